"""The host threads that pack stimuli: not made for one stimulus that a single
thread packs as fast as they are made, made for a large one or for many."""
import os

import numpy as np
import pytest

from gls import synth
from gls.capi import Simulator
from gls.netlist import Stimulus

pytestmark = pytest.mark.gpu


def threads():
    with open("/proc/self/status") as f:
        return next(int(line.split()[1]) for line in f if line.startswith("Threads:"))


def stim(nets, events):
    n = max(1, events // len(nets))
    return Stimulus(np.asarray(nets, np.uint32), (np.arange(len(nets) + 1) * n).astype(np.uint64),
                    np.tile(np.arange(n, dtype=np.uint32) * 50, len(nets)),
                    np.tile(np.where(np.arange(n) % 2, 3, 0).astype(np.uint8), len(nets))), 50 * n + 100


def test_threads_are_made_when_they_pay(gpu):
    nl = synth.make_netlist(synth.scaled(synth.CONFIGS["c1"], cells=200, cycles=10, depth=4, ppi=512), seed=1)
    results = []
    for sizes in ([200_000] * 8, [1_300_000, 200_000]):
        with Simulator() as s:
            s.load(nl)
            made = []
            for events in sizes:
                st, t_end = stim(nl.ppi_nets, events)
                s.clear_windows()
                before = threads()
                w = s.add_window(st, 0, t_end)
                made.append(threads() - before)
            s.run()
            results.append(s.saif(w).copy())
        assert made[0] == (0 if sizes[0] < 2**20 else max(made))
        assert sum(x > 0 for x in made) <= 1
        if len(sizes) > 5 and (os.cpu_count() or 1) > 1:
            assert sum(made[:5]) == 0 and max(made) > 0   # 1.0 M events alone, then the threads
    assert np.array_equal(results[0], results[1])
