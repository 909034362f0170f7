"""The host threads that pack stimuli: not made for one stimulus that a single
thread packs as fast as they are made, made for a large one or for many."""
import os

import numpy as np
import pytest

from gls import synth
from gls.capi import GlsError, Simulator
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


@pytest.mark.parametrize("times,code,match", [
    ([0, 2**31, 500], 1, "strictly increasing"),          # a late time before the last one
    ([0, 700, 500, 2**31], 1, "strictly increasing"),     # out of order, the last one late
    ([0, 700, 700], 1, "strictly increasing"),
    ([0, 700, 2**32 - 1], None, "beyond the largest"),
    ([0, 2**32 - 1, 5], None, "beyond the largest"),
])
def test_faulty_times_are_refused_in_words_of_either_size(times, code, match, gpu):
    nl = synth.make_netlist(synth.scaled(synth.CONFIGS["c1"], cells=50, cycles=10, depth=2, ppi=8), seed=1)
    nets = np.asarray(nl.ppi_nets, np.uint32)
    lists = [times] + [[0, 100, 200]] * (len(nets) - 1)
    start = np.cumsum([0] + [len(x) for x in lists]).astype(np.uint64)
    t = np.concatenate([np.array(x, np.uint64) for x in lists]).astype(np.uint32)
    v = np.concatenate([np.where(np.arange(len(x)) % 2, 3, 0) for x in lists]).astype(np.uint8)
    with Simulator() as s:
        s.load(nl)
        with pytest.raises(GlsError, match=match) as e:
            s.add_window(Stimulus(nets, start, t, v), 0, 2**32)
        assert code is None or e.value.code == code
