"""Net tables rebuilt on the device before each run, waveforms read with their
length in one launch, and VCD results that are views of the library's memory."""
import ctypes as C
import gc

import numpy as np
import pytest

from cases import random_case, standard_vcd
from gls.capi import Simulator, vcd_scan
from gls.cells import LIBRARY
from gls.levelize import assemble
from gls.netlist import Stimulus
from gpu_util import assert_same
from oracle.runner import run_oracle

pytestmark = pytest.mark.gpu

INLINE = 1 << 18   # events that one launch reads; 1024 are read without knowing the length


@pytest.mark.parametrize("base", [0, 3_000_000_000])
@pytest.mark.parametrize("n", [0, 1, 1023, 1024, 1025, INLINE - 1, INLINE, INLINE + 1, 3 * INLINE])
def test_waveform_read_at_every_length(n, base, gpu):
    """The stimulus' own lists come back as they went in, whole and cut short."""
    inv = LIBRARY["GEN_INV_D1"]
    arcs = [(e, i, o, 5.0, 5.0) for e, i, o in inv.arcs]
    nl = assemble([(inv.name, [k], [2 + k], arcs) for k in range(2)], n_nets=4)
    rng = np.random.default_rng(n)
    t = base + np.cumsum(rng.integers(1, 4, n), dtype=np.int64)
    v = rng.choice([0, 1, 2, 3], n).astype(np.uint8)
    t1, v1 = np.append(t, t[-1:] + 1 if n else [base]), np.append(v, 3).astype(np.uint8)   # one event more
    st = Stimulus(np.array([0, 1], np.uint32), np.array([0, n, 2 * n + 1], np.uint64),
                  np.concatenate([t, t1]).astype(np.uint32), np.concatenate([v, v1]))
    with Simulator() as s:
        s.load(nl)
        w = s.add_window(st, 0, 1 << 33)
        s.run()
        for net, time, val in ((0, t, v), (1, t1, v1)):
            gt, gv = s.waveform(net, w)
            assert np.array_equal(gt, time.astype(np.uint32)) and np.array_equal(gv, val)
        for cap in {0, min(n, 5), n}:
            got, gt = C.c_uint64(), np.full(cap + 1, 77, np.uint32)
            assert s.lib.gls_waveform(s.h, w, 0, gt.ctypes.data_as(C.c_void_p), None, cap, C.byref(got)) == 0
            assert got.value == n and gt[cap] == 77 and np.array_equal(gt[:cap], t[:cap].astype(np.uint32))


@pytest.mark.parametrize("batched", [False, True])
def test_tables_rebuilt_for_each_run(batched, gpu, oracle_bin):
    """One context over netlists and stimuli of other sizes, two runs each:
    nothing of the run before is left in the tables."""
    with Simulator() as s:
        for seed in (910, 911, 912, 910):
            nl, st = random_case(seed, max_gates=300 if seed == 911 else 20, max_in=9, horizon=3000, max_events=300)
            k = len(st.nets)   # one event per net
            few = Stimulus(st.nets, np.arange(k + 1, dtype=np.uint64), np.full(k, 7, np.uint32), np.zeros(k, np.uint8))
            want = [(x, run_oracle(nl, x, 0, 3500)[:2]) for x in (st, few, st)]
            s.load(nl)
            for k in (3, 1):
                s.clear_windows()
                for x, _ in want[:k]:
                    s.add_window(x, 0, 3500)
                for _ in range(2):
                    s.run_batched() if batched else s.run()
                    for w, (_, (ow, osaif)) in enumerate(want[:k]):
                        assert_same({n: s.waveform(n, w) for n in ow}, s.saif(w), ow, osaif, f"seed {seed} window {w}")


def test_vcd_arrays_outlive_the_others(gpu):
    body = standard_vcd(5).split("$enddefinitions $end", 1)[1].encode()
    codes = {c: [([k], False)] for k, c in enumerate("!\"#$%&'()*+,")}
    first = vcd_scan(body, codes)
    want = [a.copy() for a in first[:4]]
    assert want[0].size > 100
    for keep in range(4):
        arr = vcd_scan(body, codes)[keep]
        gc.collect()
        vcd_scan(body, codes)
        assert np.array_equal(arr, want[keep]) and arr.flags.writeable
    with pytest.raises(TypeError):
        vcd_scan(bytearray(body), codes)
