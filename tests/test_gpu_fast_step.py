"""The gate kernels' fast step (known input values, packed delays) at the
edges where it hands over to the general one, bit-exact against the oracle:
delays around the largest packed one (2^16 - 2), times around the last one
with room for a packed delay, X and Z inside a list, repeated values, missing
arcs, and segments down to a few events."""
import numpy as np
import pytest

from cases import stimulus
from gls.cells import LIBRARY
from gls.levelize import assemble
from gpu_util import assert_same, gpu_run
from oracle.runner import run_oracle

pytestmark = pytest.mark.gpu

NARROW_MAX = (1 << 30) - 2
CELLS = ["GEN_INV_D1", "GEN_NAND2_D1", "GEN_XOR2_D1", "GEN_MUX2_D1", "GEN_AOI21_D1", "GEN_NOR3_D1"]


def design(delays, drop_arcs=()):
    """Every cell on three stimulus nets, then a second level on the first
    one's outputs; delays are taken round robin."""
    insts, k, nn = [], 0, 3
    for level in range(2):
        src = [0, 1, 2] if level == 0 else list(range(3, 3 + len(CELLS)))
        for i, name in enumerate(CELLS):
            c = LIBRARY[name]
            arcs = []
            for n, (e, ip, op) in enumerate(c.arcs):
                arcs.append((e, ip, op, float(delays[k % len(delays)]), float(delays[(k + 1) % len(delays)])))
                k += 1
            if i in drop_arcs:
                arcs = [] if i % 2 else arcs[:-1]
            insts.append((name, [src[(i + p) % len(src)] for p in range(c.n_in)], [nn], arcs))
            nn += 1
    return assemble(insts, n_nets=nn)


def lists(seed, base, events, xz):
    rng = np.random.default_rng(seed)
    d = {}
    for net in range(3):
        t = np.cumsum(rng.integers(1, 9, events)) + base
        v = rng.choice([0, 3], events) if xz == "repeats" else np.where(np.arange(events) % 2 == net % 2, 0, 3)
        if xz in ("x", "repeats"):
            at = rng.integers(0, events, 4)
            v[at] = rng.choice([1, 2], 4)
        d[net] = list(zip(t.tolist(), v.tolist()))
    return stimulus(d)


@pytest.mark.parametrize("seg", [8, 33, 0])
@pytest.mark.parametrize("xz", ["none", "x", "repeats"])
@pytest.mark.parametrize("delays", [(1, 5, 17), (65533, 65534, 3), (65534, 65535, 2), (0, 4, 9)])
def test_fast_step_delays(delays, xz, seg, gpu, oracle_bin):
    nl = design(delays)
    st = lists(len(delays) + seg, 1, 700, xz)
    ow, osaif, _ = run_oracle(nl, st, 0, 300_000)
    gw, gs, _, _ = gpu_run(nl, st, 0, 300_000, seg=seg)
    assert_same(gw, gs, ow, osaif, f"delays {delays} {xz} seg {seg}")


@pytest.mark.parametrize("drop", [(0, 2, 4), (1, 3, 5), (0, 1, 2, 3, 4, 5)])
def test_fast_step_missing_arcs(drop, gpu, oracle_bin):
    nl = design((3, 11, 6), drop)
    st = lists(7, 0, 500, "x")
    ow, osaif, _ = run_oracle(nl, st, 0, 10_000)
    gw, gs, _, _ = gpu_run(nl, st, 0, 10_000, seg=16)
    assert_same(gw, gs, ow, osaif, f"missing arcs {drop}")


@pytest.mark.parametrize("off", [-200_000, -70_000, -66_000, -65_536, -4_000])
def test_fast_step_late_times(off, gpu, oracle_bin):
    """The lists end around the last time with room for a packed delay; the
    narrow words still hold every output."""
    nl = design((2, 9, 14))
    st = lists(11, NARROW_MAX + off - 3_500, 600, "none")
    ow, osaif, _ = run_oracle(nl, st, 0, 1 << 31)
    assert max(int(np.max(t)) for t, _ in ow.values()) <= NARROW_MAX
    gw, gs, _, stats = gpu_run(nl, st, 0, 1 << 31, seg=16)
    assert stats["wide_windows"] == 0
    assert_same(gw, gs, ow, osaif, f"late times {off}")
