"""k_gate (one level in one launch, a block per gate output) at its edges,
bit-exact against the oracle: every block size, list lengths around the
smallest segment and around one segment per thread, gates of one to six
input nets, stack and pool space that has to grow, waves of windows."""
import numpy as np
import pytest

from cases import random_case, stimulus
from gls import synth
from gls.cells import LIBRARY, CellDef
from gls.levelize import assemble, default_arcs
from gls.capi import ALLOC_EXACT
from gpu_util import assert_same, gpu_run, simulator
from oracle.runner import run_oracle

pytestmark = pytest.mark.gpu
CELLS = ["GEN_BUF_D1", "GEN_XOR2_D1", "GEN_AND2_D1", "GEN_MUX2_D1", "GEN_OAI21_D1"]


def fan_design():
    insts, nn = [], 3
    for k, name in enumerate(CELLS * 2):
        c = LIBRARY[name]
        src = [0, 1, 2] if k < len(CELLS) else [3 + (k + p) % len(CELLS) for p in range(3)]
        insts.append((name, src[:c.n_in], [nn], default_arcs(c, 3.0 + k, 7.0 + k)))
        nn += 1
    return assemble(insts, n_nets=nn)


def even_lists(events):
    return stimulus({net: [(0, 1)] + [(20 * e + 7 * net + 5, 3 if e % 2 else 0) for e in range(events)]
                     for net in range(3)})


@pytest.mark.parametrize("events", [0, 1, 7, 15, 16, 17, 255, 1023, 5000])
@pytest.mark.parametrize("threads", [32, 64, 128, 256, 512])
def test_block_sizes(threads, events, gpu, oracle_bin):
    nl, st = fan_design(), even_lists(events)
    t_end = 20 * events + 500
    ow, osaif, _ = run_oracle(nl, st, 0, t_end)
    gw, gs, _, _ = gpu_run(nl, st, 0, t_end, env={"GLS_GATE_THREADS": str(threads)})
    assert_same(gw, gs, ow, osaif, f"{threads} threads, {events} events")


@pytest.mark.parametrize("threads", [32, 512])
@pytest.mark.parametrize("alloc", [0, 1])
def test_against_the_segment_kernels(alloc, threads, gpu):
    """A netlist with lists long enough for full blocks, in both paths; a pool
    that has to grow on the way."""
    cfg = synth.scaled(synth.CONFIGS["c1"], cells=900, cycles=2500, depth=12)
    nl = synth.make_netlist(cfg, seed=5)
    st = synth.make_stimulus(cfg, nl.ppi_nets, seed=6)
    res = []
    for env in ({"GLS_GATE": "0"}, {"GLS_GATE_THREADS": str(threads)}):
        with simulator(env=env, alloc_mode=alloc, pool_events=200_000) as s:
            s.load(nl)
            w = s.add_window(st, 300, cfg.t_end - 700)
            s.run()
            assert s.stats()["overflow_retries"] > 0
            res.append((s.saif(w), s.lengths(w), [s.waveform(int(n), w) for n in range(0, nl.n_nets, 37)]))
    assert np.array_equal(res[0][0], res[1][0]) and np.array_equal(res[0][1], res[1][1])
    for (t0, v0), (t1, v1) in zip(res[0][2], res[1][2]):
        assert np.array_equal(t0, t1) and np.array_equal(v0, v1)


@pytest.mark.parametrize("threads", [32, 256])
def test_wave_with_uneven_windows(threads, gpu, oracle_bin):
    """Windows of one wave from one event a list to thousands, gates of
    up to six input nets."""
    nl, _ = random_case(3, max_gates=16, max_in=6)
    rng = np.random.default_rng(9)
    wins = []
    for events in (1, 3, 40, 900, 4000, 2):
        d = {}
        for net in nl.ppi_nets:
            t = np.cumsum(rng.integers(1, 12, events)) if events else np.zeros(0, int)
            d[int(net)] = list(zip(t.tolist(), rng.choice([0, 3, 1], events, p=[.49, .49, .02]).tolist()))
        wins.append(stimulus(d))
    with simulator(env={"GLS_GATE_THREADS": str(threads)}, alloc_mode=ALLOC_EXACT) as s:
        s.load(nl)
        ids = [s.add_window(st, 10, 60_000) for st in wins]
        s.run_batched()
        for wid, st in zip(ids, wins):
            ow, osaif, _ = run_oracle(nl, st, 10, 60_000)
            lens = s.lengths(wid)
            gw = {n: s.waveform(n, wid) for n in range(nl.n_nets) if lens[n] != 2**32 - 1}
            assert_same(gw, s.saif(wid), ow, osaif, f"wave window {wid}")


@pytest.mark.parametrize("every", [1, 3, 40, 400])
@pytest.mark.parametrize("kept", [31, 32, 33, 64, 65, 255, 257, 513])
def test_copy_of_sparse_segments(kept, every, gpu, oracle_bin):
    """Glitch trains that a slow buffer swallows, with `every` events around
    each edge that it keeps: lists of `kept` entries from segments of which
    most keep nothing, or one entry each."""
    c = LIBRARY["GEN_BUF_D1"]
    nl = assemble([(c.name, [0], [1], default_arcs(c, 100.0, 100.0))], n_nets=2)
    ev, t, v = [(0, 0)], 0, 0
    for _ in range(kept):
        for _ in range(2 * (every // 2)):   # glitches shorter than the delay
            t, v = t + 3, 3 - v
            ev.append((t, v))
        t, v = t + 3, 3 - v
        ev.append((t, v))
        t += 500
    st = stimulus({0: ev})
    ow, osaif, _ = run_oracle(nl, st, 0, t + 50)
    for threads in ("32", "128", "256"):
        gw, gs, _, _ = gpu_run(nl, st, 0, t + 50, env={"GLS_GATE_THREADS": threads})
        assert_same(gw, gs, ow, osaif, f"{threads} threads")


@pytest.mark.parametrize("events", [2, 3, 4, 5, 6, 8, 43, 85, 86, 170, 342])
def test_smallest_segments(events, gpu, oracle_bin):
    """Lists around the smallest segment, and around one smallest segment for
    every thread of a block, in every block size and the one the rule takes."""
    nl, st = fan_design(), even_lists(events)
    t_end = 20 * events + 500
    ow, osaif, _ = run_oracle(nl, st, 0, t_end)
    for env in [{"GLS_GATE_THREADS": str(t)} for t in (32, 64, 128, 256)] + [{}]:
        gw, gs, _, _ = gpu_run(nl, st, 0, t_end, env=env)
        assert_same(gw, gs, ow, osaif, f"{env}, {events} events")


def wide_cells():
    return [CellDef(f"T_{fn.upper()}{k}", [f"a{i}" for i in range(k)], ["z"], [(fn, "z", [f"a{i}" for i in range(k)])],
                    [(2, f"a{i}", "z") for i in range(k)])
            for fn, k in (("and", 4), ("xor", 4), ("nor", 5), ("or", 6), ("xor", 6))]


@pytest.mark.parametrize("base", [0, 3_000_000_000])
@pytest.mark.parametrize("events", [3, 17, 300, 4000])
@pytest.mark.parametrize("threads", [32, 64, 256])
def test_four_to_six_input_nets(threads, events, base, gpu, oracle_bin):
    """The class of four to six input nets, in both word sizes, beside a
    level's narrower gate outputs."""
    library = {**LIBRARY, **{c.name: c for c in wide_cells()}}
    names = [c.name for c in wide_cells()] + CELLS
    rng = np.random.default_rng(events)
    insts, src, nn = [], list(range(6)), 6
    for _ in range(3):
        for k, name in enumerate(names):
            c = library[name]
            ins = [int(x) for x in rng.choice(src, c.n_in, replace=False)]
            insts.append((name, ins, [nn + k], default_arcs(c, 4.0 + k, 9.0 - k % 5)))
        src, nn = list(range(nn, nn + len(names))), nn + len(names)
    nl = assemble(insts, n_nets=nn, cells=library)
    d = {}
    for net in range(6):
        t = base + np.cumsum(rng.integers(1, 30, events))
        d[net] = list(zip(t.tolist(), rng.choice([0, 3, 1, 2], events, p=[.48, .48, .02, .02]).tolist()))
    st = stimulus(d)
    t_end = base + 30 * events + 200
    ow, osaif, _ = run_oracle(nl, st, base + 5, t_end)
    gw, gs, _, _ = gpu_run(nl, st, base + 5, t_end, env={"GLS_GATE_THREADS": str(threads)})
    assert_same(gw, gs, ow, osaif, f"{threads} threads, {events} events")
