"""The gate kernel's block size: chosen by the lists that are there (the
segment count tells it), and right, against the oracle, at the largest blocks
of each class and word size."""
import numpy as np
import pytest

from cases import stimulus
from gls import synth
from gls.capi import MLP_PARAMS, Simulator
from gls.cells import LIBRARY
from gls.levelize import assemble, default_arcs
from gpu_util import assert_same, gpu_run, simulator
from oracle.runner import run_oracle
from test_gpu_gate_kernel import CELLS, even_lists, fan_design, wide_cells

pytestmark = pytest.mark.gpu
WIDE = {**LIBRARY, **{c.name: c for c in wide_cells()}}


def segments(threads, events):
    """Segments of a gate output of so many fan-in events in such a block."""
    per = max(4, -(-events // threads))
    return -(-events // per)


def level_of(gates, cells=LIBRARY):
    """One level: (cell, input nets) per gate output, nets numbered behind them."""
    first = 1 + max(max(src) for _, src in gates)
    insts = [(name, src, [first + k], default_arcs(cells[name], 3.0 + k % 5, 6.0)) for k, (name, src) in enumerate(gates)]
    return assemble(insts, n_nets=first + len(gates), cells=cells)


def ticks(events, step=20, base=0):
    return [(base + step * e, 3 if e % 2 else 0) for e in range(events)]


@pytest.mark.parametrize("events,threads", [(60_000, 512), (2_000, 128), (40, 32)])
def test_a_busy_gate_output_among_quiet_ones(events, threads, gpu, oracle_bin):
    """3,000 buffers of eight events and one of many: a level lasts as long as
    the busy one, whose list decides the block, not the mean list."""
    n = 3_000
    nl = level_of([("GEN_BUF_D1", [k]) for k in range(n + 1)])
    st = stimulus({k: ticks(events if k == n // 2 else 8) for k in range(n + 1)})
    t_end = 20 * events + 400
    gw, gs, _, stats = gpu_run(nl, st, 0, t_end)
    assert stats["segments"] == n * segments(threads, 8) + segments(threads, events)
    ow, osaif, _ = run_oracle(nl, st, 0, t_end)
    assert_same(gw, gs, ow, osaif, f"{events} events")


def test_busy_gate_outputs_among_too_many_quiet_ones(gpu, oracle_bin):
    """24,000 quiet buffers and eight busy ones: blocks that would fit the busy
    ones cost the quiet ones more than they save, and the run takes the segment
    kernels (more than one launch for the level)."""
    n = 24_000
    nl = level_of([("GEN_BUF_D1", [k]) for k in range(n + 8)])
    d = {k: ticks(3_000 if k >= n else 8) for k in range(n + 8)}
    launches = []
    for st in (stimulus(d), stimulus({**d, **{k: ticks(8) for k in range(n, n + 8)}})):
        ow, osaif, _ = run_oracle(nl, st, 0, 70_000)
        some = list(range(n - 3, n + 8)) + list(range(2 * n + 5, 2 * n + 16))
        gw, gs, _, stats = gpu_run(nl, st, 0, 70_000, nets=some)
        assert_same(gw, gs, {k: ow[k] for k in some if k in ow}, osaif, "busy among quiet")
        launches.append(stats["launches"])
    assert launches[0] > 4 and launches[1] == 2


@pytest.mark.parametrize("use_graph", [False, True])
@pytest.mark.parametrize("alloc", [0, 1, 2])
def test_wave_of_busy_among_quiet(alloc, use_graph, gpu, oracle_bin):
    """The same as a wave of windows, in every allocation mode, between waves
    that take the gate kernel."""
    n = 8_000
    nl = level_of([("GEN_BUF_D1", [k]) for k in range(n + 3)])
    quiet = {k: ticks(8) for k in range(n + 3)}
    wins = [stimulus({**quiet, **{k: ticks(3_000 - 100 * w) for k in range(n, n + 3)}}) for w in range(3)]
    model = np.zeros(MLP_PARAMS, np.float32)
    model[-1] = 3.0
    with Simulator(alloc_mode=alloc) as s:
        if alloc == 2:
            s.set_presize_model(model)
        s.load(nl)
        launches = []
        for sts in ([stimulus(quiet)] * 3, wins, [stimulus(quiet)] * 3, wins):
            s.clear_windows()
            ids = [s.add_window(st, 0, 70_000) for st in sts]
            s.run_batched(use_graph=use_graph)
            launches.append(s.stats()["launches"])
        assert launches[0] == launches[2] <= 3 and launches[1] == launches[3] > 4
        for w, st in zip(ids, wins):
            ow, osaif, _ = run_oracle(nl, st, 0, 70_000)
            some = list(range(n - 2, n + 3)) + list(range(2 * n + 1, 2 * n + 6))
            assert_same({k: s.waveform(k, w) for k in some}, s.saif(w), {k: ow[k] for k in some}, osaif, f"window {w}")


def test_a_net_that_no_gate_reads_decides_nothing(gpu):
    """A long list that feeds no gate (a clock of registers alone) leaves the
    blocks as they are without it."""
    n = 3_000
    buf = LIBRARY["GEN_BUF_D1"]
    nl = assemble([(buf.name, [k], [n + 1 + k], default_arcs(buf, 3.0 + k % 5, 6.0)) for k in range(n)],
                  n_nets=2 * n + 1)   # net n is read by no gate
    d = {k: ticks(8) for k in range(n)}
    count = []
    for lists in (d, {**d, n: ticks(60_000)}):
        with Simulator() as s:
            s.load(nl)
            s.add_window(stimulus(lists), 0, 1_300_000)
            s.run()
            count.append(s.stats()["segments"])
    assert count == [n * segments(32, 8)] * 2


def test_wide_gate_outputs_take_the_largest_blocks(gpu, oracle_bin):
    """Few gate outputs of six input nets beside others: their class takes 768
    threads, by its own number of gate outputs."""
    rng = np.random.default_rng(4)
    six, n = 40, 2_000
    gates = [("GEN_AND2_D1", [int(x) for x in rng.choice(12, 2, replace=False)]) for _ in range(n)]
    gates += [("T_XOR6", [int(x) for x in rng.choice(12, 6, replace=False)]) for _ in range(six)]
    nl = level_of(gates, WIDE)
    events = 2_400
    st = stimulus({k: ticks(events, 30, k) for k in range(12)})
    t_end = 30 * events + 400
    gw, gs, _, stats = gpu_run(nl, st, 0, t_end, nets=range(nl.n_nets - 60, nl.n_nets))
    narrow = stats["segments"] - six * segments(768, 6 * events)
    assert narrow % n == 0 and narrow // n in [segments(t, 2 * events) for t in (32, 64, 128, 256, 512)]
    ow, osaif, _ = run_oracle(nl, st, 0, t_end)
    assert_same(gw, gs, {k: w for k, w in ow.items() if k >= nl.n_nets - 60}, osaif, "six input nets")


@pytest.mark.parametrize("base", [0, 3_000_000_000])
@pytest.mark.parametrize("events", [511, 512, 513, 1_300, 9_000])
@pytest.mark.parametrize("threads", [512, 768])
def test_largest_blocks(threads, events, base, gpu, oracle_bin):
    """Lists around a segment for every thread of the largest blocks, one to
    six input nets, both word sizes (whose widest blocks are smaller)."""
    names = [c.name for c in wide_cells()] + CELLS
    rng = np.random.default_rng(events)
    insts, src, nn = [], list(range(6)), 6
    for _ in range(2):
        for k, name in enumerate(names):
            c = WIDE[name]
            ins = [int(x) for x in rng.choice(src, c.n_in, replace=False)]
            insts.append((name, ins, [nn + k], default_arcs(c, 4.0 + k, 9.0 - k % 5)))
        src, nn = list(range(nn, nn + len(names))), nn + len(names)
    nl = assemble(insts, n_nets=nn, cells=WIDE)
    d = {}
    for net in range(6):
        t = base + np.cumsum(rng.integers(1, 30, events))
        d[net] = list(zip(t.tolist(), rng.choice([0, 3, 1, 2], events, p=[.49, .49, .01, .01]).tolist()))
    st = stimulus(d)
    t_end = base + 30 * events + 200
    ow, osaif, _ = run_oracle(nl, st, base + 5, t_end)
    gw, gs, _, _ = gpu_run(nl, st, base + 5, t_end, env={"GLS_GATE_THREADS": str(threads)})
    assert_same(gw, gs, ow, osaif, f"{threads} threads, {events} events")


def test_wave_in_the_largest_blocks(gpu, oracle_bin):
    """Windows of one wave, one of which has a busy net."""
    nl = fan_design()
    wins = [even_lists(e) for e in (4, 20_000, 300)]
    with simulator() as s:
        s.load(nl)
        ids = [s.add_window(st, 0, 401_000) for st in wins]
        s.run_batched()
        for w, st in zip(ids, wins):
            ow, osaif, _ = run_oracle(nl, st, 0, 401_000)
            lens = s.lengths(w)
            gw = {n: s.waveform(n, w) for n in range(nl.n_nets) if lens[n] != 2**32 - 1}
            assert_same(gw, s.saif(w), ow, osaif, f"window {w}")


@pytest.mark.parametrize("threads", [32, 64, 128, 256, 512])
@pytest.mark.parametrize("alloc", [0, 1, 2])
def test_every_block_against_the_segment_kernels(alloc, threads, gpu):
    """Every size and allocation mode with a pool that grows on the way; in the
    learned one lists outgrow their predicted slots."""
    cfg = synth.scaled(synth.CONFIGS["c1"], cells=900, cycles=2500, depth=12)
    nl = synth.make_netlist(cfg, seed=15)
    st = synth.make_stimulus(cfg, nl.ppi_nets, seed=16)
    model = np.zeros(MLP_PARAMS, np.float32)
    model[-1] = 3.0   # some 20 events a list
    res = []
    for env in ({"GLS_GATE": "0"}, {"GLS_GATE_THREADS": str(threads)}):
        with simulator(env=env, alloc_mode=alloc, pool_events=200_000) as s:
            if alloc == 2:
                s.set_presize_model(model)
            s.load(nl)
            w = s.add_window(st, 300, cfg.t_end - 700)
            s.run()
            assert s.stats()["overflow_retries"] > 0
            if alloc == 2:
                assert s.stats()["presize_overflows"] > 0
            res.append((s.saif(w), s.lengths(w), [s.waveform(int(n), w) for n in range(0, nl.n_nets, 29)]))
    assert np.array_equal(res[0][0], res[1][0]) and np.array_equal(res[0][1], res[1][1])
    for (t0, v0), (t1, v1) in zip(res[0][2], res[1][2]):
        assert np.array_equal(t0, t1) and np.array_equal(v0, v1)
