"""Edges of runs over several windows: windows whose pool a saif_only call gave
back without running them, 64-bit windows among others, launch graphs and
schedules that fit their windows, work spaces that grow, and lists read back."""
import ctypes as C

import numpy as np
import pytest

from cases import stimulus
from gls import synth
from gls.capi import GlsError, Simulator
from gls.cells import LIBRARY
from gls.levelize import assemble, default_arcs
from gls.netlist import Stimulus

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def design():
    cfg = synth.scaled(synth.CONFIGS["c1"], cells=600, cycles=200, depth=10, ppi=96)
    return cfg, synth.make_netlist(cfg, seed=41)


def test_waveform_of_a_window_whose_pool_went(design, gpu):
    """autotune(saif_only) gives every window's pool back and runs the first
    wave only: reading another window's lists is an error, not a read of the
    buffers it no longer has; its SAIF counts stay, and a run brings the lists
    back."""
    cfg, nl = design
    out = int(nl.gate_output_nets()[0])
    with Simulator() as s:
        s.load(nl)
        ids = [s.add_window(synth.make_stimulus(cfg, nl.ppi_nets, seed=50 + k), 0, cfg.t_end) for k in range(4)]
        s.run()
        saif = [s.saif(w).copy() for w in ids]
        waves = [s.waveform(out, w) for w in ids]
        s.autotune(max_wave=2, saif_only=True)
        for w in ids:
            for net in (0, out):
                with pytest.raises(GlsError, match="saif_only"):
                    s.waveform(net, w)
            assert np.array_equal(s.saif(w), saif[w])
        s.run()
        for w in ids:
            t, v = s.waveform(out, w)
            assert np.array_equal(t, waves[w][0]) and np.array_equal(v, waves[w][1])


@pytest.mark.parametrize("late", [0, 1, 2])
def test_autotune_stops_before_a_window_of_64_bit_words(late, design, gpu):
    """Windows of 64-bit event words run alone: the wave that autotune times
    ends before one, is that one when it comes first, and leaves every window
    that it ran as gls_run leaves it."""
    cfg, nl = design
    far = synth.scaled(cfg)
    far.period = 20_000_000   # times past 2^30 - 2
    wins = [far if k == late else cfg for k in range(3)]
    with Simulator() as s:
        s.load(nl)
        ids = [s.add_window(synth.make_stimulus(c, nl.ppi_nets, seed=60 + k), 0, c.t_end) for k, c in enumerate(wins)]
        assert s.autotune()["windows"] == (1 if late == 0 else late)
        ran = [w for w in ids if w < max(1, late)]
        tuned = [s.saif(w).copy() for w in ran]
        s.run()
        assert s.stats()["wide_windows"] == 1
        for w, a in zip(ran, tuned):
            assert np.array_equal(a, s.saif(w))


def test_autotune_of_windows_that_grow_past_32_bit_times(design, gpu):
    """A window whose stimulus fits 32-bit words and whose gate outputs do not
    is found by the first run of the wave, which then goes on without it."""
    cfg, nl = design
    end = 2**30 - 2
    sts = []
    for k in range(3):
        st = synth.make_stimulus(cfg, nl.ppi_nets, seed=70 + k)
        if k == 1:   # the last event of every net at the largest 32-bit time
            last = st.ev_start[1:].astype(np.int64) - 1
            st.time[last[st.ev_start[1:] - st.ev_start[:-1] > 1]] = end
        sts.append(st)
    with Simulator() as s:
        s.load(nl)
        ids = [s.add_window(st, 0, 2**30 + 10_000) for st in sts]
        assert s.autotune()["windows"] == 1
        tuned = [s.saif(w).copy() for w in ids]
        with Simulator() as r:
            r.load(nl)
            for st in sts:
                r.add_window(st, 0, 2**30 + 10_000)
            r.run()
            assert r.stats()["wide_windows"] == 1
            for w in ids:
                assert np.array_equal(tuned[w], r.saif(w))


@pytest.mark.parametrize("order", [(30, 4000), (4000, 30)])
def test_graph_of_a_wave_fits_its_windows(order, design, gpu):
    """Waves of as many windows over the same nets, one of short and one of
    long lists, through one context: each is launched as in a context of its
    own (the segment count tells the gate kernel's block sizes), and gives the
    same counts."""
    cfg, nl = design

    def wave(s, cycles):
        s.clear_windows()
        ids = [s.add_window(synth.make_stimulus(cfg, nl.ppi_nets, seed=80 + k, cycles=cycles), 0, cycles * cfg.period)
               for k in range(40)]
        s.run_batched()
        return s.stats()["segments"], [s.saif(w).copy() for w in ids]

    with Simulator() as both:
        both.load(nl)
        for cycles in order:
            segments, saif = wave(both, cycles)
            with Simulator() as alone:
                alone.load(nl)
                s0, f0 = wave(alone, cycles)
            assert segments == s0
            assert all(np.array_equal(a, b) for a, b in zip(saif, f0))


@pytest.mark.parametrize("batched", [False, True])
def test_windows_that_all_outgrow_the_work_space(batched, gpu):
    """Glitching XOR levels need far more stack space than the stimulus lets
    expect, in every one of 40 windows of a fresh context: the space grows with
    the need, not once more for every window."""
    rng = np.random.default_rng(3)
    c = LIBRARY["GEN_XOR2_D1"]
    insts, src, nn = [], list(range(24)), 24
    for _ in range(10):
        for k in range(40):
            a, b = (int(x) for x in rng.choice(src, 2, replace=False))
            insts.append((c.name, [a, b], [nn + k], default_arcs(c, float(rng.integers(2, 9)), float(rng.integers(2, 9)))))
        src, nn = list(range(nn, nn + 40)), nn + 40
    nl = assemble(insts, n_nets=nn)

    def window(seed):
        r = np.random.default_rng(seed)
        return stimulus({n: [(0, 0)] + [(1000 * e + int(r.integers(1, 900)), 0 if e % 2 else 3) for e in range(120)]
                         for n in range(24)})

    wins = [window(100 + k) for k in range(40)]
    with Simulator() as s:
        s.load(nl)
        ids = [s.add_window(st, 0, 121_000) for st in wins]
        if batched:
            s.run_batched()
        else:
            s.run()
        for w in ids[::13]:
            with Simulator() as one:
                one.load(nl)
                v = one.add_window(wins[w], 0, 121_000)
                one.run()
                assert np.array_equal(one.saif(v), s.saif(w)) and np.array_equal(one.lengths(v), s.lengths(w))


@pytest.mark.parametrize("period", [1_000, 20_000_000])
def test_first_run_of_a_context_is_its_only_one(period, gpu):
    """Two levels of XORs whose inputs never move together: the second level's
    lists are twice the stimulus', as long as the stack space is sized for.
    The first run takes no more launches than the next, whatever the segments
    add, in 32-bit and in 64-bit event words."""
    w, events = 200, 100
    c = LIBRARY["GEN_XOR2_D1"]
    insts = [(c.name, [2 * k, 2 * k + 1], [4 * w + k], default_arcs(c, 3.0, 5.0)) for k in range(2 * w)]
    insts += [(c.name, [4 * w + 2 * k, 4 * w + 2 * k + 1], [6 * w + k], default_arcs(c, 4.0, 6.0)) for k in range(w)]
    insts += [(c.name, [4 * w + 2 * k, 4 * w + (2 * k + 3) % (2 * w)], [7 * w + k], default_arcs(c, 4.0, 6.0)) for k in range(w)]
    nl = assemble(insts, n_nets=8 * w)
    st = stimulus({n: [(0, 0)] + [(period * e + period // 4 * (n % 4), 0 if e % 2 else 3) for e in range(1, events)]
                   for n in range(4 * w)})
    with Simulator() as s:
        s.load(nl)
        v = s.add_window(st, 0, period * events)
        s.run()
        first, lens = s.stats()["launches"], s.lengths(v)
        assert lens[6 * w:].min() > 3.5 * events   # the estimate's limit: two such lists a gate output of the third level
        s.run()
        assert s.stats()["launches"] == first == 3
        assert s.stats()["wide_windows"] == (1 if period > 1_000_000 else 0)


@pytest.mark.parametrize("late", [False, True])
def test_autotune_times_equal_schedules_once(late, design, gpu):
    """Schedules that make the same launches have one time, and do not replace
    each other by chance: a level in one launch knows no segments per SM and no
    class streams, a window of 64-bit words no schedule at all."""
    cfg, nl = design
    cfg = synth.scaled(cfg)
    cfg.period = 20_000_000 if late else cfg.period
    with Simulator() as s:
        s.load(nl)
        w = s.add_window(synth.make_stimulus(cfg, nl.ppi_nets, seed=90), 0, cfg.t_end)
        t = s.autotune()
        ms = [c["ms"] for c in t["candidates"]]
        assert len(ms) == 13
        assert ms[0] == ms[1] == ms[2]
        assert len(set(ms)) == 1 if late else len(set(ms)) > 1
        if t["best"]["warp_mask"] == 0 and t["best"]["flags"] == 0:
            assert t["best"]["seg_per_sm"] == 2048 and t["candidates"][9]["ms"] == ms[0]
        assert not (t["best"]["flags"] == 1 and t["best"]["warp_mask"] == 0)
        tuned = s.saif(w).copy()
        s.run()
        assert np.array_equal(tuned, s.saif(w))


def test_segment_tables_come_with_the_segment_kernels(design, gpu):
    """Waves through the gate kernel alone hold no segment tables (117 MB a
    window at least); a schedule that asks for the segment kernels brings them,
    and going from one to the other changes no result."""
    torch = pytest.importorskip("torch")
    cfg, nl = design
    sts = [synth.make_stimulus(cfg, nl.ppi_nets, seed=110 + k) for k in range(12)]
    with Simulator() as s:
        s.load(nl)
        ids = [s.add_window(st, 0, cfg.t_end) for st in sts]
        before = torch.cuda.mem_get_info()[0]
        saif = []
        for mask, batched in ((0, True), (7, True), (0, False), (2, False), (0, True)):
            s.set_schedule(2048, mask, 0)
            if batched:
                s.run_batched()
            else:
                s.run()
            if not saif:
                assert before - torch.cuda.mem_get_info()[0] < 12 * 64 << 20
            saif.append([s.saif(w).copy() for w in ids])
        for other in saif[1:]:
            assert all(np.array_equal(a, b) for a, b in zip(saif[0], other))


@pytest.mark.parametrize("base", [0, 3_000_000_000])
def test_waveforms_around_the_staged_length(base, gpu):
    """Lists around 2^16 and 2^18 events, read with their length and by a copy,
    whole and cut off, in both word sizes."""
    c = LIBRARY["GEN_BUF_D1"]
    sizes = [1, 1024, 1025, 65_535, 65_536, 65_537, 262_143, 262_144, 262_145]
    k = len(sizes)
    nl = assemble([(c.name, [j], [k + j], default_arcs(c, 3.0, 4.0)) for j in range(k)], n_nets=2 * k)
    t = np.concatenate([base + 10 * np.arange(n, dtype=np.uint64) for n in sizes]).astype(np.uint32)
    v = np.concatenate([np.where(np.arange(n) % 2, 3, 0) for n in sizes]).astype(np.uint8)
    st = Stimulus(np.arange(k, dtype=np.uint32), np.cumsum([0] + sizes).astype(np.uint64), t, v)
    with Simulator() as s:
        s.load(nl)
        w = s.add_window(st, base, base + 2_700_000)
        s.run()
        lens = s.lengths(w)
        for j, n in enumerate(sizes):
            a, b = int(st.ev_start[j]), int(st.ev_start[j + 1])
            gt, gv = s.waveform(j, w)
            assert np.array_equal(gt, t[a:b]) and np.array_equal(gv, v[a:b])
            ot, ov = s.waveform(k + j, w)
            assert len(ot) == lens[k + j] == n + 1
            assert np.array_equal(ot[1:], t[a:b] + np.where(v[a:b] == 3, 3, 4)) and np.array_equal(ov[1:], v[a:b])
            for cap in (65_535, 65_536, 65_537):   # a caller's shorter arrays
                ct, cv, got = np.zeros(cap, np.uint32), np.zeros(cap, np.uint8), C.c_uint64()
                assert s.lib.gls_waveform(s.h, w, j, ct.ctypes.data, cv.ctypes.data, cap, C.byref(got)) == 0
                m = min(cap, n)
                assert got.value == n and np.array_equal(ct[:m], t[a:a + m]) and np.array_equal(cv[:m], v[a:a + m])
                assert not ct[m:].any()
