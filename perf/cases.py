"""Performance cases of the framework: what users have it do, through its
public Python entry points, at sizes from a first look to a large design.

Kinds of case:
  window    one stimulus window: the change lists of the undriven nets (host
            arrays, as a VCD reader leaves them) go in, every level is
            simulated, the SAIF counts and list lengths come back
  batch     many windows of one design in waves, SAIF only
  vcd       the body of a VCD text scanned into bit changes
  levelize  Kahn levels of an instance graph given in file order
  grad      loss and gradient of the presize network over one minibatch
"""
from __future__ import annotations

import sys
from pathlib import Path

import numpy as np

sys.path.insert(0, str(Path(__file__).resolve().parent.parent / "gate-level-simulator_gb300"))

from gls import capi, presize, synth  # noqa: E402
from gls.netlist import Stimulus  # noqa: E402

ALLOC = {"bound": capi.ALLOC_BOUND, "exact": capi.ALLOC_EXACT, "learned": capi.ALLOC_LEARNED}
CALC = {"fixed": capi.CALC_FIXED, "literal": capi.CALC_LITERAL}


def _window(shape, cells, depth, ppi, cycles, alloc="bound", calc="fixed", period=1000, dump=0):
    """shape names the generator (its toggle rates and fan-out); dump: that
    many nets' waveforms are read back too."""
    return {"kind": "window", "shape": shape, "cells": cells, "depth": depth, "ppi": ppi, "cycles": cycles,
            "alloc": alloc, "calc": calc, "period": period, "dump": dump}


def _batch(shape, cells, depth, ppi, windows, lo, hi):
    return {"kind": "batch", "shape": shape, "cells": cells, "depth": depth, "ppi": ppi, "windows": windows,
            "lo": lo, "hi": hi}


def listed():
    return [
        # the small configuration, as a first look or a unit-level block has
        # it: 20 levels of 100 gates, where launches and latency count; the
        # user also looks at some nets' waveforms
        dict(_window("c1", 2_000, 20, 192, 1_000, dump=16), name="small"),
        # the medium configuration in full: an ordinary block-level run with
        # the default options
        dict(_window("c2", 200_000, 60, 4_096, 10_000), name="medium"),
        # a block of odd sizes in the exact allocation
        dict(_window("c2", 37_501, 47, 1_777, 3_333, alloc="exact"), name="odd-exact"),
        # the shipped calc semantics (a user comparing with the reference's
        # own tool): many outputs stay X
        dict(_window("c2", 20_011, 31, 1_024, 2_003, calc="literal"), name="literal"),
        # the large design (2 M cells, 120 levels) over a quarter of its
        # stimulus, with the learned allocation: wide levels
        dict(_window("c3", 2_000_000, 120, 65_536, 5_000, alloc="learned"), name="large-learned"),
        # long change lists on a mid-size design: few gates, many events each
        dict(_window("c3", 200_000, 60, 16_384, 20_000, alloc="exact"), name="long-exact"),
        # times past 2^30 time units (a 2 us period in ps): 64-bit event words
        dict(_window("c2", 20_000, 30, 1_024, 2_000, period=2_000_000), name="late-times"),
        # several windows of the medium netlist for power analysis, SAIF only
        dict(_batch("c2", 200_000, 60, 4_096, 8, 500, 2_000), name="batch-medium"),
        # many short windows of a small block (a regression's test vectors)
        dict(_batch("c1", 2_000, 20, 192, 48, 100, 1_000), name="batch-small"),
        # a simulator's VCD text: 4,096 scalars and 64 buses
        {"kind": "vcd", "scalars": 4_096, "buses": 64, "cycles": 3_000, "rate": 0.2, "name": "vcd"},
        # the medium design's instances in file order
        {"kind": "levelize", "cells": 200_000, "depth": 60, "ppi": 4_096, "name": "levelize"},
        # one minibatch of the presize network's training, default batch
        {"kind": "grad", "rows": 8_192, "name": "presize-grad"},
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(lo * (hi / lo) ** rng.random()))

    kind = rng.choice(["window"] * 7 + ["batch"] * 2 + ["vcd", "levelize", "grad"])
    if kind == "window":
        cells = log(300, 200_000)
        depth = min(log(6, 120), max(6, cells // 20))
        ppi = log(64, 4_096)
        # at most the medium configuration's gate-cycles
        cycles = min(log(100, 20_000), 2_000_000_000 // cells)
        late = rng.random() < 0.12 and cells <= 40_000
        return _window(rng.choice(["c1", "c2", "c3"]), cells, depth, ppi, min(cycles, 2_000) if late else cycles,
                       alloc=rng.choice(["bound", "exact", "learned"]),
                       calc="literal" if rng.random() < 0.1 else "fixed", period=2_000_000 if late else 1_000,
                       dump=rng.choice([0, 0, 16]))
    if kind == "batch":
        cells = log(300, 100_000)
        hi = min(log(150, 2_000), 100_000_000 // cells)
        return _batch(rng.choice(["c1", "c2"]), cells, min(log(6, 60), max(6, cells // 20)), log(64, 1_024),
                      log(2, 48), max(100, hi // 8), max(110, hi))
    if kind == "vcd":
        return {"kind": "vcd", "scalars": log(16, 4_096), "buses": log(1, 64), "cycles": log(100, 3_000),
                "rate": round(rng.uniform(0.02, 0.4), 3)}
    if kind == "levelize":
        cells = log(300, 400_000)
        return {"kind": "levelize", "cells": cells, "depth": min(log(6, 120), max(6, cells // 20)),
                "ppi": log(64, 4_096)}
    return {"kind": "grad", "rows": log(64, 65_536)}


def _design(case, seed):
    cfg = synth.scaled(synth.CONFIGS[case["shape"]], cells=case["cells"], depth=case["depth"], ppi=case["ppi"],
                       cycles=case.get("cycles", case.get("hi")))
    cfg.period = case.get("period", cfg.period)
    return cfg, synth.make_netlist(cfg, seed=seed)


def _simulator(alloc, calc="fixed"):
    sim = capi.Simulator(alloc_mode=ALLOC[alloc], calc_mode=CALC[calc])
    if alloc == "learned":
        sim.set_presize_model(*presize.load(presize.DEFAULT_MODEL))
    return sim


# two printable characters per identifier code, clear of '$' and '#'
_CODE = [a + b for a in "ABCDEFGHIJKLMNOPQRSTUVWXYZabcdefghijklmnopqrstuvwxyz%&" for b in
         "!\"%&'()*+,-./0123456789:;<=>?@ABCDEFGHIJKLMNOPQRSTUVWXYZ[\\]^_`abcdefghijklmnopqrstuvwxyz{|}~"]
_BUS = 8   # bits per bus


def _vcd_text(case, seed):
    rng = np.random.default_rng(seed)
    ns, nb, cycles = case["scalars"], case["buses"], case["cycles"]
    code = np.array([[ord(c) for c in s] for s in _CODE[:ns + nb]], np.uint8)
    pieces = []
    cur = rng.integers(0, 2, ns).astype(np.uint8)
    for c in range(cycles):
        pieces.append(b"#%d\n" % (c * 1000))
        ch = np.arange(ns) if c == 0 else np.sort(rng.choice(ns, max(1, int(case["rate"] * ns)), replace=False))
        if c:
            cur[ch] ^= 1
        line = np.empty((len(ch), 4), np.uint8)
        line[:, 0] = 48 + cur[ch]
        if c == 0:
            line[rng.random(ns) < 0.01, 0] = ord("x")
        line[:, 1:3] = code[ch]
        line[:, 3] = 10
        pieces.append(line.tobytes())
        bs = np.arange(nb) if c == 0 else np.sort(rng.choice(nb, (nb + 1) // 2, replace=False))
        line = np.empty((len(bs), _BUS + 5), np.uint8)
        line[:, 0] = ord("b")
        line[:, 1:_BUS + 1] = 48 + rng.integers(0, 2, (len(bs), _BUS))
        line[:, _BUS + 1] = 32
        line[:, _BUS + 2:_BUS + 4] = code[ns + bs]
        line[:, -1] = 10
        pieces.append(line.tobytes())
    codes = {_CODE[k]: [([k], False)] for k in range(ns)}
    for k in range(nb):
        first = ns + k * _BUS
        codes[_CODE[ns + k]] = [(list(range(first, first + _BUS)), True)]
    return b"".join(pieces), codes


def _grad_inputs(rows, seed):
    """Feature rows of the presize network as a design gives them (cell one-hot,
    log list lengths, delays), targets and the network's parameters."""
    rng = np.random.default_rng(seed)
    f = np.zeros((rows, capi.MLP_IN), np.float32)
    cell = rng.integers(0, 13, rows)
    f[np.arange(rows), cell] = 1.0
    n_in = 1 + (cell >= 2) + (cell >= 10)
    f[:, 13] = f[:, 14] = n_in / 6.0
    ev = np.log1p(rng.integers(10, 10_000, (rows, 3))) / 12.0
    for k in range(3):
        f[:, 15 + k] = np.where(n_in > k, ev[:, k], 0.0)
    f[:, 18] = f[:, 15:18].max(1) * 1.05
    f[:, 19] = f[:, 15:18].max(1)
    f[:, 20] = f[:, 15]
    f[:, 21] = f[:, 18] * rng.uniform(0.5, 1.0, rows)
    f[:, 22:24] = rng.random((rows, 2))
    f[:, 24:28] = rng.uniform(0.05, 0.8, (rows, 4))
    f[:, 28] = np.log1p(rng.geometric(0.45, rows)) / 6.0
    f[:, 29] = rng.random(rows)
    f[:, 30:32] = 1.0
    target = (f[:, 21] * 12.0 + rng.normal(0.0, 0.3, rows)).astype(np.float32)
    h, i = capi.MLP_HID, capi.MLP_IN
    p = np.concatenate([rng.uniform(-1, 1, h * i) * (6.0 / i) ** 0.5, rng.uniform(-0.1, 0.1, h),
                        rng.uniform(-1, 1, h * h) * (6.0 / h) ** 0.5, rng.uniform(-0.1, 0.1, h),
                        rng.uniform(-1, 1, h) * (6.0 / h) ** 0.5, [5.0]]).astype(np.float32)
    return f, target, p


def prepare(case, seed):
    kind = case["kind"]
    if kind == "window":
        cfg, nl = _design(case, seed)
        sim = _simulator(case["alloc"], case["calc"])
        sim.load(nl)
        nets = np.linspace(0, nl.n_nets - 1, case["dump"]).astype(np.int64).tolist() if case["dump"] else []
        return {"kind": kind, "sim": sim, "stim": synth.make_stimulus(cfg, nl.ppi_nets, seed=seed + 1),
                "t_end": cfg.t_end, "dump": nets, "waves": np.zeros((2, case["dump"], 8 * case["cycles"] + 64), np.int64)}
    if kind == "batch":
        cfg, nl = _design(case, seed)
        rng = np.random.default_rng(seed + 2)
        cycles = rng.integers(case["lo"], case["hi"] + 1, case["windows"])
        sim = _simulator("learned")
        sim.load(nl)
        return {"kind": kind, "sim": sim,
                "windows": [(synth.make_stimulus(cfg, nl.ppi_nets, seed=seed + 10 + k, cycles=int(c)),
                             int(c) * cfg.period) for k, c in enumerate(cycles)]}
    if kind == "vcd":
        body, codes = _vcd_text(case, seed)
        return {"kind": kind, "body": body, "codes": codes}
    if kind == "levelize":
        cfg, nl = _design(dict(case, shape="c2", cycles=1), seed)
        n = nl.n_inst
        driver = np.full(nl.n_nets, -1, np.int64)
        n_in = np.array([c.n_in for c in nl.cells], np.int64)[nl.inst_cell]
        place = np.random.default_rng(seed + 3).permutation(n)      # file position of every instance
        start = nl.pin_start[:-1].astype(np.int64)
        driver[nl.pin_net[start + n_in]] = place
        pin_owner = np.repeat(np.arange(n), n_in + 1)
        is_in = np.ones(len(pin_owner), bool)
        is_in[start + n_in] = False
        pred = driver[nl.pin_net[is_in]]
        owner = place[pin_owner[is_in]]
        owner, pred = owner[pred >= 0], pred[pred >= 0]
        by = np.argsort(owner, kind="stable")
        ps = np.zeros(n + 1, np.uint64)
        np.cumsum(np.bincount(owner, minlength=n), out=ps[1:])
        return {"kind": kind, "pred_start": ps, "pred": pred[by].astype(np.uint32)}
    f, t, p = _grad_inputs(case["rows"], seed)
    tr = capi.Trainer(seed=0)
    tr.set_data(f, t)
    tr.set_params(p)
    return {"kind": "grad", "trainer": tr, "rows": case["rows"]}


def run(state):
    kind = state["kind"]
    if kind == "window":
        sim = state["sim"]
        sim.clear_windows()
        w = sim.add_window(state["stim"], 0, state["t_end"])
        sim.run()
        saif, lengths = sim.saif(w).view(np.int64), sim.lengths(w).view(np.int32)
        if not state["dump"]:
            return {"saif": saif, "lengths": lengths}
        waves = state["waves"]   # a table of the nets looked at, a row each
        for k, net in enumerate(state["dump"]):
            time, value = sim.waveform(net, w)
            waves[0, k, :len(time)], waves[1, k, :len(time)] = time, value
            waves[:, k, len(time):] = -1
        return {"saif": saif, "lengths": lengths, "waves": waves}
    if kind == "batch":
        sim = state["sim"]
        sim.clear_windows()
        for st, t_end in state["windows"]:
            sim.add_window(st, 0, t_end)
        sim.run_batched(saif_only=True)
        return [sim.saif(k).view(np.int64) for k in range(len(state["windows"]))]
    if kind == "vcd":
        signal, time, value, bus, fallback = capi.vcd_scan(state["body"], state["codes"])
        return {"signal": signal.view(np.int32), "time": time.view(np.int64), "value": value, "bus": bus,
                "fallback": fallback}
    if kind == "levelize":
        order, level_start = capi.levelize_gpu(state["pred_start"], state["pred"])
        return {"order": order.view(np.int32), "level_start": level_start.view(np.int32)}
    grad, loss = state["trainer"].grad(0, state["rows"])
    return {"grad": grad, "loss": loss}


# mean events per gate output and cycle of the synthetic designs (0.31 to 0.53
# from 30 to 120 levels), and per stimulus net and cycle
_OUT_RATE = 0.35
_STIM_RATE = {"c1": 0.2, "c2": 0.2, "c3": 0.125}


def work(case):
    kind = case["kind"]
    if kind in ("window", "batch"):
        cycles = case["cycles"] if kind == "window" else case["windows"] * (case["lo"] + case["hi"]) / 2
        wins = 1 if kind == "window" else case["windows"]
        stim = case["ppi"] * (wins + _STIM_RATE[case["shape"]] * cycles)
        outs = case["cells"] * (wins + _OUT_RATE * cycles)
        nets = (case["cells"] + case["ppi"]) * wins
        word = 8 if case.get("period", 1000) > 1_000_000 else 4
        # host stimulus at 5 bytes an event, every gate output's list once,
        # the netlist, SAIF rows and lengths
        return {"bytes": 5 * stim + word * outs + 64 * case["cells"] + 28 * nets, "flops": 0}
    if kind == "vcd":
        scal = case["scalars"] * (1 + case["rate"] * case["cycles"])
        bus = case["buses"] * (1 + 0.5 * case["cycles"])
        return {"bytes": 4 * scal + 13 * bus + 14 * (scal + _BUS * bus), "flops": 0}
    if kind == "levelize":
        return {"bytes": case["cells"] * (8 + 4 * 2.1 + 4), "flops": 0}
    h, i = capi.MLP_HID, capi.MLP_IN
    return {"bytes": 4 * (case["rows"] * (i + 1) + 2 * capi.MLP_PARAMS),
            "flops": 2 * case["rows"] * (2 * h * i + 3 * h * h + 3 * h)}


def exact(case, seed):
    """Only the network's gradient is a computed number; everything else is
    whole numbers."""
    if case["kind"] != "grad":
        return None
    f, t, p = _grad_inputs(case["rows"], seed)
    h, i = capi.MLP_HID, capi.MLP_IN
    x, t, p = f.astype(np.float64), t.astype(np.float64), p.astype(np.float64)
    cut = np.cumsum([h * i, h, h * h, h, h])
    w1, b1, w2, b2, w3, b3 = np.split(p, cut)
    w1, w2 = w1.reshape(h, i), w2.reshape(h, h)
    z1 = x @ w1.T + b1
    h1 = np.maximum(z1, 0)
    z2 = h1 @ w2.T + b2
    h2 = np.maximum(z2, 0)
    r = h2 @ w3 + b3 - t
    a = np.abs(r)
    loss = np.where(a <= 1, 0.5 * r * r, a - 0.5).mean()
    dy = np.clip(r, -1, 1) / len(r)
    dz2 = np.outer(dy, w3) * (z2 > 0)
    dz1 = (dz2 @ w2) * (z1 > 0)
    grad = np.concatenate([(dz1.T @ x).ravel(), dz1.sum(0), (dz2.T @ h1).ravel(), dz2.sum(0), h2.T @ dy, [dy.sum()]])
    return {"grad": grad, "loss": float(loss)}
