"""The input-dependent features of a gate output (unrolled for one to three
input nets, looped over its truth table for more) against float64.

Tolerance: est and pone are sums of at most 12 products of at most four FP32
factors, all terms positive: 16 roundings, 16 x 2^-24 = 1e-6 of the value; the
1-probabilities are rounded once more; log1p / 12 shrinks it.  1e-5 of one
plus the value leaves room for the device's logarithm."""
import itertools

import numpy as np
import pytest

from gls.capi import CALC_FIXED, Simulator, cell_lut
from gls.cells import LIBRARY, SYNTH_CELLS
from gls.levelize import assemble, default_arcs
from cases import stimulus

pytestmark = pytest.mark.gpu


def expected(lut, ins, lens, saif):
    nets = list(dict.fromkeys(ins))
    m = len(nets)
    q = []
    for n in nets:
        t0, t1 = float(saif[n][0]), float(saif[n][1])
        q.append(t1 / (t0 + t1) if t0 + t1 > 0 else 0.5)
    f = {b: lut[sum((3 if b[nets.index(n)] else 0) << (2 * p) for p, n in enumerate(ins))]
         for b in itertools.product((0, 1), repeat=m)}
    prob = lambda b, skip=None: np.prod([q[i] if b[i] else 1 - q[i] for i in range(m) if i != skip])
    pone = sum(prob(b) for b in f if f[b] == 3)
    est = sum(prob(b, j) * lens[nets[j]] for b in f for j in range(m)
              if b[j] == 0 and f[b] != f[b[:j] + (1,) + b[j + 1:]])
    return np.log1p(est) / 12, pone, sum(q) / m


@pytest.mark.parametrize("tied", [False, True])
@pytest.mark.parametrize("name", SYNTH_CELLS)
def test_features_of_every_cell(name, tied, gpu):
    c = LIBRARY[name]
    ins = [0] * c.n_in if tied and c.n_in < 3 else [0, 1, 0][:c.n_in] if tied else list(range(c.n_in))
    nl = assemble([(name, ins, [3], default_arcs(c, 3.0, 4.0))], n_nets=4)
    rng = np.random.default_rng(len(name))
    st = stimulus({n: [(10 * k + n, int(v)) for k, v in enumerate(rng.choice([0, 3, 3, 1], 20 + 40 * n))]
                   for n in sorted(set(ins))})
    cells, prims = nl.cell_arrays()
    with Simulator() as s:
        s.load(nl)
        w = s.add_window(st, 0, 2000)
        s.run()
        row = s.presize_samples(w)[0][0]
        want = expected(cell_lut(cells[0], prims, 0, CALC_FIXED), ins, s.lengths(w), s.saif(w))
    assert np.allclose(row[21:24], want, rtol=1e-5, atol=1e-5), (row[21:24], want)
