"""What waves of windows leave behind: windows whose pool a saif_only call
gave back without running them."""
import numpy as np
import pytest

from gls import synth
from gls.capi import GlsError, Simulator

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
