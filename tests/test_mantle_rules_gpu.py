"""change_phase's mantle rules (serpentinisation window, melting above the
solidus) on FP64 contexts: the FP32 test that passes over markers whose rule
certainly does nothing must leave every decision to the FP64 rules.  Markers are
put around the thresholds at distances from well inside the margins (0.001
degrees) to far outside (50 degrees), above crust that allows serpentinisation;
the new phases equal the oracle's exactly."""
import numpy as np
import pytest

from geoflac_gb300 import inpgen, new_state
from geoflac_gb300.flac import Flac
from oracle.oracle import Oracle

from ._util import oracle_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("curve", ["solidus", "window_low", "window_high", "limit"])
@pytest.mark.parametrize("spread", [1e-3, 0.3, 50.0])
def test_mantle_rules_equal_the_oracle(workdir, curve, spread):
    m = inpgen.two_phase_extension(60, 40, 300e3, 180e3)
    inp = m.write(str(workdir / f"mantle_{curve}_{spread}.inp"))
    p, c, s = new_state(inp)
    orc = Oracle(*oracle_state(inp))
    orc.finish_setflac()
    rng = np.random.default_rng(int(spread * 1e4) + len(curve))
    o = orc.s
    z, x, temp = o["cord"][..., 1], o["cord"][..., 0], o["temp"]
    z += rng.uniform(-200.0, 200.0, z.shape)  # uneven triangles
    depth = z[:1, :] - z
    press = 3000.0 * p.g * depth
    pg = np.abs(press) * 1e-9
    base = {"solidus": -5.02 * pg * pg + 132.0 * pg + 1160.0,
            "window_low": 730.0 + (press - 2.1e9) / 2.5e7,
            "window_high": 730.0 - (press - 2.1e9) / 2.3478261e7,
            "limit": 1900.0 + 0.0 * depth}[curve]  # above the solidus down to the 150 km limit
    temp[...] = base + rng.normal(0.0, spread, temp.shape)
    if curve.startswith("window"):  # rows of basalt that let the mantle above them serpentinise
        nm, ids, ph = o["nmark_elem"], o["mark_id_elem"], o["mark_phase"]
        for j in range(12, 40, 3):
            for i in range(0, 60):
                ph[ids[:nm[j, i], j, i] - 1] = 3
                o["phase_ratio"][:, j, i] = 0.0
                o["phase_ratio"][2, j, i] = 1.0
                o["iphase"][j, i] = 3
    gpu = Flac(p, c, s, "fp64")
    gpu.download()
    gpu.state.copy_from(o)
    gpu.upload()
    before = o["mark_phase"].copy()
    orc.change_phase()
    gpu.change_phase()
    gpu.download()
    n = c.nmarkers
    assert np.array_equal(gpu.state["mark_phase"][:n], o["mark_phase"][:n])
    assert np.array_equal(gpu.state["iphase"], o["iphase"])
    assert (o["mark_phase"][:n] != before[:n]).sum() > 0
    gpu.close()
