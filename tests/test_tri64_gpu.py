"""The FP64 element kernels with one thread per triangle (fl_rheol, fl_move)
at mesh sizes around a warp's eight and a CTA's 32 elements, for each
rheology and with the strain / stress mixing on and off: bit-exact with the
oracle, as the FP64 path's arithmetic is the serial reference's."""
import numpy as np
import pytest

from geoflac_gb300 import inpgen, new_state
from geoflac_gb300.flac import Flac
from oracle.oracle import Oracle

from ._util import compare_states, oracle_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nex,nez", [(7, 4), (8, 4), (11, 3), (33, 5), (43, 16)])
@pytest.mark.parametrize("irheol,mix", [(12, 1), (12, 0), (6, 1), (3, 0), (1, 1)])
def test_triangle_kernels_match_oracle(workdir, nex, nez, irheol, mix):
    m = inpgen.two_phase_extension(nex, nez, nex * 10e3, 100e3, crust_km=100.0 / nez, half_rate_cm_yr=3.0, seed_size=1)
    m.mix_strain = m.mix_stress = mix
    m.tau_heal = 1e13 if mix else 0.0
    for ph in m.phases:
        ph.irheol = irheol
        ph.coh1, ph.coh2, ph.pls2 = 2e6, 1e6, 0.01  # yields, and softens, within the steps taken
    inp = m.write(str(workdir / f"tri_{nex}_{nez}_{irheol}_{mix}.inp"))
    gpu = Flac(*new_state(inp), "fp64")
    orc = Oracle(*oracle_state(inp))
    orc.finish_setflac()
    for _ in range(3):
        orc.step(13)
        gpu.step(13)
    gpu.download()
    diffs, bad = compare_states(gpu.state, orc.s)
    assert not bad, bad
    assert max(diffs.values()) == 0.0, diffs
    assert np.isfinite(gpu.state["vel"]).all()
    gpu.close()
