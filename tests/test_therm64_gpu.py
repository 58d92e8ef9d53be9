"""FP64 fl_therm on both of its sweep kernels (one node per thread; the general
one, here forced by more nodes than the chip holds that way), with columns
shorter than, equal to and longer than a warp's 32 nodes and ragged node
counts: bit-exact with the oracle's serial in-place update, over calls whose
start is predicted from the one before."""
import numpy as np
import pytest

from geoflac_gb300 import inpgen, new_state
from geoflac_gb300.flac import Flac
from oracle.oracle import Oracle

from ._util import oracle_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nex,nez", [(2, 2), (9, 12), (4, 31), (40, 32), (7, 150), (3400, 30), (3300, 31), (900, 120)])
def test_fl_therm_equals_the_serial_update(workdir, nex, nez):
    m = inpgen.two_phase_extension(nex, nez, nex * 2e3, max(nez * 2e3, 90e3), crust_km=20.0, half_rate_cm_yr=2.0, seed_size=1)
    inp = m.write(str(workdir / f"therm_{nex}_{nez}.inp"))
    gpu = Flac(*new_state(inp), "fp64")
    orc = Oracle(*oracle_state(inp))
    orc.finish_setflac()
    rng = np.random.default_rng(nez)
    temp, shr = orc.s["temp"], orc.s["shrheat"]
    temp += rng.normal(0.0, 20.0, size=temp.shape)
    shr += rng.uniform(0.0, 1e-6, size=shr.shape)
    gpu.download()
    gpu.state.copy_from(orc.s)
    gpu.upload()
    for _ in range(3):
        orc.fl_therm()
        gpu.fl_therm()
    gpu.download()
    assert np.array_equal(gpu.state["temp"], orc.s["temp"])
    assert np.array_equal(gpu.state["temp0"], orc.s["temp0"])
    assert gpu.clock.therm_unconverged == 0
    gpu.close()
