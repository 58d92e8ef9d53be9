"""FP64 densities, time step and mass scaling on both sides of the size from
which their products and quotients run on the integer pipes (8192 elements): the
oracle's bits."""
import numpy as np
import pytest

from geoflac_gb300 import inpgen, new_state
from geoflac_gb300.flac import Flac
from oracle.oracle import Oracle

from ._util import oracle_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nex,nez", [(60, 20), (90, 91), (64, 128), (200, 61)])
def test_masses_and_time_step_bits(workdir, nex, nez):
    inp = inpgen.two_phase_extension(nex, nez, 2e3 * nex, max(2e3 * nez, 90e3)).write(str(workdir / f"mb_{nex}_{nez}.inp"))
    gpu, orc = Flac(*new_state(inp), "fp64"), Oracle(*oracle_state(inp))
    orc.finish_setflac()
    temp = orc.s["temp"]
    temp += np.random.default_rng(nex).normal(0.0, 10.0, temp.shape)
    gpu.download()
    gpu.state.copy_from(orc.s)
    gpu.upload()
    for x in (orc, gpu):
        x.rmasses()
        x.dt_mass()
    gpu.download()
    for f in ("rmass", "amass"):
        assert np.array_equal(gpu.state[f], orc.s[f]), f
    for k in ("dt", "dt_elastic", "dt_maxwell", "frac", "vel_max", "dlmin"):
        assert getattr(gpu.clock, k) == getattr(orc.c, k), k
    gpu.close()
