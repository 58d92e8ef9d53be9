"""FP64 densities, time step and mass scaling on both sides of the size from
which their products and quotients run on the integer pipes (8192 elements):
the same bits, so the fields equal the oracle's to the tolerance of the other
single-subroutine comparisons (1e-12 of the largest value)."""
import numpy as np
import pytest

from geoflac_gb300 import inpgen, new_state
from geoflac_gb300.flac import Flac
from oracle.oracle import Oracle

from ._util import oracle_state, rel_diff

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nex,nez", [(60, 20), (90, 91), (64, 128), (200, 61)])
def test_masses_and_time_step(workdir, nex, nez):
    inp = inpgen.two_phase_extension(nex, nez, 2e3 * nex, max(2e3 * nez, 90e3)).write(str(workdir / f"ip_{nex}_{nez}.inp"))
    gpu, orc = Flac(*new_state(inp), "fp64"), Oracle(*oracle_state(inp))
    orc.finish_setflac()
    rng = np.random.default_rng(nex)
    o = orc.s
    temp = o["temp"]
    temp += rng.normal(0.0, 10.0, temp.shape)
    gpu.download()
    gpu.state.copy_from(o)
    gpu.upload()
    for x in (orc, gpu):
        x.rmasses()
        x.dt_mass()
    gpu.download()
    for f in ("rmass", "amass"):
        assert rel_diff(gpu.state[f], o[f]) <= 1e-12, f
    for k in ("dt", "dt_elastic", "dt_maxwell", "frac"):
        assert getattr(gpu.clock, k) == pytest.approx(getattr(orc.c, k), rel=1e-12), k
    gpu.close()
