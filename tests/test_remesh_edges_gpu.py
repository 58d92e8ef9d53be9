"""The remesh event on distorted meshes of awkward sizes (the smallest that is
accepted, ragged against a warp, more elements than one CTA scans) and far from
the origin, where triangles get no search box: FP64 GPU against the oracle,
integer fields exact, floats within the event tolerance of
tests/test_remesh_gpu.py."""
import numpy as np
import pytest

from geoflac_gb300 import inpgen, new_state
from geoflac_gb300.flac import Flac
from oracle.oracle import Oracle

from ._util import oracle_state
from .test_remesh_gpu import EVENT_TOL, _compare

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nex,nez", [(3, 2), (34, 9), (1100, 4)])
@pytest.mark.parametrize("x0", [0.0, 5e7])
def test_distorted_mesh_remeshes_like_the_oracle(workdir, nex, nez, x0):
    m = inpgen.two_phase_extension(nex, nez, nex * 3e3, nez * 3e3, crust_km=3.0, seed_size=1)
    m.x0 = x0
    inp = m.write(str(workdir / f"edges_{nex}_{nez}_{int(x0)}.inp"))
    gpu = Flac(*new_state(inp), "fp64")
    orc = Oracle(*oracle_state(inp))
    orc.finish_setflac()
    orc.step(3)
    gpu.step(3)
    rng = np.random.default_rng(nex)
    cord = orc.s["cord"]
    shift = rng.uniform(-900.0, 900.0, size=cord.shape)
    shift[:, 0, 0] = shift[:, -1, 0] = shift[-1, :, 1] = 0.0  # walls and base keep their lines
    cord += shift
    for f in ("dhacc", "extr_acc"):
        orc.s[f][: nex] = rng.uniform(0.0, 5.0, size=nex)
    gpu.download()
    gpu.state.copy_from(orc.s)
    gpu.upload()
    orc.remesh_event()
    gpu.remesh()
    _compare(gpu, orc, EVENT_TOL, "remesh")
    for f in ("dhacc", "extr_acc"):
        assert np.array_equal(gpu.state[f][: nex], orc.s[f][: nex]), f
    gpu.close()
