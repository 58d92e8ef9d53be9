"""gf_itest_mesh's smallest angle on both sides of the size where an FP32 pass
picks the elements for the FP64 one (8192 elements): regular meshes (every
element equally good), perturbed ones, a single bad element, and one so thin
that FP32 is not trusted.  Against the rem_test expressions in numpy, 1e-12
relative (the device evaluates the same FP64 expressions; its acos may differ
in the last places)."""
import numpy as np
import pytest

from geoflac_gb300 import capi, inpgen, new_state
from geoflac_gb300.flac import Flac

pytestmark = pytest.mark.gpu


def _smallest(c):
    q = [c[:-1, :-1], c[1:, :-1], c[:-1, 1:], c[1:, 1:]]
    best = 180.0
    for t in ((0, 1, 2), (1, 3, 2), (0, 1, 3), (0, 3, 2)):
        v = [q[k] for k in t] + [q[t[0]]]
        ang = {}
        for k in (1, 2):
            a, b = v[k + 1] - v[k], v[k - 1] - v[k]
            dot = (a * b).sum(-1)
            ang[k] = np.degrees(np.arccos(dot / (np.hypot(*np.moveaxis(a, -1, 0)) * np.hypot(*np.moveaxis(b, -1, 0)))))
        best = min(best, ang[1].min(), ang[2].min(), (180.0 - ang[1] - ang[2]).min())
    return best


@pytest.mark.parametrize("nex,nez", [(60, 20), (90, 91), (64, 128), (331, 113)])
@pytest.mark.parametrize("kind", ["regular", "perturbed", "bad", "thin"])
def test_smallest_angle(workdir, nex, nez, kind):
    m = inpgen.two_phase_extension(nex, nez, 1e3 * nex, max(1e3 * nez, 90e3))
    g = Flac(*new_state(m.write(str(workdir / f"ang_{nex}_{kind}.inp"))), "fp64")
    g.download()
    c = g.state["cord"]
    rng = np.random.default_rng(nex + len(kind))
    if kind != "regular":
        c += rng.uniform(-60.0, 60.0, c.shape)
    if kind == "bad":  # one corner pulled in
        c[nez // 2, nex // 3] += 0.55 * (c[nez // 2 + 1, nex // 3 + 1] - c[nez // 2, nex // 3])
    if kind == "thin":  # a node 0.2 m from its neighbour's diagonal: an angle of about 0.01 degrees
        j, i = nez // 2, nex // 3
        mid = 0.5 * (c[j, i + 1] + c[j + 1, i])
        c[j, i] = mid + 3e-4 * (c[j, i] - mid)
    g.upload(capi.F_CORD)
    got, want = g.itest_mesh(), _smallest(np.asarray(c))
    assert abs(got - want) <= 1e-12 * want + (1e-9 if kind == "thin" else 0.0), (got, want)
    g.close()
