"""gf_batch_sample on grids finer, coarser and ragged against the members'
meshes, compared with the bilinear interpolation in numpy FP64 of the same
state.  Bounds: the FP32 result and its FP32 weights, 2^-23 of the corners'
magnitude; the grid positions, FP32 numbers f of which the library's quotient
(approximate division, 2 ulp) and numpy's differ by less than 2^-21 f, times
the field's variation around the point; 1e-9 m for the heights, whose
reference is formed in FP64."""
import numpy as np
import pytest

from geoflac_gb300 import inpgen
from geoflac_gb300.batch import Batch
from geoflac_gb300.flac import Flac, new_state

pytestmark = pytest.mark.gpu


def _index(k, n, size, shift):
    f = np.float32(k + np.float32(0.5)) * np.float32(n) / np.float32(size)
    f = np.float32(f) - np.float32(shift)
    top = np.float32(n - (1 if shift else 0))
    f = min(max(f, np.float32(0)), top)
    i0 = min(int(f), max(int(top) - 1, 0))
    return i0, np.float64(f - np.float32(i0)), float(f) * 2.0 ** -21


@pytest.mark.parametrize("H,W", [(128, 384), (33, 31), (7, 65), (1, 1)])
def test_sample_is_the_bilinear_value(workdir, H, W):
    torch = pytest.importorskip("torch")
    models = []
    for k, (nex, nez) in enumerate([(41, 13), (20, 37), (90, 28)]):
        m = inpgen.two_phase_extension(nex, nez, nex * 2.5e3, max(nez * 2.5e3, 90e3), half_rate_cm_yr=2.0)
        models.append(Flac(*new_state(m.write(str(workdir / f"sample_{k}.inp"))), "mixed"))
    b = Batch(models)
    b.step(25)
    grid = torch.empty((3, H, W, 9), dtype=torch.float32, device="cuda")
    b.sample(grid, H, W, 2)
    torch.cuda.synchronize()
    got = grid.cpu().numpy().astype(np.float64)
    rng = np.random.default_rng(H)
    for k, g in enumerate(models):
        s = g.download()
        nz, nx = s["temp"].shape
        st = s["stress0"].mean(axis=3)
        z0 = g.params.z0 + g.params.rzbo * np.arange(nz) / (nz - 1)
        node = {0: s["vel"][:, :, 0], 1: s["vel"][:, :, 1], 6: s["temp"], 8: s["cord"][:, :, 1] - z0[:, None]}
        elem = {2: st[:, :, 0], 3: st[:, :, 1], 4: st[:, :, 2], 5: s["aps"], 7: s["phase_ratio"][1]}
        for _ in range(200):
            y, x = int(rng.integers(H)), int(rng.integers(W))
            for ch in range(9):
                f, shift = (node[ch], 0.0) if ch in node else (elem[ch], 0.5)
                j, wy, ey = _index(y, nz - 1, H, shift)
                i, wx, ex = _index(x, nx - 1, W, shift)
                if shift:  # centres: nz - 1 by nx - 1 of them
                    j, i = min(j, nz - 2), min(i, nx - 2)
                j1, i1 = min(j + 1, f.shape[0] - 1), min(i + 1, f.shape[1] - 1)
                c = [f[j, i], f[j, i1], f[j1, i], f[j1, i1]]
                v = (1 - wy) * ((1 - wx) * c[0] + wx * c[1]) + wy * ((1 - wx) * c[2] + wx * c[3])
                near = f[max(j - 1, 0):j + 3, max(i - 1, 0):i + 3]
                tol = 2.0 ** -23 * max(map(abs, c)) + (ex + ey) * (near.max() - near.min()) + 1e-9 * (ch == 8)
                assert abs(got[k, y, x, ch] - v) <= tol, (k, y, x, ch)
    b.close()
    for g in models:
        g.close()
