"""gf_batch_sample keeps the precision of its FP64 fields.  On grids whose
positions are exact binary fractions (mesh and grid sides powers of two) the
sampled values are the exact bilinear sums rounded to FP32, to within half a unit
of the result and eight roundings of 2^-53 of the largest corner: for velocities
whose terms cancel to a billionth, and for values below the normal FP32 range.
Infinite corners give infinities."""
from fractions import Fraction

import numpy as np
import pytest

from geoflac_gb300 import capi, inpgen
from geoflac_gb300.batch import Batch
from geoflac_gb300.flac import Flac, new_state

pytestmark = pytest.mark.gpu
NEX, NEZ, H, W = 32, 16, 64, 64


def _sample(workdir, tag, fill):
    torch = pytest.importorskip("torch")
    m = inpgen.two_phase_extension(NEX, NEZ, 320e3, 160e3)
    g = Flac(*new_state(m.write(str(workdir / f"prec_{tag}.inp"))), "mixed")
    s = g.state
    fill(s, np.random.default_rng(11))
    g.upload(capi.F_VEL | capi.F_TEMP | capi.F_APS | capi.F_PHASE)
    b = Batch([g])
    grid = torch.empty((1, H, W, 9), dtype=torch.float32, device="cuda")
    b.sample(grid, H, W, 2)
    torch.cuda.synchronize()
    out = grid[0].cpu().numpy()
    b.close()
    return g, out


def _corners(f, y, x, shift):
    p = [Fraction(2 * k + 1, 2) * n / size - Fraction(shift, 2) for k, n, size in ((y, NEZ, H), (x, NEX, W))]
    top = [NEZ - shift, NEX - shift]
    p = [min(max(q, Fraction(0)), Fraction(t)) for q, t in zip(p, top)]
    (j, i) = (min(int(q), t - 1) for q, t in zip(p, top))
    wy, wx = p[0] - j, p[1] - i
    c = [f[j, i], f[j, i + 1], f[j + 1, i], f[j + 1, i + 1]]
    return c, [(1 - wy) * (1 - wx), (1 - wy) * wx, wy * (1 - wx), wy * wx]


@pytest.mark.parametrize("case", ["cancel", "tiny"])
def test_sums_are_exact_to_fp32(workdir, case):
    def fill(s, rng):
        v, t, a = s["vel"], s["temp"], s["aps"]
        if case == "cancel":
            sign = np.where(np.arange(v.shape[1]) % 2 == 0, 1.0, -3.0)[None, :, None]
            v[...] = 1e-9 * sign * (1.0 + 1e-9 * rng.standard_normal(v.shape))
            t[...] = 1000.0 * sign[..., 0] * (1.0 + 1e-8 * rng.standard_normal(t.shape))
        else:
            v[...] = 1e-42 * rng.standard_normal(v.shape)
            t[...] = 1e-40 * rng.random(t.shape)
            a[...] = 1e-39 * rng.random(a.shape)

    g, out = _sample(workdir, case, fill)
    s = g.state
    rng = np.random.default_rng(3)
    fields = {0: (s["vel"][..., 0], 0), 1: (s["vel"][..., 1], 0), 6: (s["temp"], 0), 5: (s["aps"].astype(np.float32), 1)}
    for _ in range(400):
        y, x = int(rng.integers(H)), int(rng.integers(W))
        for ch, (f, shift) in fields.items():
            c, w = _corners(f, y, x, shift)
            exact = sum(Fraction(float(a)) * b for a, b in zip(c, w))
            ulp = Fraction(float(np.spacing(np.float32(abs(float(exact))))))
            bound = ulp / 2 + 8 * Fraction(1, 2 ** 53) * max(abs(Fraction(float(a))) for a in c)
            assert abs(Fraction(float(out[y, x, ch])) - exact) <= bound, (ch, y, x)
    g.close()


def test_infinities(workdir):
    def fill(s, rng):
        s["vel"][4, 5, 0] = np.inf

    g, out = _sample(workdir, "inf", fill)
    v = out[..., 0]
    hit = np.zeros(v.shape, bool)
    hit[12:20, 8:12] = True  # the four cells around node (4, 5), 4 x 2 points each
    assert np.isinf(v[hit]).all() and np.isfinite(v[~hit]).all()
    g.close()
