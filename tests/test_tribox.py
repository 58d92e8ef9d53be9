"""The box test of the remesh event's search (geoflac_gb300/csrc/gf_tribox.h,
compiled for the host): it keeps out no point that the search's own test would
take.  Triangles of all shapes and places, points inside, on the edges and
corners, just outside the accepted band, far away, infinite and NaN."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from geoflac_gb300 import build

SRC = r"""
#include "gf_tribox.h"
// the search's test (rem_barcord, remesh.f90:327-439) and the box's, for n triangles
// (x1, x2, x3, y1, y2, y3) with m points each: taken[] and kept[] (by the boxes)
extern "C" void run(long n, long m, const double *t, const double *p, unsigned char *taken, unsigned char *kept) {
    const double perr = 1e-4;
    for (long i = 0; i < n; ++i) {
        const double x1 = t[6 * i], x2 = t[6 * i + 1], x3 = t[6 * i + 2], y1 = t[6 * i + 3], y2 = t[6 * i + 4], y3 = t[6 * i + 5];
        const double det = ((x2 * y3 - y2 * x3) - (x1 * y3 - y1 * x3)) + (x1 * y2 - y1 * x2);
        const double q0 = (x2 * y3 - y2 * x3) / det, q1 = (y2 - y3) / det, q2 = (x3 - x2) / det;
        const double q3 = (x3 * y1 - y3 * x1) / det, q4 = (y3 - y1) / det, q5 = (x1 - x3) / det;
        const GfTriBox box = gf_tri_box(x1, x2, x3, y1, y2, y3, det);
        for (long k = 0; k < m; ++k) {
            const double xx = p[2 * (i * m + k)], yy = p[2 * (i * m + k) + 1];
            const double a1 = q0 + xx * q1 + yy * q2, a2 = q3 + xx * q4 + yy * q5, a3 = 1.0 - a1 - a2;
            const bool out = a1 <= -perr || a1 >= (1.0 + perr) || a2 <= -perr || a2 >= (1.0 + perr) || a3 <= -perr || a3 >= (1.0 + perr);
            const float xf = (float)xx, yf = (float)yy;
            taken[i * m + k] = !out;
            kept[i * m + k] = !(gf_box_applies(xf, yf) && !gf_box_holds(box, xf, yf));
        }
    }
}
"""


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    d = tmp_path_factory.mktemp("tribox")
    (d / "t.cpp").write_text(SRC)
    subprocess.run(["g++", "-O1", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-I" + build.CSRC, "-o",
                    str(d / "t.so"), str(d / "t.cpp")], check=True)
    lib = C.CDLL(os.path.join(str(d), "t.so"))

    def call(tri, pts):
        n, m = pts.shape[:2]
        tri, pts = np.ascontiguousarray(tri, np.float64), np.ascontiguousarray(pts, np.float64)
        taken, kept = np.zeros((n, m), np.uint8), np.zeros((n, m), np.uint8)
        lib.run(C.c_long(n), C.c_long(m), *[a.ctypes.data_as(C.c_void_p) for a in (tri, pts, taken, kept)])
        return taken.astype(bool), kept.astype(bool)

    return call


@pytest.mark.parametrize("scale", [1e-3, 1.0, 1e3, 1e6])
@pytest.mark.parametrize("aspect", [1.0, 30.0, 3e3])
@pytest.mark.parametrize("offset", [0.0, 1e2, 1e5])
def test_no_taken_point_is_kept_out(run, scale, aspect, offset):
    rng = np.random.default_rng(int(aspect) + int(offset))
    n, m = 4000, 60
    v = rng.uniform(-1.0, 1.0, (n, 3, 2)) * [1.0, 1.0 / aspect] + rng.uniform(-1, 1, (n, 1, 2)) * offset
    v *= scale
    w = rng.dirichlet([1.0, 1.0, 1.0], (n, m))
    edge = rng.random((n, m)) < 0.5
    w[edge, rng.integers(0, 3)] = rng.choice([0.0, -1e-4, -0.99e-4, -1.01e-4, -1e-3], edge.sum())
    w /= w.sum(-1, keepdims=True)
    p = np.einsum("nmk,nkd->nmd", w, v)
    p[:, :3] = v  # the corners
    p[:, 3] = rng.uniform(-3, 3, (n, 2)) * scale + v[:, 0]
    p[:, 4, 0], p[:, 5, 1], p[:, 6] = np.nan, np.nan, np.nan
    p[:, 7, 0], p[:, 8, 1], p[:, 9] = np.inf, -np.inf, np.inf
    p[:, 10] = 1e300
    with np.errstate(all="ignore"):
        taken, kept = run(np.concatenate([v[..., 0], v[..., 1]], 1), p)
    assert not (taken & ~kept).any()
    assert taken[:, 4:7].all()
    if aspect * offset <= 3e6:  # (beyond, the search's own coordinates have lost their digits)
        assert taken[:, :3].mean() > 0.9
    if aspect == 1.0 and offset <= 1e2:
        assert (~kept[:, 3]).mean() > 0.3  # and it does keep points out


def test_degenerate_and_huge_triangles(run):
    v = np.array([[0, 0, 0, 0, 0, 0], [0, 1, 2, 0, 1, 2], [0, 1e200, 0, 0, 0, 1e200], [0, np.nan, 1, 0, 1, 0],
                  [1e16, 2e16, 1e16, 0, 0, 1e16], [0, 1e-20, 0, 0, 0, 1e-20]], float)
    p = np.array([[0, 0], [0.5, 0.5], [1e199, 1e199], [np.nan, 0], [1.2e16, 1e15], [2e-21, 2e-21]], float)
    taken, kept = run(v, np.broadcast_to(p, (6, 6, 2)))
    assert not (taken & ~kept).any()
