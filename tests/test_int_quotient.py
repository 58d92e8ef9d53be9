"""The quotients by a shared integer-pipe reciprocal (gf_int_recip, gf_ddiv_by,
gf_rcp_by) and the products of kernels with many of them (gf_mulq) of
geoflac_gb300/csrc/gf_kernels.cuh: restated step for step on words and checked
against IEEE arithmetic (Python floats are IEEE doubles), with what the device
code relies on asserted on every case: the rounded estimate of the quotient lies
within 3/2 of it, twice the residual fits in a signed 64-bit integer and is no
tie, and one step in either direction rounds correctly.  On the GPU, the device
functions themselves on some ten million pairs."""
import math
import random
import subprocess
from fractions import Fraction

import numpy as np
import pytest

from geoflac_gb300 import build

from .test_int_multiply import M32, funnel_l
from .test_int_reciprocal import M64, join, rcp_sig, s64, same, split


def gf_int_recip(b):
    lo, hi = split(b)
    return b, rcp_sig(hi & 0xFFFFF, lo)


def gf_ddiv_by(a, r):
    b, t = r
    la, ha = split(a)
    lb, hb = split(b)
    Ea, Eb = (ha >> 20) & 0x7FF, (hb >> 20) & 0x7FF
    za = ((ha << 1) & M32 | la) == 0
    if not ((((Ea - 573) & M32) <= 900 or za) and ((Eb - 573) & M32) <= 900):
        return None  # the IEEE division out of line
    sign = (ha ^ hb) & 0x80000000
    if za:
        return join(0, sign)
    Ma = (((ha & 0xFFFFF) | 0x100000) << 32) | la
    Mb = (((hb & 0xFFFFF) | 0x100000) << 32) | lb
    k = 52 if Ma >= Mb else 53
    hi, lo = (Ma * t) >> 64, (Ma * t) & M64
    q = ((hi << (k - 41)) + (((lo >> (104 - k)) + 1) >> 1)) & M64
    Q = Fraction(Ma * 2 ** k, Mb)
    assert abs(q - Q) < Fraction(3, 2)
    res = s64(2 * s64((Ma << k) - Mb * q))
    assert res == 2 * (Ma * 2 ** k - Mb * q) and abs(res) < 3 * Mb and abs(res) != Mb
    q += 1 if res > Mb else (-1 if res < -Mb else 0)
    assert abs(q - Q) < Fraction(1, 2)
    bits = (((1074 - k + Ea - Eb) << 52) + q) & M64
    return join(bits & M32, (bits >> 32) | sign)


def gf_rcp_by(r):
    b, t = r
    lo, hi = split(b)
    E = (hi >> 20) & 0x7FF
    if ((E - 573) & M32) > 900:
        return None
    sign = hi & 0x80000000
    if ((hi & 0xFFFFF) | lo) == 0:
        return join(0, sign | ((2046 - E) << 20))
    bits = (((2044 - E) << 52) + t) & M64
    return join(bits & M32, (bits >> 32) | sign)


def gf_mulq(a, b):
    la, ha = split(a)
    lb, hb = split(b)
    if max((ha * 2 - (573 << 21)) & M32, (hb * 2 - (573 << 21)) & M32) >= 901 << 21:
        return None  # the FP64 multiply out of line
    mh, nh = (ha & 0xFFFFF) | 0x100000, (hb & 0xFFFFF) | 0x100000
    p0 = la * lb
    t = la * nh + (p0 >> 32)
    t += mh * lb
    u = mh * nh + (t >> 32)
    assert t <= M64 and u <= M64 and u >> 32 < 1 << 10
    w2, w1, w0, wm = u >> 32, u & M32, t & M32, p0 & M32
    top = w2 >> 9
    sh = 12 - top
    mhi, mlo = funnel_l(w1, w2, sh), funnel_l(w0, w1, sh)
    rem, x = (w0 << sh) & M32, min(wm, 1) | (mlo & 1)
    up = 1 if ((rem + x) & M32) > 0x80000000 else 0
    assert rem + x <= M32
    S = ((ha & 0xFFF00000) + (hb & 0xFFF00000) - (1024 << 20) + (top << 20)) & M32
    r = ((((mhi + S) & M32) << 32 | mlo) + up) & M64
    return join(r & M32, r >> 32)


def inside(x):
    return 2.0 ** -450 <= abs(x) < 2.0 ** 451


EDGE = [2.0 ** -450, 2.0 ** 451 * (1 - 2.0 ** -53), math.nextafter(2.0 ** -450, 0.0), 2.0 ** 451, 1.0, 0.5, 3.0, 0.1,
        1.0 + 2.0 ** -52, 2.0 - 2.0 ** -52, 0.0, 5e-324, 1e-300, 1e300, math.inf]
EDGE += [-x for x in EDGE]


def quotient_cases(rng, n):
    """significands at random, at both ends, exact quotients and one unit beside
    them, and quotients next to a rounding boundary (A / B = (2 u + 1) / 2^54 - r / (2^54 B))"""
    out = []
    while len(out) < n:
        kind = rng.randrange(6)
        A, B = rng.randrange(1 << 52, 1 << 53), rng.randrange(1 << 52, 1 << 53)
        if kind == 1:
            A, B = (1 << 53) - 1 - rng.randrange(64), (1 << 52) + rng.randrange(64)
        elif kind == 2:
            A, B = (1 << 52) + rng.randrange(64), (1 << 53) - 1 - rng.randrange(64)
        elif kind == 3:
            q, B = rng.randrange(1 << 26, 1 << 27), rng.randrange(1 << 25, 1 << 26)
            A = q * B
            s = A.bit_length()
            A = (A << (53 - s)) + rng.choice([-1, 0, 1]) if s < 53 else A >> (s - 53)
            A = min(max(A, 1 << 52), (1 << 53) - 1)
            B <<= 53 - B.bit_length()
        elif kind == 4:
            B |= 1
            r = rng.choice([1, -1, 3, -3, 5, 101])
            u = r * pow(B, -1, 2 ** 54) % 2 ** 54
            A, rest = divmod(u * B - r, 2 ** 54)
            if rest or not 1 << 52 <= A < 1 << 53:
                continue
        elif kind == 5:
            B = 1 << 52
        out.append((rng.choice([1, -1]) * math.ldexp(A, rng.randint(-490, 380)), math.ldexp(B, rng.randint(-490, 380))))
    return [(a, b) for a, b in out if inside(a) and inside(b)]


def test_quotients_by_a_shared_reciprocal():
    rng = random.Random(41)
    cases = quotient_cases(rng, 30000)
    assert len(cases) > 25000
    for a, b in cases:
        r = gf_int_recip(b)
        assert same(gf_ddiv_by(a, r), a / b), (a, b)
        assert same(gf_rcp_by(r), 1.0 / b), b


def test_range_of_the_quotients():
    for a in EDGE:
        for b in EDGE:
            r = gf_int_recip(b)
            got = gf_ddiv_by(a, r)
            assert (got is not None) == ((inside(a) or a == 0.0) and inside(b)), (a, b)
            if got is not None:
                assert same(got, a / b), (a, b)
        assert (gf_rcp_by(gf_int_recip(a)) is not None) == inside(a), a


def product_cases(rng, n):
    out = []
    for _ in range(n):
        kind = rng.randrange(5)
        A, B = rng.randrange(1 << 52, 1 << 53), rng.randrange(1 << 52, 1 << 53)
        if kind == 1:  # exact ties
            A, B = (A >> 27 << 27) | (1 << 26), B >> 26 << 26 | (1 << 26)
        elif kind == 2:  # beside a tie
            A, B = (A >> 27 << 27) | (1 << 26) | rng.choice([0, 1]), B >> 27 << 27
        elif kind == 3:  # a carry out of the significand
            A, B = (1 << 53) - 1 - rng.randrange(64), (1 << 53) - 1 - rng.randrange(64)
        elif kind == 4:
            A = 1 << 52
        out.append((rng.choice([1, -1]) * math.ldexp(A, rng.randint(-502, 398)),
                    rng.choice([1, -1]) * math.ldexp(B, rng.randint(-502, 398))))
    return out


def test_products():
    rng = random.Random(42)
    cases = product_cases(rng, 60000)
    for a, b in cases:
        assert inside(a) and inside(b)
        assert same(gf_mulq(a, b), a * b), (a, b)


def test_range_of_the_products():
    """zeros go out of line too"""
    for a in EDGE:
        for b in EDGE:
            got = gf_mulq(a, b)
            assert (got is not None) == (inside(a) and inside(b)), (a, b)
            if got is not None:
                assert same(got, a * b), (a, b)


KERNELS = r"""
#include "gf_kernels.cuh"
using namespace gfk;
__global__ void k(long long n, const double *a, const double *b, double *o) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const GfIntRecip r = gf_int_recip(b[i]);
    o[i] = gf_ddiv_by(a[i], r);
    o[n + i] = gf_rcp_by(r);
    o[2 * n + i] = gf_mulq(a[i], b[i]);
    o[3 * n + i] = gf_mul(a[i], b[i]);
}
extern "C" int run(long long n, const double *a, const double *b, double *o) {
    double *d = nullptr;
    int e = cudaMalloc(&d, 6 * n * sizeof(double));
    if (!e) e = cudaMemcpy(d, a, n * sizeof(double), cudaMemcpyHostToDevice);
    if (!e) e = cudaMemcpy(d + n, b, n * sizeof(double), cudaMemcpyHostToDevice);
    if (!e) k<<<(unsigned)((n + 255) / 256), 256>>>(n, d, d + n, d + 2 * n);
    if (!e) e = cudaGetLastError();
    if (!e) e = cudaMemcpy(o, d + 2 * n, 4 * n * sizeof(double), cudaMemcpyDeviceToHost);
    cudaFree(d);
    return e;
}
"""


@pytest.mark.gpu
def test_device_functions(tmp_path):
    import ctypes as C

    src, lib = tmp_path / "q.cu", tmp_path / "q.so"
    src.write_text(KERNELS)
    subprocess.run([build._nvcc()] + build.ARCH + ["-O3", "-std=c++17", "-fmad=false", "-Xcompiler", "-fPIC", "-shared",
                                                   "-I" + build.CSRC, "-o", str(lib), str(src)], check=True)
    run = C.CDLL(str(lib)).run
    rng = np.random.default_rng(43)
    n = 1 << 23
    a, b = (np.ldexp(rng.integers(1 << 52, 1 << 53, n).astype(np.float64), rng.integers(-502, 398, n)) for _ in range(2))
    a[rng.random(n) < 0.5] *= -1.0
    m = 1 << 21  # magnitudes of the step, and all classes of value against each other
    a[:m], b[:m] = rng.uniform(-1e10, 1e10, m), rng.uniform(1e-12, 1e12, m)
    pairs = product_cases(random.Random(44), 200000) + quotient_cases(random.Random(45), 200000)
    pairs += [(x, y) for x in EDGE + [math.nan] for y in EDGE + [math.nan]]
    a = np.concatenate([a, [p[0] for p in pairs]])
    b = np.concatenate([b, [p[1] for p in pairs]])
    n = a.size
    out = np.empty((4, n))
    ptr = lambda x: x.ctypes.data_as(C.c_void_p)
    assert run(C.c_longlong(n), ptr(a), ptr(b), ptr(out)) == 0
    with np.errstate(all="ignore"):
        want = np.stack([a / b, 1.0 / b, a * b, a * b])
    same_bits = (out.view(np.uint64) == want.view(np.uint64)) | (np.isnan(out) & np.isnan(want))
    assert same_bits.all(), [(i, a[i], b[i], out[k, i]) for k, i in np.argwhere(~same_bits)[:4]]
