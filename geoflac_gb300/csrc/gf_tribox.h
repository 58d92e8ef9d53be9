// The box test of the remesh event's search for the old triangle that contains a
// new point (k_trpars, k_barcord in gf_remesh.cu), for host and device.
#pragma once

#include "gf_math.h"

struct alignas(16) GfTriBox {
    float x0, x1, y0, y1;
};

// The FP32 box outside which no point has all three barycentric coordinates in
// (-1e-4, 1 + 1e-4): the triangle's, widened by 2 % of its extent L and the
// rounding of the FP32 copies.  The coordinates that the search evaluates err by
// less than 1e-3 for triangles with |det| >= 1e-3 L^2 and coordinates up to 1e4 L
// (their numerators round at 4 2^-53 of the coordinates' squares); any other
// triangle gets an infinite box.
GFM_HD GfTriBox gf_tri_box(double x1, double x2, double x3, double y1, double y2, double y3, double det) {
    const float f1 = (float)x1, f2 = (float)x2, f3 = (float)x3, h1 = (float)y1, h2 = (float)y2, h3 = (float)y3;
    const GfTriBox b = {fminf(f1, fminf(f2, f3)), fmaxf(f1, fmaxf(f2, f3)), fminf(h1, fminf(h2, h3)),
                        fmaxf(h1, fmaxf(h2, h3))};
    const float X = fmaxf(fmaxf(fabsf(b.x0), fabsf(b.x1)), fmaxf(fabsf(b.y0), fabsf(b.y1)));
    const float L = fmaxf(b.x1 - b.x0, b.y1 - b.y0), m = 0.02f * L + 1e-6f * X;
    if (fabsf((float)det) >= 1e-3f * L * L && X <= 1e4f * L && L > 1e-15f && X < 1e15f)
        return GfTriBox{b.x0 - m, b.x1 + m, b.y0 - m, b.y1 + m};
    return GfTriBox{-INFINITY, INFINITY, -INFINITY, INFINITY};
}
// Whether boxes may be asked about the point: a NaN coordinate passes every test
// of the search (none of its comparisons holds), so no box may keep it out.
GFM_HD bool gf_box_applies(float x, float y) { return fabsf(x) < 1e15f && fabsf(y) < 1e15f; }
GFM_HD bool gf_box_holds(const GfTriBox &b, float x, float y) { return x >= b.x0 && x <= b.x1 && y >= b.y0 && y <= b.y1; }
