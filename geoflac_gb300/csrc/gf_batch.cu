// Ensemble driver: hundreds of independent models of uneven size advanced
// together, one launch per phase of the step.
//
// Each member is an ordinary mixed-precision context; a packed member table
// (device pointers, dimensions, constants) and per-kind tile tables (element,
// node, marker and max(element, node) items) describe the ensemble.  A tile
// is `threads * items` consecutive items of ONE member, so a warp never mixes
// members and the per-member reductions stay warp-local.  Every phase of the
// step (fl_therm, change_phase, fl_rheol, fl_node, fl_move, rmasses, dt_mass)
// is one launch with a CTA per tile of all members: the ensemble shares the
// step's phase order, not its dt or its size.  The per-item work is the same
// device code as the single-model kernels; a member's result does not depend
// on the other members or the tile depth (FP32 contraction may differ from
// the separately compiled single-model kernels at rounding level).
//
// The launches are chained by programmatic dependent launch (a CTA stages its
// member's record while the phase before it drains) and replayed from CUDA
// graphs.  One co-resident kernel that walks all phases between grid barriers
// was slower at both ends of the range: its registers are those of fl_rheol
// in every phase (8 warps an SM), and a barrier costs about what a dependent
// launch does (ten steps and a sample of 64 members of 80x25 to 400x120
// elements 7.24 against 6.83 ms, of 8 members of 80x25 to 120x36 1.01 against
// 0.54).  The tile depth: see build_tables.

// 32-bit indices, as in the mixed instantiation (members are mixed contexts)
#define GF_IDX int
#include "gf_kernels_impl.cuh"
#include "gf_member.h"

#include <algorithm>
#include <cstdio>
#include <cstring>
#include <vector>

namespace {

enum { K_E = 0, K_N, K_M, K_EN, K_KINDS };

struct BatchMember {
    const DevParams *P;
    DevClock *C;
    DevArrays A;
    GfDims d;
    int idt_scale, movegrid, nmarkers, pad;
    double z0, rzbo; // undeformed surface and depth of the regular start-up mesh
    long long e0;    // elements of the members before this one
};

struct BatchArgs {
    const BatchMember *members;
    int nmembers;
    const int2 *tile[K_KINDS]; // (member, first item) per tile
    int ntile[K_KINDS];
    int ipt;  // items per thread
    int opt;  // the phase's own option (viscosity update, averaging mode, time advance, sweep)
};

// One phase: CTA (t, part) works on tile t of the phase's kind.  The parts of
// a phase (grid y, the longest first) are independent of each other and share
// its launch.  The member's record is constant while steps run, so it is
// staged before the wait for the phase before.  Ph::regs caps the registers
// (at most 128, for the 512 threads a batch may be configured for).  All phases
// wait on memory: a large batch wants warps in flight, a small one many loads
// of a thread together.  A step of 64 / of 8 members: 128 for all 534 / 34.7
// us; these 511 / 34.5; b at 64, c at 48, d at 80 registers 503 / 38.6.
template <class Ph> __global__ void __maxnreg__(Ph::regs) k_phase(BatchArgs a) {
    __shared__ BatchMember m;
    const int2 tl = a.tile[Ph::kind][blockIdx.x];
    const int *src = reinterpret_cast<const int *>(a.members + tl.x);
    int *dst = reinterpret_cast<int *>(&m);
    for (int w = threadIdx.x; w < (int)(sizeof(BatchMember) / sizeof(int)); w += blockDim.x) dst[w] = src[w];
    gfk::gf_pdl_entry();
    __syncthreads();
    for (int r = 0; r < a.ipt; ++r) Ph::item(m, (int)blockIdx.y, a.opt, tl.y + r * (int)blockDim.x + (int)threadIdx.x);
}
// Per-member scalar work, one thread per member.
template <class Ph> __global__ void __launch_bounds__(128) k_phase_members(BatchArgs a) {
    gfk::gf_pdl_entry();
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < a.nmembers) Ph::member(a.members[k]);
}

#define GF_PHASE(name, k, r) struct name { static constexpr int kind = k, regs = r; \
    static __device__ __forceinline__ void item(const BatchMember &m, int part, int opt, GF_IDX i)
using namespace gfk;
// the joint launches of an ordinary step (k_step_a to k_step_d)
GF_PHASE(PhStepA, K_N, 128) {
    if (part == 0) b_k_rheol<float>(m.P, m.C, m.A, m.d, 0, 0, i);
    else b_k_therm_prep32(m.P, m.A, m.d, (float *)m.A.t_coef, i);
} };
GF_PHASE(PhStepB, K_N, 80) {
    if (part == 0) b_k_node<float>(m.P, m.C, m.A, m.d, i);
    else if (part == 1)
        b_k_therm_sweep32(m.P, m.C, m.A, m.d, (const float *)m.A.t_coef, (float *)m.A.t_delta0, m.A.t_delta1, 0, i);
    else b_k_rheol_avg<float>(m.C, m.A, m.d, opt == 2 ? 1 : 0, i);
} };
GF_PHASE(PhStepC, K_N, 64) {
    if (part == 0) {
        b_k_therm_sweep32(m.P, m.C, m.A, m.d, (const float *)m.A.t_coef, (float *)m.A.t_delta0, m.A.t_delta1, 1, i);
        if (opt == 2 && i == 0) b_k_rheol_clock(m.C, 1);
    } else if (m.movegrid && i < m.d.N) {
        b_k_move_cord(m.C, m.A, m.d, (GF_IDX)((part - 1) * m.d.N) + i);
    }
} };
GF_PHASE(PhStepD, K_N, 128) { // opt: time advances here (par.f90:86), unless dt_mass follows
    if (part == 1) b_k_therm_apply32(m.P, m.A, m.d, m.A.t_delta1, i);
    else if (m.movegrid) b_k_move_elem<float>(m.C, m.A, m.d, opt, i);
    else if (opt && i == 0) m.C->time = m.C->time + m.C->dt;
} };
// the same parts one by one, for steps that need the new temperatures first
GF_PHASE(PhPrep, K_N, 80) { b_k_therm_prep32(m.P, m.A, m.d, (float *)m.A.t_coef, i); } };
GF_PHASE(PhSweep, K_N, 64) {
    b_k_therm_sweep32(m.P, m.C, m.A, m.d, (const float *)m.A.t_coef, (float *)m.A.t_delta0, m.A.t_delta1, opt, i);
} };
GF_PHASE(PhApply, K_N, 80) { b_k_therm_apply32(m.P, m.A, m.d, m.A.t_delta1, i); } };
GF_PHASE(PhMarkers, K_M, 80) { b_k_phase_markers32(m.P, m.A, m.d, m.nmarkers, i); } };
GF_PHASE(PhRecount, K_E, 80) { b_k_phase_recount<float>(m.P, m.C, m.A, m.d, 0, i); } };
GF_PHASE(PhRheol, K_E, 128) { b_k_rheol<float>(m.P, m.C, m.A, m.d, opt, 0, i); } };
GF_PHASE(PhNode, K_N, 80) { // and fl_rheol's averaging
    if (part == 0) b_k_node<float>(m.P, m.C, m.A, m.d, i);
    else b_k_rheol_avg<float>(m.C, m.A, m.d, opt == 2 ? 1 : 0, i);
} };
GF_PHASE(PhCord, K_N, 80) {
    if (opt == 2 && part == 0 && i == 0) b_k_rheol_clock(m.C, 1);
    if (m.movegrid && i < m.d.N) b_k_move_cord(m.C, m.A, m.d, (GF_IDX)(part * m.d.N) + i);
} };
GF_PHASE(PhMove, K_E, 80) {
    if (m.movegrid) b_k_move_elem<float>(m.C, m.A, m.d, opt, i);
    else if (opt && i == 0) m.C->time = m.C->time + m.C->dt;
} };
GF_PHASE(PhDens, K_E, 80) { b_k_elem_dens<float>(m.P, m.C, m.A, m.d, i); } };
GF_PHASE(PhRmass, K_N, 80) { b_k_node_gather_tri<float>((const float *)m.A.e_tri, m.A.rmass, m.d, i); } };
GF_PHASE(PhDt, K_EN, 80) { b_k_dt_reduce<float>(m.P, m.C, m.A, m.d, i); } };
GF_PHASE(PhAm3, K_E, 80) { if (m.idt_scale != 0) b_k_elem_am3<float>(m.P, m.C, m.A, m.d, i); } };
GF_PHASE(PhAmass, K_N, 80) {
    if (m.idt_scale != 0) b_k_node_gather_tri<float>((const float *)m.A.e_tri, m.A.amass, m.d, i);
    else if (i < m.d.N) m.A.amass[i] = m.A.rmass[i];
} };
#undef GF_PHASE
struct MemFrac { static __device__ void member(const BatchMember &m) { b_k_frac_fix<float>(m.P, m.C, m.A, m.d); } };
struct MemDtReset { static __device__ void member(const BatchMember &m) { b_k_dt_reset(m.C); } };
struct MemDtScalars { static __device__ void member(const BatchMember &m) { b_k_dt_scalars(m.P, m.C); } };
// every member's status side by side (fetched one by one they cost some 7 us
// each: 0.4 ms of ten steps of 64 members)
__global__ void k_batch_status(const BatchMember *members, int n, int *out) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < n) out[k] = members[k].C->status;
}
struct MemTime { static __device__ void member(const BatchMember &m) { m.C->time = m.C->time + m.C->dt; } };

// ---------------------------------------------------------------- surrogate I/O
// Fields of every member resampled to an H x W grid (channels last, FP32):
// 0 vx, 1 vz, 2 sxx, 3 szz, 4 sxz (total stress, mean of the 4 triangles),
// 5 plastic strain, 6 temperature, 7 fraction of phase `phase_id`,
// 8 vertical displacement from the regular start-up mesh.  Bilinear in the
// node / element-centre index space of each member (the members' domains
// keep the grid's aspect).
constexpr int SAMPLE_CH = 9;

struct GridArgs {
    const BatchMember *members;
    int n, H, W, phase_id;
    float *grid;       // [n][H][W][SAMPLE_CH]
    const float *pred; // injection source, same layout
};

__device__ __forceinline__ void lerp_index(float f, int n, int &i0, float &w) {
    // f in [0, n-1] -> cell i0 in [0, n-2], weight of i0 + 1
    if (n < 2) {
        i0 = 0;
        w = 0.0f;
        return;
    }
    f = fminf(fmaxf(f, 0.0f), (float)(n - 1));
    i0 = min((int)f, n - 2);
    w = f - (float)i0;
}

// a float as a double by integer operations; only subnormals, infinities and
// NaNs take the conversion instruction (a slot of the FP64 pipe)
__device__ __forceinline__ double sample_f2d(float f) {
    const unsigned u = __float_as_uint(f), e = (u >> 23) & 0xffu;
    if (e - 1u >= 254u && (u << 1) != 0u) return (double)f;
    return gfk::gf_f2d(f);
}
// an element's mean of stress component c over its triangles, as stored (normal
// components exclude -p_ref)
__device__ __forceinline__ double mean_stress(const BatchMember &m, long long e, int c) {
    const float *st = (const float *)m.A.stress0;
    double s = gfk::gf_plus_pzero(sample_f2d(st[gf_s(m.d, e, c, 0)]));
#pragma unroll
    for (int k = 1; k < 4; ++k) s = s + sample_f2d(st[gf_s(m.d, e, c, k)]);
    return gfk::gf_scale<-2>(s);
}
__device__ double elem_value(const BatchMember &m, long long e, int ch, int phase_id) {
    switch (ch) {
    case 2: case 3: return mean_stress(m, e, ch - 2) - m.A.p_ref[e];
    case 4: return mean_stress(m, e, 2);
    case 5: return (double)((const float *)m.A.aps)[e];
    default: return m.A.phase_ratio[gf_pr(m.d, e, phase_id - 1)];
    }
}

__device__ double node_value(const BatchMember &m, long long n, int j, int ch) {
    const GfDims &d = m.d;
    switch (ch) {
    case 0: return m.A.vel[n];
    case 1: return m.A.vel[d.N + n];
    case 6: return m.A.temp[n];
    default: return m.A.cord[d.N + n] - (m.z0 + m.rzbo * (double)j / (double)(d.nz - 1));
    }
}

// A sampled value is the FP64 bilinear sum rounded to FP32 (sample_plain).  Nearly
// all of them are decided without the FP64 pipe: the sum is formed in FP32 pairs
// (hi + lo) with an error below 2^-42 of the largest corner, and where adding and
// subtracting that much rounds to the same float, that float is the result.  Only
// the others (a sum next to a rounding boundary, cancelling corners, values too
// small for pairs, infinities and NaNs) are evaluated in FP64.  All values in FP64
// (200 operations a point, the elements' means anew at each of a point's corners)
// took 1.23 ms for 64 members on a 128 x 384 grid, with the means formed once and
// half of the products on the integer pipes 0.38 ms, this 0.19 ms.
struct ff {
    float h, l;
};
__device__ __forceinline__ ff ff_two(float a, float b) { // a + b exactly
    const float s = __fadd_rn(a, b), t = __fsub_rn(s, a);
    return ff{s, __fadd_rn(__fsub_rn(a, __fsub_rn(s, t)), __fsub_rn(b, t))};
}
// v a + w b for weights v, w in [0, 1] of sum 1 (to a rounding)
__device__ __forceinline__ ff ff_mix(float v, ff a, float w, ff b) {
    const float p = __fmul_rn(v, a.h), q = __fmul_rn(w, b.h);
    const float ep = fmaf(v, a.l, fmaf(v, a.h, -p)), eq = fmaf(w, b.l, fmaf(w, b.h, -q));
    const ff s = ff_two(p, q);
    return ff{s.h, __fadd_rn(s.l, __fadd_rn(ep, eq))};
}
// The bilinear sum rounded to FP32; false where the rounding is not certain.
// With corners up to M whose lo parts are below 2^-23 M and err by 2^-47 M, the
// roundings of the lo parts add up to 14 x 2^-47 M: 6 in a sum along x (the
// corners' 1, products' ends 1.5, additions 1.5 and 2; lo parts then up to twice as
// large), 8 in the one along z (2.5, 2.5, 3).  The bound taken, 32, leaves room for
// those of the test itself and of the FP64 sum.  `floor`: what the corners' splits
// may have lost to underflow.
__device__ __forceinline__ bool ff_bilinear(ff a, ff b, ff c, ff d, float wx, float wy, float floor, float &out) {
    const float vx = 1 - wx, vy = 1 - wy;
    const ff r = ff_mix(vy, ff_mix(vx, a, wx, b), wy, ff_mix(vx, c, wx, d));
    const ff n = ff_two(r.h, r.l);
    const float m = fmaxf(fmaxf(fabsf(a.h), fabsf(b.h)), fmaxf(fabsf(c.h), fabsf(d.h)));
    const float eps = fmaf(m, 0x1p-42f, floor);
    out = __fadd_rn(n.h, __fadd_rn(n.l, eps));
    return out == __fadd_rn(n.h, __fsub_rn(n.l, eps)); // (false for NaN)
}
// the 48 leading bits of a double, truncated, without the FP64 pipe; NaN where a
// pair cannot hold them (below 2^-78 but for zero, from 2^128 on)
__device__ __forceinline__ ff ff_of(double x) {
    unsigned lo, hi;
    gfk::gf_dsplit(x, lo, hi);
    const unsigned e = ((hi >> 20) & 0x7ffu) - 1023u + 127u;
    if (e - 49u >= 206u) return ff{__uint_as_float(((hi << 1) | lo) == 0u ? 0u : 0x7fc00000u), 0.0f};
    const unsigned sg = hi & 0x80000000u;
    const float h = __uint_as_float(sg | (e << 23) | ((hi & 0xfffffu) << 3) | (lo >> 29));
    const float l = __uint2float_rz((lo >> 5) & 0xffffffu); // the next 24 bits, scaled by 2^(e - 127 - 47)
    return ff{h, l * __uint_as_float(sg | ((e - 47u) << 23))};
}

// the same for a float
__device__ __forceinline__ ff ff_of(float x) { return ff{fabsf(x) >= 0x1p-78f || x == 0.0f ? x : __uint_as_float(0x7fc00000u), 0.0f}; }

// The elements' share of a sample: total stresses (mean of the four
// triangles, as elem_value forms them) and the phase fraction as pairs, once
// per element.
__global__ void k_sample_elems(GridArgs g, const int2 *tiles, int ntile, int ipt, float4 *means) {
    for (int t = blockIdx.x; t < ntile; t += gridDim.x) {
        const int2 tl = tiles[t];
        const BatchMember &m = g.members[tl.x];
        for (int r = 0; r < ipt; ++r) {
            const int e = tl.y + r * (int)blockDim.x + (int)threadIdx.x;
            if (e >= m.d.E) continue;
            const ff xx = ff_of(elem_value(m, e, 2, 0)), zz = ff_of(elem_value(m, e, 3, 0)),
                     xz = ff_of(elem_value(m, e, 4, 0)), f = ff_of(elem_value(m, e, 7, g.phase_id));
            float4 *o = means + 2 * (m.e0 + e);
            o[0] = make_float4(xx.h, xx.l, zz.h, zz.l);
            o[1] = make_float4(xz.h, xz.l, f.h, f.l);
        }
    }
}

// The value itself: FP64 corners, weights and sums
__device__ __noinline__ float sample_plain(const BatchMember &m, int ch, int phase_id, int j0, int j1, int i0, int i1,
                                           float wx, float wy) {
    double v[4];
    const bool node = ch == 0 || ch == 1 || ch == 6 || ch == 8;
    for (int k = 0; k < 4; ++k) {
        const int j = k < 2 ? j0 : j1, i = k & 1 ? i1 : i0;
        v[k] = node ? node_value(m, gf_node(m.d, j, i), j, ch) : elem_value(m, gf_elem(m.d, j, i), ch, phase_id);
    }
    return (float)((1 - wy) * ((1 - wx) * v[0] + wx * v[1]) + wy * ((1 - wx) * v[2] + wx * v[3]));
}

// 32 x 32 grid points of one member per CTA: lanes run along the depth, the
// members' fastest index, and the points leave through shared memory in rows
// of the grid.
__global__ void __launch_bounds__(256) k_sample(GridArgs g, const float4 *means, int ty, int tx) {
    constexpr int ROW = 32 * SAMPLE_CH + 1;
    __shared__ float tile[32 * ROW];
    const int b = blockIdx.x, mi = b / (ty * tx), q = b - mi * (ty * tx);
    const int gy0 = (q / tx) * 32, gx0 = (q % tx) * 32;
    const BatchMember &m = g.members[mi];
    const GfDims d = m.d;
    const DevArrays &A = m.A;
    const int nx = d.nx, nz = d.nz, N = (int)d.N;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, gy = gy0 + lane;
    const float4 *mean = means + 2 * m.e0;
    // grid point k of `size` in the index space of n nodes
    auto at = [](int k, int n, int size) { return (k + 0.5f) * (n - 1) / size; };
    if (gy < g.H) {
        int jn, je;
        float wyn, wye;
        lerp_index(at(gy, nz, g.H), nz, jn, wyn);
        lerp_index(at(gy, nz, g.H) - 0.5f, nz - 1, je, wye);
        const int je1 = min(je + 1, nz - 2);
        // heights of rows jn and jn + 1 of the regular start-up mesh
        auto ref = [&](int j) {
            return m.z0 + gfk::gf_ddiv(gfk::gf_mul(m.rzbo, gfk::gf_f2d((float)j)), gfk::gf_f2d((float)(nz - 1)));
        };
        const double r0 = ref(jn), r1 = ref(jn + 1);
        for (int x = warp; x < 32 && gx0 + x < g.W; x += 8) {
            const int gx = gx0 + x;
            float *o = tile + lane * ROW + x * SAMPLE_CH;
            int i0;
            float wx;
            lerp_index(at(gx, nx, g.W), nx, i0, wx);
            const int a = gf_node(d, jn, i0), c = a + 1, bb = a + nz, dd = bb + 1; // (j,i), (j+1,i), (j,i+1), (j+1,i+1)
            float v[SAMPLE_CH];
            unsigned sure = 0u; // channels decided in pairs
            auto put = [&](int ch, ff p, ff r, ff q, ff w, float fx, float fy, float floor) {
                if (ff_bilinear(p, r, q, w, fx, fy, floor, v[ch])) sure |= 1u << ch;
            };
            // (a hi/lo split loses what lies below 2^-126)
            auto nodes = [&](int ch, const float *h, const float *l, int off) {
                put(ch, ff{h[off + a], l[off + a]}, ff{h[off + bb], l[off + bb]}, ff{h[off + c], l[off + c]},
                    ff{h[off + dd], l[off + dd]}, wx, wyn, 0x1p-112f);
            };
            nodes(0, A.vel_hi, A.vel_lo, 0);
            nodes(1, A.vel_hi, A.vel_lo, N);
            nodes(6, A.temp_hi, A.temp_lo, 0);
            const double *z = A.cord + N;
            put(8, ff_of(z[a] - r0), ff_of(z[bb] - r0), ff_of(z[c] - r1), ff_of(z[dd] - r1), wx, wyn, 0.0f);
            int ie;
            float wxe;
            lerp_index(at(gx, nx, g.W) - 0.5f, nx - 1, ie, wxe);
            const int ie1 = min(ie + 1, nx - 2);
            const int ea = gf_elem(d, je, ie), eb = gf_elem(d, je, ie1), ec = gf_elem(d, je1, ie), ed = gf_elem(d, je1, ie1);
            {
                const float4 p = mean[2 * ea], r = mean[2 * eb], s = mean[2 * ec], t = mean[2 * ed];
                put(2, ff{p.x, p.y}, ff{r.x, r.y}, ff{s.x, s.y}, ff{t.x, t.y}, wxe, wye, 0.0f);
                put(3, ff{p.z, p.w}, ff{r.z, r.w}, ff{s.z, s.w}, ff{t.z, t.w}, wxe, wye, 0.0f);
            }
            {
                const float4 p = mean[2 * ea + 1], r = mean[2 * eb + 1], s = mean[2 * ec + 1], t = mean[2 * ed + 1];
                put(4, ff{p.x, p.y}, ff{r.x, r.y}, ff{s.x, s.y}, ff{t.x, t.y}, wxe, wye, 0.0f);
                put(7, ff{p.z, p.w}, ff{r.z, r.w}, ff{s.z, s.w}, ff{t.z, t.w}, wxe, wye, 0.0f);
            }
            const float *aps = (const float *)A.aps;
            put(5, ff_of(aps[ea]), ff_of(aps[eb]), ff_of(aps[ec]), ff_of(aps[ed]), wxe, wye, 0.0f);
#pragma unroll
            for (int ch = 0; ch < SAMPLE_CH; ++ch) o[ch] = v[ch];
            for (unsigned rest = 0x1ffu & ~sure; rest; rest &= rest - 1u) {
                const int ch = __ffs(rest) - 1;
                const bool node = ch == 0 || ch == 1 || ch == 6 || ch == 8;
                o[ch] = node ? sample_plain(m, ch, g.phase_id, jn, jn + 1, i0, i0 + 1, wx, wyn)
                             : sample_plain(m, ch, g.phase_id, je, je1, ie, ie1, wxe, wye);
            }
        }
    }
    __syncthreads();
    const int cols = min(32, g.W - gx0) * SAMPLE_CH;
    for (int y = warp; y < 32 && gy0 + y < g.H; y += 8) {
        float *out = g.grid + (((long long)mi * g.H + gy0 + y) * g.W + gx0) * SAMPLE_CH;
        for (int k = lane; k < cols; k += 32) out[k] = tile[y * ROW + k];
    }
}

// bilinear read of one channel of member mi's grid at grid coordinates (fy, fx)
__device__ float grid_at(const GridArgs &g, int mi, float fy, float fx, int ch) {
    int i0, j0;
    float wx, wy;
    lerp_index(fx, g.W, i0, wx);
    lerp_index(fy, g.H, j0, wy);
    const float *G = g.pred + (long long)mi * g.H * g.W * SAMPLE_CH;
    auto at = [&](int j, int i) { return G[((long long)j * g.W + i) * SAMPLE_CH + ch]; };
    return (1 - wy) * ((1 - wx) * at(j0, i0) + wx * at(j0, i0 + 1)) + wy * ((1 - wx) * at(j0 + 1, i0) + wx * at(j0 + 1, i0 + 1));
}

// grid -> member nodes: velocity, temperature, vertical position
__global__ void k_inject_nodes(GridArgs g, const int2 *tiles, int ntile, int ipt) {
    for (int t = blockIdx.x; t < ntile; t += gridDim.x) {
        const int2 tl = tiles[t];
        const BatchMember &m = g.members[tl.x];
        for (int r = 0; r < ipt; ++r) {
            long long n = (long long)tl.y + (long long)r * blockDim.x + threadIdx.x;
            if (n >= m.d.N) continue;
            const int j = (int)(n % m.d.nz), i = (int)(n / m.d.nz);
            const float fx = (float)i * g.W / (m.d.nx - 1) - 0.5f, fy = (float)j * g.H / (m.d.nz - 1) - 0.5f;
            const double vx = grid_at(g, tl.x, fy, fx, 0), vz = grid_at(g, tl.x, fy, fx, 1);
            const double z = m.z0 + m.rzbo * (double)j / (double)(m.d.nz - 1) + (double)grid_at(g, tl.x, fy, fx, 8);
            m.A.vel[n] = vx;
            m.A.vel[m.d.N + n] = vz;
            const double tn = grid_at(g, tl.x, fy, fx, 6);
            m.A.temp[n] = tn;
            m.A.temp_hi[n] = (float)tn;
            m.A.temp_lo[n] = (float)(tn - (double)(float)tn);
            m.A.cord[m.d.N + n] = z;
            const float hx = (float)vx, hz = (float)vz, hc = (float)z;
            m.A.vel_hi[n] = hx;
            m.A.vel_lo[n] = (float)(vx - (double)hx);
            m.A.vel_hi[m.d.N + n] = hz;
            m.A.vel_lo[m.d.N + n] = (float)(vz - (double)hz);
            m.A.cord_hi[m.d.N + n] = hc;
            m.A.cord_lo[m.d.N + n] = (float)(z - (double)hc);
        }
    }
}

// grid -> member elements: stresses (the out-of-plane stress keeps its
// deviation from the in-plane mean), plastic strain; areas of the moved mesh
__global__ void k_inject_elems(GridArgs g, const int2 *tiles, int ntile, int ipt, DevClock *err) {
    for (int t = blockIdx.x; t < ntile; t += gridDim.x) {
        const int2 tl = tiles[t];
        const BatchMember &m = g.members[tl.x];
        const GfDims &d = m.d;
        for (int r = 0; r < ipt; ++r) {
            long long e = (long long)tl.y + (long long)r * blockDim.x + threadIdx.x;
            if (e >= d.E) continue;
            const int j = (int)(e % (d.nz - 1)), i = (int)(e / (d.nz - 1));
            const float fx = (i + 0.5f) * g.W / (d.nx - 1) - 0.5f, fy = (j + 0.5f) * g.H / (d.nz - 1) - 0.5f;
            float *st = (float *)m.A.stress0;
            const double pr = m.A.p_ref[e];
            const double sxx = grid_at(g, tl.x, fy, fx, 2), szz = grid_at(g, tl.x, fy, fx, 3),
                         sxz = grid_at(g, tl.x, fy, fx, 4);
            for (int k = 0; k < 4; ++k) {
                double oxx = (double)st[gf_s(d, e, 0, k)] - pr, ozz = (double)st[gf_s(d, e, 1, k)] - pr;
                double oyy = (double)st[gf_s(d, e, 3, k)] - pr;
                double nyy = oyy + 0.5 * ((sxx - oxx) + (szz - ozz));
                st[gf_s(d, e, 0, k)] = (float)(sxx + pr);
                st[gf_s(d, e, 1, k)] = (float)(szz + pr);
                st[gf_s(d, e, 2, k)] = (float)sxz;
                st[gf_s(d, e, 3, k)] = (float)(nyy + pr);
            }
            ((float *)m.A.aps)[e] = fmaxf(0.0f, grid_at(g, tl.x, fy, fx, 5));
            gfk::Quad q;
            gfk::load_quad(m.A.cord, d, j, i, q);
            const double *x = q.x, *y = q.y;
            double det[4] = {((x[1] * y[2] - y[1] * x[2]) - (x[0] * y[2] - y[0] * x[2])) + (x[0] * y[1] - y[0] * x[1]),
                             ((x[1] * y[3] - y[1] * x[3]) - (x[2] * y[3] - y[2] * x[3])) + (x[2] * y[1] - y[2] * x[1]),
                             ((x[1] * y[3] - y[1] * x[3]) - (x[0] * y[3] - y[0] * x[3])) + (x[0] * y[1] - y[0] * x[1]),
                             ((x[3] * y[2] - y[3] * x[2]) - (x[0] * y[2] - y[0] * x[2])) + (x[0] * y[3] - y[0] * x[3])};
            for (int k = 0; k < 4; ++k) {
                ((float *)m.A.area)[gf_ek(d, e, k)] = (float)(1.0 / det[k]);
                if (det[k] <= 0.0) gfk::set_status(m.C, 41, (int)e);
            }
        }
    }
    (void)err;
}

// Force imbalance at the free nodes (fl_node.f90 without damping): per member
// sum |F| and sum (|gravity| + sum over triangles |stress-divergence term|).
__global__ void k_force_residual(const BatchMember *members, const int2 *tiles, int ntile, int ipt, double *acc) {
    for (int t = blockIdx.x; t < ntile; t += gridDim.x) {
        const int2 tl = tiles[t];
        const BatchMember &m = members[tl.x];
        const GfDims &d = m.d;
        double sf = 0.0, ss = 0.0;
        for (int r = 0; r < ipt; ++r) {
            long long n = (long long)tl.y + (long long)r * blockDim.x + threadIdx.x;
            if (n >= d.N) continue;
            const int j = (int)(n % d.nz), i = (int)(n / d.nz);
            const int c0 = m.A.ncod[n], c1 = m.A.ncod[d.N + n];
            const int kk[4][3] = {{1, 2, 3}, {0, 1, 2}, {0, 1, 3}, {0, 2, 3}};
            const int mm[4][3] = {{2, 2, 1}, {1, 1, 1}, {2, 0, 2}, {0, 0, 0}};
            const float *st = (const float *)m.A.stress0;
            const float *area = (const float *)m.A.area;
            double fx = 0.0, fy = 0.0, mag = 0.0;
            for (int qd = 0; qd < 4; ++qd) {
                int je = j + (qd < 2 ? -1 : 0), ie = i + ((qd & 1) ? 0 : -1);
                if (je < 0 || ie < 0 || je > d.nz - 2 || ie > d.nx - 2) continue;
                long long e = gf_elem(d, je, ie);
                gfk::Quad q;
                gfk::load_quad(m.A.cord, d, je, ie, q);
                double ar[4];
                for (int k = 0; k < 4; ++k) ar[k] = (double)area[gf_ek(d, e, k)];
                double dx[3][4], dz[3][4];
                gfk::shape_derivs<double>(q, ar, dx, dz);
                const double pe = m.A.p_ref[e];
                for (int k = 0; k < 3; ++k) {
                    int tt = kk[qd][k], mq = mm[qd][k];
                    double factor = 0.25 / ar[tt];
                    double sxx = (double)st[gf_s(d, e, 0, tt)] - pe, szz = (double)st[gf_s(d, e, 1, tt)] - pe,
                           sxz = (double)st[gf_s(d, e, 2, tt)];
                    double tx = factor * (sxx * dx[mq][tt] + sxz * dz[mq][tt]);
                    double ty = factor * (sxz * dx[mq][tt] + szz * dz[mq][tt]);
                    fx -= tx;
                    fy -= ty;
                    mag += sqrt(tx * tx + ty * ty);
                }
            }
            const double grav = m.A.rmass[n] * m.P->g;
            fy -= grav;
            if (c0 == 1) fx = 0.0; // fixed velocity components carry reactions
            if (c1 == 1) fy = 0.0;
            sf += sqrt(fx * fx + fy * fy);
            ss += mag + fabs(grav);
        }
        sf = gfk::warp_sum(sf);
        ss = gfk::warp_sum(ss);
        if ((threadIdx.x & 31) == 0) {
            atomicAdd(&acc[2 * tl.x], sf);
            atomicAdd(&acc[2 * tl.x + 1], ss);
        }
    }
}

} // namespace

constexpr int GF_BATCH_CAPTURE = 8;
struct gf_batch {
    std::vector<gf_ctx *> members;
    std::vector<GfMemberView> views;
    BatchMember *d_members = nullptr;
    std::vector<BatchMember> records; // what d_members holds
    int2 *d_tiles[K_KINDS] = {};
    int ntile[K_KINDS] = {};
    cudaStream_t s = nullptr;
    std::shared_ptr<GfEvent> done = std::make_shared<GfEvent>(); // behind a call that returns before its kernels end
    gf_batch_config cfg{256, 2, 1, 10};
    int grid = 0;  // CTAs of an element phase
    int sms = 1;   // multiprocessors
    int ipt = 1;   // items per thread of the tile tables (the configuration's, or fewer for a small batch)
    int merge = 0; // every member allows the joint launches
    long long elements = 0;
    struct Graph {
        std::vector<unsigned> sigs;
        cudaGraphExec_t exec; // null: not captured yet
        int uses;             // before it is captured
    };
    std::vector<Graph> graphs;
    // device copy of the fields gf_batch_inject overwrites (restore point)
    void *backup = nullptr;
    std::vector<size_t> backup_off;
    int *status = nullptr, *h_status = nullptr; // the members' status words, device and pinned host
    float4 *means = nullptr; // gf_batch_sample's element pairs (two per element)
};

namespace {
// (device pointer, bytes) of every field of member v that injection writes
std::vector<std::pair<void *, size_t>> injected_fields(const GfMemberView &v) {
    const size_t N = (size_t)v.d.N, E = (size_t)v.d.E;
    return {{v.A.vel, 2 * N * sizeof(double)},    {v.A.temp, N * sizeof(double)},
            {v.A.cord, 2 * N * sizeof(double)},   {v.A.stress0, 16 * E * sizeof(float)},
            {v.A.aps, E * sizeof(float)},         {v.A.area, 4 * E * sizeof(float)},
            {v.A.cord_hi, 2 * N * sizeof(float)}, {v.A.cord_lo, 2 * N * sizeof(float)},
            {v.A.vel_hi, 2 * N * sizeof(float)},  {v.A.vel_lo, 2 * N * sizeof(float)},
            {v.A.temp_hi, N * sizeof(float)},     {v.A.temp_lo, N * sizeof(float)}};
}
} // namespace

namespace {

int batch_cuda(cudaError_t e, const char *what) {
    if (e == cudaSuccess) return GF_OK;
    std::fprintf(stderr, "geoflac_gb300: CUDA error in %s: %s\n", what, cudaGetErrorString(e));
    return GF_ERR_CUDA;
}
#define GB_CK(call)                                                                                                    \
    do {                                                                                                               \
        int _rc = batch_cuda((call), #call);                                                                           \
        if (_rc) return _rc;                                                                                           \
    } while (0)

void drop_graphs(gf_batch *b) {
    for (auto &g : b->graphs)
        if (g.exec) cudaGraphExecDestroy(g.exec);
    b->graphs.clear();
}

long long kind_count(const GfMemberView &v, int kind) {
    switch (kind) {
    case K_E: return v.d.E;
    case K_N: return v.d.N;
    case K_M: return v.nmarkers;
    default: return std::max(v.d.E, v.d.N);
    }
}

// Tile tables for the current configuration.  A tile of several items per
// thread saves stagings of the member record; a batch with fewer elements than
// the SMs hold threads at that depth is cut finer, since its tiles would not
// fill them once (a member's result does not depend on the tile depth).
int build_tables(gf_batch *b) {
    const gf_batch_config &c = b->cfg;
    if (c.threads != 128 && c.threads != 256 && c.threads != 512) return GF_ERR_ARG;
    if (c.items_per_thread < 1 || c.items_per_thread > 64 || c.ctas_per_sm < 1) return GF_ERR_ARG;
    int dev = 0;
    GB_CK(cudaGetDevice(&dev));
    GB_CK(cudaDeviceGetAttribute(&b->sms, cudaDevAttrMultiProcessorCount, dev));
    b->ipt = c.items_per_thread;
    while (b->ipt > 1 && b->elements < (long long)b->sms * 2048 * b->ipt) --b->ipt;
    const long long tile = (long long)c.threads * b->ipt;
    std::vector<int2> tiles[K_KINDS]; // until their copies end
    for (int kind = 0; kind < K_KINDS; ++kind) {
        std::vector<int2> &t = tiles[kind];
        for (size_t m = 0; m < b->views.size(); ++m) {
            long long n = kind_count(b->views[m], kind);
            for (long long s = 0; s < n; s += tile) {
                if (s > 0x7fffffff) return GF_ERR_ARG;
                t.push_back(make_int2((int)m, (int)s));
            }
        }
        if (b->d_tiles[kind]) cudaFree(b->d_tiles[kind]);
        b->d_tiles[kind] = nullptr;
        b->ntile[kind] = (int)t.size();
        if (!t.empty()) {
            GB_CK(cudaMalloc(&b->d_tiles[kind], t.size() * sizeof(int2)));
            GB_CK(cudaMemcpyAsync(b->d_tiles[kind], t.data(), t.size() * sizeof(int2), cudaMemcpyHostToDevice, b->s));
        }
    }
    // (a plain copy from pageable memory may return before it has landed, and is not
    // in the order of a non-blocking stream)
    GB_CK(cudaStreamSynchronize(b->s));
    b->grid = b->ntile[K_E];
    drop_graphs(b);
    return GF_OK;
}

// The members' records as they are now.
std::vector<BatchMember> member_records(const gf_batch *b) {
    std::vector<BatchMember> h(b->views.size());
    long long e0 = 0;
    for (size_t m = 0; m < h.size(); ++m) {
        const GfMemberView &v = b->views[m];
        std::memset(&h[m], 0, sizeof(BatchMember));
        h[m].P = v.P;
        h[m].C = v.C;
        h[m].A = v.A;
        h[m].d = v.d;
        h[m].idt_scale = v.idt_scale;
        h[m].movegrid = v.movegrid;
        h[m].nmarkers = v.nmarkers;
        h[m].z0 = v.z0;
        h[m].rzbo = v.rzbo;
        h[m].e0 = e0;
        e0 += v.d.E;
    }
    return h;
}
int upload_members(gf_batch *b) {
    b->records = member_records(b);
    GB_CK(cudaMemcpyAsync(b->d_members, b->records.data(), b->records.size() * sizeof(BatchMember),
                          cudaMemcpyHostToDevice, b->s));
    GB_CK(cudaStreamSynchronize(b->s)); // (as in build_tables)
    return GF_OK;
}

// Enqueue one FLAC step (flac.f90:5-91, mixed precision) of every member.
struct StepLauncher {
    gf_batch *b;
    BatchArgs a;
    cudaError_t err = cudaSuccess;
    explicit StepLauncher(gf_batch *batch) : b(batch) {
        std::memset(&a, 0, sizeof a);
        a.members = b->d_members;
        a.nmembers = (int)b->members.size();
        for (int k = 0; k < K_KINDS; ++k) {
            a.tile[k] = b->d_tiles[k];
            a.ntile[k] = b->ntile[k];
        }
        a.ipt = b->ipt;
    }
    void launch(void (*kern)(BatchArgs), dim3 grid, int threads, int opt) {
        if (grid.x == 0 || err != cudaSuccess) return;
        a.opt = opt;
        cudaLaunchConfig_t lc;
        std::memset(&lc, 0, sizeof lc);
        lc.gridDim = grid;
        lc.blockDim = dim3((unsigned)threads);
        lc.stream = b->s;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        lc.attrs = attr;
        lc.numAttrs = 1;
        err = cudaLaunchKernelEx(&lc, kern, a);
    }
    template <class Ph> void phase(unsigned parts = 1, int opt = 0) {
        launch(k_phase<Ph>, dim3((unsigned)b->ntile[Ph::kind], parts), b->cfg.threads, opt);
    }
    template <class Ph> void scalars() {
        launch(k_phase_members<Ph>, dim3((unsigned)((a.nmembers + 127) / 128)), 128, 0);
    }
    int step(unsigned sig) {
        const int avg = (sig & (8u << 8)) ? 2 : ((sig & (4u << 8)) ? 1 : 0);
        const int dtm = (sig & 32u) ? 1 : 0;
        // Steps whose fl_rheol / fl_node read nothing the thermal update
        // writes (no viscosity update, no change_phase; every member without
        // thermal stress, Winkler foundation or flux bottom condition)
        const bool joint = b->merge && (sig & 1u) && !(sig & 2u) && !(sig & 4u);
        if (joint) {
            // (the sweep coefficients beside fl_rheol while both fit the SMs at
            // once, as in the single-model step: 64 members 468 against 481 us)
            const bool beside = b->ntile[K_N] <= b->sms;
            if (!beside) phase<PhPrep>();
            phase<PhStepA>(beside ? 2 : 1);
            phase<PhStepB>(avg > 0 ? 3 : 2, avg);
            phase<PhStepC>(3, avg);
            phase<PhStepD>(2, !dtm);
        } else {
            phase<PhPrep>();
            phase<PhSweep>(1, 0);
            phase<PhSweep>(1, 1);
            phase<PhApply>();
            if (sig & 1u) {
                if (sig & 2u) { // change_phase
                    phase<PhMarkers>();
                    phase<PhRecount>();
                }
                phase<PhRheol>(1, (sig & 4u) ? 1 : 0);
                phase<PhNode>(avg > 0 ? 2 : 1, avg);
                phase<PhCord>(2, avg);
                phase<PhMove>(1, !dtm);
            }
        }
        if (sig & 1u) {
            if (sig & 16u) { // rmasses
                phase<PhDens>();
                scalars<MemFrac>();
                phase<PhRmass>();
            }
            if (dtm) { // dt_mass, then the time advance with the new dt (par.f90:86)
                scalars<MemDtReset>();
                phase<PhDt>();
                scalars<MemDtScalars>();
                phase<PhAm3>();
                phase<PhAmass>();
                scalars<MemTime>();
            }
        } else {
            scalars<MemTime>();
        }
        GB_CK(err);
        return GF_OK;
    }
};

int launch_step(gf_batch *b, unsigned sig) { return StepLauncher(b).step(sig); }

// Signatures of the next n steps (all members share them).
std::vector<unsigned> next_sigs(gf_batch *b, int n, std::vector<int> &nl, std::vector<int> &ns) {
    // simulate the host bookkeeping of member 0 without touching it
    const GfMemberView &v = b->views[0];
    std::vector<unsigned> sigs;
    int nloop = v.nloop, nsrate = v.nsrate;
    for (int k = 0; k < n; ++k) {
        unsigned sig = 0;
        if (v.itherm != 2) {
            sig |= 1u;
            if (nloop % v.ifreq_rmasses == 0) sig |= 2u | 16u;
            if (nloop % v.ifreq_visc == 0) sig |= 4u;
            if (nsrate == v.ifreq_avgsr) sig |= 8u << 8;
            else if (nsrate == -1) sig |= 4u << 8;
            if (nloop % v.ifreq_imasses == 0) sig |= 32u;
            if (sig & (8u << 8)) nsrate = 0;
            nsrate = nsrate + 1;
        }
        nloop = nloop + 1;
        sigs.push_back(sig);
    }
    nl.assign(1, nloop);
    ns.assign(1, nsrate);
    return sigs;
}

// The members as they are now: their calls between two batch calls may have
// changed their parameters (gf_set_params) or their marker counts (gf_remesh,
// gf_marker2elem, gf_set_clock).
int read_views(gf_batch *b) {
    for (size_t m = 0; m < b->members.size(); ++m) {
        int rc = gf_ctx_view(b->members[m], &b->views[m]);
        if (rc) return rc;
    }
    return GF_OK;
}
// Whether the members allow the joint launches; surface processes (diff_topo /
// resurface) are not part of the ensemble step
int members_merge(const gf_batch *b, int *merge) {
    *merge = 1;
    for (const GfMemberView &v : b->views) {
        const gf_params &p = *v.hp;
        if (p.istress_therm != 0 || p.nyhydro != 0 || p.itemp_bc == 2) *merge = 0;
        if (p.topo_kappa > 0.0) return GF_ERR_UNSUPPORTED;
    }
    return GF_OK;
}
// Order between the batch's stream and the members'.  A call first waits for
// what the members' own calls enqueued (calls with gf_set_sync(0), gf_set_clock);
// behind a call that returns before its kernels end, the members' next changes of
// their state wait for these.
int settle(const gf_batch *b) {
    for (gf_ctx *c : b->members) {
        const int rc = gf_ctx_settle(c, b->s, b->done.get());
        if (rc) return rc;
    }
    return GF_OK;
}
int release(gf_batch *b) {
    GB_CK(cudaEventRecord(b->done->e, b->s));
    for (gf_ctx *c : b->members) {
        const int rc = gf_ctx_read_until(c, b->done);
        if (rc) return rc;
    }
    return GF_OK;
}
// Device records, tile tables and captured steps follow the members: a member
// whose markers were added to or whose parameters changed has the records and
// the marker tiles rebuilt, and a change of the schedule drops what was captured.
int follow_members(gf_batch *b) {
    int rc = settle(b);
    if (!rc) rc = read_views(b);
    if (rc) return rc;
    const std::vector<BatchMember> now = member_records(b);
    if (std::memcmp(now.data(), b->records.data(), now.size() * sizeof(BatchMember)) == 0) return GF_OK;
    bool markers = false;
    for (size_t m = 0; m < now.size(); ++m) markers = markers || now[m].nmarkers != b->records[m].nmarkers;
    GB_CK(cudaStreamSynchronize(b->s)); // the old records' last readers
    rc = upload_members(b);
    return rc || !markers ? rc : build_tables(b);
}

int check_status(gf_batch *b) {
    const int n = (int)b->members.size();
    k_batch_status<<<(n + 127) / 128, 128, 0, b->s>>>(b->d_members, n, b->status);
    GB_CK(cudaMemcpyAsync(b->h_status, b->status, sizeof(int) * n, cudaMemcpyDeviceToHost, b->s));
    GB_CK(cudaStreamSynchronize(b->s));
    int first = GF_OK;
    for (int k = 0; k < n; ++k) {
        if (!b->h_status[k]) continue;
        const int st = gf_ctx_take_status(b->members[k]); // and clears it
        if (st && !first) first = st;
    }
    return first;
}

} // namespace

extern "C" {

int gf_batch_create(gf_batch **out, gf_ctx **members, int n) {
    if (!out || !members || n <= 0) return GF_ERR_ARG;
    *out = nullptr;
    gf_batch *b = new (std::nothrow) gf_batch;
    if (!b) return GF_ERR_NOMEM;
    b->members.assign(members, members + n);
    b->views.resize(n);
    int rc = read_views(b);
    if (!rc) rc = members_merge(b, &b->merge);
    for (int m = 0; m < n && !rc; ++m) {
        const GfMemberView &v = b->views[m], &v0 = b->views[0];
        if (v.mode != GF_MODE_MIXED) rc = GF_ERR_UNSUPPORTED;
        else if (v.nloop != v0.nloop || v.nsrate != v0.nsrate || v.itherm != v0.itherm ||
                 v.ifreq_rmasses != v0.ifreq_rmasses || v.ifreq_visc != v0.ifreq_visc ||
                 v.ifreq_imasses != v0.ifreq_imasses || v.ifreq_avgsr != v0.ifreq_avgsr)
            rc = GF_ERR_ARG; // the members must share the step schedule
        b->elements += v.d.E;
        if (v.g != b->views[0].g) rc = GF_ERR_ARG;
    }
    if (!rc) rc = batch_cuda(cudaStreamCreateWithFlags(&b->s, cudaStreamNonBlocking), "stream");
    if (!rc) rc = batch_cuda(cudaEventCreateWithFlags(&b->done->e, cudaEventDisableTiming), "event");
    if (!rc) rc = batch_cuda(cudaMalloc(&b->d_members, sizeof(BatchMember) * n), "members");
    if (!rc) rc = batch_cuda(cudaMalloc(&b->means, sizeof(float4) * 2 * (size_t)b->elements), "sampling scratch");
    if (!rc) rc = batch_cuda(cudaMalloc(&b->status, sizeof(int) * n), "status");
    if (!rc) rc = batch_cuda(cudaMallocHost(&b->h_status, sizeof(int) * n), "status");
    if (!rc) rc = upload_members(b);
    if (!rc) rc = build_tables(b);
    if (rc) {
        gf_batch_destroy(b);
        return rc;
    }
    *out = b;
    return GF_OK;
}

void gf_batch_destroy(gf_batch *b) {
    if (!b) return;
    if (b->s) cudaStreamSynchronize(b->s);
    drop_graphs(b);
    for (int k = 0; k < K_KINDS; ++k)
        if (b->d_tiles[k]) cudaFree(b->d_tiles[k]);
    if (b->d_members) cudaFree(b->d_members);
    if (b->backup) cudaFree(b->backup);
    if (b->means) cudaFree(b->means);
    if (b->status) cudaFree(b->status);
    if (b->h_status) cudaFreeHost(b->h_status);
    if (b->s) cudaStreamDestroy(b->s);
    delete b;
}

int gf_batch_set_config(gf_batch *b, const gf_batch_config *cfg) {
    if (!b || !cfg) return GF_ERR_ARG;
    gf_batch_config old = b->cfg;
    b->cfg = *cfg;
    int rc = build_tables(b);
    if (rc) {
        b->cfg = old;
        build_tables(b);
    }
    return rc;
}

int gf_batch_get_config(gf_batch *b, gf_batch_config *cfg) {
    if (!b || !cfg) return GF_ERR_ARG;
    *cfg = b->cfg;
    return GF_OK;
}

long long gf_batch_elements(gf_batch *b) { return b ? b->elements : 0; }

int gf_batch_grid(gf_batch *b) { return b ? b->grid : 0; }

void *gf_batch_stream(gf_batch *b) { return b ? (void *)b->s : nullptr; }

int gf_batch_step(gf_batch *b, int nsteps) {
    if (!b || nsteps < 0) return GF_ERR_ARG;
    // members must be idle: their own streams may still hold work
    for (const GfMemberView &v : b->views) GB_CK(cudaStreamSynchronize(v.s));
    int rc = follow_members(b), merge = 0;
    if (!rc) rc = members_merge(b, &merge);
    if (rc) return rc;
    if (merge != b->merge) drop_graphs(b); // (captured with the other launches)
    b->merge = merge;
    int done = 0;
    const int G = b->cfg.graph_steps;
    while (done < nsteps) {
        int chunk = G > 0 ? std::min(G, nsteps - done) : 1;
        std::vector<int> nl, ns;
        std::vector<unsigned> sigs = next_sigs(b, chunk, nl, ns);
        // (a chunk that has not come up GF_BATCH_CAPTURE times yet is launched
        // directly: capturing ten steps costs some 0.3 ms)
        gf_batch::Graph *g = nullptr;
        if (G > 0) {
            for (auto &x : b->graphs)
                if (x.sigs == sigs) g = &x;
            if (!g) {
                b->graphs.push_back(gf_batch::Graph{sigs, nullptr, 0});
                g = &b->graphs.back();
            }
            if (!g->exec && ++g->uses < GF_BATCH_CAPTURE) g = nullptr;
        }
        if (g) {
            if (!g->exec) {
                cudaGraph_t graph;
                GB_CK(cudaStreamBeginCapture(b->s, cudaStreamCaptureModeThreadLocal));
                int lrc = GF_OK;
                for (unsigned sig : sigs)
                    if (!lrc) lrc = launch_step(b, sig);
                cudaError_t e = cudaStreamEndCapture(b->s, &graph);
                if (lrc) return lrc;
                GB_CK(e);
                e = cudaGraphInstantiate(&g->exec, graph, 0);
                cudaGraphDestroy(graph);
                if (e != cudaSuccess) g->exec = nullptr;
                GB_CK(e);
            }
            GB_CK(cudaGraphLaunch(g->exec, b->s));
        } else {
            for (unsigned sig : sigs)
                if ((rc = launch_step(b, sig))) return rc;
        }
        for (unsigned sig : sigs)
            for (gf_ctx *c : b->members) gf_ctx_advance(c, sig);
        rc = read_views(b); // (the steps' counters)
        if (rc) return rc;
        done += chunk;
    }
    return check_status(b);
}

// Autotuner: every CTA shape (threads) and tile depth (items per thread), each
// timed over `trial_steps` steps
// with CUDA events after one untimed step; the fastest is kept.  The trial
// steps advance the members like any other steps.
int gf_batch_tune(gf_batch *b, int trial_steps, gf_batch_config *best, double *best_ms) {
    if (!b || trial_steps < 1) return GF_ERR_ARG;
    gf_batch_config keep = b->cfg, win = b->cfg;
    double win_ms = 1e300;
    cudaEvent_t e0, e1;
    GB_CK(cudaEventCreate(&e0));
    GB_CK(cudaEventCreate(&e1));
    const int threads[3] = {128, 256, 512};
    const int ipts[4] = {1, 2, 4, 8};
    int rc = GF_OK;
    for (int t : threads) {
        for (int ipt : ipts) {
            gf_batch_config c{t, ipt, 1, 0}; // direct launches: no capture inside the timing
            b->cfg = c;
            if (build_tables(b)) continue;
            rc = gf_batch_step(b, 1);
            if (rc) break;
            cudaEventRecord(e0, b->s);
            rc = gf_batch_step(b, trial_steps);
            if (rc) break;
            cudaEventRecord(e1, b->s);
            cudaEventSynchronize(e1);
            float ms = 0.f;
            cudaEventElapsedTime(&ms, e0, e1);
            double per = ms / trial_steps;
            if (per < win_ms) {
                win_ms = per;
                win = c;
            }
        }
        if (rc) break;
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    win.graph_steps = keep.graph_steps;
    b->cfg = rc ? keep : win;
    int rc2 = build_tables(b);
    if (rc) return rc;
    if (best) *best = win;
    if (best_ms) *best_ms = win_ms;
    return rc2;
}

int gf_batch_sample(gf_batch *b, float *grid, int H, int W, int phase_id) {
    if (!b || !grid || H < 1 || W < 1 || phase_id < 1) return GF_ERR_ARG;
    const int rc = follow_members(b);
    if (rc) return rc;
    GridArgs g{b->d_members, (int)b->members.size(), H, W, phase_id, grid, nullptr};
    if (b->ntile[K_E])
        k_sample_elems<<<b->ntile[K_E], b->cfg.threads, 0, b->s>>>(g, b->d_tiles[K_E], b->ntile[K_E],
                                                                   b->ipt, b->means);
    const int ty = (H + 31) / 32, tx = (W + 31) / 32;
    k_sample<<<(unsigned)((long long)g.n * ty * tx), 256, 0, b->s>>>(g, b->means, ty, tx);
    GB_CK(cudaGetLastError());
    return release(b);
}

int gf_batch_inject(gf_batch *b, const float *grid, int H, int W) {
    if (!b || !grid || H < 2 || W < 2) return GF_ERR_ARG;
    const int rc = follow_members(b);
    if (rc) return rc;
    for (gf_ctx *c : b->members) gf_ctx_invalidate_forces(c);
    GridArgs g{b->d_members, (int)b->members.size(), H, W, 1, nullptr, grid};
    const int T = b->cfg.threads, ipt = b->ipt;
    if (b->ntile[K_N]) k_inject_nodes<<<b->ntile[K_N], T, 0, b->s>>>(g, b->d_tiles[K_N], b->ntile[K_N], ipt);
    if (b->ntile[K_E])
        k_inject_elems<<<b->ntile[K_E], T, 0, b->s>>>(g, b->d_tiles[K_E], b->ntile[K_E], ipt, nullptr);
    GB_CK(cudaGetLastError());
    return check_status(b);
}

int gf_batch_backup(gf_batch *b) {
    if (!b) return GF_ERR_ARG;
    for (const GfMemberView &v : b->views) GB_CK(cudaStreamSynchronize(v.s));
    const int rc = settle(b);
    if (rc) return rc;
    if (!b->backup) {
        size_t total = 0;
        b->backup_off.clear();
        for (const GfMemberView &v : b->views) {
            b->backup_off.push_back(total);
            for (auto &f : injected_fields(v)) total += (f.second + 255) & ~(size_t)255;
        }
        GB_CK(cudaMalloc(&b->backup, total));
    }
    for (size_t m = 0; m < b->views.size(); ++m) {
        size_t off = b->backup_off[m];
        for (auto &f : injected_fields(b->views[m])) {
            GB_CK(cudaMemcpyAsync((char *)b->backup + off, f.first, f.second, cudaMemcpyDeviceToDevice, b->s));
            off += (f.second + 255) & ~(size_t)255;
        }
    }
    return release(b);
}

int gf_batch_restore(gf_batch *b, const int *members, int count) {
    if (!b || (count > 0 && !members)) return GF_ERR_ARG;
    if (!b->backup) return GF_ERR_ARG;
    const int rc = settle(b);
    if (rc) return rc;
    for (int k = 0; k < count; ++k) {
        int m = members[k];
        if (m < 0 || m >= (int)b->views.size()) return GF_ERR_ARG;
        gf_ctx_invalidate_forces(b->members[m]);
        size_t off = b->backup_off[m];
        for (auto &f : injected_fields(b->views[m])) {
            GB_CK(cudaMemcpyAsync(f.first, (char *)b->backup + off, f.second, cudaMemcpyDeviceToDevice, b->s));
            off += (f.second + 255) & ~(size_t)255;
        }
    }
    GB_CK(cudaStreamSynchronize(b->s));
    return GF_OK;
}

int gf_batch_force_residual(gf_batch *b, double *residual) {
    if (!b || !residual) return GF_ERR_ARG;
    const int rc = follow_members(b);
    if (rc) return rc;
    const int n = (int)b->members.size();
    double *acc = nullptr;
    GB_CK(cudaMalloc(&acc, sizeof(double) * 2 * n));
    cudaMemsetAsync(acc, 0, sizeof(double) * 2 * n, b->s);
    if (b->ntile[K_N])
        k_force_residual<<<b->ntile[K_N], b->cfg.threads, 0, b->s>>>(b->d_members, b->d_tiles[K_N], b->ntile[K_N],
                                                                     b->ipt, acc);
    std::vector<double> h(2 * n);
    cudaError_t e = cudaMemcpyAsync(h.data(), acc, sizeof(double) * 2 * n, cudaMemcpyDeviceToHost, b->s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(b->s);
    cudaFree(acc);
    GB_CK(e);
    for (int m = 0; m < n; ++m) residual[m] = h[2 * m] / (h[2 * m + 1] > 0 ? h[2 * m + 1] : 1.0);
    return GF_OK;
}

} // extern "C"
