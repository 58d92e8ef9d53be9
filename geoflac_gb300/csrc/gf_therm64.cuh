// fl_therm (fl_therm.f90:393-598) in FP64.
//
// The reference updates temp in place, i outer and j inner: node (j,i) reads
// new values at its upstream neighbours (j-1,i), (j,i-1), (j+1,i-1) and old
// values at itself and downstream.  Its result is the unique fixed point of
//   Tnew(n) = f_n(Tnew(upstream), Told(rest))
// with f_n the reference's floating-point expression.  The system is lower
// triangular, so iterating Jacobi-style sweeps of f_n reaches that fixed
// point exactly (bit for bit) after finitely many sweeps; each sweep
// contracts the distance by ~kappa*dt/h^2, so a handful of sweeps suffice.
// A sweep that changes no value proves convergence.
//
// k_therm_prep computes, per triangle A and B of every element, everything
// that does not depend on temperature (fl_therm.f90:424-567); one co-resident
// launch then runs the sweeps and the boundary conditions.
#pragma once

namespace {
namespace gfk {

// One thread per triangle (A, B) of an element: the shape-derivative products
// K_ab, real_area13 = (1/area)/6, 0.5*diff/area and src*real_area13, each with
// the reference's operations; products and quotients on the integer pipes.
__global__ void __launch_bounds__(GF_THREADS) k_therm_prep(const DevParams *__restrict__ Pp, DevClock *__restrict__ C,
                                                          DevArrays A, GfDims d, double *__restrict__ tc) {
    gf_pdl_entry();
    const GF_IDX th = (GF_IDX)blockIdx.x * blockDim.x + threadIdx.x;
    if (th < GF_THERM_KMAX) C->therm_flags[th] = 0; // before any sweep runs
    const GF_IDX e = th >> 1;
    if (e >= d.E) return;
    const int t = (int)(th & 1);
    const DevParams &P = *Pp;
    int j, i;
    tri_ji(d, e, j, i);
    const int iph = A.iphase[e] - 1;
    const double dissip = (P.ishearh == 1 && P.itherm != 2) ? ((const double *)A.shrheat)[e] : 0.0;
    // conduct / den / cp of the phase: the same two IEEE divisions as the
    // reference's cond_eff / dens / cp_eff, taken once per phase at set-up
    const double diff = P.diffu[iph];
    const double src = gf_ddiv(A.source[e] + gf_ddiv(dissip, P.den[iph]), P.cp[iph]);
    GF_IDX n[3];
    tri_nodes(d, j, i, t, n); // (q1,q2,q3) or (q3,q2,q4)
    double x[3], y[3];
#pragma unroll
    for (int m = 0; m < 3; ++m) {
        x[m] = A.cord[n[m]];
        y[m] = A.cord[d.N + n[m]];
    }
    const double a = ((const double *)A.area)[gf_ek(d, e, t)];
    const double dd[3] = {gf_mul(y[1] - y[2], a), gf_mul(y[2] - y[0], a), gf_mul(y[0] - y[1], a)};
    const double zz[3] = {gf_mul(x[2] - x[1], a), gf_mul(x[0] - x[2], a), gf_mul(x[1] - x[0], a)};
    const GF_IDX E = d.E;
#pragma unroll
    for (int m = 0; m < 3; ++m)
#pragma unroll
        for (int q = m; q < 3; ++q) tc[(t * 6 + kidx(m, q)) * E + e] = gf_mul(dd[m], dd[q]) + gf_mul(zz[m], zz[q]);
    const double inv_area = gf_rcp(a); // RN(1/a) off the FP64 pipe
    const double ra = gf_ddiv(inv_area, 6.0);
    tc[(12 + t) * E + e] = ra;
    tc[(14 + t) * E + e] = gf_mul(gf_scale<-1>(diff), inv_area);
    tc[(16 + t) * E + e] = gf_mul(src, ra);
}

// End of a sweep, bounded: every CTA adds its arrival (low half) and whether
// one of its values changed (high half) to the sweep's own counter and waits
// until all have arrived, so that the barrier's word carries the convergence
// test too.  1 / 0: some value changed / none did; -1: gave up.
#define GF_TH_POLLS (1 << 22)
__device__ __forceinline__ int therm_sync(unsigned *slot, bool changed, int polls = GF_TH_POLLS) {
    __shared__ int res;
    const int any = __syncthreads_or(changed);
    if (threadIdx.x == 0) {
        unsigned v;
        const unsigned add = any ? 0x10001u : 1u;
        asm volatile("atom.add.acq_rel.gpu.u32 %0, [%1], %2;" : "=r"(v) : "l"(slot), "r"(add) : "memory");
        v += add;
        int it = 0;
        while ((v & 0xffffu) != gridDim.x && ++it < polls)
            asm volatile("ld.acquire.gpu.u32 %0, [%1];" : "=r"(v) : "l"(slot) : "memory");
        res = (v & 0xffffu) != gridDim.x ? -1 : (v >> 16) != 0u;
    }
    __syncthreads();
    return res;
}

// The boundary conditions (fl_therm.f90:577-598) and temp0 = temp from the
// last sweep's values, and the increment that the next step's start uses
template <class Src>
__device__ __forceinline__ void therm_finish(const DevParams *Pp, const DevArrays &A, const GfDims &d, Src src,
                                             int keep_temp0, GF_IDX n) {
    int j, i;
    i = (int)((unsigned)n / (unsigned)d.nz);
    j = (int)n - i * d.nz;
    const double t = therm_bc_value(*Pp, A, d, src, j, i);
    const double told = A.temp[n];
    if (!keep_temp0) A.temp0[n] = told;
    A.temp[n] = t;
    A.t_pred[n] = t - told; // the next step's start: its Told + this increment
}
__device__ __forceinline__ void therm_count(DevClock *C, int kc, int kmax) {
    C->therm_sweeps_used = kc + 1;
    if (kc == kmax) C->therm_unconverged += 1;
}

// The sweeps with one node per thread, for meshes that the chip holds that way.
// A node's coefficients, the products with Told and the reciprocal of its
// area sum stay in registers over the sweeps, so that a sweep loads three
// upstream values and, where one of them changed, takes eleven integer-pipe
// products and twenty FP64 additions (of 26 and 31); CTAs of four warps
// spread a small mesh over all SMs.  A sweep then costs about 3 us, half of
// it the barrier: fl_therm 76 -> 39 us on 60x20 and 241x61 elements, 91 -> 53
// on 400x120, 112 -> 62 on 600x150 (events) against the general kernel's
// predecessor, where a sweep took 9 to 15 us.
//
// CL: a mesh of up to GF_TH_CL x 256 nodes runs as one cluster.  The iterates
// and the sweep's changed flags then live in the CTAs' shared memory, read
// across the cluster, and the hardware's cluster barrier ends a sweep: no trip
// to L2 and back for the values nor for the barrier (fl_therm of 60x20
// elements 40 -> 32 us).  Every CTA has as many nodes as it has threads, four
// warps (one on each FP64 pipe) up to 2048 nodes.
#define GF_TH_T 128
#define GF_TH_CTAS 5 // per SM: 102 registers
#define GF_TH_CL 16
#define GF_TH_CLT 256
__device__ __forceinline__ unsigned cl_map(const void *p, unsigned rank) { // p in CTA rank's shared memory
    unsigned a;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((unsigned)__cvta_generic_to_shared(p)), "r"(rank));
    return a;
}
__device__ __forceinline__ double cl_load(unsigned a) {
    double v;
    asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ void cl_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
template <bool CL>
__global__ void __launch_bounds__(CL ? GF_TH_CLT : GF_TH_T, CL ? 1 : GF_TH_CTAS)
    k_therm_sweeps_reg(const DevParams *__restrict__ Pp, DevClock *__restrict__ C, DevArrays A, GfDims d,
                       const double *__restrict__ tc, double *b0, double *b1, int kmax, int keep_temp0) {
    __shared__ double iter[2][CL ? GF_TH_CLT : 1];
    __shared__ unsigned moved[2][CL ? GF_TH_CL : 1]; // by the sweep's parity and the CTA that reports
    if (CL) gf_pdl_entry();
    const unsigned T_ = blockDim.x;
    const GF_IDX nn = (GF_IDX)blockIdx.x * T_ + threadIdx.x;
    const bool act = nn < d.N;
    const GF_IDX n = act ? nn : d.N - 1; // idle threads follow along and store nothing
    const int nz = d.nz, i = (int)((unsigned)n / (unsigned)nz), j = (int)n - i * nz;
    const bool up = j != 0, dn = j != nz - 1, lf = i != 0, rt = i != d.nx - 1;
    const GF_IDX E = d.E, e22 = gf_elem(d, j, i);
    const GF_IDX na = up ? n - 1 : n, nb = lf ? n - nz : n, nc = lf && dn ? n - nz + 1 : n; // upstream
    const double dt = C->dt, *T = A.temp;
    const double Ts = T[n];
    double area = 0.0;
    auto K = [&](GF_IDX e, int t, int k) { return tc[(t * 6 + k) * E + e]; };
    auto pre = [&](GF_IDX e, int t) { // and the area sum, in the reference's order of triangles
        area = area + tc[(12 + t) * E + e];
        return tc[(14 + t) * E + e];
    };
    auto heat = [&](GF_IDX e, int t) { return tc[(16 + t) * E + e]; };
    // triangles in the reference's order: 1 = B of (j-1,i-1), 2 and 3 = A and
    // B of (j-1,i), 4 and 5 = A and B of (j,i-1), 6 = A of (j,i)
    double k1a = 0, k1b = 0, c1 = 0, p1 = 0, s1 = 0, k2a = 0, c21 = 0, c22 = 0, p2 = 0, s2 = 0, q3 = 0, s3 = 0;
    double k4b = 0, k4c = 0, c4 = 0, p4 = 0, s4 = 0, k5c = 0, c50 = 0, c52 = 0, p5 = 0, s5 = 0, q6 = 0, s6 = 0;
    if (up && lf) {
        const GF_IDX e = e22 - (nz - 1) - 1;
        p1 = pre(e, 1); s1 = heat(e, 1);
        k1a = K(e, 1, 2); k1b = K(e, 1, 4);
        c1 = gf_mul(Ts, K(e, 1, 5));
    }
    if (up && rt) {
        const GF_IDX e = e22 - 1;
        const double Tr = T[n + nz - 1], Td = T[n + nz];
        p2 = pre(e, 0); s2 = heat(e, 0);
        k2a = K(e, 0, 1);
        c21 = gf_mul(Ts, K(e, 0, 3));
        c22 = gf_mul(Tr, K(e, 0, 4));
        const double p3 = pre(e, 1);
        s3 = heat(e, 1);
        q3 = gf_mul(p3, gf_mul(Tr, K(e, 1, 1)) + gf_mul(Ts, K(e, 1, 3)) + gf_mul(Td, K(e, 1, 4)));
    }
    if (dn && lf) {
        const GF_IDX e = e22 - (nz - 1);
        p4 = pre(e, 0); s4 = heat(e, 0);
        k4b = K(e, 0, 2); k4c = K(e, 0, 4);
        c4 = gf_mul(Ts, K(e, 0, 5));
        p5 = pre(e, 1); s5 = heat(e, 1);
        c50 = gf_mul(Ts, K(e, 1, 0));
        k5c = K(e, 1, 1);
        c52 = gf_mul(T[n + 1], K(e, 1, 2));
    }
    if (dn && rt) {
        const double p6 = pre(e22, 0);
        s6 = heat(e22, 0);
        q6 = gf_mul(p6, gf_mul(Ts, K(e22, 0, 0)) + gf_mul(T[n + 1], K(e22, 0, 1)) + gf_mul(T[n + nz], K(e22, 0, 2)));
    }
    const GfIntRecip ra = gf_int_recip(area);
    auto eval = [&](double a, double b, double c) {
        double r = 0.0;
        if (up && lf) r = r + s1 - gf_mul(p1, gf_mul(a, k1a) + gf_mul(b, k1b) + c1);
        if (up && rt) {
            r = r + s2 - gf_mul(p2, gf_mul(a, k2a) + c21 + c22);
            r = r + s3 - q3;
        }
        if (dn && lf) {
            r = r + s4 - gf_mul(p4, gf_mul(b, k4b) + gf_mul(c, k4c) + c4);
            r = r + s5 - gf_mul(p5, c50 + gf_mul(c, k5c) + c52);
        }
        if (dn && rt) r = r + s6 - q6;
        return Ts + gf_ddiv_by(gf_mul(r, dt), ra);
    };
    // the start (the iterate before sweep 0) is Told + the previous step's
    // increment, a guess: the fixed point does not depend on it, only how
    // many nodes the sweeps recompute before they reach it
    double a = T[na] + A.t_pred[na], b = T[nb] + A.t_pred[nb], c = T[nc] + A.t_pred[nc];
    double v = Ts + A.t_pred[n];
    auto where = [&](GF_IDX m) { return cl_map(&iter[0][(unsigned)m % T_], (unsigned)m / T_); };
    const unsigned wa = CL ? where(na) : 0u, wb = CL ? where(nb) : 0u, wc = CL ? where(nc) : 0u;
    const unsigned report = CL ? cl_map(&moved[0][blockIdx.x], threadIdx.x % gridDim.x) : 0u;
    if (CL) cl_sync(); // every CTA of the cluster runs
    int kc = kmax; // the first sweep that changed nothing
    for (int k = 0; k < kmax; ++k) {
        bool changed = false;
        bool redo = true;
        if (k > 0) {
            const double *src = (k - 1) & 1 ? b1 : b0;
            const unsigned off = ((k - 1) & 1) * (GF_TH_CLT * 8u);
            const double a1 = CL ? cl_load(wa + off) : __ldcg(src + na), c1n = CL ? cl_load(wc + off) : __ldcg(src + nc),
                         b1n = CL ? cl_load(wb + off) : __ldcg(src + nb);
            redo = (up && !gf_deq(a1, a)) || (lf && !gf_deq(b1n, b)) || (lf && dn && !gf_deq(c1n, c));
            a = a1;
            b = b1n;
            c = c1n;
        }
        if (__any_sync(0xffffffffu, redo)) { // the same inputs give the same value
            const double t = eval(a, b, c);
            changed = act && redo && !gf_deq(t, v);
            if (redo) v = t;
        }
        int s;
        if constexpr (CL) {
            iter[k & 1][threadIdx.x] = v;
            const unsigned any = __syncthreads_or(changed);
            if (threadIdx.x < gridDim.x)
                asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(report + (k & 1) * (GF_TH_CL * 4u)), "r"(any) : "memory");
            cl_sync();
            const unsigned lane = threadIdx.x & 31u;
            s = __any_sync(0xffffffffu, lane < gridDim.x && moved[k & 1][lane % GF_TH_CL] != 0u);
        } else {
            if (act) ((k & 1) ? b1 : b0)[n] = v;
            s = therm_sync(reinterpret_cast<unsigned *>(C->therm_flags + k), changed);
            if (s < 0) {
                if (nn == 0) set_status(C, GF_ERR_TIMEOUT, k);
                return;
            }
        }
        if (s == 0) {
            kc = k;
            break;
        }
    }
    if (nn == 0) therm_count(C, kc, kmax);
    const int last = (kc < kmax ? kc : kmax - 1) & 1;
    if constexpr (CL) {
        if (act)
            therm_finish(Pp, A, d, [&](GF_IDX m) { return cl_load(where(m) + last * (GF_TH_CLT * 8u)); }, keep_temp0, n);
        cl_sync(); // no CTA leaves while another reads its values
    } else {
        const double *src = last ? b1 : b0;
        if (act) therm_finish(Pp, A, d, [src](GF_IDX m) { return __ldcg(src + m); }, keep_temp0, n);
    }
}

// One node of a sweep from its coefficients in memory.  Tup holds the current
// upstream iterate; self and downstream values always come from Told.
template <class Up>
__device__ __forceinline__ double therm_node(const DevArrays &A, const GfDims &d, double dt,
                                             const double *__restrict__ tc, Up U, int j, int i, GF_IDX n) {
    const int nx = d.nx, nz = d.nz;
    const GF_IDX E = d.E, e22 = gf_elem(d, j, i);
    const double *T = A.temp;
    double rhs = 0.0, area_n = 0.0;
    // triangle t of element e; vs = local index of the updated node; the
    // three (local vertex, temperature) terms in the reference's order
    auto tri = [&](GF_IDX e, int t, int vs, int v0, double T0, int v1, double T1, int v2, double T2) {
        double ra = tc[(12 + t) * E + e];
        area_n = area_n + ra;
        const double *K = tc + (GF_IDX)t * 6 * E + e;
        rhs = rhs + tc[(16 + t) * E + e] -
              gf_mul(tc[(14 + t) * E + e], gf_mul(T0, K[kidx(v0, vs) * E]) + gf_mul(T1, K[kidx(v1, vs) * E]) +
                                               gf_mul(T2, K[kidx(v2, vs) * E]));
    };
    const double Ts = T[n];
    if (j != 0 && i != 0) tri(e22 - nz, 1, 2, 0, U(n - 1), 1, U(n - nz), 2, Ts);
    if (j != 0 && i != nx - 1) {
        tri(e22 - 1, 0, 1, 0, U(n - 1), 1, Ts, 2, T[n + nz - 1]);
        tri(e22 - 1, 1, 1, 0, T[n + nz - 1], 1, Ts, 2, T[n + nz]);
    }
    if (j != nz - 1 && i != 0) {
        const GF_IDX e = e22 - (nz - 1);
        tri(e, 0, 2, 0, U(n - nz), 1, U(n - nz + 1), 2, Ts);
        tri(e, 1, 0, 0, Ts, 1, U(n - nz + 1), 2, T[n + 1]);
    }
    if (j != nz - 1 && i != nx - 1) tri(e22, 0, 0, 0, Ts, 1, T[n + 1], 2, T[n + nz]);
    return Ts + gf_ddiv(gf_mul(rhs, dt), area_n);
}

// The sweeps of larger meshes.  A node's value depends on the sweep before
// only through its upstream neighbours, so it is evaluated again only if one
// of them changed; the changes of a sweep are kept as one bit per node.  A CTA
// goes over its nodes 256 at a time, 32 consecutive ones per warp, lists those
// to evaluate in shared memory and then evaluates the list, so that a sweep's
// cost follows the number of such nodes (from sweep 2 on some 16 % of them,
// scattered over all warps).  An unchanged value is copied into the sweep's
// buffer only if the sweep before changed it: otherwise it is there since two
// sweeps ago.  A sweep of all 301,301 nodes of 1000x300 elements takes 27 us
// (bound by latency: 31 FP64 additions and 26 integer products a node), the
// last ones 10 (were 45 and 15): fl_therm 260 -> 199 us.
#define GF_TH_IT 8 // 256-node groups listed together
__global__ void __launch_bounds__(GF_THREADS, 4)
    k_therm_sweeps(const DevParams *__restrict__ Pp, DevClock *__restrict__ C, DevArrays A, GfDims d,
                   const double *__restrict__ tc, double *b0, double *b1, int kmax, int keep_temp0) {
    constexpr int WARPS = GF_THREADS / 32;
    __shared__ unsigned short list[GF_TH_IT * GF_THREADS];
    __shared__ unsigned bits[GF_TH_IT * WARPS];
    __shared__ int count;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nz = d.nz;
    const int words = (int)((d.N + 31) / 32);
    const int first = (int)blockIdx.x * WARPS, step = (int)gridDim.x * WARPS; // words of the CTA's groups
    unsigned *chg = reinterpret_cast<unsigned *>(A.t_chg);                    // [2][words] by the sweep's parity
    const double dt = C->dt, *T = A.temp, *pred = A.t_pred;
    int kc = kmax; // the first sweep that changed nothing
    for (int k = 0; k < kmax; ++k) {
        const double *up = (k - 1) & 1 ? b1 : b0;
        double *out = (k & 1) ? b1 : b0;
        const unsigned *prev = chg + (size_t)((k - 1) & 1) * words;
        unsigned *now = chg + (size_t)(k & 1) * words;
        bool any = false;
        for (int base = first; base < words; base += GF_TH_IT * step) {
            if (threadIdx.x == 0) count = 0;
            if (threadIdx.x < GF_TH_IT * WARPS) bits[threadIdx.x] = 0u;
            __syncthreads();
            for (int it = 0; it < GF_TH_IT; ++it) {
                const int w = base + it * step + warp;
                if (w >= words) break;
                const GF_IDX n = (GF_IDX)w * 32 + lane;
                const bool act = n < d.N;
                bool redo = act;
                if (k > 0) {
                    // change bits of n-1, n and, a column back, n-nz and n-nz+1
                    const int f = w * 32 - nz; // the first of the column before (may be negative)
                    const int q = f >> 5, sh = f & 31;
                    const int at = lane == 0 ? w - 1 : lane == 1 ? w : q + lane - 2;
                    const unsigned x = lane < 4 && at >= 0 && at < words ? __ldcg(prev + at) : 0u;
                    const unsigned wm = __shfl_sync(0xffffffffu, x, 0), w0 = __shfl_sync(0xffffffffu, x, 1);
                    const unsigned y0 = __shfl_sync(0xffffffffu, x, 2), y1 = __shfl_sync(0xffffffffu, x, 3);
                    const unsigned m1 = __funnelshift_r(wm, w0, 31);                     // n - 1
                    const unsigned m2 = __funnelshift_r(y0, y1, sh);                     // n - nz
                    const unsigned m3 = sh == 31 ? y1 : __funnelshift_r(y0, y1, sh + 1); // n - nz + 1
                    if (k > 1 && (m1 | m2 | m3 | w0) == 0u) continue;
                    const int i = (int)((unsigned)n / (unsigned)nz), j = (int)n - i * nz;
                    const unsigned bit = 1u << lane;
                    redo = act && ((j != 0 && (m1 & bit)) || (i != 0 && (m2 & bit)) ||
                                   (i != 0 && j != nz - 1 && (m3 & bit)));
                    if (act && !redo && (k == 1 || (w0 & bit))) out[n] = __ldcg(up + n); // (sweep 1: nothing there yet)
                }
                const unsigned m = __ballot_sync(0xffffffffu, redo);
                int at = 0;
                if (lane == 0 && m) at = atomicAdd(&count, __popc(m));
                at = __shfl_sync(0xffffffffu, at, 0);
                if (redo) list[at + __popc(m & ((1u << lane) - 1u))] = (unsigned short)(it * GF_THREADS + threadIdx.x);
            }
            __syncthreads();
            const int total = count;
            for (int q = threadIdx.x; q < total; q += GF_THREADS) {
                const int l = list[q], it = l / GF_THREADS, th = l % GF_THREADS;
                const GF_IDX n = (GF_IDX)(base + it * step + (th >> 5)) * 32 + (th & 31);
                const int i = (int)((unsigned)n / (unsigned)nz), j = (int)n - i * nz;
                double t, old;
                if (k == 0) {
                    t = therm_node(A, d, dt, tc, [&](GF_IDX m) { return T[m] + pred[m]; }, j, i, n);
                    old = T[n] + pred[n];
                } else {
                    t = therm_node(A, d, dt, tc, [&](GF_IDX m) { return __ldcg(up + m); }, j, i, n);
                    old = __ldcg(up + n);
                }
                out[n] = t;
                if (!gf_deq(t, old)) {
                    atomicOr(&bits[it * WARPS + (th >> 5)], 1u << (th & 31));
                    any = true;
                }
            }
            __syncthreads();
            if (threadIdx.x < GF_TH_IT * WARPS) {
                const int w = base + (threadIdx.x / WARPS) * step + threadIdx.x % WARPS;
                if (w < words) now[w] = bits[threadIdx.x];
            }
        }
        const int s = therm_sync(reinterpret_cast<unsigned *>(C->therm_flags + k), any);
        if (s < 0) {
            if (blockIdx.x == 0 && threadIdx.x == 0) set_status(C, GF_ERR_TIMEOUT, k);
            return;
        }
        if (s == 0) {
            kc = k;
            break;
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) therm_count(C, kc, kmax);
    const double *src = ((kc < kmax ? kc : kmax - 1) & 1) ? b1 : b0;
    for (GF_IDX n = (GF_IDX)blockIdx.x * GF_THREADS + threadIdx.x; n < d.N; n += (GF_IDX)gridDim.x * GF_THREADS)
        therm_finish(Pp, A, d, [src](GF_IDX m) { return __ldcg(src + m); }, keep_temp0, n);
}

} // namespace gfk
} // namespace

// CTAs of the widest cluster of k_therm_sweeps_reg<true> that the device
// takes (16 needs an opt-in), 0: none
inline int cluster_ctas() {
    using namespace gfk;
    if (cudaFuncSetAttribute(k_therm_sweeps_reg<true>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess)
        (void)cudaGetLastError();
    for (int c = GF_TH_CL; c >= 8; c /= 2) {
        cudaLaunchConfig_t lc = {};
        lc.gridDim = dim3((unsigned)c);
        lc.blockDim = dim3(GF_TH_CLT);
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = (unsigned)c;
        attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
        lc.attrs = attr;
        lc.numAttrs = 1;
        int n = 0;
        if (cudaOccupancyMaxActiveClusters(&n, k_therm_sweeps_reg<true>, &lc) == cudaSuccess && n > 0) return c;
        (void)cudaGetLastError();
    }
    return 0;
}
// fl_therm after an optional temp0 = temp of the caller (keep_temp0)
inline void therm_launch(const GfLaunch &g, int kmax, int keep_temp0) {
    using namespace gfk;
    const unsigned t = gf_threads_for(2 * g.d.E, GF_THREADS);
    gf_launch_pdl(k_therm_prep, grid_for(2 * g.d.E, t), t, g.s, g.P, g.C, g.A, g.d, g.A.t_coef);
    ++*g.launches;
    // resident CTAs of the two kernels, once per device
    static int cap_reg[64] = {0}, cap_gen[64] = {0}, cap_cl[64] = {0}; // (cap_cl: CTAs of a cluster, 0: none fits)
    int dev = 0;
    cudaGetDevice(&dev);
    dev = dev & 63;
    if (cap_gen[dev] == 0) {
        int a = 0, b = 0, sms = 0;
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&a, k_therm_sweeps_reg<false>, GF_TH_T, 0);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_therm_sweeps, GF_THREADS, 0);
        cap_cl[dev] = cluster_ctas();
        cap_reg[dev] = a * sms;
        cap_gen[dev] = (b > 0 ? b : 1) * sms;
    }
    if (g.d.N <= (GF_IDX)cap_cl[dev] * GF_TH_CLT) { // one cluster holds the mesh
        const unsigned thr = (unsigned)((g.d.N + cap_cl[dev] - 1) / cap_cl[dev] + 31) & ~31u;
        cudaLaunchConfig_t lc = {};
        lc.gridDim = dim3((unsigned)cap_cl[dev]);
        lc.blockDim = dim3(thr);
        lc.stream = g.s;
        cudaLaunchAttribute attr[2];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = (unsigned)cap_cl[dev];
        attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
        attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[1].val.programmaticStreamSerializationAllowed = 1;
        lc.attrs = attr;
        lc.numAttrs = 2;
        cudaLaunchKernelEx(&lc, k_therm_sweeps_reg<true>, g.P, g.C, g.A, g.d, (const double *)g.A.t_coef, g.A.t_delta0,
                           g.A.t_delta1, kmax, keep_temp0);
        ++*g.launches;
        return;
    }
    const bool reg = g.d.N <= (GF_IDX)cap_reg[dev] * GF_TH_T; // one node per thread fits
    const int threads = reg ? GF_TH_T : GF_THREADS;
    const GF_IDX need = (g.d.N + threads - 1) / threads, cap = cap_gen[dev];
    cudaLaunchConfig_t lc = {};
    lc.gridDim = dim3((unsigned)(reg || need < cap ? need : cap));
    lc.blockDim = dim3(threads);
    lc.stream = g.s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    lc.attrs = attr;
    lc.numAttrs = 1;
    cudaLaunchKernelEx(&lc, reg ? k_therm_sweeps_reg<false> : k_therm_sweeps, g.P, g.C, g.A, g.d, (const double *)g.A.t_coef,
                       g.A.t_delta0, g.A.t_delta1, kmax, keep_temp0);
    ++*g.launches;
}
