// FP64 element kernels with one thread per triangle: lane k of a group of
// four holds triangle k of its element (fl_rheol, the element part of
// fl_move).
//
// Why this split: the FP64 pipe takes one warp instruction per 64 cycles and
// SM sub-partition, the integer pipes one per two, so these kernels are
// fastest when most products run as integer code (gf_mul, gf_ddiv_by)
// beside the FP64 additions.  With one thread per element the four
// triangles' code unrolls to more than the instruction cache holds once
// products are integer code, and holds 128 registers with spills; with one
// thread per triangle the same code appears once, and a mesh too small to
// fill the chip gives four times the warps, each with a quarter of the
// serial chain.  Sums over the four triangles keep the reference's order:
// the values are transposed within the group (lane c gets component c of
// the four triangles) and added there, one component per lane.
// Measured against one thread per element (CUDA events): fl_rheol 546 ->
// 463 us on 1000x300 elements (152 FP64 warp instructions and 5,950 in all
// per eight elements; the FP64 pipe 66 % busy), 225 -> 184 us on 600x150,
// 106 -> 51 us on 241x61, 91 -> 43 us on 60x20; fl_move 84 -> 78, 40 -> 31,
// 25 -> 14 and 21 -> 12 us.  Every size gains, so there is no other variant.
#pragma once

namespace {
namespace gfk {

__device__ __forceinline__ double grp_get(double v, int lane) { return __shfl_sync(0xffffffffu, v, lane, 4); }
__device__ __forceinline__ double grp_xor(double v, int m) { return __shfl_xor_sync(0xffffffffu, v, m, 4); }

// lane t's (v0, v1, v2, v3) -> lane c's v_c of triangles 0..3
__device__ __forceinline__ void grp_transpose(int k, double &v0, double &v1, double &v2, double &v3) {
    const bool b = k & 1, c = k & 2;
    const double y0 = grp_xor(b ? v0 : v1, 1), y1 = grp_xor(b ? v2 : v3, 1);
    const double a0 = b ? y0 : v0, a1 = b ? v1 : y0; // component (k & 1) of the pair of triangles
    const double a2 = b ? y1 : v2, a3 = b ? v3 : y1; // component 2 + (k & 1)
    const double z0 = grp_xor(c ? a0 : a2, 2), z1 = grp_xor(c ? a1 : a3, 2);
    v0 = c ? z0 : a0;
    v1 = c ? z1 : a1;
    v2 = c ? a2 : z0;
    v3 = c ? a3 : z1;
}

// the triangle's three vertices as quad nodes 0..3 = (j,i), (j+1,i), (j,i+1), (j+1,i+1)
__device__ __forceinline__ void tri_nodes(const GfDims &d, int j, int i, int k, GF_IDX n[3]) {
    const unsigned vs = k == 0 ? 0x210u : k == 1 ? 0x312u : k == 2 ? 0x310u : 0x230u;
    const GF_IDX n0 = gf_node(d, j, i);
#pragma unroll
    for (int m = 0; m < 3; ++m) {
        const unsigned v = (vs >> (4 * m)) & 3u;
        n[m] = n0 + (v & 1u) + ((v >> 1) ? d.nz : 0);
    }
}
// element e < 2^31 (a context of more would not fit the device's memory)
__device__ __forceinline__ void tri_ji(const GfDims &d, GF_IDX e, int &j, int &i) {
    i = (int)((unsigned)e / (unsigned)(d.nz - 1));
    j = (int)e - i * (d.nz - 1);
}

// Whether the phase mixture of the element lets it read the plastic table
// (plastic_table_state), the phases shared among the group's lanes.
__device__ __forceinline__ bool tri_single_phase(const DevParams &P, const DevArrays &A, const GfDims &d, GF_IDX e,
                                                 int iph, int k) {
    int single = P.itype_melting != 1;
    for (int q = k; q < P.nphase; q += 4) {
        const double r = A.phase_ratio[gf_pr(d, e, q)];
        if (q == iph) single &= __double_as_longlong(r) == 0x3ff0000000000000ll; // exactly 1
        else single &= gf_ratio_below_cut(r);
    }
    single &= __shfl_xor_sync(0xffffffffu, single, 1, 4);
    single &= __shfl_xor_sync(0xffffffffu, single, 2, 4);
    return single != 0;
}

// Eff_visc of the elements whose viscosity fl_rheol updates, ahead of it
// (one thread per element: its transcendentals are per element, not per
// triangle; fl_rheol.f90 evaluates it from the same start-of-step state).
__global__ void __launch_bounds__(GF_THREADS) k_rheol_visc(const DevParams *__restrict__ Pp, DevArrays A, GfDims d) {
    gf_pdl_entry();
    const GF_IDX e = (GF_IDX)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= d.E) return;
    const int irh = Pp->irheol[A.iphase[e] - 1];
    if (!(irh == 3 || irh >= 11)) return;
    b_k_init_visc<double>(Pp, A, d, e);
}

// CTAs of four warps, five per SM (96 registers): small CTAs even out the
// last wave, and five measured level with eight (64 registers, spills) on
// 300,000 elements and ahead of six on smaller meshes.
#define GF_TRI_T 128
// fl_rheol (fl_rheol.f90:4-389), viscosities already updated (k_rheol_visc).
__global__ void __launch_bounds__(GF_TRI_T, 5)
    k_rheol_tri(const DevParams *__restrict__ Pp, DevClock *__restrict__ C, DevArrays A, GfDims d) {
    gf_pdl_entry();
    const GF_IDX t = (GF_IDX)blockIdx.x * blockDim.x + threadIdx.x;
    const int k = (int)(t & 3);
    const bool act = (t >> 2) < d.E;
    const GF_IDX e = act ? (t >> 2) : d.E - 1; // idle groups follow along for the shuffles and store nothing
    const DevParams &P = *Pp;
    int j, i;
    tri_ji(d, e, j, i);
    const double dt = C->dt;
    if (t == 0) C->dtavg = C->dtavg + dt; // fl_rheol.f90:43 (no thread reads dtavg here)
    double *st = (double *)A.stress0;
    const double ar = ((const double *)A.area)[gf_ek(d, e, k)];
    double dx0, dx1, dx2, dz0, dz1, dz2, sr0, sr1, sr2;
    {
        GF_IDX n[3];
        tri_nodes(d, j, i, k, n);
        double x[3], y[3], u[3], v[3];
#pragma unroll
        for (int m = 0; m < 3; ++m) {
            x[m] = A.cord[n[m]];
            y[m] = A.cord[d.N + n[m]];
            u[m] = A.vel[n[m]];
            v[m] = A.vel[d.N + n[m]];
        }
        dx0 = gf_mulq(y[1] - y[2], ar); dx1 = gf_mulq(y[2] - y[0], ar); dx2 = gf_mulq(y[0] - y[1], ar);
        dz0 = gf_mulq(x[2] - x[1], ar); dz1 = gf_mulq(x[0] - x[2], ar); dz2 = gf_mulq(x[1] - x[0], ar);
        sr0 = gf_mulq(u[0], dx0) + gf_mulq(u[1], dx1) + gf_mulq(u[2], dx2);
        sr1 = gf_mulq(v[0], dz0) + gf_mulq(v[1], dz1) + gf_mulq(v[2], dz2);
        sr2 = gf_scale<-1>(gf_mulq(u[0], dz0) + gf_mulq(u[1], dz1) + gf_mulq(u[2], dz2) + gf_mulq(v[0], dx0) +
                           gf_mulq(v[1], dx1) + gf_mulq(v[2], dx2));
    }
    if (P.mix_strain == 1) {
        const double o0 = grp_xor(sr0, 1), o1 = grp_xor(sr1, 1);
        const bool odd = k & 1; // the pair's first triangle first
        const double em = gf_scale<-1>((odd ? o0 : sr0) + (odd ? o1 : sr1) + (odd ? sr0 : o0) + (odd ? sr1 : o1));
        const double ed = sr0 - sr1;
        sr0 = gf_scale<-1>(em + ed);
        sr1 = gf_scale<-1>(em - ed);
    }
    const double a0 = st[gf_s(d, e, 0, k)], a1 = st[gf_s(d, e, 1, k)], a2 = st[gf_s(d, e, 2, k)],
                 a3 = st[gf_s(d, e, 3, k)]; // start-of-step stresses
    double *se2sr = (double *)A.se2sr, *strain = (double *)A.strain, *sshrheat = (double *)A.sshrheat;
    double shr = sshrheat[e];
    {
        // component means over the triangles: lane c (xx, zz, xz) sums its
        // component of the strain rates and of the stresses
        double w0 = sr0, w1 = sr1, w2 = sr2, w3 = 0.0;
        grp_transpose(k, w0, w1, w2, w3);
        const double mr = gf_scale<-2>(w0 + w1 + w2 + w3);
        w0 = a0; w1 = a1; w2 = a2; w3 = 0.0;
        grp_transpose(k, w0, w1, w2, w3);
        const double ms = gf_scale<-2>(w0 + w1 + w2 + w3);
        if (k < 3 && act) {
            se2sr[gf_ek(d, e, k)] = se2sr[gf_ek(d, e, k)] + gf_mulq(mr, dt);
            // accumulates the element-averaged start-of-step stress
            // (s11/s22/s12 are reassigned before this point in fl_rheol.f90:181-183)
            strain[gf_ek(d, e, k)] = strain[gf_ek(d, e, k)] + gf_mulq(ms, dt);
        }
        // second invariants: lanes 0, 1 of the strain rate, lanes 2, 3 of the stress
        double c0 = grp_get(mr, 0), c1 = grp_get(mr, 1), c2 = grp_get(mr, 2);
        const double b0 = grp_get(ms, 0), b1 = grp_get(ms, 1), b2 = grp_get(ms, 2);
        if (k >= 2) { c0 = b0; c1 = b1; c2 = b2; }
        const double dif = c0 - c1;
        const double II = gf_scale<-1>(sqrt(gf_mulq(dif, dif) + gf_mulq(gf_scale<2>(c2), c2)));
        const double sI = gf_scale<-1>(c0 + c1);
        const double p = c0 - sI, q = c1 - sI;
        const double dev2 = gf_mulq(p, p) + gf_mulq(q, q) + gf_mulq(gf_scale<1>(c2), c2);
        const double srII = grp_get(II, 0), stII = grp_get(II, 2), srs2 = grp_get(dev2, 0);
        if (!gf_dzero(srII)) shr = shr + gf_mulq(gf_mulq(gf_ddiv(stII, srII), srs2), dt);
    }
    const int iph = A.iphase[e] - 1;
    const int irh = P.irheol[iph];
    const double bulkm = P.bulkm[iph], rmu = P.rm[iph];
    double stherm = 0.0;
    if (P.istress_therm > 0) {
        const GF_IDX n1 = gf_node(d, j, i);
        stherm = -P.alfa[iph] * P.bulkm[iph] * (A.temp[n1] - A.temp0[n1]);
    }
    double *aps = (double *)A.aps;
    double aps_e = aps[e];
    double hardn = 0.0;
    PlasticConsts<double> pc;
    const bool yields = irh == 6 || irh >= 11, creeps = irh == 3 || irh >= 11;
    {
        const bool single = A.plast_tab && tri_single_phase(P, A, d, e, iph, k);
        if (yields) {
            // single-phase elements outside the softening interval read the
            // per-phase table
            const int pst = single ? plastic_branch(P, iph, aps_e) : -1;
            if (pst >= 0) {
                const double *tb = (const double *)A.plast_tab + (GF_IDX)(pst * GF_MAXPH + iph) * GF_PT_W;
                pc.anphi = tb[0]; pc.anpsi = tb[1]; pc.amc = tb[2]; pc.e1 = tb[3];
                pc.e2 = tb[4]; pc.x1 = tb[5]; pc.ten_max = tb[6]; hardn = tb[7];
                plastic_consts_f32(pc);
            } else {
                double coh = 0, phi = 0, psi = 0;
                pre_plast<double>(P, A, d, e, aps_e, coh, phi, psi, hardn);
                pc = plastic_consts<double>(bulkm, rmu, coh, phi, psi, P.ten_off);
            }
        }
    }
    MaxwellConsts<double> mc;
    mc.ok = true;
    if (creeps) mc = maxwell_consts<double>(rmu, ((const double *)A.visn)[e], dt);
    if (!mc.ok && k == 0 && act) set_status(C, 22, (int)e);
    // stress update of this triangle
    const double de11 = gf_mulq(sr0, dt), de22 = gf_mulq(sr1, dt), de12 = gf_mulq(sr2, dt);
    const double dike = A.dike_released ? A.dike_released[e] : 0.0;
    const double dv = gf_sub_z(((const double *)A.dvol)[gf_ek(d, e, k)], dike);
    double p0 = gf_add_z(a0, stherm), p1 = gf_add_z(a1, stherm), p2 = a2, p3 = gf_add_z(a3, stherm);
    double v0 = p0, v1 = p1, v2 = p2, v3 = p3, depl = 0.0;
    if (irh == 1) elastic<double>(bulkm, rmu, p0, p1, p3, p2, de11, de22, de12);
    if (yields) plastic<double>(pc, rmu, depl, hardn, p0, p1, p3, p2, de11, de22, 0.0, de12);
    if (creeps) maxwell<double>(bulkm, mc, v0, v1, v3, v2, de11, de22, 0.0, de12, dv, P.ndim);
    bool use_visc = irh == 3;
    {
        // the smaller second invariant of the triangle sums: lanes 0 and 1 sum
        // s11 - s22 of the plastic and the viscous stress, lanes 2 and 3 s12
        double x0 = p0, x1 = v0, x2 = p2, x3 = v2, y0 = p1, y1 = v1, y2 = 0.0, y3 = 0.0;
        grp_transpose(k, x0, x1, x2, x3);
        grp_transpose(k, y0, y1, y2, y3);
        double s = x0 + x1 + x2 + x3;
        const double s4 = s - y0 - y1 - y2 - y3;
        if (k < 2) s = s4;
        double sq = gf_mulq(s, s);
        if (k >= 2) sq = gf_scale<2>(sq);
        sq = sq + grp_xor(sq, 2);
        const double sII_plas = grp_get(sq, 0), sII_visc = grp_get(sq, 1);
        if (irh >= 11) use_visc = !(sII_plas < sII_visc);
    }
    double s0 = use_visc ? v0 : p0, s1 = use_visc ? v1 : p1, s2 = use_visc ? v2 : p2, s3 = use_visc ? v3 : p3;
    // 1/ar of the stress mixing and the node-force factor 0.25/ar
    const double rar = gf_rcp(ar);
    if (P.mix_stress == 1) {
        const double oar = grp_xor(ar, 1), orar = grp_xor(rar, 1);
        const double sm = gf_scale<-1>(s0 + s1);
        const double q = gf_ddiv(sm, oar); // this triangle's mean by the other's area
        const double mean = gf_ddiv(q + grp_xor(q, 1), rar + orar);
        s0 = s0 - sm + mean;
        s1 = s1 - sm + mean;
    }
    s0 = gf_sub_z(s0, stherm);
    s1 = gf_sub_z(s1, stherm);
    s3 = gf_sub_z(s3, stherm);
    if (act) {
        st[gf_s(d, e, 0, k)] = s0;
        st[gf_s(d, e, 1, k)] = s1;
        st[gf_s(d, e, 2, k)] = s2;
        st[gf_s(d, e, 3, k)] = s3;
    }
    if (A.n_frc) {
        // fl_node's force terms of this triangle (fl_node.f90:50-254), each
        // the expression the node gather evaluates, from the stresses just
        // stored (the mesh does not move before fl_node); a vertex's place
        // 6c + 2q is that of corner c's q-th triangle (the inverse of
        // fl_node's kk / mm tables)
        // 0.25 * RN(1/ar) == RN(0.25/ar) while both are normal
        const double f = gf_dmid(ar) ? gf_scale<-2>(rar) : 0.25 / ar;
        const int w0 = k == 0 ? 0 : k == 1 ? 8 : k == 2 ? 2 : 4;
        const int w1 = k == 3 ? 22 : 12 + 2 * k;
        const int w2 = k == 0 ? 6 : k == 1 ? 18 : k == 2 ? 20 : 10;
        double *nf = A.n_frc;
        const double fx0 = gf_mulq(f, gf_mulq(s0, dx0) + gf_mulq(s2, dz0)), fy0 = gf_mulq(f, gf_mulq(s2, dx0) + gf_mulq(s1, dz0));
        const double fx1 = gf_mulq(f, gf_mulq(s0, dx1) + gf_mulq(s2, dz1)), fy1 = gf_mulq(f, gf_mulq(s2, dx1) + gf_mulq(s1, dz1));
        const double fx2 = gf_mulq(f, gf_mulq(s0, dx2) + gf_mulq(s2, dz2)), fy2 = gf_mulq(f, gf_mulq(s2, dx2) + gf_mulq(s1, dz2));
        if (act) {
            nf[(GF_IDX)w0 * d.E + e] = fx0;
            nf[(GF_IDX)(w0 + 1) * d.E + e] = fy0;
            nf[(GF_IDX)w1 * d.E + e] = fx1;
            nf[(GF_IDX)(w1 + 1) * d.E + e] = fy1;
            nf[(GF_IDX)w2 * d.E + e] = fx2;
            nf[(GF_IDX)(w2 + 1) * d.E + e] = fy2;
        }
    }
    {
        // plastic strain increment, area-weighted; elements without a yielded
        // triangle add +0
        const bool none = gf_is_pzero(depl) && gf_dmid(ar) && !signbit(ar);
        if (__all_sync(0xffffffffu, none || !yields)) {
            if (yields) aps_e = gf_plus_pzero(aps_e);
        } else {
            const double da = depl * ar;
            double sum = grp_get(da, 0), quad = grp_get(ar, 0);
#pragma unroll
            for (int q = 1; q < 4; ++q) {
                sum = sum + grp_get(da, q);
                quad = quad + grp_get(ar, q);
            }
            if (yields) aps_e = aps_e + gf_ddiv(sum, quad);
        }
        if (yields) {
            if (aps_e < 0.0) aps_e = 0.0;
            if (P.tau_heal != 0.0) aps_e = aps_e / (1.0 + dt / P.tau_heal);
            if (k == 0 && act) aps[e] = aps_e;
        }
    }
    if (P.ishearh == 1) {
        // the quotients by 2 mu (fl_rheol.f90:352-362) share one reciprocal
        const GfIntRecip r2mu = gf_int_recip(gf_scale<1>(rmu));
        const double lam_den = P.sh_lam_den[iph];
        const double lt0 = gf_mulq(lam_den, a0 + a1 + a3);
        const double e11a = gf_ddiv_by(a0 - lt0, r2mu), e22a = gf_ddiv_by(a1 - lt0, r2mu),
                     e33a = gf_ddiv_by(a3 - lt0, r2mu), e12a = gf_ddiv_by(a2, r2mu);
        const double lt1 = gf_mulq(lam_den, s0 + s1 + s3);
        const double e11b = gf_ddiv_by(s0 - lt1, r2mu), e22b = gf_ddiv_by(s1 - lt1, r2mu),
                     e33b = gf_ddiv_by(s3 - lt1, r2mu), e12b = gf_ddiv_by(s2, r2mu);
        const double d11 = de11 - (e11b - e11a), d22 = de22 - (e22b - e22a), d12 = de12 - (e12b - e12a);
        const double d33 = gf_zero_minus(e33b - e33a);
        const double m11 = gf_scale<-1>(a0 + s0), m22 = gf_scale<-1>(a1 + s1), m12 = gf_scale<-1>(a2 + s2),
                     m33 = gf_scale<-1>(a3 + s3);
        const double qk = gf_scale<-2>(gf_mulq(m11, d11) + gf_mulq(m22, d22) + gf_mulq(gf_scale<1>(m12), d12) +
                                       gf_mulq(m33, d33));
        double qsum = gf_plus_pzero(grp_get(qk, 0));
#pragma unroll
        for (int q = 1; q < 4; ++q) qsum = qsum + grp_get(qk, q);
        shr = shr + qsum;
    }
    if (k == 0 && act) sshrheat[e] = shr;
}

// The element part of fl_move (fl_move.f90:60-132): new area, dvol and the
// rotation of stress (each triangle its own) and of strain (by triangle A,
// one component per lane).
__global__ void __launch_bounds__(GF_THREADS) k_move_tri(DevClock *__restrict__ C, DevArrays A, GfDims d,
                                                         int advance_time) {
    gf_pdl_entry();
    const GF_IDX t = (GF_IDX)blockIdx.x * blockDim.x + threadIdx.x;
    const int k = (int)(t & 3);
    const bool act = (t >> 2) < d.E;
    const GF_IDX e = act ? (t >> 2) : d.E - 1;
    int j, i;
    tri_ji(d, e, j, i);
    const double dt = C->dt;
    if (advance_time && t == 0) C->time = C->time + dt; // par.f90:86, after every reader of time
    GF_IDX n[3];
    tri_nodes(d, j, i, k, n);
    double x[3], y[3], u[3], v[3];
#pragma unroll
    for (int m = 0; m < 3; ++m) {
        x[m] = A.cord[n[m]];
        y[m] = A.cord[d.N + n[m]];
        u[m] = A.vel[n[m]];
        v[m] = A.vel[d.N + n[m]];
    }
    double *area = (double *)A.area, *st = (double *)A.stress0, *strain = (double *)A.strain;
    const double ar = area[gf_ek(d, e, k)];
    const double s11 = st[gf_s(d, e, 0, k)], s22 = st[gf_s(d, e, 1, k)], s12 = st[gf_s(d, e, 2, k)];
    const double e11 = strain[gf_ek(d, e, 0)], e22 = strain[gf_ek(d, e, 1)], e12 = strain[gf_ek(d, e, 2)];
    const double det = ((gf_mul(x[1], y[2]) - gf_mul(y[1], x[2])) - (gf_mul(x[0], y[2]) - gf_mul(y[0], x[2]))) +
                       (gf_mul(x[0], y[1]) - gf_mul(y[0], x[1]));
    const double dv = gf_mul(det, ar) - 1.0;
    const GfIntRecip rdet = gf_int_recip(det);
    const double ar_new = gf_rcp_by(rdet);
    // half the curl of the velocity over the triangle, times dt
    const double curl = gf_mul(u[0], x[2] - x[1]) + gf_mul(u[1], x[0] - x[2]) + gf_mul(u[2], x[1] - x[0]) +
                        gf_mul(v[0], y[2] - y[1]) + gf_mul(v[1], y[0] - y[2]) + gf_mul(v[2], y[1] - y[0]);
    const double dw = gf_mul(gf_ddiv_by(gf_scale<-1>(curl), rdet), dt);
    const double ds = gf_mul(gf_scale<1>(s12), dw), dsd = gf_mul(dw, s22 - s11);
    const double wA = grp_get(dw, 0);
    // lane 0: e11 + 2 e12 w, lane 1: e22 - 2 e12 w, lane 2: e12 + w (e22 - e11)
    const double de = gf_mul(k == 2 ? wA : gf_scale<1>(e12), k == 2 ? e22 - e11 : wA);
    // (x - p and x + (-p) have the same bits)
    const double en = (k == 0 ? e11 : k == 1 ? e22 : e12) + (k == 1 ? gf_neg(de) : de);
    if (!act) return;
    area[gf_ek(d, e, k)] = ar_new;
    ((double *)A.dvol)[gf_ek(d, e, k)] = dv;
    st[gf_s(d, e, 0, k)] = s11 + ds;
    st[gf_s(d, e, 1, k)] = s22 - ds;
    st[gf_s(d, e, 2, k)] = s12 + dsd;
    if (k < 3) strain[gf_ek(d, e, k)] = en;
    if (!(ar_new > 0.0)) set_status(C, 40, (int)e);
}

} // namespace gfk
} // namespace
