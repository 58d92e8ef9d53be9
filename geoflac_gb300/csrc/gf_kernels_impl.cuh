// Kernel bodies and launchers of the FLAC step; included once per precision.
#pragma once

#include "gf_kernels.cuh"

// internal linkage: each precision's translation unit has its own copy
namespace {
namespace gfk {

__device__ __forceinline__ void elem_ji(const GfDims &d, GF_IDX e, int &j, int &i) {
    i = (int)(e / (d.nz - 1));
    j = (int)(e - (GF_IDX)i * (d.nz - 1));
}
__device__ __forceinline__ void node_ji(const GfDims &d, GF_IDX n, int &j, int &i) {
    i = (int)(n / d.nz);
    j = (int)(n - (GF_IDX)i * d.nz);
}

inline unsigned grid_for(GF_IDX n, int threads = GF_THREADS) { return (unsigned)((n + threads - 1) / threads); }

// ======================================================================
// Mixed path: the element's share of the node forces of fl_node.f90.  For
// corner c (node 1..4 = (j,i), (j+1,i), (j,i+1), (j+1,i+1)) the three
// triangles that contain it contribute -0.25/ar * (s . grad N); written as
//   F_c = -sum_t 0.25/ar_t * ((s_t - s_ref) . grad N_c,t)   (small: stress
//         variation inside the element, s_ref = triangle 1's stored stress)
//   G_c =  sum_t 0.25/ar_t * grad N_c,t
// so that a node sums F_c - (s_ref,e - s_ref,n) . G_c over its elements
// (sum_e G_c = 0 around an interior node): every FP32 term is a difference.
// The triangle/vertex tables are fl_node.f90:7-8 for quad 4 - c.
__device__ __forceinline__ void elem_corner_forces(const float dx[3][4], const float dz[3][4], const float ar[4],
                                                   const float sn[4][4], float *__restrict__ frc, GF_IDX E,
                                                   GF_IDX e) {
    const int kk[4][3] = {{1, 2, 3}, {0, 1, 2}, {0, 1, 3}, {0, 2, 3}};
    const int mm[4][3] = {{2, 2, 1}, {1, 1, 1}, {2, 0, 2}, {0, 0, 0}};
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        const int qd = 3 - c;
        float fx = 0.0f, fy = 0.0f, gx = 0.0f, gz = 0.0f;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const int t = kk[qd][k], m = mm[qd][k];
            const float factor = 0.25f / ar[t];
            const float ax = factor * dx[m][t], az = factor * dz[m][t];
            const float sxx = sn[0][t] - sn[0][1], szz = sn[1][t] - sn[1][1], sxz = sn[2][t] - sn[2][1];
            fx -= sxx * ax + sxz * az;
            fy -= sxz * ax + szz * az;
            gx += ax;
            gz += az;
        }
        frc[(4 * c + 0) * E + e] = fx;
        frc[(4 * c + 1) * E + e] = fy;
        frc[(4 * c + 2) * E + e] = gx;
        frc[(4 * c + 3) * E + e] = gz;
    }
}

// ======================================================================
// fl_rheol (fl_rheol.f90:4-389) in the mixed path: one thread per element
// (the FP64 path: k_rheol_tri).
template <class R> __device__ __forceinline__ void b_k_rheol(const DevParams *__restrict__ Pp, DevClock *__restrict__ C, DevArrays A, GfDims d, int update_visc, int nloop, GF_IDX e) {
    if (e >= d.E) return;
    const DevParams &P = *Pp;
    int j, i;
    elem_ji(d, e, j, i);
    const double dtd = C->dt;
    const R dt = gf_to<R>(dtd);
    R *st = (R *)A.stress0;
    const R *area = (const R *)A.area;

    GF_IDX n1 = gf_node(d, j, i);
    // Everything the element reads is loaded before its first store: the
    // compiler keeps a load behind any store that might alias it, and with
    // reads between the stores each field's latency came on top of the others'
    R *se2sr = (R *)A.se2sr;
    R *sshrheat = (R *)A.sshrheat;
    R *strain = (R *)A.strain;
    R *aps = (R *)A.aps;
    R *visn = (R *)A.visn;
    const R *dvol = (const R *)A.dvol;
    R vx[4], vy[4];
    R ar[4], dvl[4], se[3], sn3[3];
    R s0v[4][4]; // start-of-step stresses [comp][tri]
    for (int k = 0; k < 4; ++k) ar[k] = area[gf_ek(d, e, k)];
    R dx[3][4], dz[3][4], sr[3][4];
    // FP32 from the hi/lo splits: coordinates and velocities relative to
    // the quad's node 1 (each triangle's shape derivatives sum to zero,
    // so a common velocity offset drops out of the strain rates)
    QuadF qf;
    load_vel_rel(A, d, j, i, vx, vy);
    load_quad_rel(A, d, j, i, qf);
    int iph = A.iphase[e] - 1;
#pragma unroll
    for (int k = 0; k < 4; ++k)
#pragma unroll
        for (int c = 0; c < 4; ++c) s0v[c][k] = st[gf_s(d, e, c, k)];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        se[c] = se2sr[gf_ek(d, e, c)];
        sn3[c] = strain[gf_ek(d, e, c)];
    }
    R shr = sshrheat[e];
    R aps_e = aps[e];
    // mixed path: stored normal stresses are deviations from -pref
    const R pref = A.pr_hi[e]; // == float(p_ref)
#pragma unroll
    for (int k = 0; k < 4; ++k) dvl[k] = dvol[gf_ek(d, e, k)];
    R dike = A.dike_released ? gf_to<R>(A.dike_released[e]) : R(0);
    R vis = visn[e]; // (unless it is updated below)
    const PhaseTests pt = phase_tests(P, A, d, e);
    shape_derivs_f(qf, ar, dx, dz);
    // node triplets of triangles A,B,C,D: (1,2,3), (3,2,4), (1,2,4), (1,4,3)
    const int tn[4][3] = {{0, 1, 2}, {2, 1, 3}, {0, 1, 3}, {0, 3, 2}};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        R a0 = vx[tn[k][0]], a1 = vx[tn[k][1]], a2 = vx[tn[k][2]];
        R b0 = vy[tn[k][0]], b1 = vy[tn[k][1]], b2 = vy[tn[k][2]];
        sr[0][k] = a0 * dx[0][k] + a1 * dx[1][k] + a2 * dx[2][k];
        sr[1][k] = b0 * dz[0][k] + b1 * dz[1][k] + b2 * dz[2][k];
        sr[2][k] = gf_scale<-1>(a0 * dz[0][k] + a1 * dz[1][k] + a2 * dz[2][k] +
                                b0 * dx[0][k] + b1 * dx[1][k] + b2 * dx[2][k]);
    }
    if (P.mix_strain == 1) {
#pragma unroll
        for (int k = 0; k < 4; k += 2) {
            R em = R(0.5) * (sr[0][k] + sr[1][k] + sr[0][k + 1] + sr[1][k + 1]);
            R eda = sr[0][k] - sr[1][k];
            R edb = sr[0][k + 1] - sr[1][k + 1];
            sr[0][k] = R(0.5) * (em + eda);
            sr[1][k] = R(0.5) * (em - eda);
            sr[0][k + 1] = R(0.5) * (em + edb);
            sr[1][k + 1] = R(0.5) * (em - edb);
        }
    }
    R s11 = gf_scale<-2>(sr[0][0] + sr[0][1] + sr[0][2] + sr[0][3]);
    R s22 = gf_scale<-2>(sr[1][0] + sr[1][1] + sr[1][2] + sr[1][3]);
    R s12 = gf_scale<-2>(sr[2][0] + sr[2][1] + sr[2][2] + sr[2][3]);
    R srII = gf_scale<-1>(m_sqrt((s11 - s22) * (s11 - s22) + gf_scale<2>(s12) * s12));
    R srI = gf_scale<-1>(s11 + s22);
    R srs2 = (s11 - srI) * (s11 - srI) + (s22 - srI) * (s22 - srI) + gf_scale<1>(s12) * s12;
    se[0] = se[0] + s11 * dt;
    se[1] = se[1] + s22 * dt;
    se[2] = se[2] + s12 * dt;
    s11 = gf_scale<-2>(s0v[0][0] + s0v[0][1] + s0v[0][2] + s0v[0][3]);
    s22 = gf_scale<-2>(s0v[1][0] + s0v[1][1] + s0v[1][2] + s0v[1][3]);
    s12 = gf_scale<-2>(s0v[2][0] + s0v[2][1] + s0v[2][2] + s0v[2][3]);
    R stII = gf_scale<-1>(m_sqrt((s11 - s22) * (s11 - s22) + gf_scale<2>(s12) * s12));
    if (srII != R(0.0)) shr = shr + gf_ddiv(stII, srII) * srs2 * dt;

    int irh = P.irheol[iph];
    const R bulkm = P.f_bulkm[iph], rmu = P.f_rm[iph];
    R stherm = R(0.0);
    if (P.istress_therm > 0)
        stherm = R(-P.alfa[iph] * P.bulkm[iph] * (A.temp[n1] - A.temp0[n1]));
    R hardn = 0;
    PlasticConsts<R> pc;
    if (irh == 6 || irh >= 11) {
        // single-phase elements outside the softening interval read the
        // per-phase table
        const int pst = A.plast_tab ? plastic_table_state<R>(P, iph, aps_e, pt) : -1;
        if (pst >= 0) {
            const R *t = (const R *)A.plast_tab + (GF_IDX)(pst * GF_MAXPH + iph) * GF_PT_W;
            pc.anphi = t[0]; pc.anpsi = t[1]; pc.amc = t[2]; pc.e1 = t[3];
            pc.e2 = t[4]; pc.x1 = t[5]; pc.ten_max = t[6]; hardn = t[7];
            plastic_consts_f32(pc);
        } else {
            R coh = 0, phi = 0, psi = 0;
            pre_plast<R>(P, A, d, e, aps_e, coh, phi, psi, hardn);
            pc = plastic_consts<R>(bulkm, rmu, coh, phi, psi, P.f_ten_off);
        }
    }
    if ((irh == 3 || irh >= 11) && update_visc) {
        vis = R(visc_of<R>(P, A, d, j, i, e, st));
        visn[e] = vis;
    }
    if (e == 0) C->dtavg = C->dtavg + dtd; // fl_rheol.f90:43 (no thread reads dtavg here)
#pragma unroll
    for (int c = 0; c < 3; ++c) se2sr[gf_ek(d, e, c)] = se[c];
    R sp[4][4], sv[4][4], depl[4] = {0, 0, 0, 0};
    bool plas_mod = false;
    MaxwellConsts<R> mc;
    if (irh == 3 || irh >= 11) mc = maxwell_consts<R>(rmu, vis, dt);
    const bool ok = !(irh == 3 || irh >= 11) || mc.ok;
    R sumD = 0, sumD12 = 0; // strain-increment sums for the FP32 selection
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        R de11 = sr[0][k] * dt, de22 = sr[1][k] * dt, de12 = sr[2][k] * dt, de33 = R(0.0);
        // (dike and stherm are +0 without dikes and thermal stress:
        // gf_sub_z / gf_add_z take them on the integer pipes)
        R dv = gf_sub_z(dvl[k], dike);
        sp[0][k] = gf_add_z(s0v[0][k], stherm);
        sp[1][k] = gf_add_z(s0v[1][k], stherm);
        sp[2][k] = s0v[2][k];
        sp[3][k] = gf_add_z(s0v[3][k], stherm);
        sv[0][k] = sp[0][k]; sv[1][k] = sp[1][k]; sv[2][k] = sp[2][k]; sv[3][k] = sp[3][k];
        if (irh == 1) {
            elastic<R>(bulkm, rmu, sp[0][k], sp[1][k], sp[3][k], sp[2][k], de11, de22, de12);
        } else if (irh == 3) {
            maxwell<R>(bulkm, mc, sv[0][k], sv[1][k], sv[3][k], sv[2][k], de11, de22, de33, de12, dv, P.ndim);
        } else if (irh == 6) {
            bool m;
            plastic_sel(pc, rmu, depl[k], hardn, sp[0][k], sp[1][k], sp[3][k], sp[2][k], de11, de22, de33, de12, pref,
                        m);
        } else if (irh >= 11) {
            bool m;
            plastic_sel(pc, rmu, depl[k], hardn, sp[0][k], sp[1][k], sp[3][k], sp[2][k], de11, de22, de33, de12, pref,
                        m);
            plas_mod = plas_mod || m;
            maxwell<R>(bulkm, mc, sv[0][k], sv[1][k], sv[3][k], sv[2][k], de11, de22, de33, de12, dv, P.ndim);
            sumD = sumD + (de11 - de22);
            sumD12 = sumD12 + de12;
        }
    }
    if (!ok) set_status(C, 22, (int)e);
    R sn[4][4]; // new stresses [comp][tri]
    bool use_visc = (irh == 3);
    if (irh >= 11) {
        R a = sp[0][0] + sp[0][1] + sp[0][2] + sp[0][3] - sp[1][0] - sp[1][1] - sp[1][2] - sp[1][3];
        R b = sp[2][0] + sp[2][1] + sp[2][2] + sp[2][3];
        R sII_plas = a * a + gf_scale<2>(b * b);
        a = sv[0][0] + sv[0][1] + sv[0][2] + sv[0][3] - sv[1][0] - sv[1][1] - sv[1][2] - sv[1][3];
        b = sv[2][0] + sv[2][1] + sv[2][2] + sv[2][3];
        R sII_visc = a * a + gf_scale<2>(b * b);
        use_visc = !(sII_plas < sII_visc);
        if (!plas_mod) {
            R pa = sp[0][0] + sp[0][1] + sp[0][2] + sp[0][3] - sp[1][0] - sp[1][1] - sp[1][2] - sp[1][3];
            R pb = sp[2][0] + sp[2][1] + sp[2][2] + sp[2][3];
            R S = s0v[0][0] + s0v[0][1] + s0v[0][2] + s0v[0][3] - s0v[1][0] - s0v[1][1] - s0v[1][2] - s0v[1][3];
            R B = s0v[2][0] + s0v[2][1] + s0v[2][2] + s0v[2][3];
            use_visc = maxwell_wins_unyielded(float(pa), float(pb), float(S), float(B), float(sumD), float(sumD12),
                                              float(rmu), float(vis), float(dt));
        }
    }
#pragma unroll
    for (int k = 0; k < 4; ++k)
#pragma unroll
        for (int c = 0; c < 4; ++c) sn[c][k] = use_visc ? sv[c][k] : sp[c][k];
    if (P.mix_stress == 1) {
#pragma unroll
        for (int h = 0; h < 4; h += 2) {
            R ra = ar[h], rb = ar[h + 1];
            R s0a = gf_scale<-1>(sn[0][h] + sn[1][h]);
            R s0b = gf_scale<-1>(sn[0][h + 1] + sn[1][h + 1]);
            R quad_area = R(1.0) / ra + R(1.0) / rb;
            R s0 = (s0a / rb + s0b / ra) / quad_area;
            sn[0][h] = sn[0][h] - s0a + s0;
            sn[1][h] = sn[1][h] - s0a + s0;
            sn[0][h + 1] = sn[0][h + 1] - s0b + s0;
            sn[1][h + 1] = sn[1][h + 1] - s0b + s0;
        }
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        sn[0][k] = gf_sub_z(sn[0][k], stherm);
        sn[1][k] = gf_sub_z(sn[1][k], stherm);
        sn[3][k] = gf_sub_z(sn[3][k], stherm);
    }
#pragma unroll
    for (int k = 0; k < 4; ++k)
#pragma unroll
        for (int c = 0; c < 4; ++c) st[gf_s(d, e, c, k)] = sn[c][k];
    {
        // the node gather's corner forces of the new stresses (the mesh does
        // not move before fl_node); shape derivatives taken again rather than
        // kept live through the stress update
        float dx2[3][4], dz2[3][4];
        shape_derivs_f(qf, ar, dx2, dz2);
        elem_corner_forces(dx2, dz2, ar, sn, A.e_frc, d.E, e);
    }
    if (irh == 6 || irh >= 11) {
        R quad_area = ar[0] + ar[1] + ar[2] + ar[3];
        aps_e = aps_e + gf_ddiv(depl[0] * ar[0] + depl[1] * ar[1] + depl[2] * ar[2] + depl[3] * ar[3], quad_area);
        if (aps_e < R(0.0)) aps_e = R(0.0);
        if (P.f_tau_heal != 0.0f) aps_e = aps_e / (1.0f + dt / P.f_tau_heal);
        aps[e] = aps_e;
    }
    // accumulates the element-averaged start-of-step stress (s11/s22/s12 are
    // reassigned before this point in fl_rheol.f90:181-183)
    s11 = s11 - pref; // total stress, not the stored deviation
    s22 = s22 - pref;
    strain[gf_ek(d, e, 0)] = sn3[0] + s11 * dt;
    strain[gf_ek(d, e, 1)] = sn3[1] + s22 * dt;
    strain[gf_ek(d, e, 2)] = sn3[2] + s12 * dt;
    if (P.ishearh == 1) {
        R qsum = R(0.0);
        R lambda = bulkm - R(2.0 / 3.0) * rmu, mu = rmu;
        R den_el = R(3.0) * lambda + R(2.0) * mu;
        if (m_abs(den_el) < R(1e-30)) den_el = den_el < R(0) ? R(-1e-30) : R(1e-30);
        // the same elastic-strain differences with one reciprocal and the
        // stress changes taken first
        const float lamr = lambda / den_el, inv2mu = 1.0f / (2.0f * mu);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            float f11 = sn[0][k], f22 = sn[1][k], f12 = sn[2][k], f33 = sn[3][k];
            float dtr = ((f11 - s0v[0][k]) + (f22 - s0v[1][k])) + (f33 - s0v[3][k]);
            float d11 = sr[0][k] * dt - ((f11 - s0v[0][k]) - lamr * dtr) * inv2mu;
            float d22 = sr[1][k] * dt - ((f22 - s0v[1][k]) - lamr * dtr) * inv2mu;
            float d12 = sr[2][k] * dt - (f12 - s0v[2][k]) * inv2mu;
            float d33 = -(((f33 - s0v[3][k]) - lamr * dtr) * inv2mu);
            float a11 = 0.5f * (s0v[0][k] + f11), a22 = 0.5f * (s0v[1][k] + f22),
                  a12 = 0.5f * (s0v[2][k] + f12), a33 = 0.5f * (s0v[3][k] + f33);
            float qk = a11 * d11 + a22 * d22 + 2.0f * a12 * d12 + a33 * d33;
            qk -= pref * (d11 + d22 + d33); // isotropic reference part
            qsum = qsum + 0.25f * qk;
        }
        shr = shr + qsum;
    }
    sshrheat[e] = shr;
    (void)nloop;
}
// mixed path: 2 CTAs per SM (128 registers).  Bound by the latency of its loads
// (about half of the issue slots' wait), so they come first and together: a
// step of 1000x300 elements 102.4 -> 93.5 us, of 60x20 32.6 -> 29.4 us with
// k_move_elem's; 3 CTAs (80 registers, more spills) 97, 20 warps of 96
// registers 93.
template <class R> __global__ void __launch_bounds__(GF_THREADS, 2) k_rheol(const DevParams *__restrict__ Pp, DevClock *__restrict__ C, DevArrays A, GfDims d, int update_visc, int nloop) {
    gf_pdl_entry();
    b_k_rheol<R>(Pp, C, A, d, update_visc, nloop, (GF_IDX)blockIdx.x * blockDim.x + threadIdx.x);
}

template <class R> __device__ __forceinline__ void b_k_rheol_avg(DevClock *__restrict__ C, DevArrays A, GfDims d, int reset, GF_IDX e) {
    if (e >= d.E) return;
    R *se2sr = (R *)A.se2sr;
    R *e2sr = (R *)A.e2sr;
    R *shrheat = (R *)A.shrheat;
    R *sshrheat = (R *)A.sshrheat;
    R dtavg = R(C->dtavg);
    R a = se2sr[gf_ek(d, e, 0)], b = se2sr[gf_ek(d, e, 1)], q = se2sr[gf_ek(d, e, 2)];
    e2sr[e] = (R(0.5) * m_sqrt((a - b) * (a - b) + R(4.0) * q * q)) / dtavg;
    shrheat[e] = sshrheat[e] / dtavg;
    if (reset) {
        se2sr[gf_ek(d, e, 0)] = R(0.0);
        se2sr[gf_ek(d, e, 1)] = R(0.0);
        se2sr[gf_ek(d, e, 2)] = R(0.0);
        sshrheat[e] = R(0.0);
    }
}
template <class R> __global__ void __launch_bounds__(GF_THREADS) k_rheol_avg(DevClock *__restrict__ C, DevArrays A, GfDims d, int reset) {
    gf_pdl_entry();
    b_k_rheol_avg<R>(C, A, d, reset, (GF_IDX)blockIdx.x * blockDim.x + threadIdx.x);
}

// scalar bookkeeping of fl_rheol: dtavg += dt at entry; dtavg = 0 at a reset
__device__ __forceinline__ void b_k_rheol_clock(DevClock *C, int phase) {
    if (phase == 0)
        C->dtavg = C->dtavg + C->dt;
    else
        C->dtavg = 0.0;
}
__global__ void k_rheol_clock(DevClock *C, int phase) {
    b_k_rheol_clock(C, phase);
}

// ======================================================================
// fl_node (fl_node.f90:3-393): one thread per node, forces gathered from
// the 4 adjacent quads in the reference's order, no atomics.
//
// Threads are numbered boundary ring first (top row, bottom row, left and
// right columns), then the interior nodes (column by column, j fastest), so
// that the boundary nodes, which take the FP64 path with water load and
// Winkler foundation, run in warps of their own and start first.
__device__ __forceinline__ GF_IDX node_of_slot(const GfDims &d, GF_IDX t) {
    const int nzi = d.nz - 2;
    if (t < d.nx) return gf_node(d, 0, (int)t);
    t -= d.nx;
    if (t < d.nx) return gf_node(d, d.nz - 1, (int)t);
    t -= d.nx;
    if (t < nzi) return gf_node(d, 1 + (int)t, 0);
    t -= nzi;
    if (t < nzi) return gf_node(d, 1 + (int)t, d.nx - 1);
    t -= nzi;
    const int i = (int)(t / nzi);
    return gf_node(d, 1 + (int)(t - (GF_IDX)i * nzi), 1 + i);
}

// (hi, lo) + b in FP32 pairs: two-sum of hi and b, then renormalised
__device__ __forceinline__ void ff_add(float &hi, float &lo, float b) {
    const float s = hi + b;
    const float bb = s - hi;
    const float err = (hi - (s - bb)) + (b - bb);
    const float l = lo + err;
    hi = s + l;
    lo = l - (hi - s);
}

// Mixed path, interior node.  Stored normal stresses are deviations from
// the element's reference pressure p_ref.  The node sums its four elements'
// corner forces (elem_corner_forces, written by fl_rheol) with the
// reference-stress differences to one neighbouring triangle (sigma_n) and the
// p_ref differences, all small, so FP32 resolves the net force.  Damping and
// the velocity increment are FP32; the velocity is carried as its hi/lo FP32
// pair and written back to the FP64 array as hi + lo.
__device__ __forceinline__ void node_interior_f(const DevParams &P, const DevClock *__restrict__ C, DevArrays &A,
                                                const GfDims &d, GF_IDX n, int j, int i) {
    const float *st = (const float *)A.stress0;
    const float *frc = A.e_frc;
    const GF_IDX E = d.E;
    const GF_IDX en = gf_elem(d, j - 1, i - 1);
    const float nxx = st[gf_s(d, en, 0, 1)], nzz = st[gf_s(d, en, 1, 1)], nxz = st[gf_s(d, en, 2, 1)];
    float fx0 = 0.0f, fy0 = 0.0f;
#pragma unroll
    for (int qd = 0; qd < 4; ++qd) {
        const int je = j + (qd < 2 ? -1 : 0), ie = i + ((qd & 1) ? 0 : -1);
        const GF_IDX e = gf_elem(d, je, ie);
        const int c = 3 - qd; // this node's corner of element e
        const float dp = hl_diff(A.pr_hi, A.pr_lo, e, en);
        const float rxx = (st[gf_s(d, e, 0, 1)] - nxx) - dp;
        const float rzz = (st[gf_s(d, e, 1, 1)] - nzz) - dp;
        const float rxz = st[gf_s(d, e, 2, 1)] - nxz;
        const float gx = frc[(4 * c + 2) * E + e], gz = frc[(4 * c + 3) * E + e];
        fx0 += frc[(4 * c + 0) * E + e] - (rxx * gx + rxz * gz);
        fy0 += frc[(4 * c + 1) * E + e] - (rxz * gx + rzz * gz);
    }
    float f0 = fx0;
    float f1 = fy0 - gf_d2f(A.rmass[n]) * P.f_g;
    const float dtf = gf_d2f(C->dt);
    float drat = dtf / gf_d2f(C->dt_elastic);
    if (drat < 1.0f) drat = 1.0f;
    float h0 = A.vel_hi[n], l0 = A.vel_lo[n], h1 = A.vel_hi[d.N + n], l1 = A.vel_lo[d.N + n];
    const int c0 = A.ncod[n], c1 = A.ncod[d.N + n];
    if ((c0 & 1) != 1 && fabsf(h0) > 1.0e-13f) f0 = f0 - P.f_demf * copysignf(fabsf(f0), h0);
    if ((c1 & 2) != 2 && fabsf(h1) > 1.0e-13f) f1 = f1 - P.f_demf * copysignf(fabsf(f1), h1);
    const float s = dtf / (gf_d2f(A.amass[n]) * drat * drat);
    double v0, v1;
    if (c0 == 1) {
        v0 = A.bc[n];
        gf_split(v0, h0, l0);
    } else {
        ff_add(h0, l0, s * f0);
        v0 = gf_f2d(h0) + gf_f2d(l0);
    }
    if (c1 == 1) {
        v1 = A.bc[d.N + n];
        gf_split(v1, h1, l1);
    } else {
        ff_add(h1, l1, s * f1);
        v1 = gf_f2d(h1) + gf_f2d(l1);
    }
    A.vel[n] = v0;
    A.vel[d.N + n] = v1;
    A.vel_hi[n] = h0;
    A.vel_lo[n] = l0;
    A.vel_hi[d.N + n] = h1;
    A.vel_lo[d.N + n] = l1;
}

template <class R> __device__ __forceinline__ void b_k_node(const DevParams *__restrict__ Pp, DevClock *__restrict__ C, DevArrays A, GfDims d, GF_IDX slot, int terms = 0) {
    if (slot >= d.N) return;
    const GF_IDX n = node_of_slot(d, slot);
    const DevParams &P = *Pp;
    int j, i;
    node_ji(d, n, j, i);
    const int nx = d.nx, nz = d.nz;
    const R *st = (const R *)A.stress0;
    const R *area = (const R *)A.area;
    // kk/mm tables of fl_node.f90:7-8 (0-based)
    const int kk[4][3] = {{1, 2, 3}, {0, 1, 2}, {0, 1, 3}, {0, 2, 3}};
    const int mm[4][3] = {{2, 2, 1}, {1, 1, 1}, {2, 0, 2}, {0, 0, 0}};
    double f0, f1;
    const bool interior = j > 0 && j < nz - 1 && i > 0 && i < nx - 1;
    if constexpr (sizeof(R) == sizeof(float)) {
        if (interior) {
            node_interior_f(P, C, A, d, n, j, i);
            return;
        }
    }
    if constexpr (sizeof(R) == sizeof(float)) {
        // Mixed path, boundary node: the elements' corner forces plus their
        // total reference stress (triangle-1 stress less p_ref) against the
        // corner geometry G_c, in FP64 from the node coordinates:
        // 0.25/ar * grad N = 0.25 * (y_u - y_v, x_v - x_u) for the edge (u, v)
        // that shape_derivs uses for vertex m of triangle t.
        const int uv[4][3][2] = {{{1, 2}, {2, 0}, {0, 1}}, {{1, 3}, {3, 2}, {2, 1}},
                                 {{1, 3}, {3, 0}, {0, 1}}, {{3, 2}, {2, 0}, {0, 3}}};
        const float *frc = A.e_frc;
        const double *cx = A.cord, *cy = A.cord + d.N;
        double gx = 0.0, gy = 0.0;
#pragma unroll
        for (int qd = 0; qd < 4; ++qd) {
            int je = j + (qd < 2 ? -1 : 0), ie = i + ((qd & 1) ? 0 : -1);
            if (je < 0 || ie < 0 || je > nz - 2 || ie > nx - 2) continue;
            const GF_IDX e = gf_elem(d, je, ie);
            const int c = 3 - qd;
            GF_IDX nn[4];
            quad_nodes(d, je, ie, nn);
            double Gx = 0.0, Gz = 0.0;
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const int t = kk[qd][k], m = mm[qd][k];
                const GF_IDX u = nn[uv[t][m][0]], v = nn[uv[t][m][1]];
                Gx += cy[u] - cy[v];
                Gz += cx[v] - cx[u];
            }
            Gx *= 0.25;
            Gz *= 0.25;
            const double pe = A.p_ref[e];
            const double rxx = (double)st[gf_s(d, e, 0, 1)] - pe, rzz = (double)st[gf_s(d, e, 1, 1)] - pe,
                         rxz = (double)st[gf_s(d, e, 2, 1)];
            gx += (double)frc[(4 * c + 0) * d.E + e] - (rxx * Gx + rxz * Gz);
            gy += (double)frc[(4 * c + 1) * d.E + e] - (rxz * Gx + rzz * Gz);
        }
        f0 = gx;
        f1 = gy - A.rmass[n] * P.g;
    } else if (terms) {
        // FP64 path, terms written by fl_rheol: the reference's sum order
        R fx0 = R(0.0), fy0 = R(0.0);
#pragma unroll
        for (int qd = 0; qd < 4; ++qd) {
            int je = j + (qd < 2 ? -1 : 0), ie = i + ((qd & 1) ? 0 : -1);
            if (je < 0 || ie < 0 || je > nz - 2 || ie > nx - 2) continue;
            const GF_IDX e = gf_elem(d, je, ie);
            const int c = 3 - qd;
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                fx0 = fx0 - A.n_frc[(GF_IDX)(6 * c + 2 * k) * d.E + e];
                fy0 = fy0 - A.n_frc[(GF_IDX)(6 * c + 2 * k + 1) * d.E + e];
            }
        }
        f0 = (double)fx0;
        f1 = (double)fy0 - gf_mul(A.rmass[n], P.g);
    } else {
        // FP64 path: the reference's gather from the four quads
        R fx0 = R(0.0), fy0 = R(0.0);
#pragma unroll
        for (int qd = 0; qd < 4; ++qd) {
            int je = j + (qd < 2 ? -1 : 0), ie = i + ((qd & 1) ? 0 : -1);
            if (je < 0 || ie < 0 || je > nz - 2 || ie > nx - 2) continue;
            GF_IDX e = gf_elem(d, je, ie);
            Quad q;
            load_quad(A.cord, d, je, ie, q);
            R ar[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) ar[k] = area[gf_ek(d, e, k)];
            R dx[3][4], dz[3][4];
            shape_derivs<R>(q, ar, dx, dz);
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                int t = kk[qd][k], m = mm[qd][k];
                R factor = R(0.25) / ar[t];
                R sxx = st[gf_s(d, e, 0, t)], szz = st[gf_s(d, e, 1, t)], sxz = st[gf_s(d, e, 2, t)];
                R fx = factor * (sxx * dx[m][t] + sxz * dz[m][t]);
                R fy = factor * (sxz * dx[m][t] + szz * dz[m][t]);
                fx0 = fx0 - fx;
                fy0 = fy0 - fy;
            }
        }
        f0 = (double)fx0;
        f1 = (double)fy0 - A.rmass[n] * P.g;
    }
    const double *cord = A.cord;
    if (P.nyhydro > 0 && j == 0) { // water load on the surface
        double rho_water_g = 1030.0 * P.g;
        double water_depth = (i < nx - 1) ? 0.5 * (cord[d.N + gf_node(d, 0, i + 1)] + cord[d.N + gf_node(d, 0, i)])
                                          : 0.5 * (cord[d.N + gf_node(d, 0, i - 1)] + cord[d.N + gf_node(d, 0, i)]);
        if (water_depth < 0.0) {
            double pl = 0, dlxl = 0, dlyl = 0, pr = 0, dlxr = 0, dlyr = 0;
            if (i > 0) {
                pl = rho_water_g * ((cord[d.N + gf_node(d, 0, i - 1)] + cord[d.N + gf_node(d, 0, i)]) / 2.0);
                dlxl = cord[gf_node(d, 0, i)] - cord[gf_node(d, 0, i - 1)];
                dlyl = cord[d.N + gf_node(d, 0, i)] - cord[d.N + gf_node(d, 0, i - 1)];
            }
            if (i < nx - 1) {
                pr = rho_water_g * ((cord[d.N + gf_node(d, 0, i + 1)] + cord[d.N + gf_node(d, 0, i)]) / 2.0);
                dlxr = cord[gf_node(d, 0, i + 1)] - cord[gf_node(d, 0, i)];
                dlyr = cord[d.N + gf_node(d, 0, i + 1)] - cord[d.N + gf_node(d, 0, i)];
            }
            f0 = f0 - 0.5 * pl * dlyl - 0.5 * pr * dlyr;
            f1 = f1 + 0.5 * pl * dlxl + 0.5 * pr * dlxr;
        }
    }
    if (P.nyhydro > 0 && j == nz - 1) { // Winkler foundation
        int ips = P.iphsub - 1;
        double zb = cord[d.N + n];
        double p_est = P.pisos + 0.5 * (P.den[ips] + P.drosub) * P.g * (zb - P.rzbo);
        double rosubg = P.g * (P.den[ips] + P.drosub) * (1 - P.alfa[ips] * A.temp[n] + P.beta[ips] * p_est);
        double pl = 0, dlxl = 0, dlyl = 0, pr = 0, dlxr = 0, dlyr = 0;
        if (i > 0) {
            GF_IDX m = gf_node(d, nz - 1, i - 1);
            pl = P.pisos - rosubg * ((cord[d.N + m] + zb) / 2.0 - P.rzbo);
            dlxl = cord[n] - cord[m];
            dlyl = zb - cord[d.N + m];
        }
        if (i < nx - 1) {
            GF_IDX m = gf_node(d, nz - 1, i + 1);
            pr = P.pisos - rosubg * ((cord[d.N + m] + zb) / 2.0 - P.rzbo);
            dlxr = cord[m] - cord[n];
            dlyr = cord[d.N + m] - zb;
        }
        f0 = f0 - 0.5 * pl * dlyl - 0.5 * pr * dlyr;
        f1 = f1 + 0.5 * pl * dlxl + 0.5 * pr * dlxr;
    }
    double dt = C->dt;
    double drat = gf_ddiv(dt, C->dt_elastic); // (divisions off the FP64 pipe: gf_ddiv)
    if (drat < 1.0) drat = 1.0;
    double *vel = A.vel;
    double v0 = vel[n], v1 = vel[d.N + n];
    int c0 = A.ncod[n], c1 = A.ncod[d.N + n];
    // (the products and the |v| > 1e-13 tests on the integer pipes: gf_mul,
    // gf_abs_gt)
    if ((c0 & 1) != 1 && gf_abs_gt(v0, 1.0e-13)) f0 = f0 - gf_mul(P.demf, copysign(fabs(f0), v0));
    if ((c1 & 2) != 2 && gf_abs_gt(v1, 1.0e-13)) f1 = f1 - gf_mul(P.demf, copysign(fabs(f1), v1));
    double am = A.amass[n];
    if (sizeof(R) == sizeof(float)) {
        // FP32 increment on the FP64 velocity
        float s = gf_d2f(dt) / (gf_d2f(am) * gf_d2f(drat) * gf_d2f(drat));
        v0 = (c0 == 1) ? A.bc[n] : v0 + gf_f2d(s * gf_d2f(f0));
        v1 = (c1 == 1) ? A.bc[d.N + n] : v1 + gf_f2d(s * gf_d2f(f1));
    } else {
        const double den = gf_mul(gf_mul(am, drat), drat);
        v0 = (c0 == 1) ? A.bc[n] : v0 + gf_ddiv(gf_mul(dt, f0), den);
        v1 = (c1 == 1) ? A.bc[d.N + n] : v1 + gf_ddiv(gf_mul(dt, f1), den);
    }
    if (P.i_prestress == 1 && C->time < 600e3 * GF_SEC_YEAR) {
        if (j == nz - 1 || i == 0 || i == nx - 1) {
            v0 = 0.0;
            v1 = 0.0;
        }
    }
    vel[n] = v0;
    vel[d.N + n] = v1;
    if (sizeof(R) == sizeof(float)) {
        float h0, l0, h1, l1;
        gf_split(v0, h0, l0);
        gf_split(v1, h1, l1);
        A.vel_hi[n] = h0;
        A.vel_lo[n] = l0;
        A.vel_hi[d.N + n] = h1;
        A.vel_lo[d.N + n] = l1;
    }
}
template <class R> __global__ void __launch_bounds__(GF_THREADS) k_node(const DevParams *__restrict__ Pp, DevClock *__restrict__ C, DevArrays A, GfDims d, int terms) {
    gf_pdl_entry();
    b_k_node<R>(Pp, C, A, d, (GF_IDX)blockIdx.x * blockDim.x + threadIdx.x, terms);
}

// ======================================================================
// fl_move (fl_move.f90:3-132)
__device__ __forceinline__ void b_k_move_cord(DevClock *__restrict__ C, DevArrays A, GfDims d, GF_IDX n) {
    if (n >= 2 * d.N) return;
    const double c = A.cord[n] + A.vel[n] * C->dt;
    A.cord[n] = c;
    if (A.cord_hi) {
        float h, l;
        gf_split(c, h, l);
        A.cord_hi[n] = h;
        A.cord_lo[n] = l;
    }
}
__global__ void __launch_bounds__(GF_THREADS) k_move_cord(DevClock *__restrict__ C, DevArrays A, GfDims d) {
    gf_pdl_entry();
    b_k_move_cord(C, A, d, (GF_IDX)blockIdx.x * blockDim.x + threadIdx.x);
}

// mixed path, one element per thread (the FP64 path: k_move_tri)
template <class R> __device__ __forceinline__ void b_k_move_elem(DevClock *__restrict__ C, DevArrays A, GfDims d, int advance_time, GF_IDX e) {
    if (e >= d.E) return;
    int j, i;
    elem_ji(d, e, j, i);
    const double dtd = C->dt;
    QuadF qf;
    float rvx[4], rvy[4];
    load_quad_rel(A, d, j, i, qf);
    load_vel_rel(A, d, j, i, rvx, rvy);
    R *area = (R *)A.area;
    R *dvol = (R *)A.dvol;
    R *st = (R *)A.stress0;
    R *strain = (R *)A.strain;
    // (all loads before the first store: see b_k_rheol)
    R ar0[4], s0[3][4], e0[3];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        ar0[k] = area[gf_ek(d, e, k)];
#pragma unroll
        for (int c = 0; c < 3; ++c) s0[c][k] = st[gf_s(d, e, c, k)];
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) e0[c] = strain[gf_ek(d, e, c)];
    const int nd1[4] = {0, 2, 0, 0}, nd2[4] = {1, 1, 1, 3}, nd3[4] = {2, 3, 3, 2};
    bool neg = false;
    // the surface nodes also moved by diff_topo's dtopo (zero without it)
    float tz[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    if (j == 0) {
        tz[0] = gf_d2f(A.dtopo[i]);
        tz[2] = gf_d2f(A.dtopo[i + 1]);
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        int a = nd1[k], b = nd2[k], c = nd3[k];
        R ar_old = ar0[k];
        R dw12, ar_new;
        {
            // FP32 from edge vectors of the relative coordinates: det = B x C
            // with B = b - a, C = c - a.  dvol = det_new*area_old - 1 is taken
            // as (det_new - det_old)*area_old with the change of det expanded
            // in this step's displacements u = vel*dt, which FP32 resolves.
            const float *x = qf.x, *y = qf.y;
            const float dtf = gf_d2f(dtd);
            float Bx = x[b] - x[a], By = y[b] - y[a];
            float Cx = x[c] - x[a], Cy = y[c] - y[a];
            float dBx = (rvx[b] - rvx[a]) * dtf, dBy = (rvy[b] - rvy[a]) * dtf + (tz[b] - tz[a]);
            float dCx = (rvx[c] - rvx[a]) * dtf, dCy = (rvy[c] - rvy[a]) * dtf + (tz[c] - tz[a]);
            float Box = Bx - dBx, Boy = By - dBy, Cox = Cx - dCx, Coy = Cy - dCy;
            float ddet = (Box * dCy - Boy * dCx) + (dBx * Coy - dBy * Cox) + (dBx * dCy - dBy * dCx);
            float det = Bx * Cy - By * Cx;
            dvol[gf_ek(d, e, k)] = R(ddet * (float)ar_old);
            ar_new = R(1.0f / det);
            // 0.5 * curl of the velocity over the triangle, times dt
            float wx = rvx[a] * (x[c] - x[b]) + rvx[b] * (x[a] - x[c]) + rvx[c] * (x[b] - x[a]);
            float wy = rvy[a] * (y[c] - y[b]) + rvy[b] * (y[a] - y[c]) + rvy[c] * (y[b] - y[a]);
            dw12 = R(0.5f * (wx + wy) / det * dtf);
        }
        area[gf_ek(d, e, k)] = ar_new;
        neg |= !(ar_new > R(0));
        R s11 = s0[0][k], s22 = s0[1][k], s12 = s0[2][k];
        st[gf_s(d, e, 0, k)] = s11 + 2.0f * s12 * dw12;
        st[gf_s(d, e, 1, k)] = s22 - 2.0f * s12 * dw12;
        st[gf_s(d, e, 2, k)] = s12 + dw12 * (s22 - s11);
        if (k == 0) {
            R e11 = e0[0], e22 = e0[1], e12 = e0[2];
            strain[gf_ek(d, e, 0)] = e11 + 2.0f * e12 * dw12;
            strain[gf_ek(d, e, 1)] = e22 - 2.0f * e12 * dw12;
            strain[gf_ek(d, e, 2)] = e12 + dw12 * (e22 - e11);
        }
    }
    if (advance_time && e == 0) C->time = C->time + dtd; // par.f90:86, after every reader of time
    if (neg) set_status(C, 40, (int)e);
}
template <class R> __global__ void __launch_bounds__(GF_THREADS, 3) k_move_elem(DevClock *__restrict__ C, DevArrays A, GfDims d, int advance_time) {
    gf_pdl_entry();
    b_k_move_elem<R>(C, A, d, advance_time, (GF_IDX)blockIdx.x * blockDim.x + threadIdx.x);
}

// ======================================================================
// fl_therm (fl_therm.f90:393-598): the FP64 path in gf_therm64.cuh, the mixed
// path's two sweeps below.
// K index of (a,b), a,b in 0..2 (symmetric)
__device__ __forceinline__ int kidx(int a, int b) {
    int lo = a < b ? a : b, hi = a < b ? b : a;
    return lo == 0 ? hi : (lo == 1 ? 2 + hi : 5);
}

// Temperature after the boundary conditions of fl_therm.f90:573-598 (top
// row t_top, bottom row bot_bc or the flux condition, then the side columns
// copied from their inner neighbours), read from the swept values `src`.
template <class Src>
__device__ __forceinline__ double therm_bc_value(const DevParams &P, const DevArrays &A, const GfDims &d, Src src, int j,
                                                 int i) {
    const int nx = d.nx, nz = d.nz;
    int ii = (i == 0 || nx == 2) ? 1 : (i == nx - 1 ? nx - 2 : i);
    if (j == 0) return P.t_top;
    if (j == nz - 1) {
        if (P.itemp_bc == 1) return P.bot_bc;
        if (P.itemp_bc == 2) {
            int ie = ii < nx - 2 ? ii : nx - 2;
            double cond_eff = P.conduct[A.iphase[gf_elem(d, nz - 2, ie)] - 1];
            return src(gf_node(d, nz - 2, ii)) +
                   P.bot_bc * (A.cord[d.N + gf_node(d, nz - 2, ii)] - A.cord[d.N + gf_node(d, nz - 1, ii)]) / cond_eff;
        }
    }
    return src(gf_node(d, j, ii));
}

// ---- mixed precision: FP32 coefficients, two sweeps.
// The diffusion sum is taken over temperature differences to the updated
// node (the rows of the triangle stiffness sum to zero), so FP32 keeps the
// accuracy that a sum of ~1000 C values would lose.  Sweep 0 is the all-old
// (Jacobi) update, sweep 1 reuses the upstream increments of sweep 0, which
// leaves an error of order (kappa dt/h^2)^2 relative to the increment.
//
// The coefficients are kept per node: the weights of its six neighbours
// (sums over the node's six triangles) and the heat term, each over the node's
// area sum.  A sweep then reads 7 values a node instead of some 30 of four
// elements' 18; the prep, which does each triangle's products for its three
// nodes, runs beside fl_rheol or at full occupancy.  A step of 60x20 elements
// 29.4 -> 27.6 us, of 64 ensemble members 511 -> 468 us; 1000x300 elements
// unchanged (what the sweeps save the prep takes); the increments' error
// against FP64 is no larger (3.1e-7 to 6.5e-7 of them).
#define GF_TN 7
// offsets of the neighbours (j-1,i), (j,i-1), (j+1,i-1), (j-1,i+1), (j,i+1), (j+1,i): upstream ones first
__device__ __forceinline__ void therm_neighbours(const GfDims &d, int j, int i, GF_IDX n, GF_IDX m[6]) {
    const bool up = j != 0, dn = j != d.nz - 1, lf = i != 0, rt = i != d.nx - 1;
    m[0] = up ? n - 1 : n;
    m[1] = lf ? n - d.nz : n;
    m[2] = lf && dn ? n - d.nz + 1 : n;
    m[3] = up && rt ? n + d.nz - 1 : n;
    m[4] = rt ? n + d.nz : n;
    m[5] = dn ? n + 1 : n;
}
__device__ __forceinline__ void b_k_therm_prep32(const DevParams *__restrict__ Pp, DevArrays A, GfDims d, float *__restrict__ tc, GF_IDX n) {
    if (n >= d.N) return;
    const DevParams &P = *Pp;
    int j, i;
    node_ji(d, n, j, i);
    GF_IDX m[6];
    therm_neighbours(d, j, i, n, m);
    const float *xh = A.cord_hi, *xl = A.cord_lo, *yh = A.cord_hi + d.N, *yl = A.cord_lo + d.N;
    float x[6], y[6], w[6] = {0, 0, 0, 0, 0, 0};
#pragma unroll
    for (int q = 0; q < 6; ++q) {
        x[q] = hl_diff(xh, xl, m[q], n);
        y[q] = hl_diff(yh, yl, m[q], n);
    }
    const float *area = (const float *)A.area, *shrheat = (const float *)A.shrheat;
    float s = 0.0f, area_n = 0.0f;
    // the triangle (self, p, q) of neighbours p and q in the element's
    // orientation, area factor a, from the element's diffusivity and source
    auto tri = [&](float a, float diff, float src, int p, int q) {
        const float ds = (y[p] - y[q]) * a, dp = y[q] * a, dq = -y[p] * a;
        const float zs = (x[q] - x[p]) * a, zp = -x[q] * a, zq = x[p] * a;
        const float inv_area = 1.0f / a, ra = inv_area / 6.0f, pre = 0.5f * diff * inv_area;
        area_n += ra;
        s += src * ra;
        w[p] -= pre * (dp * ds + zp * zs);
        w[q] -= pre * (dq * ds + zq * zs);
    };
    auto elem = [&](int je, int ie, float &diff, float &src) {
        const GF_IDX e = gf_elem(d, je, ie);
        const int iph = A.iphase[e] - 1;
        const float cp = P.f_cp[iph], den = P.f_den[iph];
        const float dissip = (P.ishearh == 1 && P.itherm != 2) ? shrheat[e] : 0.0f;
        diff = P.f_cond[iph] / den / cp;
        src = (gf_d2f(A.source[e]) + dissip / den) / cp;
        return e;
    };
    // triangles A = (1,2,3) and B = (3,2,4) of the quad's nodes (j,i), (j+1,i), (j,i+1), (j+1,i+1)
    float diff, src;
    if (j != 0 && i != 0) { // self is node 4: B, (self, 3, 2)
        const GF_IDX e = elem(j - 1, i - 1, diff, src);
        tri(area[gf_ek(d, e, 1)], diff, src, 0, 1);
    }
    if (j != 0 && i != d.nx - 1) { // self is node 2: A, (self, 3, 1), and B, (self, 4, 3)
        const GF_IDX e = elem(j - 1, i, diff, src);
        tri(area[gf_ek(d, e, 0)], diff, src, 3, 0);
        tri(area[gf_ek(d, e, 1)], diff, src, 4, 3);
    }
    if (j != d.nz - 1 && i != 0) { // self is node 3: A, (self, 1, 2), and B, (self, 2, 4)
        const GF_IDX e = elem(j, i - 1, diff, src);
        tri(area[gf_ek(d, e, 0)], diff, src, 1, 2);
        tri(area[gf_ek(d, e, 1)], diff, src, 2, 5);
    }
    if (j != d.nz - 1 && i != d.nx - 1) { // self is node 1: A, (self, 2, 3)
        const GF_IDX e = elem(j, i, diff, src);
        tri(area[gf_ek(d, e, 0)], diff, src, 5, 4);
    }
    const float r = 1.0f / area_n;
#pragma unroll
    for (int q = 0; q < 6; ++q) tc[q * d.N + n] = w[q] * r;
    tc[6 * d.N + n] = s * r;
}
__global__ void __launch_bounds__(GF_THREADS) k_therm_prep32(const DevParams *__restrict__ Pp, DevArrays A, GfDims d, float *__restrict__ tc) {
    gf_pdl_entry();
    b_k_therm_prep32(Pp, A, d, tc, (GF_IDX)blockIdx.x * blockDim.x + threadIdx.x);
}

// sweep 0 (final = 0): dT0 = increment with old values; sweep 1 (final = 1):
// upstream neighbours use T + dT0, and tnew = T + dT1 (FP64) is written.
// The temperature differences come from the hi/lo FP32 split of T.
__device__ __forceinline__ void b_k_therm_sweep32(const DevParams *__restrict__ Pp, DevClock *__restrict__ C, DevArrays A, GfDims d, const float *__restrict__ tc, float *__restrict__ d0, double *__restrict__ tnew, int final_sweep, GF_IDX n) {
    if (n >= d.N) return;
    int j, i;
    node_ji(d, n, j, i);
    GF_IDX m[6];
    therm_neighbours(d, j, i, n, m);
    const float *th = A.temp_hi, *tl = A.temp_lo;
    float w[6], t[6], inc = tc[6 * d.N + n];
#pragma unroll
    for (int q = 0; q < 6; ++q) {
        w[q] = tc[q * d.N + n];
        t[q] = hl_diff(th, tl, m[q], n);
        if (q < 3 && final_sweep) t[q] += d0[m[q]]; // upstream nodes carry sweep 0's increment
    }
#pragma unroll
    for (int q = 0; q < 6; ++q) inc += w[q] * t[q];
    inc *= gf_d2f(C->dt);
    if (!final_sweep)
        d0[n] = inc;
    else
        tnew[n] = A.temp[n] + gf_f2d(inc);
}
__global__ void __launch_bounds__(GF_THREADS) k_therm_sweep32(const DevParams *__restrict__ Pp, DevClock *__restrict__ C, DevArrays A, GfDims d, const float *__restrict__ tc, float *__restrict__ d0, double *__restrict__ tnew, int final_sweep) {
    gf_pdl_entry();
    b_k_therm_sweep32(Pp, C, A, d, tc, d0, tnew, final_sweep, (GF_IDX)blockIdx.x * blockDim.x + threadIdx.x);
}

// temp0 = temp; temp = tnew with the boundary conditions (which read tnew
// at neighbours, never the temp being overwritten), and its split
__device__ __forceinline__ void b_k_therm_apply32(const DevParams *__restrict__ Pp, DevArrays A, GfDims d, const double *__restrict__ tnew, GF_IDX n) {
    if (n >= d.N) return;
    int j, i;
    node_ji(d, n, j, i);
    const double t = therm_bc_value(*Pp, A, d, [tnew](GF_IDX m) { return tnew[m]; }, j, i);
    A.temp0[n] = A.temp[n];
    A.temp[n] = t;
    float h, l;
    gf_split(t, h, l);
    A.temp_hi[n] = h;
    A.temp_lo[n] = l;
}
__global__ void __launch_bounds__(GF_THREADS) k_therm_apply32(const DevParams *__restrict__ Pp, DevArrays A, GfDims d, const double *__restrict__ tnew) {
    gf_pdl_entry();
    b_k_therm_apply32(Pp, A, d, tnew, (GF_IDX)blockIdx.x * blockDim.x + threadIdx.x);
}

// ---- mixed precision: the ordinary step in four phases.
// On steps where fl_rheol and fl_node read nothing that the thermal update
// writes (no viscosity update, no change_phase, no thermal stress, no Winkler
// foundation, whose pressure reads the new temperatures) the thermal update
// shares launches with the mechanics:
//   a: fl_rheol             beside the sweep coefficients (from the shear
//                             heating before fl_rheol's averaging rewrites it)
//   b: fl_node              beside sweep 0 and fl_rheol's averaging
//   c: the coordinates      beside sweep 1 (the sweeps read no coordinates)
//   d: fl_move's elements   beside the temperatures' boundary conditions
// so a step is four dependent launches.  Blocks of one launch take one part
// each (grid y), the longer part first: in one thread after another the
// parts' memory latencies add up (no load moves above the stores of the part
// before), which costs more than the launches saved.
// (registers as for k_rheol; d: 80 registers for 3 CTAs, 95.4 against 97.5 us
// a step of 1000x300 elements at the 106 it takes uncapped)
__global__ void __launch_bounds__(GF_THREADS, 2) k_step_a(const DevParams *__restrict__ Pp, DevClock *__restrict__ C, DevArrays A, GfDims d) {
    gf_pdl_entry();
    const GF_IDX e = (GF_IDX)blockIdx.x * blockDim.x + threadIdx.x;
    if (blockIdx.y == 0)
        b_k_rheol<float>(Pp, C, A, d, 0, 0, e);
    else
        b_k_therm_prep32(Pp, A, d, (float *)A.t_coef, e);
}
__global__ void __launch_bounds__(GF_THREADS) k_step_b(const DevParams *__restrict__ Pp, DevClock *__restrict__ C, DevArrays A, GfDims d, int avg_mode) {
    gf_pdl_entry();
    const GF_IDX n = (GF_IDX)blockIdx.x * blockDim.x + threadIdx.x;
    if (blockIdx.y == 0)
        b_k_node<float>(Pp, C, A, d, n);
    else if (blockIdx.y == 1)
        b_k_therm_sweep32(Pp, C, A, d, (const float *)A.t_coef, (float *)A.t_delta0, A.t_delta1, 0, n);
    else
        b_k_rheol_avg<float>(C, A, d, avg_mode == 2 ? 1 : 0, n);
}
__global__ void __launch_bounds__(GF_THREADS) k_step_c(const DevParams *__restrict__ Pp, DevClock *__restrict__ C, DevArrays A, GfDims d, int avg_mode) {
    gf_pdl_entry();
    const GF_IDX n = (GF_IDX)blockIdx.x * blockDim.x + threadIdx.x;
    if (blockIdx.y == 0) {
        b_k_therm_sweep32(Pp, C, A, d, (const float *)A.t_coef, (float *)A.t_delta0, A.t_delta1, 1, n);
        if (avg_mode == 2 && n == 0) b_k_rheol_clock(C, 1);
    } else if (n < d.N) {
        b_k_move_cord(C, A, d, (GF_IDX)(blockIdx.y - 1) * d.N + n);
    }
}
__global__ void __launch_bounds__(GF_THREADS, 3) k_step_d(const DevParams *__restrict__ Pp, DevClock *__restrict__ C, DevArrays A, GfDims d, int advance_time) {
    gf_pdl_entry();
    const GF_IDX n = (GF_IDX)blockIdx.x * blockDim.x + threadIdx.x;
    if (blockIdx.y == 0)
        b_k_move_elem<float>(C, A, d, advance_time, n);
    else
        b_k_therm_apply32(Pp, A, d, A.t_delta1, n);
}

// ======================================================================
// rmasses (rmasses.f90:4-63): per-element density, then a node gather in
// the reference's colour order with each element's triangles in order.
template <class R, bool I = false> __device__ __forceinline__ void b_k_elem_dens(const DevParams *__restrict__ Pp, DevClock *__restrict__ C, DevArrays A, GfDims d, GF_IDX e) {
    if (e >= d.E) return;
    int j, i;
    elem_ji(d, e, j, i);
    int wrote = 0;
    const R *area = (const R *)A.area;
    if constexpr (sizeof(R) == sizeof(float)) {
        // mixed: FP32 density and FP32 triangle shares
        float fval = 0.0f;
        const float dens = eff_dens_f32(*Pp, A, d, j, i, e, &wrote, &fval);
        A.e_dens[e] = gf_f2d(dens);
        float *tri = (float *)A.e_tri;
#pragma unroll
        for (int k = 0; k < 4; ++k) tri[k * d.E + e] = (1.0f / 12.0f) / area[gf_ek(d, e, k)] * dens;
    } else {
        double fval = 0.0;
        double dens = eff_dens<R, I>(*Pp, A, d, j, i, e, &wrote, &fval);
        A.e_dens[e] = dens;
        // each triangle's share c1d12/area*dens (rmasses.f90:35-57),
        // computed once here with the reference's operations and gathered
        // per node
        const double c1d12 = 1.0 / 12.0;
#pragma unroll
        for (int k = 0; k < 4; ++k) A.e_tri[k * d.E + e] = gf_mulc<I>(gf_divc<I>(c1d12, (double)area[gf_ek(d, e, k)]), dens);
    }
    if (wrote) {
        // serial position of this element in the coloured sweep
        int ib = i & 1, jb = j & 1;
        GF_IDX ci = (GF_IDX)(d.nx - 1 - ib + 1) / 2; // columns of this colour
        GF_IDX cj = (GF_IDX)(d.nz - 1 - jb + 1) / 2;
        GF_IDX before = 0;
        for (int b = 0; b < ib * 2 + jb; ++b) {
            int bi = b >> 1, bj = b & 1;
            before += (GF_IDX)((d.nx - 1 - bi + 1) / 2) * ((d.nz - 1 - bj + 1) / 2);
        }
        GF_IDX pos = before + (GF_IDX)(i >> 1) * cj + (j >> 1);
        (void)ci;
        atomicMax((unsigned long long *)&C->frac_writer, (unsigned long long)(pos + 1));
    }
}
template <class R, bool I = false> __global__ void __launch_bounds__(GF_THREADS) k_elem_dens(const DevParams *__restrict__ Pp, DevClock *__restrict__ C, DevArrays A, GfDims d) {
    gf_pdl_entry();
    b_k_elem_dens<R, I>(Pp, C, A, d, (GF_IDX)blockIdx.x * blockDim.x + threadIdx.x);
}

template <class R> __device__ __forceinline__ void b_k_frac_fix(const DevParams *__restrict__ Pp, DevClock *__restrict__ C, DevArrays A, GfDims d) {
    long long w = C->frac_writer;
    if (w <= 0) return;
    GF_IDX pos = w - 1;
    for (int b = 0; b < 4; ++b) {
        int bi = b >> 1, bj = b & 1;
        GF_IDX ci = (d.nx - 1 - bi + 1) / 2, cj = (d.nz - 1 - bj + 1) / 2;
        if (pos < ci * cj) {
            int i = (int)(pos / cj) * 2 + bi, j = (int)(pos % cj) * 2 + bj;
            int wrote = 0;
            double f = 0.0;
            eff_dens<R>(*Pp, A, d, j, i, gf_elem(d, j, i), &wrote, &f);
            if (wrote) C->frac = f;
            break;
        }
        pos -= ci * cj;
    }
    C->frac_writer = 0;
}
template <class R> __global__ void k_frac_fix(const DevParams *__restrict__ Pp, DevClock *__restrict__ C, DevArrays A, GfDims d) {
    b_k_frac_fix<R>(Pp, C, A, d);
}

// Contribution lists: for local vertex v of a quad (1:(j,i) 2:(j+1,i)
// 3:(j,i+1) 4:(j+1,i+1)), the triangles that contain it, in order.
__device__ __constant__ int c_vtx_tris[4][3] = {{0, 2, 3}, {0, 1, 2}, {0, 1, 3}, {1, 2, 3}};

// Node gather of per-triangle shares tri[k*E + e] in the reference's order:
// adjacent elements by colour ((ie&1)*2 + (je&1), rmasses.f90:25-30,
// dt_mass.f90:74-81), then each element's triangles containing the node in
// the order A, B, C, D.  Every element in a node's neighbourhood has a
// different colour, so this is the serial order of the coloured scatter.
// T = double: FP64 shares summed in the reference's order; T = float: the
// mixed path's FP32 shares
template <class T>
__device__ __forceinline__ void b_k_node_gather_tri(const T *__restrict__ tri, double *__restrict__ out, GfDims d, GF_IDX n) {
    if (n >= d.N) return;
    int j, i;
    node_ji(d, n, j, i);
    T acc = T(0);
    int ord[4];
    // the node is vertex 4 of quad (j-1,i-1), 2 of (j-1,i), 3 of (j,i-1), 1 of (j,i)
    int je_[4] = {j - 1, j - 1, j, j}, ie_[4] = {i - 1, i, i - 1, i}, lv[4] = {3, 1, 2, 0};
#pragma unroll
    for (int q = 0; q < 4; ++q) ord[q] = ((ie_[q] & 1) << 1) | (je_[q] & 1);
#pragma unroll
    for (int c = 0; c < 4; ++c)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            if (ord[q] != c) continue;
            int je = je_[q], ie = ie_[q];
            if (je < 0 || ie < 0 || je > d.nz - 2 || ie > d.nx - 2) continue;
            GF_IDX e = gf_elem(d, je, ie);
#pragma unroll
            for (int t = 0; t < 3; ++t) acc = acc + tri[c_vtx_tris[lv[q]][t] * d.E + e];
        }
    if constexpr (sizeof(T) == sizeof(float)) out[n] = gf_f2d(acc);
    else out[n] = acc;
}
template <class T>
__global__ void __launch_bounds__(GF_THREADS) k_node_gather_tri(const T *__restrict__ tri, double *__restrict__ out, GfDims d) {
    gf_pdl_entry();
    b_k_node_gather_tri<T>(tri, out, d, (GF_IDX)blockIdx.x * blockDim.x + threadIdx.x);
}

// ======================================================================
// dt_mass (dt_mass.f90:16-232)
// The CTA's minimum edge measure, maximum |velocity|, maximum diffusivity
// and phase mask (each warp's already reduced in its lane 0) combined in
// shared memory, then one atomic per quantity and CTA (per-warp atomics on
// the same four words serialise).  min / max are exact in any order.  Every
// thread of the CTA calls it; `diffu` (mixed path) turns the phase mask into
// the maximum diffusivity, otherwise dmax is used.
__device__ __forceinline__ void dt_block_commit(DevClock *__restrict__ C, double dl, double vmax, double dmax,
                                                unsigned pm, const double *diffu, int nphase) {
    __shared__ unsigned long long s_dl[GF_THREADS_MAX / 32], s_v[GF_THREADS_MAX / 32], s_d[GF_THREADS_MAX / 32];
    __shared__ unsigned s_pm[GF_THREADS_MAX / 32];
    const int w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
    if ((threadIdx.x & 31) == 0) {
        s_dl[w] = (unsigned long long)__double_as_longlong(dl);
        s_v[w] = (unsigned long long)__double_as_longlong(vmax);
        s_d[w] = (unsigned long long)__double_as_longlong(dmax);
        s_pm[w] = pm;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long a = s_dl[0], b = s_v[0], c = s_d[0];
        unsigned m = s_pm[0];
        for (int k = 1; k < nw; ++k) {
            a = min(a, s_dl[k]);
            b = max(b, s_v[k]);
            c = max(c, s_d[k]);
            m |= s_pm[k];
        }
        if (diffu) { // the largest diffusivity of the phases present (dt_mass.f90:130)
            double dm = 0.0;
            for (int k = 0; k < nphase; ++k)
                if (m & (1u << k)) dm = fmax(dm, diffu[k]);
            c = (unsigned long long)__double_as_longlong(dm);
        }
        atomicMin(&C->r_dlmin, a);
        atomicMax(&C->r_velmax, b);
        atomicMax(&C->r_diffmax, c);
        atomicOr(&C->phase_mask, m);
    }
    __syncthreads(); // the shared slots are free for the CTA's next item
}

template <class R, bool I = false> __device__ __forceinline__ void b_k_dt_reduce(const DevParams *__restrict__ Pp, DevClock *__restrict__ C, DevArrays A, GfDims d, GF_IDX t) {
    const DevParams &P = *Pp;
    double dl = 1e300, vmax = 0.0, dmax = 0.0;
    unsigned pm = 0;
    if constexpr (sizeof(R) == sizeof(float)) {
        // mixed: edge lengths and 1/(area*length) in FP32 from the hi/lo
        // coordinates, |vel| from the hi parts; the warp minima and maxima of
        // these FP32 values convert to FP64 exactly, and the minimum over
        // elements is taken on their FP64 values
        float df = 1e30f, vf = 0.0f;
        if (t < d.E) {
            GF_IDX e = t;
            int j, i;
            elem_ji(d, e, j, i);
            const float *area = (const float *)A.area;
            QuadF q;
            load_quad_rel(A, d, j, i, q);
            auto len = [&](int a, int b) {
                float ddx = q.x[a] - q.x[b], ddy = q.y[a] - q.y[b];
                return sqrtf(ddx * ddx + ddy * ddy);
            };
            float a0 = area[gf_ek(d, e, 0)], a1 = area[gf_ek(d, e, 1)], a2 = area[gf_ek(d, e, 2)],
                  a3 = area[gf_ek(d, e, 3)];
            float l;
            l = len(1, 0); df = fminf(df, 1.0f / (a0 * l)); df = fminf(df, 1.0f / (a2 * l));
            l = len(3, 1); df = fminf(df, 1.0f / (a1 * l)); df = fminf(df, 1.0f / (a2 * l));
            l = len(3, 2); df = fminf(df, 1.0f / (a1 * l)); df = fminf(df, 1.0f / (a3 * l));
            l = len(2, 0); df = fminf(df, 1.0f / (a0 * l)); df = fminf(df, 1.0f / (a3 * l));
            l = len(3, 0); df = fminf(df, 1.0f / (a2 * l)); df = fminf(df, 1.0f / (a3 * l));
            l = len(1, 2); df = fminf(df, 1.0f / (a0 * l)); df = fminf(df, 1.0f / (a1 * l));
            pm = 1u << (A.iphase[e] - 1);
        }
        if (t < d.N) vf = fmaxf(fabsf(A.vel_hi[t]), fabsf(A.vel_hi[d.N + t]));
        df = warp_min(df);
        vf = warp_max(vf);
        for (int o = 16; o > 0; o >>= 1) pm |= __shfl_xor_sync(0xffffffffu, pm, o);
        dt_block_commit(C, df < 1e30f ? gf_f2d(df) : 1e300, gf_f2d(vf), 0.0, pm, P.diffu, P.nphase);
        return;
    } else {
        if (t < d.E) {
            GF_IDX e = t;
            int j, i;
            elem_ji(d, e, j, i);
            const R *area = (const R *)A.area;
            Quad q;
            load_quad(A.cord, d, j, i, q);
            // (squares, products, comparisons and quotients on the integer
            // pipes; the six roots and their sums stay on the FP64 pipe)
            auto len = [&](int a, int b) {
                double ddx = q.x[a] - q.x[b], ddy = q.y[a] - q.y[b];
                return sqrt(gf_mulc<I>(ddx, ddx) + gf_mulc<I>(ddy, ddy));
            };
            double a0 = (double)area[gf_ek(d, e, 0)], a1 = (double)area[gf_ek(d, e, 1)],
                   a2 = (double)area[gf_ek(d, e, 2)], a3 = (double)area[gf_ek(d, e, 3)];
            // the smallest of the twelve quotients 1/(area*length) of
            // dlmin_prop (dt_mass.f90:174-231) is the quotient of the largest
            // product: correctly rounded division is monotone, so
            // min fl(1/x_k) = fl(1/max x_k) exactly, for one division.  The
            // largest of 0 and the products, by their bits: negative numbers
            // and NaNs, whose bits lie above infinity's, count for nothing
            unsigned long long xm = 0ull;
            auto top = [&](double ar, double l) {
                const unsigned long long u = (unsigned long long)__double_as_longlong(gf_mulc<I>(ar, l));
                if (u <= 0x7ff0000000000000ull && u > xm) xm = u;
            };
            double l;
            l = len(1, 0); top(a0, l); top(a2, l);
            l = len(3, 1); top(a1, l); top(a2, l);
            l = len(3, 2); top(a1, l); top(a3, l);
            l = len(2, 0); top(a0, l); top(a3, l);
            l = len(3, 0); top(a2, l); top(a3, l);
            l = len(1, 2); top(a0, l); top(a1, l);
            dl = fmin(dl, gf_divc<I>(1.0, __longlong_as_double((long long)xm)));
            int iph = A.iphase[e] - 1;
            dmax = gf_divc<I>(gf_divc<I>(P.conduct[iph], P.den[iph]), P.cp[iph]);
            pm = 1u << iph;
        }
        if (t < d.N) vmax = fmax(fabs(A.vel[t]), fabs(A.vel[d.N + t]));
        dl = warp_min(dl);
        vmax = warp_max(vmax);
        dmax = warp_max(dmax);
        for (int o = 16; o > 0; o >>= 1) pm |= __shfl_xor_sync(0xffffffffu, pm, o);
        dt_block_commit(C, dl, vmax, dmax, pm, nullptr, 0);
    }
}
template <class R, bool I = false> __global__ void __launch_bounds__(GF_THREADS) k_dt_reduce(const DevParams *__restrict__ Pp, DevClock *__restrict__ C, DevArrays A, GfDims d) {
    gf_pdl_entry();
    b_k_dt_reduce<R, I>(Pp, C, A, d, (GF_IDX)blockIdx.x * blockDim.x + threadIdx.x);
}

__device__ __forceinline__ void b_k_dt_scalars(const DevParams *__restrict__ Pp, DevClock *__restrict__ C) {
    const DevParams &P = *Pp;
    double dlmin = fmin(1e28, __longlong_as_double((long long)C->r_dlmin));
    double vel_max = __longlong_as_double((long long)C->r_velmax);
    double diffmax = __longlong_as_double((long long)C->r_diffmax);
    C->dlmin = dlmin;
    C->vel_max = vel_max;
    if (P.idt_scale == 1)
        C->dt_elastic = P.dt_scale;
    else if (P.idt_scale == 2) {
        if (P.vbc == 0)
            C->dt_elastic = dlmin * C->frac * P.strain_inert / (1.0 / GF_SEC_YEAR / 100);
        else
            C->dt_elastic = dlmin * C->frac * P.strain_inert / P.vbc;
    }
    // min over elements of dlmin^2/diff == dlmin^2 / max(diff) (rounded
    // division is monotone in the divisor)
    double dtmax_therm = 1e28;
    if (diffmax > 0.0) dtmax_therm = fmin(dtmax_therm, dlmin * dlmin / diffmax);
    double dt_maxwell = 1e28;
    double dt_elastic = C->dt_elastic;
    unsigned pm = C->phase_mask;
    for (int k = 0; k < P.nphase; ++k) {
        if (!(pm & (1u << k))) continue;
        if (P.idt_scale == 0) {
            // dt_mass.f90:122-126: a running minimum that starts from the
            // previous dt_elastic
            double pwave = P.rl[k] + 0.6666 * P.rm[k];
            double dte = C->frac * dlmin * sqrt(P.den[k] / pwave);
            dt_elastic = fmin(dt_elastic, dte);
        }
        if (P.ivis_present == 1 && (P.irheol[k] == 3 || P.irheol[k] == 12) && P.rm[k] < 1e11) {
            double visc_cut = 1e10;
            double rmu = (P.v_min < visc_cut) ? P.rm[k] * P.v_min / visc_cut : P.rm[k];
            double dt_m = P.v_min / rmu * P.fracm;
            dt_maxwell = fmin(dt_m, dt_maxwell);
        }
    }
    C->dt_elastic = dt_elastic;
    C->dt_maxwell = dt_maxwell;
    C->dtmax_therm = dtmax_therm;
    C->dt = fmin(fmin(dt_elastic, dt_maxwell), dtmax_therm);
}
__global__ void k_dt_scalars(const DevParams *__restrict__ Pp, DevClock *__restrict__ C) {
    b_k_dt_scalars(Pp, C);
}

// inertial mass share of each triangle c1d12*rho_inert/area
// (dt_mass.f90:83-120), one element per thread
template <class R, bool I = false> __device__ __forceinline__ void b_k_elem_am3(const DevParams *__restrict__ Pp, DevClock *__restrict__ C, DevArrays A, GfDims d, GF_IDX e) {
    if (e >= d.E) return;
    const DevParams &P = *Pp;
    const R *area = (const R *)A.area;
    if constexpr (sizeof(R) == sizeof(float)) {
        // mixed: the inertial density in FP32 (pwave / vel_sound^2 ~ 1e21,
        // well inside the FP32 range), from FP32 copies of the inputs
        const int iph = A.iphase[e] - 1;
        const float pwave = gf_d2f(P.rl[iph]) + 0.6666f * P.f_rm[iph];
        const float vel_sound = gf_d2f(C->dlmin) * gf_d2f(C->frac) / gf_d2f(C->dt_elastic);
        float rho_inert = pwave / (vel_sound * vel_sound);
        const float vel_max = gf_d2f(C->vel_max);
        if (P.i_rey == 1 && vel_max > 0.0f) {
            const float rho_inert2 = (gf_d2f(P.xReyn) * gf_d2f(P.v_min)) / (vel_max * fabsf(gf_d2f(P.rzbo)));
            if (rho_inert > rho_inert2) rho_inert = rho_inert2;
        }
        const float r = rho_inert / 12.0f;
        float *tri = (float *)A.e_tri;
#pragma unroll
        for (int k = 0; k < 4; ++k) tri[k * d.E + e] = r / area[gf_ek(d, e, k)];
        return;
    }
    const double c1d12 = 1.0 / 12.0;
    double dlmin = C->dlmin, frac = C->frac, dt_elastic = C->dt_elastic, vel_max = C->vel_max;
    int iph = A.iphase[e] - 1;
    double pwave = P.rl[iph] + 0.6666 * P.rm[iph];
    double vel_sound = gf_divc<I>(gf_mulc<I>(dlmin, frac), dt_elastic);
    double rho_inert = gf_divc<I>(pwave, gf_mulc<I>(vel_sound, vel_sound));
    if (P.i_rey == 1 && vel_max > 0.0) {
        double rho_inert2 = (P.xReyn * P.v_min) / (vel_max * fabs(P.rzbo));
        if (rho_inert > rho_inert2) rho_inert = rho_inert2;
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) A.e_tri[k * d.E + e] = gf_divc<I>(gf_mulc<I>(c1d12, rho_inert), (double)area[gf_ek(d, e, k)]);
}
template <class R, bool I = false> __global__ void __launch_bounds__(GF_THREADS) k_elem_am3(const DevParams *__restrict__ Pp, DevClock *__restrict__ C, DevArrays A, GfDims d) {
    gf_pdl_entry();
    b_k_elem_am3<R, I>(Pp, C, A, d, (GF_IDX)blockIdx.x * blockDim.x + threadIdx.x);
}

__device__ __forceinline__ void b_k_dt_reset(DevClock *C) {
    C->r_dlmin = (unsigned long long)__double_as_longlong(1e300);
    C->r_velmax = 0ull;
    C->r_diffmax = 0ull;
    C->phase_mask = 0u;
}
__global__ void k_dt_reset(DevClock *C) {
    b_k_dt_reset(C);
}

// ======================================================================
// init_visc
template <class R> __device__ __forceinline__ void b_k_init_visc(const DevParams *__restrict__ Pp, DevArrays A, GfDims d, GF_IDX e) {
    if (e >= d.E) return;
    int j, i;
    elem_ji(d, e, j, i);
    ((R *)A.visn)[e] = R(visc_of<R>(*Pp, A, d, j, i, e, (const R *)A.stress0));
}
template <class R> __global__ void __launch_bounds__(GF_THREADS) k_init_visc(const DevParams *__restrict__ Pp, DevArrays A, GfDims d) {
    gf_pdl_entry();
    b_k_init_visc<R>(Pp, A, d, (GF_IDX)blockIdx.x * blockDim.x + threadIdx.x);
}

// ======================================================================
// change_phase (change_phase.f90:35-262)
__device__ __forceinline__ void b_k_phase_markers(const DevParams *__restrict__ Pp, DevArrays A, GfDims d, int nmarkers, GF_IDX kk) {
    if (kk >= nmarkers) return;
    if (A.mark_dead[kk] == 0) return;
    const DevParams &P = *Pp;
    const int nz = d.nz;
    int n = A.mark_ntriag[kk];
    int k = (n - 1) % 2 + 1;
    int j = ((n - k) / 2) % (nz - 1);
    int i = (n - k) / 2 / (nz - 1);
    // Exclusions that change no output, ahead of the FP64 evaluation: a
    // phase without a rule, and a marker certainly deeper than its rule
    // reaches (below 200 km; 150 km for mantle phases 4 and 8).  The marker
    // lies in its triangle, so its depth is at least the surface height less
    // the highest corner; FP32 copies of those heights err by under 0.1 m
    // and the test keeps a 10 m margin.
    GF_IDX p1, p2, p3;
    if (k == 1) {
        p1 = gf_node(d, j, i); p2 = gf_node(d, j + 1, i); p3 = gf_node(d, j, i + 1);
    } else {
        p1 = gf_node(d, j, i + 1); p2 = gf_node(d, j + 1, i); p3 = gf_node(d, j + 1, i + 1);
    }
    {
        const int ph = A.mark_phase[kk];
        if (!(ph == 4 || ph == 8 || ph == 10 || ph == 3 || ph == 7 || ph == 9 || ph == 1 || ph == 11 || ph == 17 ||
              ph == 5 || ph == 16))
            return;
        const double *zc = A.cord + d.N;
        const GF_IDX q1 = gf_node(d, j, i), q3 = gf_node(d, j, i + 1);
        float zmax = fmaxf(fmaxf(gf_d2f(zc[q1]), gf_d2f(zc[q1 + 1])), fmaxf(gf_d2f(zc[q3]), gf_d2f(zc[q3 + 1])));
        const float surf = 0.5f * (gf_d2f(zc[gf_node(d, 0, i)]) + gf_d2f(zc[gf_node(d, 0, i + 1)]));
        const float lim = (ph == 4 || ph == 8) ? 150e3f : 200e3f;
        if (surf - zmax > lim + 10.0f) return;
        if (ph == 4 || ph == 8) {
            // A mantle marker whose rule certainly does nothing (outside the
            // serpentine window and below the solidus), in FP32: for heights
            // below 1e6 m and temperatures below 1e4 the depth errs by under
            // 1 m and the temperature by under 0.01; the margins are 10 m and
            // 0.5 degrees, and their effect on the pressures.  (The FP64
            // rules of 7.5 million markers: 254 us, now about 110.)
            const float a1 = gf_d2f(A.mark_a1[kk]), a2 = gf_d2f(A.mark_a2[kk]), a3 = 1.0f - a1 - a2;
            const float z1 = gf_d2f(zc[p1]), z2 = gf_d2f(zc[p2]), z3 = gf_d2f(zc[p3]);
            const float t1 = gf_d2f(A.temp[p1]), t2 = gf_d2f(A.temp[p2]), t3 = gf_d2f(A.temp[p3]);
            const float depth = surf - (z1 * a1 + z2 * a2 + z3 * a3), t = t1 * a1 + t2 * a2 + t3 * a3;
            const float rho_g = 3000.0f * P.f_g, press = rho_g * depth, m = fabsf(rho_g) * 10.0f + 1.2e7f;
            const float pg = fabsf(press) * 1e-9f;
            const bool small = fabsf(z1) + fabsf(z2) + fabsf(z3) + fabsf(surf) < 1e6f &&
                               fabsf(t1) + fabsf(t2) + fabsf(t3) < 1e4f && fabsf(a1) + fabsf(a2) < 2.0f &&
                               fabsf(rho_g) < 1e5f;
            const bool no_window = press > 2.1e9f - 2.3478261e7f * (t - 730.0f) + m || press < 2.1e9f + 2.5e7f * (t - 730.0f) - m;
            if (small && no_window && t < -5.02f * (pg * pg) + 132.0f * pg + 1160.0f - 0.5f) return;
        }
    }
    double a1 = A.mark_a1[kk], a2 = A.mark_a2[kk];
    const double *cord = A.cord, *T = A.temp;
    double yy, tmpr;
    yy = cord[d.N + p1] * a1 + cord[d.N + p2] * a2 + cord[d.N + p3] * (1 - a1 - a2);
    tmpr = T[p1] * a1 + T[p2] * a2 + T[p3] * (1 - a1 - a2);
    double depth = 0.5 * (cord[d.N + gf_node(d, 0, i)] + cord[d.N + gf_node(d, 0, i + 1)]) - yy;
    if (depth > 200e3) return;
    int iph = A.mark_phase[kk];
    GF_IDX e = gf_elem(d, j, i);
    const double mantle_density = 3000.0;
    GF_IDX total = (GF_IDX)P.nphase * d.E;
    auto pr = [&](GF_IDX eb, int ph1) {
        GF_IDX off = (GF_IDX)(ph1 - 1) + (GF_IDX)P.nphase * eb;
        return (off < 0 || off >= total) ? 0.0 : A.phase_ratio[off];
    };
    int newph = 0;
    switch (iph) {
    case 4: case 8: {
        if (depth > 150e3) break;
        // the reference's expressions, each evaluated only when its branch
        // needs it (the second pressure only below the first, the solidus
        // only outside the serpentine window)
        double press = mantle_density * P.g * depth;
        double trpres = 2.1e9 + (7.5e9 - 2.1e9) * (tmpr - 730.0) / (500.0 - 730.0);
        bool serp_window = false;
        if (press < trpres) {
            double trpres2 = 2.1e9 + (0.6e9 - 2.1e9) * (tmpr - 730.0) / (670.0 - 730.0);
            serp_window = press > trpres2;
        }
        if (serp_window) {
            int jb0 = min(j + 2, nz - 1), jb1 = min(j + 1 + P.nelem_serp, nz - 1);
            for (int jb = jb0; jb <= jb1; ++jb) {
                GF_IDX eb = gf_elem(d, jb - 1, i);
                if (pr(eb, 3) > 0.8 || pr(eb, 7) > 0.8 || pr(eb, 1) > 0.8 || pr(eb, 11) > 0.8) {
                    newph = 9;
                    break;
                }
            }
        } else {
            double pg = fabs(press * 1e-9);
            double solidus = -5.02 * (pg * pg) + 1.32e2 * pg + 1.09e3 + 35.0;
            if (tmpr >= solidus + 35.0) newph = 18;
        }
        break;
    }
    case 10: case 3: case 7: {
        double press = mantle_density * P.g * depth;
        if (P.eclogite_rule == 1) {
            if (tmpr >= 600.0 && press >= 1.5e9) newph = 13;
        } else {
            double trpres = -0.3e9 + 2.2e6 * tmpr;
            double trpres2 = 20.1e9 - 0.0375e9 * tmpr;
            if (!(tmpr < 400.0 || depth < 20e3 || press < trpres || press < trpres2)) newph = 13;
        }
        break;
    }
    case 9: {
        double trpres = 2.1e9 + (7.5e9 - 2.1e9) * (tmpr - 730.0) / (500.0 - 730.0);
        double trpres2 = 2.1e9 + (0.2e9 - 2.1e9) * (tmpr - 730.0) / (650.0 - 730.0);
        double press = mantle_density * P.g * depth;
        if (!(tmpr < 550.0 || (press < trpres && press > trpres2))) newph = 4;
        break;
    }
    case 1:
        if (!(tmpr < 80.0 && depth < 2e3)) newph = 11;
        break;
    case 11:
        if (!(tmpr < 250.0 && depth < 7e3)) newph = 17;
        break;
    case 17: {
        double trpres = 0.88e9 - (0.88e9 - 0.704e9) * (710.8 - tmpr) / (710.8 - 662.3);
        double press = mantle_density * P.g * depth;
        if (!(press < trpres)) newph = 5;
        break;
    }
    case 5: {
        double trpres = 0.0e9 - (0.0e9 - 1.2e9) * (500.0 - tmpr) / (500.0 - 600.0);
        double press = mantle_density * P.g * depth;
        if (!(press > trpres)) newph = 19;
        break;
    }
    case 16: {
        double dd = depth - 62e3;
        double trtmpr = 880 - 35e-9 * (dd * dd);
        if (!(tmpr < trtmpr)) newph = 4;
        break;
    }
    default:
        break;
    }
    if (newph) {
        A.e_flag[e] = 1;
        A.mark_phase[kk] = (int8_t)newph;
    }
}
__global__ void __launch_bounds__(GF_THREADS) k_phase_markers(const DevParams *__restrict__ Pp, DevArrays A, GfDims d, int nmarkers) {
    gf_pdl_entry();
    b_k_phase_markers(Pp, A, d, nmarkers, (GF_IDX)blockIdx.x * blockDim.x + threadIdx.x);
}

// The same rules in FP32 for the mixed path: the marker's depth below the
// surface from coordinate differences of the hi/lo splits, its temperature
// from the hi parts.  Decisions within FP32 rounding of a threshold may
// differ from the FP64 path.
__device__ __forceinline__ void b_k_phase_markers32(const DevParams *__restrict__ Pp, DevArrays A, GfDims d, int nmarkers, GF_IDX kk) {
    if (kk >= nmarkers) return;
    if (A.mark_dead[kk] == 0) return;
    const DevParams &P = *Pp;
    const int nz = d.nz;
    int n = A.mark_ntriag[kk];
    int k = (n - 1) % 2 + 1;
    int j = ((n - k) / 2) % (nz - 1);
    int i = (n - k) / 2 / (nz - 1);
    // the exclusions of the FP64 kernel (a phase without a rule; a marker
    // certainly deeper than its rule reaches, from the hi parts of the
    // corner and surface heights with a 10 m margin), before the marker's
    // own coordinates are read
    {
        const int ph = A.mark_phase[kk];
        if (!(ph == 4 || ph == 8 || ph == 10 || ph == 3 || ph == 7 || ph == 9 || ph == 1 || ph == 11 || ph == 17 ||
              ph == 5 || ph == 16))
            return;
        const float *zc = A.cord_hi + d.N;
        const GF_IDX q1 = gf_node(d, j, i), q3 = gf_node(d, j, i + 1);
        const float zmax = fmaxf(fmaxf(zc[q1], zc[q1 + 1]), fmaxf(zc[q3], zc[q3 + 1]));
        const float surf = 0.5f * (zc[gf_node(d, 0, i)] + zc[gf_node(d, 0, i + 1)]);
        const float lim = (ph == 4 || ph == 8) ? 150e3f : 200e3f;
        if (surf - zmax > lim + 10.0f) return;
    }
    const float a1 = gf_d2f(A.mark_a1[kk]), a2 = gf_d2f(A.mark_a2[kk]), a3 = 1.0f - a1 - a2;
    GF_IDX p1, p2, p3;
    if (k == 1) {
        p1 = gf_node(d, j, i); p2 = gf_node(d, j + 1, i); p3 = gf_node(d, j, i + 1);
    } else {
        p1 = gf_node(d, j, i + 1); p2 = gf_node(d, j + 1, i); p3 = gf_node(d, j + 1, i + 1);
    }
    const float *zh = A.cord_hi + d.N, *zl = A.cord_lo + d.N, *th = A.temp_hi;
    const GF_IDX s0 = gf_node(d, 0, i), s1 = gf_node(d, 0, i + 1);
    // depth = 0.5 * (z_s0 + z_s1) - sum a_k z_pk, as differences to z_s0
    const float ds1 = hl_diff(zh, zl, s1, s0);
    const float y1 = hl_diff(zh, zl, p1, s0), y2 = hl_diff(zh, zl, p2, s0), y3 = hl_diff(zh, zl, p3, s0);
    const float depth = 0.5f * ds1 - (y1 * a1 + y2 * a2 + y3 * a3);
    if (depth > 200e3f) return;
    const float tmpr = th[p1] * a1 + th[p2] * a2 + th[p3] * a3;
    int iph = A.mark_phase[kk];
    GF_IDX e = gf_elem(d, j, i);
    const float rho_g = 3000.0f * P.f_g;
    GF_IDX total = (GF_IDX)P.nphase * d.E;
    auto pr = [&](GF_IDX eb, int ph1) {
        GF_IDX off = (GF_IDX)(ph1 - 1) + (GF_IDX)P.nphase * eb;
        return (off < 0 || off >= total) ? 0.0 : A.phase_ratio[off];
    };
    int newph = 0;
    switch (iph) {
    case 4: case 8: {
        if (depth > 150e3f) break;
        float trpres = 2.1e9f + (7.5e9f - 2.1e9f) * (tmpr - 730.0f) / (500.0f - 730.0f);
        float trpres2 = 2.1e9f + (0.6e9f - 2.1e9f) * (tmpr - 730.0f) / (670.0f - 730.0f);
        float press = rho_g * depth;
        float pg = fabsf(press * 1e-9f);
        float solidus = -5.02f * (pg * pg) + 1.32e2f * pg + 1.09e3f + 35.0f;
        if (press < trpres && press > trpres2) {
            int jb0 = min(j + 2, nz - 1), jb1 = min(j + 1 + P.nelem_serp, nz - 1);
            for (int jb = jb0; jb <= jb1; ++jb) {
                GF_IDX eb = gf_elem(d, jb - 1, i);
                if (pr(eb, 3) > 0.8 || pr(eb, 7) > 0.8 || pr(eb, 1) > 0.8 || pr(eb, 11) > 0.8) {
                    newph = 9;
                    break;
                }
            }
        } else if (tmpr >= solidus + 35.0f) {
            newph = 18;
        }
        break;
    }
    case 10: case 3: case 7: {
        float press = rho_g * depth;
        if (P.eclogite_rule == 1) {
            if (tmpr >= 600.0f && press >= 1.5e9f) newph = 13;
        } else {
            float trpres = -0.3e9f + 2.2e6f * tmpr;
            float trpres2 = 20.1e9f - 0.0375e9f * tmpr;
            if (!(tmpr < 400.0f || depth < 20e3f || press < trpres || press < trpres2)) newph = 13;
        }
        break;
    }
    case 9: {
        float trpres = 2.1e9f + (7.5e9f - 2.1e9f) * (tmpr - 730.0f) / (500.0f - 730.0f);
        float trpres2 = 2.1e9f + (0.2e9f - 2.1e9f) * (tmpr - 730.0f) / (650.0f - 730.0f);
        float press = rho_g * depth;
        if (!(tmpr < 550.0f || (press < trpres && press > trpres2))) newph = 4;
        break;
    }
    case 1:
        if (!(tmpr < 80.0f && depth < 2e3f)) newph = 11;
        break;
    case 11:
        if (!(tmpr < 250.0f && depth < 7e3f)) newph = 17;
        break;
    case 17: {
        float trpres = 0.88e9f - (0.88e9f - 0.704e9f) * (710.8f - tmpr) / (710.8f - 662.3f);
        if (!(rho_g * depth < trpres)) newph = 5;
        break;
    }
    case 5: {
        float trpres = 0.0f - (0.0f - 1.2e9f) * (500.0f - tmpr) / (500.0f - 600.0f);
        if (!(rho_g * depth > trpres)) newph = 19;
        break;
    }
    case 16: {
        float dd = depth - 62e3f;
        float trtmpr = 880.0f - 35e-9f * (dd * dd);
        if (!(tmpr < trtmpr)) newph = 4;
        break;
    }
    default:
        break;
    }
    if (newph) {
        A.e_flag[e] = 1;
        A.mark_phase[kk] = (int8_t)newph;
    }
}
__global__ void __launch_bounds__(GF_THREADS) k_phase_markers32(const DevParams *__restrict__ Pp, DevArrays A, GfDims d, int nmarkers) {
    gf_pdl_entry();
    b_k_phase_markers32(Pp, A, d, nmarkers, (GF_IDX)blockIdx.x * blockDim.x + threadIdx.x);
}

// count_phase_ratio (marker_data.f90:140-172) for flagged elements + aps
template <class R> __device__ __forceinline__ void b_k_phase_recount(const DevParams *__restrict__ Pp, DevClock *__restrict__ C, DevArrays A, GfDims d, int all, GF_IDX e) {
    if (e >= d.E) return;
    if (!all && !A.e_flag[e]) return;
    const DevParams &P = *Pp;
    int nm = A.nmark_elem[e];
    if (nm == 0) {
        set_status(C, 134, (int)e);
        return;
    }
    int cnt[GF_MAXPH + 1];
#pragma unroll
    for (int k = 0; k <= GF_MAXPH; ++k) cnt[k] = 0;
    for (int m = 0; m < nm; ++m) {
        int kk = A.mark_id_elem[e * GF_MAX_MARKERS_PER_ELEM + m];
        int iph = A.mark_phase[kk - 1];
        if (iph >= 1 && iph <= GF_MAXPH) cnt[iph] += 1;
    }
    int best = 0, iph = 1;
    for (int k = 1; k <= P.nphase; ++k) {
        A.phase_ratio[gf_pr(d, e, k - 1)] = cnt[k] / (nm * 1.0);
        if (cnt[k] > best) {
            best = cnt[k];
            iph = k;
        }
    }
    A.iphase[e] = iph;
    if (!all) {
        R *aps = (R *)A.aps;
        R a0 = aps[e];
        R v = a0 - a0 / R((float)nm);
        aps[e] = v > R(0.0) ? v : R(0.0);
        A.e_flag[e] = 0;
    }
}
template <class R> __global__ void __launch_bounds__(GF_THREADS) k_phase_recount(const DevParams *__restrict__ Pp, DevClock *__restrict__ C, DevArrays A, GfDims d, int all) {
    gf_pdl_entry();
    b_k_phase_recount<R>(Pp, C, A, d, all, (GF_IDX)blockIdx.x * blockDim.x + threadIdx.x);
}

// ======================================================================
// itest_mesh angle criterion (rem_test.f90:77-118): min over all triangles.
// On large meshes a pass in FP32 comes first: the largest cosine of each
// element's angles, to about 1e-6, and of the mesh.  Only elements within 4e-6
// of the mesh's can hold the smallest angle; the FP64 pass, bound by its
// arccosines, evaluates those.  Where an angle is nearly 0 or FP32 does not
// resolve an edge the cosine counts as 2, and then every element is evaluated
// (1000x300 elements: 274 -> 56 us for the test).
__device__ __forceinline__ float elem_max_cos(const DevArrays &A, const GfDims &d, GF_IDX e) {
    int j, i;
    elem_ji(d, e, j, i);
    Quad q;
    load_quad(A.cord, d, j, i, q);
    bool ok = true;
    float cmax = -1.0f;
    // the edges from node 0 and between the others, as FP32 differences
    float x[6], y[6], r[6];
    const int ea[6] = {0, 0, 0, 1, 1, 2}, eb[6] = {1, 2, 3, 2, 3, 3};
#pragma unroll
    for (int k = 0; k < 6; ++k) {
        x[k] = gf_d2f(q.x[eb[k]] - q.x[ea[k]]);
        y[k] = gf_d2f(q.y[eb[k]] - q.y[ea[k]]);
        const float l2 = x[k] * x[k] + y[k] * y[k];
        ok = ok && l2 > 1e-24f && l2 < 1e24f;
        r[k] = 1.0f / sqrtf(l2);
    }
    // cosine between edges k and m at a common end (s: -1 where one of them points away)
    auto c = [&](int k, int m, float s) { cmax = fmaxf(cmax, s * (x[k] * x[m] + y[k] * y[m]) * (r[k] * r[m])); };
    // edges 0: 01, 1: 02, 2: 03, 3: 12, 4: 13, 5: 23; triangles 012, 132, 013, 032
    c(0, 1, 1.0f); c(0, 3, -1.0f); c(1, 3, 1.0f);
    c(3, 4, 1.0f); c(3, 5, -1.0f); c(4, 5, 1.0f);
    c(0, 2, 1.0f); c(0, 4, -1.0f); c(2, 4, 1.0f);
    c(1, 2, 1.0f); c(1, 5, -1.0f); c(2, 5, 1.0f);
    return ok && cmax < 0.9999f ? cmax : 2.0f;
}
__global__ void __launch_bounds__(GF_THREADS) k_angle_cos(DevArrays A, GfDims d, float *cosm, unsigned *top) {
    gf_pdl_entry();
    const GF_IDX e = (GF_IDX)blockIdx.x * blockDim.x + threadIdx.x;
    float c = -1.0f;
    if (e < d.E) {
        c = elem_max_cos(A, d, e);
        cosm[e] = c;
    }
    c = warp_max(c);
    if ((threadIdx.x & 31) == 0) atomicMax(top, __float_as_uint(c + 2.0f)); // (c + 2 >= 1: ordered as bits)
}
// The exact pass, a thread per triangle (local vertices as in
// rem_test.f90:84-92).  The reference's expressions; its two angles of a
// triangle share an edge (whose length and products have the same bits seen
// from either end), and products and quotients go to the integer pipes
// (60x20 elements: 39 -> 27 us for the test; eight angles ran one after another
// in an element's thread).
__device__ __forceinline__ void b_k_min_angle(DevArrays A, GfDims d, unsigned long long *out, const float *cosm,
                                              const unsigned *top, GF_IDX th) {
    double amin = 180.0;
    const GF_IDX e = th >> 2;
    // (above 2.9 some element's cosine counted as 2: all are evaluated)
    const float c = cosm ? __uint_as_float(*top) : 4.0f;
    if (e < d.E && (c > 2.9999f || cosm[e] + 2.0f >= c - 4e-6f)) {
        int j, i;
        elem_ji(d, e, j, i);
        const int t = (int)(th & 3);
        const int v0 = t == 1 ? 1 : 0, v1 = (t & 1) ? 3 : 1, v2 = t == 2 ? 3 : 2;
        auto node = [&](int v) { return gf_node(d, j + (v & 1), i + (v >> 1)); };
        const GF_IDX n0 = node(v0), n1 = node(v1), n2 = node(v2);
        const double *X = A.cord, *Y = A.cord + d.N;
        const double x0 = X[n0], x1 = X[n1], x2 = X[n2], y0 = Y[n0], y1 = Y[n1], y2 = Y[n2];
        const double raddeg = 180.0 / 3.14159265358979323846;
        // from vertex 1 to 2 and to 0, and from 2 to 0
        const double ax = x2 - x1, ay = y2 - y1, bx = x0 - x1, by = y0 - y1, cx = x0 - x2, cy = y0 - y2;
        const double al = sqrt(gf_mul(ax, ax) + gf_mul(ay, ay)), bl = sqrt(gf_mul(bx, bx) + gf_mul(by, by)),
                     cl = sqrt(gf_mul(cx, cx) + gf_mul(cy, cy));
        const double ang1 = raddeg * acos(gf_ddiv(gf_mul(ax, bx) + gf_mul(ay, by), gf_mul(al, bl)));
        const double ang2 = raddeg * acos(gf_ddiv(gf_neg(gf_mul(cx, ax) + gf_mul(cy, ay)), gf_mul(cl, al)));
        const double ang0 = 180.0 - ang1 - ang2;
        amin = fmin(amin, fmin(ang0, fmin(ang1, ang2)));
    }
    amin = warp_min(amin);
    if ((threadIdx.x & 31) == 0) atomic_min_pos(out, fmax(amin, 0.0));
}
__global__ void __launch_bounds__(GF_THREADS) k_min_angle(DevArrays A, GfDims d, unsigned long long *out, const float *cosm, const unsigned *top) {
    gf_pdl_entry();
    b_k_min_angle(A, d, out, cosm, top, (GF_IDX)blockIdx.x * blockDim.x + threadIdx.x);
}

// FP64 host array -> R device array
template <class R> __device__ __forceinline__ void b_k_convert(const double *__restrict__ src, R *__restrict__ dst, GF_IDX n, GF_IDX t) {
    if (t < n) dst[t] = R(src[t]);
}
template <class R> __global__ void k_convert(const double *__restrict__ src, R *__restrict__ dst, GF_IDX n) {
    gf_pdl_entry();
    b_k_convert<R>(src, dst, n, (GF_IDX)blockIdx.x * blockDim.x + threadIdx.x);
}
template <class R> __device__ __forceinline__ void b_k_convert_back(const R *__restrict__ src, double *__restrict__ dst, GF_IDX n, GF_IDX t) {
    if (t < n) dst[t] = (double)src[t];
}
template <class R> __global__ void k_convert_back(const R *__restrict__ src, double *__restrict__ dst, GF_IDX n) {
    gf_pdl_entry();
    b_k_convert_back<R>(src, dst, n, (GF_IDX)blockIdx.x * blockDim.x + threadIdx.x);
}

} // namespace gfk
} // namespace

#ifdef GF_FP64_UNIT
#include "gf_tri64.cuh"
#endif

// ---------------------------------------------------------------- launchers
inline int gf_sm_count() {
    static const int sms = [] {
        int dev = 0, v = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev);
        return v;
    }();
    return sms;
}
// Threads per CTA for n items.  FP64 kernels: fewer than `most`, down to 64,
// while that leaves SMs without a CTA, since warps that share an SM queue for
// its FP64 pipe (ten steps of 60x20 elements 1.055 -> 1.020 ms, 241x61 1.265
// -> 1.220; 32 threads measured the same).  The mixed kernels lose on it
// (60x20: 0.393 -> 0.416 at 32 threads): theirs is a chain of instructions
// that warps of one SM fetch once for all.
inline unsigned gf_threads_for(long long n, unsigned most) {
#ifdef GF_FP64_UNIT
    while (most > 64 && n <= (long long)(most / 2) * gf_sm_count()) most /= 2;
#else
    (void)n;
#endif
    return most;
}
#ifdef GF_FP64_UNIT
#include "gf_therm64.cuh"
#endif
#define GF_LAUNCH(kern, n, ...) GF_LAUNCH_T(kern, n, GF_THREADS, __VA_ARGS__)
#define GF_LAUNCH_T(kern, n, thr, ...)                                                                                      \
    do {                                                                                                               \
        if ((n) > 0) {                                                                                                 \
            const unsigned _t = gf_threads_for(n, thr);                                                                \
            gf_launch_pdl(kern, gfk::grid_for(n, _t), _t, g.s, __VA_ARGS__);                                           \
            ++*g.launches;                                                                                             \
        }                                                                                                              \
    } while (0)

// The table read by plastic_table_state's elements: one thread per (phase,
// state), each evaluating pre_plast_phase and plastic_consts as the element
// path does, with a plastic strain in the state's branch (-inf: before
// softening, plstrain1: at its start, +inf: after it).
namespace { // internal linkage, one copy per precision's translation unit
namespace gfk {
template <class R> __global__ void k_plastic_table(const DevParams *__restrict__ Pp, R *__restrict__ tab) {
    const DevParams &P = *Pp;
    const int t = threadIdx.x;
    if (t >= GF_MAXPH * GF_PT_STATES) return;
    const int k = t / GF_PT_STATES, s = t % GF_PT_STATES;
    R pl1, bulkm, rmu, ten_off;
    if constexpr (sizeof(R) == sizeof(float)) {
        pl1 = P.f_pl1[k]; bulkm = P.f_bulkm[k]; rmu = P.f_rm[k]; ten_off = P.f_ten_off;
    } else {
        pl1 = P.plstrain1[k]; bulkm = P.bulkm[k]; rmu = P.rm[k]; ten_off = P.ten_off;
    }
    const R pls = s == 0 ? R(-INFINITY) : (s == 1 ? pl1 : R(INFINITY));
    R phi = 0, coh = 0, psi = 0, hardn = 0;
    pre_plast_phase(P, k, R(1), pls, phi, coh, psi, hardn);
    phi = R(1) / phi;
    coh = R(1) / coh;
    const PlasticConsts<R> c = plastic_consts<R>(bulkm, rmu, coh, phi, psi, ten_off);
    R *o = tab + (s * GF_MAXPH + k) * GF_PT_W;
    o[0] = c.anphi; o[1] = c.anpsi; o[2] = c.amc; o[3] = c.e1;
    o[4] = c.e2; o[5] = c.x1; o[6] = c.ten_max; o[7] = hardn;
}
} // namespace gfk
} // namespace
template <class R> void GfKernels<R>::plastic_table(const GfLaunch &g) {
    if (g.A.plast_tab) {
        gfk::k_plastic_table<R><<<1, GF_MAXPH * GF_PT_STATES, 0, g.s>>>(g.P, (R *)g.A.plast_tab);
        ++*g.launches;
    }
}

template <class R> void GfKernels<R>::step_forces(const GfLaunch &g, int avg_mode, int move) {
    using namespace gfk;
    if (sizeof(R) != sizeof(float)) return;
    auto launch = [&](auto kern, unsigned parts, auto... args) {
        gf_launch_pdl(kern, dim3(grid_for(g.d.N), parts), GF_THREADS, g.s, args...);
        ++*g.launches;
    };
    // beside fl_rheol's CTAs (two an SM, by their registers) while both fit the
    // SMs at once; on larger meshes the prep, which wants warps in flight, is a
    // launch of its own (a step of 1000x300 elements 93.2 against 98.5 us)
    const bool beside = grid_for(g.d.N) <= (unsigned)gf_sm_count();
    if (!beside) GF_LAUNCH(k_therm_prep32, g.d.N, g.P, g.A, g.d, (float *)g.A.t_coef);
    launch(k_step_a, beside ? 2u : 1u, g.P, g.C, g.A, g.d);
    launch(k_step_b, avg_mode > 0 ? 3u : 2u, g.P, g.C, g.A, g.d, avg_mode);
    launch(k_step_c, move ? 3u : 1u, g.P, g.C, g.A, g.d, avg_mode);
    if (move)
        launch(k_step_d, 2u, g.P, g.C, g.A, g.d, g.advance_time);
    else
        GF_LAUNCH(k_therm_apply32, g.d.N, g.P, g.A, g.d, g.A.t_delta1);
}

template <class R> void GfKernels<R>::therm(const GfLaunch &g, int sweeps, int keep_temp0) {
    using namespace gfk;
    if (sizeof(R) == sizeof(float)) {
        const float *tc = (const float *)g.A.t_coef;
        float *d0 = (float *)g.A.t_delta0;
        GF_LAUNCH(k_therm_prep32, g.d.N, g.P, g.A, g.d, (float *)g.A.t_coef);
        GF_LAUNCH(k_therm_sweep32, g.d.N, g.P, g.C, g.A, g.d, tc, d0, g.A.t_delta1, 0);
        GF_LAUNCH(k_therm_sweep32, g.d.N, g.P, g.C, g.A, g.d, tc, d0, g.A.t_delta1, 1);
        GF_LAUNCH(k_therm_apply32, g.d.N, g.P, g.A, g.d, g.A.t_delta1);
        return;
    }
#ifdef GF_FP64_UNIT
    therm_launch(g, sweeps > 0 ? (sweeps < GF_THERM_KMAX ? sweeps : GF_THERM_KMAX) : GF_THERM_KMAX, keep_temp0);
#endif
}

template <class R> void GfKernels<R>::rheol(const GfLaunch &g, int update_visc, int avg_mode) {
    using namespace gfk;
#ifdef GF_FP64_UNIT
    if (update_visc) GF_LAUNCH(k_rheol_visc, g.d.E, g.P, g.A, g.d);
    GF_LAUNCH_T(k_rheol_tri, 4 * g.d.E, GF_TRI_T, g.P, g.C, g.A, g.d);
#else
    GF_LAUNCH(k_rheol<R>, g.d.E, g.P, g.C, g.A, g.d, update_visc, 0);
#endif
    if (avg_mode > 0) {
        GF_LAUNCH(k_rheol_avg<R>, g.d.E, g.C, g.A, g.d, avg_mode == 2 ? 1 : 0);
        if (avg_mode == 2) {
            k_rheol_clock<<<1, 1, 0, g.s>>>(g.C, 1);
            ++*g.launches;
        }
    }
}

namespace {
namespace gfk {
__global__ void __launch_bounds__(GF_THREADS) k_elem_forces(DevArrays A, GfDims d) {
    gf_pdl_entry();
    const GF_IDX e = (GF_IDX)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= d.E) return;
    int j, i;
    elem_ji(d, e, j, i);
    const float *st = (const float *)A.stress0;
    const float *area = (const float *)A.area;
    float ar[4], sn[4][4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        ar[k] = area[gf_ek(d, e, k)];
#pragma unroll
        for (int c = 0; c < 4; ++c) sn[c][k] = st[gf_s(d, e, c, k)];
    }
    QuadF q;
    load_quad_rel(A, d, j, i, q);
    float dx[3][4], dz[3][4];
    shape_derivs_f(q, ar, dx, dz);
    elem_corner_forces(dx, dz, ar, sn, A.e_frc, d.E, e);
}
} // namespace gfk
} // namespace

template <class R> void GfKernels<R>::elem_forces(const GfLaunch &g) {
    using namespace gfk;
    if (sizeof(R) == sizeof(float)) GF_LAUNCH(k_elem_forces, g.d.E, g.A, g.d);
}

template <class R> void GfKernels<R>::node(const GfLaunch &g) {
    using namespace gfk;
    GF_LAUNCH(k_node<R>, g.d.N, g.P, g.C, g.A, g.d, g.node_terms);
}

template <class R> void GfKernels<R>::move_cord(const GfLaunch &g) {
    using namespace gfk;
    GF_LAUNCH(k_move_cord, 2 * g.d.N, g.C, g.A, g.d);
}
template <class R> void GfKernels<R>::move_elem(const GfLaunch &g) {
    using namespace gfk;
#ifdef GF_FP64_UNIT
    GF_LAUNCH(k_move_tri, 4 * g.d.E, g.C, g.A, g.d, g.advance_time);
#else
    GF_LAUNCH(k_move_elem<R>, g.d.E, g.C, g.A, g.d, g.advance_time);
#endif
}
template <class R> void GfKernels<R>::move(const GfLaunch &g) {
    move_cord(g);
    move_elem(g);
}

// elements from which the FP64 pipe, not a thread's chain, bounds such kernels
constexpr long long GF_INT_PIPE_E = 8192;
template <class R> void GfKernels<R>::rmasses(const GfLaunch &g) {
    using namespace gfk;
    // (gf_mulc: 60x20 elements lose 1 % of ten steps on the integer pipes, 241x61
    // gain 3 %, and fl's rmasses + dt_mass of 1000x300 take 161 instead of 262 us)
    if (sizeof(R) == sizeof(double) && g.d.E >= GF_INT_PIPE_E)
        GF_LAUNCH((k_elem_dens<R, true>), g.d.E, g.P, g.C, g.A, g.d);
    else
        GF_LAUNCH(k_elem_dens<R>, g.d.E, g.P, g.C, g.A, g.d);
    k_frac_fix<R><<<1, 1, 0, g.s>>>(g.P, g.C, g.A, g.d);
    ++*g.launches;
    GF_LAUNCH(k_node_gather_tri<R>, g.d.N, (const R *)g.A.e_tri, g.A.rmass, g.d);
}

template <class R> void GfKernels<R>::dt_mass(const GfLaunch &g) {
    using namespace gfk;
    k_dt_reset<<<1, 1, 0, g.s>>>(g.C);
    ++*g.launches;
    GF_IDX n = g.d.E > g.d.N ? g.d.E : g.d.N;
    const bool ip = sizeof(R) == sizeof(double) && g.d.E >= GF_INT_PIPE_E;
    if (ip)
        GF_LAUNCH((k_dt_reduce<R, true>), n, g.P, g.C, g.A, g.d);
    else
        GF_LAUNCH(k_dt_reduce<R>, n, g.P, g.C, g.A, g.d);
    k_dt_scalars<<<1, 1, 0, g.s>>>(g.P, g.C);
    ++*g.launches;
    if (g.idt_scale == 0) {
        cudaMemcpyAsync(g.A.amass, g.A.rmass, sizeof(double) * g.d.N, cudaMemcpyDeviceToDevice, g.s);
    } else {
        if (ip)
            GF_LAUNCH((k_elem_am3<R, true>), g.d.E, g.P, g.C, g.A, g.d);
        else
            GF_LAUNCH(k_elem_am3<R>, g.d.E, g.P, g.C, g.A, g.d);
        GF_LAUNCH(k_node_gather_tri<R>, g.d.N, (const R *)g.A.e_tri, g.A.amass, g.d);
    }
}

template <class R> void GfKernels<R>::init_visc(const GfLaunch &g) {
    using namespace gfk;
    GF_LAUNCH(k_init_visc<R>, g.d.E, g.P, g.A, g.d);
}

template <class R> void GfKernels<R>::change_phase(const GfLaunch &g, int nmarkers) {
    using namespace gfk;
    if (sizeof(R) == sizeof(float))
        GF_LAUNCH(k_phase_markers32, (GF_IDX)nmarkers, g.P, g.A, g.d, nmarkers);
    else
        GF_LAUNCH(k_phase_markers, (GF_IDX)nmarkers, g.P, g.A, g.d, nmarkers);
    GF_LAUNCH(k_phase_recount<R>, g.d.E, g.P, g.C, g.A, g.d, 0);
}

namespace {
namespace gfk {
__global__ void k_split(const double *__restrict__ src, float *__restrict__ hi, float *__restrict__ lo, GF_IDX n) {
    gf_pdl_entry();
    GF_IDX t = (GF_IDX)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    const double v = src[t];
    const float h = (float)v;
    hi[t] = h;
    lo[t] = (float)(v - (double)h);
}
} // namespace gfk
} // namespace

template <class R> void GfKernels<R>::split_nodes(const GfLaunch &g) {
    using namespace gfk;
    if (!g.A.cord_hi) return;
    GF_LAUNCH(k_split, 2 * g.d.N, g.A.cord, g.A.cord_hi, g.A.cord_lo, 2 * g.d.N);
    GF_LAUNCH(k_split, 2 * g.d.N, g.A.vel, g.A.vel_hi, g.A.vel_lo, 2 * g.d.N);
    if (g.A.pr_hi) GF_LAUNCH(k_split, g.d.E, g.A.p_ref, g.A.pr_hi, g.A.pr_lo, g.d.E);
    if (g.A.temp_hi) GF_LAUNCH(k_split, g.d.N, g.A.temp, g.A.temp_hi, g.A.temp_lo, g.d.N);
}

template <class R> void GfKernels<R>::phase_recount_all(const GfLaunch &g) {
    using namespace gfk;
    GF_LAUNCH(k_phase_recount<R>, g.d.E, g.P, g.C, g.A, g.d, 1);
}

template <class R> void GfKernels<R>::min_angle(const GfLaunch &g, double *d_out) {
    using namespace gfk;
    // (the FP32 pass costs more than it saves where the FP64 pass is one chain of latencies)
    float *cosm = g.d.E >= 8192 ? (float *)g.A.t_delta0 : nullptr; // free outside fl_therm
    unsigned *top = (unsigned *)(d_out + 5 + 2 * (long long)g.d.nx);
    if (cosm) GF_LAUNCH(k_angle_cos, g.d.E, g.A, g.d, cosm, top);
    GF_LAUNCH(k_min_angle, 4 * g.d.E, g.A, g.d, (unsigned long long *)d_out, (const float *)cosm, (const unsigned *)top);
}

template <class R>
void GfKernels<R>::convert_in(const GfLaunch &g, unsigned mask, const double *src, void *dst, long long n) {
    using namespace gfk;
    if (mask)
        GF_LAUNCH(k_convert<R>, n, src, (R *)dst, n);
    else
        GF_LAUNCH(k_convert_back<R>, n, (const R *)dst, (double *)src, n);
}

namespace {
namespace gfk {
// total stress -> (p_ref, total + p_ref on the normal components)
template <class R> __device__ __forceinline__ void b_k_stress_in(const double *__restrict__ tot, R *__restrict__ st, double *__restrict__ p_ref, GfDims d, GF_IDX e) {
    if (e >= d.E) return;
    double s = 0.0;
#pragma unroll
    for (int k = 0; k < 4; ++k) s += tot[gf_s(d, e, 0, k)] + tot[gf_s(d, e, 1, k)] + tot[gf_s(d, e, 3, k)];
    double p = -s / 12.0;
    p_ref[e] = p;
#pragma unroll
    for (int k = 0; k < 4; ++k)
#pragma unroll
        for (int c = 0; c < 4; ++c) st[gf_s(d, e, c, k)] = R(c == 2 ? tot[gf_s(d, e, c, k)] : tot[gf_s(d, e, c, k)] + p);
}
template <class R> __global__ void __launch_bounds__(GF_THREADS) k_stress_in(const double *__restrict__ tot, R *__restrict__ st, double *__restrict__ p_ref, GfDims d) {
    gf_pdl_entry();
    b_k_stress_in<R>(tot, st, p_ref, d, (GF_IDX)blockIdx.x * blockDim.x + threadIdx.x);
}

template <class R> __device__ __forceinline__ void b_k_stress_out(const R *__restrict__ st, const double *__restrict__ p_ref, double *__restrict__ tot, GfDims d, GF_IDX e) {
    if (e >= d.E) return;
    double p = p_ref[e];
#pragma unroll
    for (int k = 0; k < 4; ++k)
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            double v = (double)st[gf_s(d, e, c, k)];
            tot[gf_s(d, e, c, k)] = c == 2 ? v : v - p;
        }
}
template <class R> __global__ void __launch_bounds__(GF_THREADS) k_stress_out(const R *__restrict__ st, const double *__restrict__ p_ref, double *__restrict__ tot, GfDims d) {
    gf_pdl_entry();
    b_k_stress_out<R>(st, p_ref, tot, d, (GF_IDX)blockIdx.x * blockDim.x + threadIdx.x);
}
} // namespace gfk
} // namespace

template <class R> void GfKernels<R>::stress_in(const GfLaunch &g, const double *src) {
    using namespace gfk;
    GF_LAUNCH(k_stress_in<R>, g.d.E, src, (R *)g.A.stress0, g.A.p_ref, g.d);
    if (g.A.pr_hi) GF_LAUNCH(k_split, g.d.E, g.A.p_ref, g.A.pr_hi, g.A.pr_lo, g.d.E);
}

template <class R> void GfKernels<R>::stress_out(const GfLaunch &g, double *dst) {
    using namespace gfk;
    GF_LAUNCH(k_stress_out<R>, g.d.E, (const R *)g.A.stress0, g.A.p_ref, dst, g.d);
}
