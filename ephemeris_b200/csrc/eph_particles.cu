// eph_particles.cu - massless test particles integrated against massive perturbers.
//
// A particle feels the perturbers and nothing else, and the perturbers do not feel it, so the two
// integrations separate: the perturbers run through the single-system kernel (eph_step.cu), which records
// every stage evaluation of every perturber (position, potential, Newtonian acceleration, velocity/c,
// harmonics, spin, frames: the TrajField record); then `particle_kernel` integrates each particle on its
// own thread through the same 25 stage times, reading the perturber records of each stage from shared
// memory. Per particle and stage (the reference's terms for a point-like body i and perturber j):
//   pass A  phi_i, a_N,i of mass.impl:38-46 (floored at sR2_j: the particle has no radius)
//   prepare beta_i = v_i / c, beta_i^2, phi_i / c^2, a_N,i / c^2 (mass.impl:76-80)
//   pass B  EIH 1PN (mass.impl:82-97) with the perturbers' own prepared values; j's deformation force and
//           j's Lense-Thirring field on i (mass.impl:99-125, the j-side terms)
//   fields  geopotential and ring fields of the extended perturbers at i (mass.cpp:358-371; the reaction
//           on the perturber is GM_i times the field, zero for a massless particle)
//   final   f_i = (gaccel + daccel) + naccel (mass.cpp:389-396)
// The RK12 step is RungeKutta.impl:107-194's in second-order form (only the stage accelerations are
// stored; see particle_kernel), with its state update's arithmetic. The reference has no massless bodies;
// bodies of negligible mass
// (GM = 1e-20 m^3/s^2) in one system with the perturbers are its equivalent, and the tests compare with
// exactly that.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <vector>

#include "eph_launch.cuh"
#include "eph_math.cuh"
#include "eph_models.cuh"
#include "eph_rk12_host.h"
#include "eph_system.cuh"
#include "../../include/eph_b200.h"
#include "../../include/eph_planes.h"

namespace eph {
void ctx_record_stages(eph_ctx *ctx, double *d_buf, long long base);
int ctx_rk12_begin(eph_ctx *ctx, double dt, long long n_step, double t_eph, cudaEvent_t after);
int ctx_rk12_end(eph_ctx *ctx);
}

namespace eph {
namespace {

constexpr int kPThreads = 256;          // particles per CTA
constexpr int kPMaxPert = 32;           // perturbers (their stage records live in shared memory)
constexpr size_t kPRecordBytes = 1ull << 29;   // stage records of one round of perturbers or particles
constexpr int kPRounds = 8, kPRoundSteps = 4;  // rounds of a call where its steps allow, most steps of a round
constexpr double kCP = 299792458.0;     // src/math/basic_math.h:10,18
constexpr int kPF = 3;                  // stored values per (particle, stage): the acceleration

// The Feagin table as the particle kernel uses it: c_k and the rows k = 1..25 of a (hi + lo rounded) and of the
// second-order Abar = A A without the columns where both are zero (entries p_row[k] <= q < p_row[k + 1], ascending).
__constant__ double2 p_ab[EPH_RK12_NCOEF];   // {Abar_kl, a_kl}
__constant__ int p_l[EPH_RK12_NCOEF];
__constant__ int p_row[kStages + 2];
__constant__ double p_c[kStages + 1];

struct PertInfo {
    int gp, ring;      // model indices, or -1
    int full;          // its deformation / spin act on others (full-class body)
    int nz, nt, nd;    // zonal and tesseral degree, ring disks
    double inv_r2;     // 1 / R^2
    double2 J[EPH_GP_MAX_DEGREE + 1];   // {J_n, (n + 1) J_n} of the geopotential
};
constexpr int kPartGp = 4;   // tesseral models of up to degree 6 and order 4 kept expanded in shared memory

struct PartArgs {
    int n_part, n_pert;
    long long n_step;
    double dt;
    const double *traj;         // [1 + kStages * n_step][n_pert][kTrajRec]
    int start_accel;            // 1: form f_0 from record slot 0 (first round); 0: f_0 is in the state
    double *state;              // [15][n_part]: r hi, r lo, v hi, v lo, f
    double *fstore;             // [gridDim][kStages][kPF][kPThreads]: stage accelerations
    const PertInfo *info;
    const double *gp_coef;
    const double *ring_disk;
    int *next;                  // particle-block queue
};

// Shared memory of a CTA (dynamic; every array a multiple of 16 bytes)
struct PartSmem {
    double2 ab[EPH_RK12_NCOEF];
    double X0[12][kPThreads];    // the step's start state: r hi, r lo, v hi, v lo
    double2 zonal[EPH_GP_MAX_DEGREE + 2][2];   // {(2k-1)/k, (k-1)/k}, {(2k-1)/(k-1), k/(k-1)} of the zonal recursion
    double rcp[EPH_GP_MAX_DEGREE + 2];
    int l[EPH_RK12_NCOEF + 3];
    int body[kPMaxPert];         // the perturbers, point-like ones first, then the full-class ones
    int n_point, blk;
    PertInfo info[kPMaxPert];
    double gp_x[kPartGp][kGpX];  // expanded geopotential tables (general form)
    // then: float4 Pf[n_pert][2] (mixed precision), double P[2][n_pert][kTrajRec]
};
constexpr size_t kPartFixed = (sizeof(PartSmem) + 15) / 16 * 16;
size_t part_smem(int n_pert) { return kPartFixed + (size_t)n_pert * (32 + 2 * kTrajRec * sizeof(double)); }

// Field of a purely zonal geopotential (Nt = 0), inline: the Cunningham recursion of gp_core with its two
// columns (m = 0 and m = 1, the only ones zonal terms read) advanced together in one loop over the degree,
// V_k0 for a_z and V_k1 + i W_k1 for a_x, a_y, in a handful of registers, so the particle kernel keeps its
// occupancy when its only extended perturber is zonal:
//   a_z += k J_{k-1} V_k0,  a_x += J_{k-1} V_k1,  a_y += J_{k-1} W_k1   (k - 1 = 2 .. Nz), all / R^2.
// `ir` is 1 / |r|, which the caller has formed already; Z holds the recursion's factors, J {J_n, (n + 1) J_n}.
__device__ __forceinline__ v3 gp_zonal(const double2 *J, const double2 (*Z)[2], int Nz, double R, double inv_r2, v3 r, double ir) {
    if (Nz < 2) return mk(0, 0, 0);
    const double q = R * (ir * ir);
    const double xs = r.x * q, ys = r.y * q, zs = r.z * q, rho2 = R * q, v00 = R * ir;
    double a0 = zs * v00, a0p = v00;     // column 0 at degrees k, k - 1 (from V_10)
    double b1 = xs * v00, c1 = ys * v00; // column 1 (V, W) at degree k = 1 (the diagonal)
    double b1p = 0, c1p = 0;
    double ax = 0, ay = 0, az = 0;
#pragma unroll 1
    for (int k = 2; k <= Nz + 1; ++k) {
        const double2 z0 = Z[k][0], z1 = Z[k][1];
        const double f0 = z0.x * zs, g0 = z0.y * rho2, f1 = z1.x * zs, g1 = z1.y * rho2;
        const double n0 = f0 * a0 - g0 * a0p, nb = f1 * b1 - g1 * b1p, nc = f1 * c1 - g1 * c1p;
        a0p = a0; a0 = n0;
        b1p = b1; b1 = nb;
        c1p = c1; c1 = nc;
        if (k >= 3) {
            const double2 Jn = J[k - 1];
            az += Jn.y * a0;
            ax += Jn.x * b1;
            ay += Jn.x * c1;
        }
    }
    return mk(ax * inv_r2, ay * inv_r2, az * inv_r2);
}

// What a particle's sums over the perturbers start from and add up to.
template <bool kMixed>
struct PartSums {
    dd r[3];
    v3 bi;                  // v / c
    float bfx, bfy, bfz, beta2f;
    double phi = 0, cs = 0;
    v3 na = mk(0, 0, 0), ga = mk(0, 0, 0);
    float gfx = 0, gfy = 0, gfz = 0;
};
struct PairGeom {
    v3 d;
    double q, rr, gm, sr2;
};
// The terms every perturber has (Newtonian + EIH 1PN), added to the sums; returns the pair's geometry.
// The 1PN terms of mass.impl:82-97 are regrouped: the coefficient 4 phi_i + beta_i^2 multiplies the Newtonian sum and is
// applied once after the sweep, and with b = beta_j - beta_i the last term's coefficient is r.beta_j - 4 r.b =
// 4 r.beta_i - 3 r.beta_j =: c, its sum over j sum c beta_j - beta_i sum c (59 FP64 operations a perturber, not 77).
// Nothing in it branches, so two perturbers' chains interleave.
template <bool kMixed>
__device__ __forceinline__ PairGeom pair_terms(const double *P, const float4 *Pf, int j, PartSums<kMixed> &S) {
    const double2 *rec = reinterpret_cast<const double2 *>(P + j * kTrajRec);
    const double2 p0 = rec[0], p1 = rec[1], p2 = rec[2], p3 = rec[3];   // r hi, r lo, GM, sR2
    const v3 d = mk(sep_diff(p0.x, p1.y, S.r[0].hi, S.r[0].lo), sep_diff(p0.y, p2.x, S.r[1].hi, S.r[1].lo),
                    sep_diff(p1.x, p2.y, S.r[2].hi, S.r[2].lo));
    const double q = dot(d, d);
    const double rr = inv_sqrt((q < p3.y) ? p3.y : q);
    const double tp_dphi = rr * p3.x;
    const double tp_dg = (rr * rr) * tp_dphi;
    S.phi -= tp_dphi;                                            // pass A (mass.impl:38-46)
    S.na = mk(fma(tp_dg, d.x, S.na.x), fma(tp_dg, d.y, S.na.y), fma(tp_dg, d.z, S.na.z));
    if (kMixed) {
        const float4 n4 = Pf[2 * j], b4 = Pf[2 * j + 1];   // {a_N, GM}, {beta, K}
        const float dx = (float)d.x, dy = (float)d.y, dz = (float)d.z, rf = (float)rr;
        const float tpf = rf * n4.w, tgf = (rf * rf) * tpf;
        const float rbj = dx * b4.x + dy * b4.y + dz * b4.z;
        float tp = rbj * rf;
        tp *= tp;
        const float delta1 = b4.w + S.beta2f - 4 * (S.bfx * b4.x + S.bfy * b4.y + S.bfz * b4.z) +
                             ((dx * n4.x + dy * n4.y + dz * n4.z) - 3 * tp) / 2;
        const float bx = b4.x - S.bfx, by = b4.y - S.bfy, bz = b4.z - S.bfz;
        const float h = 7 * tpf / 2, w = tgf * delta1, c = tgf * (rbj - (dx * bx + dy * by + dz * bz) * 4);
        S.gfx += h * n4.x + w * dx + c * bx;
        S.gfy += h * n4.y + w * dy + c * by;
        S.gfz += h * n4.z + w * dz + c * bz;
    } else {
        const double2 n0 = rec[4], n1 = rec[5], b1 = rec[6];   // a_N x y, a_N z and beta x, beta y z
        const double K = rec[7].x;
        const double rbj = d.x * n1.y + d.y * b1.x + d.z * b1.y;
        const double rbi = dot(d, S.bi);
        const double rn = d.x * n0.x + d.y * n0.y + d.z * n1.x;
        const double bb = S.bi.x * n1.y + S.bi.y * b1.x + S.bi.z * b1.y;
        double tp = rbj * rr;
        tp *= tp;
        const double w = tp_dg * fma(-1.5, tp, fma(0.5, rn, fma(-4.0, bb, K)));
        const double c = tp_dg * fma(4.0, rbi, -3.0 * rbj);
        const double h = 3.5 * tp_dphi;
        S.cs += c;
        S.ga.x = fma(c, n1.y, fma(w, d.x, fma(h, n0.x, S.ga.x)));
        S.ga.y = fma(c, b1.x, fma(w, d.y, fma(h, n0.y, S.ga.y)));
        S.ga.z = fma(c, b1.y, fma(w, d.z, fma(h, n1.x, S.ga.z)));
    }
    return PairGeom{d, q, rr, p3.x, p3.y};
}

// Acceleration of a particle at (r, v) at the stage whose perturber records are in P: one sweep over the point-like
// perturbers, one over the full-class ones, which deform, spin and carry fields besides.
// kGeneral = false: the fields are zonal geopotentials only (gp_zonal, inline); true: any model (gp_field_columns from
// the expanded tables, else gp_field, and ring_sum: calls, whose register saves cost the kernel some spilling).
// kMixed: the EIH 1PN terms in FP32 from the float records Pf (their sum is ~(v/c)^2 ~ 1e-8 of the
// Newtonian acceleration for solar-system speeds, so FP32 rounding is ~1e-15 of it); the separations, 1/r,
// the Newtonian terms and the deformation and Lense-Thirring terms (which can reach 1e-3 of the Newtonian
// acceleration near an oblate planet) stay FP64.
template <bool kGeneral, bool kMixed>
__device__ __forceinline__ v3 particle_accel(const PartArgs &A, const PartSmem &sm, const double *P, const float4 *Pf,
                                             const dd r[3], v3 v) {
    const int np = A.n_pert;
    const double c2 = kCP * kCP;
    PartSums<kMixed> S;
    for (int c = 0; c < 3; ++c) S.r[c] = r[c];
    S.bi = mk(v.x * (1.0 / kCP), v.y * (1.0 / kCP), v.z * (1.0 / kCP));   // PREPARE_RELATIVITY
    S.bfx = (float)S.bi.x;
    S.bfy = (float)S.bi.y;
    S.bfz = (float)S.bi.z;
    S.beta2f = S.bfx * S.bfx + S.bfy * S.bfy + S.bfz * S.bfz;
    v3 da = mk(0, 0, 0);
#pragma unroll 2
    for (int k = 0; k < sm.n_point; ++k) pair_terms<kMixed>(P, Pf, sm.body[k], S);
    // deformation, spin and fields of the full-class perturbers (mass.impl:99-125, mass.cpp:358-371)
#pragma unroll 1
    for (int k = sm.n_point; k < np; ++k) {
        const int j = sm.body[k];
        const PairGeom g = pair_terms<kMixed>(P, Pf, j, S);
        const PertInfo &in = sm.info[j];
        const double *R = P + j * kTrajRec;
        const v3 d = g.d;
        const double rr2 = g.rr * g.rr, rr3 = g.rr * rr2;
        const v3 b = mk(R[TR_BETA + 0], R[TR_BETA + 1], R[TR_BETA + 2]) - S.bi;
        const m3 Cj = m3{mk(R[TR_CPOT + 0], R[TR_CPOT + 1], R[TR_CPOT + 2]), mk(R[TR_CPOT + 3], R[TR_CPOT + 4], R[TR_CPOT + 5]),
                         mk(R[TR_CPOT + 6], R[TR_CPOT + 7], R[TR_CPOT + 8])};
        const v3 Cjr = mul(Cj, d);
        const double ck = g.gm * rr3 * rr2 * R[TR_R2];
        const double cd = ck * (dot(d, Cjr) * 5 * rr2), cc = -2 * ck;
        const double rcr32 = g.gm * rr3 * (2 / kCP);
        const v3 GLj = mk(R[TR_GL + 0], R[TR_GL + 1], R[TR_GL + 2]);
        const v3 spin = cross(rcr32 * (GLj - (3 * dot(GLj, d) * rr2) * d), b);
        da.x += fma(cd, d.x, fma(cc, Cjr.x, spin.x));
        da.y += fma(cd, d.y, fma(cc, Cjr.y, spin.y));
        da.z += fma(cd, d.z, fma(cc, Cjr.z, spin.z));
        if (in.gp >= 0) {
            const m3 fr = m3{mk(R[TR_FRAME + 0], R[TR_FRAME + 1], R[TR_FRAME + 2]), mk(R[TR_FRAME + 3], R[TR_FRAME + 4], R[TR_FRAME + 5]),
                             mk(R[TR_FRAME + 6], R[TR_FRAME + 7], R[TR_FRAME + 8])};
            const v3 rl = tolocal(fr, -d);   // r = r_particle - r_host (mass.cpp:184,198)
            v3 an;
            if (!kGeneral || in.nt == 0) {
                const double ir = g.sr2 > 0 ? inv_sqrt(g.q) : g.rr;   // the field is not softened
                an = gp_zonal(in.J, sm.zonal, in.nz, R[TR_RADIUS], in.inv_r2, rl, ir);
            } else if (in.gp < kPartGp && gp_fits_columns(in.nz, in.nt)) {
                an = gp_field_columns<kGpColK, kGpColM>(sm.gp_x[in.gp], sm.rcp, R[TR_RADIUS], rl);
            } else {
                an = gp_field(A.gp_coef + (size_t)in.gp * EPH_GP_TABLE_SIZE, in.nz, in.nt, R[TR_RADIUS], rl);
            }
            da += g.gm * toworld(fr, an);
        }
        if (kGeneral && in.ring >= 0) {
            const m3 fr = m3{mk(R[TR_RFRAME + 0], R[TR_RFRAME + 1], R[TR_RFRAME + 2]), mk(R[TR_RFRAME + 3], R[TR_RFRAME + 4], R[TR_RFRAME + 5]),
                             mk(R[TR_RFRAME + 6], R[TR_RFRAME + 7], R[TR_RFRAME + 8])};
            const v3 an = toworld(fr, ring_sum(A.ring_disk + (size_t)in.ring * EPH_RING_MAX_DISKS * 3, in.nd, R[TR_RADIUS],
                                               tolocal(fr, -d)));
            da += g.gm * an;
        }
    }
    const double phi = S.phi * (1.0 / c2);
    v3 ga;
    if (kMixed) ga = mk((double)S.gfx, (double)S.gfy, (double)S.gfz) + (4 * phi) * S.na;
    else ga = (S.ga - S.cs * S.bi) + (4 * phi + dot(S.bi, S.bi)) * S.na;
    return (ga + da) + S.na;
}

// The records of stage slot `slot` into a shared buffer (asynchronous 16-byte copies, one group per call).
__device__ __forceinline__ void fetch_records(const PartArgs &A, double *P, long long slot) {
    const double *src = A.traj + (size_t)slot * A.n_pert * kTrajRec;
    const unsigned to = (unsigned)__cvta_generic_to_shared(P);
    for (int q = threadIdx.x; q < A.n_pert * (kTrajRec / 2); q += kPThreads)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to + 16 * q), "l"(src + 2 * q) : "memory");
    asm volatile("cp.async.commit_group;" ::: "memory");
}
// Waits for the copies in flight; afterwards every thread sees the records, and no thread still reads the
// buffer of the stage before. In mixed precision also forms the float records.
template <bool kMixed>
__device__ __forceinline__ void await_records(const PartArgs &A, const double *P, float4 *Pf) {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    if (kMixed) {
        for (int q = threadIdx.x; q < 2 * A.n_pert; q += kPThreads) {
            const double *R = P + (q >> 1) * kTrajRec;
            Pf[q] = q & 1 ? make_float4((float)R[TR_BETA], (float)R[TR_BETA + 1], (float)R[TR_BETA + 2], (float)R[TR_K])
                          : make_float4((float)R[TR_NACC], (float)R[TR_NACC + 1], (float)R[TR_NACC + 2], (float)R[TR_GM]);
        }
        __syncthreads();
    }
}

// Stage combination in second-order (Runge-Kutta-Nystrom) form. A particle's stage velocities are
// themselves combinations of its stage accelerations, v_j = v0 + dt sum_l a_jl f_l, so
//   sum_j a_kj v_j = c_k v0 + dt sum_l Abar_kl f_l,   Abar = A A (strictly lower triangular),
// and only f_l (3 doubles per stage) is stored: a third of the velocity-and-acceleration store, small enough
// to stay in L2. Stage k < 25 (the columns where a or Abar is not zero, fused multiply-adds):
//   r_k = r0 + dt (c_k v0 + dt sum_l Abar_kl f_l),   v_k = v0 + dt sum_l a_kl f_l,
// r_k as an unnormalised double-double (its low word below two units in the last place of the high one), v_k,
// of which only the rounded value is used, rounded. The state update (row 25) keeps RungeKutta.impl:166-186's
// arithmetic where it sets the result's precision: v = v0 + dt sum_j b_j f_j summed term by term in ascending j over
// nonzero b_j, and r = r0 + dt (sum_j b_j v_j) in double-double with sum_j b_j v_j = c_25 v0 + dt sum_l Abar_25,l f_l. The
// rearranged sums differ from the reference's in rounding at ~1e-16 of the stage increment.
//
// What bounds it: the FP64 pipe (zonal form: about 900 FP64 instructions per particle and stage, 77 % of the pipe's
// rate on an SM that is never idle), so the terms are written for the fewest FP64 operations, a record is read 16
// bytes at a time by broadcast, and the next stage's records arrive by asynchronous copies under the present stage's
// arithmetic. 151552 particles, one step: FP64 412 -> 310 us, mixed 385 -> 293 us against the form with one
// 8-byte load per field, the library's reciprocal square root and all 325 table entries.
template <bool kGeneral, bool kMixed>
__global__ void __launch_bounds__(kPThreads, 2) particle_kernel(PartArgs A) {
    extern __shared__ __align__(16) unsigned char part_raw[];
    PartSmem &sm = *reinterpret_cast<PartSmem *>(part_raw);
    float4 *Pf = reinterpret_cast<float4 *>(part_raw + kPartFixed);
    double *P = reinterpret_cast<double *>(Pf + 2 * A.n_pert);
    const int rec = A.n_pert * kTrajRec;
    const int t = threadIdx.x;
    for (int q = t; q < EPH_RK12_NCOEF; q += kPThreads) { sm.ab[q] = p_ab[q]; sm.l[q] = p_l[q]; }
    for (int k = t; k < EPH_GP_MAX_DEGREE + 2; k += kPThreads) {
        sm.rcp[k] = GP_RCP[k];
        const double kd = k, k1 = k > 1 ? k - 1 : 1;
        sm.zonal[k][0] = make_double2((2 * kd - 1) / (k > 0 ? kd : 1), (kd - 1) / (k > 0 ? kd : 1));
        sm.zonal[k][1] = make_double2((2 * kd - 1) / k1, kd / k1);
    }
    for (int j = t; j < A.n_pert; j += kPThreads) sm.info[j] = A.info[j];
    __syncthreads();
    if (t == 0) {
        int k = 0;
        for (int full = 0; full < 2; ++full) {
            for (int j = 0; j < A.n_pert; ++j)
                if (!!sm.info[j].full == !!full) sm.body[k++] = j;
            if (!full) sm.n_point = k;
        }
    }
    if (kGeneral)
        for (int j = 0; j < A.n_pert; ++j) {
            const PertInfo &in = sm.info[j];
            if (in.gp >= 0 && in.gp < kPartGp)
                gp_expand(A.gp_coef + (size_t)in.gp * EPH_GP_TABLE_SIZE, in.nz, in.nt, sm.gp_x[in.gp], t, kPThreads);
        }
    double (*X0)[kPThreads] = sm.X0;
    double *F = A.fstore + (size_t)blockIdx.x * kStages * kPF * kPThreads + t;   // [stage][3] stride kPThreads
    const int nb = (A.n_part + kPThreads - 1) / kPThreads;
    const double dt = A.dt;
    const dd ddt = dd_make(dt);
    const long long slots = A.n_step * kStages;
#pragma unroll 1
    for (;;) {
        __syncthreads();
        if (t == 0) sm.blk = atomicAdd(A.next, 1);
        __syncthreads();
        const int blk = sm.blk;
        if (blk >= nb) return;
        int buf = 0;
        fetch_records(A, P, A.start_accel ? 0 : 1);
        const int ip = blk * kPThreads + t;
        const bool live = ip < A.n_part;
        const int n = A.n_part;
        v3 fa = mk(0, 0, 0);
        {
            dd r[3], v[3];
            for (int c = 0; c < 3; ++c) {
                r[c] = live ? dd{A.state[(0 + c) * n + ip], A.state[(3 + c) * n + ip]} : dd_make(1e30);
                v[c] = live ? dd{A.state[(6 + c) * n + ip], A.state[(9 + c) * n + ip]} : dd_make(0);
                X0[c][t] = r[c].hi; X0[3 + c][t] = r[c].lo;
                X0[6 + c][t] = v[c].hi; X0[9 + c][t] = v[c].lo;
            }
            if (live) fa = mk(A.state[12 * n + ip], A.state[13 * n + ip], A.state[14 * n + ip]);
            if (A.start_accel) {   // f_0 at the start state (the reference's loader runs accel(), mass_loader.cpp:555)
                await_records<kMixed>(A, P, Pf);
                fetch_records(A, P + rec, 1);
                fa = particle_accel<kGeneral, kMixed>(A, sm, P, Pf, r, mk(dd_val(v[0]), dd_val(v[1]), dd_val(v[2])));
                buf = 1;
            }
        }
        F[0] = fa.x;
        F[kPThreads] = fa.y;
        F[2 * kPThreads] = fa.z;
        int s = 0;
#pragma unroll 1
        for (long long slot = 0; slot < slots; ++slot) {
            const int k = s + 1, q1 = p_row[k + 1];
            double s1[3] = {0.0, 0.0, 0.0}, s2[3] = {0.0, 0.0, 0.0};
            dd r[3];
            v3 v;
            if (k < kStages) {
#pragma unroll 4
                for (int q = p_row[k]; q < q1; ++q) {
                    const double2 ab = sm.ab[q];
                    const double *Fl = F + sm.l[q];
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        const double f = Fl[c * kPThreads];
                        s1[c] = __fma_rn(ab.x, f, s1[c]);
                        s2[c] = __fma_rn(ab.y, f, s2[c]);
                    }
                }
                const double ck = p_c[k];
                double vc[3];
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    const double v0 = X0[6 + c][t];
                    double e;
                    two_sum(X0[c][t], dt * __fma_rn(ck, v0, dt * s1[c]), r[c].hi, e);
                    r[c].lo = e + X0[3 + c][t];
                    vc[c] = v0 + __fma_rn(dt, s2[c], X0[9 + c][t]);
                }
                v = mk(vc[0], vc[1], vc[2]);
                s = k;
            } else {
#pragma unroll 1
                for (int q = p_row[k]; q < q1; ++q) {
                    const double2 ab = sm.ab[q];
                    const double *Fl = F + sm.l[q];
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        const double f = Fl[c * kPThreads];
                        s1[c] = __fma_rn(ab.x, f, s1[c]);
                        if (ab.y != 0) s2[c] = __dadd_rn(s2[c], __dmul_rn(ab.y, f));
                    }
                }
                const dd c25 = dd_make(p_c[k]);
                double vc[3];
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    const dd v0 = dd{X0[6 + c][t], X0[9 + c][t]};
                    const dd sv = dd_add(dd_mul(c25, v0), dd_make(dt * s1[c]));
                    r[c] = dd_add(dd{X0[c][t], X0[3 + c][t]}, dd_mul(ddt, sv));
                    const dd vn = dd_add(v0, dd_make(dt * s2[c]));
                    X0[c][t] = r[c].hi; X0[3 + c][t] = r[c].lo;
                    X0[6 + c][t] = vn.hi; X0[9 + c][t] = vn.lo;
                    vc[c] = dd_val(vn);
                }
                v = mk(vc[0], vc[1], vc[2]);
                s = 0;   // the new state is stage 0 of the next step
            }
            await_records<kMixed>(A, P + buf * rec, Pf);
            if (slot + 1 < slots) fetch_records(A, P + (buf ^ 1) * rec, slot + 2);
            fa = particle_accel<kGeneral, kMixed>(A, sm, P + buf * rec, Pf, r, v);
            buf ^= 1;
            double *Fk = F + (size_t)s * kPF * kPThreads;
            Fk[0] = fa.x;
            Fk[kPThreads] = fa.y;
            Fk[2 * kPThreads] = fa.z;
        }
        if (live) {
            for (int c = 0; c < 3; ++c) {
                A.state[(0 + c) * n + ip] = X0[c][t];
                A.state[(3 + c) * n + ip] = X0[3 + c][t];
                A.state[(6 + c) * n + ip] = X0[6 + c][t];
                A.state[(9 + c) * n + ip] = X0[9 + c][t];
            }
            A.state[12 * n + ip] = fa.x;
            A.state[13 * n + ip] = fa.y;
            A.state[14 * n + ip] = fa.z;
        }
    }
}

using PartKernel = void (*)(PartArgs);
PartKernel kernel_of(bool general, bool mixed) {
    return general ? (mixed ? particle_kernel<true, true> : particle_kernel<true, false>)
                   : (mixed ? particle_kernel<false, true> : particle_kernel<false, false>);
}

bool g_part_ready[64];
cudaError_t particles_setup(int device) {
    if (device >= 0 && device < 64 && g_part_ready[device]) return cudaSuccess;
    double hi[EPH_RK12_NCOEF], lo[EPH_RK12_NCOEF], dtk[kStages + 1];
    rk12_expand(hi, lo, dtk);
    // Abar_kl = sum_{l<j<k} a_kj a_jl, accumulated in long double from the double-double coefficients
    auto coef = [&](int k, int j) { return (long double)hi[k * (k - 1) / 2 + j] + lo[k * (k - 1) / 2 + j]; };
    double2 ab[EPH_RK12_NCOEF] = {};
    int ll[EPH_RK12_NCOEF] = {}, row[kStages + 2] = {}, q = 0;
    for (int k = 1; k <= kStages; ++k) {
        row[k] = q;
        for (int l = 0; l < k; ++l) {
            long double acc = 0;
            bool any = hi[k * (k - 1) / 2 + l] != 0;
            for (int j = l + 1; j < k; ++j) {
                acc += coef(k, j) * coef(j, l);
                any = any || (hi[k * (k - 1) / 2 + j] != 0 && hi[j * (j - 1) / 2 + l] != 0);
            }
            if (!any) continue;
            ab[q] = make_double2((double)acc, hi[k * (k - 1) / 2 + l] + lo[k * (k - 1) / 2 + l]);
            ll[q++] = l * kPF * kPThreads;
        }
    }
    row[kStages + 1] = q;
    cudaError_t e = cudaMemcpyToSymbol(p_ab, ab, sizeof(ab));
    if (e == cudaSuccess) e = cudaMemcpyToSymbol(p_l, ll, sizeof(ll));
    if (e == cudaSuccess) e = cudaMemcpyToSymbol(p_row, row, sizeof(row));
    for (int g = 0; g < 4 && e == cudaSuccess; ++g)
        e = cudaFuncSetAttribute(kernel_of(g & 1, g & 2), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)part_smem(kPMaxPert));
    if (e == cudaSuccess) e = cudaMemcpyToSymbol(p_c, dtk, sizeof(dtk));
    if (e == cudaSuccess && device >= 0 && device < 64) g_part_ready[device] = true;
    return e;
}

}  // namespace
}  // namespace eph

using namespace eph;

struct eph_particles {
    int device = 0;
    cudaStream_t stream = nullptr;     // work stream (own_stream unless eph_particles_set_stream chose another)
    cudaStream_t own_stream = nullptr;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr, ev_begin = nullptr;
    int64_t launches = 0;              // kernels launched (step kernel, particle kernel)
    double kernel_ms = 0;              // particle_kernel device time, summed
    std::mutex mu;
    char err[512] = {0};
    eph_ctx *ctx = nullptr;            // the perturbers
    eph_ctx *ctx0 = nullptr;           // scratch context for the start-state records
    int64_t n_pert = 0, n_part = 0;
    std::vector<double> h_pert;        // perturber planes as uploaded (for the start-state records)
    std::vector<int32_t> gp_nz, gp_nt, ring_nd;
    std::vector<double> gp_coef, ring_param, ring_disk;
    bool started = false;              // f_0 of the particles formed
    double *d_state = nullptr, *d_traj[2] = {nullptr, nullptr}, *d_fstore = nullptr;   // (records of two rounds)
    int *d_next = nullptr;
    double *d_gp_coef = nullptr, *d_ring_disk = nullptr;
    PertInfo *d_info = nullptr;
    size_t traj_cap = 0;
    int grid = 0;
    int64_t cap_part = 0, cap_pert = 0;  // sizes the device buffers hold
    int cap_grid = 0, cap_gp = 0, cap_ring = 0;
    bool general = false;              // a tesseral geopotential or a ring among the perturbers
    bool mixed = false;                // EPH_PREC_MIXED
};

static int pfail(eph_particles *p, int code, const char *what, cudaError_t e = cudaSuccess) {
    if (p) {
        if (e != cudaSuccess) snprintf(p->err, sizeof(p->err), "%s: %s", what, cudaGetErrorString(e));
        else snprintf(p->err, sizeof(p->err), "%s", what);
    }
    return code;
}
#define PCK(call, what)                                                                                     \
    do {                                                                                                    \
        cudaError_t e_ = (call);                                                                            \
        if (e_ != cudaSuccess) return pfail(p, e_ == cudaErrorMemoryAllocation ? EPH_ERR_OOM : EPH_ERR_CUDA, what, e_); \
    } while (0)

static void part_free(eph_particles *p) {
    for (void *q : {(void *)p->d_state, (void *)p->d_traj[0], (void *)p->d_traj[1], (void *)p->d_fstore, (void *)p->d_next, (void *)p->d_gp_coef,
                    (void *)p->d_ring_disk, (void *)p->d_info})
        if (q) cudaFree(q);
    p->d_state = p->d_traj[0] = p->d_traj[1] = p->d_fstore = nullptr;
    p->d_next = nullptr;
    p->d_gp_coef = p->d_ring_disk = nullptr;
    p->d_info = nullptr;
    p->traj_cap = 0;
    p->cap_part = p->cap_pert = 0;
    p->cap_grid = p->cap_gp = p->cap_ring = 0;
}

// t += d in double-double (mass.cpp:441)
static void dd_advance(double *hi, double *lo, double d) {
    const double a = *hi, s = a + d, t = s - a;
    double e = (a - (s - t)) + (d - t);
    e = e + (*lo + 0.0);
    const double h = s + e;
    *lo = e - (h - s);
    *hi = h;
}

extern "C" {

int eph_particles_create(int device, eph_particles **out) {
    if (!out) return EPH_ERR_ARG;
    *out = nullptr;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || device < 0 || device >= ndev) return EPH_ERR_ARG;
    eph_particles *p = new eph_particles();
    p->device = device;
    if (cudaSetDevice(device) != cudaSuccess || cudaStreamCreateWithFlags(&p->own_stream, cudaStreamNonBlocking) != cudaSuccess ||
        cudaEventCreate(&p->ev0) != cudaSuccess || cudaEventCreate(&p->ev1) != cudaSuccess ||
        cudaEventCreateWithFlags(&p->ev_begin, cudaEventDisableTiming) != cudaSuccess ||
        particles_setup(device) != cudaSuccess || eph_ctx_create(device, &p->ctx) != EPH_OK ||
        eph_ctx_create(device, &p->ctx0) != EPH_OK) {
        eph_particles_destroy(p);
        return EPH_ERR_CUDA;
    }
    p->stream = p->own_stream;
    *out = p;
    return EPH_OK;
}

int eph_particles_destroy(eph_particles *p) {
    if (!p) return EPH_ERR_ARG;
    cudaSetDevice(p->device);
    part_free(p);
    if (p->ctx) eph_ctx_destroy(p->ctx);
    if (p->ctx0) eph_ctx_destroy(p->ctx0);
    if (p->ev0) cudaEventDestroy(p->ev0);
    if (p->ev1) cudaEventDestroy(p->ev1);
    if (p->ev_begin) cudaEventDestroy(p->ev_begin);
    if (p->own_stream) cudaStreamDestroy(p->own_stream);
    delete p;
    return EPH_OK;
}

const char *eph_particles_last_error(const eph_particles *p) { return p ? p->err : "null particle set"; }

int eph_particles_set_stream(eph_particles *p, void *stream) {
    if (!p) return EPH_ERR_ARG;
    std::lock_guard<std::mutex> lock(p->mu);
    // the perturbers keep a stream of their own, ordered after this one by an event: they run beside the particles
    p->stream = stream ? (cudaStream_t)stream : p->own_stream;
    return eph_set_stream(p->ctx0, stream);
}

int eph_particles_set_precision(eph_particles *p, int mode) {
    if (!p || (mode != EPH_PREC_FP64 && mode != EPH_PREC_MIXED)) return pfail(p, EPH_ERR_ARG, "bad precision mode");
    std::lock_guard<std::mutex> lock(p->mu);
    p->mixed = mode == EPH_PREC_MIXED;
    return EPH_OK;
}

int eph_particles_info(const eph_particles *p, int64_t *launches, double *particle_kernel_ms) {
    if (!p || !launches || !particle_kernel_ms) return EPH_ERR_ARG;
    *launches = p->launches;
    *particle_kernel_ms = p->kernel_ms;
    return EPH_OK;
}

int eph_particles_upload(eph_particles *p, int64_t n_pert, const double *pert_planes, const eph_models *models,
                         int64_t n_part, const double *part_state) {
    if (!p || n_pert <= 0 || n_pert > kPMaxPert || !pert_planes || n_part <= 0 || n_part > (1ll << 31) / 16 || !part_state)
        return pfail(p, n_pert > kPMaxPert ? EPH_ERR_LIMIT : EPH_ERR_ARG, "eph_particles_upload: bad arguments");
    std::lock_guard<std::mutex> lock(p->mu);
    PCK(cudaSetDevice(p->device), "cudaSetDevice");
    int rc = eph_upload_system(p->ctx, n_pert, pert_planes, models);
    if (rc) return pfail(p, rc, eph_last_error(p->ctx));
    p->n_pert = n_pert;
    p->n_part = n_part;
    p->h_pert.assign(pert_planes, pert_planes + (size_t)EPH_NPLANES * n_pert);
    const int n_gp = models ? models->n_gp : 0, n_ring = models ? models->n_ring : 0;
    p->gp_nz.assign(n_gp ? models->gp_nz : nullptr, n_gp ? models->gp_nz + n_gp : nullptr);
    p->gp_nt.assign(n_gp ? models->gp_nt : nullptr, n_gp ? models->gp_nt + n_gp : nullptr);
    p->gp_coef.assign(n_gp ? models->gp_coef : nullptr, n_gp ? models->gp_coef + (size_t)n_gp * EPH_GP_TABLE_SIZE : nullptr);
    p->ring_nd.assign(n_ring ? models->ring_ndisk : nullptr, n_ring ? models->ring_ndisk + n_ring : nullptr);
    p->ring_param.assign(n_ring ? models->ring_param : nullptr, n_ring ? models->ring_param + (size_t)n_ring * 4 : nullptr);
    p->ring_disk.assign(n_ring ? models->ring_disk : nullptr,
                        n_ring ? models->ring_disk + (size_t)n_ring * EPH_RING_MAX_DISKS * 3 : nullptr);
    std::vector<PertInfo> info(n_pert);
    for (int j = 0; j < n_pert; ++j) {
        auto P = [&](int q) { return pert_planes[(size_t)q * n_pert + j]; };
        info[j].gp = (int)P(EPH_P_GP_INDEX);
        info[j].ring = (int)P(EPH_P_RING_INDEX);
        bool full = P(EPH_P_K2) != 0 || P(EPH_P_K2R) != 0 || P(EPH_P_DJ2) != 0 || P(EPH_P_LUM) != 0 ||
                    P(EPH_P_RR2G_4C) != 0 || info[j].gp >= 0 || info[j].ring >= 0;
        for (int q = 0; q < 9; ++q) full = full || P(EPH_P_C_STATIC + q) != 0;
        for (int c = 0; c < 3; ++c) full = full || P(EPH_P_W + c) != 0 || P(EPH_P_GL_HI + c) != 0 || P(EPH_P_GL_LO + c) != 0;
        info[j].full = full;
        const int g = info[j].gp, rg = info[j].ring;
        info[j].nz = g >= 0 ? models->gp_nz[g] : 0;
        info[j].nt = g >= 0 ? models->gp_nt[g] : 0;
        info[j].nd = rg >= 0 ? models->ring_ndisk[rg] : 0;
        info[j].inv_r2 = 1.0 / (P(EPH_P_RADIUS) * P(EPH_P_RADIUS));
        for (int q = 0; q <= EPH_GP_MAX_DEGREE; ++q) {
            const double J = g >= 0 && q >= 2 && q <= info[j].nz ? models->gp_coef[(size_t)g * EPH_GP_TABLE_SIZE + q * q - 4] : 0.0;
            info[j].J[q] = make_double2(J, (q + 1) * J);
        }
    }
    int per_sm = 0, sms = 0;
    p->general = false;
    for (int j = 0; j < n_pert; ++j)
        p->general = p->general || info[j].ring >= 0 || (info[j].gp >= 0 && p->gp_nt[info[j].gp] > 0);
    PCK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel_of(p->general, p->mixed), kPThreads, part_smem((int)n_pert)),
        "occupancy");
    PCK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, p->device), "SM count");
    const int64_t nblk = (n_part + kPThreads - 1) / kPThreads;
    p->grid = (int)std::max<int64_t>(1, std::min<int64_t>(nblk, (int64_t)per_sm * sms));
    // device buffers are kept across uploads while they are large enough (a repeated upload of the same
    // sizes allocates nothing)
    if (n_part > p->cap_part || p->grid > p->cap_grid || n_pert > p->cap_pert || std::max(n_gp, 1) > p->cap_gp ||
        std::max(n_ring, 1) > p->cap_ring) {
        part_free(p);
        p->cap_part = n_part;
        p->cap_grid = p->grid;
        p->cap_pert = n_pert;
        p->cap_gp = std::max(n_gp, 1);
        p->cap_ring = std::max(n_ring, 1);
        PCK(cudaMalloc(&p->d_state, (size_t)15 * n_part * sizeof(double)), "cudaMalloc(particles)");
        PCK(cudaMalloc(&p->d_fstore, (size_t)p->grid * kStages * kPF * kPThreads * sizeof(double)), "cudaMalloc(stage store)");
        PCK(cudaMalloc(&p->d_info, n_pert * sizeof(PertInfo)), "cudaMalloc(perturbers)");
        PCK(cudaMalloc(&p->d_next, sizeof(int)), "cudaMalloc(queue)");
        PCK(cudaMalloc(&p->d_gp_coef, (size_t)p->cap_gp * EPH_GP_TABLE_SIZE * sizeof(double)), "cudaMalloc(gp)");
        PCK(cudaMalloc(&p->d_ring_disk, (size_t)p->cap_ring * EPH_RING_MAX_DISKS * 3 * sizeof(double)), "cudaMalloc(ring)");
    }
    // particle state [15][n_part]: r hi, r lo, v hi, v lo straight from the caller's rows (a pinned caller
    // buffer is a DMA), then f, formed at the first integration
    PCK(cudaMemcpyAsync(p->d_state, part_state, (size_t)12 * n_part * sizeof(double), cudaMemcpyHostToDevice, p->stream),
        "upload particles");
    PCK(cudaMemsetAsync(p->d_state + (size_t)12 * n_part, 0, (size_t)3 * n_part * sizeof(double), p->stream), "clear f");
    PCK(cudaStreamSynchronize(p->stream), "upload particles");
    PCK(cudaMemcpy(p->d_info, info.data(), n_pert * sizeof(PertInfo), cudaMemcpyHostToDevice), "upload perturbers");
    if (n_gp) {
        PCK(cudaMemcpy(p->d_gp_coef, p->gp_coef.data(), p->gp_coef.size() * sizeof(double), cudaMemcpyHostToDevice), "upload gp");
    }
    if (n_ring) {
        PCK(cudaMemcpy(p->d_ring_disk, p->ring_disk.data(), p->ring_disk.size() * sizeof(double), cudaMemcpyHostToDevice),
            "upload ring");
    }
    p->started = false;
    return EPH_OK;
}

int eph_particles_integrate(eph_particles *p, double dt, int64_t n_step, double *t_eph_hi, double *t_eph_lo) {
    if (!p || !t_eph_hi || !t_eph_lo) return pfail(p, EPH_ERR_ARG, "eph_particles_integrate: bad arguments");
    std::lock_guard<std::mutex> lock(p->mu);
    if (!p->n_part) return pfail(p, EPH_ERR_STATE, "no particles uploaded");
    if (n_step == 0) return EPH_OK;
    if (n_step < 0) {   // mass.cpp:401-404
        n_step = -n_step;
        dt = -dt;
    }
    PCK(cudaSetDevice(p->device), "cudaSetDevice");
    const size_t rec = (size_t)p->n_pert * kTrajRec;
    // Rounds: the perturbers of a round run beside the particles of the round before, so only the first round of
    // perturbers is waited for. 10 steps of 9 perturbers and a million particles: 4 ms of perturbers, 18 of particles.
    const int64_t fits = std::max<int64_t>(1, (int64_t)(kPRecordBytes / (sizeof(double) * kStages * rec)));
    const int64_t chunk = std::min<int64_t>(fits, std::max<int64_t>(1, std::min<int64_t>(kPRoundSteps, n_step / kPRounds)));
    const size_t need = (size_t)(1 + kStages * std::min<int64_t>(n_step, chunk)) * rec;
    if (need > p->traj_cap) {
        p->traj_cap = 0;
        for (double *&d : p->d_traj) {
            if (d) cudaFree(d);
            d = nullptr;
            PCK(cudaMalloc(&d, need * sizeof(double)), "cudaMalloc(stage records)");
        }
        p->traj_cap = need;
    }
    int rc;
    if (!p->started) {
        // the perturbers' records at the start state (slot 0), from a scratch copy so that their own
        // integration starts exactly from the uploaded state
        eph_models m{};
        m.n_gp = (int32_t)p->gp_nz.size();
        m.gp_nz = p->gp_nz.data(); m.gp_nt = p->gp_nt.data(); m.gp_coef = p->gp_coef.data();
        m.n_ring = (int32_t)p->ring_nd.size();
        m.ring_ndisk = p->ring_nd.data(); m.ring_param = p->ring_param.data(); m.ring_disk = p->ring_disk.data();
        rc = eph_upload_system(p->ctx0, p->n_pert, p->h_pert.data(), &m);
        ctx_record_stages(p->ctx0, p->d_traj[0], 0);
        if (!rc) rc = eph_accel(p->ctx0);
        ctx_record_stages(p->ctx0, nullptr, 0);
        ++p->launches;
        if (rc) return pfail(p, rc, eph_last_error(p->ctx0));
    }
    // msystem::integrate: maxima reset before, min_distance inverted after (mass.cpp:406,436)
    double *d_pl = nullptr;
    eph_device_planes(p->ctx, &d_pl);
    // On the set's stream, which the perturbers' stream waits for: nothing orders the default stream before either.
    PCK(cudaMemsetAsync(d_pl + (size_t)EPH_P_MIN_DISTANCE * p->n_pert, 0, 2 * p->n_pert * sizeof(double), p->stream), "reset maxima");
    PCK(cudaEventRecord(p->ev_begin, p->stream), "event");
    double th = *t_eph_hi, tl = *t_eph_lo;   // time at the start of the next round of perturbers
    // A round of perturbers on the context's stream: begin launches it, end waits for it. No way out of this function
    // leaves one in flight, or the context recording.
    struct Round {
        eph_ctx *ctx;
        bool open = false;
        int end() {
            open = false;
            const int r = ctx_rk12_end(ctx);
            ctx_record_stages(ctx, nullptr, 0);
            return r;
        }
        ~Round() {
            if (open) end();
        }
    } pert{p->ctx};
    auto begin = [&](int64_t steps, double *traj) {
        ctx_record_stages(p->ctx, traj, 1);
        pert.open = true;
        const int r = ctx_rk12_begin(p->ctx, dt, steps, th + tl, p->ev_begin);
        if (r) return r;
        ++p->launches;
        dd_advance(&th, &tl, dt * (double)steps);
        return (int)EPH_OK;
    };
    int64_t ready = std::min<int64_t>(n_step, chunk);   // steps of the round whose records are complete
    rc = begin(ready, p->d_traj[0]);
    if (!rc) rc = pert.end();
    if (rc) return pfail(p, rc, eph_last_error(p->ctx));
    for (int64_t done = 0, round = 0; done < n_step; ++round) {
        const int64_t next = std::min<int64_t>(n_step - done - ready, chunk);
        // the next round of perturbers first: its CTAs need an SM each, which the particle kernel would fill
        if (next > 0 && (rc = begin(next, p->d_traj[(round + 1) & 1]))) return pfail(p, rc, eph_last_error(p->ctx));
        PartArgs A;
        A.n_part = (int)p->n_part;
        A.n_pert = (int)p->n_pert;
        A.n_step = ready;
        A.dt = dt;
        A.traj = p->d_traj[round & 1];
        A.start_accel = p->started ? 0 : 1;
        A.state = p->d_state;
        A.fstore = p->d_fstore;
        A.info = p->d_info;
        A.gp_coef = p->d_gp_coef;
        A.ring_disk = p->d_ring_disk;
        A.next = p->d_next;
        PCK(cudaMemsetAsync(p->d_next, 0, sizeof(int), p->stream), "reset queue");
        PCK(cudaEventRecord(p->ev0, p->stream), "event");
        PCK(launch_kernel(kernel_of(p->general, p->mixed), p->grid, kPThreads, part_smem((int)p->n_pert), p->stream, A),
            "launch particle kernel");
        ++p->launches;
        PCK(cudaEventRecord(p->ev1, p->stream), "event");
        rc = next > 0 ? pert.end() : (int)EPH_OK;
        PCK(cudaStreamSynchronize(p->stream), "particle kernel");
        float ms = 0;
        PCK(cudaEventElapsedTime(&ms, p->ev0, p->ev1), "event time");
        p->kernel_ms += ms;
        p->started = true;
        dd_advance(t_eph_hi, t_eph_lo, dt * (double)ready);   // the particles' time; a round that fails later leaves it
        if (rc) return pfail(p, rc, eph_last_error(p->ctx));
        done += ready;
        ready = next;
    }
    std::vector<double> md(p->n_pert);
    double *d_md = d_pl + (size_t)EPH_P_MIN_DISTANCE * p->n_pert;
    PCK(cudaMemcpyAsync(md.data(), d_md, md.size() * sizeof(double), cudaMemcpyDeviceToHost, p->stream), "maxima");
    PCK(cudaStreamSynchronize(p->stream), "maxima");
    for (auto &x : md) x = 1 / x;
    PCK(cudaMemcpyAsync(d_md, md.data(), md.size() * sizeof(double), cudaMemcpyHostToDevice, p->stream), "maxima");
    PCK(cudaStreamSynchronize(p->stream), "maxima");
    return EPH_OK;
}

int eph_particles_download(eph_particles *p, double *pert_planes, double *part_state) {
    if (!p) return EPH_ERR_ARG;
    std::lock_guard<std::mutex> lock(p->mu);
    if (!p->n_part) return pfail(p, EPH_ERR_STATE, "no particles uploaded");
    PCK(cudaSetDevice(p->device), "cudaSetDevice");
    if (pert_planes) {
        const int rc = eph_download_system(p->ctx, pert_planes);
        if (rc) return pfail(p, rc, eph_last_error(p->ctx));
    }
    if (part_state) {
        PCK(cudaMemcpyAsync(part_state, p->d_state, (size_t)12 * p->n_part * sizeof(double), cudaMemcpyDeviceToHost,
                            p->stream), "download particles");
        PCK(cudaStreamSynchronize(p->stream), "download particles");
    }
    return EPH_OK;
}

}  // extern "C"
