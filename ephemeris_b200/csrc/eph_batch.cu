// eph_batch.cu - batched ensembles: many independent systems integrated in one call.
//
// Each system runs the reference's msystem::integrate (mass.cpp:399-442) on its own dt, step count and
// ephemeris time. Systems whose bodies are all point-like (no tide, rotational deformation, static
// harmonics, spin, luminosity, radiation receptance, geopotential or ring: the Newtonian + 1PN systems of
// an ensemble) run in `ensemble_kernel`: a system is integrated by one CTA, or by the CTAs of one thread-block
// cluster, so a stage needs only CTA or cluster barriers, and persistent CTAs take systems from an atomic
// queue, longest first. The bodies' stage data, and the stage accelerations where they fit, sit in shared memory.
// Any other system of the batch (a full-physics body, or more bodies than shared memory holds) is integrated by
// the per-system persistent kernel of eph_step.cu through a context, one after another.
//
// Physics per pair (the point-class branches of the reference):
//   pass A  phi_i -= GM_j / r, a_N,i += GM_j r / r^3, r^2 floored at sR2_i + sR2_j
//           (DAMPED_TIDAL_DEFORMATION_MATRIX_NK2, mass.impl:38-46)
//   prepare beta = v / c, beta^2, phi / c^2, a_N / c^2 (PREPARE_RELATIVITY, mass.impl:76-80)
//   pass B  EIH 1PN (RELATIVITY, mass.impl:82-97) and the per-pair maxima of 1/r and GM_j/r^3
//           (RungeKutta.cu:229-230), recomputed exactly for the extremal pair; in the mixed-precision form
//           (eph_batch_set_precision) the 1PN terms in FP32 (sweep_point_b32)
//   final   phi c^2, a_N c^2 (FINALIZE_RELATIVITY, mass.impl:133-135); f = (gaccel + daccel) + naccel
// For such bodies the reference's angular velocity, G*L and harmonics stay constant (w = G*L = 0), the
// frame rotations are the identity and only the end-of-step orthogonalisation of the frame acts
// (mass.h:147-150); the RK12 combination is RungeKutta.impl:148-186 in second-order form (integrate_system).
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <numeric>
#include <vector>

#include "eph_math.cuh"
#include "eph_plan.h"
#include "eph_rk12_host.h"
#include "eph_share.h"
#include "eph_system.cuh"
#include "../../include/eph_b200.h"
#include "../../include/eph_planes.h"

namespace eph {
namespace {

constexpr double kCB = 299792458.0;     // src/math/basic_math.h:10,18

// The Feagin table in second-order form: v_j = v0 + dt sum_l a_jl f_l, so sum_j a_kj v_j = c_k v0 +
// dt sum_l Abar_kl f_l with Abar = A A. Entry k(k-1)/2 + l: Abar_kl as hi + lo, a_kl rounded. The CTAs read the
// entries from shared memory: the rows are walked whole (a zero entry adds nothing), so no load depends on another.
__constant__ double b_ab_hi[EPH_RK12_NCOEF];
__constant__ double b_ab_lo[EPH_RK12_NCOEF];
__constant__ double b_a[EPH_RK12_NCOEF];
__constant__ double b_ck_hi[kStages + 1];   // c_k = sum_j a_kj, hi + lo
__constant__ double b_ck_lo[kStages + 1];
__constant__ double b_dtk[kStages + 1];     // c_k as the reference sums it (stage times)
struct RkTable {
    double2 ab[EPH_RK12_NCOEF];   // {Abar hi, a}
    double lo[EPH_RK12_NCOEF];    // Abar lo
};
static_assert(sizeof(RkTable) == kRkTableBytes, "static shared memory that eph_share.h leaves room for");

struct BatchSys {
    int n;                // bodies
    int split;            // parts that a body's j range is cut into (batch_split)
    long long n_step;     // steps (>= 1)
    double dt;            // signed step
    double t_eph;         // double(t_eph) at the start
    int accumulate;       // eph_rk12: the maxima go on from the planes' and min_distance is not inverted
    int whole;            // also write what stays constant for such bodies (harmonics, moments of inertia, J2 change)
    double *planes;       // [EPH_NPLANES][n], in and out
    double *store;        // [kStore][n] stage accelerations and start-of-step state, when shared memory has no room
};

// One CTA's share of a system: the bodies [lo, lo + cnt) of n, and its shared memory. Every CTA of a cluster has
// the same layout for the arrays that its peers write (A, and what pass B reads of all bodies: B, or F in mixed
// precision).
struct View {
    double *A[2];    // [n][kRecA], by stage parity when shared by a cluster (else the same array twice)
    double *B;       // [kRecB] records, of all bodies (FP64) or of the own bodies (mixed precision), from body b0
    float *F;        // [n][kRecF] (mixed precision only)
    double *own;     // [kOwnRows][cnt]
    double *part;    // [kPartB][split * cnt] sums of the (body, part) units
    double *store;   // [kStore] rows `ld` apart, own bodies from 0: f_l component c at row 3 l + c, then r0, v0
    int ld;
    int n, lo, cnt, b0;
    int split;       // parts of a body's j range
};
__device__ __forceinline__ double &own_row(const View &V, int r, int b) { return V.own[r * V.cnt + b]; }
__device__ __forceinline__ double *rec_b(const View &V, int i) { return V.B + (size_t)(i - V.b0) * kRecB; }

template <bool MIXED>
__device__ __forceinline__ View make_view(const BatchSys &Y, double *smem, int lo, int cnt, int peers) {
    const bool coop = peers > 1;
    const int n = Y.n;
    View V;
    V.n = n; V.lo = lo; V.cnt = cnt; V.split = Y.split;
    double *p = smem;   // every array a multiple of 16 bytes
    V.A[0] = p; p += (size_t)n * kRecA;
    V.A[1] = coop ? p : smem; p += coop ? (size_t)n * kRecA : 0;
    V.F = reinterpret_cast<float *>(p); p += MIXED ? (size_t)n * (kRecF / 2) : 0;
    V.b0 = MIXED ? lo : 0;
    V.B = p; p += (size_t)(MIXED ? cnt : n) * kRecB;
    V.part = p; p += (size_t)cnt * V.split * kPartB;
    V.own = p; p += (size_t)cnt * kOwnRows;
    bool in_smem;
    batch_smem_doubles(n, peers, Y.split, MIXED, &in_smem);
    V.store = in_smem ? p : Y.store + lo;
    V.ld = in_smem ? cnt : n;
    return V;
}

struct BodyA {   // a body's stage state
    double hx, hy, hz, lx, ly, lz, gm, sr2;
};
__device__ __forceinline__ BodyA load_a(const double *A, int i) {
    const double2 *p = reinterpret_cast<const double2 *>(A + (size_t)i * kRecA);
    const double2 a = p[0], b = p[1], c = p[2], d = p[3];
    return BodyA{a.x, a.y, b.x, b.y, c.x, c.y, d.x, d.y};
}
__device__ __forceinline__ v3 separation(const BodyA &j, const BodyA &i) {
    return mk(sep_diff(j.hx, j.lx, i.hx, i.lx), sep_diff(j.hy, j.ly, i.hy, i.ly), sep_diff(j.hz, j.lz, i.hz, i.lz));
}

// pass A over j in [j0, j1): s = {phi, a_N}. The body itself takes part with GM = 0 at unit distance, so the
// loop has no branch that differs between lanes.
__device__ __forceinline__ void sweep_point_a(const double *A, int i, int j0, int j1, double s[kPartA]) {
    const BodyA bi = load_a(A, i);
    s[0] = s[1] = s[2] = s[3] = 0;
#pragma unroll 2
    for (int j = j0; j < j1; ++j) {
        const BodyA bj = load_a(A, j);
        const v3 r = separation(bj, bi);
        const double q = dot(r, r), sm = bi.sr2 + bj.sr2;
        const double m = (q < sm) ? sm : q;
        const double rr = inv_sqrt(j == i ? 1.0 : m);
        const double tp_dphi = rr * (j == i ? 0.0 : bj.gm);
        const double tp_dg = (rr * rr) * tp_dphi;
        s[0] -= tp_dphi;
        s[1] += tp_dg * r.x;
        s[2] += tp_dg * r.y;
        s[3] += tp_dg * r.z;
    }
}

// pass B over j in [j0, j1): s = {EIH 1PN acceleration less the terms common to all j, smallest floored r^2,
// largest GM_j/r^3 and its j}. mass.impl:82-97 with the sums over j regrouped: the coefficient 4 phi_i + beta_i^2
// multiplies the Newtonian sum that pass A has formed already (point_b_common adds it), and with b = beta_j -
// beta_i the last term's coefficient is r.beta_j - 4 r.b = 4 r.beta_i - 3 r.beta_j =: c, its sum over j
// sum c beta_j - beta_i sum c: 57 FP64 operations and a reciprocal square root per pair, not 77.
__device__ __forceinline__ void sweep_point_b(const double *A, const double *B, int i, int j0, int j1, double s[kPartB]) {
    const BodyA bi = load_a(A, i);
    const double2 *pi = reinterpret_cast<const double2 *>(B + (size_t)i * kRecB);
    const double bix = pi[1].y, biy = pi[2].x, biz = pi[2].y;
    double gx = 0, gy = 0, gz = 0, cs = 0;
    double m_min = __longlong_as_double(0x7ff0000000000000ll), tq = 0;
    int tj = -1;
#pragma unroll 2
    for (int j = j0; j < j1; ++j) {
        const BodyA bj = load_a(A, j);
        const double2 *pj = reinterpret_cast<const double2 *>(B + (size_t)j * kRecB);
        const double2 p0 = pj[0], p1 = pj[1], p2 = pj[2];
        const double K = pj[3].x;
        const double nx = p0.x, ny = p0.y, nz = p1.x, bx = p1.y, by = p2.x, bz = p2.y;
        const v3 r = separation(bj, bi);
        const double q = dot(r, r), sm = bi.sr2 + bj.sr2;
        const double m = (q < sm) ? sm : q;
        const double rr = inv_sqrt(j == i ? 1.0 : m);
        const double tp_dphi = rr * (j == i ? 0.0 : bj.gm);
        const double tp_dg = (rr * rr) * tp_dphi;
        if (m < m_min && j != i) m_min = m;
        if (tp_dg > tq) { tq = tp_dg; tj = j; }
        const double rbj = r.x * bx + r.y * by + r.z * bz;
        const double rbi = r.x * bix + r.y * biy + r.z * biz;
        const double rn = r.x * nx + r.y * ny + r.z * nz;
        const double bb = bix * bx + biy * by + biz * bz;
        double tp = rbj * rr;
        tp *= tp;
        const double w = tp_dg * (((K - 4 * bb) + 0.5 * rn) - 1.5 * tp);
        const double c = tp_dg * (4 * rbi - 3 * rbj);
        const double h = 3.5 * tp_dphi;
        cs += c;
        gx += h * nx + w * r.x + c * bx;
        gy += h * ny + w * r.y + c * by;
        gz += h * nz + w * r.z + c * bz;
    }
    s[0] = gx - cs * bix;
    s[1] = gy - cs * biy;
    s[2] = gz - cs * biz;
    s[3] = m_min;
    s[4] = tq;
    s[5] = __longlong_as_double(tj);
}

// Mixed-precision form of the pass-B sweep: the separation and its floored square stay FP64 (so the per-pair
// maxima keep the reference's exact recomputation of the extremal pair), the EIH 1PN acceleration (about
// 1e-8 of the Newtonian one for solar-system speeds and potentials, so FP32's 6e-8 relative rounding is
// ~1e-15 of the total) is formed in FP32 from FP32 copies of the pass-A outputs and summed with a
// compensated FP32 sum (Fast2Sum after each add), which is converted into the FP64 totals. The
// extremal pair of max_influence is chosen on the FP32 value of GM/r^3, so in a near-tie (within FP32
// rounding) another pair's value may be the one recomputed.
struct Comp32 {    // a compensated FP32 sum
    float s, c;
};
__device__ __forceinline__ void comp_add(Comp32 &a, float x) {
    const float t = __fadd_rn(a.s, x);
    const bool keep = fabsf(a.s) >= fabsf(x);
    const float big = keep ? a.s : x, small = keep ? x : a.s;
    a.c = __fadd_rn(a.c, __fadd_rn(__fsub_rn(big, t), small));
    a.s = t;
}
__device__ __forceinline__ void sweep_point_b32(const double *A, const float *F, int i, int j0, int j1,
                                                double s[kPartB]) {
    const BodyA bi = load_a(A, i);
    const float4 *fi = reinterpret_cast<const float4 *>(F + (size_t)i * kRecF);
    const float bix = fi[1].x, biy = fi[1].y, biz = fi[1].z;
    const float phi_i = fi[1].w, beta2_i = fi[2].x;
    Comp32 gx{0, 0}, gy{0, 0}, gz{0, 0};
    double m_min = __longlong_as_double(0x7ff0000000000000ll);
    float tq = 0;
    int tj = -1;
#pragma unroll 2
    for (int j = j0; j < j1; ++j) {
        const BodyA bj = load_a(A, j);
        const float4 *fj = reinterpret_cast<const float4 *>(F + (size_t)j * kRecF);
        const float4 a = fj[0], b = fj[1];   // {a_N, GM}, {beta, phi}
        const v3 r = separation(bj, bi);
        const double q = dot(r, r), sm = bi.sr2 + bj.sr2;
        const double m = (q < sm) ? sm : q;
        if (m < m_min && j != i) m_min = m;
        const float rr = rsqrtf(j == i ? 1.0f : (float)m);
        const float tp_dphi = rr * (j == i ? 0.0f : a.w);
        const float tp_dg = (rr * rr) * tp_dphi;
        if (tp_dg > tq) { tq = tp_dg; tj = j; }
        const float rx = (float)r.x, ry = (float)r.y, rz = (float)r.z;
        const float rbj = rx * b.x + ry * b.y + rz * b.z;
        float tp = rbj * rr;
        tp *= tp;
        const float delta1 = 4 * phi_i + b.w + beta2_i + 2 * fj[2].x - 4 * (bix * b.x + biy * b.y + biz * b.z) +
                             ((rx * a.x + ry * a.y + rz * a.z) - 3 * tp) / 2;
        const float bx = b.x - bix, by = b.y - biy, bz = b.z - biz;
        const float c1 = 7 * tp_dphi / 2, c2 = tp_dg * delta1, c3 = tp_dg * (rbj - (rx * bx + ry * by + rz * bz) * 4);
        comp_add(gx, c1 * a.x + c2 * rx + c3 * bx);
        comp_add(gy, c1 * a.y + c2 * ry + c3 * by);
        comp_add(gz, c1 * a.z + c2 * rz + c3 * bz);
    }
    s[0] = (double)gx.s + (double)gx.c;
    s[1] = (double)gy.s + (double)gy.c;
    s[2] = (double)gz.s + (double)gz.c;
    s[3] = m_min;
    s[4] = (double)tq;
    s[5] = __longlong_as_double(tj);
}

// Running extremes of a body over all stages (RungeKutta.cu:229-230: the largest 1/r and GM_j/r^3 over the floored
// separations), with the reference's expressions rr2 = 1/m, rr = sqrt(rr2) (mass.impl:84-89). The smallest m = r^2
// is kept as it is (sqrt(1/m) does not decrease as m falls, so it is formed once, at the end). The stage's pair of
// the largest GM_j/r^3 is recomputed exactly only when its swept value, good to `slack`, may exceed the largest so far.
__device__ __forceinline__ void extremes_add(const View &V, const double *A, int b, double m_min, double tq, int tj,
                                             double slack) {
    if (m_min < own_row(V, OR_M, b)) own_row(V, OR_M, b) = m_min;
    const double top = own_row(V, OR_MAXI, b);
    if (tj >= 0 && tq >= top * (1 - slack)) {   // (false once the maximum is a NaN)
        const BodyA bi = load_a(A, V.lo + b), bj = load_a(A, tj);
        const v3 r = separation(bj, bi);
        const double q = dot(r, r), sm = bi.sr2 + bj.sr2;
        const double rr2 = 1.0 / ((q < sm) ? sm : q), t = rr2 * (sqrt(rr2) * bj.gm);
        if (t > top) own_row(V, OR_MAXI, b) = t;
    }
}
// The same when one of the body's sums is not a number: the sweeps' comparisons drop a NaN, the reference's
// maxima keep it (checked_maximize), so the pairs are walked again one by one.
__device__ __noinline__ void extremes_nan(const View &V, const double *A, int b) {
    const int i = V.lo + b;
    const BodyA bi = load_a(A, i);
    for (int j = 0; j < V.n; ++j) {
        if (j == i) continue;
        const BodyA bj = load_a(A, j);
        const v3 r = separation(bj, bi);
        const double q = dot(r, r), sm = bi.sr2 + bj.sr2;
        const double m = (q < sm) ? sm : q, rr2 = 1.0 / m;
        if (m != m || m < own_row(V, OR_M, b)) own_row(V, OR_M, b) = m;
        checked_maximize(own_row(V, OR_MAXI, b), rr2 * (sqrt(rr2) * bj.gm));
    }
}

// mass::orthogonalize (mass.h:147-150) of body i's frame, in place in the planes
__device__ void orthogonalize_frame(double *pl, int n, int i) {
    dd s[9];
    for (int q = 0; q < 9; ++q) s[q] = dd{pl[(size_t)(EPH_P_S_HI + q) * n + i], pl[(size_t)(EPH_P_S_LO + q) * n + i]};
    double f[9];
    for (int q = 0; q < 9; ++q) f[q] = dd_val(s[q]);
    const v3 fx = mk(f[0], f[1], f[2]), fy = mk(f[3], f[4], f[5]), fz = mk(f[6], f[7], f[8]);
    double add[9];
    for (int q = 0; q < 9; ++q) {
        const int col = q / 3, rw = q % 3;
        const v3 fc = (col == 0) ? fx : (col == 1) ? fy : fz;
        const double o0 = (col == 0 ? 1.0 : 0.0) - dot(fx, fc);
        const double o1 = (col == 1 ? 1.0 : 0.0) - dot(fy, fc);
        const double o2 = (col == 2 ? 1.0 : 0.0) - dot(fz, fc);
        add[q] = (0.5 * f[0 + rw] * o0 + 0.5 * f[3 + rw] * o1) + 0.5 * f[6 + rw] * o2;
    }
    for (int q = 0; q < 9; ++q) {
        const dd r = dd_add(s[q], dd_make(add[q]));
        pl[(size_t)(EPH_P_S_HI + q) * n + i] = r.hi;
        pl[(size_t)(EPH_P_S_LO + q) * n + i] = r.lo;
    }
}

namespace cg = cooperative_groups;

// Copies `count` 16-byte words at p (16-byte aligned, the same place in every CTA's shared memory) to the other CTAs of
// the cluster (distributed shared memory), consecutive threads consecutive words; the cluster barrier that follows
// publishes them. Stored by the threads that formed them, 8 bytes at a time and 64 apart, the records of 38 bodies
// took 1800 cycles to seven peers.
__device__ __forceinline__ void send_all(double *p, int count, int peers, int rank) {
    const double2 *from = reinterpret_cast<const double2 *>(p);
#pragma unroll 1
    for (int q = threadIdx.x; q < count * (peers - 1); q += blockDim.x) {
        const int hop = q / count, w = q - hop * count;
        const int to = rank + 1 + hop < peers ? rank + 1 + hop : rank + 1 + hop - peers;
        reinterpret_cast<double2 *>(cg::this_cluster().map_shared_rank(p, to))[w] = from[w];
    }
}

// One system on one CTA (peers = 1) or on the CTAs of a cluster, this CTA (number `rank`) owning bodies
// [lo, lo + cnt): every CTA holds the records of all bodies, computes its own bodies' stages and passes, and
// stores what the other CTAs read (state after the state update, pass-A outputs after pass A) to all of them.
//
// What bounds it: latency, of the dependent FP64 chains in the sweeps at 8 to 16 warps an SM (FP64 pipe 51 % and
// issue 52 % busy with two CTAs of 95 bodies on each SM) and of the stage's four dependent phases for small
// systems. Hence one thread per (body, component) in the state update, whose sum is one addition deep per term, one
// thread per (body, part of its j range) in the sweeps, records that a warp reads without bank conflicts, and as
// many CTAs per system as the batch needs to finish together. Stage times on one B200, one system alone, before
// (one thread per body, power-of-two lane groups, at most 4 CTAs) and now: 8 bodies 6.5 / 2.9 us, 33 9.3 / 4.6,
// 95 28.7 / 7.8, 128 16.6 / 7.5, 300 80.3 / 13.3 us.
// kEval: one evaluation of the accelerations of the loaded state (eph_accel) instead of steps.
template <bool MIXED, bool kEval = false>
__device__ void integrate_system(const BatchSys &Y, const RkTable &rk, double *smem, int peers, int rank) {
    const int n = Y.n;
    const int lo = (int)((long long)rank * n / peers);
    const int cnt = (int)((long long)(rank + 1) * n / peers) - lo;
    const View V = make_view<MIXED>(Y, smem, lo, cnt, peers);
    double *pl = Y.planes;
    const double c2 = kCB * kCB;
#define PLV(p, i) pl[(size_t)(p) * n + (i)]
    auto sync = [&]() {
        if (peers > 1) cg::this_cluster().sync();
        else __syncthreads();
    };
    // One pass over the units (body b, part `sub` of its j range), unit u = sub * cnt + b on thread u mod 256:
    // sweep(i, j0, j1, slot of the unit's sums) by the unit's thread, then take(b, value, the body's first slot) by
    // one thread per (body, value). A body's parts are summed in ascending j, so how many CTAs share a system changes
    // no result. The takes are not followed by a barrier.
    const int units = cnt * V.split;
    auto for_units = [&](auto &&sweep, auto &&take) {
#pragma unroll 1
        for (int u = threadIdx.x; u < units; u += kBThreads) {
            const int sub = u / cnt, b = u - sub * cnt;
            sweep(lo + b, sub * n / V.split, (sub + 1) * n / V.split, V.part + u);
        }
        __syncthreads();
#pragma unroll 1
        for (int idx = threadIdx.x; idx < 4 * cnt; idx += kBThreads) {
            const int c = idx / cnt, b = idx - c * cnt;
            take(b, c, V.part + b);
        }
    };
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        for (int h = 0; h < (peers > 1 ? 2 : 1); ++h) {
            double *a = V.A[h] + (size_t)i * kRecA;
            for (int c = 0; c < 3; ++c) {
                a[RA_R_HI + c] = PLV(EPH_P_R_HI + c, i);
                a[RA_R_LO + c] = PLV(EPH_P_R_LO + c, i);
            }
            a[RA_GM] = PLV(EPH_P_GM, i);
            a[RA_SR2] = PLV(EPH_P_SR2, i);
        }
    }
    for (int b = threadIdx.x; b < cnt; b += blockDim.x) {
        const int i = lo + b;
        for (int c = 0; c < 3; ++c) {
            own_row(V, OR_V_HI + c, b) = PLV(EPH_P_V_HI + c, i);
            own_row(V, OR_V_LO + c, b) = PLV(EPH_P_V_LO + c, i);
        }
        own_row(V, OR_GM0, b) = PLV(EPH_P_GM0, i);
        own_row(V, OR_DGM, b) = PLV(EPH_P_DGM, i);
        own_row(V, OR_M, b) = __longlong_as_double(0x7ff0000000000000ll);   // msystem::integrate resets the
        own_row(V, OR_MAXI, b) = 0.0;                                         // maxima (mass.cpp:406)
        if (kEval) continue;
        // the loaded auxiliaries are f_0 of the first step (RungeKutta.impl:110-116)
        const v3 fa = (mk(PLV(EPH_P_GACCEL, i), PLV(EPH_P_GACCEL + 1, i), PLV(EPH_P_GACCEL + 2, i)) +
                       mk(PLV(EPH_P_DACCEL, i), PLV(EPH_P_DACCEL + 1, i), PLV(EPH_P_DACCEL + 2, i))) +
                      mk(PLV(EPH_P_NACCEL, i), PLV(EPH_P_NACCEL + 1, i), PLV(EPH_P_NACCEL + 2, i));
        V.store[b] = fa.x;
        V.store[V.ld + b] = fa.y;
        V.store[2 * V.ld + b] = fa.z;
    }
    sync();   // the peers' copies are loaded too before the first store to them
    const double dt = Y.dt;
    int buf = 0;   // parity of the state records in use
#pragma unroll 1
    for (long long step = 0; step < (kEval ? 1 : Y.n_step); ++step) {
#pragma unroll 1
        for (int s = kEval ? kStages - 1 : 0; s < kStages; ++s) {
            const int k = s + 1;
            const double t = Y.t_eph + dt * (b_dtk[k] + (double)step);
            const bool last = kEval || (k == kStages && step + 1 == Y.n_step);
            double *A = V.A[kEval ? buf : buf ^ 1];
            if (!kEval) {
                // At s == 0 x0 = x (RungeKutta.impl:113-121). Then the state of stage k (RungeKutta.impl:148-186):
                // r = r0 + dt (c_k v0 + dt sum_l Abar_kl f_l), the sums in double-double, v = v0 + dt sum_l a_kl f_l.
#pragma unroll 1
                for (int idx = threadIdx.x; idx < 3 * cnt; idx += blockDim.x) {
                    const int b = idx / 3, c = idx - 3 * b, i = lo + b, ld = V.ld;
                    double *x0 = V.store + (size_t)(3 * kStages + c) * ld + b;
                    dd r0, v0;
                    if (s == 0) {
                        const double *a = V.A[buf] + (size_t)i * kRecA;
                        r0 = dd{a[RA_R_HI + c], a[RA_R_LO + c]};
                        v0 = dd{own_row(V, OR_V_HI + c, b), own_row(V, OR_V_LO + c, b)};
                        x0[0] = r0.hi;
                        x0[3 * ld] = r0.lo;
                        x0[6 * ld] = v0.hi;
                        x0[9 * ld] = v0.lo;
                    } else {
                        r0 = dd{x0[0], x0[3 * ld]};
                        v0 = dd{x0[6 * ld], x0[9 * ld]};
                    }
                    // r0 + dt c_k v0 does not wait for the sum
                    const dd rv = dd_add(r0, dd_mul(dd_make(dt), dd_mul(dd{b_ck_hi[k], b_ck_lo[k]}, v0)));
                    // sum_l Abar_kl f_l as a compensated dot product (Ogita, Rump and Oishi 2005, Dot2: the result of
                    // twice the working precision): one dependent addition per term instead of a double-double one
                    double s1 = 0, e1 = 0, s2 = 0;
                    const double *f = V.store + c * ld + b;
                    const int row = k * (k - 1) / 2;
#pragma unroll 4
                    for (int l = 0; l < k; ++l) {
                        const double2 ab = rk.ab[row + l];
                        const double fl = f[3 * l * ld], h = ab.x;
                        const double p = __dmul_rn(h, fl), pe = __fma_rn(rk.lo[row + l], fl, __fma_rn(h, fl, -p));
                        double sum, se;
                        two_sum(s1, p, sum, se);
                        s1 = sum;
                        e1 = __dadd_rn(e1, __dadd_rn(se, pe));
                        s2 = __dadd_rn(s2, __dmul_rn(ab.y, fl));
                    }
                    dd sf;
                    two_sum_quick(s1, e1, sf.hi, sf.lo);
                    const dd r = dd_add(rv, dd_mul(dd_make(dt), dd_mul(dd_make(dt), sf)));
                    const dd v = dd_add(v0, dd_make(dt * s2));
                    double *a = A + (size_t)i * kRecA;
                    a[RA_R_HI + c] = r.hi;
                    a[RA_R_LO + c] = r.lo;
                    own_row(V, OR_V_HI + c, b) = v.hi;
                    own_row(V, OR_V_LO + c, b) = v.lo;
                    if (c == 0) {
                        const double gm = own_row(V, OR_GM0, b) + own_row(V, OR_DGM, b) * t;
                        a[RA_GM] = gm;
                    }
                }
                if (k == kStages)
                    for (int b = threadIdx.x; b < cnt; b += blockDim.x) orthogonalize_frame(pl, n, lo + b);
                buf ^= 1;
                if (peers > 1) {
                    __syncthreads();
                    send_all(A + (size_t)lo * kRecA, cnt * (kRecA / 2), peers, rank);
                }
                // The state records alternate between two arrays when a cluster shares the system: a peer that is
                // still in the previous stage's pass B reads the other one, so one barrier per exchange is enough
                sync();
            }
            // pass A (DAMPED_TIDAL_DEFORMATION_MATRIX_NK2, mass.impl:38-46), then PREPARE_RELATIVITY
            // (mass.impl:76-80), one thread per (body, value)
            for_units([&](int i, int j0, int j1, double *part) {
                double p[kPartA];
                sweep_point_a(A, i, j0, j1, p);
                for (int c = 0; c < kPartA; ++c) part[c * units] = p[c];
            }, [&](int b, int c, const double *part) {
                double sum = 0;
#pragma unroll 8
                for (int q = 0; q < V.split; ++q) sum += part[c * units + q * cnt];
                double *rec = rec_b(V, lo + b);
                float *frec = V.F + (size_t)(lo + b) * kRecF;
                auto beta = [&](int d) {
                    return dd_val(dd{own_row(V, OR_V_HI + d, b), own_row(V, OR_V_LO + d, b)}) * (1.0 / kCB);
                };
                if (c == 0) {
                    const v3 be = mk(beta(0), beta(1), beta(2));
                    const double phi = sum / c2, b2 = dot(be, be);
                    rec[RB_PHI] = phi;
                    rec[RB_K] = phi + 2 * b2;
                    if (MIXED) {
                        frec[RF_PHI] = (float)phi;
                        frec[RF_BETA2] = (float)b2;
                        frec[RF_GM] = (float)A[(size_t)(lo + b) * kRecA + RA_GM];
                    }
                } else {
                    const double na = sum * (1.0 / c2), be = beta(c - 1);
                    rec[RB_NACC + c - 1] = na;
                    rec[RB_BETA + c - 1] = be;
                    if (MIXED) {
                        frec[RF_NACC + c - 1] = (float)na;
                        frec[RF_BETA + c - 1] = (float)be;
                    }
                }
            });
            if (peers > 1) {
                __syncthreads();
                if (MIXED) send_all(reinterpret_cast<double *>(V.F + (size_t)lo * kRecF), cnt * (kRecF / 4), peers, rank);
                else send_all(V.B + (size_t)lo * kRecB, cnt * (kRecB / 2), peers, rank);
            }
            sync();
            // pass B (RELATIVITY, mass.impl:82-97), then FINALIZE_RELATIVITY (mass.impl:133-135): f = (gaccel +
            // daccel) + naccel, kept as f_k
            for_units([&](int i, int j0, int j1, double *part) {
                double p[kPartB];
                if (MIXED) sweep_point_b32(A, V.F, i, j0, j1, p);
                else sweep_point_b(A, V.B, i, j0, j1, p);
                for (int c = 0; c < kPartB; ++c) part[c * units] = p[c];
            }, [&](int b, int c, const double *part) {
                if (c < 3) {
                    double ga = 0;
#pragma unroll 8
                    for (int q = 0; q < V.split; ++q) ga += part[c * units + q * cnt];
                    const double *rec = rec_b(V, lo + b);
                    const double na = c2 * rec[RB_NACC + c];
                    if (!MIXED) {
                        const v3 be = mk(rec[RB_BETA], rec[RB_BETA + 1], rec[RB_BETA + 2]);
                        ga += (4 * rec[RB_PHI] + dot(be, be)) * na;   // the terms common to all j
                    }
                    V.store[(3 * (k % kStages) + c) * V.ld + b] = ga + na;
                    if (last) PLV(EPH_P_GACCEL + c, lo + b) = ga;
                } else {
                    double nan = 0, m_min = __longlong_as_double(0x7ff0000000000000ll), tq = 0;
                    int tj = -1;
#pragma unroll 4
                    for (int q = 0; q < V.split; ++q) {
                        const double *p = part + q * cnt;
                        const double p0 = p[0], pm = p[3 * units], pt = p[4 * units];
                        const int pj = __double2loint(p[5 * units]);
                        nan += p0;
                        m_min = pm < m_min ? pm : m_min;
                        tj = pt > tq ? pj : tj;
                        tq = pt > tq ? pt : tq;
                    }
                    if (nan != nan) extremes_nan(V, A, b);
                    else extremes_add(V, A, b, m_min, tq, tj, MIXED ? 0x1p-18 : 0x1p-48);
                }
            });
            __syncthreads();
        }
    }
    // store (cuda_rungekutta_kernel_config::save of RungeKutta.cu:124-133); min_distance inverted (mass.cpp:436)
    for (int b = threadIdx.x; b < cnt; b += blockDim.x) {
        const int i = lo + b;
        const double *a = V.A[buf] + (size_t)i * kRecA, *rec = rec_b(V, i);
        for (int c = 0; c < 3; ++c) {
            PLV(EPH_P_R_HI + c, i) = a[RA_R_HI + c];
            PLV(EPH_P_R_LO + c, i) = a[RA_R_LO + c];
            PLV(EPH_P_V_HI + c, i) = own_row(V, OR_V_HI + c, b);
            PLV(EPH_P_V_LO + c, i) = own_row(V, OR_V_LO + c, b);
            PLV(EPH_P_NACCEL + c, i) = c2 * rec[RB_NACC + c];
            PLV(EPH_P_DACCEL + c, i) = 0.0;
            PLV(EPH_P_DTORQUE + c, i) = 0.0;
            PLV(EPH_P_BETA + c, i) = rec[RB_BETA + c];
        }
        PLV(EPH_P_GM, i) = a[RA_GM];
        PLV(EPH_P_PHI, i) = c2 * rec[RB_PHI];
        const v3 be = mk(rec[RB_BETA], rec[RB_BETA + 1], rec[RB_BETA + 2]);
        PLV(EPH_P_BETA2, i) = dot(be, be);
        double mind = sqrt(1.0 / own_row(V, OR_M, b)), maxi = own_row(V, OR_MAXI, b);   // (no pair seen: 0)
        if (Y.accumulate) {
            const double mind0 = PLV(EPH_P_MIN_DISTANCE, i), maxi0 = PLV(EPH_P_MAX_INFLUENCE, i);
            checked_maximize(mind, mind0);
            checked_maximize(maxi, maxi0);
        }
        PLV(EPH_P_MIN_DISTANCE, i) = Y.accumulate ? mind : 1 / mind;
        PLV(EPH_P_MAX_INFLUENCE, i) = maxi;
        if (Y.whole) {   // UPDATE_HARMONICS (mass.impl:48-64) of a body without tide, spin and static harmonics
            const double gi = ((-2.0) / 3 * PLV(EPH_P_R2, i)) * -PLV(EPH_P_A, i);
            for (int q = 0; q < 9; ++q) {
                PLV(EPH_P_C_POTENTIAL + q, i) = 0.0;
                PLV(EPH_P_GI + q, i) = q % 4 == 0 ? gi : 0.0;
            }
            PLV(EPH_P_EXJ2, i) = 0.0;
        }
    }
#undef PLV
    __syncthreads();
}

__device__ __forceinline__ void load_table(RkTable &rk) {
    for (int q = threadIdx.x; q < EPH_RK12_NCOEF; q += blockDim.x) {
        rk.ab[q] = make_double2(b_ab_hi[q], b_a[q]);
        rk.lo[q] = b_ab_lo[q];
    }
    __syncthreads();
}

// Persistent CTAs: every CTA (peers = 1) or thread-block cluster of `peers` CTAs takes systems from the queue
// until it is empty.
template <bool MIXED>
__global__ void __launch_bounds__(kBThreads, 2)
    ensemble_kernel(const BatchSys *sys, const int *order, int n_jobs, int *next, int peers) {
    extern __shared__ __align__(16) double bsm[];
    __shared__ RkTable rk;
    __shared__ int s_job;
    cg::cluster_group cl = cg::this_cluster();
    for (int q = threadIdx.x; q < EPH_RK12_NCOEF; q += blockDim.x) {
        rk.ab[q] = make_double2(b_ab_hi[q], b_a[q]);
        rk.lo[q] = b_ab_lo[q];
    }
    __syncthreads();
    const int rank = peers > 1 ? (int)cl.block_rank() : 0;
#pragma unroll 1
    for (;;) {
        int job;
        if (peers > 1) {
            cl.sync();   // every CTA of the cluster is done with the previous job and its shared memory
            if (rank == 0 && threadIdx.x == 0) s_job = atomicAdd(next, 1);
            cl.sync();
            job = *cl.map_shared_rank(&s_job, 0);
            cl.sync();   // read by all before rank 0 may reuse s_job, or leave
        } else {
            if (threadIdx.x == 0) s_job = atomicAdd(next, 1);
            __syncthreads();
            job = s_job;
            __syncthreads();
        }
        if (job >= n_jobs) return;
        integrate_system<MIXED>(sys[order[job]], rk, bsm, peers, rank);
    }
}

// One system on the CTAs of one cluster: its steps, or one evaluation of its accelerations (eph_accel of 33 bodies,
// with the read-back: 73 -> 45 us; of 300: 109 -> 78 us).
template <bool kEval>
__global__ void __launch_bounds__(kBThreads, 2) point_kernel(BatchSys Y, int peers) {
    extern __shared__ __align__(16) double bsm[];
    __shared__ RkTable rk;
    if (!kEval) load_table(rk);
    integrate_system<false, kEval>(Y, rk, bsm, peers, peers > 1 ? (int)cg::this_cluster().block_rank() : 0);
    if (peers > 1) cg::this_cluster().sync();   // no CTA leaves while a peer may still store to it
}

// CTA counts whose clusters the present device, or the part of it that the process may use, can hold, each CTA with the
// most shared memory it may take. Above 8 CTAs that is not a matter of course.
unsigned device_shares() {
    unsigned set = 1u << (kShares - 1);
    for (int g = 0; g < kShares - 1; ++g) {
        cudaLaunchAttribute attr{};
        attr.id = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim.x = kSharePeers[g];
        attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(kSharePeers[g]);
        cfg.blockDim = dim3(kBThreads);
        cfg.dynamicSmemBytes = kBMaxSmem;
        cfg.attrs = &attr;
        cfg.numAttrs = 1;
        int clusters = 0;
        if (cudaOccupancyMaxActiveClusters(&clusters, point_kernel<false>, &cfg) == cudaSuccess && clusters > 0) set |= 1u << g;
    }
    cudaGetLastError();   // (a size that the device refuses)
    return set;
}

std::atomic<bool> g_batch_ready[64];
unsigned g_batch_shares[64];
std::mutex g_batch_mu;   // contexts and batches may set a device up at the same time
cudaError_t batch_setup(int device, unsigned *shares) {
    const bool kept = device >= 0 && device < 64;
    if (kept && g_batch_ready[device].load(std::memory_order_acquire)) {
        *shares = g_batch_shares[device];
        return cudaSuccess;
    }
    std::lock_guard<std::mutex> lock(g_batch_mu);
    if (kept && g_batch_ready[device].load(std::memory_order_relaxed)) {
        *shares = g_batch_shares[device];
        return cudaSuccess;
    }
    double hi[EPH_RK12_NCOEF], lo[EPH_RK12_NCOEF], dtk[kStages + 1];
    rk12_expand(hi, lo, dtk);
    double ab_hi[EPH_RK12_NCOEF] = {0}, ab_lo[EPH_RK12_NCOEF] = {0}, aa[EPH_RK12_NCOEF] = {0};
    double ck_hi[kStages + 1] = {0}, ck_lo[kStages + 1] = {0};
    auto coef = [&](int k, int j) { return (long double)hi[k * (k - 1) / 2 + j] + lo[k * (k - 1) / 2 + j]; };
    auto split = [](long double x, double &h, double &l) { h = (double)x; l = (double)(x - h); };
    for (int k = 1; k <= kStages; ++k) {
        long double c = 0;
        for (int l = 0; l < k; ++l) {
            const int q = k * (k - 1) / 2 + l;
            long double acc = 0;   // Abar_kl = sum_{l<j<k} a_kj a_jl
            for (int j = l + 1; j < k; ++j) acc += coef(k, j) * coef(j, l);
            split(acc, ab_hi[q], ab_lo[q]);
            aa[q] = hi[q] + lo[q];
            c += coef(k, l);
        }
        split(c, ck_hi[k], ck_lo[k]);
    }
    cudaError_t e = cudaMemcpyToSymbol(b_ab_hi, ab_hi, sizeof(ab_hi));
    if (e == cudaSuccess) e = cudaMemcpyToSymbol(b_ab_lo, ab_lo, sizeof(ab_lo));
    if (e == cudaSuccess) e = cudaMemcpyToSymbol(b_a, aa, sizeof(aa));
    if (e == cudaSuccess) e = cudaMemcpyToSymbol(b_ck_hi, ck_hi, sizeof(ck_hi));
    if (e == cudaSuccess) e = cudaMemcpyToSymbol(b_ck_lo, ck_lo, sizeof(ck_lo));
    if (e == cudaSuccess) e = cudaMemcpyToSymbol(b_dtk, dtk, sizeof(dtk));
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(ensemble_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kBMaxSmem);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(ensemble_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kBMaxSmem);
    // clusters of 16 CTAs: twice the portable size
    if (e == cudaSuccess) e = cudaFuncSetAttribute(ensemble_kernel<false>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(ensemble_kernel<true>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    for (auto k : {point_kernel<false>, point_kernel<true>}) {
        if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kBMaxSmem);
    }
    if (e != cudaSuccess) return e;
    *shares = device_shares();
    if (kept) {
        g_batch_shares[device] = *shares;
        g_batch_ready[device].store(true, std::memory_order_release);
    }
    return cudaSuccess;
}

}  // namespace

// ---- a single point-mass system (eph_capi.cu)
// Scratch a context keeps for it (doubles).
size_t point_scratch_doubles(int n) { return (size_t)kStore * n; }
// Launches n_step steps of dt of a system of point-like bodies on `stream`, as the step kernel of eph_step.cu would
// integrate it (accumulate: eph_rk12's maxima, else eph_integrate's); n_step 0: one evaluation of its accelerations.
// cudaErrorNotSupported: the device's clusters are too small for it, nothing was launched.
cudaError_t launch_point_system(int device, cudaStream_t stream, double *planes, int n, double dt, long long n_step, double t_eph,
                                int accumulate, double *scratch) {
    unsigned shares = 0;
    cudaError_t e = batch_setup(device, &shares);
    if (e != cudaSuccess) return e;
    const int split = batch_split(n), g = shortest_stage(n, split, false, shares);
    if (g < 0) return cudaErrorNotSupported;
    const int peers = kSharePeers[g];
    BatchSys Y{};
    Y.n = n;
    Y.split = split;
    Y.n_step = n_step;
    Y.dt = dt;
    Y.t_eph = t_eph;
    Y.accumulate = accumulate;
    Y.whole = 1;
    Y.planes = planes;
    Y.store = scratch;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = peers;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(peers);
    cfg.blockDim = dim3(kBThreads);
    cfg.dynamicSmemBytes = system_smem(n, peers, split, false);
    cfg.stream = stream;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return n_step ? cudaLaunchKernelEx(&cfg, point_kernel<false>, Y, peers) : cudaLaunchKernelEx(&cfg, point_kernel<true>, Y, peers);
}
}  // namespace eph

using namespace eph;

struct eph_batch {
    int device = 0;
    cudaStream_t stream = nullptr;     // work stream (own_stream unless eph_batch_set_stream chose another)
    cudaStream_t own_stream = nullptr;
    cudaStream_t side[kShares] = {};   // the launches of one integration run beside each other
    cudaEvent_t ev_begin = nullptr, ev_end[kShares] = {};
    unsigned shares = 0;               // CTA counts that the device can hold as clusters (batch_setup)
    int mixed = 0;                     // 1: EIH 1PN terms of the ensemble kernel in FP32 (eph_batch_set_precision)
    int coop_min = kCoopMin;           // bodies from which a system is shared by a cluster (eph_batch_set_coop_min)
    std::mutex mu;
    char err[512] = {0};
    int n_sys = 0;
    std::vector<int64_t> n_body;
    std::vector<int> point;                    // 1: ensemble kernel, 0: per-system context path
    std::vector<int> split;                    // parts of a body's j range (batch_split)
    std::vector<size_t> off;                   // offset of system s in d_planes (doubles)
    std::vector<size_t> store_off;             // offset of its stage store (doubles)
    std::vector<std::vector<double>> h_full;   // host copies of the context-path systems' planes
    std::vector<std::vector<int32_t>> m_gp_nz, m_gp_nt, m_ring_nd;
    std::vector<std::vector<double>> m_gp_coef, m_ring_param, m_ring_disk;
    double *d_planes = nullptr, *d_store = nullptr;
    BatchSys *d_sys = nullptr;
    int *d_order = nullptr, *d_next = nullptr;
    eph_ctx *ctx = nullptr;                    // context path
    int64_t launches = 0;
};

static int bfail(eph_batch *b, int code, const char *what, cudaError_t e = cudaSuccess) {
    if (b) {
        if (e != cudaSuccess) snprintf(b->err, sizeof(b->err), "%s: %s", what, cudaGetErrorString(e));
        else snprintf(b->err, sizeof(b->err), "%s", what);
    }
    return code;
}
#define BCK(call, what)                                                                                     \
    do {                                                                                                    \
        cudaError_t e_ = (call);                                                                            \
        if (e_ != cudaSuccess) return bfail(b, e_ == cudaErrorMemoryAllocation ? EPH_ERR_OOM : EPH_ERR_CUDA, what, e_); \
    } while (0)

static void batch_free(eph_batch *b) {
    for (void *p : {(void *)b->d_planes, (void *)b->d_store, (void *)b->d_sys, (void *)b->d_order,
                    (void *)b->d_next})
        if (p) cudaFree(p);
    b->d_planes = b->d_store = nullptr;
    b->d_sys = nullptr;
    b->d_order = b->d_next = nullptr;
    b->n_sys = 0;
}

static bool batch_side(eph_batch *b) {   // the side streams of an integration's launches, and their events
    bool ok = cudaEventCreateWithFlags(&b->ev_begin, cudaEventDisableTiming) == cudaSuccess;
    for (int g = 0; g < kShares; ++g)
        ok = ok && cudaStreamCreateWithFlags(&b->side[g], cudaStreamNonBlocking) == cudaSuccess &&
             cudaEventCreateWithFlags(&b->ev_end[g], cudaEventDisableTiming) == cudaSuccess;
    return ok;
}

extern "C" {

int eph_batch_create(int device, eph_batch **out) {
    if (!out) return EPH_ERR_ARG;
    *out = nullptr;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || device < 0 || device >= ndev) return EPH_ERR_ARG;
    eph_batch *b = new eph_batch();
    b->device = device;
    if (cudaSetDevice(device) != cudaSuccess || cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking) != cudaSuccess ||
        batch_setup(device, &b->shares) != cudaSuccess || !batch_side(b)) {
        eph_batch_destroy(b);
        return EPH_ERR_CUDA;
    }
    *out = b;
    return EPH_OK;
}

int eph_batch_destroy(eph_batch *b) {
    if (!b) return EPH_ERR_ARG;
    cudaSetDevice(b->device);
    batch_free(b);
    for (int g = 0; g < kShares; ++g) {
        if (b->side[g]) cudaStreamDestroy(b->side[g]);
        if (b->ev_end[g]) cudaEventDestroy(b->ev_end[g]);
    }
    if (b->ev_begin) cudaEventDestroy(b->ev_begin);
    if (b->ctx) eph_ctx_destroy(b->ctx);
    if (b->own_stream) cudaStreamDestroy(b->own_stream);
    else if (b->stream) cudaStreamDestroy(b->stream);
    delete b;
    return EPH_OK;
}

const char *eph_batch_last_error(const eph_batch *b) { return b ? b->err : "null batch"; }

int eph_batch_upload(eph_batch *b, int32_t n_sys, const int64_t *n_body, const double *const *planes,
                     const eph_models *const *models) {
    if (!b || n_sys <= 0 || !n_body || !planes) return bfail(b, EPH_ERR_ARG, "eph_batch_upload: bad arguments");
    std::lock_guard<std::mutex> lock(b->mu);
    for (int s = 0; s < n_sys; ++s) {
        if (n_body[s] <= 0 || n_body[s] > (1 << 20) || !planes[s]) return bfail(b, EPH_ERR_ARG, "eph_batch_upload: bad system");
        const eph_models *m = models ? models[s] : nullptr;
        const int n_gp = m ? m->n_gp : 0, n_ring = m ? m->n_ring : 0;
        if (n_gp < 0 || n_ring < 0 || (n_gp && (!m->gp_nz || !m->gp_nt || !m->gp_coef)) ||
            (n_ring && (!m->ring_ndisk || !m->ring_param || !m->ring_disk)))
            return bfail(b, EPH_ERR_ARG, "eph_batch_upload: bad model tables");
    }
    BCK(cudaSetDevice(b->device), "cudaSetDevice");
    batch_free(b);
    b->n_sys = n_sys;
    b->n_body.assign(n_body, n_body + n_sys);
    b->point.assign(n_sys, 0);
    b->split.assign(n_sys, 1);
    b->off.assign(n_sys, 0);
    b->store_off.assign(n_sys, 0);
    b->h_full.assign(n_sys, {});
    b->m_gp_nz.assign(n_sys, {}); b->m_gp_nt.assign(n_sys, {}); b->m_ring_nd.assign(n_sys, {});
    b->m_gp_coef.assign(n_sys, {}); b->m_ring_param.assign(n_sys, {}); b->m_ring_disk.assign(n_sys, {});
    size_t tot = 0, tot_store = 0;
    for (int s = 0; s < n_sys; ++s) {
        const int n = (int)n_body[s];
        bool pt = n <= kMaxBodies;
        for (int i = 0; i < n && pt; ++i) pt = !plan_full_class(planes[s], n, i);
        if (pt) {   // (in either precision, which may be chosen after the upload)
            b->split[s] = batch_split(n);
            pt = fewest_ctas(n, b->split[s], false, b->shares) >= 0 && fewest_ctas(n, b->split[s], true, b->shares) >= 0;
        }
        b->point[s] = pt;
        if (pt) {
            b->off[s] = tot;
            b->store_off[s] = tot_store;
            tot += (size_t)EPH_NPLANES * n;
            tot_store += (size_t)kStore * n;
        } else {
            b->h_full[s].assign(planes[s], planes[s] + (size_t)EPH_NPLANES * n);
            const eph_models *m = models ? models[s] : nullptr;
            if (m && m->n_gp) {
                b->m_gp_nz[s].assign(m->gp_nz, m->gp_nz + m->n_gp);
                b->m_gp_nt[s].assign(m->gp_nt, m->gp_nt + m->n_gp);
                b->m_gp_coef[s].assign(m->gp_coef, m->gp_coef + (size_t)m->n_gp * EPH_GP_TABLE_SIZE);
            }
            if (m && m->n_ring) {
                b->m_ring_nd[s].assign(m->ring_ndisk, m->ring_ndisk + m->n_ring);
                b->m_ring_param[s].assign(m->ring_param, m->ring_param + (size_t)m->n_ring * EPH_RING_PARAMS);
                b->m_ring_disk[s].assign(m->ring_disk, m->ring_disk + (size_t)m->n_ring * EPH_RING_MAX_DISKS * 3);
            }
        }
    }
    if (tot) {
        BCK(cudaMalloc(&b->d_planes, tot * sizeof(double)), "cudaMalloc(batch planes)");
        BCK(cudaMalloc(&b->d_store, tot_store * sizeof(double)), "cudaMalloc(batch stage store)");
        BCK(cudaMalloc(&b->d_sys, (size_t)n_sys * sizeof(BatchSys)), "cudaMalloc(batch table)");
        BCK(cudaMalloc(&b->d_order, (size_t)n_sys * sizeof(int)), "cudaMalloc(batch order)");
        BCK(cudaMalloc(&b->d_next, kShares * sizeof(int)), "cudaMalloc(batch queues)");
        for (int s = 0; s < n_sys; ++s)
            if (b->point[s])
                BCK(cudaMemcpyAsync(b->d_planes + b->off[s], planes[s], (size_t)EPH_NPLANES * n_body[s] * sizeof(double),
                                    cudaMemcpyHostToDevice, b->stream), "upload batch planes");
        BCK(cudaStreamSynchronize(b->stream), "upload batch planes");
    }
    return EPH_OK;
}

int eph_batch_integrate(eph_batch *b, const double *dt, const int64_t *n_step, double *t_eph_hi, double *t_eph_lo) {
    if (!b || !dt || !n_step || !t_eph_hi || !t_eph_lo) return bfail(b, EPH_ERR_ARG, "eph_batch_integrate: bad arguments");
    std::lock_guard<std::mutex> lock(b->mu);
    if (!b->n_sys) return bfail(b, EPH_ERR_STATE, "no batch uploaded");
    BCK(cudaSetDevice(b->device), "cudaSetDevice");
    const int n_sys = b->n_sys;
    std::vector<BatchSys> tab(n_sys);
    std::vector<int> order, share(n_sys, kShares - 1);
    std::vector<double> stage(n_sys, 0.0), work(n_sys, 0.0);
    int sms = 0;
    BCK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, b->device), "SM count");
    for (int s = 0; s < n_sys; ++s) {
        if (!b->point[s] || n_step[s] == 0) continue;
        BatchSys &Y = tab[s];
        const int n = (int)b->n_body[s];
        Y.n = n;
        Y.split = b->split[s];
        Y.accumulate = Y.whole = 0;
        // msystem::integrate: a negative step count integrates backwards (mass.cpp:401-404)
        Y.n_step = n_step[s] < 0 ? -n_step[s] : n_step[s];
        Y.dt = n_step[s] < 0 ? -dt[s] : dt[s];
        Y.t_eph = t_eph_hi[s] + t_eph_lo[s];
        Y.planes = b->d_planes + b->off[s];
        Y.store = b->d_store + b->store_off[s];
        order.push_back(s);
    }
    // CTAs per system. A system on one CTA does the least work in all, one shared by a cluster is done sooner: as
    // long as the longest job would outlast the whole batch's work spread over the SMs (two CTAs each), it is given
    // twice the CTAs. The choice changes no result.
    {
        auto job = [&](int s, int g) { return (double)stage_us((int)b->n_body[s], kSharePeers[g], b->split[s]) * (double)tab[s].n_step; };
        double total = 0;
        std::vector<std::pair<double, int>> heap;   // (duration, system), longest on top
        for (int s : order) {
            share[s] = fewest_ctas((int)b->n_body[s], b->split[s], b->mixed, b->shares);
            work[s] = job(s, share[s]);
            total += work[s] * kSharePeers[share[s]];
            heap.emplace_back(work[s], s);
        }
        std::make_heap(heap.begin(), heap.end());
        while (!heap.empty() && heap.front().first > 1.1 * total / (2.0 * sms)) {
            std::pop_heap(heap.begin(), heap.end());
            const int s = heap.back().second, g = more_ctas((int)b->n_body[s], b->split[s], b->mixed, b->shares, share[s]);
            heap.pop_back();
            if (g < 0 || b->n_body[s] < b->coop_min) break;
            const double d = job(s, g);
            if (d > 0.95 * work[s]) break;
            total += d * kSharePeers[g] - work[s] * kSharePeers[share[s]];
            share[s] = g;
            work[s] = d;
            heap.emplace_back(d, s);
            std::push_heap(heap.begin(), heap.end());
        }
    }
    // one launch for each number of CTAs; in each the longest job first, so that the last to start are short ones
    std::stable_sort(order.begin(), order.end(), [&](int a, int c) {
        if (share[a] != share[c]) return share[a] < share[c];
        return work[a] > work[c];
    });
    if (!order.empty()) {
        BCK(cudaMemcpyAsync(b->d_sys, tab.data(), (size_t)n_sys * sizeof(BatchSys), cudaMemcpyHostToDevice, b->stream),
            "upload batch table");
        BCK(cudaMemcpyAsync(b->d_order, order.data(), order.size() * sizeof(int), cudaMemcpyHostToDevice, b->stream),
            "upload batch order");
        BCK(cudaMemsetAsync(b->d_next, 0, kShares * sizeof(int), b->stream), "reset batch queues");
        BCK(cudaEventRecord(b->ev_begin, b->stream), "batch event");
        auto kernel = b->mixed ? ensemble_kernel<true> : ensemble_kernel<false>;
        size_t begin = 0;
        for (int g = 0; g < kShares; ++g) {
            // side by side: the CTAs of a later launch start as the SMs come free (no CTA waits on another cluster)
            size_t end = begin, smem = 0;
            const int peers = kSharePeers[g];
            for (; end < order.size() && share[order[end]] == g; ++end)
                smem = std::max(smem, system_smem((int)b->n_body[order[end]], peers, b->split[order[end]], b->mixed));
            const int jobs = (int)(end - begin);
            if (!jobs) continue;
            cudaLaunchAttribute attr{};
            attr.id = cudaLaunchAttributeClusterDimension;
            attr.val.clusterDim.x = peers;
            attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
            cudaLaunchConfig_t cfg{};
            cfg.gridDim = dim3(peers);
            cfg.blockDim = dim3(kBThreads);
            cfg.dynamicSmemBytes = smem;
            cfg.stream = b->side[g];
            cfg.attrs = &attr;
            cfg.numAttrs = 1;
            int clusters = 0;
            BCK(cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg), "occupancy");
            if (clusters <= 0) return bfail(b, EPH_ERR_CUDA, "no room for a cluster of the ensemble kernel");
            cfg.gridDim = dim3(peers * std::min(jobs, clusters));
            BCK(cudaStreamWaitEvent(b->side[g], b->ev_begin, 0), "batch event");
            BCK(cudaLaunchKernelEx(&cfg, kernel, (const BatchSys *)b->d_sys, (const int *)b->d_order + begin, jobs,
                                   b->d_next + g, peers), "launch ensemble kernel");
            BCK(cudaEventRecord(b->ev_end[g], b->side[g]), "batch event");
            BCK(cudaStreamWaitEvent(b->stream, b->ev_end[g], 0), "batch event");
            b->launches++;
            begin = end;
        }
    }
    // the other systems through the per-system kernel, while the ensemble kernel runs
    for (int s = 0; s < n_sys; ++s) {
        if (b->point[s]) continue;
        if (!b->ctx) {
            const int rc = eph_ctx_create(b->device, &b->ctx);
            if (rc) return bfail(b, rc, "context for full-physics systems");
        }
        eph_models m{};
        m.n_gp = (int32_t)b->m_gp_nz[s].size();
        m.gp_nz = b->m_gp_nz[s].data();
        m.gp_nt = b->m_gp_nt[s].data();
        m.gp_coef = b->m_gp_coef[s].data();
        m.n_ring = (int32_t)b->m_ring_nd[s].size();
        m.ring_ndisk = b->m_ring_nd[s].data();
        m.ring_param = b->m_ring_param[s].data();
        m.ring_disk = b->m_ring_disk[s].data();
        int rc = eph_upload_system(b->ctx, b->n_body[s], b->h_full[s].data(), &m);
        double th = t_eph_hi[s], tl = t_eph_lo[s];
        if (!rc) rc = eph_integrate(b->ctx, dt[s], n_step[s], &th, &tl);
        if (!rc) rc = eph_download_system(b->ctx, b->h_full[s].data());
        if (rc) return bfail(b, rc, eph_last_error(b->ctx));
        b->launches++;
        t_eph_hi[s] = th;
        t_eph_lo[s] = tl;
    }
    BCK(cudaStreamSynchronize(b->stream), "ensemble kernel");
    // t_eph += dt*n_step in double-double (mass.cpp:441)
    for (int s : order) {
        const double d = n_step[s] < 0 ? -dt[s] : dt[s];
        const double a = t_eph_hi[s], c = d * (double)(n_step[s] < 0 ? -n_step[s] : n_step[s]);
        const double sum = a + c, t = sum - a;
        double e = (a - (sum - t)) + (c - t);
        e = e + (t_eph_lo[s] + 0.0);
        const double hi = sum + e;
        t_eph_lo[s] = e - (hi - sum);
        t_eph_hi[s] = hi;
    }
    return EPH_OK;
}

int eph_batch_download(eph_batch *b, double *const *planes) {
    if (!b || !planes) return bfail(b, EPH_ERR_ARG, "eph_batch_download: bad arguments");
    std::lock_guard<std::mutex> lock(b->mu);
    if (!b->n_sys) return bfail(b, EPH_ERR_STATE, "no batch uploaded");
    BCK(cudaSetDevice(b->device), "cudaSetDevice");
    for (int s = 0; s < b->n_sys; ++s) {
        if (!planes[s]) return bfail(b, EPH_ERR_ARG, "eph_batch_download: null planes");
        const size_t bytes = (size_t)EPH_NPLANES * b->n_body[s] * sizeof(double);
        if (b->point[s])
            BCK(cudaMemcpyAsync(planes[s], b->d_planes + b->off[s], bytes, cudaMemcpyDeviceToHost, b->stream), "download batch");
        else
            memcpy(planes[s], b->h_full[s].data(), bytes);
    }
    BCK(cudaStreamSynchronize(b->stream), "download batch");
    return EPH_OK;
}

int eph_batch_set_stream(eph_batch *b, void *stream) {
    if (!b) return EPH_ERR_ARG;
    std::lock_guard<std::mutex> lock(b->mu);
    if (!b->own_stream) b->own_stream = b->stream;
    b->stream = stream ? (cudaStream_t)stream : b->own_stream;
    return EPH_OK;
}

int eph_batch_set_coop_min(eph_batch *b, int bodies) {
    if (!b || bodies < 0) return bfail(b, EPH_ERR_ARG, "eph_batch_set_coop_min: bad arguments");
    std::lock_guard<std::mutex> lock(b->mu);
    b->coop_min = bodies == 0 ? kCoopMin : bodies;
    return EPH_OK;
}

int eph_batch_autotune(eph_batch *b, const double *dt, const int64_t *n_step, double step_frac, int *coop_min,
                       double *ms_tuned, double *ms_default) {
    if (!b || !dt || !n_step || !(step_frac > 0 && step_frac <= 1) || !coop_min || !ms_tuned || !ms_default)
        return bfail(b, EPH_ERR_ARG, "eph_batch_autotune: bad arguments");
    int n_sys = 0;
    size_t planes_doubles = 0;
    {
        std::lock_guard<std::mutex> lock(b->mu);
        if (!b->n_sys) return bfail(b, EPH_ERR_STATE, "no batch uploaded");
        n_sys = b->n_sys;
        for (int s = 0; s < n_sys; ++s) planes_doubles = std::max(planes_doubles, b->off[s] + (size_t)EPH_NPLANES * b->n_body[s]);
    }
    BCK(cudaSetDevice(b->device), "cudaSetDevice");
    // every trial runs the shared launch from the uploaded state with step counts scaled by step_frac (the
    // members keep their relative durations); the systems of the per-system path are left out
    std::vector<int64_t> steps(n_sys);
    for (int s = 0; s < n_sys; ++s) {
        const int64_t k = n_step[s] < 0 ? -n_step[s] : n_step[s];
        const int64_t t = k == 0 ? 0 : std::max<int64_t>(1, (int64_t)std::llround((double)k * step_frac));
        steps[s] = n_step[s] < 0 ? -t : t;
    }
    double *d_save = nullptr;
    BCK(cudaMalloc(&d_save, planes_doubles * sizeof(double)), "cudaMalloc(autotune)");
    BCK(cudaMemcpy(d_save, b->d_planes, planes_doubles * sizeof(double), cudaMemcpyDeviceToDevice), "save planes");
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    std::vector<double> th(n_sys), tl(n_sys);
    const int saved_coop = b->coop_min;
    for (int s = 0; s < n_sys; ++s) if (!b->point[s]) steps[s] = 0;   // ensemble members only
    int rc = EPH_OK;
    auto trial = [&](int cm, double *ms) {
        double best = 1e300;
        for (int rep = 0; rep < 2 && rc == EPH_OK; ++rep) {
            b->coop_min = cm;
            if (cudaMemcpy(b->d_planes, d_save, planes_doubles * sizeof(double), cudaMemcpyDeviceToDevice) != cudaSuccess) {
                rc = bfail(b, EPH_ERR_CUDA, "restore planes");
                break;
            }
            std::fill(th.begin(), th.end(), 0.0);
            std::fill(tl.begin(), tl.end(), 0.0);
            cudaEventRecord(e0, b->stream);
            rc = eph_batch_integrate(b, dt, steps.data(), th.data(), tl.data());
            cudaEventRecord(e1, b->stream);
            float t = 0;
            if (rc == EPH_OK && cudaEventSynchronize(e1) == cudaSuccess && cudaEventElapsedTime(&t, e0, e1) == cudaSuccess)
                best = std::min(best, (double)t);
        }
        *ms = best;
    };
    double t_def = 1e300, t_best = 1e300;
    int best = saved_coop;
    trial(saved_coop, &t_def);
    t_best = t_def;
    for (int cm : {48, 64, 128, 192, 1 << 30}) {
        if (rc || cm == saved_coop) continue;
        double t = 1e300;
        trial(cm, &t);
        if (rc == EPH_OK && t < t_best) { t_best = t; best = cm; }
    }
    b->coop_min = rc ? saved_coop : best;
    if (cudaMemcpy(b->d_planes, d_save, planes_doubles * sizeof(double), cudaMemcpyDeviceToDevice) != cudaSuccess && !rc)
        rc = bfail(b, EPH_ERR_CUDA, "restore planes");
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    cudaFree(d_save);
    if (rc) return rc;
    *coop_min = best;
    *ms_tuned = t_best;
    *ms_default = t_def;
    return EPH_OK;
}

int eph_batch_set_precision(eph_batch *b, int mode) {
    if (!b || (mode != EPH_PREC_FP64 && mode != EPH_PREC_MIXED)) return bfail(b, EPH_ERR_ARG, "eph_batch_set_precision: unknown mode");
    std::lock_guard<std::mutex> lock(b->mu);
    b->mixed = mode == EPH_PREC_MIXED;
    return EPH_OK;
}

int eph_batch_info(const eph_batch *b, int32_t *n_ensemble, int64_t *launches) {
    if (!b || !n_ensemble || !launches) return EPH_ERR_ARG;
    int k = 0;
    for (int s = 0; s < b->n_sys; ++s) k += b->point[s];
    *n_ensemble = k;
    *launches = b->launches;
    return EPH_OK;
}

}  // extern "C"
