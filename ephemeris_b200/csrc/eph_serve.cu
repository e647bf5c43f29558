// eph_serve.cu - second-stage small-body serving: massless particles integrated with adaptive RK12
// against perturbers read from a device-resident B-spline ephemeris.
//
// * Ephemeris. M perturbers, each fitted (eph_bspline_fit, src/math/interp.h:68-150) with degree-d
//   B-splines of uniform knot spacing `knot` seconds over [t0, t0 + n knot], 10 channels per body:
//   position (3), velocity (3), Newtonian acceleration / c^2 (3), potential / c^2 (1). The last four are
//   what the EIH 1PN term of a particle needs of each perturber (mass.impl:82-97); fitting them avoids an
//   O(M^2) sweep per stage, and their interpolation error enters the particle's acceleration below
//   1e-20 of it. Coefficients live in HBM as [M][n + d][10]; a stage evaluation reads, per body and
//   channel, the d + 1 coefficients of the interval and combines them with the basis values
//   B[d, x - i] (the Chebyshev form of eph_bspline_cheb_coef), as the reference's sampling does
//   (src/math/interp.h:263-280).
// * Requests. A request is P particles (double-double position and velocity), a time span and a
//   tolerance. It runs as one kernel launch of ceil(P G / 256) CTAs on one of the server's streams, G
//   lanes per particle: the smallest power of two (at most 32) that spreads the request over one block per
//   SM, so that a request's latency is that of one block's sequential stages (G = 32 up to 2352
//   particles, 16 up to 4704, 1 from 37633). Each CTA integrates its particles with
//   a shared adaptive step: one RK12 step of h and two of h/2 (step doubling); the error is the largest
//   |r_h - r_h/2| / |r_h/2 - r_0| over the CTA's particles (body 0 of the ephemeris is the central star);
//   a step is accepted when it is at most tol, and the two half steps are kept; the next step is
//   h * clamp(0.8 (tol / err)^(1/13), 0.25, 2), no larger right after a rejection. The reference has no
//   adaptive integrator (its RK12 table has no embedded pair, RungeKutta.impl:38-104); step doubling with
//   the same 25-stage method is the estimator.
// * Admission. Requests queue on the host and launch while their device memory (state, stage store)
//   fits: by default while the device's free memory (cudaMemGetInfo at admission) stays above a 1 GiB
//   reserve, or within a fixed budget set by the caller; finished requests release their memory when their
//   results are collected.
// * Particle acceleration: Newtonian + EIH 1PN against every perturber, one sweep (the 4 phi_i term of
//   mass.impl:90 factored out as 4 phi_i a_N,i), the stage combination in the second-order form of
//   eph_particles.cu (only stage accelerations stored).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <deque>
#include <map>
#include <mutex>
#include <vector>

#include "eph_bspline.h"
#include "eph_launch.cuh"
#include "eph_math.cuh"
#include "eph_rk12_host.h"
#include "eph_system.cuh"
#include "../../include/eph_b200.h"
#include "../../include/eph_planes.h"

namespace eph {
void ctx_record_stages(eph_ctx *ctx, double *d_buf, long long base);
long long ctx_size(const eph_ctx *ctx);
}

namespace eph {
namespace {

constexpr int kSThreads = 256;                 // most threads of a block that carry particles
constexpr int kSLaunch = kSThreads + 128;      // threads of a block: four warps more evaluate perturbers
constexpr size_t kFreeReserve = 1ull << 30;   // device memory kept free when admitting by free memory
constexpr int kSmemSlots = 64;   // particles per block whose stage store fits shared memory
constexpr int kSStreams = 128;   // requests in flight at once (the device runs up to 128 kernels concurrently)
constexpr int kChan = EPH_EPHEM_CHANNELS;   // x y z vx vy vz aN/c^2 (3) phi/c^2
constexpr double kCS = 299792458.0;         // src/math/basic_math.h:10,18
constexpr long long kMaxAttempts = 1ll << 22;
constexpr unsigned long long kRequestNs = 300ull * 1000000000ull;   // device-time limit of one request
// A perturber's record in shared memory: the channels at one time (velocity over c; K = phi / c^2 + 2 beta^2 in
// place of the potential), then GM. 11 doubles apart, 32 lanes reading one field of 32 consecutive records meet no bank
// conflict, and every field is a fixed offset from the record's address.
enum SRec { S_R = 0, S_B = 3, S_N = 6, S_K = 9, S_GM = 10, kSRec = 11 };
enum SStatus { SS_OK = 0, SS_STEP_UNDERFLOW = 1, SS_ATTEMPTS = 2, SS_DEADLINE = 3 };

__device__ __forceinline__ unsigned long long now_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// The Feagin table as the request kernel uses it: c_k and the rows k = 1..25 of a (hi + lo rounded) and of the
// second-order Abar = A A without the columns where both are zero (entries q_row[k] <= q < q_row[k + 1], ascending).
__constant__ double2 q_ab[EPH_RK12_NCOEF];   // {Abar_kl, a_kl}
__constant__ int q_l[EPH_RK12_NCOEF];
__constant__ int q_row[kStages + 2];
__constant__ double q_c[kStages + 1];

struct ServeArgs {
    // ephemeris
    const double *coef;        // [M][n + d][kChan]
    const double *gm, *sr2;    // [M]
    const double *cheb;        // [(d + 1)^2]: c(d, k, j)
    int M, d;
    int buffers;               // 2: the perturbers of the next stage are formed beside the present one's sums; 1: before them
    int soft;                  // any sR2 is not zero
    long long n;
    double t0, knot;
    // request
    double *state;             // [12][P] in place: r hi, r lo, v hi, v lo
    double *fstore;            // [grid][kStages][3][S] (blocks of more than kSmemSlots particles)
    int P, G, S;               // particles, lanes per particle, particles per block
    double t_start, t_end, tol, h0, hmin;
    long long *stats;          // [grid][2]: accepted, rejected
    int *status;               // [grid]
    double *hlog;              // accepted step sizes of CTA 0, or null
    int hlog_cap;
};

__device__ __forceinline__ double group_sum(double v, int G) {
    for (int o = G >> 1; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// The perturbers at time t into the shared records PR, by the warps that call it: chunks of 6 U bodies are
// taken from the counter *take until none is left. Lanes 5 b + p (b < 6, p < 5) take channels 2 p and 2 p + 1 of body
// b of six, so a warp reads 80 contiguous bytes per body and coefficient with 16-byte loads, and K is formed from
// its neighbours' channels by shuffles. No barrier.
// D > 0: degree known at compile time, U rounds of six bodies with all their coefficient loads issued before any is
// used (they come from L2: 8 bytes at a time, a body and channel per lane, the loads and their index arithmetic were a
// fifth of the kernel's instructions); D = 0: any degree. kRaw: the channels as they are fitted.
template <int D, bool kRaw>
__device__ __noinline__ void eval_rows(const double *__restrict__ coef, long long n, int deg, int M, double t0, double knot,
                                       double *PR, const double *cheb, double t, int *take) {
    const int lane = threadIdx.x & 31, d = D > 0 ? D : deg;
    constexpr int U = D > 0 ? 3 : 1;
    constexpr int NK = D > 0 ? D + 1 : EPH_BSPLINE_MAX_DEGREE + 1;
    constexpr double inv_c = 1.0 / kCS;
    const double x = (t - t0) / knot;
    long long xi = (long long)floor(x);
    xi = xi < 0 ? 0 : (xi > n - 1 ? n - 1 : xi);
    // lane k holds the basis value B[d, x - (xi + k)], k = 0..d, at u = 2 (x - xi) - 1 from its Chebyshev form
    const double u = 2 * (x - (double)xi) - 1, u2 = 2 * u;
    double mine;
    {
        const double *c = cheb + min(lane, d) * (d + 1);
        double tm, tt = 1, tp = u;
        mine = c[0] + c[1] * u;
        for (int j = 2; j <= d; ++j) {
            tm = tt;
            tt = tp;
            tp = u2 * tt - tm;
            mine += c[j] * tp;
        }
    }
    double b[NK];
#pragma unroll
    for (int k = 0; k < NK; ++k) b[k] = __shfl_sync(0xffffffffu, mine, min(k, d));
    const long long stride = (n + d) * kChan;   // doubles per body
    const int p = lane % 5, six = min(lane / 5, 5);
    const double *at = coef + xi * kChan + 2 * p;
#pragma unroll 1
    for (;;) {
        int chunk = 0;
        if (lane == 0) chunk = atomicAdd(take, 1);
        const int base = __shfl_sync(0xffffffffu, chunk, 0) * (6 * U);
        if (base >= M) break;
        double2 cf[U][NK];
#pragma unroll
        for (int q = 0; q < U; ++q) {
            const int body = min(base + q * 6 + six, M - 1);
            const double2 *c = reinterpret_cast<const double2 *>(at + body * stride);
#pragma unroll
            for (int k = 0; k < NK; ++k)
                if (D > 0 || k <= d) cf[q][k] = __ldg(c + k * (kChan / 2));
        }
#pragma unroll
        for (int q = 0; q < U; ++q) {
            const int body = base + q * 6 + lane / 5;
            double v0 = 0, v1 = 0;
#pragma unroll
            for (int k = 0; k < NK; ++k)
                if (D > 0 || k <= d) {
                    v0 += b[k] * cf[q][k].x;
                    v1 += b[k] * cf[q][k].y;
                }
            if (!kRaw) {
                // channels: p = 0 (x, y), 1 (z, vx), 2 (vy, vz), 3 (a_N x, y), 4 (a_N z, phi)
                if (p == 1) v1 *= inv_c;
                if (p == 2) { v0 *= inv_c; v1 *= inv_c; }
                const double bx = __shfl_sync(0xffffffffu, v1, max(lane - 3, 0));                     // of lane p = 1
                const double byz = __shfl_sync(0xffffffffu, v0 * v0 + v1 * v1, max(lane - 2, 0));   // of lane p = 2
                if (p == 4) v1 += 2 * (bx * bx + byz);
            }
            if (lane < 30 && body < M) {
                PR[body * kSRec + 2 * p] = v0;
                PR[body * kSRec + 2 * p + 1] = v1;
            }
        }
    }
}
__device__ __forceinline__ void eval_perturbers(const ServeArgs &A, double *PR, const double *cheb, double t, int *take) {
    if (A.d == 3) eval_rows<3, false>(A.coef, A.n, 3, A.M, A.t0, A.knot, PR, cheb, t, take);
    else eval_rows<0, false>(A.coef, A.n, A.d, A.M, A.t0, A.knot, PR, cheb, t, take);
}

// Reduce-scatter of 8 values over the GT lanes of a group (GT = 16 or 32): value v is complete on lanes
// v GT/8 .. (v + 1) GT/8 - 1 of the group. 9 shuffles (GT = 32) instead of 5 per value.
template <int GT>
__device__ __forceinline__ double group_scatter(double (&v)[8], int lane) {
#pragma unroll
    for (int h = 4, bit = GT / 2; h >= 1; h >>= 1, bit >>= 1) {
        const bool up = (lane & bit) != 0;
#pragma unroll
        for (int k = 0; k < h; ++k) {
            const double send = up ? v[k] : v[k + h], keep = up ? v[k + h] : v[k];
            v[k] = keep + __shfl_xor_sync(0xffffffffu, send, bit);
        }
    }
#pragma unroll
    for (int bit = GT / 16; bit >= 1; bit >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], bit);
    return v[0];
}

// Acceleration of a particle at (r, v): every lane of its group takes the perturbers j = lane, lane + G, ... and gets
// component c0 (GT lanes known) or all three. mass.impl:82-97 regrouped as in the ensemble and particle kernels: the
// coefficient 4 phi_i + beta_i^2 multiplies the Newtonian sum and is applied once, and with c = r.beta_j -
// 4 r.(beta_j - beta_i) = 4 r.beta_i - 3 r.beta_j the last term is c beta_j, less beta_i times the sum of the c (57 FP64
// operations a perturber, not 77). A function of its own, so that the loop has the registers to itself: inlined into
// the request loop at 128 registers it took 430 cycles a perturber and warp, with 255 registers 240.
template <int GT, bool kSoft>
__device__ __noinline__ v3 serve_accel(const double *PR, const double *SR2, int M, double rx, double rxl, double ry, double ryl,
                                       double rz, double rzl, v3 bi, int lane, int G, int c0) {
    double phi = 0, cs = 0;
    v3 na = mk(0, 0, 0), ga = mk(0, 0, 0);
    const double *R = PR + lane * kSRec;
#pragma unroll 2
    for (int j = lane; j < M; j += G, R += G * kSRec) {
        const v3 d = mk((R[S_R] - rx) - rxl, (R[S_R + 1] - ry) - ryl, (R[S_R + 2] - rz) - rzl);
        double m = dot(d, d);
        if (kSoft) {
            const double sm = SR2[j];
            m = (m < sm) ? sm : m;
        }
        const double rr = inv_sqrt(m);
        const double tp_dphi = rr * R[S_GM];
        const double tp_dg = (rr * rr) * tp_dphi;
        phi -= tp_dphi;
        na = mk(fma(tp_dg, d.x, na.x), fma(tp_dg, d.y, na.y), fma(tp_dg, d.z, na.z));
        const v3 bj = mk(R[S_B], R[S_B + 1], R[S_B + 2]), nj = mk(R[S_N], R[S_N + 1], R[S_N + 2]);
        const double rbj = dot(d, bj), rbi = dot(d, bi), rn = dot(d, nj), bb = dot(bi, bj);
        double tp = rbj * rr;
        tp *= tp;
        const double w = tp_dg * fma(-1.5, tp, fma(0.5, rn, fma(-4.0, bb, R[S_K])));
        const double c = tp_dg * fma(4.0, rbi, -3.0 * rbj);
        const double h = 3.5 * tp_dphi;
        cs += c;
        ga.x = fma(c, bj.x, fma(w, d.x, fma(h, nj.x, ga.x)));
        ga.y = fma(c, bj.y, fma(w, d.y, fma(h, nj.y, ga.y)));
        ga.z = fma(c, bj.z, fma(w, d.z, fma(h, nj.z, ga.z)));
    }
    ga = ga - cs * bi;
    const double beta2 = dot(bi, bi), c2i = 1.0 / (kCS * kCS);
    if (GT >= 16) {
        constexpr int W = GT >= 16 ? GT : 32, per = W / 8;
        double sums[8] = {phi, na.x, na.y, na.z, ga.x, ga.y, ga.z, 0.0};
        const double x = group_scatter<W>(sums, lane);
        const double p = __shfl_sync(0xffffffffu, x, 0, W), n = __shfl_sync(0xffffffffu, x, per * (1 + c0), W),
                     g = __shfl_sync(0xffffffffu, x, per * (4 + c0), W);
        return mk((g + (4 * (p * c2i) + beta2) * n) + n, 0.0, 0.0);
    }
    phi = group_sum(phi, G) * c2i;
    na = mk(group_sum(na.x, G), group_sum(na.y, G), group_sum(na.z, G));
    ga = mk(group_sum(ga.x, G), group_sum(ga.y, G), group_sum(ga.z, G));
    return (ga + (4 * phi + beta2) * na) + na;
}

// One request. GT: lanes per particle when known (16 and 32, requests of less than about 4700 particles: each lane
// then carries one component of the particle's state through the stage combination), 0 for any number.
//
// One attempt is one RK12 step of h from X0 (phase 0: its end position to RF) and two of h/2 (phase 1: X0 to X1,
// phase 2: X1 to X1), in second-order form: r_k = r0 + h (c_k v0 + h sum_l Abar_kl f_l), v_k = v0 + h sum_l a_kl f_l with
// the stage accelerations f_l in F; the same code serves every stage of the three.
//
// What bounds it: per stage, the dependent FP64 chains of serve_accel (13 perturbers a lane with 419 of them and a warp
// per particle) and the spline coefficients, 134 KB from L2. So the perturbers of the next stage are formed beside
// the present stage's sums into a second set of records, one CTA barrier a stage: four warps of a block do nothing
// else, and a warp that has its sums, or no particle, takes chunks as well. One block of 384 threads an SM: the 168
// registers a thread let two perturbers' chains overlap; at 128 registers, with two blocks of 256 an SM, a perturber
// took 430 cycles a warp instead of 240. Requests alone, 360 days, against a body and channel per lane, the
// perturbers before the sums and 128 registers: 5 particles 9.2 -> 3.7 ms, 300 (100 days) 10.4 -> 5.7, 4096 (60 days)
// 20.9 -> 12.4; 100 requests at once 285 -> 219 ms (two blocks an SM: 216). 320 threads a block: 4.1, 6.4, 13.9, 243
// ms; 512: 4.8, 6.6, 14.8, 255. Requests of more blocks than SMs (30 days, one block an SM where there were two): 20,000
// particles 61.8 -> 47.5 ms, 40,000 149 -> 119, 75,776 165.5 -> 155, 150,000 275 -> 246, 1,000,000 1563 -> 1474.
template <int GT, bool kSoft>
__global__ void __launch_bounds__(kSLaunch, 1) serve_kernel(ServeArgs A) {
    extern __shared__ __align__(16) double sm[];
    __shared__ double cheb[(EPH_BSPLINE_MAX_DEGREE + 1) * (EPH_BSPLINE_MAX_DEGREE + 1)];
    __shared__ double red[kSLaunch / 32];
    __shared__ double2 ab[EPH_RK12_NCOEF];
    __shared__ int li[EPH_RK12_NCOEF];
    __shared__ unsigned long long s_t0;
    __shared__ int s_late, s_take[2];
    constexpr bool kSplit = GT >= 16;
    constexpr int NC = kSplit ? 1 : 3;             // components per lane in the stage combination
    const int G = GT > 0 ? GT : A.G, S = A.S;
    const bool worker = (int)threadIdx.x < S * G;   // (whole warps)
    const int slot = worker ? threadIdx.x / G : 0, lane = threadIdx.x % G;
    const int c0 = kSplit ? lane % 3 : 0;          // this lane's (first) component
    const int set = A.M * kSRec;                   // doubles of one set of records
    double *rows = sm;                             // [buffers][M][kSRec], then sR2 [M] if any
    double *SR2 = rows + A.buffers * set;
    double *X0 = SR2 + (kSoft ? A.M : 0);          // [12][S]
    double *X1 = X0 + 12 * S;                      // [12][S]
    double *RF = X1 + 12 * S;                      // [6][S]
    // stage store [kStages][3][S]: shared memory for blocks of up to kSmemSlots particles, else global
    double *F = (S <= kSmemSlots ? RF + 6 * S : A.fstore + (size_t)blockIdx.x * kStages * 3 * S) + slot;
    const int ip = blockIdx.x * S + slot;
    const bool live = worker && ip < A.P;
    for (int q = threadIdx.x; q < (A.d + 1) * (A.d + 1); q += blockDim.x) cheb[q] = A.cheb[q];
    for (int q = threadIdx.x; q < EPH_RK12_NCOEF; q += blockDim.x) {
        ab[q] = q_ab[q];
        li[q] = q_l[q] * 3 * S;
    }
    for (int j = threadIdx.x; j < A.M; j += blockDim.x) {
        for (int b = 0; b < A.buffers; ++b) rows[b * set + j * kSRec + S_GM] = A.gm[j];
        if (kSoft) SR2[j] = A.sr2[j];
    }
    if (worker)
        for (int q = lane; q < 12; q += G) X0[q * S + slot] = live ? A.state[(size_t)q * A.P + ip] : (q < 3 ? 1e30 : 0.0);
    if (threadIdx.x == 0) {
        s_t0 = now_ns();
        s_take[0] = s_take[1] = 0;
    }
    __syncthreads();
    int cur = 0;               // rows of the present stage
    // Acceleration of the particle at (r, v) with the perturbers of the rows in use, this lane's component(s) to fa;
    // forms those at time t_next (if `more`) into the other rows.
    auto stage = [&](const dd r[3], v3 v, double t_now, bool fresh, double t_next, bool more, double (&fa)[NC]) {
        double *now = rows + cur * set;
        if (fresh || A.buffers == 1) {   // nothing prepared: form them now
            __syncthreads();
            eval_perturbers(A, now, cheb, t_now, &s_take[cur]);
        }
        __syncthreads();   // the rows are complete, and no warp still reads the others
        if (threadIdx.x == 0) s_take[cur] = 0;
        const int to = cur ^ 1;
        double *next = rows + to * set;
        const bool ahead = more && A.buffers == 2;
        if (ahead) cur = to;
        if (!worker) {
            if (ahead) eval_perturbers(A, next, cheb, t_next, &s_take[to]);
            return;
        }
        const v3 bi = mk(v.x * (1.0 / kCS), v.y * (1.0 / kCS), v.z * (1.0 / kCS));
        const v3 f = serve_accel<GT, kSoft>(now, SR2, A.M, r[0].hi, r[0].lo, r[1].hi, r[1].lo, r[2].hi, r[2].lo, bi, lane, G, c0);
        const double fc[3] = {f.x, f.y, f.z};
#pragma unroll
        for (int ci = 0; ci < NC; ++ci) fa[ci] = live ? fc[ci] : 0.0;
        if (ahead) eval_perturbers(A, next, cheb, t_next, &s_take[to]);
    };
    const double dir = A.t_end >= A.t_start ? 1.0 : -1.0;
    double t = A.t_start;
    double f0[NC] = {}, fm[NC] = {}, fe[NC] = {};   // f at the start, the middle and the end of the attempt
    {
        dd r[3];
        for (int c = 0; c < 3; ++c) r[c] = dd{X0[c * S + slot], X0[(3 + c) * S + slot]};
        const v3 v = mk(dd_val(dd{X0[6 * S + slot], X0[9 * S + slot]}), dd_val(dd{X0[7 * S + slot], X0[10 * S + slot]}),
                        dd_val(dd{X0[8 * S + slot], X0[11 * S + slot]}));
        stage(r, v, t, true, t, false, f0);
    }
    double h = fabs(A.h0);
    bool just_rejected = false;
    long long accepted = 0, rejected = 0;
    int status = SS_OK;
#pragma unroll 1
    for (long long attempt = 0; dir * (A.t_end - t) > 0; ++attempt) {
        if (attempt >= kMaxAttempts) { status = SS_ATTEMPTS; break; }
        if (threadIdx.x == 0) s_late = now_ns() - s_t0 > kRequestNs;
        __syncthreads();
        if (s_late) { status = SS_DEADLINE; break; }
        const double remaining = dir * (A.t_end - t);
        const bool last = h >= remaining;
        const double hs = dir * (last ? remaining : h);
        bool fresh = true;
        int phase = 0, k = 1;
#pragma unroll 1
        for (;;) {
            const double hp = phase == 0 ? hs : hs / 2, tp = phase == 2 ? t + hs / 2 : t;
            const double *Xin = (phase == 2 ? X1 : X0) + slot;
            double rh[NC] = {}, rl[NC] = {}, vv[NC] = {};
            if (worker) {
                if (k == 1) {
#pragma unroll
                    for (int ci = 0; ci < NC; ++ci)
                        if (kSplit ? lane < 3 : lane == 0) F[(c0 + ci) * S] = phase == 2 ? fm[ci] : f0[ci];
                    __syncwarp();
                }
                double s1[NC], s2[NC];
#pragma unroll
                for (int ci = 0; ci < NC; ++ci) s1[ci] = s2[ci] = 0.0;
                const int q1 = q_row[k + 1];
                if (k < kStages) {
#pragma unroll 4
                    for (int q = q_row[k]; q < q1; ++q) {
                        const double2 a = ab[q];
#pragma unroll
                        for (int ci = 0; ci < NC; ++ci) {
                            const double f = F[li[q] + (c0 + ci) * S];
                            s1[ci] = __fma_rn(a.x, f, s1[ci]);
                            s2[ci] = __fma_rn(a.y, f, s2[ci]);
                        }
                    }
                    const double ck = q_c[k];
#pragma unroll
                    for (int ci = 0; ci < NC; ++ci) {
                        const int c = c0 + ci;
                        const double v0 = Xin[(6 + c) * S];
                        double e;
                        two_sum(Xin[c * S], hp * __fma_rn(ck, v0, hp * s1[ci]), rh[ci], e);
                        rl[ci] = e + Xin[(3 + c) * S];
                        vv[ci] = v0 + __fma_rn(hp, s2[ci], Xin[(9 + c) * S]);
                    }
                } else {
#pragma unroll 1
                    for (int q = q_row[k]; q < q1; ++q) {
                        const double2 a = ab[q];
#pragma unroll
                        for (int ci = 0; ci < NC; ++ci) {
                            const double f = F[li[q] + (c0 + ci) * S];
                            s1[ci] = __fma_rn(a.x, f, s1[ci]);
                            if (a.y != 0) s2[ci] = __dadd_rn(s2[ci], __dmul_rn(a.y, f));
                        }
                    }
                    const dd ck = dd_make(q_c[k]), dh = dd_make(hp);
                    dd rn[NC], vn[NC];
#pragma unroll
                    for (int ci = 0; ci < NC; ++ci) {
                        const int c = c0 + ci;
                        const dd v0 = dd{Xin[(6 + c) * S], Xin[(9 + c) * S]};
                        const dd sv = dd_add(dd_mul(ck, v0), dd_make(hp * s1[ci]));
                        rn[ci] = dd_add(dd{Xin[c * S], Xin[(3 + c) * S]}, dd_mul(dh, sv));
                        vn[ci] = dd_add(v0, dd_make(hp * s2[ci]));
                        rh[ci] = rn[ci].hi;
                        rl[ci] = rn[ci].lo;
                        vv[ci] = dd_val(vn[ci]);
                    }
                    __syncwarp();   // every lane of the group has read Xin before it is overwritten
                    double *Xout = (phase == 0 ? RF : X1) + slot;
#pragma unroll
                    for (int ci = 0; ci < NC; ++ci) {
                        const int c = c0 + ci;
                        if (kSplit ? lane < 3 : lane == 0) {
                            Xout[c * S] = rn[ci].hi;
                            Xout[(3 + c) * S] = rn[ci].lo;
                            if (phase > 0) {
                                Xout[(6 + c) * S] = vn[ci].hi;
                                Xout[(9 + c) * S] = vn[ci].lo;
                            }
                        }
                    }
                    __syncwarp();
                }
            }
            if (k == kStages && phase == 0) {   // the whole step's end needs no acceleration
                phase = 1;
                k = 1;
                continue;
            }
            dd r[3];
            v3 v;
            if (kSplit) {
                constexpr int W = kSplit ? GT : 32;
                double vc[3];
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    r[c] = dd{__shfl_sync(0xffffffffu, rh[0], c, W), __shfl_sync(0xffffffffu, rl[0], c, W)};
                    vc[c] = __shfl_sync(0xffffffffu, vv[0], c, W);
                }
                v = mk(vc[0], vc[1], vc[2]);
            } else {
#pragma unroll
                for (int c = 0; c < 3; ++c) r[c] = dd{rh[c % NC], rl[c % NC]};
                v = mk(vv[0], vv[1 % NC], vv[2 % NC]);
            }
            // the next stage that needs the perturbers, and its time
            int np = phase, nk = k + 1;
            if (nk > kStages || (np == 0 && nk == kStages)) { ++np; nk = 1; }
            const double nh = np == 0 ? hs : hs / 2, nt = (np == 2 ? t + hs / 2 : t) + q_c[nk] * nh;
            double fa[NC] = {};
            stage(r, v, tp + q_c[k] * hp, fresh, nt, np <= 2, fa);
            fresh = false;
            if (k < kStages) {
#pragma unroll
                for (int ci = 0; ci < NC; ++ci)
                    if (worker && (kSplit ? lane < 3 : lane == 0)) F[(k * 3 + c0 + ci) * S] = fa[ci];
                __syncwarp();
                ++k;
                continue;
            }
#pragma unroll
            for (int ci = 0; ci < NC; ++ci) {
                if (phase == 1) fm[ci] = fa[ci];
                else fe[ci] = fa[ci];
            }
            if (phase == 2) break;
            phase = 2;
            k = 1;
        }
        // error of the particle: |r_h - r_h/2| / |r_h/2 - r_star(t + h)| (the last stage evaluated the
        // ephemeris at t + h)
        const double *PR = rows + cur * set;
        double e = 0;
        if (live && lane == 0) {
            double num = 0, den = 0;
            for (int c = 0; c < 3; ++c) {
                const double dr = (X1[c * S + slot] - RF[c * S + slot]) + (X1[(3 + c) * S + slot] - RF[(3 + c) * S + slot]);
                const double rs = (X1[c * S + slot] - PR[S_R + c]) + X1[(3 + c) * S + slot];
                num += dr * dr;
                den += rs * rs;
            }
            e = sqrt(num / den);
        }
        // CTA maximum, NaN-propagating
        for (int o = 16; o > 0; o >>= 1) {
            const double u = __shfl_xor_sync(0xffffffffu, e, o);
            e = (e != e || u > e || u != u) ? ((e != e) ? e : u) : e;
        }
        __syncthreads();
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = e;
        __syncthreads();
        double err = red[0];
        for (int w = 1; w < (int)(blockDim.x / 32); ++w) {
            const double u = red[w];
            err = (err != err || u > err || u != u) ? ((err != err) ? err : u) : err;
        }
        const double hused = fabs(hs);
        if (err <= A.tol) {   // accept the two half steps
            if (worker)
                for (int q = lane; q < 12; q += G) X0[q * S + slot] = X1[q * S + slot];
            if (A.hlog && blockIdx.x == 0 && threadIdx.x == 0 && accepted < A.hlog_cap) A.hlog[accepted] = hs;
#pragma unroll
            for (int ci = 0; ci < NC; ++ci) f0[ci] = fe[ci];
            t = last ? A.t_end : t + hs;
            ++accepted;
        } else {
            ++rejected;
        }
        // next step: 0.8 (tol / err)^(1/13) within [0.25, 2], no growth right after a rejection
        // (the factor only steers the step size: single precision is ample)
        double fac = (err == 0) ? 2.0 : (err != err) ? 0.25 : 0.8 * (double)powf((float)(A.tol / err), 1.0f / 13.0f);
        fac = fac < 0.25 ? 0.25 : (fac > 2.0 ? 2.0 : fac);
        if (just_rejected && fac > 1.0) fac = 1.0;
        just_rejected = !(err <= A.tol);
        h = hused * fac;
        if (h < A.hmin && dir * (A.t_end - t) > 0) { status = SS_STEP_UNDERFLOW; break; }
        __syncwarp();
    }
    __syncthreads();
    if (live)
        for (int q = lane; q < 12; q += G) A.state[(size_t)q * A.P + ip] = X0[q * S + slot];
    if (threadIdx.x == 0) {
        A.stats[2 * blockIdx.x] = accepted;
        A.stats[2 * blockIdx.x + 1] = rejected;
        A.status[blockIdx.x] = status;
    }
}

// the ephemeris at time t into out[M][kChan] (one CTA)
__global__ void __launch_bounds__(kSThreads) eval_kernel(ServeArgs A, double t, double *out) {
    extern __shared__ __align__(16) double sm[];
    __shared__ double cheb[(EPH_BSPLINE_MAX_DEGREE + 1) * (EPH_BSPLINE_MAX_DEGREE + 1)];
    for (int q = threadIdx.x; q < (A.d + 1) * (A.d + 1); q += blockDim.x) cheb[q] = A.cheb[q];
    __shared__ int take;
    if (threadIdx.x == 0) take = 0;
    __syncthreads();
    if (A.d == 3) eval_rows<3, true>(A.coef, A.n, 3, A.M, A.t0, A.knot, sm, cheb, t, &take);
    else eval_rows<0, true>(A.coef, A.n, A.d, A.M, A.t0, A.knot, sm, cheb, t, &take);
    __syncthreads();
    for (int item = threadIdx.x; item < A.M * kChan; item += blockDim.x) out[item] = sm[item / kChan * kSRec + item % kChan];
}

// step-end stage records of sampled steps into [samples][M][kChan]
__global__ void gather_samples(const double *traj, int M, int n_take, long long first_step, int stride, double *out) {
    // sample q of this chunk is the end of local step (first_step + q * stride); its record slot is
    // 1 + local_step * kStages + (kStages - 1)
    const long long total = (long long)n_take * M;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
        const long long q = i / M;
        const int j = (int)(i % M);
        const long long local = first_step + q * stride;
        const double *rec = traj + ((size_t)(1 + local * kStages + (kStages - 1)) * M + j) * kTrajRec;
        double *o = out + (size_t)i * kChan;
        for (int c = 0; c < 3; ++c) {
            o[c] = rec[TR_R_HI + c] + rec[TR_R_LO + c];
            o[3 + c] = rec[TR_BETA + c] * kCS;
            o[6 + c] = rec[TR_NACC + c];
        }
        o[9] = rec[TR_PHI];
    }
}

// Batch B-spline fit: right-hand side and the two banded substitutions of one (series, channel) per
// thread, with the grid's factorization from bspline_factor (eph_bspline.h). The double-double operations
// are those of the host fit (eph_bspline.cpp) in the same order, so the coefficients are bit-identical.
__global__ void bspline_solve_kernel(int d, long long m, int J, int channels, long long n_series, long long series_stride,
                                     const double *__restrict__ samples, const long long *__restrict__ jmin,
                                     const int *__restrict__ cnt, const double *__restrict__ bval,
                                     const double *__restrict__ rw, const double *__restrict__ lu,
                                     const double *__restrict__ rd, double *__restrict__ y, double *__restrict__ coefs) {
    const long long T = n_series * channels;
    const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (t >= T) return;
    const long long sidx = t / channels;
    const int c = (int)(t % channels);
    const int w = 2 * d + 1;
    const double *smp = samples + sidx * series_stride + c;
    // y[i] (hi, lo) at y[(2 i) * T + t], y[(2 i + 1) * T + t]
#pragma unroll 1
    for (long long i = 0; i < m; ++i) {
        dd yi = dd_make(0);
        const long long j0 = jmin[i];
#pragma unroll 1
        for (int q = 0; q < cnt[i]; ++q)
            yi = dd_add(yi, dd_mul(dd_make(smp[(j0 + q) * channels]), dd_make(bval[i * J + q])));
        yi = dd_mul(yi, dd{rw[2 * i], rw[2 * i + 1]});
#pragma unroll 1
        for (long long k = i - d < 0 ? 0 : i - d; k < i; ++k) {
            const long long qq = i * w + (k - i + d);
            yi = dd_sub(yi, dd_mul(dd{lu[2 * qq], lu[2 * qq + 1]}, dd{y[(2 * k) * T + t], y[(2 * k + 1) * T + t]}));
        }
        y[(2 * i) * T + t] = yi.hi;
        y[(2 * i + 1) * T + t] = yi.lo;
    }
#pragma unroll 1
    for (long long i = m - 1; i >= 0; --i) {
        dd yi = dd{y[(2 * i) * T + t], y[(2 * i + 1) * T + t]};
        const long long hi = i + d < m - 1 ? i + d : m - 1;
#pragma unroll 1
        for (long long j = i + 1; j <= hi; ++j) {
            const long long qq = i * w + (j - i + d);
            yi = dd_sub(yi, dd_mul(dd{lu[2 * qq], lu[2 * qq + 1]}, dd{y[(2 * j) * T + t], y[(2 * j + 1) * T + t]}));
        }
        yi = dd_mul(yi, dd{rd[2 * i], rd[2 * i + 1]});
        y[(2 * i) * T + t] = yi.hi;
        y[(2 * i + 1) * T + t] = yi.lo;
        coefs[(sidx * m + i) * channels + c] = __dadd_rn(yi.hi, yi.lo);
    }
}

using ServeKernel = void (*)(ServeArgs);
ServeKernel serve_kernel_of(int G, bool soft) {
    if (G == 32) return soft ? serve_kernel<32, true> : serve_kernel<32, false>;
    if (G == 16) return soft ? serve_kernel<16, true> : serve_kernel<16, false>;
    return soft ? serve_kernel<0, true> : serve_kernel<0, false>;
}
constexpr size_t kServeSmem = 216 * 1024;       // most dynamic shared memory of a block

bool g_serve_ready[64];
cudaError_t serve_setup(int device) {
    if (device >= 0 && device < 64 && g_serve_ready[device]) return cudaSuccess;
    double hi[EPH_RK12_NCOEF], lo[EPH_RK12_NCOEF], dtk[kStages + 1];
    rk12_expand(hi, lo, dtk);
    auto coef = [&](int k, int j) { return (long double)hi[k * (k - 1) / 2 + j] + lo[k * (k - 1) / 2 + j]; };
    double2 tab[EPH_RK12_NCOEF] = {};
    int ll[EPH_RK12_NCOEF] = {}, row[kStages + 2] = {}, q = 0;
    for (int k = 1; k <= kStages; ++k) {   // Abar = A A (second-order form), long double accumulation
        row[k] = q;
        for (int l = 0; l < k; ++l) {
            long double acc = 0;
            bool any = hi[k * (k - 1) / 2 + l] != 0;
            for (int j = l + 1; j < k; ++j) {
                acc += coef(k, j) * coef(j, l);
                any = any || (hi[k * (k - 1) / 2 + j] != 0 && hi[j * (j - 1) / 2 + l] != 0);
            }
            if (!any) continue;
            tab[q] = make_double2((double)acc, hi[k * (k - 1) / 2 + l] + lo[k * (k - 1) / 2 + l]);
            ll[q++] = l;
        }
    }
    row[kStages + 1] = q;
    cudaError_t e = cudaMemcpyToSymbol(q_ab, tab, sizeof(tab));
    if (e == cudaSuccess) e = cudaMemcpyToSymbol(q_l, ll, sizeof(ll));
    if (e == cudaSuccess) e = cudaMemcpyToSymbol(q_row, row, sizeof(row));
    if (e == cudaSuccess) e = cudaMemcpyToSymbol(q_c, dtk, sizeof(dtk));
    for (int G : {0, 16, 32})
        for (int soft = 0; soft < 2 && e == cudaSuccess; ++soft)
            e = cudaFuncSetAttribute(serve_kernel_of(G, soft), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kServeSmem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(eval_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    if (e == cudaSuccess && device >= 0 && device < 64) g_serve_ready[device] = true;
    return e;
}

size_t serve_smem(int M, int S, int buffers, bool soft) {
    return (size_t)((buffers * kSRec + (soft ? 1 : 0)) * M + 30 * S + (S <= kSmemSlots ? kStages * 3 * S : 0)) * sizeof(double);
}
// Sets of perturber records: two, where the second fits
int serve_buffers(int M, int S, bool soft) { return serve_smem(M, S, 2, soft) <= kServeSmem ? 2 : 1; }

}  // namespace
}  // namespace eph

using namespace eph;

struct eph_serve {
    int device = 0;
    std::mutex mu;
    char err[512] = {0};
    cudaStream_t streams[kSStreams] = {};
    int next_stream = 0;
    int sms = 148;
    int M = 0, d = 0;
    bool soft = false;                 // any sR2 is not zero
    long long n = 0;
    double t0 = 0, knot = 0;
    double *d_coef = nullptr, *d_gm = nullptr, *d_sr2 = nullptr, *d_cheb = nullptr;
    size_t budget = 0, in_use = 0;
    int64_t log_cap = 0;
    struct Req {
        int P = 0, G = 1, grid = 0, block = kSThreads;
        double t_start = 0, t_end = 0, tol = 0, h0 = 0;
        std::vector<double> host_in;
        double *d_state = nullptr, *d_fstore = nullptr, *d_hlog = nullptr;
        long long *d_stats = nullptr;
        int *d_status = nullptr;
        cudaEvent_t done = nullptr;
        int stream = 0;
        bool launched = false;
        size_t bytes = 0;
        int64_t log_cap = 0;
    };
    std::map<int64_t, Req> reqs;
    std::deque<int64_t> pending;
    int64_t next_id = 1;
    int64_t launches = 0;
};

static int sfail(eph_serve *s, int code, const char *what, cudaError_t e = cudaSuccess) {
    if (s) {
        if (e != cudaSuccess) snprintf(s->err, sizeof(s->err), "%s: %s", what, cudaGetErrorString(e));
        else snprintf(s->err, sizeof(s->err), "%s", what);
    }
    return code;
}
#define SCK(call, what)                                                                                     \
    do {                                                                                                    \
        cudaError_t e_ = (call);                                                                            \
        if (e_ != cudaSuccess) return sfail(s, e_ == cudaErrorMemoryAllocation ? EPH_ERR_OOM : EPH_ERR_CUDA, what, e_); \
    } while (0)

static size_t req_bytes(const eph_serve::Req &r) {
    const int S = r.block / r.G;
    return (size_t)12 * r.P * sizeof(double) + (S > kSmemSlots ? (size_t)r.grid * kStages * 3 * S * sizeof(double) : 0) +
           (size_t)r.grid * (2 * sizeof(long long) + sizeof(int)) + (size_t)r.log_cap * sizeof(double);
}

static void req_free(eph_serve::Req &r, cudaStream_t st) {
    for (void *q : {(void *)r.d_state, (void *)r.d_fstore, (void *)r.d_stats, (void *)r.d_status, (void *)r.d_hlog})
        if (q) cudaFreeAsync(q, st);
    r.d_state = r.d_fstore = r.d_hlog = nullptr;
    r.d_stats = nullptr;
    r.d_status = nullptr;
}

// launch queued requests, oldest first, while their memory fits the budget
static int pump(eph_serve *s) {
    while (!s->pending.empty()) {
        auto &r = s->reqs[s->pending.front()];
        if (s->in_use > 0) {
            if (s->budget > 0) {
                if (s->in_use + r.bytes > s->budget) break;
            } else {   // admission by free device memory
                size_t free_b = 0, total_b = 0;
                if (cudaMemGetInfo(&free_b, &total_b) != cudaSuccess || free_b < r.bytes + kFreeReserve) break;
            }
        }
        cudaStream_t st = s->streams[r.stream];
        const int S = r.block / r.G;
        cudaError_t e = cudaMallocAsync((void **)&r.d_state, (size_t)12 * r.P * sizeof(double), st);
        if (e == cudaSuccess && S > kSmemSlots)
            e = cudaMallocAsync((void **)&r.d_fstore, (size_t)r.grid * kStages * 3 * S * sizeof(double), st);
        if (e == cudaSuccess) e = cudaMallocAsync((void **)&r.d_stats, (size_t)r.grid * 2 * sizeof(long long), st);
        if (e == cudaSuccess) e = cudaMallocAsync((void **)&r.d_status, (size_t)r.grid * sizeof(int), st);
        if (e == cudaSuccess && r.log_cap > 0) e = cudaMallocAsync((void **)&r.d_hlog, (size_t)r.log_cap * sizeof(double), st);
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(r.d_state, r.host_in.data(), r.host_in.size() * sizeof(double), cudaMemcpyHostToDevice, st);
        if (e != cudaSuccess) {   // the request stays queued, holding nothing
            req_free(r, st);
            return sfail(s, e == cudaErrorMemoryAllocation ? EPH_ERR_OOM : EPH_ERR_CUDA, "admit request", e);
        }
        ServeArgs A;
        A.coef = s->d_coef; A.gm = s->d_gm; A.sr2 = s->d_sr2; A.cheb = s->d_cheb;
        A.M = s->M; A.d = s->d; A.n = s->n; A.t0 = s->t0; A.knot = s->knot;
        A.state = r.d_state; A.fstore = r.d_fstore; A.P = r.P; A.G = r.G;
        A.t_start = r.t_start; A.t_end = r.t_end; A.tol = r.tol; A.h0 = r.h0;
        A.hmin = std::max(1e-9 * std::fabs(r.t_end - r.t_start), 1e-3);
        A.stats = r.d_stats; A.status = r.d_status; A.hlog = r.d_hlog; A.hlog_cap = (int)r.log_cap;
        A.S = S;
        A.soft = s->soft;
        A.buffers = serve_buffers(s->M, S, s->soft);
        // a full block's warps whatever the particles: the warps without any evaluate perturbers
        SCK(launch_kernel(serve_kernel_of(r.G, s->soft), r.grid, kSLaunch, serve_smem(s->M, S, A.buffers, s->soft), st, A),
            "launch serve kernel");
        SCK(cudaEventRecord(r.done, st), "record event");
        r.launched = true;
        s->in_use += r.bytes;
        ++s->launches;
        r.host_in.clear();
        r.host_in.shrink_to_fit();
        s->pending.pop_front();
    }
    return EPH_OK;
}

extern "C" {

int eph_serve_create(int device, int64_t n_pert, const double *gm, const double *sr2, int degree, int64_t n_intervals,
                     double t0, double knot, const double *coefs, eph_serve **out) {
    if (!out) return EPH_ERR_ARG;
    *out = nullptr;
    if (n_pert < 1 || n_pert > EPH_SERVE_MAX_PERTURBERS || !gm || degree < 1 || degree > EPH_BSPLINE_MAX_DEGREE ||
        n_intervals < 1 || !(knot > 0) || !coefs)
        return EPH_ERR_ARG;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || device < 0 || device >= ndev) return EPH_ERR_ARG;
    eph_serve *s = new eph_serve();
    s->device = device;
    s->M = (int)n_pert;
    s->d = degree;
    s->n = n_intervals;
    s->t0 = t0;
    s->knot = knot;
    for (int64_t j = 0; sr2 && j < n_pert; ++j) s->soft = s->soft || sr2[j] != 0;
    auto bail = [&](int code, const char *what, cudaError_t e) {
        sfail(s, code, what, e);
        eph_serve_destroy(s);
        return code;
    };
    cudaError_t e = cudaSetDevice(device);
    if (e == cudaSuccess) e = serve_setup(device);
    for (int i = 0; i < kSStreams && e == cudaSuccess; ++i) e = cudaStreamCreateWithFlags(&s->streams[i], cudaStreamNonBlocking);
    if (e != cudaSuccess) return bail(EPH_ERR_CUDA, "serve setup", e);
    const size_t ncoef = (size_t)n_pert * (n_intervals + degree) * kChan;
    std::vector<double> cheb((degree + 1) * (degree + 1)), zeros(n_pert, 0.0);
    for (int k = 0; k <= degree; ++k)
        for (int j = 0; j <= degree; ++j) cheb[k * (degree + 1) + j] = eph_bspline_cheb_coef(degree, k, j);
    if ((e = cudaMalloc(&s->d_coef, ncoef * sizeof(double))) != cudaSuccess ||
        (e = cudaMalloc(&s->d_gm, n_pert * sizeof(double))) != cudaSuccess ||
        (e = cudaMalloc(&s->d_sr2, n_pert * sizeof(double))) != cudaSuccess ||
        (e = cudaMalloc(&s->d_cheb, cheb.size() * sizeof(double))) != cudaSuccess)
        return bail(e == cudaErrorMemoryAllocation ? EPH_ERR_OOM : EPH_ERR_CUDA, "cudaMalloc(ephemeris)", e);
    if ((e = cudaMemcpy(s->d_coef, coefs, ncoef * sizeof(double), cudaMemcpyHostToDevice)) != cudaSuccess ||
        (e = cudaMemcpy(s->d_gm, gm, n_pert * sizeof(double), cudaMemcpyHostToDevice)) != cudaSuccess ||
        (e = cudaMemcpy(s->d_sr2, sr2 ? sr2 : zeros.data(), n_pert * sizeof(double), cudaMemcpyHostToDevice)) != cudaSuccess ||
        (e = cudaMemcpy(s->d_cheb, cheb.data(), cheb.size() * sizeof(double), cudaMemcpyHostToDevice)) != cudaSuccess)
        return bail(EPH_ERR_CUDA, "upload ephemeris", e);
    cudaDeviceGetAttribute(&s->sms, cudaDevAttrMultiProcessorCount, device);
    s->budget = 0;   // admission by free device memory
    *out = s;
    return EPH_OK;
}

int eph_serve_destroy(eph_serve *s) {
    if (!s) return EPH_ERR_ARG;
    cudaSetDevice(s->device);
    for (auto &kv : s->reqs) {
        if (kv.second.done) cudaEventSynchronize(kv.second.done);
        req_free(kv.second, s->streams[kv.second.stream]);
        if (kv.second.done) cudaEventDestroy(kv.second.done);
    }
    for (int i = 0; i < kSStreams; ++i)
        if (s->streams[i]) {
            cudaStreamSynchronize(s->streams[i]);
            cudaStreamDestroy(s->streams[i]);
        }
    for (void *q : {(void *)s->d_coef, (void *)s->d_gm, (void *)s->d_sr2, (void *)s->d_cheb})
        if (q) cudaFree(q);
    delete s;
    return EPH_OK;
}

const char *eph_serve_last_error(const eph_serve *s) { return s ? s->err : "null server"; }

int eph_serve_set_budget(eph_serve *s, int64_t bytes) {
    if (!s || bytes < 0) return EPH_ERR_ARG;
    std::lock_guard<std::mutex> lock(s->mu);
    s->budget = (size_t)bytes;
    return EPH_OK;
}

int eph_serve_set_step_log(eph_serve *s, int64_t cap) {
    if (!s || cap < 0 || cap > (1 << 24)) return EPH_ERR_ARG;
    std::lock_guard<std::mutex> lock(s->mu);
    s->log_cap = cap;
    return EPH_OK;
}

int eph_serve_submit(eph_serve *s, int64_t n_part, const double *part_state, double t_start, double t_end, double tol,
                     double h0, int64_t *id) {
    if (!s || !part_state || !id || n_part < 1 || n_part > (1 << 24) || !(tol > 0) || !(h0 > 0) ||
        !std::isfinite(t_start) || !std::isfinite(t_end))
        return sfail(s, EPH_ERR_ARG, "eph_serve_submit: bad arguments");
    std::lock_guard<std::mutex> lock(s->mu);
    const double lo = s->t0, hi = s->t0 + (double)s->n * s->knot;
    if (std::min(t_start, t_end) < lo || std::max(t_start, t_end) > hi)
        return sfail(s, EPH_ERR_ARG, "eph_serve_submit: span outside the ephemeris");
    SCK(cudaSetDevice(s->device), "cudaSetDevice");
    eph_serve::Req r;
    r.P = (int)n_part;
    // lanes per particle: split the perturber sweep until the request spans one block per SM (its latency
    // is one block's sequential stage count), at most a warp per particle
    int G = 1;
    while (G < 32 && (n_part * G + kSThreads - 1) / kSThreads < s->sms) G *= 2;
    r.G = G;
    // small requests take a smaller block (whole warps): one warp for a single particle
    r.block = (int)std::min<int64_t>(kSThreads, (n_part * G + 31) / 32 * 32);
    r.grid = (int)((n_part * G + r.block - 1) / r.block);
    r.t_start = t_start; r.t_end = t_end; r.tol = tol; r.h0 = h0;
    r.host_in.assign(part_state, part_state + (size_t)12 * n_part);
    r.stream = s->next_stream;
    s->next_stream = (s->next_stream + 1) % kSStreams;
    r.log_cap = s->log_cap;
    r.bytes = req_bytes(r);
    SCK(cudaEventCreateWithFlags(&r.done, cudaEventDisableTiming), "cudaEventCreate");
    const int64_t rid = s->next_id++;
    s->reqs.emplace(rid, std::move(r));
    s->pending.push_back(rid);
    *id = rid;
    return pump(s);
}

int eph_serve_poll(eph_serve *s, int64_t id, int *state) {
    if (!s || !state) return EPH_ERR_ARG;
    std::lock_guard<std::mutex> lock(s->mu);
    SCK(cudaSetDevice(s->device), "cudaSetDevice");
    int rc = pump(s);
    if (rc) return rc;
    auto it = s->reqs.find(id);
    if (it == s->reqs.end()) return sfail(s, EPH_ERR_ARG, "unknown request");
    if (!it->second.launched) { *state = 0; return EPH_OK; }
    const cudaError_t e = cudaEventQuery(it->second.done);
    if (e == cudaSuccess) *state = 2;
    else if (e == cudaErrorNotReady) *state = 1;
    else return sfail(s, EPH_ERR_CUDA, "request", e);
    return EPH_OK;
}

int eph_serve_result(eph_serve *s, int64_t id, double *part_state, int64_t *n_accepted, int64_t *n_rejected,
                     double *step_log, int64_t *n_logged) {
    if (!s) return EPH_ERR_ARG;
    std::lock_guard<std::mutex> lock(s->mu);
    SCK(cudaSetDevice(s->device), "cudaSetDevice");
    auto it = s->reqs.find(id);
    if (it == s->reqs.end()) return sfail(s, EPH_ERR_ARG, "unknown request");
    if (!it->second.launched)   // collect finished requests first: their memory admits the queue
        return sfail(s, EPH_ERR_STATE, "request is still queued for device memory");
    eph_serve::Req &r = it->second;
    SCK(cudaEventSynchronize(r.done), "request");
    cudaStream_t st = s->streams[r.stream];
    std::vector<long long> stats((size_t)r.grid * 2);
    std::vector<int> status(r.grid);
    SCK(cudaMemcpyAsync(stats.data(), r.d_stats, stats.size() * sizeof(long long), cudaMemcpyDeviceToHost, st), "stats");
    SCK(cudaMemcpyAsync(status.data(), r.d_status, status.size() * sizeof(int), cudaMemcpyDeviceToHost, st), "status");
    if (part_state)
        SCK(cudaMemcpyAsync(part_state, r.d_state, (size_t)12 * r.P * sizeof(double), cudaMemcpyDeviceToHost, st), "results");
    std::vector<double> hl;
    if (r.d_hlog) {
        hl.resize(r.log_cap);
        SCK(cudaMemcpyAsync(hl.data(), r.d_hlog, hl.size() * sizeof(double), cudaMemcpyDeviceToHost, st), "step log");
    }
    SCK(cudaStreamSynchronize(st), "results");
    long long acc = 0, rej = 0;   // particle-steps: each block's step counts times its particles
    int bad = 0;
    const int S = r.block / r.G;
    for (int g = 0; g < r.grid; ++g) {
        const long long live = std::min<long long>(S, (long long)r.P - (long long)g * S);
        acc += stats[2 * g] * live;
        rej += stats[2 * g + 1] * live;
        bad = bad ? bad : status[g];
    }
    if (n_accepted) *n_accepted = acc;
    if (n_rejected) *n_rejected = rej;
    if (step_log && n_logged) {
        const int64_t k = std::min<int64_t>(stats[0], r.log_cap);   // block 0's accepted steps
        std::copy(hl.begin(), hl.begin() + k, step_log);
        *n_logged = k;
    }
    req_free(r, st);
    cudaEventDestroy(r.done);
    s->in_use -= std::min(s->in_use, r.bytes);
    s->reqs.erase(it);
    const int rc = pump(s);
    if (bad)
        return sfail(s, EPH_ERR_STEP, bad == SS_STEP_UNDERFLOW ? "adaptive step fell below the minimum"
                                      : bad == SS_ATTEMPTS ? "too many step attempts" : "request exceeded its device-time limit");
    return rc;
}

int eph_serve_eval(eph_serve *s, double t, double *out) {
    if (!s || !out) return EPH_ERR_ARG;
    std::lock_guard<std::mutex> lock(s->mu);
    if (!(t >= s->t0 && t <= s->t0 + (double)s->n * s->knot)) return sfail(s, EPH_ERR_ARG, "time outside the ephemeris");
    SCK(cudaSetDevice(s->device), "cudaSetDevice");
    cudaStream_t st = s->streams[0];
    double *d_out = nullptr;
    SCK(cudaMallocAsync((void **)&d_out, (size_t)s->M * kChan * sizeof(double), st), "cudaMallocAsync(eval)");
    ServeArgs A{};
    A.coef = s->d_coef; A.gm = s->d_gm; A.sr2 = s->d_sr2; A.cheb = s->d_cheb;
    A.M = s->M; A.d = s->d; A.n = s->n; A.t0 = s->t0; A.knot = s->knot;
    cudaError_t e = launch_kernel(eval_kernel, 1, kSThreads, (size_t)kSRec * s->M * sizeof(double), st, A, t, d_out);
    if (e == cudaSuccess) e = cudaMemcpyAsync(out, d_out, (size_t)s->M * kChan * sizeof(double), cudaMemcpyDeviceToHost, st);
    cudaFreeAsync(d_out, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return sfail(s, EPH_ERR_CUDA, "ephemeris evaluation", e);
    return EPH_OK;
}

int eph_serve_request_shape(eph_serve *s, int64_t id, int *lanes, int *particles_per_block, int *blocks) {
    if (!s || !lanes || !particles_per_block || !blocks) return EPH_ERR_ARG;
    std::lock_guard<std::mutex> lock(s->mu);
    auto it = s->reqs.find(id);
    if (it == s->reqs.end()) return sfail(s, EPH_ERR_ARG, "unknown request");
    *lanes = it->second.G;
    *particles_per_block = it->second.block / it->second.G;
    *blocks = it->second.grid;
    return EPH_OK;
}

int eph_serve_info(const eph_serve *s, int64_t *launches, int64_t *queued, int64_t *bytes_in_use) {
    if (!s || !launches || !queued || !bytes_in_use) return EPH_ERR_ARG;
    *launches = s->launches;
    *queued = (int64_t)s->pending.size();
    *bytes_in_use = (int64_t)s->in_use;
    return EPH_OK;
}

int eph_bspline_fit_batch(int device, int d, int64_t n, int64_t mn, int channels, int64_t n_series,
                          const double *samples, double *coefs) {
    if (channels < 1 || n_series < 1 || !samples || !coefs) return EPH_ERR_ARG;
    eph::BsplineFactor f;
    if (eph::bspline_factor(d, n, mn, f)) return EPH_ERR_ARG;
    if (cudaSetDevice(device) != cudaSuccess) return EPH_ERR_ARG;
    const long long m = f.m, T = n_series * channels;
    auto pack = [](const std::vector<double> &h, const std::vector<double> &l) {
        std::vector<double> o(2 * h.size());
        for (size_t i = 0; i < h.size(); ++i) { o[2 * i] = h[i]; o[2 * i + 1] = l[i]; }
        return o;
    };
    const std::vector<double> rw = pack(f.rw_hi, f.rw_lo), lu = pack(f.lu_hi, f.lu_lo), rd = pack(f.rd_hi, f.rd_lo);
    const size_t n_smp = (size_t)n_series * (mn + 1) * channels, n_coef = (size_t)n_series * m * channels;
    // One allocation, and one copy for the matrix's tables: the allocations and frees of nine arrays took longer than
    // the kernel (419 bodies, 365 knots: 5.9 -> 4.0 ms with everything, at the same sizes of the copies).
    std::vector<char> tab;
    auto put = [&](const void *p, size_t bytes) {   // the table's offset, 256-byte aligned
        const size_t at = (tab.size() + 255) / 256 * 256;
        tab.resize(at + bytes);
        memcpy(tab.data() + at, p, bytes);
        return at;
    };
    const std::vector<long long> jm(f.jmin.begin(), f.jmin.end());
    const size_t o_bval = put(f.bval.data(), f.bval.size() * sizeof(double)), o_rw = put(rw.data(), rw.size() * sizeof(double)),
                 o_lu = put(lu.data(), lu.size() * sizeof(double)), o_rd = put(rd.data(), rd.size() * sizeof(double)),
                 o_jmin = put(jm.data(), jm.size() * sizeof(long long)), o_cnt = put(f.cnt.data(), f.cnt.size() * sizeof(int));
    auto round = [](size_t bytes) { return (bytes + 255) / 256 * 256; };
    const size_t o_smp = round(tab.size()), o_coef = o_smp + round(n_smp * sizeof(double)), o_y = o_coef + round(n_coef * sizeof(double));
    char *base = nullptr;
    int rc = EPH_OK;
    cudaError_t e = cudaMalloc((void **)&base, o_y + (size_t)2 * m * T * sizeof(double));
    if (e != cudaSuccess) return e == cudaErrorMemoryAllocation ? EPH_ERR_OOM : EPH_ERR_CUDA;
    double *d_smp = (double *)(base + o_smp), *d_coef = (double *)(base + o_coef), *d_y = (double *)(base + o_y);
    const double *d_bval = (double *)(base + o_bval), *d_rw = (double *)(base + o_rw), *d_lu = (double *)(base + o_lu),
                 *d_rd = (double *)(base + o_rd);
    const long long *d_jmin = (long long *)(base + o_jmin);
    const int *d_cnt = (int *)(base + o_cnt);
    if (cudaMemcpy(base, tab.data(), tab.size(), cudaMemcpyHostToDevice) != cudaSuccess ||
        cudaMemcpy(d_smp, samples, n_smp * sizeof(double), cudaMemcpyHostToDevice) != cudaSuccess)
        rc = EPH_ERR_CUDA;
    if (!rc) {
        const int threads = 128;
        e = launch_kernel(bspline_solve_kernel, (unsigned)((T + threads - 1) / threads), threads, 0, nullptr, d, m, f.J, channels,
                          n_series, (long long)(mn + 1) * channels, d_smp, d_jmin, d_cnt, d_bval, d_rw, d_lu, d_rd, d_y, d_coef);
        if (e != cudaSuccess ||
            (e = cudaMemcpy(coefs, d_coef, n_coef * sizeof(double), cudaMemcpyDeviceToHost)) != cudaSuccess)
            rc = EPH_ERR_CUDA;
    }
    cudaFree(base);
    return rc;
}

// Ephemeris samples from a context: integrates n_step steps of dt from t_eph (advanced), and writes the
// state at the start and after every `stride` steps: out[(n_step / stride) + 1][n][EPH_EPHEM_CHANNELS]
// (position, velocity, Newtonian acceleration / c^2, potential / c^2 of every body, caller order).
int eph_record_samples(eph_ctx *ctx, double dt, int64_t n_step, int64_t stride, double *t_eph_hi, double *t_eph_lo,
                       double *out) {
    if (!ctx || n_step < 0 || stride < 1 || n_step % stride != 0 || !t_eph_hi || !t_eph_lo || !out) return EPH_ERR_ARG;
    const int64_t n = ctx_size(ctx);
    if (n < 1) return EPH_ERR_STATE;
    int rc = EPH_OK;
    const size_t rec_step = (size_t)kStages * n * kTrajRec * sizeof(double);
    const int64_t chunk = std::max<int64_t>(stride, std::min<int64_t>(n_step, (int64_t)((512ull << 20) / rec_step) / stride * stride));
    double *d_traj = nullptr, *d_out = nullptr;
    const int64_t per_chunk = chunk / stride;
    if (cudaMalloc(&d_traj, (size_t)(1 + kStages * std::max<int64_t>(chunk, 1)) * n * kTrajRec * sizeof(double)) != cudaSuccess)
        return EPH_ERR_OOM;
    if (cudaMalloc(&d_out, (size_t)std::max<int64_t>(per_chunk, 1) * n * kChan * sizeof(double)) != cudaSuccess) {
        cudaFree(d_traj);
        return EPH_ERR_OOM;
    }
    // the start: from the planes (their auxiliaries are the loader's accel of this state)
    {
        std::vector<double> pl((size_t)EPH_NPLANES * n);
        rc = eph_download_system(ctx, pl.data());
        if (rc) { cudaFree(d_traj); cudaFree(d_out); return rc; }
        const double c2 = kCS * kCS;
        for (int64_t j = 0; j < n; ++j) {
            auto P = [&](int q) { return pl[(size_t)q * n + j]; };
            double *o = out + (size_t)j * kChan;
            for (int c = 0; c < 3; ++c) {
                o[c] = P(EPH_P_R_HI + c) + P(EPH_P_R_LO + c);
                o[3 + c] = P(EPH_P_V_HI + c) + P(EPH_P_V_LO + c);
                o[6 + c] = P(EPH_P_NACCEL + c) / c2;
            }
            o[9] = P(EPH_P_PHI) / c2;
        }
    }
    int64_t written = 1;
    for (int64_t done = 0; done < n_step && rc == 0;) {
        const int64_t c = std::min<int64_t>(chunk, n_step - done);
        ctx_record_stages(ctx, d_traj, 1);
        rc = eph_rk12(ctx, dt, c, *t_eph_hi, *t_eph_lo);
        ctx_record_stages(ctx, nullptr, 0);
        if (rc) break;
        const int take = (int)(c / stride);
        cudaError_t e = launch_kernel(gather_samples, 256, 256, 0, nullptr, d_traj, (int)n, take, stride - 1, (int)stride, d_out);
        if (e == cudaSuccess) e = cudaMemcpy(out + (size_t)written * n * kChan, d_out, (size_t)take * n * kChan * sizeof(double),
                                             cudaMemcpyDeviceToHost);
        if (e != cudaSuccess) { rc = EPH_ERR_CUDA; break; }
        written += take;
        // t_eph += dt * c in double-double (mass.cpp:441)
        const double a = *t_eph_hi, b = dt * (double)c, s = a + b, tt = s - a;
        double er = (a - (s - tt)) + (b - tt);
        er = er + (*t_eph_lo + 0.0);
        const double hsum = s + er;
        *t_eph_lo = er - (hsum - s);
        *t_eph_hi = hsum;
        done += c;
    }
    cudaFree(d_traj);
    cudaFree(d_out);
    return rc;
}

}  // extern "C"
