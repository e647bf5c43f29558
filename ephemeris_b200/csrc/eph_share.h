// eph_share.h - shared memory of the ensemble and point-mass kernels (eph_batch.cu), and how many CTAs share a system:
// plain arithmetic on sizes, without CUDA calls. Nothing here changes a result: a body's sums are cut into the same
// parts (batch_split) and added in the same order whatever the number of CTAs.
#pragma once
#include <algorithm>
#include <cstddef>

#include "eph_system.cuh"
#include "../../include/eph_rk12_table.h"

#ifdef __CUDACC__
#define EPH_HD __host__ __device__
#else
#define EPH_HD
#endif

namespace eph {

constexpr int kBThreads = 256;          // threads per ensemble CTA
constexpr int kCoopMin = 32;            // default: bodies from which a system may be shared by a cluster
constexpr int kStore = 3 * kStages + 12;   // stored values per body: f_j of every stage, r0 and v0 (hi, lo)
constexpr int kMaxSplit = 32;           // most parts a body's j range is cut into
constexpr int kMaxBodies = 768;         // bodies of a system of the ensemble launch (16 CTAs hold any such)

// What a pair term reads of a body lies in records of 64 bytes, 80 apart, so that a thread fetches a body j with four
// 16-byte shared-memory loads; the lanes of a warp work on different bodies i and the same j, which makes every
// one of them a broadcast.
enum RecA { RA_R_HI = 0, RA_R_LO = 3, RA_GM = 6, RA_SR2 = 7, kRecA = 10 };          // state of the stage
enum RecB { RB_NACC = 0, RB_BETA = 3, RB_K = 6, RB_PHI = 7, kRecB = 10 };           // pass-A outputs; K = phi + 2 beta^2
// The mixed-precision form reads single-precision copies instead of RecB.
enum RecF { RF_NACC = 0, RF_GM = 3, RF_BETA = 4, RF_PHI = 7, RF_BETA2 = 8, kRecF = 12 };
enum OwnRow { OR_V_HI = 0, OR_V_LO = 3, OR_M = 6, OR_MAXI = 7, OR_GM0 = 8, OR_DGM = 9, kOwnRows = 10 };
constexpr int kPartA = 4, kPartB = 6;   // values of a unit's sums: {phi, a_N}; {gaccel, m_min, tq, j of tq}

// Shared memory (doubles) of each CTA when `peers` share a system of n bodies: room for the largest share. The
// stage store is in it while two CTAs still fit an SM; larger shares keep it in global memory (L2).
constexpr int kRkTableBytes = (EPH_RK12_NCOEF * 3 * (int)sizeof(double) + 15) / 16 * 16;   // the kernels' static table
constexpr int kPairSmem = (113 * 1024 - kRkTableBytes - 128) / 8;
constexpr size_t kBMaxSmem = 227 * 1024 - kRkTableBytes - 256;            // most dynamic shared memory of a CTA (bytes)
EPH_HD inline int batch_smem_doubles(int n, int peers, int split, bool mixed, bool *store_in_smem) {
    const int most = (n + peers - 1) / peers;
    const int base = n * ((peers > 1 ? 2 : 1) * kRecA + (mixed ? kRecF / 2 : kRecB)) +
                     most * (split * kPartB + kOwnRows + (mixed ? kRecB : 0));
    *store_in_smem = base + most * kStore <= kPairSmem;
    return *store_in_smem ? base + most * kStore : base;
}
inline size_t system_smem(int n, int peers, int split, bool mixed) {
    bool in_smem;
    return batch_smem_doubles(n, peers, split, mixed, &in_smem) * sizeof(double);
}

// ---- how many CTAs share a system
constexpr int kShares = 5;
constexpr int kSharePeers[kShares] = {16, 8, 4, 2, 1};
constexpr unsigned kAllShares = (1u << kShares) - 1;   // a set of CTA counts: bit g stands for kSharePeers[g]
constexpr int kMinOwn = 12;        // bodies per CTA below which sharing a system further does not pay
constexpr int kMaxPerThread = 4;   // units per thread, by the shared memory of their sums

// Time of one stage (us) of a system of n bodies on `peers` CTAs, its j ranges cut into `split` parts: a model
// of measurements on one B200 (single systems of 8-400 bodies on 1-16 CTAs): 2.6 us for the state update and the
// phases per body, 1.3 us for the two cluster exchanges, and per unit of a thread 0.36 us a pair (both passes;
// FP64 latency at 8 warps) and 0.3 us.
inline float stage_us(int n, int peers, int split) {
    const int per_thread = ((n + peers - 1) / peers * split + kBThreads - 1) / kBThreads;
    return 2.6f + (peers > 1 ? 1.3f : 0.0f) + (float)per_thread * (0.36f * (float)((n + split - 1) / split) + 0.3f);
}
inline bool units_fit(int n, int peers, int split) { return (n + peers - 1) / peers * split <= kMaxPerThread * kBThreads; }
inline bool share_fits(int n, int peers, int split, bool mixed) {
    return units_fit(n, peers, split) && system_smem(n, peers, split, mixed) <= kBMaxSmem;
}
// Parts that each body's j range is cut into: the number that keeps the threads busiest over the CTA counts the
// system may be shared by and on which its units fit. It depends on n alone, so that a system's sums are the same however
// it is shared. Where many parts win, the units do not fit one CTA: 85, 96, 101 to 140 and more than 144 bodies take
// two or more CTAs in any batch. On one CTA by memory alone they are slower: 96 bodies in a full batch 5.1 ms against
// 4.0 on two, 128 5.7 against 4.4, 200 9.0 against 6.4.
inline int batch_split(int n) {
    int best = 1;
    float best_cost = 1e30f;
    for (int g = 1; g <= kMaxSplit && g <= n; ++g) {
        float cost = 0;
        for (int peers : kSharePeers) {
            const int cnt = (n + peers - 1) / peers;
            if ((peers > 1 && n < kMinOwn * peers) || cnt * g > kMaxPerThread * kBThreads) continue;
            cost += stage_us(n, peers, g) / stage_us(n, peers, std::max(1, std::min(n, kBThreads / cnt)));
        }
        int counted = 0;
        for (int peers : kSharePeers)
            counted += !((peers > 1 && n < kMinOwn * peers) || (n + peers - 1) / peers * g > kMaxPerThread * kBThreads);
        if (counted && cost / counted < best_cost) { best_cost = cost / counted; best = g; }
    }
    return best;
}

// The choices below take the CTA counts that the device can hold as clusters (`shares`), and return an index of
// kSharePeers, or -1 where none of them holds the system.
// The fewest CTAs, the form with the least work in all; on a device of small clusters by memory alone.
inline int fewest_ctas(int n, int split, bool mixed, unsigned shares) {
    for (int g = kShares - 1; g >= 0; --g)
        if ((shares >> g & 1) && share_fits(n, kSharePeers[g], split, mixed)) return g;
    for (int g = kShares - 1; g >= 0; --g)
        if ((shares >> g & 1) && system_smem(n, kSharePeers[g], split, mixed) <= kBMaxSmem) return g;
    return -1;
}
// The next larger number than kSharePeers[g] that may share the system.
inline int more_ctas(int n, int split, bool mixed, unsigned shares, int g) {
    for (--g; g >= 0; --g)
        if ((shares >> g & 1) && n >= kMinOwn * kSharePeers[g] && share_fits(n, kSharePeers[g], split, mixed)) return g;
    return -1;
}
// The number with the shortest stage.
inline int shortest_stage(int n, int split, bool mixed, unsigned shares) {
    int best = fewest_ctas(n, split, mixed, shares);
    for (int g = best; g >= 0; g = more_ctas(n, split, mixed, shares, g))
        if (stage_us(n, kSharePeers[g], split) <= stage_us(n, kSharePeers[best], split)) best = g;
    return best;
}

}  // namespace eph
