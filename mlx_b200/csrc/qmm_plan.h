// Schedule and tile height of the prefill GEMM (qmm_tc.cu), as plain host arithmetic.
#pragma once
#include <algorithm>
#include <cmath>
#include <cstddef>

namespace luxcuda {

constexpr int kBK = 64;            // weights (k) per sub-block = one 128-byte swizzle row of bf16
constexpr int kSub = 2;            // sub-blocks per pipeline stage (one barrier round per 128 k)
constexpr int kTileN = 128;        // rows of W per tile (MMA M)
constexpr int kMaxBM = 256;        // rows of x per tile (MMA N)
constexpr int kStagesB = 3;        // k-stages in flight: B in shared memory, A in TMEM, one barrier pair per stage
constexpr int kStagesP = 3;        // the same in the pair kernel.  (Four, with the 64 KB more of shared memory they take
                                   // from L1, measured the same or slower.)
constexpr int kDqGroups = 3;       // groups of dequantising warps
constexpr int kEpiWarps = 8;
constexpr int kWUnitBytes = kTileN * 64;     // one unit of packed weights: 128 rows x 64 bytes (128 k at 4 bit, 64 k at 8 bit)
constexpr int kMaxWSlots = 4;      // weight units in flight per dequantising group, at most
constexpr int kEpiStageBytes = 16 * 32 * 2;  // per epilogue warp: 16 rows of y x 32 columns, bf16
constexpr int kGemmCtlBytes = 384;  // barriers and the like at the end of a CTA's shared memory
constexpr int kGemmSmemLimit = 227 * 1024;
// a finished tile of y as bf16 (the epilogue writes whole blocks of 32 rows of x)
constexpr int pair_y_bytes(int bm) { return ((bm + 31) & ~31) * kTileN * 2; }

// What the choice depends on.  ld, col0: row stride and first column of y in elements (N and 0 unless column-sharded).
struct GemmShape {
    int M, K, N, bits, group;
    bool y_bf16, sharded;
    int ld, col0;
};
struct GemmForce {  // overrides: 0, 1, or -1 for the plan's own choice
    int streamk = -1;  // stream-K or whole tiles
    int pair = -1;     // whole tiles: by pairs of CTAs or by single ones
};
struct GemmPlan {
    int bm, m_tiles, n_tiles, streamk, pair, w_slots;
    int y_tma;  // pair kernel: how y leaves (see GemmParams)
    size_t smem;
};

// False: no schedule for this shape.
//
// Tile height: the matrix instruction's N.  One CTA's (M = 128) takes multiples of 16.  The pair's (M = 256, A in tensor
// memory) is documented for multiples of 32 only, so a pair's tiles are that high whatever is left of M.
//
// Schedule and height go by a rough estimate of the time in microseconds, not a fit: on 392 shapes (32 to 2048 rows, K 512 to
// 8192, N 256 to 11008) it takes the fastest of the three kernels or one within 4 % of it on 377, within 20 % at worst, but
// the times themselves are off by up to a third for low tiles (48 rows: 0.64 us a stage measured, 0.50 here).  A k-stage of a tile costs about 0.45 + 0.001 * bm whatever the kernel (dequantisation, then the
// MMAs), so a lower tile pays where it saves no round of tiles: 777 x 2880 x 5003 took 35.6 us in 208-row tiles and
// 30.8 in 112-row ones, two rounds either way.
//   whole tiles: ceil(T/G) rounds, each with an epilogue of 3 * bm/256 that nothing else overlaps;
//   CTA pairs:   rounds of pair tiles; the epilogue overlaps where y leaves by TMA; 3 to set up;
//   stream-K:    T*nst/G stages of up to 1.6 times the cost, an epilogue more, and the exchange of partials.
inline bool choose_gemm_plan(const GemmShape& a, int sm_count, const GemmForce& force, bool no_ytma, GemmPlan* pl) {
    pl->n_tiles = (a.N + kTileN - 1) / kTileN;
    const double G = sm_count, nst = (a.K / kBK + kSub - 1) / kSub;
    const bool y_fast = a.y_bf16 && ((a.ld | a.col0) & 7) == 0;
    const int m0 = (a.M + kMaxBM - 1) / kMaxBM;
    double best = 0.0;
    bool found = false;
    for (int mt = m0; mt <= std::min(2 * m0, m0 + 8); mt++) {  // (with many tile rows a round is a small part of the whole)
        for (int k = 0; k < 3; k++) {  // 0: whole tiles, 1: pairs, 2: stream-K
            if (force.streamk >= 0 && force.streamk != (k == 2)) continue;
            if (force.pair >= 0 && k < 2 && force.pair != k) continue;
            const int step = k == 1 ? 32 : 16, bm = ((a.M + mt - 1) / mt + step - 1) / step * step;
            if ((a.M + bm - 1) / bm != mt) continue;  // (a tile row without rows)
            const double h = bm / 256.0, stage = 0.45 + 0.001 * bm, e = 3.0 * h, T = (double)pl->n_tiles * mt, rounds = std::ceil(T / G);
            double cost;
            if (k == 0) {
                cost = rounds * (nst * stage + e);
            } else if (k == 1) {
                if (sm_count & 1) continue;
                const double prounds = std::ceil((pl->n_tiles + 1) / 2 * (double)mt / (sm_count / 2));
                cost = 3.0 + prounds * (nst * stage + (y_fast ? 0.5 : e));
            } else {
                if (T * nst < G && !(force.streamk == 1 && mt == m0)) continue;
                cost = 2.0 + (1.1 + 0.5 * h) * T * nst / G * stage + (rounds + 1.0) * e + 4.0 * h * (T < G ? std::ceil(G / T) : 1.0);
            }
            if (found && cost >= best) continue;
            found = true;
            best = cost;
            pl->m_tiles = mt; pl->bm = bm; pl->pair = k == 1; pl->streamk = k == 2;
        }
    }
    if (!found) return false;
    // Shared memory: the ring of x, as tall as the tile, and the rings of weights, a stage of each group's if there is room
    // (one unit at 4 bit, two at 8 bit; more only take from L1, which holds the rows' scales: 3-5 % slower).
    pl->y_tma = 0;
    size_t fixed = 1024 + kGemmCtlBytes;
    if (pl->pair) {
        if (a.y_bf16 && !no_ytma && y_fast) pl->y_tma = a.sharded ? 2 : 1;
        fixed += (size_t)kStagesP * kSub * (pl->bm / 2) * 128 + (pl->y_tma ? pair_y_bytes(pl->bm) : 0);
    } else {
        fixed += (size_t)kStagesB * kSub * pl->bm * 128 + (size_t)kEpiWarps * kEpiStageBytes;
    }
    pl->w_slots = (int)std::min<size_t>(a.bits == 8 ? 2 : 1, (kGemmSmemLimit - fixed) / (kDqGroups * kWUnitBytes));
    pl->smem = fixed + (size_t)kDqGroups * pl->w_slots * kWUnitBytes;
    return true;
}

}  // namespace luxcuda
