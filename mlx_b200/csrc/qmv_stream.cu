// Decode-regime quantized matmul for bf16 activations, one launch for one matmul or for several of one shape, 16 rows of x at
// a time:
//   y[M,N] = x[M,K] . dequant(Wq[N,K])^T,  w^ = RNE_bf16(s*q + b)  (one bf16 FMA)
//
// HBM-bound: every packed word, scale and bias is read once; algorithmic bytes per output row: K*bits/8 + 4*K/group.
// What an SM has to issue for that comes close behind: a task (16 rows x 128 bytes) is 64 bf16x2 FMAs, 80 mask/shift
// operations and 16 MMAs of a warp at 4 bit, 300 cycles per scheduler by themselves, and the memory brings one per 390.
// So the warps that dequantise do as little else as possible:
//   * warp 16 brings the packed weights into a ring of stages in shared memory, one TMA load per tile of 16 rows x (at
//     most) 16 k-blocks: 32 KB in one instruction.  (One bulk copy per row: the copy engine takes 64 ns for each,
//     whatever its size, and 48 small ones per tile made the launch three times as long.)  The boxes are laid out
//     [k-block][row][128 bytes] under the 128-byte swizzle: the lanes' 16-byte reads are conflict-free.
//     It also brings the scales and biases of the same rows (cp.async, 16-byte pieces into padded rows).  The working
//     warps reading them from global memory, a group ahead, cost 1 us of a 25 MB layer's 6.
//   * warps 0-15: warp w owns k-block w of a stage (ts row tiles of kbc k-blocks each when K is short) and keeps the x
//     fragments of that k-block in registers for all tiles of the CTA; it reads its 16 x 128 bytes, dequantises,
//     multiplies (qmv_frag.cuh) and leaves a 16 x 8*MT fp32 partial where its weights lay.
//   * warps 17-19 take the tiles in turn, add a tile's partials in k-block order, store y and give the stage back.  (One
//     warp, which shares its scheduler with four busy ones, takes 1.3 us per tile: it alone held the launch up.)
//     There is no block barrier: the warps run from tile to tile, from matmul to matmul.
// x goes through 4 KB of shared memory per warp: read along its rows (8 lines per instruction), written in fragment
// order, read back as fragments.  (Reading the fragments from global memory takes 32 lines per instruction: 2.2 us per
// matmul with 8 rows.)
// K longer than 16 k-blocks is cut into chunks: all tiles of the CTA for the first chunk, then for the next; the sums of
// the tiles are carried along in shared memory and x is reloaded per chunk.
//
// K need not be a multiple of the k-block: x reads as zero past K, and the last box of a row is cut off there.
//
// More than 16 rows of x (the prefill kernel takes them where K is a multiple of 64) are items of 16 rows on the same
// weights, dealt over the grid's y as far as few row tiles leave SMs over.  (A launch for every 16 rows: 4096 x 96 x 16 took
// 544 us; the CUDA-core kernel 12; this way 6.)
#include <algorithm>
#include <atomic>

#include "internal.h"
#include "qmv_frag.cuh"

namespace luxcuda {

namespace {

constexpr int kWarps = 16;  // working warps
constexpr int kLoadWarp = kWarps, kSumWarp = kWarps + 1, kSumWarps = 3;
constexpr int kThreads = (kWarps + 1 + kSumWarps) * 32;
constexpr int kMaxStages = 6;
constexpr int kMaxBatch = 48;  // matmuls per launch
constexpr int kSmemLimit = 227 * 1024 - 1024;  // dynamic; the rest is for the static part
// Registers: 640 threads x 96 at launch; the working warps take what the helper warps do not need.  With 112 and 32 the
// helpers spilled at 4 bit with groups of 32 or 16 rows (88-104 bytes), which cost more than the working warps gained:
// 8 x 4096 x 5003, groups of 32: 7.13 us against 5.51, groups of 64: the same; 16 x 2880 x 5003: 7.10 against 5.67.
constexpr int kLaunchRegs = 96, kWorkRegs = 104, kHelperRegs = 56;
static_assert(kWarps * 32 * kWorkRegs + (kThreads - kWarps * 32) * kHelperRegs <= kThreads * kLaunchRegs, "register split");
// A stage: [tile][k-block][16 rows][128 bytes] of weights, then per tile the scales and biases, [rows 0-7: scales][rows 0-7:
// biases][rows 8-15: scales][rows 8-15: biases], a row's being the 16-byte pieces that hold those of the chunk.  Rows of
// sb_row bytes: 16 k-blocks' worth and up to 14 bytes of what lies before; an odd multiple of 16 bytes, for the banks.  (K cut
// off inside a k-block leaves room for the zeros behind the last group: a group of a k-block is missing, or at SPL = 2 all 272
// bytes are used.)
constexpr int sb_row(int spl) { return spl == 2 ? 16 * 16 + 16 : 16 * 8 + 16; }

__device__ __forceinline__ uint32_t s32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void bar_init(uint32_t b, uint32_t n) { asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(b), "r"(n)); }
__device__ __forceinline__ void bar_arrive(uint32_t b) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(b) : "memory"); }
__device__ __forceinline__ void bar_expect(uint32_t b, uint32_t n) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(b), "r"(n) : "memory");
}
// (the hint lets the hardware hold a waiting warp instead of having it poll: polls take issue slots from working warps)
__device__ __forceinline__ bool bar_try(uint32_t b, uint32_t parity) {
    uint32_t ok;
    asm volatile("{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3; selp.u32 %0, 1, 0, p; }"
                 : "=r"(ok) : "r"(b), "r"(parity), "r"(20000u) : "memory");
    return ok != 0;
}
// Bounded wait (about two seconds of SM clock).  False: it ran out, or another role has given up; *abort is set.
// SLEEP: of the helper warps, which are never in a hurry.
template <bool SLEEP>
__device__ __forceinline__ bool bar_wait(uint32_t b, uint32_t parity, volatile int* abort) {
    if (bar_try(b, parity)) return true;
    const uint32_t t0 = clock();
    for (;;) {
#pragma unroll 1
        for (int i = 0; i < 64; i++) {
            if (SLEEP) __nanosleep(32);
            if (bar_try(b, parity)) return true;
        }
        if (*abort || (uint32_t)clock() - t0 > 4000000000u) break;
    }
    *abort = 1;
    return false;
}
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                 ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(bar) : "memory");
}
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, int x, int y, int z, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
                 ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(z), "r"(bar) : "memory");
}
// 16 bytes, of which the first n are read and the rest are zeros
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, uint32_t n) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
}
// one arrival on the barrier once this thread's copies so far have landed
__device__ __forceinline__ void cp_async_arrive(uint32_t bar) { asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar) : "memory"); }
__device__ __forceinline__ uint32_t lds_u16(uint32_t a) {
    uint32_t v;
    asm volatile("ld.shared.u16 %0, [%1];" : "=r"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ void sts_v4(uint32_t a, const uint4& v) {
    asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(a), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
__device__ __forceinline__ uint4 lds_v4(uint32_t a) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a) : "memory");
    return v;
}
// s += v, four fp32 sums in two instructions
__device__ __forceinline__ void add_f32x4(uint4& s, const uint4& v) {
    asm("{ .reg .b64 a, b, c, d; mov.b64 a, {%0, %1}; mov.b64 b, {%2, %3}; mov.b64 c, {%4, %5}; mov.b64 d, {%6, %7};\n"
        "  add.rn.f32x2 a, a, c; add.rn.f32x2 b, b, d; mov.b64 {%0, %1}, a; mov.b64 {%2, %3}, b; }"
        : "+r"(s.x), "+r"(s.y), "+r"(s.z), "+r"(s.w) : "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w));
}
constexpr int kItemRows = 16;  // rows of x of an item, at most (more of one matmul: several items, see Params)
struct Item {
    const __nv_bfloat16* x;
    const __nv_bfloat16* scales;
    const __nv_bfloat16* biases;
    void* y;
    int M;
};
// NI: how many matmuls of a batch, at most; 1: one; 0: one whose rows of x are n_items items of 16 (M: all of them).
template <int NI>
struct Params {
    static constexpr bool kRows = NI == 0;
    static constexpr int kArray = kRows ? 1 : NI;
    alignas(64) CUtensorMap maps[kArray];  // the packed weights
    Item items[kArray];
    int n_items, K, N, gshift, y_bf16;
    __device__ __forceinline__ const Item& item(int i) const { return items[kRows ? 0 : i]; }
    int rt_q, rt_rem;       // row tiles per CTA, and how many CTAs have one more
    int ts_inv, kbc_inv;    // 65536 / ts, 65536 / kbc, rounded up
    int nkb, nch, kbc, ts, tb;  // k-blocks; chunks of K and k-blocks per chunk (at most); row tiles per stage, and per pass over K
    int k_tail;             // K is no multiple of the k-block: the last one is cut off at K
    int stages, sum_warps, stage_bytes, tile_bytes, sb_off;  // bytes of weights per tile; offset of the scales in a stage
    int xs_off, run_off, bar_off;                 // offsets in shared memory
    int x_early, x_ld;      // see launch_decode
    int x32;                // every row of every x starts on a 32-byte boundary (callers owe 16 bytes only)
    float eps;              // of the rms-norm prologue
    int* error;             // host-visible error word of the bounded waits
};

// The CTA's work, walked in the same order by every role: items, every gridDim.y-th; passes of at most tb row tiles; chunks
// of K; groups of ts tiles (one stage each).  The row tiles are dealt out in gridDim.x ranges of rt_q or rt_q + 1 tiles; the CTA takes
// range (blockIdx.x + i) mod gridDim.x of its i-th item, which evens out the one tile by which they differ.  (No divisions: they
// would be a microsecond in front of the first weight.)
struct Walk {
    int item, lo, hi, b0, c, ng;  // range [lo, hi), pass at b0, chunk, groups of this pass
    int rc;
    template <class P>
    __device__ __forceinline__ void range(const P& p) {
        lo = rc * p.rt_q + min(rc, p.rt_rem);
        hi = lo + p.rt_q + (rc < p.rt_rem ? 1 : 0);
        b0 = lo;
        groups(p);
    }
    template <class P>
    __device__ __forceinline__ void groups(const P& p) {
        ng = (int)((uint32_t)((min(p.tb, hi - b0) + p.ts - 1) * p.ts_inv) >> 16);
    }
    template <class P>
    __device__ __forceinline__ void init(const P& p) {
        item = P::kRows ? blockIdx.y : 0;
        c = 0;
        rc = blockIdx.x;
        range(p);
    }
    template <class P>
    __device__ __forceinline__ bool next_run(const P& p) {  // on to the next run of groups; false: the end
        if (++c < p.nch) return true;
        c = 0;
        b0 += p.tb;
        if (b0 < hi) {
            groups(p);
            return true;
        }
        if ((item += P::kRows ? gridDim.y : 1) >= p.n_items) return false;
        if (++rc == (int)gridDim.x) rc = 0;
        range(p);
        return true;
    }
    template <class P>
    __device__ __forceinline__ int tile_end(const P& p) const { return min(b0 + p.tb, hi); }
    template <class P>
    __device__ __forceinline__ int kb_cnt(const P& p) const { return min(p.kbc, p.nkb - c * p.kbc); }  // k-blocks of this chunk
};

// SPL: scales per lane and row of a task (2 for 4-bit weights in groups of 32).  PRO: what x is (0: as it lies; 1: the
// rms-norm of its rows, for K within one chunk; 2: the sum of three column blocks; 1 and 2 for M <= 8).
template <int BITS, int MT, int SPL, int PRO, int NI>
__global__ void __launch_bounds__(kThreads, 1) qmv_stream_kernel(const __grid_constant__ Params<NI> p) {
    static_assert(PRO == 0 || MT == 1, "prologues are built for M <= 8");
    constexpr int XV = x_frags(BITS), KB = kb_weights(BITS), KL = lane_weights(BITS), SROW = sb_row(SPL);
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ int s_abort;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    volatile int* abort = &s_abort;
    const uint32_t ring = s32(smem);
    // barriers of a stage: full (its contents have landed), sums (the working warps have left their partials), empty
    const uint32_t full = ring + p.bar_off, sums = full + 8 * kMaxStages, empty = sums + 8 * kMaxStages;
    if (tid == 0) {
        for (int i = 0; i < p.stages; i++) {
            bar_init(full + 8 * i, 1 + 32);  // the weight warp's expect_tx and the scale warp's lanes
            bar_init(sums + 8 * i, kWarps);
            bar_init(empty + 8 * i, 1);
        }
        s_abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();

    Walk wk;
    wk.init(p);
    const int role = __shfl_sync(0xffffffffu, warp, 0);  // (uniform for the compiler too: the helpers' registers are few)
    if (role >= kWarps) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kHelperRegs));
        uint32_t st = 0, ph = 0;
        bool ok = true;
        auto next_stage = [&]() {
            if (++st == (uint32_t)p.stages) { st = 0; ph ^= 1; }
        };
        if (role == kLoadWarp) {
            int issued = 0;
            // Lane (r, k) of a load: piece k of row r.  LPR pieces of a row side by side, RPI rows per load, rows r and r + 8
            // by the same distance (16*gpr bytes keep the 16-byte boundaries).
            constexpr int LPR = SPL == 2 ? 16 : 8, RPI = 32 / LPR, NB = 8 / RPI;
            // Pieces are cut off at the row's end and filled up with zeros.  Where K ends inside a k-block, the groups that the
            // lanes past K would have read their scales from are zeros, too (for those a piece of nothing else, if need be): zero
            // codes with the last group's own scale and bias would add 0 * infinity where these are infinite.
            const uint32_t gpr = (uint32_t)p.K >> p.gshift, half = 16u * gpr, k16 = 16u * (lane % LPR);
            do {
                const int t_end = wk.tile_end(p), kb0 = wk.c * p.kbc, ops = p.k_tail ? wk.kb_cnt(p) : 1;
                const CUtensorMap* map = &p.maps[p.kRows ? 0 : wk.item];
                const uint32_t g0 = (uint32_t)(wk.c * p.kbc) * KB >> p.gshift, bytes = 2u * min((uint32_t)wk.kb_cnt(p) * KB >> p.gshift, gpr - g0);
                const char *sc = reinterpret_cast<const char*>(p.item(wk.item).scales), *bi = reinterpret_cast<const char*>(p.item(wk.item).biases);
                const uint32_t need = bytes + (p.k_tail && wk.c + 1 == p.nch ? 2u * SPL : 0u);
                // where this lane's pieces of the run's first tile begin, as far as there are any, and their bytes of the row
                uint32_t lo[NB], cnt[NB], some = 0, odd = 0;
#pragma unroll
                for (int i = 0; i < NB; i++) {
                    const uint32_t at = 2u * (((uint32_t)wk.b0 * 16 + i * RPI + lane / LPR) * gpr + g0);
                    lo[i] = (at & ~15u) + k16;
                    cnt[i] = lo[i] < at + bytes ? min(16u, at + bytes - lo[i]) : 0u;
                    some |= (lo[i] < at + need ? 1u : 0u) << i;
                    odd |= (at & ~15u) + 16 * LPR < at + need ? 1u : 0u;  // a row that needs a piece more
                }
                odd = __any_sync(0xffffffffu, odd);
                for (int g = 0; g < wk.ng; g++) {
                    const int tile0 = wk.b0 + g * p.ts, tiles = min(p.ts, t_end - tile0);
                    // (the ring is full and nobody works on it before the previous kernel has ended: see the summing warps)
                    if (issued == p.stages) asm volatile("griddepcontrol.wait;" ::: "memory");
                    ok = bar_wait<true>(empty + 8 * st, ph ^ 1, abort);
                    if (!ok) break;
                    if (lane == 0) bar_expect(full + 8 * st, tiles * (p.k_tail ? ops : p.kbc) * 2048);
                    __syncwarp();
                    const uint32_t stage = ring + st * p.stage_bytes;
                    if (!p.k_tail) {
                        if (lane < tiles) tma_load_3d(stage + lane * p.tile_bytes, map, 0, (tile0 + lane) * 16, kb0, full + 8 * st);
                    } else {
                        for (int ti = 0; ti < tiles; ti++)
                            if (lane < ops) tma_load_2d(stage + ti * p.tile_bytes + lane * 2048, map, (kb0 + lane) * 128, (tile0 + ti) * 16, full + 8 * st);
                    }
                    issued++;
                    uint32_t dst = stage + p.sb_off + (lane / LPR) * SROW + k16;
                    for (int ti = 0; ti < tiles; ti++, dst += 32 * SROW) {
                        if ((tile0 + ti) * 16 + 16 <= p.N) {
#pragma unroll
                            for (int i = 0; i < NB; i++)
                                if (some >> i & 1) {
#pragma unroll
                                    for (int h = 0; h < 2; h++) {
                                        cp_async16(dst + i * RPI * SROW + h * 16 * SROW, sc + (lo[i] + h * half), cnt[i]);
                                        cp_async16(dst + i * RPI * SROW + h * 16 * SROW + 8 * SROW, bi + (lo[i] + h * half), cnt[i]);
                                    }
                                }
                        } else {
                            for (int i = 0; i < NB; i++)
                                for (int h = 0; h < 2; h++) {
                                    const uint32_t src = lo[i] + h * half;
                                    if ((some >> i & 1) && (tile0 + ti) * 16 + i * RPI + lane / LPR + 8 * h < p.N) {
                                        cp_async16(dst + i * RPI * SROW + h * 16 * SROW, sc + src, cnt[i]);
                                        cp_async16(dst + i * RPI * SROW + h * 16 * SROW + 8 * SROW, bi + src, cnt[i]);
                                    }
                                }
                        }
                        if (odd && lane < 16) {
                            const uint32_t n = (tile0 + ti) * 16 + lane, at = 2u * (n * gpr + g0), src = (at & ~15u) + 16 * LPR;
                            const uint32_t d = stage + p.sb_off + ti * (32 * SROW) + (lane >> 3) * (16 * SROW) + (lane & 7) * SROW + 16 * LPR;
                            if (n < (uint32_t)p.N && src < at + need) {
                                const uint32_t c = src < at + bytes ? min(16u, at + bytes - src) : 0u;
                                cp_async16(d, sc + src, c);
                                cp_async16(d + 8 * SROW, bi + src, c);
                            }
                        }
#pragma unroll
                        for (int i = 0; i < NB; i++) lo[i] += 2 * half;
                    }
                    cp_async_arrive(full + 8 * st);
                    next_stage();
                }
            } while (ok && wk.next_run(p));
            asm volatile("cp.async.wait_all;" ::: "memory");
            // after an abort nobody else waits for the copies in flight: they have landed before the CTA ends
            if (!ok)
                for (int i = max(0, issued - p.stages); i < issued; i++)
                    for (int k = 0; k < (1 << 16) && !bar_try(full + 8 * (i % p.stages), (i / p.stages) & 1); k++) {}
        } else if (role - kSumWarp < p.sum_warps) {
            // Stages are taken in turn.  (No more warps than stages: a warp's wait for a stage is then never a whole round
            // ahead of the stage's barrier, whose phase it tells by parity.)
            int turn = role - kSumWarp;
            // The waits below are bounded by the clock, which must not start before the previous kernel of the stream has ended:
            // it may itself be waiting, for a peer, for as long as its caller allows.
            asm volatile("griddepcontrol.wait;" ::: "memory");
            do {
                // the sums carried from chunk to chunk change hands (all these warps come here in every run, after an abort too)
                if (p.nch > 1) asm volatile("bar.sync 2, %0;" ::"r"(p.sum_warps * 32) : "memory");
                const int kn = wk.kb_cnt(p), t_end = wk.tile_end(p);
                int M = p.item(wk.item).M;
                void* y = p.item(wk.item).y;
                if (p.kRows) {
                    M = min(M - kItemRows * wk.item, kItemRows);
                    y = static_cast<char*>(y) + (size_t)wk.item * kItemRows * p.N * (p.y_bf16 ? 2 : 4);
                }
                // lane (g, t) of the MMA: rows n = g, g+8 of the tile, rows of x 2t, 2t+1 (and 8 more)
                const int m0 = 2 * (lane & 3), n0 = lane >> 2;
                for (int g = 0; g < wk.ng && ok; g++) {
                    if (turn-- != 0) {
                        next_stage();
                        continue;
                    }
                    turn = p.sum_warps - 1;
                    ok = bar_wait<true>(sums + 8 * st, ph, abort);
                    if (!ok) break;
                    const int tile0 = wk.b0 + g * p.ts, tiles = min(p.ts, t_end - tile0);
                    for (int i = 0; i < tiles * MT; i++) {
                        const int ti = MT == 1 ? i : i >> 1, mt = MT == 1 ? 0 : i & 1;
                        uint32_t src = ring + st * p.stage_bytes + ti * p.tile_bytes + mt * 512 + lane * 16;
                        const uint32_t run = ring + p.run_off + ((tile0 - wk.b0 + ti) * MT + mt) * 512 + lane * 16;
                        uint4 s = make_uint4(0, 0, 0, 0);
                        if (wk.c) s = lds_v4(run);
                        int k = kn;
                        for (; k >= 4; k -= 4, src += 4 * 2048) {
                            uint4 v[4];
#pragma unroll
                            for (int u = 0; u < 4; u++) v[u] = lds_v4(src + u * 2048);
#pragma unroll
                            for (int u = 0; u < 4; u++) add_f32x4(s, v[u]);
                        }
                        for (; k > 0; k--, src += 2048) add_f32x4(s, lds_v4(src));
                        if (wk.c + 1 < p.nch) {
                            sts_v4(run, s);
                        } else {
                            const int n = (tile0 + ti) * 16 + n0, m = mt * 8 + m0;
                            const bool two = n + 8 < p.N;
                            if (n < p.N && m < M) {
                                const size_t idx = (size_t)m * p.N + n;
                                if (p.y_bf16) {
                                    __nv_bfloat16* q = static_cast<__nv_bfloat16*>(y) + idx;
                                    q[0] = __float2bfloat16_rn(__uint_as_float(s.x));
                                    if (two) q[8] = __float2bfloat16_rn(__uint_as_float(s.z));
                                    if (m + 1 < M) {
                                        q += p.N;
                                        q[0] = __float2bfloat16_rn(__uint_as_float(s.y));
                                        if (two) q[8] = __float2bfloat16_rn(__uint_as_float(s.w));
                                    }
                                } else {
                                    float* q = static_cast<float*>(y) + idx;
                                    q[0] = __uint_as_float(s.x);
                                    if (two) q[8] = __uint_as_float(s.z);
                                    if (m + 1 < M) {
                                        q += p.N;
                                        q[0] = __uint_as_float(s.y);
                                        if (two) q[8] = __uint_as_float(s.w);
                                    }
                                }
                            }
                        }
                    }
                    // what the stage was written and read with is ordered before the copy engine's next write to it
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) bar_arrive(empty + 8 * st);
                    next_stage();
                }
            } while (wk.next_run(p));
        }
    } else {
        // ---------------- dequantise and multiply ----------------
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kWorkRegs));
        const int g = lane >> 2, t = lane & 3;
        const int tsub = warp * p.kbc_inv >> 16, kq = warp - tsub * p.kbc;
        // groups of this run in which the warp has a tile
        auto my_groups = [&]() { return tsub < p.ts && kq < wk.kb_cnt(p) ? (int)((uint32_t)((wk.tile_end(p) - wk.b0 - tsub + p.ts - 1) * p.ts_inv) >> 16) : 0; };

        // x of this warp's k-block, 8 rows at a time: read along the rows, written to the warp's buffer in shared memory in
        // fragment order ([fragment][row][t], the eight 16-byte columns permuted per pair of fragments: no bank conflicts
        // either way), read back as fragments.  Up to 8 rows of x go through in two halves (of the fragments), which leaves
        // room for a stage more; with 16 rows, rows 8..15 stay in the buffer.
        constexpr int PASS = MT == 1 ? 2 : 1, XP = XV / PASS;  // passes, fragments per pass
        const uint32_t xb = ring + p.xs_off + warp * (XP * 512);
        auto frag_addr = [&](int j, int slot) { return xb + (j % XP) * 512 + ((slot ^ (XP == 8 ? (j & 6) : XP == 4 ? (j & 2) << 1 : 0)) << 4); };
        uint4 xr[XV];
        auto pass_x = [&](int row0, bool keep) {
            // lane: a pair of fragments (16 consecutive elements, 32 bytes) of (row, t); PP pairs per t and pass
            constexpr int PP = XP / 2, CPR = 4 * PP, RPI = 32 / CPR, NL = 8 / RPI;
            const Item& it = p.item(wk.item);
            const int first = p.kRows ? wk.item * kItemRows : 0;  // row of the matmul that is the item's row 0
            const int pr = lane % PP, tt = lane / PP % 4, row = row0 + lane / CPR, ld = PRO == 0 ? p.K : p.x_ld;
            const int k0 = (wk.c * p.kbc + kq) * KB + tt * KL + pr * 16;
            V8 v[PASS][NL];
#pragma unroll
            for (int h = 0; h < PASS; h++)
#pragma unroll
                for (int i = 0; i < NL; i++) {
                    const int k = k0 + h * (KL / PASS);
#pragma unroll
                    for (int e = 0; e < 8; e++) v[h][i].v[e] = 0;
                    if (first + row + i * RPI < it.M && k < p.K) {
                        const __nv_bfloat16* s = it.x + (size_t)(first + row + i * RPI) * ld + k;
                        v[h][i] = ldg_32(s, p.x32);
                        if (PRO == 2) {
                            const V8 b = ldg_32(s + p.K, p.x32), d = ldg_32(s + 2 * p.K, p.x32);
#pragma unroll
                            for (int e = 0; e < 8; e++) v[h][i].v[e] = add3_bf16x2(v[h][i].v[e], b.v[e], d.v[e]);
                        }
                    }
                }
#pragma unroll
            for (int h = 0; h < PASS; h++) {
                __syncwarp();  // (earlier fragments have been read)
#pragma unroll
                for (int i = 0; i < NL; i++) {
                    const int slot = (i * RPI + lane / CPR) * 4 + tt, j = h * XP + 2 * pr;
                    if (first + row0 + i * RPI >= it.M) break;  // (rows past M: their columns of the result are never stored)
                    sts_v4(frag_addr(j, slot), permute_x8<BITS>(make_uint4(v[h][i].v[0], v[h][i].v[1], v[h][i].v[2], v[h][i].v[3])));
                    sts_v4(frag_addr(j + 1, slot), permute_x8<BITS>(make_uint4(v[h][i].v[4], v[h][i].v[5], v[h][i].v[6], v[h][i].v[7])));
                }
                __syncwarp();
                if (!keep)
#pragma unroll
                    for (int j = h * XP; j < (h + 1) * XP; j++) xr[j] = lds_v4(frag_addr(j, lane));
            }
        };
        auto load_x = [&]() {
            pass_x(0, false);
            if (MT == 2) pass_x(8, true);
        };
        // What precedes the wait touches only weights, scales and biases (and x where the host knows that the previous
        // kernel of the stream does not write it); behind it the next kernel of the chain may start its own fetch.  (One
        // load_x in the code, ahead of the wait or behind it: two of them cost the 16-row form 100 bytes of spills.)
        int mine = my_groups();
        bool waited = false;
        auto wait_prev = [&]() {
            asm volatile("griddepcontrol.wait;" ::: "memory");
            asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
            waited = true;
        };
        if (NI != 1 || !p.x_early) wait_prev();

        // this lane's place in the stage that comes next: 16-byte pieces 2t and 2t+1 of row g of the k-block
        const uint32_t in_tile = kq * 2048 + g * 128 + (((2 * t) ^ g) << 4), sa0 = ring + tsub * p.tile_bytes + in_tile;
        const uint32_t stage_bytes = p.stage_bytes, full_end = full + 8 * p.stages;
        uint32_t sa = sa0, bar = full, ph = 0;
        bool ok = true;
        auto next_stage = [&]() {
            sa += stage_bytes;
            bar += 8;
            if (bar == full_end) { sa = sa0; bar = full; ph ^= 1; }
        };
        for (;;) {
            const int ng = wk.ng;
            if (mine) load_x();
            if (NI == 1 && !waited) wait_prev();
            if (PRO == 1) {
                // the rows' sums of squares: a k-block's owner (tsub == 0) adds its four lanes per row, then the k-blocks in
                // order through shared memory; every working warp ends up with the factor of its rows
                __shared__ float s_rms[kWarps][8];
                float ss = mine && tsub == 0 ? sumsq_frags<XV>(xr) : 0.0f;
                ss += __shfl_xor_sync(0xffffffffu, ss, 1);
                ss += __shfl_xor_sync(0xffffffffu, ss, 2);
                if (t == 0) s_rms[warp][g] = ss;
                asm volatile("bar.sync 1, %0;" ::"n"(kWarps * 32) : "memory");
                float tot = 0.0f;
#pragma unroll
                for (int w = 0; w < kWarps; w++) tot += s_rms[w][g];
                rms_scale<XV>(xr, __fdiv_rn(1.0f, sqrtf(__fadd_rn(__fdiv_rn(tot, (float)p.K), p.eps))));
            }
            // this lane's scales in a stage, from its weights: its group (the zeros behind the row's last one where K ends before
            // it) in the row's pieces, which begin up to 14 bytes ahead of the chunk's first one (the same for rows 8 apart)
            uint32_t sb_lane;
            {
                const int kb0 = wk.c * p.kbc, gpr = p.K >> p.gshift, g0 = kb0 * KB >> p.gshift, gi = min(((kb0 + kq) * KB + t * KL) >> p.gshift, gpr);
                const int n = (wk.b0 + tsub) * 16 + g;
                sb_lane = p.sb_off + tsub * (32 * SROW - p.tile_bytes) + g * SROW + ((uint32_t)((n * gpr + g0) * 2) & 15u) + 2 * (gi - g0) - in_tile;
            }
#pragma unroll 1
            for (int gi = 0; gi < mine; gi++) {
                if (!bar_wait<false>(bar, ph, abort)) { ok = false; break; }
                uint32_t w[2][8], s[2][SPL], b[2][SPL];
#pragma unroll
                for (int r = 0; r < 2; r++)
#pragma unroll
                    for (int i = 0; i < SPL; i++) {
                        s[r][i] = lds_u16(sa + sb_lane + 2 * i + r * 16 * SROW);
                        b[r][i] = lds_u16(sa + sb_lane + 2 * i + r * 16 * SROW + 8 * SROW);
                    }
#pragma unroll
                for (int r = 0; r < 2; r++)
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        const uint4 v = lds_v4((h ? sa ^ 16u : sa) + r * 1024);
                        w[r][4 * h] = v.x; w[r][4 * h + 1] = v.y; w[r][4 * h + 2] = v.z; w[r][4 * h + 3] = v.w;
                    }
                float4 out[MT];
                auto x_hi = [&](int j) { return lds_v4(frag_addr(j, lane)); };
                if (__all_sync(0xffffffffu, scales_fast_ok<SPL>(s))) task_mma<BITS, MT, SPL, true>(w, s, b, xr, x_hi, out);
                else task_mma<BITS, MT, SPL, false>(w, s, b, xr, x_hi, out);
                // the partial takes the place of the weights it came from (nobody else's, and all of them have been used)
#pragma unroll
                for (int mt = 0; mt < MT; mt++)
                    sts_v4(sa - in_tile + kq * 2048 + mt * 512 + lane * 16,
                           make_uint4(__float_as_uint(out[mt].x), __float_as_uint(out[mt].y), __float_as_uint(out[mt].z), __float_as_uint(out[mt].w)));
                __syncwarp();
                if (lane == 0) bar_arrive(bar + 8 * kMaxStages);
                next_stage();
            }
            for (int gi = mine; gi < ng && ok; gi++) {  // groups without a tile of this warp
                ok = bar_wait<false>(bar, ph, abort);
                if (ok && lane == 0) bar_arrive(bar + 8 * kMaxStages);
                next_stage();
            }
            if (!ok || !wk.next_run(p)) break;
            mine = my_groups();
        }
    }
    __syncthreads();
    if (tid == 0 && s_abort && p.error) *p.error = 1;
}

// ---- host side ------------------------------------------------------------------------------------------------------
using Plan = QmvStreamPlan;

bool make_plan(const QmmArgs& a, int mmax, int sm_count, Plan* pl) {
    if (a.x_dtype != LUX_DTYPE_BFLOAT16 || a.sb_dtype != LUX_DTYPE_BFLOAT16 || (a.bits != 4 && a.bits != 8)) return false;
    if (mmax < 1 || mmax > 16 || a.N < 1 || sm_count < 1 || (a.group != 32 && a.group != 64 && a.group != 128) || a.K % a.group) return false;
    if (((uintptr_t)a.wq | (uintptr_t)a.x | (uintptr_t)a.scales | (uintptr_t)a.biases) & 15) return false;
    pl->gshift = a.group == 32 ? 5 : (a.group == 64 ? 6 : 7);
    const int KB = 1024 / a.bits, mt = mmax <= 8 ? 1 : 2;
    pl->nkb = (a.K + KB - 1) / KB;
    pl->n_rt = (a.N + 15) / 16;
    if ((long long)a.N * (a.K / a.group) > (1ll << 30) || (long long)pl->n_rt * pl->nkb > (1ll << 26)) return false;  // 32-bit indices
    pl->grid = std::min(pl->n_rt, sm_count);
    pl->grid_y = 1;
    const int tiles_max = (pl->n_rt + pl->grid - 1) / pl->grid;
    pl->nch = (pl->nkb + kWarps - 1) / kWarps;
    pl->kbc = (pl->nkb + pl->nch - 1) / pl->nch;
    pl->nch = (pl->nkb + pl->kbc - 1) / pl->kbc;
    pl->tile_bytes = pl->kbc * 2048;
    const int sb = 32 * sb_row(a.bits == 4 && a.group == 32 ? 2 : 1), xs = kWarps * x_frags(a.bits) * 512 / (mt == 1 ? 2 : 1), bars = 8 * 3 * kMaxStages;
    // K in one chunk: nothing is kept per tile (4096: as far as Walk::groups divides exactly); in several: the tiles' running sums
    pl->tb = std::min(tiles_max, pl->nch == 1 ? 4096 : 16 * 1024 / (mt * 512));
    const int run = pl->nch == 1 ? 0 : pl->tb * mt * 512;
    // a short K: several tiles per stage keep the warps busy (as many as leave room for two stages)
    for (pl->ts = std::max(1, std::min(kWarps / pl->kbc, tiles_max));; pl->ts--) {
        pl->sb_off = pl->ts * pl->tile_bytes;
        pl->stage_bytes = (pl->sb_off + pl->ts * sb + 1023) & ~1023;
        pl->stages = std::min(kMaxStages, (kSmemLimit - run - xs - bars) / pl->stage_bytes);
        if (pl->stages >= 2) break;
        if (pl->ts == 1) return false;
    }
    pl->xs_off = pl->stages * pl->stage_bytes;
    pl->run_off = pl->xs_off + xs;
    pl->bar_off = pl->run_off + run;
    pl->smem = (size_t)pl->bar_off + bars;
    return true;
}

// The packed weights as bytes for the copy engine, a tile of 16 rows being one box: [k-block][row][128 bytes], 128-byte
// swizzle.  With K cut off inside a k-block the boxes are single k-blocks of a plain [row][byte] tensor, whose bytes past
// the row's end read as zero.
bool encode_weights(const QmmArgs& a, const Plan& pl, CUtensorMap* map) {
    const EncodeTiledFn encode = encode_tiled_fn();
    if (!encode) return false;
    const cuuint64_t row_bytes = (cuuint64_t)a.K * a.bits / 8;
    const cuuint32_t estr[3] = {1, 1, 1};
    CUresult r;
    if (row_bytes % 128 == 0) {
        const cuuint64_t dims[3] = {128, (cuuint64_t)a.N, row_bytes / 128}, strides[2] = {row_bytes, 128};
        const cuuint32_t box[3] = {128, 16, (cuuint32_t)pl.kbc};
        r = encode(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<uint32_t*>(a.wq), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                   CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    } else {
        const cuuint64_t dims[2] = {row_bytes, (cuuint64_t)a.N}, strides[1] = {row_bytes};
        const cuuint32_t box[2] = {128, 16};
        r = encode(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<uint32_t*>(a.wq), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                   CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    }
    if (r != CUDA_SUCCESS) set_last_error("cuTensorMapEncodeTiled (weights) failed (%d)", (int)r);
    return r == CUDA_SUCCESS;
}

template <int BITS, int MT, int SPL, int PRO, int NI>
cudaError_t launch_t(const Params<NI>& p, const Plan& pl, cudaStream_t stream, bool overlap_prev) {
    auto kern = qmv_stream_kernel<BITS, MT, SPL, PRO, NI>;
    static std::atomic<bool> attr_set[64];
    if (cudaError_t e = allow_smem(kern, kSmemLimit, attr_set)) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(pl.grid, pl.grid_y);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = pl.smem;
    cfg.stream = stream;
    // As a programmatic dependent the grid may start (and fetch weights) while the previous kernel of the stream drains;
    // everything that depends on that kernel sits behind the working warps' griddepcontrol.wait.
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = overlap_prev ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kern, p);
}

template <int BITS, int SPL, int NI>
cudaError_t launch_rows(const Params<NI>& p, const Plan& pl, int mmax, int pro, cudaStream_t stream, bool overlap_prev) {
    if constexpr (NI > 0) {
        constexpr int P1 = NI == 1 ? 1 : 0, P2 = NI == 1 ? 2 : 0;  // (prologues: single calls only)
        if (mmax <= 8)
            return pro == 1   ? launch_t<BITS, 1, SPL, P1, NI>(p, pl, stream, overlap_prev)
                   : pro == 2 ? launch_t<BITS, 1, SPL, P2, NI>(p, pl, stream, overlap_prev)
                              : launch_t<BITS, 1, SPL, 0, NI>(p, pl, stream, overlap_prev);
    }
    return launch_t<BITS, 2, SPL, 0, NI>(p, pl, stream, overlap_prev);
}

template <int NI>
cudaError_t launch_items(const QmmArgs* items, int n, int mmax, const Plan& pl, cudaStream_t stream, bool overlap_prev, bool x_stable) {
    const QmmArgs& a0 = items[0];
    Params<NI> p;
    p.n_items = p.kRows ? (a0.M + kItemRows - 1) / kItemRows : n;
    p.K = a0.K; p.N = a0.N; p.gshift = pl.gshift; p.y_bf16 = a0.y_dtype == LUX_DTYPE_BFLOAT16;
    p.rt_q = pl.n_rt / pl.grid; p.rt_rem = pl.n_rt % pl.grid;
    p.ts_inv = (65536 + pl.ts - 1) / pl.ts; p.kbc_inv = (65536 + pl.kbc - 1) / pl.kbc;
    p.nkb = pl.nkb; p.nch = pl.nch; p.kbc = pl.kbc; p.ts = pl.ts; p.tb = pl.tb;
    p.stages = pl.stages; p.sum_warps = std::min(kSumWarps, pl.stages); p.stage_bytes = pl.stage_bytes; p.tile_bytes = pl.tile_bytes; p.k_tail = a0.K % (1024 / a0.bits) != 0;
    p.sb_off = pl.sb_off; p.xs_off = pl.xs_off; p.run_off = pl.run_off; p.bar_off = pl.bar_off;
    p.x_early = (!overlap_prev || x_stable) ? 1 : 0;
    p.x_ld = a0.pro ? a0.x_ld : a0.K;
    p.eps = a0.eps;
    p.error = a0.error ? a0.error : device_error_word();
    p.x32 = p.x_ld % 16 == 0;
    for (int i = 0; i < n; i++) {
        if ((uintptr_t)items[i].x & 31) p.x32 = 0;
        if (!encode_weights(items[i], pl, &p.maps[i])) return cudaErrorInvalidValue;
        p.items[i] = Item{(const __nv_bfloat16*)items[i].x, (const __nv_bfloat16*)items[i].scales,
                          (const __nv_bfloat16*)items[i].biases, items[i].y, items[i].M};
    }
    return a0.bits == 8     ? launch_rows<8, 1, NI>(p, pl, mmax, a0.pro, stream, overlap_prev)
           : a0.group == 32 ? launch_rows<4, 2, NI>(p, pl, mmax, a0.pro, stream, overlap_prev)
                            : launch_rows<4, 1, NI>(p, pl, mmax, a0.pro, stream, overlap_prev);
}

}  // namespace

bool plan_qmv_stream(const QmmArgs& a, int sm_count, QmvStreamPlan* pl) {
    if (!make_plan(a, std::min(a.M, kItemRows), sm_count, pl)) return false;
    if (a.M > kItemRows) pl->grid_y = std::min((a.M + kItemRows - 1) / kItemRows, sm_count / pl->grid);
    return true;
}

int qmv_batch_max() { return kMaxBatch; }

cudaError_t launch_qmv_stream(const QmmArgs& a, const QmvStreamPlan& pl, cudaStream_t stream, bool overlap_prev, bool x_stable) {
    // the rms-norm prologue needs the whole of x in the first fragments of the CTA's warps
    if (a.pro && (a.M > 8 || (a.pro == 1 && pl.nch != 1))) return cudaErrorNotSupported;
    return a.M > kItemRows ? launch_items<0>(&a, 1, a.M, pl, stream, overlap_prev, x_stable)
                           : launch_items<1>(&a, 1, a.M, pl, stream, overlap_prev, x_stable);
}

cudaError_t launch_qmv_stream_batch(const QmmArgs* items, int n, int sm_count, cudaStream_t stream) {
    if (n < 1 || n > kMaxBatch) return cudaErrorInvalidValue;
    const QmmArgs& a0 = items[0];
    int mmax = 0;
    for (int i = 0; i < n; i++) {
        const QmmArgs& a = items[i];
        mmax = std::max(mmax, a.M);
        if (a.K != a0.K || a.N != a0.N || a.bits != a0.bits || a.group != a0.group || a.y_dtype != a0.y_dtype || a.M < 1 || a.pro ||
            a.x_dtype != LUX_DTYPE_BFLOAT16 || a.sb_dtype != LUX_DTYPE_BFLOAT16)
            return cudaErrorNotSupported;
        if (((uintptr_t)a.wq | (uintptr_t)a.x | (uintptr_t)a.scales | (uintptr_t)a.biases) & 15) return cudaErrorInvalidValue;
    }
    Plan pl;
    if (mmax > kItemRows || !make_plan(a0, mmax, sm_count, &pl)) return cudaErrorNotSupported;
    return n == 1 ? launch_items<1>(items, n, mmax, pl, stream, false, false) : launch_items<kMaxBatch>(items, n, mmax, pl, stream, false, false);
}

}  // namespace luxcuda
