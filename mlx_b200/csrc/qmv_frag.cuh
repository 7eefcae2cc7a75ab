// What the decode kernels (qmv_mma.cu, qmv_stream.cu) share: a "task" is 16 rows of W times one k-block (128 bytes of
// packed weights per row: 256 four-bit or 128 eight-bit weights) times up to 8*MT rows of x, done by one warp with
// mma.sync.m16n8k16 on weights dequantised in registers.
//
// Lane (g = lane/4, t = lane%4) holds the 32 bytes [32t, 32t+32) of rows g and g+8 of the k-block: KL = 64 (32)
// consecutive weights per row, i.e. one quantisation group, part of one, or two groups of 32 at 4 bit (SPL scales per
// row).  The dot product is invariant under a permutation of k applied to both operands, so the weights are used in the
// order the mask/shift unpack yields them and the x fragments are brought into that order.
//
// Every decode kernel accumulates a task in the same two chains of MMAs, adds the two, and sums the tasks of an output
// in k-block order: all of them give the same bits whatever the grid, the number of rows of x, the K split or the
// sharding.
#pragma once
#include <cuda_bf16.h>

#include "dequant.cuh"

namespace luxcuda {

constexpr int kb_weights(int bits) { return 1024 / bits; }        // weights per k-block and row
constexpr int lane_weights(int bits) { return 256 / bits; }       // ... and lane
constexpr int x_frags(int bits) { return lane_weights(bits) / 8; }  // uint4 of x per lane, k-block and 8 rows of x

__device__ __forceinline__ void mma_bf16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                         uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// the first MMA of a chain: C = 0
__device__ __forceinline__ void mma_bf16_first(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                               uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.0f));
}

// all scales (raw bf16 bits, two rows) usable by the exponent-trick dequantiser?  Packed form of scale_fast_ok: exponent
// field e in [1, 121]  <=>  ((s - 0x80) & 0x7F80) <= 0x3C00 per half.
template <int SPL>
__device__ __forceinline__ bool scales_fast_ok(const uint32_t (&s)[2][SPL]) {
    uint32_t a = 0;
#pragma unroll
    for (int i = 0; i < SPL; i++) a |= (((s[0][i] | (s[1][i] << 16)) - 0x00800080u) & 0x7F807F80u) + 0x43804380u;
    return (a & 0x80008000u) == 0u;
}

// One task: w = the lane's 8 words of rows g and g+8, s / b their scales and biases, xr = the x fragments of rows 0..7,
// xs(j) = (MT == 2) fragment j of rows 8..15, in shared memory.  Result: out (the sum of the two chains).
template <int BITS, int MT, int SPL, bool FAST, class XS>
__device__ __forceinline__ void task_mma(const uint32_t (&w)[2][8], const uint32_t (&s)[2][SPL], const uint32_t (&b)[2][SPL],
                                         const uint4 (&xr)[x_frags(BITS)], const XS& xs, float4 (&out)[MT]) {
    float acc[MT][2][4];
    uint32_t sa[2], sb[2], b2[2];
#pragma unroll
    for (int j = 0; j < x_frags(BITS); j++) {
        if (j % (x_frags(BITS) / SPL) == 0) {
            const int i = j / (x_frags(BITS) / SPL);
#pragma unroll
            for (int r = 0; r < 2; r++) {
                b2[r] = dup_bf16(b[r][i]);
                sa[r] = FAST ? scale_x2_133(s[r][i]) : dup_bf16(s[r][i]);
                sb[r] = FAST && BITS == 4 ? scale_x2_129(s[r][i]) : 0u;
            }
        }
        uint32_t lo[4], hi[4];  // four pairs of weights of row g (lo) and of row g+8 (hi)
        if (BITS == 4) {
            if (FAST) {
                dequant4_fast(w[0][j], sa[0], sb[0], b2[0], lo);
                dequant4_fast(w[1][j], sa[1], sb[1], b2[1], hi);
            } else {
                dequant4_general(w[0][j], sa[0], b2[0], lo);
                dequant4_general(w[1][j], sa[1], b2[1], hi);
            }
        } else {
            constexpr int J = 7;  // (the index stays inside w for the 4-bit instantiation too)
            const int i0 = 2 * j & J, i1 = (2 * j + 1) & J;
            uint32_t l0[2], l1[2], h0[2], h1[2];
            if (FAST) {
                dequant8_fast(w[0][i0], sa[0], b2[0], l0);
                dequant8_fast(w[0][i1], sa[0], b2[0], l1);
                dequant8_fast(w[1][i0], sa[1], b2[1], h0);
                dequant8_fast(w[1][i1], sa[1], b2[1], h1);
            } else {
                dequant8_general(w[0][i0], sa[0], b2[0], l0);
                dequant8_general(w[0][i1], sa[0], b2[0], l1);
                dequant8_general(w[1][i0], sa[1], b2[1], h0);
                dequant8_general(w[1][i1], sa[1], b2[1], h1);
            }
            lo[0] = l0[0]; lo[1] = l0[1]; lo[2] = l1[0]; lo[3] = l1[1];
            hi[0] = h0[0]; hi[1] = h0[1]; hi[2] = h1[0]; hi[3] = h1[1];
        }
#pragma unroll
        for (int mt = 0; mt < MT; mt++) {
            const uint4 bx = mt == 0 ? xr[j] : xs(j);
            if (j == 0) {
                mma_bf16_first(acc[mt][0], lo[0], hi[0], lo[1], hi[1], bx.x, bx.y);
                mma_bf16_first(acc[mt][1], lo[2], hi[2], lo[3], hi[3], bx.z, bx.w);
            } else {
                mma_bf16(acc[mt][0], lo[0], hi[0], lo[1], hi[1], bx.x, bx.y);
                mma_bf16(acc[mt][1], lo[2], hi[2], lo[3], hi[3], bx.z, bx.w);
            }
        }
    }
#pragma unroll
    for (int mt = 0; mt < MT; mt++)
        out[mt] = make_float4(acc[mt][0][0] + acc[mt][1][0], acc[mt][0][1] + acc[mt][1][1], acc[mt][0][2] + acc[mt][1][2],
                              acc[mt][0][3] + acc[mt][1][3]);
}

// ---- x fragments ----------------------------------------------------------------------------------------------------
// Fragment j of lane (g, t) covers x[row g][kb*KB + t*KL + 8j .. +8), as the unpack orders the weights:
//   4-bit: (0,4) (1,5) (2,6) (3,7)      8-bit: (0,2) (1,3) (4,6) (5,7)
struct V8 {
    uint32_t v[8];
};
__device__ __forceinline__ V8 ldg_v8(const void* p) {  // 32 bytes, through L1 as an earlier launch's output (no .nc)
    V8 r;
    asm volatile("ld.global.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r.v[0]), "=r"(r.v[1]), "=r"(r.v[2]), "=r"(r.v[3]), "=r"(r.v[4]), "=r"(r.v[5]), "=r"(r.v[6]), "=r"(r.v[7])
                 : "l"(p));
    return r;
}

__device__ __forceinline__ V8 ldg_2v4(const void* p) {  // the same from a 16-byte boundary
    V8 r;
    asm volatile("ld.global.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(r.v[0]), "=r"(r.v[1]), "=r"(r.v[2]), "=r"(r.v[3]) : "l"(p));
    asm volatile("ld.global.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(r.v[4]), "=r"(r.v[5]), "=r"(r.v[6]), "=r"(r.v[7]) : "l"((const char*)p + 16));
    return r;
}
__device__ __forceinline__ V8 ldg_32(const void* p, bool aligned) { return aligned ? ldg_v8(p) : ldg_2v4(p); }
__device__ __forceinline__ uint32_t add3_bf16x2(uint32_t a, uint32_t b, uint32_t c) {
    const float lo = __fadd_rn(__fadd_rn(__uint_as_float(a << 16), __uint_as_float(b << 16)), __uint_as_float(c << 16));
    const float hi = __fadd_rn(__fadd_rn(__uint_as_float(a & 0xFFFF0000u), __uint_as_float(b & 0xFFFF0000u)), __uint_as_float(c & 0xFFFF0000u));
    const __nv_bfloat162 r = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&r);
}
// The fragments of k-block kb (all of it inside K) of one row of x (row = nullptr: a row past M, zeros), in natural k order;
// x32: rows start on 32-byte boundaries.  PRO 2: bf16(a + b + c) of the column blocks [0,K), [K,2K), [2K,3K) (fp32 adds, left to
// right, one rounding: the bits of the stand-alone sum3 kernel).
template <int BITS, int PRO>
__device__ __forceinline__ void load_x_row(const __nv_bfloat16* row, int K, int kb, int t, bool x32, uint4 (&xr)[x_frags(BITS)]) {
    const int k0 = kb * kb_weights(BITS) + t * lane_weights(BITS);
#pragma unroll
    for (int j = 0; j < x_frags(BITS); j += 2) {
        xr[j] = xr[j + 1] = make_uint4(0, 0, 0, 0);
        if (row) {
            const __nv_bfloat16* src = row + k0 + 8 * j;
            V8 v = ldg_32(src, x32);
            if (PRO == 2) {
                const V8 b = ldg_32(src + K, x32), c = ldg_32(src + 2 * K, x32);
#pragma unroll
                for (int e = 0; e < 8; e++) v.v[e] = add3_bf16x2(v.v[e], b.v[e], c.v[e]);
            }
            xr[j] = make_uint4(v.v[0], v.v[1], v.v[2], v.v[3]);
            xr[j + 1] = make_uint4(v.v[4], v.v[5], v.v[6], v.v[7]);
        }
    }
}
// natural k order -> the order of the unpacked weights
template <int BITS>
__device__ __forceinline__ uint4 permute_x8(const uint4& v) {
    if (BITS == 4) return make_uint4(prmt(v.x, v.z, 0x5410u), prmt(v.x, v.z, 0x7632u), prmt(v.y, v.w, 0x5410u), prmt(v.y, v.w, 0x7632u));
    return make_uint4(prmt(v.x, v.y, 0x5410u), prmt(v.x, v.y, 0x7632u), prmt(v.z, v.w, 0x5410u), prmt(v.z, v.w, 0x7632u));
}
template <int BITS>
__device__ __forceinline__ void permute_x(uint4 (&xr)[x_frags(BITS)]) {
#pragma unroll
    for (int j = 0; j < x_frags(BITS); j++) xr[j] = permute_x8<BITS>(xr[j]);
}
// rms-norm prologue: the sum of squares of a lane's fragments (fp32), and the fragments scaled and rounded as the
// stand-alone rms-norm kernel does it: bf16(fl32(x * inv)).
template <int XV>
__device__ __forceinline__ float sumsq_frags(const uint4 (&xr)[XV]) {
    float ss = 0.0f;
#pragma unroll
    for (int j = 0; j < XV; j++) {
        const uint32_t w[4] = {xr[j].x, xr[j].y, xr[j].z, xr[j].w};
#pragma unroll
        for (int e = 0; e < 4; e++) {
            const float lo = __uint_as_float(w[e] << 16), hi = __uint_as_float(w[e] & 0xFFFF0000u);
            ss = fmaf(lo, lo, ss);
            ss = fmaf(hi, hi, ss);
        }
    }
    return ss;
}
__device__ __forceinline__ uint32_t scale_bf16x2(uint32_t v, float inv) {
    const __nv_bfloat162 r = __floats2bfloat162_rn(__fmul_rn(__uint_as_float(v << 16), inv), __fmul_rn(__uint_as_float(v & 0xFFFF0000u), inv));
    return *reinterpret_cast<const uint32_t*>(&r);
}
template <int XV>
__device__ __forceinline__ void rms_scale(uint4 (&xr)[XV], float inv) {
#pragma unroll
    for (int j = 0; j < XV; j++)
        xr[j] = make_uint4(scale_bf16x2(xr[j].x, inv), scale_bf16x2(xr[j].y, inv), scale_bf16x2(xr[j].z, inv), scale_bf16x2(xr[j].w, inv));
}

}  // namespace luxcuda
