// Quantized matmul on CUDA cores: y[M,N] = x[M,K] . dequant(Wq[N,K])^T.
//   qmv_f32_kernel   the fp32 compute path (x fp32; w^ = fl32(fl32(s*q)+b));
//   qmv_simt_kernel  the bf16 path (w^ = one bf16 FMA) for what the tensor-core kernels do not take (index ranges past
//                    their 32-bit limits).
// HBM-bound with few rows of x: algorithmic bytes per row of W = K*bits/8 + 2*(K/group)*sizeof(scale).
#include <cuda_bf16.h>

#include <algorithm>

#include "internal.h"
#include "qmv_frag.cuh"

namespace luxcuda {

namespace {

__device__ __forceinline__ uint4 ldg_stream(const uint4* p) {
    uint4 r;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w)
                 : "l"(p));
    return r;
}

// ---- bf16 -----------------------------------------------------------------------------------------------------------
// One warp owns R consecutive rows of W.  Per step every lane fetches one 16-byte piece of each row (32 four-bit or 16
// eight-bit weights, all inside one quantisation group), dequantises it once, and reuses it for MB rows of x.
// PER consecutive activations (naturally aligned) as fp32
template <int PER>
__device__ __forceinline__ void load_x(const void* p, float* out) {
    uint32_t v[PER / 2];
    if (PER == 8) {
        const uint4 t = __ldg((const uint4*)p);
        v[0] = t.x; v[1] = t.y; v[PER / 2 - 2] = t.z; v[PER / 2 - 1] = t.w;
    } else {
        const uint2 t = __ldg((const uint2*)p);
        v[0] = t.x; v[1] = t.y;
    }
#pragma unroll
    for (int i = 0; i < PER / 2; i++) {
        out[2 * i] = __uint_as_float(v[i] << 16);
        out[2 * i + 1] = __uint_as_float(v[i] & 0xFFFF0000u);
    }
}

template <int BITS, int R, int MB>
__global__ void __launch_bounds__(256)
qmv_simt_kernel(const __nv_bfloat16* __restrict__ x, const uint32_t* __restrict__ wq, const __nv_bfloat16* __restrict__ scales,
                const __nv_bfloat16* __restrict__ biases, void* __restrict__ yv, int M, int K, int N, int group, int y_dtype) {
    constexpr int KP = 128 / BITS;  // weights per 16-byte piece
    const int lane = threadIdx.x & 31;
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int n0 = warp * R;
    if (n0 >= N) return;
    const int m0 = blockIdx.y * MB;
    const int wpr = K * BITS / 32, gpr = K / group;
    const int pieces = wpr / 4;

    float acc[R][MB];
#pragma unroll
    for (int r = 0; r < R; r++)
#pragma unroll
        for (int m = 0; m < MB; m++) acc[r][m] = 0.0f;

    for (int p = lane; p < pieces; p += 32) {
        const int k0 = p * KP;
        uint4 wv[R];
        __nv_bfloat16 s[R], b[R];
#pragma unroll
        for (int r = 0; r < R; r++) {
            const int n = min(n0 + r, N - 1);
            wv[r] = ldg_stream((const uint4*)(wq + (size_t)n * wpr) + p);
            const size_t gi = (size_t)n * gpr + k0 / group;
            s[r] = scales[gi];
            b[r] = biases[gi];
        }
#pragma unroll
        for (int w = 0; w < 4; w++) {
            constexpr int PER = 32 / BITS;  // weights per word
            float xr[MB][PER];
#pragma unroll
            for (int m = 0; m < MB; m++) {
                const int mm = min(m0 + m, M - 1);
                load_x<PER>(x + (size_t)mm * K + k0 + w * PER, xr[m]);
            }
#pragma unroll
            for (int r = 0; r < R; r++) {
                const uint32_t word = w == 0 ? wv[r].x : (w == 1 ? wv[r].y : (w == 2 ? wv[r].z : wv[r].w));
#pragma unroll
                for (int j = 0; j < PER; j++) {
                    const uint32_t q = (word >> (BITS * j)) & ((1u << BITS) - 1);
                    const float wf = __bfloat162float(__hfma(__float2bfloat16_rn((float)q), s[r], b[r]));
#pragma unroll
                    for (int m = 0; m < MB; m++) acc[r][m] = fmaf(xr[m][j], wf, acc[r][m]);
                }
            }
        }
    }
#pragma unroll
    for (int r = 0; r < R; r++)
#pragma unroll
        for (int m = 0; m < MB; m++) {
            float v = acc[r][m];
#pragma unroll
            for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            if (lane == 0 && n0 + r < N && m0 + m < M) {
                const size_t idx = (size_t)(m0 + m) * N + n0 + r;
                if (y_dtype == LUX_DTYPE_BFLOAT16) ((__nv_bfloat16*)yv)[idx] = __float2bfloat16_rn(v);
                else ((float*)yv)[idx] = v;
            }
        }
}

template <int BITS, int R, int MB>
cudaError_t launch_one(const QmmArgs& a, cudaStream_t stream) {
    const int warps = (a.N + R - 1) / R;
    dim3 grid((warps + 7) / 8, (a.M + MB - 1) / MB);
    qmv_simt_kernel<BITS, R, MB><<<grid, 256, 0, stream>>>((const __nv_bfloat16*)a.x, a.wq, (const __nv_bfloat16*)a.scales,
                                                           (const __nv_bfloat16*)a.biases, a.y, a.M, a.K, a.N, a.group, a.y_dtype);
    return cudaGetLastError();
}
template <int BITS>
cudaError_t launch_bf16(const QmmArgs& a, cudaStream_t stream) {
    if (a.M == 1) return launch_one<BITS, 4, 1>(a, stream);
    return a.M == 2 ? launch_one<BITS, 2, 2>(a, stream) : launch_one<BITS, 2, 4>(a, stream);
}

// ---- fp32 -----------------------------------------------------------------------------------------------------------
// A warp computes R rows of W times MB rows of x over its part of K; the kw warps that share these rows take the pieces
// of K in turn and add up through shared memory, in order.  A piece is 8 weights for each lane, side by side, so that
// weights and x are read along their rows, x 32 bytes at a time.  (A lane reading 32 weights at once needs x 128 bytes from
// the next lane's, 32 lines per load.)
// A sum's order follows from K alone: its P parts (f32_parts), part q adding pieces q, q + P, ... lane by lane; then the
// lanes; then the parts in order.  So one row of x and one row of W have the same bits in every call, whatever the other
// rows are, on any GPU and however the columns of a layer are sharded.  A warp may take several parts (U, their pieces side
// by side, a sum for each).
// Arithmetic runs on pairs (f32x2): per two weights two shifts, two and-ors (q + 2^23 as bits), the subtraction of 2^23,
// s*q, + b and one FMA per row of x.
// Eight 4096 x 4096 layers, 4 bit, group 64, fp32 scales, one row, call by call: 107 us with a lane's 32 weights at once and
// a launch that waits for the one before it; 82 with
// pieces; 61 as programmatic dependents (84 MB: 1.4 TB/s).  The order that follows from K alone, against parts chosen by the
// number of rows: between 0.65 and 1.37 of the time over 344 shapes, 1.02 on average (8 x 8192 x 256 10.4 -> 6.9 us,
// 1 x 1024 x 8192 3.6 -> 4.6).
__device__ __forceinline__ uint64_t pack2(uint32_t lo, uint32_t hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(lo), "r"(hi));
    return r;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
constexpr uint32_t kBits2p23 = 0x4B000000u;  // 2^23: or-ing q into it gives the float 2^23 + q
constexpr uint64_t kMinus2p23x2 = 0xCB000000CB000000ull;

// C values per lane over the 32 lanes -> every lane holds the sum of one of them, number lane >> (5 - log2 C)
template <int C>
__device__ __forceinline__ float reduce_warp(float (&v)[C], int lane) {
    int o = 16;
#pragma unroll
    for (int c = C / 2; c >= 1; c /= 2, o /= 2) {
        const bool up = lane & o;
#pragma unroll
        for (int i = 0; i < c; i++) {
            const float keep = up ? v[i + c] : v[i], send = up ? v[i] : v[i + c];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
    }
#pragma unroll
    for (; o >= 1; o /= 2) v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
    return v[0];
}

constexpr int kF32Warps = 8, kF32Rows = 4;
constexpr int kF32Piece = 8;  // weights of a lane
// log2 of the number of parts of K: 8, fewer where there is no piece for each
int f32_parts(int K) { return K > 4 * 32 * kF32Piece ? 3 : K > 2 * 32 * kF32Piece ? 2 : 1; }
// U parts per warp, D pieces of each under way at a time; BLK blocks per SM
template <int BITS, bool SB16, int MB, int U, int D, int BLK>
__global__ void __launch_bounds__(kF32Warps * 32, BLK)
qmv_f32_kernel(const float* x, const unsigned char* __restrict__ wq, const void* __restrict__ scales,
               const void* __restrict__ biases, void* yv, int M, int K, int N, int gshift, int kw_shift, int x32, int y_bf16) {
    constexpr int R = kF32Rows, V = kF32Piece, WW = BITS / 4;  // WW: words of weights per lane and piece
    __shared__ float red[kF32Warps * U][R * MB];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, kw = 1 << kw_shift, part = warp & (kw - 1);
    const int n0 = (blockIdx.x * (kF32Warps >> kw_shift) + (warp >> kw_shift)) * R, m0 = blockIdx.y * MB;
    const size_t row_bytes = (size_t)K * BITS / 8, gpr = (size_t)K >> gshift;
    const int pieces = (K + 32 * V - 1) / (32 * V);
    uint64_t acc[U][R][MB];
#pragma unroll
    for (int u = 0; u < U; u++)
#pragma unroll
        for (int r = 0; r < R; r++)
#pragma unroll
            for (int m = 0; m < MB; m++) acc[u][r][m] = 0;
    uint32_t w[U * D][R][WW], s[U * D][R], b[U * D][R];  // (piece i: part i % U)
    auto load_weights = [&](int p0) {
#pragma unroll
        for (int u = 0; u < U * D; u++) {
            const int k = (p0 + u * kw) * (32 * V) + lane * V;
#pragma unroll
            for (int r = 0; r < R; r++) {
                w[u][r][0] = w[u][r][WW - 1] = 0;
                s[u][r] = b[u][r] = 0;
                if (k >= K) continue;  // (past the end: w^ = 0, x = 0)
                const size_t n = min(n0 + r, N - 1), gi = n * gpr + (k >> gshift);
                const unsigned char* wp = wq + n * row_bytes + (size_t)k * BITS / 8;
                if (WW == 1)
                    asm volatile("ld.global.nc.L1::no_allocate.u32 %0, [%1];" : "=r"(w[u][r][0]) : "l"(wp));
                else
                    asm volatile("ld.global.nc.L1::no_allocate.v2.u32 {%0,%1}, [%2];" : "=r"(w[u][r][0]), "=r"(w[u][r][WW - 1]) : "l"(wp));
                if (SB16) {
                    s[u][r] = (uint32_t)__ldg(static_cast<const uint16_t*>(scales) + gi) << 16;
                    b[u][r] = (uint32_t)__ldg(static_cast<const uint16_t*>(biases) + gi) << 16;
                } else {
                    s[u][r] = __ldg(static_cast<const uint32_t*>(scales) + gi);
                    b[u][r] = __ldg(static_cast<const uint32_t*>(biases) + gi);
                }
            }
        }
    };
    // What precedes the wait touches only weights, scales and biases; behind it the next kernel of a chain may start its
    // own fetch.
    if (n0 < N) load_weights(part);
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (n0 < N) {
        for (int p0 = part; p0 < pieces; p0 += kw * U * D) {
            if (p0 != part) load_weights(p0);
            uint64_t xr[MB == 1 ? U * D : 1][V / 2];
            auto load_row = [&](int u, int m, uint64_t (&v)[V / 2]) {
                const int k = (p0 + u * kw) * (32 * V) + lane * V;
                V8 t;
#pragma unroll
                for (int i = 0; i < V; i++) t.v[i] = 0;
                if (k < K) t = ldg_32(x + (size_t)min(m0 + m, M - 1) * K + k, x32);
#pragma unroll
                for (int i = 0; i < V / 2; i++) v[i] = pack2(t.v[2 * i], t.v[2 * i + 1]);
            };
            if (MB == 1) {
#pragma unroll
                for (int u = 0; u < U * D; u++) load_row(u, 0, xr[MB == 1 ? u : 0]);
            }
#pragma unroll
            for (int u = 0; u < U * D; u++) {
                uint64_t wd[R][V / 2];
#pragma unroll
                for (int r = 0; r < R; r++) {
                    const uint64_t s2 = pack2(s[u][r], s[u][r]), b2 = pack2(b[u][r], b[u][r]);
#pragma unroll
                    for (int i = 0; i < V / 2; i++) {
                        constexpr uint32_t mask = (1u << BITS) - 1;
                        const int bit = 2 * i * BITS;
                        const uint32_t word = w[u][r][bit / 32 & (WW - 1)];
                        const uint64_t q2 = pack2((word >> bit % 32 & mask) | kBits2p23, (word >> (bit + BITS) % 32 & mask) | kBits2p23);
                        wd[r][i] = add2(mul2(s2, add2(q2, kMinus2p23x2)), b2);
                    }
                }
#pragma unroll
                for (int m = 0; m < MB; m++) {
                    uint64_t xv[V / 2];
                    if (MB > 1) load_row(u, m, xv);
#pragma unroll
                    for (int i = 0; i < V / 2; i++)
#pragma unroll
                        for (int r = 0; r < R; r++) acc[u % U][r][m] = fma2(MB > 1 ? xv[i] : xr[MB == 1 ? u : 0][i], wd[r][i], acc[u % U][r][m]);
                }
            }
        }
    }
    constexpr int C = U * R * MB, LPV = 32 / C;  // values, lanes that hold the same one
    float v[C];
#pragma unroll
    for (int u = 0; u < U; u++)
#pragma unroll
        for (int r = 0; r < R; r++)
#pragma unroll
            for (int m = 0; m < MB; m++)
                v[(u * MB + m) * R + r] = __uint_as_float((uint32_t)acc[u][r][m]) + __uint_as_float((uint32_t)(acc[u][r][m] >> 32));
    const float sum = reduce_warp<C>(v, lane);
    if (lane % LPV == 0) {
        const int j = lane / LPV, u = j / (R * MB);
        red[(warp - part) * U + part + u * kw][j % (R * MB)] = sum;  // [rows of W][part]
    }
    __syncthreads();
    for (int i = threadIdx.x; i < (kF32Warps >> kw_shift) * R * MB; i += kF32Warps * 32) {
        const int g = i / (R * MB), j = i % (R * MB), n = (blockIdx.x * (kF32Warps >> kw_shift) + g) * R + j % R, m = m0 + j / R;
        if (n >= N || m >= M) continue;
        const float(*parts)[R * MB] = red + (g << kw_shift) * U;
        float t = parts[0][j];
        for (int q = 1; q < kw * U; q++) t += parts[q][j];
        const size_t idx = (size_t)m * N + n;
        if (y_bf16) static_cast<__nv_bfloat16*>(yv)[idx] = __float2bfloat16_rn(t);
        else static_cast<float*>(yv)[idx] = t;
    }
}

template <int BITS, bool SB16, int MB, int U, int D, int BLK>
cudaError_t launch_f32_one(const QmmArgs& a, cudaStream_t stream, bool overlap_prev) {
    static_assert(U == 1 || U == 2, "parts are 2, 4 or 8");
    const int groups = (a.N + kF32Rows - 1) / kF32Rows, gy = (a.M + MB - 1) / MB, kw_shift = f32_parts(a.K) - (U == 2 ? 1 : 0);
    const int per_block = kF32Warps >> kw_shift;
    if (gy > 65535) return cudaErrorInvalidConfiguration;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((groups + per_block - 1) / per_block, gy);
    cfg.blockDim = dim3(kF32Warps * 32);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = overlap_prev ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, qmv_f32_kernel<BITS, SB16, MB, U, D, BLK>, (const float*)a.x, (const unsigned char*)a.wq,
                              (const void*)a.scales, (const void*)a.biases, (void*)a.y, a.M, a.K, a.N,
                              a.group == 32 ? 5 : (a.group == 64 ? 6 : 7), kw_shift, (int)(((uintptr_t)a.x & 31) == 0), (int)(a.y_dtype == LUX_DTYPE_BFLOAT16));
}
template <int BITS, bool SB16>
cudaError_t launch_f32(const QmmArgs& a, int sm_count, cudaStream_t stream, bool overlap_prev) {
    // How a warp goes about its parts leaves the bits alone.  K > 2048: more than one piece in each of the 8 parts, two of
    // them under way.  `full`: the launch fills the GPU twice over; then two rows of x take two parts per warp (half the
    // blocks; 2 x 2048 x 4096, 8 bit: 6.4 us, one part each 8.1) and more than four are taken eight at a time (32 x 4096 x 4096,
    // 4 bit: 77 us, four at a time 96), below it the other way round (2 x 1024 x 1024: 2.0 against 2.7; 8 x 1024 x 256: 2.4
    // against 3.6).
    const long long warps = (long long)((a.N + kF32Rows - 1) / kF32Rows) * ((a.M + 7) / 8) << f32_parts(a.K);
    const bool deep = a.K > 2048, full = warps > 16ll * sm_count;
    if (a.M == 1)
        return deep ? launch_f32_one<BITS, SB16, 1, 1, 2, 4>(a, stream, overlap_prev) : launch_f32_one<BITS, SB16, 1, 1, 1, 4>(a, stream, overlap_prev);
    if (a.M == 2)
        return full   ? launch_f32_one<BITS, SB16, 2, 2, 1, 2>(a, stream, overlap_prev)
               : deep ? launch_f32_one<BITS, SB16, 2, 1, 2, 2>(a, stream, overlap_prev)
                      : launch_f32_one<BITS, SB16, 2, 1, 1, 2>(a, stream, overlap_prev);
    return a.M <= 4 || !full ? launch_f32_one<BITS, SB16, 4, 1, 1, 2>(a, stream, overlap_prev)
                             : launch_f32_one<BITS, SB16, 8, 1, 1, 2>(a, stream, overlap_prev);
}

}  // namespace

cudaError_t launch_qmv_simt(const QmmArgs& a, int sm_count, cudaStream_t stream, const char** name, bool overlap_prev) {
    const bool xbf16 = a.x_dtype == LUX_DTYPE_BFLOAT16, sb16 = a.sb_dtype == LUX_DTYPE_BFLOAT16;
    if (name) *name = xbf16 ? (a.bits == 4 ? "qmv_simt<4,bf16>" : "qmv_simt<8,bf16>")
                            : (a.bits == 4 ? "qmv_simt<4,f32>" : "qmv_simt<8,f32>");
    if (xbf16) return a.bits == 4 ? launch_bf16<4>(a, stream) : launch_bf16<8>(a, stream);
    if (a.bits == 4) return sb16 ? launch_f32<4, true>(a, sm_count, stream, overlap_prev) : launch_f32<4, false>(a, sm_count, stream, overlap_prev);
    return sb16 ? launch_f32<8, true>(a, sm_count, stream, overlap_prev) : launch_f32<8, false>(a, sm_count, stream, overlap_prev);
}

}  // namespace luxcuda
