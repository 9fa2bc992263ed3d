// Mixed-precision factorization: the block schedule of gefa_f32 (one step of
// look-ahead) with the trailing update on the tensor cores (k_umma.cu), and
// the panel's top and left stages as tensor-core products with the inverted
// triangles of the FP32 diagonal block (panel_tc).  After each panel its left block column L and top
// block row T are rounded to the tensor-core operand type:
//   BF16:  Lq[m][k] = bf16(L[m][k]),  Tq[n][k] = bf16(T[k][n]);
//   E4M3:  one absmax scale per 512 x 512 block: per 512-row block of L and
//          512-wide K segment, per 512-column block of T and K segment
//          (s = absmax / 448), Lq = e4m3(L / s_L), Tq = e4m3(T^T / s_T), and
//          the update adds sum_seg s_L(seg) * s_T(seg) * (Lq_seg Tq_seg^T) in
//          FP32 (k_umma.cu accumulates every segment on its own).
// The FP32 factors the substitution uses are these rounded-update factors;
// accuracy is recovered by FP64 iterative refinement (lp_solve.cu).
//   BF16x6 (FP32 emulation): every element x of L and T is split exactly into
//          three BF16 terms x1 = bf16(x), x2 = bf16(x - x1), x3 = x - x1 - x2
//          (8 + 8 + 8 significant bits = the 24 of an FP32), and the operands
//          become six K-segments so that one tensor-core GEMM with K = 6 bs
//          accumulates x3 t1 + x2 t2 + x1 t3 + x2 t1 + x1 t2 + x1 t1 in FP32
//          (small terms first).  The three dropped products (x2 t3, x3 t2,
//          x3 t3) are below 2^-24 of x1 t1: the update has FP32 accuracy.
#include <cuda_bf16.h>
#include <cuda_fp8.h>

#include "lp_ctx.cuh"

namespace lp {
namespace {

constexpr float kE4M3Max = 448.0f;

__device__ __forceinline__ void atomic_max_nonneg(float* addr, float v) {
    atomicMax(reinterpret_cast<int*>(addr), __float_as_int(v));  // non-negative floats order as ints
}

// amax[seg * nblk + r / 512] = max |L[r][512 seg .. 512 seg + 512)| over each
// 512-row block (blockIdx.y = seg), a warp per row, eight rows per warp; rows a
// multiple of 128 and k of 128.
__global__ void __launch_bounds__(256) k_absmax_rows(const float* __restrict__ L, int ldl, int rows, int k, int nblk,
                                                     float* __restrict__ amax) {
    const int seg = blockIdx.y, lane = threadIdx.x & 31, r0 = (blockIdx.x * 8 + (threadIdx.x >> 5)) * 8;
    if (r0 >= rows) return;
    const int c1 = min(k, 512 * (seg + 1));
    float m = 0.0f;
    for (int c = 512 * seg + 4 * lane; c < c1; c += 128) {
        float4 v[8];
#pragma unroll
        for (int r = 0; r < 8; r++) v[r] = *reinterpret_cast<const float4*>(L + (size_t)(r0 + r) * ldl + c);
#pragma unroll
        for (int r = 0; r < 8; r++)
            m = fmaxf(m, fmaxf(fmaxf(fabsf(v[r].x), fabsf(v[r].y)), fmaxf(fabsf(v[r].z), fabsf(v[r].w))));
    }
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (lane == 0) atomic_max_nonneg(&amax[seg * nblk + (r0 >> 9)], m);
}

// amax[seg * nblk + c / 512] = max |T[512 seg .. 512 seg + 512)[c]| over each
// 512-column block: 128 columns x 64 rows per block (blockIdx.y: 64-row
// chunks, which lie in one segment), so that the 512 rows of a column are not
// one thread's chain.  cols a multiple of 4, k of 64; vec: rows allow 16-byte
// loads.
__global__ void __launch_bounds__(256) k_absmax_cols(const float* __restrict__ T, int ldt, int k, int cols, int nblk,
                                                     bool vec, float* __restrict__ amax) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, c = blockIdx.x * 128 + 4 * lane;
    const int r0 = blockIdx.y * 64 + warp * 8;
    float m = 0.0f;
    if (c < cols && r0 < k) {
        float4 v[8];
#pragma unroll
        for (int r = 0; r < 8; r++) {
            const float* p = T + (size_t)(r0 + r) * ldt + c;
            v[r] = vec ? *reinterpret_cast<const float4*>(p) : make_float4(p[0], p[1], p[2], p[3]);
        }
#pragma unroll
        for (int r = 0; r < 8; r++)
            m = fmaxf(m, fmaxf(fmaxf(fabsf(v[r].x), fabsf(v[r].y)), fmaxf(fabsf(v[r].z), fabsf(v[r].w))));
    }
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (lane == 0 && c < cols) atomic_max_nonneg(&amax[((blockIdx.y * 64) >> 9) * nblk + (c >> 9)], m);
}

// scale = amax / 448 (1 for an all-zero block); inv = 1 / scale.
__global__ void k_scales(const float* __restrict__ amax, float* __restrict__ scale, float* __restrict__ inv, int nb) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nb) return;
    const float a = amax[i];
    const float s = a > 0.0f ? a / kE4M3Max : 1.0f;
    scale[i] = s;
    inv[i] = 1.0f / s;
}

template <bool FP8>
__global__ void k_quant_rows(const float* __restrict__ L, int ldl, uint8_t* __restrict__ out, int rows, int k,
                             const float* __restrict__ inv, int nblk) {
    const size_t total = (size_t)rows * k / 4;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
        const size_t e = i * 4;
        const int r = (int)(e / k), c = (int)(e - (size_t)r * k);
        float4 v = *reinterpret_cast<const float4*>(L + (size_t)r * ldl + c);
        if (FP8) {
            const float s = inv[(c >> 9) * nblk + (r >> 9)];  // the four columns share a 512-wide K segment
            __nv_fp8x4_e4m3 q(make_float4(v.x * s, v.y * s, v.z * s, v.w * s));
            *reinterpret_cast<__nv_fp8x4_e4m3*>(out + e) = q;
        } else {
            __nv_bfloat162 lo = __floats2bfloat162_rn(v.x, v.y), hi = __floats2bfloat162_rn(v.z, v.w);
            __nv_bfloat162* o = reinterpret_cast<__nv_bfloat162*>(out + e * 2);
            o[0] = lo;
            o[1] = hi;
        }
    }
}

// out[c][r] = q(T[r][c]) for r < k, c < cols: 32 x 32 tiles through shared memory.
template <bool FP8>
__global__ void __launch_bounds__(256) k_quant_trans(const float* __restrict__ T, int ldt, uint8_t* __restrict__ out,
                                                     int k, int cols, const float* __restrict__ inv, int nblk) {
    __shared__ float tile[32][33];
    const int r0 = blockIdx.y * 32, c0 = blockIdx.x * 32;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
#pragma unroll
    for (int j = 0; j < 32; j += 8) {
        const int r = r0 + ty + j, c = c0 + tx;
        tile[ty + j][tx] = (r < k && c < cols) ? T[(size_t)r * ldt + c] : 0.0f;
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < 32; j += 8) {
        const int c = c0 + ty + j, r = r0 + tx;
        if (r < k && c < cols) {
            const float v = tile[tx][ty + j];
            if (FP8) {
                __nv_fp8_e4m3 q(v * inv[(r >> 9) * nblk + (c >> 9)]);
                out[(size_t)c * k + r] = *reinterpret_cast<uint8_t*>(&q);
            } else {
                __nv_bfloat16 q = __float2bfloat16_rn(v);
                reinterpret_cast<__nv_bfloat16*>(out)[(size_t)c * k + r] = q;
            }
        }
    }
}

// Exact three-term BF16 split of an FP32 value (each remainder is exact in FP32).
__device__ __forceinline__ void split3(float x, __nv_bfloat16& a, __nv_bfloat16& b, __nv_bfloat16& c) {
    a = __float2bfloat16_rn(x);
    const float r1 = x - __bfloat162float(a);
    b = __float2bfloat16_rn(r1);
    c = __float2bfloat16_rn(r1 - __bfloat162float(b));
}

// Segment s of the K = nseg k operand pairs L-term lterm(s) with T-term
// tterm(s) (term 0 = x1, the largest).  nseg 6: x3 t1 + x2 t2 + x1 t3 +
// x2 t1 + x1 t2 + x1 t1 (FP32 accuracy); nseg 3: x2 t1 + x1 t2 + x1 t1
// (about 2^-16 relative, the three-term split's first two terms); nseg 1:
// x1 t1 (plain BF16 operands).
template <int NSEG>
__host__ __device__ constexpr int lterm(int s) {
    return NSEG == 6 ? (s == 0 ? 2 : (s == 1 || s == 3) ? 1 : 0) : NSEG == 3 ? (s == 0 ? 1 : 0) : 0;
}
template <int NSEG>
__host__ __device__ constexpr int tterm(int s) {
    return NSEG == 6 ? (s == 2 ? 2 : (s == 1 || s == 4) ? 1 : 0) : NSEG == 3 ? (s == 1 ? 1 : 0) : 0;
}

// out[r][s*k + c] = term lterm(s) of L[r][c]: rows x (NSEG k) BF16.
template <int NSEG>
__global__ void k_split_rows(const float* __restrict__ L, int ldl, __nv_bfloat16* __restrict__ out, int rows, int k) {
    const size_t total = (size_t)rows * k;
    const size_t kq = NSEG * (size_t)k;
    for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < total; e += (size_t)gridDim.x * blockDim.x) {
        const int r = (int)(e / k), c = (int)(e - (size_t)r * k);
        __nv_bfloat16 t[3];
        split3(L[(size_t)r * ldl + c], t[0], t[1], t[2]);
        __nv_bfloat16* o = out + (size_t)r * kq + c;
#pragma unroll
        for (int s = 0; s < NSEG; s++) o[(size_t)s * k] = t[lterm<NSEG>(s)];
    }
}

// out[c][s*k + r] = term tterm(s) of T[r][c] (EYE: of T - I): cols x (NSEG k)
// BF16, through a 32 x 32 shared-memory transpose.
template <int NSEG, bool EYE>
__global__ void __launch_bounds__(256) k_split_trans(const float* __restrict__ T, int ldt,
                                                     __nv_bfloat16* __restrict__ out, int k, int cols) {
    __shared__ float tile[32][33];
    const int r0 = blockIdx.y * 32, c0 = blockIdx.x * 32;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
#pragma unroll
    for (int j = 0; j < 32; j += 8) {
        const int r = r0 + ty + j, c = c0 + tx;
        tile[ty + j][tx] = (r < k && c < cols) ? T[(size_t)r * ldt + c] : 0.0f;
    }
    __syncthreads();
    const size_t kq = NSEG * (size_t)k;
#pragma unroll
    for (int j = 0; j < 32; j += 8) {
        const int c = c0 + ty + j, r = r0 + tx;
        if (r < k && c < cols) {
            __nv_bfloat16 t[3];
            split3(EYE && r == c ? tile[tx][ty + j] - 1.0f : tile[tx][ty + j], t[0], t[1], t[2]);
            __nv_bfloat16* o = out + (size_t)c * kq + r;
#pragma unroll
            for (int s = 0; s < NSEG; s++) o[(size_t)s * k] = t[tterm<NSEG>(s)];
        }
    }
}

// x = identity (two n x n blocks, leading dimension n).
__global__ void k_eye2(float* __restrict__ x, float* __restrict__ y, int n) {
    const size_t total = (size_t)n * n;
    for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < total; e += (size_t)gridDim.x * blockDim.x) {
        const float v = (e / n == e % n) ? 1.0f : 0.0f;
        x[e] = v;
        y[e] = v;
    }
}

}  // namespace

// The split-BF16 operands of a product (nseg 6, 3 or 1 K-segments): aq, rows x
// nseg k, from L (rows x k).
static int split_rows(const float* L, int ldl, int rows, int k, __nv_bfloat16* a, cudaStream_t st, int nseg) {
    if (rows <= 0) return LP_OK;
    const size_t total = (size_t)rows * k;
    const int grid = (int)((total + 255) / 256 < 4736 ? (total + 255) / 256 : 4736);
    if (nseg == 6)
        k_split_rows<6><<<grid, 256, 0, st>>>(L, ldl, a, rows, k);
    else if (nseg == 3)
        k_split_rows<3><<<grid, 256, 0, st>>>(L, ldl, a, rows, k);
    else if (nseg == 1)
        k_split_rows<1><<<grid, 256, 0, st>>>(L, ldl, a, rows, k);
    else
        return fail(LP_E_INVALID, "split operands: 1, 3 or 6 segments");
    count_launch();
    LP_CUDA(cudaGetLastError());
    return LP_OK;
}

// bq, cols x nseg k, from T (k x cols), or from T - I (eye).
static int split_trans(const float* T, int ldt, int cols, int k, __nv_bfloat16* b, cudaStream_t st, int nseg,
                       bool eye = false) {
    if (cols <= 0) return LP_OK;
    const dim3 grid((cols + 31) / 32, (k + 31) / 32);
    if (nseg == 6 && eye)
        k_split_trans<6, true><<<grid, 256, 0, st>>>(T, ldt, b, k, cols);
    else if (nseg == 6)
        k_split_trans<6, false><<<grid, 256, 0, st>>>(T, ldt, b, k, cols);
    else if (nseg == 3 && eye)
        k_split_trans<3, true><<<grid, 256, 0, st>>>(T, ldt, b, k, cols);
    else if (nseg == 3)
        k_split_trans<3, false><<<grid, 256, 0, st>>>(T, ldt, b, k, cols);
    else if (nseg == 1 && eye)
        k_split_trans<1, true><<<grid, 256, 0, st>>>(T, ldt, b, k, cols);
    else if (nseg == 1)
        k_split_trans<1, false><<<grid, 256, 0, st>>>(T, ldt, b, k, cols);
    else
        return fail(LP_E_INVALID, "split operands: 1, 3 or 6 segments");
    count_launch();
    LP_CUDA(cudaGetLastError());
    return LP_OK;
}

// The left panel L (rows x k, ld ldl) rounded to the tensor-core operand type:
// aq, rows x k.  E4M3: sc holds kseg(k) * nblk block maxima, then the scales,
// then their reciprocals, indexed seg * nblk + block.  rows and k multiples of
// 128.
static int quantize_left(const float* L, int ldl, int rows, int k, bool fp8, uint8_t* aq, float* sc, int nblk,
                         cudaStream_t st) {
    if (rows <= 0) return LP_OK;
    const size_t q4 = (size_t)rows * k / 4;
    const int grid = (int)((q4 + 255) / 256 < 2368 ? (q4 + 255) / 256 : 2368);
    if (fp8) {
        const int ns = kseg(k) * nblk;
        LP_CUDA(cudaMemsetAsync(sc, 0, sizeof(float) * ns, st));
        k_absmax_rows<<<dim3((rows + 63) / 64, kseg(k)), 256, 0, st>>>(L, ldl, rows, k, nblk, sc);
        k_scales<<<(ns + 127) / 128, 128, 0, st>>>(sc, sc + ns, sc + 2 * ns, ns);
        k_quant_rows<true><<<grid, 256, 0, st>>>(L, ldl, aq, rows, k, sc + 2 * ns, nblk);
        count_launch(3);
    } else {
        k_quant_rows<false><<<grid, 256, 0, st>>>(L, ldl, aq, rows, k, nullptr, nblk);
        count_launch();
    }
    LP_CUDA(cudaGetLastError());
    return LP_OK;
}

// The same for the top panel T (k x cols, ld ldt), transposed: bq, cols x k.
static int quantize_top(const float* T, int ldt, int cols, int k, bool fp8, uint8_t* bq, float* sc, int nblk,
                        cudaStream_t st) {
    if (cols <= 0) return LP_OK;
    const dim3 grid((cols + 31) / 32, (k + 31) / 32);
    if (fp8) {
        const int ns = kseg(k) * nblk;
        LP_CUDA(cudaMemsetAsync(sc, 0, sizeof(float) * ns, st));
        k_absmax_cols<<<dim3((cols + 127) / 128, (k + 63) / 64), 256, 0, st>>>(T, ldt, k, cols, nblk,
                                                                                   ldt % 4 == 0 && aligned16(T), sc);
        k_scales<<<(ns + 127) / 128, 128, 0, st>>>(sc, sc + ns, sc + 2 * ns, ns);
        k_quant_trans<true><<<grid, 256, 0, st>>>(T, ldt, bq, k, cols, sc + 2 * ns, nblk);
        count_launch(3);
    } else {
        k_quant_trans<false><<<grid, 256, 0, st>>>(T, ldt, bq, k, cols, nullptr, nblk);
        count_launch();
    }
    LP_CUDA(cudaGetLastError());
    return LP_OK;
}

// Both panels; sc: the left panel's three arrays of kseg(k) * nblk floats, then
// the top panel's (nblk >= ceil(max(rows_l, cols_t) / 512)).
int quantize_panel(const float* L, int ldl, const float* T, int ldt, int rows_l, int cols_t, int k, bool fp8,
                   uint8_t* aq, uint8_t* bq, float* sc, int nblk, cudaStream_t st) {
    if (rows_l <= 0 || cols_t <= 0) return LP_OK;
    LP_CHECK(quantize_left(L, ldl, rows_l, k, fp8, aq, sc, nblk, st));
    return quantize_top(T, ldt, cols_t, k, fp8, bq, sc + 3 * (size_t)kseg(k) * nblk, nblk, st);
}

// One trailing (sub)update of the mixed schedule: rows [m_off, m_off+m) and
// columns [n_off, n_off+n) of the trailing matrix at c11.
static int mixed_update(lp_ctx* c, float* c11, int lda, const uint8_t* aq, const uint8_t* bq, int rest, int m_off,
                        int n_off, int m, int n, int kq, bool fp8, const float* sc, int nblk, cudaStream_t st) {
    const int ns = kseg(kq) * nblk;
    const float* scale_a = fp8 ? sc + ns : nullptr;
    const float* scale_b = fp8 ? sc + 4 * ns : nullptr;
    return launch_umma_update(c11, lda, aq, rest, bq, rest, m_off, n_off, m, n, kq, fp8, scale_a, scale_b, nblk,
                              static_cast<int*>(c->err.ptr), st);
}

// Panel of block step K for the tensor-core schedules.  lu of the diagonal
// block D as in the FP32 schedule.  top and left are triangular solves with
// D's two triangles (storage indices, k_trsm.cu):
//   top:  each column t of the block row satisfies t_k = D_kk (t0_k + sum_{i<k} D_ki t_i),
//         i.e. t = W^-1 t0 with W = diag(D)^-1 - strict-lower(D);
//   left: each row l of the block column satisfies l_i = l0_i + sum_{k<i} l_k D_ki,
//         i.e. l = l0 V with V = (I - strict-upper(D))^-1.
// W^-1 and V are the two recurrences applied to a bs x bs identity (the exact
// kernels over the nonzero triangle only, a small problem); then T = W^-1 T0
// (into the zeroed block row) and
// L += L (V - I) run as split-BF16 tensor-core products (nseg K-segments), so
// the n bs^2 flops of the recurrences per step leave the FMA pipe.  V is unit
// triangular, so L keeps its exact identity part; W^-1 is not (its diagonal
// is D_kk = -1/u_kk), and T0 + (W^-1 - I) T0 would cancel nearly all of T0.
// What reads only the panel's input -- the operands T0 and L0, and clearing the
// block row -- runs on aux2 beside the lu stage; the rounded copies q for the
// trailing update run beside the other half's product.
struct PanelOut {
    int fp8, x6;         // operand type of the trailing update (neither: BF16)
    uint8_t *aq, *bq;    // left and top operands
    float* sc;           // E4M3 scales
    int nblk;
};
static int panel_tc(lp_ctx* c, float* dA, int n, int lda, int bs, int K, int nseg, const PanelOut& q, cudaStream_t s) {
    float* d = dA + (size_t)K * bs * lda + (size_t)K * bs;
    const double b = bs;
    const int rest = n - (K + 1) * bs;  // <= 0: the last block, of n - K bs
    const size_t bb = (size_t)bs * bs, kq = (size_t)nseg * bs;
    float* winv = static_cast<float*>(c->tri.ptr);
    float* vinv = winv + bb;
    float* vlt = vinv + bb;
    float* t = d + bs;
    float* l = d + (size_t)bs * lda;
    __nv_bfloat16* a_top = static_cast<__nv_bfloat16*>(c->tq.ptr);  // bs x kq: W^-1
    __nv_bfloat16* b_left = a_top + bb * nseg;                      // bs x kq: (V - I)^T
    __nv_bfloat16* b_top = b_left + bb * nseg;                      // rest x kq: T^T
    __nv_bfloat16* a_left = b_top + (size_t)n * kq;                 // rest x kq: L
    // bs > 128: W^-1 and V are built 128 rows / columns behind the lu stage on
    // two side streams (lu_stage), rather than after it.  Measured on one B200,
    // factorization alone, after it -> beside it: BF16 n = 32768, block 1024
    // 55.3 -> 51.5 ms, E4M3 59.3 -> 54.5 ms; emulated FP32 (six segments)
    // n = 2048, block 512 1.15 -> 1.01 ms, n = 8192, block 512 6.70 -> 6.00 ms,
    // n = 16384, block 1024 22.6 -> 21.4 ms, n = 32768, block 1024 equal.
    const bool beside = rest > 0 && bs > 128;
    if (rest > 0) {
        LP_CUDA(cudaEventRecord(c->ev_side, s));
        LP_CUDA(cudaStreamWaitEvent(c->aux2, c->ev_side, 0));
        LP_CHECK(split_trans(t, lda, rest, bs, b_top, c->aux2, nseg));
        LP_CUDA(cudaMemset2DAsync(t, sizeof(float) * (size_t)lda, 0, sizeof(float) * (size_t)rest, bs, c->aux2));
        LP_CHECK(split_rows(l, lda, rest, bs, a_left, c->aux2, nseg));
        LP_CUDA(cudaEventRecord(c->ev_side_done, c->aux2));
        k_eye2<<<(int)((bb + 255) / 256 < 1184 ? (bb + 255) / 256 : 1184), 256, 0, s>>>(winv, vinv, bs);
        count_launch();
        LP_CUDA(cudaGetLastError());
    }
    const TriInverses inv{winv, vinv, vlt};
    int e = prof_begin(c, s);
    const int kb = std::min(bs, n - K * bs);
    LP_CHECK(lu_stage(c, d, lda, kb, s, beside ? &inv : nullptr));
    LP_CHECK(prof_end(c, s, LP_STAGE_LU, e, 2.0 * kb * kb * (double)kb / 3.0, 8.0 * kb * (double)kb));
    if (rest <= 0) return LP_OK;
    const double r = rest;
    int* err = static_cast<int*>(c->err.ptr);

    e = prof_begin(c, s);
    if (!beside)  // one chunk: the two recurrences in one launch
        LP_CHECK(launch_tl(d, lda, static_cast<const float*>(c->dt.ptr), bs, bs, winv, bs, bs, vinv, bs, bs, vlt, bs,
                           c->num_sms, s));
    LP_CHECK(split_rows(winv, bs, bs, bs, a_top, s, nseg));
    LP_CHECK(split_trans(vinv, bs, bs, bs, b_left, s, nseg, true));
    LP_CUDA(cudaStreamWaitEvent(s, c->ev_side_done, 0));
    LP_CHECK(launch_umma_update(t, lda, a_top, bs, b_top, rest, 0, 0, bs, rest, (int)kq, false, nullptr, nullptr, 0,
                                err, s));
    LP_CHECK(prof_end(c, s, LP_STAGE_TOP, e, b * b * r, 8.0 * b * r));
    LP_CUDA(cudaEventRecord(c->ev_side, s));
    LP_CUDA(cudaStreamWaitEvent(c->aux2, c->ev_side, 0));
    if (q.x6)
        LP_CHECK(split_trans(t, lda, rest, bs, reinterpret_cast<__nv_bfloat16*>(q.bq), c->aux2, 6));
    else
        LP_CHECK(quantize_top(t, lda, rest, bs, q.fp8 != 0, q.bq, q.sc + 3 * (size_t)kseg(bs) * q.nblk, q.nblk, c->aux2));
    LP_CUDA(cudaEventRecord(c->ev_side_done, c->aux2));
    e = prof_begin(c, s);
    LP_CHECK(launch_umma_update(l, lda, a_left, rest, b_left, bs, 0, 0, rest, bs, (int)kq, false, nullptr, nullptr, 0,
                                err, s));
    LP_CHECK(prof_end(c, s, LP_STAGE_LEFT, e, b * b * r, 8.0 * b * r));
    e = prof_begin(c, s);
    if (q.x6)
        LP_CHECK(split_rows(l, lda, rest, bs, reinterpret_cast<__nv_bfloat16*>(q.aq), s, 6));
    else
        LP_CHECK(quantize_left(l, lda, rest, bs, q.fp8 != 0, q.aq, q.sc, q.nblk, s));
    LP_CUDA(cudaStreamWaitEvent(s, c->ev_side_done, 0));
    const double esz = q.fp8 ? 1.0 : 2.0;
    return prof_end(c, s, LP_STAGE_OTHER, e, 0.0, 2.0 * 4.0 * b * rest + 2.0 * esz * b * rest);
}

// Inner block of the emulated-FP32 form, and of BF16 from order 4096 on: 1024,
// or the caller's if larger (the last block may be smaller).  Wide blocks read
// and write the FP32 trailing matrix less often and give the update a longer
// K; the chain of the 128-wide inner blocks is as long either way.  A matrix
// of one block is the FP32 lu stage alone.  E4M3 and small BF16 matrices keep
// the caller's block: what a wide block computes in FP32 instead of in rounded
// operands moves their factors by more than FP32 accuracy (E4M3, n = 12288:
// 6e-5 relative to the factors' norm; BF16 2e-5 at n = 2048, 1e-5 at 4096, 5e-6 at 12288).
// Measured on one B200, factorization alone in ms, blocks of 128 / 512 / 1024:
//   BF16          n = 4096 2.36 / 1.60 / 1.55   n = 8192 6.05 / 3.72 / 3.59   n = 32768 217 / 63.2 / 43.2
//   emulated FP32 n = 3072 2.18 / 1.37 / 1.29   n = 8192 6.80 / 4.63 / 4.70   n = 32768 270 / 145 / 141
// (Between 6144 and 16384 a block of 512 would be 1 to 5 % faster for the emulated
// form, n = 16384 19.8 against 20.7: one line for all its orders was drawn when
// the chain was longer.)
constexpr int kMixedBlock = 1024;

// Workspaces for blocks of up to bs; where one of them cannot be allocated, all
// of them are given back.
static int mixed_ensure(lp_ctx* c, int precision, int n, int bs, int nseg) {
    const size_t esz = precision == LP_FP8_IR ? 1 : 2, kq = precision == LP_F32_BF16X6 ? 6 * (size_t)bs : bs;
    const size_t nblk = (n + 511) / 512, b = bs;
    const struct { Workspace* w; size_t bytes; } need[] = {
        {&c->dt, sizeof(float) * b * b},
        {&c->q, 4 * esz * kq * n},
        {&c->qs, 2 * 6 * sizeof(float) * (size_t)kseg(bs) * nblk},
        {&c->err, sizeof(int)},
        {&c->tri, 3 * sizeof(float) * b * b},
        {&c->tq, 2 * sizeof(__nv_bfloat16) * (size_t)nseg * b * (b + n)}};
    for (const auto& x : need) {
        const int status = x.w->ensure(x.bytes);
        if (status == LP_OK) continue;
        for (const auto& y : need) y.w->release();
        return status;
    }
    return LP_OK;
}

int gefa_mixed(lp_ctx* c, int precision, float* dA, int n, int lda, int user_bs, cudaStream_t st) {
    const bool fp8 = precision == LP_FP8_IR;
    const bool x6 = precision == LP_F32_BF16X6;
    if (user_bs < 128 || user_bs % 128 != 0) return fail(LP_E_INVALID, "mixed precision needs a block size >= 128");
    // the top / left products: FP32 accuracy (six segments) for the emulated-FP32
    // form.  For BF16 / E4M3 (the panel is rounded to them for the update anyway)
    // three segments, and plain BF16 operands from block 2048 on, where the panel
    // chain is the critical path: the products cost about 9 bs / n of the update's
    // flops per three segments.  Measured on one B200 (BF16+IR): n = 65536, block
    // 2048: 582 -> 638 TFLOP/s, one refinement either way; n = 32768, block 1024: no
    // gain, the plainer factors needing a second refinement.
    const int nseg = x6 ? 6 : user_bs >= 2048 ? 1 : 3;
    // the wide block; only where its workspaces cannot be allocated, the caller's
    int bs = x6 || (!fp8 && n >= 4096) ? std::max(kMixedBlock, user_bs) : user_bs;
    int status = mixed_ensure(c, precision, n, bs, nseg);
    if (status == LP_E_NOMEM && bs > user_bs) {
        cudaGetLastError();
        bs = user_bs;
        status = mixed_ensure(c, precision, n, bs, nseg);
    }
    if (status != LP_OK) return status;
    const size_t esz = fp8 ? 1 : 2;
    const int kq = x6 ? 6 * bs : bs;    // K of the tensor-core update
    const size_t pan = (size_t)kq * n;  // one tensor-core operand
    const int nblk = (n + 511) / 512;
    LP_CUDA(cudaMemsetAsync(c->err.ptr, 0, sizeof(int), st));
    uint8_t* q = static_cast<uint8_t*>(c->q.ptr);
    uint8_t* aqb[2] = {q, q + 2 * esz * pan};
    uint8_t* bqb[2] = {q + esz * pan, q + 3 * esz * pan};
    float* scb[2] = {static_cast<float*>(c->qs.ptr), static_cast<float*>(c->qs.ptr) + 6 * (size_t)kseg(bs) * nblk};
    const int nb = (n + bs - 1) / bs;
    const double b = bs;

    auto panel_q = [&](int K, cudaStream_t s) -> int {
        return panel_tc(c, dA, n, lda, bs, K, nseg, PanelOut{fp8, x6, aqb[K & 1], bqb[K & 1], scb[K & 1], nblk}, s);
    };
    cudaStream_t aux = c->aux;
    LP_CUDA(cudaEventRecord(c->ev_fork, st));
    LP_CUDA(cudaStreamWaitEvent(aux, c->ev_fork, 0));
    LP_CHECK(panel_q(0, aux));
    for (int K = 0; K + 1 < nb; K++) {  // streams as in gefa_f32
        const int rest = n - (K + 1) * bs, nx = std::min(bs, rest);  // nx: the next block
        const double r = rest, x = nx;
        float* c11 = dA + (size_t)(K + 1) * bs * lda + (size_t)(K + 1) * bs;
        const uint8_t* aq = aqb[K & 1];
        const uint8_t* bq = bqb[K & 1];
        const float* sc = scb[K & 1];
        if (K > 0) LP_CUDA(cudaStreamWaitEvent(aux, c->ev_join, 0));  // U_b of the last step
        int e = 0;
        if (rest > bs) {
            // the block column: the panel reads it first on aux2 (split_rows), so from here down it runs
            // there, beside the block row and lu; above, where each part fills the chip, the update of the
            // rest bounds the step (n = 32768, block 1024: 44.7 ms against 43.7 with every step so;
            // n = 12288, block 512: E4M3 7.28 -> 7.00, BF16 6.68 -> 6.55 ms)
            cudaStream_t s = rest <= 12288 ? c->aux2 : aux;
            if (s != aux) {
                LP_CUDA(cudaEventRecord(c->ev_side, aux));
                LP_CUDA(cudaStreamWaitEvent(s, c->ev_side, 0));
            }
            e = prof_begin(c, s);
            LP_CHECK(mixed_update(c, c11, lda, aq, bq, rest, bs, 0, rest - bs, bs, kq, fp8, sc, nblk, s));
            LP_CHECK(prof_end(c, s, LP_STAGE_INNER, e, 2.0 * (r - x) * x * b, 8.0 * (r - x) * x));
        }
        e = prof_begin(c, aux);
        LP_CHECK(mixed_update(c, c11, lda, aq, bq, rest, 0, 0, nx, rest, kq, fp8, sc, nblk, aux));
        LP_CHECK(prof_end(c, aux, LP_STAGE_INNER, e, 2.0 * x * r * b, 8.0 * x * r));
        if (rest > bs) {
            LP_CUDA(cudaEventRecord(c->ev_fork, aux));
            LP_CUDA(cudaStreamWaitEvent(st, c->ev_fork, 0));
            const double r2 = rest - bs;
            e = prof_begin(c, st);
            LP_CHECK(mixed_update(c, c11, lda, aq, bq, rest, bs, bs, rest - bs, rest - bs, kq, fp8, sc, nblk, st));
            LP_CHECK(prof_end(c, st, LP_STAGE_INNER, e, 2.0 * r2 * r2 * b, 8.0 * r2 * r2));
            LP_CUDA(cudaEventRecord(c->ev_join, st));
        }
        LP_CHECK(panel_q(K + 1, aux));
    }
    LP_CUDA(cudaEventRecord(c->ev_fork, aux));
    LP_CUDA(cudaStreamWaitEvent(st, c->ev_fork, 0));
    int herr = 0;
    LP_CHECK(read_status(c, c->err.ptr, st, &herr));
    if (herr != 0)
        return fail(LP_E_TIMEOUT, "tensor-core trailing update: a bounded wait expired (code " +
                                      std::to_string(herr) + "); the update was abandoned");
    return LP_OK;
}

}  // namespace lp
