// Batched factor + solve of many independent systems in ONE persistent launch.
//
// Each system i is an n_i x n_i matrix in the reference encoding
// (LINPACK/src/host/linpack_data.cpp:166-229: factored in place, diagonal
// -1/u_kk, negated multipliers in storage rows, U in storage columns) with
// nrhs_i right-hand sides stored as rows of B_i, overwritten by the
// solutions.  CTAs pull systems from an atomic counter over a list sorted by
// decreasing n (largest first: the slowest systems start first, the small
// ones fill the tail), so one launch balances any size mix.
//
// Per system, one CTA of 256 threads, two CTAs per SM (128 threads with 8 x 16
// outputs each in the update tiles were slower: 21.0 against 16.2 ms for 4096
// systems of 32 .. 1024; the other phases want the threads).
//   n <= small_n_max (<= 128): the whole matrix and right-hand sides in
//     shared memory; right-looking LU with one barrier per step, then the
//     forward and back sweeps, one warp per right-hand side (n = 96: 154 -> 89
//     us a system).
//   larger n: blocked LU with panel width NB (16 or 32, per size bucket, chosen
//     by the autotuner) inside outer blocks of 128: the diagonal block factored
//     by one warp in registers (pivots and columns by shuffles); the top block
//     row (column-independent) and left block column (row-independent) by
//     their recurrences in registers, two columns or rows per thread; updates
//     in tiles whose operands are copied in with cp.async one chunk ahead.
//     (Panel widths 16 and 32 keep a recurrence in registers.)
//     Then blocked forward/back sweeps with the right-hand sides resident in
//     shared memory and each diagonal block staged before its sequential solve.
// Arithmetic uses fused multiply-add: results agree with the reference to
// rounding (checked against the oracle in tests/test_gpu_batch.py).
#include <cuda_bf16.h>
#include <cfloat>
#include <type_traits>

#include "lp_ctx.cuh"

namespace lp {
namespace {

constexpr int BT = 256;
constexpr int SMALL_MAX = 128;
constexpr int RHS_MAX = 16;
constexpr int NBUCKETS = 5;
// Flag in BatchSys::nrhs (server use only; the public entry points accept
// nrhs <= 16): the matrix already holds its factors, solve only.
constexpr int kSolveOnly = kBatchSolveOnly;

struct BatchSys {
    int n, nrhs, lda, ldb;
    long long a_off, b_off;
};
static_assert(sizeof(BatchSys) == sizeof(lp_system), "lp_system layout");

struct Tune {
    int small_n_max;
    int nb[NBUCKETS];
    int absolute;  // a_off / b_off are device addresses (bytes), not offsets into A / B
};

constexpr int kSolveBlk = 64, kSolveDL = kSolveBlk + 1;
constexpr size_t kSmallFloats = (size_t)SMALL_MAX * (SMALL_MAX + 1) + (size_t)RHS_MAX * SMALL_MAX;
// right-hand sides of n <= 1024 in the solve phase and two diagonal blocks
constexpr size_t kSolveFloats = (size_t)RHS_MAX * 1024 + 2 * kSolveBlk * kSolveDL;
// trailing_rows: a 128 x 128 piece of L and four 16 x 128 chunks of T
constexpr size_t kFactorFloats = (128 + 4 * 16) * 132;
constexpr size_t kBatchFloats = kFactorFloats > kSolveFloats ? (kFactorFloats > kSmallFloats ? kFactorFloats : kSmallFloats)
                                                             : (kSolveFloats > kSmallFloats ? kSolveFloats : kSmallFloats);
constexpr size_t kBatchSmem = sizeof(float) * kBatchFloats;  // 99 KiB: two CTAs per SM
static_assert(2 * 32 * (132 + 36) <= kFactorFloats, "update_tile smem");
// refine_system: x and the products (4 right-hand sides per unknown), the column sums, the norms' scratch
static_assert(sizeof(double) * (4 * 1024 + 4 * 1024 + 1024 + 32) <= kBatchSmem, "refinement smem");

__device__ __forceinline__ int bucket_of(int n) {
    return n <= 64 ? 0 : n <= 128 ? 1 : n <= 256 ? 2 : n <= 512 ? 3 : 4;
}

// In-place LU (reference encoding) of an m x m matrix in shared memory with
// row stride ld, all threads of the CTA; one barrier per step.  -1/pivot
// correctly rounded in float (equal to the double quotient rounded to float).
__device__ void smem_lu(float* S, int ld, int m) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    float inv_prev = 0.0f;
    for (int k = 0; k < m; k++) {
        const float inv = -__frcp_rn(S[k * ld + k]);
        if (k > 0) {
            float* rp = S + (k - 1) * ld;
            for (int i = k + tid; i < m; i += BT) rp[i] *= inv_prev;
            if (tid == 0) rp[k - 1] = inv_prev;
        }
        const float* rk = S + k * ld;
        for (int i0 = k + 1; i0 < m; i0 += 32) {
            const int i = i0 + lane;
            const bool on = i < m;
            const float sc = on ? rk[i] * inv : 0.0f;
            for (int j = k + 1 + warp; j < m; j += 4 * (BT / 32)) {  // four rows' loads before their stores
                float l[4], v[4];
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    const int jj = j + u * (BT / 32);
                    l[u] = jj < m ? S[jj * ld + k] : 0.0f;
                    v[u] = jj < m && on ? S[jj * ld + i] : 0.0f;
                }
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    const int jj = j + u * (BT / 32);
                    if (jj < m && on) S[jj * ld + i] = fmaf(sc, l[u], v[u]);
                }
            }
        }
        inv_prev = inv;
        __syncthreads();
    }
    if (tid == 0 && m > 0) S[(m - 1) * ld + (m - 1)] = inv_prev;
    __syncthreads();
}

// Forward/back sweeps on right-hand sides Y (nrhs rows of length m, stride m,
// m <= 128) with the factors in shared memory (row stride ld): one warp per
// right-hand side, its values in the lanes' registers, pivots by shuffle.
__device__ void smem_solve(const float* S, int ld, int m, float* Y, int nrhs) {
    constexpr int Q = SMALL_MAX / 32;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int q = warp; q < nrhs; q += BT / 32) {
        float* y = Y + q * m;
        float v[Q];
#pragma unroll
        for (int e = 0; e < Q; e++) v[e] = lane + 32 * e < m ? y[lane + 32 * e] : 0.0f;
#pragma unroll
        for (int e0 = 0; e0 < Q; e0++)
            for (int kk = 0; kk < min(32, m - 32 * e0); kk++) {  // y_i += y_k S[k][i] (i > k)
                const int k = 32 * e0 + kk;
                const float yk = __shfl_sync(0xffffffffu, v[e0], kk);
#pragma unroll
                for (int e = e0; e < Q; e++) {
                    const int i = lane + 32 * e;
                    if (i > k && i < m) v[e] = fmaf(yk, S[k * ld + i], v[e]);
                }
            }
#pragma unroll
        for (int e0 = Q - 1; e0 >= 0; e0--)
            for (int kk = min(32, m - 32 * e0) - 1; kk >= 0; kk--) {  // s = y_k S[k][k]; x_k = -s; y_i += s S[k][i] (i < k)
                const int k = 32 * e0 + kk;
                const float sk = __shfl_sync(0xffffffffu, v[e0], kk) * S[k * ld + k];
                if (lane == kk) v[e0] = -sk;
#pragma unroll
                for (int e = 0; e <= e0; e++) {
                    const int i = lane + 32 * e;
                    if (i < k) v[e] = fmaf(sk, S[k * ld + i], v[e]);
                }
            }
#pragma unroll
        for (int e = 0; e < Q; e++)
            if (lane + 32 * e < m) y[lane + 32 * e] = v[e];
    }
    __syncthreads();
}

__device__ __noinline__ void solve_small(float* a, int lda, int n, float* b, int ldb, int nrhs, bool factor, float* sm) {
    const int ld = n | 1;  // odd stride: column reads hit distinct banks
    float* S = sm;
    float* Y = sm + SMALL_MAX * (SMALL_MAX + 1);
    for (int idx = threadIdx.x; idx < n * n; idx += BT) {
        const int r = idx / n, c = idx - r * n;
        S[r * ld + c] = a[(size_t)r * lda + c];
    }
    for (int idx = threadIdx.x; idx < nrhs * n; idx += BT) {
        const int q = idx / n, i = idx - q * n;
        Y[idx] = b[(size_t)q * ldb + i];
    }
    __syncthreads();
    if (factor) smem_lu(S, ld, n);
    smem_solve(S, ld, n, Y, nrhs);
    if (factor)
        for (int idx = threadIdx.x; idx < n * n; idx += BT) {
            const int r = idx / n, c = idx - r * n;
            a[(size_t)r * lda + c] = S[r * ld + c];
        }
    for (int idx = threadIdx.x; idx < nrhs * n; idx += BT) {
        const int q = idx / n, i = idx - q * n;
        b[(size_t)q * ldb + i] = Y[idx];
    }
    __syncthreads();
}

// LU of the kb x kb diagonal block at d (kb <= NB), warp 0 only: lane c
// holds column c in registers, the pivot and column k are shuffled from lane
// k.  Writes the factors to d, to Ds (row stride DL) and
// transposed to Dt.  Out of line: inlined
// into the persistent loop its register array is not fully unrolled.
template <int NB, int DL>
__device__ __noinline__ void warp_diag_lu(float* d, int lda, int kb, float* Ds, float* Dt) {
    // A partial last block is padded with the identity: diag(D, I) factors as
    // diag(LU_D, I), so every step runs unconditionally (no per-step branches
    // between the shuffles) and only the kb x kb part is written back.
    const int lane = threadIdx.x & 31;
    float x[NB];
#pragma unroll
    for (int j = 0; j < NB; j++)
        x[j] = (lane < kb && j < kb) ? d[(size_t)j * lda + lane] : (j == lane ? 1.0f : 0.0f);
#pragma unroll
    for (int k = 0; k < NB; k++) {
        // -1/pivot correctly rounded in float (equal to the double quotient rounded to float)
        const float inv = -__frcp_rn(__shfl_sync(0xffffffffu, x[k], k));
        if (lane > k)
            x[k] *= inv;
        else if (lane == k)
            x[k] = inv;
#pragma unroll
        for (int j = k + 1; j < NB; j++) {
            const float sjk = __shfl_sync(0xffffffffu, x[j], k);
            if (lane > k) x[j] = fmaf(x[k], sjk, x[j]);
        }
    }
    if (lane < NB) {
#pragma unroll
        for (int j = 0; j < NB; j++) {
            Ds[j * DL + lane] = x[j];
            Dt[lane * DL + j] = x[j];
            if (lane < kb && j < kb) d[(size_t)j * lda + lane] = x[j];
        }
    }
}

// Two floats rounded to BF16 (round to nearest even) in one register, the
// first in the low half: the operand order of the warp-level MMA fragments.
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&v);
}

// D (16 x 8, FP32) += A (16 x 16, BF16, row-major fragments) * B (16 x 8, BF16).
__device__ __forceinline__ void mma_bf16_16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                               uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// C rows r .. r+3, Q groups of four columns c + cs q (columns below cend, rows
// below rend) += add(i, q).  Every load is in flight before the first store
// (the compiler keeps a load behind a store to the same array).
template <int Q, typename F>
__device__ __forceinline__ void add_quads(float* a, int lda, int cend, int rend, int r, int c, int cs, bool vec, F add) {
    float4 v[4][Q];
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int q = 0; q < Q; q++) {
            const int cc = c + cs * q;
            const float* p = a + (size_t)(r + i) * lda + cc;
            v[i][q] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (r + i < rend) {
                if (vec && cc + 3 < cend) {
                    v[i][q] = *reinterpret_cast<const float4*>(p);
                } else {
                    if (cc < cend) v[i][q].x = p[0];
                    if (cc + 1 < cend) v[i][q].y = p[1];
                    if (cc + 2 < cend) v[i][q].z = p[2];
                    if (cc + 3 < cend) v[i][q].w = p[3];
                }
            }
        }
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int q = 0; q < Q; q++) {
            const int cc = c + cs * q;
            if (r + i >= rend) continue;
            float* p = a + (size_t)(r + i) * lda + cc;
            const float4 w = add(i, q);
            const float4 u = make_float4(v[i][q].x + w.x, v[i][q].y + w.y, v[i][q].z + w.z, v[i][q].w + w.w);
            if (vec && cc + 3 < cend) {
                *reinterpret_cast<float4*>(p) = u;
            } else {
                if (cc < cend) p[0] = u.x;
                if (cc + 1 < cend) p[1] = u.y;
                if (cc + 2 < cend) p[2] = u.z;
                if (cc + 3 < cend) p[3] = u.w;
            }
        }
}

// One row r of Q 8-column MMA tiles (four neighbouring ones, the next four 64
// further), the pairs of columns that start at c: += add(q, e).
template <int Q, typename F>
__device__ __forceinline__ void add_row_pairs(float* a, int lda, int cend, int rend, int r, int c, bool vec, F add) {
    if (r >= rend) return;
    float* p = a + (size_t)r * lda + c;
    float2 v[Q];
#pragma unroll
    for (int q = 0; q < Q; q++) {
        const int o = 64 * (q >> 2) + 8 * (q & 3);
        v[q] = make_float2(0.0f, 0.0f);
        if (vec && c + o + 1 < cend) {
            v[q] = *reinterpret_cast<const float2*>(p + o);
        } else {
            if (c + o < cend) v[q].x = p[o];
            if (c + o + 1 < cend) v[q].y = p[o + 1];
        }
    }
#pragma unroll
    for (int q = 0; q < Q; q++) {
        const int o = 64 * (q >> 2) + 8 * (q & 3);
        const float2 u = make_float2(v[q].x + add(q, 0), v[q].y + add(q, 1));
        if (vec && c + o + 1 < cend) {
            *reinterpret_cast<float2*>(p + o) = u;
        } else {
            if (c + o < cend) p[o] = u.x;
            if (c + o + 1 < cend) p[o + 1] = u.y;
        }
    }
}

// One tile of an update C += L T inside a system's matrix a: rows r0 .. (below
// rend), columns c0 .. (below cend), L in columns kb .. kb+K of those rows, T
// in rows kb .. kb+K of those columns (K a multiple of 16).  WR x WC warps of
// 4 x 8 lanes with 4 x 4 outputs each (16 WR x 32 WC in all).  32-deep chunks
// of L (transposed, k-major) and T are copied in one ahead of the products; C
// goes to L2 meanwhile.
// BF16: L and T rounded to BF16 and multiplied on the tensor cores (warp-level
// m16n8k16 MMA, FP32 accumulation), a warp's piece being four such tiles; the
// row strides (4 mod 32 floats) keep the fragment reads free of bank
// conflicts.
template <int WR, int WC, bool BF16>
__device__ __noinline__ void update_tile(float* a, int lda, int r0, int rend, int c0, int cend, int kb, int K,
                                         bool vec, float* sm) {
    constexpr int TM = 16 * WR, TN = 32 * WC, SA = TM + 4, SB = TN + 4;
    static_assert(32 * WR * WC == BT, "warps");
    float* As = sm;                // 2 x 32 x SA
    float* Bs = sm + 2 * 32 * SA;  // 2 x 32 x SB
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    auto issue = [&](int k0, int buf) {
        const int kc = min(32, K - k0);
        float* A = As + buf * 32 * SA;
        float* B = Bs + buf * 32 * SB;
#pragma unroll 4
        for (int i = warp; i < TM; i += BT / 32) {  // lane = k: a row of L
            if (lane < kc && r0 + i < rend)
                cp_async4(A + lane * SA + i, a + (size_t)(r0 + i) * lda + kb + k0 + lane);
            else
                A[lane * SA + i] = 0.0f;
        }
        for (int idx = tid; idx < 32 * TN / 4; idx += BT) {
            const int k = idx / (TN / 4), j = (idx % (TN / 4)) * 4;
            const float* src = a + (size_t)(kb + k0 + k) * lda + c0 + j;
            float* dst = B + k * SB + j;
            if (k < kc && vec && c0 + j + 3 < cend) {
                cp_async_vec16(dst, src);
            } else {
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    if (k < kc && c0 + j + e < cend)
                        cp_async4(dst + e, src + e);
                    else
                        dst[e] = 0.0f;
                }
            }
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    issue(0, 0);
    for (int idx = tid; idx < TM * TN / 32; idx += BT) {
        const int r = r0 + idx / (TN / 32), c = c0 + (idx % (TN / 32)) * 32;
        if (r < rend && c < cend) asm volatile("prefetch.global.L2 [%0];\n" ::"l"(a + (size_t)r * lda + c));
    }
    const int wr = warp / WC, wc = warp % WC;
    const int g = lane >> 2, t4 = lane & 3;                                       // MMA lanes
    const int row = 16 * wr + 4 * (lane >> 3), col = 32 * wc + 4 * (lane & 7);  // FP32 lanes
    float acc[16];  // BF16: four 16 x 8 tiles' four values; FP32: 4 x 4
#pragma unroll
    for (int e = 0; e < 16; e++) acc[e] = 0.0f;
    for (int k0 = 0, buf = 0; k0 < K; k0 += 32, buf ^= 1) {
        if (k0 + 32 < K) issue(k0 + 32, buf ^ 1);
        else asm volatile("cp.async.commit_group;\n" ::: "memory");
        asm volatile("cp.async.wait_group 1;\n" ::: "memory");
        __syncthreads();
        const float* A = As + buf * 32 * SA + (BF16 ? 16 * wr + g : row);
        const float* B = Bs + buf * 32 * SB + (BF16 ? 32 * wc + g : col);
#pragma unroll 1
        for (int kq = 0; kq < min(32, K - k0); kq += 16) {
            if constexpr (BF16) {
                const float* L0 = A + (kq + 2 * t4) * SA;
                const uint32_t a0 = pack_bf16(L0[0], L0[SA]), a1 = pack_bf16(L0[8], L0[SA + 8]);
                const uint32_t a2 = pack_bf16(L0[8 * SA], L0[9 * SA]), a3 = pack_bf16(L0[8 * SA + 8], L0[9 * SA + 8]);
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    const float* T0 = B + (kq + 2 * t4) * SB + 8 * q;
                    float(&d)[4] = *reinterpret_cast<float(*)[4]>(acc + 4 * q);
                    mma_bf16_16816(d, a0, a1, a2, a3, pack_bf16(T0[0], T0[SB]), pack_bf16(T0[8 * SB], T0[9 * SB]));
                }
            } else {
#pragma unroll
                for (int k = 0; k < 16; k++) {
                    const float4 l = *reinterpret_cast<const float4*>(A + (kq + k) * SA);
                    const float4 t = *reinterpret_cast<const float4*>(B + (kq + k) * SB);
                    const float la[4] = {l.x, l.y, l.z, l.w}, ta[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
                    for (int i = 0; i < 4; i++)
#pragma unroll
                        for (int q = 0; q < 4; q++) acc[4 * i + q] = fmaf(la[i], ta[q], acc[4 * i + q]);
                }
            }
        }
        __syncthreads();
    }
    if constexpr (BF16) {
#pragma unroll
        for (int h = 0; h < 2; h++)
            add_row_pairs<4>(a, lda, cend, rend, r0 + 16 * wr + g + 8 * h, c0 + 32 * wc + 2 * t4, vec,
                             [&](int q, int e) { return acc[4 * q + 2 * h + e]; });
    } else {
        add_quads<1>(a, lda, cend, rend, r0 + row, c0 + col, 0, vec, [&](int i, int) {
            return make_float4(acc[4 * i], acc[4 * i + 1], acc[4 * i + 2], acc[4 * i + 3]);
        });
    }
    __syncthreads();
}

// The trailing update behind outer block b0: C[r0.., cbeg..] += L T for one
// block of 128 rows (rows below n) and every column from cbeg on.  L's 128 x 128
// piece (transposed, k-major) stays in shared memory for all of the row
// block's 128 x 128 tiles; T streams through a ring of four 16-row chunks
// without a break between tiles, so a tile's C is read and written while the
// next tile's first chunks arrive.  FP32: 8 x 8 outputs per thread, whose loads
// are just level with the FMA pipe; BF16: as update_tile.
template <bool BF16>
__device__ __noinline__ void trailing_rows(float* a, int lda, int n, int r0, int cbeg, int b0, bool vec, float* sm) {
    constexpr int OB = 128, SA = OB + 4, CH = 16, RINGS = 4;
    float* A = sm;                // OB x SA
    float* ring = sm + OB * SA;   // RINGS x CH x SA
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int rend = min(n, r0 + OB), ntile = (n - cbeg + OB - 1) / OB, nchunk = ntile * (OB / CH);
#pragma unroll 4
    for (int i = warp; i < OB; i += BT / 32) {  // lane = k: a row of L
#pragma unroll
        for (int k = 0; k < OB; k += 32) {
            if (r0 + i < rend)
                cp_async4(A + (k + lane) * SA + i, a + (size_t)(r0 + i) * lda + b0 + k + lane);
            else
                A[(k + lane) * SA + i] = 0.0f;
        }
    }
    auto issue = [&](int ch) {
        if (ch < nchunk) {
            const int c0 = cbeg + (ch / (OB / CH)) * OB, k0 = (ch % (OB / CH)) * CH;
            float* dst0 = ring + (ch % RINGS) * CH * SA;
#pragma unroll
            for (int idx = tid; idx < CH * OB / 4; idx += BT) {
                const int k = idx / (OB / 4), j = (idx % (OB / 4)) * 4;
                const float* src = a + (size_t)(b0 + k0 + k) * lda + c0 + j;
                float* dst = dst0 + k * SA + j;
                if (vec && c0 + j + 3 < n) {
                    cp_async_vec16(dst, src);
                } else {
#pragma unroll
                    for (int e = 0; e < 4; e++) {
                        if (c0 + j + e < n)
                            cp_async4(dst + e, src + e);
                        else
                            dst[e] = 0.0f;
                    }
                }
            }
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    for (int q = 0; q < RINGS - 1; q++) issue(q);  // the first group covers L too
    const int wr = warp >> 1, wc = warp & 1;       // 4 x 2 warps
    int ch = 0;
    for (int t = 0; t < ntile; t++) {
        const int c0 = cbeg + t * OB;
        for (int idx = tid; idx < OB * OB / 32; idx += BT) {
            const int r = r0 + idx / (OB / 32), c = c0 + (idx % (OB / 32)) * 32;
            if (r < rend && c < n) asm volatile("prefetch.global.L2 [%0];\n" ::"l"(a + (size_t)r * lda + c));
        }
        if constexpr (BF16) {
            const int g = lane >> 2, t4 = lane & 3;
            float acc[2][8][4];  // rows 16 wr + 64 m, columns 32 wc + 64 (q / 4) + 8 (q % 4)
#pragma unroll
            for (int m = 0; m < 2; m++)
#pragma unroll
                for (int q = 0; q < 8; q++)
#pragma unroll
                    for (int e = 0; e < 4; e++) acc[m][q][e] = 0.0f;
            for (int k0 = 0; k0 < OB; k0 += CH, ch++) {
                asm volatile("cp.async.wait_group %0;\n" ::"n"(RINGS - 2) : "memory");
                __syncthreads();
                issue(ch + RINGS - 1);
                const float* L = A + (k0 + 2 * t4) * SA + 16 * wr + g;
                const float* B = ring + (ch % RINGS) * CH * SA + 2 * t4 * SA + 32 * wc + g;
                uint32_t fa[2][4];
#pragma unroll
                for (int m = 0; m < 2; m++) {
                    const float* L0 = L + 64 * m;
                    fa[m][0] = pack_bf16(L0[0], L0[SA]);
                    fa[m][1] = pack_bf16(L0[8], L0[SA + 8]);
                    fa[m][2] = pack_bf16(L0[8 * SA], L0[9 * SA]);
                    fa[m][3] = pack_bf16(L0[8 * SA + 8], L0[9 * SA + 8]);
                }
#pragma unroll
                for (int q = 0; q < 8; q++) {
                    const float* T0 = B + 64 * (q >> 2) + 8 * (q & 3);
                    const uint32_t b0r = pack_bf16(T0[0], T0[SA]), b1r = pack_bf16(T0[8 * SA], T0[9 * SA]);
#pragma unroll
                    for (int m = 0; m < 2; m++)
                        mma_bf16_16816(acc[m][q], fa[m][0], fa[m][1], fa[m][2], fa[m][3], b0r, b1r);
                }
            }
#pragma unroll
            for (int m = 0; m < 2; m++)
#pragma unroll
                for (int h = 0; h < 2; h++)
                    add_row_pairs<8>(a, lda, n, rend, r0 + 16 * wr + 64 * m + g + 8 * h, c0 + 32 * wc + 2 * t4, vec,
                                     [&](int q, int e) { return acc[m][q][2 * h + e]; });
        } else {
            const int row = 16 * wr + 4 * (lane >> 3), col = 32 * wc + 4 * (lane & 7);
            float2 acc[8][4];  // rows row, row + 64; columns col, col + 64
#pragma unroll
            for (int i = 0; i < 8; i++)
#pragma unroll
                for (int q = 0; q < 4; q++) acc[i][q] = make_float2(0.0f, 0.0f);
            for (int k0 = 0; k0 < OB; k0 += CH, ch++) {
                asm volatile("cp.async.wait_group %0;\n" ::"n"(RINGS - 2) : "memory");
                __syncthreads();
                issue(ch + RINGS - 1);
                const float* L = A + k0 * SA + row;
                const float* B = ring + (ch % RINGS) * CH * SA + col;
#pragma unroll
                for (int k = 0; k < CH; k++) {
                    float l[8];
                    float2 v[4];
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        const float4 x = *reinterpret_cast<const float4*>(L + k * SA + 64 * h);
                        l[4 * h] = x.x, l[4 * h + 1] = x.y, l[4 * h + 2] = x.z, l[4 * h + 3] = x.w;
                        const float4 y = *reinterpret_cast<const float4*>(B + k * SA + 64 * h);
                        v[2 * h] = make_float2(y.x, y.y), v[2 * h + 1] = make_float2(y.z, y.w);
                    }
#pragma unroll
                    for (int i = 0; i < 8; i++)
#pragma unroll
                        for (int q = 0; q < 4; q++) acc[i][q] = __ffma2_rn(make_float2(l[i], l[i]), v[q], acc[i][q]);
                }
            }
#pragma unroll
            for (int h = 0; h < 2; h++)
                add_quads<2>(a, lda, n, rend, r0 + row + 64 * h, c0 + col, 64, vec, [&](int i, int q) {
                    const float2 x = acc[4 * h + i][2 * q], y = acc[4 * h + i][2 * q + 1];
                    return make_float4(x.x, x.y, y.x, y.y);
                });
        }
    }
    __syncthreads();
}

// top for the columns c >= cbeg of block row k0 (NB rows) with the factored
// diagonal block (Dt: transposed): t_k *= D_kk; t_j += t_k D_jk (j > k).  Two
// neighbouring columns per thread: every value of D read from shared memory
// serves both.  The compiler may order those reads freely inside one pass, but
// not move them out of the loop (NB^2 / 2 values would spill): the empty asm.
template <int NB, int DL>
__device__ __noinline__ void top_columns(float* a, int lda, int n, int k0, int cbeg, const float* Dt, bool vec) {
#pragma unroll 1
    for (int c = cbeg + 2 * threadIdx.x; c < n; c += 2 * BT) {
        asm volatile("" ::: "memory");
        const bool two = c + 1 < n, pair = two && vec;
        float x[NB], y[NB];
#pragma unroll
        for (int i = 0; i < NB; i++) {
            const float* p = a + (size_t)(k0 + i) * lda + c;
            if (pair) {
                const float2 v = *reinterpret_cast<const float2*>(p);
                x[i] = v.x, y[i] = v.y;
            } else {
                x[i] = p[0], y[i] = two ? p[1] : 0.0f;
            }
        }
#pragma unroll
        for (int k = 0; k < NB; k++) {
#pragma unroll
            for (int j = k / 4 * 4; j < NB; j += 4) {
                const float4 u = *reinterpret_cast<const float4*>(Dt + k * DL + j);
                const float d[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    if (j + e == k) x[k] *= d[e], y[k] *= d[e];
                    if (j + e > k) x[j + e] = fmaf(x[k], d[e], x[j + e]), y[j + e] = fmaf(y[k], d[e], y[j + e]);
                }
            }
        }
#pragma unroll
        for (int i = 0; i < NB; i++) {
            float* p = a + (size_t)(k0 + i) * lda + c;
            if (pair) {
                *reinterpret_cast<float2*>(p) = make_float2(x[i], y[i]);
            } else {
                p[0] = x[i];
                if (two) p[1] = y[i];
            }
        }
    }
}

// left for the rows r >= rbeg of block column k0: l_i += l_k D_ki (i > k), two
// neighbouring rows per thread, taken from the last thread on (the first ones
// have more columns of the block row).
template <int NB, int DL>
__device__ __noinline__ void left_rows(float* a, int lda, int n, int k0, int rbeg, const float* Ds, bool vec) {
#pragma unroll 1
    for (int r = rbeg + 2 * (BT - 1 - threadIdx.x); r < n; r += 2 * BT) {
        asm volatile("" ::: "memory");
        const bool two = r + 1 < n;
        float x[NB], y[NB];
        float* p = a + (size_t)r * lda + k0;
        float* q = two ? p + lda : p;
        if (vec) {  // k0 is a multiple of NB: the row segments are 16-byte aligned
#pragma unroll
            for (int i = 0; i < NB; i += 4) {
                const float4 u = *reinterpret_cast<const float4*>(p + i), v = *reinterpret_cast<const float4*>(q + i);
                x[i] = u.x, x[i + 1] = u.y, x[i + 2] = u.z, x[i + 3] = u.w;
                y[i] = v.x, y[i + 1] = v.y, y[i + 2] = v.z, y[i + 3] = v.w;
            }
        } else {
#pragma unroll
            for (int i = 0; i < NB; i++) x[i] = p[i], y[i] = q[i];
        }
#pragma unroll
        for (int k = 0; k < NB; k++) {
#pragma unroll
            for (int i = (k + 1) / 4 * 4; i < NB; i += 4) {
                const float4 u = *reinterpret_cast<const float4*>(Ds + k * DL + i);
                const float d[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
                for (int e = 0; e < 4; e++)
                    if (i + e > k) x[i + e] = fmaf(x[k], d[e], x[i + e]), y[i + e] = fmaf(y[k], d[e], y[i + e]);
            }
        }
        if (vec) {
#pragma unroll
            for (int i = 0; i < NB; i += 4) {
                *reinterpret_cast<float4*>(p + i) = make_float4(x[i], x[i + 1], x[i + 2], x[i + 3]);
                if (two) *reinterpret_cast<float4*>(q + i) = make_float4(y[i], y[i + 1], y[i + 2], y[i + 3]);
            }
        } else {
#pragma unroll
            for (int i = 0; i < NB; i++) {
                p[i] = x[i];
                if (two) q[i] = y[i];
            }
        }
    }
}

// Blocked factorization of one system in global memory (see file comment):
// outer blocks of 128, inner panels of NB.  Inside an outer block the panels
// are left-looking (each panel's block column and row first take all of the
// outer block's earlier panels at once), and everything beyond the outer block
// takes its 128 steps in one update: C is read and written n / 128 times, not
// n / NB.  4096 systems of 32 .. 1024: 19.4 -> 15.6 ms with the solve's changes;
// one system of n = 1000 spends half of its time in the trailing update, at
// 49 % of the FMA pipe with both of an SM's CTAs in it.
template <int NB, bool BF16>
__device__ __noinline__ void factor_blocked(float* a, int lda, int n, float* sm) {
    constexpr int OB = 128, DL = NB + 4;
    float* Ds = sm;           // the factored diagonal block and its transpose (row stride DL); the updates' operands
    float* Dt = sm + NB * DL; // take the same space when neither is needed any more
    const int tid = threadIdx.x;
    const bool vec = ((lda & 3) == 0) && ((reinterpret_cast<uintptr_t>(a) & 15) == 0);
    for (int b0 = 0; b0 < n; b0 += OB) {
        const int bend = min(n, b0 + OB);
        for (int k0 = b0; k0 < bend; k0 += NB) {
            const int kb = min(NB, bend - k0), r0 = k0 + kb, done = k0 - b0;
            if (done > 0) {
                // the block column (with the diagonal block), then the block row right of it
                for (int r = k0; r < n; r += 128)
                    update_tile<8, 1, BF16>(a, lda, r, n, k0, r0, b0, done, vec, sm);
                for (int c = r0; c < n; c += 128)
                    update_tile<2, 4, BF16>(a, lda, k0, r0, c, n, b0, done, vec, sm);
            }
            if (tid < 32) warp_diag_lu<NB, DL>(a + (size_t)k0 * lda + k0, lda, kb, Ds, Dt);
            __syncthreads();
            if (r0 < n) {  // (the panel is full: kb == NB)
                top_columns<NB, DL>(a, lda, n, k0, r0, Dt, vec);
                left_rows<NB, DL>(a, lda, n, k0, r0, Ds, vec);
                __syncthreads();
            }
        }
        for (int r = bend; r < n; r += OB) trailing_rows<BF16>(a, lda, n, r, bend, b0, vec, sm);
    }
}

// Blocked forward/back sweeps, right-hand sides resident in shared memory
// (Y[i * NR + q], nrhs <= NR).  Per 64-unknown block: the diagonal block is
// staged in shared memory (copied in while the block before it is applied) and
// one warp per right-hand side walks its 64-step chain (values in lanes,
// pivots by shuffle); then every thread updates up to four later (forward) /
// earlier (backward) unknowns with the block's rows, four rows' loads in
// flight, each factor element and each of the block's values read once for
// all right-hand sides / unknowns of the thread.

// Y[i] += sgn * sum_k Y[k0 + k] S[k0 + k][i] for i = i0 + threadIdx.x + e * BT < i1, e < PT.
template <int NR, int PT>
__device__ __forceinline__ void apply_block(const float* __restrict__ a, int lda, int k0, int kb, int i0, int i1,
                                            float sgn, float* Y) {
    float acc[PT][NR];
#pragma unroll
    for (int e = 0; e < PT; e++)
#pragma unroll
        for (int q = 0; q < NR; q++) acc[e][q] = 0.0f;
    const float* col = a + (size_t)k0 * lda + i0 + threadIdx.x;
    for (int kc = 0; kc < kb; kc += 4) {
        float v[4][PT];
#pragma unroll
        for (int k = 0; k < 4; k++)
#pragma unroll
            for (int e = 0; e < PT; e++)
                v[k][e] = (kc + k < kb && i0 + (int)threadIdx.x + e * BT < i1) ? col[(size_t)(kc + k) * lda + e * BT] : 0.0f;
#pragma unroll
        for (int k = 0; k < 4; k++) {
            if (kc + k >= kb) break;
            float y[NR];
            const float* yk = Y + (k0 + kc + k) * NR;
            if constexpr (NR >= 4) {
#pragma unroll
                for (int q = 0; q < NR; q += 4) {
                    const float4 u = *reinterpret_cast<const float4*>(yk + q);
                    y[q] = u.x, y[q + 1] = u.y, y[q + 2] = u.z, y[q + 3] = u.w;
                }
            } else {
#pragma unroll
                for (int q = 0; q < NR; q++) y[q] = yk[q];
            }
#pragma unroll
            for (int e = 0; e < PT; e++)
#pragma unroll
                for (int q = 0; q < NR; q++) acc[e][q] = fmaf(y[q], v[k][e], acc[e][q]);
        }
    }
#pragma unroll
    for (int e = 0; e < PT; e++) {
        const int i = i0 + threadIdx.x + e * BT;
        if (i < i1)
#pragma unroll
            for (int q = 0; q < NR; q++) Y[i * NR + q] = fmaf(sgn, acc[e][q], Y[i * NR + q]);
    }
}

template <int NR>
__device__ __forceinline__ void apply_range(const float* a, int lda, int k0, int kb, int i0, int i1, float sgn,
                                            float* Y) {
    const int pt = (i1 - i0 + BT - 1) / BT;  // n <= 1024: at most four unknowns per thread
    if (pt <= 0) return;
    if (pt == 1)
        apply_block<NR, 1>(a, lda, k0, kb, i0, i1, sgn, Y);
    else if (pt == 2)
        apply_block<NR, 2>(a, lda, k0, kb, i0, i1, sgn, Y);
    else
        apply_block<NR, 4>(a, lda, k0, kb, i0, i1, sgn, Y);
}

template <int NR>
__device__ __noinline__ void solve_blocked(const float* a, int lda, int n, float* b, int ldb, int nrhs, float* sm) {
    constexpr int SBK = kSolveBlk, DL = kSolveDL;
    float* Y = sm;                         // n x NR
    float* dblk = sm + RHS_MAX * 1024;     // two diagonal blocks, alternating
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nblk = (n + SBK - 1) / SBK;
    // step s: forward block s, then backward blocks nblk - 1 .. 0
    auto stage = [&](int s) {
        const int k0 = (s < nblk ? s : 2 * nblk - 1 - s) * SBK, kb = min(SBK, n - k0);
        float* D = dblk + (s & 1) * SBK * DL;
        for (int r = warp; r < kb; r += BT / 32)
            for (int c = lane; c < kb; c += 32) cp_async4(D + r * DL + c, a + (size_t)(k0 + r) * lda + k0 + c);
    };
    stage(0);
    for (int idx = tid; idx < NR * n; idx += BT) {
        const int q = idx / n, i = idx - q * n;
        Y[i * NR + q] = q < nrhs ? b[(size_t)q * ldb + i] : 0.0f;
    }
    for (int s = 0; s < 2 * nblk; s++) {
        const bool fwd = s < nblk;
        const int k0 = (fwd ? s : 2 * nblk - 1 - s) * SBK, kb = min(SBK, n - k0);
        const float* D = dblk + (s & 1) * SBK * DL;
        cp_async_wait_all();
        __syncthreads();
        if (s + 1 < 2 * nblk) stage(s + 1);
        for (int q = warp; q < nrhs; q += BT / 32) {
            float* y = Y + k0 * NR + q;
            float v0 = lane < kb ? y[lane * NR] : 0.0f, v1 = lane + 32 < kb ? y[(lane + 32) * NR] : 0.0f;
            if (fwd) {  // y_i += y_k S[k][i] (i > k)
                for (int k = 0; k < kb; k++) {
                    const float yk = __shfl_sync(0xffffffffu, k < 32 ? v0 : v1, k & 31);
                    if (lane > k && lane < kb) v0 = fmaf(yk, D[k * DL + lane], v0);
                    if (lane + 32 > k && lane + 32 < kb) v1 = fmaf(yk, D[k * DL + lane + 32], v1);
                }
            } else {  // s = y_k S[k][k]; x_k = -s; y_i += s S[k][i] (i < k)
                for (int k = kb - 1; k >= 0; k--) {
                    const float yk = __shfl_sync(0xffffffffu, k < 32 ? v0 : v1, k & 31);
                    const float sk = yk * D[k * DL + k];
                    if (lane == (k & 31)) {
                        if (k < 32) v0 = -sk; else v1 = -sk;
                    }
                    if (lane < k) v0 = fmaf(sk, D[k * DL + lane], v0);
                    if (lane + 32 < k) v1 = fmaf(sk, D[k * DL + lane + 32], v1);
                }
            }
            if (lane < kb) y[lane * NR] = v0;
            if (lane + 32 < kb) y[(lane + 32) * NR] = v1;
        }
        __syncthreads();
        // the unknowns after (forward) or before (backward, coefficients s_k = -x_k) the block
        if (fwd)
            apply_range<NR>(a, lda, k0, kb, k0 + kb, n, 1.0f, Y);
        else
            apply_range<NR>(a, lda, k0, kb, 0, k0, -1.0f, Y);
    }
    __syncthreads();
    for (int idx = tid; idx < nrhs * n; idx += BT) {
        const int q = idx / n, i = idx - q * n;
        b[(size_t)q * ldb + i] = Y[i * NR + q];
    }
    __syncthreads();
}

__device__ __forceinline__ void solve_factored(const float* a, int lda, int n, float* b, int ldb, int nrhs, float* sm) {
    if (nrhs == 1)
        solve_blocked<1>(a, lda, n, b, ldb, nrhs, sm);
    else if (nrhs <= 4)
        solve_blocked<4>(a, lda, n, b, ldb, nrhs, sm);
    else if (nrhs <= 8)
        solve_blocked<8>(a, lda, n, b, ldb, nrhs, sm);
    else
        solve_blocked<16>(a, lda, n, b, ldb, nrhs, sm);
}

__global__ void __launch_bounds__(BT, 2) k_batch_solve(const BatchSys* __restrict__ sys, int count, float* A, float* B,
                                                    int* next, Tune tune) {
    extern __shared__ float sm[];
    __shared__ int s_item;
    for (;;) {
        if (threadIdx.x == 0) s_item = atomicAdd(next, 1);
        __syncthreads();
        const int t = s_item;
        __syncthreads();
        if (t >= count) break;
        const BatchSys s = sys[t];
        float* a = tune.absolute ? reinterpret_cast<float*>(s.a_off) : A + s.a_off;
        float* b = tune.absolute ? reinterpret_cast<float*>(s.b_off) : B + s.b_off;
        const bool factor = (s.nrhs & kSolveOnly) == 0;
        const int nrhs = s.nrhs & (kSolveOnly - 1);
        if (s.n <= tune.small_n_max) {
            solve_small(a, s.lda, s.n, b, s.ldb, nrhs, factor, sm);
        } else {
            if (factor) {
                if (tune.nb[bucket_of(s.n)] == 16)
                    factor_blocked<16, false>(a, s.lda, s.n, sm);
                else
                    factor_blocked<32, false>(a, s.lda, s.n, sm);
            }
            solve_factored(a, s.lda, s.n, b, s.ldb, nrhs, sm);
        }
    }
}

// max over the CTA of v[0..3] (non-negative values; NaN marks a non-finite
// input and wins), into out[0..3] for every thread.
__device__ __forceinline__ void block_max4(double (&v)[4], double* red) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int q = 0; q < 4; q++) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const double w = __shfl_xor_sync(0xffffffffu, v[q], o);
            v[q] = (isnan(w) || w > v[q]) ? w : v[q];
        }
    }
    __syncthreads();
    if (lane == 0)
#pragma unroll
        for (int q = 0; q < 4; q++) red[warp * 4 + q] = v[q];
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 4; q++) {
        double m = red[q];
        for (int w = 1; w < BT / 32; w++) {
            const double x = red[w * 4 + q];
            m = (isnan(x) || x > m) ? x : m;
        }
        v[q] = m;
    }
    __syncthreads();
}

// One warp's part of M x (M = S0^T, S0 the FP32 original a0 widened exactly,
// FP64 accumulation): columns c0 .. c0+127 of S0 (lane: four neighbouring
// ones) over rows j0 .. j1, NQ right-hand sides x[j * 4 + q]; with NORM the
// columns' absolute sums too.  Four columns per thread, so that a value of x
// read from shared memory serves four FP64 products; eight or sixteen rows'
// loads in flight.
template <int NQ, bool NORM>
__device__ __forceinline__ void residual_part(const float* __restrict__ a0, int lda, int n, int c0, int j0, int j1,
                                              bool vec, const double* x, double (&acc)[4][NQ], double (&col)[4]) {
    const int c = c0 + 4 * (threadIdx.x & 31);
#pragma unroll
    for (int e = 0; e < 4; e++) {
        col[e] = 0.0;
#pragma unroll
        for (int q = 0; q < NQ; q++) acc[e][q] = 0.0;
    }
    constexpr int U = NQ <= 2 ? 16 : 8;
    for (int jc = j0; jc < j1; jc += U) {
        float v[U][4];
#pragma unroll
        for (int k = 0; k < U; k++) {
            const float* p = a0 + (size_t)(jc + k) * lda + c;
            if (jc + k < j1 && vec && c + 3 < n) {
                const float4 u = *reinterpret_cast<const float4*>(p);
                v[k][0] = u.x, v[k][1] = u.y, v[k][2] = u.z, v[k][3] = u.w;
            } else {
#pragma unroll
                for (int e = 0; e < 4; e++) v[k][e] = jc + k < j1 && c + e < n ? p[e] : 0.0f;
            }
        }
#pragma unroll
        for (int k = 0; k < U; k++) {
            if (jc + k >= j1) break;
            double xj[NQ];
#pragma unroll
            for (int q = 0; q < NQ; q++) xj[q] = x[(jc + k) * 4 + q];
#pragma unroll
            for (int e = 0; e < 4; e++) {
                const double w = (double)v[k][e];
                if (NORM) col[e] += fabs(w);
#pragma unroll
                for (int q = 0; q < NQ; q++) acc[e][q] = fma(w, xj[q], acc[e][q]);
            }
        }
    }
}

// M x for NQ right-hand sides into part (splits x 128 G columns x NQ doubles,
// G = ceil(n / 128) column groups, splits = the row ranges that the warps
// allow), and the columns' absolute sums (NORM) into pcol alike.
template <int NQ, bool NORM>
__device__ __noinline__ void residual_product(const float* __restrict__ a0, int lda, int n, bool vec, const double* x,
                                              double* part, double* pcol, int G, int splits) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rows = (n + splits - 1) / splits;
    for (int item = warp; item < G * splits; item += BT / 32) {
        const int g = item % G, sp = item / G;
        double acc[4][NQ], col[4];
        residual_part<NQ, NORM>(a0, lda, n, 128 * g, min(n, sp * rows), min(n, (sp + 1) * rows), vec, x, acc, col);
#pragma unroll
        for (int e = 0; e < 4; e++) {
            const int i = (sp * G + g) * 128 + 4 * lane + e;
#pragma unroll
            for (int q = 0; q < NQ; q++) part[i * NQ + q] = acc[e][q];
            if (NORM) pcol[i] = col[e];
        }
    }
}

// FP64 iterative refinement of one factored system (all threads of the CTA),
// the per-system form of refine_core: x = the FP32 solution in b32, widened;
// repeat r = b - M x (M = S0^T, the original FP32 matrix widened exactly, FP64
// accumulation), HPL scaled residual per right-hand side
// ||r||_inf / ((||M||_inf ||x||_inf + ||b||_inf) n eps), eps = DBL_EPSILON/2
// (LINPACK/src/host/gmres.c:182-193); stop at <= 16 or after max_iters
// refinements, else d = LU \ r (FP32 factors, r rounded to FP32), x += d.
// Returns the refinements made; *resid = the largest scaled residual (NaN if
// any value is not finite).
__device__ int refine_system(const float* __restrict__ lu, const float* __restrict__ a0, int lda, int n,
                             float* b32, const double* __restrict__ b64, double* x64, int ldb, int nrhs,
                             int max_iters, bool small, float* sm, double* resid) {
    const int tid = threadIdx.x;
    const bool vec = ((lda & 3) == 0) && ((reinterpret_cast<uintptr_t>(a0) & 15) == 0);
    const int G = (n + 127) / 128, splits = max(1, (BT / 32) / G), cols = 128 * G;
    double* xs = reinterpret_cast<double*>(sm);  // n x 4 right-hand sides (FP64)
    double* part = xs + 4 * 1024;                // splits x cols x (right-hand sides at a time, at most 4)
    double* pcol = part + 4 * 1024;              // splits x cols
    double* red = pcol + 1024;                   // one row of 4 per warp
    for (int idx = tid; idx < nrhs * n; idx += BT) {
        const int q = idx / n, i = idx - q * n;
        x64[(size_t)q * ldb + i] = (double)b32[(size_t)q * ldb + i];
    }
    __syncthreads();
    double normM = 0.0;
    double worst = 0.0;
    int it = 0;
    for (;; it++) {
        worst = 0.0;
        for (int q0 = 0; q0 < nrhs; q0 += 4) {
            const int nq = min(4, nrhs - q0), nt = nq == 3 ? 4 : nq;  // nt: products formed
            for (int idx = tid; idx < nt * n; idx += BT) {
                const int q = idx / n, j = idx - q * n;
                xs[j * 4 + q] = q < nq ? x64[(size_t)(q0 + q) * ldb + j] : 0.0;
            }
            __syncthreads();
            const bool norm = it == 0 && q0 == 0;
            auto product = [&](auto nqc) {
                constexpr int NQ = decltype(nqc)::value;
                if (norm) residual_product<NQ, true>(a0, lda, n, vec, xs, part, pcol, G, splits);
                else residual_product<NQ, false>(a0, lda, n, vec, xs, part, pcol, G, splits);
            };
            if (nt == 1) product(std::integral_constant<int, 1>());
            else if (nt == 2) product(std::integral_constant<int, 2>());
            else product(std::integral_constant<int, 4>());
            __syncthreads();
            // r = b - M x into b32 (FP32, the next correction's right-hand side); norms of r, x, b and M's columns
            double rm[4] = {0.0, 0.0, 0.0, 0.0}, xm[4] = {0.0, 0.0, 0.0, 0.0}, bm[4] = {0.0, 0.0, 0.0, 0.0};
            double cm[4] = {0.0, 0.0, 0.0, 0.0};
            auto larger = [](double& m, double w) { m = (isnan(w) || w > m) ? w : m; };
            for (int i = tid; i < n; i += BT) {
                if (norm) {
                    double s = 0.0;
                    for (int sp = 0; sp < splits; sp++) s += pcol[sp * cols + i];
                    larger(cm[0], s);
                }
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    if (q >= nq) continue;
                    double s = 0.0;
                    for (int sp = 0; sp < splits; sp++) s += part[(sp * cols + i) * nt + q];
                    const double bv = b64[(size_t)(q0 + q) * ldb + i], r = bv - s;
                    b32[(size_t)(q0 + q) * ldb + i] = (float)r;
                    larger(rm[q], fabs(r));
                    larger(xm[q], fabs(xs[i * 4 + q]));
                    larger(bm[q], fabs(bv));
                }
            }
            block_max4(rm, red);
            block_max4(xm, red);
            block_max4(bm, red);
            if (norm) {
                block_max4(cm, red);
                normM = cm[0];
            }
            for (int q = 0; q < nq; q++) {
                const double h = rm[q] / (normM * xm[q] + bm[q]) / (double)n / (DBL_EPSILON / 2.0);
                worst = (isnan(h) || !(h <= worst)) ? h : worst;
            }
        }
        if (!(worst > 16.0) || isnan(worst) || isinf(worst) || it >= max_iters) break;
        // d = LU \ r, x += d
        if (small)
            solve_small(const_cast<float*>(lu), lda, n, b32, ldb, nrhs, false, sm);
        else
            solve_factored(lu, lda, n, b32, ldb, nrhs, sm);
        for (int idx = tid; idx < nrhs * n; idx += BT) {
            const int q = idx / n, i = idx - q * n;
            x64[(size_t)q * ldb + i] += (double)b32[(size_t)q * ldb + i];
        }
        __syncthreads();
    }
    *resid = worst;
    return it;
}

// The refined form of k_batch_solve: per system, b32 = (float) b64; factor
// in place (BF16: the blocked path's trailing updates on the tensor cores,
// the diagonal blocks and triangular stages in FP32; systems solved whole in
// shared memory are factored in FP32); FP32 solve into b32; FP64 refinement
// against the original a0 into x64.  iters / resid: per descriptor position.
template <bool BF16>
__global__ void __launch_bounds__(BT, 2)
    k_batch_solve_ir(const BatchSys* __restrict__ sys, int count, float* A, const float* __restrict__ A0, float* B32,
                     const double* __restrict__ B64, double* X64, int* next, Tune tune, int max_iters,
                     int* __restrict__ iters, double* __restrict__ resid) {
    extern __shared__ float sm[];
    __shared__ int s_item;
    for (;;) {
        if (threadIdx.x == 0) s_item = atomicAdd(next, 1);
        __syncthreads();
        const int t = s_item;
        __syncthreads();
        if (t >= count) break;
        const BatchSys s = sys[t];
        float* a = A + s.a_off;
        const float* a0 = A0 + s.a_off;
        float* b = B32 + s.b_off;
        const double* b64 = B64 + s.b_off;
        double* x64 = X64 + s.b_off;
        const int nrhs = s.nrhs;
        for (int idx = threadIdx.x; idx < nrhs * s.n; idx += BT) {
            const int q = idx / s.n, i = idx - q * s.n;
            b[(size_t)q * s.ldb + i] = (float)b64[(size_t)q * s.ldb + i];
        }
        __syncthreads();
        const bool small = s.n <= tune.small_n_max;
        const int nb = tune.nb[bucket_of(s.n)];
        if (small) {
            solve_small(a, s.lda, s.n, b, s.ldb, nrhs, true, sm);
        } else {
            if (nb == 16)
                factor_blocked<16, BF16>(a, s.lda, s.n, sm);
            else
                factor_blocked<32, BF16>(a, s.lda, s.n, sm);
            solve_factored(a, s.lda, s.n, b, s.ldb, nrhs, sm);
        }
        double r = 0.0;
        const int k = refine_system(a, a0, s.lda, s.n, b, b64, x64, s.ldb, nrhs, max_iters, small, sm, &r);
        if (threadIdx.x == 0) {
            iters[t] = k;
            resid[t] = r;
        }
    }
}

}  // namespace

int batch_init_attrs() {
    LP_CUDA(cudaFuncSetAttribute(k_batch_solve, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kBatchSmem));
    LP_CUDA(cudaFuncSetAttribute(k_batch_solve_ir<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)kBatchSmem));
    LP_CUDA(cudaFuncSetAttribute(k_batch_solve_ir<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)kBatchSmem));
    return LP_OK;
}

int validate_batch(int count, const lp_system* systems) {
    if (count < 0 || (count > 0 && systems == nullptr)) return fail(LP_E_INVALID, "batch: bad system list");
    for (int i = 0; i < count; i++) {
        const lp_system& s = systems[i];
        if (s.n <= 0 || s.n > 1024 || s.nrhs <= 0 || s.nrhs > RHS_MAX || s.lda < s.n || s.ldb < s.n || s.a_off < 0 ||
            s.b_off < 0)
            return fail(LP_E_INVALID, "batch: system " + std::to_string(i) +
                                          " needs 1 <= n <= 1024, 1 <= nrhs <= 16, lda >= n, ldb >= n");
    }
    return LP_OK;
}

int launch_batch(lp_ctx* c, const lp_system* d_sorted, int count, float* dA, float* dB, const lp_batch_config& cfg,
                 int* d_next, cudaStream_t st, bool absolute) {
    static_assert(kSolveOnly > RHS_MAX, "solve-only flag above the nrhs range");
    Tune tune;
    tune.absolute = absolute ? 1 : 0;
    tune.small_n_max = cfg.small_n_max;
    for (int i = 0; i < NBUCKETS; i++) tune.nb[i] = cfg.nb[i];
    const int per_sm = cfg.ctas_per_sm < 1 ? 1 : (cfg.ctas_per_sm > 3 ? 3 : cfg.ctas_per_sm);
    int grid = c->num_sms * per_sm;
    if (grid > count) grid = count;
    if (grid < 1) return LP_OK;
    LP_CUDA(cudaMemsetAsync(d_next, 0, sizeof(int), st));
    k_batch_solve<<<grid, BT, kBatchSmem, st>>>(reinterpret_cast<const BatchSys*>(d_sorted), count, dA, dB, d_next,
                                                 tune);
    count_launch();
    LP_CUDA(cudaGetLastError());
    return LP_OK;
}

int launch_batch_ir(lp_ctx* c, bool bf16, const lp_system* d_sorted, int count, float* dA, const float* dA0,
                    float* dB32, const double* dB64, double* dX, const lp_batch_config& cfg, int max_iters,
                    int* d_iters, double* d_resid, int* d_next, cudaStream_t st) {
    Tune tune;
    tune.absolute = 0;
    tune.small_n_max = cfg.small_n_max;
    for (int i = 0; i < NBUCKETS; i++) tune.nb[i] = cfg.nb[i];
    const int per_sm = cfg.ctas_per_sm < 1 ? 1 : (cfg.ctas_per_sm > 3 ? 3 : cfg.ctas_per_sm);
    int grid = c->num_sms * per_sm;
    if (grid > count) grid = count;
    if (grid < 1) return LP_OK;
    LP_CUDA(cudaMemsetAsync(d_next, 0, sizeof(int), st));
    const auto* sys = reinterpret_cast<const BatchSys*>(d_sorted);
    if (bf16)
        k_batch_solve_ir<true><<<grid, BT, kBatchSmem, st>>>(sys, count, dA, dA0, dB32, dB64, dX, d_next, tune,
                                                             max_iters, d_iters, d_resid);
    else
        k_batch_solve_ir<false><<<grid, BT, kBatchSmem, st>>>(sys, count, dA, dA0, dB32, dB64, dX, d_next, tune,
                                                              max_iters, d_iters, d_resid);
    count_launch();
    LP_CUDA(cudaGetLastError());
    return LP_OK;
}

}  // namespace lp
