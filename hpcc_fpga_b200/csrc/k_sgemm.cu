// inner stage, FP32: C(m x n) += At^T * B on k-major operands
// (At: k x m, B: k x n, rows of contiguous floats).
//
// The trailing update of one block step runs as one or a few launches over
// the whole trailing matrix (the reference issues one inner_update_mm task
// per b x b block, hpl_torus_PCIE.cl:711-865, execution_pcie.hpp:523-583):
// C += L * T with L given transposed.
//
// Both operands are k-major, so every tile load is a run of 16-byte cp.async
// copies into a ST-deep shared-memory ring.  Accumulators are pairs updated
// with Blackwell's packed FP32 FMA (FFMA2, fma.rn.f32x2: two independent
// correctly rounded fused multiply-adds per issued instruction, so each
// element is computed exactly as fmaf would).  C is read and written once per
// launch.
//
// Shared memory delivers 128 bytes a clock to an SM's registers, whether the
// lanes of a load share addresses or not, and the FMA pipe takes 128 products
// a clock: R x C outputs per thread cost R + C clocks of loads against R C / 4
// of products per warp and k.  At 8 x 8 the two are level (and the kernel
// reached 75 % of the pipe); the large form takes 8 x 16, 24 against 32
// (7680^2 x 512 1093 -> 993 us, 60.8 TFLOP/s; x 128 313 -> 274).  The small
// forms trade that for more CTAs (launch_sgemm_update).  Every element
// gets the same sum in the same order in each form, so they agree bit for
// bit.
#include "lp_common.cuh"

namespace lp {
namespace {

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem, int src_bytes) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem), "r"(src_bytes));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }

// A CTA computes a TM x TN tile with WR x WC warps of 4 x 8 lanes; a thread
// holds RG row groups and CG column groups of four.
template <int WR, int WC, int RG, int CG, int BK, int ST>
struct Form {
    static constexpr int NT = 32 * WR * WC, TM = 16 * WR * RG, TN = 32 * WC * CG;
    static constexpr size_t smem = sizeof(float) * ST * BK * (TM + TN);
};

template <int WR, int WC, int RG, int CG, int BK, int ST, int MINB>
__global__ void __launch_bounds__(32 * WR * WC, MINB)
    k_sgemm_update(float* __restrict__ C, int ldc, const float* __restrict__ At, int ldat, const float* __restrict__ B,
                   int ldb, int M, int N, int K) {
    using F = Form<WR, WC, RG, CG, BK, ST>;
    constexpr int NT = F::NT, TM = F::TM, TN = F::TN, R = 4 * RG;
    extern __shared__ __align__(16) float sm[];
    float* As = sm;
    float* Bs = sm + ST * BK * TM;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int m0 = blockIdx.y * TM, n0 = blockIdx.x * TN;
    const int row = 16 * (warp / WC) + 4 * (lane >> 3), col = 32 * (warp % WC) + 4 * (lane & 7);

    auto load_stage = [&](int stage, int kt) {
#pragma unroll
        for (int i = 0; i < BK * TM / 4 / NT; i++) {
            const int idx = tid + i * NT, r = idx / (TM / 4), c = (idx % (TM / 4)) * 4, kr = kt * BK + r;
            const bool ok = m0 + c < M && (BK == 16 || kr < K);
            cp_async16(&As[(stage * BK + r) * TM + c], ok ? At + (size_t)kr * ldat + m0 + c : At, ok ? 16 : 0);
        }
#pragma unroll
        for (int i = 0; i < BK * TN / 4 / NT; i++) {
            const int idx = tid + i * NT, r = idx / (TN / 4), c = (idx % (TN / 4)) * 4, kr = kt * BK + r;
            const bool ok = n0 + c < N && (BK == 16 || kr < K);
            cp_async16(&Bs[(stage * BK + r) * TN + c], ok ? B + (size_t)kr * ldb + n0 + c : B, ok ? 16 : 0);
        }
    };

    // acc[i][h]: the pair of columns (2h, 2h + 1) of the thread's row i
    float2 acc[R][2 * CG];
#pragma unroll
    for (int i = 0; i < R; i++)
#pragma unroll
        for (int j = 0; j < 2 * CG; j++) acc[i][j] = make_float2(0.0f, 0.0f);

    const int KT = (K + BK - 1) / BK;
    if constexpr (TM < 128) {  // the forms of the panel's chain; big grids lose SM slots to waiting blocks
        pdl_start();
        pdl_wait();
    }
#pragma unroll
    for (int s = 0; s < ST - 1; s++) {
        if (s < KT) load_stage(s, s);
        cp_async_commit();
    }
    // the tile of C on its way to L2 while the products run: the epilogue's reads are its only use
#pragma unroll
    for (int i = 0; i < TM * TN / 32 / NT; i++) {
        const int idx = tid + i * NT, r = m0 + idx / (TN / 32), c = n0 + (idx % (TN / 32)) * 32;
        if (r < M && c < N) asm volatile("prefetch.global.L2 [%0];\n" ::"l"(C + (size_t)r * ldc + c));
    }
    for (int kt = 0; kt < KT; kt++) {
        cp_async_wait<ST - 2>();
        __syncthreads();
        const int nk = kt + ST - 1;
        if (nk < KT) load_stage(nk % ST, nk);
        cp_async_commit();
        const float* as = As + (kt % ST) * BK * TM + row;
        const float* bs = Bs + (kt % ST) * BK * TN + col;
        // K is a multiple of 16: with BK = 32 the last step may hold 16 rows
        const int kend = (BK > 16 && K - kt * BK < BK) ? 16 : BK;
#pragma unroll 16
        for (int k = 0; k < kend; k++) {
            float a[R];
            float2 b[2 * CG];
#pragma unroll
            for (int i = 0; i < RG; i++) {
                const float4 v = *reinterpret_cast<const float4*>(as + k * TM + 16 * WR * i);
                a[4 * i] = v.x, a[4 * i + 1] = v.y, a[4 * i + 2] = v.z, a[4 * i + 3] = v.w;
            }
#pragma unroll
            for (int j = 0; j < CG; j++) {
                const float4 v = *reinterpret_cast<const float4*>(bs + k * TN + 32 * WC * j);
                b[2 * j] = make_float2(v.x, v.y), b[2 * j + 1] = make_float2(v.z, v.w);
            }
#pragma unroll
            for (int i = 0; i < R; i++) {
                const float2 ai = make_float2(a[i], a[i]);
#pragma unroll
                for (int j = 0; j < 2 * CG; j++) acc[i][j] = __ffma2_rn(ai, b[j], acc[i][j]);
            }
        }
    }
    cp_async_wait<0>();

    // four rows' loads in flight before their first store (the compiler keeps a load behind a store to the same array)
#pragma unroll
    for (int i0 = 0; i0 < R; i0 += 4) {
        float4 v[4][CG];
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int j = 0; j < CG; j++) {
                const int r = m0 + row + 4 * WR * i0 + i, c = n0 + col + 32 * WC * j;
                if (r < M && c < N) v[i][j] = *reinterpret_cast<const float4*>(C + (size_t)r * ldc + c);
            }
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int j = 0; j < CG; j++) {
                const int r = m0 + row + 4 * WR * i0 + i, c = n0 + col + 32 * WC * j;
                if (r < M && c < N)
                    *reinterpret_cast<float4*>(C + (size_t)r * ldc + c) =
                        make_float4(v[i][j].x + acc[i0 + i][2 * j].x, v[i][j].y + acc[i0 + i][2 * j].y,
                                    v[i][j].z + acc[i0 + i][2 * j + 1].x, v[i][j].w + acc[i0 + i][2 * j + 1].y);
            }
    }
}

#define LP_LARGE 4, 1, 2, 4, 16, 4   // 128 x 128 tiles, 8 x 16 outputs per thread
#define LP_MIDDLE 2, 2, 2, 1, 32, 3  // 64 x 64, 8 x 4
#define LP_SMALL 2, 1, 1, 1, 32, 4   // 32 x 32, 4 x 4
using Large = Form<LP_LARGE>;
using Middle = Form<LP_MIDDLE>;
using Small = Form<LP_SMALL>;

constexpr int kSms = 148;

}  // namespace

int sgemm_init_attrs() {
    LP_CUDA(cudaFuncSetAttribute(k_sgemm_update<LP_LARGE, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)Large::smem));
    LP_CUDA(cudaFuncSetAttribute(k_sgemm_update<LP_MIDDLE, 4>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)Middle::smem));
    LP_CUDA(cudaFuncSetAttribute(k_sgemm_update<LP_SMALL, 8>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)Small::smem));
    return LP_OK;
}

int launch_sgemm_update(float* c, int ldc, const float* lt, int ldlt, const float* t, int ldt, int m, int n, int k,
                        cudaStream_t st) {
    if (m <= 0 || n <= 0) return LP_OK;
    if (k % 16 != 0 || m % 4 != 0 || n % 4 != 0 || ldc % 4 != 0 || ldlt % 4 != 0 || ldt % 4 != 0 || !aligned16(c) ||
        !aligned16(lt) || !aligned16(t))
        return fail(LP_E_INVALID, "inner_update: k must be a multiple of 16; m, n, leading dimensions multiples of 4; "
                                  "pointers 16-byte aligned");
    if ((m + Large::TM - 1) / Large::TM > 65535) return fail(LP_E_INVALID, "inner_update: m too large");
    auto grid = [&](int tm, int tn) { return dim3((n + tn - 1) / tn, (m + tm - 1) / tm); };
    // The form whose busiest SM has the least to do: tiles per SM x clocks per k of a tile (products or loads,
    // whichever is more: 128, 48, 16).
    auto cost = [&](int tm, int tn, long long clocks) {
        const dim3 g = grid(tm, tn);
        return ((long long)g.x * g.y + kSms - 1) / kSms * clocks;
    };
    const long long large = cost(Large::TM, Large::TN, 128), middle = cost(Middle::TM, Middle::TN, 48),
                    small = cost(Small::TM, Small::TN, 16);
    if (large <= middle && large <= small) {
        k_sgemm_update<LP_LARGE, 2><<<grid(Large::TM, Large::TN), Large::NT, Large::smem, st>>>(c, ldc, lt, ldlt, t, ldt, m,
                                                                                              n, k);
    } else if (middle <= small) {
        LP_CUDA(launch_pdl(k_sgemm_update<LP_MIDDLE, 4>, grid(Middle::TM, Middle::TN), dim3(Middle::NT), Middle::smem, st,
                           c, ldc, lt, ldlt, t, ldt, m, n, k));
    } else {
        LP_CUDA(launch_pdl(k_sgemm_update<LP_SMALL, 8>, grid(Small::TM, Small::TN), dim3(Small::NT), Small::smem, st, c,
                           ldc, lt, ldlt, t, ldt, m, n, k));
    }
    count_launch();
    LP_CUDA(cudaGetLastError());
    return LP_OK;
}

}  // namespace lp
