// inner stage, FP64 (the reference's _DP build, DATA_TYPE double): C(m x n) +=
// At^T * B on k-major operands (At: k x m, B: k x n, rows of contiguous
// doubles) — inner_update_mm (hpl_torus_PCIE.cl:711-865) in double.
//
// tcgen05 has no FP64 kind, and this part's FP64 tensor rate equals its DFMA
// rate; the warp-level FP64 MMA still wins because of its operand traffic.
// Shared memory delivers 128 bytes a clock to the registers: 8 x 4 DFMA
// outputs per thread need 96 bytes per 32 products, 43 products a clock of the
// pipe's 64 (that form ran at 19 TFLOP/s, 0.52 of it), where a 32 x 32 warp
// tile of m16n8k8 MMAs loads 128 bytes a lane for 256 (31 TFLOP/s).  Products are fused
// and accumulated in ascending k, as the DFMA form did.  Operands are staged
// by 16-byte cp.async into a ring; C is read and written once per launch.
#include "lp_common.cuh"

namespace lp {
namespace {

constexpr int BK = 16, ST = 3;

__device__ __forceinline__ void cp_async16z(void* smem, const void* gmem, int src_bytes) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem), "r"(src_bytes));
}

// D (16 x 8) += A (16 x 8) * B (8 x 8) in FP64, one warp.
__device__ __forceinline__ void mma_f64(double (&d)[4], const double (&a)[4], double b0, double b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
        : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3])
        : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(b0), "d"(b1));
}

// WR x WC warps, each 16 MT rows x 8 NC columns.
template <int WR, int WC, int MT, int NC>
struct Form {
    static constexpr int NT = 32 * WR * WC, TM = 16 * MT * WR, TN = 8 * NC * WC;
    // row strides: 4 mod 16 doubles, so that the fragment loads (4 k x 8 rows or columns) hit distinct banks
    static constexpr int SA = TM + 4, SB = TN + 4;
    static constexpr size_t smem = sizeof(double) * ST * BK * (SA + SB);
};

template <int WR, int WC, int MT, int NC>
__global__ void __launch_bounds__(32 * WR * WC) k_dgemm_update(double* __restrict__ C, int ldc,
                                                               const double* __restrict__ At, int ldat,
                                                               const double* __restrict__ B, int ldb, int M, int N,
                                                               int K) {
    using F = Form<WR, WC, MT, NC>;
    constexpr int NT = F::NT, TM = F::TM, TN = F::TN, SA = F::SA, SB = F::SB;
    extern __shared__ __align__(16) double dsm[];
    double* As = dsm;                  // ST x BK x SA
    double* Bs = dsm + ST * BK * SA;   // ST x BK x SB
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int m0 = blockIdx.y * TM, n0 = blockIdx.x * TN;
    const int g = lane >> 2, t4 = lane & 3;
    const int wm = (warp / WC) * 16 * MT, wn = (warp % WC) * 8 * NC;

    auto load_stage = [&](int stage, int kt) {
#pragma unroll
        for (int i = 0; i < BK * TM / 2 / NT; i++) {
            const int idx = tid + i * NT, row = idx / (TM / 2), col = (idx % (TM / 2)) * 2;
            const bool ok = m0 + col < M;
            cp_async16z(&As[(stage * BK + row) * SA + col], ok ? At + (size_t)(kt * BK + row) * ldat + m0 + col : At,
                        ok ? 16 : 0);
        }
#pragma unroll
        for (int i = 0; i < BK * TN / 2 / NT; i++) {
            const int idx = tid + i * NT, row = idx / (TN / 2), col = (idx % (TN / 2)) * 2;
            const bool ok = n0 + col < N;
            cp_async16z(&Bs[(stage * BK + row) * SB + col], ok ? B + (size_t)(kt * BK + row) * ldb + n0 + col : B,
                        ok ? 16 : 0);
        }
    };

    double acc[MT][NC][4];
#pragma unroll
    for (int i = 0; i < MT; i++)
#pragma unroll
        for (int j = 0; j < NC; j++)
#pragma unroll
            for (int e = 0; e < 4; e++) acc[i][j][e] = 0.0;

    const int KT = K / BK;
#pragma unroll
    for (int s = 0; s < ST - 1; s++) {
        if (s < KT) load_stage(s, s);
        asm volatile("cp.async.commit_group;\n" ::);
    }
    // the tile of C on its way to L2 while the products run
#pragma unroll
    for (int i = 0; i < TM * TN / 16 / NT; i++) {
        const int idx = tid + i * NT, r = m0 + idx / (TN / 16), c = n0 + (idx % (TN / 16)) * 16;
        if (r < M && c < N) asm volatile("prefetch.global.L2 [%0];\n" ::"l"(C + (size_t)r * ldc + c));
    }
    for (int kt = 0; kt < KT; kt++) {
        asm volatile("cp.async.wait_group %0;\n" ::"n"(ST - 2));
        __syncthreads();
        const int nk = kt + ST - 1;
        if (nk < KT) load_stage(nk % ST, nk);
        asm volatile("cp.async.commit_group;\n" ::);
        const double* as = As + (kt % ST) * BK * SA + wm + g;
        const double* bs = Bs + (kt % ST) * BK * SB + wn + g;
#pragma unroll
        for (int k = 0; k < BK; k += 8) {
            double a[MT][4], b[NC][2];
#pragma unroll
            for (int i = 0; i < MT; i++) {
                a[i][0] = as[(k + t4) * SA + 16 * i];
                a[i][1] = as[(k + t4) * SA + 16 * i + 8];
                a[i][2] = as[(k + 4 + t4) * SA + 16 * i];
                a[i][3] = as[(k + 4 + t4) * SA + 16 * i + 8];
            }
#pragma unroll
            for (int j = 0; j < NC; j++) {
                b[j][0] = bs[(k + t4) * SB + 8 * j];
                b[j][1] = bs[(k + 4 + t4) * SB + 8 * j];
            }
#pragma unroll
            for (int i = 0; i < MT; i++)
#pragma unroll
                for (int j = 0; j < NC; j++) mma_f64(acc[i][j], a[i], b[j][0], b[j][1]);
        }
    }
    asm volatile("cp.async.wait_group 0;\n" ::);

#pragma unroll
    for (int i = 0; i < MT; i++)
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int r = m0 + wm + 16 * i + 8 * h + g;
            if (r >= M) continue;
            double2 v[NC];
            double2* p = reinterpret_cast<double2*>(C + (size_t)r * ldc + n0 + wn + 2 * t4);
#pragma unroll
            for (int j = 0; j < NC; j++)
                if (n0 + wn + 8 * j + 2 * t4 < N) v[j] = p[4 * j];
#pragma unroll
            for (int j = 0; j < NC; j++)
                if (n0 + wn + 8 * j + 2 * t4 < N) {
                    v[j].x += acc[i][j][2 * h];
                    v[j].y += acc[i][j][2 * h + 1];
                    p[4 * j] = v[j];
                }
        }
}

#define LP_D_TILE 2, 2, 2, 4   // 64 x 64 tiles
#define LP_D_SMALL 2, 2, 1, 2  // 32 x 32
using Tile = Form<LP_D_TILE>;
using Small = Form<LP_D_SMALL>;

}  // namespace

int dgemm_init_attrs() {
    LP_CUDA(cudaFuncSetAttribute(k_dgemm_update<LP_D_TILE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)Tile::smem));
    LP_CUDA(cudaFuncSetAttribute(k_dgemm_update<LP_D_SMALL>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)Small::smem));
    return LP_OK;
}

int launch_dgemm_update(double* c, int ldc, const double* lt, int ldlt, const double* t, int ldt, int m, int n, int k,
                        cudaStream_t st) {
    if (m <= 0 || n <= 0) return LP_OK;
    if (k % BK != 0 || m % 4 != 0 || n % 4 != 0 || ldc % 2 != 0 || ldlt % 2 != 0 || ldt % 2 != 0 || !aligned16(c) ||
        !aligned16(lt) || !aligned16(t))
        return fail(LP_E_INVALID, "FP64 inner update: k a multiple of 16; m, n multiples of 4; leading dimensions "
                                  "even; pointers 16-byte aligned");
    auto grid = [&](int tm, int tn) { return dim3((n + tn - 1) / tn, (m + tm - 1) / tm); };
    // 64 x 64 tiles, several CTAs per SM (128 x 128 with one CTA per SM: 669 us against 565 at 5888^2 x 256, 31.4
    // TFLOP/s); a quarter of that while they would not give every SM two (512^2 x 128: 10.7 -> 7.3 us)
    const dim3 g = grid(Tile::TM, Tile::TN);
    if (g.y > 65535) return fail(LP_E_INVALID, "FP64 inner update: m too large");
    if ((long long)g.x * g.y < 2 * 148)
        k_dgemm_update<LP_D_SMALL><<<grid(Small::TM, Small::TN), Small::NT, Small::smem, st>>>(c, ldc, lt, ldlt, t, ldt,
                                                                                             m, n, k);
    else
        k_dgemm_update<LP_D_TILE><<<g, Tile::NT, Tile::smem, st>>>(c, ldc, lt, ldlt, t, ldt, m, n, k);
    count_launch();
    LP_CUDA(cudaGetLastError());
    return LP_OK;
}

}  // namespace lp
