// FP64 form of the path — the reference's _DP build (DATA_TYPE / HOST_DATA_TYPE
// double, LINPACK/src/host/parameters.h.in; CI's double-precision variant):
// the same blocked right-looking LU without pivoting (lu / top / left / inner,
// gefa_ref_nopvt's encoding) and the same substitution, in double.
//
// lu, top and left are the float kernels instantiated for double
// (k_lu.cu, k_trsm.cu: reference operation order, bit-identical on one
// block); inner is k_dgemm_update.  The substitution below is blocked by 64
// unknowns, one launch for both sweeps: every CTA runs a block's recurrence
// itself, then updates its share of the other
// unknowns with the block's rows (a GEMV over contiguous rows, each factor
// element read once per sweep).
#include <string>

#include "lp_ctx.cuh"

namespace lp {
namespace {

constexpr int SB = 64;       // substitution block
constexpr int GT = 256;      // threads per CTA
constexpr int RMAX = 16;     // right-hand sides per pass
constexpr int NW = GT / 32;  // warps; in the updates each takes SB / NW rows of the block
constexpr int RPW = SB / NW;
constexpr unsigned kSpinLimit64 = 1u << 22;

// The dependent steps of one block for Q right-hand sides, one warp; lane holds
// the unknowns lane and lane + 32 (v[q][0], v[q][1]); D: the kb x kb diagonal
// block (FP32 factors, for the GMRES refinement, widened exactly as they are
// read).  Forward: v_i += v_k D_ki (i > k).  Backward: s = v_k D_kk, v_i += s D_ki
// (i < k); v_k = s.  Four steps at a time: one exchange brings their values to
// every lane, which forms the four results itself (the operations of the
// unknowns' own lanes, in the same order), so a step costs a quarter of an
// exchange's latency (n = 6144: 0.07 ms); G = 1 is the plain step of a ragged
// block's end.
template <int G, int Q, typename FT>
__device__ __forceinline__ void steps_forward(double (&v)[Q][2], const FT* D, int h, int kk, int lane) {
    const FT* row = D + (32 * h + kk) * SB;  // row of the first step
#pragma unroll
    for (int q = 0; q < Q; q++) {
        double y[G];
#pragma unroll
        for (int j = 0; j < G; j++) y[j] = __shfl_sync(0xffffffffu, v[q][h], kk + j);
#pragma unroll
        for (int j = 1; j < G; j++)
#pragma unroll
            for (int i = 0; i < j; i++) y[j] = fma(y[i], (double)row[i * SB + 32 * h + kk + j], y[j]);
#pragma unroll
        for (int j = 0; j < G; j++) {
            if (lane > kk + j) v[q][h] = fma(y[j], (double)row[j * SB + 32 * h + lane], v[q][h]);
            if (h == 0) v[q][1] = fma(y[j], (double)row[j * SB + 32 + lane], v[q][1]);
        }
    }
}
template <int G, int Q, typename FT>
__device__ __forceinline__ void steps_backward(double (&v)[Q][2], const FT* D, int h, int kk, int lane) {
    const FT* row = D + (32 * h + kk) * SB;  // row of the last step (the lowest unknown)
#pragma unroll
    for (int q = 0; q < Q; q++) {
        double s[G];
#pragma unroll
        for (int j = 0; j < G; j++) s[j] = __shfl_sync(0xffffffffu, v[q][h], kk + j);
#pragma unroll
        for (int j = G - 1; j >= 0; j--) {
#pragma unroll
            for (int i = G - 1; i > j; i--) s[j] = fma(s[i], (double)row[i * SB + 32 * h + kk + j], s[j]);
            s[j] *= (double)row[j * SB + 32 * h + kk + j];
        }
#pragma unroll
        for (int j = G - 1; j >= 0; j--) {
            if (lane < kk + j)
                v[q][h] = fma(s[j], (double)row[j * SB + 32 * h + lane], v[q][h]);
            else if (lane == kk + j)
                v[q][h] = s[j];
            if (h == 1) v[q][0] = fma(s[j], (double)row[j * SB + lane], v[q][0]);
        }
    }
}
template <int Q, typename FT>
__device__ __forceinline__ void block_forward(double (&v)[Q][2], const FT* D, int kb, int lane) {
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const int m = min(32, kb - 32 * h);
        int kk = 0;
#pragma unroll 2
        for (; kk + 4 <= m; kk += 4) steps_forward<4>(v, D, h, kk, lane);
        for (; kk < m; kk++) steps_forward<1>(v, D, h, kk, lane);
    }
}
template <int Q, typename FT>
__device__ __forceinline__ void block_backward(double (&v)[Q][2], const FT* D, int kb, int lane) {
#pragma unroll
    for (int h = 1; h >= 0; h--) {
        int kk = min(32, kb - 32 * h);
        while (kk > 0 && (kk & 3) != 0) steps_backward<1>(v, D, h, --kk, lane);
#pragma unroll 2
        for (kk -= 4; kk >= 0; kk -= 4) steps_backward<4>(v, D, h, kk, lane);
    }
}

// Bounded grid barrier of a cooperative launch; the counter only grows.
// absent (tests): this CTA does not arrive.
__device__ __forceinline__ bool grid_sync64(unsigned* bar, unsigned target, unsigned limit, bool absent, int* err) {
    __shared__ int s_ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        if (!absent) atomicAdd(bar, 1u);
        int ok = 1;
        unsigned spins = 0, v;
        for (;;) {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(bar) : "memory");
            if (v >= target) break;
            if ((++spins & 255u) == 0 && (*reinterpret_cast<volatile int*>(err) != 0 || spins > limit)) {
                atomicExch(err, 1);
                ok = 0;
                break;
            }
        }
        __threadfence();
        s_ok = ok;
    }
    __syncthreads();
    return s_ok != 0;
}

// Forward and back substitution of one group of right-hand sides (rows of b,
// overwritten by the solutions), one cooperative launch.  Per block of SB
// unknowns every CTA runs the block's own recurrence (one warp per right-hand
// side, two above eight; the diagonal block was copied in before the barrier),
// then updates its share of the unknowns after (forward) or before (backward)
// it with rows loaded before the barrier; one barrier per block.  w1, w2: n x
// nrhs accumulating values of the two sweeps (the forward sweep's results are
// the second's input).  A chain of 2 n / 64 short steps, where one launch per block and direction took
// 15 us each (n = 6144: 192 launches, 2.9 ms; now 1.0).  Products with the blocks'
// inverses in place of the recurrences took 0.20 ms less, but lost what the
// condition of a block's triangles allows.  A barrier that gives up leaves
// NaN in the solutions and sets *gave_up, a word in page-locked host memory.
// stall (tests): CTA 0 never arrives at the first barrier.
template <typename FT>
__global__ void __launch_bounds__(GT, 1)
    k_gesl64(const FT* __restrict__ a, int lda, int n, double* w1, double* w2, double* b, int ldb, int nrhs,
             unsigned* sync, int* gave_up, int stall) {
    extern __shared__ __align__(16) double sm[];
    double* ys = sm;                          // RMAX x SB: the block's solved values
    double* part = ys + RMAX * SB;            // NW x 32 x RMAX partial sums
    FT* Db = reinterpret_cast<FT*>(part + NW * 32 * RMAX);  // 2 x SB x SB: the diagonal block, alternating
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, G = gridDim.x, g = blockIdx.x;
    int* err = reinterpret_cast<int*>(sync + 1);
    const int nblk = (n + SB - 1) / SB, steps = 2 * nblk;
    // step s: forward block s, then backward blocks nblk - 1 .. 0
    auto block_of = [&](int s) { return s < nblk ? s : steps - 1 - s; };
    auto range = [&](int s, int& i0, int& i1) {
        const int k0 = block_of(s) * SB, lo = s < nblk ? min(n, k0 + SB) : 0, hi = s < nblk ? n : k0;
        const int ch = (hi - lo + G - 1) / G;
        i0 = min(hi, lo + g * ch);
        i1 = min(hi, i0 + ch);
    };
    auto stage = [&](int s) {
        const int k0 = block_of(s) * SB, kb = min(SB, n - k0);
        for (int idx = tid; idx < SB * SB; idx += GT) {
            const int r = idx / SB, c = idx % SB;
            if (r < kb && c < kb) cp_async_elem(Db + (s & 1) * SB * SB + idx, a + (size_t)(k0 + r) * lda + k0 + c);
        }
    };
    double v[RPW];
    auto load_rows = [&](int s, int i, bool ok) {
        const int k0 = block_of(s) * SB + RPW * warp;
#pragma unroll
        for (int q = 0; q < RPW; q++) v[q] = ok && k0 + q < n ? (double)__ldg(a + (size_t)(k0 + q) * lda + i) : 0.0;
    };
    int i0, i1;
    stage(0);
    range(0, i0, i1);
    load_rows(0, i0 + lane, i0 + lane < i1);
    for (int s = 0; s < steps; s++) {
        const bool fwd = s < nblk;
        const int k0 = block_of(s) * SB, kb = min(SB, n - k0);
        double* w = fwd ? w1 : w2;
        double y[2][2];  // this warp's right-hand sides: warp and warp + NW
#pragma unroll
        for (int q = 0; q < 2; q++)
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int r = warp + NW * q, i = lane + 32 * h;
                y[q][h] = r < nrhs && i < kb ? __ldcg(w + (size_t)r * n + k0 + i) : 0.0;
            }
        cp_async_wait_all();
        __syncthreads();
        if (s + 1 < steps) stage(s + 1);
        if (warp < nrhs) {
            const FT* D = Db + (s & 1) * SB * SB;
            if (nrhs <= NW) {
                double(&y1)[1][2] = reinterpret_cast<double(&)[1][2]>(y);
                if (fwd) block_forward<1>(y1, D, kb, lane);
                else block_backward<1>(y1, D, kb, lane);
            } else if (fwd) {
                block_forward<2>(y, D, kb, lane);
            } else {
                block_backward<2>(y, D, kb, lane);
            }
        }
#pragma unroll
        for (int q = 0; q < 2; q++)
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int r = warp + NW * q, i = lane + 32 * h;
                if (r >= nrhs) continue;
                ys[r * SB + i] = i < kb ? y[q][h] : 0.0;
                if (g == 0 && i < kb) {
                    if (fwd)
                        w2[(size_t)r * n + k0 + i] = y[q][h];  // (w1's block is still being read by other CTAs)
                    else
                        b[(size_t)r * ldb + k0 + i] = -y[q][h];
                }
            }
        __syncthreads();
        // unknowns after (forward) or before (backward) the block: += y^T S[block][i]
        for (int ib = i0; ib < i1; ib += 32) {
            if (ib != i0) load_rows(s, ib + lane, ib + lane < i1);
            for (int r = 0; r < nrhs; r++) {
                const double* y = ys + r * SB + RPW * warp;
                double t = 0.0;
#pragma unroll
                for (int q = 0; q < RPW; q++) t = fma(y[q], v[q], t);
                part[(r * NW + warp) * 32 + lane] = t;
            }
            __syncthreads();
            for (int idx = tid; idx < nrhs * 32; idx += GT) {
                const int r = idx >> 5, i = ib + (idx & 31);
                if (i < i1) {
                    const double* q = part + r * NW * 32 + (idx & 31);
                    double t = 0.0;
#pragma unroll
                    for (int e = 0; e < NW; e++) t += q[32 * e];
                    double* p = w + (size_t)r * n + i;
                    *p = __ldcg(p) + t;
                }
            }
            __syncthreads();
        }
        if (s + 1 == steps) break;
        range(s + 1, i0, i1);
        load_rows(s + 1, i0 + lane, i0 + lane < i1);
        if (!grid_sync64(sync, (unsigned)(s + 1) * (unsigned)G, stall != 0 ? kSpinLimit64 / 16 : kSpinLimit64,
                         stall != 0 && g == 0 && s == 0, err)) {
            if (tid == 0) {
                *reinterpret_cast<volatile int*>(gave_up) = 1;
                __threadfence_system();
            }
            for (int idx = g * GT + tid; idx < nrhs * n; idx += G * GT)
                b[(size_t)(idx / n) * ldb + idx % n] = __longlong_as_double(0x7ff8000000000000ll);
            return;
        }
    }
}
constexpr size_t kGesl64Smem = sizeof(double) * (2 * SB * SB + RMAX * SB + (size_t)NW * 32 * RMAX);
static_assert(RMAX <= 2 * NW, "a warp takes two right-hand sides");

double event_s64(cudaEvent_t a, cudaEvent_t b) {
    float ms = 0.0f;
    cudaEventElapsedTime(&ms, a, b);
    return 1e-3 * ms;
}

int validate64(const void* a, int n, int lda, int bs, const char* who) {
    if (a == nullptr) return fail(LP_E_INVALID, std::string(who) + ": null matrix pointer");
    if (n <= 0 || lda < n) return fail(LP_E_INVALID, std::string(who) + ": need n > 0 and lda >= n");
    if (bs != 64 && bs != 128 && bs != 256)
        return fail(LP_E_INVALID, std::string(who) + ": FP64 block size must be 64, 128 or 256");
    if (n % bs != 0) return fail(LP_E_INVALID, std::string(who) + ": n must be a multiple of the block size");
    if (lda % 2 != 0 || !aligned16(a))
        return fail(LP_E_INVALID, std::string(who) + ": matrix must be 16-byte aligned with an even lda");
    return LP_OK;
}

}  // namespace

// Blocks wider than 128 (256): the same blocked algorithm inside the block
// with 128-wide inner blocks, as the FP32 path does for its 512 blocks — the
// lu of the diagonal block recursively, top and left as 128-row / -column
// exact chunks plus FP64 GEMM updates of the rest.  `dt` holds one transposed
// 128-wide sub-block (128 x 128) of the diagonal block.
static int lu_stage64(double* d, int lda, int bs, double* lti, cudaStream_t st) {
    if (bs <= 128) return launch_lu_small_f64(d, lda, bs, st);
    const int ib = 128;
    for (int kk = 0; kk < bs / ib; kk++) {
        double* dd = d + (size_t)kk * ib * lda + (size_t)kk * ib;
        LP_CHECK(launch_lu_small_f64(dd, lda, ib, st));
        const int r = bs - (kk + 1) * ib;
        if (r <= 0) break;
        LP_CHECK(launch_top_chunk_f64(dd, lda, dd + ib, lda, ib, r, st));
        LP_CHECK(launch_left_chunk_f64(dd, lda, dd + (size_t)ib * lda, lda, ib, r, lti, r, st));
        LP_CHECK(launch_dgemm_update(dd + (size_t)ib * lda + ib, lda, lti, r, dd + ib, lda, r, r, ib, st));
    }
    return LP_OK;
}

static int top_blocked64(const double* d, int lda, double* t, int ldt, int bs, int ncols, double* dt,
                         cudaStream_t st) {
    if (bs <= 128) return launch_top_chunk_f64(d, lda, t, ldt, bs, ncols, st);
    const int ib = 128;
    for (int kk = 0; kk < bs / ib; kk++) {
        const double* dkk = d + (size_t)kk * ib * lda + (size_t)kk * ib;
        double* tk = t + (size_t)kk * ib * ldt;
        LP_CHECK(launch_top_chunk_f64(dkk, lda, tk, ldt, ib, ncols, st));
        const int m2 = bs - (kk + 1) * ib;
        if (m2 <= 0) break;
        // T[below] += D[below][chunk] * T[chunk]: D's sub-block transposed into the k-major operand
        LP_CHECK(launch_transpose_f64(dkk + (size_t)ib * lda, lda, dt, m2, m2, ib, st));
        LP_CHECK(launch_dgemm_update(tk + (size_t)ib * ldt, ldt, dt, m2, tk, ldt, m2, ncols, ib, st));
    }
    return LP_OK;
}

static int left_blocked64(const double* d, int lda, double* l, int ldl, int bs, int nrows, double* lt, int ldlt,
                          cudaStream_t st) {
    if (bs <= 128) return launch_left_chunk_f64(d, lda, l, ldl, bs, nrows, lt, ldlt, st);
    const int ib = 128;
    for (int kk = 0; kk < bs / ib; kk++) {
        const double* dkk = d + (size_t)kk * ib * lda + (size_t)kk * ib;
        double* lk = l + (size_t)kk * ib;
        double* ltk = lt + (size_t)kk * ib * ldlt;
        LP_CHECK(launch_left_chunk_f64(dkk, lda, lk, ldl, ib, nrows, ltk, ldlt, st));
        const int m2 = bs - (kk + 1) * ib;
        if (m2 <= 0) break;
        // L[:, after] += L[:, chunk] * D[chunk][after]
        LP_CHECK(launch_dgemm_update(lk + ib, ldl, ltk, ldlt, dkk + ib, lda, nrows, m2, ib, st));
    }
    return LP_OK;
}

// One step of look-ahead, as gefa_f32: the next block row and column first,
// then the panel of the next step (a latency-bound chain, top on its stream and
// left beside it) on the auxiliary stream beside the update of the rest on the
// main stream.  n = 6144, block 256, against the panel behind an event: 10.3 ms
// for 10.0 of factorization; with the block column's update on left's stream,
// beside the block row's and lu, another 4 % less.
int gefa_f64(lp_ctx* c, double* a, int n, int lda, int bs, cudaStream_t st) {
    const size_t pan = (size_t)bs * n;
    LP_CHECK(c->f64lt.ensure(sizeof(double) * (2 * pan + (bs > 128 ? 2 * (size_t)128 * bs : 0))));
    double* lts[2] = {static_cast<double*>(c->f64lt.ptr), static_cast<double*>(c->f64lt.ptr) + pan};
    double* scratch = lts[1] + pan;  // bs > 128: inner Lt of the lu stage, then transposed D sub-blocks
    auto panel = [&](int k0, double* lt, cudaStream_t s) -> int {
        double* d = a + (size_t)k0 * lda + k0;
        const int rest = n - k0 - bs;
        int e = prof_begin(c, s);
        LP_CHECK(lu_stage64(d, lda, bs, scratch, s));
        LP_CHECK(prof_end(c, s, LP_STAGE_LU, e, 2.0 * bs * bs * bs / 3.0, 16.0 * bs * bs));
        if (rest <= 0) return LP_OK;
        LP_CUDA(cudaEventRecord(c->ev_side, s));
        LP_CUDA(cudaStreamWaitEvent(c->aux2, c->ev_side, 0));
        e = prof_begin(c, c->aux2);
        LP_CHECK(left_blocked64(d, lda, d + (size_t)bs * lda, lda, bs, rest, lt, rest, c->aux2));
        LP_CHECK(prof_end(c, c->aux2, LP_STAGE_LEFT, e, (double)bs * bs * rest, 24.0 * bs * rest));
        LP_CUDA(cudaEventRecord(c->ev_side_done, c->aux2));
        e = prof_begin(c, s);
        LP_CHECK(top_blocked64(d, lda, d + bs, lda, bs, rest, scratch, s));
        LP_CHECK(prof_end(c, s, LP_STAGE_TOP, e, (double)bs * bs * rest, 16.0 * bs * rest));
        LP_CUDA(cudaStreamWaitEvent(s, c->ev_side_done, 0));
        return LP_OK;
    };
    cudaStream_t aux = c->aux;
    auto update = [&](double* cc, const double* lt, const double* t, int rest, int m, int nn, cudaStream_t s) -> int {
        const int e = prof_begin(c, s);
        LP_CHECK(launch_dgemm_update(cc, lda, lt, rest, t, lda, m, nn, bs, s));
        return prof_end(c, s, LP_STAGE_INNER, e, 2.0 * m * nn * bs, 8.0 * (2.0 * m * nn + (double)bs * (m + nn)));
    };
    LP_CUDA(cudaEventRecord(c->ev_fork, st));
    LP_CUDA(cudaStreamWaitEvent(aux, c->ev_fork, 0));
    LP_CHECK(panel(0, lts[0], aux));
    for (int k0 = 0, K = 0; k0 + bs < n; k0 += bs, K++) {
        const int rest = n - k0 - bs;
        double* top = a + (size_t)k0 * lda + k0 + bs;
        double* c11 = a + (size_t)(k0 + bs) * lda + k0 + bs;
        const double* lt = lts[K & 1];
        if (K > 0) LP_CUDA(cudaStreamWaitEvent(aux, c->ev_join, 0));  // U_b of the last step
        if (rest > bs) {  // the block column: only left reads it, on the same stream
            LP_CUDA(cudaEventRecord(c->ev_side, aux));
            LP_CUDA(cudaStreamWaitEvent(c->aux2, c->ev_side, 0));
            LP_CHECK(update(c11 + (size_t)bs * lda, lt + bs, top, rest, rest - bs, bs, c->aux2));
        }
        LP_CHECK(update(c11, lt, top, rest, bs, rest, aux));
        if (rest > bs) {
            LP_CUDA(cudaEventRecord(c->ev_fork, aux));
            LP_CUDA(cudaStreamWaitEvent(st, c->ev_fork, 0));
            LP_CHECK(update(c11 + (size_t)bs * lda + bs, lt + bs, top + bs, rest, rest - bs, rest - bs, st));
            LP_CUDA(cudaEventRecord(c->ev_join, st));
        }
        LP_CHECK(panel(k0 + bs, lts[(K + 1) & 1], aux));
    }
    LP_CUDA(cudaEventRecord(c->ev_fork, aux));
    LP_CUDA(cudaStreamWaitEvent(st, c->ev_fork, 0));
    return LP_OK;
}

template <typename FT>
static int gesl64_any(lp_ctx* c, const FT* a, int n, int lda, double* b, int nrhs, int ldb, int* gave_up,
                      cudaStream_t st) {
    const int g0 = nrhs < RMAX ? nrhs : RMAX;
    LP_CHECK(c->f64w.ensure(sizeof(double) * (2 * (size_t)n * g0 + 2)));
    unsigned* sync = static_cast<unsigned*>(c->f64w.ptr);  // barrier counter, error word
    double* w1 = static_cast<double*>(c->f64w.ptr) + 2;
    double* w2 = w1 + (size_t)n * g0;
    const int e = prof_begin(c, st);
    int stall = c->stall_site == LP_STALL_GESL64;  // (failure-path tests: the first group)
    if (stall) c->stall_site = LP_STALL_NONE;
    // enough CTAs that a step's products are one pass of 32 unknowns each, at most one per SM
    const int grid = std::max(1, std::min(c->num_sms, (n + 31) / 32));
    for (int r0 = 0; r0 < nrhs; r0 += RMAX) {
        int g = nrhs - r0 < RMAX ? nrhs - r0 : RMAX;
        double* bb = b + (size_t)r0 * ldb;
        LP_CUDA(cudaMemcpy2DAsync(w1, sizeof(double) * n, bb, sizeof(double) * ldb, sizeof(double) * n, g,
                                  cudaMemcpyDeviceToDevice, st));
        LP_CUDA(cudaMemsetAsync(sync, 0, 2 * sizeof(unsigned), st));
        void* args[] = {&a, &lda, &n, &w1, &w2, &bb, &ldb, &g, &sync, &gave_up, &stall};
        LP_CUDA(cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(k_gesl64<FT>), dim3(grid), dim3(GT), args,
                                            kGesl64Smem, st));
        count_launch();
        stall = 0;
    }
    return prof_end(c, st, LP_STAGE_GESL, e, 2.0 * n * n * nrhs,
                    (double)sizeof(FT) * n * n * ((nrhs + RMAX - 1) / RMAX));
}

int gesl64_init_attrs() {
    LP_CUDA(cudaFuncSetAttribute(k_gesl64<double>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kGesl64Smem));
    LP_CUDA(cudaFuncSetAttribute(k_gesl64<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kGesl64Smem));
    return LP_OK;
}

// The host words that a substitution sets when it gives up (page-locked, so
// they can be read once the stream was waited for): [0] for lp_gesl_f64_dev,
// which does not wait, [1] for the calls that do.
static int gesl64_words(lp_ctx* c) {
    if (c->f64stat != nullptr) return LP_OK;
    LP_CUDA(cudaHostAlloc(&c->f64stat, 2 * sizeof(int), cudaHostAllocPortable));
    c->f64stat[0] = c->f64stat[1] = 0;
    return LP_OK;
}

int gesl64_status(lp_ctx* c, int slot, const char* who) {
    if (c->f64stat == nullptr) return LP_OK;
    volatile int* w = c->f64stat + slot;
    if (*w == 0) return LP_OK;
    *w = 0;
    return fail(LP_E_TIMEOUT, std::string(who) + ": a bounded wait of the FP64 substitution expired "
                                                 "(its solutions are NaN)");
}

int gesl_f64(lp_ctx* c, const double* a, int n, int lda, double* b, int nrhs, int ldb, int slot, cudaStream_t st) {
    LP_CHECK(gesl64_words(c));
    return gesl64_any(c, a, n, lda, b, nrhs, ldb, c->f64stat + slot, st);
}

int gesl_f64_on_f32(lp_ctx* c, const float* a, int n, int lda, double* b, int nrhs, int ldb, cudaStream_t st) {
    LP_CHECK(gesl64_words(c));
    return gesl64_any(c, a, n, lda, b, nrhs, ldb, c->f64stat + 1, st);
}

}  // namespace lp

using namespace lp;

extern "C" {

int lp_gefa_f64_dev(lp_ctx* c, double* dA, int n, int lda, int bs) {
    if (c == nullptr) return fail(LP_E_INVALID, "lp_gefa_f64_dev: null context");
    LP_CHECK(validate64(dA, n, lda, bs, "lp_gefa_f64_dev"));
    LP_CUDA(cudaSetDevice(c->device));
    return gefa_f64(c, dA, n, lda, bs, c->stream);
}

int lp_gesl_f64_dev(lp_ctx* c, const double* dLU, int n, int lda, double* dB, int nrhs, int ldb) {
    if (c == nullptr || dLU == nullptr || dB == nullptr) return fail(LP_E_INVALID, "lp_gesl_f64_dev: null argument");
    if (n <= 0 || lda < n || nrhs <= 0 || ldb < n) return fail(LP_E_INVALID, "lp_gesl_f64_dev: bad sizes");
    LP_CUDA(cudaSetDevice(c->device));
    return gesl_f64(c, dLU, n, lda, dB, nrhs, ldb, 0, c->stream);
}

int lp_calculate_f64(lp_ctx* c, int n, int lda, int bs, int repetitions, double* A, double* b, double* gefa_times,
                     double* gesl_times) {
    if (c == nullptr || A == nullptr || b == nullptr || gefa_times == nullptr || gesl_times == nullptr)
        return fail(LP_E_INVALID, "lp_calculate_f64: null argument");
    if (repetitions <= 0) return fail(LP_E_INVALID, "lp_calculate_f64: repetitions must be positive");
    if (n <= 0 || lda < n || lda % 2 != 0 || (bs != 64 && bs != 128 && bs != 256) || n % bs != 0)
        return fail(LP_E_INVALID, "lp_calculate_f64: n a multiple of bs (64, 128 or 256), lda >= n and even");
    LP_CUDA(cudaSetDevice(c->device));
    const size_t abytes = sizeof(double) * (size_t)n * lda;
    LP_CHECK(c->f64a.ensure(abytes));
    LP_CHECK(c->f64b.ensure(sizeof(double) * (size_t)n));
    double* dA = static_cast<double*>(c->f64a.ptr);
    double* dB = static_cast<double*>(c->f64b.ptr);
    cudaStream_t st = c->stream;
    for (int rep = 0; rep < repetitions; rep++) {
        LP_CUDA(cudaMemcpyAsync(dA, A, abytes, cudaMemcpyHostToDevice, st));
        LP_CUDA(cudaMemcpyAsync(dB, b, sizeof(double) * n, cudaMemcpyHostToDevice, st));
        LP_CUDA(cudaEventRecord(c->ev[0], st));
        LP_CHECK(gefa_f64(c, dA, n, lda, bs, st));
        LP_CUDA(cudaEventRecord(c->ev[1], st));
        LP_CHECK(gesl_f64(c, dA, n, lda, dB, 1, n, 1, st));
        LP_CUDA(cudaEventRecord(c->ev[2], st));
        LP_CUDA(cudaStreamSynchronize(st));
        LP_CHECK(gesl64_status(c, 1, "lp_calculate_f64"));
        gefa_times[rep] = event_s64(c->ev[0], c->ev[1]);
        gesl_times[rep] = event_s64(c->ev[1], c->ev[2]);
    }
    LP_CUDA(cudaMemcpyAsync(A, dA, abytes, cudaMemcpyDeviceToHost, st));
    LP_CUDA(cudaMemcpyAsync(b, dB, sizeof(double) * n, cudaMemcpyDeviceToHost, st));
    LP_CUDA(cudaStreamSynchronize(st));
    return LP_OK;
}

}  // extern "C"
