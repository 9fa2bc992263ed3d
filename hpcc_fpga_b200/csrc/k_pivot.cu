// LU with partial pivoting (LINPACK dgefa / dgesl convention) — the
// reference's gefa_ref / gesl_ref (LINPACK/src/host/linpack_data.cpp:72-156),
// used by the harness for non-diagonally-dominant ("--uniform") matrices
// (linpack_benchmark.hpp:69, 440-447).
//
// Storage S[r][c] = a[r*lda + c]; the factored matrix is M = S^T, so M's
// column k is storage row k (contiguous) and the pivot search of step k is a
// scan of one storage row.  Encoding on return (reference): diagonal u_kk,
// storage row k right of the diagonal the negated multipliers -l_ik, left of
// it U; ipvt[k] = the pivot row of step k.  In LINPACK's convention the
// interchange of step k touches only M's columns >= k, so the multipliers of
// earlier columns stay in the row order of the step that produced them.
//
// Blocked right-looking form, panel width PB (128, or 64 when a 128-wide
// panel of the tallest column does not fit the SMs' shared memory):
//   k_piv_panel  the PB columns of M (PB storage rows x the trailing length),
//                one cooperative launch: each CTA holds a slice of rows in
//                shared memory; per step it publishes its best candidate and
//                that row, all CTAs agree on the pivot (largest |v|, then
//                smallest index), the two rows are exchanged across CTAs and
//                each CTA scales and updates its rows with the reference's
//                rounding (multiplier in double, product and sum rounded to
//                float separately).
//                Inside the panel whole panel rows are exchanged ("block
//                form"); the earlier multipliers of the same panel are put
//                back into LINPACK order by k_piv_convert at the end.
//   k_piv_rows   every trailing storage row: the panel's interchanges as one
//                composite permutation (gathered, then scattered), the unit
//                lower triangular solve with the panel's diagonal block (U12),
//                and the transposed copy the trailing update reads.
//   inner        k_sgemm_update: C += U12 * L21, the same contraction as the
//                no-pivoting path (hpl_torus_PCIE.cl:711-865).
//   k_piv_gesl   forward (interchanges, then the block's triangular solve and
//                the update of everything below it, per panel) and back
//                substitution, one cooperative launch with one bounded grid
//                barrier per panel and direction.
//
// Every spin-wait is bounded: a message or barrier that does not arrive within
// the iteration limit sets the error word and every CTA returns; the host
// reports LP_E_TIMEOUT.
#include "lp_ctx.cuh"

namespace lp {
namespace {

constexpr int PT = 256;                  // threads per CTA
constexpr int GMAX = 256;                // CTAs of one panel launch, at most
constexpr int PBMAX = 128;               // panel width, at most
constexpr unsigned kSpinLimit = 1u << 21;

// Device scratch of one factorization or solve: a barrier counter, an error
// word, then the panel's messages, 64-bit words (tag << 32 | 32-bit value)
// that are valid on their own, alternating by pivot step.
constexpr int RW = PBMAX + 2;                                                          // a row and its reciprocal
constexpr size_t kKeysOff = 16;                                                        // u64 [2][GMAX]
constexpr size_t kRowsOff = kKeysOff + 2 * (size_t)GMAX * sizeof(unsigned long long);  // u64 [2][GMAX][RW]
constexpr size_t kKrowOff = kRowsOff + 2 * (size_t)GMAX * RW * sizeof(unsigned long long);  // u64 [2][PBMAX]
constexpr size_t kSyncBytes = kKrowOff + 2 * (size_t)PBMAX * sizeof(unsigned long long);

__device__ __forceinline__ unsigned ld_acquire_u32(const unsigned* p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];\n" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// Grid-wide barrier among the co-resident CTAs of a cooperative launch: the
// counter only grows; barrier number b of a launch completes at base + b * G.
// Returns false (and leaves the error word set) if it did not complete
// within the iteration limit or another CTA gave up.
__device__ __forceinline__ bool grid_sync(unsigned* bar, unsigned target, int* err) {
    __shared__ int s_ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        atomicAdd(bar, 1u);
        int ok = 1;
        unsigned spins = 0;
        while (ld_acquire_u32(bar) < target) {
            if (*reinterpret_cast<volatile int*>(err) != 0 || ++spins > kSpinLimit) {
                atomicExch(err, 1);
                ok = 0;
                break;
            }
            __nanosleep(32);
        }
        __threadfence();
        s_ok = ok;
    }
    __syncthreads();
    return s_ok != 0;
}

// Rank of M row value v in the pivot search: larger magnitudes rank higher
// (the bit pattern of a non-negative float orders like the value), equal ones
// are told apart by the index (the smaller wins, as the reference's strict "<"
// scan keeps the first).  NaN never wins, except at the diagonal itself, which
// the reference's scan then never leaves.
__device__ __forceinline__ unsigned pivot_rank(float v, bool diag) {
    const float a = fabsf(v);
    if (a != a) return diag ? 0xFFFFFFFFu : 0u;
    return __float_as_uint(a) + 1u;
}

__device__ __forceinline__ void st_word(unsigned long long* p, unsigned tag, unsigned v) {
    const unsigned long long w = ((unsigned long long)tag << 32) | v;
    asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p), "l"(w) : "memory");
}
__device__ __forceinline__ unsigned long long ld_word(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}

// A CTA's candidate in one word: its rank, its row within the CTA and the
// step (20 bits: a matrix of that order would take 4 TB).
constexpr int kKeyTagBits = 20, kKeyRowBits = 12;
__device__ __forceinline__ unsigned long long key_word(unsigned rank, unsigned row, unsigned tag) {
    return ((unsigned long long)rank << 32) | (row << kKeyTagBits) | tag;
}

// One more unsuccessful poll: false (and the error word set) past the limit or
// when another CTA gave up.
__device__ __forceinline__ bool keep_polling(unsigned& spins, unsigned limit, int* err) {
    if ((++spins & 255u) != 0) return true;
    if (*reinterpret_cast<volatile int*>(err) != 0) return false;
    if (spins > limit) {
        atomicExch(err, 1);
        return false;
    }
    return true;
}

// The value of the message word at p once it carries `tag`.
__device__ __forceinline__ unsigned poll_word(const unsigned long long* p, unsigned tag, unsigned limit, int* err,
                                              bool& ok) {
    unsigned spins = 0;
    unsigned long long w = ld_word(p);
    while ((unsigned)(w >> 32) != tag) {
        if (!keep_polling(spins, limit, err)) {
            ok = false;
            break;
        }
        w = ld_word(p);
    }
    return (unsigned)w;
}

// One panel.  A pivot step is a chain through all CTAs, so what counts is its
// latency.  Each CTA brings only the next column up to date, finds its
// candidate there and publishes it with its row (the row's other columns
// brought up to date on the way out); the rank-1 update of everything else
// runs while the messages travel.  Messages are words that carry their step,
// so a consumer needs one L2 round trip for the candidates and one for the
// winner's row, without barrier or fence.  The winner's reciprocal, a double
// division, travels with its row: it is formed while the candidates do.  Two
// buffers suffice: a CTA publishes step s + 2 only after every CTA published
// s + 1, and so had read all it needs of s.  Measured on one B200, 128 steps:
// m = 4500 855 -> 330 us (a grid barrier, then keys and row, each an L2 round
// trip, before), m = 900 280 us.
// R is a multiple of 4.  A wait of more than `limit` polls gives up: the error
// word is set and every CTA returns.  The panel's pivots start as "no exchange",
// so that the kernels already queued behind it then find valid rows in ipvt
// whatever it held before.  STALL (tests): the last CTA never sends its first
// candidate.
template <bool STALL>
__global__ void __launch_bounds__(PT, 1)
    k_piv_panel(float* __restrict__ a, int lda, int n, int k0, int kb, int R, int* __restrict__ ipvt,
                unsigned char* __restrict__ sync) {
    extern __shared__ __align__(16) float slab[];  // kb columns of M x R rows: slab[c * R + r]
    __shared__ float newk[PBMAX];    // the pivot row of the last step
    __shared__ unsigned red_v[PT / 32], red_i[PT / 32];
    __shared__ int s_p, s_ok;
    __shared__ double s_rcp;         // its -1 / pivot
    int* err = reinterpret_cast<int*>(sync + 4);
    unsigned long long* keys = reinterpret_cast<unsigned long long*>(sync + kKeysOff);
    unsigned long long* rows = reinterpret_cast<unsigned long long*>(sync + kRowsOff);
    unsigned long long* krow = reinterpret_cast<unsigned long long*>(sync + kKrowOff);
    const int G = gridDim.x, g = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int row0 = g * R;                       // M rows k0 + row0 ... belong to this CTA
    const int nr = max(0, min(R, n - k0 - row0));
    const size_t cbase = (size_t)k0 + row0;       // their storage column
    constexpr unsigned limit = STALL ? kSpinLimit / 8 : kSpinLimit;
    if (g == 0 && tid < kb) ipvt[k0 + tid] = k0 + tid;  // (kb <= PT; see above)
    for (int c = 0; c < kb; c++) {  // every copy in flight before the first wait
        const float* src = a + (size_t)(k0 + c) * lda + cbase;
        for (int r = tid; r < nr; r += PT) cp_async4(slab + c * R + r, src + r);
    }
    cp_async_wait_all();
    __syncthreads();
    for (int kk = 0; kk < kb; kk++) {
        const int k = k0 + kk, par = k & 1;
        const unsigned tag = (unsigned)k + 1u;
        const int rk = kk - row0;  // local index of M row k (in range only in its owner)
        const bool own_k = rk >= 0 && rk < nr;
        const int lo = max(0, rk);  // this CTA's rows from k on
        float* colm = slab + (kk - 1) * R;  // (kk > 0) the last step's column: its multipliers
        // the last step's multipliers (the reciprocal in double, the product rounded to float), column k up to date
        // (product and sum rounded separately), and the best row of it
        unsigned best = 0, bi = 0xFFFFFFFFu;
        {
            const double s = s_rcp;
            const float u = newk[kk];
            float* colk = slab + kk * R;
            for (int r = lo + tid; r < nr; r += PT) {
                float v = colk[r];
                if (kk > 0) {
                    const float m = (float)((double)colm[r] * s);
                    colm[r] = m;
                    v = __fadd_rn(v, __fmul_rn(m, u));
                    colk[r] = v;
                }
                const unsigned q = pivot_rank(v, r == rk);
                if (q > best) best = q, bi = (unsigned)r;  // rows in ascending order: the first stays
            }
        }
        {
            const unsigned m = __reduce_max_sync(0xffffffffu, best);
            const unsigned i = __reduce_min_sync(0xffffffffu, best == m ? bi : 0xFFFFFFFFu);
            if (lane == 0) red_v[warp] = m, red_i[warp] = i;
        }
        __syncthreads();
        {
            const unsigned v = lane < PT / 32 ? red_v[lane] : 0u, i = lane < PT / 32 ? red_i[lane] : 0xFFFFFFFFu;
            best = __reduce_max_sync(0xffffffffu, v);
            bi = __reduce_min_sync(0xffffffffu, v == best ? i : 0xFFFFFFFFu);
        }
        // publish the candidate, its panel row and, from the owner, row k
        if (tid == PT - 1 && !(STALL && kk == 0 && g == G - 1)) {
            const unsigned long long w = key_word(best, bi & ((1u << kKeyRowBits) - 1u), tag);
            asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(keys + par * GMAX + g), "l"(w) : "memory");
        }
        const int half = tid >> 7, c0 = tid & 127;
        unsigned long long* mine = rows + ((size_t)par * GMAX + g) * RW;
        if (c0 < kb && (half == 0 ? best != 0u : own_k)) {
            const int r = half == 0 ? (int)bi : rk;
            float v = slab[c0 * R + r];
            if (kk > 0 && c0 > kk) v = __fadd_rn(v, __fmul_rn(colm[r], newk[c0]));
            st_word(half == 0 ? mine + c0 : krow + par * PBMAX + c0, tag, __float_as_uint(v));
        }
        if (warp == 1 && best != 0u && lane == 0) {
            const double s = -1.0 / (double)slab[kk * R + (int)bi];
            st_word(mine + PBMAX, tag, (unsigned)__double2loint(s));
            st_word(mine + PBMAX + 1, tag, (unsigned)__double2hiint(s));
        }
        __syncthreads();  // the rows above are read before the update below changes them
        if (warp == 0) {
            constexpr int KQ = GMAX / 32;
            bool ok = true;
            unsigned long long w[KQ];
#pragma unroll
            for (int j = 0; j < KQ; j++)  // every candidate's word in flight at once
                w[j] = lane + 32 * j < G ? ld_word(keys + par * GMAX + lane + 32 * j) : tag;
            unsigned v = 0, i = 0xFFFFFFFFu;
#pragma unroll
            for (int j = 0; j < KQ; j++) {
                const int q = lane + 32 * j;
                if (q < G) {
                    unsigned spins = 0;
                    while (((unsigned)w[j] & ((1u << kKeyTagBits) - 1u)) != tag && ok) {
                        ok = keep_polling(spins, limit, err);
                        w[j] = ld_word(keys + par * GMAX + q);
                    }
                    const unsigned x = (unsigned)(w[j] >> 32), y = (unsigned)(k0 + q * R) + ((unsigned)w[j] >> kKeyTagBits);
                    if (x > v || (x == v && y < i)) v = x, i = y;
                }
            }
            const unsigned m = __reduce_max_sync(0xffffffffu, v);
            const unsigned im = __reduce_min_sync(0xffffffffu, v == m ? i : 0xFFFFFFFFu);
            const int all = __all_sync(0xffffffffu, ok);
            if (lane == 0) s_p = (int)im, s_ok = all;
        } else if (kk > 0) {
            // rank-1 update of the panel's later columns (product and sum rounded separately): a warp takes every
            // seventh column, a lane four rows, four columns' loads in flight
            constexpr int CB = 4, CS = PT / 32 - 1;
            for (int r = 4 * lane; r < nr; r += 128) {
                if (r + 3 < lo) continue;
                const float4 m = *reinterpret_cast<const float4*>(colm + r);
                for (int c = kk + warp; c < kb; c += CB * CS) {
                    float4 x[CB];
                    float u[CB];
#pragma unroll
                    for (int j = 0; j < CB; j++)
                        if (c + j * CS < kb) {
                            x[j] = *reinterpret_cast<const float4*>(slab + (c + j * CS) * R + r);
                            u[j] = newk[c + j * CS];
                        }
#pragma unroll
                    for (int j = 0; j < CB; j++)
                        if (c + j * CS < kb) {
                            if (r >= lo) x[j].x = __fadd_rn(x[j].x, __fmul_rn(m.x, u[j]));
                            if (r + 1 >= lo) x[j].y = __fadd_rn(x[j].y, __fmul_rn(m.y, u[j]));
                            if (r + 2 >= lo) x[j].z = __fadd_rn(x[j].z, __fmul_rn(m.z, u[j]));
                            x[j].w = __fadd_rn(x[j].w, __fmul_rn(m.w, u[j]));
                            *reinterpret_cast<float4*>(slab + (c + j * CS) * R + r) = x[j];
                        }
                }
            }
        }
        __syncthreads();
        if (!s_ok) return;
        const int p = s_p, wg = (p - k0) / R, rp = p - (int)cbase;
        const bool own_p = p != k && rp >= 0 && rp < nr;
        bool ok = true;
        const unsigned long long* won = rows + ((size_t)par * GMAX + wg) * RW;
        if (c0 < kb) {
            if (half == 0) {
                const float v = __uint_as_float(poll_word(won + c0, tag, limit, err, ok));
                newk[c0] = v;
                if (p != k && own_k) slab[c0 * R + rk] = v;  // exchange M rows k and p over the whole panel
            } else if (own_p) {
                slab[c0 * R + rp] = __uint_as_float(poll_word(krow + par * PBMAX + c0, tag, limit, err, ok));
            }
        }
        if (warp == PT / 32 - 1) {  // the reciprocal, by two lanes
            const unsigned h = lane < 2 ? poll_word(won + PBMAX + lane, tag, limit, err, ok) : 0u;
            const unsigned hi = __shfl_sync(0xffffffffu, h, 1);
            if (lane == 0) s_rcp = __hiloint2double((int)hi, (int)h);
        }
        if (g == 0 && tid == 0) ipvt[k] = p;
        if (!__syncthreads_and(ok)) return;
    }
    // the last column's multipliers
    {
        const double s = s_rcp;
        for (int r = max(0, kb - row0) + tid; r < nr; r += PT)
            slab[(kb - 1) * R + r] = (float)((double)slab[(kb - 1) * R + r] * s);
    }
    __syncthreads();
    for (int c = 0; c < kb; c++) {
        float* dst = a + (size_t)(k0 + c) * lda + cbase;
        for (int r = tid; r < nr; r += PT) dst[r] = slab[c * R + r];
    }
}

// The interchanges of one panel (M rows k0 .. k0+kb-1 with ipvt) as one
// composite permutation: after it, panel position k0+t holds the value that
// was at psrc[t], and outside position odst[e] (>= r0) the value that was at
// osrc[e].  Every position is traced back through the interchanges by a thread
// of its own, the outside ones (distinct ipvt values beyond the panel) by the
// first step that names them.  pv: the panel's ipvt entries in shared memory;
// all threads of the block.
__device__ void build_perm(const int* pv, int k0, int kb, int r0, int* psrc, int* odst, int* osrc, int* s_nout) {
    auto trace = [&](int pos) {
        for (int kk = kb - 1; kk >= 0; kk--) {
            const int p = pv[kk], q = k0 + kk;
            pos = pos == q ? p : (pos == p ? q : pos);
        }
        return pos;
    };
    for (int t = threadIdx.x; t < kb; t += blockDim.x) psrc[t] = trace(k0 + t);
    if (threadIdx.x < 32) {
        int nout = 0;
        for (int b = 0; b < kb; b += 32) {
            const int t = b + threadIdx.x;
            bool first = t < kb && pv[t] >= r0;
            for (int u = 0; first && u < t; u++) first = pv[u] != pv[t];
            const unsigned who = __ballot_sync(0xffffffffu, first);
            if (first) odst[nout + __popc(who & ((1u << threadIdx.x) - 1u))] = pv[t];
            nout += __popc(who);
        }
        if (threadIdx.x == 0) *s_nout = nout;
    }
    __syncthreads();
    for (int e = threadIdx.x; e < *s_nout; e += blockDim.x) osrc[e] = trace(odst[e]);
}

// Trailing storage rows [r0 + first, r0 + last) (M's trailing columns): interchanges, then
// x_t += L[k][t] x_k (t > k) with the panel's unit lower block, written in
// place and transposed into at (at[t * ldat + c - r0]).  One warp per row.
template <int PB>
__global__ void __launch_bounds__(PT)
    k_piv_rows(float* __restrict__ a, int lda, int k0, int first, int last, const int* __restrict__ ipvt,
               float* __restrict__ at, int ldat) {
    constexpr int Q = PB / 32, SS = PB + 4;
    extern __shared__ float sm[];
    float* L = sm;               // L[k * PB + t] = S[k0 + k][k0 + t]
    float* stage = L + PB * PB;  // 8 rows x SS
    __shared__ int pv[PB], psrc[PB], odst[PB], osrc[PB];
    __shared__ int s_nout;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int r0 = k0 + PB;
    for (int t = tid; t < PB; t += PT) pv[t] = ipvt[k0 + t];
    for (int idx = tid; idx < PB * PB; idx += PT) {
        const int k = idx / PB, t = idx - k * PB;
        cp_async4(L + idx, a + (size_t)(k0 + k) * lda + k0 + t);
    }
    cp_async_wait_all();
    __syncthreads();
    build_perm(pv, k0, PB, r0, psrc, odst, osrc, &s_nout);
    __syncthreads();
    const int nout = s_nout;
    for (int base = first + blockIdx.x * 8; base < last; base += gridDim.x * 8) {
        const int c = r0 + base + warp;
        if (base + warp < last) {
            float* row = a + (size_t)c * lda;
            float x[Q], ov[Q];
#pragma unroll
            for (int q = 0; q < Q; q++) {
                const int e = lane + 32 * q;
                x[q] = row[psrc[e]];
                ov[q] = e < nout ? row[osrc[e]] : 0.0f;
            }
            __syncwarp();
#pragma unroll
            for (int q = 0; q < Q; q++) {
                const int e = lane + 32 * q;
                if (e < nout) row[odst[e]] = ov[q];
            }
#pragma unroll
            for (int k = 0; k < PB; k++) {
                const float xk = __shfl_sync(0xffffffffu, x[k >> 5], k & 31);
#pragma unroll
                for (int q = 0; q < Q; q++) {
                    const int t = lane + 32 * q;
                    if (t > k) x[q] = fmaf(L[k * PB + t], xk, x[q]);
                }
            }
#pragma unroll
            for (int q = 0; q < Q; q++) {
                row[k0 + lane + 32 * q] = x[q];
                stage[warp * SS + lane + 32 * q] = x[q];
            }
        }
        __syncthreads();
        for (int idx = tid; idx < PB * 8; idx += PT) {
            const int t = idx >> 3, j = idx & 7;
            if (base + j < last) at[(size_t)t * ldat + base + j] = stage[j * SS + t];
        }
        __syncthreads();
    }
}

// One composite permutation per panel (layout: psrc[PB], odst[PB], osrc[PB],
// count at [3 PB]), one block per panel.
template <int PB>
__global__ void k_piv_desc(const int* __restrict__ ipvt, int n, int* __restrict__ desc) {
    __shared__ int pv[PB], psrc[PB], odst[PB], osrc[PB];
    __shared__ int s_nout;
    const int j = blockIdx.x, k0 = j * PB, kb = min(PB, n - k0);
    for (int t = threadIdx.x; t < kb; t += blockDim.x) pv[t] = ipvt[k0 + t];
    __syncthreads();
    build_perm(pv, k0, kb, k0 + kb, psrc, odst, osrc, &s_nout);
    __syncthreads();
    int* d = desc + (size_t)j * 4 * PB;
    for (int t = threadIdx.x; t < PB; t += blockDim.x) {
        d[t] = t < kb ? psrc[t] : k0 + t;
        d[PB + t] = odst[t];
        d[2 * PB + t] = osrc[t];
    }
    if (threadIdx.x == 0) d[3 * PB] = s_nout;
}

// Between block form (whole panel rows exchanged inside a panel) and the
// reference encoding: storage row kp's multipliers take the interchanges of
// the later steps of its own panel (to block form, in step order) or give
// them back (to the reference encoding, in reverse order).  One thread per
// storage row.
__global__ void k_piv_convert(float* __restrict__ a, int lda, int n, int pb, const int* __restrict__ ipvt,
                              int to_reference) {
    const int kp = blockIdx.x * blockDim.x + threadIdx.x;
    if (kp >= n) return;
    const int kend = min((kp / pb + 1) * pb, n);
    float* row = a + (size_t)kp * lda;
    if (to_reference) {
        for (int k = kend - 1; k > kp; k--) {
            const int p = __ldg(ipvt + k);
            if (p != k) {
                const float t = row[k];
                row[k] = row[p];
                row[p] = t;
            }
        }
    } else {
        for (int k = kp + 1; k < kend; k++) {
            const int p = __ldg(ipvt + k);
            if (p != k) {
                const float t = row[k];
                row[k] = row[p];
                row[p] = t;
            }
        }
    }
}

// One warp's share of the products with a block's rows: the sums over rows
// [16 part, +16) of ys[t] S[k0 + t][i], lane = column; all 16 loads in flight
// before they are used.
struct DotRows {
    float v[16];
    __device__ __forceinline__ void load(const float* __restrict__ a, int lda, int k0, int kb, int part, int i, bool in) {
        const float* col = a + (size_t)(k0 + 16 * part) * lda + i;
#pragma unroll
        for (int j = 0; j < 16; j++) v[j] = in && 16 * part + j < kb ? __ldg(col + (size_t)j * lda) : 0.0f;
    }
    __device__ __forceinline__ float dot(const float* ys) const {
        float s = 0.0f;
#pragma unroll
        for (int j = 0; j < 16; j++) s = fmaf(ys[j], v[j], s);
        return s;
    }
};

// The block's diagonal block into D (row stride PB), 16-byte copies where the
// rows allow them (k0 is a multiple of PB).
template <int PB>
__device__ __forceinline__ void stage_diag(float* D, const float* __restrict__ a, int lda, int k0, int kb, bool vec) {
    const float* src = a + (size_t)k0 * lda + k0;
    if (vec && kb == PB) {
        for (int idx = threadIdx.x; idx < PB * PB / 4; idx += PT) {
            const int k = idx / (PB / 4), t = (idx % (PB / 4)) * 4;
            cp_async_vec16(D + k * PB + t, src + (size_t)k * lda + t);
        }
    } else {
        for (int idx = threadIdx.x; idx < kb * kb; idx += PT) {
            const int k = idx / kb, t = idx - k * kb;
            cp_async4(D + k * PB + t, src + (size_t)k * lda + t);
        }
    }
}

// Forward and back substitution on block-form factors, nrhs right-hand
// sides (rows of b, solutions overwrite them).  w: 3 n floats (the forward
// values y, two alternating trailing vectors).  Per panel every CTA computes
// the block's values itself (warp 0, from the diagonal block staged in
// shared memory), then updates its share of the positions after (forward) or
// before (backward) the block; one grid barrier per panel.  A chain of two
// panels' work per barrier, so latency counts: the next diagonal block is
// copied in and the first products' rows are loaded before the barrier, and
// the 128 terms of a position are split over eight warps (n = 5000: 2.46 ms ->
// 1.02; one thread per position and 40 CTAs before).
template <int PB>
__global__ void __launch_bounds__(PT, 1)
    k_piv_gesl(const float* __restrict__ a, int lda, int n, const int* __restrict__ desc, float* b, int ldb, int nrhs,
               float* w, unsigned char* __restrict__ sync) {
    constexpr int Q = PB / 32, NP = PB / 16;  // NP warps share the terms of a position (the others idle there)
    extern __shared__ __align__(16) float sm[];
    float* Dbuf = sm;                                     // 2 x PB x PB diagonal blocks, alternating
    int* ovr = reinterpret_cast<int*>(Dbuf + 2 * PB * PB);  // this CTA's positions: override source or -1
    __shared__ float ys[PB], part[NP][32], rd[PB];
    __shared__ int od[PB], os[PB];
    __shared__ int ps[PB];
    __shared__ int s_nout;
    unsigned* bar = reinterpret_cast<unsigned*>(sync);
    int* err = reinterpret_cast<int*>(sync + 4);
    const int G = gridDim.x, g = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int np = (n + PB - 1) / PB;
    const bool vec = (lda & 3) == 0 && (reinterpret_cast<uintptr_t>(a) & 15u) == 0;
    unsigned nbar = 0;
    float* y = w;
    float* buf0 = w + n;
    float* buf1 = w + 2 * (size_t)n;
    // this CTA's positions of panel j: [i0, i1) after (forward) or before (backward) the block
    auto range = [&](int j, bool fwd, int& i0, int& i1) {
        const int k0 = j * PB, lo = fwd ? min(n, k0 + PB) : 0, hi = fwd ? n : k0, ch = (hi - lo + G - 1) / G;
        i0 = min(hi, lo + g * ch);
        i1 = min(hi, i0 + ch);
    };
    // dst[i] = src[i] (or its override) + sgn * sum_t ys[t] S[k0 + t][i] over [i0, i1); pre: the first group's rows
    auto products = [&](int j, int i0, int i1, float sgn, DotRows& pre, const float* src, const int* over, float* dst) {
        const int k0 = j * PB, kb = min(PB, n - k0);
        for (int ib = i0; ib < i1; ib += 32) {
            const int i = ib + lane;
            if (warp < NP) {
                if (ib != i0) pre.load(a, lda, k0, kb, warp, i, i < i1);
                part[warp][lane] = pre.dot(ys + 16 * warp);
            }
            __syncthreads();
            if (warp == 0 && i < i1) {
                float s = 0.0f;
#pragma unroll
                for (int q = 0; q < NP; q++) s += part[q][lane];
                const int o = over != nullptr ? over[i - i0] : -1;
                dst[i] = __ldcg(src + (o >= 0 ? o : i)) + sgn * s;
            }
            __syncthreads();
        }
    };
    for (int q = 0; q < nrhs; q++) {
        float* bq = b + (size_t)q * ldb;
        DotRows pre;
        int i0, i1;
        // forward: phase j reads cur, writes nxt (positions after the block) and y (the block)
        stage_diag<PB>(Dbuf, a, lda, 0, min(PB, n), vec);
        range(0, true, i0, i1);
        if (warp < NP) pre.load(a, lda, 0, min(PB, n), warp, i0 + lane, i0 + lane < i1);
        for (int j = 0; j < np; j++) {
            const int k0 = j * PB, kb = min(PB, n - k0);
            const float* cur = j == 0 ? bq : ((j & 1) ? buf0 : buf1);
            float* nxt = (j & 1) ? buf1 : buf0;
            const float* D = Dbuf + (j & 1) * PB * PB;
            const int* dj = desc + (size_t)j * 4 * PB;
            for (int t = tid; t < PB; t += PT) {
                ps[t] = dj[t], od[t] = dj[PB + t], os[t] = dj[2 * PB + t];
                ys[t] = 0.0f;
            }
            if (tid == 0) s_nout = dj[3 * PB];
            cp_async_wait_all();
            for (int i = tid; i < i1 - i0; i += PT) ovr[i] = -1;
            __syncthreads();
            const int nout = s_nout;
            for (int e = tid; e < nout; e += PT) {
                const int d = od[e];
                if (d >= i0 && d < i1) ovr[d - i0] = os[e];
            }
            // the next diagonal block on its way: the forward sweep's, or the backward sweep's first (this last one)
            if (j + 1 < np) stage_diag<PB>(Dbuf + ((j + 1) & 1) * PB * PB, a, lda, k0 + PB, min(PB, n - k0 - PB), vec);
            if (warp == 0) {
                float x[Q];
#pragma unroll
                for (int qq = 0; qq < Q; qq++) {
                    const int t = lane + 32 * qq;
                    x[qq] = t < kb ? __ldcg(cur + ps[t]) : 0.0f;
                }
#pragma unroll
                for (int k = 0; k < PB; k++) {
                    const float xk = __shfl_sync(0xffffffffu, x[k >> 5], k & 31);
#pragma unroll
                    for (int qq = 0; qq < Q; qq++) {
                        const int t = lane + 32 * qq;
                        if (t > k && t < kb) x[qq] = fmaf(xk, D[k * PB + t], x[qq]);
                    }
                }
#pragma unroll
                for (int qq = 0; qq < Q; qq++) {
                    const int t = lane + 32 * qq;
                    if (t < kb) {
                        ys[t] = x[qq];
                        if (g == 0) y[k0 + t] = x[qq];
                    }
                }
            }
            __syncthreads();
            products(j, i0, i1, 1.0f, pre, cur, ovr, nxt);
            if (j + 1 < np) {
                range(j + 1, true, i0, i1);
                if (warp < NP) pre.load(a, lda, k0 + PB, min(PB, n - k0 - PB), warp, i0 + lane, i0 + lane < i1);
            } else {
                range(np - 1, false, i0, i1);
                if (warp < NP) pre.load(a, lda, k0, kb, warp, i0 + lane, i0 + lane < i1);
            }
            if (!grid_sync(bar, (++nbar) * (unsigned)G, err)) return;
        }
        // backward: x_k = y_k / u_kk; y_t -= x_k u_tk (t < k).  Block j's diagonal block is in buffer j & 1, as in
        // the forward sweep; the last one is still there.
        for (int j = np - 1; j >= 0; j--) {
            const int k0 = j * PB, kb = min(PB, n - k0);
            const float* D = Dbuf + (j & 1) * PB * PB;
            cp_async_wait_all();
            __syncthreads();
            for (int t = tid; t < PB; t += PT) {
                ys[t] = 0.0f;
                rd[t] = t < kb ? __frcp_rn(D[t * PB + t]) : 0.0f;
            }
            if (j > 0) stage_diag<PB>(Dbuf + ((j - 1) & 1) * PB * PB, a, lda, k0 - PB, PB, vec);
            __syncthreads();
            if (warp == 0) {
                float x[Q];
#pragma unroll
                for (int qq = 0; qq < Q; qq++) {
                    const int t = lane + 32 * qq;
                    x[qq] = t < kb ? __ldcg(y + k0 + t) : 0.0f;
                }
#pragma unroll
                for (int k = PB - 1; k >= 0; k--) {
                    if (k < kb) {
                        // the quotient: the product with the reciprocal and one correction; where that is not finite
                        // (a zero or infinite pivot, overflow) the division itself
                        const float v = __shfl_sync(0xffffffffu, x[k >> 5], k & 31), d = D[k * PB + k], r = rd[k];
                        const float q0 = v * r;
                        float xk = fmaf(fmaf(-q0, d, v), r, q0);
                        if (!(fabsf(xk) < 3.0e38f)) xk = v / d;
                        if (lane == (k & 31)) x[k >> 5] = xk;
#pragma unroll
                        for (int qq = 0; qq < Q; qq++) {
                            const int t = lane + 32 * qq;
                            if (t < k) x[qq] = fmaf(-xk, D[k * PB + t], x[qq]);
                        }
                    }
                }
#pragma unroll
                for (int qq = 0; qq < Q; qq++) {
                    const int t = lane + 32 * qq;
                    if (t < kb) {
                        ys[t] = x[qq];
                        if (g == 0) bq[k0 + t] = x[qq];
                    }
                }
            }
            __syncthreads();
            products(j, i0, i1, -1.0f, pre, y, nullptr, y);
            if (j > 0) {
                range(j - 1, false, i0, i1);
                if (warp < NP) pre.load(a, lda, k0 - PB, PB, warp, i0 + lane, i0 + lane < i1);
            }
            if (!grid_sync(bar, (++nbar) * (unsigned)G, err)) return;
        }
    }
}

int g_panel_smem_max = 0;  // dynamic shared memory available to k_piv_panel
int g_gesl_smem_max = 0;

template <int PB>
constexpr size_t rows_smem() {
    return sizeof(float) * ((size_t)PB * PB + 8 * (PB + 4));
}

}  // namespace

int piv_init_attrs() {
    int dev = 0, optin = 0;
    LP_CUDA(cudaGetDevice(&dev));
    LP_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    cudaFuncAttributes fa{};
    LP_CUDA(cudaFuncGetAttributes(&fa, k_piv_panel<false>));
    g_panel_smem_max = optin - (int)fa.sharedSizeBytes;
    LP_CUDA(cudaFuncSetAttribute(k_piv_panel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, g_panel_smem_max));
    LP_CUDA(cudaFuncSetAttribute(k_piv_panel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, g_panel_smem_max));
    LP_CUDA(cudaFuncSetAttribute(k_piv_rows<128>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)rows_smem<128>()));
    LP_CUDA(cudaFuncSetAttribute(k_piv_rows<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)rows_smem<64>()));
    LP_CUDA(cudaFuncGetAttributes(&fa, k_piv_gesl<128>));
    g_gesl_smem_max = optin - (int)fa.sharedSizeBytes;
    LP_CUDA(cudaFuncSetAttribute(k_piv_gesl<128>, cudaFuncAttributeMaxDynamicSharedMemorySize, g_gesl_smem_max));
    LP_CUDA(cudaFuncGetAttributes(&fa, k_piv_gesl<64>));
    LP_CUDA(cudaFuncSetAttribute(k_piv_gesl<64>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 optin - (int)fa.sharedSizeBytes));
    return LP_OK;
}

size_t piv_sync_bytes() { return kSyncBytes; }

int piv_panel_width(int n, int sms) {
    const long long rows = ((n + sms - 1) / sms + 3) / 4 * 4;
    return rows * 128 * (long long)sizeof(float) <= g_panel_smem_max ? 128 : 64;
}

// CTAs and rows per CTA of the panel launch for m trailing rows: about 128
// rows per CTA, at most one CTA per SM, the slice within shared memory.
static void panel_grid(int m, int kb, int sms, int* G, int* R) {
    int g = std::min(sms, std::max(1, (m + 127) / 128));
    auto rows = [&]() { return ((m + g - 1) / g + 3) / 4 * 4; };
    while ((long long)rows() * kb * (long long)sizeof(float) > g_panel_smem_max && g < sms) g = std::min(sms, g * 2);
    *R = rows();
    *G = (m + *R - 1) / *R;
}

// stall (tests): the first pivot step's wait runs out, after some 0.2 s.
int launch_piv_panel(float* a, int lda, int n, int k0, int kb, int* ipvt, unsigned char* sync, bool stall, int sms,
                     cudaStream_t st) {
    const int m = n - k0;
    int G = 0, R = 0;
    panel_grid(m, kb, sms, &G, &R);
    const size_t smem = (size_t)kb * R * sizeof(float);
    if (kb > PBMAX || G > GMAX || R >= 1 << kKeyRowBits || n >= 1 << kKeyTagBits || (long long)smem > g_panel_smem_max)
        return fail(LP_E_INVALID, "pivoting panel: matrix too large for the panel width");
    void* args[] = {&a, &lda, &n, &k0, &kb, &R, &ipvt, &sync};
    const void* fn = stall ? reinterpret_cast<const void*>(k_piv_panel<true>)
                           : reinterpret_cast<const void*>(k_piv_panel<false>);
    LP_CUDA(cudaLaunchCooperativeKernel(fn, dim3(G), dim3(PT), args, smem, st));
    count_launch();
    return LP_OK;
}

// Storage rows [r0 + first, r0 + last) of the trailing matrix, r0 = k0 + pb.
int launch_piv_rows(float* a, int lda, int k0, int pb, int first, int last, const int* ipvt, float* at, int ldat,
                    int sms, cudaStream_t st) {
    if (last <= first) return LP_OK;
    const int grid = std::max(1, std::min(2 * sms, (last - first + 7) / 8));
    if (pb == 128)
        k_piv_rows<128><<<grid, PT, rows_smem<128>(), st>>>(a, lda, k0, first, last, ipvt, at, ldat);
    else
        k_piv_rows<64><<<grid, PT, rows_smem<64>(), st>>>(a, lda, k0, first, last, ipvt, at, ldat);
    count_launch();
    LP_CUDA(cudaGetLastError());
    return LP_OK;
}

int launch_piv_desc(const int* ipvt, int n, int pb, int* desc, cudaStream_t st) {
    const int np = (n + pb - 1) / pb;
    if (pb == 128)
        k_piv_desc<128><<<np, 128, 0, st>>>(ipvt, n, desc);
    else
        k_piv_desc<64><<<np, 128, 0, st>>>(ipvt, n, desc);
    count_launch();
    LP_CUDA(cudaGetLastError());
    return LP_OK;
}

int launch_piv_convert(float* a, int lda, int n, int pb, const int* ipvt, bool to_reference, cudaStream_t st) {
    k_piv_convert<<<(n + 127) / 128, 128, 0, st>>>(a, lda, n, pb, ipvt, to_reference ? 1 : 0);
    count_launch();
    LP_CUDA(cudaGetLastError());
    return LP_OK;
}

int launch_piv_gesl(const float* a, int lda, int n, int pb, const int* desc, float* b, int ldb, int nrhs, float* w,
                    unsigned char* sync, int sms, cudaStream_t st) {
    const int G = std::max(1, std::min(sms, (n + 31) / 32));
    const size_t smem = sizeof(float) * 2 * (size_t)pb * pb + sizeof(int) * (size_t)((n + G - 1) / G);
    if ((long long)smem > g_gesl_smem_max) return fail(LP_E_INVALID, "pivoting solve: matrix too large");
    void* args[] = {&a, &lda, &n, &desc, &b, &ldb, &nrhs, &w, &sync};
    const void* fn = pb == 128 ? reinterpret_cast<const void*>(k_piv_gesl<128>)
                               : reinterpret_cast<const void*>(k_piv_gesl<64>);
    LP_CUDA(cudaLaunchCooperativeKernel(fn, dim3(G), dim3(PT), args, smem, st));
    count_launch();
    return LP_OK;
}

}  // namespace lp
