// Panel kernels of the FP32 and tensor-core schedules: the LU of a 128 x 128
// diagonal block and the triangular updates of the block row and column
// beside it.  They compute the recurrences of k_lu.cu / k_trsm.cu (gefa's lu,
// top and left, LINPACK/src/host/linpack_data.cpp:166-196) with fused
// multiply-adds and sums in another order, so their results agree with those to
// rounding; the entry points that promise the reference's exact operation order
// (lp_lu_block_dev up to 128, lp_top_update_dev, lp_left_update_dev) keep the
// other kernels.
//
// k_lu128 is a chain of 128 dependent pivots on one SM, so what counts is the
// latency per pivot.  Eight worker warps hold the block in registers (8 x 8
// per thread) and factor it 8 columns at a time: 128 of their threads finish
// one row of the block column each, the other 128 one column of the block
// row, then all apply the rank-8 update from shared memory.  Meanwhile the
// diagonal warp brings the next 8 x 8 diagonal block up to date and factors
// it, redundantly in every lane's registers (a chain of eight reciprocals
// without an exchange between threads).  It has an SM partition to itself:
// beside two workers on one scheduler its instructions wait for theirs.
// Measured on one B200 per block, beside 31 us for k_lu_block<128>: 19.6 us.
//
// k_tl applies top and left to strips of 32 or 64 columns / rows, all bs of
// the block's unknowns at once.  With X the strip (left: transposed) each
// 32-wide chunk c of it becomes X0_c + sum_{b<c} D_cb X_b and then runs the
// recurrence of its own triangle, one column per lane (solve32): a product with
// the triangle's inverse in its place was 1 us shorter per 128 rows, but lost
// what the condition of the triangle allows on matrices that are not dominant,
// and the inversions cost k_lu128 2 us.  One launch covers the block row and the
// block column (they are independent), the strip stays in shared memory, and
// per 128 rows a thread keeps its outputs in registers.  9.9 us beside a 128
// block (384 rows and columns), 22.6 us beside 256 and 61 us beside 512 (512
// rows and columns), where top and left took 13 us each beside 128 and a chain
// of such launches, transposes and GEMMs beside wider blocks.  The whole chain of
// a 128 step (LU, top and left, update of the 384 behind it): 36 us, was 70.
#include "lp_ctx.cuh"

namespace lp {
namespace {

constexpr int PB = 128;     // block
constexpr int PS = PB + 4;  // row stride of the panels in shared memory

__device__ __forceinline__ float2 fma2(float a, float2 b, float2 c) { return __ffma2_rn(make_float2(a, a), b, c); }

template <int ID, int COUNT>
__device__ __forceinline__ void bar_sync() { asm volatile("bar.sync %0, %1;\n" ::"n"(ID), "n"(COUNT) : "memory"); }

// -1 / x, correctly rounded over the whole range of floats, as in the exact
// kernels: an approximate reciprocal flushes subnormal results, so that a pivot
// above 2^126 would get multipliers of zero.  0.3 us more per 128 pivots than
// that reciprocal and one Newton step.
__device__ __forceinline__ float neg_rcp(float x) { return -__frcp_rn(x); }

__device__ __forceinline__ void ld4(float* d, const float* s) {
    const float4 v = *reinterpret_cast<const float4*>(s);
    d[0] = v.x, d[1] = v.y, d[2] = v.z, d[3] = v.w;
}

// Rank-8 update of a thread's piece with the panels Ls (8 x PS, row of the
// block) and Ts (8 x PS, column of the block): its low (R0) and high rows, its
// low (C0) and high columns.  Shared memory delivers 128 bytes a clock to the
// registers whether lanes share addresses or not, so 8 x 8 outputs per 16
// loaded values keep the loads just level with the FMA pipe.
template <bool R0, bool C0>
__device__ __forceinline__ void rank8(float2 (&c)[2][4][4], const float* Ls, const float* Ts) {
#pragma unroll
    for (int k = 0; k < 8; k++) {
        const float4 t1 = *reinterpret_cast<const float4*>(Ts + k * PS + 64);
        float4 t0 = t1;
        if (C0) t0 = *reinterpret_cast<const float4*>(Ts + k * PS);
#pragma unroll
        for (int h = R0 ? 0 : 1; h < 2; h++) {
            const float4 l = *reinterpret_cast<const float4*>(Ls + k * PS + 64 * h);
            const float la[4] = {l.x, l.y, l.z, l.w};
#pragma unroll
            for (int i = 0; i < 4; i++) {
                if (C0) {
                    c[h][i][0] = fma2(la[i], make_float2(t0.x, t0.y), c[h][i][0]);
                    c[h][i][1] = fma2(la[i], make_float2(t0.z, t0.w), c[h][i][1]);
                }
                c[h][i][2] = fma2(la[i], make_float2(t1.x, t1.y), c[h][i][2]);
                c[h][i][3] = fma2(la[i], make_float2(t1.z, t1.w), c[h][i][3]);
            }
        }
    }
}

// Four rows of a thread's piece into the block row's panel.
__device__ __forceinline__ void store_rows(float* dst, const float2 (&c)[4][4]) {
#pragma unroll
    for (int i = 0; i < 4; i++) {
        *reinterpret_cast<float4*>(dst + i * PS) = make_float4(c[i][0].x, c[i][0].y, c[i][1].x, c[i][1].y);
        *reinterpret_cast<float4*>(dst + i * PS + 64) = make_float4(c[i][2].x, c[i][2].y, c[i][3].x, c[i][3].y);
    }
}

// Four columns (pairs P0, P0 + 1) of four rows into the block column's panel.
template <int P0>
__device__ __forceinline__ void store_cols(float* dst, const float2 (&c)[4][4]) {
    *reinterpret_cast<float4*>(dst) = make_float4(c[0][P0].x, c[1][P0].x, c[2][P0].x, c[3][P0].x);
    *reinterpret_cast<float4*>(dst + PS) = make_float4(c[0][P0].y, c[1][P0].y, c[2][P0].y, c[3][P0].y);
    *reinterpret_cast<float4*>(dst + 2 * PS) = make_float4(c[0][P0 + 1].x, c[1][P0 + 1].x, c[2][P0 + 1].x, c[3][P0 + 1].x);
    *reinterpret_cast<float4*>(dst + 3 * PS) = make_float4(c[0][P0 + 1].y, c[1][P0 + 1].y, c[2][P0 + 1].y, c[3][P0 + 1].y);
}

// A 4 x 4 quarter of an 8 x 8 diagonal block (row stride 8).
template <int P0>
__device__ __forceinline__ void store_diag(float* dst, const float2 (&c)[4][4]) {
#pragma unroll
    for (int i = 0; i < 4; i++)
        *reinterpret_cast<float4*>(dst + 8 * i) = make_float4(c[i][P0].x, c[i][P0].y, c[i][P0 + 1].x, c[i][P0 + 1].y);
}

// rank-8 contribution of the panels to the 8 x 8 diagonal block at row q0, two
// neighbouring elements per lane, added to dg (row-major).
__device__ __forceinline__ void diag_rank8(float* dg, const float* Ls, const float* Ts, int q0, int lane) {
    const int r = lane >> 2, i = 2 * (lane & 3);
    float2* p = reinterpret_cast<float2*>(dg + 8 * r + i);
    float2 v = *p;
#pragma unroll
    for (int k = 0; k < 8; k++)
        v = fma2(Ls[k * PS + q0 + r], *reinterpret_cast<const float2*>(Ts + k * PS + q0 + i), v);
    *p = v;
}

// The 8 x 8 block at dg factored in every lane's registers (lane 0 writes it
// to fd).
__device__ __forceinline__ void diag_lu8(const float* dg, float* fd, int lane) {
    float d[8][8];
#pragma unroll
    for (int j = 0; j < 8; j++) {
        const float4 u = *reinterpret_cast<const float4*>(dg + 8 * j);
        const float4 v = *reinterpret_cast<const float4*>(dg + 8 * j + 4);
        d[j][0] = u.x, d[j][1] = u.y, d[j][2] = u.z, d[j][3] = u.w;
        d[j][4] = v.x, d[j][5] = v.y, d[j][6] = v.z, d[j][7] = v.w;
    }
#pragma unroll
    for (int k = 0; k < 8; k++) {
        const float r = neg_rcp(d[k][k]);
        d[k][k] = r;
#pragma unroll
        for (int i = k + 1; i < 8; i++) d[k][i] *= r;
#pragma unroll
        for (int j = k + 1; j < 8; j++)
#pragma unroll
            for (int i = k + 1; i < 8; i++) d[j][i] = fmaf(d[k][i], d[j][k], d[j][i]);
    }
    if (lane == 0) {
#pragma unroll
        for (int j = 0; j < 8; j++) {
            *reinterpret_cast<float4*>(fd + 8 * j) = make_float4(d[j][0], d[j][1], d[j][2], d[j][3]);
            *reinterpret_cast<float4*>(fd + 8 * j + 4) = make_float4(d[j][4], d[j][5], d[j][6], d[j][7]);
        }
    }
}

// Warps of k_lu128 (warp % 4 is its SM partition): 0 the diagonal warp, 4 and 8
// leave at once, the other eight the workers.
constexpr int LUT = 352;

// dt (leading dimension lddt): the block's lower triangle transposed (rows of
// 32-wide chunks whole, so a chunk's own upper triangle comes along).
__global__ void __launch_bounds__(LUT, 1) k_lu128(float* __restrict__ a, int lda, float* __restrict__ dt, int lddt) {
    extern __shared__ __align__(16) float sm[];
    float* F = sm;                     // the factored block
    float* panels = F + PB * PS;       // two pairs of panels, alternating by step
    float* dgs = panels + 2 * 16 * PS;  // the next diagonal 8 x 8 block, updated up to the last step (alternating)
    float* fds = dgs + 2 * 64;          // the current one factored (alternating)
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    pdl_start();
    pdl_wait();
    if (warp == 0) {
        for (int idx = lane; idx < 32; idx += 32) {
            const int q = idx >> 4, r = (idx >> 1) & 7, i = (idx & 1) * 4;
            *reinterpret_cast<float4*>(dgs + 64 * q + r * 8 + i) =
                *reinterpret_cast<const float4*>(a + (size_t)(8 * q + r) * lda + 8 * q + i);
        }
        __syncwarp();
        diag_lu8(dgs, fds, lane);
        bar_sync<1, 288>();
#pragma unroll 1
        for (int b = 0; b < 16; b++) {
            const float* Ls = panels + (b & 1) * (16 * PS);
            bar_sync<1, 288>();  // the panels of step b are final
            if (b == 15) break;
            float* dg = dgs + ((b + 1) & 1) * 64;
            diag_rank8(dg, Ls, Ls + 8 * PS, 8 * (b + 1), lane);
            __syncwarp();
            diag_lu8(dg, fds + ((b + 1) & 1) * 64, lane);
            bar_sync<1, 288>();
        }
        return;
    }
    if ((warp & 3) == 0) return;
    const int w = (warp >> 2) * 3 + (warp & 3) - 1;  // worker 0..7: four groups of 16 rows, two of 32 columns
    const int ty = 4 * (w >> 1) + (lane >> 3), tx = 8 * (w & 1) + (lane & 7);
    // c[h][i][p]: row 64h + 4ty + i, columns 4tx + {0,1}, {2,3}, 64 + 4tx + {0,1}, {2,3}
    float2 c[2][4][4];
#pragma unroll
    for (int h = 0; h < 2; h++)
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const float* row = a + (size_t)(64 * h + 4 * ty + i) * lda + 4 * tx;
            const float4 u = *reinterpret_cast<const float4*>(row);
            const float4 v = *reinterpret_cast<const float4*>(row + 64);
            c[h][i][0] = make_float2(u.x, u.y);
            c[h][i][1] = make_float2(u.z, u.w);
            c[h][i][2] = make_float2(v.x, v.y);
            c[h][i][3] = make_float2(v.z, v.w);
        }
    const bool left = w < 4;            // in the panel step: one row of the block column, else one column of the row
    const int e = 32 * (w & 3) + lane;  // which
#pragma unroll 1
    for (int b = 0; b < 16; b++) {
        const int k0 = 8 * b;
        float* Ls = panels + (b & 1) * (16 * PS);  // 8 x PS: block column, k-major
        float* Ts = Ls + 8 * PS;                   // 8 x PS: block row
        const int hk = k0 >> 6, jk = (k0 & 63) >> 3;  // rows and columns k0 .. k0+7: half hk, ty / tx 2jk and 2jk + 1
        if ((ty >> 1) == jk) {
            float* dst = Ts + (4 * (ty & 1)) * PS + 4 * tx;
            if (hk == 0) store_rows(dst, c[0]);
            else store_rows(dst, c[1]);
        }
        if ((tx >> 1) == jk) {
            float* dst = Ls + (4 * (tx & 1)) * PS + 4 * ty;
            if (hk == 0) {
                store_cols<0>(dst, c[0]);
                store_cols<0>(dst + 64, c[1]);
            } else {
                store_cols<2>(dst, c[0]);
                store_cols<2>(dst + 64, c[1]);
            }
        }
        if (b > 0 && b < 15) {  // the diagonal block after this one (the first two: read by the diagonal warp itself)
            const int hn = (k0 + 8) >> 6, jn = ((k0 + 8) & 63) >> 3;
            if ((ty >> 1) == jn && (tx >> 1) == jn) {
                float* dst = dgs + ((b + 1) & 1) * 64 + 32 * (ty & 1) + 4 * (tx & 1);
                if (hn == 0) store_diag<0>(dst, c[0]);
                else store_diag<2>(dst, c[1]);
            }
        }
        bar_sync<1, 288>();
        const float* fd = fds + (b & 1) * 64;
        float x[8];
        if (e >= k0 + 8) {
            float d[8][8];
#pragma unroll
            for (int j = 0; j < 8; j++) {
                ld4(d[j], fd + 8 * j);
                ld4(d[j] + 4, fd + 8 * j + 4);
            }
            float* p = left ? Ls + e : Ts + e;
#pragma unroll
            for (int k = 0; k < 8; k++) x[k] = p[k * PS];
            if (left) {  // l_i += l_k D_ki (i > k)
#pragma unroll
                for (int k = 0; k < 8; k++)
#pragma unroll
                    for (int i = k + 1; i < 8; i++) x[i] = fmaf(x[k], d[k][i], x[i]);
            } else {  // t_k *= D_kk; t_j += t_k D_jk (j > k)
#pragma unroll
                for (int k = 0; k < 8; k++) {
                    x[k] *= d[k][k];
#pragma unroll
                    for (int j = k + 1; j < 8; j++) x[j] = fmaf(x[k], d[j][k], x[j]);
                }
            }
#pragma unroll
            for (int k = 0; k < 8; k++) p[k * PS] = x[k];
        } else if (left && e >= k0) {  // a row of the diagonal block
#pragma unroll
            for (int k = 0; k < 8; k++) x[k] = fd[8 * (e - k0) + k];
        }
        bar_sync<1, 288>();
        // the finished values into F
        if (left && e >= k0) {
            float4* g = reinterpret_cast<float4*>(F + e * PS + k0);
            g[0] = make_float4(x[0], x[1], x[2], x[3]);
            g[1] = make_float4(x[4], x[5], x[6], x[7]);
        } else if (!left && e >= k0 + 8) {
#pragma unroll
            for (int k = 0; k < 8; k++) F[(k0 + k) * PS + e] = x[k];
        }
        if (b == 15) break;
        // rank-8 update of what is still open (warps skip finished groups of rows and columns; values left of or
        // above the open part are never read again)
        const int k1 = k0 + 8, rhi = 16 * (w >> 1) + 16, chi = 32 * (w & 1) + 32;
        const float* lp = Ls + 4 * ty;
        const float* tp = Ts + 4 * tx;
        if (64 + rhi > k1 && 64 + chi > k1) {
            if (rhi > k1 && chi > k1)
                rank8<true, true>(c, lp, tp);
            else if (rhi > k1)
                rank8<true, false>(c, lp, tp);
            else if (chi > k1)
                rank8<false, true>(c, lp, tp);
            else
                rank8<false, false>(c, lp, tp);
        }
    }
    bar_sync<2, 256>();
    // the factored block, and its lower triangle transposed (lane = row)
    for (int idx = w * 32 + lane; idx < PB * PB / 4; idx += 256) {
        const int r = idx >> 5, i = (idx & 31) * 4;
        *reinterpret_cast<float4*>(a + (size_t)r * lda + i) = *reinterpret_cast<const float4*>(F + r * PS + i);
    }
    for (int q = w; q < 80; q += 8) {  // 32 rows x 4 columns each
        const int rb = q < 8 ? 0 : (q < 24 ? 1 : (q < 48 ? 2 : 3)), k = 4 * (q - 4 * rb * (rb + 1));
        const int r = 32 * rb + lane;
        const float4 v = *reinterpret_cast<const float4*>(F + r * PS + k);
        float* o = dt + (size_t)k * lddt + r;
        o[0] = v.x;
        o[lddt] = v.y;
        o[2 * (size_t)lddt] = v.z;
        o[3 * (size_t)lddt] = v.w;
    }
}

constexpr size_t kLu128Smem = sizeof(float) * (PB * PS + 32 * PS + 4 * 64);

// ---- top and left --------------------------------------------------------------

struct TlArgs {
    const float* d;    // factored diagonal block (bs x bs, leading dimension ldd)
    const float* dt;   // its lower triangle transposed (leading dimension lddt; top only)
    int ldd, bs, lddt;
    float* t;          // block row: bs x ncols
    int ldt, ncols, ntop;  // ntop: strips of the block row (CTAs 0 .. ntop - 1)
    float* l;          // block column: nrows x bs, and its transposed copy lt
    int ldl, nrows;
    float* lt;
    int ldlt;
};

constexpr int TT = 256;   // threads
constexpr int TR = 3;     // operator tiles (32 x 128, k-major, row stride PS) in flight

template <int TW>
constexpr size_t tl_smem(int bs) {
    return sizeof(float) * ((size_t)bs * (TW + 4) + TR * 32 * PS);
}

__device__ __forceinline__ void cp_group() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }

// y (RT rows x 4 columns) += sum_k op[k][rows] x[k][columns] over k < kn.
template <int RT, int XS>
__device__ __forceinline__ void tile_mul(float2 (&y)[RT][2], const float* op, const float* x, int kn) {
#pragma unroll 8
    for (int k = 0; k < kn; k++) {
        float o[RT];
        if constexpr (RT >= 4) {
#pragma unroll
            for (int i = 0; i < RT; i += 4) ld4(o + i, op + k * PS + i);
        } else if constexpr (RT == 2) {
            const float2 v = *reinterpret_cast<const float2*>(op + k * PS);
            o[0] = v.x, o[1] = v.y;
        } else {
            o[0] = op[k * PS];
        }
        const float4 v = *reinterpret_cast<const float4*>(x + k * XS);
#pragma unroll
        for (int i = 0; i < RT; i++) {
            y[i][0] = fma2(o[i], make_float2(v.x, v.y), y[i][0]);
            y[i][1] = fma2(o[i], make_float2(v.z, v.w), y[i][1]);
        }
    }
}

// The recurrence of a 32-row chunk, one column per lane: x_k *= D_kk (scale),
// x_i += x_k D_ki (i > k).  x: the column in the strip (row stride XS), d: D_ki
// at d[k * PS + i]; out: the column in global memory, or null.
template <int XS>
__device__ __forceinline__ void solve32(float* xs, const float* d, bool scale, float* out, int ldo) {
    float x[32];
#pragma unroll
    for (int i = 0; i < 32; i++) x[i] = xs[i * XS];
#pragma unroll
    for (int k = 0; k < 32; k++) {
        x[k] *= scale ? d[k * PS + k] : 1.0f;
#pragma unroll
        for (int i = (k + 1) / 4 * 4; i < 32; i += 4) {
            const float4 v = *reinterpret_cast<const float4*>(d + k * PS + i);
            if (i > k) x[i] = fmaf(x[k], v.x, x[i]);
            if (i + 1 > k) x[i + 1] = fmaf(x[k], v.y, x[i + 1]);
            if (i + 2 > k) x[i + 2] = fmaf(x[k], v.z, x[i + 2]);
            if (i + 3 > k) x[i + 3] = fmaf(x[k], v.w, x[i + 3]);
        }
    }
#pragma unroll
    for (int i = 0; i < 32; i++) {
        xs[i * XS] = x[i];
        if (out != nullptr) out[(size_t)i * ldo] = x[i];
    }
}

// Per 128 rows B of the block: acc = sum over the rows before B of D X (tiles
// of 32 x 128), then four chunks of 32 rows: the recurrence of X0_c + acc_c
// within the chunk, and acc of the later chunks += D X_c.  256 threads even for
// narrow strips: 128 with twice the outputs each load less per product but
// were slower (12.5 against 10.4 us for 128 rows, 72 against 61 us for 512).
template <int TW>
__global__ void __launch_bounds__(TT, 2) k_tl(const TlArgs p) {
    constexpr int XS = TW + 4;       // row stride of the strip
    constexpr int CG = TW / 32;      // warps side by side; each covers 32 columns
    constexpr int RT = 4 * CG;       // rows of acc per thread (128 rows over 8 / CG warps of 4 threads)
    extern __shared__ __align__(16) float sm[];
    float* X = sm;                   // bs x XS: the strip, unknowns by rows
    float* ring = X + p.bs * XS;     // TR x 32 x PS operator tiles, ring[k][i]
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const bool top = (int)blockIdx.x < p.ntop;
    const int s0 = (top ? blockIdx.x : blockIdx.x - p.ntop) * TW;  // first column (top) or row (left) of the strip
    const int width = min(TW, (top ? p.ncols : p.nrows) - s0);     // a multiple of 4
    const int nb = p.bs / PB, ntiles = 2 * nb * (nb + 1);          // 4 (B + 1) tiles for each B
    // the operator's off-diagonal values, k-major: top D^T, left D
    const float* off = top ? p.dt : p.d;
    const int ldo = top ? p.lddt : p.ldd;
    pdl_start();
    pdl_wait();

    int iB = 0, ik = 0, in = 0;  // next tile to issue: rows [128 iB, +128), k chunk ik
    auto issue = [&]() {
        if (in < ntiles) {
            float* dst = ring + (in % TR) * (32 * PS);
            const int own = ik - 4 * iB;  // >= 0: chunk `own` of the block itself
            const float* src = off + (size_t)(32 * ik) * ldo + PB * iB;
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int k = (tid >> 5) + 8 * q, i = lane * 4;
                if (i >= 32 * own) cp_async_vec16(dst + k * PS + i, src + (size_t)k * ldo + i);
            }
            if (own == 3)
                iB++, ik = 0;
            else
                ik++;
            in++;
        }
        cp_group();
    };
    if (top) {
        for (int idx = tid; idx < p.bs * (TW / 4); idx += TT) {
            const int k = idx / (TW / 4), j = (idx - k * (TW / 4)) * 4;
            if (j < width)
                cp_async_vec16(X + k * XS + j, p.t + (size_t)k * p.ldt + s0 + j);
            else
                *reinterpret_cast<float4*>(X + k * XS + j) = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        }
    }
#pragma unroll
    for (int q = 0; q < TR - 1; q++) issue();  // the first group covers the block row's strip too
    if (!top) {  // rows of the block column transposed into X: lane = row, so the stores do not conflict
        for (int q0 = warp; q0 < CG * (p.bs / 4); q0 += 4 * (TT / 32)) {
            float4 v[4];
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const int q = q0 + u * (TT / 32), r = (q % CG) * 32 + lane, k = (q / CG) * 4;
                v[u] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                if (k < p.bs && r < width) v[u] = *reinterpret_cast<const float4*>(p.l + (size_t)(s0 + r) * p.ldl + k);
            }
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const int q = q0 + u * (TT / 32), r = (q % CG) * 32 + lane, k = (q / CG) * 4;
                if (k < p.bs) {
                    X[k * XS + r] = v[u].x;
                    X[(k + 1) * XS + r] = v[u].y;
                    X[(k + 2) * XS + r] = v[u].z;
                    X[(k + 3) * XS + r] = v[u].w;
                }
            }
        }
    }
    // a warp covers 4 RT rows x 32 columns (4 x 8 threads)
    const int wr = warp / CG, wc = warp - wr * CG;
    const int row = RT * (4 * wr + (lane >> 3)), col = 32 * wc + 4 * (lane & 7);
    int tile = 0;
    for (int B = 0; B < nb; B++) {
        float2 acc[RT][2];
#pragma unroll
        for (int i = 0; i < RT; i++) acc[i][0] = acc[i][1] = make_float2(0.0f, 0.0f);
        float* XB = X + PB * B * XS;
        for (int ck = 0; ck < 4 * B + 4; ck++, tile++) {
            asm volatile("cp.async.wait_group %0;\n" ::"n"(TR - 2) : "memory");
            __syncthreads();
            issue();  // into the slot that was read before this barrier
            const float* op = ring + (tile % TR) * (32 * PS);
            if (ck < 4 * B) {
                tile_mul<RT, XS>(acc, op + row, X + 32 * ck * XS + col, 32);
                continue;
            }
            const int c = ck - 4 * B;
            if ((row >> 5) == c) {  // X0_c + acc and its recurrence, by the two warps that hold it
#pragma unroll
                for (int i = 0; i < RT; i++) {
                    float4* q = reinterpret_cast<float4*>(XB + (row + i) * XS + col);
                    float4 v = *q;
                    v.x += acc[i][0].x, v.y += acc[i][0].y, v.z += acc[i][1].x, v.w += acc[i][1].y;
                    *q = v;
                }
                if (CG == 1)
                    bar_sync<1, 64>();  // (each warp holds half of the rows)
                else
                    __syncwarp();
                const int cl = 32 * wc + lane, k = PB * B + 32 * c;
                if (CG == 2 || (warp & 1) == 0) {
                    float* o = top ? p.t + (size_t)k * p.ldt : p.lt + (size_t)k * p.ldlt;
                    solve32<XS>(X + k * XS + cl, op + 32 * c, top, cl < width ? o + s0 + cl : nullptr,
                                top ? p.ldt : p.ldlt);
                }
            }
            if (c < 3) {
                __syncthreads();
                if ((row >> 5) > c) tile_mul<RT, XS>(acc, op + row, XB + 32 * c * XS + col, 32);
            }
        }
    }
    if (!top) {  // rows of the block column back, lane = row
        __syncthreads();
        for (int q = warp; q < CG * (p.bs / 8); q += TT / 32) {
            const int r = (q % CG) * 32 + lane, k = (q / CG) * 8;
            if (r < width) {
                float4* o = reinterpret_cast<float4*>(p.l + (size_t)(s0 + r) * p.ldl + k);
                const float* x = X + k * XS + r;
                o[0] = make_float4(x[0], x[XS], x[2 * XS], x[3 * XS]);
                o[1] = make_float4(x[4 * XS], x[5 * XS], x[6 * XS], x[7 * XS]);
            }
        }
    }
}

}  // namespace

int panel_init_attrs() {
    LP_CUDA(cudaFuncSetAttribute(k_lu128, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kLu128Smem));
    LP_CUDA(cudaFuncSetAttribute(k_tl<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tl_smem<64>(512)));
    LP_CUDA(cudaFuncSetAttribute(k_tl<32>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tl_smem<32>(512)));
    return LP_OK;
}

int launch_lu128(float* a, int lda, float* dt, int lddt, cudaStream_t st) {
    if (lda % 4 != 0 || !aligned16(a)) return fail(LP_E_INVALID, "128 block LU: block must be 16-byte aligned, lda % 4 == 0");
    LP_CUDA(launch_pdl(k_lu128, dim3(1), dim3(LUT), kLu128Smem, st, a, lda, dt, lddt));
    count_launch();
    return LP_OK;
}

// T (bs x ncols) and L (nrows x bs, with its transposed copy lt) beside the
// factored block d, in place; bs a multiple of 128, at most 512; ncols and
// nrows multiples of 4 (either may be 0).  dt: d's lower triangle transposed
// (needed for ncols > 0).
int launch_tl(const float* d, int ldd, const float* dt, int lddt, int bs, float* t, int ldt,
              int ncols, float* l, int ldl, int nrows, float* lt, int ldlt, int sms, cudaStream_t st) {
    if (ncols <= 0 && nrows <= 0) return LP_OK;
    if (bs % PB != 0 || bs > 512 || ncols % 4 != 0 || nrows % 4 != 0 || ldd % 4 != 0 || ldt % 4 != 0 || ldl % 4 != 0 ||
        ldlt % 4 != 0 || lddt % 4 != 0 || !aligned16(d) || !aligned16(t) || !aligned16(l) || !aligned16(lt))
        return fail(LP_E_INVALID, "top/left update: sizes must be multiples of 4, the block of 128, pointers 16-byte aligned");
    TlArgs p{d, dt, ldd, bs, lddt, t, ldt, ncols, 0, l, ldl, nrows, lt, ldlt};
    // narrow strips while they leave SMs idle (less work per CTA), wide ones (fewer loads per product) once they do not
    const int wide = (ncols + 63) / 64 + (nrows + 63) / 64;
    if (wide >= sms) {
        p.ntop = (ncols + 63) / 64;
        LP_CUDA(launch_pdl(k_tl<64>, dim3(wide), dim3(TT), tl_smem<64>(bs), st, p));
    } else {
        p.ntop = (ncols + 31) / 32;
        LP_CUDA(launch_pdl(k_tl<32>, dim3(p.ntop + (nrows + 31) / 32), dim3(TT), tl_smem<32>(bs), st, p));
    }
    count_launch();
    return LP_OK;
}

}  // namespace lp
