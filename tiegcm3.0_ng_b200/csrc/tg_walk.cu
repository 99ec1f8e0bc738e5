// The column walk of the three-pass assembly routines: the Thomas solve
// (src/trsolv_ng.F90:14-26) of rows already formed by a level-parallel pass,
// stored through the routines' post-solve steps.
//
// In the two-pass form each walk forms its rows as it goes (hundreds of
// dependent instructions per level, one thread per column); with few columns
// per SM every level then waits on its own instruction latencies.  Here the
// rows come from planes p, q, r, f (level-major, k*ld + col) that one thread
// per (level, column) wrote, so a walk level is the recurrence alone: two
// divisions sharing one correctly rounded reciprocal, a product and a
// difference.
//
//   top = 0 (minor_ng): rows 0..K-1 with K = nk, no extrapolation;
//   top = 1 (dt_ng, oplus_ng): rows 0..K-1 with K = nk-1 and
//         x(nk-1) = x(nk-2)**2/x(nk-3) from the unfiltered values
//         (dt_ng.F90:167, oplus_ng.F90:307).
// With a PostStep every row is stored through post_store: the lateral
// boundary overwrite, the time filter and the floors.  Same operations in the
// same order as the fused walks, so the same bits.
#include <cfloat>
#include <cstdint>

#include "tg_internal.h"
#include "tg_arith.cuh"
#include "tg_stage.cuh"
#include "tg_tile.cuh"

namespace tg {
namespace {
__device__ __forceinline__ double xm(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double xs(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double xd(double a, double b) { return __ddiv_rn(a, b); }

// The walk with the column tile held in shared memory, for launches of
// few columns.  A block of kWalkTileThreads threads takes kTileCols columns:
// together they copy the p, q, r, f rows of every level (every copy in flight
// at once) and read the post-step inputs of their own levels into registers;
// one thread per column walks (tile_thomas); then all store the rows through
// the post-solve steps, each its own levels.  16 columns a block spread a
// launch of few columns over twice the SMs a 32-column tile does, and 29 KB of
// rows (57 levels) leave seven blocks per SM (a 32-column tile that also held
// the post-step inputs took 87 KB: two).  The walk's chain bounds it; dt_ng
// with its rows, 11,248 columns x 57 levels 61 -> 45 us, 2,072 columns 21.5 ->
// 18.7 (the post-step stores had waited on the boundary values one by one).
constexpr int kWalkTileThreads = 128;
template <bool WIDE>
__global__ void __launch_bounds__(kWalkTileThreads) k_thomas_post_tile(const double *P, const double *Q,
                                                                       const double *R, const double *Fv, double *x,
                                                                       int nk, int K, int top, int ncol, long ld,
                                                                       unsigned *status, PostStep post, int has_post)
{
    constexpr int T = kTileCols, NG = kWalkTileThreads / T;
    extern __shared__ __align__(16) double tile_walk[];
    const int t = threadIdx.x % T, g = threadIdx.x / T;
    const long c0 = (long)blockIdx.x * T, col = c0 + t;
    const bool live = col < ncol;
    const int KS = top == 1 ? K + 1 : K;   // q holds the KS solved rows
    double *sp = tile_walk, *sr = sp + K * T, *sf = sr + K * T, *sq = sf + K * T;
    double *dst[4] = {sp, sq, sr, sf};
    const double *src[4] = {P + c0, Q + c0, R + c0, Fv + c0};
    if (WIDE) {   // 8 lanes a row, 16 bytes each
        const int c2 = (threadIdx.x % (T / 2)) * 2;
        for (int k = threadIdx.x / (T / 2); k < K; k += 2 * NG)
#pragma unroll
            for (int v = 0; v < 4; ++v) cp_async16_ca(dst[v] + k * T + c2, src[v] + (long)k * ld + c2);
    } else if (live) {
        for (int k = g; k < K; k += NG)
#pragma unroll
            for (int v = 0; v < 4; ++v) cp_async8(dst[v] + k * T + t, src[v] + (long)k * ld + t);
    }
    cp_async_commit();
    const bool bcol = live && has_post && post.bnd_mask && post.bnd_mask[col];
    TilePost<NG, 8> ps;
    if (live) ps.load(post, has_post, bcol, g, KS, ld, col);
    cp_async_wait<0>();
    __syncthreads();
    if (threadIdx.x < T && live) tile_thomas<T>(sp, sq, sr, sf, K, top, t, status);
    __syncthreads();
    if (live) ps.template store<T>(post, has_post, bcol, sq, x, t, g, KS, ld, col);
}

// The walk for launches of more columns, one warp per 32-column block.
// The rows stream through a shared-memory ring of kRingStages stages of
// kRingLevels levels (WIDE: 16-byte asynchronous copies, two rows per
// instruction).  w2 and w3 of a level replace its p and q in the planes (each
// lane its own column, behind the copies), and come back with the post-step
// inputs, every lane its own values, through the same ring for the back sweep,
// which stores each row as it solves it.  Alone on 43,216 columns x 57 levels
// the walk took 107 us with w2 in shared memory, w3 parked in x and the stores
// waiting on their inputs level by level (issue 20%, 6.6 long-scoreboard stalls
// per issue); dt_ng there went from 203 to 130 us, minor_ng from 252 to 186.
// The tile walk is taken while shared memory alone would hold its blocks all at
// once: 35,520 columns at 29 levels, 16,576 at 57, 7,104 at 113.  (Its registers
// hold 5 blocks per SM, 11,840 columns, so that the upper part of the range runs
// in two or three rounds.)  dt_ng with its rows, us with tile and ring:
//   29 levels  11,760 columns 21.9, 27.2; 13,440 29.0, 29.1; 22,080 40.3, 40.1;
//              29,000 52.7, 48.3; 36,000 64.8, 55.4
//   57         11,760 40.5, 49.5; 13,440 51.5, 53.1; 16,320 57.7, 58.6; 22,080
//              71.9, 71.0; 29,000 93.2, 87.1
//   113        7,000 53.2, 72.3; 8,400 76.5, 77.5; 11,280 90.3, 88.3; 16,320 128,
//              108
// The limit lies where the two meet at 57 and 113 levels; at 29 they meet near
// 14,000 columns, part by 1% up to 22,000 and by 9% at 29,000.
constexpr int kRingLevels = 4, kRingStages = 3;
constexpr int kRingDoubles = 5 * 32;   // a level of the back sweep: w2, w3, prev, cur, bnd
template <bool WIDE>
__global__ void __launch_bounds__(32) k_thomas_post_ring(double *P, double *Q, const double *R, const double *Fv,
                                                         double *x, int nk, int K, int top, int ncol, long ld,
                                                         unsigned *status, PostStep post, int has_post)
{
    constexpr int L = kRingLevels, C = kRingStages, RD = kRingDoubles;
    extern __shared__ __align__(16) double ring_walk[];
    const int t = threadIdx.x;
    const long c0 = (long)blockIdx.x * 32, col = c0 + t;
    const bool live = col < ncol;
    const int nch = (K + L - 1) / L;
    const int half = t >> 4, c2 = (t & 15) * 2;
    const double *a0 = WIDE ? (half ? Q : P) + c0 + c2 : P + col, *a1 = WIDE ? (half ? Fv : R) + c0 + c2 : R + col;
    auto issue = [&](int st, int j) {
        double *d = ring_walk + st * L * RD;
#pragma unroll
        for (int l = 0; l < L; ++l) {
            const int k = j * L + l;
            if (k < K) {
                const long o = (long)k * ld;
                if (WIDE) {
                    cp_async16_cg(d + l * RD + half * 32 + c2, a0 + o);
                    cp_async16_cg(d + l * RD + 64 + half * 32 + c2, a1 + o);
                } else if (live) {
                    cp_async8(d + l * RD + t, a0 + o);
                    cp_async8(d + l * RD + 32 + t, Q + o + col);
                    cp_async8(d + l * RD + 64 + t, a1 + o);
                    cp_async8(d + l * RD + 96 + t, Fv + o + col);
                }
            }
        }
        cp_async_commit();
    };
#pragma unroll 1
    for (int j = 0; j < C; ++j) issue(j, j);
    bool ok = true;
    double w2 = 0.0, w3 = 0.0;
    int st = 0;
#pragma unroll 1
    for (int j = 0; j < nch; ++j) {
        cp_async_wait<C - 1>();
        __syncwarp();
        double *stg = ring_walk + st * L * RD + t;
        if (j == 0) stg[0] = 0.0;   // row 0 has no p: x - 0*0 = x
        auto step = [&](int l) {
            const double p = stg[l * RD], q = stg[l * RD + 32], r = stg[l * RD + 64], f = stg[l * RD + 96];
            const double w1 = xs(q, xm(p, w2));
            const double y1 = __drcp_rn(w1);
            const double num = xs(f, xm(p, w3));
            if (max(exp_dist(w1), max(exp_dist(num), exp_dist(r))) < kExpSpan) {
                w3 = div_markstein(num, w1, y1);
                w2 = div_markstein(r, w1, y1);
            } else {
                const bool w1s = exp_safe(w1);
                w3 = qdiv_pivot(num, w1, y1, w1s);
                w2 = qdiv_pivot(r, w1, y1, w1s);
                if (!w1s) ok = ok && finite_nz(w1);
            }
            const long o = (long)(j * L + l) * ld + col;
            P[o] = w2;
            Q[o] = w3;
        };
        if (live) {
            if ((j + 1) * L <= K) {
#pragma unroll
                for (int l = 0; l < L; ++l) step(l);
            } else {
                for (int l = 0; j * L + l < K; ++l) step(l);
            }
        }
        __syncwarp();
        issue(st, j + C);
        st = st + 1 == C ? 0 : st + 1;
    }
    cp_async_wait<0>();
    __syncwarp();
    if (!live) return;
    // back sweep: x(k) = w3(k) - w2(k)*x(k+1), levels kh - L + 1 .. kh of stage
    // d, kh = K - 2 - d*L; no lane reads another's copies
    const bool bcol = has_post && post.bnd_mask && post.bnd_mask[col];
    const int KB = K - 1, nbk = (KB + L - 1) / L;
    auto issue_b = [&](int sb, int d) {
        double *db = ring_walk + sb * L * RD + t;
#pragma unroll
        for (int l = 0; l < L; ++l) {
            const int k = KB - 1 - d * L - l;
            if (k >= 0) {
                const long o = (long)k * ld + col;
                cp_async8(db + l * RD, P + o);
                cp_async8(db + l * RD + 32, Q + o);
                if (has_post) {
                    cp_async8(db + l * RD + 64, post.prev + o);
                    cp_async8(db + l * RD + 96, post.cur + o);
                    if (bcol) cp_async8(db + l * RD + 128, post.bnd + o);
                }
            }
        }
        cp_async_commit();
    };
#pragma unroll 1
    for (int d = 0; d < C; ++d) issue_b(d, d);
    // the rows above the ring: K-1 now, for top = 1 row K when x(K-2) is known
    const long ot = (long)(K - 1) * ld + col;
    const double xtop = w3;
    double pk = 0.0, ck = 0.0, xn = w3;
    if (top == 1 && has_post) {
        pk = post.prev[ot + ld];
        ck = post.cur[ot + ld];
    }
    post_store(post, has_post, bcol, x, ot, xtop);
    st = 0;
#pragma unroll 1
    for (int d = 0; d < nbk; ++d) {
        cp_async_wait<C - 1>();
        const double *g = ring_walk + st * L * RD + t;
#pragma unroll
        for (int l = 0; l < L; ++l) {
            const int k = KB - 1 - d * L - l;
            if (k >= 0) {
                xn = xs(g[l * RD + 32], xm(g[l * RD], xn));
                const long o = (long)k * ld + col;
                if (has_post)
                    post_store_v(post, false, x, o, bcol ? g[l * RD + 128] : xn, g[l * RD + 64], g[l * RD + 96]);
                else
                    x[o] = xn;
                if (top == 1 && d == 0 && l == 0) {   // x(nk-1) = x(nk-2)**2/x(nk-3) from the unfiltered values
                    const double xe = xd(xm(xtop, xtop), xn);
                    if (has_post) post_store_v(post, bcol, x, ot + ld, xe, pk, ck);
                    else x[ot + ld] = xe;
                }
            }
        }
        issue_b(st, d + C);
        st = st + 1 == C ? 0 : st + 1;
    }
    cp_async_wait<0>();
    // x(k) = w3 - w2*x(k+1) carries a non-finite value down to x(0)
    const bool fin = finite(xn) && finite(xtop);
    if (status && (!ok || !fin)) atomicOr(status, (ok ? 0u : FLAG_PIVOT) | (fin ? 0u : FLAG_NONFINITE));
}
}  // namespace

cudaError_t launch_thomas_post(double *p, double *q, const double *r, const double *f, double *x, int nk, int K,
                               int top, int ncol, long ld, unsigned *status, const PostStep *post, cudaStream_t st)
{
    if (ncol <= 0) return cudaSuccess;
    if (K < 1 || K > nk || (top == 1 && (K != nk - 1 || K < 2))) return cudaErrorInvalidValue;
    const PostStep pv = post ? *post : PostStep{};
    const int hp = post != nullptr, KS = top == 1 ? K + 1 : K;
    auto aligned = [](const double *v) { return ((uintptr_t)v & 15) == 0; };
    auto wide = [&](int T) {   // whole 16-byte pieces of rows of T columns lie in the planes
        return ld % 2 == 0 && ld >= (long)(ncol + T - 1) / T * T && aligned(p) && aligned(q) && aligned(r) && aligned(f);
    };
    const size_t tile = (size_t)kTileCols * (3 * K + KS) * sizeof(double);
    if (tile <= (size_t)smem_optin() && (ncol + kTileCols - 1) / kTileCols <= resident_by_smem(tile)) {
        once_per_device([] {
            cudaFuncSetAttribute(k_thomas_post_tile<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_optin());
            cudaFuncSetAttribute(k_thomas_post_tile<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_optin());
        });
        auto k = wide(kTileCols) ? k_thomas_post_tile<true> : k_thomas_post_tile<false>;
        k<<<(ncol + kTileCols - 1) / kTileCols, kWalkTileThreads, tile, st>>>(p, q, r, f, x, nk, K, top, ncol, ld,
                                                                             status, pv, hp);
        return cudaGetLastError();
    }
    auto k = wide(32) ? k_thomas_post_ring<true> : k_thomas_post_ring<false>;
    k<<<(ncol + 31) / 32, 32, sizeof(double) * kRingStages * kRingLevels * kRingDoubles, st>>>(
        p, q, r, f, x, nk, K, top, ncol, ld, status, pv, hp);
    return cudaGetLastError();
}
}  // namespace tg
