// A column tile of the assembly routines' walks in shared memory: T columns,
// rows of T, every level.  One thread per column walks the rows; one thread
// per (level, column) stores the solution through the post-solve steps.
#pragma once
#include "tg_arith.cuh"
#include "tg_internal.h"
#include "tg_stage.cuh"

namespace tg {

// The Thomas walk of column t of the tile: rows 0..K-1 of p, q, r, f into the
// solution, left in sq (KS = K rows; top = 1: one more, x(K) = x(K-1)**2/x(K-2)
// from the unfiltered values).
//
// Level k divides by its pivot w1(k) twice: w3(k) and the next level's w2 =
// r(k)/w1(k) (the reference's operands, so the same quotients), kept where
// r(k) was.  The walk's chain is the recurrence alone: every quotient by
// Markstein's sequence, no branch, each level's operands read one level ahead.
// A level whose operands leave the sequence's safe range (zeros, non-finite or
// extreme values) stops the stores; the levels from the first such one are then
// walked again with the IEEE fallback (qdiv2, qdiv1).
template <int T>
__device__ __forceinline__ void tile_thomas(const double *sp, double *sq, double *sr, const double *sf, int K, int top,
                                            int t, unsigned *status)
{
    bool ok = true;
    int bad = K;
    double w1 = 0.0, y1 = 0.0, w2 = 0.0, w3 = 0.0;
    auto level = [&](int k, double p, double q, double r, double f, bool top_level) {
        w1 = k == 0 ? q : xsub(q, xmul(p, w2));
        y1 = __drcp_rn(w1);
        const double num = k == 0 ? f : xsub(f, xmul(p, w3));
        ok = ok && (bad < K || finite_nz(w1));
        const unsigned d = max(exp_dist(w1), max(exp_dist(num), top_level ? 0u : exp_dist(r)));
        bad = d >= kExpSpan && bad == K ? k : bad;
        w3 = div_markstein(num, w1, y1);
        w2 = div_markstein(r, w1, y1);
        if (bad > k) {
            sr[k * T + t] = w2;
            sq[k * T + t] = w3;
        }
    };
    double pn = sp[t], qn = sq[t], rn = sr[t], fn = sf[t];
    for (int k = 0; k < K - 1; ++k) {
        const int s = k * T + t;
        const double p = pn, q = qn, r = rn, f = fn;
        pn = sp[s + T];
        qn = sq[s + T];
        rn = sr[s + T];
        fn = sf[s + T];
        level(k, p, q, r, f, false);
    }
    level(K - 1, pn, qn, rn, fn, true);
    if (bad < K) {
        w2 = bad > 0 ? sr[(bad - 1) * T + t] : 0.0;
        w3 = bad > 0 ? sq[(bad - 1) * T + t] : 0.0;
        for (int k = bad; k < K; ++k) {
            const int s = k * T + t;
            const double p = sp[s], q = sq[s], f = sf[s];
            w1 = k == 0 ? q : xsub(q, xmul(p, w2));
            y1 = __drcp_rn(w1);
            const double num = k == 0 ? f : xsub(f, xmul(p, w3));
            if (k + 1 < K) {
                qdiv2(num, sr[s], w1, y1, w3, w2);
                sr[s] = w2;
            } else {
                w3 = qdiv1(num, w1, y1);
            }
            ok = ok && finite_nz(w1);
            sq[s] = w3;
        }
    }
    const double xtop = w3;
    back_sweep<T>(sq, sr, K, t, w3);
    // x(k) = w3 - w2*x(k+1) carries a non-finite value down to x(0)
    const bool fin = finite(sq[t]) && finite(xtop);
    if (top == 1) sq[K * T + t] = xdiv(xmul(xtop, xtop), sq[(K - 2) * T + t]);
    if (status && (!ok || !fin)) atomicOr(status, (ok ? 0u : FLAG_PIVOT) | (fin ? 0u : FLAG_NONFINITE));
}

// The post-solve inputs of this thread's levels k = g + m*NG (m < R), read
// before the walk; levels past R*NG are read when they are stored, four at a
// time (nm may alias prev or cur, so no read may pass a store by itself).
template <int NG, int R>
struct TilePost {
    double pv[R > 0 ? R : 1], cv[R > 0 ? R : 1], bv[R > 0 ? R : 1];
    __device__ __forceinline__ void load(const PostStep &post, bool on, bool bcol, int g, int KS, long ld, long col)
    {
        if (!on) return;
#pragma unroll
        for (int m = 0; m < R; ++m) {
            const int k = g + m * NG;
            if (k < KS) {
                const long o = (long)k * ld + col;
                pv[m] = post.prev[o];
                cv[m] = post.cur[o];
                bv[m] = bcol ? __ldg(post.bnd + o) : 0.0;
            }
        }
        for (int k = g + R * NG; k < KS; k += NG) {
            const long o = (long)k * ld + col;
            asm volatile("prefetch.global.L2 [%0];" ::"l"(post.prev + o));
            asm volatile("prefetch.global.L2 [%0];" ::"l"(post.cur + o));
        }
    }
    // the solution rows sx (rows of T) of column t to out, through the steps when on
    template <int T>
    __device__ __forceinline__ void store(const PostStep &post, bool on, bool bcol, const double *sx, double *out, int t,
                                          int g, int KS, long ld, long col) const
    {
        if (!on) {
            for (int k = g; k < KS; k += NG) out[(long)k * ld + col] = sx[k * T + t];
            return;
        }
#pragma unroll
        for (int m = 0; m < R; ++m) {
            const int k = g + m * NG;
            if (k < KS)
                post_store_v(post, false, out, (long)k * ld + col, bcol ? bv[m] : sx[k * T + t], pv[m], cv[m]);
        }
        for (int k0 = g + R * NG; k0 < KS; k0 += 4 * NG) {
            double p[4], c[4], x[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int k = k0 + u * NG;
                if (k < KS) {
                    const long o = (long)k * ld + col;
                    p[u] = post.prev[o];
                    c[u] = post.cur[o];
                    x[u] = bcol ? __ldg(post.bnd + o) : sx[k * T + t];
                }
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int k = k0 + u * NG;
                if (k < KS) post_store_v(post, false, out, (long)k * ld + col, x[u], p[u], c[u]);
            }
        }
    }
};

constexpr int kTileCols = 16;   // columns of a tile: one 128-byte line of a row

}  // namespace tg
