// Horizontal operators that feed the column assembly: advec_ng
// (src/advec_ng.F90) and smooth_ng (src/smooth_ng.F90), over one nest held as
// a single subdomain.  Every lateral edge is then a boundary (is_bndry all
// true, src/fields_ng.F90:143-147) and the halo syncs of src/sync_ng.F90
// exchange nothing, so the operators are plain stencils over the
// ghost-inclusive (nlon+4) x (nlat+4) plane of each level.
//
// Layout: level-major planes, (k, i, j) at k*ld + i + nlond*j with
// nlond = nlon+4, i.e. the column index of the other device entries.  One
// thread per point; a block covers 32 longitudes x 8 latitudes of one level
// (blockIdx.z), so the lat neighbours are rows that the block's other warps
// bring into L1.
//
// Arithmetic follows the reference's operation order with separately rounded
// operations.  Divisions by 2 and 4 are written as multiplications by 0.5
// and 0.25 (the same correctly rounded number); divisions by 3, 12, dlamda
// and dphi are correctly rounded (qdiv with the reciprocal from the host).
#include <cmath>

#include "tg_internal.h"
#include "tg_arith.cuh"

namespace tg {
namespace {

constexpr int kTx = 32, kTy = 8;

struct AdvecRcp {
    double r3, r12, rlam, rphi;  // correctly rounded 1/3, 1/12, 1/dlamda, 1/dphi
    int lam_safe, phi_safe;      // dlamda, dphi inside the Markstein range
};

// a/b correctly rounded, y the reciprocal of b, b known to be in range
__device__ __forceinline__ double qdiv_by(double a, double b, double y, bool b_safe)
{
    return b_safe && exp_safe(a) ? div_markstein(a, b, y) : __ddiv_rn(a, b);
}

// One direction of advec_ng (:33-37 lon, :44-48 lat) at index t of an axis
// of n points with element stride s (p: the field, u: the wind, both at the
// point).  df_3d and fm_3d (src/dffm_ng.F90:66-110, :166-205) of order 1 are
// (p[+1]-p[-1])/2 and (u[+1]+u[-1])/2 inside, and on the edge rows the
// one-sided difference and the value itself; with the neighbour indices
// clamped into the axis, p[+1]-p[-1] is the one-sided difference there.  The
// term is dfdx1*2*2/3*ubar1 - dfdx2*4/12*ubar2 on rows 2..n-3 (where the
// order-2 helpers take their centred form) and dfdx1*ubar1 on the two ghost
// rows of each boundary side.  (d*2)*2 is d*4 exactly; x/2 and x/4 are the
// same numbers as x*0.5 and x*0.25.
__device__ __forceinline__ double advec_dir(const double *p, const double *u, int t, int n, int s,
                                            const AdvecRcp &rc)
{
    const int dm = t > 0 ? -s : 0, dp = t < n - 1 ? s : 0;
    const bool edge = t == 0 || t == n - 1;
    const double dif = xsub(__ldg(p + dp), __ldg(p + dm));
    const double d1 = edge ? dif : xmul(dif, 0.5);
    const double m1 = edge ? __ldg(u) : xmul(xadd(__ldg(u + dp), __ldg(u + dm)), 0.5);
    if (t <= 1 || t >= n - 2) return xmul(d1, m1);
    const double d2 = xmul(xsub(__ldg(p + 2 * s), __ldg(p - 2 * s)), 0.25);
    const double m2 = xmul(xadd(__ldg(u + 2 * s), __ldg(u - 2 * s)), 0.5);
    const double lhs = xmul(qdiv_by(xmul(d1, 4.0), 3.0, rc.r3, true), m1);
    const double rhs = xmul(qdiv_by(xmul(d2, 4.0), 12.0, rc.r12, true), m2);
    return xsub(lhs, rhs);
}

// Several fields in one launch: blockIdx.z counts planes, nk of each field.
constexpr int kMaxBatch = 8;
struct HorizBatch {
    const double *in[kMaxBatch];
    double *out[kMaxBatch];
};

__device__ __forceinline__ void advec_point(const double *f, const double *un, const double *vn, const double *racs,
                                            double dlamda, double dphi, double re_inv, const AdvecRcp &rc, int i, int j,
                                            int nlond, int nlatd, long o, double *hadvec)
{
    const double wk1 = xmul(advec_dir(f + o, un + o, i, nlond, 1, rc), __ldg(racs + j));
    const double wk2 = advec_dir(f + o, vn + o, j, nlatd, nlond, rc);
    // hadvec = wk1/dlamda + wk2*re_inv/dphi (:50)
    hadvec[o] = xadd(qdiv_by(wk1, dlamda, rc.rlam, rc.lam_safe), qdiv_by(xmul(wk2, re_inv), dphi, rc.rphi, rc.phi_safe));
}

// The lat pass lands in a shared tile of the block's 8 rows x (32 + 4)
// longitudes (the lon pass needs +-2 neighbours): its 288 points are dealt
// to the 256 threads in order, so only one warp takes a second point.  Then
// the lon pass reads the tile.
__device__ __forceinline__ void smooth_point(const double *fin, double sh, int i0, int j0, int nlond, int nlatd,
                                             long plane, double *fout)
{
    constexpr int W = kTx + 4;
    __shared__ double ft[kTy][W + 1];
    for (int q = threadIdx.y * kTx + threadIdx.x; q < W * kTy; q += kTx * kTy) {
        const int r = q / W, c = q - r * W;
        const int i = i0 - 2 + c, j = j0 + r;
        if (i < 0 || i >= nlond || j >= nlatd) continue;
        const double *p = fin + plane + i + (long)nlond * j;
        ft[r][c] = shapiro_at([&](int d) { return p[d * nlond]; }, j, nlatd, sh);
    }
    __syncthreads();
    const int i = i0 + threadIdx.x, j = j0 + threadIdx.y;
    if (i >= nlond || j >= nlatd) return;
    // every longitude the lon pass reads (i-2..i+2 where used) is in the tile
    const double *p = &ft[threadIdx.y][threadIdx.x + 2];
    fout[plane + i + (long)nlond * j] = shapiro_at([&](int d) { return p[d]; }, i, nlond, sh);
}

// KIND 1: advec_ng of n_adv fields, 2: smooth_ng, 3: both, the advected fields
// first.  One field of a small grid is a launch gap and a quarter of a wave
// (56 x 37 x 57: 4.2 us for 3 MB), so a routine's fields share a launch: one
// advec + one smooth 6.2 us against 8.4, three of each 10.3 against 25 (147 x
// 76 x 57: 14.4 against 18.5, 35 against 56).  Bound by the loads' latency and
// the issue slots, hence 8 blocks per SM: at 32 registers instead of 38 to 40
// advec_ng of 580 x 292 x 20 falls from 42.9 to 37.0 us and three of each of
// 147 x 76 x 57 from 38 to 35; 4 levels per thread with every load in flight
// took 60.  ONE: one field, whose plane needs no loop (smooth_ng of 580 x 292 x
// 20: 22.6 us, 23.7 with it).  The lists stay in the parameter bank (__grid_constant__): indexed as a plain
// parameter they are copied to the stack, and advec_ng takes 71 us.
template <int KIND, bool ONE>
__global__ void __launch_bounds__(kTx * kTy, 8)
    k_horiz_ng(const __grid_constant__ HorizBatch hb, int n_adv, const double *un, const double *vn, const double *racs,
               double dlamda, double dphi, double re_inv, AdvecRcp rc, double sh, int nk, int nlond, int nlatd, long ld)
{
    int n = 0, k = blockIdx.z;
    if (!ONE)
        for (; k >= nk; k -= nk) ++n;
    const long plane = (long)k * ld;
    const int i0 = blockIdx.x * kTx, j0 = blockIdx.y * kTy;
    if (KIND == 1 || (KIND == 3 && n < n_adv)) {
        const int i = i0 + threadIdx.x, j = j0 + threadIdx.y;
        if (i < nlond && j < nlatd)
            advec_point(hb.in[n], un, vn, racs, dlamda, dphi, re_inv, rc, i, j, nlond, nlatd,
                        plane + i + (long)nlond * j, hb.out[n]);
    } else {
        smooth_point(hb.in[n], sh, i0, j0, nlond, nlatd, plane, hb.out[n]);
    }
}

dim3 plane_grid(int nk, int nlond, int nlatd)
{
    return dim3((unsigned)((nlond + kTx - 1) / kTx), (unsigned)((nlatd + kTy - 1) / kTy), (unsigned)nk);
}

}  // namespace

cudaError_t launch_horiz_ng(int n_adv, const double *const *f, double *const *hadvec, int n_smooth,
                            const double *const *fin, double *const *fout, const double *un, const double *vn,
                            const double *racs, double dlamda, double dphi, double re_inv, double shapiro, int nk,
                            int nlon, int nlat, long ld, cudaStream_t st)
{
    const int nlond = nlon + 4, nlatd = nlat + 4;
    // host IEEE division: the correctly rounded reciprocals the Markstein step needs
    auto in_range = [](double b) { return std::fabs(b) >= 0x1p-500 && std::fabs(b) < 0x1p500; };
    const AdvecRcp rc{1.0 / 3.0, 1.0 / 12.0, 1.0 / dlamda, 1.0 / dphi, in_range(dlamda), in_range(dphi)};
    // grid.z counts planes: at most 65535
    const int most = nk > 65535 / kMaxBatch ? 65535 / nk : kMaxBatch;
    for (int a = 0, s = 0; a < n_adv || s < n_smooth;) {
        HorizBatch hb{};
        int n = 0, na = 0;
        for (; a < n_adv && n < most; ++a, ++n, ++na) {
            hb.in[n] = f[a];
            hb.out[n] = hadvec[a];
        }
        for (; s < n_smooth && n < most; ++s, ++n) {
            hb.in[n] = fin[s];
            hb.out[n] = fout[s];
        }
        auto k = n == 1 ? na ? k_horiz_ng<1, true> : k_horiz_ng<2, true>
                 : na == n ? k_horiz_ng<1, false> : na ? k_horiz_ng<3, false> : k_horiz_ng<2, false>;
        k<<<plane_grid(nk * n, nlond, nlatd), dim3(kTx, kTy), 0, st>>>(hb, na, un, vn, racs, dlamda, dphi, re_inv, rc,
                                                                       shapiro, nk, nlond, nlatd, ld);
    }
    return cudaGetLastError();
}

cudaError_t launch_advec_ng(const double *f, const double *un, const double *vn, const double *racs, double dlamda,
                            double dphi, double re_inv, int nk, int nlon, int nlat, long ld, double *hadvec,
                            cudaStream_t st)
{
    return launch_horiz_ng(1, &f, &hadvec, 0, nullptr, nullptr, un, vn, racs, dlamda, dphi, re_inv, 0.0, nk, nlon, nlat,
                           ld, st);
}

cudaError_t launch_smooth_ng(const double *fin, double shapiro, int nk, int nlon, int nlat, long ld, double *fout,
                             cudaStream_t st)
{
    return launch_horiz_ng(0, nullptr, nullptr, 1, &fin, &fout, nullptr, nullptr, nullptr, 1.0, 1.0, 1.0, shapiro, nk,
                           nlon, nlat, ld, st);
}

}  // namespace tg
