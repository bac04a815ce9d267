// Matrix-free derivatives of the convex-inversion model (PS_FORM_FAST
// arithmetic, FP64): chi2 and beta = J^T W (y_obs - y) -- the chi2 gradient is
// -2 beta -- and Gauss-Newton products J^T W (J v), one or kAdjDirs at a time,
// without forming J.
//
// The shape block of J is J_pk = Scale_p sum_f Darea_f s_pf g_f Dsph_fk
// (bright.c:78-85 with Dg = g Dsph, curv.c:31-35).  Its products with a vector
// and its transpose need no p x k array:
//   (J v)_p   = Scale_p sum_f Area_f s_pf z_f,      z = Dsph v        (forward)
//   (J^T l)_k = sum_f (sum_p l_p Scale_p s_pf) Area_f Dsph_fk       (adjoint)
// so one product costs two passes over the (point, facet) pairs plus two
// F x C contractions instead of the N F C of the explicit Jacobian.  The eight
// non-shape columns are formed per point, and so is the first shape column:
// Dsph_f0 = 1, so it is the model itself, and z leaves the first coefficient
// out.  The relative-lightcurve normalisation (mrqcof.c:92-104),
// J'_r = coef_r (J_r - y_r dave / ave) with dave = sum_r J_r and J'_r1 = 0,
// becomes per-lightcurve scalars:
//   (J' v)_r  = coef_r ((J v)_r - y_r sum_{r'} (J v)_{r'} / ave)   (v_1 left out)
//   J'^T u    = J^T l,  l_r = coef_r u_r - sum_{r'} coef_{r'} y_{r'} u_{r'} / ave;
// coef_r = sigma_r L / ave: a curve's sigmas need not be equal.
// A convexity row (conv.c:12-29) is a point whose s_pf is a component of the
// facet's normal, so its weights join the facet sums.  Every reduction runs in
// a fixed order, so results are deterministic.
//
// Six kernels, or seven, each spread over the GPU by how many CTAs its sizes give:
// adj_curv (warp per facet: scalars, areas, z, facet sums), adj_points (point
// blocks x facet slices), adj_sums (CTA per block of points of one curve: the
// slices' sums, model, columns of J; part of adj_rows where no relative curve is
// long), adj_rows (CTA per relative lightcurve or block of calibrated points:
// residual, adjoint weights), adj_facets (facet blocks x point blocks), adj_cols
// (blocks of facets: the F x C contraction), adj_out (CTA per free parameter).
#include <cuda_runtime.h>
#include <math.h>

#include "ps_adjoint.hpp"
#include "ps_device.hpp"
#include "ps_fit_common.cuh"

namespace psb {
namespace {

using namespace fitcommon;

constexpr int kCurvFacets = 8;    // adj_curv: facets per CTA (a warp each)
constexpr int kPtThreads = 128;   // adj_points: points per CTA
constexpr int kPairChunk = 64;    // adj_points: facet pairs staged at a time
constexpr int kRowThreads = 256;  // adj_rows
constexpr int kFcThreads = 128;   // adj_facets: facets per CTA
constexpr int kPtStage = 64;      // adj_facets: points staged at a time
constexpr int kColFacets = 32;    // adj_cols: facets per CTA
constexpr int kOutThreads = 1024; // adj_out: the non-shape columns run over all points
constexpr int kFixed = 9;         // adj_points: sums besides the directions'
constexpr int kMaxSlices = 32;    // adj_points: facet slices at most
constexpr int kMaxPointBlocks = 64;  // adj_facets: point blocks at most
constexpr int kFill = 8 * 148;    // CTAs that fill the GPU

// misc slots (X_CHK and X_SAREA are read by the host: kAdjMiscChk, kAdjMiscSarea)
enum { X_B = 0, X_D = 9, X_CL = 27, X_CLS = 28, X_OMG = 29, X_P1 = 30, X_P2 = 31, X_P3 = 32, X_CHK = kAdjMiscChk,
       X_SAREA = kAdjMiscSarea, X_UC = 40, X_N = X_UC + 3 * kAdjDirs };

// Device work arrays of one evaluation, carved from one buffer of
// adjoint_work_doubles doubles; K directions.
struct AdjWork {
    double* misc;    // scalars, then u of the convexity rows [K][3]
    double* dir;     // [K][9]: v of the first shape coefficient, then of the non-shape parameters
    double* area;    // [F]
    double* z;       // [K][F]
    double* cpart;   // [4 + 3 K][curv CTAs]: chck, area sum, J v of the convexity rows
    double* e6;      // [6][N]: e, e0
    double* pp;      // [kFixed + K][nfs][N]
    double* jns;     // [9][N]: non-shape columns, first shape column (0 on relative rows)
    double *y, *scale;  // [N]
    double* jv;      // [K][N]
    double* lam;     // [K][N] adjoint weights
    double* ls;      // [K][N] times Scale
    double* x2part;  // [row items]
    double* q;       // [K][npb][F]
    double* cols;    // [K][col CTAs][C]
    double* out;     // [K][mfit]
    double* chi2;
    int nfs, npb, ppb;  // facet slices; point blocks and their points
    int ncurv, ncol;
    AdjMode mode;
};

inline int cdiv(int a, int b) { return (a + b - 1) / b; }

// Facet slices of adj_points: enough CTAs to fill the GPU, 16 pairs or more.
inline int facet_slices(const DevProblem& P) {
    const int blocks = cdiv(P.n_points, kPtThreads);
    int s = cdiv(kFill, blocks);
    if (s > P.F / 2 / 16) s = P.F / 2 / 16;
    return s < 1 ? 1 : s > kMaxSlices ? kMaxSlices : s;
}

// Points per CTA of adj_facets: likewise, 32 or more.
inline int points_per_block(const DevProblem& P) {
    int blocks = cdiv(kFill, cdiv(P.F, kFcThreads));
    if (blocks > kMaxPointBlocks) blocks = kMaxPointBlocks;
    const int n = cdiv(P.n_points, blocks);
    return n < 32 ? 32 : n;
}

__device__ double block_sum(double v, double* red) {
    // fixed-order tree: warp shuffles, then warp 0 over the warp partials
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    __syncthreads();
    if (lane == 0) red[warp] = v;
    __syncthreads();
    double s = 0;
    if (warp == 0) {
        s = lane < (int)(blockDim.x >> 5) ? red[lane] : 0.0;
        for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
        if (lane == 0) red[0] = s;
    }
    __syncthreads();
    s = red[0];
    __syncthreads();
    return s;
}

__device__ __forceinline__ double warp_sum(double v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// blmatrix, the scattering and phase scalars and the directions' non-shape
// parts (block 0); curv (curv.c:15-37 through Dsph = Fc/Fs Pleg), z without the
// first coefficient, and each CTA's share of the facet sums: a warp per facet,
// lanes over the coefficients.  (A thread per facet read its rows uncoalesced:
// 26 us at 2048 facets and 81 coefficients.)
template <int K>
__global__ void __launch_bounds__(32 * kCurvFacets) adj_curv(const DevProblem* __restrict__ Pp, AdjWork W, const AdjArgs A) {
    const DevProblem& P = *Pp;
    const int C = P.C, F = P.F, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    __shared__ double part[4 + 3 * K][kCurvFacets];
    if (blockIdx.x == 0) {
        double* x = W.misc;
        if (tid == 0) {
            blmatrix(A.a[C], A.a[C + 1], x + X_B, x + X_D);
            x[X_CL] = exp(A.a[C + 6]);
            x[X_CLS] = A.a[C + 7];
            x[X_OMG] = A.a[C + 2];
            x[X_P1] = A.a[C + 3];
            x[X_P2] = A.a[C + 4];
            x[X_P3] = A.a[C + 5];
        }
        for (int i = tid; i < 9 * K; i += blockDim.x) {
            const int d = i / 9, j = i - 9 * d, k = j == 0 ? 0 : C + j - 1;
            W.dir[i] = W.mode == kAdjUnits ? (A.unit[d] == k ? 1.0 : 0.0) : W.mode == kAdjProduct ? A.v[k] : 0.0;
        }
    }
    const int f = blockIdx.x * kCurvFacets + warp;
    double x = 0, z[K], n[3] = {0, 0, 0}, area = 0;
#pragma unroll
    for (int d = 0; d < K; d++) z[d] = 0;
    if (f < F) {
        const double* ds = P.dsph + (size_t)f * P.NCB;
        for (int k = lane; k < C; k += 32) {
            const double b = ds[k];
            x = fma(A.a[k], b, x);
            if (K == 1 && W.mode == kAdjProduct && k > 0) z[0] = fma(A.v[k], b, z[0]);
        }
        x = warp_sum(x);
        if (K == 1) z[0] = warp_sum(z[0]);
        if constexpr (K > 1) {
#pragma unroll
            for (int d = 0; d < K; d++) {
                const int k = A.unit[d];
                z[d] = k > 0 && k < C ? ds[k] : 0.0;
            }
        }
        const double* fa = P.fac + (size_t)f * 4;
        area = fa[3] * exp(x);
        for (int c = 0; c < 3; c++) n[c] = fa[c];
        if (lane == 0) {
            W.area[f] = area;
#pragma unroll
            for (int d = 0; d < K; d++) W.z[(size_t)d * F + f] = z[d];
        }
    }
    if (lane == 0) {
        for (int c = 0; c < 3; c++) part[c][warp] = area * n[c];
        part[3][warp] = area;
#pragma unroll
        for (int d = 0; d < K; d++) {
            double v0 = 0;
            if (W.mode == kAdjUnits) v0 = A.unit[d] == 0 ? 1.0 : 0.0;
            if (W.mode == kAdjProduct) v0 = A.v[0];
            for (int c = 0; c < 3; c++) part[4 + 3 * d + c][warp] = area * n[c] * (z[d] + v0);
        }
    }
    __syncthreads();
    if (tid < 4 + 3 * K) {
        double s = 0;
        for (int w = 0; w < kCurvFacets; w++) s += part[tid][w];
        W.cpart[(size_t)tid * W.ncurv + blockIdx.x] = s;
    }
}

// Per point and facet slice: the slice's sums of the model brightness and of
// what the non-shape columns and the shape parts of J v need (Area s z per
// direction, the Lambert / Lommel-Seeliger sums, T = sum Area dsmu n,
// S = sum Area dsmu0 n); grid (point blocks, facet slices).  Facets come in
// antipodal pairs, of which a point sees at most one: an FP32 cosine picks the
// side, so a warp's lanes work on a facet they see in nine of ten pairs, where
// facet by facet 45 % of the lanes were active and points in time order share
// no facets to skip (20 000 points, 2048 facets: 174 us).  Where the FP32 sign
// is wrong (a facet within 1e-6 of grazing) the pair's two facets are tested in
// FP64.  A facet that is not seen counts with area 0; kMasked: with no terms, where
// parameters or directions are so large that these may be infinite.
template <int K, bool kMasked>
__global__ void __launch_bounds__(kPtThreads) adj_points(const DevProblem* __restrict__ Pp, AdjWork W) {
    const DevProblem& P = *Pp;
    __shared__ double sf[4 + K][2 * kPairChunk];  // nx, ny, nz, Area, z; [pair][side]
    const int tid = threadIdx.x, F = P.F, N = P.n_points;
    const int p = blockIdx.x * kPtThreads + tid;
    const bool act = p < N;
    const int pairs = F / 2, per = (pairs + W.nfs - 1) / W.nfs;
    const int j0 = blockIdx.y * per, j1 = min(pairs, j0 + per);
    const double* x = W.misc;
    const double cl = x[X_CL], cls = x[X_CLS];
    double e[3] = {0, 0, 0}, e0[3] = {0, 0, 0};
    if (act) {
        PointGeom G;
        point_geometry(P, p, x + X_B, x + X_D, x[X_OMG], x[X_P1], x[X_P2], x[X_P3], G);
        for (int c = 0; c < 3; c++) {
            e[c] = G.e[c];
            e0[c] = G.e0[c];
        }
        if (!visible_geometry(e, e0))
            for (int c = 0; c < 3; c++) e[c] = e0[c] = 0;
        if (blockIdx.y == 0)
            for (int c = 0; c < 3; c++) {
                W.e6[(size_t)c * N + p] = e[c];
                W.e6[(size_t)(3 + c) * N + p] = e0[c];
            }
    }
    const float e32[3] = {(float)e[0], (float)e[1], (float)e[2]};
    double acc[kFixed + K] = {};
    for (int c0 = j0; c0 < j1; c0 += kPairChunk) {
        const int np = min(kPairChunk, j1 - c0);
        __syncthreads();
        for (int i = tid; i < 2 * np; i += kPtThreads) {
            const int f = P.apair[2 * c0 + i];
            const double* fa = P.fac + (size_t)f * 4;
            sf[0][i] = fa[0];
            sf[1][i] = fa[1];
            sf[2][i] = fa[2];
            sf[3][i] = W.area[f];
#pragma unroll
            for (int d = 0; d < K; d++) sf[4 + d][i] = W.z[(size_t)d * F + f];
        }
        __syncthreads();
#pragma unroll 2
        for (int j = 0; j < np; j++) {
            const float m32 = e32[0] * (float)sf[0][2 * j] + e32[1] * (float)sf[1][2 * j] + e32[2] * (float)sf[2][2 * j];
            int i = 2 * j + (m32 < 0.f);
            double nx = sf[0][i], ny = sf[1][i], nz = sf[2][i];
            double mu = fma(e[2], nz, fma(e[1], ny, e[0] * nx));
            if (mu < 0) {  // the other side after all
                i ^= 1;
                nx = sf[0][i], ny = sf[1][i], nz = sf[2][i];
                mu = fma(e[2], nz, fma(e[1], ny, e[0] * nx));
            }
            const double mu0 = fma(e0[2], nz, fma(e0[1], ny, e0[0] * nx));
            const bool vis = mu > kTinyD && mu0 > kTinyD;
            if (kMasked && !vis) continue;
            const double ar = vis ? sf[3][i] : 0.0;
            const double r = rcp_newton(vis ? mu + mu0 : 1.0);
            const double am = ar * mu, am0 = ar * mu0, mm = am * mu0, cr = cls * r, crr = cr * r;
            const double t = mm * (cr + cl);
            acc[0] += t;                      // br
            acc[1] += mm;                     // sum mu mu0 Area
            acc[2] = fma(mm, r, acc[2]);      // sum mu mu0 Area / (mu + mu0)
            const double w = am0 * fma(crr, mu0, cl), w0 = am * fma(crr, mu, cl);
            acc[3] = fma(w, nx, acc[3]);
            acc[4] = fma(w, ny, acc[4]);
            acc[5] = fma(w, nz, acc[5]);
            acc[6] = fma(w0, nx, acc[6]);
            acc[7] = fma(w0, ny, acc[7]);
            acc[8] = fma(w0, nz, acc[8]);
#pragma unroll
            for (int d = 0; d < K; d++) acc[kFixed + d] = fma(t, sf[4 + d][i], acc[kFixed + d]);
        }
    }
    if (!act) return;
#pragma unroll
    for (int j = 0; j < kFixed + K; j++) W.pp[((size_t)j * W.nfs + blockIdx.y) * N + p] = acc[j];
}

// A block of at most kAdjRowBlock points of one lightcurve, by kRowThreads
// threads: the slices' sums in slice order, kRowThreads / kAdjRowBlock threads
// per point, then a thread per point the model, the non-shape columns of J and
// J v; the thread's y and J v are added to sy and sj.
template <int K>
__device__ __forceinline__ void block_sums(const DevProblem& P, const AdjWork& W, int first, int last, bool rel,
                                           double& sy, double* sj) {
    __shared__ double sums[kFixed + K][kAdjRowBlock];
    const int tid = threadIdx.x, N = P.n_points;
    const double* x = W.misc;
    const double cl = x[X_CL];
    const int np = last - first, i0 = tid % kAdjRowBlock;
    if (i0 < np)
        for (int j = tid / kAdjRowBlock; j < kFixed + K; j += kRowThreads / kAdjRowBlock) {
            const double* src = W.pp + (size_t)j * W.nfs * N + first + i0;
            double v = 0;
#pragma unroll 8
            for (int k = 0; k < W.nfs; k++) v += src[(size_t)k * N];
            sums[j][i0] = v;
        }
    __syncthreads();
    if (tid >= np) return;
    const int p = first + tid;
    PointGeom G;
    point_geometry(P, p, x + X_B, x + X_D, x[X_OMG], x[X_P1], x[X_P2], x[X_P3], G);
    double acc[kFixed + K];
#pragma unroll
    for (int j = 0; j < kFixed + K; j++) acc[j] = sums[j][tid];
    const double br = acc[0], sc = G.scale, yy = br * sc;
    double jn[9];
    for (int k = 0; k < 3; k++) {
        double v = 0;
        for (int c = 0; c < 3; c++) v = fma(acc[3 + c], G.de[c][k], fma(acc[6 + c], G.de0[c][k], v));
        jn[k] = sc * v;
    }
    jn[3] = br * G.dphp[0];
    jn[4] = br * G.dphp[1];
    jn[5] = br * G.dphp[2];
    jn[6] = sc * acc[1] * cl;
    jn[7] = sc * acc[2];
    jn[8] = rel ? 0.0 : yy;  // first shape coefficient
    for (int j = 0; j < 9; j++) W.jns[(size_t)j * N + p] = jn[j];
    W.y[p] = yy;
    W.scale[p] = sc;
    sy += yy;
#pragma unroll
    for (int d = 0; d < K; d++) {
        const double* v = W.dir + 9 * d;
        double s = jn[8] * v[0];
        for (int j = 0; j < 8; j++) s = fma(jn[j], v[1 + j], s);
        s = fma(sc, acc[kFixed + d], s);
        W.jv[(size_t)d * N + p] = s;
        sj[d] += s;
    }
}

// A block of points per CTA, where some relative lightcurve is longer than
// kAdjOwnBlocks of them: its own kernel, whose blocks spread over the GPU however
// long a lightcurve is.  Inside adj_rows, a CTA per relative lightcurve, they took
// 3 us each in turn: a gradient on one curve of 1000 / 5000 / 20 000 points and
// 800 facets 184 / 673 / 1313 us, 79 / 113 / 238 as a kernel of their own.  Where
// no curve is longer, adj_rows forms its item's blocks itself and the launch is
// saved, which costs as much as two blocks in turn: 40 calibrated points and 8
// facets 58 against 62 us, two nights of 80 points among 760 73 against 76.
template <int K>
__global__ void __launch_bounds__(kRowThreads) adj_sums(const DevProblem* __restrict__ Pp, AdjWork W) {
    const int4 item = reinterpret_cast<const int4*>(Pp->ablocks)[blockIdx.x];  // first point, last + 1, relative
    double sy = 0, sj[K] = {};  // adj_rows forms the curve's
    block_sums<K>(*Pp, W, item.x, item.y, item.z != 0, sy, sj);
}

// One item of the row list per CTA: a relative lightcurve, a block of
// calibrated points, or (the last) the three convexity rows.  Per relative
// lightcurve ave = sum y and S = sum J v without v_1 (mrqcof.c:53-58, 92-104);
// per row the normalised model and J v, the residual, u = W (y_obs - y') or
// W J' v, and the item's share of chi2; the adjoint weights l.  (y S) / ave in
// mrqcof's order: where it overflows, as at a Lambert coefficient of 1e200, J' is
// infinite there and a fit freezes.  kOwnSums: the item's blocks are formed here
// (see adj_sums).
template <int K, bool kOwnSums>
__global__ void __launch_bounds__(kRowThreads) adj_rows(const DevProblem* __restrict__ Pp, AdjWork W) {
    const DevProblem& P = *Pp;
    __shared__ double red[32];
    const int tid = threadIdx.x, N = P.n_points;
    const int4 item = reinterpret_cast<const int4*>(P.arows)[blockIdx.x];  // first row, last + 1, relative, points of the curve
    double* x = W.misc;
    double x2 = 0;
    if (item.x >= N) {
        // the facet sums of adj_curv's CTAs, a warp per sum
        const int lane = tid & 31;
        for (int j = tid >> 5; j < 4 + 3 * K; j += kRowThreads / 32) {
            double s = 0;
            for (int b = lane; b < W.ncurv; b += 32) s += W.cpart[(size_t)j * W.ncurv + b];
            s = warp_sum(s);
            if (lane == 0) {
                if (j < 4)
                    x[X_CHK + j] = s;
                else if (W.mode != kAdjGradient) {
                    const int r = N + (j - 4) % 3;
                    x[X_UC + j - 4] = P.sig2i[r] * P.wght[r] * s;
                }
            }
        }
        __syncthreads();
        if (tid < 3) {
            const int r = N + tid;
            const double dy = P.yobs[r] - x[X_CHK + tid], w = P.sig2i[r] * P.wght[r];
            x2 = dy * dy * w;
            if (W.mode == kAdjGradient) x[X_UC + tid] = w * dy;
        }
        x2 = block_sum(x2, red);
        if (tid == 0) W.x2part[blockIdx.x] = x2;
        return;
    }
    const bool rel = item.z != 0;
    double sy = 0, sj[K];
#pragma unroll
    for (int d = 0; d < K; d++) sj[d] = 0;
    if constexpr (kOwnSums) {
        for (int p = item.x; p < item.y; p += kAdjRowBlock) {
            block_sums<K>(P, W, p, min(p + kAdjRowBlock, item.y), rel, sy, sj);
            __syncthreads();
        }
    } else if (rel) {
#pragma unroll 2
        for (int p = item.x + tid; p < item.y; p += kRowThreads) {
            sy += W.y[p];
#pragma unroll
            for (int d = 0; d < K; d++) sj[d] += W.jv[(size_t)d * N + p];
        }
    }
    // coef of a row: L sigma / ave; rs is its sigma over the curve's first, one
    // for the per-curve mean
    double ave = 0, sjv[K], kap[K], coefn = 0;
    const double sig0 = rel ? P.sig[item.x] : 1.0;
    auto ratio = [&](double sig) { return sig == sig0 ? 1.0 : sig / sig0; };
#pragma unroll
    for (int d = 0; d < K; d++) sjv[d] = kap[d] = 0;
    if (rel) {
        ave = block_sum(sy, red);
        coefn = (double)item.w / ave;
#pragma unroll
        for (int d = 0; d < K; d++) sjv[d] = block_sum(sj[d], red);
    }
    for (int p = item.x + tid; p < item.y; p += kRowThreads) {
        const double y = W.y[p], coef = rel ? P.sig[p] * coefn : 1.0, rs = rel ? ratio(P.sig[p]) : 1.0;
        const double w = P.sig2i[p] * P.wght[p], dy = P.yobs[p] - coef * y;
        x2 = fma(dy * w, dy, x2);
#pragma unroll
        for (int d = 0; d < K; d++) {
            const double jv = W.jv[(size_t)d * N + p];
            const double u = W.mode == kAdjGradient ? w * dy : w * (rel ? coef * (jv - y * sjv[d] / ave) : jv);
            W.lam[(size_t)d * N + p] = u;
            kap[d] = fma(rs * y, u, kap[d]);
        }
    }
    if (rel) {
#pragma unroll
        for (int d = 0; d < K; d++) kap[d] = block_sum(kap[d], red) / ave;
    }
    for (int p = item.x + tid; p < item.y; p += kRowThreads) {
        const double sc = W.scale[p], coef0 = sig0 * coefn, rs = rel ? ratio(P.sig[p]) : 1.0;
#pragma unroll
        for (int d = 0; d < K; d++) {
            double l = W.lam[(size_t)d * N + p];
            if (rel) l = coef0 * (rs * l - kap[d]);
            W.lam[(size_t)d * N + p] = l;
            W.ls[(size_t)d * N + p] = l * sc;
        }
    }
    x2 = block_sum(x2, red);
    if (tid == 0) W.x2part[blockIdx.x] = x2;
}

// q_f = sum_p ls_p s_pf over a block of points; thread per facet (neighbours
// see nearly the same points), points staged in shared memory, two points at a
// time without a branch (a facet that a point does not see adds zero times the
// point's weight, nothing where a weight staged is not finite).  Blocks of points small enough to fill the GPU: in
// blocks of 512, 760 points and 800 facets made 14 CTAs and 62 us.
template <int K>
__global__ void __launch_bounds__(kFcThreads) adj_facets(const DevProblem* __restrict__ Pp, AdjWork W) {
    const DevProblem& P = *Pp;
    constexpr int kU = 2;
    __shared__ double sp[6 + K][kPtStage];  // e (3), e0 (3), ls
    const int f = blockIdx.x * kFcThreads + threadIdx.x, N = P.n_points, F = P.F;
    const int p0 = blockIdx.y * W.ppb, p1 = min(N, p0 + W.ppb);
    const double cl = W.misc[X_CL], cls = W.misc[X_CLS];
    double nx = 0, ny = 0, nz = 0, q[K];
    if (f < F) {
        nx = P.fac[(size_t)f * 4];
        ny = P.fac[(size_t)f * 4 + 1];
        nz = P.fac[(size_t)f * 4 + 2];
    }
#pragma unroll
    for (int d = 0; d < K; d++) q[d] = 0;
    for (int b = p0; b < p1; b += kPtStage) {
        const int np = min(kPtStage, p1 - b), npu = (np + kU - 1) / kU * kU;
        __syncthreads();
        bool fine = true;
        for (int i = threadIdx.x; i < npu * (6 + K); i += kFcThreads) {
            const int c = i / npu, j = i - c * npu;
            const double* src = c < 6 ? W.e6 + (size_t)c * N : W.ls + (size_t)(c - 6) * N;
            const double v = j < np ? src[b + j] : 0.0;
            fine = fine && isfinite(v);
            sp[c][j] = v;
        }
        fine = __syncthreads_and(fine);
        for (int i = 0; i < npu; i += kU) {
            double mu[kU], mu0[kU];
            bool vis[kU], some = false;
#pragma unroll
            for (int u = 0; u < kU; u++) {
                mu[u] = fma(sp[2][i + u], nz, fma(sp[1][i + u], ny, sp[0][i + u] * nx));
                mu0[u] = fma(sp[5][i + u], nz, fma(sp[4][i + u], ny, sp[3][i + u] * nx));
                vis[u] = mu[u] > kTinyD && mu0[u] > kTinyD;
                some = some || vis[u];
            }
            if (!__any_sync(0xffffffffu, some)) continue;
#pragma unroll
            for (int u = 0; u < kU; u++) {
                const double r = rcp_newton(vis[u] ? mu[u] + mu0[u] : 1.0);
                const double s = vis[u] ? mu[u] * mu0[u] * fma(cls, r, cl) : 0.0;
#pragma unroll
                for (int d = 0; d < K; d++)
                    if (fine || vis[u]) q[d] = fma(sp[6 + d][i + u], s, q[d]);
            }
        }
    }
    if (f >= F) return;
#pragma unroll
    for (int d = 0; d < K; d++) W.q[((size_t)d * W.npb + blockIdx.y) * F + f] = q[d];
}

// A block of facets: Q_f = Area_f (sum of q over the point blocks + the
// convexity rows' n_f . u), then its share of sum_f Q_f Dsph_fk, thread per
// coefficient.
template <int K>
__global__ void __launch_bounds__(128) adj_cols(const DevProblem* __restrict__ Pp, AdjWork W) {
    const DevProblem& P = *Pp;
    __shared__ double sq[K][kColFacets];
    const int f0 = blockIdx.x * kColFacets, F = P.F, C = P.C, nf = min(kColFacets, F - f0), tid = threadIdx.x;
    for (int i = tid; i < K * kColFacets; i += 128) {
        const int d = i / kColFacets, ff = i - d * kColFacets, f = f0 + ff;
        double s = 0;
        if (ff < nf) {
            for (int b = 0; b < W.npb; b++) s += W.q[((size_t)d * W.npb + b) * F + f];
            for (int c = 0; c < 3; c++) s = fma(P.fac[(size_t)f * 4 + c], W.misc[X_UC + 3 * d + c], s);
            s *= W.area[f];
        }
        sq[d][ff] = s;
    }
    __syncthreads();
    if (tid >= C) return;
    double s[K];
#pragma unroll
    for (int d = 0; d < K; d++) s[d] = 0;
#pragma unroll 4
    for (int ff = 0; ff < nf; ff++) {
        const double b = P.dsph[(size_t)(f0 + ff) * P.NCB + tid];
#pragma unroll
        for (int d = 0; d < K; d++) s[d] = fma(sq[d][ff], b, s[d]);
    }
#pragma unroll
    for (int d = 0; d < K; d++) W.cols[((size_t)d * W.ncol + blockIdx.x) * C + tid] = s[d];
}

// One CTA per free parameter and direction: a shape column's shares in block
// order, or sum_p l_p J_p for a non-shape column; the first shape column is
// J_p = y_p over the points plus the convexity rows' facet sum.  The last CTA
// of direction 0 sums chi2.
template <int K>
__global__ void __launch_bounds__(kOutThreads) adj_out(const DevProblem* __restrict__ Pp, AdjWork W, int items) {
    const DevProblem& P = *Pp;
    __shared__ double red[32];
    const int i = blockIdx.x, d = blockIdx.y, C = P.C, N = P.n_points, tid = threadIdx.x;
    double s = 0;
    if (i == P.mfit) {
        if (d > 0) return;
        for (int b = tid; b < items; b += blockDim.x) s += W.x2part[b];
        s = block_sum(s, red);
        if (tid == 0) *W.chi2 = s;
        return;
    }
    const int k = P.free_idx[i];
    if (k > 0 && k < C) {
        for (int b = tid; b < W.ncol; b += blockDim.x) s += W.cols[((size_t)d * W.ncol + b) * C + k];
    } else {
        const double* col = W.jns + (size_t)(k == 0 ? 8 : k - C) * N;
        const double* lam = W.lam + (size_t)d * N;
#pragma unroll 4
        for (int p = tid; p < N; p += kOutThreads) s = fma(__ldg(lam + p), __ldg(col + p), s);
        if (k == 0 && tid < 3) s = fma(W.misc[X_CHK + tid], W.misc[X_UC + 3 * d + tid], s);
    }
    s = block_sum(s, red);
    if (tid == 0) W.out[(size_t)d * P.mfit + i] = s;
}

template <int K>
size_t carve(const DevProblem& P, double* base, AdjWork& W) {
    const size_t N = P.n_points, F = P.F;
    W.nfs = facet_slices(P);
    W.ppb = points_per_block(P);
    W.npb = cdiv(P.n_points, W.ppb);
    W.ncurv = cdiv(P.F, kCurvFacets);
    W.ncol = cdiv(P.F, kColFacets);
    size_t o = 0;
    auto take = [&](size_t n) {
        double* r = base + o;
        o += (n + 1) & ~(size_t)1;
        return r;
    };
    W.misc = take(X_N);  // first: the host reads chck and the area sum there
    W.dir = take(9 * K);
    W.area = take(F);
    W.z = take(K * F);
    W.cpart = take((size_t)(4 + 3 * K) * W.ncurv);
    W.e6 = take(6 * N);
    W.pp = take((size_t)(kFixed + K) * W.nfs * N);
    W.jns = take(9 * N);
    W.y = take(N);
    W.scale = take(N);
    W.jv = take(K * N);
    W.lam = take(K * N);
    W.ls = take(K * N);
    W.x2part = take(P.n_arows);
    W.q = take((size_t)K * W.npb * F);
    W.cols = take((size_t)K * W.ncol * P.C);
    return o;
}

template <int K>
cudaError_t launch(const DevProblem& P, const DevProblem* dP, double* work, const AdjArgs& args, AdjMode mode,
                   double* d_out, double* d_chi2, cudaStream_t s) {
    AdjWork W{};
    carve<K>(P, work, W);
    W.out = d_out;
    W.chi2 = d_chi2;
    W.mode = mode;
    adj_curv<K><<<W.ncurv, 32 * kCurvFacets, 0, s>>>(dP, W, args);
    bool masked = !ordinary_scattering(exp(args.a[P.C + 6]), args.a[P.C + 7]);
    for (int k = 0; mode == kAdjProduct && k < P.C; k++) masked = masked || !(fabs(args.v[k]) < 1e200);
    const dim3 pgrid(cdiv(P.n_points, kPtThreads), W.nfs);
    if (masked)
        adj_points<K, true><<<pgrid, kPtThreads, 0, s>>>(dP, W);
    else
        adj_points<K, false><<<pgrid, kPtThreads, 0, s>>>(dP, W);
    if (P.n_ablocks > 0) {
        adj_sums<K><<<P.n_ablocks, kRowThreads, 0, s>>>(dP, W);
        adj_rows<K, false><<<P.n_arows, kRowThreads, 0, s>>>(dP, W);
    } else {
        adj_rows<K, true><<<P.n_arows, kRowThreads, 0, s>>>(dP, W);
    }
    adj_facets<K><<<dim3(cdiv(P.F, kFcThreads), W.npb), kFcThreads, 0, s>>>(dP, W);
    adj_cols<K><<<W.ncol, 128, 0, s>>>(dP, W);
    adj_out<K><<<dim3(P.mfit + 1, K), kOutThreads, 0, s>>>(dP, W, P.n_arows);
    return cudaGetLastError();
}

}  // namespace

size_t adjoint_work_doubles(const DevProblem& P, bool batched) {
    AdjWork W{};
    const size_t one = carve<1>(P, nullptr, W);
    if (!batched) return one;
    const size_t all = carve<kAdjDirs>(P, nullptr, W);
    return one > all ? one : all;
}

cudaError_t launch_adjoint(const DevProblem& P, const DevProblem* dP, double* work, const AdjArgs& args, AdjMode mode,
                           double* d_out, double* d_chi2, cudaStream_t s) {
    if (mode == kAdjUnits) return launch<kAdjDirs>(P, dP, work, args, mode, d_out, d_chi2, s);
    return launch<1>(P, dP, work, args, mode, d_out, d_chi2, s);
}

}  // namespace psb
