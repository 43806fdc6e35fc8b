// cpb_groups.cu -- many small simultaneous fits in one persistent launch.
//
// A "group" is a small field holding a blend of a few stars; each group is an
// independent fit_all_stars_simultaneous call
// (src/photometry/psf_photometry_simultaneous.jl:953-1431).  One thread
// block owns one group for the whole fit and keeps every working array of it
// in shared memory:
//
//   * the union U of the stars' fit-box pixels (_touched_pixels, :329-335),
//     sorted in the group image's column-major order, with the weighted
//     residual and the LSQR u vector per pixel of U (data_work and sqrt(w) in
//     the block's slice of global memory) -- the reference's npix-long vectors
//     are zero outside U, so nothing else is kept;
//   * per pixel of U, bit masks of the (Morton-ordered) active stars whose fit
//     box and model box contain it.  J v, the renders and the frozen-star
//     subtraction are gathers over those bits in ascending (Morton) order,
//     which is the order in which the reference's scatter-adds reach the pixel
//     (apply_J! :95-137, _render_model! :545-673, _freeze_star! :739-754);
//   * the stamp derivatives V (StampDerivatives, :19-43) with, per stamp
//     entry, its index in U (0 = unusable entry, as the reference's pixel 0);
//   * per star the solver state (theta, colnorm, D, b, LSQR x / v / w).
//
// Renders are evaluated only on U: the residual, cost and data_work are read
// only there (_residual_cost! :675-684, _cost! :686-693), so values of the
// model boxes outside U never influence the fit.  The final residual image
// and the diagnostics evaluate the full model boxes.  Blocks take groups from
// a device work queue (an atomic counter), so groups of uneven size share the
// GPU without a host round trip.  All reductions use a fixed order (results
// are bitwise reproducible run to run); the host never reads anything back
// until the batch is done.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <limits>
#include <string>
#include <vector>

#include "cpb_internal.cuh"
#include "cpb_linalg.cuh"

namespace cpb {

namespace {

constexpr double kEpsG = 2.220446049250313e-16;
constexpr int kMaxGroupStars = 64;
constexpr int kNoU = 0x7fffffff;
constexpr uint16_t kNoU16 = 0xffff;  // unusable stamp entry

struct GroupConst {
    int p;
    int gc[3];     // grad_col of free parameter k (1 = dy, 2 = dx, 3 = dflux)
    int ky, kx;    // position of y / x in the free list, -1 if fixed
    double fixed_y, fixed_x, fixed_flux, fixed_bkg;
    int R, S, S2;  // fit box
    int mR;        // model radius (scalar model_rad)
    int nmax;      // star capacity of the shared-memory layout
    int umax;      // union-pixel capacity
    int keyn;      // power-of-two key buffer for the union sort (>= nmax * S2)
    int same;      // model radius = fit half-width: one star mask a pixel
    unsigned Smag; // quot_magic(S)
    int max_iter, max_trials, itmax;
    double linear_tol, max_step, x_tol, f_tol, g_tol;
    double lambda_init, lambda_up, lambda_down, lambda_min, lambda_max;
    int eltype;
    int reweighted;
    double fit_rad;
    // spread_model: on when requested and its disk width is NaN (derived per
    // group) or finite and positive; the disk table length and the fit box
    // capacity ((2 R + 2)^2 pixels)
    int sp_on, sp_tab, sp_box;
    double sp_param;     // spread_model_fwhm (NaN: _spread_fwhm of the group's first star)
    double sp_psf_fwhm;  // the PSF object's own FWHM, which _spread_fwhm renders
};

struct GroupIn {
    const int64_t* pix_off;
    const int32_t* ny;
    const int32_t* nx;
    const void* pix;
    const void* iv;   // nullable
    const void* bkg;  // nullable
    const int64_t* star_off;
    const double *y0, *x0, *f0;
};

struct GroupOut {
    double *y, *x, *flux, *y_err, *x_err, *flux_err;
    uint8_t *converged, *valid;
    int32_t* n_iter;
    double *chisq, *qfit, *qfit_expected, *qfit_z, *crowding;
    double* residual;
    int32_t *n_passes, *n_failed, *status, *error_kind, *n_active, *n_union, *n_trials, *n_lsqr;
    double *spread, *spread_err;
    double* px;             // a block: data_work and sqrt(w) of its group's union, 2 umax doubles
    double* sp_rw;          // per star: residual and weight over its box, 2 sp_box doubles (spread_model)
    const double* sp_rule;  // kSpreadRuleLen doubles (spread_rule)
};

// q / d for q < 2^31 without a division: quot_magic(d) = min(floor(2^32 / d), 2^32 - 1),
// whose product with q is short of 2^32 q / d by less than 2^32, so the high word is the
// quotient or one below it.
__host__ __device__ inline unsigned quot_magic(unsigned d) {
    return d <= 1 ? 0xffffffffu : (unsigned)(0x100000000ull / d);
}
__device__ __forceinline__ int quot(int q, int d, unsigned magic, int& rem) {
    int k = (int)__umulhi((unsigned)q, magic);
    rem = q - k * d;
    if (rem >= d) {
        rem -= d;
        ++k;
    }
    return k;
}

// Byte offsets of the shared-memory layout (same computation on host and device).
// node: single-node image PSF (a NodeStar a star).
struct Layout {
    size_t coef, ns, theta, delta, dsc, cn, D, bsc, xl, vt, wl;
    size_t ay, ax, act, frozen, live, conv, newf;
    size_t V, uidx;
    size_t wr, u, upix, fmask, mmask;
    size_t total;
};

__host__ __device__ inline size_t align16(size_t v) { return (v + 15) & ~(size_t)15; }

template <typename MaskT>
__host__ __device__ inline Layout make_layout(int nmax, int S2, int umax, int keyn, bool node, bool same) {
    Layout L;
    size_t o = 0;
    auto take = [&](size_t bytes) {
        size_t at = o;
        o = align16(o + bytes);
        return at;
    };
    const size_t np = (size_t)3 * nmax;
    L.coef = take(sizeof(StarCoef) * nmax);
    L.ns = take(node ? sizeof(NodeStar<false>) * nmax : 0);
    L.theta = take(8 * np);
    L.delta = take(8 * np);
    L.dsc = take(8 * np);
    L.cn = take(8 * np);
    L.D = take(8 * np);
    L.bsc = take(8 * np);
    L.xl = take(8 * np);
    L.vt = take(8 * np);
    L.wl = take(8 * np);
    L.ay = take(4 * nmax);
    L.ax = take(4 * nmax);
    L.act = take(4 * nmax);
    L.frozen = take(4 * nmax);
    L.live = take(nmax);
    L.conv = take(nmax);
    L.newf = take(nmax);
    // V doubles as the bit map (or key buffer) of the union (keyn int32 <= 3 * 8 * nmax * S2 bytes)
    size_t vbytes = (size_t)24 * nmax * S2;
    if (vbytes < (size_t)4 * keyn) vbytes = (size_t)4 * keyn;
    L.V = take(vbytes);
    L.uidx = take((size_t)2 * nmax * S2);
    L.wr = take((size_t)8 * umax);
    L.u = take((size_t)8 * umax);
    L.upix = take((size_t)4 * umax);
    L.fmask = take(sizeof(MaskT) * umax);
    L.mmask = same ? L.fmask : take(sizeof(MaskT) * umax);
    L.total = o;
    return L;
}

__device__ __forceinline__ uint64_t spread_bits(uint64_t v) {
    v &= 0x00000000ffffffffULL;
    v = (v | (v << 16)) & 0x0000ffff0000ffffULL;
    v = (v | (v << 8)) & 0x00ff00ff00ff00ffULL;
    v = (v | (v << 4)) & 0x0f0f0f0f0f0f0f0fULL;
    v = (v | (v << 2)) & 0x3333333333333333ULL;
    v = (v | (v << 1)) & 0x5555555555555555ULL;
    return v;
}

// Block-wide sum / max whose result every thread receives.  `buf` alternates
// between two 32-entry halves so that consecutive reductions need one barrier each.
template <int NT>
__device__ __forceinline__ double block_allsum(double v, double* sh, int& flip) {
    double* b = sh + 32 * (flip & 1);
    ++flip;
    v = warp_sum(v);
    if ((threadIdx.x & 31) == 0) b[threadIdx.x >> 5] = v;
    __syncthreads();
    double r = 0.0;
#pragma unroll
    for (int k = 0; k < NT / 32; ++k) r += b[k];
    return r;
}
template <int NT>
__device__ __forceinline__ double block_allmax(double v, double* sh, int& flip) {
    double* b = sh + 32 * (flip & 1);
    ++flip;
    v = warp_max(v);
    if ((threadIdx.x & 31) == 0) b[threadIdx.x >> 5] = v;
    __syncthreads();
    double r = 0.0;
#pragma unroll
    for (int k = 0; k < NT / 32; ++k) r = nan_max(r, b[k]);
    return r;
}

template <typename MaskT>
__device__ __forceinline__ int next_bit(MaskT& m) {
    int a;
    if (sizeof(MaskT) == 8) a = __ffsll((long long)m) - 1;
    else a = __ffs((int)m) - 1;
    m &= m - 1;
    return a;
}

// Per-group view of the inputs.
struct GView {
    GroupIn in;
    int eltype;
    int64_t off;
    int ny, nx;
    __device__ double ld(const void* p, int64_t q) const {
        return eltype == CPB_F64 ? ((const double*)p)[off + q] : (double)((const float*)p)[off + q];
    }
    // sanitised data (image - background; non-finite -> 0) and weight (:1056-1084)
    __device__ void data_w(int64_t q, double& d, double& w) const {
        d = ld(in.pix, q) - (in.bkg ? ld(in.bkg, q) : 0.0);
        if (in.iv) {
            const double v = ld(in.iv, q);
            w = (isfinite(v) && v > 0) ? v : 0.0;
        } else {
            w = 1.0;
        }
        if (!isfinite(d)) {
            d = 0.0;
            w = 0.0;
        }
    }
};

__device__ __forceinline__ double psf_value(const DevPsf& P, const StarCoef& c, int gy, int gx) {
    return model_value<double, double>(P, P.data64, c, (double)gy, (double)gx);
}
__device__ __forceinline__ void psf_grad(const DevPsf& P, const StarCoef& c, int gy, int gx, double* g) {
    model_grad<double, double>(P, P.data64, c, (double)gy, (double)gx, g);
}

// One group's fit by one block.  What bounds it: latency -- a group is a few hundred to
// two thousand pixels, so every step is a short dependent chain between block barriers.
// Hence two resident 256-thread blocks an SM (see plan_tiers); per-star cubic weights
// (NodeStar) instead of a stencil worked out at every pixel; the accepted candidate's
// residual kept as the next iteration's; and in LSQR the scalar recurrences, stopping
// tests and the update of x and w on warp 0 while the other warps already gather the next
// J v.  4,000 groups of 2-12 stars measured on the
// B200: 13.6 ms with one block an SM, generic stencils and three barriers an iteration,
// 7.2 ms now; 60 Gaussian groups 421 and 350 us.
template <int NT, typename MaskT, bool NODE>
struct GroupFit {
    static constexpr int NW = NT / 32;
    // warps that leave the next J v to the others while warp 0 works the scalars: with two
    // warps that would be half the block, so there both gather
    static constexpr bool kSplit = NW >= 4;
    const GroupConst& C;
    const DevPsf& P;
    const PPNode& N;
    const GroupOut& O;
    GView G;
    char* smem;
    Layout L;
    double *dw, *sw;  // data_work and sqrt(w) of the union, in global memory: read in order, once a render
    double* sh;       // 64 doubles of reduction scratch
    int* s_stop;      // 2 flags, used in turn
    int flip = 0;
    int n_act = 0, nU = 0;
    unsigned nymag = 0;

    __device__ StarCoef* coef() const { return (StarCoef*)(smem + L.coef); }
    __device__ NodeStar<false>* ns() const { return (NodeStar<false>*)(smem + L.ns); }
    __device__ double* dp(size_t o) const { return (double*)(smem + o); }
    __device__ int32_t* ip(size_t o) const { return (int32_t*)(smem + o); }
    __device__ uint16_t* hp(size_t o) const { return (uint16_t*)(smem + o); }
    __device__ uint8_t* bp(size_t o) const { return (uint8_t*)(smem + o); }
    __device__ MaskT* mp(size_t o) const { return (MaskT*)(smem + o); }

    // model_from_vector (psf_fitting.jl:23-26) for active slot a at theta (+ delta).
    __device__ void make_coef(int a, const double* th, const double* dl, StarCoef& c) const {
        c.y = C.fixed_y;
        c.x = C.fixed_x;
        c.flux = C.fixed_flux;
        c.bkg = C.fixed_bkg;
        for (int k = 0; k < C.p; ++k) {
            double v = th[a * C.p + k];
            if (dl) v = v + dl[a * C.p + k];
            if (C.gc[k] == 1) c.y = v;
            else if (C.gc[k] == 2) c.x = v;
            else c.flux = v;
        }
        if (!NODE) grid_corners_dw(P, c.y, c.x, c);
    }
    // Star a's model at pixel (gy, gx) of its model box.
    __device__ double mval(int a, int gy, int gx) const {
        if (NODE) {
            const StarCoef& c = coef()[a];
            return c.flux * ns()[a].value(N, N.pp, gy - ip(L.ay)[a] + C.mR, gx - ip(L.ax)[a] + C.mR) + c.bkg;
        }
        return psf_value(P, coef()[a], gy, gx);
    }
    __device__ void uxy(int u, int& gy, int& gx) const {
        int r;
        gx = quot(ip(L.upix)[u], G.ny, nymag, r) + 1;
        gy = r + 1;
    }
    // stamp entry m = row + col S
    __device__ int srow(int m, int& col) const {
        int r;
        col = quot(m, C.S, C.Smag, r);
        return r;
    }

    // Block-wide sum of the warps' lane-0 values, in warp order; one barrier.
    __device__ double warps_sum(double lane0) {
        double* b = sh + 32 * (flip & 1);
        ++flip;
        if ((threadIdx.x & 31) == 0) b[threadIdx.x >> 5] = lane0;
        __syncthreads();
        double r = 0.0;
#pragma unroll
        for (int k = 0; k < NW; ++k) r += b[k];
        return r;
    }

    // coef[a] (and the star's weights over its model box) for every active slot at theta
    // (+ delta), a warp a star.
    __device__ void coefs(bool cand) {
        const double* th = dp(L.theta);
        for (int a = threadIdx.x >> 5; a < n_act; a += NW) {
            StarCoef c;
            make_coef(a, th, cand ? dp(L.delta) : nullptr, c);
            if (NODE) {
                NodeStar<false> S;
                const int n = 2 * C.mR + 1;
                S.set(N, c.y, c.x, ip(L.ay)[a] - C.mR, ip(L.ax)[a] - C.mR, n, n);
                if ((threadIdx.x & 31) == 0) {
                    ns()[a] = S;
                    StarCoef& t = coef()[a];
                    t.y = c.y;
                    t.x = c.x;
                    t.flux = c.flux;
                    t.bkg = c.bkg;
                }
            } else if ((threadIdx.x & 31) == 0) {
                coef()[a] = c;
            }
        }
        __syncthreads();
    }

    // _fill_stamps! (:342-543) for the live stars (all when `all`); with `gram`
    // the per-star p x p Gram block of the raw columns is written instead of V
    // (errors pass, :1302-1329).  One warp per star.  V is zero at unusable entries.
    __device__ void fill(bool all, double* gram) {
        const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
        const int p = C.p, S2 = C.S2, R = C.R;
        double* V = dp(L.V);
        const uint16_t* ui = hp(L.uidx);
        double* cn = dp(L.cn);
        const uint8_t* live = bp(L.live);
        for (int a = wid; a < n_act; a += NW) {
            if (!all && !live[a]) continue;
            StarCoef c;
            NodeStar<false> T;
            if (NODE) {
                T = ns()[a];
                c.flux = coef()[a].flux;
            } else {
                c = coef()[a];
            }
            const int ay = ip(L.ay)[a], ax = ip(L.ax)[a];
            double s0 = 0, s1 = 0, s2 = 0, g01 = 0, g02 = 0, g12 = 0;
            for (int m = lane; m < S2; m += 32) {
                const int u = ui[a * S2 + m];
                double r[3] = {0, 0, 0};
                if (u != kNoU16) {
                    int col;
                    const int row = srow(m, col);
                    double g[3];
                    if (NODE) {
                        const int i = row - R + C.mR, j = col - R + C.mR;
                        g[0] = g[1] = c.flux * 0.0;
                        g[2] = N.nd.fill;
                        if (i >= T.sy.lo && i <= T.sy.hi && j >= T.sx.lo && j <= T.sx.hi) {
                            double rv[4], rd[4];
                            T.template rows<true>(N.pp, i, j, rv, rd);
                            const double dv = T.dy[0] * rv[0] + T.dy[1] * rv[1] + T.dy[2] * rv[2] + T.dy[3] * rv[3];
                            const double du = T.wy[0] * rd[0] + T.wy[1] * rd[1] + T.wy[2] * rd[2] + T.wy[3] * rd[3];
                            g[0] = c.flux * -(N.nd.sy * dv);
                            g[1] = c.flux * -(N.nd.sx * du);
                            g[2] = T.wy[0] * rv[0] + T.wy[1] * rv[1] + T.wy[2] * rv[2] + T.wy[3] * rv[3];
                        }
                    } else {
                        psf_grad(P, c, ay + row - R, ax + col - R, g);
                    }
                    const double swv = sw[u];
#pragma unroll
                    for (int k = 0; k < 3; ++k)
                        if (k < p) r[k] = swv * (C.gc[k] == 1 ? g[0] : (C.gc[k] == 2 ? g[1] : g[2]));
                }
                if (!gram) {
#pragma unroll
                    for (int k = 0; k < 3; ++k)
                        if (k < p) V[(a * S2 + m) * p + k] = r[k];
                }
                s0 += r[0] * r[0];
                s1 += r[1] * r[1];
                s2 += r[2] * r[2];
                g01 += r[0] * r[1];
                g02 += r[0] * r[2];
                g12 += r[1] * r[2];
            }
            s0 = warp_sum(s0);
            s1 = warp_sum(s1);
            s2 = warp_sum(s2);
            if (gram) {
                g01 = warp_sum(g01);
                g02 = warp_sum(g02);
                g12 = warp_sum(g12);
                if (lane == 0) {
                    double* gr = gram + a * 6;
                    gr[0] = s0;
                    gr[1] = g01;
                    gr[2] = g02;
                    gr[3] = s1;
                    gr[4] = g12;
                    gr[5] = s2;
                }
                continue;
            }
            const double ss[3] = {__shfl_sync(0xffffffffu, s0, 0), __shfl_sync(0xffffffffu, s1, 0),
                                  __shfl_sync(0xffffffffu, s2, 0)};
            double inv[3] = {0, 0, 0};
#pragma unroll
            for (int k = 0; k < 3; ++k)
                if (k < p) {
                    double cv = sqrt(ss[k]);
                    cv = cv < kEpsG ? kEpsG : cv;
                    inv[k] = 1.0 / cv;
                    if (lane == 0) cn[a * p + k] = cv;
                }
            for (int m = lane; m < S2; m += 32) {
#pragma unroll
                for (int k = 0; k < 3; ++k)
                    if (k < p) V[(a * S2 + m) * p + k] *= inv[k];
            }
        }
        __syncthreads();
    }

    // sqrt(w) (model - data_work) on U into `to` and its cost, for the stars in `sel` (bit
    // a = active slot a); `freeze`: data_work -= model (frozen-star subtraction) instead.
    __device__ double render(bool freeze, MaskT sel, double* to) {
        const MaskT* mm = mp(L.mmask);
        double part = 0.0;
        for (int u = threadIdx.x; u < nU; u += NT) {
            int gy, gx;
            uxy(u, gy, gx);
            MaskT m = mm[u] & sel;
            if (freeze) {
                double d = dw[u];
                while (m) d -= mval(next_bit(m), gy, gx);
                dw[u] = d;
                continue;
            }
            double acc = 0.0;
            while (m) acc += mval(next_bit(m), gy, gx);
            const double v = sw[u] * (acc - dw[u]);
            to[u] = v;
            part += v * v;
        }
        if (freeze) {
            __syncthreads();
            return 0.0;
        }
        return block_allsum<NT>(part, sh, flip);
    }

    // z = J^T src * scale for the live stars (apply_JT!, :55-85), one warp per
    // star.  LSQR form: v_new = z - beta v_old / alpha, returns ||v_new||^2.
    __device__ double jt(const double* src, double scale, bool lsqr, double beta, double inv_alpha, double* z) {
        const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
        const int p = C.p, S2 = C.S2;
        const double* V = dp(L.V);
        const uint16_t* ui = hp(L.uidx);
        const uint8_t* live = bp(L.live);
        double part = 0.0;
        for (int a = wid; a < n_act; a += NW) {
            if (!live[a]) continue;
            double z0 = 0, z1 = 0, z2 = 0;
#pragma unroll 2
            for (int m = lane; m < S2; m += 32) {
                const int u = ui[a * S2 + m];
                double uv = u == kNoU16 ? 0.0 : src[u];
                if (lsqr) uv *= scale;
                const double* v = V + (a * S2 + m) * p;
                z0 += v[0] * uv;
                if (p > 1) z1 += v[1] * uv;
                if (p > 2) z2 += v[2] * uv;
            }
            z0 = warp_sum(z0);
            if (p > 1) z1 = warp_sum(z1);
            if (p > 2) z2 = warp_sum(z2);
            if (lane == 0) {
                for (int k = 0; k < p; ++k) {
                    double val = k == 0 ? z0 : (k == 1 ? z1 : z2);
                    if (lsqr) {
                        val = val - beta * (z[a * p + k] * inv_alpha);
                        part += val * val;
                    }
                    z[a * p + k] = val;
                }
            }
        }
        if (!lsqr) {
            __syncthreads();
            return 0.0;
        }
        return warps_sum(part);
    }

    // u_new = J v / alpha - alpha u_old (apply_J!, :95-137, gathered per pixel of
    // U in Morton order); u_old = src * uscale.  Returns the calling thread's part of
    // ||u_new||^2 over the pixels t0, t0 + tn, ...
    __device__ double jv(const double* src, double uscale, double alpha, double inv_alpha, MaskT live_bits, int t0,
                         int tn) {
        const int p = C.p, S = C.S, S2 = C.S2, R = C.R;
        const double* V = dp(L.V);
        const double* vt = dp(L.vt);
        const MaskT* fm = mp(L.fmask);
        const int32_t* ay = ip(L.ay);
        const int32_t* ax = ip(L.ax);
        double* uu = dp(L.u);
        double part = 0.0;
        for (int u = t0; u < nU; u += tn) {
            int gy, gx;
            uxy(u, gy, gx);
            MaskT m = fm[u] & live_bits;
            double acc = 0.0;
            while (m) {
                const int a = next_bit(m);
                const int mi = (gy - ay[a] + R) + (gx - ax[a] + R) * S;
                const double* v = V + (a * S2 + mi) * p;
                double t = v[0] * (vt[a * p] * inv_alpha);
                if (p > 1) t += v[1] * (vt[a * p + 1] * inv_alpha);
                if (p > 2) t += v[2] * (vt[a * p + 2] * inv_alpha);
                acc += t;
            }
            const double un = acc - alpha * (src[u] * uscale);
            uu[u] = un;
            part += un * un;
        }
        return part;
    }

    // Damped LSQR (Paige & Saunders 1982, Krylov.jl 0.10 stopping rules) on
    // min ||J d + r||^2 + lambda ||d||^2, right-hand side -wr, zero start.
    // Returns the iterations run.  Two barriers an iteration: after J' u, and after the
    // step in which warp 0 works the scalars, x, w and the stopping tests while the others
    // gather the next iteration's J v (whose u is simply not used after a stop).
    __device__ int lsqr(double cost, double lam, MaskT live_bits) {
        const int n = n_act * C.p, lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
        double* xl = dp(L.xl);
        double* vt = dp(L.vt);
        double* wl = dp(L.wl);
        const double* bsc = dp(L.bsc);
        const double beta1 = sqrt(cost);
        if (wid == 0)
            for (int i = lane; i < n; i += 32) xl[i] = 0.0;
        if (beta1 == 0.0) {
            __syncthreads();
            return 0;
        }
        const double inv_b1 = 1.0 / beta1;
        // v1 = A'u1 = -b / beta1 (the gradient pass already holds A'r); every warp sums its norm
        double part = 0.0;
        for (int i = lane; i < n; i += 32) {
            const double v = -(bsc[i] * inv_b1);
            if (wid == 0) vt[i] = v;
            part += v * v;
        }
        const double a2 = __shfl_sync(0xffffffffu, warp_sum(part), 0);
        double alpha = sqrt(a2);
        const double t0 = (alpha * beta1) / (alpha * beta1);
        if (alpha == 0.0 || t0 <= 1.4901161193847656e-08 || 1.0 + t0 <= 1.0) {
            __syncthreads();
            return 0;
        }
        double inv_alpha = 1.0 / alpha;
        double wnorm2 = 0.0, c1 = 0, s1 = 0, rhobar1 = 0;
        const double lambda = sqrt(lam);
        if (wid == 0) {
            part = 0.0;
            for (int i = lane; i < n; i += 32) {
                const double v = vt[i] * inv_alpha;
                wl[i] = v;
                part += v * v;
            }
            wnorm2 = __shfl_sync(0xffffffffu, warp_sum(part), 0);
            sym_givens(alpha, lambda, c1, s1, rhobar1);
        }
        __syncthreads();
        double Anorm2 = a2, dNorm2 = 0, xNorm2 = 0, c2 = -1, s2 = 0, xENorm2 = 0, res2 = 0, rhs = 0, gamma = 1;
        double phibar = beta1, inv_beta = inv_b1;
        double err_vec[5] = {0, 0, 0, 0, 0};
        const double atol = C.linear_tol, btol = C.linear_tol;
        const double axtol = 1.4901161193847656e-08, etol = axtol, ctol = axtol;
        // beta u = A v - alpha u
        double b2 = block_allsum<NT>(jv(dp(L.wr), -inv_beta, alpha, inv_alpha, live_bits, threadIdx.x, NT), sh, flip);
        for (int it = 0;; ++it) {
            const double beta = sqrt(b2);
            const double alpha_old = alpha;
            if (beta != 0.0) {
                inv_beta = 1.0 / beta;
                // alpha v = A'u - beta v
                const double an2 = jt(dp(L.u), inv_beta, true, beta, inv_alpha, vt);
                alpha = sqrt(an2);
                inv_alpha = alpha != 0.0 ? 1.0 / alpha : 0.0;
            }
            const bool last = it + 1 >= C.itmax;
            if (wid == 0) {
                const int iter = it + 1;
                if (beta != 0.0) {
                    Anorm2 = Anorm2 + alpha_old * alpha_old + beta * beta;
                    if (lambda > 0) Anorm2 += lambda * lambda;
                }
                // An FP64 division or root is a chain of 150-250 cycles, and an iteration has 28
                // of them.  The independent ones go to different lanes of one instruction,
                // which leaves 8 in a row (6,000 -> 4,900 cycles an iteration beside the
                // other warps of two blocks an SM): lane k's operands below, results by shuffle.
                const double psi = s1 * phibar;
                phibar = c1 * phibar;
                Rotation g2(rhobar1, beta);
                // z of the iteration before (lane 1) beside this rotation's tangent (the rest)
                double d = (lane == 1 ? rhs : g2.lo) / (lane == 1 ? gamma : g2.hi);
                const double z = __shfl_sync(0xffffffffu, d, 1);
                xNorm2 = xNorm2 + z * z;
                double c, s, rho;
                {
                    const double t = __shfl_sync(0xffffffffu, d, 0);
                    const double q = g2.sign() / sqrt(1.0 + t * t);
                    g2.finish(t, q, g2.hi / q, c, s, rho);
                }
                const double phi = c * phibar;
                phibar = s * phibar;
                const double theta = s * alpha, tau = s * phi;
                const double delta = s2 * rho, gambar = -c2 * rho;
                rhs = phi - delta * z;
                // lane 4: the rotation of (gambar, theta); lane 5: the next iteration's of
                // (rhobar, lambda); lanes 0-3: sigma, the w factor, |w|^2 / rho^2, zbar
                Rotation g3(lane == 4 ? gambar : -c * alpha, lane == 4 ? theta : lambda);
                const bool rot = lane == 4 || lane == 5;
                {
                    const double num = rot ? g3.lo : (lane == 1 ? -theta : (lane == 2 ? wnorm2 : (lane == 3 ? rhs : phi)));
                    const double den = rot ? g3.hi : (lane == 2 ? rho * rho : (lane == 3 ? gambar : rho));
                    d = num / den;
                }
                const double tan3 = d;
                const double sigma = __shfl_sync(0xffffffffu, d, 0), tr = __shfl_sync(0xffffffffu, d, 1);
                dNorm2 = dNorm2 + __shfl_sync(0xffffffffu, d, 2);
                const double zbar = __shfl_sync(0xffffffffu, d, 3);
                part = 0.0;
                for (int i = lane; i < n; i += 32) {
                    const double wi = wl[i];
                    xl[i] = xl[i] + sigma * wi;
                    const double wn = vt[i] * inv_alpha + tr * wi;
                    wl[i] = wn;
                    part += wn * wn;
                }
                wnorm2 = __shfl_sync(0xffffffffu, warp_sum(part), 0);
                xENorm2 = xENorm2 + phi * phi;
                double e2 = 0;
#pragma unroll
                for (int k = 0; k < 5; ++k) {
                    if (k == iter % 5) err_vec[k] = phi;
                    e2 += err_vec[k] * err_vec[k];
                }
                const double res1 = phibar * phibar;
                res2 = res2 + psi * psi;
                d = sqrt(rot         ? 1.0 + tan3 * tan3
                         : lane == 1 ? dNorm2
                         : lane == 2 ? res1 + res2
                         : lane == 3 ? e2
                         : lane == 6 ? Anorm2
                         : lane == 7 ? xENorm2
                                     : xNorm2 + zbar * zbar);
                const double xNorm = __shfl_sync(0xffffffffu, d, 0);
                const double rNorm = __shfl_sync(0xffffffffu, d, 2);
                const double err_lbnd = __shfl_sync(0xffffffffu, d, 3);
                const double Anorm = __shfl_sync(0xffffffffu, d, 6);
                const double Acond = Anorm * __shfl_sync(0xffffffffu, d, 1);
                const double xENorm = __shfl_sync(0xffffffffu, d, 7);
                const double ArNorm = alpha * fabs(tau);
                {
                    const double num = rot         ? g3.sign()
                                       : lane == 1 ? ArNorm
                                       : lane == 2 ? 1.0
                                       : lane == 3 ? Anorm * xNorm
                                       : lane == 6 ? axtol * Anorm * xNorm
                                                   : rNorm;
                    const double den = rot ? d : (lane == 1 ? Anorm * rNorm : (lane == 2 ? Acond : beta1));
                    d = num / den;
                }
                const double q3 = d;
                const double test1 = __shfl_sync(0xffffffffu, d, 0);
                const double test2 = __shfl_sync(0xffffffffu, d, 1);
                const double test3 = __shfl_sync(0xffffffffu, d, 2);
                const double xrel = __shfl_sync(0xffffffffu, d, 3);
                const double rNormtol = btol + __shfl_sync(0xffffffffu, d, 6);
                d = (rot ? g3.hi : test1) / (rot ? q3 : 1.0 + xrel);
                const double t1 = __shfl_sync(0xffffffffu, d, 0);
                double cr, sr, rr;
                g3.finish(tan3, q3, d, cr, sr, rr);
                c2 = __shfl_sync(0xffffffffu, cr, 4);
                s2 = __shfl_sync(0xffffffffu, sr, 4);
                gamma = __shfl_sync(0xffffffffu, rr, 4);
                c1 = __shfl_sync(0xffffffffu, cr, 5);
                s1 = __shfl_sync(0xffffffffu, sr, 5);
                rhobar1 = __shfl_sync(0xffffffffu, rr, 5);
                const bool ill = (1.0 + test3 <= 1.0) || (test3 <= ctol);
                const bool zr = (1.0 + t1 <= 1.0) || (test1 <= rNormtol);
                const bool fwd = iter >= 5 && err_lbnd <= etol * xENorm;
                const bool solved = (1.0 + test2 <= 1.0) || (test2 <= axtol) || (ArNorm <= atol) || zr || fwd;
                if (lane == 0) s_stop[it & 1] = solved || ill;
            }
            part = 0.0;
            if (!last && (!kSplit || wid != 0))
                part = jv(dp(L.u), inv_beta, alpha, inv_alpha, live_bits, kSplit ? threadIdx.x - 32 : threadIdx.x,
                          kSplit ? NT - 32 : NT);
            b2 = block_allsum<NT>(part, sh, flip);
            if (last || s_stop[it & 1]) return it + 1;
        }
    }
};

// Groups come from glist[0 .. nlist) through the queue counter, then from ovf_in (nullable;
// its count *ovf_n_in, complete before the launch).  A group whose union exceeds the
// layout's umax is appended to ovf_out and left to the next launch (without ovf_out the
// layout holds any union of its groups).
template <int NT, typename MaskT, bool NODE>
__global__ void __launch_bounds__(NT, 512 / NT) k_groups(GroupConst C, DevPsf P, GroupIn in, GroupOut O,
                                                         const int32_t* __restrict__ glist, int nlist, int* queue,
                                                         const int32_t* __restrict__ ovf_in, const int* ovf_n_in,
                                                         int32_t* ovf_out, int* ovf_n_out) {
    extern __shared__ __align__(16) char smem[];
    __shared__ double sh[64];
    __shared__ int s_g;
    __shared__ double s_gram[kMaxGroupStars * 6];
    __shared__ uint64_t s_key[kMaxGroupStars];
    __shared__ int s_ay0[kMaxGroupStars], s_ax0[kMaxGroupStars];
    __shared__ uint8_t s_ok[kMaxGroupStars];
    const double NaN = __longlong_as_double(0x7ff8000000000000LL);
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    __shared__ PPNode s_node;
    __shared__ int s_stop[2];
    if (NODE && tid == 0) node_of(P, s_node);
    const int n_ovf = ovf_in ? *ovf_n_in : 0;
    GroupFit<NT, MaskT, NODE> F{C, P, s_node, O};
    F.smem = smem;
    F.L = make_layout<MaskT>(C.nmax, C.S2, C.umax, C.keyn, NODE, C.same);
    F.sh = sh;
    F.s_stop = s_stop;
    F.dw = O.px + (size_t)blockIdx.x * 2 * C.umax;
    F.sw = F.dw + C.umax;
    F.G.in = in;
    F.G.eltype = C.eltype;
    const int p = C.p, S = C.S, S2 = C.S2, R = C.R;
    for (;;) {
        if (tid == 0) s_g = atomicAdd(queue, 1);
        __syncthreads();
        const int li = s_g;
        __syncthreads();
        if (li >= nlist + n_ovf) break;
        const int g = li < nlist ? glist[li] : ovf_in[li - nlist];
        const int64_t soff = in.star_off[g];
        const int ng = (int)(in.star_off[g + 1] - soff);
        F.G.off = in.pix_off[g];
        F.G.ny = in.ny[g];
        F.G.nx = in.nx[g];
        const int ny = F.G.ny, nx = F.G.nx;
        F.nymag = quot_magic((unsigned)ny);
        const int64_t npix = (int64_t)ny * nx;
        const double* y0 = in.y0 + soff;
        const double* x0 = in.x0 + soff;
        const double* f0 = in.f0 + soff;
        // outputs that hold the catalogue (failed / empty groups, inactive stars)
        auto write_catalogue = [&](int i) {
            const int64_t o = soff + i;
            O.y[o] = y0[i];
            O.x[o] = x0[i];
            O.flux[o] = f0[i];
            O.y_err[o] = NaN;
            O.x_err[o] = NaN;
            O.flux_err[o] = NaN;
            O.converged[o] = 0;
            O.valid[o] = 0;
            O.n_iter[o] = 0;
            if (O.chisq) O.chisq[o] = 0.0;
            if (O.qfit) O.qfit[o] = NaN;
            if (O.qfit_expected) O.qfit_expected[o] = NaN;
            if (O.qfit_z) O.qfit_z[o] = NaN;
            if (O.crowding) O.crowding[o] = NaN;
            if (O.spread) O.spread[o] = NaN;
            if (O.spread_err) O.spread_err[o] = NaN;
        };
        auto fixed_fix = [&](int64_t o) {  // fixed parameters take the fixed values, error 0
            bool fy = false, fx = false, ff = false;
            for (int k = 0; k < p; ++k) {
                fy |= C.gc[k] == 1;
                fx |= C.gc[k] == 2;
                ff |= C.gc[k] == 3;
            }
            if (!fy) {
                O.y[o] = C.fixed_y;
                O.y_err[o] = 0.0;
            }
            if (!fx) {
                O.x[o] = C.fixed_x;
                O.x_err[o] = 0.0;
            }
            if (!ff) {
                O.flux[o] = C.fixed_flux;
                O.flux_err[o] = 0.0;
            }
        };
        auto zero_residual = [&]() {
            if (O.residual)
                for (int64_t q = tid; q < npix; q += NT) O.residual[F.G.off + q] = 0.0;
        };
        auto group_stats = [&](int passes, int failed, int status, int kind, int nact, int nun, int ntr, int nls) {
            if (tid != 0) return;
            O.n_passes[g] = passes;
            O.n_failed[g] = failed;
            O.status[g] = status;
            if (O.error_kind) O.error_kind[g] = kind;
            if (O.n_active) O.n_active[g] = nact;
            if (O.n_union) O.n_union[g] = nun;
            if (O.n_trials) O.n_trials[g] = ntr;
            if (O.n_lsqr) O.n_lsqr[g] = nls;
        };
        auto fail_group = [&](int kind) {
            for (int i = tid; i < ng; i += NT) {
                write_catalogue(i);
                fixed_fix(soff + i);
            }
            zero_residual();
            group_stats(0, ng, CPB_ERR_ARGUMENT, kind, 0, 0, 0, 0);
            __syncthreads();
        };
        if (ng == 0) {
            zero_residual();
            group_stats(0, 0, 0, 0, 0, 0, 0, 0);
            __syncthreads();
            continue;
        }
        if (ng > C.nmax || ng > kMaxGroupStars) {  // the host routes such groups elsewhere
            group_stats(0, ng, CPB_ERR_INTERNAL, 0, 0, 0, 0, 0);
            __syncthreads();
            continue;
        }
        // ---- non-finite data without inv_var is an ArgumentError (:1065-1072)
        if (!in.iv) {
            int bad = 0;
            for (int64_t q = tid; q < npix; q += NT) {
                const double d = F.G.ld(in.pix, q) - (in.bkg ? F.G.ld(in.bkg, q) : 0.0);
                bad |= !isfinite(d);
            }
            if (__syncthreads_or(bad)) {
                fail_group(1);
                continue;
            }
        }
        // ---- anchors and usable stamps (_build_stamps!, :245-323)
        for (int i = wid; i < ng; i += NT / 32) {
            const double yy = y0[i], xx = x0[i];
            const bool fin = isfinite(yy) && isfinite(xx) && fabs(yy) < 1e9 && fabs(xx) < 1e9;
            const int ay = fin ? (int)rint(yy) : 0, ax = fin ? (int)rint(xx) : 0;
            int any = 0;
            if (fin)
                for (int m = lane; m < S2; m += 32) {
                    int col;
                    const int row = F.srow(m, col);
                    const int gy = ay + row - R, gx = ax + col - R;
                    if (gy >= 1 && gy <= ny && gx >= 1 && gx <= nx) {
                        double d, w;
                        F.G.data_w((gy - 1) + (int64_t)(gx - 1) * ny, d, w);
                        any |= w > 0;
                    }
                }
            any = __any_sync(0xffffffffu, any);
            if (lane == 0) {
                s_ok[i] = (any && fin && isfinite(f0[i])) ? 1 : 0;
                s_ay0[i] = ay;
                s_ax0[i] = ax;
                s_key[i] = (ay >= 0 && ax >= 0) ? (spread_bits((uint64_t)ay) | (spread_bits((uint64_t)ax) << 1)) : 0;
            }
        }
        __syncthreads();
        // active set in stable Morton order (:306); negative anchors fail (Morton key of a negative Int)
        int* act = F.ip(F.L.act);
        {
            int nok = 0, neg = 0;
            for (int j = 0; j < ng; ++j) {
                nok += s_ok[j];
                neg |= s_ok[j] && (s_ay0[j] < 0 || s_ax0[j] < 0);
            }
            F.n_act = nok;
            if (neg) {
                fail_group(2);
                continue;
            }
            if (tid < ng && s_ok[tid]) {
                const uint64_t k = s_key[tid];
                int rank = 0;
                for (int j = 0; j < ng; ++j)
                    rank += s_ok[j] && (s_key[j] < k || (s_key[j] == k && j < tid));
                act[rank] = tid;
            }
        }
        const int n_act = F.n_act;
        if (n_act == 0) {  // _empty_simultaneous_result (:1433-1445)
            for (int i = tid; i < ng; i += NT) {
                write_catalogue(i);
                fixed_fix(soff + i);
            }
            zero_residual();
            group_stats(0, ng, 0, 0, 0, 0, 0, 0);
            __syncthreads();
            continue;
        }
        __syncthreads();
        int32_t* ay = F.ip(F.L.ay);
        int32_t* ax = F.ip(F.L.ax);
        double* theta = F.dp(F.L.theta);
        uint8_t* live = F.bp(F.L.live);
        uint8_t* conv = F.bp(F.L.conv);
        uint8_t* newf = F.bp(F.L.newf);
        int32_t* frozen = F.ip(F.L.frozen);
        double* cn = F.dp(F.L.cn);
        double* D = F.dp(F.L.D);
        double* bsc = F.dp(F.L.bsc);
        double* delta = F.dp(F.L.delta);
        double* dsc = F.dp(F.L.dsc);
        for (int a = tid; a < n_act; a += NT) {
            const int i = act[a];
            ay[a] = s_ay0[i];
            ax[a] = s_ax0[i];
            for (int k = 0; k < p; ++k)
                theta[a * p + k] = C.gc[k] == 1 ? y0[i] : (C.gc[k] == 2 ? x0[i] : f0[i]);
            live[a] = 1;
            conv[a] = 0;
            newf[a] = 0;
            frozen[a] = 0;
            for (int k = 0; k < p; ++k) cn[a * p + k] = 0.0;
        }
        // ---- union of usable stamp pixels (_touched_pixels, :329-335), in column-major
        // order: a bit map of the boxes' bounding box, where it fits the V region, gives
        // each pixel's place by counting bits (66 sorting steps with a barrier each for a
        // full 12-star group otherwise: 10 % of the fit); stars far apart sort the entries'
        // pixel indices (bitonic) and drop duplicates
        int32_t* upix = F.ip(F.L.upix);
        uint16_t* uidx = F.hp(F.L.uidx);
        const int ne = n_act * S2;
        __shared__ int s_wsum[32];
        // places by a chunked block scan of each thread's count; returns the thread's first
        auto scan = [&](int cnt) {
            int incl = cnt;
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += t;
            }
            if (lane == 31) s_wsum[wid] = incl;
            __syncthreads();
            int wbase = 0, tot = 0;
            for (int k = 0; k < NT / 32; ++k) {
                if (k < wid) wbase += s_wsum[k];
                tot += s_wsum[k];
            }
            F.nU = tot;
            return wbase + incl - cnt;
        };
        int by0 = ny, by1 = 1, bx0 = nx, bx1 = 1;  // the boxes' bounding box, clipped to the image
        for (int j = 0; j < ng; ++j)
            if (s_ok[j]) {
                by0 = min(by0, max(s_ay0[j] - R, 1));
                by1 = max(by1, min(s_ay0[j] + R, ny));
                bx0 = min(bx0, max(s_ax0[j] - R, 1));
                bx1 = max(bx1, min(s_ax0[j] + R, nx));
            }
        const int bh = by1 - by0 + 1, bw = bx1 - bx0 + 1;
        const size_t vbytes = F.L.uidx - F.L.V;
        const int64_t area = (int64_t)bh * bw;
        const bool by_map = ((area + 31) / 32) * 8 <= (int64_t)vbytes;
        if (by_map) {
            const int nwords = (int)((area + 31) / 32);
            unsigned* map = (unsigned*)F.ip(F.L.V);
            int* place = (int*)(map + nwords);
            for (int i = tid; i < nwords; i += NT) map[i] = 0;
            __syncthreads();
            for (int e = tid; e < ne; e += NT) {
                const int a = e / S2;
                int col;
                const int row = F.srow(e - a * S2, col);
                const int gy = ay[a] + row - R, gx = ax[a] + col - R;
                if (gy >= 1 && gy <= ny && gx >= 1 && gx <= nx) {
                    double d, w;
                    F.G.data_w((gy - 1) + (int64_t)(gx - 1) * ny, d, w);
                    const int b = (gy - by0) + (gx - bx0) * bh;
                    if (w > 0) atomicOr(&map[b >> 5], 1u << (b & 31));
                }
            }
            __syncthreads();
            const int per = (nwords + NT - 1) / NT;
            const int b0 = min(tid * per, nwords), b1 = min(b0 + per, nwords);
            int cnt = 0;
            for (int i = b0; i < b1; ++i) cnt += __popc(map[i]);
            int pos = scan(cnt);
            const unsigned bmag = quot_magic((unsigned)bh);
            for (int i = b0; i < b1; ++i) {
                unsigned m = map[i];
                place[i] = pos;
                while (m) {
                    const int b = 32 * i + __ffs((int)m) - 1;
                    m &= m - 1;
                    int r;
                    const int c = quot(b, bh, bmag, r);
                    if (pos < C.umax) upix[pos] = (by0 - 1 + r) + (bx0 - 1 + c) * ny;
                    ++pos;
                }
            }
        } else {
            int32_t* keys = F.ip(F.L.V);
            int kn = 2;
            while (kn < ne) kn <<= 1;
            for (int e = tid; e < kn; e += NT) {
                int key = kNoU;
                if (e < ne) {
                    const int a = e / S2, m = e % S2;
                    const int gy = ay[a] + (m % S) - R, gx = ax[a] + (m / S) - R;
                    if (gy >= 1 && gy <= ny && gx >= 1 && gx <= nx) {
                        const int q = (gy - 1) + (gx - 1) * ny;
                        double d, w;
                        F.G.data_w(q, d, w);
                        if (w > 0) key = q;
                    }
                }
                keys[e] = key;
            }
            __syncthreads();
            for (int k = 2; k <= kn; k <<= 1)
                for (int j = k >> 1; j > 0; j >>= 1) {
                    for (int i = tid; i < kn; i += NT) {
                        const int l = i ^ j;
                        if (l > i) {
                            const int ki = keys[i], kl = keys[l];
                            const bool up = (i & k) == 0;
                            if ((ki > kl) == up) {
                                keys[i] = kl;
                                keys[l] = ki;
                            }
                        }
                    }
                    __syncthreads();
                }
            // compaction of the distinct keys
            const int per = (kn + NT - 1) / NT;
            const int b0 = min(tid * per, kn), b1 = min(b0 + per, kn);
            int cnt = 0;
            for (int e = b0; e < b1; ++e) cnt += keys[e] != kNoU && (e == 0 || keys[e] != keys[e - 1]);
            int pos = scan(cnt);
            for (int e = b0; e < b1; ++e)
                if (keys[e] != kNoU && (e == 0 || keys[e] != keys[e - 1])) {
                    if (pos < C.umax) upix[pos] = keys[e];
                    ++pos;
                }
        }
        if (F.nU > C.umax) {  // block-uniform: left to the launch with the full layout
            if (tid == 0) {
                if (ovf_out) ovf_out[atomicAdd(ovf_n_out, 1)] = g;
                else group_stats(0, ng, CPB_ERR_INTERNAL, 0, 0, 0, 0, 0);
            }
            __syncthreads();
            continue;
        }
        __syncthreads();
        const int nU = F.nU;
        // per stamp entry: its position in U, kNoU16 when unusable
        for (int e = tid; e < ne; e += NT) {
            const int a = e / S2;
            int col;
            const int row = F.srow(e - a * S2, col);
            const int gy = ay[a] + row - R, gx = ax[a] + col - R;
            int r = kNoU16;
            if (gy >= 1 && gy <= ny && gx >= 1 && gx <= nx && by_map) {
                const int b = (gy - by0) + (gx - bx0) * bh;
                const unsigned* map = (const unsigned*)F.ip(F.L.V);
                const unsigned m = map[b >> 5];
                const int* place = (const int*)(map + (area + 31) / 32);
                if (m >> (b & 31) & 1) r = place[b >> 5] + __popc(m & ((1u << (b & 31)) - 1));
            } else if (gy >= 1 && gy <= ny && gx >= 1 && gx <= nx) {
                const int q = (gy - 1) + (gx - 1) * ny;
                int lo = 0, hi = nU;
                while (lo < hi) {
                    const int mid = (lo + hi) >> 1;
                    if (upix[mid] < q) lo = mid + 1;
                    else hi = mid;
                }
                if (lo < nU && upix[lo] == q) r = lo;
            }
            uidx[e] = (uint16_t)r;
        }
        // per pixel of U: data_work, w and the star masks
        {
            MaskT* fm = F.mp(F.L.fmask);
            MaskT* mm = F.mp(F.L.mmask);
            for (int u = tid; u < nU; u += NT) {
                const int q = upix[u];
                double d, w;
                F.G.data_w(q, d, w);
                F.dw[u] = d;
                F.sw[u] = sqrt(w);
                int gy, gx;
                F.uxy(u, gy, gx);
                MaskT f = 0, mo = 0;
                for (int a = 0; a < n_act; ++a) {
                    const int dy = abs(gy - ay[a]), dx = abs(gx - ax[a]);
                    if (dy <= R && dx <= R) f |= (MaskT)1 << a;
                    if (dy <= C.mR && dx <= C.mR) mo |= (MaskT)1 << a;
                }
                fm[u] = f;
                if (!C.same) mm[u] = mo;
            }
        }
        const MaskT all_bits = n_act >= (int)(8 * sizeof(MaskT)) ? ~(MaskT)0 : (((MaskT)1 << n_act) - 1);
        MaskT live_bits = all_bits;
        const int n = n_act * p;
        const double dof = (double)max(nU - n, 1);
        __syncthreads();

        // ---- initial fill and cost (:1171-1178)
        F.coefs(false);
        F.fill(false, nullptr);
        double cost = F.render(false, live_bits, F.dp(F.L.wr));
        for (int i = tid; i < n; i += NT) D[i] = cn[i];
        // the last iteration's step was accepted: coef is at theta and wr, cost are the
        // candidate's (rendered again when stars were frozen, their models gone from
        // data_work); after a rejected one nothing has changed but lambda
        bool moved = false, froze = false;
        double lam = C.lambda_init;
        int n_run = 0, n_trials = 0, n_lsqr = 0;
        // ---- outer loop (:1186-1284)
        for (int iter = 1; iter <= C.max_iter; ++iter) {
            if (moved) {
                F.fill(false, nullptr);
                if (froze) cost = F.render(false, live_bits, F.dp(F.L.wr));
            }
            moved = froze = false;
            for (int i = tid; i < n; i += NT) bsc[i] = 0.0;
            __syncthreads();
            F.jt(F.dp(F.L.wr), 1.0, false, 0.0, 0.0, bsc);
            // global gradient cosine (:1199-1213)
            const double C_r = cost / dof;
            double gmax = 0.0;
            for (int i = tid; i < n; i += NT) {
                const double bt = cn[i] * bsc[i], Aii = cn[i] * cn[i];
                gmax = nan_max(gmax, fabs(bt) / (sqrt(Aii * C_r) + kEpsG));
            }
            const double gnorm = block_allmax<NT>(gmax, sh, F.flip);
            if (gnorm <= C.g_tol) {
                for (int a = tid; a < n_act; a += NT)
                    if (live[a]) {
                        live[a] = 0;
                        frozen[a] = iter - 1;
                        conv[a] = 1;
                    }
                live_bits = 0;
                n_run = iter - 1;
                __syncthreads();
                break;
            }
            bool accepted = false, f_conv = false;
            for (int trial = 1; trial <= C.max_trials; ++trial) {
                ++n_trials;
                n_lsqr += F.lsqr(cost, lam, live_bits);
                // delta = x / colnorm, position step cap (:700-716), delta_scaled
                const double* xl = F.dp(F.L.xl);
                for (int a = tid; a < n_act; a += NT) {
                    double d[3];
                    for (int k = 0; k < p; ++k) d[k] = xl[a * p + k] / cn[a * p + k];
                    if (C.ky >= 0 || C.kx >= 0) {
                        const double dy = C.ky < 0 ? 0.0 : d[C.ky];
                        const double dx = C.kx < 0 ? 0.0 : d[C.kx];
                        const double len = sqrt(dy * dy + dx * dx);
                        if (len > C.max_step) {
                            const double scl = C.max_step / len;
                            if (C.ky >= 0) d[C.ky] *= scl;
                            if (C.kx >= 0) d[C.kx] *= scl;
                        }
                    }
                    for (int k = 0; k < p; ++k) {
                        delta[a * p + k] = d[k];
                        dsc[a * p + k] = cn[a * p + k] * d[k];
                    }
                }
                __syncthreads();
                F.coefs(true);
                const double cost_cand = F.render(false, live_bits, F.dp(F.L.u));
                f_conv = (cost_cand < cost) && ((cost - cost_cand) / cost <= C.f_tol);
                if (cost_cand < cost) {
                    accepted = true;
                    lam = fmax(lam / C.lambda_down, C.lambda_min);
                    // accepted step (:1245-1251) and per-star freeze tests (:1265-1283)
                    int nf = 0;
                    for (int a = tid; a < n_act; a += NT) {
                        for (int k = 0; k < p; ++k) {
                            const int i = a * p + k;
                            theta[i] = theta[i] + delta[i];
                            D[i] = fmax(D[i], cn[i]);
                        }
                        newf[a] = 0;
                        if (!live[a] || f_conv) continue;
                        double num = 0, xn = 0, gn = 0;
                        for (int k = 0; k < p; ++k) {
                            const int i = a * p + k;
                            const double v = (D[i] / cn[i]) * dsc[i];
                            num += v * v;
                            const double xv = D[i] * theta[i];
                            xn += xv * xv;
                            const double bt = cn[i] * bsc[i], Aii = cn[i] * cn[i];
                            gn = nan_max(gn, fabs(bt) / (sqrt(Aii * C_r) + kEpsG));
                        }
                        const bool xt = sqrt(num) <= C.x_tol * (sqrt(xn) + C.x_tol);
                        const bool gt = gn <= C.g_tol;
                        if (xt || gt) {
                            live[a] = 0;
                            newf[a] = 1;
                            frozen[a] = iter;
                            conv[a] = 1;
                            nf = 1;
                        }
                    }
                    cost = cost_cand;
                    moved = true;
                    const size_t t = F.L.wr;
                    F.L.wr = F.L.u;
                    F.L.u = t;
                    if (__syncthreads_or(nf)) {
                        froze = true;
                        MaskT nb = 0;
                        for (int a = 0; a < n_act; ++a)
                            if (newf[a]) nb |= (MaskT)1 << a;
                        live_bits &= ~nb;
                        F.render(true, nb, nullptr);  // _freeze_star! in Morton order
                    }
                    break;
                }
                lam = fmin(lam * C.lambda_up, C.lambda_max);
            }
            n_run = iter;
            if (f_conv) {
                for (int a = tid; a < n_act; a += NT)
                    if (live[a]) {
                        live[a] = 0;
                        frozen[a] = iter;
                        conv[a] = 1;
                    }
                live_bits = 0;
                __syncthreads();
                break;
            }
            if (accepted && live_bits == 0) break;
        }
        __syncthreads();
        // ---- errors at the final theta, every active star (:1302-1329)
        F.coefs(false);
        F.fill(true, s_gram);
        const StarCoef* cf = F.coef();
        double* err = F.dp(F.L.delta);  // reuse: per-star errors
        for (int a = tid; a < n_act; a += NT) {
            double A[9], inv[9];
            const double* gr = s_gram + a * 6;
            const double gfull[3][3] = {{gr[0], gr[1], gr[2]}, {gr[1], gr[3], gr[4]}, {gr[2], gr[4], gr[5]}};
            for (int k = 0; k < p; ++k)
                for (int l = 0; l < p; ++l) A[k + l * p] = gfull[k][l];
            double tr = 0;
            for (int k = 0; k < p; ++k) tr += A[k + k * p];
            for (int k = 0; k < p; ++k) A[k + k * p] += 1.0e-12 * tr;
            if (!chol_inv_small(A, p, inv)) pinv_small(A, p, inv);
            const double fsc = C.reweighted ? cost / dof : 1.0;
            for (int k = 0; k < p; ++k) err[a * p + k] = sqrt(fmax(0.0, inv[k + k * p] * fsc));
        }
        __syncthreads();
        // ---- outputs in catalogue order (:1289-1337, :1404-1430)
        for (int i = tid; i < ng; i += NT) {
            write_catalogue(i);
            fixed_fix(soff + i);
        }
        __syncthreads();
        for (int a = tid; a < n_act; a += NT) {
            const int64_t o = soff + act[a];
            for (int k = 0; k < p; ++k) {
                const double v = theta[a * p + k], e = err[a * p + k];
                if (C.gc[k] == 1) {
                    O.y[o] = v;
                    O.y_err[o] = e;
                } else if (C.gc[k] == 2) {
                    O.x[o] = v;
                    O.x_err[o] = e;
                } else {
                    O.flux[o] = v;
                    O.flux_err[o] = e;
                }
            }
            const StarCoef& c = cf[a];
            O.valid[o] = (isfinite(c.y) && isfinite(c.x) && isfinite(c.flux) && c.flux > 0) ? 1 : 0;
            O.converged[o] = conv[a];
            O.n_iter[o] = live[a] ? n_run : frozen[a];
        }
        // ---- final residual against the original data (:1344-1356), every active star
        if (O.residual) {
            for (int64_t q = tid; q < npix; q += NT) {
                int gy;
                const int gx = quot((int)q, ny, F.nymag, gy) + 1;
                ++gy;
                double acc = 0.0;
                for (int a = 0; a < n_act; ++a)
                    if (abs(gy - ay[a]) <= C.mR && abs(gx - ax[a]) <= C.mR) acc += F.mval(a, gy, gx);
                double d, w;
                F.G.data_w(q, d, w);
                O.residual[F.G.off + q] = d - acc;
            }
        }
        // ---- chisq and the qfit / crowding diagnostics (:1358-1397,
        // psf_photometry_diagnostics.jl:154-231), one warp per valid star; with
        // spread_model on, each box pixel's residual and weight also go to the
        // star's planes for k_group_spread
        for (int a = wid; a < n_act; a += NT / 32) {
            const StarCoef c = cf[a];
            const int64_t o = soff + act[a];
            if (!(isfinite(c.y) && isfinite(c.x) && isfinite(c.flux) && c.flux > 0)) continue;
            const int ylo = max((int)floor(c.y - C.fit_rad), 1), yhi = min((int)ceil(c.y + C.fit_rad), ny);
            const int xlo = max((int)floor(c.x - C.fit_rad), 1), xhi = min((int)ceil(c.x + C.fit_rad), nx);
            double num = 0, qv = 0, ncl = 0, ndi = 0, den = 0, ss = 0, ss2 = 0;
            int ng_ = 0, ngi = 0;
            const int h = yhi - ylo + 1, wd = xhi - xlo + 1;
            const double inv_flux = 1.0 / c.flux;
            double* rw = C.sp_on ? O.sp_rw + (size_t)o * 2 * C.sp_box : nullptr;
            NodeStar<false> T;  // the star's own weights: its box may have moved off the anchor's
            if (NODE) T.set(s_node, c.y, c.x, ylo, xlo, max(h, 0), max(wd, 0));
            const unsigned hmag = quot_magic((unsigned)max(h, 1));
            if (h > 0 && wd > 0)
                for (int e = lane; e < h * wd; e += 32) {
                    int er;
                    const int ec = quot(e, h, hmag, er);
                    const int gy = ylo + er, gx = xlo + ec;
                    const int64_t q = (gy - 1) + (int64_t)(gx - 1) * ny;
                    double acc = 0.0;
                    for (int b = 0; b < n_act; ++b)
                        if (abs(gy - ay[b]) <= C.mR && abs(gx - ax[b]) <= C.mR) acc += F.mval(b, gy, gx);
                    double d, wsan;
                    F.G.data_w(q, d, wsan);
                    const double r = d - acc;
                    const double wp = in.iv ? F.G.ld(in.iv, q) : 1.0;
                    if (rw) {
                        rw[e] = r;
                        rw[C.sp_box + e] = (isfinite(wp) && wp > 0) ? wp : 0.0;
                    }
                    if (isfinite(wp) && wp > 0) {
                        num += wp * (r * r);
                        ng_ += 1;
                        const double mv = NODE ? c.flux * T.value(s_node, s_node.pp, er, ec) + c.bkg
                                               : psf_value(P, c, gy, gx);
                        qv += fabs(r);
                        const double Pp = (mv - c.bkg) * inv_flux;
                        const double wP = wp * Pp;
                        ncl += wP * (r + mv - c.bkg);
                        const double im = F.G.ld(in.pix, q) - (in.bkg ? F.G.ld(in.bkg, q) : 0.0);
                        ndi += wP * (im - c.bkg);
                        den += wP * Pp;
                        if (in.iv) {
                            const double si = 1.0 / sqrt(wp);
                            ss += si;
                            ss2 += si * si;
                            ngi += 1;
                        }
                    }
                }
            num = warp_sum(num);
            qv = warp_sum(qv);
            ncl = warp_sum(ncl);
            ndi = warp_sum(ndi);
            den = warp_sum(den);
            ss = warp_sum(ss);
            ss2 = warp_sum(ss2);
            ng_ = warp_sum(ng_);
            ngi = warp_sum(ngi);
            if (lane == 0) {
                if (O.chisq) O.chisq[o] = (ng_ - p > 0) ? num / (double)(ng_ - p) : 0.0;
                if (O.qfit) O.qfit[o] = qv * inv_flux;
                if (O.crowding) O.crowding[o] = (den > 0 && ncl > 0 && ndi > 0) ? 2.5 * log10(ndi / ncl) : NaN;
                if (in.iv) {
                    if (O.qfit_expected) O.qfit_expected[o] = sqrt(2.0 / 3.141592653589793) * ss * inv_flux;
                    if (O.qfit_z) {
                        if (ss2 > 0 && ngi > p) {
                            const double dfac = sqrt(1.0 - (double)p / (double)ngi);
                            O.qfit_z[o] = (qv - sqrt(2.0 / 3.141592653589793) * dfac * ss) /
                                          (sqrt((1.0 - 2.0 / 3.141592653589793) * ss2) * dfac);
                        }
                    }
                }
            }
        }
        group_stats(n_run, ng - n_act, 0, 0, n_act, nU, n_trials, n_lsqr);
        __syncthreads();
    }
}

// spread_model of the kernel-fitted groups (_star_diagnostics!,
// psf_photometry_diagnostics.jl:200-231, with the disk of
// psf_photometry_simultaneous.jl:1361-1365), after k_groups: one block per group
// (grid-stride over the group list), one warp per valid star.  The block builds
// the group's disk into shared memory, its width from the first catalogue
// star's final parameters; each warp renders its star's model stamp over the
// fit box and correlates it with the disk one component at a time (x pass, then
// the y pass added into the correlated stamp; boxes up to kLine px in register
// lines, spread_lines_warp), all in its own stamp and two planes of shared
// memory, and sums against the residual and weight planes k_groups
// saved for the star.  Kept out of k_groups so that the fit's register
// allocation does not carry it.
__global__ void __launch_bounds__(128) k_group_spread(GroupConst C, DevPsf P, GroupIn in, GroupOut O,
                                                      const int32_t* __restrict__ glist, int nlist) {
    extern __shared__ __align__(16) double sm[];
    __shared__ double red[2 * 4 + 1];
    const double NaN = __longlong_as_double(0x7ff8000000000000LL);
    const int kh = C.R, box = C.sp_box, n = 2 * kh + 1;
    const int nw = blockDim.x >> 5, lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    double* tab = sm;
    double* pan = tab + ((C.sp_tab + 1) & ~1);
    const bool lines = spread_lines_fit(kh);
    const int ld = lines ? spread_plane(box, kh) : box;
    double* M = pan + (7 + kh) * kSpreadGL + (size_t)wid * (box + 2 * ld);  // the warp's model stamp
    double* T = M + box;                                                   // one component's x pass
    double* Gs = T + ld;                                                   // the disk-correlated stamp
    PPNode N;
    const bool one_node = node_of(P, N);
    DevPsf Ps = P;
    Ps.fwhm = C.sp_psf_fwhm;  // _spread_fwhm renders the PSF object's own width
    for (int li = blockIdx.x; li < nlist; li += gridDim.x) {
        const int g = glist[li];
        const int64_t soff = in.star_off[g];
        const int ng = (int)(in.star_off[g + 1] - soff);
        int any = 0;
        for (int i = threadIdx.x; i < ng; i += blockDim.x) any |= O.valid[soff + i];
        if (!__syncthreads_or(any)) continue;  // also: the previous group's disk is no longer read
        spread_disk_block(Ps, C.sp_param, kh, O.y[soff], O.x[soff], O.sp_rule, tab, red, pan);
        if (!spread_tab_on(tab)) continue;
        const SpreadDev D = spread_dev(tab, kh);
        const int ny = in.ny[g], nx = in.nx[g];
        for (int i = wid; i < ng; i += nw) {
            const int64_t o = soff + i;
            if (!O.valid[o]) continue;
            StarCoef c;
            c.y = O.y[o];
            c.x = O.x[o];
            c.flux = O.flux[o];
            c.bkg = C.fixed_bkg;
            grid_corners_dw(P, c.y, c.x, c);
            const int ylo = max((int)floor(c.y - C.fit_rad), 1), yhi = min((int)ceil(c.y + C.fit_rad), ny);
            const int xlo = max((int)floor(c.x - C.fit_rad), 1), xhi = min((int)ceil(c.x + C.fit_rad), nx);
            const int h = yhi - ylo + 1, wd = xhi - xlo + 1, nb = h * wd;
            if (h <= 0 || wd <= 0 || nb > box) continue;
            const double* Rr = O.sp_rw + (size_t)o * 2 * box;
            const double* Wt = Rr + box;
            __syncwarp();  // the warp's previous stamp is no longer read
            const unsigned hmag = quot_magic((unsigned)h);
            if (one_node) {
                NodeStar<false> S;
                S.set(N, c.y, c.x, ylo, xlo, h, wd);
                for (int e = lane; e < nb; e += 32) {
                    int r;
                    const int col = quot(e, h, hmag, r);
                    M[e] = c.flux * S.value(N, N.pp, r, col) + c.bkg;
                }
            } else {
                for (int e = lane; e < nb; e += 32) M[e] = psf_value(P, c, ylo + e % h, xlo + e / h);
            }
            if (lines) spread_lines_warp(D, D.I, M, T, Gs, h | 1, h, wd);
            for (int cc = 0; cc < 6 && !lines; ++cc) {
                const int L = D.L[cc];
                const double* I = D.I + cc * n + kh;
                __syncwarp();
                for (int e = lane; e < nb; e += 32) {  // x pass
                    const int r = e % h, col = e / h;
                    const int q0 = max(-L, -col), q1 = min(L, wd - 1 - col);
                    double t = 0.0;
                    for (int q = q0; q <= q1; ++q) t += I[q] * M[r + (col + q) * h];
                    T[e] = t;
                }
                __syncwarp();
                for (int e = lane; e < nb; e += 32) {  // y pass
                    const int r = e % h, col = e / h;
                    const int p0 = max(-L, -r), p1 = min(L, h - 1 - r);
                    double t = 0.0;
                    for (int p = p0; p <= p1; ++p) t += I[p] * T[r + p + col * h];
                    Gs[e] = (cc ? Gs[e] : 0.0) + D.alpha[cc] * t;
                }
            }
            __syncwarp();
            const int pad = lines ? (h | 1) - h : 0;  // of a Gs column
            const double inv_flux = 1.0 / c.flux;
            double Sp = 0, Sq = 0, Sp0 = 0, Sq0 = 0, SqG = 0;
            for (int e = lane; e < nb; e += 32) {
                const double wp = Wt[e];
                if (wp > 0) {
                    const double mv = M[e];
                    const double Pp = (mv - c.bkg) * inv_flux;
                    const double wP = wp * Pp;
                    const double p_i = Rr[e] + mv - c.bkg;
                    int r;
                    const double g_i = (Gs[e + pad * quot(e, h, hmag, r)] - c.bkg) * inv_flux;
                    Sp += wP * p_i;
                    Sq += wp * g_i * p_i;
                    Sp0 += wP * Pp;
                    Sq0 += wp * Pp * g_i;
                    SqG += wp * g_i * g_i;
                }
            }
            Sp = warp_sum(Sp);
            Sq = warp_sum(Sq);
            Sp0 = warp_sum(Sp0);
            Sq0 = warp_sum(Sq0);
            SqG = warp_sum(SqG);
            if (lane == 0 && Sp > 0) {
                if (O.spread) O.spread[o] = Sq / Sp - Sq0 / Sp0;
                if (O.spread_err)
                    O.spread_err[o] =
                        in.iv ? sqrt(fmax(0.0, Sp * Sp * SqG + Sq * Sq * Sp0 - 2 * Sq * Sp * Sq0)) / (Sp * Sp) : NaN;
            }
        }
    }
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
inline int next_pow2(int v) {
    int p = 1;
    while (p < v) p <<= 1;
    return p;
}

// Groups are launched in buckets of star count, each launch with a
// shared-memory layout sized for its largest group.  Measured on the B200 with
// the blended-group workload (2-12 stars), one launch over all groups (20,000
// groups: 56 ms) beats four launches by size class (65 ms): the class
// launches run one after another and each fills the GPU less.  So groups up to
// 32 stars share one bucket; larger ones (up to 64) get a second.
constexpr int kBucketEdges[] = {32, 64};
constexpr int kNumBuckets = sizeof(kBucketEdges) / sizeof(int);

// One launch over a bucket's groups or part of them.
struct Tier {
    int64_t first = 0, n = 0;  // its groups within the bucket's list
    size_t smem = 0;
    GroupConst C{};
};

struct Bucket {
    std::vector<int32_t> groups;  // most stars first
    int nmax = 1, umax = 1, keyn = 2;
    bool wide = false;
    Tier full, half;    // half.n > 0: two launches, half then full (plan_tiers)
    int threads = 256;  // default block size
};
constexpr int kQueueInts = 3;  // a bucket's counters: the two launches' queues, deferred groups


struct GroupPlan {
    std::vector<Bucket> buckets;  // non-empty buckets only
    std::vector<int32_t> routed_groups;
    int64_t n_kernel = 0;
};

// Everything a launch needs, derived once from the arguments.
struct GroupSetup {
    GroupConst C{};
    DevPsf dp{};
    GroupPlan plan;
    GroupIn gin{};
    GroupOut go{};
    std::vector<int64_t> h_off, h_soff;
    std::vector<int32_t> h_ny, h_nx;
    int64_t total_pixels = 0;
    int32_t eltype = CPB_F64;
    int sp_nw = 0;        // spread_model: warps a k_group_spread block (0: off)
    size_t sp_smem = 0;   // its dynamic shared memory
    int64_t n_stars = 0;  // catalogue length (sizes the residual / weight planes)
};

constexpr size_t kStaticSmem = 6 * 1024;  // the kernel's static shared arrays, rounded up

// Single-node image PSFs take the per-star weights (NODE).
inline bool group_node(const DevPsf& P) { return P.kind != CPB_PSF_CIRCULAR_GAUSSIAN && P.n_nodes == 1; }

// The size rule of a group that the kernel takes (others go to the full-field fit): two
// coefficient sets, 32-bit stamp indices and separate masks, within the block's shared
// memory less 8 KB.  The layout proper needs less at every size near that limit.
size_t group_rule_bytes(int nmax, int S2, int umax, int keyn) {
    const size_t n = (size_t)nmax, mask = nmax > 32 ? 8 : 4;
    return 2 * align16(sizeof(StarCoef) * n) + 9 * align16(24 * n) + 4 * align16(4 * n) + 3 * align16(n) +
           align16(std::max((size_t)24 * n * S2, (size_t)4 * keyn)) + align16(4 * n * S2) +
           4 * align16((size_t)8 * umax) + align16((size_t)4 * umax) + 2 * align16(mask * umax);
}

size_t layout_bytes(const GroupConst& C, int nmax, int umax, int keyn, bool node) {
    return nmax > 32 ? make_layout<uint64_t>(nmax, C.S2, umax, keyn, node, C.same).total
                     : make_layout<uint32_t>(nmax, C.S2, umax, keyn, node, C.same).total;
}

// The bucket's launches.  One block of the layout for the largest group an SM leaves its
// schedulers 80 % idle (4,000 groups of 2-12 stars, 152 KB: 12.3 ms, 20 % of issue slots).
// With data_work and sqrt(w) in global memory (read in order, once a render) two blocks of
// 12-star groups of 13 px boxes fit; with both in shared memory 40 % of those groups were
// deferred and the batch took 9.6 ms instead of 7.2.
// The union of a blend's boxes is usually well below the bound its layout allows for, so
// where two such blocks do not fit an SM, the groups of up to `nA` stars run first with a
// layout of half an SM: its union capacity is what is left beside the stars' arrays, at
// least half the bound.  A group whose union is larger appends itself to a list, and a
// second launch with the full layout takes those and the groups of more stars.
void plan_tiers(Bucket& B, const GroupConst& C, bool node, size_t smem_sm, const std::vector<int64_t>& soff,
                const std::vector<int32_t>& ny, const std::vector<int32_t>& nx) {
    auto stars = [&](int32_t g) { return (int)(soff[g + 1] - soff[g]); };
    std::stable_sort(B.groups.begin(), B.groups.end(), [&](int32_t a, int32_t b) { return stars(a) > stars(b); });
    auto tier = [&](Tier& t, int nmax, int umax, int keyn) {
        t.C = C;
        t.C.nmax = nmax;
        t.C.umax = umax;
        t.C.keyn = keyn;
        t.smem = layout_bytes(C, nmax, umax, keyn, node);
    };
    tier(B.full, B.nmax, B.umax, B.keyn);
    B.full.first = 0;
    B.full.n = (int64_t)B.groups.size();
    B.half.n = 0;
    const size_t half = smem_sm / 2 - 1024 - kStaticSmem;
    if (B.full.smem <= half || B.wide) return;
    for (size_t i = 0; i < B.groups.size(); ++i) {  // B.groups[i ..) in the half launch
        const int nA = stars(B.groups[i]);
        if (i && nA == stars(B.groups[i - 1])) continue;
        int um = 1;
        for (size_t k = i; k < B.groups.size(); ++k)
            um = std::max(um, (int)std::min<int64_t>((int64_t)stars(B.groups[k]) * C.S2,
                                                     (int64_t)ny[B.groups[k]] * nx[B.groups[k]]));
        const int keyn = next_pow2(std::max(nA * C.S2, 2));
        auto fits = [&](int u) { return layout_bytes(C, std::max(nA, 1), u, keyn, node) <= half; };
        if (!fits((um + 1) / 2)) continue;
        int lo = (um + 1) / 2, hi = um;  // the largest capacity that fits
        while (lo < hi) {
            const int mid = (lo + hi + 1) / 2;
            if (fits(mid)) lo = mid;
            else hi = mid - 1;
        }
        tier(B.half, std::max(nA, 1), lo, keyn);
        B.half.first = (int64_t)i;
        B.half.n = (int64_t)(B.groups.size() - i);
        B.full.n = (int64_t)i;
        return;
    }
}

// Argument checks (the reference's, :984-1051), constants, group metadata on
// the host and the shared-memory plan: which groups one block can hold.
void setup_groups(cpb_ctx* ctx, const cpb_psf* psf, const cpb_sim_params* P, int64_t G, const int64_t* d_off,
                  const int32_t* d_ny, const int32_t* d_nx, const void* d_pix, int32_t eltype, const void* d_iv,
                  const void* d_bkg, const int64_t* d_soff, const double* d_y0, const double* d_x0,
                  const double* d_f0, int64_t total_pixels, const cpb_group_result* out, const int64_t* h_off_opt,
                  const int32_t* h_ny_opt, const int32_t* h_nx_opt, const int64_t* h_soff_opt, GroupSetup& su) {
    cudaStream_t st = ctx->stream;
    // argument checks in the reference's order (:984-997), shared by every group
    if (!(P->max_iter > 0)) throw ArgError{"max_iter must be positive"};
    if (!(P->inner_iterations > 0)) throw ArgError{"inner_iterations must be positive"};
    if (!(P->linear_tol > 0)) throw ArgError{"linear_tol must be positive"};
    if (!(P->max_trials > 0)) throw ArgError{"max_trials must be positive"};
    if (!P->model_rad_auto && !(P->model_rad > 0)) throw ArgError{"model_rad must be :auto or a positive real"};
    const double model_rad_max = P->model_rad_max < 0 ? 10 * P->fit_rad : P->model_rad_max;
    if (!(model_rad_max >= P->fit_rad)) throw ArgError{"model_rad_max must be >= fit_rad"};
    if (!(P->model_rad_nsigma > 0)) throw ArgError{"model_rad_nsigma must be positive"};
    if (P->solver != CPB_SOLVER_LSQR && P->solver != CPB_SOLVER_LSMR) throw ArgError{"solver must be :lsqr or :lsmr"};
    if (P->damping == CPB_DAMP_LEVENBERG)
        throw ArgError{
            "LevenbergDamping is not supported by fit_all_stars_simultaneous: it conflicts with the "
            "column-equilibrated x_tol scaling. Use MarquardtDamping."};
    if (!(P->fit_rad > 0)) throw ArgError{"fit_rad must be positive"};
    if (eltype != CPB_F32 && eltype != CPB_F64) throw ArgError{"unsupported image eltype"};
    if (P->model_rad_auto && !d_iv)
        throw ArgError{
            "model_rad=:auto requires inv_var (it needs a noise scale); pass inv_var or an explicit scalar model_rad"};
    if (G < 0) throw ArgError{"n_groups must be >= 0"};
    if (!out->y || !out->x || !out->flux || !out->y_err || !out->x_err || !out->flux_err || !out->converged ||
        !out->valid || !out->n_iter || !out->n_passes || !out->n_failed || !out->status)
        throw ArgError{"null output array"};
    GroupConst& C = su.C;
    C.p = 0;
    if (P->free_mask & CPB_FREE_Y) C.gc[C.p++] = 1;
    if (P->free_mask & CPB_FREE_X) C.gc[C.p++] = 2;
    if (P->free_mask & CPB_FREE_FLUX) C.gc[C.p++] = 3;
    if (P->free_mask & ~(CPB_FREE_Y | CPB_FREE_X | CPB_FREE_FLUX))
        throw ArgError{
            "fit_all_stars_simultaneous fits only (y, x, flux) per star. Fix `bkg` (subtract the background first "
            "and pass `fixed = (; bkg = zero(eltype(image)))`), and fix all shape parameters."};
    if (C.p == 0) throw ArgError{"all model parameters are fixed; nothing to fit"};
    C.ky = C.kx = -1;
    for (int k = 0; k < C.p; ++k) {
        if (C.gc[k] == 1) C.ky = k;
        if (C.gc[k] == 2) C.kx = k;
    }
    for (int k = C.p; k < 3; ++k) C.gc[k] = 3;
    C.fixed_y = P->fixed_y;
    C.fixed_x = P->fixed_x;
    C.fixed_flux = P->fixed_flux;
    C.fixed_bkg = P->fixed_bkg;
    C.R = (int)std::ceil(P->fit_rad);
    C.S = 2 * C.R + 1;
    C.S2 = C.S * C.S;
    {
        const int R_cap = (int)std::ceil(std::max(P->model_rad, P->fit_rad));
        C.mR = std::min(std::max((int)std::ceil(P->model_rad), C.R), R_cap);
    }
    C.max_iter = P->max_iter;
    C.max_trials = P->max_trials;
    C.itmax = P->inner_iterations;
    C.linear_tol = P->linear_tol;
    C.max_step = P->max_step;
    C.x_tol = P->x_tol;
    C.f_tol = P->f_tol;
    C.g_tol = P->g_tol;
    C.lambda_init = P->lambda_init;
    C.lambda_up = P->lambda_up;
    C.lambda_down = P->lambda_down;
    C.lambda_min = P->lambda_min;
    C.lambda_max = P->lambda_max;
    C.same = C.mR == C.R;
    C.Smag = quot_magic((unsigned)C.S);
    C.eltype = eltype;
    C.reweighted = (P->covariance == CPB_COV_REWEIGHTED || (P->covariance == CPB_COV_AUTO && d_iv == nullptr)) ? 1 : 0;
    C.fit_rad = P->fit_rad;
    {
        const double spp = P->spread_model_fwhm;
        C.sp_on = (out->spread_model || out->spread_model_err) && (std::isnan(spp) || (std::isfinite(spp) && spp > 0));
        C.sp_tab = spread_tab_len(C.R);
        C.sp_box = (2 * C.R + 2) * (2 * C.R + 2);
        C.sp_param = spp;
        C.sp_psf_fwhm = psf->dev.fwhm;
    }
    su.dp = psf->dev;
    su.dp.fwhm = P->fixed_fwhm;

    su.total_pixels = total_pixels;
    su.eltype = eltype;
    su.gin = GroupIn{d_off, d_ny, d_nx, d_pix, d_iv, d_bkg, d_soff, d_y0, d_x0, d_f0};
    su.go = GroupOut{out->y, out->x, out->flux, out->y_err, out->x_err, out->flux_err, out->converged, out->valid,
                     out->n_iter, out->chisq, out->qfit, out->qfit_expected, out->qfit_z, out->crowding,
                     out->residual, out->n_passes, out->n_failed, out->status, out->error_kind, out->n_active,
                     out->n_union, out->n_trials, out->n_lsqr_iters, out->spread_model, out->spread_model_err,
                     nullptr, nullptr, nullptr};
    if (G == 0) return;
    // group sizes on the host (plan the shared-memory layout, route oversized groups)
    std::vector<int64_t>& h_off = su.h_off;
    std::vector<int64_t>& h_soff = su.h_soff;
    std::vector<int32_t>& h_ny = su.h_ny;
    std::vector<int32_t>& h_nx = su.h_nx;
    h_off.resize(G);
    h_soff.resize(G + 1);
    h_ny.resize(G);
    h_nx.resize(G);
    if (h_off_opt) {
        std::memcpy(h_off.data(), h_off_opt, sizeof(int64_t) * G);
        std::memcpy(h_soff.data(), h_soff_opt, sizeof(int64_t) * (G + 1));
        std::memcpy(h_ny.data(), h_ny_opt, sizeof(int32_t) * G);
        std::memcpy(h_nx.data(), h_nx_opt, sizeof(int32_t) * G);
    } else {
        check(cudaMemcpyAsync(h_off.data(), d_off, sizeof(int64_t) * G, cudaMemcpyDeviceToHost, st), "d2h");
        check(cudaMemcpyAsync(h_soff.data(), d_soff, sizeof(int64_t) * (G + 1), cudaMemcpyDeviceToHost, st), "d2h");
        check(cudaMemcpyAsync(h_ny.data(), d_ny, sizeof(int32_t) * G, cudaMemcpyDeviceToHost, st), "d2h");
        check(cudaMemcpyAsync(h_nx.data(), d_nx, sizeof(int32_t) * G, cudaMemcpyDeviceToHost, st), "d2h");
        check(cudaStreamSynchronize(st), "sync");
    }
    for (int64_t g = 0; g < G; ++g) {
        if (h_ny[g] <= 0 || h_nx[g] <= 0 || (int64_t)h_ny[g] * h_nx[g] >= (1LL << 31))
            throw ArgError{"group image size out of range"};
        if (h_soff[g + 1] < h_soff[g]) throw ArgError{"star_offsets must be non-decreasing"};
        if (out->residual && h_off[g] + (int64_t)h_ny[g] * h_nx[g] > total_pixels)
            throw ArgError{"total_pixels is smaller than the pixels the groups span"};
    }
    int smem_optin = 0, smem_sm = 0;
    check(cudaDeviceGetAttribute(&smem_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, ctx->device), "attr");
    check(cudaDeviceGetAttribute(&smem_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, ctx->device), "attr");
    const size_t cap = (size_t)smem_optin - 8 * 1024;  // of the size rule
    su.n_stars = h_soff[G];
    if (C.sp_on) {
        // k_group_spread: the disk table and one panel of the quadrature, then
        // the stamp and two planes a warp (3 sp_box doubles or a little more); up to 4 warps within 96 KB, else fewer; a fit
        // box beyond shared memory even for one warp leaves spread_model NaN
        const size_t fixed = ((size_t)((C.sp_tab + 1) & ~1) + (size_t)(7 + C.R) * kSpreadGL) * sizeof(double);
        const size_t per_warp =
            (C.sp_box + 2 * (size_t)(spread_lines_fit(C.R) ? spread_plane(C.sp_box, C.R) : C.sp_box)) * sizeof(double);
        int nw = 4;
        while (nw > 1 && fixed + nw * per_warp > 96 * 1024) --nw;
        if (fixed + nw * per_warp > cap) C.sp_on = 0;
        su.sp_nw = C.sp_on ? nw : 0;
        su.sp_smem = fixed + nw * per_warp;
    }
    GroupPlan& plan = su.plan;
    const bool node = group_node(su.dp);
    auto need_of = [&](int ng, int um, int kn) {
        return group_rule_bytes(std::max(ng, 1), C.S2, std::max(um, 1), kn);
    };
    // a group runs in the kernel when it has <= 64 stars and its own layout fits;
    // the kernel computes in FP64 with LSQR and one scalar model radius, so
    // solver = :lsmr, model_rad = :auto or the mixed form route every group to
    // the full-field fit
    const bool route_all = P->solver == CPB_SOLVER_LSMR || P->model_rad_auto || P->precision != CPB_PREC_FP64;
    std::vector<Bucket> bk(kNumBuckets);
    for (int64_t g = 0; g < G; ++g) {
        const int ng = (int)(h_soff[g + 1] - h_soff[g]);
        const int um = (int)std::min<int64_t>((int64_t)ng * C.S2, (int64_t)h_ny[g] * h_nx[g]);
        const int kn = next_pow2(std::max(ng * C.S2, 2));
        if (route_all || ng > kMaxGroupStars || need_of(ng, um, kn) > cap) {
            plan.routed_groups.push_back((int32_t)g);
            continue;
        }
        int b = 0;
        while (kBucketEdges[b] < ng) ++b;
        Bucket& B = bk[b];
        // the bucket's layout must still fit with this group's sizes folded in
        const int nm2 = std::max(B.nmax, ng), um2 = std::max(B.umax, um), kn2 = std::max(B.keyn, kn);
        if (need_of(nm2, um2, kn2) > cap) {
            plan.routed_groups.push_back((int32_t)g);
            continue;
        }
        B.groups.push_back((int32_t)g);
        B.nmax = nm2;
        B.umax = um2;
        B.keyn = kn2;
    }
    std::sort(plan.routed_groups.begin(), plan.routed_groups.end());
    for (Bucket& B : bk) {
        if (B.groups.empty()) continue;
        B.wide = B.nmax > 32;
        if (layout_bytes(C, B.nmax, B.umax, B.keyn, node) > (size_t)smem_optin - kStaticSmem)
            throw CudaError{cudaErrorInvalidConfiguration, "group layout"};  // the size rule excludes it
        plan_tiers(B, C, node, (size_t)smem_sm, h_soff, h_ny, h_nx);
        // default block size: about 512 threads an SM (the kernel's register budget
        // allows 512 threads of 128 registers), in as many blocks as shared memory holds
        const int by_smem = std::max(1, (int)((size_t)smem_sm / ((B.half.n ? B.half.smem : B.full.smem) + kStaticSmem + 1024)));
        const int blocks = std::min(by_smem, 8);
        B.threads = blocks >= 8 ? 64 : (blocks >= 4 ? 128 : 256);
        plan.n_kernel += (int64_t)B.groups.size();
        plan.buckets.push_back(std::move(B));
    }
}

using GroupKernel = void (*)(GroupConst, DevPsf, GroupIn, GroupOut, const int32_t*, int, int*, const int32_t*,
                             const int*, int32_t*, int*);
template <int NT>
GroupKernel group_kernel(bool wide, bool node) {
    return wide ? (node ? k_groups<NT, uint64_t, true> : k_groups<NT, uint64_t, false>)
                : (node ? k_groups<NT, uint32_t, true> : k_groups<NT, uint32_t, false>);
}

GroupKernel group_kernel_for(int threads, bool wide, bool node) {
    return threads == 64 ? group_kernel<64>(wide, node)
                         : (threads == 128 ? group_kernel<128>(wide, node) : group_kernel<256>(wide, node));
}

inline int valid_threads(int t) { return t == 64 ? 64 : (t == 128 ? 128 : 256); }

// Resident blocks per SM of the group kernel with a launch's layout and this block size.
int tier_occupancy(const Bucket& B, const Tier& T, int threads, bool node) {
    GroupKernel kfn = group_kernel_for(threads, B.wide, node);
    allow_smem(kfn, T.smem);
    int per_sm = 0;
    check(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kfn, threads, T.smem), "occupancy");
    return std::max(per_sm, 1);
}
// Doubles of the blocks' union arrays (GroupOut::px) for any block size of any launch.
size_t group_px_doubles(const cpb_ctx* ctx, const GroupSetup& su) {
    size_t most = 0;
    const bool node = group_node(su.dp);
    for (const Bucket& B : su.plan.buckets)
        for (const Tier* T : {&B.half, &B.full})
            for (int t = 64; t <= 256; t *= 2)
                if (T->C.umax) {
                    const int64_t grid = std::min<int64_t>((int64_t)B.groups.size(),
                                                           (int64_t)ctx->n_sm * tier_occupancy(B, *T, t, node));
                    most = std::max(most, (size_t)2 * T->C.umax * (size_t)grid);
                }
    return most;
}
int group_occupancy(const Bucket& B, int threads, bool node) {
    return tier_occupancy(B, B.half.n ? B.half : B.full, valid_threads(threads), node);
}

// The group kernel over one bucket's groups: resets its counters and starts, for each of
// its launches, min(groups, SMs x blocks_per_sm) persistent blocks.  threads: 64, 128 or
// 256 (<= 0: the bucket's default); blocks_per_sm <= 0 means the occupancy limit.  d_ovf:
// room for the half launch's deferred groups; d_queue: kQueueInts counters.
void launch_bucket(cpb_ctx* ctx, cudaStream_t st, const GroupSetup& su, const Bucket& B, const int32_t* d_list,
                   int32_t* d_ovf, int* d_queue, int threads, int blocks_per_sm) {
    const int64_t nk = (int64_t)B.groups.size();
    if (nk <= 0) return;
    threads = valid_threads(threads <= 0 ? B.threads : threads);
    const bool node = group_node(su.dp);
    GroupKernel kern = group_kernel_for(threads, B.wide, node);
    check(cudaMemsetAsync(d_queue, 0, sizeof(int) * kQueueInts, st), "memset");
    auto go = [&](const Tier& T, bool half) {
        KernelScope ks_(ctx, "k_groups",
                        (double)su.total_pixels * (su.eltype == CPB_F64 ? 8 : 4) * (su.gin.iv ? 2 : 1) * T.n /
                            std::max<int64_t>(su.plan.n_kernel, 1));
        const int occ = tier_occupancy(B, T, threads, node);
        const int per_sm = blocks_per_sm <= 0 ? occ : std::min(blocks_per_sm, occ);
        const int64_t grid = std::min<int64_t>(half ? T.n : nk, (int64_t)ctx->n_sm * per_sm);
        const bool rest = !half && B.half.n;  // takes the half launch's deferred groups
        kern<<<(unsigned)grid, threads, T.smem, st>>>(T.C, su.dp, su.gin, su.go, d_list + T.first, (int)T.n,
                                                      d_queue + (half ? 0 : 1), rest ? d_ovf : nullptr, d_queue + 2,
                                                      half ? d_ovf : nullptr, d_queue + 2);
        check(cudaGetLastError(), "k_groups");
    };
    if (B.half.n) go(B.half, true);
    go(B.full, false);
}

// k_group_spread over the kernel-fitted groups (after their bucket launches).
void launch_spread(cpb_ctx* ctx, cudaStream_t st, const GroupSetup& su, const int32_t* d_list, int64_t nk) {
    if (!su.C.sp_on || nk <= 0) return;
    const int threads = 32 * su.sp_nw;
    allow_smem(k_group_spread, su.sp_smem);
    int per_sm = 0;
    check(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_group_spread, threads, su.sp_smem), "occupancy");
    const int64_t grid = std::min<int64_t>(nk, (int64_t)ctx->n_sm * std::max(per_sm, 1));
    KernelScope ks_(ctx, "k_group_spread", 0.0);
    k_group_spread<<<(unsigned)grid, threads, su.sp_smem, st>>>(su.C, su.dp, su.gin, su.go, d_list, (int)nk);
    check(cudaGetLastError(), "k_group_spread");
}

}  // namespace

int fit_groups_dev(cpb_ctx* ctx, const cpb_psf* psf, const cpb_sim_params* P, int64_t G, const int64_t* d_off,
                   const int32_t* d_ny, const int32_t* d_nx, const void* d_pix, int32_t eltype, const void* d_iv,
                   const void* d_bkg, const int64_t* d_soff, const double* d_y0, const double* d_x0,
                   const double* d_f0, int64_t total_pixels, cpb_group_result* out, const int64_t* h_off_opt,
                   const int32_t* h_ny_opt, const int32_t* h_nx_opt, const int64_t* h_soff_opt) {
    NvtxRange nv_("cpb:group_batch");
    cudaStream_t st = ctx->stream;
    GroupSetup su;
    setup_groups(ctx, psf, P, G, d_off, d_ny, d_nx, d_pix, eltype, d_iv, d_bkg, d_soff, d_y0, d_x0, d_f0,
                 total_pixels, out, h_off_opt, h_ny_opt, h_nx_opt, h_soff_opt, su);
    out->n_kernel_groups = 0;
    out->n_routed_groups = 0;
    out->device_seconds = 0;
    if (G == 0) return 0;
    const GroupPlan& plan = su.plan;
    const std::vector<int64_t>& h_off = su.h_off;
    const std::vector<int64_t>& h_soff = su.h_soff;
    const std::vector<int32_t>& h_ny = su.h_ny;
    const std::vector<int32_t>& h_nx = su.h_nx;
    check(cudaEventRecord(ctx->ev0, st), "event");
    const int64_t nk = plan.n_kernel;
    if (nk > 0) {
        // every bucket's group list back to back, one queue counter per bucket
        std::vector<int32_t> lists;
        for (const Bucket& B : plan.buckets) lists.insert(lists.end(), B.groups.begin(), B.groups.end());
        if (su.C.sp_on) {
            double h_rule[kSpreadRuleLen];
            spread_rule(h_rule);
            auto* d_rule = (double*)scratch(ctx, "grp_sp_rule", sizeof(h_rule));
            check(cudaMemcpyAsync(d_rule, h_rule, sizeof(h_rule), cudaMemcpyHostToDevice, st), "h2d");
            su.go.sp_rule = d_rule;
            su.go.sp_rw = (double*)scratch(ctx, "grp_sp_rw", sizeof(double) * 2 * su.C.sp_box * su.n_stars);
        }
        su.go.px = (double*)scratch(ctx, "grp_px", sizeof(double) * group_px_doubles(ctx, su));
        int32_t* d_list = (int32_t*)scratch(ctx, "grp_list", sizeof(int32_t) * 2 * nk);  // and the deferred groups
        int* d_queue = (int*)scratch(ctx, "grp_queue", sizeof(int) * kQueueInts * plan.buckets.size());
        check(cudaMemcpyAsync(d_list, lists.data(), sizeof(int32_t) * nk, cudaMemcpyHostToDevice, st), "h2d");
        int64_t at = 0;
        for (size_t b = 0; b < plan.buckets.size(); ++b) {
            launch_bucket(ctx, st, su, plan.buckets[b], d_list + at, d_list + nk + at, d_queue + kQueueInts * b, 0, 0);
            at += (int64_t)plan.buckets[b].groups.size();
        }
        launch_spread(ctx, st, su, d_list, nk);
    }
    check(cudaEventRecord(ctx->ev1, st), "event");
    check(cudaStreamSynchronize(st), "sync");
    float ms = 0;
    cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1);
    out->device_seconds = ms * 1e-3;
    out->n_kernel_groups = nk;
    out->n_routed_groups = (int64_t)plan.routed_groups.size();
    // groups too large for one block: the full-field path, one at a time
    for (int32_t g : plan.routed_groups) {
        const int64_t s0 = h_soff[g], ng = h_soff[g + 1] - h_soff[g];
        const int ny = h_ny[g], nx = h_nx[g];
        const size_t esz = eltype == CPB_F64 ? 8 : 4;
        const int64_t off = h_off[g];
        std::vector<double> y(ng), x(ng), f(ng), b(ng), ey(ng), ex(ng), ef(ng), eb(ng), chi(ng), q1(ng), q2(ng),
            q3(ng), cr(ng), sm(ng), sme(ng);
        std::vector<uint8_t> cv(ng), va(ng);
        std::vector<int32_t> it(ng);
        std::vector<double> res(out->residual ? (size_t)ny * nx : 0);
        cpb_sim_result r{};
        r.y = y.data();
        r.x = x.data();
        r.flux = f.data();
        r.bkg = b.data();
        r.y_err = ey.data();
        r.x_err = ex.data();
        r.flux_err = ef.data();
        r.bkg_err = eb.data();
        r.converged = cv.data();
        r.valid = va.data();
        r.chisq = chi.data();
        r.qfit = q1.data();
        r.qfit_expected = q2.data();
        r.qfit_z = q3.data();
        r.crowding = cr.data();
        r.spread_model = sm.data();
        r.spread_model_err = sme.data();
        r.n_iter = it.data();
        r.residual = out->residual ? res.data() : nullptr;
        int32_t status = 0, kind = 0;
        try {
            fit_simultaneous_dev(ctx, psf, P, (const char*)d_pix + esz * off, eltype, ny, nx,
                                 d_iv ? (const char*)d_iv + esz * off : nullptr,
                                 d_bkg ? (const char*)d_bkg + esz * off : nullptr, ng, d_y0 + s0, d_x0 + s0,
                                 d_f0 + s0, &r);
        } catch (const ArgError& e) {
            status = CPB_ERR_ARGUMENT;
            kind = e.msg.find("non-finite") != std::string::npos ? 1 : 2;
            std::vector<double> hy(ng), hx(ng), hf(ng);
            if (ng > 0) {
                // on the context's stream (non-blocking: a legacy-stream copy would not
                // wait for the catalogue's upload)
                check(cudaMemcpyAsync(hy.data(), d_y0 + s0, 8 * ng, cudaMemcpyDeviceToHost, ctx->stream), "d2h");
                check(cudaMemcpyAsync(hx.data(), d_x0 + s0, 8 * ng, cudaMemcpyDeviceToHost, ctx->stream), "d2h");
                check(cudaMemcpyAsync(hf.data(), d_f0 + s0, 8 * ng, cudaMemcpyDeviceToHost, ctx->stream), "d2h");
                check(cudaStreamSynchronize(ctx->stream), "d2h");
            }
            const double NaN = std::numeric_limits<double>::quiet_NaN();
            for (int64_t i = 0; i < ng; ++i) {
                y[i] = (P->free_mask & CPB_FREE_Y) ? hy[i] : P->fixed_y;
                x[i] = (P->free_mask & CPB_FREE_X) ? hx[i] : P->fixed_x;
                f[i] = (P->free_mask & CPB_FREE_FLUX) ? hf[i] : P->fixed_flux;
                ey[i] = (P->free_mask & CPB_FREE_Y) ? NaN : 0.0;
                ex[i] = (P->free_mask & CPB_FREE_X) ? NaN : 0.0;
                ef[i] = (P->free_mask & CPB_FREE_FLUX) ? NaN : 0.0;
                cv[i] = 0;
                va[i] = 0;
                it[i] = 0;
                chi[i] = 0.0;
                q1[i] = q2[i] = q3[i] = cr[i] = sm[i] = sme[i] = NaN;
            }
            std::fill(res.begin(), res.end(), 0.0);
            r.n_passes = 0;
            r.n_failed = (int32_t)ng;
            r.n_active = 0;
            r.n_union = 0;
            r.n_trials = 0;
            r.n_lsqr_iters = 0;
        }
        auto up = [&](void* dst, const void* src, size_t bytes) {
            if (dst && bytes) check(cudaMemcpy(dst, src, bytes, cudaMemcpyHostToDevice), "h2d routed group");
        };
        up(out->y + s0, y.data(), 8 * ng);
        up(out->x + s0, x.data(), 8 * ng);
        up(out->flux + s0, f.data(), 8 * ng);
        up(out->y_err + s0, ey.data(), 8 * ng);
        up(out->x_err + s0, ex.data(), 8 * ng);
        up(out->flux_err + s0, ef.data(), 8 * ng);
        up(out->converged + s0, cv.data(), ng);
        up(out->valid + s0, va.data(), ng);
        up(out->n_iter + s0, it.data(), 4 * ng);
        if (out->chisq) up(out->chisq + s0, chi.data(), 8 * ng);
        if (out->qfit) up(out->qfit + s0, q1.data(), 8 * ng);
        if (out->qfit_expected) up(out->qfit_expected + s0, q2.data(), 8 * ng);
        if (out->qfit_z) up(out->qfit_z + s0, q3.data(), 8 * ng);
        if (out->crowding) up(out->crowding + s0, cr.data(), 8 * ng);
        if (out->spread_model) up(out->spread_model + s0, sm.data(), 8 * ng);
        if (out->spread_model_err) up(out->spread_model_err + s0, sme.data(), 8 * ng);
        if (out->residual) up(out->residual + off, res.data(), 8 * res.size());
        const int32_t na = (int32_t)r.n_active, nu = (int32_t)r.n_union, ntr = (int32_t)r.n_trials,
                      nls = (int32_t)r.n_lsqr_iters;
        up(out->n_passes + g, &r.n_passes, 4);
        up(out->n_failed + g, &r.n_failed, 4);
        up(out->status + g, &status, 4);
        if (out->error_kind) up(out->error_kind + g, &kind, 4);
        if (out->n_active) up(out->n_active + g, &na, 4);
        if (out->n_union) up(out->n_union + g, &nu, 4);
        if (out->n_trials) up(out->n_trials + g, &ntr, 4);
        if (out->n_lsqr_iters) up(out->n_lsqr_iters + g, &nls, 4);
        out->device_seconds += r.device_seconds;
    }
    return 0;
}


// ---------------------------------------------------------------------------
// A bound batch over fixed device buffers (CUDA-graph capture and tuning)
// ---------------------------------------------------------------------------
struct GroupBatch {
    GroupSetup su;
    void* block = nullptr;      // owned, from the device's pool: spread_model rule, the lists, the stars'
                                // residual / weight planes, the blocks' union arrays (GroupOut::px) and
                                // the counters
    int32_t* d_list = nullptr;  // every bucket's groups back to back, then as much for deferred ones
    int* d_queue = nullptr;     // kQueueInts counters per bucket
    std::vector<int64_t> at;    // first list entry of each bucket
    std::vector<int> threads;   // chosen block size per bucket
};

GroupBatch* group_batch_create(cpb_ctx* ctx, const cpb_psf* psf, const cpb_sim_params* P, int64_t G,
                               const int64_t* d_off, const int32_t* d_ny, const int32_t* d_nx, const void* d_pix,
                               int32_t eltype, const void* d_iv, const void* d_bkg, const int64_t* d_soff,
                               const double* d_y0, const double* d_x0, const double* d_f0, int64_t total_pixels,
                               const cpb_group_result* out) {
    if (G > 0 && (!d_off || !d_ny || !d_nx || !d_pix || !d_soff || !d_y0 || !d_x0 || !d_f0 || !out))
        throw ArgError{"null argument"};
    auto* b = new GroupBatch();
    try {
        if (G > 0)
            setup_groups(ctx, psf, P, G, d_off, d_ny, d_nx, d_pix, eltype, d_iv, d_bkg, d_soff, d_y0, d_x0, d_f0,
                         total_pixels, out, nullptr, nullptr, nullptr, nullptr, b->su);
        const GroupPlan& plan = b->su.plan;
        if (!plan.routed_groups.empty() &&
            (P->solver == CPB_SOLVER_LSMR || P->model_rad_auto || P->precision != CPB_PREC_FP64))
            throw ArgError{"groups with solver :lsmr, model_rad = :auto or mixed precision are fitted one by one "
                           "by the full-field fit; use cpb_fit_simultaneous_batch instead of a captured batch"};
        if (!plan.routed_groups.empty())
            throw ArgError{"group " + std::to_string(plan.routed_groups[0]) +
                           " is too large for one thread block (more than 64 stars, or a working set beyond shared "
                           "memory); fit it with cpb_fit_simultaneous_batch instead of a captured batch"};
        std::vector<int32_t> lists;
        for (const Bucket& B : plan.buckets) {
            b->at.push_back((int64_t)lists.size());
            b->threads.push_back(B.threads);
            lists.insert(lists.end(), B.groups.begin(), B.groups.end());
        }
        // One block from the pool, whose first chunk a scratch buffer keeps, and one copy: three or
        // four cudaMalloc, and the memory the driver maps for each above 1 MB, took a tenth of
        // binding a small batch (milliseconds on some hosts).
        scratch(ctx, "grp_keep", 256);
        GroupSetup& su = b->su;
        const bool sp = su.C.sp_on && !plan.buckets.empty();
        size_t bytes = 0;
        auto place = [&](size_t n) {
            const size_t at = bytes;
            bytes = (at + n + 255) & ~size_t(255);
            return at;
        };
        const size_t o_rule = place(sp ? sizeof(double) * kSpreadRuleLen : 0);
        const size_t o_list = place(sizeof(int32_t) * 2 * lists.size());
        const size_t o_rw = place(sp ? sizeof(double) * 2 * su.C.sp_box * su.n_stars : 0);
        const size_t o_queue = place(sizeof(int) * kQueueInts * plan.buckets.size());
        const size_t o_px = place(plan.buckets.empty() ? 0 : sizeof(double) * group_px_doubles(ctx, su));
        if (cudaMallocAsync(&b->block, std::max<size_t>(bytes, 256), ctx->stream) != cudaSuccess) {
            cudaGetLastError();
            throw OomError{"device memory exhausted allocating the groups' work queues, pixel arrays and "
                           "spread_model planes"};
        }
        char* base = (char*)b->block;
        b->d_list = (int32_t*)(base + o_list);
        b->d_queue = (int*)(base + o_queue);
        su.go.px = (double*)(base + o_px);
        std::vector<char> head(o_list + sizeof(int32_t) * lists.size());
        if (sp) {
            spread_rule((double*)head.data());
            su.go.sp_rule = (const double*)(base + o_rule);
            su.go.sp_rw = (double*)(base + o_rw);
        }
        if (!lists.empty()) {
            std::copy(lists.begin(), lists.end(), (int32_t*)(head.data() + o_list));
            check(cudaMemcpyAsync(base, head.data(), head.size(), cudaMemcpyHostToDevice, ctx->stream), "h2d");
            check(cudaStreamSynchronize(ctx->stream), "sync");
        }
    } catch (...) {
        group_batch_destroy(ctx, b);
        throw;
    }
    return b;
}

int group_batch_buckets(const GroupBatch* b) { return (int)b->su.plan.buckets.size(); }

// bucket < 0: every bucket, each with its chosen block size; threads <= 0: the chosen one.
void group_batch_enqueue(cpb_ctx* ctx, GroupBatch* b, cudaStream_t st, int bucket, int threads) {
    const auto& bks = b->su.plan.buckets;
    for (int k = 0; k < (int)bks.size(); ++k) {
        if (bucket >= 0 && k != bucket) continue;
        launch_bucket(ctx, st, b->su, bks[k], b->d_list + b->at[k], b->d_list + b->su.plan.n_kernel + b->at[k],
                      b->d_queue + kQueueInts * k, threads > 0 ? threads : b->threads[k], 0);
    }
    if (bucket < 0) launch_spread(ctx, st, b->su, b->d_list, group_batch_size(b));
}

void group_batch_set_threads(GroupBatch* b, int bucket, int threads) { b->threads[bucket] = valid_threads(threads); }
int group_batch_threads(const GroupBatch* b, int bucket) { return b->threads[bucket]; }
int group_batch_occupancy(GroupBatch* b, int bucket, int threads) {
    return group_occupancy(b->su.plan.buckets[bucket], threads, group_node(b->su.dp));
}
int64_t group_batch_size(const GroupBatch* b) { return b->su.plan.n_kernel; }

// Tuning signature of one bucket: what its best block size depends on.
std::string group_batch_signature(const GroupBatch* b, int bucket) {
    const GroupSetup& su = b->su;
    const Bucket& B = su.plan.buckets[bucket];
    char buf[256];
    std::snprintf(buf, sizeof(buf), "groups psf%d nodes%d el%d p%d S2_%d mR%d nmax%d umax%d G2^%d", su.dp.kind,
                  su.dp.n_nodes, su.eltype, su.C.p, su.C.S2, su.C.mR, B.nmax, B.umax,
                  (int)std::log2((double)std::max<size_t>(B.groups.size(), 1)));
    return buf;
}

void group_batch_destroy(cpb_ctx* ctx, GroupBatch* b) {
    if (!b) return;
    if (b->block) cudaFreeAsync(b->block, ctx->stream);
    delete b;
}

}  // namespace cpb
