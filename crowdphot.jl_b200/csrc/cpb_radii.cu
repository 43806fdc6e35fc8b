// cpb_radii.cu -- model_rad = :auto: per-star model-render radii (the PSF's curve of
// growth on the host, the noise quantile and the radii on the device).
//
// Restates, for the library's device path,
//   _model_radii (:auto branch)       src/photometry/psf_photometry_simultaneous.jl:209-243
//   curve_of_growth                    src/curve_of_growth.jl:143-212
//   CircularAperture ExactOverlap      src/apertures.jl:52-66, 93-103, 160-166, 196-290
// The unit PSF's annular surface brightness depends only on the PSF, R_cap and
// (for the Gaussian) its FWHM, so it is computed once per PSF handle and kept.
// Arithmetic is FP64 throughout.
#include <algorithm>
#include <cmath>
#include <mutex>
#include <vector>

#include "cpb_internal.cuh"

namespace cpb {
namespace {

const double kPi = 3.141592653589793;

// Exact area of a unit pixel / circle overlap (apertures.jl:196-290).
double area_triangle(double x0, double y0, double x1, double y1, double x2, double y2) {
    return std::fabs(x0 * (y1 - y2) + x1 * (y2 - y0) + x2 * (y0 - y1)) / 2;
}

double area_arc(double x0, double y0, double x1, double y1, double r) {
    const double a = std::sqrt((x1 - x0) * (x1 - x0) + (y1 - y0) * (y1 - y0));
    const double th = 2 * std::asin(a / (2 * r));
    return r * r * (th - std::sin(th)) / 2;
}

// Rectangle [xmin, xmax] x [ymin, ymax] in the first quadrant (0 <= xmin, 0 <= ymin).
double overlap_core(double xmin, double ymin, double xmax, double ymax, double r) {
    if (xmin * xmin + ymin * ymin > r * r) return 0.0;
    if (xmax * xmax + ymax * ymax < r * r) return (xmax - xmin) * (ymax - ymin);
    const double d1 = std::sqrt(xmax * xmax + ymin * ymin);
    const double d2 = std::sqrt(xmin * xmin + ymax * ymax);
    if (d1 < r && d2 < r) {
        const double x1 = std::sqrt(r * r - ymax * ymax), y1 = ymax;
        const double x2 = xmax, y2 = std::sqrt(r * r - xmax * xmax);
        return (xmax - xmin) * (ymax - ymin) - area_triangle(x1, y1, x2, y2, xmax, ymax) +
               area_arc(x1, y1, x2, y2, r);
    }
    if (d1 < r) {
        const double x1 = xmin, y1 = std::sqrt(r * r - xmin * xmin);
        const double x2 = xmax, y2 = std::sqrt(r * r - xmax * xmax);
        return area_arc(x1, y1, x2, y2, r) + area_triangle(x1, y1, x1, ymin, xmax, ymin) +
               area_triangle(x1, y1, x2, ymin, x2, y2);
    }
    if (d2 < r) {
        const double x1 = std::sqrt(r * r - ymin * ymin), y1 = ymin;
        const double x2 = std::sqrt(r * r - ymax * ymax), y2 = ymax;
        return area_arc(x1, y1, x2, y2, r) + area_triangle(x1, y1, xmin, y1, xmin, ymax) +
               area_triangle(x1, y1, xmin, y2, x2, y2);
    }
    const double x1 = std::sqrt(r * r - ymin * ymin), y1 = ymin;
    const double x2 = xmin, y2 = std::sqrt(r * r - xmin * xmin);
    return area_arc(x1, y1, x2, y2, r) + area_triangle(x1, y1, x2, y2, xmin, ymin);
}

// Any rectangle, split at the axes into first-quadrant pieces.
double overlap_single(double xmin, double ymin, double xmax, double ymax, double r) {
    if (r <= 0) return 0.0;
    if (0 <= xmin) {
        if (0 <= ymin) return overlap_core(xmin, ymin, xmax, ymax, r);
        if (0 >= ymax) return overlap_core(-ymax, xmin, -ymin, xmax, r);
        return overlap_single(xmin, ymin, xmax, 0, r) + overlap_single(xmin, 0, xmax, ymax, r);
    }
    if (0 >= xmax) {
        if (0 <= ymin) return overlap_core(-xmax, ymin, -xmin, ymax, r);
        if (0 >= ymax) return overlap_core(-xmax, -ymax, -xmin, -ymin, r);
        return overlap_single(xmin, ymin, xmax, 0, r) + overlap_single(xmin, 0, xmax, ymax, r);
    }
    if (0 <= ymin) return overlap_single(xmin, ymin, 0, ymax, r) + overlap_single(0, ymin, xmax, ymax, r);
    if (0 >= ymax) return overlap_single(xmin, ymin, 0, ymax, r) + overlap_single(0, ymin, xmax, ymax, r);
    return overlap_single(xmin, ymin, 0, 0, r) + overlap_single(0, ymin, xmax, 0, r) +
           overlap_single(xmin, 0, 0, ymax, r) + overlap_single(0, 0, xmax, ymax, r);
}

// aperture_weight(::CircularAperture at the origin, i, j, ExactOverlap()).
double aperture_weight(int i, int j, double r) {
    const double dy = (double)i, dx = (double)j;
    const double d2 = dx * dx + dy * dy;
    const double dr = std::sqrt(2.0) / 2;
    if (d2 > (r + dr) * (r + dr)) return 0.0;
    if (r > dr && d2 < (r - dr) * (r - dr)) return 1.0;
    if (r <= 0) return 0.0;
    return overlap_single(dx - 0.5, dy - 0.5, dx + 0.5, dy + 0.5, r);
}

// bicubic_interpolate value of one node at detector offset (dy, dx) = pixel
// minus star centre (empirical_models.jl:185-292).
double node_value(const cpb_psf* ps, const DevNode& nd, double dy, double dx) {
    const double* data = ps->h_data64.data() + nd.off;
    const double u = nd.sx * dx + nd.ox;
    const double v = nd.sy * dy + nd.oy;
    const int nyd = nd.ny, nxd = nd.nx;
    if (!(std::isfinite(u) && std::isfinite(v) && u >= 1 && u <= nxd && v >= 1 && v <= nyd)) return nd.fill;
    const int lx = std::min(std::max((int)std::floor(u), 1), nxd - 1);
    const int ly = std::min(std::max((int)std::floor(v), 1), nyd - 1);
    const double du = u - lx, dv = v - ly;
    auto cl = [](int t, int n) { return std::min(std::max(t, 1), n) - 1; };
    const int ix[4] = {cl(lx - 1, nxd), lx - 1, lx, cl(lx + 2, nxd)};
    const int iy[4] = {cl(ly - 1, nyd), ly - 1, ly, cl(ly + 2, nyd)};
    double row[4];
    for (int r = 0; r < 4; ++r) {
        const double a = data[iy[r] + (int64_t)ix[0] * nyd], b = data[iy[r] + (int64_t)ix[1] * nyd];
        const double c = data[iy[r] + (int64_t)ix[2] * nyd], e = data[iy[r] + (int64_t)ix[3] * nyd];
        const double k1 = (c - a) / 2, k4 = c - b - k1, k2 = 3 * k4 - (e - b) / 2 + k1, k3 = k4 - k2;
        row[r] = du * (du * (du * k3 + k2) + k1) + b;
    }
    const double v1 = (row[2] - row[0]) / 2, v4 = row[2] - row[1] - v1, v2 = 3 * v4 - (row[3] - row[1]) / 2 + v1,
                 v3 = v4 - v2;
    return dv * (dv * (dv * v3 + v2) + v1) + row[1];
}

// Node weights of GriddedPSFModel at (Y, X) (_grid_corners_dw, gridded_psf.jl:176-208,
// weights only); single-node and ImagePSF models: node 0 with weight 1.
int host_corners(const cpb_psf* ps, double Y, double X, int idx[4], double wts[4]) {
    const DevPsf& P = ps->dev;
    if (P.n_nodes == 1 || P.kind != CPB_PSF_GRIDDED_IMAGE) {
        idx[0] = 0;
        wts[0] = 1.0;
        return 1;
    }
    const auto& yg = ps->h_ygrid;
    const auto& xg = ps->h_xgrid;
    const int gny = (int)yg.size(), gnx = (int)xg.size();
    int iy = 0, ix = 0;
    for (int k = 0; k < gny; ++k) iy += yg[k] <= Y ? 1 : 0;
    for (int k = 0; k < gnx; ++k) ix += xg[k] <= X ? 1 : 0;
    iy = std::min(std::max(iy, 1), gny - 1);
    ix = std::min(std::max(ix, 1), gnx - 1);
    const double y0 = yg[iy - 1], y1 = yg[iy], x0 = xg[ix - 1], x1 = xg[ix];
    const double Yc = std::min(std::max(Y, y0), y1), Xc = std::min(std::max(X, x0), x1);
    const double inv = 1.0 / ((x1 - x0) * (y1 - y0));
    const double w4[4] = {(x1 - Xc) * (y1 - Yc) * inv, (Xc - x0) * (y1 - Yc) * inv, (x1 - Xc) * (Yc - y0) * inv,
                          (Xc - x0) * (Yc - y0) * inv};
    const int i4[4] = {ps->h_index_grid[(iy - 1) + (ix - 1) * gny], ps->h_index_grid[(iy - 1) + ix * gny],
                       ps->h_index_grid[iy + (ix - 1) * gny], ps->h_index_grid[iy + ix * gny]};
    int k = 0;
    for (int q = 0; q < 4; ++q)
        if (w4[q] != 0.0) {
            idx[k] = i4[q];
            wts[k] = w4[q];
            ++k;
        }
    return k;
}

}  // namespace

// The unit model (flux = 1, bkg = 0) centred at (Y, X), at pixel (i, j).
double host_unit_value(const cpb_psf* ps, double fwhm, double Y, double X, int i, int j) {
    if (ps->dev.kind == CPB_PSF_CIRCULAR_GAUSSIAN) {
        const double g = -4.0 * std::log(2.0);
        const double r2 = ((double)i - Y) * ((double)i - Y) + ((double)j - X) * ((double)j - X);
        const double norm = -(kPi * fwhm * fwhm / g);
        return (1.0 / norm) * std::exp(g * r2 / (fwhm * fwhm));
    }
    int idx[4];
    double wts[4];
    const int nc = host_corners(ps, Y, X, idx, wts);
    double s = 0;
    for (int k = 0; k < nc; ++k) s += wts[k] * node_value(ps, ps->h_nodes[idx[k]], (double)i - Y, (double)j - X);
    return s;
}

// PSF.extent of the model centred at (Y, X) (PSF.jl:285-296, empirical_models.jl:167-176,
// gridded_psf.jl:281-300): (ymin, ymax, xmin, xmax).
void host_extent(const cpb_psf* ps, double fwhm, double Y, double X, double e[4]) {
    if (ps->dev.kind == CPB_PSF_CIRCULAR_GAUSSIAN) {
        const double a = 5.0 * fwhm / 2;  // fwhm_factor 5, no rotation
        e[0] = Y - a;
        e[1] = Y + a;
        e[2] = X - a;
        e[3] = X + a;
        return;
    }
    int idx[4];
    double wts[4];
    const int nc = host_corners(ps, Y, X, idx, wts);
    for (int k = 0; k < nc; ++k) {
        const DevNode& nd = ps->h_nodes[idx[k]];
        const double lo_y = Y - (nd.oy - 1.0) / nd.sy, hi_y = Y + ((double)nd.ny - nd.oy) / nd.sy;
        const double lo_x = X - (nd.ox - 1.0) / nd.sx, hi_x = X + ((double)nd.nx - nd.ox) / nd.sx;
        if (k == 0) {
            e[0] = lo_y;
            e[1] = hi_y;
            e[2] = lo_x;
            e[3] = hi_x;
        } else {
            e[0] = std::min(e[0], lo_y);
            e[1] = std::max(e[1], hi_y);
            e[2] = std::min(e[2], lo_x);
            e[3] = std::max(e[3], hi_x);
        }
    }
}

namespace {

// The unit model (y = x = 0, flux = 1, bkg = 0) at pixel (i, j).
double unit_value(const cpb_psf* ps, int i, int j) { return host_unit_value(ps, 0.0, 0.0, 0.0, i, j); }

// Annular mean surface brightness of the unit PSF for radii 1..R_cap
// (_model_radii, :226-236), from its curve of growth.
std::vector<double> unit_sb(const cpb_psf* ps, double fwhm, int R_cap) {
    std::vector<double> cog(R_cap);
    if (ps->dev.kind == CPB_PSF_CIRCULAR_GAUSSIAN) {
        // analytic overload (curve_of_growth.jl:180-195); integral(model) = flux = 1
        const double g = -4.0 * std::log(2.0);
        for (int r = 1; r <= R_cap; ++r) cog[r - 1] = 1.0 * (1.0 - std::exp(g * ((double)r * r) / (fwhm * fwhm)));
    } else {
        // generic curve_of_growth: exact-overlap apertures over the unit model's pixels
        const int W = 2 * R_cap + 1;
        std::vector<double> val((size_t)W * W);
        for (int j = -R_cap; j <= R_cap; ++j)
            for (int i = -R_cap; i <= R_cap; ++i) val[(i + R_cap) + (size_t)(j + R_cap) * W] = unit_value(ps, i, j);
        for (int r = 1; r <= R_cap; ++r) {
            double flux = 0;
            for (int j = -r; j <= r; ++j)
                for (int i = -r; i <= r; ++i) {
                    const double w = aperture_weight(i, j, (double)r);
                    if (!(w > 0)) continue;
                    flux += w * val[(i + R_cap) + (size_t)(j + R_cap) * W];
                }
            cog[r - 1] = flux;
        }
    }
    std::vector<double> sb(R_cap);
    double prev = 0;
    for (int r = 1; r <= R_cap; ++r) {
        const double ee = cog[r - 1] / cog[R_cap - 1];
        sb[r - 1] = std::max((ee - prev) / (kPi * (double)(r * r - (r - 1) * (r - 1))), 0.0);
        prev = ee;
    }
    return sb;
}

}  // namespace

namespace {

constexpr int kQuantThreads = 1024, kDigit = 11, kBins = 1 << kDigit;

// sigma_bg of _model_radii (:192-225): the 0.84 quantile (type 7) of the positive
// finite weights of the sample w[0], w[step], ... (nsamp of them), then
// sqrt(1 / quantile).  One block: the sample is copied to `buf` once and the two
// order statistics found by a radix select, 11 bits a pass (positive doubles order
// as their bit patterns), counting in shared memory with one atomic per distinct
// digit of a warp.  res[0] = sigma_bg, res[1] = the number of positive weights.
// Rounding steps are those of the host arithmetic (no contraction).
// Bound by the latency of one block's passes over at most 131,071 samples; a strided
// read-back and a host sort of them took half of a 613 x 421 field's call (whole call
// 9.9 -> 5.1 ms).
__global__ void __launch_bounds__(kQuantThreads) k_noise_quantile(const double* __restrict__ w, int64_t step,
                                                                  int64_t nsamp, double* buf, double* res) {
    __shared__ unsigned hist[kBins];
    __shared__ unsigned wsum[kQuantThreads / 32];
    __shared__ unsigned long long s_prefix;
    __shared__ unsigned s_rank, s_cnt;
    __shared__ unsigned long long s_next;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    if (tid == 0) s_cnt = 0;
    __syncthreads();
    unsigned good = 0;
    for (int64_t i = tid; i < nsamp; i += kQuantThreads) {
        double v = w[i * step];
        const bool ok = v > 0 && isfinite(v);
        good += ok;
        buf[i] = ok ? v : 0.0;  // 0: not in the sample
    }
    good = __reduce_add_sync(0xffffffffu, good);
    if (lane == 0 && good) atomicAdd(&s_cnt, good);
    __syncthreads();
    const unsigned n = s_cnt;
    if (tid == 0) res[1] = (double)n;
    if (n == 0) {
        if (tid == 0) res[0] = 1.0;
        return;
    }
    const double h = __dmul_rn((double)(n - 1), 0.84);
    const unsigned lo = (unsigned)floor(h);
    if (tid == 0) {
        s_prefix = 0;
        s_rank = lo;
    }
    unsigned long long mask = 0;
    for (int shift = 64 - kDigit; ; shift = shift > kDigit ? shift - kDigit : 0) {
        for (int b = tid; b < kBins; b += kQuantThreads) hist[b] = 0;
        __syncthreads();
        const unsigned long long prefix = s_prefix;
        for (int64_t i0 = 0; i0 < nsamp; i0 += kQuantThreads) {
            const int64_t i = i0 + tid;
            const unsigned long long key = i < nsamp ? (unsigned long long)__double_as_longlong(buf[i]) : 0ull;
            const bool in = key != 0 && (key & mask) == prefix;
            const unsigned d = in ? (unsigned)(key >> shift) & (kBins - 1) : kBins;
            const unsigned same = __match_any_sync(0xffffffffu, d);
            if (in && lane == __ffs(same) - 1) atomicAdd(&hist[d], __popc(same));
        }
        __syncthreads();
        // the bin holding rank s_rank: two bins a thread, block prefix sums
        const unsigned c0 = hist[2 * tid], c1 = hist[2 * tid + 1];
        unsigned incl = c0 + c1;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned t = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += t;
        }
        if (lane == 31) wsum[wid] = incl;
        __syncthreads();
        unsigned before = 0;
        for (int q = 0; q < wid; ++q) before += wsum[q];
        const unsigned excl = before + incl - (c0 + c1), rank = s_rank;
        __syncthreads();  // every thread has read s_rank
        if (rank >= excl && rank < excl + c0 + c1) {
            const bool second = rank >= excl + c0;
            s_prefix = prefix | (unsigned long long)(2 * tid + (second ? 1 : 0)) << shift;
            s_rank = rank - excl - (second ? c0 : 0);
        }
        mask |= (unsigned long long)(kBins - 1) << shift;
        __syncthreads();
        if (shift == 0) break;
    }
    // ws[lo] = the selected value; ws[lo + 1]: the same value when more than one
    // sample past rank lo has it, else the smallest larger one
    const unsigned long long key_lo = s_prefix;
    if (tid == 0) {
        s_next = ~0ull;
        s_cnt = 0;
    }
    __syncthreads();
    unsigned long long nxt = ~0ull;
    unsigned le = 0;
    for (int64_t i = tid; i < nsamp; i += kQuantThreads) {
        const unsigned long long key = (unsigned long long)__double_as_longlong(buf[i]);
        if (key == 0) continue;
        if (key <= key_lo) ++le;
        else nxt = key < nxt ? key : nxt;
    }
    le = __reduce_add_sync(0xffffffffu, le);
    if (lane == 0) atomicAdd(&s_cnt, le);
    atomicMin(&s_next, nxt);
    __syncthreads();
    if (tid == 0) {
        const double a = __longlong_as_double((long long)key_lo);
        const double b = lo + 1 >= n || s_cnt > lo + 1 ? a : __longlong_as_double((long long)s_next);
        const double wval = __dadd_rn(a, __dmul_rn(h - (double)lo, b - a));
        res[0] = wval > 0 ? sqrt(1.0 / wval) : 1.0;
    }
}

// Per active star: the radius where its flux times the unit annular surface
// brightness falls below nsigma * sigma_bg (:237-243).
__global__ void k_model_radii(int64_t n_act, const int32_t* __restrict__ act, const double* __restrict__ f0,
                              const double* __restrict__ sb, const double* __restrict__ res, double nsigma, int R_fit,
                              int R_cap, int32_t* out) {
    const int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (j >= n_act) return;
    const double thr = __dmul_rn(nsigma, res[0]);
    const double F = fmax(f0[act[j]], 0.0);
    int r = R_fit;
    while (r < R_cap && __dmul_rn(F, sb[r - 1]) > thr) ++r;
    out[j] = r;
}

}  // namespace

void model_radii_auto(cpb_ctx* ctx, const cpb_psf* psf, double fwhm, double nsigma, int R_fit, int R_cap,
                      const double* d_w, int64_t npix, double* d_buf, double* d_sb, const int32_t* d_act,
                      int64_t n_act, const double* d_f0, int32_t* d_R, std::vector<int32_t>& out) {
    cudaStream_t st = ctx->stream;
    const int64_t step = std::max<int64_t>(1, npix / 65536), nsamp = (npix + step - 1) / step;
    cpb_psf* ps = const_cast<cpb_psf*>(psf);
    std::vector<double> sb;
    {
        std::lock_guard<std::mutex> lk(ps->cog_mu);
        const auto key = std::make_pair(R_cap, psf->dev.kind == CPB_PSF_CIRCULAR_GAUSSIAN ? fwhm : 0.0);
        auto it = ps->cog_sb.find(key);
        if (it == ps->cog_sb.end()) it = ps->cog_sb.emplace(key, unit_sb(psf, fwhm, R_cap)).first;
        sb = it->second;
    }
    double* d_res = d_sb + sb.size();
    check(cudaMemcpyAsync(d_sb, sb.data(), sizeof(double) * sb.size(), cudaMemcpyHostToDevice, st), "h2d");
    k_noise_quantile<<<1, kQuantThreads, 0, st>>>(d_w, step, nsamp, d_buf, d_res);
    check(cudaGetLastError(), "k_noise_quantile");
    k_model_radii<<<(unsigned)((n_act + 255) / 256), 256, 0, st>>>(n_act, d_act, d_f0, d_sb, d_res, nsigma, R_fit,
                                                                   R_cap, d_R);
    check(cudaGetLastError(), "k_model_radii");
    out.resize(n_act);
    double res[2] = {0, 0};
    check(cudaMemcpyAsync(res, d_res, sizeof(res), cudaMemcpyDeviceToHost, st), "d2h");
    check(cudaMemcpyAsync(out.data(), d_R, sizeof(int32_t) * n_act, cudaMemcpyDeviceToHost, st), "d2h");
    check(cudaStreamSynchronize(st), "sync");
    if (res[1] == 0) throw ArgError{"model_rad=:auto found no positive finite weights to estimate the noise"};
}

}  // namespace cpb
