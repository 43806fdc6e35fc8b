// cpb_api.cu -- the extern "C" boundary (include/crowdphot_b200.h).
//
// Context and PSF handles, argument validation that mirrors the reference's
// constructors, host<->device staging, and error translation: C++ exceptions
// never cross the ABI; every entry point returns a CPB_* status and leaves a
// message for cpb_last_error().
#include <algorithm>
#include <cmath>
#include <cstring>
#include <memory>
#include <type_traits>
#include <set>
#include <string>
#include <vector>

#include "cpb_internal.cuh"

namespace cpb {

// A named grow-only scratch buffer of at least `bytes`.  Growth frees and
// allocates in stream order on the context's stream (cudaFreeAsync /
// cudaMallocAsync from the device's memory pool): no device-wide
// synchronisation, so contexts sharing the GPU -- the server's slots -- keep
// running while one of them grows.  The copy stream's work is ordered before
// the free and after the new allocation.
void* scratch(cpb_ctx* ctx, const char* name, size_t bytes) {
    if (ctx->arena) return arena_carve(ctx->arena, name, bytes);
    auto& b = ctx->bufs[name];
    if (b.bytes >= bytes && b.p) return b.p;
    if (b.p) {
        check(cudaEventRecord(ctx->grow_ev, ctx->copy_stream), "grow order");
        check(cudaStreamWaitEvent(ctx->stream, ctx->grow_ev, 0), "grow order");
        check(cudaFreeAsync(b.p, ctx->stream), "cudaFreeAsync");
        b.p = nullptr;
        b.bytes = 0;
    }
    size_t want = std::max<size_t>(bytes, 256);
    void* p = nullptr;
    cudaError_t e = cudaMallocAsync(&p, want, ctx->stream);
    if (e == cudaErrorMemoryAllocation) {
        cudaGetLastError();
        throw OomError{std::string("device memory exhausted allocating ") + name};
    }
    check(e, "cudaMallocAsync");
    check(cudaEventRecord(ctx->grow_ev, ctx->stream), "grow order");
    check(cudaStreamWaitEvent(ctx->copy_stream, ctx->grow_ev, 0), "grow order");
    b.p = p;
    b.bytes = want;
    return p;
}

static cudaEvent_t pool_event(cpb_ctx* ctx) {
    if (!ctx->event_pool.empty()) {
        cudaEvent_t e = ctx->event_pool.back();
        ctx->event_pool.pop_back();
        return e;
    }
    cudaEvent_t e;
    check(cudaEventCreate(&e), "cudaEventCreate");
    return e;
}

KernelScope::KernelScope(cpb_ctx* c, const char* n, double by) : ctx(c), name(n), bytes(by) {
    ctx->launches += 1;
    if (ctx->profile) {
        a = pool_event(ctx);
        b = pool_event(ctx);
        cudaEventRecord(a, ctx->stream);
    }
}

KernelScope::~KernelScope() {
    if (a) {
        cudaEventRecord(b, ctx->stream);
        ctx->pending.push_back({name, a, b, bytes});
    }
}

void resolve_kernel_events(cpb_ctx* ctx) {
    if (ctx->pending.empty()) return;
    cudaStreamSynchronize(ctx->stream);
    for (auto& p : ctx->pending) {
        float ms = 0;
        cudaEventElapsedTime(&ms, p.a, p.b);
        auto& k = ctx->kstats[p.name];
        k.launches += 1;
        k.seconds += ms * 1e-3;
        k.bytes += p.bytes;
        ctx->event_pool.push_back(p.a);
        ctx->event_pool.push_back(p.b);
    }
    ctx->pending.clear();
}

}  // namespace cpb

using namespace cpb;

extern "C" {

const char* cpb_version(void) { return "crowdphot_b200 0.1 (sm_100a)"; }

int cpb_ctx_create(int device, cpb_ctx** out) {
    if (!out) return CPB_ERR_ARGUMENT;
    *out = nullptr;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
        cudaGetLastError();
        return CPB_ERR_NO_DEVICE;
    }
    if (device < 0 || device >= ndev) return CPB_ERR_ARGUMENT;
    auto* ctx = new cpb_ctx();
    ctx->device = device;
    if (cudaSetDevice(device) != cudaSuccess || cudaStreamCreateWithFlags(&ctx->stream, cudaStreamNonBlocking) != cudaSuccess ||
        cudaEventCreate(&ctx->ev0) != cudaSuccess || cudaEventCreate(&ctx->ev1) != cudaSuccess ||
        cudaEventCreateWithFlags(&ctx->grow_ev, cudaEventDisableTiming) != cudaSuccess ||
        cudaMallocHost(&ctx->pinned, 4096) != cudaSuccess ||
        cudaStreamCreateWithFlags(&ctx->copy_stream, cudaStreamNonBlocking) != cudaSuccess) {
        cudaGetLastError();
        delete ctx;
        return CPB_ERR_CUDA;
    }
    for (int k = 0; k < cpb_ctx::kCopyEvents; ++k)
        if (cudaEventCreateWithFlags(&ctx->copy_ev[k], cudaEventDisableTiming) != cudaSuccess) {
            cudaGetLastError();
            return CPB_ERR_CUDA;
        }
    cudaDeviceGetAttribute(&ctx->n_sm, cudaDevAttrMultiProcessorCount, device);
    *out = ctx;
    return CPB_OK;
}

int cpb_ctx_destroy(cpb_ctx* ctx) {
    if (!ctx) return CPB_OK;
    {
        std::lock_guard<std::mutex> lk(ctx->mu);
        cudaSetDevice(ctx->device);
        if (ctx->copy_stream) cudaStreamSynchronize(ctx->copy_stream);
        ctx->copier.reset();
        for (auto& kv : ctx->bufs)
            if (kv.second.p) cudaFreeAsync(kv.second.p, ctx->stream);
        ctx->bufs.clear();
        cudaStreamSynchronize(ctx->stream);
        if (ctx->pinned) cudaFreeHost(ctx->pinned);
        for (auto e : ctx->event_pool) cudaEventDestroy(e);
        for (auto& p : ctx->pending) {
            cudaEventDestroy(p.a);
            cudaEventDestroy(p.b);
        }
        if (ctx->ev0) cudaEventDestroy(ctx->ev0);
        if (ctx->ev1) cudaEventDestroy(ctx->ev1);
        if (ctx->grow_ev) cudaEventDestroy(ctx->grow_ev);
        if (ctx->copy_stream) cudaStreamSynchronize(ctx->copy_stream);
        for (auto e : ctx->copy_ev)
            if (e) cudaEventDestroy(e);
        if (ctx->copy_stream) cudaStreamDestroy(ctx->copy_stream);
        if (ctx->stream) cudaStreamDestroy(ctx->stream);
    }
    delete ctx;
    return CPB_OK;
}

const char* cpb_last_error(const cpb_ctx* ctx) { return ctx ? ctx->err.c_str() : "null context"; }

int cpb_ctx_set_profiling(cpb_ctx* ctx, int enable) {
    return guarded(ctx, [&]() -> int {
        resolve_kernel_events(ctx);
        ctx->profile = enable != 0;
        return CPB_OK;
    });
}

int cpb_ctx_set_wait_limit(cpb_ctx* ctx, int64_t polls) {
    return guarded(ctx, [&]() -> int {
        ctx->wait_limit = polls;
        return CPB_OK;
    });
}

int cpb_ctx_inject_fault(cpb_ctx* ctx, int32_t fault) {
    return guarded(ctx, [&]() -> int {
        if (fault != CPB_FAULT_NONE && fault != CPB_FAULT_HOLD_READY_STAR) throw ArgError{"unknown fault kind"};
        ctx->fault = fault;
        return CPB_OK;
    });
}

int cpb_ctx_kernel_stats(cpb_ctx* ctx, cpb_kernel_stat* out, int max_out, int* n_out, int64_t* launches, int reset) {
    return guarded(ctx, [&]() -> int {
        resolve_kernel_events(ctx);
        int k = 0;
        for (auto& kv : ctx->kstats) {
            if (out && k < max_out) {
                std::memset(&out[k], 0, sizeof(cpb_kernel_stat));
                std::strncpy(out[k].name, kv.first.c_str(), sizeof(out[k].name) - 1);
                out[k].launches = kv.second.launches;
                out[k].seconds = kv.second.seconds;
                out[k].bytes = kv.second.bytes;
            }
            ++k;
        }
        if (n_out) *n_out = k;
        if (launches) *launches = ctx->launches;
        if (reset) {
            ctx->kstats.clear();
            ctx->launches = 0;
        }
        return CPB_OK;
    });
}

int cpb_psf_upload(cpb_ctx* ctx, const cpb_psf_desc* d, cpb_psf** out) {
    return guarded(ctx, [&]() -> int {
        if (!d || !out) throw ArgError{"null argument"};
        *out = nullptr;
        auto* ps = new cpb_psf();
        DevPsf& dp = ps->dev;
        std::memset(&dp, 0, sizeof(dp));
        dp.kind = d->kind;
        dp.fwhm = d->fwhm;
        try {
            if (d->kind == CPB_PSF_CIRCULAR_GAUSSIAN) {
                if (!(std::isfinite(d->fwhm))) throw ArgError{"CircularGaussianPSF fwhm must be finite"};
                dp.n_nodes = 0;
                *out = ps;
                return CPB_OK;
            }
            if (d->kind != CPB_PSF_GRIDDED_IMAGE && d->kind != CPB_PSF_IMAGE) throw ArgError{"unsupported PSF kind"};
            const int nn = d->n_nodes;
            if (nn < 1) throw ArgError{"`psfs` must be non-empty"};
            if (d->kind == CPB_PSF_IMAGE && nn != 1) throw ArgError{"ImagePSF takes exactly one node"};
            if (nn > kMaxNodes) throw ArgError{"too many PSF nodes"};
            if (d->eltype != CPB_F32 && d->eltype != CPB_F64) throw ArgError{"unsupported PSF eltype"};
            // ImagePSF checks (empirical_models.jl:101-140)
            std::vector<double> h64;
            std::vector<DevNode> nodes(nn);
            int64_t off = 0;
            for (int k = 0; k < nn; ++k) {
                DevNode& nd = nodes[k];
                const int64_t nyd = d->node_ny[k], nxd = d->node_nx[k];
                if (nyd < 4 || nxd < 4) throw ArgError{"each axis of `data` must have at least 4 samples"};
                nd.ny = (int32_t)nyd;
                nd.nx = (int32_t)nxd;
                nd.off = off;
                nd.sx = (double)d->node_os[2 * k];
                nd.sy = (double)d->node_os[2 * k + 1];
                if (!(nd.sx > 0 && nd.sy > 0)) throw ArgError{"`oversampling` values must be positive"};
                nd.oy = d->node_origin[2 * k];
                nd.ox = d->node_origin[2 * k + 1];
                if (!std::isfinite(nd.oy) || !std::isfinite(nd.ox)) throw ArgError{"`origin` must be finite"};
                nd.fill = d->node_fill_value ? d->node_fill_value[k] : 0.0;
                const int64_t ne = nyd * nxd;
                const int64_t padded = (ne + 3) / 4 * 4;  // 32-byte (FP64) / 16-byte (FP32) node alignment
                h64.resize(off + padded, 0.0);
                for (int64_t q = 0; q < ne; ++q) {
                    double v = d->eltype == CPB_F64 ? ((const double*)d->node_data[k])[q]
                                                    : (double)((const float*)d->node_data[k])[q];
                    if (!std::isfinite(v)) throw ArgError{"all elements of `data` must be finite"};
                    h64[off + q] = v;
                }
                off += padded;
            }
            // node grid (gridded_psf.jl:106-134)
            std::vector<double> yg, xg;
            std::vector<int32_t> ig;
            if (nn == 1 || d->kind == CPB_PSF_IMAGE) {
                yg = {d->grid_y ? d->grid_y[0] : 0.0};
                xg = {d->grid_x ? d->grid_x[0] : 0.0};
                ig = {0};
            } else {
                for (int k = 0; k < nn; ++k)
                    if (!std::isfinite(d->grid_y[k]) || !std::isfinite(d->grid_x[k]))
                        throw ArgError{"`grid_y` and `grid_x` must be finite"};
                std::set<double> ys(d->grid_y, d->grid_y + nn), xs(d->grid_x, d->grid_x + nn);
                yg.assign(ys.begin(), ys.end());
                xg.assign(xs.begin(), xs.end());
                if (yg.size() < 2 || xg.size() < 2)
                    throw ArgError{
                        "`grid_y` and `grid_x` must each contain at least 2 unique values unless a single PSF is "
                        "supplied"};
                if ((size_t)nn != yg.size() * xg.size())
                    throw ArgError{"`grid_y`/`grid_x` positions do not form a complete rectangular grid"};
                ig.assign(yg.size() * xg.size(), -1);
                for (int k = 0; k < nn; ++k) {
                    size_t iy = std::lower_bound(yg.begin(), yg.end(), d->grid_y[k]) - yg.begin();
                    size_t ix = std::lower_bound(xg.begin(), xg.end(), d->grid_x[k]) - xg.begin();
                    int32_t& slot = ig[iy + ix * yg.size()];
                    if (slot != -1) throw ArgError{"duplicate node position"};
                    slot = k;
                }
            }
            // geometry of the copies (DevNode) and their places in one device block (256-byte
            // aligned pieces).  The edge-padded and row-phase copies are read for single-node
            // PSFs only, the row-phase ones where they fit the kernels' shared memory.
            int optin = 0;
            check(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, ctx->device), "attr");
            size_t n_pp = 0, n_lpp = 0, n_row[3] = {0, 0, 0};
            for (int k = 0; k < nn; ++k) {
                DevNode& nd = nodes[k];
                nd.isy = (int32_t)d->node_os[2 * k + 1];
                nd.isx = (int32_t)d->node_os[2 * k];
                nd.PY = (nd.ny + nd.isy - 1) / nd.isy;
                nd.PX = (nd.nx + nd.isx - 1) / nd.isx;
                nd.LPY = (nd.ny + 3 + nd.isy - 1) / nd.isy;
                nd.LPX = (nd.nx + 3 + nd.isx - 1) / nd.isx;
                nd.RPX = (nd.nx + 3) | 1;
                nd.poff = (int64_t)n_pp;
                n_pp += ((size_t)nd.PY * nd.PX * nd.isy * nd.isx + 3) / 4 * 4;
                for (int c = 0; c < 3; ++c) {
                    const int ph = kRowPhase[c] * nd.isy;
                    nd.RPY[c] = (nd.ny + 3 + ph - 1) / ph;
                    if (nn == 1 && row_phase_staged(nd, c, optin)) n_row[c] = row_phase_len(nd, c);
                }
                if (nn == 1) n_lpp = ((size_t)nd.LPY * nd.LPX * nd.isy * nd.isx + 3) / 4 * 4;
            }
            nodes[0].rpoff[2] = (int64_t)n_row[0];  // copies 0 and 2 share rpp64
            size_t bytes = 0;
            auto place = [&](size_t n, size_t size) {
                const size_t at = bytes;
                bytes = (at + n * size + 255) & ~size_t(255);
                return at;
            };
            const size_t n64 = h64.size();
            const size_t o_d64 = place(n64, 8), o_d32 = place(n64, 4), o_pp64 = place(n_pp, 8),
                         o_pp32 = place(n_pp, 4), o_lpp = place(n_lpp, 8), o_r64 = place(n_row[0] + n_row[2], 8),
                         o_r32 = place(n_row[1], 4), o_nd = place(nn, sizeof(DevNode)), o_yg = place(yg.size(), 8),
                         o_xg = place(xg.size(), 8), o_ig = place(ig.size(), 4);
            std::unique_ptr<char[]> block(new char[bytes]);
            char* host = block.get();
            std::memset(host, 0, bytes);
            std::memcpy(host + o_d64, h64.data(), 8 * n64);
            std::memcpy(host + o_nd, nodes.data(), sizeof(DevNode) * nn);
            std::memcpy(host + o_yg, yg.data(), 8 * yg.size());
            std::memcpy(host + o_xg, xg.data(), 8 * xg.size());
            std::memcpy(host + o_ig, ig.data(), 4 * ig.size());
            auto round_all = [](float* to, const double* from, size_t n) {
                for (size_t q = 0; q < n; ++q) to[q] = (float)from[q];
            };
            round_all((float*)(host + o_d32), h64.data(), n64);
            // Offsets of an axis' n entries in a copy that regroups them by their index modulo
            // `ph`, and the samples they come from (before: replicates in front).  Tabulated: a
            // few divisions an axis instead of four a sample of each copy.
            struct AxisMap {
                std::vector<int64_t> at, src;
            };
            auto axis_map = [](int64_t n, int64_t samples, int64_t before, int64_t ph, int64_t phase_step, int64_t step) {
                AxisMap m;
                m.at.resize(n);
                m.src.resize(n);
                for (int64_t i = 0; i < n; ++i) {
                    m.at[i] = (i % ph) * phase_step + (i / ph) * step;
                    m.src[i] = std::min(std::max<int64_t>(i - before, 0), samples - 1);
                }
                return m;
            };
            auto regroup = [&](auto* to, const AxisMap& y, const AxisMap& x, const DevNode& nd) {
                for (size_t k = 0; k < x.at.size(); ++k) {
                    const double* from = h64.data() + nd.off + x.src[k] * nd.ny;
                    auto* col = to + x.at[k];
                    for (size_t i = 0; i < y.at.size(); ++i)
                        col[y.at[i]] = (std::decay_t<decltype(*to)>)from[y.src[i]];
                }
            };
            for (const DevNode& nd : nodes) {
                const int64_t plane = (int64_t)nd.PY * nd.PX;
                regroup((double*)(host + o_pp64) + nd.poff, axis_map(nd.ny, nd.ny, 0, nd.isy, plane, 1),
                        axis_map(nd.nx, nd.nx, 0, nd.isx, plane * nd.isy, nd.PY), nd);
            }
            round_all((float*)(host + o_pp32), (const double*)(host + o_pp64), n_pp);
            if (nn == 1) {
                const DevNode& nd = nodes[0];
                const int64_t plane = (int64_t)nd.LPY * nd.LPX;
                regroup((double*)(host + o_lpp), axis_map(nd.ny + 3, nd.ny, 1, nd.isy, plane, 1),
                        axis_map(nd.nx + 3, nd.nx, 1, nd.isx, plane * nd.isy, nd.LPY), nd);
                const AxisMap cols = axis_map(nd.nx + 3, nd.nx, 1, nd.nx + 3, 1, 1);
                for (int c = 0; c < 3; ++c) {
                    if (!n_row[c]) continue;
                    const AxisMap rows = axis_map(nd.ny + 3, nd.ny, 1, kRowPhase[c] * nd.isy,
                                                  (int64_t)nd.RPY[c] * nd.RPX, nd.RPX);
                    if (c == 1) regroup((float*)(host + o_r32), rows, cols, nd);
                    else regroup((double*)(host + o_r64) + nd.rpoff[c], rows, cols, nd);
                }
            }
            // from the device's pool, as the scratch: a loop over new models takes back what the
            // last one gave
            check(cudaMallocAsync(&ps->d_blob, bytes, ctx->stream), "cudaMallocAsync");
            check(cudaMemcpyAsync(ps->d_blob, host, bytes, cudaMemcpyHostToDevice, ctx->stream), "h2d");
            check(cudaStreamSynchronize(ctx->stream), "sync");
            const char* base = (const char*)ps->d_blob;
            dp.data64 = (const double*)(base + o_d64);
            dp.data32 = (const float*)(base + o_d32);
            dp.pp64 = (const double*)(base + o_pp64);
            dp.pp32 = (const float*)(base + o_pp32);
            dp.lpp64 = n_lpp ? (const double*)(base + o_lpp) : nullptr;
            dp.rpp64 = n_row[0] + n_row[2] ? (const double*)(base + o_r64) : nullptr;
            dp.rpp32 = n_row[1] ? (const float*)(base + o_r32) : nullptr;
            dp.nodes = (const DevNode*)(base + o_nd);
            dp.ygrid = (const double*)(base + o_yg);
            dp.xgrid = (const double*)(base + o_xg);
            dp.index_grid = (const int32_t*)(base + o_ig);
            dp.n_nodes = nn;
            dp.gny = (int32_t)yg.size();
            dp.gnx = (int32_t)xg.size();
            dp.total_elems = (int64_t)n64;
            ps->h_nodes = nodes;
            ps->h_data64 = std::move(h64);
            ps->h_ygrid = yg;
            ps->h_xgrid = xg;
            ps->h_index_grid = ig;
            ps->smem_bytes64 = (int64_t)n64 * 8;
            ps->smem_bytes32 = (int64_t)n64 * 4;
        } catch (...) {
            if (ps->d_blob) cudaFreeAsync(ps->d_blob, ctx->stream);
            delete ps;
            throw;
        }
        *out = ps;
        return CPB_OK;
    });
}

int cpb_psf_free(cpb_ctx* ctx, cpb_psf* ps) {
    if (!ps) return CPB_OK;
    return guarded(ctx, [&]() -> int {
        cudaStreamSynchronize(ctx->stream);
        if (ps->d_blob) cudaFreeAsync(ps->d_blob, ctx->stream);
        delete ps;
        return CPB_OK;
    });
}

int cpb_fit_simultaneous_device(cpb_ctx* ctx, const cpb_psf* psf, const cpb_sim_params* params, const void* d_image,
                                int32_t eltype, int64_t ny, int64_t nx, const void* d_inv_var,
                                const void* d_background, int64_t n, const double* d_y0, const double* d_x0,
                                const double* d_flux0, cpb_sim_result* out) {
    return guarded(ctx, [&]() -> int {
        if (!psf || !params || !out || (n > 0 && (!d_y0 || !d_x0 || !d_flux0)) || !d_image)
            throw ArgError{"null argument"};
        return fit_simultaneous_dev(ctx, psf, params, d_image, eltype, ny, nx, d_inv_var, d_background, n, d_y0, d_x0,
                                    d_flux0, out);
    });
}

int cpb_fit_simultaneous(cpb_ctx* ctx, const cpb_psf* psf, const cpb_sim_params* params, const void* image,
                         int32_t eltype, int64_t ny, int64_t nx, const void* inv_var, const void* background,
                         int64_t n, const double* y0, const double* x0, const double* flux0, cpb_sim_result* out) {
    return guarded(ctx, [&]() -> int {
        if (!psf || !params || !out || !image || (n > 0 && (!y0 || !x0 || !flux0))) throw ArgError{"null argument"};
        if (eltype != CPB_F32 && eltype != CPB_F64) throw ArgError{"unsupported image eltype"};
        if (ny <= 0 || nx <= 0) throw ArgError{"image must be non-empty"};
        const size_t esz = eltype == CPB_F64 ? 8 : 4;
        const size_t bytes = esz * (size_t)ny * (size_t)nx;
        cudaStream_t st = ctx->stream;
        void* d_img = scratch(ctx, "in_image", bytes);
        void* d_iv = inv_var ? scratch(ctx, "in_inv_var", bytes) : nullptr;
        void* d_bk = background ? scratch(ctx, "in_background", bytes) : nullptr;
        double* d_y = (double*)scratch(ctx, "in_y", sizeof(double) * std::max<int64_t>(n, 1));
        double* d_x = (double*)scratch(ctx, "in_x", sizeof(double) * std::max<int64_t>(n, 1));
        double* d_f = (double*)scratch(ctx, "in_flux", sizeof(double) * std::max<int64_t>(n, 1));
        const HostCopy in[3] = {{d_img, image, bytes}, {d_iv, inv_var, bytes}, {d_bk, background, bytes}};
        host_to_device(ctx, in, 3);
        if (n > 0) {
            check(cudaMemcpyAsync(d_y, y0, sizeof(double) * n, cudaMemcpyHostToDevice, st), "h2d y");
            check(cudaMemcpyAsync(d_x, x0, sizeof(double) * n, cudaMemcpyHostToDevice, st), "h2d x");
            check(cudaMemcpyAsync(d_f, flux0, sizeof(double) * n, cudaMemcpyHostToDevice, st), "h2d flux");
        }
        return fit_simultaneous_dev(ctx, psf, params, d_img, eltype, ny, nx, d_iv, d_bk, n, d_y, d_x, d_f, out);
    });
}

int cpb_fit_simultaneous_batch_device(cpb_ctx* ctx, const cpb_psf* psf, const cpb_sim_params* params,
                                      int64_t n_groups, const int64_t* d_pix_offsets, const int32_t* d_ny,
                                      const int32_t* d_nx, const void* d_pixels, int32_t eltype,
                                      const void* d_inv_var, const void* d_background,
                                      const int64_t* d_star_offsets, const double* d_y0, const double* d_x0,
                                      const double* d_flux0, int64_t total_pixels, cpb_group_result* out) {
    return guarded(ctx, [&]() -> int {
        if (!psf || !params || !out || (n_groups > 0 && (!d_pix_offsets || !d_ny || !d_nx || !d_pixels ||
                                                         !d_star_offsets || !d_y0 || !d_x0 || !d_flux0)))
            throw ArgError{"null argument"};
        return fit_groups_dev(ctx, psf, params, n_groups, d_pix_offsets, d_ny, d_nx, d_pixels, eltype, d_inv_var,
                              d_background, d_star_offsets, d_y0, d_x0, d_flux0, total_pixels, out, nullptr,
                              nullptr, nullptr, nullptr);
    });
}

int cpb_fit_simultaneous_batch(cpb_ctx* ctx, const cpb_psf* psf, const cpb_sim_params* params, int64_t n_groups,
                               const int64_t* pix_offsets, const int32_t* ny, const int32_t* nx, const void* pixels,
                               int32_t eltype, const void* inv_var, const void* background,
                               const int64_t* star_offsets, const double* y0, const double* x0, const double* flux0,
                               cpb_group_result* out) {
    return guarded(ctx, [&]() -> int {
        if (!psf || !params || !out || n_groups < 0 || (n_groups > 0 && (!pix_offsets || !ny || !nx || !pixels ||
                                                                          !star_offsets || !y0 || !x0 || !flux0)))
            throw ArgError{"null argument"};
        if (eltype != CPB_F32 && eltype != CPB_F64) throw ArgError{"unsupported image eltype"};
        if (!out->y || !out->x || !out->flux || !out->y_err || !out->x_err || !out->flux_err || !out->converged ||
            !out->valid || !out->n_iter || !out->n_passes || !out->n_failed || !out->status)
            throw ArgError{"null output array"};
        const int64_t G = n_groups;
        if (G == 0) {
            out->n_kernel_groups = out->n_routed_groups = 0;
            out->device_seconds = 0;
            return CPB_OK;
        }
        int64_t npx = 0;
        for (int64_t g = 0; g < G; ++g) {
            if (ny[g] <= 0 || nx[g] <= 0) throw ArgError{"group image size out of range"};
            if (pix_offsets[g] < 0) throw ArgError{"pixel offsets must be non-negative"};
            npx = std::max<int64_t>(npx, pix_offsets[g] + (int64_t)ny[g] * nx[g]);
        }
        if (star_offsets[0] != 0) throw ArgError{"star_offsets[0] must be 0"};
        for (int64_t g = 0; g < G; ++g)
            if (star_offsets[g + 1] < star_offsets[g]) throw ArgError{"star_offsets must be non-decreasing"};
        const int64_t ns = star_offsets[G];
        const size_t esz = eltype == CPB_F64 ? 8 : 4;
        cudaStream_t st = ctx->stream;
        auto up = [&](const char* name, const void* src, size_t bytes) -> void* {
            void* d = scratch(ctx, name, std::max<size_t>(bytes, 8));
            if (src && bytes) check(cudaMemcpyAsync(d, src, bytes, cudaMemcpyHostToDevice, st), "h2d batch input");
            return d;
        };
        const void* d_pix = up("gb_pix", pixels, esz * npx);
        const void* d_iv = inv_var ? up("gb_iv", inv_var, esz * npx) : nullptr;
        const void* d_bk = background ? up("gb_bkg", background, esz * npx) : nullptr;
        const int64_t* d_off = (const int64_t*)up("gb_off", pix_offsets, 8 * G);
        const int32_t* d_ny = (const int32_t*)up("gb_ny", ny, 4 * G);
        const int32_t* d_nx = (const int32_t*)up("gb_nx", nx, 4 * G);
        const int64_t* d_so = (const int64_t*)up("gb_soff", star_offsets, 8 * (G + 1));
        const double* d_y = (const double*)up("gb_y0", y0, 8 * ns);
        const double* d_x = (const double*)up("gb_x0", x0, 8 * ns);
        const double* d_f = (const double*)up("gb_f0", flux0, 8 * ns);
        // device outputs
        cpb_group_result d = *out;
        auto dout = [&](const char* name, void* host, size_t bytes) -> void* {
            return host ? scratch(ctx, name, std::max<size_t>(bytes, 8)) : nullptr;
        };
        d.y = (double*)dout("gb_o_y", out->y, 8 * ns);
        d.x = (double*)dout("gb_o_x", out->x, 8 * ns);
        d.flux = (double*)dout("gb_o_f", out->flux, 8 * ns);
        d.y_err = (double*)dout("gb_o_ey", out->y_err, 8 * ns);
        d.x_err = (double*)dout("gb_o_ex", out->x_err, 8 * ns);
        d.flux_err = (double*)dout("gb_o_ef", out->flux_err, 8 * ns);
        d.converged = (uint8_t*)dout("gb_o_cv", out->converged, ns);
        d.valid = (uint8_t*)dout("gb_o_va", out->valid, ns);
        d.n_iter = (int32_t*)dout("gb_o_it", out->n_iter, 4 * ns);
        d.chisq = (double*)dout("gb_o_chi", out->chisq, 8 * ns);
        d.qfit = (double*)dout("gb_o_q1", out->qfit, 8 * ns);
        d.qfit_expected = (double*)dout("gb_o_q2", out->qfit_expected, 8 * ns);
        d.qfit_z = (double*)dout("gb_o_q3", out->qfit_z, 8 * ns);
        d.crowding = (double*)dout("gb_o_cr", out->crowding, 8 * ns);
        d.spread_model = (double*)dout("gb_o_sm", out->spread_model, 8 * ns);
        d.spread_model_err = (double*)dout("gb_o_sme", out->spread_model_err, 8 * ns);
        d.residual = (double*)dout("gb_o_res", out->residual, 8 * npx);
        d.n_passes = (int32_t*)dout("gb_o_np", out->n_passes, 4 * G);
        d.n_failed = (int32_t*)dout("gb_o_nf", out->n_failed, 4 * G);
        d.status = (int32_t*)dout("gb_o_st", out->status, 4 * G);
        d.error_kind = (int32_t*)dout("gb_o_ek", out->error_kind, 4 * G);
        d.n_active = (int32_t*)dout("gb_o_na", out->n_active, 4 * G);
        d.n_union = (int32_t*)dout("gb_o_nu", out->n_union, 4 * G);
        d.n_trials = (int32_t*)dout("gb_o_nt", out->n_trials, 4 * G);
        d.n_lsqr_iters = (int32_t*)dout("gb_o_nl", out->n_lsqr_iters, 4 * G);
        fit_groups_dev(ctx, psf, params, G, d_off, d_ny, d_nx, d_pix, eltype, d_iv, d_bk, d_so, d_y, d_x, d_f, npx, &d,
                       pix_offsets, ny, nx, star_offsets);
        auto down = [&](void* host, const void* dev, size_t bytes) {
            if (host && bytes) check(cudaMemcpyAsync(host, dev, bytes, cudaMemcpyDeviceToHost, st), "d2h batch output");
        };
        down(out->y, d.y, 8 * ns);
        down(out->x, d.x, 8 * ns);
        down(out->flux, d.flux, 8 * ns);
        down(out->y_err, d.y_err, 8 * ns);
        down(out->x_err, d.x_err, 8 * ns);
        down(out->flux_err, d.flux_err, 8 * ns);
        down(out->converged, d.converged, ns);
        down(out->valid, d.valid, ns);
        down(out->n_iter, d.n_iter, 4 * ns);
        down(out->chisq, d.chisq, 8 * ns);
        down(out->qfit, d.qfit, 8 * ns);
        down(out->qfit_expected, d.qfit_expected, 8 * ns);
        down(out->qfit_z, d.qfit_z, 8 * ns);
        down(out->crowding, d.crowding, 8 * ns);
        down(out->spread_model, d.spread_model, 8 * ns);
        down(out->spread_model_err, d.spread_model_err, 8 * ns);
        down(out->residual, d.residual, 8 * npx);
        down(out->n_passes, d.n_passes, 4 * G);
        down(out->n_failed, d.n_failed, 4 * G);
        down(out->status, d.status, 4 * G);
        down(out->error_kind, d.error_kind, 4 * G);
        down(out->n_active, d.n_active, 4 * G);
        down(out->n_union, d.n_union, 4 * G);
        down(out->n_trials, d.n_trials, 4 * G);
        down(out->n_lsqr_iters, d.n_lsqr_iters, 4 * G);
        check(cudaStreamSynchronize(st), "sync");
        out->n_kernel_groups = d.n_kernel_groups;
        out->n_routed_groups = d.n_routed_groups;
        out->device_seconds = d.device_seconds;
        return CPB_OK;
    });
}

int cpb_fit_all_stars(cpb_ctx* ctx, const cpb_psf* psf, const cpb_lm_params* params, double fit_rad,
                      int32_t n_passes, double spread_model_fwhm, const void* image, int32_t eltype, int64_t ny,
                      int64_t nx, const void* inv_var, int64_t n, const double* init, cpb_multipass_result* out) {
    return guarded(ctx, [&]() -> int {
        if (!psf || !params || !out || !image || (n > 0 && !init)) throw ArgError{"null argument"};
        if (eltype != CPB_F32 && eltype != CPB_F64) throw ArgError{"unsupported image eltype"};
        if (ny <= 0 || nx <= 0) throw ArgError{"image must be non-empty"};
        const size_t bytes = (eltype == CPB_F64 ? 8 : 4) * (size_t)ny * (size_t)nx;
        void* d_img = scratch(ctx, "mp_in_image", bytes);
        void* d_iv = inv_var ? scratch(ctx, "mp_in_inv_var", bytes) : nullptr;
        const HostCopy in[2] = {{d_img, image, bytes}, {d_iv, inv_var, bytes}};
        host_to_device(ctx, in, 2);
        return fit_all_stars_dev(ctx, psf, params, fit_rad, n_passes, spread_model_fwhm, d_img, eltype, ny, nx, d_iv,
                                 n, init, out);
    });
}

int cpb_fit_lm_batch(cpb_ctx* ctx, const cpb_psf* psf, const cpb_lm_params* params, int64_t n_cutouts,
                     const int64_t* offsets, const int32_t* ny, const int32_t* nx, const int32_t* y_origin,
                     const int32_t* x_origin, const void* pixels, int32_t eltype, const void* inv_var,
                     const double* init, cpb_lm_result* out) {
    return guarded(ctx, [&]() -> int {
        if (!psf || !params || !out || (n_cutouts > 0 && (!offsets || !ny || !nx || !y_origin || !x_origin ||
                                                          !pixels || !init || !out->params || !out->iterations ||
                                                          !out->status)))
            throw ArgError{"null argument"};
        return fit_lm_batch(ctx, psf, params, n_cutouts, offsets, ny, nx, y_origin, x_origin, pixels, eltype, inv_var,
                            init, out);
    });
}

int cpb_fit_lm_batch_device(cpb_ctx* ctx, const cpb_psf* psf, const cpb_lm_params* params, int64_t n_cutouts,
                            const int64_t* d_offsets, const int32_t* d_ny, const int32_t* d_nx,
                            const int32_t* d_y_origin, const int32_t* d_x_origin, const void* d_pixels,
                            int32_t eltype, const void* d_inv_var, const double* d_init, int64_t total_pixels,
                            cpb_lm_result* out) {
    return guarded(ctx, [&]() -> int {
        if (!psf || !params || !out || (n_cutouts > 0 && (!d_offsets || !d_ny || !d_nx || !d_y_origin ||
                                                          !d_x_origin || !d_pixels || !d_init || !out->status)))
            throw ArgError{"null argument"};
        return fit_lm_batch_device(ctx, psf, params, n_cutouts, d_offsets, d_ny, d_nx, d_y_origin, d_x_origin,
                                   d_pixels, eltype, d_inv_var, d_init, total_pixels, out);
    });
}

}  // extern "C"
