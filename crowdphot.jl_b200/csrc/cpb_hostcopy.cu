// cpb_hostcopy.cu -- large copies between pageable host memory and the device.
//
// A pageable cudaMemcpyAsync is staged by one driver thread: it moved the three
// 16.8 MB images of a 2048^2 field and the 33.5 MB residual (into memory the caller
// has not touched yet, so every page faults) at a few GB/s while the GPU waited.
// Here a few worker threads each own a stream and two pinned chunks and take the chunks of
// the job in turn: the host copies, the page faults and the DMA
// transfers run side by side (2048^2 field with residual, whole call: 44.4 -> 35.5 ms),
// and the residual leaves while the diagnostics run.  Memory the caller has pinned goes to the driver as
// before.  One copier per context, made at its first large pageable copy and given
// back with the context; kThreads * 2 chunks of pinned memory.  A process' copiers together
// have a worker a processor it may run on, each copier at least one.
#include <sched.h>
#include <stdlib.h>
#include <string.h>
#include <sys/mman.h>

#include <atomic>
#include <condition_variable>
#include <mutex>
#include <thread>
#include <vector>

#include "cpb_internal.cuh"

namespace cpb {

namespace {

constexpr int kThreads = 4;                 // at most
constexpr size_t kChunk = size_t(1) << 18;
// The pinned memory: one huge page, registered.  Making a copier falls into a context's first
// large request, and cudaMallocHost of 2 MB took 1.2-3.9 ms of it, registering a huge page
// 0.35 (2.2 where the host has none to give); the first pass of a new server of four slots
// 30.6 -> 26.5 ms (22.0 from then on).
constexpr size_t kPage = size_t(2) << 20;
static_assert(kThreads * 2 * kChunk <= kPage, "the workers' chunks");
// Below this the workers' wake-up and scheduling costs more than they save.  Whole calls on
// square fields, by workers and by the driver.  Up, three Float32 images read from memory (a
// new field each call) and from the processor's cache (the same one again):
//    3.2 MB 2.0 and 1.9 ms, 2.0 and 1.8;   8.4 MB 2.4 and 2.45, 2.4 and 2.1;
//   17.3 MB 3.2 and 3.5,    3.2 and 2.9;  27.0 MB 4.0 and 4.9,  4.1 and 3.9;
//   50.3 MB 5.0 and 6.7,    5.1 and 5.1.
// Down, the residual to memory not touched before (results are kept) and used again:
//    3.9 MB 2.3 and 3.7,    2.7 and 2.4;   8.4 MB 3.2 and 4.6,  3.6 and 3.3;
//   18.0 MB 5.7 and 8.3,    5.7 and 5.8;  23.1 MB 6.3 and 9.7,  6.9 and 7.1.
// Six served fields, two of them above the line: 21.9 ms, and 20.7 with every one below it,
// from the cache; 22.6 and 22.9 from memory.
constexpr size_t kMinBytes = size_t(8) << 20;

std::atomic<int> n_workers{0};  // of every copier

int processors() {
    cpu_set_t set;
    CPU_ZERO(&set);
    return sched_getaffinity(0, sizeof(set), &set) == 0 ? CPU_COUNT(&set) : 1;
}

bool pinned_host(const void* p) {
    cudaPointerAttributes a{};
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return a.type != cudaMemoryTypeUnregistered;
}

}  // namespace

class HostCopier {
  public:
    struct Part {
        char* dst;
        const char* src;
        size_t bytes;
    };

    explicit HostCopier(int device) : device_(device) {
        int others = n_workers.load();
        do {
            n_ = std::min(std::max(processors() - others, 1), kThreads);
        } while (!n_workers.compare_exchange_weak(others, others + n_));
        pin_ = (char*)aligned_alloc(kPage, kPage);
        if (pin_) {
            madvise(pin_, kPage, MADV_HUGEPAGE);
            memset(pin_, 0, (size_t)n_ * 2 * kChunk);
            registered_ = cudaHostRegister(pin_, (size_t)n_ * 2 * kChunk, cudaHostRegisterDefault) == cudaSuccess;
        }
        if (!registered_) {  // no room to lock it
            cudaGetLastError();
            free(pin_);
            pin_ = nullptr;
            if (cudaMallocHost((void**)&pin_, (size_t)n_ * 2 * kChunk) != cudaSuccess) ok_ = false;
        }
        for (int k = 0; k < n_; ++k) {
            Worker& w = w_[k];
            w.pin = pin_ + k * 2 * kChunk;
            if (cudaStreamCreateWithFlags(&w.stream, cudaStreamNonBlocking) != cudaSuccess) ok_ = false;
            for (auto& e : w.ev)
                if (cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess) ok_ = false;
        }
        if (cudaEventCreateWithFlags(&start_, cudaEventDisableTiming) != cudaSuccess) ok_ = false;
        if (!ok_) {
            cudaGetLastError();
            return;
        }
        try {
            for (int k = 0; k < n_; ++k) w_[k].th = std::thread([this, k] { loop(k); });
        } catch (...) {  // no threads to be had: the caller copies through the driver
            ok_ = false;
        }
    }

    ~HostCopier() {
        {
            std::lock_guard<std::mutex> lk(mu_);
            quit_ = true;
        }
        cv_.notify_all();
        for (auto& w : w_) {
            if (w.th.joinable()) w.th.join();
            for (auto& e : w.ev)
                if (e) cudaEventDestroy(e);
            if (w.stream) cudaStreamDestroy(w.stream);
        }
        if (registered_) {
            cudaHostUnregister(pin_);
            free(pin_);
        } else if (pin_) {
            cudaFreeHost(pin_);
        }
        if (start_) cudaEventDestroy(start_);
        n_workers -= n_;
    }

    bool ok() const { return ok_; }

    // Starts copying `parts` behind what `st` holds now; wait() ends it.
    void begin(std::vector<Part> parts, bool to_device, cudaStream_t st) {
        check(cudaEventRecord(start_, st), "event");
        {
            std::lock_guard<std::mutex> lk(mu_);
            parts_ = std::move(parts);
            to_device_ = to_device;
            err_ = cudaSuccess;
            running_ = n_;
            ++job_;
        }
        cv_.notify_all();
    }

    // Every byte has left (to_device) or reached the host memory; `st` (to_device)
    // continues behind the transfers.  Returns the first error.
    cudaError_t wait(cudaStream_t st) {
        std::unique_lock<std::mutex> lk(mu_);
        done_.wait(lk, [this] { return running_ == 0; });
        cudaError_t e = err_;
        if (to_device_)
            for (int k = 0; k < n_; ++k)
                for (auto& ev : w_[k].ev)
                    if (e == cudaSuccess) e = cudaStreamWaitEvent(st, ev, 0);
        return e;
    }

  private:
    struct Worker {
        std::thread th;
        cudaStream_t stream = nullptr;
        cudaEvent_t ev[2] = {};
        char* pin = nullptr;
        unsigned n = 0;  // chunks so far: chunk n uses half n & 1
    };

    void loop(int k) {
        cudaSetDevice(device_);
        unsigned seen = 0;
        for (;;) {
            {
                std::unique_lock<std::mutex> lk(mu_);
                cv_.wait(lk, [&] { return quit_ || job_ != seen; });
                if (quit_) return;
                seen = job_;
            }
            const cudaError_t e = copy(k);
            {
                std::lock_guard<std::mutex> lk(mu_);
                if (e != cudaSuccess && err_ == cudaSuccess) err_ = e;
                if (--running_ == 0) done_.notify_all();
            }
        }
    }

    cudaError_t copy(int k) {
        Worker& w = w_[k];
#define CPB_TRY(x)                                  \
    do {                                            \
        const cudaError_t e_ = (x);                 \
        if (e_ != cudaSuccess) return e_;           \
    } while (0)
        CPB_TRY(cudaStreamWaitEvent(w.stream, start_, 0));
        size_t c = 0;  // running chunk number over all parts
        char* pend_dst = nullptr;  // D2H: the transfer whose host copy is due
        size_t pend_n = 0;
        int pend_half = 0;
        auto drain = [&]() -> cudaError_t {
            if (!pend_dst) return cudaSuccess;
            const cudaError_t e = cudaEventSynchronize(w.ev[pend_half]);
            if (e == cudaSuccess) memcpy(pend_dst, w.pin + pend_half * kChunk, pend_n);
            pend_dst = nullptr;
            return e;
        };
        for (const Part& p : parts_)
            for (size_t at = 0; at < p.bytes; at += kChunk, ++c) {
                if (c % (size_t)n_ != (size_t)k) continue;
                const size_t n = p.bytes - at < kChunk ? p.bytes - at : kChunk;
                const int half = (int)(w.n++ & 1);
                char* pin = w.pin + half * kChunk;
                if (to_device_) {
                    CPB_TRY(cudaEventSynchronize(w.ev[half]));  // the half's previous transfer
                    memcpy(pin, p.src + at, n);
                    CPB_TRY(cudaMemcpyAsync(p.dst + at, pin, n, cudaMemcpyHostToDevice, w.stream));
                    CPB_TRY(cudaEventRecord(w.ev[half], w.stream));
                } else {
                    CPB_TRY(cudaMemcpyAsync(pin, p.src + at, n, cudaMemcpyDeviceToHost, w.stream));
                    CPB_TRY(cudaEventRecord(w.ev[half], w.stream));
                    CPB_TRY(drain());  // the other half, while this one is in flight
                    pend_dst = p.dst + at;
                    pend_n = n;
                    pend_half = half;
                }
            }
        return drain();
#undef CPB_TRY
    }

    int device_;
    bool ok_ = true, registered_ = false;
    int n_ = 0;  // workers
    char* pin_ = nullptr;
    Worker w_[kThreads];
    cudaEvent_t start_ = nullptr;
    std::mutex mu_;
    std::condition_variable cv_, done_;
    std::vector<Part> parts_;
    bool to_device_ = false, quit_ = false;
    cudaError_t err_ = cudaSuccess;
    int running_ = 0;
    unsigned job_ = 0;
};

void HostCopierDelete::operator()(HostCopier* p) const { delete p; }

namespace {

// The context's copier, or null where the driver copies: small or pinned memory,
// the allocation-free entry point, no workers to be had.
HostCopier* copier_for(cpb_ctx* ctx, size_t bytes, const void* host) {
    if (bytes < kMinBytes || ctx->arena || pinned_host(host)) return nullptr;
    if (!ctx->copier) ctx->copier.reset(new HostCopier(ctx->device));
    return ctx->copier->ok() ? ctx->copier.get() : nullptr;
}

}  // namespace

void host_to_device(cpb_ctx* ctx, const HostCopy* parts, int n) {
    std::vector<HostCopier::Part> big;
    size_t bytes = 0;
    for (int k = 0; k < n; ++k)
        if (parts[k].host) bytes += parts[k].bytes;
    HostCopier* c = nullptr;
    for (int k = 0; k < n; ++k) {
        const HostCopy& p = parts[k];
        if (!p.host || !p.bytes) continue;
        HostCopier* q = copier_for(ctx, bytes, p.host);
        if (q) {
            c = q;
            big.push_back({(char*)p.device, (const char*)p.host, p.bytes});
        } else {
            check(cudaMemcpyAsync(p.device, p.host, p.bytes, cudaMemcpyHostToDevice, ctx->stream), "h2d");
        }
    }
    if (!c) return;
    c->begin(std::move(big), true, ctx->stream);
    check(c->wait(ctx->stream), "h2d");
}

DeviceToHost::DeviceToHost(cpb_ctx* ctx, void* host, const void* device, size_t bytes) : ctx_(ctx) {
    if (!host || !bytes) return;
    HostCopier* c = copier_for(ctx, bytes, host);
    if (!c) {
        host_ = host;
        device_ = device;
        bytes_ = bytes;
        return;
    }
    c->begin({{(char*)host, (const char*)device, bytes}}, false, ctx->stream);
    copier_ = c;
}

void DeviceToHost::finish() {
    if (copier_) {
        HostCopier* c = copier_;
        copier_ = nullptr;
        check(c->wait(ctx_->stream), "d2h");
    } else if (host_) {
        check(cudaMemcpyAsync(host_, device_, bytes_, cudaMemcpyDeviceToHost, ctx_->stream), "d2h");
        host_ = nullptr;
    }
}

DeviceToHost::~DeviceToHost() {
    if (copier_) copier_->wait(ctx_->stream);
}

}  // namespace cpb
