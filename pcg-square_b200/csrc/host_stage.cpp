// Transfers between pageable host buffers and the device for the entry points
// that take and return host arrays.
//
// cudaMemcpyAsync on pageable memory stages each array on its own through the
// driver's pinned buffers, with one host thread that also takes the page
// faults of a fresh output buffer.  Here small sets of arrays are gathered into
// one copy through a pinned buffer of the device (an expansion of 2^16 through
// the host API: 541 -> 421 us), and large ones are moved in chunks by helper
// threads, which touch their part of a destination while the kernels run.
//
// The buffer is bounded (kStageBytes), is released by pcgb_trim_pool, and is
// used by one call at a time; a call that finds it taken (another host
// thread) copies straight from and to its own memory.
#include "pcgb_internal.h"

#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <cstring>
#include <memory>
#include <mutex>
#include <thread>

namespace pcgb {
namespace {

constexpr size_t kStageBytes = size_t{32} << 20;
constexpr size_t kChunk = size_t{1} << 20;
constexpr int kChunks = static_cast<int>(kStageBytes / kChunk);
constexpr size_t kPage = 4096;
// Ranges up to kSmall are staged by this thread alone: one copy instead of one
// per array.  From kLarge on helper threads pay for their start (a product with
// 3 x 16 MB: 2.9 -> 2.6 ms; 3 x 32 MB: 12.9 -> 5.9 ms).  Between the two the
// driver's own staging is as good.
constexpr size_t kSmall = size_t{4} << 20, kLarge = size_t{16} << 20;

struct Stage {
    std::mutex mu;
    char* pinned = nullptr;
    size_t bytes = 0;
    cudaEvent_t ev[kChunks] = {};
};

Stage& stage_for_device(int* dev_out) {
    static Stage stages[64];
    int dev = 0;
    check_cuda(cudaGetDevice(&dev), "cudaGetDevice");
    if (dev < 0 || dev >= 64) fail(PCGB_EINVAL, "device index out of range");
    if (dev_out) *dev_out = dev;
    return stages[dev];
}

bool is_pinned(const void* p) {
    cudaPointerAttributes a = {};
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return a.type != cudaMemoryTypeUnregistered;
}

constexpr int kHelpers = 4;

inline void pause() {
#if defined(__x86_64__)
    __builtin_ia32_pause();
#endif
}

// Up to kHelpers threads running f(), joined on destruction; fewer (count)
// where the system gives fewer.  The threads call the caller's own f, which is
// declared before them and so outlives them: a temporary does not bind.
struct Helpers {
    std::thread th[kHelpers];
    int count = 0;
    template <class F>
    Helpers(int want, F& f) {
        try {
            for (; count < want; ++count) th[count] = std::thread([&f] { f(); });
        } catch (...) {   // no thread or no memory for one: those that run are enough
        }
    }
    ~Helpers() {
        for (int i = 0; i < count; ++i) th[i].join();
    }
};

// f(c) for every chunk c < n, on helpers when the whole range is large.
template <class F>
void each_chunk(int n, size_t bytes, const F& f) {
    std::atomic<int> next{0};
    auto share = [&] {
        for (int c; (c = next.fetch_add(1, std::memory_order_relaxed)) < n;) f(c);
    };
    Helpers h(bytes >= kLarge ? std::min(kHelpers, n) : 0, share);
    if (h.count == 0) share();
}

// Chunks announced by the one thread that waits on the driver.  The others
// look a few microseconds (chunks of a running copy are 20 us apart), then
// sleep: the first chunk comes only after the call's kernels, 15 ms for an
// expansion of 2^20.
class Progress {
  public:
    // Chunks [0, r) are there; r < 0: no more will come.
    void announce(int r) {
        {
            std::lock_guard<std::mutex> lk(mu);
            ready.store(r, std::memory_order_release);
        }
        cv.notify_all();
    }
    // Whether chunk c is there, waiting for it or for the end.
    bool wait(int c) {
        for (int k = 0; k < kLooks; ++k) {
            const int r = ready.load(std::memory_order_acquire);
            if (r > c || r < 0) return r > c;
            pause();
        }
        std::unique_lock<std::mutex> lk(mu);
        cv.wait(lk, [&] { return ready.load() > c || ready.load() < 0; });
        return ready.load() > c;
    }

  private:
    static constexpr int kLooks = 1000;
    std::mutex mu;
    std::condition_variable cv;
    std::atomic<int> ready{0};
};

}  // namespace

struct HostStage::Impl {
    Stage* s;
    int dev;
    std::unique_lock<std::mutex> lk;
};

HostStage::HostStage() {
    auto p = std::make_unique<Impl>();
    p->s = &stage_for_device(&p->dev);
    p->lk = std::unique_lock<std::mutex>(p->s->mu, std::try_to_lock);
    usable = p->lk.owns_lock();
    im = p.release();
}

// Makes the buffer hold a transfer of `total` bytes (kSmall, or kStageBytes
// for the large ones: 32 MB of pinned memory take 13 ms to get, 4 MB 2).
bool HostStage::reserve(size_t total) {
    if (!usable || (total > kSmall && total < kLarge)) return false;
    Stage& s = *im->s;
    const size_t want = total <= kSmall ? kSmall : kStageBytes;
    if (s.bytes >= want) return true;
    if (pending) check_cuda(cudaStreamSynchronize(pending), "host copy");
    pending = nullptr;
    used = 0;
    if (s.pinned) cudaFreeHost(s.pinned);
    s.pinned = nullptr;
    s.bytes = 0;
    bool ok = true;
    for (auto& e : s.ev)
        if (!e && cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess) {
            e = nullptr;
            ok = false;
        }
    if (!ok || cudaMallocHost(&s.pinned, want) != cudaSuccess) {
        cudaGetLastError();
        s.pinned = nullptr;
        usable = false;
        return false;
    }
    s.bytes = want;
    return true;
}

HostStage::~HostStage() {
    // A call that failed half way; its own error is the one reported.
    if (pending && cudaStreamSynchronize(pending) != cudaSuccess) cudaGetLastError();
    delete im;
}

void HostStage::trim() {
    Stage& s = stage_for_device(nullptr);
    std::lock_guard<std::mutex> lk(s.mu);
    if (s.pinned) cudaFreeHost(s.pinned);
    s.pinned = nullptr;
    s.bytes = 0;
}

namespace {

// Calls f(pointer, offset from `a`, bytes) for the parts of bytes [a, b) of the
// concatenated pieces.
template <class Ptr, class F>
void parts_of(Ptr const* piece, const size_t* len, int pieces, size_t a, size_t b, const F& f) {
    size_t o = 0;
    for (int i = 0; i < pieces; ++i) {
        const size_t lo = std::max(a, o), hi = std::min(b, o + len[i]);
        if (lo < hi) f(i, lo - o, lo - a, hi - lo);
        o += len[i];
    }
}

}  // namespace

void HostStage::upload(void* d_dst, const void* const* src, const size_t* len, int pieces,
                       cudaStream_t st) {
    size_t total = 0;
    bool direct = false;
    for (int i = 0; i < pieces; ++i) {
        total += len[i];
        direct = direct || (len[i] && is_pinned(src[i]));
    }
    direct = direct || !reserve(total);
    if (direct) {
        if (pending && pending != st) check_cuda(cudaStreamSynchronize(pending), "host upload");
        pending = st;   // pinned sources are read until the stream gets there
        size_t o = 0;
        for (int i = 0; i < pieces; ++i) {
            check_cuda(cudaMemcpyAsync(static_cast<char*>(d_dst) + o, src[i], len[i],
                                       cudaMemcpyHostToDevice, st), "host upload");
            o += len[i];
        }
        return;
    }
    Stage& s = *im->s;
    for (size_t at = 0; at < total;) {
        if (used == s.bytes) {   // earlier copies still read the buffer
            check_cuda(cudaStreamSynchronize(pending), "host upload");
            used = 0;
        }
        const size_t round = std::min(s.bytes - used, total - at);
        const int n = static_cast<int>((round + kChunk - 1) / kChunk);
        char* base = s.pinned + used;
        pending = st;
        std::atomic<int> bad{0};
        each_chunk(n, total, [&](int c) {
            const size_t o = static_cast<size_t>(c) * kChunk, l = std::min(kChunk, round - o);
            parts_of(src, len, pieces, at + o, at + o + l,
                     [&](int i, size_t in, size_t from, size_t m) {
                         std::memcpy(base + o + from, static_cast<const char*>(src[i]) + in, m);
                     });
            cudaError_t e = cudaSetDevice(im->dev);
            if (e == cudaSuccess)
                e = cudaMemcpyAsync(static_cast<char*>(d_dst) + at + o, base + o, l,
                                    cudaMemcpyHostToDevice, st);
            if (e != cudaSuccess) bad = static_cast<int>(e);
        });
        if (bad) check_cuda(static_cast<cudaError_t>(bad.load()), "host upload");
        at += round;
        used = std::min(s.bytes, (used + round + 255) & ~size_t{255});
    }
}

void HostStage::download(void* const* dst, const size_t* len, int pieces, const void* d_src,
                         cudaStream_t st) {
    size_t total = 0;
    bool direct = false;
    for (int i = 0; i < pieces; ++i) {
        total += len[i];
        direct = direct || (len[i] && is_pinned(dst[i]));
    }
    direct = direct || !reserve(total);
    if (pending && pending != st) check_cuda(cudaStreamSynchronize(pending), "host download");
    pending = st;   // until the end: a failure leaves copies queued
    if (direct) {
        size_t o = 0;
        for (int i = 0; i < pieces; ++i) {
            check_cuda(cudaMemcpyAsync(dst[i], static_cast<const char*>(d_src) + o, len[i],
                                       cudaMemcpyDeviceToHost, st), "host download");
            o += len[i];
        }
        check_cuda(cudaStreamSynchronize(st), "host download");
        pending = nullptr;
        used = 0;
        return;
    }
    Stage& s = *im->s;
    for (size_t at = 0; at < total; at += s.bytes) {
        const size_t round = std::min(s.bytes, total - at);
        const int n = static_cast<int>((round + kChunk - 1) / kChunk);
        for (int c = 0; c < n; ++c) {
            const size_t o = static_cast<size_t>(c) * kChunk, l = std::min(kChunk, round - o);
            check_cuda(cudaMemcpyAsync(s.pinned + o, static_cast<const char*>(d_src) + at + o, l,
                                       cudaMemcpyDeviceToHost, st), "host download");
            check_cuda(cudaEventRecord(s.ev[c], st), "host download");
        }
        // Helpers take the page faults of their chunks while the device is at
        // work (a write that keeps the byte), then move each chunk as this thread,
        // which alone waits on the driver, announces it.
        Progress progress;
        auto touch = [&](int c) {
            const size_t o = static_cast<size_t>(c) * kChunk, l = std::min(kChunk, round - o);
            parts_of(dst, len, pieces, at + o, at + o + l, [&](int i, size_t in, size_t, size_t m) {
                char* p = static_cast<char*>(dst[i]) + in;
                for (size_t k = 0; k < m; k += kPage) __atomic_fetch_or(p + k, 0, __ATOMIC_RELAXED);
            });
        };
        auto move = [&](int c) {
            const size_t o = static_cast<size_t>(c) * kChunk, l = std::min(kChunk, round - o);
            parts_of(dst, len, pieces, at + o, at + o + l,
                     [&](int i, size_t in, size_t from, size_t m) {
                         std::memcpy(static_cast<char*>(dst[i]) + in, s.pinned + o + from, m);
                     });
        };
        std::atomic<int> next{0};
        auto share = [&] {
            static_assert(kChunks <= 32, "a bit per chunk");
            uint32_t mine = 0;   // a chunk is moved by the thread that touched it
            for (int c; (c = next.fetch_add(1, std::memory_order_relaxed)) < n;) {
                touch(c);
                mine |= uint32_t{1} << c;
            }
            for (int c = 0; c < n; ++c) {
                if (!(mine >> c & 1)) continue;
                if (!progress.wait(c)) return;
                move(c);
            }
        };
        cudaError_t err = cudaSuccess;
        {
            Helpers helpers(total >= kLarge ? std::min(kHelpers, n) : 0, share);
            if (helpers.count == 0)
                for (int c = 0; c < n; ++c) touch(c);
            for (int c = 0; c < n && err == cudaSuccess; ++c) {
                err = cudaEventSynchronize(s.ev[c]);
                progress.announce(err == cudaSuccess ? c + 1 : -1);
                if (helpers.count == 0 && err == cudaSuccess) move(c);
            }
        }
        check_cuda(err, "host download");
    }
    // The stream has passed every copy that used the buffer.
    pending = nullptr;
    used = 0;
}

}  // namespace pcgb
