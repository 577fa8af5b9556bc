// Runs host_stage.cpp against a CUDA runtime of plain host memory: streams
// complete at once, device pointers are host pointers.  Modes (argv[1]):
//   move MB    an upload and a download of MB megabytes in three pieces
//   threads MB  as move, where only N threads can be had, N = 0 .. 4
//   failed MB  transfers that fail half way leave nothing in flight
//   idle MB    processor time of a download whose first chunk comes after 300 ms
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <atomic>
#include <chrono>
#include <ctime>
#include <new>
#include <thread>
#include <vector>

#include "pcgb_internal.h"

namespace pcgb {
void fail(int code, const std::string& msg) { throw Error(code, msg); }
void check_cuda(cudaError_t e, const char* what) {
    if (e == cudaSuccess) return;
    cudaGetLastError();
    throw Error(PCGB_ECUDA, what);
}
}  // namespace pcgb

static std::atomic<int> event_delay_ms{0};   // of the next event wait
static std::atomic<int> events_left{-1};     // event waits until one fails; < 0: none does
static std::atomic<int> in_flight{0};        // copies the stream was not waited for since
static bool sync_fails = false;
static cudaError_t last_error = cudaSuccess;
static const void* pinned_at = nullptr;      // an address that counts as pinned memory
// Allocations until one throws (those of a transfer are its threads' states); < 0: none does.
static thread_local int allocations_left = -1;

void* operator new(std::size_t n) {
    if (allocations_left == 0) throw std::bad_alloc();
    if (allocations_left > 0) --allocations_left;
    if (void* p = std::malloc(n)) return p;
    throw std::bad_alloc();
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, std::size_t) noexcept { std::free(p); }

extern "C" {
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetLastError() {
    const cudaError_t e = last_error;
    last_error = cudaSuccess;
    return e;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {
    a->type = p == pinned_at ? cudaMemoryTypeHost : cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { *p = std::malloc(n); return cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { std::free(p); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
    std::memcpy(d, s, n);
    ++in_flight;
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) {
    in_flight = 0;
    return last_error = sync_fails ? cudaErrorStreamCaptureUnsupported : cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
    *e = reinterpret_cast<cudaEvent_t>(1);
    return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) {
    std::this_thread::sleep_for(std::chrono::milliseconds(event_delay_ms.exchange(0)));
    if (events_left == 0) return last_error = cudaErrorUnknown;
    if (events_left > 0) --events_left;
    return cudaSuccess;
}
}

namespace {

const cudaStream_t kStream = reinterpret_cast<cudaStream_t>(8);

// Three ragged pieces of `total` bytes and a "device" buffer of as many.
struct Arrays {
    std::vector<char> part[3], out[3], dev;
    size_t len[3];
    explicit Arrays(size_t total) : dev(total) {
        len[0] = total / 3 + 5;
        len[1] = total / 7;
        len[2] = total - len[0] - len[1];
        unsigned s = 12345;
        for (int i = 0; i < 3; ++i) {
            part[i].resize(len[i]);
            for (auto& c : part[i]) c = static_cast<char>((s = s * 1664525u + 1013904223u) >> 24);
            out[i].assign(len[i], 0x5a);
        }
    }
};

void expect(bool ok, const char* what) {
    if (ok) return;
    std::fprintf(stderr, "FAILED: %s\n", what);
    std::exit(1);
}

void move(Arrays& a) {
    const void* src[3];
    void* dst[3];
    for (int i = 0; i < 3; ++i) {
        src[i] = a.part[i].data();
        dst[i] = a.out[i].data();
    }
    pcgb::HostStage io;
    io.upload(a.dev.data(), src, a.len, 3, kStream);
    io.download(dst, a.len, 3, a.dev.data(), kStream);
}

int run_move(size_t mb) {
    Arrays a(mb << 20);
    move(a);
    for (int i = 0; i < 3; ++i) expect(a.out[i] == a.part[i], "bytes after the round trip");
    pcgb::HostStage::trim();
    return 0;
}

int run_threads(size_t mb) {
    for (int threads = 0; threads <= 4; ++threads) {
        Arrays a(mb << 20);
        const void* src[3];
        void* dst[3];
        for (int i = 0; i < 3; ++i) {
            src[i] = a.part[i].data();
            dst[i] = a.out[i].data();
        }
        pcgb::HostStage io;
        allocations_left = threads;
        io.upload(a.dev.data(), src, a.len, 3, kStream);
        allocations_left = threads;
        io.download(dst, a.len, 3, a.dev.data(), kStream);
        allocations_left = -1;
        for (int i = 0; i < 3; ++i) expect(a.out[i] == a.part[i], "bytes with fewer threads");
    }
    return 0;
}

int run_failed(size_t mb) {
    Arrays a(mb << 20);
    const void* src[3];
    void* dst[3];
    for (int i = 0; i < 3; ++i) {
        src[i] = a.part[i].data();
        dst[i] = a.out[i].data();
    }
    pinned_at = src[1];
    {
        pcgb::HostStage io;   // a call that fails between its upload and its download
        io.upload(a.dev.data(), src, a.len, 3, kStream);
        expect(in_flight > 0, "the upload is queued");
    }
    expect(in_flight == 0, "copies from pinned sources have ended");
    pinned_at = nullptr;
    for (int good = 0; good < 2; ++good) {
        bool thrown = false;
        try {
            pcgb::HostStage io;
            events_left = good;
            io.download(dst, a.len, 3, a.dev.data(), kStream);
        } catch (const pcgb::Error&) {
            thrown = true;
        }
        events_left = -1;
        expect(thrown, "the error is reported");
        expect(in_flight == 0, "copies into the buffer have ended");
        // Chunks that did not come leave their part of the outputs alone.
        size_t at = 0;
        for (int i = 0; i < 3; ++i)
            for (size_t k = 0; k < a.len[i]; ++k, ++at)
                expect(at < static_cast<size_t>(good) << 20 || a.out[i][k] == 0x5a,
                       "outputs a failed call does not reach");
    }
    // Nor an error for the next launch's check to find.
    try {
        pcgb::HostStage io;
        events_left = 0;
        sync_fails = true;
        io.download(dst, a.len, 3, a.dev.data(), kStream);
    } catch (const pcgb::Error&) {
    }
    events_left = -1;
    sync_fails = false;
    expect(cudaGetLastError() == cudaSuccess, "no error left behind");
    return 0;
}

// Four threads that wait by spinning would burn 1200 ms; touching and copying
// 16 MB takes 10 to 30.
int run_idle(size_t mb) {
    Arrays a(mb << 20);
    move(a);   // threads, pages and the buffer are warm
    event_delay_ms = 300;
    const std::clock_t t0 = std::clock();   // all threads of the process
    move(a);
    const double ms = 1e3 * static_cast<double>(std::clock() - t0) / CLOCKS_PER_SEC;
    std::fprintf(stderr, "%.1f ms of processor time\n", ms);
    expect(ms < 150, "helpers sleep while the device works");
    return 0;
}

}  // namespace

int main(int argc, char** argv) {
    const std::string mode = argc > 1 ? argv[1] : "";
    if (mode == "move" && argc > 2) return run_move(std::strtoul(argv[2], nullptr, 10));
    if (mode == "threads" && argc > 2) return run_threads(std::strtoul(argv[2], nullptr, 10));
    if (mode == "failed" && argc > 2) return run_failed(std::strtoul(argv[2], nullptr, 10));
    if (mode == "idle" && argc > 2) return run_idle(std::strtoul(argv[2], nullptr, 10));
    return 2;
}
