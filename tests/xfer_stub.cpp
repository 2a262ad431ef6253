// The host transfer ring (csrc/host_xfer.cpp) against a stand-in for the part of
// the CUDA runtime that it calls, so that its paths run without a GPU: "device"
// memory is host memory and a copy is complete when the call returns.
//
//   xfer_stub MODE      exit status 0: as it should be
#include "../aocl-data-analytics_b200/csrc/host_xfer.hpp"
#include <cuda.h>
#include <atomic>
#include <chrono>
#include <csignal>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <sys/mman.h>
#include <sys/wait.h>
#include <thread>
#include <unistd.h>
#include <vector>

// ----------------------------------------------------------- the stand-in --
namespace {
std::mutex g_mu;
int g_ring_copies = 0; // copies issued by threads other than the caller's
int g_row_copies = 0;  // two-dimensional copies: the driver's row by row
int g_strays = 0;      // calls of theirs that name their own stream, not the caller's
std::thread::id g_main;
void note_thread(cudaStream_t s) {
    if (std::this_thread::get_id() != g_main) {
        std::lock_guard<std::mutex> lk(g_mu);
        ++g_ring_copies;
        if (s == cudaStreamPerThread) ++g_strays;
    }
}

// contexts: the primary one of device 0 (its id changes when it is reset) and one
// that a program makes by itself; page-locked memory and events belong to the
// context that they are made in
std::atomic<unsigned long long> g_primary{1};
std::atomic<int> g_active{1};
thread_local int t_ctx = 0; // 0: primary, 1: the program's own
unsigned long long ctx_id() { return t_ctx ? 77 : g_primary.load(); }
struct Locked {
    size_t n;
    unsigned long long ctx;
};
std::map<void *, Locked> g_locked;
std::map<cudaEvent_t, unsigned long long> g_events;
// a thread of the program's captures a graph in the global mode, which calls that
// page-lock or free memory in any thread end unless that thread's mode is relaxed
std::atomic<bool> g_capture{false};
std::atomic<int> g_spoilt{0};
thread_local cudaStreamCaptureMode t_mode = cudaStreamCaptureModeGlobal;
void unsafe_call() {
    if (g_capture && t_mode != cudaStreamCaptureModeRelaxed) ++g_spoilt;
}
int g_bad = 0; // uses of memory or events of another context, or of none
std::atomic<int> g_freed{0};
void use_event(cudaEvent_t e) {
    std::lock_guard<std::mutex> lk(g_mu);
    if (!g_events.count(e) || g_events[e] != ctx_id()) ++g_bad;
}
void use_memory(const void *p) { // a slot that is gone faults by itself
    std::lock_guard<std::mutex> lk(g_mu);
    auto it = g_locked.upper_bound(const_cast<void *>(p));
    if (it == g_locked.begin()) return;
    --it;
    if ((const char *)p < (const char *)it->first + it->second.n && it->second.ctx != ctx_id())
        ++g_bad;
}
// cudaDeviceReset: page-locked memory is unmapped, events are gone
void reset(bool again) {
    std::lock_guard<std::mutex> lk(g_mu);
    for (auto it = g_locked.begin(); it != g_locked.end();)
        if (it->second.ctx == g_primary) {
            mprotect(it->first, it->second.n, PROT_NONE);
            it = g_locked.erase(it);
        } else {
            ++it;
        }
    for (auto it = g_events.begin(); it != g_events.end();)
        it = it->second == g_primary ? g_events.erase(it) : std::next(it);
    ++g_primary;
    g_active = again;
}
CUresult ctx_get_current(CUcontext *c) {
    *c = reinterpret_cast<CUcontext>(t_ctx ? 0x200 : 0x100);
    return CUDA_SUCCESS;
}
CUresult ctx_get_id(CUcontext c, unsigned long long *id) {
    *id = c == reinterpret_cast<CUcontext>(0x200) ? 77 : g_primary.load();
    return CUDA_SUCCESS;
}
CUresult primary_state(CUdevice, unsigned *flags, int *active) {
    *flags = 0;
    *active = g_active;
    return CUDA_SUCCESS;
}
CUresult primary_retain(CUcontext *c, CUdevice) {
    *c = reinterpret_cast<CUcontext>(0x100);
    return CUDA_SUCCESS;
}
CUresult primary_release(CUdevice) { return CUDA_SUCCESS; }
} // namespace

extern "C" {
cudaError_t cudaGetDriverEntryPoint(const char *name, void **p, unsigned long long,
                                    cudaDriverEntryPointQueryResult *q) {
    const std::string n = name;
    *p = n == "cuCtxGetCurrent"              ? (void *)ctx_get_current
         : n == "cuCtxGetId"                 ? (void *)ctx_get_id
         : n == "cuDevicePrimaryCtxGetState" ? (void *)primary_state
         : n == "cuDevicePrimaryCtxRetain"   ? (void *)primary_retain
         : n == "cuDevicePrimaryCtxRelease"  ? (void *)primary_release
                                             : nullptr;
    *q = *p ? cudaDriverEntryPointSuccess : cudaDriverEntryPointSymbolNotFound;
    return cudaSuccess;
}
cudaError_t cudaThreadExchangeStreamCaptureMode(cudaStreamCaptureMode *m) {
    std::swap(*m, t_mode);
    return cudaSuccess;
}
cudaError_t cudaMallocHost(void **p, size_t n) {
    unsafe_call();
    *p = mmap(nullptr, n, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
    std::lock_guard<std::mutex> lk(g_mu);
    g_locked[*p] = {n, ctx_id()};
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void *p) {
    unsafe_call();
    std::lock_guard<std::mutex> lk(g_mu);
    if (!g_locked.count(p)) {
        ++g_bad;
        return cudaErrorInvalidValue;
    }
    munmap(p, g_locked[p].n);
    g_locked.erase(p);
    ++g_freed;
    return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) {
    static uintptr_t next = 0x5000;
    std::lock_guard<std::mutex> lk(g_mu);
    *e = reinterpret_cast<cudaEvent_t>(next += 16);
    g_events[*e] = ctx_id();
    return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t e) {
    use_event(e);
    std::lock_guard<std::mutex> lk(g_mu);
    g_events.erase(e);
    return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e) {
    use_event(e);
    return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t) {
    use_event(e);
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *to, const void *from, size_t n, cudaMemcpyKind, cudaStream_t s) {
    note_thread(s);
    use_memory(to);
    use_memory(from);
    std::memcpy(to, from, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpy2DAsync(void *to, size_t tp, const void *from, size_t fp, size_t w, size_t h,
                              cudaMemcpyKind, cudaStream_t) {
    ++g_row_copies;
    for (size_t r = 0; r < h; ++r) std::memcpy((char *)to + r * tp, (const char *)from + r * fp, w);
    return cudaSuccess;
}
cudaError_t cudaMemset2DAsync(void *p, size_t pitch, int v, size_t w, size_t h, cudaStream_t) {
    for (size_t r = 0; r < h; ++r) std::memset((char *)p + r * pitch, v, w);
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus *s) {
    *s = cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
cudaError_t cudaGetDevice(int *d) {
    *d = 0;
    return cudaSuccess;
}
cudaError_t cudaSetDevice(int) {
    t_ctx = 0;
    g_active = 1;
    return cudaSuccess;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *) {
    std::memset(a, 0, sizeof *a);
    a->type = cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
} // extern "C"

// ---------------------------------------------------------------- checks --
using namespace b200;
namespace {
#define CHECK(c)                                                                              \
    do {                                                                                      \
        if (!(c)) {                                                                           \
            std::fprintf(stderr, "line %d: %s\n", __LINE__, #c);                              \
            std::exit(1);                                                                     \
        }                                                                                     \
    } while (0)

cudaStream_t const S = reinterpret_cast<cudaStream_t>(0x1000);

// bytes copied through the driver's path until the ring takes a copy
bool warm(cudaStream_t s = S) {
    std::vector<char> host(8 << 20, 1), dev(8 << 20);
    for (int i = 0; i < 20; ++i) {
        const XferSeg g{host.data(), host.size(), dev.data(), host.size(), host.size(), 1};
        cudaError_t e = cudaSuccess;
        if (xfer_up(&g, 1, s, e)) return true;
    }
    return false;
}

// rows of w bytes, pitched on either side, up and down again: the rows arrive,
// the device rows' pads are zero, the host's bytes between rows stay
void round_trip(size_t rows, size_t w, size_t host_pitch, size_t dev_pitch, int times) {
    std::vector<unsigned char> from(rows * host_pitch), dev(rows * dev_pitch + 64, 0xFF),
        to(rows * host_pitch, 0xAA);
    for (size_t i = 0; i < from.size(); ++i) from[i] = (unsigned char)(i * 31 + i / 251 + 1);
    for (int t = 0; t < times; ++t) {
        std::fill(dev.begin(), dev.end(), 0xFF);
        CHECK(copy_up({from.data(), host_pitch, dev.data(), dev_pitch, w, rows}, S) == cudaSuccess);
        for (size_t r = 0; r < rows; ++r) {
            CHECK(std::memcmp(&dev[r * dev_pitch], &from[r * host_pitch], w) == 0);
            for (size_t c = w; c < dev_pitch; ++c) CHECK(dev[r * dev_pitch + c] == 0);
        }
        for (int i = 0; i < 64; ++i) CHECK(dev[rows * dev_pitch + i] == 0xFF);
        std::fill(to.begin(), to.end(), 0xAA);
        CHECK(copy_down({to.data(), host_pitch, dev.data(), dev_pitch, w, rows}, S) == cudaSuccess);
        for (size_t r = 0; r < rows; ++r) {
            CHECK(std::memcmp(&to[r * host_pitch], &from[r * host_pitch], w) == 0);
            for (size_t c = w; c < host_pitch; ++c) CHECK(to[r * host_pitch + c] == 0xAA);
        }
    }
}

int copies() {
    for (int pass = 0; pass < 2; ++pass) { // without the ring, then with it
        round_trip(1, 12, 12, 16, 1);
        round_trip(1, 3 << 20, 3 << 20, (3 << 20) + 12, 1); // one padded row of many pieces
        round_trip(1, (512 * 1024) * 5 - 8, (512 * 1024) * 5 - 8, 512 * 1024 * 5, 1);
        round_trip(1, 512 * 1024 * 5, 512 * 1024 * 5, 512 * 1024 * 5 + 16, 1); // a piece of pad alone
        round_trip(5, 600'004, 600'004, 600'016, 1);                         // rows over a slot
        round_trip(30'000, 148, 148, 160, 1);
        round_trip(30'000, 148, 152, 160, 1);
        round_trip(30'001, 96, 96, 96, 1);
        round_trip(30'001, 96, 100, 96, 1);
        if (pass == 0) CHECK(warm());
    }
    CHECK(g_ring_copies > 0);
    return 0;
}

// Results that are dense on the device come down in runs, whatever the caller's row
// pitch, with the ring and without.
int pitched_results() {
    for (int pass = 0; pass < 2; ++pass) {
        for (size_t rows : {1, 17, 2000, 30'001, 120'000})
            for (size_t pitch : {256, 268}) {
                std::vector<unsigned char> dev(rows * 256), to(rows * pitch, 0xAA);
                for (size_t i = 0; i < dev.size(); ++i) dev[i] = (unsigned char)(i * 31 + i / 251);
                CHECK(copy_down({to.data(), pitch, dev.data(), 256, 256, rows}, S) == cudaSuccess);
                for (size_t r = 0; r < rows; ++r) {
                    CHECK(std::memcmp(&to[r * pitch], &dev[r * 256], 256) == 0);
                    for (size_t c = 256; c < pitch; ++c) CHECK(to[r * pitch + c] == 0xAA);
                }
            }
        if (pass == 0) CHECK(warm());
    }
    CHECK(g_row_copies == 0);
    return 0;
}

// cudaStreamPerThread names another stream in every thread: all of a copy's
// pieces have to be the caller's
int per_thread() {
    CHECK(warm());
    const size_t w = 8 << 20;
    std::vector<char> from(w, 7), dev(w), to(w);
    CHECK(copy_up({from.data(), w, dev.data(), w, w, 1}, cudaStreamPerThread) == cudaSuccess);
    CHECK(copy_down({to.data(), w, dev.data(), w, w, 1}, cudaStreamPerThread) == cudaSuccess);
    CHECK(to == from);
    CHECK(g_strays == 0);
    const int before = g_ring_copies;
    CHECK(copy_up({from.data(), w, dev.data(), w, w, 1}, S) == cudaSuccess);
    CHECK(g_ring_copies > before); // other streams: as before
    return 0;
}

// Ends by exit() in a child forked while the ring's threads wait, and copies the
// driver's way there; then the parent's ring goes on.
int forked(int idle) {
    CHECK(warm());
    std::this_thread::sleep_for(std::chrono::milliseconds(idle));
    const pid_t child = fork();
    if (child == 0) {
        const size_t w = 8 << 20;
        std::vector<char> from(w, 5), dev(w);
        for (int i = 0; i < 20; ++i) {
            const XferSeg g{from.data(), w, dev.data(), w, w, 1};
            cudaError_t e = cudaSuccess;
            if (xfer_up(&g, 1, S, e)) _exit(3);
        }
        std::exit(0);
    }
    int status = -1;
    for (int i = 0; i < 100 && waitpid(child, &status, WNOHANG) == 0; ++i)
        std::this_thread::sleep_for(std::chrono::milliseconds(50));
    if (!WIFEXITED(status)) kill(child, SIGKILL);
    CHECK(WIFEXITED(status) && WEXITSTATUS(status) == 0);
    round_trip(30'000, 148, 148, 160, 1);
    CHECK(warm());
    return 0;
}

// A reset of the device takes the slots and events; a context of the program's own
// has none.
int contexts() {
    CHECK(warm());
    reset(true);
    round_trip(30'000, 148, 148, 160, 2);
    CHECK(g_bad == 0);
    CHECK(warm()); // a ring in the new context
    t_ctx = 1;
    const int before = g_ring_copies;
    round_trip(30'000, 148, 148, 160, 1);
    CHECK(g_ring_copies == before);
    CHECK(!warm()); // none is set up there either
    t_ctx = 0;
    round_trip(30'000, 148, 148, 160, 1);
    CHECK(g_ring_copies > before); // the primary's is still there
    CHECK(g_bad == 0);
    return 0;
}
// The same with the ring's context gone when it is given back: nothing is made
// again for it, and the program ends.
int reset_idle() {
    CHECK(warm());
    reset(false);
    std::this_thread::sleep_for(std::chrono::milliseconds(2500));
    CHECK(g_bad == 0 && g_freed == 0 && g_active == 0);
    g_active = 1;
    CHECK(warm());
    std::this_thread::sleep_for(std::chrono::milliseconds(2500));
    CHECK(g_freed == 1);
    CHECK(warm());
    reset(true);
    return 0;
}

// The ring is set up, given back and set up again while another thread captures.
int capture() {
    g_capture = true;
    CHECK(warm());
    CHECK(t_mode == cudaStreamCaptureModeGlobal); // the caller's mode is its own again
    std::this_thread::sleep_for(std::chrono::milliseconds(2500));
    CHECK(g_freed == 1);
    CHECK(warm());
    CHECK(g_spoilt == 0);
    return 0;
}
} // namespace

int main(int argc, char **argv) {
    g_main = std::this_thread::get_id();
    const char *m = argc > 1 ? argv[1] : "";
    if (!std::strcmp(m, "copies")) return copies();
    if (!std::strcmp(m, "per_thread")) return per_thread();
    if (!std::strcmp(m, "fork")) return forked(50);
    if (!std::strcmp(m, "fork_idle")) return forked(2500);
    if (!std::strcmp(m, "contexts")) return contexts();
    if (!std::strcmp(m, "reset_idle")) return reset_idle();
    if (!std::strcmp(m, "capture")) return capture();
    if (!std::strcmp(m, "pitched_results")) return pitched_results();
    return 2;
}
