// The pinned ring of host_xfer.hpp.  One per process, for the first device that
// uses it, in the runtime's (primary) context of that device: 8 MB of pinned
// memory and its threads, set up once XFER_AFTER bytes
// have gone the driver's way (page-locking takes 7 ms: a program that moves
// little never pays it) and given back after XFER_IDLE seconds without a copy.
// A copy holds the ring alone; a second thread's copy meanwhile goes the
// driver's way.
#include "host_xfer.hpp"
#include "cuda_context.hpp"
#include <algorithm>
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <cstdint>
#include <cstring>
#if defined(__SSE2__)
#include <emmintrin.h>
#endif
#include <memory>
#include <mutex>
#include <new>
#include <thread>
#include <unistd.h>
#include <vector>

namespace b200 {

namespace {

constexpr size_t XFER_SLOT = 512 * 1024;   // bytes per slot, two slots a thread
constexpr size_t XFER_MIN = 2 << 20;       // smaller copies: the driver is as fast
constexpr size_t XFER_AFTER = 64u << 20;   // bytes before the ring is set up
constexpr int XFER_THREADS = 8;            // with the caller's, at most
#ifndef XFER_IDLE_SECONDS // (a test's build sets fewer)
#define XFER_IDLE_SECONDS 20
#endif
constexpr int XFER_IDLE = XFER_IDLE_SECONDS;

struct Job {
    const XferSeg *segs = nullptr;
    std::vector<size_t> first; // of each segment, and the number of pieces
    bool up = false;
    int device = 0;
    cudaStream_t s = nullptr;
    std::atomic<size_t> next{0};
    std::atomic<int> error{0};
};

// A piece of a segment: rows r .. r + n - 1, or (n = 0) bytes of row r, the last
// `pad` of them past the row (zeros, going up).
struct Piece {
    size_t r, n, off, bytes, pad;
};
// One run of bytes on both sides.  Going up, a single row that is padded on the
// device is not: its pad is written too.
bool flat(const XferSeg &g, bool up) {
    return (g.rows == 1 && !(up && g.dev_pitch > g.row_bytes)) ||
           (g.host_pitch == g.row_bytes && g.dev_pitch == g.row_bytes);
}
// bytes that one row takes on the device
size_t row_span(const XferSeg &g, bool up) { return up ? g.dev_pitch : g.row_bytes; }
size_t pieces(const XferSeg &g, bool up) {
    if (flat(g, up)) return (g.rows * g.row_bytes + XFER_SLOT - 1) / XFER_SLOT;
    if (g.dev_pitch <= XFER_SLOT) {
        const size_t per = XFER_SLOT / g.dev_pitch;
        return (g.rows + per - 1) / per;
    }
    return g.rows * ((row_span(g, up) + XFER_SLOT - 1) / XFER_SLOT);
}
Piece piece(const XferSeg &g, size_t i, bool up) {
    if (flat(g, up)) {
        const size_t off = i * XFER_SLOT;
        return {0, 0, off, std::min(XFER_SLOT, g.rows * g.row_bytes - off), 0};
    }
    if (g.dev_pitch <= XFER_SLOT) {
        const size_t per = XFER_SLOT / g.dev_pitch, r = i * per, n = std::min(per, g.rows - r);
        // the last row's pad may lie past the device buffer on the way down
        return {r, n, 0, (n - 1) * g.dev_pitch + g.row_bytes, 0};
    }
    const size_t span = row_span(g, up), per = (span + XFER_SLOT - 1) / XFER_SLOT;
    const size_t off = i % per * XFER_SLOT, bytes = std::min(XFER_SLOT, span - off);
    const size_t past = off + bytes > g.row_bytes ? off + bytes - g.row_bytes : 0;
    return {i / per, 0, off, bytes, std::min(past, bytes)};
}

// Into a pinned slot past the caches: the device reads lines that a core's
// cache holds modified at 4 GB/s at times (120 us for a slot against 14).
void stream_copy(char *to, const char *from, size_t bytes) {
#if defined(__SSE2__)
    if (((uintptr_t)to & 15) == 0) {
        for (; bytes >= 64; bytes -= 64, to += 64, from += 64) {
            const __m128i *f = reinterpret_cast<const __m128i *>(from);
            __m128i *t = reinterpret_cast<__m128i *>(to);
            const __m128i a = _mm_loadu_si128(f), b = _mm_loadu_si128(f + 1),
                          c = _mm_loadu_si128(f + 2), d = _mm_loadu_si128(f + 3);
            _mm_stream_si128(t, a);
            _mm_stream_si128(t + 1, b);
            _mm_stream_si128(t + 2, c);
            _mm_stream_si128(t + 3, d);
        }
        _mm_sfence(); // before the copy to the device is queued
    }
#endif
    std::memcpy(to, from, bytes);
}

// What the ring page-locks and frees belongs to no capture: such calls must not
// end one that another thread of the program has in progress.
struct RelaxedCapture {
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
    ~RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
};

class Ring {
  public:
    // The process ends, or the library is unloaded.  A copy that stays in progress
    // keeps the ring: its threads end with the process.
    void end() {
        if (foreign()) return;
        std::unique_lock<std::mutex> use(use_mu_, std::try_to_lock);
        for (int i = 0; i < 100 && !use.owns_lock(); ++i) {
            std::this_thread::sleep_for(std::chrono::milliseconds(1));
            (void)use.try_lock();
        }
        if (!use.owns_lock()) return;
        const RelaxedCapture relaxed;
        closed_ = true;
        join();
        if (threads_ > 0 && current_context_id() == ctx_id_) free_memory();
    }
    bool run(const XferSeg *segs, int n, bool up, cudaStream_t s, cudaError_t &e) {
        size_t total = 0;
        for (int i = 0; i < n; ++i) total += segs[i].rows * segs[i].row_bytes;
        if (total < XFER_MIN) return false;
        // this name means another stream in each of the ring's threads
        if (s == cudaStreamPerThread) return false;
        if (foreign()) return false;
        // what the device reads or writes itself, at the link's rate
        const XferSeg *big = std::max_element(segs, segs + n, [](const XferSeg &a, const XferSeg &b) {
            return a.rows * a.row_bytes < b.rows * b.row_bytes;
        });
        if (flat(*big, up) && host_pinned(big->host)) return false;
        cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
        if (cudaStreamIsCapturing(s, &cap) != cudaSuccess || cap != cudaStreamCaptureStatusNone) {
            cudaGetLastError();
            return false;
        }
        std::unique_lock<std::mutex> use(use_mu_, std::try_to_lock);
        if (!use.owns_lock() || closed_) return false;
        const RelaxedCapture relaxed;
        int dev = 0;
        if (cudaGetDevice(&dev) != cudaSuccess) {
            cudaGetLastError();
            return false;
        }
        if (threads_ > 0 && dev == device_ && current_context_id() != ctx_id_) {
            // another context of the caller's, or the ring's is gone
            // (cudaDeviceReset), and the slots and events with it
            if (!in_primary_context(dev)) return false;
            join();
            forget_memory();
        }
        if (threads_ == 0) {
            seen_ += total;
            if (seen_ < XFER_AFTER || !set_up(dev)) return false;
        }
        if (dev != device_) return false;
        Job job;
        job.segs = segs;
        job.first.assign(1, 0);
        for (int i = 0; i < n; ++i) job.first.push_back(job.first.back() + pieces(segs[i], up));
        job.up = up;
        job.device = dev;
        job.s = s;
        {
            std::lock_guard<std::mutex> lk(mu_);
            job_ = &job;
            ++ticket_;
            busy_ = (int)workers_.size();
            used_ = std::chrono::steady_clock::now();
        }
        wake_.notify_all();
        work(job, 0);
        std::unique_lock<std::mutex> lk(mu_);
        done_.wait(lk, [&] { return busy_ == 0; });
        job_ = nullptr;
        e = (cudaError_t)job.error.load();
        return true;
    }

  private:
    // a forked child: threads, locks and waiters are the parent's
    bool foreign() const {
        const pid_t p = pid_;
        return p != 0 && p != getpid();
    }

    std::mutex use_mu_; // one copy at a time
    std::mutex mu_;     // the fields below
    std::condition_variable wake_, done_;
    std::vector<std::thread> workers_;
    Job *job_ = nullptr;
    unsigned long ticket_ = 0;
    int busy_ = 0;
    bool stop_ = false;
    std::chrono::steady_clock::time_point used_;
    // set while use_mu_ is held
    int threads_ = 0, device_ = -1;
    unsigned long long ctx_id_ = 0; // the context of the slots and events
    bool closed_ = false;
    std::atomic<pid_t> pid_{0}; // of the process that set the ring up
    size_t seen_ = 0;
    char *pinned_ = nullptr;
    std::vector<cudaEvent_t> ev_;
    std::vector<char> recorded_;

    bool set_up(int dev) {
        if (!in_primary_context(dev)) return false; // the one that the threads use
        join(); // threads of a ring that was given back
        const unsigned hw = std::thread::hardware_concurrency();
        const int t = std::max(2, std::min(XFER_THREADS, (int)hw / 2));
        void *p = nullptr;
        if (cudaMallocHost(&p, XFER_SLOT * 2 * t) != cudaSuccess) {
            cudaGetLastError();
            seen_ = 0; // tried again later
            return false;
        }
        pinned_ = static_cast<char *>(p);
        device_ = dev;
        ctx_id_ = current_context_id();
        pid_ = getpid();
        threads_ = t;
        ev_.assign(2 * t, nullptr);
        recorded_.assign(2 * t, 0);
        bool ok = true;
        for (auto &x : ev_)
            ok = ok && cudaEventCreateWithFlags(&x, cudaEventDisableTiming) == cudaSuccess;
        stop_ = false;
        used_ = std::chrono::steady_clock::now();
        try {
            const unsigned long now = ticket_;
            for (int i = 1; ok && i < t; ++i)
                workers_.emplace_back([this, i, now] { serve(i, now); });
        } catch (...) {
            ok = false;
        }
        if (!ok) {
            cudaGetLastError();
            join();
            free_memory();
        }
        return ok;
    }
    void join() {
        {
            std::lock_guard<std::mutex> lk(mu_);
            stop_ = true;
        }
        wake_.notify_all();
        for (auto &t : workers_) t.join();
        workers_.clear();
        stop_ = false;
    }
    void free_memory() { // no worker touches a slot
        for (auto &x : ev_)
            if (x) {
                cudaEventSynchronize(x);
                cudaEventDestroy(x);
            }
        if (pinned_) cudaFreeHost(pinned_);
        cudaGetLastError();
        forget_memory();
    }
    void forget_memory() {
        ev_.clear();
        pinned_ = nullptr;
        threads_ = 0;
        seen_ = 0;
    }

    void serve(int id, unsigned long last) {
        const RelaxedCapture relaxed;
        for (;;) {
            Job *job = nullptr;
            {
                std::unique_lock<std::mutex> lk(mu_);
                const bool woken = wake_.wait_for(lk, std::chrono::seconds(XFER_IDLE), [&] {
                    return stop_ || ticket_ != last;
                });
                if (stop_) return;
                if (!woken) {
                    // idle: the first worker gives the memory back and ends the
                    // others (their threads are joined at the next set-up)
                    if (id != 1 || std::chrono::steady_clock::now() - used_ <
                                       std::chrono::seconds(XFER_IDLE))
                        continue;
                    lk.unlock();
                    std::unique_lock<std::mutex> use(use_mu_, std::try_to_lock);
                    if (!use.owns_lock()) continue;
                    lk.lock();
                    if (stop_) return;
                    if (ticket_ != last) continue; // a copy came in between
                    stop_ = true;
                    lk.unlock();
                    wake_.notify_all();
                    // (a context that is gone is not made again for it)
                    if (primary_context_active(device_) &&
                        cudaSetDevice(device_) == cudaSuccess && current_context_id() == ctx_id_)
                        free_memory();
                    else
                        forget_memory();
                    return;
                }
                last = ticket_;
                job = job_;
            }
            if (job) {
                cudaSetDevice(job->device);
                work(*job, id);
            }
            std::lock_guard<std::mutex> lk(mu_);
            if (--busy_ == 0) done_.notify_one();
        }
    }

    bool take(Job &job, const XferSeg *&g, Piece &p) {
        const size_t i = job.next.fetch_add(1);
        if (i >= job.first.back() || job.error.load() != 0) return false;
        const size_t k = std::upper_bound(job.first.begin(), job.first.end(), i) -
                         job.first.begin() - 1;
        g = &job.segs[k];
        p = piece(*g, i - job.first[k], job.up);
        return true;
    }
    static char *dev_at(const XferSeg &g, const Piece &p) {
        return static_cast<char *>(g.dev) + p.r * g.dev_pitch + p.off;
    }
    static char *host_at(const XferSeg &g, const Piece &p) {
        return static_cast<char *>(g.host) + p.r * g.host_pitch + p.off;
    }
    void work(Job &job, int id) {
        auto check = [&](cudaError_t r) {
            int none = 0;
            if (r != cudaSuccess) job.error.compare_exchange_strong(none, (int)r);
            return r == cudaSuccess;
        };
        char *const slot[2] = {pinned_ + (size_t)id * 2 * XFER_SLOT,
                               pinned_ + ((size_t)id * 2 + 1) * XFER_SLOT};
        // a slot's last transfer, possibly of an earlier copy, is complete
        auto wait = [&](int k) {
            if (!recorded_[2 * id + k]) return true;
            recorded_[2 * id + k] = 0;
            return check(cudaEventSynchronize(ev_[2 * id + k]));
        };
        auto record = [&](int k) {
            recorded_[2 * id + k] = 1;
            return check(cudaEventRecord(ev_[2 * id + k], job.s));
        };
        const XferSeg *g[2];
        Piece p[2];
        if (job.up) {
            for (int k = 0; take(job, g[0], p[0]); k ^= 1) {
                if (!wait(k)) return;
                size_t bytes = p[0].bytes;
                if (p[0].n == 0) {
                    if (bytes > p[0].pad) stream_copy(slot[k], host_at(*g[0], p[0]), bytes - p[0].pad);
                    std::memset(slot[k] + bytes - p[0].pad, 0, p[0].pad);
                } else {
                    const size_t pad = g[0]->dev_pitch - g[0]->row_bytes;
                    for (size_t r = 0; r < p[0].n; ++r) {
                        char *to = slot[k] + r * g[0]->dev_pitch;
                        stream_copy(to, host_at(*g[0], p[0]) + r * g[0]->host_pitch, g[0]->row_bytes);
                        if (pad) std::memset(to + g[0]->row_bytes, 0, pad);
                    }
                    bytes = p[0].n * g[0]->dev_pitch;
                }
                if (!check(cudaMemcpyAsync(dev_at(*g[0], p[0]), slot[k], bytes,
                                           cudaMemcpyHostToDevice, job.s)) ||
                    !record(k))
                    return;
            }
            return;
        }
        // down: the next piece is on its way while this one is copied out
        auto fetch = [&](int k) {
            return wait(k) &&
                   check(cudaMemcpyAsync(slot[k], dev_at(*g[k], p[k]), p[k].bytes,
                                         cudaMemcpyDeviceToHost, job.s)) &&
                   record(k);
        };
        int k = 0;
        bool have = take(job, g[0], p[0]) && fetch(0);
        while (have) {
            const bool more = take(job, g[k ^ 1], p[k ^ 1]) && fetch(k ^ 1);
            if (!wait(k)) return;
            if (p[k].n == 0) {
                std::memcpy(host_at(*g[k], p[k]), slot[k], p[k].bytes);
            } else {
                for (size_t r = 0; r < p[k].n; ++r)
                    std::memcpy(host_at(*g[k], p[k]) + r * g[k]->host_pitch,
                                slot[k] + r * g[k]->dev_pitch, g[k]->row_bytes);
            }
            have = more;
            k ^= 1;
        }
    }
};

// The object stays: in a forked child, destroying a condition variable waits for
// the parent's waiting threads for ever.
Ring &ring() {
    static Ring *const r = new Ring;
    static const struct End {
        ~End() { r->end(); }
    } at_exit;
    (void)at_exit;
    return *r;
}

} // namespace

bool host_pinned(const void *p) {
    cudaPointerAttributes a{};
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return a.type == cudaMemoryTypeHost;
}
bool xfer_up(const XferSeg *segs, int n, cudaStream_t s, cudaError_t &e) {
    return ring().run(segs, n, true, s, e);
}
bool xfer_down(const XferSeg *segs, int n, cudaStream_t s, cudaError_t &e) {
    return ring().run(segs, n, false, s, e);
}

cudaError_t copy_up(const XferSeg &g, cudaStream_t s) {
    cudaError_t e = cudaSuccess;
    if (xfer_up(&g, 1, s, e)) return e;
    if (flat(g, true))
        return cudaMemcpyAsync(g.dev, g.host, g.rows * g.row_bytes, cudaMemcpyHostToDevice, s);
    e = cudaMemcpy2DAsync(g.dev, g.dev_pitch, g.host, g.host_pitch, g.row_bytes, g.rows,
                          cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess && g.dev_pitch > g.row_bytes)
        e = cudaMemset2DAsync(static_cast<char *>(g.dev) + g.row_bytes, g.dev_pitch, 0,
                              g.dev_pitch - g.row_bytes, g.rows, s);
    return e;
}
cudaError_t copy_down(const XferSeg &g, cudaStream_t s) {
    cudaError_t e = cudaSuccess;
    if (xfer_down(&g, 1, s, e)) return e;
    if (flat(g, false)) {
        e = cudaMemcpyAsync(g.host, g.dev, g.rows * g.row_bytes, cudaMemcpyDeviceToHost, s);
        return e == cudaSuccess ? cudaStreamSynchronize(s) : e;
    }
    // Short rows that are dense on the device come down in runs and are dealt out
    // here: the driver takes 0.2 us a row (1.5 MB of 256-byte rows: 1.0 ms against
    // 0.30; of 2,048-byte rows 0.27 each way, of 4,096-byte ones 0.20 against 0.26).
    const size_t per = std::max<size_t>(1, (4u << 20) / g.row_bytes);
    const std::unique_ptr<char[]> tmp(
        g.dev_pitch == g.row_bytes && g.row_bytes < 2048
            ? new (std::nothrow) char[std::min(per, g.rows) * g.row_bytes]
            : nullptr);
    if (tmp) {
        for (size_t r = 0; r < g.rows; r += per) {
            const size_t n = std::min(per, g.rows - r);
            e = cudaMemcpyAsync(tmp.get(), static_cast<char *>(g.dev) + r * g.row_bytes,
                                n * g.row_bytes, cudaMemcpyDeviceToHost, s);
            if (e == cudaSuccess) e = cudaStreamSynchronize(s);
            if (e != cudaSuccess) return e;
            char *to = static_cast<char *>(g.host) + r * g.host_pitch;
            for (size_t i = 0; i < n; ++i)
                std::memcpy(to + i * g.host_pitch, tmp.get() + i * g.row_bytes, g.row_bytes);
        }
    } else {
        e = cudaMemcpy2DAsync(g.host, g.host_pitch, g.dev, g.dev_pitch, g.row_bytes, g.rows,
                              cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    }
    return e;
}

} // namespace b200
