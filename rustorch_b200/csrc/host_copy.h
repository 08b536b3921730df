// Staged copies between pageable host memory and the device for the blocking *_host entry points.
//
// A cudaMemcpyAsync on pageable memory blocks its caller while the driver moves the data through its own pinned
// buffers with one thread: 10 to 15 GB/s here against the 50 GB/s of the link, and nothing of the call overlaps.  A
// HostJob cuts the tensors of a call into 64 KB pieces; a few worker threads copy pieces into a pinned ring (and out
// of one, for the results) while the calling thread enqueues the transfers in order, launches each chunk's kernels
// once its inputs are on the way, and hands finished downloads to the workers.  Pieces are small so that eight threads
// share even a small tensor (4 MB in 35 us), transfers are runs of pieces because a transfer costs 3 us apart from its
// bytes (16 MB: 52 GB/s in 4 MB transfers, 39 in 512 KB, 12 in 64 KB), and 8 us when an event follows it: runs of 1 to
// 2 MB (a short first one, so that the link starts early), with events only where ring slots are used again.  With f32 host data and bf16 kernels the
// workers convert as they copy, which halves what crosses the link.  Pinned host memory skips the ring.
//
// The workers and the ring (16 MB up, 8 MB down) are made by the first call that needs them, serve one call at a time
// (the entry points hold a lock) and are given back when the library is unloaded.  The workers sleep while there is
// nothing to copy; the calling thread polls until the call ends, as in any blocking CUDA call.
#pragma once
#include <cuda_runtime.h>
#if defined(__x86_64__)
#include <immintrin.h>
#endif

#include <atomic>
#include <chrono>
#include <condition_variable>
#include <cstdint>
#include <cstring>
#include <exception>
#include <functional>
#include <mutex>
#include <new>
#include <thread>
#include <vector>

namespace rt {

enum class HostMode { kCopy, kF32ToBf16, kBf16ToF32 };  // what happens between the host side and the device side

inline uint16_t f32_bits_to_bf16(uint32_t u) {  // round to nearest even; NaN as the device conversion gives it
    const uint32_t rounded = (u + 0x7fffu + ((u >> 16) & 1u)) >> 16;
    return (u & 0x7fffffffu) > 0x7f800000u ? (uint16_t)0x7fffu : (uint16_t)rounded;
}

// The two conversions, compiled for AVX2 where the processor has it (0.34 -> 0.19 ms for a million values a thread).
inline void f32_to_bf16_row(uint16_t* d, const uint32_t* s, size_t n) {
    for (size_t i = 0; i < n; ++i) d[i] = f32_bits_to_bf16(s[i]);
}
inline void bf16_to_f32_row(uint32_t* d, const uint16_t* s, size_t n) {
    for (size_t i = 0; i < n; ++i) d[i] = (uint32_t)s[i] << 16;
}
#if defined(__x86_64__)
// Streaming stores, see copy_streaming; dst is 32-byte aligned.
__attribute__((target("avx2"))) inline void f32_to_bf16_row_avx2(uint16_t* d, const uint32_t* s, size_t n) {
    const __m256i half = _mm256_set1_epi32(0x7fff), one = _mm256_set1_epi32(1), inf = _mm256_set1_epi32(0x7f800000),
                  abs = _mm256_set1_epi32(0x7fffffff);
    size_t i = 0;
    for (; i + 16 <= n; i += 16) {
        __m256i r[2];
        for (int k = 0; k < 2; ++k) {
            const __m256i u = _mm256_loadu_si256(reinterpret_cast<const __m256i*>(s + i + 8 * k));
            const __m256i odd = _mm256_and_si256(_mm256_srli_epi32(u, 16), one);
            const __m256i x = _mm256_srli_epi32(_mm256_add_epi32(_mm256_add_epi32(u, half), odd), 16);
            r[k] = _mm256_blendv_epi8(x, half, _mm256_cmpgt_epi32(_mm256_and_si256(u, abs), inf));
        }
        const __m256i packed = _mm256_permute4x64_epi64(_mm256_packus_epi32(r[0], r[1]), 0xd8);
        _mm256_stream_si256(reinterpret_cast<__m256i*>(d + i), packed);
    }
    _mm_sfence();
    for (; i < n; ++i) d[i] = f32_bits_to_bf16(s[i]);
}
__attribute__((target("avx2"))) inline void bf16_to_f32_row_avx2(uint32_t* __restrict__ d, const uint16_t* __restrict__ s,
                                                                 size_t n) {
    for (size_t i = 0; i < n; ++i) d[i] = (uint32_t)s[i] << 16;
}
inline bool has_avx2() {
    static const bool yes = __builtin_cpu_supports("avx2");
    return yes;
}
#endif

// Copy into the upload ring past the caches: the link reads what the threads have just written, and from a core's
// cache it does so a sixth slower (12 MB: 342 against 292 us).
inline void copy_streaming(void* dst, const void* src, size_t n) {
#if defined(__x86_64__)
    __m128i* d = static_cast<__m128i*>(dst);  // ring slots are aligned
    const __m128i* s = static_cast<const __m128i*>(src);
    for (size_t i = 0; i < n / 64; ++i, d += 4, s += 4) {
        const __m128i a = _mm_loadu_si128(s), b = _mm_loadu_si128(s + 1), c = _mm_loadu_si128(s + 2), e = _mm_loadu_si128(s + 3);
        _mm_stream_si128(d, a);
        _mm_stream_si128(d + 1, b);
        _mm_stream_si128(d + 2, c);
        _mm_stream_si128(d + 3, e);
    }
    _mm_sfence();
    memcpy(d, s, n % 64);
#else
    memcpy(dst, src, n);
#endif
}

// One piece of work for a thread: n elements (f32 <-> bf16) or bytes (copy) from src to dst.
struct HostTask {
    void* dst;
    const void* src;
    size_t n;
    HostMode mode;
    bool up;
    void run() const {
        if (mode == HostMode::kCopy) {
            if (up) copy_streaming(dst, src, n);
            else memcpy(dst, src, n);
        } else if (mode == HostMode::kF32ToBf16) {
            const uint32_t* s = static_cast<const uint32_t*>(src);
            uint16_t* d = static_cast<uint16_t*>(dst);
#if defined(__x86_64__)
            if (has_avx2()) return f32_to_bf16_row_avx2(d, s, n);
#endif
            f32_to_bf16_row(d, s, n);
        } else {
            const uint16_t* s = static_cast<const uint16_t*>(src);
            uint32_t* d = static_cast<uint32_t*>(dst);
#if defined(__x86_64__)
            if (has_avx2()) return bf16_to_f32_row_avx2(d, s, n);
#endif
            bf16_to_f32_row(d, s, n);
        }
    }
};

// Tasks that any thread may take, in order, as far as they have been released.
class HostQueue {
  public:
    void reset(size_t n) {
        tasks.assign(n, HostTask{});
        done_ = std::vector<std::atomic<uint8_t>>(n);
        next_.store(0);
        limit_.store(0);
    }
    std::vector<HostTask> tasks;
    void release(size_t upto) { limit_.store(upto, std::memory_order_release); }  // tasks below `upto` are filled in
    bool waiting() const { return next_.load() < limit_.load(); }                 // a released task that nobody has taken
    bool done(size_t i) const { return done_[i].load(std::memory_order_acquire) != 0; }
    bool run_one() {
        size_t i = next_.load(std::memory_order_relaxed);
        do {
            if (i >= limit_.load(std::memory_order_acquire)) return false;
        } while (!next_.compare_exchange_weak(i, i + 1));
        tasks[i].run();
        done_[i].store(1, std::memory_order_release);
        return true;
    }

  private:
    std::vector<std::atomic<uint8_t>> done_;
    std::atomic<size_t> next_{0}, limit_{0};
};

// The status for the exception being handled.  The C entry points catch all (memory, a thread or a lock that the system
// refuses): none may reach a caller whose frames need not be C++.
inline int exception_status() noexcept {
    try {
        throw;
    } catch (const std::bad_alloc&) {
        return (int)cudaErrorMemoryAllocation;
    } catch (...) {
        return (int)cudaErrorUnknown;
    }
}

// The worker threads and the pinned ring of the process.
class HostWorkers {
  public:
    static constexpr size_t kPiece = size_t(64) << 10;
    static constexpr size_t kUp = 256, kDown = 128;
    HostQueue up, down;
    uint8_t* ring = nullptr;  // kUp slots, then kDown slots
    uint8_t* up_slot(size_t i) { return ring + (i % kUp) * kPiece; }
    uint8_t* down_slot(size_t i) { return ring + (kUp + i % kDown) * kPiece; }

    cudaError_t init() {
        if (!ring) {
            void* p = nullptr;
            const cudaError_t e = cudaHostAlloc(&p, (kUp + kDown) * kPiece, cudaHostAllocPortable);
            if (e != cudaSuccess) return e;
            ring = static_cast<uint8_t*>(p);
        }
        const size_t cores = std::thread::hardware_concurrency(), n = cores > 15 ? 7 : cores > 2 ? cores / 2 - 1 : 0;
        // A process that gets no more threads works with the ones it has, none at worst: the calling thread copies as
        // well.  The next call asks again.
        try {
            threads_.reserve(n);
            while (threads_.size() < n) threads_.emplace_back([this] { work(); });
        } catch (const std::exception&) {
        }
        return cudaSuccess;
    }
    // Tasks of q below `upto` may be taken from now on.
    void release(HostQueue& q, size_t upto) {
        {
            std::lock_guard<std::mutex> lock(mu_);
            q.release(upto);
            if (asleep_ == 0) return;
        }
        cv_.notify_all();
    }
    // Between begin and end the workers take tasks from both queues; end returns once none of them looks at them.
    void begin() {
        active_.store(true);
        {
            std::lock_guard<std::mutex> lock(mu_);
            ++generation_;
        }
        cv_.notify_all();
    }
    void end() {
        {
            std::lock_guard<std::mutex> lock(mu_);  // a worker enters under this lock, or sees active_ false
            active_.store(false);
        }
        cv_.notify_all();
        while (inside_.load() != 0) std::this_thread::yield();
    }
    ~HostWorkers() {
        {
            std::lock_guard<std::mutex> lock(mu_);
            stop_ = true;
        }
        cv_.notify_all();
        for (std::thread& t : threads_) t.join();
        if (ring) cudaFreeHost(ring);
    }

  private:
    void work() {
        uint64_t seen = 0;
        for (;;) {
            {
                std::unique_lock<std::mutex> lock(mu_);
                cv_.wait(lock, [&] { return stop_ || generation_ != seen; });
                if (stop_) return;
                seen = generation_;
                if (!active_.load()) continue;
                inside_.fetch_add(1);
            }
            int idle = 0;
            std::chrono::steady_clock::time_point idle_since;
            while (active_.load(std::memory_order_relaxed)) {
                if (down.run_one() || up.run_one()) {
                    idle = 0;
                    continue;
                }
                if (++idle <= 256) continue;
                std::this_thread::yield();
                if (idle == 257) idle_since = std::chrono::steady_clock::now();
                if (idle % 16 != 0 || std::chrono::steady_clock::now() - idle_since < kSpin) continue;
                std::unique_lock<std::mutex> lock(mu_);  // tasks are released under this lock
                ++asleep_;
                cv_.wait(lock, [&] { return !active_.load() || down.waiting() || up.waiting(); });
                --asleep_;
                idle = 0;
            }
            inside_.fetch_sub(1);
        }
    }
    // A worker without a task looks for one this long and then sleeps until one is released.  To be woken takes some 50 us,
    // which would come on top of a short kernel; while a longer one runs, or only pinned data moves, the cores stay free.
    static constexpr std::chrono::microseconds kSpin{200};
    std::vector<std::thread> threads_;
    std::mutex mu_;
    std::condition_variable cv_;
    uint64_t generation_ = 0;
    int asleep_ = 0;  // in the middle of a call
    bool stop_ = false;
    std::atomic<bool> active_{false};
    std::atomic<int> inside_{0};
};

inline bool is_pageable(const void* p) {
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return true;
    }
    return a.type == cudaMemoryTypeUnregistered;
}

// The copies and launches of one blocking call: chunk by chunk, the inputs up, `launch`, the results down.
class HostJob {
  public:
    struct Device {  // streams and events of the current device
        static constexpr int kComp = 4, kMaxChunks = 32;
        cudaStream_t in = nullptr, out = nullptr, comp[kComp] = {};
        static constexpr int kTransfers = 32;  // transfers of one direction that may be under way
        cudaEvent_t ev_in[kMaxChunks] = {}, ev_comp[kMaxChunks] = {}, ev_up[kTransfers] = {}, ev_down[kTransfers] = {};
        bool ready = false;
        cudaError_t init() {
            if (ready) return cudaSuccess;
            cudaError_t e = cudaStreamCreateWithFlags(&in, cudaStreamNonBlocking);
            if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&out, cudaStreamNonBlocking);
            for (int i = 0; i < kComp && e == cudaSuccess; ++i) e = cudaStreamCreateWithFlags(&comp[i], cudaStreamNonBlocking);
            auto events = [&](cudaEvent_t* ev, int n) {
                for (int i = 0; i < n && e == cudaSuccess; ++i) e = cudaEventCreateWithFlags(&ev[i], cudaEventDisableTiming);
            };
            events(ev_in, kMaxChunks);
            events(ev_comp, kMaxChunks);
            events(ev_up, kTransfers);
            events(ev_down, kTransfers);
            ready = e == cudaSuccess;
            return e;
        }
    };
    HostJob(HostWorkers& w, Device& d) : w_(w), d_(d) {}

    // n elements of `size` bytes on the device; the host side has the same, or f32 where the mode converts.
    // Calls are in chunk order.
    void upload(int chunk, void* dev, const void* host, size_t n, size_t size, HostMode mode, bool staged) {
        add(up_, chunk, dev, const_cast<void*>(host), n, size, mode, staged);
    }
    void download(int chunk, void* host, const void* dev, size_t n, size_t size, HostMode mode, bool staged) {
        add(down_, chunk, const_cast<void*>(dev), host, n, size, mode, staged);
    }

    // launch(chunk, stream) enqueues the kernels of a chunk and returns a status; chunks may run side by side.
    template <class Launch>
    int run(int n_chunks, Launch&& launch) {
        size_t n_up = 0, n_down = 0;
        for (const Piece& p : up_) n_up += p.staged;
        for (const Piece& p : down_) n_down += p.staged;
        bool working = false;
        int rc = 0;
        try {
            if (n_up + n_down > 0) {
                rc = (int)w_.init();
                if (rc == 0) {
                    w_.up.reset(n_up);
                    w_.down.reset(n_down);
                    size_t k = 0;
                    for (const Piece& p : up_)
                        if (p.staged) w_.up.tasks[k] = HostTask{w_.up_slot(k), p.host, p.n, p.mode, true}, ++k;
                    w_.release(w_.up, n_up < HostWorkers::kUp ? n_up : HostWorkers::kUp);
                    w_.begin();
                    working = true;
                }
            }
            if (rc == 0) rc = drive(n_chunks, n_up, launch);
        } catch (...) {
            rc = exception_status();
        }
        if (working) w_.end();
        // nothing may still use the ring or the caller's memory when the call returns
        for (cudaStream_t s : {d_.in, d_.comp[0], d_.comp[1], d_.comp[2], d_.comp[3], d_.out}) {
            const cudaError_t e = cudaStreamSynchronize(s);
            if (rc == 0 && e != cudaSuccess) rc = (int)e;
        }
        return rc;
    }

  private:
    struct Piece {
        int chunk;
        void *dev, *host;
        size_t n, bytes;  // elements to convert (or bytes to copy), and bytes on the device
        HostMode mode;
        bool staged, first;  // first: of its tensor
    };
    void add(std::vector<Piece>& to, int chunk, void* dev, void* host, size_t n, size_t size, HostMode mode, bool staged) {
        const size_t host_size = mode == HostMode::kCopy ? size : sizeof(float);
        const size_t most = staged ? HostWorkers::kPiece / size : n;
        for (size_t at = 0; at < n; at += most) {
            const size_t m = n - at < most ? n - at : most;
            to.push_back(Piece{chunk, static_cast<char*>(dev) + at * size, static_cast<char*>(host) + at * host_size,
                               mode == HostMode::kCopy ? m * size : m, m * size, mode, staged, at == 0});
        }
    }
    // Transfers of one direction under way, oldest first: the staged pieces up to end[] are done with the newest of them.
    struct Transfers {
        size_t head = 0, tail = 0, end[Device::kTransfers];
        size_t under_way() const { return head - tail; }
        size_t start(size_t upto) {  // the new transfer's event
            end[head % Device::kTransfers] = upto;
            return head++ % Device::kTransfers;
        }
    };
    // Pieces from `at` on that one transfer can take: ready, next to each other in the ring, of one tensor and chunk
    // (two buffers may happen to be neighbours, but a transfer must not run from one allocation into the next).
    template <class Ready>
    static size_t run_of(const std::vector<Piece>& v, size_t at, size_t slot, size_t slots, size_t most_bytes, bool& whole,
                         Ready&& ready) {
        size_t n = 0;
        for (whole = true; at + n < v.size() && n < most_bytes / HostWorkers::kPiece; ++n) {
            const Piece& p = v[at + n];
            if (!p.staged || (n > 0 && p.first) || slot % slots + n >= slots) break;
            if (!ready(slot + n)) {
                whole = false;
                break;
            }
        }
        return n;
    }
    static size_t bytes_of(const std::vector<Piece>& v, size_t at, size_t n) {
        return (n - 1) * HostWorkers::kPiece + v[at + n - 1].bytes;  // only a tensor's last piece is short
    }
    template <class Launch>
    int drive(int n_chunks, size_t n_up, Launch&& launch) {
#define RT_TRY(expr)                                 \
    do {                                             \
        const cudaError_t e_ = (expr);               \
        if (e_ != cudaSuccess) return (int)e_;       \
    } while (0)
        Transfers ups, downs;
        size_t u = 0, us = 0;   // input pieces enqueued, staged ones among them
        size_t dn = 0, ds = 0;  // the same of the results
        int launched = 0;
        while (u < up_.size() || launched < n_chunks || dn < down_.size() || (ds > 0 && !all_done(ds))) {
            bool moved = false;
            // ---- finished transfers: ring slots of inputs take the next pieces, results can be copied out
            for (bool is_up : {true, false}) {
                Transfers& t = is_up ? ups : downs;
                while (t.under_way() > 0) {
                    const cudaError_t e = cudaEventQuery((is_up ? d_.ev_up : d_.ev_down)[t.tail % Device::kTransfers]);
                    if (e == cudaErrorNotReady) break;
                    RT_TRY(e);
                    const size_t upto = t.end[t.tail++ % Device::kTransfers];
                    if (is_up) w_.release(w_.up, upto + HostWorkers::kUp < n_up ? upto + HostWorkers::kUp : n_up);
                    else w_.release(w_.down, upto);
                    moved = true;
                }
            }
            // ---- the next input pieces, once they are in the ring
            if (u < up_.size() && up_[u].chunk == launched) {
                if (!up_[u].staged) {
                    RT_TRY(cudaMemcpyAsync(up_[u].dev, up_[u].host, up_[u].bytes, cudaMemcpyHostToDevice, d_.in));
                    ++u, moved = true;
                } else if (ups.under_way() < Device::kTransfers) {
                    bool whole;  // the run ends because nothing can follow, not because a piece is not ready yet
                    const size_t run = run_of(up_, u, us, HostWorkers::kUp, 2u << 20, whole, [&](size_t k) { return w_.up.done(k); });
                    if (run > 0 && (whole || run * HostWorkers::kPiece >= (us == 0 ? 256u << 10 : 1u << 20))) {
                        RT_TRY(cudaMemcpyAsync(up_[u].dev, w_.up_slot(us), bytes_of(up_, u, run), cudaMemcpyHostToDevice, d_.in));
                        u += run, us += run, moved = true;
                        if (n_up > HostWorkers::kUp) RT_TRY(cudaEventRecord(d_.ev_up[ups.start(us)], d_.in));
                    }
                }
            } else if (launched < n_chunks) {  // all inputs of this chunk are on the way
                cudaStream_t s = d_.comp[launched % Device::kComp];
                RT_TRY(cudaEventRecord(d_.ev_in[launched], d_.in));
                RT_TRY(cudaStreamWaitEvent(s, d_.ev_in[launched], 0));
                const int rc = launch(launched, s);
                if (rc != 0) return rc;
                RT_TRY(cudaEventRecord(d_.ev_comp[launched], s));
                RT_TRY(cudaStreamWaitEvent(d_.out, d_.ev_comp[launched], 0));
                ++launched, moved = true;
            }
            // ---- results of launched chunks, into ring slots that have been copied out
            if (dn < down_.size() && down_[dn].chunk < launched) {
                if (!down_[dn].staged) {
                    RT_TRY(cudaMemcpyAsync(down_[dn].host, down_[dn].dev, down_[dn].bytes, cudaMemcpyDeviceToHost, d_.out));
                    ++dn, moved = true;
                } else if (downs.under_way() < Device::kTransfers) {
                    bool whole;
                    const size_t run = run_of(down_, dn, ds, HostWorkers::kDown, 1u << 20, whole, [&](size_t k) {
                        return k < HostWorkers::kDown || w_.down.done(k - HostWorkers::kDown);
                    });
                    if (run > 0) {
                        RT_TRY(cudaMemcpyAsync(w_.down_slot(ds), down_[dn].dev, bytes_of(down_, dn, run),
                                               cudaMemcpyDeviceToHost, d_.out));
                        for (size_t i = 0; i < run; ++i)
                            w_.down.tasks[ds + i] = HostTask{down_[dn + i].host, w_.down_slot(ds + i), down_[dn + i].n,
                                                             down_[dn + i].mode, false};
                        dn += run, ds += run, moved = true;
                        RT_TRY(cudaEventRecord(d_.ev_down[downs.start(ds)], d_.out));
                    }
                }
            }
            // ---- nothing to enqueue: this thread copies as well
            if (!moved && !w_.down.run_one()) w_.up.run_one();
        }
        return 0;
#undef RT_TRY
    }
    bool all_done(size_t n) {
        while (finished_ < n && w_.down.done(finished_)) ++finished_;
        return finished_ == n;
    }
    HostWorkers& w_;
    Device& d_;
    std::vector<Piece> up_, down_;
    size_t finished_ = 0;
};

}  // namespace rt
