// Drives csrc/host_copy.h against a stand-in for the CUDA runtime in which every copy is done at once, so that what the
// staging threads do can be tested without a GPU and with a system that refuses threads or memory.
//   host_copy_check threads | memory | idle
#include "../rustorch_b200/csrc/host_copy.h"

#include <dlfcn.h>
#include <pthread.h>
#include <sys/resource.h>
#include <time.h>

#include <chrono>
#include <cstdio>
#include <cstdlib>

// ---- the stand-in
extern "C" {
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { return (*p = aligned_alloc(4096, n)) ? cudaSuccess : cudaErrorMemoryAllocation; }
cudaError_t cudaFreeHost(void* p) { free(p); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) { memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t*, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t*, unsigned) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventQuery(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes*, const void*) { return cudaErrorInvalidValue; }
cudaError_t cudaGetLastError() { return cudaSuccess; }

// ---- a system that gives a number of threads, or of allocations, and then no more
static int threads_left = 1 << 30, threads_made = 0;
int pthread_create(pthread_t* t, const pthread_attr_t* a, void* (*f)(void*), void* x) {
    static auto real = (int (*)(pthread_t*, const pthread_attr_t*, void* (*)(void*), void*))dlsym(RTLD_NEXT, "pthread_create");
    if (threads_left-- <= 0) return EAGAIN;
    ++threads_made;
    return real(t, a, f, x);
}
}
static thread_local long news_left = 1l << 60;
void* operator new(size_t n) {
    if (news_left-- <= 0) throw std::bad_alloc();
    void* p = malloc(n ? n : 1);
    if (!p) abort();
    return p;
}
void operator delete(void* p) noexcept { free(p); }
void operator delete(void* p, size_t) noexcept { free(p); }

static rt::HostWorkers workers;
static rt::HostJob::Device device;

// Up in two chunks and down again: 24 MB each way, more pieces than the ring has slots.  Returns the call's status, as an
// entry point would; -1 for a wrong result.
constexpr size_t n = 6 << 20;
static std::vector<float> host(n), dev(n), back(n);
static int call(int sleep_ms = 0) {
    for (size_t i = 0; i < n; ++i) host[i] = (float)i, back[i] = 0.f;
    int rc;
    try {
        rt::HostJob job(workers, device);
        for (int c = 0; c < 2; ++c) {
            job.upload(c, dev.data() + c * n / 2, host.data() + c * n / 2, n / 2, 4, rt::HostMode::kCopy, true);
            job.download(c, back.data() + c * n / 2, dev.data() + c * n / 2, n / 2, 4, rt::HostMode::kCopy, true);
        }
        rc = job.run(2, [&](int, cudaStream_t) {
            if (sleep_ms) std::this_thread::sleep_for(std::chrono::milliseconds(sleep_ms));
            return 0;
        });
    } catch (...) {
        rc = rt::exception_status();
    }
    return rc != 0 ? rc : back == host ? 0 : -1;
}

static double cpu_ms(clockid_t c) {
    timespec t;
    clock_gettime(c, &t);
    return t.tv_sec * 1e3 + t.tv_nsec * 1e-6;
}

#define CHECK(x)                                                     \
    do {                                                             \
        if (!(x)) {                                                  \
            printf("line %d: %s does not hold\n", __LINE__, #x);     \
            fflush(stdout);                                          \
            _Exit(1);                                                \
        }                                                            \
    } while (0)

int main(int argc, char** argv) {
    const char what = argc > 1 ? argv[1][0] : 0;
    const int cores = (int)std::thread::hardware_concurrency(), full = cores > 15 ? 7 : cores > 2 ? cores / 2 - 1 : 0;
    device.init();
    if (what == 't') {  // no thread, then one, then all: every call works, and later ones start what was missing
        threads_left = 0;
        CHECK(call() == 0 && threads_made == 0);
        threads_left = 1;
        CHECK(call() == 0 && threads_made == (full ? 1 : 0));
        threads_left = 1 << 30;
        CHECK(call() == 0 && threads_made == full);
        CHECK(call() == 0 && threads_made == full);
    } else if (what == 'm') {  // memory refused at each request of a call in turn
        int refused = 0;
        for (long given = 0; given < 1000; ++given) {
            news_left = given;
            const int rc = call();
            const bool short_of = news_left < 0;
            news_left = 1l << 60;
            CHECK(rc == 0 || rc == (int)cudaErrorMemoryAllocation);
            CHECK(call() == 0);
            refused += rc != 0;
            if (!short_of) break;
        }
        CHECK(refused > 3);
    } else if (what == 'i') {  // while a kernel runs and there is nothing to copy, the staging threads sleep
        CHECK(call() == 0);
        const double all = cpu_ms(CLOCK_PROCESS_CPUTIME_ID), own = cpu_ms(CLOCK_THREAD_CPUTIME_ID);
        CHECK(call(300) == 0);  // 0.6 s of waiting
        const double others = cpu_ms(CLOCK_PROCESS_CPUTIME_ID) - all - (cpu_ms(CLOCK_THREAD_CPUTIME_ID) - own);
        printf("%.1f ms by the staging threads\n", others);
        CHECK(others < 100);
        for (int i = 0; i < 200; ++i) CHECK(call(i % 3) == 0);  // to sleep and back, often
    } else {
        return 2;
    }
    printf("ok\n");
}
