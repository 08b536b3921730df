// Shared device helpers for the sm_100a attention kernels.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace rt {

constexpr float kLog2e = 1.4426950408889634f;
constexpr float kLn2 = 0.6931471805599453f;
constexpr unsigned kFullMask = 0xffffffffu;

// Device status word: 0 = clean; kernels record here which bounded wait gave up.  The word
// lives in api.cu; kernels receive its device address as a parameter.  Read (and cleared)
// by rt_attn_device_status().
__device__ __forceinline__ void report_timeout(int* status, int code) { atomicCAS(status, 0, code); }

// 16-byte streaming load that bypasses L1 allocation (KV cache is read exactly once).
__device__ __forceinline__ uint4 ld_stream_16B(const void* p) {
    uint4 r;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w)
                 : "l"(p));
    return r;
}

// Two bf16 packed in a 32-bit word -> (low element, high element) as f32.
__device__ __forceinline__ float2 bf16x2_to_float2(uint32_t w) {
    return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u));
}

__device__ __forceinline__ uint32_t float2_to_bf16x2(float lo, float hi) {
    __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);  // .x = lo (low half), RNE
    return *reinterpret_cast<uint32_t*>(&h);
}

__device__ __forceinline__ float fast_exp2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// max(a, b, c) in one instruction (three-input max exists from sm_100 on).
__device__ __forceinline__ float max3(float a, float b, float c) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

__device__ __forceinline__ float fast_log2(float x) {
    float y;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// How a decode launch cuts its sequences into chunks, one CTA each; see pick_split for the rule.
enum { kSplitFixed = 0, kSplitEven, kSplitShare, kSplitCluster };
struct DecodeSplit {
    int n_chunks;  // chunks of a sequence at most
    int chunk;     // kSplitFixed: tokens per chunk (grid: chunk, KV head, sequence)
    int mode;      // kSplitEven: n_chunks equal parts of every sequence's own length (same grid)
                   // kSplitCluster: the same parts, merged by the cluster of n_chunks CTAs that streams them (no partials)
                   // kSplitShare: chunks of one size for all `batch` <= 32 sequences, about `target` of them in all,
    int batch;     //              dealt to a flat grid of `ctas` CTAs
    int ctas;
    int slots;     //              CTAs resident at a time
    float target;
};

// The chunk of the calling CTA: tokens [lo, hi) of the sequence's visible range.
struct DecodeChunk {
    int b, kvh, idx, lo, hi;
    int rest;  // kSplitShare: chunks after the sequence's last, which the CTA with the last marks empty for the merge
    bool none;  // kSplitShare: a CTA beyond the last chunk
};

__device__ __forceinline__ int round_up_64(int x) { return max(64, (x + 63) & ~63); }

// Called by all threads of a warp; every warp comes to the same answer on its own.  visible_of(b): tokens of sequence b.
template <bool kShare, class VisibleOf>
__device__ __forceinline__ DecodeChunk find_chunk(const DecodeSplit& sp, int n_kv, VisibleOf&& visible_of) {
    DecodeChunk c;
    c.none = false;
    c.rest = 0;
    if (!kShare) {
        c.idx = blockIdx.x, c.kvh = blockIdx.y, c.b = blockIdx.z;
        const int visible = visible_of(c.b);
        const int size = sp.mode == kSplitFixed ? sp.chunk : round_up_64((visible + sp.n_chunks - 1) / sp.n_chunks);
        c.lo = c.idx * size;
        c.hi = min(c.lo + size, visible);
        return c;
    }
    // Lane b holds sequence b: the sum of the lengths gives the chunk size, a scan of the chunk counts the place of
    // every sequence in the list of chunks (sequence, KV head, chunk).
    const int lane = threadIdx.x & 31;
    const int visible = lane < sp.batch ? visible_of(lane) : 0;
    float total = (float)visible;
#pragma unroll
    for (int off = 16; off; off >>= 1) total += __shfl_xor_sync(kFullMask, total, off);
    int share = (int)ceilf(total * (float)n_kv / sp.target);
    int n, size, mine, end;
    for (int tries = 0;; ++tries) {
        const int most = round_up_64(max(share, (visible + sp.n_chunks - 1) / sp.n_chunks));
        n = max(1, (visible + most - 1) / most);
        size = round_up_64((visible + n - 1) / n);  // equal chunks: the last one would end early otherwise
        end = mine = lane < sp.batch ? n * n_kv : 0;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const int y = __shfl_up_sync(kFullMask, end, off);
            if (lane >= off) end += y;
        }
        // Lengths alike can all just miss one chunk less; a few CTAs more than fit at once cost a second wave.
        if (tries == 3 || __shfl_sync(kFullMask, end, 31) <= sp.slots) break;
        share += share >> 3;
    }
    const int want = blockIdx.x;
    const unsigned owner = __ballot_sync(kFullMask, want >= end - mine && want < end);
    c.none = owner == 0;
    c.b = owner ? __ffs(owner) - 1 : 0;
    const int at = want - __shfl_sync(kFullMask, end - mine, c.b), size_b = __shfl_sync(kFullMask, size, c.b),
              n_b = __shfl_sync(kFullMask, n, c.b), visible_b = __shfl_sync(kFullMask, visible, c.b);
    c.kvh = at / n_b;
    c.idx = at - c.kvh * n_b;
    c.lo = c.idx * size_b;
    c.hi = min(c.lo + size_b, visible_b);
    if (c.idx == n_b - 1) c.rest = sp.n_chunks - n_b;
    return c;
}

}  // namespace rt
