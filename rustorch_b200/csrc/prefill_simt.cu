// f32 flash-attention forward on CUDA cores, plus the f32 <-> bf16 conversion kernels.
//
// The exact-arithmetic companions of the tensor-core kernel: f32 inputs, f32
// accumulation, CUDA's exponentials, any head dim up to 256, seq_q != seq_kv and grouped KV heads.
// They back the host mirrors of flash_forward_masked (crates/rustorch-attention/src/cpu_forward.rs:193-242)
// and gqa_forward_f32 (crates/rustorch-nn/src/gqa.rs:94-210) at the reference's own 1e-4
// tolerance.  The online-softmax recurrence is the reference's (cpu_forward.rs:355-386) with the
// leading-masked-tile case resolved to the finite answer.
//   prefill_f32_tiled_kernel  16 query rows and more: 64 rows per CTA, register tiles, exp2f (simt_tile.cuh)
//   prefill_f32_kernel        fewer rows: one warp owns one query row and walks the keys in tiles of 32 staged in
//                             shared memory, expf
#include <algorithm>
#include <atomic>
#include <cstdlib>

#include "common.cuh"
#include "kernels.h"
#include "simt_tile.cuh"

namespace rt {

constexpr int kSimtRows = 8;   // query rows (warps) per CTA
constexpr int kSimtKeys = 32;  // keys per tile (one per lane)

struct SimtParams {
    const float *q, *k, *v;
    float *out, *lse;
    int64_t heads_q, heads_kv, seq_q, seq_kv;
    int dim, causal;
    const int32_t* kv_lens;
    const int32_t* q_offsets;
    const uint8_t* key_keep;
    int64_t keep_batch_stride;
    float scale;
    int split;  // CTAs (one cluster) that share the keys of a row block
};

__global__ void __launch_bounds__(kSimtRows * 32) prefill_f32_kernel(const SimtParams p) {
    extern __shared__ float smem[];
    const int D = p.dim;
    float* Ks = smem;                              // [32][D+1]
    float* Vs = Ks + kSimtKeys * (D + 1);          // [32][D]
    float* Qs = Vs + kSimtKeys * D;                // [rows][D]

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t b = blockIdx.z, hq = blockIdx.y;
    const int64_t hkv = hq / (p.heads_q / p.heads_kv);
    const int64_t row0 = (int64_t)blockIdx.x * kSimtRows;
    const int64_t qi = row0 + warp;
    const bool row_valid = qi < p.seq_q;

    const float* qptr = p.q + ((b * p.heads_q + hq) * p.seq_q) * D;
    const float* kptr = p.k + ((b * p.heads_kv + hkv) * p.seq_kv) * D;
    const float* vptr = p.v + ((b * p.heads_kv + hkv) * p.seq_kv) * D;
    const uint8_t* keep = p.key_keep ? p.key_keep + b * p.keep_batch_stride : nullptr;

    for (int i = threadIdx.x; i < kSimtRows * D; i += blockDim.x) {
        const int64_t r = row0 + i / D;
        Qs[i] = (r < p.seq_q) ? qptr[r * D + i % D] : 0.f;
    }

    int64_t k_hi = p.seq_kv;
    if (p.kv_lens && p.kv_lens[b] < k_hi) k_hi = p.kv_lens[b] < 0 ? 0 : p.kv_lens[b];
    const int64_t q_off = p.q_offsets ? p.q_offsets[b] : 0;  // query row i sits at key position i + q_off
    int64_t k_loop = k_hi;
    if (p.causal) {
        int64_t last = row0 + kSimtRows;  // keys <= position of the last query row of the CTA
        if (last > p.seq_q) last = p.seq_q;
        last += q_off;
        if (last < 0) last = 0;
        if (last < k_loop) k_loop = last;
    }

    float m = -INFINITY, l = 0.f;
    float o[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) o[i] = 0.f;

    for (int64_t kj = 0; kj < k_loop; kj += kSimtKeys) {
        __syncthreads();
        for (int i = threadIdx.x; i < kSimtKeys * D; i += blockDim.x) {
            const int r = i / D, d = i % D;
            const bool in = kj + r < k_hi;
            Ks[r * (D + 1) + d] = in ? kptr[(kj + r) * D + d] : 0.f;
            Vs[r * D + d] = in ? vptr[(kj + r) * D + d] : 0.f;
        }
        __syncthreads();
        if (!row_valid) continue;

        const int64_t key = kj + lane;
        float s = 0.f;
        const float* qrow = Qs + warp * D;
        const float* krow = Ks + lane * (D + 1);
        for (int d = 0; d < D; ++d) s = fmaf(qrow[d], krow[d], s);
        s *= p.scale;
        bool masked = key >= k_hi;
        if (p.causal && key > qi + q_off) masked = true;
        if (keep && key < p.seq_kv && !keep[key]) masked = true;
        if (masked) s = -INFINITY;

        float m_tile = s;
#pragma unroll
        for (int off = 16; off; off >>= 1) m_tile = fmaxf(m_tile, __shfl_xor_sync(kFullMask, m_tile, off));
        const float m_new = fmaxf(m, m_tile);
        const float m_use = (m_new == -INFINITY) ? 0.f : m_new;
        const float alpha = (m == -INFINITY) ? 0.f : expf(m - m_use);
        const float pe = masked ? 0.f : expf(s - m_use);
        float psum = pe;
#pragma unroll
        for (int off = 16; off; off >>= 1) psum += __shfl_xor_sync(kFullMask, psum, off);
        l = l * alpha + psum;
        m = m_new;
#pragma unroll
        for (int i = 0; i < 8; ++i) o[i] *= alpha;
        for (int jj = 0; jj < kSimtKeys; ++jj) {
            const float pj = __shfl_sync(kFullMask, pe, jj);
            const float* vrow = Vs + jj * D;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int d = lane + 32 * i;
                if (d < D) o[i] = fmaf(pj, vrow[d], o[i]);
            }
        }
    }

    if (!row_valid) return;
    float* dst = p.out + ((b * p.heads_q + hq) * p.seq_q + qi) * D;
    const bool ok = (l > 0.f) && isfinite(l);  // cpu_forward.rs:411
    const float inv = ok ? 1.f / l : 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int d = lane + 32 * i;
        if (d < D) dst[d] = ok ? o[i] * inv : NAN;
    }
    if (p.lse && lane == 0)
        p.lse[(b * p.heads_q + hq) * p.seq_q + qi] = (l > 0.f) ? m + logf(l) : (l == 0.f ? -INFINITY : NAN);
}

// ---------------------------------------------------------------------------------------------
// Register-tiled variant: a CTA owns 64 query rows and walks the keys in tiles of 64; see simt_tile.cuh for the
// split of the two products.  Same recurrence, masks and NaN rules as the kernel above.  With G = 2 groups each has
// its own K and V buffers and its own running maximum, sum and output, merged at the end: at these sizes (a few
// hundred row blocks) the launch lasts as long as its longest block, and two groups walk that in half the steps.
// Head dims above 128 leave no room for the second group's tiles.  K and V have one buffer each per group: K of the
// next tile is copied while P V runs, V while Q K^T runs, so two group barriers per tile order everything.  The row
// sum stays per thread until the end.  NC = ceil(D / 32) column groups of the output.
// Against the 256-thread kernel with 4 x 4 scores a thread that this replaces (scalar loads transposed into shared
// memory with 16-way conflicts): B=1 H=8 N=2048 D=64 causal 371 -> 113 us (38 TFLOP/s), B=2 H=16 N=1000 D=128 causal
// 520 -> 218 us, B=4 H=16 N=1024 D=64 656 -> 408 us (42 TFLOP/s of the FP32 pipe's 74).
// Launches of few row blocks leave SMs idle while each block walks its keys alone; there a cluster of 2, 4 or 8 CTAs shares
// them (kSplit): each takes every split-th pair of tiles, leaves its partial rows in shared memory, and merges 64 / split rows out
// of all of them.  (N=2048 D=64 causal, H=1 112 -> 37 us, H=2 112 -> 52; H=4 N=600 D=80 without a mask 51 -> 41; H=2 64 rows
// against 4096 keys D=128 402 -> 64; the merge costs about half a step.)
__device__ __forceinline__ void f32_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ float f32_remote(const float* a, int rank) {
    uint32_t r;
    float v;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"((uint32_t)__cvta_generic_to_shared(a)), "r"(rank));
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(r) : "memory");
    return v;
}

template <int NC, int G, bool kSplit>
__global__ void __launch_bounds__(simt::kGroup * G, 1)
prefill_f32_tiled_kernel(const SimtParams p, const bool vec, const bool pairs, const int64_t row_blocks) {
    using namespace simt;
    extern __shared__ __align__(16) float smem[];
    const int group = G == 1 ? 0 : (int)threadIdx.x >> 7, tid = (int)threadIdx.x & (kGroup - 1);
    constexpr int kPitch = pitch_of(NC * 32), tile = tile_floats(kRows, kPitch);
    const int D = p.dim;
    float* Qs = smem;
    float* Ks = Qs + tile + group * (2 * tile + kWFloats);
    float* Vs = Ks + tile;
    float* Ws = Vs + tile;
    const Lane ln;
    const Share share = Share::of<kGroup>(tid, D, vec), q_share = Share::of<kGroup * G>((int)threadIdx.x, D, vec);

    // CTA order: under a causal mask the longest row blocks of all heads first
    const int rank = kSplit ? (int)blockIdx.x % p.split : 0, split = kSplit ? p.split : 1;
    const int64_t n_bh = (int64_t)gridDim.x / split / row_blocks, x = blockIdx.x / split;
    const int64_t bh = p.causal ? x % n_bh : x / row_blocks;
    const int64_t row0 = (p.causal ? row_blocks - 1 - x / n_bh : x % row_blocks) * kRows;
    const int64_t b = bh / p.heads_q, hq = bh % p.heads_q, hkv = hq / (p.heads_q / p.heads_kv);
    const float* kptr = p.k + ((b * p.heads_kv + hkv) * p.seq_kv) * D;
    const float* vptr = p.v + ((b * p.heads_kv + hkv) * p.seq_kv) * D;
    const uint8_t* keep = p.key_keep ? p.key_keep + b * p.keep_batch_stride : nullptr;

    int64_t k_hi = p.seq_kv;
    if (p.kv_lens && p.kv_lens[b] < k_hi) k_hi = p.kv_lens[b] < 0 ? 0 : p.kv_lens[b];
    const int64_t q_off = p.q_offsets ? p.q_offsets[b] : 0;  // query row i sits at key position i + q_off
    int64_t k_loop = k_hi;
    if (p.causal) {
        int64_t last = row0 + kRows;  // keys <= position of the last query row of the CTA
        if (last > p.seq_q) last = p.seq_q;
        last += q_off;
        if (last < 0) last = 0;
        if (last < k_loop) k_loop = last;
    }

    const float c2 = p.scale * kLog2e;
    float m[8], l[8];  // maximum (log2 units) and this thread's share of the sum
    float2 z[4][2 * NC];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        m[i] = -INFINITY;
        l[i] = 0.f;
    }
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < 2 * NC; ++c) z[r][c] = make_float2(0.f, 0.f);

    const int64_t first = (int64_t)(rank * G + group) * kRows, step = (int64_t)(G * split) * kRows;
    load_tile<kRows, kGroup * G, kPitch>(Qs, p.q + (bh * p.seq_q) * D, row0, p.seq_q, D, vec, q_share);
    if (first < k_loop) load_tile<kRows, kGroup, kPitch>(Ks, kptr, first, k_hi, D, vec, share);
    cp_async_commit();
    cp_async_wait<0>();
    __syncthreads();  // both groups have copied their share of Q
    for (int64_t kj = first; kj < k_loop; kj += step) {
        cp_async_wait<0>();
        group_sync(group);  // this tile's K is visible and nobody reads the last tile's V any more
        load_tile<kRows, kGroup, kPitch>(Vs, vptr, kj, k_hi, D, vec, share);
        cp_async_commit();
        float s[8][4];
        product<4, kPitch>(s, Qs, Ks, D, ln);
        cp_async_wait<0>();
        group_sync(group);  // V is visible, K is free
        if (kj + step < k_loop) {
            load_tile<kRows, kGroup, kPitch>(Ks, kptr, kj + step, k_hi, D, vec, share);
            cp_async_commit();
        }
        // ---- masks, in tiles that the length, the diagonal or flags cut
        if (keep || kj + kRows > k_hi || (p.causal && kj + kRows - 1 > row0 + q_off)) {
            const int hi = (int)(k_hi - kj < kRows ? k_hi - kj : kRows);
            const int64_t d64 = row0 + q_off - kj;
            const int diag = (int)(d64 < -kRows ? -kRows : d64 > kRows ? kRows : d64);  // tile row r sees keys <= r + diag
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int key = ln.h + 16 * j;
                const bool off = key >= hi || (keep && !keep[kj + key]);
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    if (off || (p.causal && key > ln.g + 8 * i + diag)) s[i][j] = -INFINITY;
            }
        }
        // ---- online softmax in units of log2; the 16 lanes of a row agree on the maximum through shuffles
        float2 alpha[4];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const float mt = fmaxf(fmaxf(s[i][0], s[i][1]), fmaxf(s[i][2], s[i][3]));
            const float m_new = fmaxf(m[i], row_max(mt) * c2);
            const float m_use = (m_new == -INFINITY) ? 0.f : m_new;
            const float a = exp2f(m[i] - m_use);  // 0 while m is -inf
#pragma unroll
            for (int j = 0; j < 4; ++j) s[i][j] = exp2f(fmaf(s[i][j], c2, -m_use));  // masked: 0
            l[i] = l[i] * a + ((s[i][0] + s[i][1]) + (s[i][2] + s[i][3]));
            m[i] = m_new;
            if (i & 1) alpha[i >> 1].y = a;
            else alpha[i >> 1].x = a;
        }
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int c = 0; c < 2 * NC; ++c) z[r][c] = __fmul2_rn(z[r][c], alpha[r]);
        accumulate<4, NC, kPitch>(z, s, Vs, Ws, ln);
    }

    // ---- the two groups' partial rows: the second hands over (max, per-thread sum, output), the first merges
    if (G == 2) {
        __syncthreads();  // both are done with their tiles; the exchange starts at the first group's K
        float2* ex = reinterpret_cast<float2*>(Qs + tile);
        if (group == 1) {
            put(ex, z, tid);
#pragma unroll
            for (int i = 0; i < 8; ++i) ex[(8 * NC + i) * kGroup + tid] = make_float2(m[i], l[i]);
        }
        __syncthreads();
        if (!kSplit && group == 1) return;
        float2 f0[4], f1[4];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const float2 o = ex[(8 * NC + i) * kGroup + tid];
            const float mm = fmaxf(m[i], o.x), m_use = (mm == -INFINITY) ? 0.f : mm;
            const float a = exp2f(m[i] - m_use), c = exp2f(o.x - m_use);
            l[i] = l[i] * a + o.y * c;  // (a NaN sum stays one: NaN * 0)
            m[i] = mm;
            if (i & 1) { f0[i >> 1].y = a; f1[i >> 1].y = c; }
            else { f0[i >> 1].x = a; f1[i >> 1].x = c; }
        }
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int c = 0; c < 2 * NC; ++c)
                z[r][c] = __ffma2_rn(f0[r], z[r][c], __fmul2_rn(f1[r], ex[(r * 2 * NC + c) * kGroup + tid]));
    }

    if constexpr (kSplit) {
        // ---- the cluster's partial rows, over the Q tile; (max, sum) of each behind what the groups have exchanged, which
        // other warps may still be reading (4224 of the first group's 7168 floats at the narrowest width)
        float* const part = Qs;
        float* const ml = Qs + tile + (8 * NC + 8) * 2 * kGroup;
        if (group == 0) {
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const float sum = row_sum(l[i]);
                const int r = ln.g + 8 * i;
                store_row<NC>(part + r * kPitch, z, i, 1.f, 0, D, D % 2 == 0, ln);
                if (ln.h == 0) ml[2 * r] = m[i], ml[2 * r + 1] = sum;
            }
        }
        f32_cluster_sync();
        const int rows = kRows / split;
        for (int i = (int)threadIdx.x; i < rows * D; i += kGroup * G) {
            const int r = rank * rows + i / D, d = i % D;
            if (row0 + r >= p.seq_q) break;  // (rows ascend)
            float ms[8], ls[8], zs[8], mm = -INFINITY;
#pragma unroll
            for (int c = 0; c < 8; ++c)
                if (c < split) {
                    ms[c] = f32_remote(ml + 2 * r, c);
                    ls[c] = f32_remote(ml + 2 * r + 1, c);
                    zs[c] = f32_remote(part + r * kPitch + d, c);
                    mm = fmaxf(mm, ms[c]);
                }
            const float m_use = (mm == -INFINITY) ? 0.f : mm;
            float sum = 0.f, o = 0.f;
#pragma unroll
            for (int c = 0; c < 8; ++c)
                if (c < split) {
                    const float w = exp2f(ms[c] - m_use);
                    sum = fmaf(ls[c], w, sum);  // (a NaN sum stays one: NaN * 0)
                    o = fmaf(zs[c], w, o);
                }
            const bool ok = (sum > 0.f) && isfinite(sum);  // cpu_forward.rs:411
            const int64_t qi = row0 + r;
            p.out[(bh * p.seq_q + qi) * D + d] = o * (ok ? 1.f / sum : NAN);
            if (p.lse && d == 0)
                p.lse[bh * p.seq_q + qi] = (sum > 0.f) ? fmaf(mm, kLn2, logf(sum)) : (sum == 0.f ? -INFINITY : NAN);
        }
        f32_cluster_sync();  // no CTA leaves while its partial rows are being read
        return;
    } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const float sum = row_sum(l[i]);
        const int64_t qi = row0 + ln.g + 8 * i;
        if (qi >= p.seq_q) continue;
        const bool ok = (sum > 0.f) && isfinite(sum);  // cpu_forward.rs:411
        store_row<NC>(p.out + (bh * p.seq_q + qi) * D, z, i, ok ? 1.f / sum : NAN, 0, D, pairs, ln);
        if (p.lse && ln.h == 0)
            p.lse[bh * p.seq_q + qi] = (sum > 0.f) ? fmaf(m[i], kLn2, logf(sum)) : (sum == 0.f ? -INFINITY : NAN);
    }
    }
}

template <int NC, int G>
constexpr int f32_tiled_bytes() {
    return (int)sizeof(float) * ((1 + 2 * G) * simt::tile_floats(simt::kRows, simt::pitch_of(NC * 32)) + G * simt::kWFloats);
}

template <int NC, int G, bool kSplit>
static cudaError_t launch_tiled_s(const SimtParams& p, int64_t n, bool vec, bool pairs, int64_t row_blocks, cudaStream_t stream) {
    cudaError_t e = set_max_dynamic_smem_once<prefill_f32_tiled_kernel<NC, G, kSplit>>(f32_tiled_bytes<NC, G>());
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(n * p.split));
    cfg.blockDim = dim3(simt::kGroup * G);
    cfg.dynamicSmemBytes = f32_tiled_bytes<NC, G>();
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    if (kSplit) {
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = (unsigned)p.split;
        attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
    }
    return cudaLaunchKernelEx(&cfg, prefill_f32_tiled_kernel<NC, G, kSplit>, p, vec, pairs, row_blocks);
}

// CTAs that clusters of `split` CTAs of the widest kernel can have resident on the current device (one CTA per SM; GPCs hold
// whole clusters only).  Asked once per device and size.
static int f32_cluster_slots(int split) {
    static std::atomic<int> known[64][3];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
    std::atomic<int>& slot = known[dev][split == 2 ? 0 : split == 4 ? 1 : 2];
    const int have = slot.load(std::memory_order_relaxed);
    if (have > 0) return have - 1;
    int n = 0;
    if (set_max_dynamic_smem_once<prefill_f32_tiled_kernel<4, 2, true>>(f32_tiled_bytes<4, 2>()) == cudaSuccess) {
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = (unsigned)split;
        attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)(split * 256));
        cfg.blockDim = dim3(simt::kGroup * 2);
        cfg.dynamicSmemBytes = f32_tiled_bytes<4, 2>();
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        if (cudaOccupancyMaxActiveClusters(&n, prefill_f32_tiled_kernel<4, 2, true>, &cfg) != cudaSuccess) {
            cudaGetLastError();
            n = 0;
        }
    }
    slot.store(n * split + 1, std::memory_order_relaxed);
    return n * split;
}

template <int NC, int G>
static cudaError_t launch_tiled(SimtParams p, int64_t batch, cudaStream_t stream) {
    const int64_t row_blocks = (p.seq_q + simt::kRows - 1) / simt::kRows, n = row_blocks * p.heads_q * batch;
    if (n > 0x7fffffff) return cudaErrorInvalidValue;
    const uintptr_t in = reinterpret_cast<uintptr_t>(p.q) | reinterpret_cast<uintptr_t>(p.k) | reinterpret_cast<uintptr_t>(p.v);
    const bool vec = p.dim % 4 == 0 && (in & 15) == 0;
    const bool pairs = p.dim % 2 == 0 && (reinterpret_cast<uintptr_t>(p.out) & 7) == 0;
    // How many CTAs share the keys of a row block: the launch lasts as long as its longest CTA or as the SMs' share of all,
    // whichever is more (causal blocks are started heaviest first and fill up to within 8 %, equal ones come in whole waves).
    // In us: a step of 64 keys per group, per CTA, and for the merge across a cluster.
    p.split = 1;
    if constexpr (G == 2) {
        // RT_ATTN_PREFILL_F32_CLUSTER=1|2|4|8 takes that many for every launch (read once per process).
        static const int env = [] {
            const char* e = getenv("RT_ATTN_PREFILL_F32_CLUSTER");
            const int c = e ? atoi(e) : 0;
            return c == 1 || c == 2 || c == 4 || c == 8 ? c : 0;
        }();
        if (env > 0) {
            if (n * env <= 0x7fffffff && (env == 1 || f32_cluster_slots(env) > 0)) p.split = env;
        } else if (n < 2 * (int64_t)sm_count()) {
            const double step = 1.0 + 0.1 * p.dim, cta = 3.0, merge = 4.0;
            const int64_t all = (p.seq_kv + simt::kRows - 1) / simt::kRows,
                          off = p.causal && p.q_offsets && p.seq_kv > p.seq_q ? p.seq_kv - p.seq_q : 0;
            double best = 0;
            for (int c = 1; c <= 8; c *= 2) {
                const int64_t slots = c == 1 ? sm_count() : f32_cluster_slots(c) / c;
                if (slots == 0 || all < 2 * c) break;
                double sum = 0, mx = 0;
                for (int64_t i = 0; i < row_blocks; ++i) {
                    const int64_t tiles = p.causal ? std::min(all, (off + std::min((i + 1) * simt::kRows, p.seq_q) + simt::kRows - 1) / simt::kRows) : all;
                    const double t = (double)((tiles + 2 * c - 1) / (2 * c)) * step + cta + (c > 1 ? merge : 0.0);
                    sum += t;
                    mx = std::max(mx, t);
                }
                const int64_t heads = n / row_blocks;
                const double t = p.causal ? std::max(mx, 1.08 * sum * (double)heads / (double)slots) : mx * (double)((n + slots - 1) / slots);
                if (c == 1 || t < best) best = t, p.split = c;
            }
        }
        if (p.split > 1) return launch_tiled_s<NC, G, true>(p, n, vec, pairs, row_blocks, stream);
    }
    return launch_tiled_s<NC, G, false>(p, n, vec, pairs, row_blocks, stream);
}

cudaError_t launch_prefill_f32(const float* q, const float* k, const float* v, float* out, float* lse,
                               int64_t batch, int64_t heads_q, int64_t heads_kv, int64_t seq_q,
                               int64_t seq_kv, int dim, int causal, const int32_t* kv_lens,
                               const int32_t* q_offsets, const uint8_t* key_keep, int64_t keep_batch_stride,
                               float scale, cudaStream_t stream) {
    if (batch == 0 || heads_q == 0 || seq_q == 0) return cudaSuccess;
    SimtParams p{q, k, v, out, lse, heads_q, heads_kv, seq_q, seq_kv, dim, causal, kv_lens, q_offsets, key_keep,
                 keep_batch_stride, scale, 1};
    // The register-tiled kernel is the path for 16 query rows and more; a decode-shaped call (a few rows against
    // a long cache) would waste most of its 64-row tile and keeps the warp-per-row kernel, which
    // RT_ATTN_PREFILL_F32_IMPL=rows selects for every shape (comparisons).
    static const bool rows_impl = [] {
        const char* e = getenv("RT_ATTN_PREFILL_F32_IMPL");
        return e && e[0] == 'r';
    }();
    if (!rows_impl && dim <= 256 && seq_q >= 16) {
        if (dim <= 32) return launch_tiled<1, 2>(p, batch, stream);
        if (dim <= 64) return launch_tiled<2, 2>(p, batch, stream);
        if (dim <= 96) return launch_tiled<3, 2>(p, batch, stream);
        if (dim <= 128) return launch_tiled<4, 2>(p, batch, stream);
        return launch_tiled<8, 1>(p, batch, stream);
    }
    const size_t smem = sizeof(float) * ((size_t)kSimtKeys * (dim + 1) + (size_t)kSimtKeys * dim +
                                         (size_t)kSimtRows * dim);
    cudaError_t e = cudaFuncSetAttribute(prefill_f32_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)smem);
    if (e != cudaSuccess) return e;
    const int64_t row_blocks = (seq_q + kSimtRows - 1) / kSimtRows;
    if (row_blocks > 0x7fffffff || heads_q > 65535 || batch > 65535) return cudaErrorInvalidValue;
    dim3 grid((unsigned)row_blocks, (unsigned)heads_q, (unsigned)batch);
    prefill_f32_kernel<<<grid, kSimtRows * 32, smem, stream>>>(p);
    return cudaGetLastError();
}

__global__ void f32_to_bf16_kernel(const float* __restrict__ src, __nv_bfloat16* __restrict__ dst, int64_t n) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride)
        dst[i] = __float2bfloat16_rn(src[i]);
}

__global__ void bf16_to_f32_kernel(const __nv_bfloat16* __restrict__ src, float* __restrict__ dst, int64_t n) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride)
        dst[i] = __bfloat162float(src[i]);
}

static unsigned grid_for(int64_t n) {
    int64_t g = (n + 255) / 256;
    const int64_t cap = (int64_t)sm_count() * 16;
    return (unsigned)(g > cap ? cap : (g < 1 ? 1 : g));
}

cudaError_t launch_f32_to_bf16(const float* src, void* dst, int64_t n, cudaStream_t stream) {
    if (n == 0) return cudaSuccess;
    f32_to_bf16_kernel<<<grid_for(n), 256, 0, stream>>>(src, (__nv_bfloat16*)dst, n);
    return cudaGetLastError();
}

cudaError_t launch_bf16_to_f32(const void* src, float* dst, int64_t n, cudaStream_t stream) {
    if (n == 0) return cudaSuccess;
    bf16_to_f32_kernel<<<grid_for(n), 256, 0, stream>>>((const __nv_bfloat16*)src, dst, n);
    return cudaGetLastError();
}

}  // namespace rt
