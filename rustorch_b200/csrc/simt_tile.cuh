// Building blocks of the exact f32 kernels (prefill_simt.cu, backward_simt.cu): 64-row tiles in shared memory, the
// two kinds of product the attention passes are made of, register-tiled on the CUDA cores with packed f32x2 math.
//
// A group is 128 threads; a CTA is one group, or two that share their own 64 rows and take the other side's tiles
// alternately, which halves the CTA's chain of steps (merged at the end, in a fixed order).  Warp w of a group owns
// rows 2w, 2w+1 (mod 8) of a 64-row tile, i.e. 16 rows; inside it a lane has a row class g (2w or 2w + 1) and a column
// class h (0 to 15).  A thread holds rows g + 8 i (i < 8) and, of the other side's tile, rows h + 16 j.  So
//   * tiles stay in their natural [row][d] layout for both products: the score-like product reads 16 bytes along d of
//     8 + J rows for 32 J multiply-adds, the accumulating one 8 scores and the thread's columns of one row per row, so
//     nothing is transposed on the way in, and global -> shared is a plain 16-byte cp.async;
//   * the row pitch is an odd multiple of 16 bytes, so the 8 lanes of a shared-memory wavefront hit 8 different
//     16-byte bank groups;
//   * a score row lives in 16 lanes of one warp: the row maximum is four shuffles, and the scores reach the second
//     product through a warp-private piece of shared memory without a CTA barrier.
// Bound: the FP32 pipe (128 multiply-adds per clock and SM) and, next to it, shared-memory wavefronts (2.7 per 16-byte read);
// with two warps per scheduler the products run at three quarters of the pipe.  What two warps do not hide is the latency of
// the first reads behind a loop's end and the integer work on row addresses: products unrolled 4 and 16 deep over tiles of
// constant pitch take 6 % less than 2 and 4 deep over a pitch that follows the head dim.  (8 deep, or the next step's operands
// read ahead, spill: level and 2 % slower.  A third group at 168 registers 3 % slower; lanes h and h ^ 8 sharing 8 x 8
// scores over half of d each, a third fewer reads per multiply-add but scalar ones, 6 %.)
#pragma once
#include "common.cuh"

namespace rt {
namespace simt {

constexpr int kGroup = 128, kRows = 64;
constexpr int kWKeys = 32, kWPitch = 20;                // one warp's exchange buffer: [32 keys][16 rows + pad]
constexpr int kWFloats = 4 * kWKeys * kWPitch;          // of a group

// Floats between rows of a tile for head dims up to `cols`, an odd multiple of 4.  It is a constant of the kernel, not of
// the call: row offsets are immediates of the loads then and take no registers.
__host__ __device__ constexpr int pitch_of(int cols) { return 4 * ((cols + 3) / 4 | 1); }
// Floats of a tile.
__host__ __device__ constexpr int tile_floats(int rows, int pitch) { return rows * pitch; }

struct Lane {
    int warp, g, h;
    __device__ __forceinline__ Lane() {
        const int t = (int)threadIdx.x & (kGroup - 1);
        warp = t >> 5;
        g = warp * 2 + (t >> 3 & 1);
        h = (t & 7) | (t >> 1 & 8);
    }
};

// Maximum or sum over the 16 lanes that share a row class.
__device__ __forceinline__ float row_max(float x) {
    x = fmaxf(x, __shfl_xor_sync(kFullMask, x, 1));
    x = fmaxf(x, __shfl_xor_sync(kFullMask, x, 2));
    x = fmaxf(x, __shfl_xor_sync(kFullMask, x, 4));
    return fmaxf(x, __shfl_xor_sync(kFullMask, x, 16));
}
__device__ __forceinline__ float row_sum(float x) {
    x += __shfl_xor_sync(kFullMask, x, 1);
    x += __shfl_xor_sync(kFullMask, x, 2);
    x += __shfl_xor_sync(kFullMask, x, 4);
    return x + __shfl_xor_sync(kFullMask, x, 16);
}

// Column (within the accumulated group) of a thread's c-th pair: lanes hold 4 neighbouring columns of every full 64,
// 2 of a last 32.
template <int NC>
__device__ __forceinline__ int pair_col(int c, int h) {
    return c < NC / 2 * 2 ? c / 2 * 64 + h * 4 + c % 2 * 2 : NC / 2 * 64 + h * 2;
}

// Barrier of one group of the CTA.
__device__ __forceinline__ void group_sync(int group) { asm volatile("bar.sync %0, 128;" ::"r"(1 + group) : "memory"); }

__device__ __forceinline__ void cp_async16(float* dst, const float* src, bool in) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src),
                 "r"(in ? 16 : 0)
                 : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int kPending>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(kPending) : "memory");
}

// A thread's share of a tile copy by kThreads threads: column piece c of rows r, r + step, ...  Worked out once, because
// the head dim is a run-time value and a division per 16 bytes costs as much as a fifth of a product.
struct Share {
    int r, c, step;
    template <int kThreads>
    static __device__ __forceinline__ Share of(int tid, int dim, bool vec) {
        const int cpr = vec ? dim / 4 : (dim + 3) & ~3;  // pieces (16 bytes, or single floats) per row, at most 256
        if (cpr >= kThreads) return Share{0, tid, 0};    // a row is one or two rounds of all threads
        const int step = kThreads / cpr, r = tid / cpr;
        return r < step ? Share{r, tid - r * cpr, step} : Share{kRows, 0, step};
    }
};

// Starts the copy of rows [r0, r0 + kTileRows) of a [n_rows, dim] matrix; rows beyond n_rows and the padding up to a
// multiple of 4 columns become zero.  vec: dim is a multiple of 4 and the matrix 16-byte aligned.  The copy is the work
// of kThreads threads, each doing its share; the caller commits.
template <int kTileRows, int kThreads, int pitch>
__device__ __forceinline__ void load_tile(float* tile, const float* src, int64_t r0, int64_t n_rows, int dim, bool vec,
                                          const Share& sh) {
    const int n = (int)(n_rows - r0 < kTileRows ? n_rows - r0 : kTileRows);  // rows that exist (may be negative)
    if (vec) {
        const float* g = src + r0 * dim + sh.c * 4;
        for (int r = sh.r; r < kTileRows; r += sh.step) {
            const bool in = r < n;
            cp_async16(tile + r * pitch + sh.c * 4, in ? g + r * dim : src, in);
        }
    } else {
        const int dp = (dim + 3) & ~3, step = sh.step ? sh.step : 1;
        for (int r = sh.r; r < kTileRows; r += step)
            for (int c = sh.c; c < dp; c += sh.step ? dp : kThreads)
                tile[r * pitch + c] = (r < n && c < dim) ? src[(r0 + r) * dim + c] : 0.f;
    }
}

// t[i][j] = sum over d of X[g + 8 i][d] Y[h + 16 j][d].  Even and odd d accumulate in the two halves of an f32x2.
template <int J, int pitch>
__device__ __forceinline__ void product(float (&t)[8][J], const float* X, const float* Y, int dim, const Lane& ln) {
    const int steps = (dim + 3) / 4;
    const float* x = X + ln.g * pitch;
    const float* y = Y + ln.h * pitch;
    float2 acc[8][J];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < J; ++j) acc[i][j] = make_float2(0.f, 0.f);
#pragma unroll 4
    for (int s = 0; s < steps; ++s) {
        float4 b[J];
#pragma unroll
        for (int j = 0; j < J; ++j) b[j] = *reinterpret_cast<const float4*>(y + j * 16 * pitch + s * 4);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const float4 a = *reinterpret_cast<const float4*>(x + i * 8 * pitch + s * 4);
#pragma unroll
            for (int j = 0; j < J; ++j) {
                acc[i][j] = __ffma2_rn(make_float2(a.x, a.y), make_float2(b[j].x, b[j].y), acc[i][j]);
                acc[i][j] = __ffma2_rn(make_float2(a.z, a.w), make_float2(b[j].z, b[j].w), acc[i][j]);
            }
        }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < J; ++j) t[i][j] = acc[i][j].x + acc[i][j].y;
}

// z[p][c] (+)= sum over the other tile's rows k of t[row][k] Y[k][col]: p = row pair (g + 16 p, g + 16 p + 8), c = 2 cc + e
// stands for column pair_col(cc) + e.  t goes through the warp's exchange buffer, 32 rows of Y at a time.
template <int J, int NC, int pitch>
__device__ __forceinline__ void accumulate(float2 (&z)[4][2 * NC], const float (&t)[8][J], const float* Y, float* w_sm,
                                           const Lane& ln) {
    float* w = w_sm + ln.warp * kWKeys * kWPitch;
    const float* wr = w + (ln.g & 1) * 8;
#pragma unroll
    for (int half = 0; half < J / 2; ++half) {
        __syncwarp();
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            float* dst = w + (ln.h + 16 * u) * kWPitch + (ln.g & 1) * 8;
            const int j = half * 2 + u;
            *reinterpret_cast<float4*>(dst) = make_float4(t[0][j], t[1][j], t[2][j], t[3][j]);
            *reinterpret_cast<float4*>(dst + 4) = make_float4(t[4][j], t[5][j], t[6][j], t[7][j]);
        }
        __syncwarp();
        const float* y = Y + half * 32 * pitch;
#pragma unroll 16
        for (int k = 0; k < kWKeys; ++k) {
            const float4 a = *reinterpret_cast<const float4*>(wr + k * kWPitch);
            const float4 b = *reinterpret_cast<const float4*>(wr + k * kWPitch + 4);
            const float2 rows[4] = {make_float2(a.x, a.y), make_float2(a.z, a.w), make_float2(b.x, b.y), make_float2(b.z, b.w)};
            float2 v[NC];
#pragma unroll
            for (int c = 0; c < NC / 2; ++c) {
                const float4 q = *reinterpret_cast<const float4*>(y + k * pitch + c * 64 + ln.h * 4);
                v[2 * c] = make_float2(q.x, q.y);
                v[2 * c + 1] = make_float2(q.z, q.w);
            }
            if (NC % 2) v[NC - 1] = *reinterpret_cast<const float2*>(y + k * pitch + NC / 2 * 64 + ln.h * 2);
#pragma unroll
            for (int c = 0; c < NC; ++c)
#pragma unroll
                for (int p = 0; p < 4; ++p) {
                    z[p][2 * c] = __ffma2_rn(rows[p], make_float2(v[c].x, v[c].x), z[p][2 * c]);
                    z[p][2 * c + 1] = __ffma2_rn(rows[p], make_float2(v[c].y, v[c].y), z[p][2 * c + 1]);
                }
        }
    }
}

// Lays n f32x2 values of every thread of a group out in shared memory, thread by thread next to each other.
template <int A, int B>
__device__ __forceinline__ void put(float2* dst, const float2 (&z)[A][B], int tid) {
#pragma unroll
    for (int r = 0; r < A; ++r)
#pragma unroll
        for (int c = 0; c < B; ++c) dst[(r * B + c) * kGroup + tid] = z[r][c];
}

// Stores this thread's columns of row i (of the 8) with a factor; col0 is the first column of the accumulated group.
template <int NC>
__device__ __forceinline__ void store_row(float* dst, const float2 (&z)[4][2 * NC], int i, float mul, int col0, int dim,
                                          bool pairs, const Lane& ln) {
#pragma unroll
    for (int c = 0; c < NC; ++c) {
        const int d = col0 + pair_col<NC>(c, ln.h);
        const float a = ((i & 1) ? z[i >> 1][2 * c].y : z[i >> 1][2 * c].x) * mul;
        const float b = ((i & 1) ? z[i >> 1][2 * c + 1].y : z[i >> 1][2 * c + 1].x) * mul;
        if (pairs) {  // dim even and dst 8-byte aligned
            if (d < dim) *reinterpret_cast<float2*>(dst + d) = make_float2(a, b);
        } else {
            if (d < dim) dst[d] = a;
            if (d + 1 < dim) dst[d + 1] = b;
        }
    }
}

}  // namespace simt
}  // namespace rt
