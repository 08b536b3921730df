// f32 flash-attention backward on CUDA cores: (dQ, dK, dV) from Q, K, V, O, dO and the saved
// row statistics LSE = m + ln(l) of the forward pass.
//
// Replaces rustorch_attention::flash_backward (crates/rustorch-attention/src/cpu_backward.rs:46-185),
// which recomputes the full N x N probability matrix per (batch, head).  Same math (:16-27):
//   P = exp(scale * Q K^T - LSE),  dV = P^T dO,  dP = dO V^T,
//   dS = P o (dP - delta),  delta_i = sum_j P_ij dP_ij = dO_i . O_i,
//   dQ = scale * dS K,  dK = scale * dS^T Q
// evaluated tile by tile, so nothing of size N x N is stored.  Deterministic, without atomics: a CTA owns 64 query
// rows and accumulates dQ over the key tiles, or owns 64 key rows and accumulates dK and dV over the query tiles
// (recomputing S and dP).  Both kinds run in one launch, so that one side's long rows fill the other side's tail.
// The products are the register-tiled ones of simt_tile.cuh.  A causal launch skips the tiles above the diagonal.
#include "common.cuh"
#include "kernels.h"
#include "simt_tile.cuh"

namespace rt {

struct BwdParams {
    const float *q, *k, *v, *out, *d_out, *lse;
    float *dq, *dk, *dv, *delta;
    int64_t seq;
    int dim, causal;
    float scale;
};

// delta_i = dO_i . O_i (the row sum of P o dP), one warp per row.
__global__ void __launch_bounds__(256) bwd_delta_kernel(const float* __restrict__ out, const float* __restrict__ d_out,
                                                        float* __restrict__ delta, int64_t rows, int dim) {
    const int64_t row = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (row >= rows) return;
    float acc = 0.f;
    for (int d = lane; d < dim; d += 32) acc = fmaf(out[row * dim + d], d_out[row * dim + d], acc);
#pragma unroll
    for (int off = 16; off; off >>= 1) acc += __shfl_xor_sync(kFullMask, acc, off);
    if (lane == 0) delta[row] = acc;
}

// Tiles hold whole rows: the gradient columns of a launch with one column group, all 256 with two.
template <int NC, int G>
__host__ __device__ constexpr int bwd_pitch() { return simt::pitch_of(G == 1 ? 256 : NC * 32); }

// One CTA's 64 rows of one side.  X1, X2 are its own rows of (Q, dO) or (K, V), Y1, Y2 the other side's tiles of
// (K, V) or (Q, dO), 16 J rows at a time; col0 is the first of the NC x 32 gradient columns it accumulates.
// Every step computes dP (Y2) before S (Y1) and accumulates with Y2 before Y1, so each single-buffered tile is
// copied while a product that does not need it runs.  With G = 2 groups each takes every second tile of the other
// side, with buffers and sums of its own; the first adds the second's sums at the end.
template <int NC, int J, int G, bool kKeySide>
__device__ __forceinline__ void bwd_rows(const BwdParams& p, float* smem, int64_t bh, int64_t own0, int col0, bool vec,
                                         bool pairs) {
    using namespace simt;
    const int D = p.dim;
    const int group = G == 1 ? 0 : (int)threadIdx.x >> 7, tid = (int)threadIdx.x & (kGroup - 1);
    constexpr int kPitch = bwd_pitch<NC, G>(), x_tile = tile_floats(kRows, kPitch), y_tile = tile_floats(16 * J, kPitch);
    float* X1 = smem;
    float* X2 = X1 + x_tile;
    float* Y1 = X2 + x_tile + group * (2 * y_tile + kWFloats);
    float* Y2 = Y1 + y_tile;
    float* Ws = Y2 + y_tile;
    const Lane ln;
    const Share share = Share::of<kGroup>(tid, D, vec), x_share = Share::of<kGroup * G>((int)threadIdx.x, D, vec);
    const int64_t N = p.seq, base = bh * N * D;
    const float* lse = p.lse + bh * N;
    const float* delta = p.delta + bh * N;
    const float* oth1 = (kKeySide ? p.q : p.k) + base;
    const float* oth2 = (kKeySide ? p.d_out : p.v) + base;

    // the other side's rows that the own rows meet: keys up to the last own query, queries from the first own key on
    const int64_t t_lo = (kKeySide && p.causal) ? own0 / (16 * J) * (16 * J) : 0;
    const int64_t t_hi = (!kKeySide && p.causal && own0 + kRows < N) ? own0 + kRows : N;

    const int64_t first = t_lo + group * 16 * J, step = (int64_t)G * 16 * J;
    load_tile<kRows, kGroup * G, kPitch>(X1, (kKeySide ? p.k : p.q) + base, own0, N, D, vec, x_share);
    load_tile<kRows, kGroup * G, kPitch>(X2, (kKeySide ? p.v : p.d_out) + base, own0, N, D, vec, x_share);
    if (first < t_hi) load_tile<16 * J, kGroup, kPitch>(Y2, oth2, first, N, D, vec, share);
    cp_async_commit();

    // LSE in units of log2.  A row without a visible key has LSE = -inf: +inf in its place makes every probability 0.
    auto lse2_of = [&](int64_t r) {
        const float x = r < N ? lse[r] : INFINITY;
        return x == -INFINITY ? INFINITY : x * kLog2e;
    };
    auto delta_of = [&](int64_t r) { return r < N ? delta[r] : 0.f; };
    const float c2 = p.scale * kLog2e;
    float r_lse[kKeySide ? 1 : 8], r_delta[kKeySide ? 1 : 8];
    if (!kKeySide) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            r_lse[i] = lse2_of(own0 + ln.g + 8 * i);
            r_delta[i] = delta_of(own0 + ln.g + 8 * i);
        }
    }
    float2 z1[4][2 * NC], z2[kKeySide ? 4 : 1][2 * NC];  // dQ, or dK and dV
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < 2 * NC; ++c) z1[r][c] = z2[kKeySide ? r : 0][c] = make_float2(0.f, 0.f);

    cp_async_wait<0>();
    __syncthreads();  // both groups have copied their share of the own rows
    for (int64_t t0 = first; t0 < t_hi; t0 += step) {
        const bool more = t0 + step < t_hi;
        float c_lse[kKeySide ? J : 1], c_delta[kKeySide ? J : 1];
        if (kKeySide) {
#pragma unroll
            for (int j = 0; j < J; ++j) {
                c_lse[j] = lse2_of(t0 + ln.h + 16 * j);
                c_delta[j] = delta_of(t0 + ln.h + 16 * j);
            }
        }
        cp_async_wait<0>();
        group_sync(group);  // Y2 is visible, the last step's Y1 is free
        load_tile<16 * J, kGroup, kPitch>(Y1, oth1, t0, N, D, vec, share);
        cp_async_commit();
        float dp[8][J], pr[8][J];
        product<J, kPitch>(dp, X2, Y2, D, ln);
        cp_async_wait<0>();
        group_sync(group);  // Y1 is visible (and, on the query side, Y2 free)
        if (!kKeySide && more) {
            load_tile<16 * J, kGroup, kPitch>(Y2, oth2, t0 + step, N, D, vec, share);
            cp_async_commit();
        }
        product<J, kPitch>(pr, X1, Y1, D, ln);

#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < J; ++j)
                pr[i][j] = exp2f(fmaf(pr[i][j], c2, -(kKeySide ? c_lse[j] : r_lse[i])));
        if (t0 + 16 * J > N || (p.causal && (kKeySide ? t0 < own0 + kRows : t0 + 16 * J > own0))) {
            const int hi = (int)(N - t0 < 16 * J ? N - t0 : 16 * J);
            const int diag = (int)(own0 - t0);  // within a tile of zero wherever the causal mask cuts
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < J; ++j) {
                    const int own = ln.g + 8 * i + diag, oth = ln.h + 16 * j;
                    if (oth >= hi || (p.causal && (kKeySide ? own > oth : oth > own))) pr[i][j] = 0.f;
                }
        }
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < J; ++j) dp[i][j] = pr[i][j] * (dp[i][j] - (kKeySide ? c_delta[j] : r_delta[i]));
        if constexpr (kKeySide) {
            accumulate<J, NC, kPitch>(z2, pr, Y2 + col0, Ws, ln);  // dV += P^T dO
            group_sync(group);                                // Y2 is free
            if (more) {
                load_tile<16 * J, kGroup, kPitch>(Y2, oth2, t0 + step, N, D, vec, share);
                cp_async_commit();
            }
        }
        accumulate<J, NC, kPitch>(z1, dp, Y1 + col0, Ws, ln);  // dQ += dS K, or dK += dS^T Q
    }

    if (G == 2) {
        __syncthreads();  // both are done with their tiles; the exchange starts at the first group's Y1
        float2* ex = reinterpret_cast<float2*>(X2 + x_tile);
        if (group == 1) {
            put(ex, z1, tid);
            if constexpr (kKeySide) put(ex + 8 * NC * kGroup, z2, tid);
        }
        __syncthreads();
        if (group == 1) return;
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int c = 0; c < 2 * NC; ++c) {
                z1[r][c] = __fadd2_rn(z1[r][c], ex[(r * 2 * NC + c) * kGroup + tid]);
                if constexpr (kKeySide) z2[r][c] = __fadd2_rn(z2[r][c], ex[(8 * NC + r * 2 * NC + c) * kGroup + tid]);
            }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int64_t r = own0 + ln.g + 8 * i;
        if (r >= N) continue;
        store_row<NC>((kKeySide ? p.dk : p.dq) + base + r * D, z1, i, p.scale, col0, D, pairs, ln);
        if constexpr (kKeySide) store_row<NC>(p.dv + base + r * D, z2, i, 1.f, col0, D, pairs, ln);
    }
}

// CTA order: rank (0 = most other-side tiles under a causal mask), then side, column group, head.
// Against the kernel that gave every own row to one warp (a shared-memory load per multiply-add): B=2 H=8 N=1000 D=64
// causal 1814 -> 193 us, B=4 H=16 N=1024 D=64 12.1 -> 1.35 ms (45 TFLOP/s executed), B=4 H=16 N=161 D=80 causal 312 -> 62 us.
// Scalar multiply-adds in place of the packed ones were 4 % slower, one group per CTA (two CTAs an SM) 15 % at N=1000.
template <int NC, int J, int G>
__global__ void __launch_bounds__(simt::kGroup * G, 1)
bwd_tiled_kernel(const BwdParams p, const bool vec, const bool pairs, const int n_tiles, const int n_bh, const int groups) {
    extern __shared__ __align__(16) float smem[];
    const int x = (int)blockIdx.x;
    const int bh = x % n_bh, rest = x / n_bh, col0 = rest % groups * (NC * 32), side = rest / groups & 1,
              rank = rest / groups / 2;
    if (side == 0)
        bwd_rows<NC, J, G, true>(p, smem, bh, (int64_t)rank * simt::kRows, col0, vec, pairs);
    else
        bwd_rows<NC, J, G, false>(p, smem, bh, (int64_t)(p.causal ? n_tiles - 1 - rank : rank) * simt::kRows, col0, vec,
                                  pairs);
}

template <int NC, int J, int G>
static cudaError_t launch_bwd_tiled(const BwdParams& p, int64_t bh, cudaStream_t stream) {
    constexpr int kPitch = bwd_pitch<NC, G>(),
                  bytes = (int)sizeof(float) * (2 * simt::tile_floats(simt::kRows, kPitch) +
                                                G * (2 * simt::tile_floats(16 * J, kPitch) + simt::kWFloats));
    cudaError_t e = set_max_dynamic_smem_once<bwd_tiled_kernel<NC, J, G>>(bytes);
    if (e != cudaSuccess) return e;
    const int64_t n_tiles = (p.seq + simt::kRows - 1) / simt::kRows;
    const int groups = (p.dim + NC * 32 - 1) / (NC * 32);
    const int64_t n = 2 * n_tiles * bh * groups;
    if (n > 0x7fffffff) return cudaErrorInvalidValue;
    const uintptr_t in = reinterpret_cast<uintptr_t>(p.q) | reinterpret_cast<uintptr_t>(p.k) |
                         reinterpret_cast<uintptr_t>(p.v) | reinterpret_cast<uintptr_t>(p.d_out);
    const uintptr_t outs = reinterpret_cast<uintptr_t>(p.dq) | reinterpret_cast<uintptr_t>(p.dk) | reinterpret_cast<uintptr_t>(p.dv);
    const bool vec = p.dim % 4 == 0 && (in & 15) == 0, pairs = p.dim % 2 == 0 && (outs & 7) == 0;
    bwd_tiled_kernel<NC, J, G><<<(unsigned)n, simt::kGroup * G, bytes, stream>>>(p, vec, pairs, (int)n_tiles,
                                                                                         (int)bh, groups);
    return cudaGetLastError();
}

cudaError_t launch_backward_f32(const float* q, const float* k, const float* v, const float* out, const float* d_out,
                                const float* lse, float* dq, float* dk, float* dv, float* delta_ws, int64_t batch,
                                int64_t heads, int64_t seq, int dim, int causal, float scale, cudaStream_t stream) {
    const int64_t bh = batch * heads;
    if (bh == 0 || seq == 0) return cudaSuccess;
    if (bh > 65535) return cudaErrorInvalidValue;
    const int64_t rows = bh * seq;
    bwd_delta_kernel<<<(unsigned)((rows + 7) / 8), 256, 0, stream>>>(out, d_out, delta_ws, rows, dim);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    BwdParams p{q, k, v, out, d_out, lse, dq, dk, dv, delta_ws, seq, dim, causal, scale};
    // Tiles of 64 x 64 while the scores of both products fit the registers next to the gradients, 64 x 32 beyond; a
    // head dim above 128 is accumulated in two column groups of 128, and its tiles leave no room for a second group.
    if (dim <= 32) return launch_bwd_tiled<1, 4, 2>(p, bh, stream);
    if (dim <= 64) return launch_bwd_tiled<2, 4, 2>(p, bh, stream);
    if (dim <= 96) return launch_bwd_tiled<3, 2, 2>(p, bh, stream);
    if (dim <= 128) return launch_bwd_tiled<4, 2, 2>(p, bh, stream);
    return launch_bwd_tiled<4, 2, 1>(p, bh, stream);
}

}  // namespace rt
