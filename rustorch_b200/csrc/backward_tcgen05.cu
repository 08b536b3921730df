// bf16 flash-attention backward on the Blackwell tensor cores (tcgen05 + TMEM + TMA).
//
// Same math as rustorch_attention::flash_backward (crates/rustorch-attention/src/cpu_backward.rs:16-27,
// 96-189) with the saved row statistics in place of the N x N probability matrix:
//   P = exp(scale * Q K^T - LSE),  dP = dO V^T,  dS = P o (dP - delta),  delta_i = dO_i . O_i,
//   dV = P^T dO,  dQ = scale * dS K,  dK = scale * dS^T Q.
// Two deterministic passes (no atomics, fixed summation order) run in one launch, each on its own CTAs, one per SM, which
// work through a list of tiles (tile_schedule.cuh).  For each tile a CTA takes
// 128 rows of one side, keeps them in shared memory, and walks the other side in 64-row steps that TMA
// streams through a four-slot ring:
//   query side: own X1 = Q_i, X2 = dO_i;  per key tile (Y1 = K_j, Y2 = V_j)
//               T1 = Q K^T, T2 = dO V^T (SS MMAs into TMEM) -> dS (bf16, back into TMEM) -> dQ += dS K_j (TS MMA)
//   key side:   own X1 = K_j, X2 = V_j;   per query tile (Y1 = Q_i, Y2 = dO_i)
//               T1 = K Q^T = S^T, T2 = V dO^T = dP^T -> P^T, dS^T (bf16, into TMEM)
//               -> dV += P^T dO_i, dK += dS^T Q_i (TS MMAs)
// Every product is "own rows x other tile": the score-like ones take both operands K-major from
// 128-byte-swizzled shared memory, the accumulating ones take A from TMEM and the other tile MN-major,
// exactly as TMA lands it (the forward's P V product has the same shape).  The thread that owns TMEM lane
// r owns own-row r: on the query side the statistics (LSE_i, delta_i) are per thread, on the key side
// they belong to the columns and are staged in shared memory per tile.  P and dS are rounded to bf16 for
// the accumulating products, as the forward rounds P.  A causal launch skips the tiles beyond the diagonal.
// An other-side tile is consumed in two 64-row steps, and the score-like results are double-buffered in
// TMEM, so the element-wise work of step u+1 runs while the accumulating MMAs of step u and the score
// MMAs of step u+2 occupy the tensor pipe (the forward kernel pipelines S and P the same way).
// TMEM (512 columns): buffer b of step u (b = u & 1) holds T1 at [128 b, 128 b + 64) and T2 at
// [128 b + 64, 128 b + 128); accumulators from 256 (dQ, or dV then dK), D columns each; P^T / dS (bf16)
// overwrite 32 of the columns of T1 / T2 (query side at D = 128: 32 columns of their own per buffer, see kApart).
// From one tile to the next the pipeline does not drain: the next own rows load once the last score MMAs have read the
// present ones, and the next tile's first score MMAs run while the accumulators are read out (through shared memory
// and TMA stores).  One CTA per tile, with its set-up, first loads and read-out exposed each time, took 651 us on
// B=4 H=32 N=2048 D=128 causal (498 with one issuing warp, 456 with two and what follows), 45 on B=1 H=32 N=658 D=64 (23).
//  384 threads: warps 0-7 element-wise work and the final read-out,
// two threads per own row (warp w owns rows 32 (w % 4).. and the 32 score columns of half w / 4; its bf16
// results go back into the first 16 of its OWN columns, so the two threads of a row never touch each other's
// inputs, and the accumulating MMAs take K elements 0-31 from columns [0,16) and 32-63 from [32,48));
// warp 8 TMA producer, warp 9 TMEM allocation and the accumulating MMAs, warp 10 the score MMAs, warp 11 the columns' statistics.
// What bounds a step, by its clocks and those of its MMAs at the rates of back-to-back issue: the MMAs on the key side at
// D = 128 (1270 and 1280: the pipe does not idle), MMAs and their hand-over on its query side (1140 and 1024), the element-wise
// chain at D = 64 (key side 1030 and 640, query side 980 and 512); between two items the read-out, 4000 clocks of f32 stores at
// D = 128, and the refill.
// Every mbarrier wait is bounded; on expiry the kernel records a code in the device status word and
// leaves through the common teardown.
#include <cuda.h>
#include <algorithm>
#include <cstdlib>
#include <type_traits>

#include "kernels.h"
#include "tc_ptx.cuh"
#include "tile_schedule.cuh"

namespace rt {

using namespace ptx;

bool make_tensor_map_bf16_4d(CUtensorMap* map, const void* base, int64_t batch, int64_t heads, int64_t seq, int dim,
                             int64_t stride_b, int64_t stride_h, int64_t stride_row, int box_rows);  // prefill_tc.cu

namespace {

enum { kToBwdX = 201, kToBwdYFull, kToBwdYEmpty, kToBwdT, kToBwdA, kToBwdAcc, kToBwdDrain, kToBwdStat, kToBwdXEmpty, kToBwdAlign };

__device__ __forceinline__ void grid_dep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Q, K, V and dO up to this size are taken to stay in L2 (126 MB) with their gradients passing through.
constexpr int64_t kLevelsBytes = 96ll << 20;

constexpr int kBwdThreads = 384;

template <int D>
struct BwdCfg {
    static constexpr int TILE_BYTES = 128 * D * 2;
    static constexpr int SUB_BYTES = 128 * 64 * 2;  // one 64-column (128-byte) swizzled sub-tile
    static constexpr int NSUB = D / 64;
    static constexpr int HALF_BYTES = 64 * D * 2;   // 64 other-side rows: NSUB sub-tiles of 64 rows x 128 bytes
    static constexpr int HSUB_BYTES = 64 * 64 * 2;
    static constexpr int STAGES = 4;                // ring slots, each (Y1 | Y2) of one 64-row step
    static constexpr int STAGE_OUT = 8 * 32 * 128;  // per element-wise warp: 32 rows x 32 f32 columns on their way out
    static constexpr int NBARS = 2 + 2 * STAGES + 13;
    static constexpr int STAT_BYTES = 2 * 2 * 128 * 4;  // two slots of -LSE * log2(e) and -delta of a 128-row other tile
    static constexpr int SMEM_BYTES = 2 * TILE_BYTES + STAGES * 2 * HALF_BYTES + STAGE_OUT + STAT_BYTES + NBARS * 8 + 16;
    static constexpr uint32_t COL_T = 0, COL_ACC = 256;  // T1 of buffer b at COL_T + 128 b, T2 64 columns further
    static_assert(SMEM_BYTES <= 232448, "exceeds the 227 KB of shared memory a CTA can opt into");
};

struct Bwd5Params {
    const float* lse;    // [B*H, N]
    const float* delta;  // [B*H, N]
    int seq, heads;
    int causal;
    float scale, scale_log2;
    int* status;
    int q_ctas;          // CTAs of the query side; the rest of the grid is the key side's
    LevelSchedule list[2];  // the query side's and the key side's 128-row tiles
};

// One 128-row tile of a CTA's own side.
struct BwdItem {
    int bh, b, h;
    int own0;     // first own row
    int s_lo;     // first other-side 64-row step (even)
    int n_u;      // steps
};

template <int D, bool kKeySide>
__device__ __forceinline__ void bwd_side(const CUtensorMap* tm_x1, const CUtensorMap* tm_x2, const CUtensorMap* tm_y1,
                                         const CUtensorMap* tm_y2, const CUtensorMap* tm_o1, const CUtensorMap* tm_o2,
                                         const Bwd5Params& p, uint8_t* smem, int warp, int lane, int cta, int n_ctas) {
    using C = BwdCfg<D>;
    constexpr int TILE = C::TILE_BYTES, SUB = C::SUB_BYTES, STAGES = C::STAGES, HALFT = C::HALF_BYTES, HSUB = C::HSUB_BYTES;
    // On the query side at D = 128 dS has columns of its own behind the accumulator (32 per buffer): the score MMAs of step
    // u + 2 then follow the reading of T(u), not the accumulating MMAs of step u.
    constexpr bool kApart = !kKeySide && D == 128;
    constexpr uint32_t COL_A = C::COL_ACC + D, A_BUF = 32;
    static_assert(!kApart || COL_A + 2 * A_BUF <= 512, "TMEM columns");
    uint8_t* sX1 = smem;
    uint8_t* sX2 = sX1 + TILE;
    uint8_t* sY = sX2 + TILE;  // [STAGES][Y1 | Y2], 64 rows each
    uint8_t* sOut = sY + STAGES * 2 * HALFT;
    float* stat = reinterpret_cast<float*>(sOut + C::STAGE_OUT);  // [2][lse2[128] | delta[128]]
    uint64_t* bars = reinterpret_cast<uint64_t*>(reinterpret_cast<uint8_t*>(stat) + C::STAT_BYTES);
    uint64_t* x_full = bars;                // [1] one phase per item
    uint64_t* x_empty = x_full + 1;         // [1] one phase per item: its last score MMAs have retired
    uint64_t* y_full = x_empty + 1;         // [STAGES]
    uint64_t* y_empty = y_full + STAGES;    // [STAGES]
    uint64_t* t_full = y_empty + STAGES;    // [2] per buffer, one phase per use: T1, T2 are in TMEM
    uint64_t* a_full = t_full + 2;          // [2] per buffer, one phase per use: the bf16 A operands are in TMEM
    uint64_t* acc_done = a_full + 2;        // [1] one phase per item: its last accumulating MMA has retired
    uint64_t* stat_bar = acc_done + 1;      // [2] key side, per slot, one phase per other tile: the column statistics are in shared memory
    uint64_t* acc_step = stat_bar + 2;      // [2] per buffer, one phase per use: the MMAs that read the A operands have retired
    uint64_t* t_read = acc_step + 2;        // [2] per buffer, one phase per use: T1, T2 are in registers (kApart)
    uint64_t* acc_half = t_read + 2;        // [2] key side, as acc_step: the MMAs that read P^T have
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_half + 2);

    const int N = p.seq;
    const LevelSchedule& list = p.list[kKeySide ? 1 : 0];
    // Entry j of the CTA's list and on to the next that holds a tile (all roles walk the same list).  Heaviest first:
    // under a causal mask the query side's last tiles and the key side's first tiles walk the most steps.
    auto fetch = [&](int& j, BwdItem& it) {
        for (;;) {
            bool end = false, valid;
            int rank = 0;
            if (p.causal) {
                valid = level_item(list, j, cta, n_ctas, it.bh, rank, end);
            } else {
                const int pos = j * n_ctas + cta;
                end = pos >= list.units * list.n;
                valid = !end;
                it.bh = pos / list.n;
                rank = pos % list.n;
            }
            ++j;
            if (end) return false;
            if (!valid) continue;
            const int own = (kKeySide || !p.causal) ? rank : list.n - 1 - rank;
            it.b = it.bh / p.heads;
            it.h = it.bh % p.heads;
            it.own0 = own * 128;
            const int all = (N + 63) / 64;
            it.s_lo = (kKeySide && p.causal) ? 2 * own : 0;
            it.n_u = ((!kKeySide && p.causal) ? min(all, 2 * own + 2) : all) - it.s_lo;
            return true;
        }
    };

    if (warp == 8 && lane == 0) {
        prefetch_tensormap(tm_x1);
        prefetch_tensormap(tm_x2);
        prefetch_tensormap(tm_y1);
        prefetch_tensormap(tm_y2);
        prefetch_tensormap(tm_o1);
        mbar_init(x_full, 1);
        mbar_init(x_empty, 1);
        for (int i = 0; i < STAGES; ++i) {
            mbar_init(&y_full[i], 1);
            mbar_init(&y_empty[i], 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&t_full[i], 1);
            mbar_init(&a_full[i], 256);
            mbar_init(&acc_step[i], 1);
            mbar_init(&t_read[i], 256);
            mbar_init(&acc_half[i], 1);
        }
        mbar_init(acc_done, 1);
        mbar_init(&stat_bar[0], 32);
        mbar_init(&stat_bar[1], 32);
        fence_barrier_init();
        fence_proxy_async();
    }
    if (warp == 9) {
        tmem_alloc(tmem_slot, 512);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    grid_dep_wait();  // delta is the previous kernel's output; the set-up above overlaps that kernel

    if (warp == 8) {
        // ============================================================== TMA producer
        if (lane == 0) {
            int g = 0, k = 0;  // steps requested so far (ring position and phase), items begun
            bool ok = true;
            BwdItem it;
            for (int j = 0; ok && fetch(j, it); ++k) {
                if (k > 0 && !mbar_wait(x_empty, (uint32_t)(k - 1) & 1u, p.status, kToBwdXEmpty)) break;
                mbar_arrive_expect_tx(x_full, 2 * TILE);
#pragma unroll
                for (int s = 0; s < C::NSUB; ++s)
#pragma unroll
                    for (int r = 0; r < 2; ++r) {
                        tma_load_4d(sX1 + s * SUB + r * HSUB, tm_x1, x_full, s * 64, it.own0 + r * 64, it.h, it.b);
                        tma_load_4d(sX2 + s * SUB + r * HSUB, tm_x2, x_full, s * 64, it.own0 + r * 64, it.h, it.b);
                    }
                for (int u = 0; u < it.n_u; ++u) {
                    const int st = g % STAGES;
                    if (g >= STAGES && !mbar_wait(&y_empty[st], (uint32_t)(g / STAGES - 1) & 1u, p.status, kToBwdYEmpty)) {
                        ok = false;
                        break;
                    }
                    mbar_arrive_expect_tx(&y_full[st], 2 * HALFT);
                    uint8_t* dst = sY + st * 2 * HALFT;
                    const int r0 = (it.s_lo + u) * 64;
#pragma unroll
                    for (int s = 0; s < C::NSUB; ++s) {
                        tma_load_4d(dst + s * HSUB, tm_y1, &y_full[st], s * 64, r0, it.h, it.b);
                        tma_load_4d(dst + HALFT + s * HSUB, tm_y2, &y_full[st], s * 64, r0, it.h, it.b);
                    }
                    ++g;
                }
            }
            // Drain: every copy this thread issued must have landed before the CTA may exit.
            if (k > 0) mbar_wait(x_full, (uint32_t)(k - 1) & 1u, p.status, kToBwdDrain);
            for (int u = max(0, g - STAGES); u < g; ++u)
                mbar_wait(&y_full[u % STAGES], (uint32_t)(u / STAGES) & 1u, p.status, kToBwdDrain);
        }
    } else if (warp == 11) {
        // ============================================================== key side: the columns' statistics
        // -LSE (as log2; -inf, which makes every probability 0, for absent queries and rows without a visible key) and -delta
        // of the 128 queries of each other tile, negated here once rather than per score, into the slot that was last
        // read two tiles ago (its last step's rows are free: every thread has handed that step's operands over).
        if (kKeySide) {
            int g = 0, gt = 0, before = 0, before2 = 0;  // steps and tiles so far, last step of the tile before and of the one before that
            bool ok = true;
            BwdItem it;
            for (int j = 0; ok && fetch(j, it); g += it.n_u) {
                const float* lse = p.lse + (int64_t)it.bh * N;
                const float* delta = p.delta + (int64_t)it.bh * N;
                for (int u = 0; u < it.n_u && ok; u += 2, ++gt) {
                    float l[4], d[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const int qi = (it.s_lo + u) * 64 + i * 32 + lane;
                        const float raw = qi < N ? __ldg(lse + qi) : INFINITY;
                        l[i] = (raw > -INFINITY && raw < INFINITY) ? raw * -kLog2e : -INFINITY;
                        d[i] = qi < N ? -__ldg(delta + qi) : 0.f;
                    }
                    if (gt >= 2)
                        ok = __all_sync(kFullMask, mbar_wait(&y_empty[before2 % STAGES], (uint32_t)(before2 / STAGES) & 1u, p.status, kToBwdStat));
                    float* to = stat + (gt & 1) * 256;
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        to[i * 32 + lane] = l[i];
                        to[128 + i * 32 + lane] = d[i];
                    }
                    mbar_arrive(&stat_bar[gt & 1]);
                    before2 = before;
                    before = g + min(u + 1, it.n_u - 1);
                }
            }
        }
    } else if (warp >= 9) {
        // ============================================================== MMA issuers
        // One warp for the score MMAs, one for the accumulating ones: an issuing warp is held until the pipe takes its MMA, so
        // what a single one did between two steps (two waits that were already over, commits: 345 clocks of 1625 a key-side
        // step at D=128) left the pipe idle.
        const bool leader = elect_one();
        const uint32_t tT = tmem_base + C::COL_T, tAcc = tmem_base + C::COL_ACC;
        auto wait = [&](uint64_t* bar, uint32_t parity, int code) -> bool {
            return __all_sync(kFullMask, mbar_wait(bar, parity, p.status, code));
        };
        bool ok = true;
        BwdItem it;
        if (warp == 10) {
            // T1 = X1 Y1^T, T2 = X2 Y2^T over the 64 other-side rows of every step, two steps ahead of the accumulating MMAs.  The
            // first ones of an item run while the element-wise warps read the accumulators of the one before out.
            constexpr uint32_t idesc_t = make_idesc_bf16(128, 64, 0, 0);
            const uint64_t dx1 = make_smem_desc_sw128(smem_u32(sX1), 16, 1024);
            const uint64_t dx2 = make_smem_desc_sw128(smem_u32(sX2), 16, 1024);
            const uint64_t dy = make_smem_desc_sw128(smem_u32(sY), 16, 1024);  // other tile as a K-major operand
            int st = 0;                       // ring slot of the step
            uint32_t ph = 0, b = 0, pb = 3;   // its phase; the step's buffer; bit b: phase in which the buffer is free
            for (int j = 0, k = 0; ok && fetch(j, it); ++k) {
                ok = wait(x_full, (uint32_t)k & 1u, kToBwdX);
                for (int u = 0; u < it.n_u && ok; ++u) {
                    ok = wait(&y_full[st], ph, kToBwdYFull) && wait(kApart ? &t_read[b] : kKeySide ? &acc_half[b] : &acc_step[b], (pb >> b) & 1u, kToBwdAcc);
                    if (!ok) break;
                    tc_fence_after();
                    const uint64_t y1 = dy + (uint64_t)((st * 2 * HALFT) >> 4), y2 = y1 + (uint64_t)(HALFT >> 4);
                    const uint32_t t1 = tT + b * 128, t2 = t1 + 64;
#pragma unroll
                    for (int kk = 0; kk < D / 16; ++kk) {
                        const uint32_t offx = (uint32_t)(((kk / 4) * SUB + (kk % 4) * 32) >> 4);
                        const uint32_t offy = (uint32_t)(((kk / 4) * HSUB + (kk % 4) * 32) >> 4);
                        if (leader) mma_ss(t1, dx1 + offx, y1 + offy, idesc_t, kk > 0);
                    }
                    if (kKeySide) {  // T1 overwrites P^T while the MMAs that read dS^T, in T2, still run
                        ok = wait(&acc_step[b], (pb >> b) & 1u, kToBwdAcc);
                        if (!ok) break;
                        tc_fence_after();
                    }
#pragma unroll
                    for (int kk = 0; kk < D / 16; ++kk) {
                        const uint32_t offx = (uint32_t)(((kk / 4) * SUB + (kk % 4) * 32) >> 4);
                        const uint32_t offy = (uint32_t)(((kk / 4) * HSUB + (kk % 4) * 32) >> 4);
                        if (leader) mma_ss(t2, dx2 + offx, y2 + offy, idesc_t, kk > 0);
                    }
                    if (leader) mma_commit(&t_full[b]);
                    if (leader && u == it.n_u - 1) mma_commit(x_empty);
                    pb ^= 1u << b;
                    b ^= 1;
                    if (++st == STAGES) st = 0, ph ^= 1;
                }
            }
        } else {
            constexpr uint32_t idesc_a = make_idesc_bf16(128, D, 0, 1);
            const uint64_t dy = make_smem_desc_sw128(smem_u32(sY), HSUB, 1024);  // the other tile's rows as an MN-major operand
            int st = 0;                      // ring slot of the step
            uint32_t b = 0, pa = 0;          // the step's buffer; bit b: phase of its A operands
            for (int j = 0; ok && fetch(j, it);) {
                // (The first A operands of an item come after the element-wise warps have read the accumulators out.)
                for (int u = 0; u < it.n_u; ++u) {
                    ok = wait(&a_full[b], (pa >> b) & 1u, kToBwdA);
                    if (!ok) break;
                    tc_fence_after();
                    const uint64_t y1 = dy + (uint64_t)((st * 2 * HALFT) >> 4), y2 = y1 + (uint64_t)(HALFT >> 4);
                    // P^T and dS^T (or dS): the first 16 of every 32 columns of T1 and T2, or contiguous
                    const uint32_t a1 = tT + b * 128, a2 = kApart ? tmem_base + COL_A + b * A_BUF : a1 + 64;
                    auto k16 = [](int kk) { return (uint32_t)(kk * 8 + (!kApart && kk >= 2 ? 16 : 0)); };
                    const uint32_t acc0 = u > 0 ? 1u : 0u;
                    if (kKeySide) {
                        // dV += P^T dO (B = Y2 = dO), dK += dS^T Q (B = Y1 = Q)
#pragma unroll
                        for (int kk = 0; kk < 4; ++kk)
                            if (leader) mma_ts(tAcc, a1 + k16(kk), y2 + (uint64_t)((kk * 2048) >> 4), idesc_a, kk > 0 ? 1u : acc0);
                        if (leader) mma_commit(&acc_half[b]);
#pragma unroll
                        for (int kk = 0; kk < 4; ++kk)
                            if (leader) mma_ts(tAcc + D, a2 + k16(kk), y1 + (uint64_t)((kk * 2048) >> 4), idesc_a, kk > 0 ? 1u : acc0);
                    } else {
                        // dQ += dS K (B = Y1 = K)
#pragma unroll
                        for (int kk = 0; kk < 4; ++kk)
                            if (leader) mma_ts(tAcc, a2 + k16(kk), y1 + (uint64_t)((kk * 2048) >> 4), idesc_a, kk > 0 ? 1u : acc0);
                    }
                    if (leader) mma_commit(&acc_step[b]);
                    if (leader) mma_commit(&y_empty[st]);  // the step's rows: its score MMAs have retired before
                    if (leader && u == it.n_u - 1) mma_commit(acc_done);
                    pa ^= 1u << b;
                    b ^= 1;
                    if (++st == STAGES) st = 0;
                }
            }
        }
    } else {
        // ============================================================== element-wise warps (two threads per own row)
        const int half = warp >> 2;  // which 32 of a step's 64 score columns
        const int r = (warp & 3) * 32 + lane;
        const uint32_t lane_sel = (uint32_t)((warp & 3) * 32) << 16;
        const uint32_t tT = tmem_base + lane_sel + C::COL_T;
        const uint32_t tAcc = tmem_base + lane_sel + C::COL_ACC;
        uint8_t* const stage = sOut + warp * 4096;
        const float c = p.scale_log2;
        // Query side: the row's own statistics (see warp 11 for the key side's), requested an item ahead.
        float raw_lse = 0.f, raw_delta = 0.f;
        auto request = [&](const BwdItem& it) {
            const int qi = it.own0 + r;
            raw_lse = qi < N ? __ldg(p.lse + (int64_t)it.bh * N + qi) : INFINITY;
            raw_delta = qi < N ? -__ldg(p.delta + (int64_t)it.bh * N + qi) : 0.f;
        };
        int j = 0, g = 0, gt = 0;  // list entry, first step of the item, other tiles so far (key side)
        BwdItem it, nx;
        bool ok = true, more = fetch(j, it);
        if (!kKeySide && more) request(it);
        for (int k = 0; more && ok; ++k, it = nx) {
        more = fetch(j, nx);
        const int own_row = it.own0 + r, n_u = it.n_u;
        float my_lse2 = 0.f, my_delta = 0.f;  // query side: this row's statistics
        if (!kKeySide) {
            my_lse2 = (raw_lse > -INFINITY && raw_lse < INFINITY) ? raw_lse * -kLog2e : -INFINITY;
            my_delta = raw_delta;
            if (more) request(nx);
        }
        for (int u = 0; u < n_u && ok; ++u) {
            const int step = it.s_lo + u, buf = (g + u) & 1, sub = step & 1;
            const int other0 = step * 64;  // first other-side row of this step
            const float* s_lse2 = stat + (gt & 1) * 256;
            const float* s_delta = s_lse2 + 128;
            if (kKeySide && sub == 0) ok &= mbar_wait(&stat_bar[gt & 1], (uint32_t)(gt >> 1) & 1u, p.status, kToBwdStat);
            ok &= mbar_wait(&t_full[buf], (uint32_t)((g + u) >> 1) & 1u, p.status, kToBwdT);
            // its A operands: the MMAs of two steps ago have read them
            if (kApart && g + u >= 2) ok &= mbar_wait(&acc_step[buf], (uint32_t)(((g + u) >> 1) - 1) & 1u, p.status, kToBwdAcc);
            if (!__all_sync(kFullMask, ok)) {  // (one vote for the waits of the step)
                ok = false;
                break;
            }
            tc_fence_after();
            // Is any (own row, other index) pair of this step masked?  Only the diagonal tile of a causal
            // launch and the last tile of a ragged sequence are.
            const bool diag = p.causal && (step >> 1) == (it.own0 >> 7);
            const bool ragged = other0 + 64 > N;
            const uint32_t t1 = tT + buf * 128, t2 = t1 + 64;
            const float2 c2 = make_float2(c, c);
            {
                const int cbase = half * 32;  // this thread's score columns of the step: [32 half, 32 half + 32)
                uint32_t a1[32], a2[32];
                tmem_ld32(t1 + cbase, a1);
                tmem_ld32(t2 + cbase, a2);
                tc_wait_ld();
                if (kApart) {
                    tc_fence_before();
                    mbar_arrive(&t_read[buf]);
                }
                uint32_t pk_p[16], pk_ds[16];
                // (Compiled twice: a test per four columns cuts the step into eight pieces whose exponentials cannot overlap.)
                auto columns = [&](auto masked) {
#pragma unroll
                for (int i = 0; i < 32; i += 4) {
                    // statistics of four columns: the row's own on the query side, one 16-byte broadcast read each
                    // on the key side (a negated LSE of -inf makes the probability 0: absent queries, rows without a key)
                    float4 l4, d4;
                    if (kKeySide) {
                        l4 = *reinterpret_cast<const float4*>(s_lse2 + sub * 64 + cbase + i);
                        d4 = *reinterpret_cast<const float4*>(s_delta + sub * 64 + cbase + i);
                    } else {
                        l4 = make_float4(my_lse2, my_lse2, my_lse2, my_lse2);
                        d4 = make_float4(my_delta, my_delta, my_delta, my_delta);
                    }
                    const float2 xa = __ffma2_rn(make_float2(__uint_as_float(a1[i]), __uint_as_float(a1[i + 1])), c2,
                                                 make_float2(l4.x, l4.y));
                    const float2 xb = __ffma2_rn(make_float2(__uint_as_float(a1[i + 2]), __uint_as_float(a1[i + 3])), c2,
                                                 make_float2(l4.z, l4.w));
                    float2 pa = make_float2(fast_exp2(xa.x), fast_exp2(xa.y));
                    float2 pb = make_float2(fast_exp2(xb.x), fast_exp2(xb.y));
                    if constexpr (decltype(masked)::value) {
                        const int o0 = other0 + cbase + i;
                        auto hidden = [&](int other) {
                            return other >= N || (p.causal && (kKeySide ? own_row > other : other > own_row));
                        };
                        if (hidden(o0)) pa.x = 0.f;
                        if (hidden(o0 + 1)) pa.y = 0.f;
                        if (hidden(o0 + 2)) pb.x = 0.f;
                        if (hidden(o0 + 3)) pb.y = 0.f;
                    }
                    const float2 ta = __fadd2_rn(make_float2(__uint_as_float(a2[i]), __uint_as_float(a2[i + 1])),
                                                 make_float2(d4.x, d4.y));
                    const float2 tb = __fadd2_rn(make_float2(__uint_as_float(a2[i + 2]), __uint_as_float(a2[i + 3])),
                                                 make_float2(d4.z, d4.w));
                    const float2 da = __fmul2_rn(pa, ta), db = __fmul2_rn(pb, tb);
                    pk_p[i / 2] = float2_to_bf16x2(pa.x, pa.y);
                    pk_p[i / 2 + 1] = float2_to_bf16x2(pb.x, pb.y);
                    pk_ds[i / 2] = float2_to_bf16x2(da.x, da.y);
                    pk_ds[i / 2 + 1] = float2_to_bf16x2(db.x, db.y);
                }
                };
                if (diag || ragged) columns(std::true_type{});
                else columns(std::false_type{});
                if constexpr (kApart) {
                    tmem_st16(tmem_base + lane_sel + COL_A + buf * A_BUF + half * 16, pk_ds);
                } else {  // into the first 16 of this thread's own 32 columns (in registers by now)
                    if (kKeySide) tmem_st16(t1 + cbase, pk_p);
                    tmem_st16(t2 + cbase, pk_ds);
                }
            }
            tc_wait_st();
            tc_fence_before();
            mbar_arrive(&a_full[buf]);
            if (kKeySide && (sub == 1 || u == n_u - 1)) ++gt;
        }
        g += n_u;
        // ---- read-out: accumulators -> f32 (scale folded into dQ and dK) -> 32 rows x 32 columns of this warp in shared
        // memory, swizzled as the tensor map has it -> one TMA store, which clips the rows past N.  (Stored straight
        // from registers, 16 bytes of 32 rows per instruction, the tile took 8192 store cycles.)
        ok = ok && __all_sync(kFullMask, mbar_wait(acc_done, (uint32_t)k & 1u, p.status, kToBwdAcc));
        if (ok) {
            tc_fence_after();
            constexpr int kOuts = kKeySide ? 2 : 1;
            constexpr int OC = D / 2;  // accumulator columns per thread
            const int row0 = it.own0 + (warp & 3) * 32;
#pragma unroll
            for (int o = 0; o < kOuts; ++o) {
                const float mul = (kKeySide && o == 0) ? 1.f : p.scale;  // dV is not scaled
#pragma unroll
                for (int ch = 0; ch < OC / 32; ++ch) {
                    uint32_t a[32];
                    tmem_ld32(tAcc + o * D + half * OC + ch * 32, a);
                    tc_wait_ld();
                    if (lane == 0) tma_store_wait_read();  // the warp's previous store has read the staging rows
                    __syncwarp();
#pragma unroll
                    for (int i = 0; i < 32; i += 4)
                        *reinterpret_cast<float4*>(stage + lane * 128 + (((i >> 2) ^ (lane & 7)) << 4)) =
                            make_float4(__uint_as_float(a[i]) * mul, __uint_as_float(a[i + 1]) * mul,
                                        __uint_as_float(a[i + 2]) * mul, __uint_as_float(a[i + 3]) * mul);
                    fence_proxy_async();
                    __syncwarp();
                    if (lane == 0 && row0 < N) {
                        // the map counts in 2-byte elements
                        tma_store_4d(o == 0 ? tm_o1 : tm_o2, stage, (half * OC + ch * 32) * 2, row0, it.h, it.b);
                        tma_store_commit();
                    }
                }
            }
        }
        }
        if (lane == 0) tma_store_wait_read();  // shared memory stays until the last store has read it
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 9) {
        tc_fence_after();
        tmem_dealloc(tmem_base, 512);
    }
}

// CTAs [0, q_ctas) work through the query side's tiles, the others through the key side's.
template <int D>
__global__ void __launch_bounds__(kBwdThreads, 1)
bwd_tcgen05_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                   const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_do,
                   const __grid_constant__ CUtensorMap tm_dq, const __grid_constant__ CUtensorMap tm_dk,
                   const __grid_constant__ CUtensorMap tm_dv, const Bwd5Params p) {
    extern __shared__ __align__(1024) uint8_t smem[];
    const int warp = __shfl_sync(kFullMask, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    if (smem_u32(smem) & 1023u) {  // the swizzled tiles need it; all 227 KB are in use, so none is spent on rounding up
        if (threadIdx.x == 0) atomicCAS(p.status, 0, (int)kToBwdAlign);
        return;
    }
    const int cta = (int)blockIdx.x, nq = p.q_ctas;
    if (cta < nq) bwd_side<D, false>(&tm_q, &tm_do, &tm_k, &tm_v, &tm_dq, &tm_dq, p, smem, warp, lane, cta, nq);
    else bwd_side<D, true>(&tm_k, &tm_v, &tm_q, &tm_do, &tm_dv, &tm_dk, p, smem, warp, lane, cta - nq, (int)gridDim.x - nq);
}

template <int D>
cudaError_t launch_sides(const CUtensorMap (&m)[7], Bwd5Params p, int64_t bh, cudaStream_t stream) {
    cudaError_t e = set_max_dynamic_smem_once<bwd_tcgen05_kernel<D>>(BwdCfg<D>::SMEM_BYTES);
    if (e != cudaSuccess) return e;
    const int64_t n_tiles = (p.seq + 127) / 128, n_items = n_tiles * bh;
    if (n_items > 0x3fffffff) return cudaErrorNotSupported;
    const int64_t n_sm = sm_count();
    // Both sides' tiles go out in one launch: small grids run side by side, and large ones have one tail instead of
    // two.  Where the tiles exceed the SMs, the query side gets fewer of them: it has one accumulating product
    // a step, the key side two (share: measured best of 0.39 .. 0.50 on 16 shapes; equal tiles come in whole
    // waves, so without a mask the split with the shortest longer side is taken, 77 -> 72 us at B=2 H=16 N=1024 D=128).
    int64_t nq = n_items, nk = n_items;
    if (2 * n_items > n_sm) {
        constexpr double share = D == 128 ? 0.45 : 0.46;
        nq = std::max<int64_t>(1, (int64_t)((double)n_sm * share + 0.5));
        if (!p.causal) {
            double best = 1e30;
            for (int64_t x = n_sm / 4; x <= n_sm / 2; ++x) {
                auto waves = [&](int64_t ctas) { return (double)((n_items + ctas - 1) / ctas); };
                const double t = std::max(waves(x) * share, waves(n_sm - x) * (1 - share));
                if (t < best) best = t, nq = x;
            }
        }
        nq = std::min(n_items, nq);
        nk = std::min(n_items, n_sm - nq);
    }
    p.q_ctas = (int)nq;
    const bool paired = 8 * bh * p.seq * D > kLevelsBytes;
    p.list[0] = make_level_schedule(bh, n_tiles, nq, paired);
    p.list[1] = make_level_schedule(bh, n_tiles, nk, paired);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(nq + nk));
    cfg.blockDim = dim3(kBwdThreads);
    cfg.dynamicSmemBytes = BwdCfg<D>::SMEM_BYTES;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, bwd_tcgen05_kernel<D>, m[0], m[1], m[2], m[3], m[4], m[5], m[6], p);
}

}  // namespace

// Returns cudaErrorNotSupported when this kernel does not cover the shape (the caller then uses the
// mma.sync kernel).
cudaError_t launch_backward_tcgen05(const void* q, const void* k, const void* v, const void* d_out, const float* lse,
                                    const float* delta, float* dq, float* dk, float* dv, int64_t batch, int64_t heads,
                                    int64_t seq, int dim, int causal, float scale, cudaStream_t stream) {
    const int64_t bh = batch * heads;
    if ((dim != 64 && dim != 128) || bh > 65535 || seq > (1 << 30)) return cudaErrorNotSupported;
    // inputs in boxes of 64 rows; outputs, f32 seen as pairs of 2-byte elements, in boxes of 32 rows x 32 columns
    CUtensorMap m[7];
    const TensorStrides s = TensorStrides::contiguous(heads, seq, dim);
    const void* ptrs[7] = {q, k, v, d_out, dq, dk, dv};
    for (int i = 0; i < 7; ++i) {
        const int f = i < 4 ? 1 : 2;
        if (!make_tensor_map_bf16_4d(&m[i], ptrs[i], batch, heads, seq, f * dim, f * s.batch, f * s.head, f * s.row, i < 4 ? 64 : 32))
            return cudaErrorNotSupported;
    }
    Bwd5Params p;
    p.lse = lse;
    p.delta = delta;
    p.seq = (int)seq;
    p.heads = (int)heads;
    p.causal = causal;
    p.scale = scale;
    p.scale_log2 = scale * kLog2e;
    p.status = device_status_ptr();
    if (!p.status) return cudaErrorInvalidSymbol;
    return dim == 128 ? launch_sides<128>(m, p, bh, stream) : launch_sides<64>(m, p, bh, stream);
}

}  // namespace rt
