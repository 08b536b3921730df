// Flash-attention forward on the Blackwell tensor cores (tcgen05 + TMEM + TMA), bf16.
//
// Replaces rustorch_attention::flash_forward_masked (crates/rustorch-attention/src/cpu_forward.rs:193-425)
// for bf16 device tensors of head dim 64 or 128.  The recurrence is the reference's online
// softmax (cpu_forward.rs:355-386) evaluated in the log2 domain; unlike the reference, KV tiles
// that a causal mask or a per-batch kv_len hides completely are never visited.
//
// Work item = 256 query rows of one (batch, head) = two 128-row Q tiles that share the K/V tiles
// in shared memory and ping-pong on the tensor pipe.  The kernel is persistent: one CTA per SM
// walks a static list of items (see tc_item), and every barrier runs on phase counters that
// carry over from item to item, so the next item's loads and first score MMAs overlap the
// previous item's last steps and write-back.  384 threads = 3 warpgroups:
//   warps 0-3  : softmax + lazy O rescale + epilogue of Q tile 0 (one thread per query row)
//   warps 4-7  : the same for Q tile 1
//   warp  8    : TMA producer (Q per item, K_j / V_j through their rings)
//   warp  9    : TMEM allocation; issues the tcgen05.mma of Q tile 0
//   warp  10   : issues the tcgen05.mma of Q tile 1 (two issuers, so that the barrier waits and
//                commits of one tile hide behind the queued MMAs of the other, and one tile can
//                move on to the next item while the other finishes)
//   warp  11   : idle (it completes the third warpgroup so that setmaxnreg can move its
//                registers to the softmax warpgroups: 72 vs 216 registers per thread; the split
//                must stay below the 64 K register file or setmaxnreg.inc never returns)
// TMEM (512 columns x 128 lanes, f32): per Q tile two 64-column S buffers (S[w][b] at w*128 + b*64),
// O0 [256,256+D), O1 [256+D,256+2D).  K/V are loaded as 128-key tiles but multiplied in 64-key
// steps; P (bf16) overwrites the first 32 columns of its S buffer and feeds the PV MMA from TMEM.
// S = Q K^T is an SS MMA with both operands K-major in 128-byte-swizzled shared memory; O += P V
// is a TS MMA whose B operand (V) is MN-major, i.e. V is used exactly as TMA lands it.
// The normalised O tile is staged in shared memory (at D = 64 in a buffer of its own, at D = 128, where
// the rings leave no room, in the tile's by then idle Q buffer) and leaves through TMA stores.  Every
// mbarrier wait is bounded; on expiry the kernel records a code in the device status word, drains its
// own copies and MMAs, frees TMEM and returns.
#include <algorithm>
#include <atomic>
#include <cuda.h>
#include <cstdlib>
#include <cstring>
#include <mutex>

#include "kernels.h"
#include "tc_ptx.cuh"
#include "tile_schedule.cuh"
#include "tensor_map.h"

namespace rt {

using namespace ptx;

template <int D>
struct TcCfg {
    static constexpr int BM = 128;                      // query rows per tile
    static constexpr int BL = 128;                      // keys per TMA-loaded K/V tile
    static constexpr int BN = 64;                       // keys per MMA / softmax step
    static constexpr int KS = (D == 128) ? 3 : 4;       // K ring depth (runs one tile ahead of V)
    static constexpr int VS = (D == 128) ? 2 : 4;       // V ring depth
    static constexpr int TILE_BYTES = 128 * D * 2;
    static constexpr int SUB_BYTES = 128 * 64 * 2;      // one 64-column (128-byte) swizzled sub-tile
    static constexpr int HALF_BYTES = 64 * 128;         // 64 rows inside a sub-tile
    static constexpr int NSUB = D / 64;
    static constexpr int NBARS = 2 + 2 + 3 * KS + 3 * VS + 4 + 4 + 2 + 2 + 2 + 2 + 1 + 1;
    // (batch, query block) pairs the length-sorted schedule can hold (two uint16 per pair); what is left of
    // the 227 KB of shared memory at D = 128 bounds it there
    static constexpr int SCHED_CAP = (D == 128) ? 384 : 2048;
    // The O tiles on their way out have shared memory of their own: B=4 H=32 D=64 N=300 15.0 -> 14.0 us, N=600 causal 26.7 -> 25.2,
    // 16 heads of 16 sequences of up to 1024 61.5 -> 56.4; items of 24 steps and more without a mask take up to 2 % longer
    // (N=3000 415 -> 420, N=4096 726 -> 739).
    static constexpr bool OWN_STAGE = (D == 64);
    static constexpr int SMEM_BYTES = (2 + KS + VS + (OWN_STAGE ? 2 : 0)) * TILE_BYTES + NBARS * 8 + 48 + 4 * SCHED_CAP + 1024;
    static_assert(SMEM_BYTES <= 232448, "exceeds the 227 KB of shared memory a CTA can opt into");
    static constexpr uint32_t TMEM_COLS = 512;
    static constexpr uint32_t COL_S = 0, COL_O = 256;   // S: tile w, buffer b at COL_S + w*128 + b*64
};

struct TcParams {
    __nv_bfloat16* out;
    float* lse;
    const int32_t* kv_lens;
    const uint8_t* key_keep;
    int64_t keep_batch_stride;
    int seq, heads;        // query rows per head, query heads
    int seq_kv, heads_kv;  // key rows per KV head, KV heads (query head h reads KV head h / (heads/heads_kv))
    const int32_t* q_offsets;  // NULL or [B]: causal position of query row 0 inside the key sequence
    float scale_log2;  // scale * log2(e)
    int* status;       // device status word (bounded-wait expiry codes)
    int64_t o_stride_b, o_stride_h, o_stride_row;  // element strides of the output (inner dim contiguous)
    int n_qb;          // 256-row blocks per head
    int n_items, units;  // static schedule, see tc_item: items of the launch, (batch, query head) pairs
    int by_level;      // single-tile items: level after level instead of head after head
    LevelSchedule list;  // causal launches
    int sorted;        // length-sorted order (launches with per-batch kv_lens), see tc_item
    int keep_tab;      // sorted schedule with key_keep: index of the per-batch step bounds behind the order in the table, else 0
    int stagger_clocks;  // single-tile items: head start of tile 0 over tile 1, in SM clocks
    int direct_out;    // one item per CTA: the epilogue stores its rows straight from registers (no staged tile, no TMA store)
    int tighten;       // key_keep launches of one item per CTA: trailing hidden keys are found at start-up and not visited
    int split;         // CTAs (one cluster) that share the keys of a single-tile item
    int single_tile;   // items are 128-row blocks whose 64-key steps alternate between the two tiles (small launches, see tc_item)
};


// Timeout codes written to the device status word (100 + site).
enum { kToQ = 101, kToKFull, kToKEmpty, kToVFull, kToVEmpty, kToSFull, kToPFull, kToOFull, kToDone, kToDrain,
       kToQEmpty, kToOFree, kToStage, kToMerge };

// 2^x for a pair of arguments on the FMA and integer pipes (x <= ~100): round to the nearest
// integer n with the 1.5*2^23 trick, a cubic for 2^r on r = x - n in [-0.5, 0.5] (relative error
// 7.5e-5, far below the bf16 rounding of P), and n added into the exponent field.  Arguments
// below -125 (masked scores are -inf) give 2^-125, not 0: invisible next to any visible score,
// and a row without one is recognised by a flag instead of by a zero sum.
// The MUFU pipe (16 ex2 per clock per SM) is the softmax warps' bottleneck; sending a share of
// the exponentials here balances it against the FMA pipe.
__device__ __forceinline__ float2 exp2_poly2(float2 x) {
    x.x = fmaxf(x.x, -125.f);
    x.y = fmaxf(x.y, -125.f);
    const float2 magic = make_float2(12582912.f, 12582912.f), nmagic = make_float2(-12582912.f, -12582912.f);
    const float2 t = __fadd2_rn(x, magic);
    const float2 nf = __fadd2_rn(t, nmagic);
    const float2 r = __fadd2_rn(x, make_float2(-nf.x, -nf.y));
    float2 y = __ffma2_rn(r, make_float2(0.0551716685f, 0.0551716685f), make_float2(0.242611125f, 0.242611125f));
    y = __ffma2_rn(y, r, make_float2(0.693260968f, 0.693260968f));
    y = __ffma2_rn(y, r, make_float2(0.999928057f, 0.999928057f));
    y.x = __int_as_float(__float_as_int(y.x) + (__float_as_int(t.x) << 23));
    y.y = __int_as_float(__float_as_int(y.y) + (__float_as_int(t.y) << 23));
    return y;
}
// Which of the 16 element pairs of a 32-column chunk take the polynomial path (a quarter: more
// than that costs more issue slots on the FMA pipe than it frees on the MUFU pipe).
__host__ __device__ constexpr bool poly_pair(int q) { return (q & 3) == 3; }

// All threads of the cluster: their shared-memory writes before it are visible to all after it.  (Threads that have
// exited count as arrived; every wait on the way here is bounded.)
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
// The address in CTA `rank` of the cluster of what lies at `a` in this one.
__device__ __forceinline__ uint32_t map_cluster(uint32_t a, int rank) {
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    return r;
}
__device__ __forceinline__ float2 ld_cluster_f2(uint32_t a) {
    float2 v;
    asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ float4 ld_cluster_f4(uint32_t a) {
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ void grid_dep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_dep_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// One work item of a CTA's static list.
struct TcItem {
    int bh, b, h, h_kv, q0, kv_hi, q_off;  // bh = b * heads + h indexes LSE; h_kv is the KV head h reads
    int U0, U1;    // 64-key steps of each Q tile; scalars, so nothing is indexed dynamically
    int n_tiles;   // 128-key K/V tiles to load
    int t0;        // first of them (split items: each CTA of the cluster takes its own run of tiles)
    bool end;      // the list is exhausted
    bool valid;    // false: this position of the list holds no item
    __device__ __forceinline__ int steps(int w) const { return w ? U1 : U0; }
    // first query row of tile w: the tiles are stacked (q0, q0 + 128), or both sit on the item's one block
    __device__ __forceinline__ int qrow(int w, bool single) const { return q0 + ((w || single) ? 128 : 0); }
};

// Static schedule.  Under a causal mask the 256-row block of rank n_qb-1 of a head costs n_qb times the first one, so
// what a launch costs over its work is the balance of the CTAs' lists.  Level t holds the t-th heaviest block of
// every head; the levels one after the other are dealt to the CTAs boustrophedon (0..G-1, G-1..0, ...), heaviest
// first.  Without a mask the blocks go out head after head, the ragged last ones (a tile or two of fewer rows: cheaper)
// at the end.  Where the K/V of all heads exceed L2, `rounds` paired rounds come first: a slot holds the blocks r and
// n_qb-1-r of one head, so all slots of a round cost the same and its CTAs work on a few neighbouring heads and share
// their K/V in L2; only the heads left over are dealt by levels.  (Pairs alone left the last round half empty: B=2
// H=32 N=2409 D=128 141 us against 118, B=4 H=12 N=1794 D=64 62 / 51, B=14 H=16 N=584 D=64 52 / 41.)
// Small launches use 128-row items instead (single_tile, see choose_items): twice the CTAs,
// and inside a CTA the item's 64-key steps alternate between the two tiles (tile 0 takes the even steps = the first
// half of every 128-key K/V tile, tile 1 the odd ones), each with its own running max, sum and accumulator;
// the epilogue merges the two partial results straight out of TMEM and stores the rows directly (no staged
// tile: such a CTA has no further item).  Both softmax warpgroups and both MMA issuers then work on the one
// block, which nearly halves the critical path of a small problem.  More such items than SMs are started level by
// level as well, heaviest first (H=8 N=4096 D=128: 53 us head after head, 37 by levels).
// Sorted mode (per-batch kv_lens, where an item's cost is only known on the device): every CTA ranks the
// (batch, query block) pairs by their step count at start-up (the same deterministic sort in every CTA, so
// no queue, no atomics and no scratch memory are needed), the item list is that order with all heads of a
// pair side by side, and it is dealt to the CTAs boustrophedon (0..G-1, G-1..0, ...), heaviest first: the
// persistent kernel's overlap of one item's set-up with the previous item's tail, and a balanced finish.
// 128-row items start in that order too where choose_items finds that it pays.
template <bool kCausal, bool kSingle>
__device__ __forceinline__ void tc_steps(const TcParams& p, int b, int q0, int& kv_hi, int& q_off, int& U0, int& U1,
                                         int keep_hi = 0x7fffffff, int* t0 = nullptr) {
    kv_hi = min(p.seq_kv, keep_hi);
    if (p.kv_lens) {
        const int l = p.kv_lens[b];
        kv_hi = l < 0 ? 0 : (l < kv_hi ? l : kv_hi);
    }
    q_off = p.q_offsets ? p.q_offsets[b] : 0;   // query row i sits at key position i + q_off
    const int n_steps = (kv_hi + 63) / 64;      // 64-key steps that hold a visible key
    const int last0 = q0 + 127 + q_off, last1 = last0 + 128;  // last key each tile's last row may see
    U0 = !kCausal ? n_steps : (last0 < 0 ? 0 : min(n_steps, last0 / 64 + 1));
    U1 = !kCausal ? n_steps : (last1 < 0 ? 0 : min(n_steps, last1 / 64 + 1));
    if (!kSingle && q0 + 128 >= p.seq) U1 = 0;  // the second tile of a ragged last block holds no row
    if (kSingle && t0) {  // this CTA's share of the steps
        const int per = ((U1 + 1) / 2 + p.split - 1) / p.split;
        *t0 = ((int)blockIdx.x % p.split) * per;
        U1 = max(0, min(U1 - 2 * *t0, 2 * per));
    }
    if (kSingle) {  // the block's U1 steps are dealt alternately: even ones to tile 0, odd ones to tile 1
        U0 = (U1 + 1) >> 1;
        U1 = U1 >> 1;
    }
}

template <bool kCausal, bool kSingle, bool kByLength>
__device__ __forceinline__ TcItem tc_item(int j, const TcParams& p, const uint16_t* sched, int keep_hi = 0x7fffffff) {
    TcItem it;
    it.valid = false;
    it.t0 = 0;
    int qb;
    if (kSingle) {  // the CTA's only item
        it.end = j > 0;
        if (it.end) return it;
        if (kByLength) {
            const int pair = sched[(int)blockIdx.x / p.heads];
            qb = pair % p.n_qb;
            it.b = pair / p.n_qb;
            it.h = (int)blockIdx.x % p.heads;
            it.bh = it.b * p.heads + it.h;
        } else {
            const int n = p.by_level ? p.units : p.n_qb, item = (int)blockIdx.x / p.split, a = item / n, r = item % n;
            it.bh = p.by_level ? r : a;
            qb = p.n_qb - 1 - (p.by_level ? a : r);
            it.b = it.bh / p.heads;
            it.h = it.bh % p.heads;
        }
    } else if (p.sorted) {
        const int G = (int)gridDim.x;
        it.end = (int64_t)j * G >= (int64_t)p.n_items;
        if (it.end) return it;
        const int pos = j * G + ((j & 1) ? G - 1 - (int)blockIdx.x : (int)blockIdx.x);
        if (pos >= p.n_items) return it;
        const int pair = sched[pos / p.heads];
        qb = pair % p.n_qb;
        it.b = pair / p.n_qb;
        it.h = pos % p.heads;
        it.bh = it.b * p.heads + it.h;
        if (p.keep_tab) keep_hi = 64 * sched[p.keep_tab + it.b];
    } else {
        const int G = (int)gridDim.x;
        if (kCausal) {
            int rank;
            if (!level_item(p.list, j, (int)blockIdx.x, G, it.bh, rank, it.end)) return it;
            qb = p.n_qb - 1 - rank;
        } else {
            // head after head; the lighter ragged blocks last
            it.end = j * G >= p.n_items;
            const int pos = j * G + ((j & 1) ? G - 1 - (int)blockIdx.x : (int)blockIdx.x);
            if (pos >= p.n_items) return it;
            const int whole = p.seq / 256, n_whole = p.units * whole;
            it.bh = pos < n_whole ? pos / whole : pos - n_whole;
            qb = pos < n_whole ? pos % whole : whole;
        }
        it.b = it.bh / p.heads;
        it.h = it.bh % p.heads;
    }
    it.valid = true;
    it.h_kv = it.h / (p.heads / p.heads_kv);
    // Single-tile items: block qb covers rows [128 qb, 128 qb + 128); the item's origin is kept 128 rows
    // earlier so that the block sits where tile 1 sits in a two-tile item (TcItem::qrow).
    it.q0 = kSingle ? qb * 128 - 128 : qb * 256;
    tc_steps<kCausal, kSingle>(p, it.b, it.q0, it.kv_hi, it.q_off, it.U0, it.U1, keep_hi, kSingle ? &it.t0 : nullptr);
    it.n_tiles = kSingle ? it.U0 : (max(it.U0, it.U1) + 1) / 2;
    return it;
}

// The rows of a split item: thread i of the 256 takes 4 columns of every (1024 / D)-th row of this CTA's 128 / C rows
// from the shared memory of all C CTAs, merges them and stores them.  All of a thread's remote loads are in flight
// together (read row by row, the 0.7 us of each round trip added 5 us to an item).
template <int D, int C>
__device__ __forceinline__ void merge_cluster(const TcParams& p, const TcItem& it, uint32_t parts, uint32_t stats) {
    constexpr int kPer = 128 / C * (D / 4) / 256;
    const int row0 = (int)blockIdx.x % C * (128 / C);
    float2 ml[kPer][C];
    float4 x[kPer][C];
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
        const int i = threadIdx.x + k * 256, row = row0 + i / (D / 4), ch = i % (D / 4);
#pragma unroll
        for (int r = 0; r < C; ++r) {
            ml[k][r] = ld_cluster_f2(map_cluster(stats + row * 8, r));
            x[k][r] = ld_cluster_f4(map_cluster(parts + row * (D * 4) + ((ch ^ (row & 7)) << 4), r));
        }
    }
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
        const int i = threadIdx.x + k * 256, ch = i % (D / 4), row = it.qrow(1, true) + row0 + i / (D / 4);
        float m = -INFINITY, l = 0.f;
#pragma unroll
        for (int r = 0; r < C; ++r) m = fmaxf(m, ml[k][r].x);
        float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int r = 0; r < C; ++r)
            if (ml[k][r].x > -INFINITY) {
                const float f = fast_exp2((ml[k][r].x - m) * p.scale_log2);
                l += f * ml[k][r].y;
                o = make_float4(o.x + f * x[k][r].x, o.y + f * x[k][r].y, o.z + f * x[k][r].z, o.w + f * x[k][r].w);
            }
        const bool seen = m > -INFINITY, valid = seen && l > 0.f;
        const float inv = valid ? 1.f / l : 0.f;
        if (row < p.seq) {
            *reinterpret_cast<uint2*>(p.out + it.b * p.o_stride_b + it.h * p.o_stride_h + (int64_t)row * p.o_stride_row + ch * 4) =
                valid ? make_uint2(float2_to_bf16x2(o.x * inv, o.y * inv), float2_to_bf16x2(o.z * inv, o.w * inv))
                      : make_uint2(0x7fc07fc0u, 0x7fc07fc0u);
            if (ch == 0 && p.lse)
                p.lse[(int64_t)it.bh * p.seq + row] =
                    valid ? (m * p.scale_log2 + fast_log2(l)) * kLn2 : (seen ? NAN : -INFINITY);
        }
    }
}

// Pipeline, per Q tile w and 64-key step u (buffer b = u & 1):
//   MMA:     S_w(u) -> TMEM S[w][b]            (SS, N = 64, D/16 k-steps)       commit s_full[w][b]
//   softmax: S[w][b] -> registers -> P (bf16) over the first 32 columns of S[w][b]   arrive p_full[w][b]
//   MMA:     O_w += P V(u)                      (TS, N = D, 4 k-steps)
//            then S_w(u+2) into the same buffer (in-order after the PV that read P from it)   commit s_full[w][b]
// S is double-buffered, so the softmax of step u+1 never waits for the PV of step u.  One commit a step: S_w(u+2) has
// retired only if PV(u) has, so a softmax warp that moves the reference maximum at step u+1 reads 'O is at rest' off
// the barrier of the next scores; only an item's last step but one has a commit for it (o_full).
// Per item and tile: q_full (Q landed) -> ... -> o_done (last PV retired) -> epilogue reads O
// (o_free: the next item's first PV may overwrite it), stages it (stage_full), and one thread stores it.
// q_empty, the next item's Q may land: at D = 64 behind the item's last score MMA, at D = 128 when the store has
// read the staged tile.  A tile that sees no key in an item takes no part in these (its rows are written as
// NaN directly).
template <int D, bool kCausal, bool kKeep, bool kSingle, bool kSplit, bool kByLength>
__global__ void __launch_bounds__(384, 1)
prefill_tc_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                  const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_o,
                  const TcParams p) {
    using C = TcCfg<D>;
    constexpr int KS = C::KS, VS = C::VS, TILE = C::TILE_BYTES, SUB = C::SUB_BYTES, HALF = C::HALF_BYTES;

    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* sQ = smem;
    uint8_t* sK = sQ + 2 * TILE;
    uint8_t* sV = sK + KS * TILE;
    uint8_t* sO = C::OWN_STAGE ? sV + VS * TILE : sQ;  // [2] staged O tiles
    uint64_t* bars = reinterpret_cast<uint64_t*>(sV + (VS + (C::OWN_STAGE ? 2 : 0)) * TILE);
    uint64_t* q_full = bars;              // [2]
    uint64_t* q_empty = q_full + 2;       // [2]  the next Q may land (see early_q)
    uint64_t* k_full = q_empty + 2;       // [KS]
    uint64_t* k_empty = k_full + KS;      // [2 tiles][KS]: the issuer of tile w is done with the slot
    uint64_t* v_full = k_empty + 2 * KS;  // [VS]
    uint64_t* v_empty = v_full + VS;      // [2 tiles][VS]
    uint64_t* s_full = v_empty + 2 * VS;  // [2 tiles][2 buffers]
    uint64_t* p_full = s_full + 4;        // [2 tiles][2 buffers]
    uint64_t* o_full = p_full + 4;        // [2]  one phase per item of two steps or more: its last PV but one has retired
    uint64_t* o_done = o_full + 2;        // [2]  one phase per item: the last PV of the tile has retired
    uint64_t* o_free = o_done + 2;        // [2]  one phase per item: the epilogue has read O out of TMEM
    uint64_t* stage_full = o_free + 2;    // [2]  one phase per item: the O tile is staged in shared memory
    uint64_t* done_bar = stage_full + 2;  // [1]
    uint64_t* merge_bar = done_bar + 1;   // [1]  single-tile items: both tiles have published their (max, sum)
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(merge_bar + 1);
    uint16_t* sched = reinterpret_cast<uint16_t*>(tmem_slot + 12);  // (after 8 words of the keep-flag scan) [SCHED_CAP] pair order, then [SCHED_CAP] step counts

    // Broadcasting the warp index makes it provably warp-uniform, so role dispatch and the MMA
    // operands stay on the uniform datapath.
    const int warp = __shfl_sync(kFullMask, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    const int N = p.seq;
    const int Nkv = p.seq_kv;

    // ------------------------------------------------------------------ setup
    // Launched with programmatic stream serialization, the CTA may start while the previous kernel of
    // the stream is still running: barrier set-up and the TMEM allocation then overlap that kernel's tail.
    // grid_dep_wait returns once the previous kernel has completed and its writes are visible (at once under
    // a normal launch); every global access of this kernel comes after one.
    if (p.sorted) {
        grid_dep_wait();  // kv_lens may be the previous kernel's output
        // Rank sort of the (batch, query block) pairs by their step count, descending, ties by index:
        // every CTA computes the same table.
        uint16_t* cost = sched + C::SCHED_CAP;
        const int n_pairs = p.n_items / p.heads;
        if (kKeep && p.keep_tab) {
            // The last kept key of every batch bounds its steps as a length would: each warp looks for it from the
            // end, 256 flags at a time (hidden tails beyond 4096 keys are not searched further).  At least one
            // step stays, so that rows without a kept key are recognised as in the other schedules.
            for (int b = warp; b < n_pairs / p.n_qb; b += 12) {
                const uint8_t* keep = p.key_keep + (int64_t)b * p.keep_batch_stride;
                int hi = 0, end = Nkv;
                for (int round = 0; round < 16 && end > 0 && hi == 0; ++round, end -= 256) {
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const int k = end - 1 - (i * 32 + lane);
                        if (k >= 0 && __ldg(keep + k) != 0) hi = max(hi, k + 1);
                    }
                    hi = __reduce_max_sync(kFullMask, hi);
                }
                hi = max(hi, max(end, 1));  // end: where the search stopped
                if (lane == 0) sched[p.keep_tab + b] = (uint16_t)((hi + 63) / 64);
            }
            __syncthreads();
        }
        for (int i = threadIdx.x; i < n_pairs; i += blockDim.x) {
            int kv_hi, q_off, U0, U1;
            const int keep_hi = (kKeep && p.keep_tab) ? 64 * sched[p.keep_tab + i / p.n_qb] : 0x7fffffff;
            tc_steps<kCausal, kSingle>(p, i / p.n_qb, kByLength ? (i % p.n_qb) * 128 - 128 : (i % p.n_qb) * 256, kv_hi,
                                       q_off, U0, U1, keep_hi);
            cost[i] = (uint16_t)min(U0 + U1, 65535);
        }
        __syncthreads();
        for (int i = threadIdx.x; i < n_pairs; i += blockDim.x) {
            const int ci = cost[i];
            int rank = 0;
            for (int k2 = 0; k2 < n_pairs; ++k2) {
                const int ck = cost[k2];
                rank += (ck > ci || (ck == ci && k2 < i)) ? 1 : 0;
            }
            sched[rank] = (uint16_t)i;
        }
        __syncthreads();
    }
    bool first_preloaded = false;  // meaningful in the producer thread only
    if (warp == 8) {
        // The barriers are initialised by the 32 lanes side by side (one thread doing all of them costs
        // ~0.4 us at the head of every CTA's critical path); all counts are 1 except the ones named here.
        for (int i = lane; i < C::NBARS; i += 32) {
            uint64_t* bar = bars + i;
            uint32_t count = 1;
            if (bar >= p_full && bar < p_full + 4) count = 128;
            else if (bar >= o_free && bar < o_free + 2) count = 128;
            else if (bar >= stage_full && bar < stage_full + 2) count = 128;
            else if (bar == done_bar) count = 2;
            else if (bar == merge_bar) count = 256;
            mbar_init(bar, count);
        }
        fence_barrier_init();
        __syncwarp();
    }
    if (warp == 8 && lane == 0) {
        prefetch_tensormap(&tm_q);
        prefetch_tensormap(&tm_k);
        prefetch_tensormap(&tm_v);
        prefetch_tensormap(&tm_o);
        fence_barrier_init();
        fence_proxy_async();
        grid_dep_wait();
        // Q and the first K tile of the first item are requested right away, so their latency
        // overlaps the TMEM allocation and the CTA-wide barrier below.
        const TcItem it = tc_item<kCausal, kSingle, kByLength>(0, p, sched);
        if (!it.end && it.valid && it.n_tiles > 0) {
            first_preloaded = true;
            if constexpr (kSingle) {
                // one Q tile serves both issuers (buffer 1, which also stages the output); K tile 0 follows
                mbar_arrive_expect_tx(&q_full[1], TILE);
#pragma unroll
                for (int s = 0; s < C::NSUB; ++s)
                    tma_load_4d(sQ + TILE + s * SUB, &tm_q, &q_full[1], s * 64, it.qrow(1, true), it.h, it.b);
                mbar_arrive_expect_tx(&k_full[0], TILE);
#pragma unroll
                for (int s = 0; s < C::NSUB; ++s)
                    tma_load_4d(sK + s * SUB, &tm_k, &k_full[0], s * 64, it.t0 * 128, it.h_kv, it.b);
            }
            for (int w = 0; w < 2 && !kSingle; ++w) {
                if (it.steps(w) == 0) continue;
                mbar_arrive_expect_tx(&q_full[w], TILE);
#pragma unroll
                for (int s = 0; s < C::NSUB; ++s)
                    tma_load_4d(sQ + w * TILE + s * SUB, &tm_q, &q_full[w], s * 64, it.qrow(w, kSingle), it.h, it.b);
                if (w == 0 || it.U0 == 0) {
                    mbar_arrive_expect_tx(&k_full[0], TILE);
#pragma unroll
                    for (int s = 0; s < C::NSUB; ++s)
                        tma_load_4d(sK + s * SUB, &tm_k, &k_full[0], s * 64, 0, it.h_kv, it.b);
                }
            }
        }
    }
    if (warp == 9) {
        tmem_alloc(tmem_slot, C::TMEM_COLS);
        tmem_relinquish();
    }
    if (kKeep && p.tighten) {
        // Keep flags mostly hide the tail of a sequence (its padding): the last kept key bounds the keys this CTA's
        // only item visits.  At least one key stays, so that an item has steps here exactly if it has them without
        // the bound (the preload above relies on that); a row that sees no kept key is recognised as before.
        grid_dep_wait();
        if (warp < 8) {
            const uint8_t* keep = p.key_keep + (int64_t)tc_item<kCausal, kSingle, kByLength>(0, p, sched).b * p.keep_batch_stride;
            int hi = 1;
            for (int i = threadIdx.x; i < Nkv; i += 256)
                if (__ldg(keep + i)) hi = i + 1;
            hi = __reduce_max_sync(kFullMask, hi);
            if (lane == 0) reinterpret_cast<int*>(tmem_slot + 4)[warp] = hi;
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    int keep_hi = 0x7fffffff;
    if (kKeep && p.tighten) {
        keep_hi = 1;
#pragma unroll
        for (int i = 0; i < 8; ++i) keep_hi = max(keep_hi, reinterpret_cast<const int*>(tmem_slot + 4)[i]);
    }
    grid_dep_wait();
    // The next kernel of the stream may be scheduled as SMs fall free (it waits as above before it reads or
    // writes anything): its launch latency and set-up hide behind the tail of this grid.
    grid_dep_launch();

    // The register hand-over sits inside each role's own branch: the compiler budgets the code
    // that follows a setmaxnreg only when no path with a different budget merges into it.
    if (warp >= 8) {
      asm volatile("setmaxnreg.dec.sync.aligned.u32 72;");
      if (warp == 8) {
        // ============================================================== TMA producer
        if (lane == 0 && kSingle) {
            // A single-tile item is its CTA's only item; Q and K tile 0 were requested during setup.  Each
            // issuer reads every tile once and asks for K tile u + 2 right after the PV of step u, so K runs
            // two tiles ahead of V in the request order: K1 | K2 V0 | K3 V1 | ...
            const TcItem it = tc_item<kCausal, kSingle, kByLength>(0, p, sched, keep_hi);
            if (first_preloaded) {
                bool ok = true;
                int kg = 1, vg = 0;
                auto load_k = [&](int t) {
                    const int ks = t % KS;
                    const uint32_t par = ((uint32_t)(t / KS) & 1u) ^ 1u;
                    if (!mbar_wait(&k_empty[ks], par, p.status, kToKEmpty) ||
                        !mbar_wait(&k_empty[KS + ks], par, p.status, kToKEmpty))
                        return false;
                    mbar_arrive_expect_tx(&k_full[ks], TILE);
#pragma unroll
                    for (int s = 0; s < C::NSUB; ++s)
                        tma_load_4d(sK + ks * TILE + s * SUB, &tm_k, &k_full[ks], s * 64, (it.t0 + t) * 128, it.h_kv, it.b);
                    ++kg;
                    return true;
                };
                if (it.n_tiles > 1) ok = load_k(1);
                for (int t = 0; t < it.n_tiles && ok; ++t) {
                    if (t + 2 < it.n_tiles && !load_k(t + 2)) break;
                    const int vs = t % VS;
                    const uint32_t par = ((uint32_t)(t / VS) & 1u) ^ 1u;
                    if (!mbar_wait(&v_empty[vs], par, p.status, kToVEmpty) ||
                        !mbar_wait(&v_empty[VS + vs], par, p.status, kToVEmpty))
                        break;
                    mbar_arrive_expect_tx(&v_full[vs], TILE);
#pragma unroll
                    for (int s = 0; s < C::NSUB; ++s)
                        tma_load_4d(sV + vs * TILE + s * SUB, &tm_v, &v_full[vs], s * 64, (it.t0 + t) * 128, it.h_kv, it.b);
                    ++vg;
                }
                // Drain: every copy this thread issued must have landed before the CTA may exit.
                mbar_wait(&q_full[1], 0u, p.status, kToDrain);
                for (int t = max(0, kg - KS); t < kg; ++t)
                    mbar_wait(&k_full[t % KS], (uint32_t)(t / KS) & 1u, p.status, kToDrain);
                for (int t = max(0, vg - VS); t < vg; ++t)
                    mbar_wait(&v_full[t % VS], (uint32_t)(t / VS) & 1u, p.status, kToDrain);
            }
        } else if (lane == 0) {
            int kg = 0, vg = 0;    // K / V tiles requested so far (ring position and phase)
            int na0 = 0, na1 = 0;  // items so far in which tile w took part (phase of its per-item barriers)
            bool ok = true;
            for (int j = 0; ok; ++j) {
                const TcItem it = tc_item<kCausal, kSingle, kByLength>(j, p, sched, keep_hi);
                if (it.end) break;
                if (!it.valid || it.n_tiles == 0) continue;  // nothing to load
                auto load_q = [&](int w, int na) {
                    // the previous item's O tile must have left the buffer
                    if (!mbar_wait(&q_empty[w], ((uint32_t)na & 1u) ^ 1u, p.status, kToQEmpty)) return false;
                    mbar_arrive_expect_tx(&q_full[w], TILE);
#pragma unroll
                    for (int s = 0; s < C::NSUB; ++s)
                        tma_load_4d(sQ + w * TILE + s * SUB, &tm_q, &q_full[w], s * 64, it.qrow(w, kSingle), it.h, it.b);
                    return true;
                };
                const bool pre = first_preloaded && j == 0;  // Q and K tile 0 were requested during setup
                if (it.U0 > 0) {
                    if (!pre && !load_q(0, na0)) break;
                    ++na0;
                }
                for (int t = 0; t < it.n_tiles && ok; ++t) {
                    // A slot is free once both issuers have released the tile it held.
                    const int ks = kg % KS, vs = vg % VS;
                    const uint32_t kpar = ((uint32_t)(kg / KS) & 1u) ^ 1u, vpar = ((uint32_t)(vg / VS) & 1u) ^ 1u;
                    if (!(pre && t == 0)) {
                        if (!mbar_wait(&k_empty[ks], kpar, p.status, kToKEmpty) ||
                            !mbar_wait(&k_empty[KS + ks], kpar, p.status, kToKEmpty)) {
                            ok = false;
                            break;
                        }
                        mbar_arrive_expect_tx(&k_full[ks], TILE);
#pragma unroll
                        for (int s = 0; s < C::NSUB; ++s)
                            tma_load_4d(sK + ks * TILE + s * SUB, &tm_k, &k_full[ks], s * 64, t * 128, it.h_kv, it.b);
                    }
                    ++kg;
                    if (t == 0 && it.U1 > 0) {  // tile 1 usually still works on the previous item: its Q comes second
                        if (!pre && !load_q(1, na1)) {
                            ok = false;
                            break;
                        }
                        ++na1;
                    }
                    if (!mbar_wait(&v_empty[vs], vpar, p.status, kToVEmpty) ||
                        !mbar_wait(&v_empty[VS + vs], vpar, p.status, kToVEmpty)) {
                        ok = false;
                        break;
                    }
                    mbar_arrive_expect_tx(&v_full[vs], TILE);
#pragma unroll
                    for (int s = 0; s < C::NSUB; ++s)
                        tma_load_4d(sV + vs * TILE + s * SUB, &tm_v, &v_full[vs], s * 64, t * 128, it.h_kv, it.b);
                    ++vg;
                }
            }
            // Drain: every copy this thread issued must have landed before the CTA may exit.
            if (na0 > 0) mbar_wait(&q_full[0], (uint32_t)(na0 - 1) & 1u, p.status, kToDrain);
            if (na1 > 0) mbar_wait(&q_full[1], (uint32_t)(na1 - 1) & 1u, p.status, kToDrain);
            for (int t = max(0, kg - KS); t < kg; ++t)
                mbar_wait(&k_full[t % KS], (uint32_t)(t / KS) & 1u, p.status, kToDrain);
            for (int t = max(0, vg - VS); t < vg; ++t)
                mbar_wait(&v_full[t % VS], (uint32_t)(t / VS) & 1u, p.status, kToDrain);
        }
      } else if (warp == 9 || warp == 10) {
        // ============================================================== MMA issuer of Q tile w
        // The whole warp runs this loop with uniform control flow and only the elected lane
        // executes the tcgen05 instructions: descriptors, addresses and loop state then live in
        // uniform registers, which is what the MMA instruction takes its operands from.
        {
            const int w = warp - 9;
            const bool leader = elect_one();
            constexpr uint32_t idesc_s = make_idesc_bf16(128, 64, 0, 0);
            constexpr uint32_t idesc_o = make_idesc_bf16(128, D, 0, 1);
            // Descriptors are built once; each MMA only adds an offset (in 16-byte units) to the
            // start-address field, so the issuing thread keeps ahead of the tensor pipe.
            const uint64_t dq = make_smem_desc_sw128(smem_u32(sQ + (kSingle ? 1 : w) * TILE), 16, 1024);
            const uint64_t dk = make_smem_desc_sw128(smem_u32(sK), 16, 1024);
            const uint64_t dv = make_smem_desc_sw128(smem_u32(sV), SUB, 1024);
            const uint32_t tS = tmem_base + C::COL_S + w * 128, tO = tmem_base + C::COL_O + w * D;
            uint64_t* const ke = k_empty + w * KS;
            uint64_t* const ve = v_empty + w * VS;
            uint64_t* const sf = s_full + w * 2;
            uint64_t* const pf = p_full + w * 2;
            // Ring slots and phases are carried along: every instruction between a P that has arrived and the score MMA
            // behind its PV is on the critical path of the softmax warps, and so is whatever this loop does instead of
            // looking for the next P.
            uint32_t ks = 0, kph = 0, vs = 0, vph = 0;  // slot and phase of the next K / V tile
            uint32_t p0 = 0, p1 = 0;                    // phase of the next P in each score buffer
            uint32_t na = 0;                            // items so far in which this tile took part
            auto wait = [&](uint64_t* bar, uint32_t parity, int code) {
                return __all_sync(kFullMask, mbar_wait(bar, parity, p.status, code));
            };
            auto next_k = [&] {
                if (++ks == KS) ks = 0, kph ^= 1;
            };
            auto next_v = [&] {
                if (++vs == VS) vs = 0, vph ^= 1;
            };
            // (called by the elected lane)
            auto issue_S = [&](int b, uint64_t bk) {
#pragma unroll
                for (int kk = 0; kk < D / 16; ++kk) {
                    const uint32_t off = (uint32_t)(((kk / 4) * SUB + (kk % 4) * 32) >> 4);
                    mma_ss(tS + b * 64, dq + off, bk + off, idesc_s, kk > 0);
                }
                mma_commit(&sf[b]);
            };
            auto issue_PV = [&](int b, uint64_t bv, uint32_t acc) {  // P (bf16) sits in the first 32 columns of the score buffer
#pragma unroll
                for (int kk = 0; kk < 4; ++kk)
                    mma_ts(tO, tS + b * 64 + kk * 8, bv + (uint64_t)((kk * 2048) >> 4), idesc_o, kk > 0 ? 1u : acc);
            };
            constexpr uint32_t kTileEnc = TILE >> 4, kHalfEnc = HALF >> 4;
            constexpr bool early_q = C::OWN_STAGE;  // nothing is staged in the Q buffer: it is free behind the item's last scores
            bool ok = true;
            for (int j = 0; ok; ++j) {
                const TcItem it = tc_item<kCausal, kSingle, kByLength>(j, p, sched, keep_hi);
                if (it.end) break;
                if (!it.valid || it.n_tiles == 0) continue;
                const int n_u = it.steps(w);
                if (kSingle) {
                    // ---- the tile's steps are every second 64-key step: half w of every K/V tile
                    const uint64_t bk0 = dk + w * kHalfEnc, bv0 = dv + w * kHalfEnc;
                    if (n_u > 0) {
                        ok = wait(&k_full[ks], kph, kToKFull) && wait(&q_full[1], na & 1u, kToQ);
                        if (!ok) break;
                        tc_fence_after();
                        if (leader) {
                            issue_S(0, bk0 + ks * kTileEnc);
                            mma_commit(&ke[ks]);
                        }
                        next_k();
                        if (n_u > 1) {
                            if (!wait(&k_full[ks], kph, kToKFull)) { ok = false; break; }
                            tc_fence_after();
                            if (leader) {
                                issue_S(1, bk0 + ks * kTileEnc);
                                mma_commit(&ke[ks]);
                            }
                            next_k();
                        }
                        for (int u = 0; u < n_u && ok; u += 2) {
#pragma unroll
                            for (int b = 0; b < 2; ++b) {
                                if (b == 1 && u + 1 >= n_u) break;
                                const bool more = u + b + 2 < n_u;
                                ok = wait(&v_full[vs], vph, kToVFull) && (!more || wait(&k_full[ks], kph, kToKFull)) &&
                                     wait(&pf[b], b ? p1 : p0, kToPFull);
                                if (!ok) break;
                                (b ? p1 : p0) ^= 1;
                                tc_fence_after();
                                if (leader) {
                                    issue_PV(b, bv0 + vs * kTileEnc, (u + b > 0) ? 1u : 0u);
                                    if (more) {
                                        issue_S(b, bk0 + ks * kTileEnc);
                                        mma_commit(&ke[ks]);
                                    }
                                    mma_commit(&ve[vs]);
                                    if (u + b == n_u - 2) mma_commit(&o_full[w]);
                                    if (u + b == n_u - 1) mma_commit(&o_done[w]);
                                }
                                next_v();
                                if (more) next_k();
                            }
                        }
                        ++na;
                    }
                } else {
                    // ---- steps 2t and 2t + 1 read the halves of K/V tile t and use score buffers 0 and 1
                    if (n_u > 0) {
                        ok = wait(&k_full[ks], kph, kToKFull) && wait(&q_full[w], na & 1u, kToQ);
                        if (!ok) break;
                        tc_fence_after();
                        if (leader) {
                            const uint64_t bk = dk + ks * kTileEnc;
                            issue_S(0, bk);
                            if (n_u > 1) issue_S(1, bk + kHalfEnc);
                            mma_commit(&ke[ks]);
                            if (early_q && n_u <= 2) mma_commit(&q_empty[w]);
                        }
                        next_k();
                    }
                    for (int u = 0; u < n_u; u += 2) {
                        const bool more = u + 2 < n_u;
                        ok = wait(&v_full[vs], vph, kToVFull) && (!more || wait(&k_full[ks], kph, kToKFull)) &&
                             // the previous item's epilogue must have read O_w before it is overwritten
                             (u > 0 || na == 0 || wait(&o_free[w], (na - 1) & 1u, kToOFree)) && wait(&pf[0], p0, kToPFull);
                        if (!ok) break;
                        p0 ^= 1;
                        const uint64_t bk = dk + ks * kTileEnc, bv = dv + vs * kTileEnc;
                        tc_fence_after();
                        if (leader) {
                            issue_PV(0, bv, u > 0 ? 1u : 0u);
                            if (more) issue_S(0, bk);
                            if (early_q && u + 3 == n_u) mma_commit(&q_empty[w]);
                            if (u + 2 == n_u) mma_commit(&o_full[w]);
                        }
                        if (u + 1 < n_u) {
                            ok = wait(&pf[1], p1, kToPFull);
                            if (!ok) break;
                            p1 ^= 1;
                            tc_fence_after();
                            if (leader) {
                                issue_PV(1, bv + kHalfEnc, 1u);
                                if (u + 3 < n_u) issue_S(1, bk + kHalfEnc);
                                if (early_q && u + 4 == n_u) mma_commit(&q_empty[w]);
                                if (u + 3 == n_u) mma_commit(&o_full[w]);
                            }
                        }
                        if (leader) {
                            if (more) mma_commit(&ke[ks]);
                            else mma_commit(&o_done[w]);
                            mma_commit(&ve[vs]);
                        }
                        next_v();
                        if (more) next_k();
                    }
                    if (n_u > 0) ++na;
                }
                if (!ok) break;
                // Tiles this Q tile does not read (it sees fewer keys than the other one) are passed on
                // once they have landed, which keeps this issuer inside the ring window.
                for (int t = kSingle ? n_u : (n_u + 1) / 2; t < it.n_tiles && ok; ++t) {
                    ok = wait(&k_full[ks], kph, kToKFull) && wait(&v_full[vs], vph, kToVFull);
                    if (ok && leader) {
                        mma_commit(&ke[ks]);
                        mma_commit(&ve[vs]);
                    }
                    next_k();
                    next_v();
                }
            }
            // All MMAs of both issuers must retire before TMEM is freed.
            if (leader) mma_commit(done_bar);
            wait(done_bar, 0, kToDone);
        }
      }  // warp 11 idle: it only completes the warpgroup for setmaxnreg
      if constexpr (kSplit) {
          __syncwarp();
          cluster_sync_all();
          cluster_sync_all();
      }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 216;");
        // ============================================================== softmax / epilogue warps
        const int w = warp >> 2;                       // Q tile
        const int row_in_tile = (warp & 3) * 32 + lane;
        const uint32_t lane_sel = (uint32_t)((warp & 3) * 32) << 16;
        const uint32_t tS = tmem_base + lane_sel + C::COL_S + w * 128;
        const uint32_t tO = tmem_base + lane_sel + C::COL_O + w * D;
        const float c = p.scale_log2;
        const float grow = c > 0.f ? fminf(8.f / c, 3.0e38f) : 3.0e38f;  // raw scores that a factor of 2^8 stands for
        int na = 0;            // items so far in which this tile took part
        int cs0 = 0, cs1 = 0;  // s_full phases of each S buffer consumed before the item
        int co = 0;            // items of two steps or more before this one (phase of o_full)
        bool ok = true;

        for (int j = 0; ok; ++j) {
            const TcItem it = tc_item<kCausal, kSingle, kByLength>(j, p, sched, keep_hi);
            if (it.end) break;
            if (!it.valid) continue;
            const int n_iter = it.steps(w);
            constexpr bool il = kSingle;  // this tile's steps are every second 64-key step of the block
            const int bh = it.bh, kv_hi = it.kv_hi, q_off = it.q_off;
            const int row = it.qrow(w, il) + row_in_tile;  // query index within the sequence
            const uint8_t* keep = kKeep ? p.key_keep + (int64_t)it.b * p.keep_batch_stride : nullptr;

            // The tile sees no key: NaN rows, LSE = -inf (cpu_forward.rs:411-420).  A single-tile item whose
            // other tile has a step still goes through the merge below with an empty partial result.
            if (n_iter == 0 && !kSplit && !(il && it.n_tiles > 0)) {
                if (row < N && !(il && w == 0)) {
                    uint4* dst = reinterpret_cast<uint4*>(p.out + it.b * p.o_stride_b + it.h * p.o_stride_h +
                                                          (int64_t)row * p.o_stride_row);
#pragma unroll
                    for (int i = 0; i < D / 8; ++i) dst[i] = make_uint4(0x7fc07fc0u, 0x7fc07fc0u, 0x7fc07fc0u, 0x7fc07fc0u);
                    if (p.lse) p.lse[(int64_t)bh * N + row] = -INFINITY;
                }
                continue;
            }

            // The tile's last O has been read out of its staging buffer; the other threads learn it through o_done, below.
            if (C::OWN_STAGE && !il && row_in_tile == 0) tma_store_wait_read();
            float m_ref = -INFINITY;  // reference max (raw score units) the running sums are relative to; -inf: no score was visible yet
            float l = 0.f;
            for (int u = 0; u < n_iter; ++u) {
                const int buf = u & 1;
                const int col0 = (il ? 2 * (it.t0 + u) + w : u) * 64;
                uint32_t keep0 = 0xffffffffu, keep1 = 0xffffffffu;
                if (kKeep) {
                    // Mask::Padding keep flags (mask.rs:44) of the step's 64 keys as two 32-bit words: each lane reads
                    // two flags, issued before the wait for the scores so that their latency hides behind it.  (One
                    // flag load per key in every thread, as this replaces, cost 6 x the rest of the step.)
                    const int k0 = col0 + lane, k1 = k0 + 32;
                    const bool f0 = k0 >= Nkv || __ldg(keep + k0) != 0, f1 = k1 >= Nkv || __ldg(keep + k1) != 0;
                    keep0 = __ballot_sync(kFullMask, f0);
                    keep1 = __ballot_sync(kFullMask, f1);
                }
                // (No vote on the outcome: a wait that gives up clears the thread's `ok`, which the vote below sees.)
                ok &= mbar_wait(&s_full[w * 2 + buf], (uint32_t)((buf ? cs1 : cs0) + (u >> 1)) & 1u, p.status, kToSFull);
                tc_fence_after();
                if (il && w == 1 && u == 0 && p.stagger_clocks > 0) {
                    // The two tiles of a single-tile item start together and would stay in step: both
                    // warps of a scheduler would then wait for TMEM at the same moments.  Half a step of
                    // offset lets one tile's loads and stores hide behind the other's arithmetic
                    // (measured: 0.5-1 us of 21 on B=1 H=8 N=2048 D=64; RT_ATTN_PREFILL_STAGGER sets the clocks).
                    const long long t0 = clock64();
                    while (clock64() - t0 < p.stagger_clocks) {}
                }

                uint32_t s[64];
                {
                    uint32_t(&s0)[32] = *reinterpret_cast<uint32_t(*)[32]>(&s[0]);
                    uint32_t(&s1)[32] = *reinterpret_cast<uint32_t(*)[32]>(&s[32]);
                    tmem_ld32(tS + buf * 64, s0);
                    tmem_ld32(tS + buf * 64 + 32, s1);
                    tc_wait_ld();
                }

                // ---- masks: keys beyond kv_hi, causal diagonal, keep flags
                int lim = kv_hi - 1 - col0;                       // last visible column in this step
                if (kCausal) lim = min(lim, row + q_off - col0);
                if (lim < 63) {
#pragma unroll
                    for (int i = 0; i < 64; ++i)
                        if (i > lim) s[i] = 0xff800000u;  // -inf
                }
                if (kKeep && (keep0 & keep1) != 0xffffffffu) {
#pragma unroll
                    for (int i = 0; i < 32; ++i) {
                        if (!(keep0 & (1u << i))) s[i] = 0xff800000u;
                        if (!(keep1 & (1u << i))) s[32 + i] = 0xff800000u;
                    }
                }

                // ---- row max (three-input max halves the instruction count)
                float mx0 = -INFINITY, mx1 = -INFINITY, mx2 = -INFINITY, mx3 = -INFINITY;
#pragma unroll
                for (int i = 0; i < 64; i += 8) {
                    mx0 = max3(mx0, __uint_as_float(s[i]), __uint_as_float(s[i + 1]));
                    mx1 = max3(mx1, __uint_as_float(s[i + 2]), __uint_as_float(s[i + 3]));
                    mx2 = max3(mx2, __uint_as_float(s[i + 4]), __uint_as_float(s[i + 5]));
                    mx3 = max3(mx3, __uint_as_float(s[i + 6]), __uint_as_float(s[i + 7]));
                }
                const float mx = fmaxf(fmaxf(mx0, mx1), fmaxf(mx2, mx3));

                // ---- lazy rescale: move the reference max only when it would grow by > 2^8
                if (__any_sync(kFullMask, mx > m_ref + grow || !ok)) {
                    if (u > 0) {
                        // O must be at rest: the PV of step u - 1 has to be complete.  The scores of step u + 1 were
                        // requested right behind it; the last step has a barrier of its own for this.
                        ok &= u + 1 < n_iter
                            ? mbar_wait(&s_full[w * 2 + 1 - buf], (uint32_t)((buf ? cs0 : cs1) + ((u + 1) >> 1)) & 1u, p.status, kToOFull)
                            : mbar_wait(&o_full[w], (uint32_t)co & 1u, p.status, kToOFull);
                    }
                    ok = __all_sync(kFullMask, ok);
                    if (!ok) break;
                    tc_fence_after();
                    const float m_new = fmaxf(m_ref, mx);
                    const float alpha = (m_new == -INFINITY) ? 1.f : fast_exp2((m_ref - m_new) * c);
                    l *= alpha;
                    m_ref = m_new;
                    if (u > 0) {
#pragma unroll
                        for (int ch = 0; ch < D / 32; ++ch) {
                            uint32_t o[32];
                            tmem_ld32(tO + ch * 32, o);
                            tc_wait_ld();
#pragma unroll
                            for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
                            tmem_st32(tO + ch * 32, o);
                        }
                        tc_wait_st();
                    }
                }

                // ---- P = exp2(s*c - m*c), row sum, bf16 pack, store to TMEM over S (packed f32x2 math)
                const float mc = (m_ref == -INFINITY) ? 0.f : m_ref * c;
                const float2 c2 = make_float2(c, c), nmc2 = make_float2(-mc, -mc);
                float2 sum_a = make_float2(0.f, 0.f), sum_b = make_float2(0.f, 0.f);
#pragma unroll
                for (int ch = 0; ch < 2; ++ch) {
                    uint32_t pk[16];
#pragma unroll
                    for (int i = 0; i < 16; i += 2) {
                        const float2 xa = __ffma2_rn(
                            make_float2(__uint_as_float(s[ch * 32 + 2 * i]), __uint_as_float(s[ch * 32 + 2 * i + 1])), c2,
                            nmc2);
                        const float2 xb = __ffma2_rn(
                            make_float2(__uint_as_float(s[ch * 32 + 2 * i + 2]), __uint_as_float(s[ch * 32 + 2 * i + 3])),
                            c2, nmc2);
                        // a quarter of the exponentials go to the polynomial (see exp2_poly2)
                        const float2 pa = poly_pair(i) ? exp2_poly2(xa) : make_float2(fast_exp2(xa.x), fast_exp2(xa.y));
                        const float2 pb = poly_pair(i + 1) ? exp2_poly2(xb) : make_float2(fast_exp2(xb.x), fast_exp2(xb.y));
                        sum_a = __fadd2_rn(sum_a, pa);
                        sum_b = __fadd2_rn(sum_b, pb);
                        pk[i] = float2_to_bf16x2(pa.x, pa.y);
                        pk[i + 1] = float2_to_bf16x2(pb.x, pb.y);
                    }
                    tmem_st16(tS + buf * 64 + ch * 16, pk);
                }
                l += (sum_a.x + sum_a.y) + (sum_b.x + sum_b.y);
                tc_wait_st();  // warp-wide: every lane's part of the store has completed
                tc_fence_before();
                mbar_arrive(&p_full[w * 2 + buf]);
            }
            ok = __all_sync(kFullMask, ok);
            if (!ok) break;
            const bool seen = m_ref > -INFINITY;  // the row has met a score that no mask hides

            // ---- epilogue: O / l -> bf16 into the (now idle) shared-memory tile of Q_w in the swizzled
            // layout of the output tensor map, then one TMA store per 64-column half: 16-byte shared
            // stores instead of row-strided global stores, and rows past N are clipped by the hardware.
            if (n_iter > 0 && !__all_sync(kFullMask, mbar_wait(&o_done[w], (uint32_t)na & 1u, p.status, kToOFull))) {
                ok = false;
                break;
            }
            tc_fence_after();
            if (il) {
                // ---- single-tile item: the two tiles hold partial results of the same 128 rows (even and odd
                // 64-key steps).  Each thread publishes its (max, sum, seen) in the first columns of its tile's
                // idle score buffer, TMEM being readable by the other warpgroup's warp of the same lane
                // quarter; after the barrier every thread knows both partials of its row.  The merged row is
                //   O = (f0 O_0 + f1 O_1) / (f0 l_0 + f1 l_1),  f_w = 2^((m_w - max(m_0, m_1)) c),
                // and warpgroup w produces columns [w D/2, (w+1) D/2) of it from both accumulators.
                {
                    uint32_t ex[16];
#pragma unroll
                    for (int i = 0; i < 16; ++i) ex[i] = 0u;
                    ex[0] = __float_as_uint(m_ref);
                    ex[1] = __float_as_uint(l);
                    ex[2] = seen ? 1u : 0u;
                    tmem_st16(tS, ex);
                    tc_wait_st();
                    tc_fence_before();
                    mbar_arrive(merge_bar);
                }
                if (!__all_sync(kFullMask, mbar_wait(merge_bar, (uint32_t)na & 1u, p.status, kToMerge))) {
                    ok = false;
                    break;
                }
                tc_fence_after();
                const uint32_t tS_other = tmem_base + lane_sel + C::COL_S + (1 - w) * 128;
                const uint32_t tO_other = tmem_base + lane_sel + C::COL_O + (1 - w) * D;
                uint32_t exo[16];
                tmem_ld16(tS_other, exo);
                tc_wait_ld();
                const float m_o = __uint_as_float(exo[0]), l_o = __uint_as_float(exo[1]);
                const bool seen_any = seen || (exo[2] != 0u);
                const float m_all = fmaxf(m_ref, m_o);
                const float f_own = (m_ref == -INFINITY) ? 0.f : fast_exp2((m_ref - m_all) * c);
                const float f_oth = (m_o == -INFINITY) ? 0.f : fast_exp2((m_o - m_all) * c);
                const float l_all = f_own * l + f_oth * l_o;
                const bool valid = seen_any && (l_all > 0.f);
                const float inv = valid ? 1.f / l_all : 0.f;
                const float a_own = kSplit ? f_own : f_own * inv, a_oth = kSplit ? f_oth : f_oth * inv;
                const bool has_own = n_iter > 0, has_oth = it.steps(1 - w) > 0;  // an idle tile's accumulator was never written
                // The merged half rows go straight to global memory (64 or 128 contiguous bytes per thread): the CTA
                // has no further item, and a staged tile, its barrier and a TMA store would only lengthen the
                // tail of a launch whose time is its longest CTA.
                __nv_bfloat16* dst = p.out + it.b * p.o_stride_b + it.h * p.o_stride_h + (int64_t)row * p.o_stride_row;
#pragma unroll
                for (int cq = 0; cq < D / 64; ++cq) {
                    const int ch = w * (D / 64) + cq;
                    uint32_t oa[32], ob[32];
                    float part[32];
                    if (has_own) tmem_ld32(tO + ch * 32, oa);
                    if (has_oth) tmem_ld32(tO_other + ch * 32, ob);
                    tc_wait_ld();
#pragma unroll
                    for (int v4 = 0; v4 < 4; ++v4) {
                        uint4 pack;
                        uint32_t* pw = reinterpret_cast<uint32_t*>(&pack);
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const int e = v4 * 8 + 2 * i;
                            const float x0 = (has_own ? __uint_as_float(oa[e]) * a_own : 0.f) +
                                             (has_oth ? __uint_as_float(ob[e]) * a_oth : 0.f);
                            const float x1 = (has_own ? __uint_as_float(oa[e + 1]) * a_own : 0.f) +
                                             (has_oth ? __uint_as_float(ob[e + 1]) * a_oth : 0.f);
                            pw[i] = valid ? float2_to_bf16x2(x0, x1) : 0x7fc07fc0u;
                            if constexpr (kSplit) part[e] = x0, part[e + 1] = x1;
                        }
                        if (!kSplit && row < N) *reinterpret_cast<uint4*>(dst + ch * 32 + v4 * 8) = pack;
                    }
                    if constexpr (kSplit) {
                        // This CTA's partial row, relative to m_all, in f32 over the K ring (every MMA of the CTA has
                        // retired): 16-byte chunks swizzled by the row, so that 8 lanes' rows meet 8 bank groups.
#pragma unroll
                        for (int i = 0; i < 8; ++i)
                            *reinterpret_cast<float4*>(sK + row_in_tile * (D * 4) + (((ch * 8 + i) ^ (row_in_tile & 7)) << 4)) =
                                make_float4(part[4 * i], part[4 * i + 1], part[4 * i + 2], part[4 * i + 3]);
                    }
                }
                if (kSplit && w == 1)
                    reinterpret_cast<float2*>(sV)[row_in_tile] = make_float2(seen_any ? m_all : -INFINITY, l_all);
                if (!kSplit && w == 1 && p.lse && row < N)
                    p.lse[(int64_t)bh * N + row] =
                        valid ? (m_all * c + fast_log2(l_all)) * kLn2 : (seen_any ? NAN : -INFINITY);
            } else {
                // A masked score costs the polynomial path 2^-125 instead of 0, so a row counts as
                // empty when it never saw a visible score, not when its sum is exactly 0.
                const bool valid = seen && (l > 0.f);
                const float inv = valid ? 1.f / l : 0.f;
                uint8_t* stage = sO + w * TILE + row_in_tile * 128;  // (in the Q buffer: every score MMA that read Q_w has retired)
                __nv_bfloat16* dst = p.out + it.b * p.o_stride_b + it.h * p.o_stride_h + (int64_t)row * p.o_stride_row;
#pragma unroll
                for (int ch = 0; ch < D / 32; ++ch) {
                    uint32_t o[32];
                    tmem_ld32(tO + ch * 32, o);
                    tc_wait_ld();
                    if (ch == D / 32 - 1) {  // O_w is in registers: the next item's first PV may overwrite it
                        tc_fence_before();
                        mbar_arrive(&o_free[w]);
                    }
#pragma unroll
                    for (int v4 = 0; v4 < 4; ++v4) {
                        uint4 pack;
                        uint32_t* pw = reinterpret_cast<uint32_t*>(&pack);
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const float a = __uint_as_float(o[v4 * 8 + 2 * i]) * inv;
                            const float bb = __uint_as_float(o[v4 * 8 + 2 * i + 1]) * inv;
                            pw[i] = valid ? float2_to_bf16x2(a, bb) : 0x7fc07fc0u;
                        }
                        const int cc = ch * 4 + v4;  // 16-byte chunk of the row: sub-tile cc/8, chunk cc%8
                        if (p.direct_out) {  // the CTA's only item: no overlap to win, the staged store would just add to the tail
                            if (row < N) *reinterpret_cast<uint4*>(dst + cc * 8) = pack;
                        } else {
                            *reinterpret_cast<uint4*>(stage + (cc / 8) * SUB + (((cc % 8) ^ (row_in_tile & 7)) << 4)) = pack;
                        }
                    }
                }
                if (p.lse && row < N)
                    p.lse[(int64_t)bh * N + row] =
                        valid ? (m_ref * c + fast_log2(l)) * kLn2 : (seen ? NAN : -INFINITY);
                if (!p.direct_out) {
                    fence_proxy_async();  // generic-proxy writes above -> visible to the TMA (async proxy) read
                    mbar_arrive(&stage_full[w]);
                }
            }
            if (row_in_tile == 0 && !il && !p.direct_out) {
                if (!mbar_wait(&stage_full[w], (uint32_t)na & 1u, p.status, kToStage)) {
                    ok = false;
                } else {
#pragma unroll
                    for (int s = 0; s < C::NSUB; ++s)
                        tma_store_4d(&tm_o, sO + w * TILE + s * SUB, s * 64, it.qrow(w, il), it.h, it.b);
                    tma_store_commit();
                    if (!C::OWN_STAGE) {
                        tma_store_wait_read();  // the staged tile has been read: the next Q may land
                        mbar_arrive(&q_empty[w]);
                    }
                }
            }
            ok = __all_sync(kFullMask, ok);
            ++na;
            cs0 += (n_iter + 1) / 2;
            cs1 += n_iter / 2;
            co += n_iter > 1 ? 1 : 0;
        }
        if (C::OWN_STAGE && !kSingle && row_in_tile == 0) tma_store_wait_read();  // shared memory stays until the last store has read it
        if constexpr (kSplit) {
            // ---- the cluster's partial rows: CTA r reads its 128 / split rows from every CTA's shared memory, merges them
            // as above and stores them.  (A CTA that gave up on a wait still meets the barriers.)
            cluster_sync_all();
            const TcItem it = tc_item<kCausal, kSingle, kByLength>(0, p, sched, keep_hi);
            if (ok) {
                if (p.split == 2) merge_cluster<D, 2>(p, it, smem_u32(sK), smem_u32(sV));
                else if (p.split == 4) merge_cluster<D, 4>(p, it, smem_u32(sK), smem_u32(sV));
                else merge_cluster<D, 8>(p, it, smem_u32(sK), smem_u32(sV));
            }
            cluster_sync_all();  // no CTA leaves while its partial rows are being read
        }
    }

    // ------------------------------------------------------------------ teardown
    tc_fence_before();
    __syncthreads();
    if (warp == 9) {
        tc_fence_after();
        tmem_dealloc(tmem_base, C::TMEM_COLS);
    }
}

// ---------------------------------------------------------------------- host side

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn get_encode_fn() {
    static EncodeTiledFn fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* sym = nullptr;
        cudaDriverEntryPointQueryResult qres;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &qres) == cudaSuccess &&
            qres == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(sym);
    });
    return fn;
}

bool encode_bf16_map_cached(CUtensorMap* out, int rank, const void* base, const uint64_t* dims,
                            const uint64_t* strides_bytes, const uint32_t* box) {
    struct Key {
        const void* base;
        uint64_t dims[4], strides[3];
        uint32_t box[4];
        int rank;
    };
    // 64 sets of two entries, the older of a set replaced.  A training step uses 12 maps per set of tensors and a
    // caller often rotates several sets; the 32-entry list this replaces was searched front to back (up to 0.3 us a
    // map) and re-encoded every map (~1 us) once three such sets took turns.
    constexpr int kSets = 64;
    struct Cache {
        Key key[kSets][2];
        CUtensorMap map[kSets][2];
        uint8_t used[kSets] = {}, newest[kSets] = {};
    };
    thread_local Cache cache;
    if (rank < 1 || rank > 4) return false;
    Key k;
    memset(&k, 0, sizeof(k));
    k.base = base;
    k.rank = rank;
    for (int i = 0; i < rank; ++i) {
        k.dims[i] = dims[i];
        k.box[i] = box[i];
        if (i + 1 < rank) k.strides[i] = strides_bytes[i];
    }
    uint64_t h = (uint64_t)(uintptr_t)base >> 9;
    h = (h ^ (uint64_t)box[rank > 1 ? 1 : 0] ^ (dims[rank > 1 ? 1 : 0] << 7)) * 0x9E3779B97F4A7C15ull;
    const int set = (int)(h >> 58);
    for (int i = 0; i < cache.used[set]; ++i)
        if (memcmp(&cache.key[set][i], &k, sizeof(Key)) == 0) {
            *out = cache.map[set][i];
            return true;
        }
    EncodeTiledFn enc = get_encode_fn();
    if (!enc) return false;
    cuuint64_t d[4], st[3];
    cuuint32_t bx[4], estr[4] = {1, 1, 1, 1};
    for (int i = 0; i < rank; ++i) {
        d[i] = dims[i];
        bx[i] = box[i];
        if (i + 1 < rank) st[i] = strides_bytes[i];
    }
    if (enc(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, (cuuint32_t)rank, const_cast<void*>(base), d, st, bx, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return false;
    const int slot = cache.used[set] < 2 ? cache.used[set]++ : 1 - cache.newest[set];
    cache.newest[set] = (uint8_t)slot;
    cache.key[set][slot] = k;
    cache.map[set][slot] = *out;
    return true;
}

bool make_tensor_map_bf16_4d(CUtensorMap* map, const void* base, int64_t batch, int64_t heads, int64_t seq, int dim,
                             int64_t stride_b, int64_t stride_h, int64_t stride_row, int box_rows = 128);

// View of a [B, H, N, D] bf16 tensor with arbitrary batch / head / row strides (inner dim contiguous)
// as a 4-D TMA tensor (d, row, head, batch); box = 64 columns x box_rows (128, or 64) rows of one (b,h), 128-byte
// swizzle.  Rows past N are zero-filled on loads and clipped on stores, so tiles never touch a
// neighbouring head.  Strides are in elements and must be multiples of 8 (16 bytes).
bool make_tensor_map_bf16_4d(CUtensorMap* map, const void* base, int64_t batch, int64_t heads, int64_t seq, int dim,
                             int64_t stride_b, int64_t stride_h, int64_t stride_row, int box_rows) {
    const uint64_t dims[4] = {(uint64_t)dim, (uint64_t)seq, (uint64_t)heads, (uint64_t)batch};
    const uint64_t strides[3] = {(uint64_t)stride_row * 2, (uint64_t)stride_h * 2, (uint64_t)stride_b * 2};
    const uint32_t box[4] = {64, (uint32_t)box_rows, 1, 1};
    return encode_bf16_map_cached(map, 4, base, dims, strides, box);
}

// The contiguous [B*H, N, D] view used by the self-test kernel.
bool make_tensor_map_bf16_3d(CUtensorMap* map, const void* base, int64_t bh, int64_t seq, int dim) {
    const uint64_t dims[3] = {(uint64_t)dim, (uint64_t)seq, (uint64_t)bh};
    const uint64_t strides[2] = {(uint64_t)dim * 2, (uint64_t)seq * dim * 2};
    const uint32_t box[3] = {64, 128, 1};
    return encode_bf16_map_cached(map, 3, base, dims, strides, box);
}

template <int D, bool kCausal, bool kKeep, bool kSingle, bool kSplit, bool kByLength = false>
static cudaError_t launch_tc_s(const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv, const CUtensorMap& mo,
                             const TcParams& p, int64_t n_ctas, cudaStream_t stream) {
    auto kern = prefill_tc_kernel<D, kCausal, kKeep, kSingle, kSplit, kByLength>;
    cudaError_t e = set_max_dynamic_smem_once<prefill_tc_kernel<D, kCausal, kKeep, kSingle, kSplit, kByLength>>(TcCfg<D>::SMEM_BYTES);
    if (e != cudaSuccess) return e;
    // RT_ATTN_PREFILL_PDL=0|1 forces programmatic stream serialization off or on.
    static const int env_pdl = [] {
        const char* s = getenv("RT_ATTN_PREFILL_PDL");
        return s ? (s[0] == '0' ? 0 : 1) : -1;
    }();
    // The next launch's set-up, and its first CTAs on SMs that run out of work, overlap this one's tail: 2 to 25 % of
    // launches below 50 us, 0.5 to 2 % of ones up to 1 ms, over 1100 shapes of all kinds and 1 to 30 items per SM.  One
    // kind is faster without: a wave of 128-row items at D = 128 of which many walk one long K/V in step (CTAs that start
    // where SMs fall free lose the step).  16 and more on one K/V: N=4352 H=3 without a mask 35.1 against 38.5 us, causal
    // 34.2 / 36.3, N=8192 H=2 59.7 / 64.0; level at 2000 keys, 0 to 5 % either way at 3000.  4 to 15 on one: 1 to 2.5 %
    // from 7000 keys on, below them the overlap gains 1 to 5 %, as it does at D = 64 everywhere.
    const int share = p.n_qb * (p.heads / p.heads_kv);
    const bool in_step = D == 128 && kSingle && !kSplit && p.n_items <= sm_count() &&
                         p.seq_kv >= (share >= 16 ? 3500 : share >= 4 ? 7000 : INT32_MAX);
    const bool pdl = env_pdl >= 0 ? env_pdl == 1 : !in_step;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)n_ctas);
    cfg.blockDim = dim3(384);
    cfg.dynamicSmemBytes = TcCfg<D>::SMEM_BYTES;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    cfg.attrs = attr;
    if (pdl) {
        attr[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[cfg.numAttrs++].val.programmaticStreamSerializationAllowed = 1;
    }
    if constexpr (kSplit) {
        attr[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
        attr[cfg.numAttrs].val.clusterDim.x = (unsigned)p.split;
        attr[cfg.numAttrs].val.clusterDim.y = attr[cfg.numAttrs].val.clusterDim.z = 1;
        ++cfg.numAttrs;
    }
    return cudaLaunchKernelEx(&cfg, kern, mq, mk, mv, mo, p);
}

template <int D, bool kCausal, bool kKeep>
static cudaError_t launch_tc(const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv, const CUtensorMap& mo,
                             const TcParams& p, int64_t n_ctas, cudaStream_t stream) {
    if constexpr (!kKeep) {
        if (p.split > 1) return launch_tc_s<D, kCausal, false, true, true>(mq, mk, mv, mo, p, n_ctas * p.split, stream);
        if (p.single_tile && p.sorted) return launch_tc_s<D, kCausal, false, true, false, true>(mq, mk, mv, mo, p, n_ctas, stream);
    }
    return p.single_tile ? launch_tc_s<D, kCausal, kKeep, true, false>(mq, mk, mv, mo, p, n_ctas, stream)
                         : launch_tc_s<D, kCausal, kKeep, false, false>(mq, mk, mv, mo, p, n_ctas, stream);
}

// CTAs that clusters of `split` CTAs can have resident on the current device: GPCs hold whole clusters only, and how many
// depends on the part (this one: 74 clusters of 2, 33 of 4, 15 of 8).  Asked once per device and size.
static int cluster_slots(int split) {
    static std::atomic<int> known[64][3];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
    std::atomic<int>& slot = known[dev][split == 2 ? 0 : split == 4 ? 1 : 2];
    int n = slot.load(std::memory_order_relaxed);
    if (n > 0) return n - 1;
    auto kern = prefill_tc_kernel<128, true, false, true, true, false>;
    if (set_max_dynamic_smem_once<prefill_tc_kernel<128, true, false, true, true, false>>(TcCfg<128>::SMEM_BYTES) != cudaSuccess) return 0;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)split;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(split * 256));
    cfg.blockDim = dim3(384);
    cfg.dynamicSmemBytes = TcCfg<128>::SMEM_BYTES;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) {
        cudaGetLastError();
        n = 0;
    }
    slot.store(n * split + 1, std::memory_order_relaxed);
    return n * split;
}

// What a launch's items are: 0 for 256-row items (one CTA per SM works through several), 1 for 128-row items (one per
// CTA, keys split inside it), 2, 4 or 8 for 128-row items whose keys a cluster of so many CTAs shares.  The second
// kind has twice the CTAs and half the time per key, the third a shorter chain still for launches that leave SMs idle
// (a prompt chunk against a long cache), the first the least total work: each is priced as the longer of
// its heaviest CTA and the SMs' share of all CTAs.  Costs in us, from launches timed over B*H = 8..448, N = 37..4096:
// per 128 keys, per item, and for the merge across a cluster.
// (Clusters: B=2 H=16/2 123 rows against 8400 keys D=128 50 -> 23 us, H=8/1 64 rows against 2048 keys 18 -> 11, H=4/1
// 100 rows against 20000 keys D=64 130 -> 24.)  (Between the first two they picked the faster kind
// or one within 10 % of it on 57 of 57 shapes, within 3 % on 54; the block-count rule that this replaces took
// 33 us instead of 23 on H=16 N=1795 D=128, 49 / 27 on H=8 N=3500 D=64.)  Lengths that only the
// device knows (`uneven`) are taken at their largest, but not as equal: without a mask, whole waves of the longest took
// 256-row items for B=5 H=8 400 rows against 6000 keys D=64 (79 us, 50 with 128 rows) and 128-row items for B=24 H=16
// D=128 (440 us, 324 with 256 rows by length).
// *by_length: whether 128-row items are better started in the order of their lengths, where all items of a sequence are
// about as long (`sortable`: no mask, or a chunk's offsets).  That costs every item about 2 us before its first load
// (the lengths, the ranking).  Without it a longest item may start last, with nothing to hide behind: over 360 shapes of
// 2 to 24 sequences, lengths an eighth to all of the cache, that cost between a tenth and a half of its time.  B=4 H=8
// 700 rows against 8192 keys D=128 78 us in batch order, 59 by length; B=3 H=32 1000 against 3000 D=64 80 and 88.
static int choose_items(int64_t bh, int64_t seq, int64_t seq_kv, int64_t dim, bool causal, bool offsets, bool uneven, bool sortable,
                        bool may_split, int n_sm, bool* by_length) {
    *by_length = false;
    const int64_t n1 = (seq + 127) / 128, n2 = (seq + 255) / 256;
    if (bh * n2 >= 8 * (int64_t)n_sm) return 0;  // many items: the lower total wins, and no loop over long heads
    const double key1 = dim == 128 ? 1.0 : 0.84, item1 = dim == 128 ? 4.8 : 4.2, merge = 4.0;  // 128-row items
    const double key2 = dim == 128 ? 2.0 : 1.7, key2_one = 1.1, item2 = 3.0, first2 = 2.5;     // 256-row items
    const int64_t all = (seq_kv + 127) / 128, off = (causal && offsets && seq_kv > seq) ? seq_kv - seq : 0;
    auto tiles = [&](int64_t row_end) { return causal ? std::min(all, (off + std::min(row_end, seq) + 127) / 128) : all; };
    // equal CTAs come in whole waves; a list of unequal ones is dealt out to within about 8 % (of 256-row items that only
    // the lengths make unequal, 12 %: over 240 shapes the faster kind or within 0.4 % of it on average, 1.2 % with 8 and
    // 2.5 % with 16)
    auto span = [&](double sum, double mx, int64_t n, int slots, double over = 1.08) {
        return causal || uneven ? std::max(mx, over * sum * (double)bh / slots) : mx * (double)((bh * n + slots - 1) / slots);
    };
    double sum = 0, mx = 0;
    for (int64_t i = 0; i < n2; ++i) {
        const double c = (double)tiles((i + 1) * 256) * (i * 256 + 128 >= seq ? key2_one : key2) + item2;
        sum += c;
        mx = std::max(mx, c);
    }
    double best = span(sum, mx, n2, n_sm, uneven && !causal ? 1.12 : 1.08) + first2;
    int kind = 0;
    for (int split = 1; split <= (may_split ? 8 : 1); split *= 2) {
        sum = mx = 0;
        for (int64_t i = 0; i < n1; ++i) {
            const double c = (double)((tiles((i + 1) * 128) + split - 1) / split) * key1 + item1 + (split > 1 ? merge : 0);
            sum += c * split;
            mx = std::max(mx, c);
        }
        // a second wave of clusters starts only when whole clusters end (10 us and more a wave)
        if (split > 1 && (bh * n1 * split > n_sm || bh * n1 * split > cluster_slots(split))) break;
        const double t = span(sum, mx, n1 * split, n_sm);
        if (split == 1 && sortable && bh * n1 > n_sm) *by_length = span(sum + 2.0 * n1, mx + 2.0, n1, n_sm) < t + 0.12 * mx;
        if (t < best) {
            best = t;
            kind = split;
        }
    }
    return kind;
}

cudaError_t launch_prefill_tc(const void* q, const void* k, const void* v, void* out, float* lse, int64_t batch,
                              int64_t heads, int64_t heads_kv, int64_t seq, int64_t seq_kv, int dim,
                              const TensorStrides& sq, const TensorStrides& sk, const TensorStrides& sv,
                              const TensorStrides& so, int causal, const int32_t* kv_lens, const int32_t* q_offsets,
                              const uint8_t* key_keep, int64_t keep_batch_stride, float scale, cudaStream_t stream) {
    const int64_t bh = batch * heads;
    if (bh == 0 || seq == 0) return cudaSuccess;
    CUtensorMap mq, mk, mv, mo;
    // With no key at all nothing is loaded through the K/V maps; they still have to be valid.
    const void* kk = seq_kv > 0 ? k : q;
    const void* vv = seq_kv > 0 ? v : q;
    const int64_t skv = seq_kv > 0 ? seq_kv : 1;
    if (!make_tensor_map_bf16_4d(&mq, q, batch, heads, seq, dim, sq.batch, sq.head, sq.row) ||
        !make_tensor_map_bf16_4d(&mo, out, batch, heads, seq, dim, so.batch, so.head, so.row) ||
        !make_tensor_map_bf16_4d(&mk, kk, batch, heads_kv, skv, dim, sk.batch, sk.head, sk.row) ||
        !make_tensor_map_bf16_4d(&mv, vv, batch, heads_kv, skv, dim, sv.batch, sv.head, sv.row))
        return cudaErrorInvalidValue;
    TcParams p;
    p.o_stride_b = so.batch;
    p.o_stride_h = so.head;
    p.o_stride_row = so.row;
    p.out = (__nv_bfloat16*)out;
    p.lse = lse;
    p.kv_lens = kv_lens;
    p.key_keep = key_keep;
    p.keep_batch_stride = keep_batch_stride;
    p.seq = (int)seq;
    p.heads = (int)heads;
    p.seq_kv = (int)seq_kv;
    p.heads_kv = (int)heads_kv;
    p.q_offsets = q_offsets;
    p.scale_log2 = scale * kLog2e;
    p.status = device_status_ptr();
    if (!p.status) return cudaErrorInvalidSymbol;
    // Schedule (tc_item).  A launch whose items' costs the host knows (no per-batch lengths, and no keep flags unless
    // a causal mask already orders the items) and that has more items than SMs runs one CTA per SM over a static
    // list: the set-up of an item overlaps the item before.  With per-batch lengths the list is sorted on the
    // device.  Other launches use one CTA per item and leave the balancing to the hardware scheduler.
    // A causal launch whose K and V stay in L2 deals out whole levels, which balances best; a larger one works
    // through paired rounds, in which the CTAs share a few heads' K/V, down to the last one or two, and deals only
    // the rest by levels.  (Levels throughout cost 12 % on B=4 H=32 N=4096 D=128, 268 MB of K and V, at full clocks; at
    // 52 to 140 MB the two are within 1.5 %; at 30 MB and below levels win by up to 18 %.)
    constexpr int64_t kLevelsKvBytes = 96ll << 20;
    const int n_sm = sm_count();
    // RT_ATTN_PREFILL_TILES=1|2 and RT_ATTN_PREFILL_SCHED=persistent|percta override the choices below
    // (read once per process).
    static const int env_tiles = [] {
        const char* s = getenv("RT_ATTN_PREFILL_TILES");
        return (s && s[0] == '1') ? 1 : (s && s[0] == '2') ? 2 : 0;
    }();
    static const int env_sched = [] {
        const char* s = getenv("RT_ATTN_PREFILL_SCHED");
        return (s && !strcmp(s, "persistent")) ? 1 : (s && !strcmp(s, "percta")) ? 2 : 0;
    }();
    const bool uneven = kv_lens != nullptr && batch > 1;
    // (the ranking of 128-row items: one pass of the CTA's first 128 threads)
    const bool sortable = uneven && (q_offsets != nullptr || !causal) && key_keep == nullptr && batch * ((seq + 127) / 128) <= 128;
    bool by_length;
    const int kind = choose_items(bh, seq, seq_kv, dim, causal, q_offsets != nullptr, uneven, sortable,
                                  key_keep == nullptr && env_tiles == 0, n_sm, &by_length);
    p.single_tile = kind > 0 ? 1 : 0;
    p.split = kind > 1 ? kind : 1;
    static const int env_stagger = [] {
        const char* s = getenv("RT_ATTN_PREFILL_STAGGER");
        return s ? atoi(s) : 900;
    }();
    p.stagger_clocks = env_stagger;
    if (env_tiles == 1) p.single_tile = 1;
    if (env_tiles == 2) p.single_tile = 0;
    const int64_t n_qb = p.single_tile ? (seq + 127) / 128 : (seq + 255) / 256;
    const int64_t n_items = bh * n_qb;
    if (n_items > 0x3fffffff) return cudaErrorInvalidValue;
    p.n_qb = (int)n_qb;
    bool persistent = kv_lens == nullptr && (causal || key_keep == nullptr) && n_items > (int64_t)n_sm && !p.single_tile;
    if (env_sched == 1 && !p.single_tile) persistent = true;  // a single-tile item is its CTA's only item (the merge reuses barriers)
    if (env_sched == 2) persistent = false;
    // Per-batch lengths: the length-sorted persistent schedule, if its table fits (tc_item).  Keep flags are the same
    // with a length that every CTA has to look up first, about 0.7 us for 12 sequences; an item saves 3 us of set-up,
    // so at least 12 blocks per sequence are asked for.  (B=8 H=12 N=777 D=64 with padding: 45 us one CTA per item.)
    p.sorted = p.keep_tab = 0;
    const int64_t n_pairs = batch * n_qb, cap = dim == 128 ? TcCfg<128>::SCHED_CAP : TcCfg<64>::SCHED_CAP;
    const bool keep_sorted = key_keep != nullptr && heads * n_qb >= 12 && n_pairs + batch <= cap && seq_kv <= 4000000 && seq_kv > 0;
    if ((kv_lens != nullptr || keep_sorted) && !p.single_tile && env_sched != 2 && n_items > (int64_t)n_sm &&
        n_pairs <= cap && n_pairs <= 65535) {
        p.sorted = 1;
        p.keep_tab = keep_sorted ? (int)n_pairs : 0;
        persistent = true;
    }
    if (p.single_tile && p.split == 1 && by_length && env_sched != 2) p.sorted = 1;
    const int64_t n_ctas = (persistent && n_items > n_sm) ? n_sm : n_items;
    p.n_items = (int)n_items;
    p.units = (int)bh;
    p.list = make_level_schedule(bh, n_qb, n_ctas, batch * heads_kv * seq_kv * dim * 4 > kLevelsKvBytes && n_ctas < n_items);
    p.by_level = n_items * p.split > n_sm ? 1 : 0;
    p.direct_out = n_ctas == n_items ? 1 : 0;  // every CTA has exactly one item
    const bool keep = key_keep != nullptr;
    p.tighten = (keep && p.direct_out && seq_kv > 0) ? 1 : 0;
#define RT_TC_DISPATCH(DD)                                                                         \
    if (causal) {                                                                                  \
        return keep ? launch_tc<DD, true, true>(mq, mk, mv, mo, p, n_ctas, stream)                     \
                    : launch_tc<DD, true, false>(mq, mk, mv, mo, p, n_ctas, stream);                   \
    } else {                                                                                       \
        return keep ? launch_tc<DD, false, true>(mq, mk, mv, mo, p, n_ctas, stream)                    \
                    : launch_tc<DD, false, false>(mq, mk, mv, mo, p, n_ctas, stream);                  \
    }
    if (dim == 128) { RT_TC_DISPATCH(128) }
    if (dim == 64) { RT_TC_DISPATCH(64) }
#undef RT_TC_DISPATCH
    return cudaErrorInvalidValue;
}

}  // namespace rt
