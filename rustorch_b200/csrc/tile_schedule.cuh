// Static lists of work for kernels that run one CTA per SM under a causal mask, shared by the prefill and the
// backward kernels.
//
// A launch has `units` equal heads of `n` blocks; the block of rank 0 is the heaviest and cost falls with the rank.  The
// blocks of rank t of all heads form level t.  The levels one after the other are dealt to the G CTAs boustrophedon
// (0..G-1, G-1..0, ...), heaviest first, which balances the CTAs' lists to a few per cent.  A launch whose
// operands exceed L2 first works through `rounds` paired rounds: a slot holds the blocks r and n-1-r of one head, so
// all slots of a round cost the same and its CTAs work on a few neighbouring heads; only what they leave is dealt by levels.
#pragma once
#include <cstdint>

namespace rt {

struct LevelSchedule {
    int units, n;
    int rounds;     // paired rounds
    int tail_head;  // first head that they leave blocks of, and the ranks (from either end) that it has lost
    int tail_skip;
    int n_tail;     // blocks dealt by levels
};

// The list over G CTAs; with `paired`, all rounds but the last one or two are paired.
inline LevelSchedule make_level_schedule(int64_t units, int64_t n, int64_t G, bool paired) {
    LevelSchedule s;
    s.units = (int)units;
    s.n = (int)n;
    const int64_t per_head = (n + 1) / 2, all = units * per_head / G;
    s.rounds = (paired && all > 1) ? (int)(all - 1) : 0;
    const int64_t taken = s.rounds * G;
    s.tail_head = (int)(taken / per_head);
    s.tail_skip = (int)(taken % per_head);
    s.n_tail = s.tail_head == units ? 0 : (int)((units - s.tail_head) * n - 2 * s.tail_skip);
    return s;
}

// Entry j of CTA `cta`'s list: its head and rank.  False where the entry is empty; `end` once the list is over.
__device__ __forceinline__ bool level_item(const LevelSchedule& s, int j, int cta, int G, int& unit, int& rank, bool& end) {
    end = false;
    if (j < 2 * s.rounds) {
        const int slot = cta + (j >> 1) * G, per_head = (s.n + 1) >> 1, r = slot % per_head;
        unit = slot / per_head;
        rank = (j & 1) ? s.n - 1 - r : r;
        return !((j & 1) && rank == r);  // the middle block of an odd count has no partner
    }
    const int jt = j - 2 * s.rounds;
    end = jt * G >= s.n_tail;
    const int pos = jt * G + ((jt & 1) ? G - 1 - cta : cta);
    if (end || pos >= s.n_tail) return false;
    // the head that the rounds end in is missing from the first and last tail_skip levels
    const int full = s.units - s.tail_head - 1, mid = s.tail_skip * full, hi = mid + (s.n - 2 * s.tail_skip) * (full + 1);
    if (pos < mid) {
        rank = pos / full;
        unit = s.tail_head + 1 + pos % full;
    } else if (pos < hi) {
        rank = s.tail_skip + (pos - mid) / (full + 1);
        unit = s.tail_head + (pos - mid) % (full + 1);
    } else {
        rank = s.n - s.tail_skip + (pos - hi) / full;
        unit = s.tail_head + 1 + (pos - hi) % full;
    }
    return true;
}

}  // namespace rt
