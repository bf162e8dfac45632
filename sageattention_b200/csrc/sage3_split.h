// The last rounds of attention work dealt out by key blocks: the plan, formed on the host, and how a kernel's slot finds its tiles.
#pragma once

#include "sage3_kernels.h"

namespace sage3 {

// Units are pairs of tiles, and 5.5 pairs per SM take as long as 6, 0.86 as long as 1: the tiles of the
// round that is not full (of the one before too, where that leaves less than a tile per SM) are cut into slots of as many key blocks as come to one SM, in the
// order tile after tile, blocks of a tile from its first key on (McNaughton 1959).  A CTA draws one slot and takes its parts in that order.  A tile lies in
// one slot or two: the one behind has its last keys, at its own start, walks them, and leaves the accumulator, row sums and maxima in memory; the one
// before has its first keys, at its end, and goes on from there.  So the same operations in the same order, and the same bits, as in one walk.  Slots are
// drawn from the last to the first: the part that is waited for belongs to a slot drawn before, where it comes first and waits for nothing, so some CTA can
// always go on, however many of them are resident.
// us per call, without / with: 1 000 queries x 9 192 keys, 32 heads 139.3 / 127.9, 1 500 x 12 000, 28 heads 246.8 / 200.9, 600 x 5 000 84.5 / 61.3; 4 250 tokens
// of 48 heads, D = 64 349.0 / 333.9; N tokens of H heads, D = 128 (64): 16 x 2 500 72.4 / 63.7 (63.8 / 55.4), 10 x 4 100 104.5 / 90.2 (94.3 / 80.4), 16 x 5 000 194.9
// / 180.4 (174.3 / 162.3), 24 x 5 000 269.2 / 259.0 (239.7 / 233.2), 5 x 16 384 532 / 476 (498 / 454).
// What it costs: some 8 blocks per slot (two more changes of units, 64 KB of accumulator in and out), and at D = 64 without a mask the rolled halves.  So: from 10 blocks
// of gain, 1 / 80 of the call (less shows nothing: 16 384 x 24 heads, 1.15 %, 2 192 / 2 182, 8 192 x 32, 1.1 %, 792 / 794), there 1 / 25 (24 x 6 000, 3.2 %, 312 / 313, 40 x 5 000,
// 1.6 %, 372 / 379).  With a mask only where it is that of a chunk of a longer sequence (tiles differ by a quarter of their blocks at most): pairs in order of their
// length level out by themselves otherwise.  The rounds ahead have to be even, since a CTA's slot is as long as any other's: 2 x 32 heads x 10 590 tokens, 83 tiles per head of which
// one was a unit of its own in them, 2 526 / 2 555.
struct SplitPlan {
    int whole = 0, slots = 0;         // pairs ahead of the slots; slots (0: nothing is dealt out by blocks)
    int blocks = 0, rest = 0;         // key blocks per slot; of slot 0
    int rest0 = 0;                    // see rest_tile
    uint32_t first[kSplitSlots];      // first tile of a slot (12 bits) and first key block of it
};
static_assert(4 * kSplitSlots <= 1 << 12, "fewer than four tiles per SM are dealt out");

// Tile number j of those dealt out by key blocks.  Without a mask the last ones of an odd number of tiles per head (whole units are pairs then, so that the rounds
// ahead are even), and the tiles from pair number rest0 / 2 on; with one in the order of the pairs, of which the first rest0 have one tile.
template <bool CAUSAL>
__host__ __device__ __forceinline__ void rest_tile(int j, int nqt, int BHq, int whole, int rest0, int& bhq, int& mt) {
    if (!CAUSAL) {
        const int odd = nqt & 1 ? BHq : 0;
        if (j < odd) {
            bhq = j;
            mt = nqt - 1;
        } else {
            bhq = (rest0 + j - odd) / (nqt & ~1);
            mt = rest0 + j - odd - bhq * (nqt & ~1);
        }
        return;
    }
    const int npair = (nqt + 1) >> 1, one = rest0;
    const int pair = j < one ? whole + j : whole + one + ((j - one) >> 1);
    bhq = pair % BHq;
    mt = 2 * (npair - 1 - pair / BHq) + (j < one ? 0 : 1 - ((j - one) & 1));
}

// Key blocks of a query tile.
template <bool CAUSAL>
__host__ __device__ __forceinline__ int tile_blocks(int mt, int Nk, int shift) {
    const int last = CAUSAL && mt * kBlock + kBlock - 1 + shift < Nk - 1 ? mt * kBlock + kBlock - 1 + shift : Nk - 1;
    return last < 0 ? 0 : last / kBlock + 1;
}

// The tiles dealt out, in rest_tile's order, as runs of groups of a tile or two with the same numbers of blocks: go(groups, blocks of the first tile, of the second or 0).
// (Host time of an attention call with 256 such tiles, 512: 3.9, 4.6 us by a walk over single tiles, 1.7 so, of which the plan is 0.5.)
template <bool CAUSAL, typename F>
inline void for_each_run(const SplitPlan& plan, int BHq, int nqt, int Nk, int shift, int tiles, F&& go) {
    if (!CAUSAL) return go(tiles, tile_blocks<CAUSAL>(0, Nk, shift), 0);
    if (plan.rest0 > 0) go(plan.rest0, tile_blocks<CAUSAL>(nqt - 1, Nk, shift), 0);
    const int npair = (nqt + 1) >> 1;
    int pair = plan.whole + plan.rest0;
    for (int row = pair / BHq; row < npair; ++row) {
        const int mt = 2 * (npair - 1 - row), end = (row + 1) * BHq;
        go(end - pair, tile_blocks<CAUSAL>(mt + 1, Nk, shift), tile_blocks<CAUSAL>(mt, Nk, shift));
        pair = end;
    }
}

template <bool CAUSAL>
inline SplitPlan plan_split(int BHq, int nqt, int Nk, int shift, int D, int sms) {
    SplitPlan none, plan;
    const int last = tile_blocks<CAUSAL>(nqt - 1, Nk, shift), pairs = BHq * ((nqt + 1) / 2);
    if (sms > kSplitSlots || last < kSplitMinBlocks || 4 * tile_blocks<CAUSAL>(0, Nk, shift) < 3 * last) return none;
    const bool odd = (nqt & 1) != 0;
    const int full = pairs / sms, over = pairs % sms;
    int tiles;                        // dealt out by blocks
    double before;                    // blocks per SM without slots
    if (CAUSAL) {
        const bool that_round = 2 * over > sms;      // the round that is not full is enough
        if (over == 0 || (!that_round && full == 0)) return none;
        plan.whole = pairs - over - (that_round ? 0 : sms);
        if (odd && plan.whole > 0) return none;      // (the rounds ahead of the slots are not even)
        plan.rest0 = odd ? BHq : 0;
        tiles = plan.rest0 + 2 * (pairs - plan.whole - plan.rest0);
        before = nqt == 1 ? (full + 1) * (double)last : (2 * full + (that_round ? 2 : 1) - (odd ? 0.5 : 0)) * last;      // (odd: units of one tile among them level out)
    } else {
        // rounds of whole pairs ahead such that one to three tiles per SM are left
        const int64_t all = (int64_t)BHq * nqt;
        const int whole_pairs = BHq * (nqt / 2);
        int64_t rounds = all / (2 * sms);
        if (rounds > 0 && all - rounds * 2 * sms < sms) --rounds;
        if (rounds * sms > whole_pairs || all <= sms) return none;
        plan.whole = (int)rounds * sms;
        plan.rest0 = 2 * plan.whole;
        tiles = (int)(all - plan.rest0);
        // (an odd number of tiles per head: one unit of a head is a single tile, which levels out half of a tile)
        before = nqt == 1 ? (double)((all + sms - 1) / sms) * last
               : odd      ? ((double)all / sms + 0.5) * last
                          : (2 * full + (over == 0 ? 0 : 2 * over > sms ? 2 : 1)) * (double)last;
    }
    int sum = 0;
    for_each_run<CAUSAL>(plan, BHq, nqt, Nk, shift, tiles, [&](int groups, int n0, int n1) { sum += groups * (n0 + n1); });
    const int per = (sum + sms - 1) / sms > last ? (sum + sms - 1) / sms : last;
    const double gain = before - per - plan.whole / sms * 2.0 * last;
    if (gain < 10 || gain * (D == 64 && !CAUSAL ? 25 : 80) < before) return none;
    plan.slots = (sum + per - 1) / per;
    plan.blocks = per;
    plan.rest = sum - (plan.slots - 1) * per;
    int i = 0, tile = 0, at = 0;      // slot plan.slots - 1 - i begins at block i * per of all tiles' blocks; the run's first tile, and that tile's first block
    for_each_run<CAUSAL>(plan, BHq, nqt, Nk, shift, tiles, [&](int groups, int n0, int n1) {
        const int each = n1 > 0 ? 2 : 1;
        for (; i < plan.slots && i * per < at + groups * (n0 + n1); ++i) {
            const int g = (i * per - at) / (n0 + n1), in = i * per - at - g * (n0 + n1), second = each == 2 && in >= n0 ? 1 : 0;
            plan.first[plan.slots - 1 - i] = (uint32_t)(tile + g * each + second) | (uint32_t)(in - second * n0) << 12;
        }
        at += groups * (n0 + n1);
        tile += groups * each;
    });
    return plan;
}

}  // namespace sage3
