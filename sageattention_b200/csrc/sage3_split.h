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
// What it costs: two more changes of units per slot, 64 KB of accumulator in and out, and at D = 64 without a mask the rolled halves.  Over 600 calls of 1 to 96 heads the blocks that an SM walks less
// (see longest_walk), less what was measured to be saved, are 5.4 (D = 64 under a mask 3.1), there 3.4 and 2.9 % of the call, each to 2.  So: from 6.5 blocks of gain on, 1 / 80
// of the call (less shows nothing: 16 384 x 24 heads, 1.15 %, 2 192 / 2 182, 8 192 x 32, 1.1 %, 792 / 794), 1 / 160 with an odd number of tiles per head, where the walk that is counted is the
// least there can be (6 979 x 64 heads, 0.9 %, 1 147 / 1 139, 119 056 x 24, 0.7 %, 106 670 / 106 200); there from 4 and 3 % (40 x 5 000, 1.6 %, 372 / 379).  Of the 473 of them that pass,
// one is slower, by 0.3 % (with 6 blocks three, by up to 1.2 %).  With a mask only where it is that of a chunk of a longer sequence (tiles differ by a quarter of their blocks at most): pairs in order of their
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

// Pairs that are whole units without slots: when the last round of pairs fills at most half of the SMs it is dealt out as single tiles (half the time for the round, twice
// the SMs).  With more than that single tiles need two rounds and lose the shared K and V stages.  148 SMs, heads x 2 048 tokens, D = 128, never / this rule / always
// single: 68 pairs over 81.8 / 71.8 / 71.7 us, 76 over 82.8 / 82.8 / 85.9 us, 140 over 87.5 / 87.4 / 92.9 us.
inline int whole_pairs(int nqt, int pairs, int sms) {
    const int rest = pairs % sms;
    return nqt > 1 && 2 * rest <= sms ? pairs - rest : pairs;
}

// Tiles one after the other on the SM that has most of them, without slots: units of two tiles and of one (the last of an odd number of a head's; the last round's), in order,
// each drawn when the CTA begins the one before, so that a unit of one tile at the end may well go to a CTA that has just begun one of two: of units that are drawn together those of two
// tiles' CTAs come first.  In steps of a tile: how many SMs end a unit in this step and in the next one, by the tiles of the unit that they have drawn.
template <bool CAUSAL>
inline int longest_walk(int BHq, int nqt, int sms) {
    const int npair = (nqt + 1) / 2, pairs = BHq * npair, whole = whole_pairs(nqt, pairs, sms);
    auto singles = [&](int n) { return nqt % 2 == 0 ? 0 : !CAUSAL ? n / npair : n < BHq ? n : BHq; };      // among the first n pairs
    const int units = whole + 2 * (pairs - whole) - (singles(pairs) - singles(whole));
    int next = 0;
    struct Count { int none, one, two; };
    auto draw = [&](int n) {
        const int begin = next, end = units - next < n ? units : next + n;
        const int p0 = begin < whole ? begin : whole, p1 = end < whole ? end : whole;
        const int two = p1 - p0 - (singles(p1) - singles(p0));
        next = end;
        return Count{n - (end - begin), end - begin - two, two};
    };
    const Count first = draw(sms < units ? sms : units);
    Count later = draw(first.two), now = draw(first.one);      // end in the step after the next; in the next one
    int steps = 0;
    for (int t = 1; now.none + now.one + now.two + later.none + later.one + later.two > 0; ++t) {
        const Count ended = now;
        if (ended.none + ended.one + ended.two > 0) steps = t;
        now = later;
        later = draw(ended.two);
        const Count again = draw(ended.one);
        now.none += again.none; now.one += again.one; now.two += again.two;
    }
    return steps;
}

template <bool CAUSAL>
inline SplitPlan plan_split(int BHq, int nqt, int Nk, int shift, int D, int sms) {
    SplitPlan none, plan;
    const int last = tile_blocks<CAUSAL>(nqt - 1, Nk, shift), pairs = BHq * ((nqt + 1) / 2);
    if (sms > kSplitSlots || last < kSplitMinBlocks || 4 * tile_blocks<CAUSAL>(0, Nk, shift) < 3 * last) return none;
    const int64_t all = (int64_t)BHq * nqt;
    if (all > 320 * (int64_t)sms) return none;      // (slots save two tiles of a walk at most, which has to be 1 / 160 of it)
    const bool odd = (nqt & 1) != 0;
    if (CAUSAL) {
        const int over = pairs % sms;
        const bool that_round = 2 * over > sms;      // the round that is not full is enough
        if (over == 0 || (!that_round && pairs < sms)) return none;
        plan.whole = pairs - over - (that_round ? 0 : sms);
        if (odd && plan.whole > 0) return none;      // (the rounds ahead of the slots are not even)
        plan.rest0 = odd ? BHq : 0;
    } else {
        // rounds of whole pairs ahead such that one to three tiles per SM are left
        int64_t rounds = all / (2 * sms);
        if (rounds > 0 && all - rounds * 2 * sms < sms) --rounds;
        if (rounds * sms > BHq * (nqt / 2)) return none;
        plan.whole = (int)rounds * sms;
        plan.rest0 = 2 * plan.whole;
    }
    const int tiles = (int)(all - 2 * plan.whole), ahead = 2 * (plan.whole / sms);      // dealt out by blocks; of an SM ahead of its slot
    int sum = 0;
    for_each_run<CAUSAL>(plan, BHq, nqt, Nk, shift, tiles, [&](int groups, int n0, int n1) { sum += groups * (n0 + n1); });
    const int per = (sum + sms - 1) / sms > last ? (sum + sms - 1) / sms : last;
    // key blocks of an SM without slots, behind the rounds ahead (under a mask tiles have different numbers of them), less those of a slot
    const double gain = (longest_walk<CAUSAL>(BHq, nqt, sms) - ahead) * ((double)sum / tiles) - per;
    const double before = gain + per + ahead * (double)last;
    if (D == 64 && !CAUSAL ? gain < 4 + 0.03 * before : gain < 6.5 || gain * (odd ? 160 : 80) < before) return none;
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
