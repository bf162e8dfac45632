// Block-scaled FP4 attention for sm_100a: TMA-staged E2M1 tiles, tcgen05 NVFP4 MMAs with the S and O
// accumulators in tensor memory, exp2 online softmax, P re-quantized to NVFP4 before the PV MMA.
//
// One CTA per SM; each draws units of work from a counter.  A unit is a PAIR of 128-row query tiles of one head (every K / V^T
// stage in shared memory serves both tiles), a stream of items (key block, tile), the two tiles in turn; all pipelines run on
// from unit to unit.  Six warpgroups (setmaxnreg moves registers to the softmax warpgroups):
//   warps 0, 1   Q K^T MMA issuers, for keys [0, 64) and [64, 128) of every item; warp 1 owns the tensor-memory allocation
//   warp 2       P V MMA issuer
//   warp 3       draws and publishes the units; TMA producer: Q tiles, then K (+ one delta_s row per tile) / V^T / scale atoms per block
//                (Each on a scheduler of its own; which role on which makes little difference.  With the producer as warp 0 and the issuers as 1
//                and 3, in turns on one machine: packed prompts 607.0 / 603.5 us, 3 001 tokens 90.6 / 90.3, 16 384 keys 5 788 / 5 780.)
//   warps 4-19   four softmax groups of four warps; group g takes the items g, g + 4, ...  A thread owns one row of the block
//                and walks its 128 keys in two halves of 64 (the scores of a half live in registers).
//   warps 20-23  O rescale ("correction"), one warp per tensor-memory lane quarter: when a row of the quarter moved
//                its maximum, the warp multiplies the 32 O rows of its quarter by their factors before the block's
//                P V MMA is issued; it also keeps the running row sums and writes O / l while the softmax groups are
//                already at work on the next unit.
// Per half a softmax thread pulls its 64 scores out of tensor memory (the S buffer is free again at once) and runs the
// exp2 pass microblock by microblock, the maxima of the next microblock found under the exponentials of the current one:
// with E = P~ / sf = 6 * 2^((S - bm) s), the exp2 values and FP4 codes of a microblock depend on the maximum bm of that
// microblock only.  The running row maximum enters just the E4M3 scales, the row sum and the O rescale factor; it is handed
// from the group that has a tile's block to the group that has the next one as soon as all maxima of the row are known, and
// nothing else connects the groups: four independent chains per scheduler, a quarter of an item apart.
// What bounds it: the exp2 unit (16 results per clock and SM: 1 096 cycles per 128 x 128 block with the exponentials of the
// scales), the other instructions of the softmax warps (some 700 issue slots per block and scheduler) and fetching them; the tensor pipe
// needs 580 cycles.  Measured (1 965 MHz): 1 522 cycles per block at D = 128 and 1 458 at D = 64 for N = 16 384, 1 483 and 1 425 for N = 32 768;
// the exp2 unit 78 %, issue slots 63 % busy.
// Code size is a cost of its own: the softmax warps of a scheduler are in different places of their loop, and the issuers' and correction
// warps' loops come on top.  Taking out code that never ran (carried state, masks, second copies of waits) and rolling the two halves of
// an item into one loop gave more than any instruction saved in it: 2 x 48 heads, 17 550 queries x 226 keys, D = 64 298 -> 246 us per call, 2 x 40
// heads, 9 000 x 300, D = 128 230 -> 195, packed prompts of 256 to 2 048 tokens 697 -> 621, 8 192 keys causal 3 253 -> 3 203, 16 384
// keys 5 848 -> 5 802.  Two copies of the item, one with and one without masks, came out at 336 (226 keys) and 6 050 us (16 384).
// Units in place of one CTA per pair took the drain and refill of the pipeline, 10 us per pair, out: B = 2, H = 32, N = 8 192 causal
// 960 -> 776 us, B = 4, H = 32, N = 1 024 99 -> 77 us.
// Halves of 64 keys because a thread's registers hold 64 scores, and because tensor memory has room for three 64-key buffers
// next to two O tiles at D = 128.

// Arithmetic follows (paths inside the reference project, sageattention3_blackwell/sageattn3/blackwell/...):
//   mainloop_tma_ws.h:509, 532-551, 865     KV blocks are walked from the last to the first
//   mainloop_tma_ws.h:691-704, 718          S starts from the delta_s row of the query tile (here: a rank-1
//                                           16-bit MMA, ones (x) delta_s, issued before the FP4 MMAs)
//   mainloop_tma_ws.h:732-748               masks (applied here on the real key index)
//   softmax_fused.h:39-137                  running max per 128 keys, P~ = 2^(S s - m s) * 2688, row sum of the
//                                           unquantized P~, microblock scale max(P~)/6 (E4M3 in the MMA)
//   softmax_fused.h:139-170                 O = O alpha + P^ V^;  out = O / l  (0 when l == 0)
// Every wait is bounded (see mbar_wait); a wait that gives up records a code in the status word and the
// CTA winds down without touching tensor memory it does not own.
#include <cuda.h>

#include <type_traits>

#include "sage3_common.cuh"
#include "sage3_kernels.h"
#include "sage3_split.h"

namespace sage3 {

constexpr float kNoKey = -1e30f;                      // maximum of a microblock without visible keys (keeps -inf - -inf out of the arithmetic)
constexpr float kLog2Of6 = 2.584962500721156f;
constexpr float kPScaleLog2 = -11.392317422778762f;   // log2(1 / (448 * 6)), softmax_fused.h:33

struct AttnParams {
    int BHq, Hq, Hkv, Nq, Nk, nqt, nkb, nqm;   // nqt = query tiles per head, nkb = KV blocks per head
    int units, whole_units;             // units of work; those from whole_units on are single query tiles instead of pairs
    int pack_heads, pack_tiles;         // PACK kernels: query heads per tile, tiles per kv head
    int* unit_counter;                  // zero at launch: next unit after the first gridDim.x (CARRY == 2 and no whole units: all are drawn)
    float sm_scale_log2;
    const float* sm_scale_per_head;
    const uint8_t *q_sf, *k_sf, *v_sf;
    const uint16_t* delta;              // 16-bit elements [B*Hq][nqm][nkb*128]
    void* out[kMaxParts];               // output buffers; out_rows == 0: one buffer
    int out_wide;                       // rows of the output start on 32-byte boundaries: 256-bit stores
    int out_rows;                       // query rows per output part (rows of one (batch, head) go to part row / out_rows)
    int64_t os0, os1, os2;
    float* lse;                         // optional fp32 [B*Hq][Nq]
    const float* qkm;                   // fp32 [B*Hq][nqt*128]: q . km per query row
    float sm_scale;
    int* status;
    const int* prepass_status;
    // accumulator state carried between calls that walk consecutive key ranges of one attention (nullptr: none)
    const float *carry_o_in, *carry_m_in, *carry_l_in;   // fp32 [B*Hq][Nq][D] unnormalized O; [B*Hq][Nq] running max; [B*Hq][Nq][2] partial row sums
    float *carry_o_out, *carry_m_out, *carry_l_out;
    int causal_shift;                   // key j is visible to query i iff j <= i + causal_shift
    const int *cu_q, *cu_k;             // packed variable-length sequences (VARLEN kernels): entry b owns rows cu[b] .. cu[b + 1]
    const int* nonfinite;               // PACK: per (batch, kv head), delta_s holds values that are not finite
};

// Of the kernels whose last rounds are dealt out by key blocks: units from whole_units on are slots, see SplitPlan.
struct SplitParams : AttnParams {
    int slot_blocks, slot_rest;         // key blocks per slot; of slot 0
    int rest0;                          // see rest_tile
    int* split_flags;
    float* split_state;
    uint32_t slot_first[kSplitSlots];
};

constexpr int kUnitRing = 4;

// PACK: few query rows and several query heads per kv head.  The rows of all these heads share one 128-row tile (row = head * Nq +
// token), so the keys are walked once instead of once per head.  Mode 1: 2 sequences x 32 heads x 16 tokens against 8 192 keys of 8
// kv heads 90.1 -> 88.3 us per call (without packing its 64 tiles leave SMs idle too; 8 sequences x 32 heads x 1 token, which
// mode 2 has now: 225.8 -> 166.4 us).
//
// PACK == 2: at most 32 such rows.  A thread owns a row of scores, so one warp of the four would have work and do the exponentials
// of all 128 keys for it.  The rows stand in every quarter of the tile instead (rows 0..31 = 32..63 = ...), and the warp of quarter
// w takes keys 32 w .. 32 w + 31 of the block for all of them: a quarter of the exponentials per warp.  The four exchange their
// maxima through shared memory; P, its scales and the accumulator are those of rows 0..31.  Same operations per score, and the row
// sums are added in the same order, so the same bits.  D = 128, 8 sequences x 32 heads x 1 token against 8 192 keys of 8 kv heads:
// 166.4 -> 143.1 us per call, pre-pass included (D = 64: 116.8 -> 92.2 us).  The copy warps' and the MMA issuer's instructions bound it: K, V and delta_s have
// a copy warp each.
template <int D, int PACK>
struct Cfg {
    // K and V^T stages, each shared by the two query tiles (as many as fit: PACK, see oP)
    static constexpr int kStages = PACK == 2 ? (D == 128 ? 7 : 11) : PACK ? (D == 128 ? 5 : 8) : (D == 128 ? 4 : 8);
    static constexpr int kQTiles = PACK ? 1 : 2;              // query tiles per unit
    static constexpr int kGroups = 4;                         // softmax groups
    static constexpr int kThreads = 256 + 128 * kGroups;      // and two more warpgroups, see the kernel
    // S buffers of 128 rows x 64 keys: a rotation for the first halves of the items and one for the second halves (D = 64 has room for
    // a second one of the latter: 1 % slower)
    static constexpr int kSBufs0 = 2, kSBufs1 = PACK ? 2 : 1, kSBufs = kSBufs0 + kSBufs1;
    static constexpr int kQBytes = 128 * D / 2;               // per query tile
    static constexpr int kSfQkBytes = (D / 64) * 512;
    static constexpr int kKBytes = 128 * D / 2;
    static constexpr int kVBytes = D * 64;
    static constexpr int kSfVBytes = 1024;
    static constexpr int kDeltaBytes = 256;
    // P slot to slot. PACK == 2 writes rows 0 .. 31 only, and lets the other rows of the operand be the next slots' bytes: finite codes, and scales of 0
    static constexpr int kPBytes = PACK == 2 ? 2048 : 8192;
    // shared-memory map (bytes from a 1024-aligned base)
    static constexpr int oQ = 0;                              // [buffer][tile] 8192
    static constexpr int oK = oQ + 2 * kQTiles * 8192;
    static constexpr int oV = oK + kStages * kKBytes;
    static constexpr int oP = oV + kStages * kVBytes;            // [slot] 8192
    static constexpr int oSfQ = oP + 7 * kPBytes + 8192;      // [buffer][tile] 1024
    static constexpr int oSfK = oSfQ + 2 * kQTiles * 1024;
    static constexpr int oSfV = oSfK + kStages * 1024;
    static constexpr int oSfP = oSfV + kStages * 1024;        // [slot] 1024
    // delta_s per stage: one row per tile, 256 B + 256 B that stay zero; PACK: [16 chunks of 8 keys][8 heads] 16 B, all finite, + 128 B that
    // stay zero, or the row of one head over the first 256 B
    static constexpr int kDeltaPitch = 512, kDeltaStage = PACK ? 16 * 128 + 128 : 2 * kDeltaPitch;
    static constexpr int oDelta = oSfP + 8 * 1024;            // [stage] kDeltaStage
    static constexpr int oOnes = oDelta + kStages * kDeltaStage;   // 128 x 16 tile: 1.0 in column 0 (PACK: in the column of the row's head), rest 0
    static constexpr int oStat = oOnes + 4096;                // float2 [slot][128 rows]: running maximum, rescale factor
    static constexpr int oSum = oStat + 8192;                 // float2 [slot][128 rows]: row sums of the two key halves of a block
    static constexpr int oMax = oSum + (PACK == 2 ? 16384 : 8192);      // PACK == 2: float [slot][quarter][32 rows]; oSum: float4 [slot][quarter][32 rows]
    static constexpr int oL = oMax + (PACK == 2 ? 4096 : 0);                    // float2 [tile][128 rows]: running row sums of the two key halves
    static constexpr int oM = oL + 2048;                      // float [tile][128 rows]: running maximum
    static constexpr int oBar = oM + 1024;
    static constexpr int kNumBars = 4 + 4 * kStages + kSBufs + 2 * kGroups + 7 * 8 + (PACK == 2 ? 4 : 0) + 2 * kUnitRing;
    static constexpr int oUnit = (oBar + kNumBars * 8 + 15) / 16 * 16;      // descriptors of the units being worked on
    static constexpr int oMisc = oUnit + kUnitRing * 64;
    static constexpr int kSmemBytes = oMisc + 64 + 1024;      // + slack for the manual 1024-byte alignment
    static_assert(kSmemBytes <= 227 * 1024, "shared memory");
    // tensor-memory columns: the S buffers, one O accumulator per tile, scale factors (Q, K: one copy per issuer)
    static constexpr uint32_t cS = 0, cO = 64 * kSBufs, cSfQ = cO + (PACK ? 1 : 2) * D, cSfK = cSfQ + 32, cSfV = cSfK + 16, cSfP = cSfV + 8;
    static_assert(cSfP + 8 <= 512, "tensor memory");
    static constexpr uint64_t kSwzQK = (D == 128) ? kSwz64 : kSwz32;
    static constexpr uint32_t kSboQK = (D == 128) ? 512 : 256;
    static constexpr size_t kState = split_state_floats(D);      // of a tile that two CTAs share
};

template <typename OutT> __device__ __forceinline__ uint32_t pack2(float a, float b);
template <> __device__ __forceinline__ uint32_t pack2<__nv_bfloat16>(float a, float b) {
    __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&v);
}
template <> __device__ __forceinline__ uint32_t pack2<__half>(float a, float b) {
    __half2 v = __floats2half2_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&v);
}

// 32 bytes to a 32-byte aligned address in one store: a whole sector per lane, since the rows of the output are far apart.  (Two
// 16-byte stores: 2 to 4 % of the attention time at two to four key blocks per tile.)
__device__ __forceinline__ void store_32b(void* p, const uint32_t* v) {
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                 ::"l"(p), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]) : "memory");
}

// A value that is the same in all lanes, marked as such for the compiler (uniform registers feed the tcgen05 instructions).
__device__ __forceinline__ int uniform(int v) { return __shfl_sync(0xffffffffu, v, 0); }

// Wait executed by a whole converged warp; the verdict is made warp-uniform so that no lane leaves a loop alone.
template <bool kBackoff = false>
__device__ __forceinline__ bool warp_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag, int* status, int code) {
    if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;       // (0.5 to 1.5 % over going through the loop's first look)
    const bool ok = mbar_wait<kBackoff>(bar, parity, abort_flag, status, code);
    return __all_sync(0xffffffffu, ok);
}

// One unit of work of a CTA: one or two query tiles of one head, walked over their key blocks.
struct __align__(16) Unit {
    // The unit is a stream of (block step jj, tile t) items, s = 0 ... ns - 1; with sd = s + d, t = sd & two and jj = sd >> two: two
    // tiles alternate (d = 1: under a causal mask tile 1 may start one block before tile 0), a single tile walks alone.
    int ns, two, d;               // ns < 0: no more units
    int nbmax;                    // the unit walks key block n = nbmax - 1 ... 0
    int mt0, nv;                  // first query tile, number of tiles
    int Nq, Nk, shift;            // lengths of this batch entry; key j is visible to query i iff j <= i + shift
    int nb[2];                    // key blocks per tile (PACK: nb[1] = query heads in the tile, bhq, hq = the first of them)
    int bhq, hq, bhkv;
    int64_t out_base;
};

// Unit number u of the launch; false when it is empty (beyond a short sequence of a packed batch).
// Order: without a mask pairs of tiles of one head are neighbours (its K and V are shared in L2); under a causal mask the
// pairs with the most keys of all heads come first, so that the short ones level out the end of the launch.
template <bool CAUSAL, bool VARLEN, int PACK, bool SPLIT>
__device__ __forceinline__ bool make_unit(const AttnParams& p, int u, Unit& w) {
    if constexpr (PACK) {
        w.bhkv = u / p.pack_tiles;
        const int h0 = (u % p.pack_tiles) * p.pack_heads, group = p.Hq / p.Hkv, b = w.bhkv / p.Hkv;
        w.hq = (w.bhkv % p.Hkv) * group + h0;
        w.bhq = b * p.Hq + w.hq;
        w.mt0 = 0;
        w.nv = 1;
        w.Nq = p.Nq;
        w.Nk = p.Nk;
        w.shift = p.causal_shift;
        w.out_base = b * p.os0;
        const int max_key = CAUSAL ? min(w.Nk - 1, w.Nq - 1 + w.shift) : w.Nk - 1;
        w.nb[0] = w.nbmax = w.ns = max_key < 0 ? 0 : max_key / kBlock + 1;
        w.nb[1] = min(p.pack_heads, group - h0);
        w.two = w.d = 0;
        return true;
    }
    const int npair = (p.nqt + (SPLIT && !CAUSAL ? 0 : 1)) >> 1;      // (SPLIT, see rest_tile)
    int pair = u, half = -1;
    if (u >= p.whole_units) {                      // the last units are single tiles
        pair = p.whole_units + ((u - p.whole_units) >> 1);
        half = (u - p.whole_units) & 1;
    }
    int pr;
    if (CAUSAL) {
        pr = npair - 1 - pair / p.BHq;
        w.bhq = pair % p.BHq;
    } else {
        w.bhq = pair / npair;
        pr = pair % npair;
    }
    w.mt0 = 2 * pr + (half > 0 ? 1 : 0);
    const int b = w.bhq / p.Hq;
    w.hq = w.bhq % p.Hq;
    w.bhkv = b * p.Hkv + w.hq / (p.Hq / p.Hkv);
    // p.Nq, p.Nk, p.nqt, p.nkb stay the strides of the workspace layouts; with packed variable-length sequences they are the
    // maxima and the entry's own lengths come from the cu arrays.
    w.Nq = p.Nq;
    w.Nk = p.Nk;
    w.shift = p.causal_shift;
    w.out_base = b * p.os0;
    int nqt = p.nqt, nkb = p.nkb;
    if constexpr (VARLEN) {
        const int q0 = p.cu_q[b], k0 = p.cu_k[b];
        w.Nq = min(max(p.cu_q[b + 1] - q0, 0), p.Nq);
        w.Nk = min(max(p.cu_k[b + 1] - k0, 0), p.Nk);
        nqt = (w.Nq + kBlock - 1) / kBlock;
        nkb = (w.Nk + kBlock - 1) / kBlock;
        w.shift = w.Nk - w.Nq;
        w.out_base = (int64_t)q0 * p.os2;
    }
    w.nv = min(half < 0 ? 2 : 1, nqt - w.mt0);
    if (w.nv <= 0) return false;
#pragma unroll
    for (int t = 0; t < 2; ++t) {
        int nb = nkb;
        if (CAUSAL) {
            const int max_key = min(w.Nk - 1, (w.mt0 + t) * kBlock + kBlock - 1 + w.shift);
            nb = max_key < 0 ? 0 : max_key / kBlock + 1;
        }
        w.nb[t] = t < w.nv ? nb : 0;
    }
    w.nbmax = max(w.nb[0], w.nb[1]);
    w.two = w.nv == 2 ? 1 : 0;
    w.d = w.two ? w.nb[1] - w.nb[0] : 0;
    w.ns = w.nb[0] + w.nb[1];
    return true;
}

__device__ __forceinline__ float4 load_state(const float4* p) {
    float4 v;
    asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p) : "memory");
    return v;
}

// The part of tile j of the rest from key block lo on, `left` blocks of it at most, in slot m.
template <bool CAUSAL>
__device__ __forceinline__ void make_part(const SplitParams& p, int j, int lo, int left, int m, Unit& w) {
    rest_tile<CAUSAL>(j, p.nqt, p.BHq, p.whole_units, p.rest0, w.bhq, w.mt0);
    const int b = w.bhq / p.Hq, nb = tile_blocks<CAUSAL>(w.mt0, p.Nk, p.causal_shift), hi = min(nb, lo + left);
    w.hq = w.bhq % p.Hq;
    w.bhkv = b * p.Hkv + w.hq / (p.Hq / p.Hkv);
    w.Nq = p.Nq;
    w.Nk = p.Nk;
    w.shift = p.causal_shift;
    w.out_base = b * p.os0;
    w.nv = 1;
    w.two = w.d = 0;
    w.nbmax = hi;
    w.ns = w.nb[0] = hi - lo;
    w.nb[1] = (hi < nb ? m : 0) | (lo > 0 ? m + 1 : 0) << 16;      // goes on from slot m - 1's part; leaves its own under m
}

template <int D, bool CAUSAL, typename OutT, bool VARLEN, int PACK, int CARRY, bool ROLL>
__global__ void __launch_bounds__(Cfg<D, PACK>::kThreads, 1)
attn_fwd_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_d,
                const __grid_constant__ std::conditional_t<CARRY == 2, SplitParams, AttnParams> p) {
    using C = Cfg<D, PACK>;
    constexpr int S = C::kStages;
    extern __shared__ uint8_t smem_dyn[];
    const uint32_t sbase = (smem_u32(smem_dyn) + 1023u) & ~1023u;
    uint8_t* sgen = smem_dyn + (sbase - smem_u32(smem_dyn));

    const int warp = uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;

    // barriers
    const uint32_t bars = uniform(sbase + C::oBar);
    auto bar = [&](int i) { return bars + 8u * i; };
    constexpr int bQF = 0, bQE = 2, bKF = 4, bKE = bKF + S, bVF = bKE + S, bVE = bVF + S, bSF = bVE + S, bSE = bSF + 2 * C::kGroups, bM = bSE + C::kSBufs,
                  bPF = bM + 32, bPV = bPF + 8, bOS = bPV + 8, bX = bOS + 8, bWF = bX + (PACK == 2 ? 4 : 0), bWE = bWF + kUnitRing, bEnd = bWE + kUnitRing;
    static_assert(bEnd == C::kNumBars, "barriers");
    volatile int* abort_flag = reinterpret_cast<volatile int*>(sgen + C::oMisc);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sgen + C::oMisc + 8);

    // One barrier per thread: the number of arrivals that completes a phase.
    if (threadIdx.x < C::kNumBars) {
        const int i = threadIdx.x;
        uint32_t count = 1;                                      // copies landed, MMAs complete, one warp's statistics
        if (i >= bQE && i < bKF) count = PACK == 2 ? 1 : 2;      // Q buffer free: the Q K^T issuers are done with it
        if (i >= bKE && i < bKE + S) count = PACK == 2 ? 1 : 2;  // K stage free: likewise
        if (i >= bKF && i < bKE) count = PACK == 2 ? 2 : 1;      // K and its scales; delta_s by a warp of its own
        if (i >= bSE && i < bM) count = 4;                       // S buffer free: the four warps of its group hold the scores
        if (i >= bPF && i < bPV) count = 4;                      // P, its scales and the row sums written
        if (i >= bOS && i < bX) count = PACK == 2 ? 1 : 4;       // the correction warps are done with O (and have seen P written)
        if (i >= bX && i < bWF) count = 4;                       // maxima exchanged
        if (i >= bWE) count = C::kThreads / 32 - 1;              // unit descriptor free: every warp but the producer has finished the unit
        mbar_init(bar(i), count);
        mbar_fence_init();
    }
    if (threadIdx.x == 0) {
        *abort_flag = 0;
    }
    // delta_s stages: the bytes behind the rows stay zero for the whole kernel; ones tile:
    // [k chunk][row group][8 rows][16 bytes], 1.0 in element 0 of every row of chunk 0 (PACK: in the element of the row's head);
    // PACK: rows beyond the packed ones stay zero, codes and scales
    {
        uint4* z = reinterpret_cast<uint4*>(sgen + C::oDelta);
        constexpr int nd = S * C::kDeltaStage / 16;
        const uint32_t one = std::is_same<OutT, __nv_bfloat16>::value ? 0x3F80u : 0x3C00u;
        for (int i = threadIdx.x; i < nd + 4096 / 16; i += C::kThreads) {
            uint4 v = make_uint4(0, 0, 0, 0);
            if (i >= nd && i < nd + 128) {
                const int g = PACK ? (PACK == 2 ? (i - nd) & 31 : i - nd) / p.Nq : 0;
                const uint32_t w = one << (16 * (g & 1));
                if (!PACK || g < p.pack_heads) v = make_uint4(g >> 1 == 0 ? w : 0, g >> 1 == 1 ? w : 0, g >> 1 == 2 ? w : 0, g >> 1 == 3 ? w : 0);
            }
            z[i] = v;
        }
        if constexpr (PACK) {
            for (int i = threadIdx.x; i < 2 * C::kQTiles * 8192 / 16; i += C::kThreads) reinterpret_cast<uint4*>(sgen + C::oQ)[i] = make_uint4(0, 0, 0, 0);
            for (int i = threadIdx.x; i < 2 * C::kQTiles * 1024 / 16; i += C::kThreads) reinterpret_cast<uint4*>(sgen + C::oSfQ)[i] = make_uint4(0, 0, 0, 0);
            // rows 32 .. 127 of P have no writer: scale 0
            for (int i = threadIdx.x; PACK == 2 && i < 8 * 1024 / 16; i += C::kThreads) reinterpret_cast<uint4*>(sgen + C::oSfP)[i] = make_uint4(0, 0, 0, 0);
        }
        fence_proxy_async_smem();
    }
    if (warp == 1) {
        tmem_alloc(smem_u32(tmem_slot), 512);
        tmem_relinquish();
    }
    if (warp == 0 && lane == 0) {
        prefetch_tmap(&tm_q);
        prefetch_tmap(&tm_k);
        prefetch_tmap(&tm_v);
    }
    pdl_wait();                       // nothing above reads what the pre-pass writes
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = uniform(*tmem_slot);
    constexpr bool STATE = CARRY == 1, SPLIT = CARRY == 2;       // carried from call to call; from CTA to CTA
    const bool carry_in = STATE && p.carry_o_in != nullptr, carry_out = STATE && p.carry_o_out != nullptr;
    // SPLIT: slot whose accumulator this unit goes on from, and slot under which it leaves its own (-1: none).  A unit of one tile keeps them in nb[1].
    auto part_in = [](const Unit& u) { return SPLIT && u.nv == 1 ? (u.nb[1] & 0xffff) - 1 : -1; };
    auto part_out = [](const Unit& u) { return SPLIT && u.nv == 1 ? (u.nb[1] >> 16) - 1 : -1; };

    // Register budget: 768 threads start with 80 registers each, and that allocation (61 440) is all the CTA can
    // ever hold: 128 x kRoleRegs for warpgroup 0 (the copy and MMA roles) + 128 x kCorrRegs for the correction
    // warpgroup + 512 x kSoftRegs for the softmax warpgroups.  (An increase beyond the launch allocation would wait forever.)  With
    // the halves of an item in one loop the softmax code needs 88, which leaves the other warps 64: bytes spilled (stores / loads) 0 at D = 128 and at D = 64
    // without a mask, 22 / 30 at D = 64 with one, 10 / 14 with carried state at D = 64, 4 / 4 with packed heads at D = 64.  Unrolled it needs 96 and the others have 48:
    // 58 / 82 at D = 64, 82 / 114 for packed batches, 66 / 98 and (with a mask) 70 / 102 with carried state at D = 128; up to 32 rows 78 / 98.
    constexpr int kRoleRegs = PACK == 2 || !ROLL ? 48 : 64, kSoftRegs = PACK == 2 || !ROLL ? 96 : 88;
    constexpr int kCorrRegs = PACK == 2 || !ROLL ? 48 : 64;
    static_assert(128 * (kRoleRegs + kCorrRegs + C::kGroups * kSoftRegs) <= C::kThreads * 80, "registers");
    constexpr int kRescaleUnroll = D == 128 ? 2 : 8;
    // Carried state, us per three ranges attended (16 heads, 8 192 queries, ranges of 8 192 keys; D = 128 without / with a mask, D = 64 likewise): halves rolled, one
    // wait per item, row sums in registers 1 134, 676, 1 061, 603.  Sums in shared memory and, at D = 128, the halves unrolled 1 129, 660; at D = 64 rolled, the
    // factor waited for ahead of P and the output loop unrolled 1 048, 594.  Across: D = 128 rolled with the rest 1 130, 672, D = 64 unrolled 1 057, 610.
    constexpr bool kFactorFirst = STATE && ROLL;
    // A CTA runs unit after unit (the grid is one CTA per SM): the producer draws the next unit's number from a counter and
    // publishes the unit in shared memory, so the loads, scores and exponentials of the next unit fill in while the last one
    // drains, and uneven units (causal masks, packed batches) level out.
    const Unit* units = reinterpret_cast<const Unit*>(sgen + C::oUnit);
    auto next_unit = [&](int i) -> const Unit* {       // nullptr: none, or a wait gave up
        const int e = i % kUnitRing;
        if (!warp_wait(bar(bWF + e), (i / kUnitRing) & 1, abort_flag, p.status, kWaitUnit)) return nullptr;
        return units[e].ns < 0 ? nullptr : &units[e];
    };
    auto unit_done = [&](int i) { warp_arrive(bar(bWE + i % kUnitRing), lane); };
    int base = 0;                 // items of the units before this one: groups, slots and phases count through all units
    if (warp >= 4 + 4 * C::kGroups) {
      reg_dealloc<kCorrRegs>();
      // ------------------------------------------------------------------ O rescale (correction) and output, one warp per lane quarter
      // Also keeps the running row sums: l = l alpha + (sum over the block), for each half of the keys.
      const int quarter = warp & 3, row = quarter * 32 + lane;
      const int prow_head = PACK ? row / p.Nq : 0, prow_tok = PACK ? row - prow_head * p.Nq : 0;      // packed row -> head, token
      const uint32_t lane_addr = static_cast<uint32_t>(quarter * 32) << 16;
      const float2* stat = reinterpret_cast<const float2*>(sgen + C::oStat) + row;
      const float2* sum = reinterpret_cast<const float2*>(sgen + C::oSum) + row;
      float2* l_s = reinterpret_cast<float2*>(sgen + C::oL) + row;
      float* m_s = reinterpret_cast<float*>(sgen + C::oM) + row;
      // The pre-pass gave up (the workspace is then incomplete): the units are walked, but nothing is written.  (Read here, needed at
      // the first epilogue: off the path to the first scores.)
      const int broken = *reinterpret_cast<const volatile int*>(p.prepass_status);
      int dst = 0, dst_parity = 1;              // PACK == 2: stage of delta_s
      const Unit* u;
      bool ok = true;
      for (int i = 0; ok && (u = next_unit(i)) != nullptr; ++i) {
          const Unit& w = *u;
          const int ns = w.ns, two = w.two, d = w.d;
          const int pin = part_in(w);
          if constexpr (SPLIT) if (pin >= 0) {
              // resume another CTA's tile
              if (!warp_wait_word(p.split_flags + pin, 4, abort_flag, p.status, kWaitPart)) { ok = false; break; }
              const float* state = p.split_state + (size_t)pin * C::kState;
              l_s[0] = make_float2(load_written(state + 128 * D + 2 * row), load_written(state + 128 * D + 2 * row + 1));
              const float4* from = reinterpret_cast<const float4*>(state) + row;
#pragma unroll 1
              for (uint32_t o_addr = tmem + lane_addr + C::cO, end = o_addr + D; o_addr != end; o_addr += 32, from += 8 * 128) {
                  float o[32];
#pragma unroll
                  for (int q = 0; q < 8; ++q) {
                      const float4 v4 = load_state(from + q * 128);
                      o[4 * q] = v4.x; o[4 * q + 1] = v4.y; o[4 * q + 2] = v4.z; o[4 * q + 3] = v4.w;
                  }
                  tmem_st16(o_addr, o);
                  tmem_st16(o_addr + 16, o + 16);
              }
              tc_wait_st();
          }
          for (int t = 0; (!SPLIT || pin < 0) && t < w.nv; ++t) {
              l_s[t * 128] = make_float2(0.f, 0.f);
              m_s[t * 128] = -INFINITY;
              const int grow = (w.mt0 + t) * kBlock + row;
              if (carry_in && grow < w.Nq) {
                  const size_t crow = (size_t)w.bhq * p.Nq + grow;
                  l_s[t * 128] = *reinterpret_cast<const float2*>(p.carry_l_in + 2 * crow);
                  m_s[t * 128] = p.carry_m_in[crow];
              }
              if (carry_in) {
                  // resume: O continues from the state an earlier call left (its key range came later in the walk)
                  const float* src = p.carry_o_in + ((size_t)w.bhq * p.Nq + min(grow, w.Nq - 1)) * D;
                  for (int c = 0; c < D; c += 16) {
                      float o[16];
#pragma unroll
                      for (int q = 0; q < 4; ++q) {
                          const float4 v4 = *reinterpret_cast<const float4*>(src + c + 4 * q);
                          o[4 * q] = v4.x; o[4 * q + 1] = v4.y; o[4 * q + 2] = v4.z; o[4 * q + 3] = v4.w;
                      }
                      tmem_st16(tmem + lane_addr + C::cO + t * D + c, o);
                  }
                  tc_wait_st();
              }
          }
          if constexpr (PACK == 2) {
              if (quarter == 1) {
                  // delta_s of the unit's blocks: a copy less for the warp that has K.  One token of 8 x 32 heads, 8 192 keys of 8 kv heads 117.2 -> 116.8 us per call
                  // (D = 64 77.5 -> 76.2), of one sequence, 16 000 keys 76.8 -> 76.2 (63.6 -> 62.1).
                  const bool box = w.nb[1] > 1;
                  const uint16_t* src = p.delta + (size_t)w.bhq * p.nqm * ((size_t)p.nkb * kBlock);
                  for (int n = w.nbmax - 1; n >= 0; --n) {
                      if (!warp_wait<true>(bar(bKE + dst), dst_parity, abort_flag, p.status, kWaitKEmpty)) { ok = false; break; }
                      if (lane == 0) {
                          mbar_expect_tx(bar(bKF + dst), (box ? 8 : 1) * C::kDeltaBytes);
                          if (box) tma_load_3d(sbase + C::oDelta + dst * C::kDeltaStage, &tm_d, bar(bKF + dst), 0, w.bhq, n * (kBlock / 8));
                          else bulk_load(sbase + C::oDelta + dst * C::kDeltaStage, src + (size_t)n * kBlock, C::kDeltaBytes, bar(bKF + dst));
                      }
                      __syncwarp();
                      if (++dst == S) { dst = 0; dst_parity ^= 1; }
                  }
              }
              // One warp holds all rows: it waits for P alone (the factor was written before), reads all it needs, and keeps the sums in
              // registers.  (Waiting for the factor and for P with the sums in shared memory took it 1 000 cycles per block.)
              float2 l = make_float2(0.f, 0.f);
              float m = -INFINITY;
              const uint32_t o_addr = tmem + C::cO;
              for (int s = 0; quarter == 0 && s < ns; ++s) {
                  const int sg = base + s, slot = sg & 7;
                  if (!warp_wait(bar(bPF + slot), (sg >> 3) & 1, abort_flag, p.status, kWaitPFull)) { ok = false; break; }
                  const float2 ma = stat[slot * 128];
                  // scale and sum of every microblock, two per softmax warp
                  const float4* mb = reinterpret_cast<const float4*>(sgen + C::oSum) + slot * 128 + lane;
                  const float4 a = mb[0], b = mb[32], c = mb[64], e = mb[96];
                  if (s > 0 && __any_sync(0xffffffffu, ma.y != 1.0f)) {
                      if (!warp_wait(bar(bPV + ((sg - 1) & 7)), ((sg - 1) >> 3) & 1, abort_flag, p.status, kWaitOReady)) { ok = false; break; }
                      tc_fence_after();
#pragma unroll
                      for (int cc = 0; cc < D / 16; ++cc) {
                          float o0[16];
                          tmem_ld16(o_addr + cc * 16, o0);
                          tc_wait_ld();
#pragma unroll
                          for (int q = 0; q < 16; ++q) o0[q] *= ma.y;
                          tmem_st16(o_addr + cc * 16, o0);
                      }
                      tc_wait_st();
                      tc_fence_before();
                  }
                  warp_arrive(bar(bOS + slot), lane);
                  l.x = fmaf(l.x, ma.y, fmaf(b.z, b.w, fmaf(b.x, b.y, fmaf(a.z, a.w, fmaf(a.x, a.y, 0.f)))));
                  l.y = fmaf(l.y, ma.y, fmaf(e.z, e.w, fmaf(e.x, e.y, fmaf(c.z, c.w, fmaf(c.x, c.y, 0.f)))));
                  m = ma.x;
              }
              l_s[0] = l;
              m_s[0] = m;
          }
          float2 l0 = make_float2(0.f, 0.f), l1 = l0;              // running row sums of the two tiles (carried state: in l_s)
          if (SPLIT && pin >= 0) l0 = l_s[0];
          for (int s = 0; PACK != 2 && s < ns; ++s) {
              const int sg = base + s, slot = sg & 7, ph = (sg >> 3) & 1;
              const int t = (s + d) & two;
              const bool first = s <= two;                            // the tile's first block
              // One wait per item: P, its scales, the row sums and the factor are all written.  (kFactorFirst elsewhere, a wait for the factor first, so that the rescale
              // runs under the rest of the softmax: 226 keys 255 instead of 248 us, 300 keys at D = 128 202 instead of 198.)
              if (kFactorFirst && !warp_wait(bar(bM + slot * 4 + quarter), ph, abort_flag, p.status, kWaitAlpha)) { ok = false; break; }
              if (!kFactorFirst && !warp_wait(bar(bPF + slot), ph, abort_flag, p.status, kWaitPFull)) { ok = false; break; }
              float2 rs = make_float2(0.f, 0.f);
              if (!kFactorFirst) rs = sum[slot * 128];
              const float2 ma = stat[slot * 128];
              const float alpha = ma.y;
              // the first block has nothing to rescale unless the accumulator was carried in
              if ((!first || carry_in || (SPLIT && part_in(w) >= 0)) && __any_sync(0xffffffffu, alpha != 1.0f)) {
                  // the P V MMA of the tile's previous block must have landed first
                  if (!first) {
                      const int sp = sg - 1 - two;
                      if (!warp_wait(bar(bPV + (sp & 7)), (sp >> 3) & 1, abort_flag, p.status, kWaitOReady)) { ok = false; break; }
                  }
                  tc_fence_after();
                  const uint64_t a2 = pack2f(alpha, alpha);
                  const uint32_t o_addr = tmem + lane_addr + C::cO + t * D;
#pragma unroll kRescaleUnroll
                  for (int cc = 0; cc < D / 16; ++cc) {
                      float o0[16];
                      tmem_ld16(o_addr + cc * 16, o0);
                      tc_wait_ld();
#pragma unroll
                      for (int q = 0; q < 8; ++q)
                          unpack2f(mul2(pack2f(o0[2 * q], o0[2 * q + 1]), a2), o0[2 * q], o0[2 * q + 1]);
                      tmem_st16(o_addr + cc * 16, o0);
                  }
                  tc_wait_st();
              }
              tc_fence_before();
              // P V issue waits for this warpgroup only, so its arrival also stands for "P is written"
              if (kFactorFirst) {
                  if (!warp_wait(bar(bPF + slot), ph, abort_flag, p.status, kWaitPFull)) { ok = false; break; }
                  rs = sum[slot * 128];
              }
              warp_arrive(bar(bOS + slot), lane);
              float2 l = STATE ? l_s[t * 128] : t ? l1 : l0;
              l.x = fmaf(l.x, alpha, rs.x);
              l.y = fmaf(l.y, alpha, rs.y);
              if (STATE) l_s[t * 128] = l; else if (t) l1 = l; else l0 = l;
              m_s[t * 128] = ma.x;
          }
          if (PACK != 2 && !STATE) {
              l_s[0] = l0;
              l_s[128] = l1;
          }
          const int pout = part_out(w);
          // ---------------------------------------------------------------- O / l of the unit's tiles
          // (The accumulators belong to the next unit once this warpgroup arrives for its first items.  PACK == 2: the warps without rows
          // stay away, the pipeline does not wait for them, and the barrier below may be two phases on by the time they look.)
          for (int t = 0; ok && broken == 0 && (PACK != 2 || quarter == 0) && t < w.nv; ++t) {
              const int grow = PACK ? prow_tok : (w.mt0 + t) * kBlock + row;
              const bool live = PACK ? prow_head < w.nb[1] : grow < w.Nq && (!SPLIT || pout < 0);
              const int bhq = w.bhq + prow_head, hq = w.hq + prow_head;
              const bool have = w.nb[t] > 0 || carry_in;
              const float2 l2 = l_s[t * 128];
              const float l_tot = l2.x + l2.y;
              if (live && (p.lse != nullptr || carry_out)) {
                  const float m_fin = m_s[t * 128];
                  const size_t crow = (size_t)bhq * p.Nq + grow;
                  if (p.lse != nullptr) {
                      // ln sum_k exp(scale * q.k): the kernel's row sum is 2688 * sum_k 2^((S_k - m) s) over the smoothed
                      // scores S (delta_s included); K smoothing took scale * q.km out of every score of the row
                      const float scale = p.sm_scale_per_head ? p.sm_scale_per_head[hq] : p.sm_scale;
                      const float ms_fin = (m_fin == -INFINITY ? 0.f : m_fin) * (p.sm_scale_per_head ? scale * 1.4426950408889634f : p.sm_scale_log2);
                      const float v = (ms_fin + __log2f(l_tot) + kPScaleLog2) * 0.6931471805599453f +
                                      scale * p.qkm[(size_t)bhq * p.nqt * kBlock + grow];
                      p.lse[crow] = (l_tot == 0.f) ? -INFINITY : v;
                  }
                  if (carry_out) {
                      p.carry_m_out[crow] = m_fin > kNoKey ? m_fin : -INFINITY;
                      *reinterpret_cast<float2*>(p.carry_l_out + 2 * crow) = l2;
                  }
              }
              const float inv_l = (l_tot == 0.f || l_tot != l_tot) ? 0.f : __frcp_rn(l_tot);
              // the row's home: one output buffer, or the part that owns this token (another GPU's memory when the
              // output goes straight back to the token shards of a sequence-parallel group: plain stores)
              const int opart = (p.out_rows == 0) ? 0 : min(grow / p.out_rows, kMaxParts - 1);
              OutT* orow = p.out[opart] == nullptr || !live ? nullptr
                         : static_cast<OutT*>(p.out[opart]) + w.out_base + hq * p.os1 + (int64_t)(grow - opart * p.out_rows) * p.os2;
              if (w.nb[t] > 0) {
                  const int sl = base + (w.two ? 2 * (w.nbmax - 1) + t - w.d : w.nb[t] - 1);       // the tile's last item
                  if (!warp_wait(bar(bPV + (sl & 7)), (sl >> 3) & 1, abort_flag, p.status, kWaitOReady)) { ok = false; break; }
              }
              tc_fence_after();
              // All address arithmetic ahead of the wait for the last P V, products in pairs: the warp shares its scheduler with four softmax
              // warps, so what is behind the wait costs several cycles an instruction (300 keys at D = 128 191.9 -> 190.7 us, packed prompts
              // 610.3 -> 607.6, 226 keys 247.6 -> 246.1).  Its stores cost nothing that shows, wider loads did not help.
              const uint64_t inv2 = pack2f(inv_l, inv_l);
#pragma unroll (kFactorFirst ? D / 16 : PACK == 2 ? 8 : 1)
              for (int c = 0; c < D; c += 16) {
                  float o[16];
                  if (have) {
                      tmem_ld16(tmem + lane_addr + C::cO + t * D + c, o);
                      tc_wait_ld();
                  } else {
#pragma unroll
                      for (int q = 0; q < 16; ++q) o[q] = 0.f;
                  }
                  if constexpr (SPLIT) if (pout >= 0) {
                      float4* state = reinterpret_cast<float4*>(p.split_state + (size_t)pout * C::kState) + row;
#pragma unroll
                      for (int q = 0; q < 4; ++q) state[(c / 4 + q) * 128] = make_float4(o[4 * q], o[4 * q + 1], o[4 * q + 2], o[4 * q + 3]);
                  }
                  if (carry_out && live) {
#pragma unroll
                      for (int q = 0; q < 4; ++q)
                          *reinterpret_cast<float4*>(p.carry_o_out + ((size_t)bhq * p.Nq + grow) * D + c + 4 * q) =
                              make_float4(o[4 * q], o[4 * q + 1], o[4 * q + 2], o[4 * q + 3]);
                  }
                  if (orow != nullptr) {
                      uint32_t v[8];
#pragma unroll
                      for (int q = 0; q < 8; ++q) {
                          float x, y;
                          unpack2f(mul2(pack2f(o[2 * q], o[2 * q + 1]), inv2), x, y);
                          v[q] = pack2<OutT>(x, y);
                      }
                      if (p.out_wide) {
                          store_32b(orow + c, v);
                      } else {
                          *reinterpret_cast<uint4*>(orow + c) = make_uint4(v[0], v[1], v[2], v[3]);
                          *reinterpret_cast<uint4*>(orow + c + 8) = make_uint4(v[4], v[5], v[6], v[7]);
                      }
                  }
              }
          }
          if constexpr (SPLIT) if (ok && pout >= 0) {
              float* state = p.split_state + (size_t)pout * C::kState + 128 * D;
              *reinterpret_cast<float2*>(state + 2 * row) = l_s[0];
              state[256 + row] = m_s[0];
              warp_raise_word(p.split_flags + pout, lane);
          }
          unit_done(i);
          base += ns;
      }
      __syncwarp();
    } else if (warp < 4) {
      reg_dealloc<kRoleRegs>();
      auto load_v = [&](int st, int n, int bhkv) {
          mbar_expect_tx(bar(bVF + st), C::kVBytes + C::kSfVBytes);
          tma_load_3d(sbase + C::oV + st * C::kVBytes, &tm_v, bar(bVF + st), n * 64, 0, bhkv);
          bulk_load(sbase + C::oSfV + st * 1024, p.v_sf + ((size_t)bhkv * p.nkb + n) * C::kSfVBytes, C::kSfVBytes, bar(bVF + st));
      };
      if (warp == 3) {
        // ------------------------------------------------------------------ TMA producer
        int st = 0, st_parity = 1;                // K / V stage; parity of its "free" phase (a fresh barrier passes parity 1)
        int u = blockIdx.x, k = 0, kq = 0;        // unit number; units published, units with items
        // SPLIT: a slot is always drawn, the first unit too where that is one, so that the slots before it are in the hands of CTAs that run, in whatever order CTAs
        // are started.  (Its CTA draws on at its end: ahead of that it would take the slot of one that has just been started.)
        const int drawn = SPLIT && p.whole_units == 0 ? 0 : gridDim.x;
        if (drawn == 0) u = uniform(lane == 0 ? atomicAdd(p.unit_counter, 1) : 0);
        int next = 0, head = 0;                   // the unit after this one (lane 0); PACK: next head of a unit whose heads go one by one; SPLIT: next part of a slot
        int tile = 0, lo = 0, left = 0;           // SPLIT: of the slot, tile and first key block of its next part, key blocks left
        // V is loaded kLag blocks behind K.  A V stage is free four blocks after its K stage (scores, softmax and P lie between), and
        // with as few stages as D = 128 has room for, the K that the issuers want next would otherwise queue behind a V that
        // nobody is waiting for yet: they waited 740 cycles for every second item in an earlier kernel.  In this one the lag is worth little (us per call,
        // with / without: 1 000 queries x 9 192 keys 141.7 / 142.0, packed prompts 604.6 / 607.8, 3 001 tokens 92.7 / 92.5, 8 192 keys 801.3 / 802.5, 119 056
        // keys 106 640 / 106 790; carried state, three ranges of 8 192 keys 1 129 / 1 143).
        // What is held back must not keep the producer itself waiting: a ring entry is free when the unit four before it is finished, which
        // takes all of that unit's V.  Behind units with keys every block loaded brings a V in; an empty unit and the end marker load
        // nothing, so ahead of publishing one of these all V that is pending is loaded.
        constexpr int kLag = PACK == 2 || D == 64 ? 0 : 2;
        int vst = 0, vst_parity = 1, pend = 0;    // V stage; blocks whose V is still to be loaded: key block, kv head, oldest first
        int pend_n[2], pend_kv[2];
        auto next_v = [&](int n, int bhkv) {      // V of the block; waits until its stage is free
            if (!warp_wait<true>(bar(bVE + vst), vst_parity, abort_flag, p.status, kWaitVEmpty)) return false;
            if (lane == 0) load_v(vst, n, bhkv);
            if (++vst == S) { vst = 0; vst_parity ^= 1; }
            return true;
        };
        bool ok = true;
        while (ok) {
            if (!(PACK || SPLIT) || head == 0) next = 0;     // (where heads never go one by one nothing is carried round the loop: 0.3 % at 8 192 keys)
            if (lane == 0 && head == 0 && (!SPLIT || u < p.whole_units)) next = drawn + atomicAdd(p.unit_counter, 1);
            Unit w;
            const bool more = u < p.units;
            if (!more) w.ns = -1;
            else if (SPLIT && u >= p.whole_units) {
                if constexpr (SPLIT) {
                    const int m = u - p.whole_units;
                    if (head == 0) {
                        const uint32_t first = p.slot_first[m];
                        tile = first & 0xfff;
                        lo = first >> 12;
                        left = m == 0 ? p.slot_rest : p.slot_blocks;
                    }
                    make_part<CAUSAL>(p, tile, lo, left, m, w);
                }
            } else if (!make_unit<CAUSAL, VARLEN, PACK, SPLIT>(p, u, w)) { u = uniform(next); continue; }
            // Heads that share a tile share the operand that adds delta_s (eight rows of it, the next heads' too), and 0 x NaN is NaN: where
            // one of the kv heads behind these rows has a delta_s that is not finite, the unit's heads are published one by one.
            bool last_head = true;
            if constexpr (PACK) {
                if (more && w.ns > 0 && w.nb[1] > 1) {
                    const int kv = min(w.bhq + 7, p.BHq - 1) / (p.Hq / p.Hkv) - w.bhkv;
                    if (__any_sync(0xffffffffu, lane <= kv && p.nonfinite[w.bhkv + lane] != 0)) {
                        last_head = head + 1 == w.nb[1];
                        w.bhq += head;
                        w.hq += head;
                        w.nb[1] = 1;
                    }
                }
            }
            if (SPLIT && more && u >= p.whole_units) last_head = left == w.ns;
            const int lowest = SPLIT && more && u >= p.whole_units ? lo : 0;
            auto advance = [&] {
                if (SPLIT && u >= p.whole_units) {
                    ++tile;
                    lo = 0;
                    left -= w.ns;
                    if (last_head && lane == 0) next = drawn + atomicAdd(p.unit_counter, 1);
                }
                if (last_head) u = uniform(next);
                head = last_head ? 0 : head + 1;
            };
            if constexpr (kLag == 2) {
                if (w.ns <= 0) {
                    for (; ok && pend > 0; --pend) ok = next_v(pend == 2 ? pend_n[0] : pend_n[1], pend == 2 ? pend_kv[0] : pend_kv[1]);
                    if (!ok) break;
                }
            }
            if (!warp_wait<true>(bar(bWE + k % kUnitRing), ((k / kUnitRing) & 1) ^ 1, abort_flag, p.status, kWaitUnit)) break;
            if (lane == 0) {
                *reinterpret_cast<Unit*>(sgen + C::oUnit + (k % kUnitRing) * 64) = w;
                mbar_arrive(bar(bWF + k % kUnitRing));
            }
            ++k;
            if (!more) break;
            if (w.ns == 0) { advance(); continue; }
            const int qb = kq & 1;                // Q buffer
            if (!warp_wait<true>(bar(bQE + qb), ((kq >> 1) & 1) ^ 1, abort_flag, p.status, kWaitKEmpty)) break;
            ++kq;
            const uint16_t* dptr0 = p.delta + ((size_t)w.bhq * p.nqm + ((p.nqm > 1) ? w.mt0 : 0)) * ((size_t)p.nkb * kBlock);
            const size_t dstep = (p.nqm > 1) ? (size_t)p.nkb * kBlock : 0;
            const bool box = PACK && w.nb[1] > 1;        // (a head on its own brings its delta_s as a plain row, as a tile does)
            if constexpr (PACK) {
                // one box holds the rows of all heads; the scales move one word (four scales of a row) at a time into the packed row's place
                const int live = w.nb[1] * p.Nq;
                for (int r = lane; r < live; r += 32) {
                    const int g = r / p.Nq, i = r - g * p.Nq;
#pragma unroll
                    for (int a = 0; a < D / 64; ++a) {
                        const uint32_t sf = *reinterpret_cast<const uint32_t*>(p.q_sf + (size_t)(w.bhq + g) * C::kSfQkBytes + sf_atom_offset(i, 4 * a));
#pragma unroll
                        for (int c = 0; c < (PACK == 2 ? 4 : 1); ++c)
                            *reinterpret_cast<uint32_t*>(sgen + C::oSfQ + qb * C::kQTiles * 1024 + sf_atom_offset(r + 32 * c, 4 * a)) = sf;
                    }
                }
                fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0) {
                    constexpr int copies = PACK == 2 ? 4 : 1;
                    mbar_expect_tx(bar(bQF + qb), copies * p.pack_heads * p.Nq * (D / 2));
                    for (int c = 0; c < copies; ++c)
                        tma_load_3d(sbase + C::oQ + qb * C::kQTiles * 8192 + c * 32 * (D / 2), &tm_q, bar(bQF + qb), 0, 0, w.bhq);
                }
            } else if (lane == 0) {
                mbar_expect_tx(bar(bQF + qb), w.nv * (C::kQBytes + C::kSfQkBytes));
                for (int t = 0; t < w.nv; ++t) {
                    tma_load_3d(sbase + C::oQ + (qb * C::kQTiles + t) * 8192, &tm_q, bar(bQF + qb), 0, (w.mt0 + t) * kBlock, w.bhq);
                    bulk_load(sbase + C::oSfQ + (qb * C::kQTiles + t) * 1024, p.q_sf + ((size_t)w.bhq * p.nqt + w.mt0 + t) * C::kSfQkBytes,
                              C::kSfQkBytes, bar(bQF + qb));
                }
            }
            for (int n = w.nbmax - 1; n >= lowest; --n) {
                if (!warp_wait<true>(bar(bKE + st), st_parity, abort_flag, p.status, kWaitKEmpty)) { ok = false; break; }
                if (lane == 0) {
                    mbar_expect_tx(bar(bKF + st), C::kKBytes + C::kSfQkBytes + (PACK == 2 ? 0 : box ? 8 : w.nv) * C::kDeltaBytes);
                    tma_load_3d(sbase + C::oK + st * C::kKBytes, &tm_k, bar(bKF + st), 0, n * kBlock, w.bhkv);
                    bulk_load(sbase + C::oSfK + st * 1024, p.k_sf + ((size_t)w.bhkv * p.nkb + n) * C::kSfQkBytes,
                              C::kSfQkBytes, bar(bKF + st));
                    // box: [16 chunks of 8 keys][8 heads], the canonical core matrices of an MN-major operand (heads beyond the packed ones
                    // bring finite data that meets zeros).  One tensor copy: 64 copies of 16 bytes took 2.9 us per key block.
                    if (PACK != 2 && box) tma_load_3d(sbase + C::oDelta + st * C::kDeltaStage, &tm_d, bar(bKF + st), 0, w.bhq, n * (kBlock / 8));
                    for (int t = 0; PACK != 2 && !box && t < w.nv; ++t)
                        bulk_load(sbase + C::oDelta + (PACK ? st * C::kDeltaStage : (st * 2 + t) * C::kDeltaPitch), dptr0 + t * dstep + (size_t)n * kBlock,
                                  C::kDeltaBytes, bar(bKF + st));
                }
                if constexpr (PACK != 2) {
                    int vn = n, vkv = w.bhkv;
                    bool now = true;
                    if constexpr (kLag == 2) {
                        vn = pend_n[0]; vkv = pend_kv[0];
                        pend_n[0] = pend_n[1]; pend_kv[0] = pend_kv[1];
                        pend_n[1] = n; pend_kv[1] = w.bhkv;
                        now = pend == 2;
                        if (!now) ++pend;
                    }
                    if (now && !next_v(vn, vkv)) { ok = false; break; }
                }
                __syncwarp();
                if (++st == S) { st = 0; st_parity ^= 1; }
            }
            advance();
        }
        __syncwarp();
      } else if (PACK == 2 && warp == 1) {
        // ------------------------------------------------------------------ TMA producer of V
        // The waits and five copies of a block cost one producer 1 100 cycles, more than anything else does per block here (8 192
        // keys, 64 kv heads: 44 -> 40 us with a warp for K and one for V, D = 64 43 -> 33).
        int st = 0, st_parity = 1;
        bool ok = true;
        const Unit* u;
        for (int i = 0; ok && (u = next_unit(i)) != nullptr; ++i) {
            const int nbmax = uniform(u->nbmax), bhkv = uniform(u->bhkv);
            unit_done(i);
            for (int n = nbmax - 1; n >= 0; --n) {
                if (!warp_wait<true>(bar(bVE + st), st_parity, abort_flag, p.status, kWaitVEmpty)) { ok = false; break; }
                if (lane == 0) load_v(st, n, bhkv);
                __syncwarp();
                if (++st == S) { st = 0; st_parity ^= 1; }
            }
        }
        __syncwarp();
      } else if (warp == 0 || warp == 1) {
        // ------------------------------------------------------------------ Q K^T MMA issuers
        // The scores of an item are formed in two halves of 64 keys; warp 0 issues the first halves, warp 1 the second
        // ones, each into its own S buffers (issuing one half takes a few hundred cycles next to busy softmax warps: one
        // issuer for both would be the slowest part of the pipeline).  The whole warp walks the loop and one elected lane
        // issues, so loop state and descriptors stay in uniform registers.
        // (PACK == 2: softmax is short there, and the tensor pipe's cost per instruction counts; warp 0 issues all 128 keys at once, warp 1 loads V.)
        const int h = warp;
        constexpr int kKeys = PACK == 2 ? 128 : 64;
        constexpr uint32_t idesc_qk = make_idesc_nvfp4(kKeys);
        constexpr uint32_t idesc_delta = make_idesc_f16_bmn(kKeys, std::is_same<OutT, __nv_bfloat16>::value);
        // descriptors: constant high words, low words that move with the stage, tile and key half (bytes / 16)
        constexpr uint32_t hi_qk = sdesc_hi(C::kSboQK, C::kSwzQK), hi_ones = sdesc_hi(128, kSwzNone);
        const uint32_t ones_lo = sdesc_lo(sbase + C::oOnes, 2048), q_lo0 = sdesc_lo(sbase + C::oQ, 16), sfq_lo0 = sdesc_lo(sbase + C::oSfQ, 0);
        const uint32_t k_lo0 = sdesc_lo(sbase + C::oK + h * (64 * D / 2), 16), delta_row_lo = sdesc_lo(sbase + C::oDelta + h * 128, 16);
        const uint32_t sfk_lo0 = sdesc_lo(sbase + C::oSfK, 0);
        // each issuer has its own copies of the scale factors in tensor memory, so that its MMAs and copies stay in one order
        const uint32_t sfk_col = tmem + C::cSfK + 8 * h;        // the 128-key atoms; keys 64 .. 127 start two columns in
        const uint32_t sfq_col0 = tmem + C::cSfQ + 16 * h;
        const int nbuf = h == 0 ? C::kSBufs0 : C::kSBufs1, buf0 = h == 0 ? 0 : C::kSBufs0;
        int grp = 0;                              // softmax group of the next item
        int buf = 0, buf_parity = 1;              // next S buffer; parity of its "empty" phase (a fresh barrier passes parity 1)
        int st = 0, st_parity = 0;                // K stage
        bool ok = true;
        const Unit* u;
        for (int i = 0, k = 0; ok && (u = next_unit(i)) != nullptr; ++i) {
            const int ns = uniform(u->ns), two = uniform(u->two), d = uniform(u->d), nv = uniform(u->nv);
            uint32_t delta_lo0 = delta_row_lo, hi_delta = sdesc_hi(16, kSwzNone);
            if constexpr (PACK) {
                if (uniform(u->nb[1]) > 1) {       // the box of several heads: 128 bytes from 8 keys to the next 8
                    delta_lo0 = sdesc_lo(sbase + C::oDelta + h * 1024, 128);
                    hi_delta = sdesc_hi(128, kSwzNone);
                }
            }
            unit_done(i);
            if (ns == 0) continue;
            const int qb = k & 1;
            if (!warp_wait(bar(bQF + qb), (k >> 1) & 1, abort_flag, p.status, kWaitQFull)) break;
            ++k;
            tc_fence_after();
            if (elect_one()) {
                for (int t = 0; t < nv; ++t)
#pragma unroll
                    for (int ks = 0; ks < D / 64; ++ks)
                        tc_cp_sf(sfq_col0 + 8 * t + 4 * ks, sdesc(sfq_lo0 + (qb * C::kQTiles + t) * 64 + ks * 32, sdesc_hi(128, kSwzNone)));
            }
            __syncwarp();
            for (int s = 0; s < ns; ++s) {
                const int t = (s + d) & two;
                const bool opens = t == 0 || s == 0, closes = t == two;       // first / last item of its K block
                if (opens && !warp_wait(bar(bKF + st), st_parity, abort_flag, p.status, kWaitKFull)) { ok = false; break; }
                if (!warp_wait(bar(bSE + buf0 + buf), buf_parity, abort_flag, p.status, kWaitSEmpty)) { ok = false; break; }
                tc_fence_after();
                const uint32_t k_lo = k_lo0 + st * (C::kKBytes / 16), delta_lo = delta_lo0 + st * (C::kDeltaStage / 16) + t * (C::kDeltaPitch / 16);
                const uint32_t sfk_lo = sfk_lo0 + st * (1024 / 16), q_lo = q_lo0 + (qb * C::kQTiles + t) * (8192 / 16);
                const uint32_t s_col = tmem + C::cS + kKeys * (buf0 + buf), sfq_col = sfq_col0 + 8 * t;
                if (elect_one()) {
                    if (opens) {
#pragma unroll
                        for (int ks = 0; ks < D / 64; ++ks) tc_cp_sf(sfk_col + 4 * ks, sdesc(sfk_lo + ks * 32, sdesc_hi(128, kSwzNone)));
                    }
                    // S <- 1 (x) delta_s: A = [128 x 16] with ones in column 0 (K-major), B = 64 elements of the delta_s row read as an
                    // MN-major [16 x 64] operand whose rows 1..15 alias later keys of the row or finite data and meet zeros in A (PACK, several
                    // heads: rows 0..7 are the heads', all finite)
                    tc_mma_f16(s_col, sdesc(ones_lo, hi_ones), sdesc(delta_lo, hi_delta), idesc_delta, false);
#pragma unroll
                    for (int ks = 0; ks < D / 64; ++ks)
                        tc_mma_nvfp4(s_col, sdesc(q_lo + 2 * ks, hi_qk), sdesc(k_lo + 2 * ks, hi_qk), idesc_qk, sfq_col + 4 * ks,
                                     sfk_col + 4 * ks + 2 * h, true);
                    tc_commit(bar(bSF + 2 * grp + h));
                    if (closes) tc_commit(bar(bKE + st));
                    if (s == ns - 1) tc_commit(bar(bQE + qb));
                }
                __syncwarp();
                if (++grp == C::kGroups) grp = 0;
                if (++buf == nbuf) { buf = 0; buf_parity ^= 1; }
                if (closes && ++st == S) { st = 0; st_parity ^= 1; }
            }
            base += ns;
        }
        __syncwarp();
      } else {
        // ------------------------------------------------------------------ PV MMA issuer
        constexpr uint32_t idesc_pv = make_idesc_nvfp4(D);
        constexpr uint32_t hi_pv = sdesc_hi(512, kSwz64), hi_sf = sdesc_hi(128, kSwzNone);
        const uint32_t v_lo0 = sdesc_lo(sbase + C::oV, 16), p_lo0 = sdesc_lo(sbase + C::oP, 16);
        const uint32_t sfv_lo0 = sdesc_lo(sbase + C::oSfV, 0), sfp_lo0 = sdesc_lo(sbase + C::oSfP, 0);
        const uint32_t sfp_col = tmem + C::cSfP, sfv_col = tmem + C::cSfV;
        int st = 0, st_parity = 0;
        bool ok = true;
        const Unit* u;
        for (int i = 0; ok && (u = next_unit(i)) != nullptr; ++i) {
            const int ns = uniform(u->ns), two = uniform(u->two), d = uniform(u->d);
            const bool resumed = carry_in || uniform(part_in(*u)) >= 0;
            unit_done(i);
            for (int s = 0; s < ns; ++s) {
                const int slot = (base + s) & 7, t = (s + d) & two;
                const bool opens = t == 0 || s == 0, closes = t == two;       // first / last item of its V block
                if (opens && !warp_wait(bar(bVF + st), st_parity, abort_flag, p.status, kWaitVFull)) { ok = false; break; }
                if (!warp_wait(bar(bOS + slot), ((base + s) >> 3) & 1, abort_flag, p.status, kWaitOScaled)) { ok = false; break; }
                tc_fence_after();
                const uint32_t v_lo = v_lo0 + st * (C::kVBytes / 16), p_lo = p_lo0 + slot * (C::kPBytes / 16);
                const uint32_t sfv_lo = sfv_lo0 + st * (1024 / 16), sfp_lo = sfp_lo0 + slot * (1024 / 16), o_col = tmem + C::cO + t * D;
                if (elect_one()) {
                    if (opens) {
#pragma unroll
                        for (int ks = 0; ks < 2; ++ks) tc_cp_sf(sfv_col + 4 * ks, sdesc(sfv_lo + ks * 32, hi_sf));
                    }
#pragma unroll
                    for (int ks = 0; ks < 2; ++ks) tc_cp_sf(sfp_col + 4 * ks, sdesc(sfp_lo + ks * 32, hi_sf));
#pragma unroll
                    for (int ks = 0; ks < 2; ++ks)
                        tc_mma_nvfp4(o_col, sdesc(p_lo + 2 * ks, hi_pv), sdesc(v_lo + 2 * ks, hi_pv), idesc_pv, sfp_col + 4 * ks, sfv_col + 4 * ks,
                                     s > two || (ks > 0) || resumed);
                    tc_commit(bar(bPV + slot));
                    if (closes) tc_commit(bar(bVE + st));
                }
                __syncwarp();
                if (closes && ++st == S) { st = 0; st_parity ^= 1; }
            }
            base += ns;
        }
        __syncwarp();
      }
    } else if constexpr (PACK == 2) {
        reg_alloc<kSoftRegs>();
        // ------------------------------------------------------------------ softmax groups, at most 32 rows
        // As below, but the thread's row is its lane and the warp's keys are 32 * quarter .. + 31 of the block.
        const int g = (warp >> 2) - 1, quarter = warp & 3;
        const uint32_t s_addr = tmem + (static_cast<uint32_t>(quarter * 32) << 16) + C::cS + 32 * quarter;
        const int head = lane / p.Nq, tok = lane - head * p.Nq;
        float* wmax = reinterpret_cast<float*>(sgen + C::oMax) + lane;
        float2* stat = reinterpret_cast<float2*>(sgen + C::oStat) + quarter * 32 + lane;
        uint8_t* prow = sgen + C::oP + lane * 64 + ((quarter ^ ((lane >> 1) & 3)) << 4);
        bool alive = true;
        const Unit* u;
        for (int i = 0; alive && (u = next_unit(i)) != nullptr; ++i) {
            const int ns = uniform(u->ns), Nk = uniform(u->Nk), shift = CAUSAL ? uniform(u->shift) : 0;
            const float sl2 = p.sm_scale_per_head ? p.sm_scale_per_head[u->hq + min(head, u->nb[1] - 1)] * 1.4426950408889634f : p.sm_scale_log2;
            const uint64_t sl2x2 = pack2f(sl2, sl2);
            for (int s = (g - base) & 3; s < ns; s += 4) {
                const int sg = base + s, slot = sg & 7, slot_prev = (sg - 1) & 7, buf = sg % C::kSBufs0;
                const int key0 = (ns - 1 - s) * kBlock + 32 * quarter;
                if (!warp_wait(bar(bSF + 2 * g), (sg >> 2) & 1, abort_flag, p.status, kWaitSFull)) { alive = false; break; }
                tc_fence_after();
                float x[32];
                tmem_ld32(s_addr + 128 * buf, x);
                tc_wait_ld();
                tc_fence_before();
                warp_arrive(bar(bSE + buf), lane);
                if (key0 + 31 > (CAUSAL ? min(Nk - 1, shift) : Nk - 1)) {
                    const float vis = (float)((CAUSAL ? min(Nk - 1, tok + shift) : Nk - 1) - key0);
#pragma unroll
                    for (int q = 0; q < 32; ++q)
                        if ((float)q > vis) x[q] = -INFINITY;
                }
                float bm[2], se[2];
                uint32_t codes[4];
#pragma unroll
                for (int b = 0; b < 2; ++b) {
                    const float* y = x + 16 * b;
                    const float a = fmax3(fmax3(y[0], y[1], y[2]), y[12], y[13]);
                    const float c = fmax3(fmax3(y[3], y[4], y[5]), y[14], y[15]);
                    bm[b] = fmax3(a, c, fmax3(fmax3(y[6], y[7], y[8]), fmax3(y[9], y[10], y[11]), kNoKey));
                }
                wmax[(slot * 4 + quarter) * 32] = fmaxf(bm[0], bm[1]);
                warp_arrive(bar(bX + g), lane);
#pragma unroll
                for (int b = 0; b < 2; ++b) {
                    const float negc = fmaf(bm[b], -sl2, kLog2Of6);
                    const uint64_t negc2 = pack2f(negc, negc);
                    float e[16];
#pragma unroll
                    for (int q = 0; q < 8; ++q) {
                        float a, c;
                        unpack2f(fma2(pack2f(x[16 * b + 2 * q], x[16 * b + 2 * q + 1]), sl2x2, negc2), a, c);
                        e[2 * q] = ex2_approx(a);
                        e[2 * q + 1] = ex2_approx(c);
                    }
                    uint64_t acc0 = pack2f(e[0], e[1]), acc1 = pack2f(e[2], e[3]);
#pragma unroll
                    for (int q = 4; q < 16; q += 4) {
                        acc0 = add2(acc0, pack2f(e[q], e[q + 1]));
                        acc1 = add2(acc1, pack2f(e[q + 2], e[q + 3]));
                    }
                    float se0, se1;
                    unpack2f(add2(acc0, acc1), se0, se1);
                    se[b] = se0 + se1;
                    codes[2 * b] = cvt_e2m1x8(e[0], e[1], e[2], e[3], e[4], e[5], e[6], e[7]);
                    codes[2 * b + 1] = cvt_e2m1x8(e[8], e[9], e[10], e[11], e[12], e[13], e[14], e[15]);
                }
                if (sg >= 7 && !warp_wait(bar(bPV + ((sg - 7) & 7)), ((sg - 7) >> 3) & 1, abort_flag, p.status, kWaitPEmpty)) { alive = false; break; }
                *reinterpret_cast<uint4*>(prow + slot * C::kPBytes) = make_uint4(codes[0], codes[1], codes[2], codes[3]);
                if (!warp_wait(bar(bX + g), (sg >> 2) & 1, abort_flag, p.status, kWaitPair)) { alive = false; break; }
                float m_old = -INFINITY;
                if (s > 0) {
                    if (!warp_wait(bar(bM + slot_prev * 4 + quarter), ((sg - 1) >> 3) & 1, abort_flag, p.status, kWaitPair)) { alive = false; break; }
                    m_old = stat[slot_prev * 128].x;
                }
                const float* wm = wmax + slot * 128;
                const float m_run = fmax3(fmax3(wm[0], wm[32], wm[64]), wm[96], m_old);
                const float alpha = ex2_approx((m_old - m_run) * sl2);
                stat[slot * 128] = make_float2(m_run, alpha);
                warp_arrive(bar(bM + slot * 4 + quarter), lane);
                const float max_scaled = (m_run == kNoKey) ? 0.f : fmaf(m_run, sl2, kPScaleLog2);
                const float sf0 = ex2_approx(fmaf(bm[0], sl2, -max_scaled) - kLog2Of6), sf1 = ex2_approx(fmaf(bm[1], sl2, -max_scaled) - kLog2Of6);
                *reinterpret_cast<uint16_t*>(sgen + C::oSfP + slot * 1024 + 512 * (quarter >> 1) + lane * 16 + 2 * (quarter & 1)) =
                    static_cast<uint16_t>((cvt_e4m3x2(sf0, 0.f) & 0xffu) | (cvt_e4m3x2(sf1, 0.f) & 0xffu) << 8);
                reinterpret_cast<float4*>(sgen + C::oSum)[slot * 128 + quarter * 32 + lane] = make_float4(sf0, se[0], sf1, se[1]);
                fence_proxy_async_smem();
                warp_arrive(bar(bPF + slot), lane);
            }
            unit_done(i);
            base += ns;
        }
        __syncwarp();
    } else {
        reg_alloc<kSoftRegs>();
        // ------------------------------------------------------------------ softmax groups (4 x 4 warps)
        // Group g (one warpgroup) takes the stream items s = g, g + 4, ...; a thread owns one row (tensor-memory lane) of the
        // block and walks its 128 keys in two halves of 64.  With two tiles a group always serves the same tile.
        const int g = (warp >> 2) - 1;
        const int quarter = warp & 3;            // tensor-memory lane quarter this warp may touch
        const int r = quarter * 32 + lane;       // row inside the tile
        const uint32_t lane_addr = static_cast<uint32_t>(quarter * 32) << 16;
        const int prow_head = PACK ? r / p.Nq : 0, tok = PACK ? r - prow_head * p.Nq : r;      // packed row -> head, token
        const int sw = (r >> 1) & 3;
        float2* stat = reinterpret_cast<float2*>(sgen + C::oStat) + r;
        bool alive = true;
        int sg = g, sf_parity = 0;               // next item of this group (items count through all units), parity of its scores' barriers
        const Unit* u;
        for (int i = 0; alive && (u = next_unit(i)) != nullptr; ++i) {
        const int ns = uniform(u->ns), two = uniform(u->two), d = uniform(u->d), nb1 = uniform(u->nbmax) - 1, row0 = uniform(u->mt0) * kBlock;
        const int Nk = uniform(u->Nk), shift = CAUSAL ? uniform(u->shift) : 0;
        const float sl2 = p.sm_scale_per_head ? p.sm_scale_per_head[u->hq + (PACK ? min(prow_head, u->nb[1] - 1) : 0)] * 1.4426950408889634f : p.sm_scale_log2;
        const uint64_t sl2x2 = pack2f(sl2, sl2);
        for (; sg < base + ns; sg += C::kGroups, sf_parity ^= 1) {
            const int s = sg - base;
            const int t = (s + d) & two, n = nb1 - ((s + d) >> two);      // tile, key block
            const int trow = row0 + t * kBlock;                           // the tile's first query row
            // Mask only where it can change a score: asked per half and warp (the warp's first row sees least).
            const int lim_min = CAUSAL ? min(Nk - 1, trow + (PACK ? 0 : 32 * quarter) + shift) : Nk - 1;
            // Slot of the item (P buffer, statistics, barriers): each group alternates between two, so that it need not wait for the
            // P V MMA of its previous item.
            const int slot = sg & 7, slot_prev = (sg - 1 - two) & 7;      // ... and of the tile's previous block
            uint8_t* prow = sgen + C::oP + slot * C::kPBytes + r * 64;
            // Waits of an item besides the scores': its P slot and the running maximum of the tile's previous block.  The compiler interleaves
            // the exponentials only between waits, so these stand apart from them: the slot's at the start of the item and the maximum's
            // where all maxima of the row are known (D = 128; 16 384 keys 5 824 -> 5 781 us against the slot's in the middle of the
            // first half), or both while the scores come in (D = 64 rolled, 5 577 -> 5 509; D = 128 spills with that).
            constexpr int kWaits = !ROLL ? 0 : D == 64 ? 2 : 1;
            // The P slot was last read by the P V MMA of the item eight before.  The wait is for the item six before, though: the ring of
            // maxima has eight places too, and the one this item writes was read by the items up to six before, maybe of an earlier unit,
            // which have run through P V then.
            auto p_slot_free = [&]() { return sg < 6 || warp_wait(bar(bPV + ((sg - 6) & 7)), ((sg - 6) >> 3) & 1, abort_flag, p.status, kWaitPEmpty); };
            float m_old = -INFINITY;
            auto previous_max = [&]() {
                if (s > two) {
                    if (!warp_wait(bar(bM + slot_prev * 4 + quarter), ((sg - 1 - two) >> 3) & 1, abort_flag, p.status, kWaitPair)) return false;
                    m_old = stat[slot_prev * 128].x;
                } else if constexpr (SPLIT) {
                    const int pin = uniform(part_in(*u));
                    if (pin >= 0) {
                        if (!warp_wait_word(p.split_flags + pin, 4, abort_flag, p.status, kWaitPart)) return false;
                        m_old = load_written(p.split_state + (size_t)pin * C::kState + 128 * (D + 2) + r);
                    }
                } else if (STATE) {
                    if (carry_in && trow + r < u->Nq) m_old = p.carry_m_in[(size_t)u->bhq * p.Nq + trow + r];
                }
                return true;
            };
            if (kWaits == 1 && !p_slot_free()) { alive = false; break; }
            // The two halves share one copy of the code (17 -> 9 KB of it; the scale phase below takes both halves' maxima and sums).  The
            // softmax warps of a scheduler are in different places of the loop, and what they fetch is a cost of its own: see the head.
            float bm[4], se[4], bm0[4], se0[4], m_run = 0.f;      // of this half; of the first half
#pragma unroll (ROLL ? 1 : 2)
            for (int h = 0; h < 2; ++h) {
                const int buf = h == 0 ? sg % C::kSBufs0 : C::kSBufs0 + sg % C::kSBufs1;
                if (!warp_wait(bar(bSF + 2 * g + h), sf_parity, abort_flag, p.status, kWaitSFull)) { alive = false; break; }
                tc_fence_after();
                float x[64];
                const uint32_t s_addr = tmem + lane_addr + C::cS + 64 * buf;
                const bool masked = n * kBlock + 64 * h + 63 > lim_min;
                auto mask = [&](int i0, int i1) {
                    int lim = Nk - 1;
                    if (CAUSAL) lim = min(lim, trow + tok + shift);
                    const float vis = (float)(lim - (n * kBlock + 64 * h));      // x[0 .. vis] are visible
#pragma unroll
                    for (int i = i0; i < i1; ++i)
                        if ((float)i > vis) x[i] = -INFINITY;
                };
                tmem_ld32(s_addr, x);
                tmem_ld32(s_addr + 32, x + 32);
                if constexpr (kWaits == 2) {           // while the scores come in
                    if (h == 0) {
                        if (!p_slot_free()) alive = false;
                    } else if (!previous_max()) alive = false;
                }
                tc_wait_ld();
                tc_fence_before();
                warp_arrive(bar(bSE + buf), lane);     // in registers: the buffer may be overwritten
                if (kWaits == 2 && !alive) break;
                if (masked) mask(0, 64);
                // Microblock maxima interleaved with the exp2 pass: E = P~ / sf = 6 * 2^((S - bm) s) of a microblock needs only that
                // microblock's maximum, so the maxima of microblock i + 1 are found while the exponentials of microblock i are
                // in flight.
                auto mb_max = [&](int i) {
                    const float* y = x + 16 * i;
                    float a = fmax3(y[0], y[1], y[2]);
                    float b = fmax3(y[3], y[4], y[5]);
                    const float c = fmax3(y[6], y[7], y[8]);
                    const float e = fmax3(y[9], y[10], y[11]);
                    a = fmax3(a, y[12], y[13]);
                    b = fmax3(b, y[14], y[15]);
                    bm[i] = fmax3(a, b, fmax3(c, e, kNoKey));
                };
                mb_max(0);
                uint32_t codes[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float bmi = bm[i];
                    const float negc = fmaf(bmi, -sl2, kLog2Of6);
                    const uint64_t negc2 = pack2f(negc, negc);
                    float e[16];
#pragma unroll
                    for (int q = 0; q < 8; ++q) {
                        float a, b2;
                        unpack2f(fma2(pack2f(x[16 * i + 2 * q], x[16 * i + 2 * q + 1]), sl2x2, negc2), a, b2);
                        e[2 * q] = ex2_approx(a);
                        e[2 * q + 1] = ex2_approx(b2);
                    }
                    if (i < 3) mb_max(i + 1);
                    if (h == 1 && i == 2) {
                        // All maxima of the row are known: running maximum (with the previous block's, from the group that has it)
                        // and O rescale factor, handed to the next block's group and to the correction warps.
                        if (kWaits != 2 && !previous_max()) { alive = false; break; }
                        m_run = fmax3(fmax3(fmaxf(bm0[0], bm0[1]), bm0[2], bm0[3]), fmax3(bm[0], bm[1], bm[2]), fmaxf(bm[3], m_old));
                        const float alpha = ex2_approx((m_old - m_run) * sl2);        // m_old = -inf  ->  0
                        stat[slot * 128] = make_float2(m_run, alpha);
                        warp_arrive(bar(bM + slot * 4 + quarter), lane);
                    }
                    uint64_t acc0 = pack2f(e[0], e[1]), acc1 = pack2f(e[2], e[3]);
                    acc0 = add2(acc0, pack2f(e[4], e[5]));
                    acc1 = add2(acc1, pack2f(e[6], e[7]));
                    acc0 = add2(acc0, pack2f(e[8], e[9]));
                    acc1 = add2(acc1, pack2f(e[10], e[11]));
                    acc0 = add2(acc0, pack2f(e[12], e[13]));
                    acc1 = add2(acc1, pack2f(e[14], e[15]));
                    float sum_lo, sum_hi;
                    unpack2f(add2(acc0, acc1), sum_lo, sum_hi);
                    se[i] = sum_lo + sum_hi;
                    codes[2 * (i & 1)] = cvt_e2m1x8(e[0], e[1], e[2], e[3], e[4], e[5], e[6], e[7]);
                    codes[2 * (i & 1) + 1] = cvt_e2m1x8(e[8], e[9], e[10], e[11], e[12], e[13], e[14], e[15]);
                    if (i & 1) {
                        // P codes of 32 keys: one 16-byte chunk of the 64-byte-swizzled K-major row
                        if (kWaits == 0 && h == 0 && i == 1 && !p_slot_free()) { alive = false; break; }
                        *reinterpret_cast<uint4*>(prow + ((h * 32 + (i >> 1) * 16) ^ (sw << 4))) = make_uint4(codes[0], codes[1], codes[2], codes[3]);
                    }
                }
                if (!alive) break;
                if (h == 0) {
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        bm0[i] = bm[i];
                        se0[i] = se[i];
                    }
                }
            }
            if (!alive) break;
            // E4M3 scale sf = max(P~) / 6 = 2^(bm s - max_scaled - log2 6) of every microblock, weighted sums of the two halves
            const float max_scaled = (m_run == kNoKey) ? 0.f : fmaf(m_run, sl2, kPScaleLog2);       // no key yet: every scale is 2^-huge = 0
            float rowsum[2];
            uint32_t* sfp_row = reinterpret_cast<uint32_t*>(sgen + C::oSfP + slot * 1024 + (r & 31) * 16 + (r >> 5) * 4);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                uint32_t sfb = 0;
                rowsum[h] = 0.f;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float bmi = h == 0 ? bm0[i] : bm[i];
                    const float sfv = ex2_approx(fmaf(bmi, sl2, -max_scaled) - kLog2Of6);
                    rowsum[h] = fmaf(sfv, h == 0 ? se0[i] : se[i], rowsum[h]);
                    sfb |= (cvt_e4m3x2(sfv, 0.f) & 0xffu) << (8 * i);
                }
                sfp_row[128 * h] = sfb;
            }
            reinterpret_cast<float2*>(sgen + C::oSum)[slot * 128 + r] = make_float2(rowsum[0], rowsum[1]);
            fence_proxy_async_smem();
            warp_arrive(bar(bPF + slot), lane);
        }
        unit_done(i);
        base += ns;
        }
        __syncwarp();
    }

    // ---------------------------------------------------------------------- teardown
    tc_fence_before();
    __syncthreads();
    if (*abort_flag != 0) {
        // a wait gave up: give copies that may still be in flight time to land before the CTA retires
        const long long t0 = clock64();
        while (clock64() - t0 < 200000) __nanosleep(1000);
        __syncthreads();
    }
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem, 512);
    }
}

// ------------------------------------------------------------------------------------------------
// host side: tensor maps + launch
// ------------------------------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn get_encode_fn() {
    static EncodeTiledFn fn = nullptr;
    if (fn) return fn;
    void* sym = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &qres) != cudaSuccess ||
        qres != cudaDriverEntryPointSuccess)
        return nullptr;
    fn = reinterpret_cast<EncodeTiledFn>(sym);
    return fn;
}

// byte tensor [n2][n1][n0] (n0 contiguous), box [b2][b1][b0]
static CUresult make_map(EncodeTiledFn fn, CUtensorMap* m, const void* base, uint64_t n0, uint64_t n1, uint64_t n2,
                         uint32_t b0, uint32_t b1, CUtensorMapSwizzle swz, uint32_t b2 = 1) {
    cuuint64_t dims[3] = {n0, n1, n2};
    cuuint64_t strides[2] = {n0, n0 * n1};
    cuuint32_t box[3] = {b0, b1, b2};
    cuuint32_t estr[3] = {1, 1, 1};
    return fn(m, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<void*>(base), dims, strides, box, estr,
              CU_TENSOR_MAP_INTERLEAVE_NONE, swz, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
}

int encode_tiled_bytes(void* map64, const void* base, uint64_t n0, uint64_t n1, uint64_t n2, uint32_t b0, uint32_t b1, int swizzle) {
    EncodeTiledFn fn = get_encode_fn();
    if (!fn) return -1;
    const CUtensorMapSwizzle swz = swizzle == 3 ? CU_TENSOR_MAP_SWIZZLE_128B : swizzle == 2 ? CU_TENSOR_MAP_SWIZZLE_64B
                                 : swizzle == 1 ? CU_TENSOR_MAP_SWIZZLE_32B : CU_TENSOR_MAP_SWIZZLE_NONE;
    return (int)make_map(fn, static_cast<CUtensorMap*>(map64), base, n0, n1, n2, b0, b1, swz);
}

template <int D, bool CAUSAL, typename OutT, bool VARLEN, int PACK, int CARRY = 0, bool ROLL = true>
static cudaError_t launch_v(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const CUtensorMap& td,
                            const SplitParams& p, int grid, cudaStream_t st) {
    constexpr auto kern = attn_fwd_kernel<D, CAUSAL, OutT, VARLEN, PACK, CARRY, ROLL>;
    using C = Cfg<D, PACK>;
    cudaError_t e = allow_smem<kern>(C::kSmemBytes);
    if (e != cudaSuccess) return e;
    return launch(true, kern, dim3(grid), dim3(C::kThreads), C::kSmemBytes, st, tq, tk, tv, td, static_cast<const std::conditional_t<CARRY == 2, SplitParams, AttnParams>&>(p));
}

// D = 64 without a mask, more key blocks than this: the halves of an item unrolled.  us per call, rolled / unrolled: 226 keys (2 x 48 heads,
// 17 550 queries) 245.5 / 282.2, 512 (4 x 24 x 2 000) 60.8 / 62.4, 1 024 98.6 / 98.8, 2 048 (2 x 24 x 2 048) 100.3 / 98.7, 4 250 356.3 / 351.1, 16 384
// (2 x 32 heads) 5 542 / 5 441.  Under a causal mask rolled is faster throughout (1 024: 45.3 / 47.4, 6 000: 328.4 / 335.1), as it is at D = 128.
// Packed batches hold sequences shorter than the longest, which is what the host knows: 24 heads, 24 sequences of 300 to 2 048 tokens 522.8 / 545.1,
// of 400 to 3 072 948.7 / 973.6, of 500 to 4 096 1 620 / 1 641, 12 of 1 000 to 8 192 3 597 / 3 556; of one length, 8 x 3 072 684.5 / 678.1,
// 8 x 4 096 1 150 / 1 137, 8 x 6 144 2 464 / 2 424, 4 x 16 384 (12 heads) 4 161 / 4 089.
constexpr int kRolledBlocks = 8, kRolledBlocksPacked = 32;

template <int D, bool CAUSAL, typename OutT>
static cudaError_t launch_t(const AttnArgs& a, const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const CUtensorMap& td,
                            const SplitParams& p, int pack_mode, int grid, cudaStream_t st) {
    // packed variable-length batches and carried state run their own instantiations, so that the other kernels carry none of it
    const bool carry = a.carry_o_in != nullptr || a.carry_o_out != nullptr;
    constexpr bool roll = D == 128 || CAUSAL;        // at every length
    return a.cu_q != nullptr && !roll && p.nkb > kRolledBlocksPacked ? launch_v<D, CAUSAL, OutT, true, 0, 0, roll>(tq, tk, tv, td, p, grid, st)
           : a.cu_q != nullptr ? launch_v<D, CAUSAL, OutT, true, 0>(tq, tk, tv, td, p, grid, st)
           : carry            ? launch_v<D, CAUSAL, OutT, false, 0, 1, D == 64>(tq, tk, tv, td, p, grid, st)
           : pack_mode == 2   ? launch_v<D, CAUSAL, OutT, false, 2>(tq, tk, tv, td, p, grid, st)
           : pack_mode == 1   ? launch_v<D, CAUSAL, OutT, false, 1>(tq, tk, tv, td, p, grid, st)
           : p.slot_blocks > 0 ? launch_v<D, CAUSAL, OutT, false, 0, 2>(tq, tk, tv, td, p, grid, st)
           : !roll && p.nkb > kRolledBlocks ? launch_v<D, CAUSAL, OutT, false, 0, 0, roll>(tq, tk, tv, td, p, grid, st)
                              : launch_v<D, CAUSAL, OutT, false, 0>(tq, tk, tv, td, p, grid, st);
}

cudaError_t launch_attn(const AttnArgs& a, cudaStream_t st, int* driver_rc) {
    *driver_rc = 0;
    EncodeTiledFn fn = get_encode_fn();
    if (!fn) return cudaErrorNotSupported;
    CUtensorMap tq, tk, tv, td;
    const uint32_t rowb = a.D / 2;
    const CUtensorMapSwizzle swz_qk = (a.D == 128) ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B;
    const int group = a.Hq / a.Hkv;
    const PackRule rule(a.Nq, group, a.cu_q == nullptr && a.carry_o_in == nullptr && a.carry_o_out == nullptr);
    const int pack = rule.heads, mode = rule.mode;
    CUresult r = make_map(fn, &tq, a.q_codes, rowb, a.Nq_p, (uint64_t)a.B * a.Hq, rowb, mode ? a.Nq : kBlock, swz_qk, pack);
    if (r == CUDA_SUCCESS) r = make_map(fn, &tk, a.k_codes, rowb, a.Nk_p, (uint64_t)a.B * a.Hkv, rowb, kBlock, swz_qk);
    if (r == CUDA_SUCCESS)
        r = make_map(fn, &tv, a.v_codes, a.Nk_p / 2, a.D, (uint64_t)a.B * a.Hkv, 64, a.D, CU_TENSOR_MAP_SWIZZLE_64B);
    td = tv;                            // (only the PACK kernels use it)
    if (r == CUDA_SUCCESS && mode) {
        // delta_s as [Nk_p / 8][B * Hq][8 keys]: eight keys of eight heads are one core matrix
        const cuuint64_t dims[3] = {16, (cuuint64_t)a.B * a.Hq, (cuuint64_t)a.Nk_p / 8}, strides[2] = {(cuuint64_t)a.Nk_p * 2, 16};
        const cuuint32_t box[3] = {16, 8, kBlock / 8}, estr[3] = {1, 1, 1};
        r = fn(&td, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<void*>(a.delta), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    }
    if (r != CUDA_SUCCESS) {
        *driver_rc = (int)r;
        return cudaErrorInvalidValue;
    }
    int dev = 0;
    DeviceInfo info;
    const cudaError_t e = current_device(&dev, &info);
    if (e != cudaSuccess) return e;
    const int sms = info.sms;
    SplitParams p;
    // Units of work: pairs of query tiles; in the last rounds single tiles or slots of key blocks.
    const int nqt = a.Nq_p / kBlock, pairs = a.B * a.Hq * ((nqt + 1) / 2), whole = whole_pairs(nqt, pairs, sms);
    p.unit_counter = a.unit_counter;
    SplitPlan plan;
    if (a.split_flags != nullptr && mode == 0 && a.cu_q == nullptr && a.carry_o_in == nullptr && a.carry_o_out == nullptr)
        plan = a.is_causal ? plan_split<true>(a.B * a.Hq, nqt, a.Nk, a.causal_shift, a.D, sms) : plan_split<false>(a.B * a.Hq, nqt, a.Nk, a.causal_shift, a.D, sms);
    p.slot_blocks = plan.blocks; p.slot_rest = plan.rest; p.rest0 = plan.rest0;
    p.split_flags = a.split_flags; p.split_state = a.split_state;
    for (int i = 0; i < plan.slots; ++i) p.slot_first[i] = plan.first[i];
    p.whole_units = plan.slots > 0 ? plan.whole : whole;
    p.pack_heads = pack;
    p.pack_tiles = (group + pack - 1) / pack;
    p.units = mode ? a.B * a.Hkv * p.pack_tiles : plan.slots > 0 ? plan.whole + plan.slots : whole + 2 * (pairs - whole);
    const int grid = p.units < sms ? p.units : sms;
    p.BHq = a.B * a.Hq;
    p.Hq = a.Hq; p.Hkv = a.Hkv; p.Nq = a.Nq; p.Nk = a.Nk;
    p.nqt = a.Nq_p / kBlock; p.nkb = a.Nk_p / kBlock; p.nqm = a.nqm;
    p.sm_scale_log2 = a.sm_scale * 1.4426950408889634f;
    p.sm_scale_per_head = a.sm_scale_per_head;
    p.q_sf = a.q_sf; p.k_sf = a.k_sf; p.v_sf = a.v_sf;
    p.delta = static_cast<const uint16_t*>(a.delta);
    for (int i = 0; i < kMaxParts; ++i) p.out[i] = a.out.base[i];
    p.out_rows = a.out.rows;
    p.out_wide = a.os[0] % 16 == 0 && a.os[1] % 16 == 0 && a.os[2] % 16 == 0;
    for (int i = 0; i < kMaxParts; ++i) p.out_wide &= reinterpret_cast<uintptr_t>(a.out.base[i]) % 32 == 0;
    p.lse = a.lse; p.qkm = a.qkm; p.sm_scale = a.sm_scale;
    p.os0 = a.os[0]; p.os1 = a.os[1]; p.os2 = a.os[2];
    p.status = a.status;
    p.prepass_status = a.prepass_status;
    p.nonfinite = a.nonfinite;
    p.carry_o_in = a.carry_o_in; p.carry_m_in = a.carry_m_in; p.carry_l_in = a.carry_l_in;
    p.carry_o_out = a.carry_o_out; p.carry_m_out = a.carry_m_out; p.carry_l_out = a.carry_l_out;
    p.causal_shift = a.causal_shift;
    p.cu_q = a.cu_q; p.cu_k = a.cu_k;
    if (a.is_bf16) {
        if (a.D == 128) return a.is_causal ? launch_t<128, true, __nv_bfloat16>(a, tq, tk, tv, td, p, mode, grid, st)
                                           : launch_t<128, false, __nv_bfloat16>(a, tq, tk, tv, td, p, mode, grid, st);
        return a.is_causal ? launch_t<64, true, __nv_bfloat16>(a, tq, tk, tv, td, p, mode, grid, st)
                           : launch_t<64, false, __nv_bfloat16>(a, tq, tk, tv, td, p, mode, grid, st);
    }
    if (a.D == 128) return a.is_causal ? launch_t<128, true, __half>(a, tq, tk, tv, td, p, mode, grid, st)
                                       : launch_t<128, false, __half>(a, tq, tk, tv, td, p, mode, grid, st);
    return a.is_causal ? launch_t<64, true, __half>(a, tq, tk, tv, td, p, mode, grid, st)
                       : launch_t<64, false, __half>(a, tq, tk, tv, td, p, mode, grid, st);
}

}  // namespace sage3
