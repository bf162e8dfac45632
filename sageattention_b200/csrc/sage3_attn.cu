// Block-scaled FP4 attention for sm_100a: TMA-staged E2M1 tiles, tcgen05 NVFP4 MMAs with the S and O
// accumulators in tensor memory, exp2 online softmax, P re-quantized to NVFP4 before the PV MMA.
//
// One CTA per PAIR of 128-row query tiles of one head; every K / V^T stage in shared memory serves both tiles.  The
// CTA's work is one stream of items (key block, tile), the two tiles in turn.  Six warpgroups (setmaxnreg moves
// registers to the softmax warpgroups):
//   warp 0       TMA producer (one lane): both Q tiles once, then K (+ one delta_s row per tile) / V^T / scale atoms per block
//   warps 1, 3   Q K^T MMA issuers, for keys [0, 64) and [64, 128) of every item; warp 1 owns the tensor-memory allocation
//   warp 2       P V MMA issuer
//   warps 4-19   four softmax groups of four warps; group g takes the items g, g + 4, ...  A thread owns one row of the block
//                and walks its 128 keys in two halves of 64 (the scores of a half live in registers).
//   warps 20-23  O rescale ("correction"), one warp per tensor-memory lane quarter: when a row of the quarter moved
//                its maximum, the warp multiplies the 32 O rows of its quarter by their factors before the block's
//                P V MMA is issued; it also keeps the running row sums.  The softmax warps never touch O inside the loop.
// Per half a softmax thread pulls its 64 scores out of tensor memory (the S buffer is free again at once) and runs the
// exp2 pass microblock by microblock, the maxima of the next microblock found under the exponentials of the current one:
// with E = P~ / sf = 6 * 2^((S - bm) s), the exp2 values and FP4 codes of a microblock depend on the maximum bm of that
// microblock only.  The running row maximum enters just the E4M3 scales, the row sum and the O rescale factor; it is handed
// from the group that has a tile's block to the group that has the next one as soon as all maxima of the row are known, and
// nothing else connects the groups: four independent chains per scheduler, a quarter of an item apart.
// What bounds it: the exp2 unit (16 results per clock and SM: 1 096 cycles per 128 x 128 block with the exponentials of the
// scales) and, next to it, the instruction latency of the softmax warps; the tensor pipe needs 580 cycles.  Measured (B = 2,
// H = 32, N = 16 384): 1 545 cycles per block at D = 128 and 1 525 at D = 64, the exp2 unit 77 % busy.  (With a row shared by two
// threads and all warps of a tile in step, as this kernel was before: 1 640 and 1 590.)  Halves of 64 keys because a thread's
// registers hold 64 scores, and because tensor memory has room for three 64-key buffers next to two O tiles at D = 128.

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

namespace sage3 {

constexpr float kNoKey = -1e30f;                      // maximum of a microblock without visible keys (keeps -inf - -inf out of the arithmetic)
constexpr float kLog2Of6 = 2.584962500721156f;
constexpr float kPScaleLog2 = -11.392317422778762f;   // log2(1 / (448 * 6)), softmax_fused.h:33

struct AttnParams {
    int Hq, Hkv, Nq, Nk, nqt, nkb, nqm;   // nqt = query tiles per head, nkb = KV blocks per head
    float sm_scale_log2;
    const float* sm_scale_per_head;
    const uint8_t *q_sf, *k_sf, *v_sf;
    const uint16_t* delta;              // 16-bit elements [B*Hq][nqm][nkb*128]
    void* out[kMaxParts];               // output buffers; out_rows == 0: one buffer
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
};

template <int D>
struct Cfg {
    static constexpr int kStages = (D == 128) ? 5 : 8;        // K and V^T stages, each shared by the two query tiles
    static constexpr int kThreads = 768;                      // 6 warpgroups, see the kernel
    // S buffers of 128 rows x 64 keys: a rotation for the first halves of the items and one for the second halves
    static constexpr int kSBufs0 = 2, kSBufs1 = (D == 128) ? 1 : 2, kSBufs = kSBufs0 + kSBufs1;
    static constexpr int kQBytes = 128 * D / 2;               // per query tile
    static constexpr int kSfQkBytes = (D / 64) * 512;
    static constexpr int kKBytes = 128 * D / 2;
    static constexpr int kVBytes = D * 64;
    static constexpr int kSfVBytes = 1024;
    static constexpr int kDeltaBytes = 256;
    static constexpr int kPBytes = 8192;
    // shared-memory map (bytes from a 1024-aligned base)
    static constexpr int oQ = 0;                              // [tile] 8192
    static constexpr int oK = oQ + 2 * 8192;
    static constexpr int oV = oK + kStages * kKBytes;
    static constexpr int oP = oV + kStages * kVBytes;            // [slot] 8192
    static constexpr int oSfQ = oP + 8 * kPBytes;             // [tile] 1024
    static constexpr int oSfK = oSfQ + 2 * 1024;
    static constexpr int oSfV = oSfK + kStages * 1024;
    static constexpr int oSfP = oSfV + kStages * 1024;        // [slot] 1024
    static constexpr int kDeltaPitch = 512;                   // 256 B of delta_s + 256 B that stay zero
    static constexpr int oDelta = oSfP + 8 * 1024;            // [stage][tile] kDeltaPitch
    static constexpr int oOnes = oDelta + kStages * 2 * kDeltaPitch;   // 128 x 16 tile: column 0 = 1.0, rest 0
    static constexpr int oStat = oOnes + 4096;                // float2 [slot][128 rows]: running maximum, rescale factor
    static constexpr int oSum = oStat + 8192;                 // float2 [slot][128 rows]: row sums of the two key halves of a block
    static constexpr int oL = oSum + 8192;                    // float2 [tile][128 rows]: running row sums of the two key halves
    static constexpr int oBar = oL + 2048;
    static constexpr int kNumBars = 2 + 4 * kStages + kSBufs + 8 + 7 * 8 + 8;
    static constexpr int oMisc = oBar + kNumBars * 8;
    static constexpr int kSmemBytes = oMisc + 64 + 1024;      // + slack for the manual 1024-byte alignment
    // tensor-memory columns: the S buffers, one O accumulator per tile, scale factors (K: one copy per issuer)
    static constexpr uint32_t cS = 0, cO = 64 * kSBufs, cSfQ = cO + 2 * D, cSfK = cSfQ + 16, cSfV = cSfK + 16, cSfP = cSfV + 8;
    static_assert(cSfP + 8 <= 512, "tensor memory");
    static constexpr uint64_t kSwzQK = (D == 128) ? kSwz64 : kSwz32;
    static constexpr uint32_t kSboQK = (D == 128) ? 512 : 256;
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

// A value that is the same in all lanes, marked as such for the compiler (uniform registers feed the tcgen05 instructions).
__device__ __forceinline__ int uniform(int v) { return __shfl_sync(0xffffffffu, v, 0); }

// Wait executed by a whole converged warp; the verdict is made warp-uniform so that no lane leaves a loop alone.
__device__ __forceinline__ bool warp_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag, int* status, int code) {
    const bool ok = mbar_wait(bar, parity, abort_flag, status, code);
    return __all_sync(0xffffffffu, ok);
}

template <int D, bool CAUSAL, typename OutT, bool VARLEN>
__global__ void __launch_bounds__(Cfg<D>::kThreads, 1)
attn_fwd_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ AttnParams p) {
    using C = Cfg<D>;
    constexpr int S = C::kStages;
    extern __shared__ uint8_t smem_dyn[];
    const uint32_t sbase = (smem_u32(smem_dyn) + 1023u) & ~1023u;
    uint8_t* sgen = smem_dyn + (sbase - smem_u32(smem_dyn));

    const int warp = uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;

    // barriers
    const uint32_t bars = uniform(sbase + C::oBar);
    auto bar = [&](int i) { return bars + 8u * i; };
    constexpr int bQ = 0, bSQ = 1, bKF = 2, bKE = bKF + S, bVF = bKE + S, bVE = bVF + S, bSF = bVE + S, bSE = bSF + 8, bM = bSE + C::kSBufs,
                  bPF = bM + 32, bPV = bPF + 8, bOS = bPV + 8, bL = bOS + 8;
    volatile int* abort_flag = reinterpret_cast<volatile int*>(sgen + C::oMisc);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sgen + C::oMisc + 8);

    // CTA -> (batch*head, pair of query tiles); heavier causal pairs are scheduled first
    const int npair = (p.nqt + 1) >> 1;
    const int bhq = blockIdx.x / npair;
    int pr = blockIdx.x % npair;
    if (CAUSAL) pr = npair - 1 - pr;
    const int mt0 = 2 * pr;
    const int b = bhq / p.Hq, hq = bhq % p.Hq;
    const int bhkv = b * p.Hkv + hq / (p.Hq / p.Hkv);
    // Lengths of this batch entry.  p.Nq, p.Nk, p.nqt, p.nkb stay the strides of the workspace layouts; with packed
    // variable-length sequences they are the maxima and the entry's own lengths come from the cu arrays.
    int Nq = p.Nq, Nk = p.Nk, nqt = p.nqt, nkb = p.nkb, shift = p.causal_shift;
    int64_t out_base = b * p.os0;
    if constexpr (VARLEN) {
        const int q0 = p.cu_q[b], k0 = p.cu_k[b];
        Nq = min(max(p.cu_q[b + 1] - q0, 0), p.Nq);
        Nk = min(max(p.cu_k[b + 1] - k0, 0), p.Nk);
        nqt = (Nq + kBlock - 1) / kBlock;
        nkb = (Nk + kBlock - 1) / kBlock;
        shift = Nk - Nq;
        out_base = (int64_t)q0 * p.os2;
    }
    const int nv = (mt0 + 1 < nqt) ? 2 : (VARLEN && mt0 >= nqt ? 0 : 1);   // query tiles this CTA really has
    // an earlier CTA of this launch gave up, or the pre-pass did (the workspace is then incomplete)
    const bool dead_launch = (*reinterpret_cast<volatile int*>(p.status) != 0) || (*reinterpret_cast<const volatile int*>(p.prepass_status) != 0);
    // KV blocks of tile t: [0, nbt[t]); the CTA walks block n = nbmax - 1 ... 0.  Under a causal mask tile 1 may start one
    // block earlier than tile 0 (their rows differ by one block), never more.
    int nbt[2];
#pragma unroll
    for (int t = 0; t < 2; ++t) {
        int nb = nkb;
        if (CAUSAL) {
            const int max_key = min(Nk - 1, (mt0 + t) * kBlock + kBlock - 1 + shift);
            nb = max_key < 0 ? 0 : max_key / kBlock + 1;
        }
        nbt[t] = (dead_launch || t >= nv) ? 0 : nb;
    }
    const int nbmax = uniform(max(nbt[0], nbt[1]));
    // The work is one stream of (block step jj, tile t) items, s = 0 ... ns - 1: with two tiles they alternate, sd = s + d,
    // t = sd & 1, jj = sd >> 1 (d = 1: the stream starts with tile 1 alone); with one tile jj = s.
    const int two = uniform(nv == 2 ? 1 : 0);
    const int d = uniform(two ? nbt[1] - nbt[0] : 0);
    const int ns = uniform(nbt[0] + nbt[1]);

    // One barrier per thread: the number of arrivals that completes a phase.
    if (threadIdx.x < C::kNumBars) {
        const int i = threadIdx.x;
        uint32_t count = 1;                                      // copies landed, MMAs complete, one warp's statistics
        if (i >= bKE && i < bKE + S) count = 2;                  // K stage free: both Q K^T issuers are done with it
        if (i >= bSE && i < bM) count = 4;                       // S buffer free: the four warps of its group hold the scores
        if (i >= bPF && i < bPV) count = 4;                      // P, its scales and the row sums written
        if (i >= bOS && i < bL) count = 4;                       // the correction warps are done with O (and have seen P written)
        mbar_init(bar(i), count);
        mbar_fence_init();
    }
    if (threadIdx.x == 0) *abort_flag = 0;
    // delta_s stages: the 256 bytes behind each row stay zero for the whole kernel; ones tile:
    // [k chunk][row group][8 rows][16 bytes], 1.0 in element 0 of every row of chunk 0
    {
        uint4* z = reinterpret_cast<uint4*>(sgen + C::oDelta);
        constexpr int nd = S * 2 * C::kDeltaPitch / 16;
        const uint32_t one = std::is_same<OutT, __nv_bfloat16>::value ? 0x3F80u : 0x3C00u;
        for (int i = threadIdx.x; i < nd + 4096 / 16; i += C::kThreads) z[i] = make_uint4(i >= nd && i < nd + 128 ? one : 0u, 0, 0, 0);
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
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = uniform(*tmem_slot);

    const float sl2 = p.sm_scale_per_head ? p.sm_scale_per_head[hq] * 1.4426950408889634f : p.sm_scale_log2;
    const bool carry_in = (p.carry_o_in != nullptr);
    if (carry_in) {
        // resume: O continues from the state an earlier call left (its key range came later in the walk)
        if (warp >= 4 && warp < 4 + 4 * 2) {
            const int t = (warp >> 2) - 1, r = (warp & 3) * 32 + lane, grow = (mt0 + t) * kBlock + r;
            const bool live = t < nv && grow < Nq && !dead_launch;
            const float* src = p.carry_o_in + ((size_t)bhq * p.Nq + grow) * D;
            for (int cc = 0; cc < D / 16; ++cc) {
                float o[16];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float4 v4 = live ? *reinterpret_cast<const float4*>(src + cc * 16 + 4 * i) : make_float4(0.f, 0.f, 0.f, 0.f);
                    o[4 * i] = v4.x; o[4 * i + 1] = v4.y; o[4 * i + 2] = v4.z; o[4 * i + 3] = v4.w;
                }
                tmem_st16(tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16) + C::cO + t * D + cc * 16, o);
            }
            tc_wait_st();
        }
        tc_fence_before();
        __syncthreads();
        tc_fence_after();
    }

    // Register budget: 768 threads start with 80 registers each, and that allocation (61 440) is all the CTA can
    // ever hold: 128 x kRoleRegs for warpgroup 0 (three single-lane roles) + 128 x kCorrRegs for the correction
    // warpgroup + 512 x 104 for the softmax warpgroups.  (An increase beyond the launch allocation would wait forever.)
    constexpr int kRoleRegs = (D == 64) ? 24 : 32, kCorrRegs = 64 - kRoleRegs;
    if (warp >= 20) {
      reg_dealloc<kCorrRegs>();
      // ------------------------------------------------------------------ O rescale (correction), one warp per lane quarter
      // Also keeps the running row sums: l = l alpha + (sum over the block), for each half of the keys.
      const int quarter = warp & 3, row = quarter * 32 + lane;
      const uint32_t lane_addr = static_cast<uint32_t>(quarter * 32) << 16;
      const float2* stat = reinterpret_cast<const float2*>(sgen + C::oStat);
      const float2* sum = reinterpret_cast<const float2*>(sgen + C::oSum);
      float2* l_s = reinterpret_cast<float2*>(sgen + C::oL);
      for (int t = 0; t < 2; ++t) {
          const int grow = (mt0 + t) * kBlock + row;
          const bool from = p.carry_l_in != nullptr && t < nv && grow < Nq && !dead_launch;
          l_s[t * 128 + row] = from ? *reinterpret_cast<const float2*>(p.carry_l_in + 2 * ((size_t)bhq * p.Nq + grow)) : make_float2(0.f, 0.f);
      }
      bool ok = true;
      for (int s = 0; s < ns; ++s) {
          const int g = s & 7, ph = (s >> 3) & 1;
          const int t = two ? (s + d) & 1 : 0;
          const bool first = s <= two;                              // the tile's first block
          if (!warp_wait(bar(bM + g * 4 + quarter), ph, abort_flag, p.status, kWaitAlpha)) { ok = false; break; }
          const float alpha = stat[g * 128 + row].y;
          // the first block has nothing to rescale unless the accumulator was carried in
          if ((!first || carry_in) && __any_sync(0xffffffffu, alpha != 1.0f)) {
              // the P V MMA of the tile's previous block must have landed first
              if (!first) {
                  const int sp = s - 1 - two;
                  if (!warp_wait(bar(bPV + (sp & 7)), (sp >> 3) & 1, abort_flag, p.status, kWaitOReady)) { ok = false; break; }
              }
              tc_fence_after();
              const uint64_t a2 = pack2f(alpha, alpha);
              const uint32_t o_addr = tmem + lane_addr + C::cO + t * D;
#pragma unroll
              for (int cc = 0; cc < D / 16; ++cc) {
                  float o0[16];
                  tmem_ld16(o_addr + cc * 16, o0);
                  tc_wait_ld();
#pragma unroll
                  for (int i = 0; i < 8; ++i)
                      unpack2f(mul2(pack2f(o0[2 * i], o0[2 * i + 1]), a2), o0[2 * i], o0[2 * i + 1]);
                  tmem_st16(o_addr + cc * 16, o0);
              }
              tc_wait_st();
          }
          tc_fence_before();
          // P V issue waits for this warpgroup only, so its arrival also stands for "P is written"
          if (!warp_wait(bar(bPF + g), ph, abort_flag, p.status, kWaitPFull)) { ok = false; break; }
          const float2 rs = sum[g * 128 + row];
          warp_arrive(bar(bOS + g), lane);
          float2 l = l_s[t * 128 + row];
          l.x = fmaf(l.x, alpha, rs.x);
          l.y = fmaf(l.y, alpha, rs.y);
          l_s[t * 128 + row] = l;
      }
      if (ok && !dead_launch) {
          for (int t = 0; t < nv; ++t) {
              const int grow = (mt0 + t) * kBlock + row;
              if (p.carry_l_out != nullptr && grow < Nq)
                  *reinterpret_cast<float2*>(p.carry_l_out + 2 * ((size_t)bhq * p.Nq + grow)) = l_s[t * 128 + row];
              warp_arrive(bar(bL + t * 4 + quarter), lane);
          }
      }
      __syncwarp();
    } else if (warp < 4) {
      reg_dealloc<kRoleRegs>();
      if (warp == 0) {
        // ------------------------------------------------------------------ TMA producer
        if (lane == 0 && nbmax > 0) {
            mbar_expect_tx(bar(bQ), nv * (C::kQBytes + C::kSfQkBytes));
            const uint16_t* dptr[2];
            for (int t = 0; t < nv; ++t) {
                tma_load_3d(sbase + C::oQ + t * 8192, &tm_q, bar(bQ), 0, (mt0 + t) * kBlock, bhq);
                bulk_load(sbase + C::oSfQ + t * 1024, p.q_sf + ((size_t)bhq * p.nqt + mt0 + t) * C::kSfQkBytes,
                          C::kSfQkBytes, bar(bQ));
                const int drow = (p.nqm > 1) ? mt0 + t : 0;
                dptr[t] = p.delta + ((size_t)bhq * p.nqm + drow) * ((size_t)p.nkb * kBlock);
            }
            for (int jj = 0; jj < nbmax; ++jj) {
                const int n = nbmax - 1 - jj, st = jj % S;
                if (jj >= S && !mbar_wait<true>(bar(bKE + st), ((jj / S) - 1) & 1, abort_flag, p.status, kWaitKEmpty)) break;
                mbar_expect_tx(bar(bKF + st), C::kKBytes + C::kSfQkBytes + nv * C::kDeltaBytes);
                tma_load_3d(sbase + C::oK + st * C::kKBytes, &tm_k, bar(bKF + st), 0, n * kBlock, bhkv);
                bulk_load(sbase + C::oSfK + st * 1024, p.k_sf + ((size_t)bhkv * p.nkb + n) * C::kSfQkBytes,
                          C::kSfQkBytes, bar(bKF + st));
                for (int t = 0; t < nv; ++t)
                    bulk_load(sbase + C::oDelta + (st * 2 + t) * C::kDeltaPitch, dptr[t] + (size_t)n * kBlock,
                              C::kDeltaBytes, bar(bKF + st));
                if (jj >= S && !mbar_wait<true>(bar(bVE + st), ((jj / S) - 1) & 1, abort_flag, p.status, kWaitVEmpty)) break;
                mbar_expect_tx(bar(bVF + st), C::kVBytes + C::kSfVBytes);
                tma_load_3d(sbase + C::oV + st * C::kVBytes, &tm_v, bar(bVF + st), n * 64, 0, bhkv);
                bulk_load(sbase + C::oSfV + st * 1024, p.v_sf + ((size_t)bhkv * p.nkb + n) * C::kSfVBytes,
                          C::kSfVBytes, bar(bVF + st));
            }
        }
        __syncwarp();
      } else if (warp == 1 || warp == 3) {
        // ------------------------------------------------------------------ Q K^T MMA issuers
        // The scores of a stream item are formed in two halves of 64 keys; warp 1 issues the first halves, warp 3 the second
        // ones, each into its own S buffers (issuing one half takes a few hundred cycles next to busy softmax warps: one
        // issuer for both would be the slowest part of the pipeline).  The whole warp walks the loop and one elected lane
        // issues, so loop state and descriptors stay in uniform registers.
        const int h = warp >> 1;
        if (ns > 0) {
            constexpr uint32_t idesc_qk = make_idesc_nvfp4(64);
            constexpr uint32_t idesc_delta = make_idesc_f16_bmn(64, std::is_same<OutT, __nv_bfloat16>::value);
            // descriptors: constant high words, low words that move with the stage, tile and key half (bytes / 16)
            constexpr uint32_t hi_qk = sdesc_hi(C::kSboQK, C::kSwzQK), hi_ones = sdesc_hi(128, kSwzNone), hi_delta = sdesc_hi(16, kSwzNone);
            const uint32_t ones_lo = sdesc_lo(sbase + C::oOnes, 2048), q_lo = sdesc_lo(sbase + C::oQ, 16);
            const uint32_t k_lo0 = sdesc_lo(sbase + C::oK + h * (64 * D / 2), 16), delta_lo0 = sdesc_lo(sbase + C::oDelta + h * 128, 16);
            const uint32_t sfk_lo0 = sdesc_lo(sbase + C::oSfK, 0);
            const uint32_t sfk_col = tmem + C::cSfK + 8 * h;        // the 128-key atoms; keys 64 .. 127 start two columns in
            bool ok;
            if (h == 0) {
                ok = warp_wait(bar(bQ), 0, abort_flag, p.status, kWaitQFull);
                if (ok && elect_one()) {
                    for (int t = 0; t < nv; ++t)
#pragma unroll
                        for (int ks = 0; ks < D / 64; ++ks)
                            tc_cp_sf(tmem + C::cSfQ + 8 * t + 4 * ks, make_sdesc(sbase + C::oSfQ + t * 1024 + ks * 512, 0, 128, kSwzNone));
                    tc_commit(bar(bSQ));
                }
                __syncwarp();
            } else {
                ok = warp_wait(bar(bSQ), 0, abort_flag, p.status, kWaitQFull);
            }
            const int nbuf = h == 0 ? C::kSBufs0 : C::kSBufs1, buf0 = h == 0 ? 0 : C::kSBufs0;
            int buf = 0, buf_parity = 1;              // next S buffer; parity of its "empty" phase (a fresh barrier passes parity 1)
            int st = 0, st_parity = 0;                // K stage
            for (int s = 0; ok && s < ns; ++s) {
                const int t = two ? (s + d) & 1 : 0;
                const bool opens = t == 0 || s == 0, closes = t == two;       // first / last item of its K block
                if (opens && !warp_wait(bar(bKF + st), st_parity, abort_flag, p.status, kWaitKFull)) break;
                if (!warp_wait(bar(bSE + buf0 + buf), buf_parity, abort_flag, p.status, kWaitSEmpty)) break;
                tc_fence_after();
                const uint32_t k_lo = k_lo0 + st * (C::kKBytes / 16), delta_lo = delta_lo0 + (st * 2 + t) * (C::kDeltaPitch / 16);
                const uint32_t sfk_lo = sfk_lo0 + st * (1024 / 16), qt_lo = q_lo + t * (8192 / 16);
                const uint32_t s_col = tmem + C::cS + 64 * (buf0 + buf), sfq_col = tmem + C::cSfQ + 8 * t;
                if (elect_one()) {
                    if (opens) {
#pragma unroll
                        for (int ks = 0; ks < D / 64; ++ks) tc_cp_sf(sfk_col + 4 * ks, sdesc(sfk_lo + ks * 32, sdesc_hi(128, kSwzNone)));
                    }
                    // S <- 1 (x) delta_s: A = [128 x 16] with ones in column 0 (K-major), B = 64 elements of the delta_s row read as an
                    // MN-major [16 x 64] operand whose rows 1..15 alias finite data and meet zeros in A
                    tc_mma_f16(s_col, sdesc(ones_lo, hi_ones), sdesc(delta_lo, hi_delta), idesc_delta, false);
#pragma unroll
                    for (int ks = 0; ks < D / 64; ++ks)
                        tc_mma_nvfp4(s_col, sdesc(qt_lo + 2 * ks, hi_qk), sdesc(k_lo + 2 * ks, hi_qk), idesc_qk, sfq_col + 4 * ks,
                                     sfk_col + 4 * ks + 2 * h, true);
                    tc_commit(bar(bSF + 2 * (s & 3) + h));
                    if (closes) tc_commit(bar(bKE + st));
                }
                __syncwarp();
                if (++buf == nbuf) { buf = 0; buf_parity ^= 1; }
                if (closes && ++st == S) { st = 0; st_parity ^= 1; }
            }
        }
        __syncwarp();
      } else if (warp == 2) {
        // ------------------------------------------------------------------ PV MMA issuer
        if (ns > 0) {
            constexpr uint32_t idesc_pv = make_idesc_nvfp4(D);
            constexpr uint32_t hi_pv = sdesc_hi(512, kSwz64), hi_sf = sdesc_hi(128, kSwzNone);
            const uint32_t v_lo0 = sdesc_lo(sbase + C::oV, 16), p_lo0 = sdesc_lo(sbase + C::oP, 16);
            const uint32_t sfv_lo0 = sdesc_lo(sbase + C::oSfV, 0), sfp_lo0 = sdesc_lo(sbase + C::oSfP, 0);
            const uint32_t sfp_col = tmem + C::cSfP, sfv_col = tmem + C::cSfV;
            int st = 0, st_parity = 0;
            for (int s = 0; s < ns; ++s) {
                const int g = s & 7, t = two ? (s + d) & 1 : 0;
                const bool opens = t == 0 || s == 0, closes = t == two;       // first / last item of its V block
                if (opens && !warp_wait(bar(bVF + st), st_parity, abort_flag, p.status, kWaitVFull)) break;
                if (!warp_wait(bar(bOS + g), (s >> 3) & 1, abort_flag, p.status, kWaitOScaled)) break;
                tc_fence_after();
                const uint32_t v_lo = v_lo0 + st * (C::kVBytes / 16), p_lo = p_lo0 + g * (C::kPBytes / 16);
                const uint32_t sfv_lo = sfv_lo0 + st * (1024 / 16), sfp_lo = sfp_lo0 + g * (1024 / 16), o_col = tmem + C::cO + t * D;
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
                                     s > two || (ks > 0) || carry_in);
                    tc_commit(bar(bPV + g));
                    if (closes) tc_commit(bar(bVE + st));
                }
                __syncwarp();
                if (closes && ++st == S) { st = 0; st_parity ^= 1; }
            }
        }
        __syncwarp();
      }
    } else {
        reg_alloc<104>();
        // ------------------------------------------------------------------ softmax groups (4 x 4 warps)
        // Group g (one warpgroup) takes the stream items s = g, g + 4, ...; a thread owns one row (tensor-memory lane) of the
        // block and walks its 128 keys in two halves of 64.  With two tiles a group always serves the same tile.
        const int g = (warp >> 2) - 1;
        const int quarter = warp & 3;            // tensor-memory lane quarter this warp may touch
        const int r = quarter * 32 + lane;       // row inside the tile
        const uint32_t lane_addr = static_cast<uint32_t>(quarter * 32) << 16;
        const int t = two ? (g + d) & 1 : 0;
        const int mt = mt0 + t;
        const int grow = mt * kBlock + r;        // query index
        const int sw = (r >> 1) & 3;
        const uint64_t sl2x2 = pack2f(sl2, sl2);
        float2* stat = reinterpret_cast<float2*>(sgen + C::oStat) + r;
        const size_t crow = (size_t)bhq * p.Nq + grow;           // row of the carried state
        float m_run = -INFINITY;
        if (carry_in && t < nv && grow < Nq) m_run = p.carry_m_in[crow];
        bool alive = true;
        for (int s = g; s < ns; s += 4) {
            const int n = nbmax - 1 - (two ? (s + d) >> 1 : s);      // key block
            const bool need_mask = ((n + 1) * kBlock > Nk) || (CAUSAL && (n * kBlock + kBlock - 1 > mt * kBlock + shift));
            // Slot of the item (P buffer, statistics, barriers): each group alternates between two, so that it need not wait for the
            // P V MMA of its previous item.
            const int slot = s & 7, slot_prev = (s - 1 - two) & 7;      // ... and of the tile's previous block
            uint8_t* prow = sgen + C::oP + slot * C::kPBytes + r * 64;
            float bm[8], se[8];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int buf = h == 0 ? s % C::kSBufs0 : C::kSBufs0 + s % C::kSBufs1;
                if (!warp_wait(bar(bSF + 2 * g + h), (s >> 2) & 1, abort_flag, p.status, kWaitSFull)) { alive = false; break; }
                tc_fence_after();
                float x[64];
                tmem_ld32(tmem + lane_addr + C::cS + 64 * buf, x);
                tmem_ld32(tmem + lane_addr + C::cS + 64 * buf + 32, x + 32);
                tc_wait_ld();
                tc_fence_before();
                warp_arrive(bar(bSE + buf), lane);     // in registers: the buffer may be overwritten
                if (need_mask) {
                    int lim = Nk - 1;
                    if (CAUSAL) lim = min(lim, grow + shift);
                    const int key0 = n * kBlock + 64 * h;
#pragma unroll
                    for (int i = 0; i < 64; ++i)
                        if (key0 + i > lim) x[i] = -INFINITY;
                }
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
                    bm[4 * h + i] = fmax3(a, b, fmax3(c, e, kNoKey));
                };
                mb_max(0);
                uint32_t codes[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float bmi = bm[4 * h + i];
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
                        if (s > two) {
                            if (!warp_wait(bar(bM + slot_prev * 4 + quarter), ((s - 1 - two) >> 3) & 1, abort_flag, p.status, kWaitPair)) { alive = false; break; }
                            m_run = stat[slot_prev * 128].x;
                        }
                        const float m_old = m_run;
                        m_run = fmax3(fmax3(fmaxf(bm[0], bm[1]), bm[2], bm[3]), fmax3(bm[4], bm[5], bm[6]), fmaxf(bm[7], m_run));
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
                    float se0, se1;
                    unpack2f(add2(acc0, acc1), se0, se1);
                    se[4 * h + i] = se0 + se1;
                    codes[2 * (i & 1)] = cvt_e2m1x8(e[0], e[1], e[2], e[3], e[4], e[5], e[6], e[7]);
                    codes[2 * (i & 1) + 1] = cvt_e2m1x8(e[8], e[9], e[10], e[11], e[12], e[13], e[14], e[15]);
                    if (i & 1) {
                        // P codes of 32 keys: one 16-byte chunk of the 64-byte-swizzled K-major row.  The P buffer was last read
                        // by the P V MMA of the group's item before the previous one.
                        if (h == 0 && i == 1 && s >= 8 &&
                            !warp_wait(bar(bPV + slot), ((s >> 3) - 1) & 1, abort_flag, p.status, kWaitPEmpty)) { alive = false; break; }
                        *reinterpret_cast<uint4*>(prow + (((2 * h + (i >> 1)) ^ sw) << 4)) = make_uint4(codes[0], codes[1], codes[2], codes[3]);
                    }
                }
                if (!alive) break;
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
                    const float bmi = bm[4 * h + i];
                    const float sfv = ex2_approx(fmaf(bmi, sl2, -max_scaled) - kLog2Of6);
                    rowsum[h] = fmaf(sfv, se[4 * h + i], rowsum[h]);
                    sfb |= (cvt_e4m3x2(sfv, 0.f) & 0xffu) << (8 * i);
                }
                sfp_row[128 * h] = sfb;
            }
            reinterpret_cast<float2*>(sgen + C::oSum)[slot * 128 + r] = make_float2(rowsum[0], rowsum[1]);
            fence_proxy_async_smem();
            warp_arrive(bar(bPF + slot), lane);
        }
        // ------------------------------------------------------------------ epilogue: O / l
        // The groups of a tile take equal shares of its columns.
        if (alive && !dead_launch && nv > 0) {
            const int nb = nbt[t];
            const int share = two ? D / 2 : D / 4, c0 = (two ? g >> 1 : g) * share;
            const int s_last = two ? 2 * (nbmax - 1) + t - d : nb - 1;
            alive = warp_wait(bar(bL + t * 4 + quarter), 0, abort_flag, p.status, kWaitPair);
            if (alive && nb > 0) alive = warp_wait(bar(bPV + (s_last & 7)), (s_last >> 3) & 1, abort_flag, p.status, kWaitOReady);
            tc_fence_after();
            const float2 l2 = reinterpret_cast<const float2*>(sgen + C::oL)[t * 128 + r];
            const float l_tot = l2.x + l2.y;
            if (alive && grow < Nq && (nb > 0 ? g == (s_last & 3) : c0 == 0)) {      // the group that has the final maximum
                if (p.lse != nullptr) {
                    // ln sum_k exp(scale * q.k): the kernel's row sum is 2688 * sum_k 2^((S_k - m) s) over the smoothed
                    // scores S (delta_s included); K smoothing took scale * q.km out of every score of the row
                    const float ms_fin = m_run * sl2;       // (without keys l is 0, whatever this is)
                    const float scale = p.sm_scale_per_head ? p.sm_scale_per_head[hq] : p.sm_scale;
                    const float v = (ms_fin + __log2f(l_tot) + kPScaleLog2) * 0.6931471805599453f +
                                    scale * p.qkm[(size_t)bhq * p.nqt * kBlock + grow];
                    p.lse[(size_t)bhq * p.Nq + grow] = (l_tot == 0.f) ? -INFINITY : v;
                }
                if (p.carry_o_out != nullptr) p.carry_m_out[crow] = m_run > kNoKey ? m_run : -INFINITY;
            }
            if (alive) {
                const float inv_l = (l_tot == 0.f || l_tot != l_tot) ? 0.f : __frcp_rn(l_tot);
                const bool want_out = (p.out[0] != nullptr);
                // the row's home: one output buffer, or the part that owns this token (another GPU's memory when the
                // output goes straight back to the token shards of a sequence-parallel group: plain stores)
                const int opart = (p.out_rows == 0) ? 0 : min(grow / p.out_rows, kMaxParts - 1);
                const int orow_l = grow - opart * p.out_rows;
                OutT* orow = static_cast<OutT*>(p.out[opart]) + out_base + hq * p.os1 + (int64_t)orow_l * p.os2;
                for (int c = c0; c < c0 + share; c += 16) {
                    float o[16];
                    if (nb > 0 || carry_in) {
                        tmem_ld16(tmem + lane_addr + C::cO + t * D + c, o);
                        tc_wait_ld();
                    } else {
#pragma unroll
                        for (int i = 0; i < 16; ++i) o[i] = 0.f;
                    }
                    if (p.carry_o_out != nullptr && grow < Nq) {
#pragma unroll
                        for (int i = 0; i < 4; ++i)
                            *reinterpret_cast<float4*>(p.carry_o_out + crow * D + c + 4 * i) = make_float4(o[4 * i], o[4 * i + 1], o[4 * i + 2], o[4 * i + 3]);
                    }
                    if (want_out && grow < Nq) {
#pragma unroll
                        for (int i = 0; i < 2; ++i) {
                            uint4 w;
                            w.x = pack2<OutT>(o[8 * i] * inv_l, o[8 * i + 1] * inv_l);
                            w.y = pack2<OutT>(o[8 * i + 2] * inv_l, o[8 * i + 3] * inv_l);
                            w.z = pack2<OutT>(o[8 * i + 4] * inv_l, o[8 * i + 5] * inv_l);
                            w.w = pack2<OutT>(o[8 * i + 6] * inv_l, o[8 * i + 7] * inv_l);
                            *reinterpret_cast<uint4*>(orow + c + i * 8) = w;
                        }
                    }
                }
            }
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

// byte tensor [n2][n1][n0] (n0 contiguous), box [1][b1][b0]
static CUresult make_map(EncodeTiledFn fn, CUtensorMap* m, const void* base, uint64_t n0, uint64_t n1, uint64_t n2,
                         uint32_t b0, uint32_t b1, CUtensorMapSwizzle swz) {
    cuuint64_t dims[3] = {n0, n1, n2};
    cuuint64_t strides[2] = {n0, n0 * n1};
    cuuint32_t box[3] = {b0, b1, 1};
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

template <int D, bool CAUSAL, typename OutT, bool VARLEN>
static cudaError_t launch_v(const AttnArgs& a, const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv,
                            const AttnParams& p, cudaStream_t st) {
    auto kern = attn_fwd_kernel<D, CAUSAL, OutT, VARLEN>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg<D>::kSmemBytes);
    if (e != cudaSuccess) return e;
    const int grid = a.B * a.Hq * ((a.Nq_p / kBlock + 1) / 2);      // one CTA per pair of query tiles
    kern<<<grid, Cfg<D>::kThreads, Cfg<D>::kSmemBytes, st>>>(tq, tk, tv, p);
    return cudaGetLastError();
}

template <int D, bool CAUSAL, typename OutT>
static cudaError_t launch_t(const AttnArgs& a, const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv,
                            const AttnParams& p, cudaStream_t st) {
    // packed variable-length batches run their own instantiation, so that the uniform kernels carry none of it
    return a.cu_q != nullptr ? launch_v<D, CAUSAL, OutT, true>(a, tq, tk, tv, p, st)
                             : launch_v<D, CAUSAL, OutT, false>(a, tq, tk, tv, p, st);
}

cudaError_t launch_attn(const AttnArgs& a, cudaStream_t st, int* driver_rc) {
    *driver_rc = 0;
    EncodeTiledFn fn = get_encode_fn();
    if (!fn) return cudaErrorNotSupported;
    CUtensorMap tq, tk, tv;
    const uint32_t rowb = a.D / 2;
    const CUtensorMapSwizzle swz_qk = (a.D == 128) ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B;
    CUresult r = make_map(fn, &tq, a.q_codes, rowb, a.Nq_p, (uint64_t)a.B * a.Hq, rowb, kBlock, swz_qk);
    if (r == CUDA_SUCCESS) r = make_map(fn, &tk, a.k_codes, rowb, a.Nk_p, (uint64_t)a.B * a.Hkv, rowb, kBlock, swz_qk);
    if (r == CUDA_SUCCESS)
        r = make_map(fn, &tv, a.v_codes, a.Nk_p / 2, a.D, (uint64_t)a.B * a.Hkv, 64, a.D, CU_TENSOR_MAP_SWIZZLE_64B);
    if (r != CUDA_SUCCESS) {
        *driver_rc = (int)r;
        return cudaErrorInvalidValue;
    }
    AttnParams p;
    p.Hq = a.Hq; p.Hkv = a.Hkv; p.Nq = a.Nq; p.Nk = a.Nk;
    p.nqt = a.Nq_p / kBlock; p.nkb = a.Nk_p / kBlock; p.nqm = a.nqm;
    p.sm_scale_log2 = a.sm_scale * 1.4426950408889634f;
    p.sm_scale_per_head = a.sm_scale_per_head;
    p.q_sf = a.q_sf; p.k_sf = a.k_sf; p.v_sf = a.v_sf;
    p.delta = static_cast<const uint16_t*>(a.delta);
    for (int i = 0; i < kMaxParts; ++i) p.out[i] = a.out.base[i];
    p.out_rows = a.out.rows;
    p.lse = a.lse; p.qkm = a.qkm; p.sm_scale = a.sm_scale;
    p.os0 = a.os[0]; p.os1 = a.os[1]; p.os2 = a.os[2];
    p.status = a.status;
    p.prepass_status = a.prepass_status;
    p.carry_o_in = a.carry_o_in; p.carry_m_in = a.carry_m_in; p.carry_l_in = a.carry_l_in;
    p.carry_o_out = a.carry_o_out; p.carry_m_out = a.carry_m_out; p.carry_l_out = a.carry_l_out;
    p.causal_shift = a.causal_shift;
    p.cu_q = a.cu_q; p.cu_k = a.cu_k;
    if (a.is_bf16) {
        if (a.D == 128) return a.is_causal ? launch_t<128, true, __nv_bfloat16>(a, tq, tk, tv, p, st)
                                           : launch_t<128, false, __nv_bfloat16>(a, tq, tk, tv, p, st);
        return a.is_causal ? launch_t<64, true, __nv_bfloat16>(a, tq, tk, tv, p, st)
                           : launch_t<64, false, __nv_bfloat16>(a, tq, tk, tv, p, st);
    }
    if (a.D == 128) return a.is_causal ? launch_t<128, true, __half>(a, tq, tk, tv, p, st)
                                       : launch_t<128, false, __half>(a, tq, tk, tv, p, st);
    return a.is_causal ? launch_t<64, true, __half>(a, tq, tk, tv, p, st)
                       : launch_t<64, false, __half>(a, tq, tk, tv, p, st);
}

}  // namespace sage3
