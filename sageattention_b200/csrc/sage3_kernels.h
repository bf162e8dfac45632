// Host-visible launch interface between the C ABI (sage3_abi.cu) and the kernel translation units.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>

namespace sage3 {

constexpr int kBlock = 128;          // query-tile rows and keys per KV block
constexpr int kRowsPerChunk = 512;   // rows per partial column sum (fixes the summation order)
constexpr int kMaxParts = 8;         // a tensor's tokens may be split over this many buffers (one per GPU of a node)

// A tensor whose token dimension is split into equal parts living in different buffers (e.g. the token shards of the
// ranks of a sequence-parallel group, mapped into this process): part p holds tokens [p * rows, (p + 1) * rows).
// rows == 0: one buffer, base[0].
struct PartsPtr {
    void* base[kMaxParts];
    int rows;
};

struct PrepassArgs {
    PartsPtr q, k, v;
    int64_t qs[3], ks[3], vs[3];   // element strides for (b, h, n)
    int B, Hq, Hkv, Nq, Nk, D, Nq_p, Nk_p, nqm;
    int per_block_mean, is_bf16;
    int km_given;                  // the K mean is already in `km` (computed elsewhere): skip its two kernels
    int kchunks_k, kchunks_q;
    float* kpart;
    void *km, *qm, *delta;
    uint8_t *q_codes, *q_sf, *k_codes, *k_sf, *v_codes, *v_sf;
    float* qkm;                    // fp32 [B][Hq][Nq_p]: q . km per query row
    int* status;                   // device status words (bounded waits report here)
    int want_qkm;                  // q . km per query row is wanted (the LSE output needs it)
    int* clear;                    // words the first kernel zeroes: status words, the attention kernel's work counter and flags, `nonfinite`
    int n_clear;
    int* nonfinite;                // per (batch, kv head): set when a delta_s value is not finite; nullptr: nobody asks (see PackRule)
    // packed variable-length sequences (both nullptr: every batch entry has Nq / Nk tokens): device int32 [B + 1], entry b
    // owns rows cu[b] .. cu[b + 1] of the packed tensor; Nq / Nk are then the maximum lengths, stride 0 is unused
    const int *cu_q, *cu_k;
};

struct AttnArgs {
    int B, Hq, Hkv, Nq, Nk, D, Nq_p, Nk_p, nqm;
    int is_causal, is_bf16;
    float sm_scale;                 // already resolved (> 0)
    const float* sm_scale_per_head; // device [Hq] or nullptr
    const void* delta;              // dtype [B][Hq][nqm][Nk_p]
    const uint8_t *q_codes, *q_sf, *k_codes, *k_sf, *v_codes, *v_sf;
    PartsPtr out;
    int64_t os[3];
    float* lse;                     // optional fp32 [B][Hq][Nq]; nullptr if not wanted
    const float* qkm;               // fp32 [B][Hq][Nq_p] from the pre-pass
    int* status;                    // the attention kernel's status word
    int* unit_counter;              // work counter, zeroed before the launch
    // accumulator state carried between calls (all nullptr: none); fp32, unnormalized O [B][Hq][Nq][D], m [B][Hq][Nq], l [B][Hq][Nq][2]
    const float *carry_o_in, *carry_m_in, *carry_l_in;
    float *carry_o_out, *carry_m_out, *carry_l_out;
    int causal_shift;               // key j visible to query i iff j <= i + causal_shift (Nk - Nq unless the caller offsets it)
    const int* prepass_status;      // the pre-pass's status word (non-zero: the workspace is incomplete, do nothing)
    const int* nonfinite;           // per (batch, kv head), from the pre-pass: delta_s holds values that are not finite
    const int *cu_q, *cu_k;         // packed variable-length sequences, as in PrepassArgs (nullptr: uniform lengths)
    // Last rounds of units dealt out by key blocks (see SplitPlan): flags, zeroed before the launch, and scratch.  nullptr: not possible for these sizes.
    int* split_flags;
    float* split_state;
};

// The accumulator of a query tile whose keys two CTAs of the attention kernel share: fp32 O [D / 4][128 rows][4], row sums [128][2], maxima [128] per slot.
constexpr int kSplitSlots = 160;      // CTAs (one per SM)
constexpr int kSplitMinBlocks = 16;   // key blocks of a call, below which no tile is shared
constexpr size_t split_state_floats(size_t D) { return 128 * D + 128 * 3; }

// Few query rows and several heads per kv head (token generation): as many heads as fit share a 128-row tile, eight at most (the
// operand that adds delta_s has eight rows); uniform lengths and no carried state only (`plain`).  Mode 2, where a warp takes a
// quarter of the keys for all rows, when the rows of these heads (of one head, too) fit one warp: it would need more tiles otherwise.
struct PackRule {
    int heads = 1, mode = 0;       // query heads per tile; kernel: 0 pairs of tiles, 1 packed, 2 packed with at most 32 rows
    PackRule(int Nq, int group, bool plain) {
        if (!plain) return;
        const int most = group < 8 ? group : 8;
        if (Nq <= 64) heads = 128 / Nq < most ? 128 / Nq : most;
        mode = Nq * most <= 32 ? 2 : heads > 1 ? 1 : 0;
    }
};

// Device the calling thread has current, its SM count and whether it is compute capability 10.0 (looked up once per device).
struct DeviceInfo { int sms; bool ok; };
cudaError_t current_device(int* dev, DeviceInfo* info);

// Result of a runtime call, an error taken off the thread's record: the caller gets it as a return code, and whoever asks the runtime
// next must not find it.
inline cudaError_t checked(cudaError_t e) {
    if (e != cudaSuccess) (void)cudaGetLastError();
    return e;
}

// Dynamic shared memory of a kernel beyond 48 KB: set once per kernel and device, which every kernel remembers for itself (the call into
// the runtime would come on top of every launch).
template <auto Kernel>
cudaError_t allow_smem(int bytes) {
    static std::atomic<uint64_t> devices{0};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const uint64_t bit = dev < 64 ? 1ull << dev : 0;
    if (devices.load(std::memory_order_acquire) & bit) return cudaSuccess;
    e = checked(cudaFuncSetAttribute(Kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
    if (e == cudaSuccess) devices.fetch_or(bit, std::memory_order_release);
    return e;
}

// Launch, with its result.  `early`: it may begin (up to its griddepcontrol.wait) while the kernel before it in the stream is still running.
template <typename... P, typename... A>
cudaError_t launch(bool early, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A... args) {
    cudaLaunchAttribute attr = {};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &attr;
    cfg.numAttrs = early ? 1 : 0;
    return checked(cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...));
}

// Encodes a tensor map over a byte tensor [n2][n1][n0] (n0 contiguous) with box [1][b1][b0]; swizzle: 0 none, 1 32 B, 2 64 B,
// 3 128 B.  Returns 0, or the driver's error code (-1: the driver entry point could not be resolved).
int encode_tiled_bytes(void* map64, const void* base, uint64_t n0, uint64_t n1, uint64_t n2, uint32_t b0, uint32_t b1, int swizzle);

cudaError_t launch_prepass(const PrepassArgs& a, cudaStream_t st);
// returns cudaSuccess, or an error; `driver_rc` receives a CUresult when tensor-map encoding failed
cudaError_t launch_attn(const AttnArgs& a, cudaStream_t st, int* driver_rc);

}  // namespace sage3
