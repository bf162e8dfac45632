// Pre-pass kernels: K smoothing, Q smoothing, delta_s = qm . k'^T, and NVFP4 quantization of Q, K and
// V-transposed into the layouts the attention kernel consumes.  HBM-bound; 128-bit loads, staged and
// coalesced stores.
//
// Math follows (paths inside the reference project, sageattention3_blackwell/sageattn3/...):
//   api.py:84            k' = k - mean_N(k)                 (mean: fp32 sum, rounded to the input type)
//   api.py:26-72, 86-90  q' = q - mean of each 128-row block (16-bit additions in the Triton kernel's order) or of all padded rows
//   api.py:91            delta_s = qm . k'^T, rounded to the input type (tcgen05 16-bit MMA, accumulator in TMEM)
//   quantization/fp4_quantization_4d.cu:185-225   SF = e4m3(amax / 6), code = e2m1(x * (1 / SF))
//   quantization/fp4_quantization_4d.cu:300-349   V: microblocks are 16 consecutive tokens of one channel
// Quotients and reciprocals are those of IEEE arithmetic (see micro_scale), so the result can be checked bit for bit.
#include <mutex>
#include <type_traits>

#include "../../include/sage3_b200.h"
#include <cuda.h>

#include "sage3_common.cuh"
#include "sage3_kernels.h"

namespace sage3 {

// Division of block indices by a run-time constant: q = (mulhi(n, m) + n) >> s for 0 <= n < 2^31 (Granlund and Montgomery 1994);
// a plain integer division costs every thread of a block some 25 instructions.
struct FastDiv {
    uint32_t d, m, s;
    FastDiv() = default;
    explicit FastDiv(int div) : d((uint32_t)div), s(0) {
        while ((1ull << s) < d) ++s;
        m = (uint32_t)((((1ull << s) - d) << 32) / d + 1);
    }
    __device__ __forceinline__ int div(int n) const { return (int)((__umulhi((uint32_t)n, m) + (uint32_t)n) >> s); }
    __device__ __forceinline__ int divmod(int n, int& rem) const {
        const int q = div(n);
        rem = n - q * (int)d;
        return q;
    }
};

template <typename T> struct Num;
template <> struct Num<__nv_bfloat16> {
    using T2 = __nv_bfloat162;
    static constexpr bool kIsBf16 = true;
    static __device__ __forceinline__ float to_f(__nv_bfloat16 x) { return __bfloat162float(x); }
    static __device__ __forceinline__ __nv_bfloat16 from_f(float x) { return __float2bfloat16_rn(x); }
    static __device__ __forceinline__ float2 to_f2(uint32_t w) {
        return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u));
    }
    static __device__ __forceinline__ uint32_t pack2(float lo, float hi) {     // two values rounded to T, lo in bits 0..15
        const __nv_bfloat162 pr = __floats2bfloat162_rn(lo, hi);
        return *reinterpret_cast<const uint32_t*>(&pr);
    }
    // packed pairs: each result rounded once to T, which for sums and differences of two T values equals fp32
    // arithmetic followed by a rounding to T (the fp32 result is exact unless the smaller operand lies below a
    // quarter ulp of the larger, where both roundings return the larger operand)
    static __device__ __forceinline__ uint32_t sub2(uint32_t a, uint32_t b) {
        const __nv_bfloat162 r = __hsub2(*reinterpret_cast<const __nv_bfloat162*>(&a), *reinterpret_cast<const __nv_bfloat162*>(&b));
        return *reinterpret_cast<const uint32_t*>(&r);
    }
    static __device__ __forceinline__ uint32_t add2(uint32_t a, uint32_t b) {
        const __nv_bfloat162 r = __hadd2(*reinterpret_cast<const __nv_bfloat162*>(&a), *reinterpret_cast<const __nv_bfloat162*>(&b));
        return *reinterpret_cast<const uint32_t*>(&r);
    }
    static __device__ __forceinline__ uint32_t absmax2(uint32_t m, uint32_t a) {   // max(m, |a|) per half
        const __nv_bfloat162 r = __hmax2(*reinterpret_cast<const __nv_bfloat162*>(&m), __habs2(*reinterpret_cast<const __nv_bfloat162*>(&a)));
        return *reinterpret_cast<const uint32_t*>(&r);
    }
    static __device__ __forceinline__ uint32_t zero_fma2(uint32_t a, uint32_t z) {   // 0 a + z: stays 0 while every a is finite, then NaN
        const __nv_bfloat162 r = __hfma2(*reinterpret_cast<const __nv_bfloat162*>(&a), __floats2bfloat162_rn(0.f, 0.f), *reinterpret_cast<const __nv_bfloat162*>(&z));
        return *reinterpret_cast<const uint32_t*>(&r);
    }
};
template <> struct Num<__half> {
    using T2 = __half2;
    static constexpr bool kIsBf16 = false;
    static __device__ __forceinline__ float to_f(__half x) { return __half2float(x); }
    static __device__ __forceinline__ __half from_f(float x) { return __float2half_rn(x); }
    static __device__ __forceinline__ float2 to_f2(uint32_t w) {
        return __half22float2(*reinterpret_cast<const __half2*>(&w));
    }
    static __device__ __forceinline__ uint32_t pack2(float lo, float hi) {
        const __half2 pr = __floats2half2_rn(lo, hi);
        return *reinterpret_cast<const uint32_t*>(&pr);
    }
    static __device__ __forceinline__ uint32_t sub2(uint32_t a, uint32_t b) {
        const __half2 r = __hsub2(*reinterpret_cast<const __half2*>(&a), *reinterpret_cast<const __half2*>(&b));
        return *reinterpret_cast<const uint32_t*>(&r);
    }
    static __device__ __forceinline__ uint32_t add2(uint32_t a, uint32_t b) {
        const __half2 r = __hadd2(*reinterpret_cast<const __half2*>(&a), *reinterpret_cast<const __half2*>(&b));
        return *reinterpret_cast<const uint32_t*>(&r);
    }
    static __device__ __forceinline__ uint32_t absmax2(uint32_t m, uint32_t a) {
        const __half2 r = __hmax2(*reinterpret_cast<const __half2*>(&m), __habs2(*reinterpret_cast<const __half2*>(&a)));
        return *reinterpret_cast<const uint32_t*>(&r);
    }
    static __device__ __forceinline__ uint32_t zero_fma2(uint32_t a, uint32_t z) {
        const __half2 r = __hfma2(*reinterpret_cast<const __half2*>(&a), __floats2half2_rn(0.f, 0.f), *reinterpret_cast<const __half2*>(&z));
        return *reinterpret_cast<const uint32_t*>(&r);
    }
};

// Rows of an input tensor that may be split over several buffers along the token dimension.
template <typename T>
struct Src {
    const T* part[kMaxParts];
    int rows;                       // tokens per part; 0 = everything in part[0]
    const int* cu;                  // packed variable-length sequences: batch entry b owns rows cu[b] .. cu[b + 1]; nullptr: uniform
    // Element offset of (batch entry b, head h); with `cu` also replaces N (the maximum length) by the entry's own length.
    __device__ __forceinline__ int64_t base(int b, int h, int64_t sb, int64_t sh, int64_t sn, int& N) const {
        if (cu != nullptr) {
            const int r0 = cu[b];
            N = min(max(cu[b + 1] - r0, 0), N);
            return (int64_t)r0 * sn + h * sh;
        }
        return b * sb + h * sh;
    }
    // Visits rows r0, r0 + step, ... (n of them): f(i, pointer to the row).  One buffer: the pointer is stepped.
    template <int n, typename F>
    __device__ __forceinline__ void rows_each(int64_t bh_off, int r0, int step, int64_t sn, F f) const {
        if (rows == 0) {
            const T* p = part[0] + bh_off + (int64_t)r0 * sn;
            const int64_t d = (int64_t)step * sn;
#pragma unroll
            for (int i = 0; i < n; ++i, p += d) f(i, p);
        } else {
#pragma unroll
            for (int i = 0; i < n; ++i) f(i, row(bh_off, r0 + i * step, sn));
        }
    }
    __device__ __forceinline__ const T* row(int64_t bh_off, int r, int64_t sn) const {
        if (rows == 0) return part[0] + bh_off + (int64_t)r * sn;
        const int pi = min(r / rows, kMaxParts - 1);
        return part[pi] + bh_off + (int64_t)(r - pi * rows) * sn;
    }
};
template <typename T>
static Src<T> make_src(const PartsPtr& a, const int* cu = nullptr) {
    Src<T> s;
    for (int i = 0; i < kMaxParts; ++i) s.part[i] = static_cast<const T*>(a.base[i]);
    s.rows = a.rows;
    s.cu = cu;
    return s;
}

// 16 elements stay packed in two 128-bit registers until they are needed (keeps the register count, and with it
// the number of resident CTAs, where an HBM-bound kernel needs it)
template <typename T>
__device__ __forceinline__ void load16_packed(const T* p, bool valid, uint4& a, uint4& b) {
    a = make_uint4(0, 0, 0, 0);
    b = a;
    if (valid) {
        a = __ldg(reinterpret_cast<const uint4*>(p));
        b = __ldg(reinterpret_cast<const uint4*>(p) + 1);
    }
}
template <typename T>
__device__ __forceinline__ void unpack16(const uint4& a, const uint4& b, float* f) {   // 16 elements -> fp32
    const uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        float2 v = Num<T>::to_f2(w[i]);
        f[2 * i] = v.x;
        f[2 * i + 1] = v.y;
    }
}

// Scale byte of a microblock with maximum magnitude amax, SF = e4m3(amax / 6), and the factor 1 / SF its values are scaled with
// (0 when SF is 0).  Both without the division and reciprocal routines (a quarter of the stage kernel's instructions):
//   amax * RN(1/6) and RN(amax / 6) round to the same E4M3 value for every 16-bit amax.  A quotient on a rounding boundary of E4M3 (a
//   significand of at most 5 bits) means amax = 6 x boundary, and RN(1/6) = 1/6 (1 + 2^-25.0) is close enough for the product to
//   round to the boundary itself (half an ulp is more than 2^-24.96 of it); any other quotient is at least 2^-14 away from one.
//   rcp.approx of the 126 positive E4M3 values is their correctly rounded reciprocal (checked for each of them).
__device__ __forceinline__ float micro_scale(float amax, uint32_t& sf_byte) {
    sf_byte = cvt_e4m3x2(__fmul_rn(amax, 1.0f / 6.0f), 0.f) & 0xffu;
    float inv;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(inv) : "f"(e4m3_to_float(sf_byte)));
    return sf_byte == 0u ? 0.f : inv;
}

// One NVFP4 microblock, eight packed words of the input type (16 values) -> 8 bytes of codes + scale byte: the maximum magnitude is found on the packed pairs
// (exact, as fp4_quantization_4d.cu:186-196 does), the scaling runs in fp32.
template <typename T>
__device__ __forceinline__ void quant16_packed(const uint32_t* w, uint32_t& lo, uint32_t& hi, uint32_t& sf_byte) {
    uint32_t m = Num<T>::absmax2(0u, w[0]);
#pragma unroll
    for (int i = 1; i < 8; ++i) m = Num<T>::absmax2(m, w[i]);
    const float2 mm = Num<T>::to_f2(m);
    const float amax = fmaxf(mm.x, mm.y);
    const float inv = micro_scale(amax, sf_byte);
    const uint64_t inv2 = pack2f(inv, inv);
    float y[16];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const float2 v = Num<T>::to_f2(w[i]);
        unpack2f(mul2(pack2f(v.x, v.y), inv2), y[2 * i], y[2 * i + 1]);
    }
    lo = cvt_e2m1x8(y[0], y[1], y[2], y[3], y[4], y[5], y[6], y[7]);
    hi = cvt_e2m1x8(y[8], y[9], y[10], y[11], y[12], y[13], y[14], y[15]);
}

// ------------------------------------------------------------------------------------------------
// column sums over tokens: partial sums per chunk of kRowsPerChunk rows, then a fixed-order finalize
// (deterministic: no atomics, the summation order depends on N only)
// ------------------------------------------------------------------------------------------------
template <typename T, int D>
__device__ __forceinline__ void colsum_chunk(const Src<T>& x, int64_t sb, int64_t sh, int64_t sn, FastDiv H, int N, float* __restrict__ part,
                                             int chunks, int chunk, int bh, float* red) {   // red: shared, [RPP][D + 1]
    constexpr int TPR = D / 8;           // threads per row (8 elements = 16 bytes each)
    constexpr int RPP = 256 / TPR;       // rows per pass
    int h;
    const int b = H.divmod(bh, h);
    const int64_t bh_off = x.base(b, h, sb, sh, sn, N);
    const int c8 = threadIdx.x % TPR, rl = threadIdx.x / TPR;
    const int r0 = chunk * kRowsPerChunk;
    const int r1 = min(N, r0 + kRowsPerChunk);
    float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    // Eight rows in flight per thread (a load per addition made the two CTAs of a 1 024-token head take 19 us); the additions
    // keep their order.
    constexpr int U = D == 64 ? 4 : 8;
    for (int r = r0 + rl; r < r1; r += U * RPP) {
        uint4 a[U];
        x.template rows_each<U>(bh_off, r, RPP, sn, [&](int u, const T* p) {
            a[u] = make_uint4(0, 0, 0, 0);
            if (r + u * RPP < r1) a[u] = __ldg(reinterpret_cast<const uint4*>(p + c8 * 8));
        });
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const uint32_t w[4] = {a[u].x, a[u].y, a[u].z, a[u].w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                float2 v = Num<T>::to_f2(w[i]);
                acc[2 * i] += v.x;
                acc[2 * i + 1] += v.y;
            }
        }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) red[rl * (D + 1) + c8 * 8 + i] = acc[i];
    __syncthreads();
    if (threadIdx.x < D) {
        float s = 0.f;
#pragma unroll
        for (int i = 0; i < RPP; ++i) s += red[i * (D + 1) + threadIdx.x];
        part[((int64_t)bh * chunks + chunk) * D + threadIdx.x] = s;
    }
}

// One sum of a column's partial sums, in the order of the chunks.
__device__ __forceinline__ float sum_chunks(const float* __restrict__ part, int chunks, int D) {
    float s = 0.f;
    for (int c = 0; c < chunks; c += 16) {
        float v[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i] = c + i < chunks ? load_written(part + (int64_t)(c + i) * D) : 0.f;
#pragma unroll
        for (int i = 0; i < 16; ++i) s += v[i];       // (+ 0 beyond the last chunk: no change)
    }
    return s;
}

template <typename T, int D>
__global__ void __launch_bounds__(256) colsum_partial_kernel(const __grid_constant__ Src<T> x, int64_t sb, int64_t sh, int64_t sn, FastDiv H, int N,
                                                             float* __restrict__ part, int chunks) {
    __shared__ float red[(2048 / D) * (D + 1)];
    colsum_chunk<T, D>(x, sb, sh, sn, H, N, part, chunks, blockIdx.x, blockIdx.y, red);
}

template <typename T, int D>
__global__ void colmean_finalize_kernel(const float* __restrict__ part, int chunks, float inv_count,
                                        T* __restrict__ mean, const int* __restrict__ cu, int H, int pad_to_block) {
    const int bh = blockIdx.x, d = threadIdx.x;
    if (cu != nullptr) {
        // the entry's own token count (rounded up to whole 128-row blocks where the mean is over the padded rows);
        // chunks beyond it hold zeros, so the sum is the one a call on this entry alone would form
        int n = max(cu[bh / H + 1] - cu[bh / H], 0);
        if (pad_to_block) n = (n + kBlock - 1) / kBlock * kBlock;
        inv_count = n > 0 ? 1.0f / (float)n : 0.f;
    }
    const float s = sum_chunks(part + (int64_t)bh * chunks * D + d, chunks, D);
    mean[(int64_t)bh * D + d] = Num<T>::from_f(s * inv_count);
}

// ------------------------------------------------------------------------------------------------
// Q: smooth + quantize one 128-row tile per CTA
// ------------------------------------------------------------------------------------------------
enum { kModeQBlockMean = 0, kModeQGlobalMean = 1 };

// Partial column sums for the blocks that form the means they need themselves (nullptr: the means are in memory).
struct MeanParts {
    const float *k, *q;                // [B*Hkv][chunks_k][D], [B*H][chunks_q][D]
    int chunks_k, chunks_q, Nk;
    const int* cu_k;
    bool wait;                         // the sums come from the launch before this one (programmatic dependent launch)
};

// Microblock column and (first) row of a thread in a tile of 128 rows: eight neighbouring lanes have four columns of two rows.  With the 16-byte chunks of odd
// rows in swapped pairs (or in the swizzle of an MMA operand) these eight lie on different banks.
template <int D> __device__ __forceinline__ int micro_col(int lane) { return (lane & 3) | (D == 128 ? (lane >> 1) & 4 : 0); }
template <int D> __device__ __forceinline__ int micro_row(int warp, int lane) {
    return D == 128 ? warp * 4 + (((lane >> 2) & 1) | ((lane >> 3) & 2)) : warp * 8 + (lane >> 2);
}

// Scale bytes of a tile, from threads that hold those of rows rl, rl + RPP, ... in bytes 0, 1, ...: four neighbouring lanes have the four columns of a word of the
// atom, and store the word of one microblock each.
template <int D>
__device__ __forceinline__ void store_scales(uint8_t* tile, uint32_t sf, int c, int rl, int lane) {
    constexpr int CH = D / 16, RPP = 256 / CH, ITEMS = kBlock / RPP;
    const int l = lane & 3;
    const uint32_t y = __shfl_xor_sync(0xffffffffu, sf, 1);
    const uint32_t v = __byte_perm(sf, y, l & 1 ? 0x3715 : 0x6240);
    const uint32_t z = __shfl_xor_sync(0xffffffffu, v, 2);
    const uint32_t word = __byte_perm(v, z, l & 2 ? 0x3276 : 0x5410);
    if (ITEMS == 4 || l < 2) *reinterpret_cast<uint32_t*>(tile + (c >> 2) * 512 + sf_atom_offset(rl + RPP * l, 0)) = word;
}

template <typename T, int D, int MODE>
__device__ __forceinline__ void quant_q_tile(
    const Src<T>& x, int64_t sb, int64_t sh, int64_t sn, FastDiv H, int N, int Np,
    const T* __restrict__ mean_in,     // one mean per head: qm [B*H][D]; unused for block mean
    T* __restrict__ qm_out,            // block mean: [B*H][Np/128][D]
    uint8_t* __restrict__ codes,       // [B*H][Np][D/2]
    uint8_t* __restrict__ sfs,         // [B*H][Np/128][D/64][512]
    const T* __restrict__ km,          // K means [B*Hkv][D]
    int group,                         // query heads per kv head
    float* __restrict__ qkm,           // [B*H][Np]: x . km per row (the score part that K smoothing removes); nullptr: not wanted
    const MeanParts& mp,
    int tile, int bh, uint8_t* smem_raw) {
    constexpr int CH = D / 16;            // microblocks per row
    constexpr int RPP = 256 / CH;         // rows per pass
    constexpr int ITEMS = kBlock / RPP;   // microblocks per thread

    int h;
    const int b = H.divmod(bh, h);
    const int t = threadIdx.x, lane = t & 31;
    const int c = micro_col<D>(lane), rl = micro_row<D>(t >> 5, lane);
    const int64_t bh_off = x.base(b, h, sb, sh, sn, N);
    const int row0 = tile * kBlock;
    if (row0 >= N && row0 > 0) return;    // a tile beyond this entry's padded length (variable-length batches only)

    T* s_mean = reinterpret_cast<T*>(smem_raw);                                // [D]
    uint8_t* s_more = smem_raw + D * 4;                                        // block mean only: staged tile, chain sums

    uint4 raw[ITEMS][2];
    x.template rows_each<ITEMS>(bh_off, row0 + rl, RPP, sn, [&](int i, const T* p) {
        load16_packed<T>(p + c * 16, row0 + rl + RPP * i < N, raw[i][0], raw[i][1]);
    });

    if (mp.wait) pdl_wait();               // the rows above are inputs; the means are not
    // x . km of every row: 16 products per thread, then a sum over the CH neighbouring lanes that share the row
    if (qkm != nullptr) {
        const int bhk = b * ((int)H.d / group) + h / group;
        float kf[16];
        if (mp.k != nullptr) {
            if (t < D) {
                const int nk = mp.cu_k != nullptr ? min(max(mp.cu_k[b + 1] - mp.cu_k[b], 0), mp.Nk) : mp.Nk;
                const float m = sum_chunks(mp.k + (int64_t)bhk * mp.chunks_k * D + t, mp.chunks_k, D) * (nk > 0 ? 1.0f / (float)nk : 0.f);
                s_mean[t] = Num<T>::from_f(m);
            }
            __syncthreads();
            unpack16<T>(reinterpret_cast<const uint4*>(s_mean)[2 * c], reinterpret_cast<const uint4*>(s_mean)[2 * c + 1], kf);
            __syncthreads();               // s_mean takes the Q mean next
        } else {
            const uint4* km4 = reinterpret_cast<const uint4*>(km + (int64_t)bhk * D + c * 16);
            const uint4 k0 = load_written(km4), k1 = load_written(km4 + 1);
            unpack16<T>(k0, k1, kf);
        }
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) {
            float f[16];
            unpack16<T>(raw[i][0], raw[i][1], f);
            float dot = 0.f;
#pragma unroll
            for (int j = 0; j < 16; ++j) dot = fmaf(f[j], kf[j], dot);
#pragma unroll
            for (int off = 1; off < CH; off <<= 1) dot += __shfl_xor_sync(0xffffffffu, dot, off == 4 ? 8 : off);      // (see micro_col)
            if (c == 0) qkm[(int64_t)bh * Np + row0 + rl + RPP * i] = dot;
        }
    }

    if (MODE == kModeQBlockMean) {
        // Block mean exactly as the reference's Triton kernel forms it (api.py:45-48): a sum of 16-bit values whose every
        // addition rounds to the input type, in the order of that kernel's 4-warp blocked layout:
        //   chain (w, l): rows rep * R + w * L + l, rep = 0 .. 128 / R - 1, added in order of rep
        //                 (L = 32 / (D / 8) rows of a warp, R = 4 L rows per repetition),
        //   then a butterfly over l inside each warp (distance L/2, L/4, ...), then (w0 + w2) + (w1 + w3).
        // Rows beyond N are zero and take part (padding precedes the mean).  The tile is staged in shared memory so
        // that one thread can walk one chain for four columns.
        constexpr int L = 32 / (D / 8), R = 4 * L, REPS = kBlock / R;
        static_assert(R * (D / 4) == 256, "one thread per (chain, group of four columns)");
        T* s_tile = reinterpret_cast<T*>(s_more);                              // [128][D]
        constexpr int PITCH = D + 8;                                           // (the four lanes' rows on different banks)
        T* s_part = s_tile + kBlock * D;                                       // [R][PITCH]
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) {
            uint8_t* dst = reinterpret_cast<uint8_t*>(s_tile + (rl + RPP * i) * D);
            *reinterpret_cast<uint4*>(dst + ((2 * c ^ (rl & 1)) << 4)) = raw[i][0];
            *reinterpret_cast<uint4*>(dst + (((2 * c ^ (rl & 1)) ^ 1) << 4)) = raw[i][1];
        }
        __syncthreads();
        {
            const int chain = t / (D / 4), c4 = (t % (D / 4)) * 4;
            static_assert(R % 2 == 0, "the rows of a chain are all odd or all even");
            const T* place = s_tile + chain * D + (((c4 >> 3) ^ (chain & 1)) << 3) + (c4 & 4);
            uint2 acc = *reinterpret_cast<const uint2*>(place);
#pragma unroll
            for (int rep = 1; rep < REPS; ++rep) {
                const uint2 w1 = *reinterpret_cast<const uint2*>(place + rep * R * D);
                acc.x = Num<T>::add2(acc.x, w1.x);
                acc.y = Num<T>::add2(acc.y, w1.y);
            }
            *reinterpret_cast<uint2*>(s_part + chain * PITCH + c4) = acc;
        }
        __syncthreads();
        // Four lanes per pair of columns, one for each w; packed additions round as the order above asks.  The means stay packed, here and in
        // the K kernel: every thread takes its 16 with two 128-bit loads.  (One thread per column with fp32 additions and roundings, and
        // means as floats that every thread packs again: 8 x 32 heads x 1 token against 8 192 keys 141.0 -> 137.1 us per call, packed prompts
        // of 256 to 2 048 tokens 621 -> 610, a 3 001-token prompt 92.2 -> 90.7, 1 000 queries x 9 192 keys 141.5 -> 140.3.)
        if (t < 2 * D) {
            const int w = (t >> 3) & 3, c2 = (t >> 5) * 8 + (t & 7);
            uint32_t v[L];
#pragma unroll
            for (int l = 0; l < L; ++l) v[l] = *reinterpret_cast<const uint32_t*>(s_part + (w * L + l) * PITCH + 2 * c2);
#pragma unroll
            for (int n = L / 2; n > 0; n >>= 1)
#pragma unroll
                for (int l = 0; l < n; ++l) v[l] = Num<T>::add2(v[l], v[l + n]);
            uint32_t sum = Num<T>::add2(v[0], __shfl_xor_sync(0xffffffffu, v[0], 16));
            sum = Num<T>::add2(sum, __shfl_xor_sync(0xffffffffu, sum, 8));
            if (w == 0) {
                const float2 f = Num<T>::to_f2(sum);
                const uint32_t m = Num<T>::pack2(f.x * (1.0f / kBlock), f.y * (1.0f / kBlock));
                reinterpret_cast<uint32_t*>(s_mean)[c2] = m;
                reinterpret_cast<uint32_t*>(qm_out + ((int64_t)bh * (Np / kBlock) + tile) * D)[c2] = m;
            }
        }
    } else {
        if (t < D) {
            if (mp.q != nullptr) {         // mean over the rows padded to whole blocks (api.py:88-90)
                const int np = (N + kBlock - 1) / kBlock * kBlock;
                const T m = Num<T>::from_f(sum_chunks(mp.q + (int64_t)bh * mp.chunks_q * D + t, mp.chunks_q, D) * (np > 0 ? 1.0f / (float)np : 0.f));
                if (tile == 0) qm_out[(int64_t)bh * D + t] = m;
                s_mean[t] = m;
            } else {
                s_mean[t] = mean_in[(int64_t)bh * D + t];
            }
        }
    }
    __syncthreads();

    uint32_t mu2[8];       // the 16 means of this thread's columns, packed (they are values of the input type)
    *reinterpret_cast<uint4*>(mu2) = reinterpret_cast<const uint4*>(s_mean)[2 * c];
    *reinterpret_cast<uint4*>(mu2 + 4) = reinterpret_cast<const uint4*>(s_mean)[2 * c + 1];

    uint8_t* code = codes + ((int64_t)bh * Np + row0 + rl) * (D / 2) + c * 8;
    uint32_t sf = 0;
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
        // rows beyond N hold 0 - mean (Q is padded before smoothing); they are never read back
        const uint32_t x2[8] = {raw[i][0].x, raw[i][0].y, raw[i][0].z, raw[i][0].w, raw[i][1].x, raw[i][1].y, raw[i][1].z, raw[i][1].w};
        uint32_t d2[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) d2[j] = Num<T>::sub2(x2[j], mu2[j]);
        uint32_t lo, hi, sfb;
        quant16_packed<T>(d2, lo, hi, sfb);
        *reinterpret_cast<uint2*>(code + i * RPP * (D / 2)) = make_uint2(lo, hi);
        sf |= sfb << (8 * i);
    }
    store_scales<D>(sfs + ((int64_t)bh * (Np / kBlock) + tile) * (D / 64) * 512, sf, c, rl, lane);
}

// ------------------------------------------------------------------------------------------------
// K: smooth + quantize one 128-key tile per CTA, and its delta_s columns on the tensor core:
// delta_s[qb][key] = sum_d qm[qb][d] * k'[key][d] as 128 x 128 x D tcgen05 MMAs (16-bit operands from shared
// memory in the 128-byte-swizzled K-major layout, fp32 accumulator in tensor memory), one per 128 query blocks, counted
// through all query heads of the kv head (their means follow one another): four query heads of one block each took four
// rounds of copy, MMA and store, 150 us for 4 096 key tiles, and take one now, 68 us.
// The query-block means arrive through TMA (a tensor map over qm) and the delta_s tiles leave through TMA (a tensor
// map over delta), so the threads' load / store instructions carry only the K rows, the codes and the staging of
// the converted accumulator.
// ------------------------------------------------------------------------------------------------
// AROWS = 64: up to 64 query blocks (the A tile then has 64 rows, the MMA's other 64 read what lies behind it, for accumulator rows nobody looks at; four blocks
// per SM) where few tiles come to an SM, see launch_prepass_t.  Up to 64 query blocks are otherwise quant_k_delta_run_kernel's.
// FLAG: notes whether a value of delta_s is not finite, for calls whose heads share a tile in the attention kernel.
template <typename T, int D, int AROWS, bool FLAG>
__global__ void __launch_bounds__(256, AROWS == 128 ? 3 : 4) quant_k_delta_kernel(
    const __grid_constant__ Src<T> x, int64_t sb, int64_t sh, int64_t sn, FastDiv H, int N, int Np,
    T* __restrict__ km,                // [B*H][D]
    const float* __restrict__ part,    // partial column sums to form the mean from ([B*H][chunks][D]), or nullptr: `km` holds it
    int chunks,
    uint8_t* __restrict__ codes,       // [B*H][Np][D/2]
    uint8_t* __restrict__ sfs,         // [B*H][Np/128][D/64][512]
    int rows,                          // query blocks of all query heads of a kv head
    int* __restrict__ status,
    int* __restrict__ nonfinite,       // FLAG: [B*H], set when a delta_s value is not finite
    const __grid_constant__ CUtensorMap tm_qm,       // bytes [B*H][rows][2 D], box AROWS rows x 128 bytes, 128-byte swizzle
    const __grid_constant__ CUtensorMap tm_delta) {  // bytes [B*H][rows][2 Np], box 32 rows x 128 bytes, 128-byte swizzle
    constexpr int CH = D / 16;            // microblocks per row
    constexpr int RPP = 256 / CH;         // rows per pass
    constexpr int ITEMS = kBlock / RPP;   // microblocks per thread
    constexpr int SUB = D / 64;           // 64-element (128-byte) sub-tiles along K
    constexpr uint32_t kTmemCols = 128;
    constexpr bool kBf16 = sizeof(T) == 2 && Num<T>::kIsBf16;

    const int tile = blockIdx.x, bh = blockIdx.y;
    int h;
    const int b = H.divmod(bh, h);
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    const int c = t % CH, rl = t / CH;
    const int64_t bh_off = x.base(b, h, sb, sh, sn, N);
    const int row0 = tile * kBlock;
    if (row0 >= N && row0 > 0) return;    // a tile beyond this entry's padded length (variable-length batches only)

    extern __shared__ uint8_t smem_dyn[];
    const uint32_t sbase = (smem_u32(smem_dyn) + 1023u) & ~1023u;
    uint8_t* sgen = smem_dyn + (sbase - smem_u32(smem_dyn));
    // [A tile: qm chunk | B tile: k'] as SUB sub-tiles of (A: AROWS) 128 rows x 128 bytes each (in this order: the MMA reads 128 rows
    // from the start of every A sub-tile, which has to stay inside the block's shared memory), then small things, then (where the
    // A tile is too small for it, or stays) the staging tile of the epilogue: 32 rows x 128 bytes per warp that has rows
    constexpr int kARows = AROWS, kASub = kARows * 128;
    constexpr int oA = 0, oB = SUB * kASub, oMean = oB + SUB * 16384, oSf = oMean + D * 4, oBar = oSf + SUB * 512;
    static_assert(oA + (SUB - 1) * kASub + 16384 <= oMean, "the MMA's 128 A rows stay inside the tiles");
    constexpr int oStg = D == 128 ? oA : ((oBar + 64 + 1023) / 1024) * 1024;
    T* s_mean = reinterpret_cast<T*>(sgen + oMean);
    uint8_t* s_sf = sgen + oSf;
    const uint32_t bar = sbase + oBar;
    volatile int* abort_flag = reinterpret_cast<volatile int*>(sgen + oBar + 8);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sgen + oBar + 12);

    const uint32_t bar_a = bar + 16;        // "the A tile has landed" (the bytes between hold the abort flag and the tensor-memory slot)
    if (t == 224) {
        *abort_flag = 0;
        mbar_init(bar, 1);
        mbar_init(bar_a, 1);
        mbar_fence_init();
        prefetch_tmap(&tm_qm);
        prefetch_tmap(&tm_delta);
    }
    if (warp == 0) {
        tmem_alloc(smem_u32(tmem_slot), kTmemCols);
        tmem_relinquish();
        // Not before this block has its tensor memory: a dependent that takes all of it and then waits for this launch would keep it from
        // going on.  (The attention kernel's shared memory leaves no room next to a block of this one; another's may.)
        pdl_launch_dependents();
    }
    uint4 raw[ITEMS][2];
    x.template rows_each<ITEMS>(bh_off, row0 + rl, RPP, sn, [&](int i, const T* p) {
        load16_packed<T>(p + c * 16, row0 + rl + RPP * i < N, raw[i][0], raw[i][1]);
    });
    pdl_wait();                           // the K rows above are inputs; from here on results of the launches before are read
    // the first A tile (see below) comes in while K is quantized
    auto load_a = [&](int m0) {
        mbar_expect_tx(bar_a, SUB * kASub);
#pragma unroll
        for (int sub = 0; sub < SUB; ++sub)
            tma_load_3d(sbase + oA + sub * kASub, &tm_qm, bar_a, sub * 128, m0, bh);
    };
    if (t == 224) load_a(0);       // (a warp with nothing else to do here)
    if (t < D) {
        if (part != nullptr) {
            const T m = Num<T>::from_f(sum_chunks(part + (int64_t)bh * chunks * D + t, chunks, D) * (N > 0 ? 1.0f / (float)N : 0.f));
            if (tile == 0) km[(int64_t)bh * D + t] = m;
            s_mean[t] = m;
        } else {
            s_mean[t] = km[(int64_t)bh * D + t];
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    uint32_t mu2[8];       // the 16 means of this thread's columns, packed (they are values of the input type)
    *reinterpret_cast<uint4*>(mu2) = reinterpret_cast<const uint4*>(s_mean)[2 * c];
    *reinterpret_cast<uint4*>(mu2 + 4) = reinterpret_cast<const uint4*>(s_mean)[2 * c + 1];
    uint32_t iter = 0;
    bool alive = true;
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
        const int rt = rl + RPP * i;          // row inside the tile
        const int r = row0 + rt;
        const bool zero_row = (r >= N);       // K is padded after smoothing: pad rows are 0
        const uint32_t x2[8] = {raw[i][0].x, raw[i][0].y, raw[i][0].z, raw[i][0].w, raw[i][1].x, raw[i][1].y, raw[i][1].z, raw[i][1].w};
        uint32_t w[8];         // k' of this item, packed: quantized below and stored as the MMA operand as it is
#pragma unroll
        for (int j = 0; j < 8; ++j) w[j] = zero_row ? 0u : Num<T>::sub2(x2[j], mu2[j]);
        uint32_t lo, hi, sfb;
        quant16_packed<T>(w, lo, hi, sfb);
        *reinterpret_cast<uint2*>(codes + ((int64_t)bh * Np + r) * (D / 2) + c * 8) = make_uint2(lo, hi);
        s_sf[sf_atom_offset(rt, c)] = static_cast<uint8_t>(sfb);
        // k' into the B tile: this item's 16 elements are the 16-byte chunks 2c, 2c+1 of row rt
#pragma unroll
        for (int q2 = 0; q2 < 2; ++q2) {
            // (the two sub-tiles lie on the same banks: where one half of a row's threads store even chunks, the other store odd ones)
            const bool odd = (q2 ^ (c >> 2)) & 1;
            const int chunk = 2 * c + (odd ? 1 : 0), sub = chunk >> 3, cw = chunk & 7;
            *reinterpret_cast<uint4*>(sgen + oB + sub * 16384 + rt * 128 + ((cw ^ (rt & 7)) << 4)) =
                make_uint4(odd ? w[4] : w[0], odd ? w[5] : w[1], odd ? w[6] : w[2], odd ? w[7] : w[3]);
        }
    }
    __syncthreads();
    {
        uint8_t* dst = sfs + ((int64_t)bh * (Np / kBlock) + tile) * (D / 64) * 512;
        if (t < (D / 64) * 32) reinterpret_cast<uint4*>(dst)[t] = reinterpret_cast<const uint4*>(s_sf)[t];
    }

    // delta_s of all query heads of this kv head, 128 query blocks per MMA group
    constexpr uint32_t idesc = make_idesc_f16_kk(128, kBf16);
    const int quarter = warp & 3, chalf = warp >> 2;       // tensor-memory lane quarter, column half of the epilogue
    for (int m0 = 0; m0 < rows && alive; m0 += 128, ++iter) {
        // A tile: 128 query-block means, fetched by the copy engine in the 128-byte swizzle the MMA reads.  Rows beyond
        // the tensor arrive as zeros; rows of a shorter sequence of a packed batch only feed accumulator rows
        // that nobody reads.
        fence_proxy_async_smem();       // this thread's stores (the k' tile; the previous epilogue's staging) before the engine touches the tiles
        if (m0 > 0) {
            __syncthreads();
            if (t == 0) load_a(m0);
        }
        alive = mbar_wait(bar_a, iter & 1, abort_flag, status, kWaitDeltaA);
        tc_fence_before();
        alive = __syncthreads_and(alive ? 1 : 0) != 0;
        if (!alive) break;
        if (t == 0) {
            tc_fence_after();
#pragma unroll
            for (int ks = 0; ks < D / 16; ++ks) {
                const uint32_t off = (ks >> 2) * 16384 + (ks & 3) * 32, off_a = (ks >> 2) * kASub + (ks & 3) * 32;
                tc_mma_f16(tmem, make_sdesc(sbase + oA + off_a, 16, 1024, kSwz128), make_sdesc(sbase + oB + off, 16, 1024, kSwz128),
                           idesc, ks > 0);
            }
            tc_commit(bar);
        }
        alive = mbar_wait(bar, iter & 1, abort_flag, status, kWaitDeltaMma);
        alive = __syncthreads_and(alive ? 1 : 0) != 0;
        if (!alive) break;
        tc_fence_after();
        // epilogue: thread = query block (row) of the accumulator, 64 keys of its row = 128 contiguous bytes of delta_s.
        // The warp's 32 rows x 128 bytes are staged in shared memory in the 128-byte swizzle (at D = 128 in the A tile,
        // which is free once the MMAs have completed) and leave as one TMA tile store; the engine clips rows beyond nqm.
        if (m0 + quarter * 32 < rows) {
            const uint32_t acc = tmem + (static_cast<uint32_t>(quarter * 32) << 16) + chalf * 64;
            const int stg_off = oStg + (chalf * (kARows / 32) + quarter) * 4096;
            uint8_t* stg = sgen + stg_off;
            uint32_t z = 0;               // FLAG: 0 while all values are finite
#pragma unroll
            for (int cc = 0; cc < 2; ++cc) {
                float v[32];
                tmem_ld32(acc + cc * 32, v);
                tc_wait_ld();
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    uint32_t p4[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) p4[e] = Num<T>::pack2(v[8 * i + 2 * e], v[8 * i + 2 * e + 1]);
                    *reinterpret_cast<uint4*>(stg + lane * 128 + (((cc * 4 + i) ^ (lane & 7)) << 4)) =
                        make_uint4(p4[0], p4[1], p4[2], p4[3]);
                    if constexpr (FLAG) {
#pragma unroll
                        for (int e = 0; e < 4; ++e) z = Num<T>::zero_fma2(p4[e], z);
                    }
                }
            }
            if (FLAG && (z & 0x7fff7fffu) != 0 && m0 + quarter * 32 + lane < rows) nonfinite[bh] = 1;
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) {
                tma_store_3d(&tm_delta, sbase + stg_off, (row0 + chalf * 64) * 2, m0 + quarter * 32, bh);
                bulk_commit_group();
                bulk_wait_group_read0();      // the engine has read the staging tile: it may be written again
            }
            __syncwarp();
        }
        tc_fence_before();
        __syncthreads();      // the accumulator and the A tile are free again
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        tmem_dealloc(tmem, kTmemCols);
    }
}

// ------------------------------------------------------------------------------------------------
// K for up to 64 query blocks per kv head, D = 64 up to 128 (token generation, chunks of a prompt, calls with one Q mean per head, packed prompts): two blocks per SM
// walk runs of tiles, all of one length, that go on from head to head.
//   warps 0-7   hold the next tile's rows in registers (a row's load is issued as soon as the one before it in that place is used), smooth and quantize
//               them, store k' as the operand of the MMA, and write delta_s of the tile before: nothing in their loop waits for a copy or an MMA
//               that has just been started, and a barrier of all eight is met once per head
//   warp 8      the MMAs, as delta_s^T: the 128 keys are the rows of the accumulator and the query blocks its columns, so that an MMA costs
//               what the query blocks ask for and a warp's store covers 32 keys of a row
// The kernel above spends a chain of load, quantization, copy, MMA and read-out per tile, with four block-wide barriers, and accumulator rows of 128 query
// blocks where there are four.  What bounds this one: instructions (5 100 per tile, issue slots 63 % busy) and, at 5.0 TB/s, nearly HBM.  One token of 8 x 32
// heads against 8 192 keys of 8 kv heads, this kernel's time 51.5 -> 34.3 us (D = 64 32.3 -> 23.0).  Pre-pass of 4 096 / 2 048 / 512 / 296 tiles, 8 kv
// heads, us: 4 query blocks 108.1 / 55.6 / 19.6 / 16.6 -> 90.5 / 47.3 / 18.7 / 15.0, 64 blocks 158.3 / 83.0 / 24.3 / 20.7 -> 143.3 / 74.7 / 22.8 / 19.6, D = 64
// 4 blocks 58.2 / 33.5 / 15.0 / 14.8 -> 50.1 / 29.0 / 14.6 / 14.5, 64 blocks 92.2 / 47.7 / 17.5 / 15.9 -> 84.4 / 45.1 / 18.5 / 14.6.  Variants of it, first figure
// (51.5 before): rows copied to shared memory ahead by all warps 44.5, by a warp of its own 44.1 (shared memory then moves 160 KB per tile: the copy, the
// read, k', and the MMA's operands), three blocks per SM 38.6 (two 36.0), one store per key and row 36.0 -> 35.5, row addresses ahead 34.3.
// NR = 32 instead of 64 columns: up to 32 query blocks (half of the read-out and of its registers).  Pre-pass with 64 / 32 columns, us: one token of 4 x 32 heads, 8 kv heads, 4 096
// keys 28.7 / 27.6 (D = 64 20.5 / 19.3), 8 192 47.1 / 46.0 (30.5 / 28.1), of 8 x 32 heads 92.2 / 90.3 (53.3 / 49.2), of 8 x 28 heads, 4 kv heads, 9 000 keys 53.7 / 53.2 (34.8 / 31.9); 24
// query blocks, 2 x 8 x 16 000 keys 50.9 / 50.7 (32.6 / 31.2).
// ------------------------------------------------------------------------------------------------
// A place in the list of tiles: entry by entry, head by head, tile by tile.
template <typename T>
struct KCursor {
    int bh, b, h, tile, nt, N;
    int64_t off;
    __device__ __forceinline__ void enter(const Src<T>& x, int64_t sb, int64_t sh, int64_t sn, int Nmax) {
        N = Nmax;
        off = x.base(b, h, sb, sh, sn, N);
        nt = max(1, (N + kBlock - 1) / kBlock);
    }
    __device__ __forceinline__ bool next(int H) {             // true: another head, to be entered
        if (++tile < nt) return false;
        tile = 0;
        ++bh;
        if (++h == H) { h = 0; ++b; }
        return true;
    }
};

__device__ __forceinline__ void bar_sync(int id, int threads) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory"); }

template <int D, int NR>
struct KRunCfg {
    static constexpr int SUB = D / 64;                        // 64-element (128-byte) sub-tiles along K
    static constexpr int kThreads = 256 + 32;
    static constexpr int kBlocks = 2;                         // per SM
    static constexpr int oK = 0, oQ = 2 * SUB * 16384, oMean = oQ + SUB * NR * 128, oBar = oMean + 2 * D * 2, kSmem = oBar + 64 + 1024;      // + slack for the alignment
    static constexpr uint32_t kCols = 2 * NR < 32 ? 32 : 2 * NR;      // tensor memory: two accumulators
};

template <typename T, int D, int NR, bool FLAG>
__global__ void __launch_bounds__(KRunCfg<D, NR>::kThreads, KRunCfg<D, NR>::kBlocks) quant_k_delta_run_kernel(
    const __grid_constant__ Src<T> x, int64_t sb, int64_t sh, int64_t sn, FastDiv H, FastDiv tiles, int B, int Nmax, int Np,
    T* __restrict__ km, const float* __restrict__ part, int chunks, uint8_t* __restrict__ codes, uint8_t* __restrict__ sfs, T* __restrict__ delta, int rows,
    int* __restrict__ status, int* __restrict__ nonfinite, const __grid_constant__ CUtensorMap tm_qm) {
    using C = KRunCfg<D, NR>;
    constexpr int CH = D / 16, RPP = 256 / CH, ITEMS = kBlock / RPP, SUB = C::SUB;
    extern __shared__ uint8_t smem_dyn[];
    const uint32_t sbase = (smem_u32(smem_dyn) + 1023u) & ~1023u;
    uint8_t* sgen = smem_dyn + (sbase - smem_u32(smem_dyn));
    const int t = threadIdx.x, warp = __shfl_sync(0xffffffffu, t >> 5, 0), lane = t & 31;
    const uint32_t bar_ready = sbase + C::oBar, bar_mma = bar_ready + 16, bar_q = bar_mma + 16;
    volatile int* abort_flag = reinterpret_cast<volatile int*>(sgen + C::oBar + 48);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sgen + C::oBar + 52);
    if (t == 0) {
        *abort_flag = 0;
        for (int i = 0; i < 2; ++i) {
            mbar_init(bar_ready + 8 * i, 8);
            mbar_init(bar_mma + 8 * i, 1);
        }
        mbar_init(bar_q, 1);
        mbar_fence_init();
    }
    if (warp == 8) {
        tmem_alloc(smem_u32(tmem_slot), C::kCols);
        tmem_relinquish();
        pdl_launch_dependents();          // (not before the tensor memory is this block's, see above)
    }
    // This block's run of tiles, the same number for every block.
    KCursor<T> at;
    int n;
    {
        int p0;
        if (x.cu == nullptr) {
            const int64_t total = (int64_t)B * H.d * tiles.d;
            p0 = (int)(total * blockIdx.x / gridDim.x);
            n = (int)(total * (blockIdx.x + 1) / gridDim.x) - p0;
            at.bh = tiles.divmod(p0, at.tile);
            at.b = H.divmod(at.bh, at.h);
        } else {
            auto tiles_of = [&](int b) { return b < B ? max(1, (min(max(x.cu[b + 1] - x.cu[b], 0), Nmax) + kBlock - 1) / kBlock) : 0; };
            int all = 0;
            for (int b0 = 0; b0 < B; b0 += 32) all += __reduce_add_sync(0xffffffffu, tiles_of(b0 + lane));
            const int64_t total = (int64_t)all * H.d;
            p0 = (int)(total * blockIdx.x / gridDim.x);
            n = (int)(total * (blockIdx.x + 1) / gridDim.x) - p0;
            at.b = at.h = at.tile = 0;
            for (int b0 = 0; n > 0; b0 += 32) {
                const int mine = tiles_of(b0 + lane);
                const int here = __reduce_add_sync(0xffffffffu, mine) * (int)H.d;
                if (p0 >= here) { p0 -= here; continue; }
                for (int i = 0;; ++i) {
                    const int nt = __shfl_sync(0xffffffffu, mine, i);
                    if (p0 < nt * (int)H.d) {
                        at.b = b0 + i;
                        at.h = p0 / nt;
                        at.tile = p0 - at.h * nt;
                        break;
                    }
                    p0 -= nt * (int)H.d;
                }
                break;
            }
            at.bh = at.b * (int)H.d + at.h;
        }
        if (n > 0) at.enter(x, sb, sh, sn, Nmax);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);
    if (warp < 8) {
        // ------------------------------------------------------------------ smoothing and quantization; delta_s of the tile before
        const int c = micro_col<D>(lane), rl = micro_row<D>(warp, lane);
        const uint32_t place = (uint32_t)((c >> 2) * 16384 + rl * 128 + ((((2 * c) & 7) ^ (rl & 7)) << 4));      // of the microblock's first 16 bytes; the others: ^ 16
        KCursor<T> ahead = at;
        uint4 raw[ITEMS][2];
        const T* src[ITEMS];              // this thread's rows of the tile `ahead`
        int rows_ahead = 0;               // ... of which those are there whose number in the tile is less
        auto locate = [&]() {
            const int r = ahead.tile * kBlock + rl;
            rows_ahead = ahead.N - r;
            x.template rows_each<ITEMS>(ahead.off + c * 16, r, RPP, sn, [&](int i, const T* p) { src[i] = p; });
        };
        if (n > 0) {
            locate();
#pragma unroll
            for (int i = 0; i < ITEMS; ++i) load16_packed<T>(src[i], RPP * i < rows_ahead, raw[i][0], raw[i][1]);
        }
        pdl_wait();                       // the K rows are inputs; from here on results of the launches before are read
        uint32_t mu2[8];                  // the 16 means of this thread's columns, packed
        bool fresh = true;                // this head's mean is not in mu2 yet
        int seg = 0;
        // delta_s of a tile: a thread is a key (tensor-memory lane), the warps 0-3 and 4-7 have half of the query blocks each
        auto write_delta = [&](int it, int bh, int tile) {
            constexpr int HALF = NR / 2;
            const int quarter = warp & 3, r0 = (warp >> 2) * HALF;
            if (!mbar_try_wait(bar_mma + 8 * (it & 1), (it >> 1) & 1)) mbar_wait(bar_mma + 8 * (it & 1), (it >> 1) & 1, abort_flag, status, kWaitDeltaMma);
            __syncwarp();
            if (r0 < rows) {
                tc_fence_after();
                // Two neighbouring lanes swap one of two rows: each has two keys of one row then, and a store covers 64 bytes of both rows.
                const int row = r0 + (lane & 1);
                T* dst = delta + ((int64_t)bh * rows + row) * Np + tile * kBlock + quarter * 32 + (lane & ~1);
                uint32_t z = 0;           // FLAG: 0 while all values are finite
                constexpr int STEP = HALF < 32 ? HALF : 32;
#pragma unroll
                for (int c0 = 0; c0 < HALF; c0 += STEP) {
                    if (c0 > 0 && r0 + c0 >= rows) break;
                    float v[STEP];
                    const uint32_t acc = tmem + (static_cast<uint32_t>(quarter * 32) << 16) + (it & 1) * NR + r0 + c0;
                    if constexpr (STEP == 16) tmem_ld16(acc, v);
                    else tmem_ld32(acc, v);
                    tc_wait_ld();
#pragma unroll
                    for (int r = 0; r < STEP; r += 2, dst += 2 * Np) {
                        const uint32_t w = Num<T>::pack2(v[r], v[r + 1]), y = __shfl_xor_sync(0xffffffffu, w, 1);
                        const uint32_t pair = __byte_perm(w, y, lane & 1 ? 0x3276 : 0x5410);
                        if (row + c0 + r < rows) {
                            *reinterpret_cast<uint32_t*>(dst) = pair;
                            if (FLAG) z = Num<T>::zero_fma2(pair, z);
                        }
                    }
                }
                tc_fence_before();
                if (FLAG && (z & 0x7fff7fffu) != 0) nonfinite[bh] = 1;
            }
        };
        int bh_before = 0, tile_before = 0;
        for (int it = 0; it < n; ++it) {
            if (fresh) {
                T* s_mean = reinterpret_cast<T*>(sgen + C::oMean) + (seg & 1) * D;
                if (t < D) {
                    T m;
                    if (part != nullptr) {
                        m = Num<T>::from_f(sum_chunks(part + (int64_t)at.bh * chunks * D + t, chunks, D) * (at.N > 0 ? 1.0f / (float)at.N : 0.f));
                        if (at.tile == 0) km[(int64_t)at.bh * D + t] = m;
                    } else {
                        m = km[(int64_t)at.bh * D + t];
                    }
                    s_mean[t] = m;
                }
                bar_sync(1, 256);
                *reinterpret_cast<uint4*>(mu2) = reinterpret_cast<const uint4*>(s_mean)[2 * c];
                *reinterpret_cast<uint4*>(mu2 + 4) = reinterpret_cast<const uint4*>(s_mean)[2 * c + 1];
                ++seg;
            }
            const bool more = it + 1 < n;
            const int here = rows_ahead;
            if (more) {
                if (ahead.next((int)H.d)) ahead.enter(x, sb, sh, sn, Nmax);
                locate();
            }
            const int row0 = at.tile * kBlock;
            const bool edge = row0 + kBlock > at.N;
            uint8_t *lo_half = sgen + C::oK + (it & 1) * SUB * 16384 + place, *hi_half = sgen + C::oK + (it & 1) * SUB * 16384 + (place ^ 16u);
            uint32_t sf = 0;              // scale bytes of this thread's microblocks
            uint8_t* code = codes + ((int64_t)at.bh * Np + row0 + rl) * (D / 2) + c * 8;
#pragma unroll
            for (int i = 0; i < ITEMS; ++i) {
                const uint32_t x2[8] = {raw[i][0].x, raw[i][0].y, raw[i][0].z, raw[i][0].w, raw[i][1].x, raw[i][1].y, raw[i][1].z, raw[i][1].w};
                uint32_t w[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) w[j] = Num<T>::sub2(x2[j], mu2[j]);
                if (edge) {                   // K is padded after smoothing: pad rows are 0
#pragma unroll
                    for (int j = 0; j < 8; ++j) w[j] = RPP * i < here ? w[j] : 0u;
                }
                if (more) load16_packed<T>(src[i], RPP * i < rows_ahead, raw[i][0], raw[i][1]);
                // k', the operand of the MMA: [row][16-byte chunk], 128-byte swizzle
                *reinterpret_cast<uint4*>(lo_half + i * RPP * 128) = make_uint4(w[0], w[1], w[2], w[3]);
                *reinterpret_cast<uint4*>(hi_half + i * RPP * 128) = make_uint4(w[4], w[5], w[6], w[7]);
                uint32_t lo, hi, sfb;
                quant16_packed<T>(w, lo, hi, sfb);
                *reinterpret_cast<uint2*>(code + i * RPP * (D / 2)) = make_uint2(lo, hi);
                sf |= sfb << (8 * i);
            }
            fence_proxy_async_smem();
            warp_arrive(bar_ready + 8 * (it & 1), lane);
            store_scales<D>(sfs + ((int64_t)at.bh * (Np / kBlock) + at.tile) * SUB * 512, sf, c, rl, lane);
            if (it > 0) write_delta(it - 1, bh_before, tile_before);
            bh_before = at.bh;
            tile_before = at.tile;
            fresh = at.next((int)H.d);
            if (fresh && more) at.enter(x, sb, sh, sn, Nmax);
        }
        if (n > 0) write_delta(n - 1, bh_before, tile_before);
    } else {
        // ------------------------------------------------------------------ MMAs: delta_s^T [128 keys][query blocks] = k' qm^T
        pdl_wait();
        constexpr uint32_t idesc = make_idesc_f16_kk(NR, Num<T>::kIsBf16);
        constexpr uint32_t hi_k = sdesc_hi(1024, kSwz128);
        const uint32_t k_lo0 = __shfl_sync(0xffffffffu, sdesc_lo(sbase + C::oK, 16), 0), q_lo = __shfl_sync(0xffffffffu, sdesc_lo(sbase + C::oQ, 16), 0);
        bool fresh = true;
        uint32_t q_parity = 0;
        for (int it = 0; it < n; ++it) {
            const int st = it & 1;
            if (fresh) {                  // this head's query-block means; the MMAs with the last ones' must be complete
                if (it > 0) mbar_wait<true>(bar_mma + 8 * (st ^ 1), ((it - 1) >> 1) & 1, abort_flag, status, kWaitDeltaMma);
                if (lane == 0) {
                    mbar_expect_tx(bar_q, SUB * NR * 128);
#pragma unroll
                    for (int sub = 0; sub < SUB; ++sub) tma_load_3d(sbase + C::oQ + sub * NR * 128, &tm_qm, bar_q, sub * 128, 0, at.bh);
                }
                __syncwarp();
                mbar_wait<true>(bar_q, q_parity, abort_flag, status, kWaitDeltaA);
                q_parity ^= 1;
            }
            mbar_wait<true>(bar_ready + 8 * st, (it >> 1) & 1, abort_flag, status, kWaitDeltaA);
            __syncwarp();
            tc_fence_after();
            if (elect_one()) {
                const uint32_t k_lo = k_lo0 + st * (SUB * 16384 / 16), acc = tmem + st * NR;
#pragma unroll
                for (int ks = 0; ks < D / 16; ++ks)
                    tc_mma_f16(acc, sdesc(k_lo + ((ks >> 2) * 16384 + (ks & 3) * 32) / 16, hi_k), sdesc(q_lo + ((ks >> 2) * NR * 128 + (ks & 3) * 32) / 16, hi_k),
                               idesc, ks > 0);
                tc_commit(bar_mma + 8 * st);
            }
            __syncwarp();
            fresh = at.next((int)H.d);
            if (fresh && it + 1 < n) at.enter(x, sb, sh, sn, Nmax);
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 8) {
        tc_fence_after();
        tmem_dealloc(tmem, C::kCols);
    }
}

// ------------------------------------------------------------------------------------------------
// V: one tile of 128 tokens x D channels per CTA -> V^T codes (microblocks along tokens) + scale atoms
// ------------------------------------------------------------------------------------------------
template <typename T, int D>
__device__ __forceinline__ void quant_vt_tile(const Src<T>& x, int64_t sb, int64_t sh, int64_t sn, FastDiv H, int N, int Np,
                                              uint8_t* __restrict__ codes, uint8_t* __restrict__ sfs, int tile, int bh, uint8_t* smem_raw) {
    constexpr int PITCH = D;              // elements (rows are stored in 16-byte pieces, and read a word per lane along a row)
    int h;
    const int b = H.divmod(bh, h);
    const int t = threadIdx.x;
    const int64_t bh_off = x.base(b, h, sb, sh, sn, N);
    const int row0 = tile * kBlock;
    if (row0 >= N && row0 > 0) return;    // a tile beyond this entry's padded length (variable-length batches only)

    T* s_v = reinterpret_cast<T*>(smem_raw);                                  // [128][PITCH]
    constexpr int OPITCH = 72;            // bytes per staged output row (64 + 8: 8-byte stores stay conflict-free)
    uint8_t* s_out = smem_raw + ((kBlock * PITCH * 2 + 15) / 16) * 16;          // [D][OPITCH] codes
    uint8_t* s_sf = s_out + D * OPITCH;                                        // [2 * 512]

    // zero the scale atoms (rows >= D of a 128-row atom stay zero)
    if (t < 64) reinterpret_cast<uint4*>(s_sf)[t] = make_uint4(0, 0, 0, 0);
    // coalesced load: 16 bytes per thread per pass
    constexpr int TPR = D / 8, RPP = 256 / TPR;
    {
        const int c8 = t % TPR, rl = t / TPR;
        uint4 val[kBlock / RPP];
        x.template rows_each<kBlock / RPP>(bh_off, row0 + rl, RPP, sn, [&](int i, const T* p) {
            val[i] = make_uint4(0, 0, 0, 0);
            if (row0 + rl + i * RPP < N) val[i] = __ldg(reinterpret_cast<const uint4*>(p + c8 * 8));
        });
#pragma unroll
        for (int i = 0; i < kBlock / RPP; ++i) {
            *reinterpret_cast<uint4*>(s_v + (rl + i * RPP) * PITCH + c8 * 8) = val[i];
        }
    }
    __syncthreads();
    // two microblocks per item: (channels 2*dp and 2*dp + 1, token group mb); channel pair fastest across
    // threads, so every shared-memory read is one conflict-free 32-bit word holding both channels
    for (int item = t; item < (D / 2) * 8; item += 256) {
        const int dp = item % (D / 2), mb = item / (D / 2);
        uint32_t w[16];             // 16 tokens of both channels
        uint32_t m2 = 0u;           // running maximum magnitude of both channels, packed
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            w[i] = *reinterpret_cast<const uint32_t*>(s_v + (mb * 16 + i) * PITCH + 2 * dp);
            m2 = Num<T>::absmax2(m2, w[i]);
        }
        const float2 amax2 = Num<T>::to_f2(m2);
#pragma unroll
        for (int ch = 0; ch < 2; ++ch) {
            uint32_t sfb;
            const float inv = micro_scale(ch == 0 ? amax2.x : amax2.y, sfb);
            const uint64_t inv2 = pack2f(inv, inv);
            uint32_t code[2];
#pragma unroll
            for (int g = 0; g < 2; ++g) {
                float y[8];
#pragma unroll
                for (int i = 0; i < 8; i += 2) {
                    const float2 v2 = Num<T>::to_f2(w[8 * g + i]), v3 = Num<T>::to_f2(w[8 * g + i + 1]);
                    unpack2f(mul2(ch == 0 ? pack2f(v2.x, v3.x) : pack2f(v2.y, v3.y), inv2), y[i], y[i + 1]);
                }
                code[g] = cvt_e2m1x8(y[0], y[1], y[2], y[3], y[4], y[5], y[6], y[7]);
            }
            *reinterpret_cast<uint2*>(s_out + (2 * dp + ch) * OPITCH + mb * 8) = make_uint2(code[0], code[1]);
            s_sf[sf_atom_offset(2 * dp + ch, mb)] = static_cast<uint8_t>(sfb);
        }
    }
    __syncthreads();
    // coalesced stores: D rows of 64 bytes
    for (int idx = t; idx < D * 8; idx += 256) {
        const int d = idx >> 3, q = idx & 7;
        *reinterpret_cast<uint2*>(codes + ((int64_t)bh * D + d) * (Np / 2) + tile * 64 + q * 8) =
            *reinterpret_cast<const uint2*>(s_out + d * OPITCH + q * 8);
    }
    if (t < 64) {
        uint8_t* dst = sfs + ((int64_t)bh * (Np / kBlock) + tile) * 1024;
        reinterpret_cast<uint4*>(dst)[t] = reinterpret_cast<const uint4*>(s_sf)[t];
    }
}

// ------------------------------------------------------------------------------------------------
// Everything of the pre-pass that reads raw inputs only, in one launch: partial column sums of K (and of Q, when it is smoothed
// by one mean per head), V quantization, and Q quantization when it needs no mean of a whole head.  Block b works on the b-th
// piece of the list; the parts have nothing to wait for from one another, so their tails and launch gaps disappear.
// With the status words cleared here, the K mean formed by the K kernel where that is cheap, and the K and attention kernels
// launched early (griddepcontrol), a call is 3 launches instead of 6 and 2 memsets: 1 024 tokens of two heads 51 -> 26 us, a
// 3 001-token prompt 151 -> 106 us.  HBM-bound at size: 0.47 GB read and 0.16 GB written in 85 us for 17 550 queries of 96 heads.
// ------------------------------------------------------------------------------------------------
template <typename T>
struct StageArgs {
    Src<T> q, k, v;
    int64_t qs[3], ks[3], vs[3];
    FastDiv Hq, Hkv, chunks_k, chunks_q, tiles_q, tiles_k;
    int group, Nq, Nk, Nq_p, Nk_p;
    int n_colk, n_colq, n_q, n_v;      // pieces of each kind, in this order
    int q_block_mean;
    float *part_k, *part_q;
    T *km, *qm;
    uint8_t *q_codes, *q_sf, *v_codes, *v_sf;
    float* qkm;                        // nullptr: not wanted
    MeanParts means;
    int* clear;                        // words to zero: status, work counter, flags, `nonfinite` (nullptr: not in this launch)
    int n_clear;
};

constexpr int kMostCleared = 512;      // words

template <typename T, int D>
struct StageCfg {
    static constexpr int kQ = D * 4 + (kBlock * D + 4 * (32 / (D / 8)) * (D + 8)) * (int)sizeof(T);   // staged tile and chain sums
    static constexpr int kV = kBlock * D * (int)sizeof(T) + D * 72 + 1024;
    static constexpr int kCol = (2048 / D) * (D + 1) * 4;
    static constexpr int kSmem = kQ > kV ? (kQ > kCol ? kQ : kCol) : (kV > kCol ? kV : kCol);
};

// Next to HBM the shared-memory pipe bounds it (62 to 65 % busy, issue slots 52 %), so the tiles stand there without bank conflicts: Q's rows in pairs of swapped chunks, V's in
// 16-byte pieces (as words of padded rows every store took four turns), the scale bytes put together by shuffles instead of in a staged atom behind one more barrier.  Stage
// kernel, us: 17 550 queries of 96 heads, D = 64 67.4 -> 62.3, D = 128 115.0 -> 109.5; K sums and V of 8 x 8 x 8 192 keys 55.4 -> 52.4 (5.8 TB/s), D = 64 27.6 -> 26.4.
// Six resident blocks at D = 64 (40 registers, column sums four rows deep): 17 550 queries of 96 heads 71 -> 58 us against four.  At
// D = 128 four: five spill (131 -> 149 us for 8 x 8 x 8 192 keys with their K kernel).
template <typename T, int D>
__global__ void __launch_bounds__(256, D == 64 ? 6 : 4) prepass_stage_kernel(const __grid_constant__ StageArgs<T> a) {
    extern __shared__ __align__(16) uint8_t smem_raw[];
    pdl_launch_dependents();
    int i = blockIdx.x;
    if (i == 0 && a.clear != nullptr) {
#pragma unroll
        for (int j = 0; j < kMostCleared; j += 256)
            if (threadIdx.x + j < a.n_clear) a.clear[threadIdx.x + j] = 0;
    }
    int tile, bh;
    if (i < a.n_colk) {
        bh = a.chunks_k.divmod(i, tile);
        colsum_chunk<T, D>(a.k, a.ks[0], a.ks[1], a.ks[2], a.Hkv, a.Nk, a.part_k, a.chunks_k.d, tile, bh, reinterpret_cast<float*>(smem_raw));
        return;
    }
    i -= a.n_colk;
    if (i < a.n_colq) {
        bh = a.chunks_q.divmod(i, tile);
        colsum_chunk<T, D>(a.q, a.qs[0], a.qs[1], a.qs[2], a.Hq, a.Nq, a.part_q, a.chunks_q.d, tile, bh, reinterpret_cast<float*>(smem_raw));
        return;
    }
    i -= a.n_colq;
    if (i < a.n_q) {
        bh = a.tiles_q.divmod(i, tile);
        if (a.q_block_mean)
            quant_q_tile<T, D, kModeQBlockMean>(a.q, a.qs[0], a.qs[1], a.qs[2], a.Hq, a.Nq, a.Nq_p, nullptr, a.qm, a.q_codes, a.q_sf, a.km,
                                                a.group, a.qkm, a.means, tile, bh, smem_raw);
        else
            quant_q_tile<T, D, kModeQGlobalMean>(a.q, a.qs[0], a.qs[1], a.qs[2], a.Hq, a.Nq, a.Nq_p, a.qm, a.qm, a.q_codes, a.q_sf, a.km,
                                                 a.group, a.qkm, a.means, tile, bh, smem_raw);
        return;
    }
    i -= a.n_q;
    bh = a.tiles_k.divmod(i, tile);
    quant_vt_tile<T, D>(a.v, a.vs[0], a.vs[1], a.vs[2], a.Hkv, a.Nk, a.Nk_p, a.v_codes, a.v_sf, tile, bh, smem_raw);
}

// ------------------------------------------------------------------------------------------------
// host-side launch
// ------------------------------------------------------------------------------------------------
// Up to this many chunks (16 384 rows) the blocks that need a mean form it themselves from the partial sums (an 8 KB read from L2 at
// 8 192 keys); beyond, one small kernel does, because every block adds up all chunks.  Inside / by a launch of its own, us per call:
// 1 024 queries of 32 heads (8 kv heads) 8 192 keys 129.6 / 134.3, 16 384 241.9 / 245.6, 24 576 356.6 / 359.1, 65 536 916 / 903; one
// token of 8 x 32 heads 8 192 keys 143.4 / 146.7, 16 384 271.7 / 268.2, of 4 x 32 heads 32 768 keys 330.3 / 317.0; LSE and one Q mean
// per head, 2 x 16 heads, D = 64, 16 384 tokens 2 764 / 2 752, 24 576 6 090 / 6 053.  The sides meet between 16 384 and 24 576.
constexpr int kInlineMeanChunks = 32;

template <typename T, int D>
static cudaError_t launch_prepass_t(const PrepassArgs& a, cudaStream_t st) {
    T* km = static_cast<T*>(a.km);
    T* qm = static_cast<T*>(a.qm);
    T* delta = static_cast<T*>(a.delta);
    const int BHq = a.B * a.Hq, BHkv = a.B * a.Hkv;
    cudaError_t e = allow_smem<prepass_stage_kernel<T, D>>(StageCfg<T, D>::kSmem);
    if (e != cudaSuccess) return e;

    StageArgs<T> s = {};
    s.q = make_src<T>(a.q, a.cu_q);
    s.k = make_src<T>(a.k, a.cu_k);
    s.v = make_src<T>(a.v, a.cu_k);
    for (int i = 0; i < 3; ++i) {
        s.qs[i] = a.qs[i];
        s.ks[i] = a.ks[i];
        s.vs[i] = a.vs[i];
    }
    const int tiles_q = a.Nq_p / kBlock, tiles_k = a.Nk_p / kBlock;
    s.Hq = FastDiv(a.Hq); s.Hkv = FastDiv(a.Hkv);
    s.chunks_k = FastDiv(a.kchunks_k); s.chunks_q = FastDiv(a.kchunks_q); s.tiles_q = FastDiv(tiles_q); s.tiles_k = FastDiv(tiles_k);
    s.group = a.Hq / a.Hkv; s.Nq = a.Nq; s.Nk = a.Nk; s.Nq_p = a.Nq_p; s.Nk_p = a.Nk_p;
    s.q_block_mean = a.per_block_mean;
    s.part_k = a.kpart; s.part_q = a.kpart + (size_t)BHkv * a.kchunks_k * D;
    s.km = km; s.qm = qm;
    s.q_codes = a.q_codes; s.q_sf = a.q_sf; s.v_codes = a.v_codes; s.v_sf = a.v_sf;
    s.clear = a.clear; s.n_clear = a.n_clear < kMostCleared ? a.n_clear : kMostCleared;
    if (a.n_clear > kMostCleared && (e = checked(cudaMemsetAsync(a.clear + kMostCleared, 0, (a.n_clear - kMostCleared) * sizeof(int), st))) != cudaSuccess) return e;
    // Q waits for the means when it is smoothed by one mean per head (api.py:88-90) or when q . km is wanted
    const bool q_late = !a.per_block_mean || a.want_qkm;
    const bool km_here = !a.km_given;
    const bool km_inline = km_here && a.kchunks_k <= kInlineMeanChunks, qm_inline = !a.per_block_mean && a.kchunks_q <= kInlineMeanChunks;
    s.n_colk = km_here ? a.kchunks_k * BHkv : 0;
    s.n_colq = a.per_block_mean ? 0 : a.kchunks_q * BHq;
    s.n_q = q_late ? 0 : tiles_q * BHq;
    s.n_v = tiles_k * BHkv;
    // Every launch is checked: the ones behind a failed one would work on what an earlier call left (the work counter among it).
    if ((e = launch(false, prepass_stage_kernel<T, D>, dim3(s.n_colk + s.n_colq + s.n_q + s.n_v), dim3(256), (size_t)StageCfg<T, D>::kSmem, st, s)) != cudaSuccess)
        return e;
    if (km_here && !km_inline &&
        (e = launch(false, colmean_finalize_kernel<T, D>, dim3(BHkv), dim3(D), 0, st, (const float*)s.part_k, a.kchunks_k, 1.0f / (float)a.Nk, km, a.cu_k, a.Hkv, 0)) != cudaSuccess)
        return e;
    if (!a.per_block_mean && !qm_inline &&
        (e = launch(false, colmean_finalize_kernel<T, D>, dim3(BHq), dim3(D), 0, st, (const float*)s.part_q, a.kchunks_q, 1.0f / (float)a.Nq_p, qm, a.cu_q, a.Hq, 1)) != cudaSuccess)
        return e;
    if (q_late) {
        s.n_colk = s.n_colq = s.n_v = 0;
        s.n_q = tiles_q * BHq;
        s.qkm = a.want_qkm ? a.qkm : nullptr;
        s.clear = nullptr;
        s.means.k = km_inline ? s.part_k : nullptr;
        s.means.q = qm_inline ? s.part_q : nullptr;
        s.means.chunks_k = a.kchunks_k;
        s.means.chunks_q = a.kchunks_q;
        s.means.Nk = a.Nk;
        s.means.cu_k = a.cu_k;
        s.means.wait = true;
        if ((e = launch(true, prepass_stage_kernel<T, D>, dim3(s.n_q), dim3(256), (size_t)StageCfg<T, D>::kSmem, st, s)) != cudaSuccess) return e;
    }
    // tensor maps for the K kernel: the Q means and delta_s of a kv head's query heads follow one another, so both are byte
    // tensors [B*Hkv][group * nqm][...] and one MMA takes the blocks of several heads
    const uint64_t rows = (uint64_t)(a.Hq / a.Hkv) * a.nqm;
    int dev = 0;
    DeviceInfo info;
    if ((e = current_device(&dev, &info)) != cudaSuccess) return e;
    const int64_t tiles = (int64_t)tiles_k * BHkv;
    auto by_flag = [&](auto go) { return a.nonfinite != nullptr ? go(std::true_type()) : go(std::false_type()); };
    auto run = [&](auto rows_) {
        return by_flag([&](auto flag_) {
            constexpr int NR = decltype(rows_)::value;
            using C = KRunCfg<D, NR>;
            constexpr auto kern = quant_k_delta_run_kernel<T, D, NR, decltype(flag_)::value>;
            const cudaError_t allowed = allow_smem<kern>(C::kSmem);
            if (allowed != cudaSuccess) return allowed;
            alignas(64) CUtensorMap tm_qm;
            if (encode_tiled_bytes(&tm_qm, qm, (uint64_t)D * 2, rows, (uint64_t)BHkv, 128, NR, 3) != 0) return cudaErrorInvalidValue;
            const int64_t slots = (int64_t)C::kBlocks * info.sms;
            return launch(true, kern, dim3((unsigned)(tiles < slots ? tiles : slots)), dim3(C::kThreads), (size_t)C::kSmem, st, s.k, a.ks[0], a.ks[1], a.ks[2],
                          s.Hkv, s.tiles_k, a.B, a.Nk, a.Nk_p, km, km_inline ? (const float*)s.part_k : (const float*)nullptr, a.kchunks_k, a.k_codes, a.k_sf,
                          delta, (int)rows, a.status, a.nonfinite, tm_qm);
        });
    };
    auto one_tile = [&](auto a_rows_) {
        return by_flag([&](auto flag_) {
            constexpr int AR = decltype(a_rows_)::value;
            constexpr auto kern = quant_k_delta_kernel<T, D, AR, decltype(flag_)::value>;
            constexpr size_t smem = (D / 64) * (128 + AR) * 128 + D * 4 + (D / 64) * 512 + 64 + 1024 + (D == 64 ? 1024 + AR * 256 : 0);
            const cudaError_t allowed = allow_smem<kern>((int)smem);
            if (allowed != cudaSuccess) return allowed;
            alignas(64) CUtensorMap tm_qm, tm_delta;
            if (encode_tiled_bytes(&tm_qm, qm, (uint64_t)D * 2, rows, (uint64_t)BHkv, 128, AR, 3) != 0 ||
                encode_tiled_bytes(&tm_delta, delta, (uint64_t)a.Nk_p * 2, rows, (uint64_t)BHkv, 128, 32, 3) != 0)
                return cudaErrorInvalidValue;
            return launch(true, kern, dim3(tiles_k, BHkv), dim3(256), smem, st, s.k, a.ks[0], a.ks[1], a.ks[2],
                          s.Hkv, a.Nk, a.Nk_p, km, km_inline ? (const float*)s.part_k : (const float*)nullptr, a.kchunks_k, a.k_codes, a.k_sf, (int)rows,
                          a.status, a.nonfinite, tm_qm, tm_delta);
        });
    };
    // Which kernel, us per call with a block per tile / runs.
    // Up to one tile per SM nothing goes on in a run: the pre-pass alone is shorter with runs (1 024 tokens of 16 heads 15.2 / 12.8), but the attention kernel starts later behind
    // them: D = 128, 1 024 of 16 25.1 / 26.1, 500 queries of 32 heads, 1 000 keys of 8 24.6 / 26.4, 1 500 of 12 29.8 / 30.6, 256 of 8 16.4 / 16.7, 2 048 of 8 32.7 / 32.8; D = 64, 1 829 of
    // 4 x 2 26.7 / 28.7, 700 of 2 x 8, causal, 19.2 / 20.5.
    // At D = 64 four blocks of one tile fit an SM at once, two of the other kernel: a block per tile between two and three tiles per SM, too.  Up to 64 query blocks, 2.2 tiles per SM 70.2
    // / 71.3, 73.8 / 74.6, 2.6 21.4 / 21.9, 2.7 42.0 / 42.7, 37.5 / 37.9, 2.8 89.3 / 89.7; 3.1 35.4 / 35.0, 96.3 / 96.3, 3.4 69.5 / 67.8, 78.5 / 78.1, 3.7 73.8 / 72.0, 161.1 / 160.9, 3.8 54.4 /
    // 53.3, 3.9 23.8 / 22.6, 59.1 / 57.4, 204.7 / 203.9.  Up to 32 also between one and two, where it is by turns the faster and the slower: 1.1 20.5 / 21.7, 47.2 / 48.0, 1.4 51.1 / 51.1, 34.9 /
    // 35.8, 1.6 40.9 / 41.0, 18.4 / 18.0, 1.8 44.3 / 43.5, 43.0 / 43.1, 2.0 28.5 / 27.1, 67.6 / 67.6.
    // 65 to 128 query blocks at D = 64 alike (at D = 128 the wider accumulator spills: 3 000 tokens of 4 x 32 heads, 96 blocks 57.5 / 59.0 us of pre-pass).  Pre-pass: 16 000 tokens of
    // 2 x 32 heads 211.7 / 192.3, 9 000 of 40 71.5 / 64.5, 4 000 of 8 x 32 (8 kv heads) 84.3 / 81.7, of 2 x 32 (512 tiles) 26.7 / 24.8, 4 096 of 32 (256) 18.4 / 16.8; between two and three 2 600
    // of 2 x 32 (336) 18.6 / 20.5, 3 400 (432) 22.5 / 22.6.
    const bool runs = D == 64 ? rows <= 128 && (tiles > 3 * info.sms || (rows > 32 && tiles > info.sms && tiles <= 2 * info.sms)) : rows <= 64 && tiles > info.sms;
    if (!runs) return rows > 64 ? one_tile(std::integral_constant<int, 128>()) : one_tile(std::integral_constant<int, 64>());
    if constexpr (D == 64)
        if (rows > 64) return run(std::integral_constant<int, 128>());
    return rows > 32 ? run(std::integral_constant<int, 64>()) : run(std::integral_constant<int, 32>());
}

cudaError_t launch_prepass(const PrepassArgs& a, cudaStream_t st) {
    if (a.is_bf16) {
        return a.D == 128 ? launch_prepass_t<__nv_bfloat16, 128>(a, st) : launch_prepass_t<__nv_bfloat16, 64>(a, st);
    }
    return a.D == 128 ? launch_prepass_t<__half, 128>(a, st) : launch_prepass_t<__half, 64>(a, st);
}

}  // namespace sage3

// ------------------------------------------------------------------------------------------------
// K mean without any allocation by anybody: the partial column sums live in a static device array
// ------------------------------------------------------------------------------------------------
namespace {

// Scratch for sage3_kmean_noalloc: partial column sums [B*Hkv][chunks][D] in fp32.  Every GPU that loads this
// library holds these 4 MiB until the process exits.  Inside host code this name is only a stand-in for the
// device array; the device address is obtained once per device with cudaGetSymbolAddress (below).
static __device__ __align__(256) float g_kmean_scratch[SAGE3_KMEAN_NOALLOC_MAX_FLOATS];

constexpr int kMaxDevices = 64;
std::mutex g_scratch_mutex;
float* g_scratch_addr[kMaxDevices] = {};   // device address of g_kmean_scratch on each device, once resolved

// Device address of the scratch array on the current device; resolved on the first call per device.
int scratch_for_current_device(float** out) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return SAGE3_E_CUDA;
    if (dev < 0 || dev >= kMaxDevices) return SAGE3_E_TOO_LARGE;
    std::lock_guard<std::mutex> lock(g_scratch_mutex);
    if (g_scratch_addr[dev] == nullptr) {
        void* p = nullptr;
        if (cudaGetSymbolAddress(&p, g_kmean_scratch) != cudaSuccess || p == nullptr) return SAGE3_E_CUDA;
        g_scratch_addr[dev] = static_cast<float*>(p);
    }
    *out = g_scratch_addr[dev];
    return SAGE3_OK;
}

template <typename T, int D>
cudaError_t launch_kmean_t(const Sage3Desc* d, const void* k, void* km, float* scratch, int chunks, cudaStream_t st) {
    const int BH = d->B * d->Hkv;
    sage3::PartsPtr one = {};
    one.base[0] = const_cast<void*>(k);
    const cudaError_t e = sage3::launch(false, sage3::colsum_partial_kernel<T, D>, dim3(chunks, BH), dim3(256), 0, st, sage3::make_src<T>(one),
                                        d->k_stride[0], d->k_stride[1], d->k_stride[2], sage3::FastDiv(d->Hkv), d->Nk, scratch, chunks);
    if (e != cudaSuccess) return e;
    return sage3::launch(false, sage3::colmean_finalize_kernel<T, D>, dim3(BH), dim3(D), 0, st, (const float*)scratch, chunks,
                         1.0f / (float)d->Nk, static_cast<T*>(km), (const int*)nullptr, d->Hkv, 0);
}

}  // namespace

// Column means from partial column sums: mean[r][d] = round(dtype, (sum over c, in order, of part[r][c][d]) * (1 / count)).
// The second half of the K-mean stage on its own, for callers that gather the partial sums of several token shards
// (one 512-row chunk after the other, shard after shard) and need the mean the single call forms, bit for bit.
extern "C" SAGE3_API int sage3_mean_from_partial_sums(const float* part, int32_t rows, int32_t chunks, int32_t D, int32_t dtype,
                                                      int64_t count, void* mean_out, void* stream) {
    if (!part || !mean_out) return SAGE3_E_NULL;
    if (rows <= 0 || chunks <= 0 || count <= 0 || (D != 64 && D != 128)) return SAGE3_E_SHAPE;
    if (dtype != SAGE3_FP16 && dtype != SAGE3_BF16) return SAGE3_E_DTYPE;
    if ((reinterpret_cast<uintptr_t>(part) % 4) != 0 || (reinterpret_cast<uintptr_t>(mean_out) % 2) != 0) return SAGE3_E_ALIGN;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const float inv = 1.0f / (float)count;
    if (dtype == SAGE3_BF16) {
        if (D == 128) sage3::colmean_finalize_kernel<__nv_bfloat16, 128><<<rows, 128, 0, st>>>(part, chunks, inv, static_cast<__nv_bfloat16*>(mean_out), nullptr, 1, 0);
        else sage3::colmean_finalize_kernel<__nv_bfloat16, 64><<<rows, 64, 0, st>>>(part, chunks, inv, static_cast<__nv_bfloat16*>(mean_out), nullptr, 1, 0);
    } else {
        if (D == 128) sage3::colmean_finalize_kernel<__half, 128><<<rows, 128, 0, st>>>(part, chunks, inv, static_cast<__half*>(mean_out), nullptr, 1, 0);
        else sage3::colmean_finalize_kernel<__half, 64><<<rows, 64, 0, st>>>(part, chunks, inv, static_cast<__half*>(mean_out), nullptr, 1, 0);
    }
    return cudaGetLastError() == cudaSuccess ? SAGE3_OK : SAGE3_E_CUDA;
}

extern "C" SAGE3_API int sage3_kmean_noalloc(const Sage3Desc* desc, const void* k, void* km_out, void* stream) {
    if (!desc || !k || !km_out) return SAGE3_E_NULL;
    if (desc->B <= 0 || desc->Hkv <= 0 || desc->Nk <= 0 || (desc->D != 64 && desc->D != 128)) return SAGE3_E_SHAPE;
    if (desc->dtype != SAGE3_FP16 && desc->dtype != SAGE3_BF16) return SAGE3_E_DTYPE;
    for (int i = 0; i < 3; ++i)
        if (desc->k_stride[i] < 0 || (desc->k_stride[i] % 8) != 0) return SAGE3_E_STRIDE;
    if ((reinterpret_cast<uintptr_t>(k) % 16) != 0 || (reinterpret_cast<uintptr_t>(km_out) % 2) != 0) return SAGE3_E_ALIGN;
    const int64_t chunks = ((int64_t)desc->Nk + sage3::kRowsPerChunk - 1) / sage3::kRowsPerChunk;
    const int64_t need = (int64_t)desc->B * desc->Hkv * chunks * desc->D;
    if (need > (int64_t)SAGE3_KMEAN_NOALLOC_MAX_FLOATS || chunks > 65535) return SAGE3_E_TOO_LARGE;
    int dev = 0, major = 0, minor = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&minor, cudaDevAttrComputeCapabilityMinor, dev) != cudaSuccess)
        return SAGE3_E_CUDA;
    if (major != 10 || minor != 0) return SAGE3_E_ARCH;
    float* scratch = nullptr;
    const int rc = scratch_for_current_device(&scratch);
    if (rc != SAGE3_OK) return rc;
    // Nothing in the scratch has to start at zero: every partial sum the finalize step reads is written by the
    // first kernel of this very call.
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    cudaError_t e;
    if (desc->dtype == SAGE3_BF16)
        e = desc->D == 128 ? launch_kmean_t<__nv_bfloat16, 128>(desc, k, km_out, scratch, (int)chunks, st)
                           : launch_kmean_t<__nv_bfloat16, 64>(desc, k, km_out, scratch, (int)chunks, st);
    else
        e = desc->D == 128 ? launch_kmean_t<__half, 128>(desc, k, km_out, scratch, (int)chunks, st)
                           : launch_kmean_t<__half, 64>(desc, k, km_out, scratch, (int)chunks, st);
    return e == cudaSuccess ? SAGE3_OK : SAGE3_E_CUDA;
}
