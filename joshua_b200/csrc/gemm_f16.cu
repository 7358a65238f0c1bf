// Prefill / batched matmul (from five rows on) over raw GGUF blocks on the 5th-generation tensor cores, in half precision
// terms that keep f32's precision.
//
// dst[m, n] = lhs[m, k] . W[n, k]^T with W left in its GGUF bytes.  A CTA owns 128 rows of W and up to N_TILE rows of
// lhs.  Per window of 256 columns (one super-block of the K formats) the weights of a row are one f32 factor times
// numbers that f16 holds exactly, or as two terms:
//
//   Q4_K, Q2_K   d  * (scale * code)            <= 945, 45: one term; the minima below
//   IQ2_XXS      d/8 * (2 s + 1) * (+-grid)     <= 1333: one term
//   MXFP4        2^(e_max - 139) * (E2M1 * 2^(e - e_max + 12))   one term
//   Q8_0         2^p * (code * d_block / 2^p)   18 bits: two terms, the second by an exact fused multiply-subtract
//   Q6_K         d  * (scale * code)            13 bits: two terms
//
// f16 has 40 powers of two.  What lies further apart than that inside one factor (MXFP4 blocks 2^-35 below the largest
// beside them, Q8_0 blocks 2^-22 below it, a dmin 2^28 times d or 2^-9 of it) would lose bits: such a block, or such a
// window of the K formats, is converted as zeros, and the CTA that met one adds its f32 weights' products at the end on
// the CUDA cores (`add_lost`).  Weights of one layer do not differ that much; the check rides in branches not taken.
//
// The activations are split once per launch (`split_f16_kernel`): a row is scaled by a power of two that puts its largest
// value just below 2^15, hi = f16(x), lo = f16(x - hi): 22 to 24 bits of every value within 2^17 of the largest one, an
// absolute error below 2^-39 of it otherwise.  A window whose own largest value lies more than 2^8 below the row's (an
// outlier elsewhere) is scaled further by itself, so the error stays below 2^-31 of the window's largest value (the int8
// planes of the decode kernel, scaled over the same 256 values: 2^-24 of it), and the read-back undoes that scale token
// by token.  Rows with such a window say so by the sign of their scale; a tile without one, the usual one, never asks.
// The tensor core's products of f16 terms are exact; two or three products (hi*hi, hi*lo, lo*hi) replace three TF32
// products (gemm_tc.cu) at twice their rate: 32 to 48 instructions per window instead of 96.
//
// Minima (Q4_K, Q2_K): sum_c dmin m_g x_c = sum_g (dmin m_g) (sum of x over the group), an inner product of 16 terms per
// window.  The split kernel also writes the sums of each 16 values, times 2^-5 so that they fit, as two f16 terms, the
// converters write -2^5 (dmin / f) m_g as two f16 terms, and three more instructions add their product to the same
// accumulator.
//
// The tensor core adds into its f32 accumulator with truncation, an error that grows with the instructions behind one
// another, so accumulators are short and the converter warps read them back with tcgen05.ld and add f * acc,
// round-to-nearest, to running sums in registers.  Tiles of 128 rows of lhs: one accumulator per window, two of them
// in turn, a column share for every warp.  Tiles of up to 32 rows are as exact as the decode kernel's integer sums:
// every 64 columns have an accumulator (the small products first, then four instructions of full size), read back by
// the warps that converted the columns, whose four partial tiles meet in shared memory at the end.
//
// Tensor memory, 512 columns: the accumulators, then stages of 64 weights: 32 columns of first terms (two per column)
// and 32 of second terms where the type has them, weight row r in lane r; then 16 columns of minima per window in
// flight.  The activation ring in shared memory has the same stages, 64 columns of k each.  A window is four stages;
// narrow tiles keep two windows in flight, because their products take less time than a conversion.
//
// Order of k inside four columns: 0, 2, 1, 3, for the activations and the weights alike, so that a mask picks two
// codes out of a word of nibbles or bytes.  MXFP4: i, i + 16 of a block, the two nibbles of a byte, which one instruction
// converts.
//
// What bounds it: the converters' chain and its issue slots; a window of a tile is 7 700 warp instructions at 128 rows, at 2.0 a
// cycle (Q4_K 28672 x 4096, 512 rows: the tensor pipe 59 % of the active cycles).
//
// Warps: 16 converters, warp (q = w % 4, g = w / 4) owns weight rows 32q .. 32q+31 (the tensor-memory lanes it may touch) and
// the columns 64g .. 64g+63 of every window.  Warps 16 to 19 issue the MMAs and the TMA copies: an instruction takes about 30
// cycles to issue, so narrow tiles have an issuer per step, which also copies its step's activation tiles; wide ones, whose
// steps share an accumulator, have one, and another warp copies.  Warps 20 to 23 copy raw weights (cp.async, eight lanes a
// row, so that an address serves all of a row's vectors; a whole window completes on one mbarrier): when the converters
// copied their own rows and met on a named barrier, that was an eighth of their instructions and a fifth of their waits.
// Against that form, and with the issuer of wide tiles waiting for its next step between the halves of the one it issues:
// Q2_K 4096 x 14336, 333 rows 146 -> 121 us, Q4_K 28672 x 4096, 512 rows 250 -> 239 (at 1.4 GHz under the power cap) and
// 4096 x 14336 127 -> 122, Q8_0 5120 x 2048, 1000 rows 86 -> 81, Q4_K 28672 x 4096, 16 rows 50.5 -> 47.3.  MXFP4, whose nibbles
// one conversion instruction a pair now unpacks (64 a cycle and SM) instead of three byte permutes and masks: 28672 x 7168,
// 20 / 64 / 200 rows 102 / 203 / 252 -> 76 / 150 / 206 us.  It costs launches of one or two windows a CTA 0.2 to 0.9 us
// (Q4_K 2048 x 4096, 33 rows 13.3 -> 13.8; Q6_K, whose rows are copied by the word, 2048 x 4096, 33 rows 15.4 -> 16.3, 4096 x 4096
// 20 rows 15.4 -> 15.9, 128 rows 46.7 -> 43.4).
// Two further forms were slower: an owner per window instead of per step (half the instructions, but a chain of single warps:
// 28672 x 4096, 16 rows 56 us) and a persistent loop over tiles on top of it.
//
// Few tiles (small n, or few rows of lhs) leave SMs idle: then a cluster of S CTAs splits k, every CTA leaves its
// partial tile in its shared memory, and each adds a share of the tile over the cluster in rank order (distributed
// shared memory), so results do not depend on timing.
//
// Every wait on an mbarrier is bounded; a wait that runs out raises the device status flag, and every thread still
// reaches the common exit where tensor memory is released.  Running out takes seconds; copies and products that were in
// flight when progress stopped have landed long before.
#include <algorithm>
#include <type_traits>

#include <cudaTypedefs.h>

#include "common.cuh"
#include "tc5.cuh"

namespace jq {

cudaError_t tables_gemm_f16() { return upload_tables(); }

namespace {

constexpr int HM = 128;           // weight rows per CTA = MMA M = TMEM lanes
constexpr int H_CONV = 16;        // converter / epilogue warps
constexpr int H_ISSUE = 4;        // issuing warps: one per 64-column step where the steps have their own accumulators
constexpr int H_COPY = 4;         // warps that copy raw weights
constexpr int H_THREADS = (H_CONV + H_ISSUE + H_COPY) * 32;
// Registers a thread: the launch has 768 x 80 = 61440; the converters take 512 x 96 of them, the others 256 x 48.
constexpr int H_REGS_CONV = 96, H_REGS_REST = 48;
static_assert(H_CONV * 32 * H_REGS_CONV + (H_ISSUE + H_COPY) * 32 * H_REGS_REST <= H_THREADS * 80, "registers");
constexpr uint32_t H_STEPS = 4;   // 64-column steps per 256-column window = ring stages

template <uint32_t TYPE>
struct HT;  // UNIT: bytes of 256 columns of a row; UNITS: windows staged together (whole 32-bit words); VEC: bytes a copy
template <>
struct HT<T_Q4_K> {
    static constexpr uint32_t UNIT = 144, UNITS = 1, VEC = 16;
    static constexpr bool TWO = false, MIN = true, LOSES = true;
};
template <>
struct HT<T_Q2_K> {
    static constexpr uint32_t UNIT = 84, UNITS = 1, VEC = 4;
    static constexpr bool TWO = false, MIN = true, LOSES = true;
};
template <>
struct HT<T_IQ2_XXS> {
    static constexpr uint32_t UNIT = 66, UNITS = 2, VEC = 4;
    static constexpr bool TWO = false, MIN = false, LOSES = false;
};
template <>
struct HT<T_MXFP4> {
    static constexpr uint32_t UNIT = 136, UNITS = 1, VEC = 8;
    static constexpr bool TWO = false, MIN = false, LOSES = true;
};
template <>
struct HT<T_Q8_0> {
    static constexpr uint32_t UNIT = 272, UNITS = 1, VEC = 8;
    static constexpr bool TWO = true, MIN = false, LOSES = true;
};
template <>
struct HT<T_Q6_K> {
    static constexpr uint32_t UNIT = 210, UNITS = 2, VEC = 4;
    static constexpr bool TWO = true, MIN = false, LOSES = false;
};
// Row stride of the staged bytes in words.  Rows copied by the word: odd, so that 32 lanes reading the same word of their
// rows hit 32 banks.  Q4_K rows are read as 16-byte vectors, which 36 words spread over the banks; rows copied by
// eight bytes take 34 or 70 words, two lanes a bank.
template <uint32_t TYPE>
constexpr uint32_t raw_stride() {
    constexpr uint32_t words = HT<TYPE>::UNIT * HT<TYPE>::UNITS / 4;
    return HT<TYPE>::VEC == 4 ? words | 1u : HT<TYPE>::VEC == 8 && words % 4 == 0 ? words + 2 : words;
}
// Shape of a tile: windows in flight, buffers of raw bytes (narrow tiles stream weights at memory speed and want tens
// of kilobytes on their way), accumulators.
template <uint32_t TYPE, int N_TILE>
struct Tile {
    static constexpr bool FINE = N_TILE <= 32;
    static constexpr int NB = FINE ? 2 : 8;  // blocks of 32 columns behind one accumulator
    static constexpr uint32_t WINDOWS = N_TILE <= 32 && !HT<TYPE>::TWO ? 2 : 1;
    static constexpr uint32_t STAGES = H_STEPS * WINDOWS;
    static constexpr uint32_t ACCS = FINE ? H_STEPS : 2;
    static constexpr uint32_t ACC_COLS = ACCS * N_TILE;
    static constexpr uint32_t A_COLS = HT<TYPE>::TWO ? 64 : 32;
    static constexpr uint32_t MIN_COL0 = ACC_COLS + STAGES * A_COLS;
    static_assert(MIN_COL0 + (HT<TYPE>::MIN ? 16 * WINDOWS : 0) <= 512, "tensor memory");
    static constexpr uint32_t PLANE_B = N_TILE * 128;  // 64 f16 columns of N_TILE rows
    static constexpr uint32_t STAGE_B = 2 * PLANE_B;   // hi | lo
    static constexpr uint32_t RAW_BUF = HM * raw_stride<TYPE>() * 4;
    static constexpr uint32_t SCALE_B = H_CONV * 32 * 16;  // every converter warp's tokens: what scales of windows need
    static constexpr uint32_t FIXED = STAGES * STAGE_B + (HT<TYPE>::MIN ? WINDOWS * PLANE_B : 0) +
                                      (TYPE == T_IQ2_XXS ? 2048 : 0) + SCALE_B + 1024;
    static constexpr uint32_t ROOM = (226 * 1024 - FIXED) / RAW_BUF;
    static constexpr uint32_t WANT = N_TILE <= 32 ? 4 : 2;
    static constexpr uint32_t BUFS = ROOM < WANT ? ROOM : WANT;
    static_assert(BUFS >= 2, "shared memory");
    static constexpr uint32_t LOOP_SMEM = FIXED + BUFS * RAW_BUF;
    static constexpr uint32_t RED_SMEM = (FINE ? 4 : 1) * N_TILE * HM * 4 + 1024;  // the partial tiles at the end
    static constexpr uint32_t SMEM = LOOP_SMEM > RED_SMEM ? LOOP_SMEM : RED_SMEM;
    static_assert(SMEM <= 226 * 1024, "shared memory");
};

// ── activations ──
// One CTA per row; a thread takes 16 consecutive values at a time, half a warp a window.  hi / lo [m][k];
// sums [m][k / 256][32]: the 16 group sums of a window, first terms then second terms; inv[m]: the inverse of the row's
// scale, negative where some window has one of its own; rel[k / 256][m]: the inverse of that.  With norm_w (KEEP = 0) the
// rows are RMS-normalised first: the values split are x * rs * norm_w.  With a list, row r is row list[r] of x, and rows from
// *n_list on stay as they are.  KEEP: 16-value groups that a thread holds between finding the largest value and splitting;
// 0 reads them twice.  Bound by memory, and for short rows by the CTAs that an SM holds, so that a CTA is no wider than its
// row.  Q4_K 4096 x 14336 at 13 rows 26.8 -> 24.8 us with the product; a routed layer of 1000 tokens, eight experts each, 14 us
// less by the copy of the listed rows that stood before.
template <int THREADS, int KEEP>
__global__ void __launch_bounds__(THREADS) split_f16_kernel(const float* __restrict__ x, uint32_t k,
                                                            const float* __restrict__ norm_w, float eps,
                                                            const uint32_t* __restrict__ list, const uint32_t* __restrict__ n_list,
                                                            int nibble_pairs, __half* __restrict__ hi,
                                                            __half* __restrict__ lo, __half* __restrict__ sums,
                                                            float* __restrict__ inv, float* __restrict__ rel) {
    constexpr int WARPS = THREADS / 32;
    __shared__ float s_max[WARPS], s_sq[WARPS];
    pdl_trigger();
    pdl_wait();
    const uint32_t row = blockIdx.x, tid = threadIdx.x, groups = k / 16;
    if (list != nullptr && row >= *n_list) return;
    const float4* xr = reinterpret_cast<const float4*>(x + (uint64_t)(list ? list[row] : row) * k);
    // vector j of group g: 16 values in a row, or 0 .. 7 and 16 .. 23 (8 .. 15 and 24 .. 31) of 32
    auto place = [&](uint32_t g, int j) {
        return nibble_pairs ? 8 * (g >> 1) + 2 * (g & 1) + 4 * (j >> 1) + (j & 1) : 4 * g + j;
    };
    auto largest = [](float m, const float4& v) { return fmaxf(m, fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w)))); };
    float4 kept[KEEP > 0 ? KEEP : 1][4];
    const float4* nr = reinterpret_cast<const float4*>(norm_w);
    float row_max = 0.0f, sq = 0.0f;
    if constexpr (KEEP > 0) {
#pragma unroll
        for (int i = 0; i < KEEP; ++i)
            if (const uint32_t g = tid + i * THREADS; g < groups) {
#pragma unroll
                for (int j = 0; j < 4; ++j) kept[i][j] = __ldg(xr + place(g, j));
            }
#pragma unroll
        for (int i = 0; i < KEEP; ++i)
            if (tid + i * THREADS < groups) {
#pragma unroll
                for (int j = 0; j < 4; ++j) row_max = largest(row_max, kept[i][j]);
            }
    } else {
#pragma unroll 4
        for (uint32_t i = tid; i < k / 4; i += THREADS) {
            float4 v = __ldg(xr + i);
            if (norm_w) {
                sq = fmaf(v.x, v.x, fmaf(v.y, v.y, fmaf(v.z, v.z, fmaf(v.w, v.w, sq))));
                const float4 g = __ldg(nr + i);
                v.x *= g.x, v.y *= g.y, v.z *= g.z, v.w *= g.w;
            }
            row_max = largest(row_max, v);
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        row_max = fmaxf(row_max, __shfl_xor_sync(0xFFFFFFFFu, row_max, o));
        sq += __shfl_xor_sync(0xFFFFFFFFu, sq, o);
    }
    if ((tid & 31) == 0) s_max[tid >> 5] = row_max, s_sq[tid >> 5] = sq;
    __syncthreads();
    row_max = s_max[0], sq = s_sq[0];
#pragma unroll
    for (int i = 1; i < WARPS; ++i) row_max = fmaxf(row_max, s_max[i]), sq += s_sq[i];
    const float rs = norm_w ? rsqrtf(sq / (float)k + eps) : 1.0f;
    // scale 2^(141 - e): the largest value lands in [2^14, 2^15) (a rounding of the norm aside).  Clamped where the scale
    // itself would leave f32 (below 2^-113); infinities keep theirs.
    auto scale_bits = [](float amax) {
        const uint32_t e = __float_as_uint(amax) >> 23;
        return e == 255 ? 127u : min(254u, 268u - e);
    };
    const uint32_t row_bits = scale_bits(row_max * rs);
    bool own = false;  // a window of this thread has a scale of its own
    auto split_group = [&](uint32_t g, const float4 (&val)[4]) {  // groups is a multiple of 16: whole half-warps
        float amax = 0.0f;
#pragma unroll
        for (int j = 0; j < 4; ++j) amax = largest(amax, val[j]);
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xFFFFu << (tid & 16), amax, o));
        int extra = amax == 0.0f ? 0 : (int)scale_bits(amax) - (int)row_bits;
        extra = extra <= 8 ? 0 : min(extra, 60);
        own |= extra != 0;
        const float scale = __uint_as_float((row_bits + extra) << 23);
        if ((g & 15) == 0) rel[(uint64_t)(g >> 4) * gridDim.x + row] = __uint_as_float((uint32_t)(127 - extra) << 23);
        uint32_t h[8], l[8];
        float sum = 0.0f;
        float f[16];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float4 v = val[j];
            f[4 * j] = v.x * scale, f[4 * j + 1] = v.y * scale, f[4 * j + 2] = v.z * scale, f[4 * j + 3] = v.w * scale;
            sum += (f[4 * j] + f[4 * j + 1]) + (f[4 * j + 2] + f[4 * j + 3]);
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int p = 4 * (j >> 1) + (j & 1);  // 0, 2 and 1, 3 of four
            const float x0 = nibble_pairs ? f[j] : f[p], x1 = nibble_pairs ? f[8 + j] : f[p + 2];
            const __half2 t = __floats2half2_rn(x0, x1);
            const float2 back = __half22float2(t);
            const __half2 rest = __floats2half2_rn(x0 - back.x, x1 - back.y);
            h[j] = *reinterpret_cast<const uint32_t*>(&t), l[j] = *reinterpret_cast<const uint32_t*>(&rest);
        }
        uint4* hp = reinterpret_cast<uint4*>(hi + (uint64_t)row * k + 16 * g);
        uint4* lp = reinterpret_cast<uint4*>(lo + (uint64_t)row * k + 16 * g);
        hp[0] = make_uint4(h[0], h[1], h[2], h[3]), hp[1] = make_uint4(h[4], h[5], h[6], h[7]);
        lp[0] = make_uint4(l[0], l[1], l[2], l[3]), lp[1] = make_uint4(l[4], l[5], l[6], l[7]);
        sum *= 0.03125f;  // 16 values below 2^15: at most 2^14
        const __half sh = __float2half_rn(sum);
        __half* sp = sums + ((uint64_t)row * (k / 256) + (g >> 4)) * 32 + (g & 15);
        sp[0] = sh;
        sp[16] = __float2half_rn(sum - __half2float(sh));
    };
    if constexpr (KEEP > 0) {
#pragma unroll
        for (int i = 0; i < KEEP; ++i)
            if (tid + i * THREADS < groups) split_group(tid + i * THREADS, kept[i]);
    } else {
        for (uint32_t g = tid; g < groups; g += THREADS) {
            float4 val[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const uint32_t at = place(g, j);
                val[j] = __ldg(xr + at);
                if (norm_w) {
                    const float4 w = __ldg(nr + at);
                    val[j].x = val[j].x * rs * w.x, val[j].y = val[j].y * rs * w.y, val[j].z = val[j].z * rs * w.z, val[j].w = val[j].w * rs * w.w;
                }
            }
            split_group(g, val);
        }
    }
    const int any_own = __syncthreads_or(own);
    if (tid == 0) {
        const float v = row_bits == 254 ? __uint_as_float(0x00400000u) : __uint_as_float((254u - row_bits) << 23);
        inv[row] = any_own ? -v : v;
    }
}

// ── weights: 32 columns of a row -> packed f16 terms ──
__device__ __forceinline__ uint32_t s32(uint32_t addr) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr));
    return v;
}
__device__ __forceinline__ uint32_t s16(uint32_t addr) {
    uint32_t v;
    asm volatile("{\n\t.reg .u16 t;\n\tld.shared.u16 t, [%1];\n\tcvt.u32.u16 %0, t;\n\t}" : "=r"(v) : "r"(addr));
    return v;
}
__device__ __forceinline__ uint32_t s8(uint32_t addr) { return (s32(addr & ~3u) >> ((addr & 3u) * 8)) & 0xFFu; }
__device__ __forceinline__ uint4 s128(uint32_t addr) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
    return v;
}
// N consecutive words from any byte address
template <int N>
__device__ __forceinline__ void s_words(uint32_t addr, uint32_t (&w)[N]) {
    const uint32_t al = addr & ~3u, sh = (addr & 3u) * 8;
    uint32_t prev = s32(al);
#pragma unroll
    for (int i = 0; i < N; ++i) {
        // the word behind an aligned run may lie outside the row: it is not needed and not read
        const uint32_t next = (i + 1 < N || sh) ? s32(al + 4 * (i + 1)) : 0u;
        w[i] = __funnelshift_r(prev, next, sh);
        prev = next;
    }
}
__device__ __forceinline__ __half2 as_h2(uint32_t v) { return *reinterpret_cast<__half2*>(&v); }
__device__ __forceinline__ uint32_t as_u32(__half2 v) { return *reinterpret_cast<uint32_t*>(&v); }
// Bytes 0 and 2, and 1 and 3, of a word of values below 256 as two half2 of 1024 + byte: exact, and one fused
// multiply-add away from scale * byte.
__device__ __forceinline__ void bytes_1024(uint32_t b, __half2* even, __half2* odd) {
    *even = as_h2(__byte_perm(b, 0x64646464u, 0x4240));
    *odd = as_h2(__byte_perm(b, 0x64646464u, 0x4341));
}
// (w & mask) | bits
__device__ __forceinline__ uint32_t and_or(uint32_t w, uint32_t mask, uint32_t bits) {
    uint32_t r;
    asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(r) : "r"(w), "r"(mask), "r"(bits));
    return r;
}
// a small integer (0..255) in both halves, exact
__device__ __forceinline__ __half2 int_h2(uint32_t v) {
    return __hsub2(as_h2(__byte_perm(v, 0x64646464u, 0x4040)), __float2half2_rn(1024.0f));
}
__device__ __forceinline__ float pow2_f32(int e) {  // 2^e for -149 <= e <= 127
    return e >= -126 ? __uint_as_float((uint32_t)(e + 127) << 23) : __uint_as_float(1u << (e + 149));
}

// Per window and row: the f32 factor of the accumulated products, and what the terms need of it.
struct RowWin {
    float f;       // result = f * accumulator
    float aux;     // Q4_K / Q2_K: scale of the codes (a power of two); Q8_0: 1 / f; MXFP4: e_max
    float d, dmin; // Q4_K / Q2_K
    bool lost;     // Q4_K / Q2_K: the window is converted as zeros
};

// The codes' factor f = d 2^e.  Usually e = 0; where dmin is 32 times d or more the codes are scaled down by 2^-e
// (exact, f16 has subnormals down to 2^-24) so that the minima stay inside f16: |2^5 dmin / f * m| <= 1024 * 63.
// Below 2^-9 of d the minima's second terms would end in f16's subnormals, above 2^28 the codes.
__device__ __forceinline__ RowWin min_factors(uint32_t dd) {
    const float d = f16_bits_to_f32(dd & 0xFFFF), dmin = f16_bits_to_f32(dd >> 16), ad = fabsf(d), am = fabsf(dmin);
    if (dmin == 0.0f || !(am >= 32.0f * ad || am < ad * (1.0f / 512.0f)) || ad > 65504.0f) return {d, 1.0f, d, dmin, false};
    if (d == 0.0f) return {dmin * (1.0f / 16.0f), 0.0f, d, dmin, false};
    const int e = (int)(__float_as_uint(am / ad) >> 23) - 127 - 4;
    if (e < 0 || e > 24) return {d, 0.0f, d, 0.0f, true};
    return {d * pow2_f32(e), pow2_f32(-e), d, dmin, false};
}
// Q8_0: the largest |d| / f lies in [128, 256), codes times it stay below 2^15.  mx: the largest |d|'s bits
__device__ __forceinline__ int q8_power(uint32_t mx) {
    return mx == 0 ? 0 : (int)(__float_as_uint(f16_bits_to_f32(mx)) >> 23) - 127 - 7;
}
__device__ __forceinline__ bool q8_lost(float ratio) { return ratio != 0.0f && fabsf(ratio) < 6.103515625e-5f; }  // |d| / f < 2^-14
// MXFP4: 2^(e - e_max + 12) is the unit, half of it the smallest value.
__device__ __forceinline__ bool mxfp4_lost(uint32_t e, uint32_t mx) { return e + 35 < mx; }

// NB blocks of 32 columns have one factor (MXFP4, Q8_0): eight, or the two of a step with its own accumulator.
// u: shared address of the row's 256 columns, b0: the first of the blocks.
template <uint32_t TYPE, int NB>
__device__ __forceinline__ RowWin row_window(uint32_t u, uint32_t b0) {
    if constexpr (TYPE == T_Q4_K) {
        return min_factors(s32(u));
    } else if constexpr (TYPE == T_Q2_K) {
        return min_factors(s32(u + 80));
    } else if constexpr (TYPE == T_IQ2_XXS) {
        return {f16_bits_to_f32(s16(u)) * 0.125f, 0.0f, 0.0f, 0.0f, false};
    } else if constexpr (TYPE == T_Q6_K) {
        return {f16_bits_to_f32(s16(u + 208)), 0.0f, 0.0f, 0.0f, false};
    } else if constexpr (TYPE == T_Q8_0) {
        uint32_t mx = 0;
#pragma unroll
        for (int b = 0; b < NB; ++b) mx = max(mx, s16(u + 34 * (b0 + b)) & 0x7FFFu);
        const int p = q8_power(mx);
        return {pow2_f32(p), pow2_f32(-p), 0.0f, 0.0f, false};
    } else {
        uint32_t mx = 0;
#pragma unroll
        for (int b = 0; b < NB; ++b) {
            const uint32_t e = s8(u + 17 * (b0 + b));
            mx = max(mx, e == 255u ? 0u : e);
        }
        return {pow2_f32((int)mx - 139), (float)mx, 0.0f, 0.0f, false};
    }
}
// Whether row_window / convert64 leave block b of a row's window, in global memory, to add_lost.
template <uint32_t TYPE, int NB>
__device__ bool block_lost(const uint8_t* win, uint32_t b) {
    const uint32_t b0 = b / NB * NB;
    if constexpr (TYPE == T_Q4_K || TYPE == T_Q2_K) {
        return min_factors(ld_u32(win + (TYPE == T_Q4_K ? 0 : 80))).lost;
    } else if constexpr (TYPE == T_Q8_0) {
        uint32_t mx = 0;
#pragma unroll 1
        for (uint32_t i = b0; i < b0 + NB; ++i) mx = max(mx, ld_u16(win + 34 * i) & 0x7FFFu);
        return q8_lost(f16_bits_to_f32(ld_u16(win + 34 * b)) * pow2_f32(-q8_power(mx)));
    } else {
        uint32_t mx = 0;
#pragma unroll 1
        for (uint32_t i = b0; i < b0 + NB; ++i) {
            const uint32_t e = ld_u8(win + 17 * i);
            mx = max(mx, e == 255u ? 0u : e);
        }
        return mxfp4_lost(ld_u8(win + 17 * b), mx);
    }
}

// Columns 64 g .. 64 g + 63 of the window: h = 0, 1 are its two groups of 32; put(h, a, b) takes 16 packed first terms
// and (two-term types) 16 second terms.  *lost (shared memory) is set where a block was converted as zeros.
template <uint32_t TYPE, class Put>
__device__ __forceinline__ void convert64(uint32_t u, uint32_t g, const RowWin& rw, const uint2* s_grid, volatile int* lost, Put put) {
    if constexpr (TYPE == T_Q4_K || TYPE == T_Q2_K) {
        if (rw.lost) *lost = 1;
    }
    if constexpr (TYPE == T_Q4_K) {
        const uint4 hd = s128(u), v0 = s128(u + 16 + 32 * g), v1 = s128(u + 32 + 32 * g);
        const uint32_t w[8] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
        // scales of pairs 2g and 2g + 1 in bytes 0 and 1
        const uint32_t j = 16 * (g & 1);
        const uint32_t sc = g < 2 ? (hd.y >> j) & 0x3F3Fu : ((hd.w >> j) & 0x0F0Fu) | ((hd.y >> (j + 2)) & 0x3030u);
        const __half2 aux = __float2half2_rn(rw.aux);
#pragma unroll
        for (uint32_t h = 0; h < 2; ++h) {
            // low nibbles: 1024 + q; high nibbles in place: 64 + q (their unit is 1/16 of 64's last place)
            const uint32_t mask = h ? 0x00F000F0u : 0x000F000Fu, bits = h ? 0x54005400u : 0x64006400u;
            const __half2 s2 = __hmul2(int_h2((sc >> (8 * h)) & 0xFFu), aux), off = __hmul2(s2, __float2half2_rn(h ? -64.0f : -1024.0f));
            uint32_t a[16];
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                a[2 * q] = as_u32(__hfma2(as_h2(and_or(w[q], mask, bits)), s2, off));
                a[2 * q + 1] = as_u32(__hfma2(as_h2(and_or(w[q] >> 8, mask, bits)), s2, off));
            }
            put(h, a, a);
        }
    } else if constexpr (TYPE == T_Q2_K) {
        // 32 bytes of four 2-bit fields; this step takes fields 2 (g % 2) and the next.  Field i in place is q in
        // units of 4^i: 1024 / 4^i + q.
        const uint32_t qb = u + 16 + 32 * (g >> 1), scs = s32(u + 4 * g);
        uint32_t w[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) w[q] = s32(qb + 4 * q);
        const __half2 aux = __float2half2_rn(rw.aux);
#pragma unroll
        for (uint32_t h = 0; h < 2; ++h) {
            const uint32_t i = 2 * (g & 1) + h, mask = 0x00030003u << (2 * i), bits = 0x64006400u - i * 0x08000800u;
            const __half2 base = as_h2(bits | 0x80008000u);
            uint32_t a[16];
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const __half2 s2 = __hmul2(int_h2((scs >> (16 * h + 8 * (q >> 2))) & 15u), aux), off = __hmul2(s2, base);
                a[2 * q] = as_u32(__hfma2(as_h2(and_or(w[q], mask, bits)), s2, off));
                a[2 * q + 1] = as_u32(__hfma2(as_h2(and_or(w[q] >> 8, mask, bits)), s2, off));
            }
            put(h, a, a);
        }
    } else if constexpr (TYPE == T_IQ2_XXS) {
        uint32_t gw[4];
        s_words<4>(u + 2 + 16 * g, gw);
#pragma unroll
        for (uint32_t h = 0; h < 2; ++h) {
            const uint32_t codes = gw[2 * h], sw = gw[2 * h + 1];
            const __half2 s2 = int_h2(2 * (sw >> 28) + 1), off = __hmul2(s2, __float2half2_rn(-1024.0f));
            uint32_t a[16];
#pragma unroll
            for (int l = 0; l < 4; ++l) {
                const uint2 gr = s_grid[(codes >> (8 * l)) & 0xFFu];
                const uint32_t sg = iq2_signs((sw >> (7 * l)) & 127u);
                __half2 v[4];
                bytes_1024(gr.x, &v[0], &v[1]);
                bytes_1024(gr.y, &v[2], &v[3]);
#pragma unroll
                for (int p = 0; p < 4; ++p) {  // values e and e + 2: their sign bits -> bits 15 and 31
                    const int e = 4 * (p >> 1) + (p & 1);
                    a[4 * l + p] = as_u32(__hfma2(v[p], s2, off)) ^ (((sg << (15 - e)) & 0x8000u) | ((sg << (29 - e)) & 0x80000000u));
                }
            }
            put(h, a, a);
        }
    } else if constexpr (TYPE == T_MXFP4) {
#pragma unroll
        for (uint32_t h = 0; h < 2; ++h) {
            const uint32_t blk = u + 17 * (2 * g + h), e = s8(blk);
            uint32_t w[4];
            s_words<4>(blk + 1, w);
            const bool gone = mxfp4_lost(e, (uint32_t)rw.aux);
            const __half2 s2 = __float2half2_rn(e == 255u || gone ? 0.0f : pow2_f32((int)e - (int)rw.aux + 12));
            if (gone && ((w[0] | w[1] | w[2] | w[3]) & 0x77777777u)) *lost = 1;  // a block of zeros has exponent 0
            uint32_t a[16];
#pragma unroll
            for (int q = 0; q < 4; ++q) {  // a byte: values i and i + 16
                uint32_t v[4];
                e2m1_pairs(w[q], v);
#pragma unroll
                for (int j = 0; j < 4; ++j) a[4 * q + j] = as_u32(__hmul2(as_h2(v[j]), s2));
            }
            put(h, a, a);
        }
    } else if constexpr (TYPE == T_Q8_0) {
#pragma unroll
        for (uint32_t h = 0; h < 2; ++h) {
            const uint32_t blk = u + 34 * (2 * g + h);
            const float r = f16_bits_to_f32(s16(blk)) * rw.aux;
            const bool gone = q8_lost(r);
            const __half2 r2 = __float2half2_rn(gone ? 0.0f : r);
            if (gone) *lost = 1;
            uint32_t w[8], a[16], b[16];
            s_words<8>(blk + 2, w);
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                __half2 v[2];
                bytes_1024(w[q] ^ 0x80808080u, &v[0], &v[1]);
#pragma unroll
                for (int p = 0; p < 2; ++p) {
                    const __half2 c = __hsub2(v[p], __float2half2_rn(1152.0f)), hi = __hmul2(c, r2);
                    a[2 * q + p] = as_u32(hi);
                    b[2 * q + p] = as_u32(__hfma2(c, r2, __hneg2(hi)));
                }
            }
            put(h, a, b);
        }
    } else {  // Q6_K: half = g / 2; part = 2 (g % 2) + h takes nibble g % 2 of low run h and bit pair `part`
        uint32_t qh[8];
        s_words<8>(u + 128 + 32 * (g >> 1), qh);
#pragma unroll
        for (uint32_t h = 0; h < 2; ++h) {
            uint32_t ql[8], a[16], b[16];
            s_words<8>(u + 64 * (g >> 1) + 32 * h, ql);
            const uint32_t nsh = 4 * (g & 1), part = 2 * (g & 1) + h;
            const __half2 r[2] = {__float2half2_rn((float)(int8_t)s8(u + 192 + 4 * g + 2 * h)),
                                  __float2half2_rn((float)(int8_t)s8(u + 193 + 4 * g + 2 * h))};
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const uint32_t code = ((ql[q] >> nsh) & 0x0F0F0F0Fu) | (((qh[q] >> (2 * part)) & 0x03030303u) << 4);
                __half2 v[2];
                bytes_1024(code, &v[0], &v[1]);
#pragma unroll
                for (int p = 0; p < 2; ++p) {
                    const __half2 c = __hsub2(v[p], __float2half2_rn(1056.0f)), hi = __hmul2(c, r[q >> 2]);
                    a[2 * q + p] = as_u32(hi);
                    b[2 * q + p] = as_u32(__hfma2(c, r[q >> 2], __hneg2(hi)));
                }
            }
            put(h, a, b);
        }
    }
}

// The products that the tensor core did not form: blocks converted as zeros, their weights in f32 as the float kernels
// decode them, times the split activations.  One warp: its lanes' rows, n_chunks windows from win0 on, steps S0 .. S1 - 1 of
// each, tokens tok0 .. tok0 + n_tok - 1; add(t, v) takes token t's share in units of the row's scale.  Inlined and rolled
// up: as a call it cost the kernel seven per cent where it never ran (Q4_K 28672 x 4096, 8 rows 53.5 us instead of 50.4).
template <uint32_t TYPE, int NB, class Add>
__device__ __forceinline__ void add_lost(const uint8_t* row, uint32_t win0, uint32_t n_chunks, uint32_t S0, uint32_t S1, uint64_t k,
                                      const __half* __restrict__ x_hi, const __half* __restrict__ x_lo,
                                      const float* __restrict__ rel, uint64_t m_rows, uint64_t tok0, uint32_t n_tok, Add add) {
#pragma unroll 1
    for (uint32_t c = win0; c < win0 + n_chunks; ++c) {
        const uint8_t* win = row + (uint64_t)c * HT<TYPE>::UNIT;
#pragma unroll 1
        for (uint32_t b = 2 * S0; b < 2 * S1; ++b) {
            const bool mine = block_lost<TYPE, NB>(win, b);
            if (!__any_sync(0xFFFFFFFFu, mine)) continue;
#pragma unroll 1
            for (uint32_t u = 4 * b; u < 4 * b + 4; ++u) {
                float w[8];
                decode_unit<TYPE>(win, u, w, false);
#pragma unroll 1
                for (uint32_t t = 0; t < n_tok; ++t) {
                    // where the split kernel put the values: 0, 2, 1, 3 of four, or value i of a block's half at 2 i (+ 1)
                    const uint64_t at = (tok0 + t) * k + (uint64_t)c * 256 + (TYPE == T_MXFP4 ? (u & ~3u) * 8 + (u & 1) * 16 + (u >> 1 & 1) : u * 8);
                    float v = 0.0f;
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        const int o = TYPE == T_MXFP4 ? 2 * j : (j & 4) | ((j & 1) << 1) | ((j >> 1) & 1);
                        v = fmaf(w[j], __half2float(x_hi[at + o]) + __half2float(x_lo[at + o]), v);
                    }
                    if (mine) add(t, v * rel[c * m_rows + tok0 + t]);
                }
            }
        }
    }
}

// The window's 16 minima, -2^5 (dmin / f) m, as eight packed first and eight packed second terms.  The ratio is two f16
// terms, m at most six bits: the first products' remainders are exact.
template <uint32_t TYPE>
__device__ __forceinline__ void convert_minima(uint32_t u, const RowWin& rw, uint32_t (&a)[16]) {
    // f is d, d 2^e or (d = 0) dmin / 16
    const float ratio = rw.dmin == 0.0f ? 0.0f : -32.0f * (rw.dmin / rw.f);
    const __half2 rh = __float2half2_rn(ratio), rl = __float2half2_rn(ratio - __low2float(rh));
    const uint4 hd = TYPE == T_Q4_K ? s128(u) : make_uint4(s32(u), s32(u + 4), s32(u + 8), s32(u + 12));
    // Q4_K: eight minima of 32 values, a byte each; Q2_K: sixteen of 16 values in the high nibbles
    const uint32_t m4[4] = {TYPE == T_Q4_K ? hd.z & 0x3F3F3F3Fu : hd.x >> 4 & 0x0F0F0F0Fu,
                            TYPE == T_Q4_K ? (hd.w >> 4 & 0x0F0F0F0Fu) | (hd.z >> 2 & 0x30303030u) : hd.y >> 4 & 0x0F0F0F0Fu,
                            hd.z >> 4 & 0x0F0F0F0Fu, hd.w >> 4 & 0x0F0F0F0Fu};
#pragma unroll
    for (int p = 0; p < 8; ++p) {  // groups of 16 values 2p, 2p + 1
        const uint32_t pair = TYPE == T_Q4_K ? __byte_perm(m4[p >> 2], 0x64646464u, 0x4040 + 0x0101 * (p & 3))
                                             : __byte_perm(m4[p >> 1], 0x64646464u, p & 1 ? 0x4342 : 0x4140);
        const __half2 m = __hsub2(as_h2(pair), __float2half2_rn(1024.0f)), hi = __hmul2(m, rh);
        a[p] = as_u32(hi);
        a[8 + p] = as_u32(__hfma2(m, rl, __hfma2(m, rh, __hneg2(hi))));
    }
}

// Loads of what a kernel in front wrote, for places directly behind pdl_wait: read-only loads (__ldg, or plain ones through
// __restrict__) may be moved above the wait, volatile ones stay.  (The sign of a row's scale, read too early: in one call out
// of eight of 200 rows x 14336 columns a window with a scale of its own, where the call before had none, counted some 500 times.)
__device__ __forceinline__ float ld_behind_wait(const float* p) {
    float v;
    asm volatile("ld.global.cg.f32 %0, [%1];" : "=f"(v) : "l"(p) : "memory");
    return v;
}
// The same for the list of expert tiles, which every CTA of an SM reads: kept in L1 (the lists of two launches that could overlap are
// one layer's, and equal).  Through L2 the routed-expert model's prompt of 1000 tokens took 36.7 ms instead of 35.7.
__device__ __forceinline__ uint32_t ld_list(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ uint4 ld_list(const GemmTile* p) {
    uint4 v;
    asm volatile("ld.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
    return v;
}

// VEC: bytes a copy of raw weights, HT's or (a tensor that starts on a word boundary only) 4.
template <uint32_t TYPE, int N_TILE, uint32_t VEC>
__global__ void __launch_bounds__(H_THREADS, 1)
    gemm_f16_kernel(const uint8_t* __restrict__ w_a, uint64_t n, uint64_t k, const __grid_constant__ CUtensorMap map_hi,
                    const __grid_constant__ CUtensorMap map_lo, const __grid_constant__ CUtensorMap map_sums,
                    const float* __restrict__ inv, const float* __restrict__ rel, const __half* __restrict__ x_hi,
                    const __half* __restrict__ x_lo, uint64_t m_rows, float* dst_a, const float* residual, int* __restrict__ error_flag,
                    const GemmTile* __restrict__ tiles, const uint32_t* __restrict__ n_tiles, uint64_t expert_bytes,
                    const uint8_t* __restrict__ w_b, float* dst_b, uint32_t split) {
    using T = HT<TYPE>;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    using S = Tile<TYPE, N_TILE>;
    constexpr uint32_t PLANE_B = S::PLANE_B, STAGE = S::STAGE_B, RAW_BUF = S::RAW_BUF, BUFS = S::BUFS;
    constexpr uint32_t RAW_STRIDE = raw_stride<TYPE>();
    constexpr uint32_t WIN_WORDS = T::UNIT * T::UNITS / 4;
    constexpr int MY_COLS = S::FINE ? N_TILE : N_TILE / 4;  // accumulator columns a converter thread keeps
    uint8_t* s_sums = smem + (size_t)S::STAGES * STAGE;
    uint8_t* raw = s_sums + (T::MIN ? S::WINDOWS * PLANE_B : 0);
    const uint32_t scales = smem_u32(raw + BUFS * RAW_BUF);
    uint2* s_grid = reinterpret_cast<uint2*>(raw + BUFS * RAW_BUF + S::SCALE_B);
    // full[s]: the step's four converter warps + the TMA thread (and the tiles' bytes); empty[s]: the MMAs' commit
    // raw_full / raw_empty: the copying threads, the converter warps
    __shared__ uint64_t full[S::STAGES], empty[S::STAGES], acc_full[2], acc_empty[S::ACCS], raw_full[BUFS], raw_empty[BUFS];
    __shared__ uint64_t scales_known;  // wide tiles: scaled_groups, by converter group, whether some token has windows with own scales
    __shared__ uint32_t scaled_groups, tmem_base_slot;
    __shared__ int abort_flag, lost_flag;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    pdl_trigger();
    // blockIdx.z: the bank (gate and up in one launch) and this CTA's place in its cluster along k.
    // Grouped form: tile blockIdx.y of the list, its expert's slice of the bank; rows of the tile box beyond the tile's count
    // belong to other experts, are multiplied along and never stored.  The launch covers the list's capacity, not its length.
    uint64_t tok0 = (uint64_t)blockIdx.y * N_TILE, m = m_rows;
    const uint32_t bank = blockIdx.z / split, rank = blockIdx.z - bank * split;
    const uint8_t* w = bank ? w_b : w_a;
    float* dst = bank ? dst_b : dst_a;
    if (tiles != nullptr) {
        pdl_wait();
        if (blockIdx.y >= ld_list(n_tiles)) return;
        const uint4 t = ld_list(tiles + blockIdx.y);  // expert, row0, cnt
        w += (uint64_t)t.x * expert_bytes;
        tok0 = t.y;
        m = tok0 + t.z;
    }
    const uint64_t row0 = (uint64_t)blockIdx.x * HM;
    const uint64_t row_bytes = k / 256 * T::UNIT;
    // this CTA's share of k, in staged windows
    const uint32_t all_windows = (uint32_t)(k / (256 * T::UNITS));
    const uint32_t win0 = (uint32_t)((uint64_t)all_windows * rank / split);
    const uint32_t n_windows = (uint32_t)((uint64_t)all_windows * (rank + 1) / split) - win0;
    const uint32_t n_chunks = n_windows * T::UNITS;  // accumulated windows of 256 columns

    // A staged window of the tile's rows: eight lanes a row, a warp 32 rows, four at a time; the rest of a row of vectors that
    // is no multiple of eight falls to the first lanes.
    constexpr uint32_t ROW_VECS = WIN_WORDS * 4 / VEC, COPIERS = H_COPY * 32;
    static_assert(COPIERS == HM, "a copying warp takes 32 rows");
    // rows r0, r0 + 4, .. of window wn by a warp whose lanes' first row is r0
    auto copy_rows = [&](uint32_t wn, uint32_t r0, auto n_rows) {
        const uint32_t buf = wn % BUFS, v0 = lane & 7;
        const uint32_t last = (uint32_t)min((uint64_t)HM, n - row0) - 1;  // rows past n repeat the last one
        const uint8_t* base = w + row0 * row_bytes + (uint64_t)(win0 + wn) * (WIN_WORDS * 4) + v0 * VEC;
        const uint32_t dst0 = smem_u32(raw) + buf * RAW_BUF + r0 * (RAW_STRIDE * 4) + v0 * VEC;
#pragma unroll
        for (uint32_t j = 0; j < n_rows.value; ++j) {
            const uint8_t* src = base + (uint64_t)min(r0 + 4 * j, last) * (uint32_t)row_bytes;
            const uint32_t dst = dst0 + 4 * j * (RAW_STRIDE * 4);
#pragma unroll
            for (uint32_t c = 0; c < (ROW_VECS + 7) / 8; ++c) {
                if (8 * c + 8 > ROW_VECS && v0 >= ROW_VECS - 8 * c) continue;
                if constexpr (VEC == 16)
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 8 * c * VEC), "l"(src + 8 * c * VEC) : "memory");
                else
                    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(dst + 8 * c * VEC), "l"(src + 8 * c * VEC), "n"(VEC) : "memory");
            }
        }
    };
    auto copy_window = [&](uint32_t wn) {
        copy_rows(wn, (warp & 3) * 32 + (lane >> 3), std::integral_constant<uint32_t, 8>{});
        asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(&raw_full[wn % BUFS])) : "memory");
    };
    // The first window is on its way before anything else is set up (more of them would hold up the rest: Q6_K, 4096 x 4096, 20
    // rows 16.6 -> 18.0 us).  A window of Q6_K, 512 columns copied by the word, is a hundred instructions a copying thread, which
    // launches of one or two windows a CTA wait for: there the converters, idle until it arrives, copy it among themselves
    // (4096 x 4096, 64 rows 26.8 -> 25.9 us, 2048 x 4096 19.0 -> 18.6; Q2_K and IQ2_XXS, half of it, lose up to 0.6 us).
    constexpr bool SHARED_FIRST = TYPE == T_Q6_K;
    if (SHARED_FIRST && warp < H_CONV) {
        copy_rows(0, warp * 8 + (lane >> 3), std::integral_constant<uint32_t, 2>{});
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    if (warp >= H_CONV + H_ISSUE) {
        if (tid == (H_CONV + H_ISSUE) * 32) {
            for (uint32_t b = 0; b < BUFS; ++b) mbar_init(&raw_full[b], COPIERS), mbar_init(&raw_empty[b], H_CONV);
            mbar_fence_init();
        }
        asm volatile("bar.sync 2, %0;" ::"n"(COPIERS) : "memory");
        if (SHARED_FIRST) asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(&raw_full[0])) : "memory");
        else copy_window(0);
    }
    if (tid == 0) {
        for (uint32_t s = 0; s < S::STAGES; ++s) {
            mbar_init(&full[s], 4 + 1);
            mbar_init(&empty[s], 1);
        }
        for (uint32_t b = 0; b < S::ACCS; ++b) {
            if (!S::FINE) mbar_init(&acc_full[b & 1], 1);
            mbar_init(&acc_empty[b], S::FINE ? 4 : H_CONV);
        }
        mbar_init(&scales_known, 1);
        abort_flag = lost_flag = 0;
        mbar_fence_init();
    }
    if (warp == H_CONV) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_slot)),
                     "r"(512u)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if constexpr (TYPE == T_IQ2_XXS)
        for (int i = tid; i < 256; i += H_THREADS) s_grid[i] = g_iq2xxs_grid[i];
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_d = tmem_base_slot;

    if (warp < H_CONV) {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(H_REGS_CONV));
        // narrow tiles: polls, a chain of short waits is what they spend their time on; wide ones sleep and leave the issue slots
        auto converter_wait = [](uint64_t* bar, uint32_t parity) { return S::FINE ? mbar_wait_polling(bar, parity) : mbar_wait(bar, parity); };
        const uint32_t q = warp & 3, g = warp >> 2;
        const uint32_t lane_base = (q * 32) << 16;  // this warp's quarter of the tensor-memory lanes
        float sums[MY_COLS];
#pragma unroll
        for (int c = 0; c < MY_COLS; ++c) sums[c] = 0.0f;
        // Some token of this warp's columns has windows with scales of their own.  Its running sum then is in units of the
        // scale of the window that was added last (the first one's, to begin with), and is brought to the next one's where
        // they differ.  What that needs lies in shared memory and in a loop of its own, so that the usual tile spends no
        // registers on it (in one loop Q6_K, 28672 x 4096, 40 rows took 202 us instead of 172).
        bool scaled = false;
        const uint32_t slot = scales + warp * 32 * 16;  // per token: its address in rel, its scale so far, its change
        // On wide tiles an idle issuer reads the signs and tells: the load in the converters' chain cost Q2_K 4096 x 14336, 333 rows
        // 2.8 of 125 us.  On narrow ones, whose issuers have no time, waiting for one costs more than the load (Q4_K 512 x 2048, 33
        // rows 10.4 and 9.9 us).
        auto find_scales = [&] {
            if constexpr (!S::FINE) {
                scaled = scaled_groups >> g & 1;
                if (!scaled) return;
            }
            pdl_wait();  // the scales belong to the kernel in front
            const uint64_t tok = min(tok0 + (S::FINE ? 0 : g * MY_COLS) + lane % MY_COLS, m_rows - 1);  // the last row, past it
            if constexpr (S::FINE) {
                scaled = __any_sync(0xFFFFFFFFu, ld_behind_wait(inv + tok) < 0.0f);
                if (!scaled) return;
            }
            const float* p = rel + (uint64_t)win0 * T::UNITS * m_rows + tok;
            asm volatile("st.shared.u64 [%0], %1;" ::"r"(slot + lane * 8), "l"(p) : "memory");
            asm volatile("st.shared.f32 [%0], %1;" ::"r"(slot + 256 + lane * 4), "f"(ld_behind_wait(p)) : "memory");
        };
        auto rescale = [&](uint32_t c) {  // to window c's scales; c = n_chunks: to the rows'
            const float* p;
            asm volatile("ld.shared.u64 %0, [%1];" : "=l"(p) : "r"(slot + lane * 8));
            const float was = __uint_as_float(s32(slot + 256 + lane * 4)), now = c < n_chunks ? ld_behind_wait(p + (uint64_t)c * m_rows) : 1.0f;
            if (!__any_sync(0xFFFFFFFFu, was != now)) return;
            asm volatile("st.shared.f32 [%0], %1;" ::"r"(slot + 256 + lane * 4), "f"(now) : "memory");
            asm volatile("st.shared.f32 [%0], %1;" ::"r"(slot + 384 + lane * 4), "f"(was / now) : "memory");  // powers of two
            __syncwarp();
#pragma unroll
            for (int i = 0; i < MY_COLS; ++i) sums[i] *= __uint_as_float(s32(slot + 384 + i * 4));
            __syncwarp();
        };
        // sums += f * (this warp's columns of the accumulator at column `col`)
        auto add_acc = [&](uint32_t col, float f) {
            constexpr int PART = 16;
            const uint32_t taddr = tmem_d + lane_base + col;
#pragma unroll
            for (int part = 0; part < MY_COLS / PART; ++part) {
                uint32_t rr[PART];
                tmem_ld16(taddr + part * 16, rr);
#pragma unroll
                for (int i = 0; i < PART; ++i) sums[part * PART + i] = fmaf(f, __uint_as_float(rr[i]), sums[part * PART + i]);
            }
        };
        // read back window c: this warp's columns of its accumulator, or all columns of the accumulator of its own step
        auto drain = [&](uint32_t c, float f) -> bool {
            uint64_t* ready = S::FINE ? &empty[(c % S::WINDOWS) * H_STEPS + g] : &acc_full[c & 1];
            if (!__all_sync(0xFFFFFFFFu, converter_wait(ready, (S::FINE ? c / S::WINDOWS : c >> 1) & 1))) return false;
            tc_fence_after();
            add_acc(S::FINE ? g * N_TILE : (c & 1) * N_TILE + g * MY_COLS, f);
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&acc_empty[S::FINE ? g : c & 1]);
            return true;
        };
        const uint32_t raw_q = smem_u32(raw) + q * 32 * RAW_STRIDE * 4;
        if (SHARED_FIRST) {  // the first window, which they copied
            asm volatile("cp.async.wait_all;" ::: "memory");
            asm volatile("bar.sync 1, %0;" ::"n"(H_CONV * 32) : "memory");
        }
        bool ok = true;
        float f_prev = 0.0f;
        auto window = [&](uint32_t wn, auto with_scales) {
            const uint32_t buf = wn % BUFS;
            ok = __all_sync(0xFFFFFFFFu, converter_wait(&raw_full[buf], (wn / BUFS) & 1));
#pragma unroll 1
            for (uint32_t cc = 0; cc < T::UNITS && ok; ++cc) {
                const uint32_t c = wn * T::UNITS + cc;
                const uint32_t u = raw_q + buf * RAW_BUF + lane * RAW_STRIDE * 4 + cc * T::UNIT;
                const RowWin rw = row_window<TYPE, S::NB>(u, S::FINE ? 2 * g : 0);
                // the stage's columns must have been read by the MMAs that used them last
                const uint32_t ph = c % S::WINDOWS, st = ph * H_STEPS + g;
                ok = __all_sync(0xFFFFFFFFu, converter_wait(&empty[st], ((c / S::WINDOWS) & 1) ^ 1));
                if (!ok) break;
                tc_fence_after();
                const uint32_t acol = tmem_d + lane_base + S::ACC_COLS + st * S::A_COLS;
                convert64<TYPE>(u, g, rw, s_grid, &lost_flag, [&](uint32_t h, const uint32_t (&a)[16], const uint32_t (&b)[16]) {
                    tmem_st16(acol + 16 * h, a);
                    if constexpr (T::TWO) tmem_st16(acol + 32 + 16 * h, b);
                });
                if constexpr (T::MIN) {
                    if (g == H_STEPS - 1) {
                        uint32_t a[16];
                        convert_minima<TYPE>(u, rw, a);
                        tmem_st16(tmem_d + lane_base + S::MIN_COL0 + 16 * ph, a);
                    }
                }
                if (cc == T::UNITS - 1) {
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&raw_empty[buf]);
                }
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&full[st]);
                // read back the window before this one while this one accumulates
                if (c > 0) {
                    if constexpr (with_scales.value) rescale(c - 1);
                    ok = drain(c - 1, f_prev);
                } else {
                    if constexpr (!S::FINE) ok = __all_sync(0xFFFFFFFFu, converter_wait(&scales_known, 0));
                    if (ok) find_scales();
                }
                f_prev = rw.f;
            }
        };
        uint32_t wn = 0;
        for (; wn < n_windows && !scaled && ok; ++wn) window(wn, std::false_type{});  // the first window tells
        for (; wn < n_windows && ok; ++wn) window(wn, std::true_type{});
        if (scaled) rescale(n_chunks - 1);
        if (ok && n_chunks > 0) ok = drain(n_chunks - 1, f_prev);
        if (scaled) rescale(n_chunks);
        if (!ok) abort_flag = 1;
        pdl_wait();  // dst and the rows' scales belong to the kernels before this one
        // The ring and the staged bytes are idle once every converter is here: the last read-back waited for this CTA's
        // last products.
        asm volatile("bar.sync 1, %0;" ::"n"(H_CONV * 32) : "memory");
        const uint64_t out_row = row0 + q * 32 + lane, first_tok = tok0 + (S::FINE ? 0 : g * MY_COLS);
        float* red = reinterpret_cast<float*>(smem);
        if (!S::FINE && split == 1) {
            if (ok && out_row < n) {
#pragma unroll
                for (int c = 0; c < MY_COLS; ++c) {
                    const uint64_t tok = tok0 + g * MY_COLS + c;
                    if (tok < m) {
                        const float v = sums[c] * fabsf(__ldg(inv + tok));
                        dst[tok * n + out_row] = residual ? residual[tok * n + out_row] + v : v;
                    }
                }
            }
        } else {
            // leave the partial tile in shared memory, [token][row] (four of them where the warps of a quarter hold sums
            // of their own steps)
#pragma unroll
            for (int c = 0; c < MY_COLS; ++c) red[(g * MY_COLS + c) * HM + q * 32 + lane] = sums[c];
        }
        if constexpr (T::LOSES) {
            if (lost_flag && ok && first_tok < m) {  // each thread adds to what it has just stored
                add_lost<TYPE, S::NB>(w + min(out_row, n - 1) * row_bytes, win0 * T::UNITS, n_chunks, S::FINE ? g : 0,
                                      S::FINE ? g + 1 : H_STEPS, k, x_hi, x_lo, rel, m_rows, first_tok,
                                      (uint32_t)min((uint64_t)MY_COLS, m - first_tok), [&](uint32_t t, float v) {
                                          if (S::FINE || split > 1)
                                              red[(g * MY_COLS + t) * HM + q * 32 + lane] += v;
                                          else if (out_row < n)
                                              dst[(first_tok + t) * n + out_row] += v * fabsf(__ldg(inv + first_tok + t));
                                      });
            }
        }
    } else if (warp < H_CONV + H_ISSUE) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(H_REGS_REST));
        // ── issuers (their waits sleep: polling warps take issue slots from the converters) ──
        constexpr uint32_t idesc = umma_idesc_f16(N_TILE);
        const uint32_t base0 = smem_u32(smem);
        const uint64_t d0_hi = umma_desc(base0), d0_lo = umma_desc(base0 + PLANE_B);
        [[maybe_unused]] const uint64_t d_sums = umma_desc(smem_u32(s_sums));
        bool ok = true;
        // the activation tiles of window c's step g, once the products that read the stage last are through
        auto load = [&](uint32_t c, uint32_t g) -> bool {
            const uint32_t ph = c % S::WINDOWS, st = ph * H_STEPS + g;
            if (!__all_sync(0xFFFFFFFFu, mbar_wait(&empty[st], ((c / S::WINDOWS) & 1) ^ 1))) return false;
            if (lane == 0) {
                uint8_t* tile = smem + (size_t)st * STAGE;
                const uint32_t col = (win0 * T::UNITS + c) * 256 + 64 * g;
                const bool with_sums = T::MIN && g == H_STEPS - 1;
                mbar_arrive_expect_tx(&full[st], (with_sums ? 3 : 2) * PLANE_B);
                tma_load_2d(tile, &map_hi, col, (uint32_t)tok0, &full[st]);
                tma_load_2d(tile + PLANE_B, &map_lo, col, (uint32_t)tok0, &full[st]);
                if (with_sums)
                    tma_load_2d(s_sums + ph * PLANE_B, &map_sums, ((win0 + c) >> 1) * 64, (uint32_t)tok0, &full[st]);
            }
            __syncwarp();
            return true;
        };
        // wide tiles: whether some token of a converter warp's columns has windows with scales of their own
        auto tell_scales = [&] {
            constexpr uint32_t COLS = S::FINE ? N_TILE : N_TILE / 4;
            uint32_t bits = 0;
#pragma unroll
            for (uint32_t i = 0; i < N_TILE / COLS; ++i) {
                const uint64_t tok = min(tok0 + i * COLS + lane % COLS, m_rows - 1);  // the last row, past it
                bits |= (__any_sync(0xFFFFFFFFu, ld_behind_wait(inv + tok) < 0.0f) ? 1u : 0u) << i;
            }
            if (lane == 0) {
                *static_cast<volatile uint32_t*>(&scaled_groups) = bits;
                mbar_arrive(&scales_known);
            }
            __syncwarp();
        };
        // Steps G0 .. G1 - 1 of every window; compile-time, so that the descriptors need no arithmetic but a stage's offset.
        // The tensor pipe takes few instructions ahead: on wide tiles the waits for the next step stand between the two halves of
        // this one's, or the pipe runs dry at every step (some 220 cycles, 600 at a new window).
        auto issue = [&](auto G0, auto G1) {
            // whether step g of window c can start: its accumulator's last contents have been read back, its operands are there
            auto can_start = [&](uint32_t c, uint32_t g) {
                if (S::FINE ? c >= 1 : g == 0 && c >= 2)
                    if (!mbar_wait(&acc_empty[S::FINE ? g : c & 1], (S::FINE ? c - 1 : (c >> 1) - 1) & 1)) return false;
                return mbar_wait(&full[c % S::WINDOWS * H_STEPS + g], (c / S::WINDOWS) & 1);
            };
            if (S::FINE) {
                pdl_wait();
                for (uint32_t c = 0; c < S::WINDOWS && c < n_chunks && ok; ++c) ok = load(c, G0.value);
            }
            if (ok && n_chunks > 0) ok = __all_sync(0xFFFFFFFFu, can_start(0, G0.value));
            const bool leader = elect_one();
            for (uint32_t c = 0; c < n_chunks && ok; ++c) {
                const uint32_t ph = c % S::WINDOWS;
#pragma unroll
                for (uint32_t g = G0.value; g < G1.value; ++g) {
                    const uint32_t st = ph * H_STEPS + g, acc = S::FINE ? g : c & 1, d = tmem_d + acc * N_TILE;
                    const uint64_t so = (uint64_t)st * (STAGE >> 4);
                    const uint32_t a1 = tmem_d + S::ACC_COLS + st * S::A_COLS;
                    [[maybe_unused]] const uint32_t a2 = a1 + 32;
                    const bool fresh = S::FINE || g == 0;
                    tc_fence_after();  // the converters' tcgen05.st / .ld
                    if (leader) {
                        // small products first, while the accumulator is small.  16 columns an instruction: 8 columns of A,
                        // 32 bytes of B's swizzled rows.
#pragma unroll
                        for (uint32_t kk = 0; kk < 4; ++kk) {
                            umma_f16_ts(d, a1 + kk * 8, d0_lo + so + kk * 2, idesc, !fresh || kk != 0);
                            if constexpr (T::TWO) umma_f16_ts(d, a2 + kk * 8, d0_hi + so + kk * 2, idesc, 1);
                        }
                        if constexpr (T::MIN) {
                            if (g == H_STEPS - 1) {
                                // a tile of sums holds two windows, 64 bytes each: first terms, second terms
                                const uint64_t ds = d_sums + ph * (PLANE_B >> 4) + ((win0 + c) & 1) * 4;
                                const uint32_t am = tmem_d + S::MIN_COL0 + 16 * ph;
                                umma_f16_ts(d, am + 8, ds, idesc, 1);
                                umma_f16_ts(d, am, ds + 2, idesc, 1);
                                umma_f16_ts(d, am, ds, idesc, 1);
                            }
                        }
                    }
                    bool next = true;
                    if (!S::FINE) {  // the next step does not depend on this one's products
                        __syncwarp();
                        if (!(g == G1.value - 1 && c + 1 == n_chunks))
                            next = g + 1 < G1.value ? can_start(c, g + 1) : can_start(c + 1, G0.value);
                        next = __all_sync(0xFFFFFFFFu, next);
                    }
                    if (leader) {
#pragma unroll
                        for (uint32_t kk = 0; kk < 4; ++kk) umma_f16_ts(d, a1 + kk * 8, d0_hi + so + kk * 2, idesc, 1);
                        umma_commit(&empty[st]);  // the weight columns and the activation tiles of the stage are free
                        if (!S::FINE && g == H_STEPS - 1) umma_commit(&acc_full[acc]);
                    }
                    __syncwarp();
                    ok = next;
                    if (!ok) break;
                }
                if (!S::FINE) continue;
                // the next window's tiles: its stage's last products are a window behind, or (one window) the ones above
                if (ok && c + 1 >= S::WINDOWS && c + 1 < n_chunks) ok = load(c + 1, G0.value);
                if (ok && c + 1 < n_chunks) ok = __all_sync(0xFFFFFFFFu, can_start(c + 1, G0.value));
            }
        };
        using std::integral_constant;
        const uint32_t mine = warp - H_CONV;
        if constexpr (S::FINE) {
            if (mine == 0) issue(integral_constant<uint32_t, 0>{}, integral_constant<uint32_t, 1>{});
            else if (mine == 1) issue(integral_constant<uint32_t, 1>{}, integral_constant<uint32_t, 2>{});
            else if (mine == 2) issue(integral_constant<uint32_t, 2>{}, integral_constant<uint32_t, 3>{});
            else issue(integral_constant<uint32_t, 3>{}, integral_constant<uint32_t, 4>{});
        } else if (mine == 0) {
            issue(integral_constant<uint32_t, 0>{}, integral_constant<uint32_t, H_STEPS>{});
        } else if (mine == 1) {
            pdl_wait();
            for (uint32_t c = 0; c < n_chunks && ok; ++c)
                for (uint32_t g = 0; g < H_STEPS && ok; ++g) ok = load(c, g);
        } else if (mine == 2) {
            pdl_wait();
            tell_scales();
        }
        if (!ok && lane == 0) abort_flag = 1;
    } else {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(H_REGS_REST));
        // ── copies of raw weights ──
        bool ok = true;
        for (uint32_t wn = 1; wn < n_windows && ok; ++wn) {
            ok = __all_sync(0xFFFFFFFFu, mbar_wait(&raw_empty[wn % BUFS], ((wn / BUFS) & 1) ^ 1));
            if (ok) copy_window(wn);
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        if (!ok && lane == 0) abort_flag = 1;
    }
    tc_fence_before();
    __syncthreads();
    if (S::FINE || split > 1) {
        if (split > 1) cluster_sync_all();
        // tile element i = token * 128 + row; rank r adds the tokens t = r (mod split), over the ranks and their partial
        // tiles in order
        if (abort_flag == 0 && tid < H_CONV * 32) {
            const uint32_t red = smem_u32(smem), row = tid & (HM - 1);
            constexpr uint32_t TILES = S::FINE ? 4 : 1;
            for (uint32_t t = rank + split * (tid / HM); t < N_TILE; t += split * (H_CONV * 32 / HM)) {
                const uint64_t tok = tok0 + t, at = tok * n + row0 + row;
                if (tok >= m || row0 + row >= n) continue;
                float v = 0.0f;
                for (uint32_t r = 0; r < split; ++r)
#pragma unroll
                    for (uint32_t p = 0; p < TILES; ++p) {
                        const uint32_t addr = red + ((p * N_TILE + t) * HM + row) * 4;
                        v += split > 1 ? ld_cluster_f32(addr, r) : __uint_as_float(s32(addr));
                    }
                v *= fabsf(__ldg(inv + tok));
                dst[at] = residual ? residual[at] + v : v;
            }
        }
        if (split > 1) cluster_sync_all();  // no CTA leaves while another reads its shared memory
    }
    if (abort_flag && tid == 0) *reinterpret_cast<volatile int*>(error_flag) = 1;
    if (warp == H_CONV) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_d), "r"(512u) : "memory");
    }
}

// ── host side ──
PFN_cuTensorMapEncodeTiled g_encode_f16 = nullptr;

cudaError_t f16_map(const __half* base, uint64_t rows, uint64_t cols, uint32_t n_tile, CUtensorMap* out) {
    if (!g_encode_f16) {
        void* fn = nullptr;
        cudaDriverEntryPointQueryResult qres;
        cudaError_t e = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qres);
        if (e != cudaSuccess) return e;
        if (qres != cudaDriverEntryPointSuccess || !fn) return cudaErrorNotSupported;
        g_encode_f16 = reinterpret_cast<PFN_cuTensorMapEncodeTiled>(fn);
    }
    const cuuint64_t dims[2] = {cols, rows};
    const cuuint64_t strides[1] = {cols * 2};  // a multiple of 64: cols is a multiple of 32
    const cuuint32_t box[2] = {64, n_tile};    // 64 halves = one 128-byte swizzled row
    const cuuint32_t estr[2] = {1, 1};
    CUresult r = g_encode_f16(out, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<__half*>(base), dims, strides, box, estr,
                              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);  // rows and columns beyond the array read as zeros
    return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

struct SplitX {  // the split activations inside the caller's scratch
    __half *hi, *lo, *sums;
    float *inv, *rel;
};
uint64_t up128(uint64_t v) { return (v + 127) & ~(uint64_t)127; }
SplitX split_in(void* scratch, uint64_t m, uint64_t k) {
    SplitX x;
    uint8_t* b = static_cast<uint8_t*>(scratch);
    x.hi = reinterpret_cast<__half*>(b);
    b += up128(2 * m * k);
    x.lo = reinterpret_cast<__half*>(b);
    b += up128(2 * m * k);
    x.sums = reinterpret_cast<__half*>(b);
    b += up128(m * k / 4);
    x.inv = reinterpret_cast<float*>(b);
    b += up128(4 * m);
    x.rel = reinterpret_cast<float*>(b);
    return x;
}

// Everything of a launch but the weights' type and the tile width.
struct F16Launch {
    const uint8_t *w_a, *w_b;
    uint64_t n, k, rows, expert_bytes;
    SplitX x;
    float *dst_a, *dst_b;
    const float* residual;
    const GemmTile* tiles;
    uint32_t max_tiles;
    const uint32_t* n_tiles;
    int* error_flag;
};

template <uint32_t TYPE, int N_TILE, uint32_t VEC = HT<TYPE>::VEC>
cudaError_t launch_f16_tile(const F16Launch& l, cudaStream_t s) {
    if constexpr (VEC == 8)
        if ((reinterpret_cast<uintptr_t>(l.w_a) | reinterpret_cast<uintptr_t>(l.w_b)) % 8 != 0) return launch_f16_tile<TYPE, N_TILE, 4>(l, s);
    constexpr size_t smem = Tile<TYPE, N_TILE>::SMEM;
    auto kern = gemm_f16_kernel<TYPE, N_TILE, VEC>;
    static bool configured[MAX_DEVICES] = {};
    if (cudaError_t ce = set_max_smem_once(kern, 226 * 1024, configured); ce != cudaSuccess) return ce;
    CUtensorMap hi, lo, sums;
    cudaError_t e = f16_map(l.x.hi, l.rows, l.k, N_TILE, &hi);
    if (e == cudaSuccess) e = f16_map(l.x.lo, l.rows, l.k, N_TILE, &lo);
    if (e == cudaSuccess) e = f16_map(l.x.sums, l.rows, l.k / 8, N_TILE, &sums);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cfg.blockDim = dim3(H_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    const unsigned gx = (unsigned)((l.n + HM - 1) / HM);
    uint32_t split = 1;
    if (l.tiles) {
        if (l.max_tiles > 65535) return cudaErrorInvalidValue;  // the tile list is walked along grid.y
        cfg.gridDim = dim3(gx, l.max_tiles, l.w_b ? 2 : 1);
    } else {
        // Split k over a cluster where whole tiles fill the SMs badly: waves x (a CTA's windows + about three windows'
        // worth of filling the pipeline and storing the tile).  Clusters of up to four pack the GPCs without loss.
        const unsigned banks = l.w_b ? 2 : 1;
        const uint64_t gy = (l.rows + N_TILE - 1) / N_TILE, tiles = gx * gy * banks, sms = (uint64_t)num_sms();
        const uint64_t windows = l.k / (256 * HT<TYPE>::UNITS);
        uint64_t best = ~0ull;
        for (uint32_t c = 1; c <= 4 && c <= windows; ++c) {
            const uint64_t waves = (tiles * c + sms - 1) / sms;
            const uint64_t cost = waves * ((windows + c - 1) / c * HT<TYPE>::UNITS + 3 + (c > 1));
            if (cost < best) best = cost, split = c;
        }
        cfg.gridDim = dim3(gx, (unsigned)gy, split * banks);
        if (split > 1) {
            attr[1].id = cudaLaunchAttributeClusterDimension;
            attr[1].val.clusterDim.x = 1;
            attr[1].val.clusterDim.y = 1;
            attr[1].val.clusterDim.z = split;
            cfg.numAttrs = 2;
        }
    }
    e = cudaLaunchKernelEx(&cfg, kern, l.w_a, l.n, l.k, hi, lo, sums, (const float*)l.x.inv, (const float*)l.x.rel,
                           (const __half*)l.x.hi, (const __half*)l.x.lo, l.rows, l.dst_a, l.residual, l.error_flag, l.tiles,
                           l.n_tiles, l.expert_bytes, l.w_b, l.dst_b, split);
    return e != cudaSuccess ? e : cudaGetLastError();
}

template <int N_TILE>
cudaError_t launch_f16_typed(uint32_t type, const F16Launch& l, cudaStream_t s) {
    switch (type) {
        case T_Q8_0:
            if constexpr (N_TILE > 16) return launch_f16_tile<T_Q8_0, N_TILE>(l, s);
            return cudaErrorInvalidValue;
        case T_Q2_K: return launch_f16_tile<T_Q2_K, N_TILE>(l, s);
        case T_Q4_K: return launch_f16_tile<T_Q4_K, N_TILE>(l, s);
        case T_IQ2_XXS: return launch_f16_tile<T_IQ2_XXS, N_TILE>(l, s);
        case T_MXFP4: return launch_f16_tile<T_MXFP4, N_TILE>(l, s);
        case T_Q6_K:
            if constexpr (N_TILE <= 32) return launch_f16_tile<T_Q6_K, N_TILE>(l, s);
            return cudaErrorInvalidValue;
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t split_activations_f16(uint32_t type, const float* x, uint64_t m, uint64_t k, const float* norm_w, float eps, const SplitX& o,
                                  cudaStream_t s, const uint32_t* list = nullptr, const uint32_t* n_list = nullptr) {
    // a row's groups in the threads' registers where 512 threads can hold them
    unsigned threads = 256;
    auto kern = split_f16_kernel<256, 0>;
    if (norm_w == nullptr && k <= 16384) {
        threads = k <= 1024 ? 64 : k <= 2048 ? 128 : k <= 4096 ? 256 : 512;
        kern = k <= 1024   ? split_f16_kernel<64, 1>
               : k <= 2048 ? split_f16_kernel<128, 1>
               : k <= 4096 ? split_f16_kernel<256, 1>
                           : split_f16_kernel<512, 2>;
    }
    return launch_pdl(kern, dim3((unsigned)m), threads, 0, s, x, (uint32_t)k, norm_w, eps, list, n_list, type == T_MXFP4 ? 1 : 0,
                      o.hi, o.lo, o.sums, o.inv, o.rel);
}

}  // namespace

// Rows of a tile for m rows of lhs.  Up to 64 rows the other route is the decode kernel: they stay on the exact tiles.
// Q6_K always does (no 128-row form of it was built).  Q8_0 comes with 17 rows and more.
static uint32_t tile_rows(uint32_t type, uint64_t m) { return m <= 16 && type != T_Q8_0 ? 16 : m <= 64 || type == T_Q6_K ? 32 : 128; }

// Whole staged windows in every row, made of the vectors they are copied by (Q4_K tensors and slices always start on 16
// bytes); the tiles of lhs fit grid.y.
bool gemm_f16_supports(uint32_t type, const uint8_t* w, uint64_t n, uint64_t k, uint64_t m) {
    if (m == 0 || n == 0 || k == 0 || k % 256 != 0 || k > 0x7FFFFFFFu || m > 65535ull * tile_rows(type, m)) return false;
    const uintptr_t a = reinterpret_cast<uintptr_t>(w);
    switch (type) {
        case T_Q4_K: return a % 16 == 0;
        case T_Q8_0:
        case T_MXFP4:
        case T_Q2_K: return a % 4 == 0;
        case T_IQ2_XXS:
        case T_Q6_K: return a % 4 == 0 && k % 512 == 0;
        default: return false;
    }
}

size_t gemm_f16_scratch_bytes(uint64_t m, uint64_t k) {
    return (size_t)(2 * up128(2 * m * k) + up128(m * k / 4) + up128(4 * m) + up128(m * k / 64));
}

// dst_a = residual + norm(lhs) . W^T; with w_b the same rows through a second tensor into dst_b.
cudaError_t launch_gemm_f16(uint32_t type, const uint8_t* w_a, const uint8_t* w_b, uint64_t n, uint64_t k, const float* lhs,
                            uint64_t m, const float* norm_w, float eps, const float* residual, float* dst_a, float* dst_b,
                            void* scratch, int* error_flag, cudaStream_t s) {
    F16Launch l = {};
    l.w_a = w_a, l.w_b = w_b;
    l.n = n, l.k = k, l.rows = m;
    l.x = split_in(scratch, m, k);
    l.dst_a = dst_a, l.dst_b = dst_b;
    l.residual = residual;
    l.error_flag = error_flag;
    if (cudaError_t e = split_activations_f16(type, lhs, m, k, norm_w, eps, l.x, s); e != cudaSuccess) return e;
    switch (tile_rows(type, m)) {
        case 16: return launch_f16_typed<16>(type, l, s);
        case 32: return launch_f16_typed<32>(type, l, s);
        default: return launch_f16_typed<128>(type, l, s);
    }
}

bool gemm_f16_grouped_supports(uint32_t type, const uint8_t* bank, uint64_t n, uint64_t k) {
    return type != T_Q6_K && gemm_f16_supports(type, bank, n, k, 128);
}

cudaError_t launch_gemm_f16_grouped(uint32_t type, const uint8_t* bank_a, const uint8_t* bank_b, uint64_t expert_bytes,
                                   uint64_t n, uint64_t k, const float* x, const uint32_t* list, const uint32_t* n_list,
                                   uint64_t rows, float* dst_a, float* dst_b, const GemmTile* narrow, uint32_t max_narrow, const GemmTile* wide, uint32_t max_wide,
                                   const uint32_t* counts, void* scratch, int* error_flag, cudaStream_t s) {
    F16Launch l = {};
    l.w_a = bank_a, l.w_b = bank_b;
    l.n = n, l.k = k, l.rows = rows, l.expert_bytes = expert_bytes;
    l.x = split_in(scratch, rows, k);
    l.dst_a = dst_a, l.dst_b = dst_b;
    l.error_flag = error_flag;
    if (cudaError_t e = split_activations_f16(type, x, rows, k, nullptr, 0.0f, l.x, s, list, n_list); e != cudaSuccess) return e;
    if (max_narrow) {
        l.tiles = narrow, l.max_tiles = max_narrow, l.n_tiles = counts;
        if (cudaError_t e = launch_f16_typed<32>(type, l, s); e != cudaSuccess) return e;
    }
    if (max_wide) {
        l.tiles = wide, l.max_tiles = max_wide, l.n_tiles = counts + 1;
        return launch_f16_typed<128>(type, l, s);
    }
    return cudaSuccess;
}

}  // namespace jq
