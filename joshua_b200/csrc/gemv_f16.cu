// Decode-time matmul of small batches (3 .. 8 rows) over raw GGUF blocks in half-precision terms that keep f32's precision.
//
// dst[m, n] = lhs[m, k] . W[n, k]^T with W left in its GGUF bytes, streamed once.  As in gemv_mma.cu the arithmetic is
// regrouped around the formats' small codes,
//
//     sum_c x_c (s_g q_c - o_g)  =  s_g sum_c x_c q_c  -  o_g sum_c x_c     (per group of 32 columns g)
//
// but the products are mma.sync.m16n8k16 on f16: the codes are exact f16 numbers (Q4_K: a nibble left in place under the
// exponent of 1024 or 64, less that; MXFP4: one conversion instruction a pair), and an activation is two f16
// terms under a power-of-two scale of its 256 columns (largest value just below 2^15): 22 to 24 bits of every value within 2^17
// of the largest.  A group is four chained instructions, low terms first, whose exact products the tensor core adds with
// truncation; its sum is scaled and added round-to-nearest.  The minima of Q4_K are one more instruction per 256 columns:
// eight six-bit minima against the groups' sums of x, two terms each.  (Codes as f16 subnormals would need no subtraction,
// but the tensor core aligns them by their unnormalised exponents: 1.3e-6 instead of 2.0e-7 against float64.)  Eight rows fill
// the instruction's columns; up to four rows the high terms take columns 0 .. 3, the low terms 4 .. 7, half the instructions.
//
// Structure: persistent, one CTA an SM.  One thread copies: a TMA box of 16 rows x a stage's units, padded to a row stride
// without bank conflicts (a bulk copy a row, as in gemv_mma.cu, costs its warp more instructions than 16 busy consumer warps
// leave it time for: 10 bytes a cycle).  16 warps consume, in teams; a team owns a tile of 16 rows at a time and adds its
// warps' partial sums itself (one warp that added for all was the bottleneck at 2000 cycles a tile).  The activations of the
// CTA's columns stay in shared memory; where they do not fit, a cluster of S CTAs splits k, walks the same tiles, and the
// teams send their partial tiles to one of the ranks in turn (distributed shared memory, an mbarrier a slot), which adds them
// in rank order, so that results do not depend on timing.
//
// Error against float64 (2-norm, N(0, 1) rows): Q4_K 2.1e-7 to 2.9e-7, MXFP4 0.9e-7 to 1.1e-7; the routes before 3.3e-7 to
// 3.8e-7 and 1.3e-7 to 1.5e-7.  Positive rows (1 + |N(0, 1)|), Q4_K weights of mean zero: up to four rows 1.2e-6, before 1.8e-6 to
// 2.8e-6; five to eight 1.4e-6 to 1.6e-6, before 2.4e-6 to 5.6e-6.
// Algorithmic bytes per launch: n*k/B*S (weights) + 4*m*(k + n).  What bounds it: the consumers' instructions, 460 (four rows) to 600 (eight)
// per 16 x 256 unit at 1.8 to 2.8 a cycle.  Measured, four / eight rows, before (the integer kernel / the tile GEMM and its
// split) and now: Q4_K 28672 x 4096 27.4 / 49.5 and 22.2 / 27.5 us, 6144 x 4096 11.4 /
// 25.9 and 9.2 / 12.2, 4096 x 4096 9.8 / 11.5 and 7.4 / 10.2, 4096 x 14336 24.6 / 28.5 and 18.3 / 22.8, 128256 x 4096 94 / 169 and
// 73 / 96; MXFP4 28672 x 4096 41.5 (three rows) / 54.7 and 23.7 / 30.3, 7168 x 2048 11.6 / 18.2 and 6.8 / 8.6.
//
// Every wait is bounded and raises the device status flag; threads that gave up still take part in the CTA's and the
// cluster's barriers.
#include <cuda_fp16.h>

#include <algorithm>
#include <type_traits>

#include <cudaTypedefs.h>

#include "common.cuh"
#include "tc5.cuh"

namespace jq {

namespace {

constexpr uint32_t ROWS = 16;      // weight rows of a tile = MMA M
constexpr uint32_t NCW = 16;       // consumer warps
constexpr uint32_t THREADS = (NCW + 1) * 32;
constexpr uint32_t MAX_TEAMS = 8;  // a named barrier each
constexpr uint32_t SLOTS = 2;      // partial tiles a rank can hold of every other one
constexpr uint32_t MAX_SPLIT = 8;
constexpr uint32_t SMEM_MAX = 225 * 1024;
constexpr uint32_t MAX_STAGES = 48;  // of all teams
// Shorter rows stay with the routes they had, although they lose there: k = 512, four / eight rows, Q4_K 4096 rows 5.0 / 6.3 us
// (here 4.5 / 5.1), 28672 rows 16.4 / 13.1 (6.6 / 7.5), MXFP4 5.9 / 8.4 (5.0 / 5.7) and 22.4 / 35.1 (7.0 / 8.4).  One and two
// rows of x stay with the integer kernel: 28672 x 4096 17.0 and 18.7 us there, 21.9 and 22.0 here.
constexpr uint64_t MIN_K = 1024;

template <uint32_t TYPE>
struct FT;
template <>
struct FT<T_Q4_K> {
    static constexpr uint32_t UNIT = 144, STRIDE_MOD = 8;  // row stride mod 32 words: 64-bit fragment loads
    static constexpr uint32_t STEP = 1;                    // units that end on 16 bytes
    static constexpr bool MIN = true;
};
template <>
struct FT<T_MXFP4> {
    static constexpr uint32_t UNIT = 136, STRIDE_MOD = 4;  // 32-bit loads
    static constexpr uint32_t STEP = 2;
    static constexpr bool MIN = false;
};

// PACK: up to four rows, high terms in columns 0 .. 3 of the instruction, low terms in 4 .. 7
constexpr uint32_t COLS = 8;
template <bool PACK>
struct Shape {
    static constexpr uint32_t TOK = PACK ? 4 : COLS, PLANES = PACK ? 1 : 2;
    static constexpr uint32_t GROUP_B = PLANES * COLS * 64 + 64;  // 32 columns; the 64 bytes spread the stores of eight groups over the banks
    static constexpr uint32_t UNIT_B = 8 * GROUP_B;
    static constexpr uint32_t ACT_UNIT = UNIT_B + COLS * 32 + COLS * 4;  // + group sums (two terms) + scales
    static constexpr uint32_t TILE_F = ROWS * TOK;                       // floats of a partial tile
};

struct F16Args {
    uint64_t n, k;
    const float* x;            // [m, k]
    float* dst;                // [m, n]
    uint32_t m;
    const float* norm_w;       // RMS-normalise the rows of x first
    float norm_eps;
    const float* residual;     // added to the product; may be dst
    float clamp;               // pair
    uint32_t split, row_stride, stages, act_bytes;
    uint32_t cu;               // units of a stage = warps of a team
    uint32_t two_red;          // two buffers of partial sums, or one that a second barrier guards
    int* error_flag;
};

__device__ __forceinline__ void mma_f16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// the same from zero: the accumulator's registers need no clearing
__device__ __forceinline__ void mma_f16_first(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.0f));
}
// (w & mask) | bits
__device__ __forceinline__ uint32_t and_or(uint32_t w, uint32_t mask, uint32_t bits) {
    uint32_t r;
    asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(r) : "r"(w), "r"(mask), "r"(bits));
    return r;
}

// a - b of two pairs of halves
__device__ __forceinline__ uint32_t less(uint32_t a, uint32_t b) {
    const __half2 v = __hsub2(*reinterpret_cast<__half2*>(&a), *reinterpret_cast<__half2*>(&b));
    return *reinterpret_cast<const uint32_t*>(&v);
}

// One unit (256 columns x 16 rows): u0 / u1 its bytes of rows g and g + 8, act its activations.  acc[0, 1]: row g,
// columns 2t and 2t + 1; [2, 3]: row g + 8.
template <uint32_t TYPE, bool PACK>
__device__ __forceinline__ void f16_unit(const uint8_t* u0, const uint8_t* u1, const uint8_t* act, uint32_t lane,
                                         float (&acc)[4]) {
    using S = Shape<PACK>;
    const uint32_t t = lane & 3;
    const uint8_t* b_lane = act + lane * 16;  // lane (g, t): column g, its 16 bytes
    float us[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    // The products of groups G0 .. G0 + GB - 1; a[j]: the weights of a group's two instructions, s0[j] / s1[j] their scales
    // (rows g / g + 8).  Four chains side by side: an instruction takes some 30 cycles to the next one of its chain.
    constexpr uint32_t GB = 4;
    auto groups = [&](uint32_t G0, const uint32_t (&a)[GB][2][4], const float (&s0)[GB], const float (&s1)[GB]) {
        float c[GB][4];
        uint4 b[GB];
#pragma unroll
        for (int plane = PACK ? 1 : 0; plane < 2; ++plane) {  // low terms, then high terms
#pragma unroll
            for (uint32_t j = 0; j < GB; ++j) b[j] = lds128(b_lane + (G0 + j) * S::GROUP_B + (plane ? 0 : COLS * 64));
#pragma unroll
            for (uint32_t j = 0; j < GB; ++j) {
                if (plane == (PACK ? 1 : 0)) mma_f16_first(c[j], a[j][0], b[j].x, b[j].y);
                else mma_f16(c[j], a[j][0], b[j].x, b[j].y);
            }
#pragma unroll
            for (uint32_t j = 0; j < GB; ++j) mma_f16(c[j], a[j][1], b[j].z, b[j].w);
        }
#pragma unroll
        for (uint32_t j = 0; j < GB; ++j) {
            us[0] = fmaf(c[j][0], s0[j], us[0]), us[1] = fmaf(c[j][1], s0[j], us[1]);
            us[2] = fmaf(c[j][2], s1[j], us[2]), us[3] = fmaf(c[j][3], s1[j], us[3]);
        }
    };
    if constexpr (TYPE == T_Q4_K) {
        const uint4 h0 = lds128(u0), h1 = lds128(u1);
        // six-bit scales and minima of pairs 0 .. 3 and 4 .. 7 as bytes (src/kquant_dot.rs:106-118)
        const uint32_t sc0[2] = {h0.y & 0x3F3F3F3Fu, and_or(h0.y >> 2, 0x30303030u, h0.w & 0x0F0F0F0Fu)};
        const uint32_t sc1[2] = {h1.y & 0x3F3F3F3Fu, and_or(h1.y >> 2, 0x30303030u, h1.w & 0x0F0F0F0Fu)};
        // minima: lane t holds those of groups 2t and 2t + 1, for the first and the second terms of the sums
        auto minima = [&](const uint4& h) {
            const uint32_t w = t < 2 ? h.z & 0x3F3F3F3Fu : and_or(h.z >> 2, 0x30303030u, (h.w >> 4) & 0x0F0F0F0Fu);
            return less(__byte_perm(w, 0x64646464u, t & 1 ? 0x4342u : 0x4140u), 0x64006400u);
        };
        const uint32_t m0 = minima(h0), m1 = minima(h1), am[4] = {m0, m1, m0, m1};
        float cm[4];
        const uint2 bm = lds64(act + S::UNIT_B + lane * 8);
        mma_f16_first(cm, am, bm.x, bm.y);
#pragma unroll
        for (uint32_t c0 = 0; c0 < 4; c0 += GB / 2) {
            uint32_t a[GB][2][4];
            float s0[GB], s1[GB];
#pragma unroll
            for (uint32_t cc = 0; cc < GB / 2; ++cc) {
                const uint32_t c = c0 + cc;
                const uint2 p = lds64(u0 + 16 + 32 * c + 8 * t), q = lds64(u1 + 16 + 32 * c + 8 * t);
                const uint32_t w[2][4] = {{p.x, q.x, p.x >> 8, q.x >> 8}, {p.y, q.y, p.y >> 8, q.y >> 8}};
#pragma unroll
                for (uint32_t nib = 0; nib < 2; ++nib) {
                    // columns 8t + (0, 2), (1, 3), (4, 6), (5, 7) of the group: 1024 + q (low nibbles) or 64 + q (high ones, in
                    // place), less that
                    const uint32_t G = 2 * c + nib, j = 2 * cc + nib, mask = nib ? 0x00F000F0u : 0x000F000Fu, one = nib ? 0x54005400u : 0x64006400u;
#pragma unroll
                    for (int h = 0; h < 2; ++h)
#pragma unroll
                        for (int i = 0; i < 4; ++i) a[j][h][i] = less(and_or(w[h][i], mask, one), one);
                    // the scale's byte under the exponent of 2^23
                    const uint32_t sel = 0x7440u | (G & 3);
                    s0[j] = __uint_as_float(__byte_perm(sc0[G >> 2], 0x4B000000u, sel)) - 8388608.0f;
                    s1[j] = __uint_as_float(__byte_perm(sc1[G >> 2], 0x4B000000u, sel)) - 8388608.0f;
                }
            }
            groups(2 * c0, a, s0, s1);
        }
        const float2 f0 = __half22float2(*reinterpret_cast<const __half2*>(&h0.x)), f1 = __half22float2(*reinterpret_cast<const __half2*>(&h1.x));
        const float e0 = f0.y * -32.0f, e1 = f1.y * -32.0f;  // the sums are stored / 32
        const float2 sx = *reinterpret_cast<const float2*>(act + S::UNIT_B + COLS * 32 + t * 8);
        acc[0] = fmaf(fmaf(cm[0], e0, us[0] * f0.x), sx.x, acc[0]);
        acc[1] = fmaf(fmaf(cm[1], e0, us[1] * f0.x), sx.y, acc[1]);
        acc[2] = fmaf(fmaf(cm[2], e1, us[2] * f1.x), sx.x, acc[2]);
        acc[3] = fmaf(fmaf(cm[3], e1, us[3] * f1.x), sx.y, acc[3]);
    } else {
        auto block_scale = [](uint32_t e) {  // 2^(e - 127); e = 255 zeroes the block, e = 0 is subnormal
            return e == 255u ? 0.0f : __uint_as_float(e ? e << 23 : 0x00400000u);
        };
#pragma unroll
        for (uint32_t G0 = 0; G0 < 8; G0 += GB) {
            uint32_t a[GB][2][4];
            float s[2][GB];
#pragma unroll
            for (uint32_t j = 0; j < GB; ++j) {
                const uint32_t at = 17 * (G0 + j) + 1, mis = at & 3;  // the unit is 4-byte aligned
#pragma unroll
                for (uint32_t r = 0; r < 2; ++r) {
                    const uint8_t* p = (r ? u1 : u0) + at - mis + 4 * t;
                    uint32_t w = lds32(p);
                    if (mis) w = __funnelshift_r(w, lds32(p + 4), 8 * mis);
                    uint32_t v[4];
                    e2m1_pairs(w, v);  // values 4t + i and 16 + 4t + i of the block
                    a[j][0][r] = v[0], a[j][0][2 + r] = v[1], a[j][1][r] = v[2], a[j][1][2 + r] = v[3];
                    s[r][j] = block_scale((r ? u1 : u0)[17 * (G0 + j)]);
                }
            }
            groups(G0, a, s[0], s[1]);
        }
        const float2 sx = *reinterpret_cast<const float2*>(act + S::UNIT_B + COLS * 32 + t * 8);
        acc[0] = fmaf(us[0], sx.x, acc[0]), acc[1] = fmaf(us[1], sx.y, acc[1]);
        acc[2] = fmaf(us[2], sx.x, acc[2]), acc[3] = fmaf(us[3], sx.y, acc[3]);
    }
}

// The two 16-byte pieces of a unit that lane l splits: they are what lane t = l % 4 of a quad multiplies in group l / 4.
template <uint32_t TYPE>
__device__ __forceinline__ void load_run(const float* xu, uint32_t lane, float (&v)[8]) {
    const uint32_t o0 = TYPE == T_MXFP4 ? (lane >> 2) * 32 + (lane & 3) * 4 : lane * 8, o1 = o0 + (TYPE == T_MXFP4 ? 16 : 4);
    const float4 a = __ldg(reinterpret_cast<const float4*>(xu + o0)), b = __ldg(reinterpret_cast<const float4*>(xu + o1));
    v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w, v[4] = b.x, v[5] = b.y, v[6] = b.z, v[7] = b.w;
}

// A row's 256 columns into the terms of activation column `col`, by a warp.  act: the unit's region.
template <uint32_t TYPE, bool PACK>
__device__ __forceinline__ void split_unit(float (&v)[8], uint32_t lane, uint32_t col, uint8_t* act) {
    using S = Shape<PACK>;
    const uint32_t G = lane >> 2, t = lane & 3;
    float amax = 0.0f;
#pragma unroll
    for (int j = 0; j < 8; ++j) amax = fmaxf(amax, fabsf(v[j]));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, o));
    // 2^(141 - e) puts the largest value into [2^14, 2^15); infinities keep theirs
    const uint32_t e = __float_as_uint(amax) >> 23, bits = e == 255 ? 127u : min(254u, 268u - e);
    const float scale = __uint_as_float(bits << 23);
    float sum = 0.0f;
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] *= scale, sum += v[j];
    uint32_t hi[4], lo[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        // pairs as the weights come: Q4_K 0 2, 1 3, 4 6, 5 7; MXFP4 0 16, 1 17, 2 18, 3 19 (the run is 0 .. 3, 16 .. 19)
        const int p = TYPE == T_MXFP4 ? j : (j >> 1) * 4 + (j & 1), q = p + (TYPE == T_MXFP4 ? 4 : 2);
        const __half2 h = __floats2half2_rn(v[p], v[q]);
        const float2 f = __half22float2(h);
        const __half2 l = __floats2half2_rn(v[p] - f.x, v[q] - f.y);
        hi[j] = *reinterpret_cast<const uint32_t*>(&h), lo[j] = *reinterpret_cast<const uint32_t*>(&l);
    }
    uint8_t* b = act + G * S::GROUP_B + col * 64 + t * 16;
    *reinterpret_cast<uint4*>(b) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
    *reinterpret_cast<uint4*>(b + (PACK ? 4 * 64 : COLS * 64)) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
    if constexpr (FT<TYPE>::MIN) {
        sum += __shfl_xor_sync(0xFFFFFFFFu, sum, 1);
        sum += __shfl_xor_sync(0xFFFFFFFFu, sum, 2);
        if (t == 0) {
            sum *= 0.03125f;  // 32 values below 2^15
            const __half h = __float2half_rn(sum), l = __float2half_rn(sum - __half2float(h));
            __half* s = reinterpret_cast<__half*>(act + S::UNIT_B + col * 32 + (G >> 1) * 8) + (G & 1);
            // Second terms: behind the first ones, or (PACK) in the low terms' columns, which keeps the first ones' products
            // exact.  Beside them the tensor core cuts off the second ones' last bits, a bias that the codes' exact products
            // do not share.
            const __half zero = __float2half_rn(0.0f);
            s[0] = h, s[2] = PACK ? zero : l;
            if constexpr (PACK) s[4 * 16] = l, s[4 * 16 + 2] = zero;
        }
    }
    if (lane == 0) {
        const float inv = bits == 254 ? __uint_as_float(0x00400000u) : __uint_as_float((254u - bits) << 23);
        float* f = reinterpret_cast<float*>(act + S::UNIT_B + COLS * 32) + col;
        f[0] = inv;
        if constexpr (PACK) f[4] = inv;
    }
}

__device__ __forceinline__ float silu_f16k(float v) { return v / (1.0f + expf(-v)); }

// ── distributed shared memory ──
__device__ __forceinline__ uint32_t map_rank(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void arrive_rank(uint64_t* bar, uint32_t rank) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(map_rank(smem_u32(bar), rank)) : "memory");
}
// mbar_wait whose completion also orders other CTAs' stores
__device__ __forceinline__ bool mbar_wait_cluster(uint64_t* bar, uint32_t parity) {
    const uint32_t addr = smem_u32(bar);
    for (uint32_t it = 0; it < (1u << 26); ++it) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(addr), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}
template <uint32_t TYPE, bool PACK, bool PAIR>
__global__ void __launch_bounds__(THREADS, 1) gemv_f16_kernel(const __grid_constant__ F16Args ga, const __grid_constant__ CUtensorMap map_a,
                                                              const __grid_constant__ CUtensorMap map_b) {
    using S = Shape<PACK>;
    constexpr uint32_t UNIT = FT<TYPE>::UNIT, TOK = S::TOK, TILE_F = S::TILE_F, N_SUB = PAIR ? 2 : 1;
    extern __shared__ __align__(128) uint8_t smem[];
    const uint32_t NS = ga.stages, split = ga.split;
    const uint64_t n = ga.n, k = ga.k;
    const uint32_t rank = split > 1 ? blockIdx.x % split : 0, cid = blockIdx.x / split, n_clusters = gridDim.x / split;
    const uint32_t units = (uint32_t)(k / 256), row_tiles = (uint32_t)((n + ROWS - 1) / ROWS);
    // this rank's units of a row; u_max, the largest share, decides how many tiles a stage holds
    constexpr uint32_t STEP = FT<TYPE>::STEP;
    const uint32_t unit0 = (uint32_t)((uint64_t)(units / STEP) * rank / split) * STEP,
                   U = (uint32_t)((uint64_t)(units / STEP) * (rank + 1) / split) * STEP - unit0;
    const uint32_t u_max = (units / STEP + split - 1) / split * STEP;
    // A stage is `cu` units of a tile.  The consumers form teams of cu warps; a team takes every n_teams-th tile of an item, a warp
    // one unit of each of the tile's stages; the stages of a round of teams come chunk by chunk.  Every team has a ring of its
    // own, `depth` stages that it takes one after another: with one ring for all, a team's wait for a stage's next round could
    // find the round before still on its way, whose parity an mbarrier cannot tell from the one asked for.
    const uint32_t cu = ga.cu, n_teams = min(NCW / cu, MAX_TEAMS), n_chunks = (u_max + cu - 1) / cu, depth = NS / n_teams;
    const uint32_t stage_bytes = ROWS * ga.row_stride;
    // layout: activations | ring | two buffers of the warps' partial sums | partial tiles of the cluster's ranks | mbarriers
    uint8_t* ring = smem + ga.act_bytes;
    float* s_red = reinterpret_cast<float*>(ring + NS * stage_bytes);
    const bool two_red = ga.two_red != 0;
    float* s_x = s_red + (two_red ? 2 : 1) * NCW * TILE_F;  // [team][slot][rank][gate, up][TILE_F]
    uint64_t* full = reinterpret_cast<uint64_t*>(s_x + (split > 1 ? n_teams * SLOTS * split * N_SUB * TILE_F : 0));
    uint64_t *empty = full + NS, *x_full = empty + NS, *x_free = x_full + n_teams * SLOTS;  // x_full[team][slot], x_free[team][rank][slot]
    __shared__ float s_rs[MAX_SPLIT * GEMV_F16_MAX_M];  // sums of squares [rank][row]
    __shared__ uint64_t norm_full;

    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t out_warps = min(cu, TILE_F / 32);  // warps of a team that add a tile's partial sums
    if (tid == 0) {
        for (uint32_t s = 0; s < NS; ++s) mbar_init(&full[s], 1), mbar_init(&empty[s], cu);
        mbar_init(&norm_full, split);
        if (split > 1) {
            for (uint32_t b = 0; b < n_teams * SLOTS; ++b) mbar_init(&x_full[b], split * out_warps);
            for (uint32_t b = 0; b < n_teams * split * SLOTS; ++b) mbar_init(&x_free[b], out_warps);
        }
        mbar_fence_init();
    }
    __syncthreads();
    if (split > 1) cluster_sync_all();  // the ranks' mbarriers exist
    pdl_trigger();
    if (warp != 0) pdl_wait();  // the weights do not depend on the kernel in front
    const uint32_t tiles = cid < row_tiles ? (row_tiles - cid + n_clusters - 1) / n_clusters : 0;  // cid, cid + n_clusters, ...
    bool ok = true;
    auto check = [&](bool done) {
        if (!done) {
            ok = false;
            *reinterpret_cast<volatile int*>(ga.error_flag) = 1;
        }
    };

    if (warp == 0) {
        // ── producer: one thread, one box of 16 rows per tile of a stage ──
        if (lane == 0) {
            uint32_t next[MAX_TEAMS];  // per team: its next stage, parity in bit 16
            for (uint32_t i = 0; i < n_teams; ++i) next[i] = 0;
            for (uint32_t t0 = 0; t0 < tiles && ok; t0 += n_teams) {
                const uint32_t nt = min(n_teams, tiles - t0);
                for (uint32_t ch = 0; ch < N_SUB * n_chunks && ok; ++ch) {
                    const bool up = ch >= n_chunks;
                    const uint32_t x = (unit0 + (up ? ch - n_chunks : ch) * cu) * (UNIT / 8);
                    for (uint32_t team = 0; team < nt; ++team) {
                        const uint32_t at = next[team] & 0xFFFFu, par = next[team] >> 16, st = team * depth + at;
                        check(mbar_wait(&empty[st], par ^ 1));
                        if (!ok) break;
                        mbar_arrive_expect_tx(&full[st], stage_bytes);  // (what lies behind the row's end comes as zeros)
                        tma_load_2d(ring + st * stage_bytes, PAIR && up ? &map_b : &map_a, x, (cid + (t0 + team) * n_clusters) * ROWS, &full[st]);
                        next[team] = at + 1 == depth ? (par ^ 1) << 16 : next[team] + 1;
                    }
                }
            }
        }
        __syncwarp();
    } else {
        // ── consumers ──
        const uint32_t cw = warp - 1, g = lane >> 2, t = lane & 3;
        const uint32_t team = cw / cu, uw = cw % cu, mine_at = g * ga.row_stride + uw * UNIT;
        constexpr uint32_t OUT = TILE_F / 64;  // of a tile's values, a thread's at most (a team has two warps or more)
        const uint32_t tt = uw * 32 + lane, hop = cu * 32;
        auto store = [&](uint32_t tile, const float (&gate)[OUT], const float (&v)[OUT]) {
#pragma unroll
            for (uint32_t q = 0; q < OUT; ++q) {
                const uint32_t o = tt + hop * q, row = o / TOK, tok = o % TOK;
                if (o >= TILE_F || tok >= ga.m || (uint64_t)tile * ROWS + row >= n) continue;
                float y = v[q];
                if constexpr (PAIR) {
                    float gv = gate[q];
                    if (ga.clamp > 0.0f) {
                        gv = fminf(gv, ga.clamp);
                        y = fmaxf(-ga.clamp, fminf(y, ga.clamp));
                    }
                    y = silu_f16k(gv) * y;
                }
                const uint64_t at = (uint64_t)tok * n + (uint64_t)tile * ROWS + row;
                if (!PAIR && ga.residual != nullptr) y += ga.residual[at];
                ga.dst[at] = y;
            }
        };
        // Split: tile number seq of a team goes to that team in rank seq % split, which finishes it when it has sent its part of
        // its next one: the other ranks are through by then, and none waits for another tile by tile.
        uint32_t seq = 0, held_seq = 0, held_tile = 0;
        bool held = false;
        float* s_xt = s_x + team * SLOTS * split * N_SUB * TILE_F;
        auto finish = [&] {
            if (!held || !ok) return;
            held = false;
            const uint32_t slot = held_seq / split % SLOTS;
            check(__all_sync(0xFFFFFFFFu, mbar_wait_cluster(&x_full[team * SLOTS + slot], held_seq / split / SLOTS & 1)));
            if (!ok) return;
            float gate[OUT], v[OUT];
#pragma unroll
            for (uint32_t q = 0; q < OUT; ++q) gate[q] = v[q] = 0.0f;
            for (uint32_t r = 0; r < split; ++r)
#pragma unroll
                for (uint32_t q = 0; q < OUT; ++q) {
                    if (tt + hop * q >= TILE_F) continue;
                    const float* p = s_xt + (slot * split + r) * N_SUB * TILE_F + tt + hop * q;
                    if (PAIR) gate[q] += p[0];
                    v[q] += p[PAIR ? TILE_F : 0];
                }
            __syncwarp();
            if (lane < split) arrive_rank(&x_free[(team * split + rank) * SLOTS + slot], lane);
            store(held_tile, gate, v);
        };
        uint32_t at = 0, par = 0, rb = 0;  // the team's next stage, its buffer of partial sums
        // Activations: a warp takes one unit (or every 16th) of every row (of every pn-th, where the units are few), four rows'
        // loads ahead of their use.
        const uint32_t pn = U < NCW ? NCW / U : 1, pu = U < NCW ? cw % U : cw, pr = cw / max(U, 1u) * (U < NCW ? 1 : 0);
        const uint32_t p_rows = U < NCW && pr >= pn ? 0 : TOK;  // 16 is no multiple of U: the last warps rest
        float row_scale = 1.0f;                                 // of row `lane`
        if (ga.norm_w != nullptr) {
            // the rows' sums of squares: units in unit order (in the idle buffers of partial sums), ranks in rank order
            for (uint32_t u = pu; u < U; u += NCW > U ? U : NCW)
                for (uint32_t r0 = pr; r0 < min(p_rows, ga.m); r0 += 4 * pn) {
                    float v[4][8];
#pragma unroll
                    for (uint32_t j = 0; j < 4; ++j)
                        load_run<TYPE>(ga.x + (uint64_t)min(r0 + j * pn, ga.m - 1) * k + (uint64_t)(unit0 + u) * 256, lane, v[j]);
#pragma unroll
                    for (uint32_t j = 0; j < 4; ++j) {
                        float ss = 0.0f;
#pragma unroll
                        for (int i = 0; i < 8; ++i) ss = fmaf(v[j][i], v[j][i], ss);
#pragma unroll
                        for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xFFFFFFFFu, ss, o);
                        if (lane == 0 && r0 + j * pn < ga.m) s_red[u * TOK + r0 + j * pn] = ss;
                    }
                }
            asm volatile("bar.sync 1, %0;" ::"n"(NCW * 32) : "memory");
            float ss = 0.0f;
            if (lane < ga.m)
#pragma unroll 4
                for (uint32_t u = 0; u < U; ++u) ss += s_red[u * TOK + lane];
            if (split > 1) {
                if (warp == 1) {
                    if (lane < ga.m)
                        for (uint32_t r = 0; r < split; ++r)
                            asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(map_rank(smem_u32(s_rs + rank * GEMV_F16_MAX_M + lane), r)),
                                         "f"(ss)
                                         : "memory");
                    asm volatile("fence.acq_rel.cluster;" ::: "memory");
                    __syncwarp();
                    if (lane < split) arrive_rank(&norm_full, lane);
                }
                check(__all_sync(0xFFFFFFFFu, mbar_wait_cluster(&norm_full, 0)));
                ss = 0.0f;
                if (lane < ga.m)
                    for (uint32_t r = 0; r < split; ++r) ss += s_rs[r * GEMV_F16_MAX_M + lane];
            }
            row_scale = rsqrtf(ss / (float)k + ga.norm_eps);
        }
        for (uint32_t u = pu; u < U; u += NCW > U ? U : NCW) {
            float w[8];
            if (ga.norm_w != nullptr) load_run<TYPE>(ga.norm_w + (uint64_t)(unit0 + u) * 256, lane, w);
            for (uint32_t r0 = pr; r0 < p_rows; r0 += 4 * pn) {
                float v[4][8];
#pragma unroll
                for (uint32_t j = 0; j < 4; ++j)
                    load_run<TYPE>(ga.x + (uint64_t)min(r0 + j * pn, ga.m - 1) * k + (uint64_t)(unit0 + u) * 256, lane, v[j]);
#pragma unroll
                for (uint32_t j = 0; j < 4; ++j) {
                    const uint32_t row = r0 + j * pn;
                    if (row >= TOK) break;
                    if (row >= ga.m) {
#pragma unroll
                        for (int i = 0; i < 8; ++i) v[j][i] = 0.0f;
                    } else if (ga.norm_w != nullptr) {
                        const float rs = __shfl_sync(0xFFFFFFFFu, row_scale, row);
#pragma unroll
                        for (int i = 0; i < 8; ++i) v[j][i] = v[j][i] * rs * w[i];
                    }
                    split_unit<TYPE, PACK>(v[j], lane, row, smem + u * S::ACT_UNIT);
                }
            }
        }
        asm volatile("bar.sync 1, %0;" ::"n"(NCW * 32) : "memory");
        for (uint32_t ti = team < n_teams ? team : tiles; ti < tiles; ti += n_teams) {  // (warps that do not fill a team: none)
            const uint32_t tile = cid + ti * n_clusters;
            float gate[OUT], v[OUT];
#pragma unroll
            for (uint32_t sub = 0; sub < N_SUB; ++sub, rb ^= two_red ? 1 : 0) {
                float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
                for (uint32_t u = uw; u < n_chunks * cu; u += cu) {
                    const uint32_t st = team * depth + at;
                    if (ok) check(__all_sync(0xFFFFFFFFu, mbar_wait(&full[st], par)));
                    if (ok && u < U) {
                        const uint8_t* sp = ring + st * stage_bytes + mine_at;
                        f16_unit<TYPE, PACK>(sp, sp + 8 * ga.row_stride, smem + u * S::ACT_UNIT, lane, acc);
                    }
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&empty[st]);
                    if (++at == depth) at = 0, par ^= 1;
                }
                // the team's partial sums, [warp][row][token], added in unit order
                if (!two_red) asm volatile("bar.sync %0, %1;" ::"r"(2 + team), "r"(hop) : "memory");
                float* red = s_red + (rb * NCW + team * cu) * TILE_F;
                if constexpr (PACK) {
#pragma unroll
                    for (int j = 0; j < 4; ++j) acc[j] += __shfl_xor_sync(0xFFFFFFFFu, acc[j], 2);  // high + low terms
                }
                if (!PACK || t < 2) {
                    *reinterpret_cast<float2*>(red + uw * TILE_F + g * TOK + 2 * t) = make_float2(acc[0], acc[1]);
                    *reinterpret_cast<float2*>(red + uw * TILE_F + (g + 8) * TOK + 2 * t) = make_float2(acc[2], acc[3]);
                }
                asm volatile("bar.sync %0, %1;" ::"r"(2 + team), "r"(hop) : "memory");
                if (PAIR && sub == 1)
#pragma unroll
                    for (uint32_t q = 0; q < OUT; ++q) gate[q] = v[q];
#pragma unroll
                for (uint32_t q = 0; q < OUT; ++q) v[q] = 0.0f;
                if (uw < out_warps)
#pragma unroll 4
                    for (uint32_t p = 0; p < cu; ++p)
#pragma unroll
                        for (uint32_t q = 0; q < OUT; ++q)
                            if (q == 0 || tt + hop * q < TILE_F) v[q] += red[p * TILE_F + tt + hop * q];
            }
            if (uw >= out_warps || !ok) continue;
            if (split == 1) {
                store(tile, gate, v);
                continue;
            }
            const uint32_t dest = seq % split, slot = seq / split % SLOTS;
            check(__all_sync(0xFFFFFFFFu, mbar_wait_cluster(&x_free[(team * split + dest) * SLOTS + slot], (seq / split / SLOTS & 1) ^ 1)));
            if (!ok) continue;
            const uint32_t to = map_rank(smem_u32(s_xt + (slot * split + rank) * N_SUB * TILE_F + tt), dest);
#pragma unroll
            for (uint32_t q = 0; q < OUT; ++q) {
                if (tt + hop * q >= TILE_F) continue;
                if (PAIR) asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(to + hop * q * 4), "f"(gate[q]) : "memory");
                asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(to + (PAIR ? TILE_F * 4 : 0) + hop * q * 4), "f"(v[q]) : "memory");
            }
            asm volatile("fence.acq_rel.cluster;" ::: "memory");
            __syncwarp();
            if (lane == 0) arrive_rank(&x_full[team * SLOTS + slot], dest);
            if (dest == rank) {
                finish();
                held = true, held_seq = seq, held_tile = tile;
            }
            ++seq;
        }
        finish();
    }
    if (split > 1) {
        __syncthreads();
        cluster_sync_all();  // no CTA leaves while another writes to its shared memory
    }
}

// ── host side ──
struct F16Plan {
    uint32_t split, cu, row_stride, stages, act_bytes, two_red, total;
};

// The smallest split of k whose activations leave room for two stages a team.
template <uint32_t TYPE, bool PACK>
bool f16_plan(uint64_t n, uint64_t k, bool pair, F16Plan* p) {
    using S = Shape<PACK>;
    constexpr uint32_t STEP = FT<TYPE>::STEP;
    const uint32_t units = (uint32_t)(k / 256);
    if (units % STEP != 0) return false;
    for (uint32_t split = 1; split <= MAX_SPLIT && split * STEP <= units; split *= 2) {
        const uint32_t u_max = (units / STEP + split - 1) / split * STEP;
        // the teams' rounds over a cluster's tiles x (a warp's units of one + handing its sums over, about half a unit's time)
        const uint64_t steps = ((n + ROWS - 1) / ROWS * split + num_sms() - 1) / num_sms();
        uint64_t best = ~0ull;
        for (uint32_t cu = std::max(2u, std::min(u_max, NCW / 2)); cu >= std::max(2u, std::min(u_max, 3u)); --cu) {
            const uint32_t teams = std::min(NCW / cu, MAX_TEAMS), words = cu * FT<TYPE>::UNIT / 4;
            const uint64_t cost = (steps + teams - 1) / teams * (2 * ((u_max + cu - 1) / cu) + 1);
            if (cu % STEP != 0 || cost >= best) continue;
            const uint32_t stride = (words + (FT<TYPE>::STRIDE_MOD + 32 - words % 32) % 32) * 4;
            const uint64_t stage = (uint64_t)ROWS * stride, act = ((uint64_t)u_max * S::ACT_UNIT + 127) / 128 * 128, red = NCW * S::TILE_F * 4;
            const uint64_t fixed = act + red + (split > 1 ? teams * SLOTS * split * (pair ? 2 : 1) * S::TILE_F * 4 : 0) +
                                   8 * (2 * MAX_STAGES + teams * SLOTS * (1 + split));
            const uint64_t ring = 2 * teams * stage;
            if (fixed + ring > SMEM_MAX) continue;
            best = cost;
            p->split = split, p->cu = cu, p->row_stride = stride, p->act_bytes = (uint32_t)act;
            p->two_red = fixed + red + ring <= SMEM_MAX;
            p->stages = teams * (uint32_t)std::min<uint64_t>(MAX_STAGES / teams, (SMEM_MAX - fixed - p->two_red * red) / stage / teams);
            p->total = (uint32_t)(fixed + p->two_red * red + p->stages * stage);
        }
        if (best != ~0ull) return true;
    }
    return false;
}

// The blocks as rows of 64-bit words; a box is 16 rows of a stage's units and what pads them to the fragment loads' stride.
cudaError_t f16_weight_map(const uint8_t* w, uint64_t rows, uint64_t row_bytes, uint32_t box_bytes, CUtensorMap* out) {
    static PFN_cuTensorMapEncodeTiled encode = nullptr;
    if (!encode) {
        void* fn = nullptr;
        cudaDriverEntryPointQueryResult qres;
        if (cudaError_t e = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qres); e != cudaSuccess) return e;
        if (qres != cudaDriverEntryPointSuccess || !fn) return cudaErrorNotSupported;
        encode = reinterpret_cast<PFN_cuTensorMapEncodeTiled>(fn);
    }
    const cuuint64_t dims[2] = {row_bytes / 8, rows}, strides[1] = {row_bytes};
    const cuuint32_t box[2] = {box_bytes / 8, ROWS}, estr[2] = {1, 1};
    const CUresult r = encode(out, CU_TENSOR_MAP_DATA_TYPE_INT64, 2, const_cast<uint8_t*>(w), dims, strides, box, estr,
                              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);  // rows and columns beyond the array read as zeros
    return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

template <uint32_t TYPE, bool PACK, bool PAIR>
cudaError_t f16_launch(F16Args& ga, const uint8_t* w_a, const uint8_t* w_b, cudaStream_t s) {
    F16Plan p;
    if (!f16_plan<TYPE, PACK>(ga.n, ga.k, PAIR, &p)) return cudaErrorInvalidValue;
    ga.split = p.split, ga.cu = p.cu, ga.two_red = p.two_red, ga.row_stride = p.row_stride, ga.stages = p.stages, ga.act_bytes = p.act_bytes;
    auto kern = gemv_f16_kernel<TYPE, PACK, PAIR>;
    static bool configured[MAX_DEVICES] = {};
    if (cudaError_t ce = set_max_smem_once(kern, (int)SMEM_MAX, configured); ce != cudaSuccess) return ce;
    CUtensorMap map_a, map_b;
    const uint64_t row_bytes = ga.k / 256 * FT<TYPE>::UNIT;
    if (cudaError_t e = f16_weight_map(w_a, ga.n, row_bytes, p.row_stride, &map_a); e != cudaSuccess) return e;
    if constexpr (PAIR) {
        if (cudaError_t e = f16_weight_map(w_b, ga.n, row_bytes, p.row_stride, &map_b); e != cudaSuccess) return e;
    } else {
        map_b = map_a;  // not read
    }
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = p.split;
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = p.split > 1 ? 2 : 1;
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = p.total;
    cfg.stream = s;
    // clusters that are resident at once (the GPCs' SM counts are no multiples of every cluster size)
    static int resident[MAX_DEVICES][MAX_SPLIT + 1] = {};
    int& fit = resident[current_device()][p.split];
    if (fit == 0) {
        int c = num_sms() / (int)p.split;
        if (p.split > 1) {
            cfg.gridDim = dim3(p.split);
            if (cudaError_t e = cudaOccupancyMaxActiveClusters(&c, kern, &cfg); e != cudaSuccess) return e;
        }
        fit = std::max(1, c);
    }
    const uint64_t row_tiles = (ga.n + ROWS - 1) / ROWS;
    const uint64_t clusters = std::min<uint64_t>((uint64_t)fit, row_tiles);
    cfg.gridDim = dim3((unsigned)(clusters * p.split));
    cudaError_t e = cudaLaunchKernelEx(&cfg, kern, ga, map_a, map_b);
    return e != cudaSuccess ? e : cudaGetLastError();
}

template <uint32_t TYPE, bool PAIR>
cudaError_t f16_rows(F16Args& ga, const uint8_t* w_a, const uint8_t* w_b, cudaStream_t s) {
    return ga.m <= 4 ? f16_launch<TYPE, true, PAIR>(ga, w_a, w_b, s) : f16_launch<TYPE, false, PAIR>(ga, w_a, w_b, s);
}

}  // namespace

bool gemv_f16_supports(uint32_t type, const uint8_t* w, uint64_t n, uint64_t k, uint64_t m, bool pair) {
    if (m < GEMV_F16_MIN_M || m > GEMV_F16_MAX_M || n == 0 || k < MIN_K || k % 256 != 0 || n > 0x7FFFFFFFu || k > 0x7FFFFFFFu) return false;
    const uintptr_t a = reinterpret_cast<uintptr_t>(w);
    F16Plan p;
    auto fits = [&](auto t) {
        constexpr uint32_t TYPE = decltype(t)::value;
        return m <= 4 ? f16_plan<TYPE, true>(n, k, pair, &p) : f16_plan<TYPE, false>(n, k, pair, &p);
    };
    switch (type) {
        case T_Q4_K: return a % 16 == 0 && fits(std::integral_constant<uint32_t, T_Q4_K>{});
        // five to eight rows with k split stay on tiles: 4096 x 7168 14.2 us there and 16.8 here, 7168 x 16384 40.7 and 46.1,
        // 4096 x 14336 23.8 and 25.6 (the other way round for few rows of weights and very many: 1536 x 7168 13.9 and 12.7,
        // 24576 x 7168 61.2 and 57.5)
        case T_MXFP4: return a % 16 == 0 && fits(std::integral_constant<uint32_t, T_MXFP4>{}) && (m <= 4 || p.split == 1);
        default: return false;
    }
}

cudaError_t launch_gemv_f16(uint32_t type, const uint8_t* w_a, const uint8_t* w_b, uint64_t n, uint64_t k, const float* lhs,
                            uint64_t m, const float* norm_w, float eps, const float* residual, float clamp, float* dst,
                            int* error_flag, cudaStream_t s) {
    F16Args ga = {};
    ga.n = n, ga.k = k, ga.m = (uint32_t)m;
    ga.x = lhs, ga.dst = dst;
    ga.norm_w = norm_w, ga.norm_eps = eps;
    ga.residual = residual, ga.clamp = clamp;
    ga.error_flag = error_flag;
    switch (type) {
        case T_Q4_K: return w_b ? f16_rows<T_Q4_K, true>(ga, w_a, w_b, s) : f16_rows<T_Q4_K, false>(ga, w_a, w_b, s);
        case T_MXFP4: return w_b ? f16_rows<T_MXFP4, true>(ga, w_a, w_b, s) : f16_rows<T_MXFP4, false>(ga, w_a, w_b, s);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace jq
