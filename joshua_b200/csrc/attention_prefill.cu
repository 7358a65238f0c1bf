// Causal attention of a prompt's tokens over the KV cache on the 5th-generation tensor cores, in 16-bit terms that keep
// f32's precision.
//
// `seq` new tokens of ONE sequence at positions pos0 .. pos0 + seq - 1 (the cache already holds their k / v rows):
// out[s, head, :] = softmax(q_s . K[0 .. pos0 + s]^T / sqrt(hd)) V (src/quantized_qwen3_moe.rs:366-386 with the causal
// mask of :805-812).  One CTA per (128 queries, q head), 64 keys at a time, running maximum and sum in f32.
//
// Queries and keys are split into two f16 terms under a power-of-two scale of their row that puts its largest value just
// below 2^15, which keeps 22 to 24 bits of every value within 2^17 of the largest and an absolute error below 2^-39 of it
// otherwise; a product is three products of terms (lo * hi, hi * lo, hi * hi).  Probabilities and values are three bf16
// terms each, which hold f32's 24 bits at any size: values share tiles of keys with values that a query must not see, and
// with a scale over them (f16 terms had one) a later token would move an earlier one's result.  Their product is the six
// products of terms above 2^-24.  The tensor core forms the products exactly and adds with truncation, so accumulators are
// short: 64 dimensions of a score, the 64 keys of a tile for the output, small products first; they are read back and added
// round-to-nearest in registers, where the running output lives.  A value that is not finite stands as zero in the products
// and is added at the end, where it is seen.  Error against float64 (2-norm, N(0, 1)
// rows, 1000 tokens, 32 q / 4 kv heads of 128): 1.8e-7, an f32 kernel on the CUDA cores 3.9e-7 (queries four times as large:
// 3.8e-7, 1.08e-6; a value of 1e6 beside the others, that dimension: 1.0e-7 to 1.7e-7, 1.5e-7 to 2.7e-7).
//
// Warps: 0 .. 7 softmax, two threads a query (32 keys and half of the output dimensions each); 8 .. 15 convert the key and
// value tiles into swizzled K-major tiles (values transposed: keys run along a row), two stages; 16 issues the products.
// Tensor memory: the query's terms (the A operand of the scores), scores, probabilities (A of the output), output of a tile.
//
// What bounds it: a tile of 64 keys takes 2.9 us (hd 128, 4096 tokens), of which the tensor pipe works 2304 cycles; the rest is
// the softmax threads' chain (read the scores, maximum, exponentials, terms, add the output before) and the issue slots that
// they share with the converters.  The f32 rows come by one bulk copy a tile, ahead of the converters: with loads into
// registers instead a tile took 1.7 times as long.  Measured against an f32 kernel on the CUDA cores, 32 heads of 128 (in a
// graph): 1000 tokens 57.9 us (248), 512 29.7 (128), 256 19.5 (62), 128 14.8 (29), 16 6.0 (10.7), one 5.8 (10.2); heads of 64,
// 1000 tokens 34.1 (152): ahead at every size, so it is the only route.  (Values in two f16 terms: 52.0, 26.7, 17.8, 13.7, 5.9,
// 5.6; 32.5.)
//
// Every wait on an mbarrier is bounded.  A warp whose wait ran out hands nothing on (the waits that depend on it run out in
// turn) but still comes to every named barrier that others expect it at, so that all warps reach the common exit, where
// tensor memory is released.  The status flag is raised and the rows of the CTA are NaN.
#include <cuda_fp16.h>

#include <algorithm>
#include <cmath>

#include "common.cuh"
#include "tc5.cuh"

namespace jq {

namespace {

constexpr uint32_t AQ = 128, AK = 64;        // queries and keys of a tile
constexpr uint32_t A_SOFT = 8, A_CONV = 8;   // warps
constexpr uint32_t A_THREADS = (A_SOFT + A_CONV + 4) * 32;  // whole warpgroups: they trade registers
// Registers a thread: the launch has 640 x 96 = 61440, of which the issuer's warpgroup keeps 128 x 32, the converters
// 256 x 72 and the softmax threads (64 running outputs, 32 scores, 48 terms) 256 x 152: all of it.
constexpr int A_REGS_ISSUE = 32, A_REGS_CONV = 72, A_REGS_SOFT = 152;
static_assert(128 * A_REGS_ISSUE + A_CONV * 32 * A_REGS_CONV + A_SOFT * 32 * A_REGS_SOFT <= A_THREADS * 96, "registers");

// what the warps share beside the tiles
struct AttShared {
    uint16_t ks[4][AK];       // inverse scales of key rows, by tile % 4: powers of two (or infinity), so their upper halves
    float row[2][2][AQ];      // row maxima of the two halves
    uint64_t k_full[2], k_empty[2], v_full[2], v_empty[2], s_full, s_free, p_full, o_full;
    uint64_t rk_full, rk_empty, rv_full, rv_empty;  // the raw rows
    uint64_t drained;         // the products of a CTA that gives up
    uint32_t tmem_slot;
    int abort_flag;
    uint32_t odd_first, odd_end;  // key tiles that hold a value that is not finite: none, or within these
};

template <uint32_t HD>
struct AttTile {
    static constexpr uint32_t HALVES = HD / 64;              // 64-dimension accumulators of a score
    static constexpr uint32_t K_PLANE = AK * 128;            // 64 dimensions of the tile's keys, one term
    static constexpr uint32_t K_STAGE = 2 * HALVES * K_PLANE;
    static constexpr uint32_t V_PLANE = HD * 128;            // the tile's keys of every dimension, one term
    static constexpr uint32_t V_STAGE = 3 * V_PLANE;
    static constexpr uint32_t RAW = AK * HD * 4;             // the f32 rows of a tile's keys or values
    static constexpr uint32_t SMEM = 2 * (K_STAGE + V_STAGE) + 2 * RAW + sizeof(AttShared);
    static_assert(SMEM <= 227 * 1024, "shared memory");
    // tensor memory columns
    static constexpr uint32_t Q_HI = 0, Q_LO = HD / 2, S0 = HD, P0 = S0 + 64 * HALVES, O = P0 + 128;
    static_assert(O + HD <= 512, "tensor memory");
};

// power of two that puts a largest magnitude just below 2^15, as exponent bits; infinities keep theirs
__device__ __forceinline__ uint32_t term_scale_bits(float amax) {
    const uint32_t e = __float_as_uint(amax) >> 23;
    return e == 255 ? 127u : min(254u, 268u - e);
}
__device__ __forceinline__ float bits_scale(uint32_t bits) { return __uint_as_float(bits << 23); }
__device__ __forceinline__ float bits_inverse(uint32_t bits) {  // 2^-127 is a subnormal
    return bits == 254 ? __uint_as_float(0x00400000u) : __uint_as_float((254u - bits) << 23);
}
__device__ __forceinline__ void split_pair(float a, float b, uint32_t* hi, uint32_t* lo) {
    const __half2 h = __floats2half2_rn(a, b);
    const float2 f = __half22float2(h);
    const __half2 l = __floats2half2_rn(a - f.x, b - f.y);
    *hi = *reinterpret_cast<const uint32_t*>(&h);
    *lo = *reinterpret_cast<const uint32_t*>(&l);
}
// a and b as the sum of three bf16 terms each, rounded one after another
__device__ __forceinline__ void split3_pair(float a, float b, uint32_t (&t)[3]) {
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(t[i]) : "f"(b), "f"(a));
        a -= __uint_as_float(t[i] << 16), b -= __uint_as_float(t[i] & 0xFFFF0000u);
    }
}
// the same, exact and without overflow: cut off, not rounded
__device__ __forceinline__ void cut3_pair(float a, float b, uint32_t (&t)[3]) {
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        t[i] = __byte_perm(__float_as_uint(a), __float_as_uint(b), 0x7632);
        a -= __uint_as_float(__float_as_uint(a) & 0xFFFF0000u), b -= __uint_as_float(__float_as_uint(b) & 0xFFFF0000u);
    }
}
__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float lds_f32(uint32_t addr) {
    float v;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(addr));
    return v;
}
__device__ __forceinline__ float4 lds_f32x4(uint32_t addr) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr));
    return v;
}
__device__ __forceinline__ void st_shared_v4(uint32_t addr, const uint32_t (&v)[4]) {
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]) : "memory");
}

template <uint32_t HD>
__global__ void __launch_bounds__(A_THREADS, 1)
    attention_prefill_kernel(const float* __restrict__ q, const float* __restrict__ cache_k, const float* __restrict__ cache_v,
                             const int32_t* __restrict__ pos, uint32_t seq, uint32_t nq, uint32_t nkv, uint32_t max_ctx,
                             float* __restrict__ out, int32_t* __restrict__ bad_pos, int* __restrict__ error_flag) {
    using T = AttTile<HD>;
    extern __shared__ __align__(1024) uint8_t smem[];  // K and V stages | raw rows | AttShared
    const uint32_t k_base = smem_u32(smem), v_base = k_base + 2 * T::K_STAGE;
    uint8_t* raw_k = smem + 2 * (T::K_STAGE + T::V_STAGE);
    uint8_t* raw_v = raw_k + T::RAW;
    AttShared& sh = *reinterpret_cast<AttShared*>(raw_v + T::RAW);

    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    pdl_trigger();
    if (k_base % 1024 != 0) {  // the swizzle's period; no static shared memory stands in front
        if (tid == 0 && error_flag) *reinterpret_cast<volatile int*>(error_flag) = 1;
        return;
    }
    if (tid == 0) {
        sh.odd_first = 0xFFFFFFFFu, sh.odd_end = 0;
        for (int i = 0; i < 2; ++i) {
            mbar_init(&sh.k_full[i], A_CONV);
            mbar_init(&sh.v_full[i], A_CONV);
            mbar_init(&sh.k_empty[i], 1);
            mbar_init(&sh.v_empty[i], 1);
        }
        mbar_init(&sh.s_full, 1);
        mbar_init(&sh.s_free, A_SOFT);
        mbar_init(&sh.p_full, A_SOFT);
        mbar_init(&sh.o_full, 1);
        mbar_init(&sh.rk_full, 1);
        mbar_init(&sh.rv_full, 1);
        mbar_init(&sh.rk_empty, A_CONV);
        mbar_init(&sh.rv_empty, A_CONV);
        mbar_init(&sh.drained, 1);
        sh.abort_flag = 0;
        mbar_fence_init();
    }
    if (warp == A_SOFT + A_CONV) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sh.tmem_slot)), "r"(512u)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = sh.tmem_slot;
    pdl_wait();
    // heads run fastest, the last queries first: they see the most keys, and a long CTA in the last wave leaves the
    // other SMs waiting
    const uint32_t head = blockIdx.x, kvh = head / (nq / nkv), s0 = (gridDim.y - 1 - blockIdx.y) * AQ;
    const int32_t p0 = pos[0];
    const bool in_cache = p0 >= 0 && (uint64_t)p0 + seq <= max_ctx;
    if (!in_cache && tid == 0 && bad_pos) atomicExch(bad_pos, 1);
    const uint32_t n_keys = in_cache ? (uint32_t)p0 + min(seq, s0 + AQ) : 0;  // keys the newest query of the tile sees
    const uint32_t n_tiles = (n_keys + AK - 1) / AK;
    bool ok = true;  // the same in all lanes of a warp; once false, the warp waits for nothing more
    auto wait_all = [&](uint64_t* bar, uint32_t parity) {
        return ok = __all_sync(0xFFFFFFFFu, mbar_wait(bar, parity));
    };
    // The common exit, where all warps meet: whether some wait of the CTA ran out.
    auto leave = [&] {
        if (!ok && lane == 0) *static_cast<volatile int*>(&sh.abort_flag) = 1;
        tc_fence_before();
        asm volatile("bar.sync 6, %0;" ::"n"(A_THREADS) : "memory");
        return *static_cast<volatile int*>(&sh.abort_flag) != 0;
    };

    if (warp < A_SOFT) {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(A_REGS_SOFT));
        if (in_cache) {
            // ── softmax: thread = (query row, half) ──
            const uint32_t quarter = warp & 3, half = warp >> 2, row = quarter * 32 + lane, sr = s0 + row;
            const uint32_t lanes = tmem + ((quarter * 32) << 16);
            constexpr uint32_t DN = HD / 2;  // dimensions of this thread
            float rf;                        // inverse scale of the query row, times log2(e) / sqrt(hd)
            auto pair_bar = [&] { asm volatile("bar.sync %0, 64;" ::"r"(1 + quarter) : "memory"); };
            float o[DN];
            {
                const float4* src = reinterpret_cast<const float4*>(q + ((uint64_t)min(sr, seq - 1) * nq + head) * HD + half * DN);
                float amax = 0.0f;
#pragma unroll
                for (uint32_t i = 0; i < DN / 4; ++i) {
                    const float4 v = sr < seq ? __ldg(src + i) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                    o[4 * i] = v.x, o[4 * i + 1] = v.y, o[4 * i + 2] = v.z, o[4 * i + 3] = v.w;
                    amax = fmaxf(amax, fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w))));
                }
                sh.row[1][half][row] = amax;
                pair_bar();
                const uint32_t bits = term_scale_bits(fmaxf(amax, sh.row[1][half ^ 1][row]));
                const float sc = bits_scale(bits);
                rf = bits_inverse(bits) * (rsqrtf((float)HD) * 1.44269504f);
#pragma unroll
                for (uint32_t c = 0; c < DN / 32; ++c) {
                    uint32_t hi[16], lo[16];
#pragma unroll
                    for (uint32_t i = 0; i < 16; ++i) split_pair(o[32 * c + 2 * i] * sc, o[32 * c + 2 * i + 1] * sc, &hi[i], &lo[i]);
                    tmem_st16(lanes + T::Q_HI + half * (DN / 2) + 16 * c, hi);
                    tmem_st16(lanes + T::Q_LO + half * (DN / 2) + 16 * c, lo);
                }
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&sh.s_free);  // the first scores wait for the query's terms
            }
#pragma unroll
            for (uint32_t i = 0; i < DN; ++i) o[i] = 0.0f;
            float mx = -INFINITY, sum = 0.0f, alpha_prev = 0.0f;
            const uint32_t visible = (uint32_t)p0 + sr + 1;                         // keys 0 .. p0 + s (rows past seq: never stored)
            const uint32_t all_see = (uint32_t)p0 + s0 + quarter * 32 + 1;          // keys that every query of the warp sees
            // o = o * alpha + the tile's output
            auto add_tile = [&](uint32_t j, float alpha) {
                if (__any_sync(0xFFFFFFFFu, alpha != 1.0f)) {  // while the products run; the maxima settle after a few tiles
#pragma unroll
                    for (uint32_t i = 0; i < DN; ++i) o[i] *= alpha;
                }
                if (!wait_all(&sh.o_full, j & 1)) return;
                tc_fence_after();
#pragma unroll
                for (uint32_t c = 0; c < DN / 32; ++c) {
                    uint32_t r[32];
                    tmem_ld32(lanes + T::O + half * DN + 32 * c, r);
#pragma unroll
                    for (uint32_t i = 0; i < 32; ++i) o[32 * c + i] += __uint_as_float(r[i]);
                }
            };
            uint32_t j = 0;  // tiles whose barrier this warp has come to
            while (j < n_tiles) {
                const uint32_t t0 = j * AK + half * 32;  // this thread's first key
                float sc[32];
                if (!wait_all(&sh.s_full, j & 1)) break;
                tc_fence_after();
                {
                    uint32_t r[32];
                    tmem_ld32(lanes + T::S0 + half * 32, r);
#pragma unroll
                    for (int i = 0; i < 32; ++i) sc[i] = __uint_as_float(r[i]);
                    if constexpr (T::HALVES == 2) {
                        tmem_ld32(lanes + T::S0 + 64 + half * 32, r);
#pragma unroll
                        for (int i = 0; i < 32; ++i) sc[i] += __uint_as_float(r[i]);
                    }
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&sh.s_free);
                const uint4* ks = reinterpret_cast<const uint4*>(&sh.ks[j & 3][half * 32]);
                float cm = -INFINITY;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const uint4 f = ks[i];
                    const uint32_t w[4] = {f.x, f.y, f.z, f.w};
#pragma unroll
                    for (int h = 0; h < 4; ++h) {
                        sc[8 * i + 2 * h] *= __uint_as_float(w[h] << 16);
                        sc[8 * i + 2 * h + 1] *= __uint_as_float(w[h] & 0xFFFF0000u);
                    }
                }
                if (t0 + 32 > all_see) {
#pragma unroll
                    for (int i = 0; i < 32; ++i) sc[i] = t0 + i < visible ? sc[i] : -INFINITY;
                }
#pragma unroll
                for (int i = 0; i < 32; ++i) cm = fmaxf(cm, sc[i]);
                sh.row[j & 1][half][row] = cm;
                pair_bar();
                // logarithms to base 2 of the probabilities; the maximum is finite from the first tile on: key 0 is
                // visible to every query
                const float nm = fmaxf(mx, fmaxf(cm, sh.row[j & 1][half ^ 1][row]) * rf);
                const float alpha = ex2(mx - nm);  // 0 on the first tile (mx = -inf)
                float ps = 0.0f;
                uint32_t w0[16], w1[16], w2[16];
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    const float a = ex2(fmaf(sc[2 * i], rf, -nm)), b = ex2(fmaf(sc[2 * i + 1], rf, -nm));  // 0 for masked keys
                    ps += a + b;
                    uint32_t t[3];
                    split3_pair(a, b, t);
                    w0[i] = t[0], w1[i] = t[1], w2[i] = t[2];
                }
                sum = sum * alpha + ps;
                mx = nm;
                if (j++ > 0) add_tile(j - 2, alpha_prev);  // its products have read the probabilities before these
                if (!ok) break;
                alpha_prev = alpha;
                tmem_st16(lanes + T::P0 + half * 16, w0);
                tmem_st16(lanes + T::P0 + 32 + half * 16, w1);
                tmem_st16(lanes + T::P0 + 64 + half * 16, w2);
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&sh.p_full);
            }
            for (; j < n_tiles; ++j) pair_bar();  // the other half of the rows may not have given up
            if (ok) add_tile(n_tiles - 1, alpha_prev);
            sh.row[n_tiles & 1][half][row] = sum;
            pair_bar();
            const float inv = 1.0f / (sum + sh.row[n_tiles & 1][half ^ 1][row]);
            const float bad = leave() ? NAN : 0.0f;
            if (sh.odd_end != 0) {
                // values that are not finite stood as zeros in the products: they go where a query sees them, and nowhere else
                const float* V = cache_v + (uint64_t)kvh * max_ctx * HD + half * DN;
                for (uint32_t t = sh.odd_first * AK; t < min(sh.odd_end * AK, visible) && sr < seq; ++t)
#pragma unroll
                    for (uint32_t i = 0; i < DN; ++i) {
                        const float v = __ldg(V + (uint64_t)t * HD + i);
                        if (!(fabsf(v) < INFINITY)) o[i] += v;
                    }
            }
            if (sr < seq) {
                float4* dst = reinterpret_cast<float4*>(out + ((uint64_t)sr * nq + head) * HD + half * DN);
#pragma unroll
                for (uint32_t i = 0; i < DN / 4; ++i)
                    dst[i] = make_float4(fmaf(o[4 * i], inv, bad), fmaf(o[4 * i + 1], inv, bad), fmaf(o[4 * i + 2], inv, bad),
                                         fmaf(o[4 * i + 3], inv, bad));
            }
        } else {
            leave();
        }
    } else if (warp < A_SOFT + A_CONV) {
        // ── converters ──
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(A_REGS_CONV));
        const uint32_t cw = warp - A_SOFT;
        // keys: eight dimensions a thread, HD / 8 neighbouring lanes a row
        constexpr uint32_t CPR = HD / 8, RPW = 32 / CPR, KIT = AK / (RPW * A_CONV);
        const uint32_t chunk = lane % CPR, krow = cw * RPW + lane / CPR;
        // a thread's two 16-byte pieces: every other four lanes take the second one first, so that eight lanes hit 32 banks
        const uint32_t k_src = smem_u32(raw_k) + krow * (HD * 4) + chunk * 32, swap = (lane & 4) << 2;
        // values: one dimension a thread, KN consecutive keys
        constexpr uint32_t DB = HD / 32, KP = A_CONV / DB, KN = AK / KP;
        const uint32_t vd = (cw % DB) * 32 + lane, part = cw / DB;
        const uint32_t v_src = smem_u32(raw_v) + part * KN * (HD * 4) + vd * 4;
        auto publish = [&](uint64_t* bar) {
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(bar);
        };
        auto convert_keys = [&](uint32_t j, uint32_t st, uint32_t live) {
            // all loads, then all row maxima, then the terms: rows after one another took three times as long
            float4 kr[KIT][2];
            float row_max[KIT];
#pragma unroll
            for (uint32_t i = 0; i < KIT; ++i) {
                const uint32_t src = k_src + i * RPW * A_CONV * (HD * 4);
                kr[i][0] = lds_f32x4(src + swap), kr[i][1] = lds_f32x4(src + (swap ^ 16));
                if (krow + i * RPW * A_CONV >= live) kr[i][0] = kr[i][1] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&sh.rk_empty);
#pragma unroll
            for (uint32_t i = 0; i < KIT; ++i) {
                const float4 a = kr[i][0], b = kr[i][1];
                row_max[i] = fmaxf(fmaxf(fmaxf(fabsf(a.x), fabsf(a.y)), fmaxf(fabsf(a.z), fabsf(a.w))),
                                   fmaxf(fmaxf(fabsf(b.x), fabsf(b.y)), fmaxf(fabsf(b.z), fabsf(b.w))));
            }
#pragma unroll
            for (uint32_t off = CPR / 2; off > 0; off >>= 1)
#pragma unroll
                for (uint32_t i = 0; i < KIT; ++i) row_max[i] = fmaxf(row_max[i], __shfl_xor_sync(0xFFFFFFFFu, row_max[i], off));
#pragma unroll
            for (uint32_t i = 0; i < KIT; ++i) {
                const uint32_t bits = term_scale_bits(row_max[i]), r = krow + i * RPW * A_CONV;
                const float sc = bits_scale(bits);
                const bool infinite = row_max[i] == INFINITY;
                if (infinite) {  // the others of the row no longer count: signs under a scale of infinity
#pragma unroll
                    for (int p = 0; p < 2; ++p)
                        for (float* v : {&kr[i][p].x, &kr[i][p].y, &kr[i][p].z, &kr[i][p].w})
                            *v = fabsf(*v) == INFINITY ? copysignf(1.0f, *v) : *v != *v ? *v : 0.0f;
                }
                uint32_t x[2][2], y[2][2];  // terms of the two pieces
#pragma unroll
                for (int p = 0; p < 2; ++p) {
                    split_pair(kr[i][p].x * sc, kr[i][p].y * sc, &x[p][0], &y[p][0]);
                    split_pair(kr[i][p].z * sc, kr[i][p].w * sc, &x[p][1], &y[p][1]);
                }
                const uint32_t hi[4] = {swap ? x[1][0] : x[0][0], swap ? x[1][1] : x[0][1], swap ? x[0][0] : x[1][0], swap ? x[0][1] : x[1][1]};
                const uint32_t lo[4] = {swap ? y[1][0] : y[0][0], swap ? y[1][1] : y[0][1], swap ? y[0][0] : y[1][0], swap ? y[0][1] : y[1][1]};
                // 128-byte swizzle: the 16-byte piece's place in its row of 64 dimensions, exclusive-or the row
                const uint32_t at = k_base + st * T::K_STAGE + (chunk >> 3) * T::K_PLANE + r * 128 + (((chunk ^ r) & 7) << 4);
                st_shared_v4(at, hi);
                st_shared_v4(at + T::HALVES * T::K_PLANE, lo);
                if (chunk == 0) sh.ks[j & 3][r] = __float_as_uint(infinite ? INFINITY : bits_inverse(bits)) >> 16;
            }
            publish(&sh.k_full[st]);
        };
        for (uint32_t j = 0; j < n_tiles; ++j) {
            const uint32_t st = j & 1, freed = ((j >> 1) & 1) ^ 1;
            const uint32_t live = n_keys - j * AK;  // rows of the tile that hold keys; the others are zeros
            if (!wait_all(&sh.k_empty[st], freed) || !wait_all(&sh.rk_full, j & 1)) break;
            convert_keys(j, st, live);
            if (!wait_all(&sh.rv_full, j & 1)) break;
            float vr[KN], zero = 0.0f;
#pragma unroll
            for (uint32_t i = 0; i < KN; ++i) {
                vr[i] = part * KN + i < live ? lds_f32(v_src + i * (HD * 4)) : 0.0f;
                zero = fmaf(vr[i], 0.0f, zero);  // NaN if some value is not finite
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&sh.rv_empty);
            if (zero != 0.0f) {
#pragma unroll
                for (uint32_t i = 0; i < KN; ++i) vr[i] = fabsf(vr[i]) < INFINITY ? vr[i] : 0.0f;
                atomicMin(&sh.odd_first, j);
                atomicMax(&sh.odd_end, j + 1);
            }
            if (!wait_all(&sh.v_empty[st], freed)) break;
#pragma unroll
            for (uint32_t c = 0; c < KN / 8; ++c) {
                uint32_t t[4][3];
#pragma unroll
                for (uint32_t i = 0; i < 4; ++i) cut3_pair(vr[8 * c + 2 * i], vr[8 * c + 2 * i + 1], t[i]);
                const uint32_t piece = part * (KN / 8) + c;
                const uint32_t at = v_base + st * T::V_STAGE + vd * 128 + (((piece ^ vd) & 7) << 4);
#pragma unroll
                for (int p = 0; p < 3; ++p) st_shared_v4(at + p * T::V_PLANE, {t[0][p], t[1][p], t[2][p], t[3][p]});
            }
            publish(&sh.v_full[st]);
        }
        leave();
    } else {
        // ── issuer (one warp issues, one copies, two have nothing to do) ──
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(A_REGS_ISSUE));
        if (warp == A_SOFT + A_CONV) {
            constexpr uint32_t idesc_s = umma_idesc_f16(AK), idesc_o = umma_idesc_bf16(HD);
            const uint64_t dk = umma_desc(k_base), dv = umma_desc(v_base);
            auto scores = [&](uint32_t j) {  // one accumulator per 64 dimensions, small products first
                // the scores before have been read (the first: the query is in place)
                if (!wait_all(&sh.s_free, j & 1) || !wait_all(&sh.k_full[j & 1], (j >> 1) & 1)) return;
                tc_fence_after();
                if (elect_one()) {
                    const uint64_t d0 = dk + (uint64_t)(j & 1) * (T::K_STAGE >> 4);
#pragma unroll
                    for (uint32_t h = 0; h < T::HALVES; ++h) {
                        const uint64_t hi = d0 + h * (T::K_PLANE >> 4), lo = hi + T::HALVES * (T::K_PLANE >> 4);
                        const uint32_t d = tmem + T::S0 + 64 * h, a_hi = tmem + T::Q_HI + 32 * h, a_lo = tmem + T::Q_LO + 32 * h;
#pragma unroll
                        for (uint32_t kk = 0; kk < 4; ++kk) {
                            umma_f16_ts(d, a_lo + 8 * kk, hi + 2 * kk, idesc_s, kk != 0);
                            umma_f16_ts(d, a_hi + 8 * kk, lo + 2 * kk, idesc_s, 1);
                        }
#pragma unroll
                        for (uint32_t kk = 0; kk < 4; ++kk) umma_f16_ts(d, a_hi + 8 * kk, hi + 2 * kk, idesc_s, 1);
                    }
                    umma_commit(&sh.k_empty[j & 1]);
                    umma_commit(&sh.s_full);
                }
                __syncwarp();
            };
            if (n_tiles) scores(0);
            for (uint32_t j = 0; j < n_tiles && ok; ++j) {
                if (j + 1 < n_tiles) scores(j + 1);
                // the probabilities are in place, the output before has been read
                if (!ok || !wait_all(&sh.v_full[j & 1], (j >> 1) & 1) || !wait_all(&sh.p_full, j & 1)) break;
                tc_fence_after();
                if (elect_one()) {
                    const uint64_t b = dv + (uint64_t)(j & 1) * (T::V_STAGE >> 4);
                    const uint32_t d = tmem + T::O, a = tmem + T::P0, steps = (min(n_keys - j * AK, AK) + 15) / 16;
#pragma unroll
                    for (int order = 2; order >= 0; --order)  // terms p of the probabilities and order - p of the values
#pragma unroll
                        for (uint32_t kk = 0; kk < 4; ++kk) {
                            if (kk >= steps) break;  // zeros
#pragma unroll
                            for (int p = 0; p <= order; ++p)
                                umma_f16_ts(d, a + 32 * p + 8 * kk, b + (order - p) * (T::V_PLANE >> 4) + 2 * kk, idesc_o,
                                            order < 2 || kk != 0 || p != 0);
                        }
                    umma_commit(&sh.v_empty[j & 1]);
                    umma_commit(&sh.o_full);
                }
                __syncwarp();
            }
            if (!ok) {  // products in flight still use tensor memory and the tiles
                if (elect_one()) umma_commit(&sh.drained);
                __syncwarp();
                mbar_wait(&sh.drained, 0);
            }
        } else if (warp == A_SOFT + A_CONV + 1) {
            // ── loader: a tile's rows are one run of memory ──
            const float* K = cache_k + (uint64_t)kvh * max_ctx * HD;
            const float* V = cache_v + (uint64_t)kvh * max_ctx * HD;
            uint32_t k_sent = 0, v_sent = 0;
            for (uint32_t j = 0; j < n_tiles && ok; ++j) {
                const uint32_t bytes = min(n_keys - j * AK, AK) * (HD * 4);
                if (!wait_all(&sh.rk_empty, (j & 1) ^ 1)) break;
                ++k_sent;
                if (lane == 0) {
                    mbar_arrive_expect_tx(&sh.rk_full, bytes);
                    bulk_g2s(raw_k, K + (uint64_t)j * AK * HD, bytes, &sh.rk_full);
                }
                if (!wait_all(&sh.rv_empty, (j & 1) ^ 1)) break;
                ++v_sent;
                if (lane == 0) {
                    mbar_arrive_expect_tx(&sh.rv_full, bytes);
                    bulk_g2s(raw_v, V + (uint64_t)j * AK * HD, bytes, &sh.rv_full);
                }
            }
            if (!ok) {  // copies in flight still write to shared memory
                if (k_sent) mbar_wait(&sh.rk_full, (k_sent - 1) & 1);
                if (v_sent) mbar_wait(&sh.rv_full, (v_sent - 1) & 1);
            }
        }
        leave();
    }
    if (tid == 0 && sh.abort_flag && error_flag) *reinterpret_cast<volatile int*>(error_flag) = 1;
    tc_fence_after();
    if (warp == A_SOFT + A_CONV)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
}

}  // namespace

cudaError_t launch_attention_prefill(const float* q, const float* cache_k, const float* cache_v, const int32_t* pos,
                                     uint32_t seq, uint32_t nq, uint32_t nkv, uint32_t hd, uint32_t max_ctx, float* out,
                                     int32_t* bad_pos, int* error_flag, cudaStream_t s) {
    const dim3 grid(nq, (seq + AQ - 1) / AQ);
    auto launch = [&](auto kern, size_t smem, bool* configured) {
        if (cudaError_t ce = set_max_smem_once(kern, (int)smem, configured); ce != cudaSuccess) return ce;
        cudaError_t e = launch_pdl(kern, grid, A_THREADS, smem, s, q, cache_k, cache_v, pos, seq, nq, nkv, max_ctx, out, bad_pos,
                                   error_flag);
        return e != cudaSuccess ? e : cudaGetLastError();
    };
    static bool configured[2][MAX_DEVICES] = {};
    if (hd == 64) return launch(attention_prefill_kernel<64>, AttTile<64>::SMEM, configured[0]);
    if (hd == 128) return launch(attention_prefill_kernel<128>, AttTile<128>::SMEM, configured[1]);
    return cudaErrorInvalidValue;
}

}  // namespace jq
