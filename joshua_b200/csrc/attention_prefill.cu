// Causal attention of a prompt's tokens over the KV cache on the 5th-generation tensor cores, in half-precision terms that
// keep f32's precision.
//
// `seq` new tokens of ONE sequence at positions pos0 .. pos0 + seq - 1 (the cache already holds their k / v rows):
// out[s, head, :] = softmax(q_s . K[0 .. pos0 + s]^T / sqrt(hd)) V (src/quantized_qwen3_moe.rs:366-386 with the causal
// mask of :805-812).  One CTA per (128 queries, q head), 64 keys at a time, running maximum and sum in f32.
//
// Every operand is split into two f16 terms under a power-of-two scale that puts its largest value just below 2^15 (a
// query row, a key row, a value column of the tile), which keeps 22 to 24 bits of every value within 2^17 of the largest
// and an absolute error below 2^-39 of it otherwise; the probabilities are split the same way under 2^14.  A product is
// three products of terms (lo * hi, hi * lo, hi * hi; the tensor core forms them exactly).  It adds with truncation, so
// accumulators are short: 64 dimensions of a score, the 64 keys of a tile for the output, small products first; they are
// read back and added round-to-nearest in registers, where the running output lives.  Error against float64 (2-norm,
// N(0, 1) rows, 1000 tokens, 32 q / 4 kv heads of 128): 2.8e-7; the f32 kernel before it 3.8e-7 (queries four times as
// large: 4.0e-7, 1.1e-6).  The limit: a value 2^17 above the others of its dimension in the same 64 keys costs those bits
// (1e6 beside N(0, 1), masked: 4.8e-7 and 6.9e-7 in that dimension at 16 and 64 tokens, 3.6e-7 and 2.8e-7 before).
//
// Warps: 0 .. 7 softmax, two threads a query (32 keys and half of the output dimensions each); 8 .. 15 convert the key and
// value tiles into swizzled K-major tiles (values transposed: keys run along a row), two stages; 16 issues the products.
// Tensor memory: the query's terms (the A operand of the scores), scores, probabilities (A of the output), output of a tile.
//
// What bounds it: a tile of 64 keys takes some 3000 to 3900 cycles, of which the tensor pipe works 1536 (hd 128); the rest
// is the softmax threads' chain (read the scores, maximum, exponentials, terms, add the output before) and the issue slots
// that they share with the converters (12500 warp instructions a tile, two a cycle).  The f32 rows come by one bulk copy a
// tile, ahead of the converters: with loads into registers instead a tile took 6600 cycles.  Measured against the f32
// kernel on the CUDA cores, 32 heads of 128 (in a graph): 1000 tokens 53.0 us (248), 512 27.0 (127), 256 17.6 (59.5),
// 128 13.7 (27.0), 16 6.0 (10.8), one 5.8 (10.3); heads of 64, 1000 tokens 33.1 (152): ahead at every size, so it is the
// only route.
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
// Registers a thread: the launch has 640 x 96 = 61440, of which the issuer's warpgroup keeps 128 x 40, the converters
// 256 x 72 and the softmax threads (64 running outputs, 32 scores) 256 x 144: 60416.
constexpr int A_REGS_ISSUE = 40, A_REGS_CONV = 72, A_REGS_SOFT = 144;
static_assert(128 * A_REGS_ISSUE + A_CONV * 32 * A_REGS_CONV + A_SOFT * 32 * A_REGS_SOFT <= A_THREADS * 96, "registers");
constexpr float P_LOG2 = 14.0f;              // probabilities (and their sum) are formed times 2^14

template <uint32_t HD>
struct AttTile {
    static constexpr uint32_t HALVES = HD / 64;              // 64-dimension accumulators of a score
    static constexpr uint32_t K_PLANE = AK * 128;            // 64 dimensions of the tile's keys, one term
    static constexpr uint32_t K_STAGE = 2 * HALVES * K_PLANE;
    static constexpr uint32_t V_PLANE = HD * 128;            // the tile's keys of every dimension, one term
    static constexpr uint32_t V_STAGE = 2 * V_PLANE;
    static constexpr uint32_t RAW = AK * HD * 4;             // the f32 rows of a tile's keys or values
    static constexpr uint32_t SMEM = 2 * (K_STAGE + V_STAGE) + 2 * RAW + 1024;
    // tensor memory columns
    static constexpr uint32_t Q_HI = 0, Q_LO = HD / 2, S0 = HD, P_HI = S0 + 64 * HALVES, P_LO = P_HI + 32, O = P_LO + 32;
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
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const uint32_t k_base = smem_u32(smem), v_base = k_base + 2 * T::K_STAGE;
    uint8_t* raw_k = smem + 2 * (T::K_STAGE + T::V_STAGE);
    uint8_t* raw_v = raw_k + T::RAW;
    __shared__ __align__(16) float s_ks[4][AK], s_vs[4][HD];  // inverse scales of key rows and value columns, by tile % 4
    __shared__ float s_vmax[2][8 * 32];                       // column maxima of the key parts
    __shared__ float s_row[2][2][AQ];                         // row maxima of the two halves
    __shared__ uint64_t k_full[2], k_empty[2], v_full[2], v_empty[2], s_full, s_free, p_full, o_full;
    __shared__ uint64_t rk_full, rk_empty, rv_full, rv_empty;  // the raw rows
    __shared__ uint64_t drained;                               // the products of a CTA that gives up
    __shared__ uint32_t tmem_slot;
    __shared__ int abort_flag;

    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    pdl_trigger();
    if (tid == 0) {
        for (int i = 0; i < 2; ++i) {
            mbar_init(&k_full[i], A_CONV);
            mbar_init(&v_full[i], A_CONV);
            mbar_init(&k_empty[i], 1);
            mbar_init(&v_empty[i], 1);
        }
        mbar_init(&s_full, 1);
        mbar_init(&s_free, A_SOFT);
        mbar_init(&p_full, A_SOFT);
        mbar_init(&o_full, 1);
        mbar_init(&rk_full, 1);
        mbar_init(&rv_full, 1);
        mbar_init(&rk_empty, A_CONV);
        mbar_init(&rv_empty, A_CONV);
        mbar_init(&drained, 1);
        abort_flag = 0;
        mbar_fence_init();
    }
    if (warp == A_SOFT + A_CONV) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(512u)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;
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
        if (!ok && lane == 0) *static_cast<volatile int*>(&abort_flag) = 1;
        tc_fence_before();
        asm volatile("bar.sync 6, %0;" ::"n"(A_THREADS) : "memory");
        return *static_cast<volatile int*>(&abort_flag) != 0;
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
                s_row[1][half][row] = amax;
                pair_bar();
                const uint32_t bits = term_scale_bits(fmaxf(amax, s_row[1][half ^ 1][row]));
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
                if (lane == 0) mbar_arrive(&s_free);  // the first scores wait for the query's terms
            }
#pragma unroll
            for (uint32_t i = 0; i < DN; ++i) o[i] = 0.0f;
            float mx = -INFINITY, sum = 0.0f, alpha_prev = 0.0f;
            const uint32_t visible = (uint32_t)p0 + sr + 1;                         // keys 0 .. p0 + s (rows past seq: never stored)
            const uint32_t all_see = (uint32_t)p0 + s0 + quarter * 32 + 1;          // keys that every query of the warp sees
            // o = o * alpha + the tile's output, whose value columns have scales
            auto add_tile = [&](uint32_t j, float alpha) {
                if (__any_sync(0xFFFFFFFFu, alpha != 1.0f)) {  // while the products run; the maxima settle after a few tiles
#pragma unroll
                    for (uint32_t i = 0; i < DN; ++i) o[i] *= alpha;
                }
                if (!wait_all(&o_full, j & 1)) return;
                tc_fence_after();
#pragma unroll
                for (uint32_t c = 0; c < DN / 32; ++c) {
                    uint32_t r[32];
                    tmem_ld32(lanes + T::O + half * DN + 32 * c, r);
                    const float4* vs = reinterpret_cast<const float4*>(&s_vs[j & 3][half * DN + 32 * c]);
#pragma unroll
                    for (uint32_t i = 0; i < 8; ++i) {
                        const float4 f = vs[i];
                        float* d = o + 32 * c + 4 * i;
                        d[0] = fmaf(__uint_as_float(r[4 * i]), f.x, d[0]);
                        d[1] = fmaf(__uint_as_float(r[4 * i + 1]), f.y, d[1]);
                        d[2] = fmaf(__uint_as_float(r[4 * i + 2]), f.z, d[2]);
                        d[3] = fmaf(__uint_as_float(r[4 * i + 3]), f.w, d[3]);
                    }
                }
            };
            uint32_t j = 0;  // tiles whose barrier this warp has come to
            while (j < n_tiles) {
                const uint32_t t0 = j * AK + half * 32;  // this thread's first key
                float sc[32];
                if (!wait_all(&s_full, j & 1)) break;
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
                if (lane == 0) mbar_arrive(&s_free);
                const float4* ks = reinterpret_cast<const float4*>(&s_ks[j & 3][half * 32]);
                float cm = -INFINITY;
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const float4 f = ks[i];
                    sc[4 * i] *= f.x, sc[4 * i + 1] *= f.y, sc[4 * i + 2] *= f.z, sc[4 * i + 3] *= f.w;
                }
                if (t0 + 32 > all_see) {
#pragma unroll
                    for (int i = 0; i < 32; ++i) sc[i] = t0 + i < visible ? sc[i] : -INFINITY;
                }
#pragma unroll
                for (int i = 0; i < 32; ++i) cm = fmaxf(cm, sc[i]);
                s_row[j & 1][half][row] = cm;
                pair_bar();
                // logarithms to base 2 of the probabilities; the maximum is finite from the first tile on: key 0 is
                // visible to every query
                const float nm = fmaxf(mx, fmaxf(cm, s_row[j & 1][half ^ 1][row]) * rf);
                const float alpha = ex2(mx - nm);  // 0 on the first tile (mx = -inf)
                const float shift = P_LOG2 - nm;
                float ps = 0.0f;
                uint32_t hi[16], lo[16];
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    const float a = ex2(fmaf(sc[2 * i], rf, shift)), b = ex2(fmaf(sc[2 * i + 1], rf, shift));  // 0 for masked keys
                    ps += a + b;
                    split_pair(a, b, &hi[i], &lo[i]);
                }
                sum = sum * alpha + ps;
                mx = nm;
                if (j++ > 0) add_tile(j - 2, alpha_prev);  // its products have read the probabilities before these
                if (!ok) break;
                alpha_prev = alpha;
                tmem_st16(lanes + T::P_HI + half * 16, hi);
                tmem_st16(lanes + T::P_LO + half * 16, lo);
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&p_full);
            }
            for (; j < n_tiles; ++j) pair_bar();  // the other half of the rows may not have given up
            if (ok) add_tile(n_tiles - 1, alpha_prev);
            s_row[n_tiles & 1][half][row] = sum;
            pair_bar();
            const float inv = 1.0f / (sum + s_row[n_tiles & 1][half ^ 1][row]);
            const float bad = leave() ? NAN : 0.0f;
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
            if (lane == 0) mbar_arrive(&rk_empty);
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
                if (chunk == 0) s_ks[j & 3][r] = bits_inverse(bits);
            }
            publish(&k_full[st]);
        };
        auto meet = [&] { asm volatile("bar.sync 5, %0;" ::"n"(A_CONV * 32) : "memory"); };
        uint32_t j = 0;  // tiles whose barrier this warp has come to
        while (j < n_tiles) {
            const uint32_t st = j & 1, freed = ((j >> 1) & 1) ^ 1;
            const uint32_t live = n_keys - j * AK;  // rows of the tile that hold keys; the others are zeros
            if (!wait_all(&k_empty[st], freed) || !wait_all(&rk_full, j & 1)) break;
            convert_keys(j, st, live);
            if (!wait_all(&rv_full, j & 1)) break;
            float amax = 0.0f, vr[KN];
#pragma unroll
            for (uint32_t i = 0; i < KN; ++i) {
                vr[i] = part * KN + i < live ? lds_f32(v_src + i * (HD * 4)) : 0.0f;
                amax = fmaxf(amax, fabsf(vr[i]));
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&rv_empty);
            s_vmax[st][part * HD + vd] = amax;
            meet();
            const uint32_t vs_at = j++ & 3;
            if (!wait_all(&v_empty[st], freed)) break;
#pragma unroll
            for (uint32_t p = 0; p < KP; ++p) amax = fmaxf(amax, s_vmax[st][p * HD + vd]);
            const uint32_t bits = term_scale_bits(amax);
            const float sc = bits_scale(bits);
#pragma unroll
            for (uint32_t c = 0; c < KN / 8; ++c) {
                uint32_t hi[4], lo[4];
#pragma unroll
                for (uint32_t i = 0; i < 4; ++i) split_pair(vr[8 * c + 2 * i] * sc, vr[8 * c + 2 * i + 1] * sc, &hi[i], &lo[i]);
                const uint32_t piece = part * (KN / 8) + c;
                const uint32_t at = v_base + st * T::V_STAGE + vd * 128 + (((piece ^ vd) & 7) << 4);
                st_shared_v4(at, hi);
                st_shared_v4(at + T::V_PLANE, lo);
            }
            if (part == 0) s_vs[vs_at][vd] = bits_inverse(bits);
            publish(&v_full[st]);
        }
        for (; j < n_tiles; ++j) meet();  // the others may not have given up
        leave();
    } else {
        // ── issuer (one warp issues, one copies, two have nothing to do) ──
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(A_REGS_ISSUE));
        if (warp == A_SOFT + A_CONV) {
            constexpr uint32_t idesc_s = umma_idesc_f16(AK), idesc_o = umma_idesc_f16(HD);
            const uint64_t dk = umma_desc(k_base), dv = umma_desc(v_base);
            auto scores = [&](uint32_t j) {  // one accumulator per 64 dimensions, small products first
                // the scores before have been read (the first: the query is in place)
                if (!wait_all(&s_free, j & 1) || !wait_all(&k_full[j & 1], (j >> 1) & 1)) return;
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
                    umma_commit(&k_empty[j & 1]);
                    umma_commit(&s_full);
                }
                __syncwarp();
            };
            if (n_tiles) scores(0);
            for (uint32_t j = 0; j < n_tiles && ok; ++j) {
                if (j + 1 < n_tiles) scores(j + 1);
                // the probabilities are in place, the output before has been read
                if (!ok || !wait_all(&v_full[j & 1], (j >> 1) & 1) || !wait_all(&p_full, j & 1)) break;
                tc_fence_after();
                if (elect_one()) {
                    const uint64_t hi = dv + (uint64_t)(j & 1) * (T::V_STAGE >> 4), lo = hi + (T::V_PLANE >> 4);
                    const uint32_t d = tmem + T::O, a_hi = tmem + T::P_HI, a_lo = tmem + T::P_LO;
#pragma unroll
                    for (uint32_t kk = 0; kk < 4; ++kk) {
                        umma_f16_ts(d, a_lo + 8 * kk, hi + 2 * kk, idesc_o, kk != 0);
                        umma_f16_ts(d, a_hi + 8 * kk, lo + 2 * kk, idesc_o, 1);
                    }
#pragma unroll
                    for (uint32_t kk = 0; kk < 4; ++kk) umma_f16_ts(d, a_hi + 8 * kk, hi + 2 * kk, idesc_o, 1);
                    umma_commit(&v_empty[j & 1]);
                    umma_commit(&o_full);
                }
                __syncwarp();
            }
            if (!ok) {  // products in flight still use tensor memory and the tiles
                if (elect_one()) umma_commit(&drained);
                __syncwarp();
                mbar_wait(&drained, 0);
            }
        } else if (warp == A_SOFT + A_CONV + 1) {
            // ── loader: a tile's rows are one run of memory ──
            const float* K = cache_k + (uint64_t)kvh * max_ctx * HD;
            const float* V = cache_v + (uint64_t)kvh * max_ctx * HD;
            uint32_t k_sent = 0, v_sent = 0;
            for (uint32_t j = 0; j < n_tiles && ok; ++j) {
                const uint32_t bytes = min(n_keys - j * AK, AK) * (HD * 4);
                if (!wait_all(&rk_empty, (j & 1) ^ 1)) break;
                ++k_sent;
                if (lane == 0) {
                    mbar_arrive_expect_tx(&rk_full, bytes);
                    bulk_g2s(raw_k, K + (uint64_t)j * AK * HD, bytes, &rk_full);
                }
                if (!wait_all(&rv_empty, (j & 1) ^ 1)) break;
                ++v_sent;
                if (lane == 0) {
                    mbar_arrive_expect_tx(&rv_full, bytes);
                    bulk_g2s(raw_v, V + (uint64_t)j * AK * HD, bytes, &rv_full);
                }
            }
            if (!ok) {  // copies in flight still write to shared memory
                if (k_sent) mbar_wait(&rk_full, (k_sent - 1) & 1);
                if (v_sent) mbar_wait(&rv_full, (v_sent - 1) & 1);
            }
        }
        leave();
    }
    if (tid == 0 && abort_flag) *reinterpret_cast<volatile int*>(error_flag) = 1;
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
