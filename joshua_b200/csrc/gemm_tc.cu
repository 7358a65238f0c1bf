// Prefill / batched matmul (m > 8) over raw GGUF blocks on the 5th-generation tensor cores.
//
// dst[m, n] = lhs[m, k] . W[n, k]^T with W left in its GGUF bytes.  A CTA owns a 128-row tile of W and a tile
// of up to 128 activation rows.  Per 32-column K step its converter warps decode the 128 x 32 weight block to
// the exact f32 weights the reference forms (formats.cuh) and split them into two TF32 terms (hi = top 11
// significant bits, lo = the exact remainder); the activations are split the same way once per launch by a
// small kernel (two f32 arrays) and reach shared memory by TMA (`cp.async.bulk.tensor.2d`, 128-byte swizzle).
// One thread issues tcgen05.mma (kind::tf32) for the three significant products hi*hi + hi*lo + lo*hi into a
// 128 x N f32 accumulator in tensor memory; each product is exact and the split carries ~2^-22 relative error
// per term.  The tensor core adds into its f32 accumulator with truncation, an error that grows linearly with
// the number of accumulated instructions, so the accumulator only ever holds a chunk of 4 K steps (128
// columns): the converter warps read each finished chunk back with tcgen05.ld and add it, round-to-nearest, to
// running sums in registers while the next chunk accumulates in the other half of tensor memory.  The result
// then matches f32 accumulation (src/kquant_dot.rs:268-483) to the tolerance the path is held to.
//
// The weights are decoded straight from global memory into swizzled shared-memory tiles.  This form serves the shapes
// that gemm_f16.cu does not take (k not a whole number of 256-column windows, 512 for IQ2_XXS; tensors that
// are not word-aligned).
//
// Every wait on an mbarrier is bounded; a wait that runs out raises the device status flag, and every thread
// still reaches the common exit where tensor memory is released.
//
// Tensor-pipe bound for large m: 3 x 2*m*n*k TF32 flops per launch.  Algorithmic flops: 2*m*n*k.
#include <algorithm>
#include <cstdlib>

#include <cuda.h>
#include <cudaTypedefs.h>

#include "common.cuh"
#include "tc5.cuh"

namespace jq {

cudaError_t tables_gemm_tc() { return upload_tables(); }

namespace {

constexpr int TC_M = 128;          // weight rows per CTA = MMA M = TMEM lanes
constexpr int TC_K = 32;           // K per stage: 32 tf32 = one 128-byte swizzled row
constexpr int TC_CHUNK = 4;        // K steps accumulated in tensor memory before a read-back
constexpr int TC_CONV_WARPS = 16;  // converter / epilogue warps: 4 per quarter of the accumulator's lanes
constexpr int TC_THREADS = (TC_CONV_WARPS + 1) * 32;
constexpr uint32_t PLANE_A = TC_M * 128;  // bytes of one term of the weight tile

__device__ __forceinline__ unsigned long long tc_now() {
    return (unsigned long long)clock64();  // SM cycles: both traced threads run on the same SM
}
// Profiling aid (jq_debug_gemm_trace, a buffer of 512 values): CTA (0, 0) stores eight SM-cycle stamps per K step
// for its first 64 steps.  Converter thread 0: [0] stage free, [1] stage handed over.  Issuer: [2] top of the
// step, [3] accumulator half free, [4] operands complete, [5] MMAs issued, [6] stage commit issued, [7] end.
unsigned long long* g_gemm_trace = nullptr;

// x -> its TF32 part (top 11 significant bits) and the exact remainder, element-wise.
__global__ void __launch_bounds__(256) split_tf32_kernel(const float* __restrict__ x, uint64_t n4, float* __restrict__ hi,
                                                         float* __restrict__ lo) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n4; i += (uint64_t)gridDim.x * blockDim.x) {
        const float4 v = __ldg(reinterpret_cast<const float4*>(x) + i);
        float4 h;
        h.x = __uint_as_float(__float_as_uint(v.x) & 0xFFFFE000u);
        h.y = __uint_as_float(__float_as_uint(v.y) & 0xFFFFE000u);
        h.z = __uint_as_float(__float_as_uint(v.z) & 0xFFFFE000u);
        h.w = __uint_as_float(__float_as_uint(v.w) & 0xFFFFE000u);
        reinterpret_cast<float4*>(hi)[i] = h;
        reinterpret_cast<float4*>(lo)[i] = make_float4(v.x - h.x, v.y - h.y, v.z - h.z, v.w - h.w);
    }
}

// Instruction descriptor: D f32, A and B tf32, both K-major, M = 128, N = n_tile.
__device__ __forceinline__ uint32_t umma_idesc(uint32_t n_tile) {
    return (1u << 4) | (2u << 7) | (2u << 10) | ((n_tile >> 3) << 17) | ((uint32_t)(TC_M >> 4) << 24);
}

__device__ __forceinline__ void umma_tf32(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc,
                                          uint32_t accumulate) {
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t"
        "}\n" ::"r"(tmem_d),
        "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate), "r"(0u), "r"(0u), "r"(0u), "r"(0u)
        : "memory");
}
// Split 4 floats into their TF32 hi parts and exact remainders and store both 16-byte chunks.  `row_base`
// is the byte offset of the row inside a term's tile; `chunk` the 16-byte chunk inside the 128-byte row.
__device__ __forceinline__ void store_split(uint8_t* hi_tile, uint8_t* lo_tile, uint32_t row, uint32_t chunk,
                                            const float v[4]) {
    float4 h, l;
    h.x = __uint_as_float(__float_as_uint(v[0]) & 0xFFFFE000u);
    h.y = __uint_as_float(__float_as_uint(v[1]) & 0xFFFFE000u);
    h.z = __uint_as_float(__float_as_uint(v[2]) & 0xFFFFE000u);
    h.w = __uint_as_float(__float_as_uint(v[3]) & 0xFFFFE000u);
    l = make_float4(v[0] - h.x, v[1] - h.y, v[2] - h.z, v[3] - h.w);
    // 128-byte swizzle: chunk index XOR (row mod 8) inside each 8-row x 128-byte atom
    const uint32_t off = row * 128 + ((chunk ^ (row & 7)) << 4);
    *reinterpret_cast<float4*>(hi_tile + off) = h;
    *reinterpret_cast<float4*>(lo_tile + off) = l;
}

template <uint32_t TYPE, uint32_t ELEMS, uint32_t BYTES, int N_TILE>
__global__ void __launch_bounds__(TC_THREADS, 1)
    gemm_tc_kernel(const uint8_t* __restrict__ w, uint64_t n, uint64_t k, const __grid_constant__ CUtensorMap map_hi,
                   const __grid_constant__ CUtensorMap map_lo, uint64_t m, float* __restrict__ dst, uint32_t n_stages,
                   int* __restrict__ error_flag, unsigned long long* __restrict__ trace, int dbg_skip) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    // stage layout: A hi | A lo | B hi | B lo, every tile 1024-byte aligned
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    constexpr uint32_t PLANE_B = N_TILE * 128;
    constexpr uint32_t STAGE = 2 * PLANE_A + 2 * PLANE_B;
    __shared__ uint64_t full[8], empty[8], acc_full[2], acc_empty[2];
    __shared__ uint32_t tmem_base_slot;
    __shared__ int abort_flag;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint64_t row0 = (uint64_t)blockIdx.x * TC_M;
    const uint64_t tok0 = (uint64_t)blockIdx.y * N_TILE;
    const uint32_t k_steps = (uint32_t)(k / TC_K);
    const uint32_t n_chunks = (k_steps + TC_CHUNK - 1) / TC_CHUNK;
    const uint64_t row_bytes = k / ELEMS * BYTES;
    constexpr uint32_t UPB = ELEMS / 8;
    constexpr uint32_t TMEM_COLS = 2 * N_TILE < 32 ? 32 : 2 * N_TILE;  // two accumulators; a power of two >= 32
    // Converter mapping: warp w owns weight rows 8w .. 8w+7, lane l the unit l % 4 (8 of the step's 32 columns)
    // of row 8w + l / 4, so a warp's loads touch 8 rows (8 L1 wavefronts per load, not 32) and its 16-byte
    // stores to the swizzled tile fall on distinct banks.  The decode reads global memory directly: this form
    // serves the shapes the tensor-memory form (gemm_f16.cu) does not take.
    constexpr uint32_t ROWS_PER_WARP = TC_M / TC_CONV_WARPS;                // 8

    if (tid == 0) {
        for (uint32_t s = 0; s < n_stages; ++s) {
            mbar_init(&full[s], TC_CONV_WARPS + 1);  // the converter warps and the thread that starts the TMA copies
            mbar_init(&empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&acc_full[b], 1);
            mbar_init(&acc_empty[b], TC_CONV_WARPS);
        }
        abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == TC_CONV_WARPS) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_slot)),
                     "r"(TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_d = tmem_base_slot;

    if (warp < TC_CONV_WARPS) {
        // ── converters: per K step a thread decodes 8 weights of its row and stores their two TF32 terms;
        // thread 0 also starts the TMA copies of the step's activation tiles.
        // Between chunks they read the finished accumulator back: warp w reads TMEM lanes 32 (w % 4) .. + 31
        // (its weight rows) and the quarter w / 4 of the columns (tokens). ──
        const uint32_t r = warp * ROWS_PER_WARP + (lane >> 2), unit = lane & 3;  // this thread's row and unit
        const uint64_t wrow = row0 + r < n ? row0 + r : n - 1;                  // rows past n repeat the last one
        const uint32_t q = warp & 3, grp = warp >> 2;
        constexpr int MY_COLS = N_TILE / 4;  // columns this thread accumulates
        float sums[MY_COLS];
#pragma unroll
        for (int c = 0; c < MY_COLS; ++c) sums[c] = 0.0f;
        // read chunk `c`'s accumulator and add it to the running sums
        auto drain = [&](uint32_t c) -> bool {
            const uint32_t buf = c & 1;
            if (!__all_sync(0xFFFFFFFFu, mbar_wait(&acc_full[buf], (c >> 1) & 1))) return false;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t taddr = tmem_d + ((q * 32) << 16) + buf * N_TILE + grp * MY_COLS;
            if constexpr (MY_COLS == 8) {
                uint32_t rr[8];
                tmem_ld8(taddr, rr);
#pragma unroll
                for (int i = 0; i < 8; ++i) sums[i] += __uint_as_float(rr[i]);
            } else if constexpr (MY_COLS == 16) {
                uint32_t rr[16];
                tmem_ld16(taddr, rr);
#pragma unroll
                for (int i = 0; i < 16; ++i) sums[i] += __uint_as_float(rr[i]);
            } else {
#pragma unroll
                for (int part = 0; part < MY_COLS / 32; ++part) {
                    uint32_t rr[32];
                    tmem_ld32(taddr + part * 32, rr);
#pragma unroll
                    for (int i = 0; i < 32; ++i) sums[part * 32 + i] += __uint_as_float(rr[i]);
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&acc_empty[buf]);
            return true;
        };
        bool ok = true;
        uint32_t drained = 0;
        for (uint32_t ks = 0; ks < k_steps && ok; ++ks) {
            const uint32_t s = ks % n_stages, round = ks / n_stages;
            // decode before waiting for the stage (the loads overlap the wait)
            float v[8];
            if (!(dbg_skip & 1)) {
                const uint32_t u = ks * 4 + unit;  // 8-value unit of the row
                decode_unit<TYPE>(w + wrow * row_bytes + (uint64_t)(u / UPB) * BYTES, u % UPB, v, false);
            }
            ok = __all_sync(0xFFFFFFFFu, mbar_wait(&empty[s], (round & 1) ^ 1));  // warp-uniform
            if (!ok) break;
            const bool tr = trace != nullptr && tid == 0 && blockIdx.x == 0 && blockIdx.y == 0 && ks < 64;
            if (tr) trace[8 * ks] = tc_now();
            uint8_t* st = smem + (size_t)s * STAGE;
            if (tid == 0) {
                // the stage is free: start the two activation tiles (hi, lo) of this K step on their way
                if (dbg_skip & 2) {
                    mbar_arrive(&full[s]);
                } else {
                    mbar_arrive_expect_tx(&full[s], 2 * PLANE_B);
                    tma_load_2d(st + 2 * PLANE_A, &map_hi, ks * TC_K, (uint32_t)tok0, &full[s]);
                    tma_load_2d(st + 2 * PLANE_A + PLANE_B, &map_lo, ks * TC_K, (uint32_t)tok0, &full[s]);
                }
            }
            if (!(dbg_skip & 1)) {
                store_split(st, st + PLANE_A, r, unit * 2, v);
                store_split(st, st + PLANE_A, r, unit * 2 + 1, v + 4);
            }
            // make the generic-proxy stores visible to the tensor core's async proxy, then hand over
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&full[s]);
            if (tr) trace[8 * ks + 1] = tc_now();
            // drain every finished chunk but the newest (which is still accumulating)
            while (ok && drained + 1 < (ks + 1) / TC_CHUNK) ok = drain(drained++);
        }
        while (ok && drained < n_chunks) ok = drain(drained++);
        if (!ok) abort_flag = 1;
        if (ok) {
            const uint64_t out_row = row0 + q * 32 + lane;
#pragma unroll
            for (int c = 0; c < MY_COLS; ++c) {
                const uint64_t tok = tok0 + grp * MY_COLS + c;
                if (tok < m && out_row < n) dst[tok * n + out_row] = sums[c];
            }
        }
    } else {
        // ── issuer: the whole warp walks the K steps and waits on the barriers (warp-uniform control flow); one
        // elected lane issues the tensor-core instructions and their commits ──
        const uint32_t idesc = umma_idesc(N_TILE);
        const uint32_t base0 = smem_u32(smem);
        const uint64_t d0_a_hi = umma_desc(base0), d0_a_lo = umma_desc(base0 + PLANE_A);
        const uint64_t d0_b_hi = umma_desc(base0 + 2 * PLANE_A), d0_b_lo = umma_desc(base0 + 2 * PLANE_A + PLANE_B);
        bool ok = true;
        uint32_t s = 0, round = 0;  // stage and its use count, stepped without a division
        for (uint32_t ks = 0; ks < k_steps && ok; ++ks) {
            const uint32_t chunk = ks / TC_CHUNK, buf = chunk & 1;
            const bool tr = trace != nullptr && lane == 0 && blockIdx.x == 0 && blockIdx.y == 0 && ks < 64;
            if (tr) trace[8 * ks + 2] = tc_now();
            if (ks % TC_CHUNK == 0 && chunk >= 2) {
                // the accumulator half must have been read back before it is overwritten
                ok = __all_sync(0xFFFFFFFFu, mbar_wait(&acc_empty[buf], ((chunk >> 1) - 1) & 1));
                if (!ok) break;
                // orders the MMAs below after the converters' reads of this half of tensor memory; the
                // shared-memory operands need no tensor-core fence (proxy fence + mbarrier)
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            }
            if (tr) trace[8 * ks + 3] = tc_now();
            ok = __all_sync(0xFFFFFFFFu, mbar_wait(&full[s], round & 1));
            if (!ok) break;
            if (tr) trace[8 * ks + 4] = tc_now();
            if (elect_one()) {
                // descriptors differ from the stage-0 ones only in the start-address field (bytes / 16, no carry
                // out of its 14 bits below 256 KB): one add each instead of rebuilding them
                const uint64_t so = (uint64_t)s * (STAGE >> 4);
                const uint64_t da_hi = d0_a_hi + so, da_lo = d0_a_lo + so, db_hi = d0_b_hi + so, db_lo = d0_b_lo + so;
                const uint32_t d = tmem_d + buf * N_TILE;
#pragma unroll
                for (uint32_t kk = 0; kk < TC_K / 8; ++kk) {
                    // one instruction covers K = 8 tf32 = 32 bytes of the swizzled row
                    const uint64_t adv = kk * 2;
                    umma_tf32(d, da_hi + adv, db_hi + adv, idesc, (ks % TC_CHUNK != 0) || kk != 0);
                    if (dbg_skip & 4) continue;  // measurement only: one product of the three
                    umma_tf32(d, da_hi + adv, db_lo + adv, idesc, 1);
                    umma_tf32(d, da_lo + adv, db_hi + adv, idesc, 1);
                }
                if (tr) trace[8 * ks + 5] = tc_now();
                umma_commit(&empty[s]);  // arrives when the instructions above have finished reading the stage
                if (tr) trace[8 * ks + 6] = tc_now();
                if ((ks + 1) % TC_CHUNK == 0 || ks + 1 == k_steps) umma_commit(&acc_full[buf]);
            }
            __syncwarp();
            if (tr) trace[8 * ks + 7] = tc_now();
            if (++s == n_stages) {
                s = 0;
                ++round;
            }
        }
        if (!ok && lane == 0) abort_flag = 1;
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (abort_flag && tid == 0) *reinterpret_cast<volatile int*>(error_flag) = 1;
    if (warp == TC_CONV_WARPS) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_d), "r"(TMEM_COLS) : "memory");
    }
}


PFN_cuTensorMapEncodeTiled g_encode_tiled = nullptr;

cudaError_t tensor_map_for(const float* base, uint64_t m, uint64_t k, uint32_t n_tile, CUtensorMap* out) {
    if (!g_encode_tiled) {
        void* fn = nullptr;
        cudaDriverEntryPointQueryResult qres;
        cudaError_t e = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qres);
        if (e != cudaSuccess) return e;
        if (qres != cudaDriverEntryPointSuccess || !fn) return cudaErrorNotSupported;
        g_encode_tiled = reinterpret_cast<PFN_cuTensorMapEncodeTiled>(fn);
    }
    const cuuint64_t dims[2] = {k, m};
    const cuuint64_t strides[1] = {k * 4};             // bytes between rows (a multiple of 16: k % 32 == 0)
    const cuuint32_t box[2] = {(cuuint32_t)TC_K, n_tile};  // 32 floats = one 128-byte swizzled row, n_tile rows
    const cuuint32_t estr[2] = {1, 1};
    CUresult r = g_encode_tiled(out, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(base), dims, strides, box, estr,
                                CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);  // rows beyond m read as zeros
    return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

template <uint32_t TYPE, uint32_t ELEMS, uint32_t BYTES, int N_TILE>
cudaError_t launch_tile(const uint8_t* w, uint64_t n, uint64_t k, const float* x_hi, const float* x_lo, uint64_t m,
                        float* dst, int* error_flag, cudaStream_t s) {
    constexpr uint32_t STAGE = 2 * PLANE_A + 2 * N_TILE * 128;
    uint32_t n_stages = std::min<uint32_t>(8, std::min<uint32_t>((uint32_t)(k / TC_K), (216 * 1024) / STAGE));
    size_t smem = (size_t)n_stages * STAGE + 1024;
    auto kern = gemm_tc_kernel<TYPE, ELEMS, BYTES, N_TILE>;
    static bool configured[MAX_DEVICES] = {};
    if (cudaError_t ce = set_max_smem_once(kern, 226 * 1024, configured); ce != cudaSuccess) return ce;
    CUtensorMap map_hi, map_lo;
    cudaError_t e = tensor_map_for(x_hi, m, k, N_TILE, &map_hi);
    if (e == cudaSuccess) e = tensor_map_for(x_lo, m, k, N_TILE, &map_lo);
    if (e != cudaSuccess) return e;
    dim3 grid((unsigned)((n + TC_M - 1) / TC_M), (unsigned)((m + N_TILE - 1) / N_TILE));
    // JQ_DEBUG_TC_SKIP (measurement only, results are wrong): bit 0 = no weight decode / stores, bit 1 = no TMA,
    // bit 2 = one tensor-core product instead of three
#ifdef JQ_PROFILING
    static const int dbg_skip = std::getenv("JQ_DEBUG_TC_SKIP") ? std::atoi(std::getenv("JQ_DEBUG_TC_SKIP")) : 0;
#else
    constexpr int dbg_skip = 0;  // the measurement switch exists in profiling builds only
#endif
    kern<<<grid, TC_THREADS, smem, s>>>(w, n, k, map_hi, map_lo, m, dst, n_stages, error_flag, g_gemm_trace, dbg_skip);
    return cudaGetLastError();
}

// Splits the activations once (hi and lo arrays of m * k floats each), then the tiles.
template <uint32_t TYPE, uint32_t ELEMS, uint32_t BYTES>
cudaError_t launch_type(const uint8_t* w, uint64_t n, uint64_t k, const float* lhs, uint64_t m, float* dst,
                        float* scratch, int* error_flag, cudaStream_t s) {
    float* x_hi = scratch;
    float* x_lo = scratch + ((m * k + 63) & ~(uint64_t)63);
    const uint64_t n4 = m * k / 4;
    split_tf32_kernel<<<(unsigned)std::min<uint64_t>((n4 + 255) / 256, 148 * 16), 256, 0, s>>>(lhs, n4, x_hi, x_lo);
    if (cudaError_t e = cudaGetLastError(); e != cudaSuccess) return e;
    if (m <= 32) return launch_tile<TYPE, ELEMS, BYTES, 32>(w, n, k, x_hi, x_lo, m, dst, error_flag, s);
    if (m <= 64) return launch_tile<TYPE, ELEMS, BYTES, 64>(w, n, k, x_hi, x_lo, m, dst, error_flag, s);
    return launch_tile<TYPE, ELEMS, BYTES, 128>(w, n, k, x_hi, x_lo, m, dst, error_flag, s);
}

}  // namespace

bool gemm_tc_supports(uint32_t type, const uint8_t* w, uint64_t n, uint64_t k, uint64_t m) {
    if (m == 0 || n == 0 || k == 0 || k % 32 != 0) return false;
    Format f;
    if (!format_of(type, &f)) return false;
    uint64_t row_bytes = k / f.elems * f.bytes;
    uintptr_t a = reinterpret_cast<uintptr_t>(w);
    // decode_unit's alignment needs hold for every row
    switch (type) {
        case T_Q8_0: return a % 2 == 0 && row_bytes % 2 == 0;
        case T_IQ2_XXS: return a % 2 == 0;
        case T_MXFP4: return true;
        default: return false;
    }
}

void gemm_tc_set_trace(unsigned long long* dev_buf) { g_gemm_trace = dev_buf; }

size_t gemm_tc_scratch_bytes(uint64_t m, uint64_t k) { return (size_t)(2 * ((m * k + 63) & ~(uint64_t)63) * 4 + 256); }

cudaError_t launch_gemm_tc(uint32_t type, const uint8_t* w, uint64_t n, uint64_t k, const float* lhs, uint64_t m,
                           float* dst, void* scratch_v, int* error_flag, cudaStream_t s) {
    float* scratch = static_cast<float*>(scratch_v);
    switch (type) {
        case T_Q8_0: return launch_type<T_Q8_0, 32, 34>(w, n, k, lhs, m, dst, scratch, error_flag, s);
        case T_IQ2_XXS: return launch_type<T_IQ2_XXS, 256, 66>(w, n, k, lhs, m, dst, scratch, error_flag, s);
        case T_MXFP4: return launch_type<T_MXFP4, 32, 17>(w, n, k, lhs, m, dst, scratch, error_flag, s);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace jq
