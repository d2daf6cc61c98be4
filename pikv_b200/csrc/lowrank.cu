// Low-rank projection GEMM on 5th-generation tensor cores:
//   out[M,N] = act(x[M,K] . w[N,K]^T + bias) (+ residual),  bf16 operands, fp32 accumulate.
//
// Persistent grid, one CTA per SM, 10 warps; an item is a 128-row tile of x times a block of bn <= 256 outputs, the
// blocks of one row tile next to each other (the tile comes from L2 after the first):
//   warp 0   TMA producer: cp.async.bulk.tensor 2D loads of a [128 x 64] tile of x and a
//            [bn x 64] tile of w (128-byte swizzle) into a shared-memory ring that runs on across items
//   warp 1   allocates tensor memory, one lane issues tcgen05.mma (M=128, N=bn, K=16; four
//            per 64-wide k block) straight from shared-memory descriptors into one of two accumulators
//            and signals stage release / accumulator completion with tcgen05.commit
//   warps 2-9 epilogue: tcgen05.ld their accumulator rows (two warps per 32 rows, alternate 128-byte column
//            chunks), bias + ReLU (+ residual) in registers, rows into a swizzled [128 x 128 B] staging tile that a
//            TMA store writes out in whole lines; it runs beside the loads and MMAs of the next item
// Bound by HBM (60 FLOP/B at rank 64, far below the ridge): what matters is that loads stay in flight through the
// epilogue and that stores leave as full lines.  With one CTA per item and a row per thread storing 32 bytes at a
// stride of a whole output row, the reconstruction 262144 x 64 -> 1024 took 560 us for 570 MB and the projection
// 1024 -> 64 107 us; now 182 us (a plain fill of that output takes 140) and 98 us = 5.8 TB/s.
// Every mbarrier wait is bounded; on a timeout the CTA sets an error word and drains.
#include "tc_common.cuh"

namespace pikv {

constexpr int LR_EPI_WARPS = 8;
constexpr int LR_THREADS = 64 + 32 * LR_EPI_WARPS;
constexpr int LR_MAX_BN = 256;
constexpr int LR_STAGING = LR_BM * 128;        // one staging tile: 128 rows of 128 bytes
constexpr int LR_BIAS_SMEM = 4096;             // output columns whose bias is kept in shared memory

__device__ unsigned g_lowrank_error = 0;   // sticky: set when a bounded wait ran out

struct LowrankArgs {
    const void* bias;
    const __nv_bfloat16* residual;
    int bias_bf16, M, N, K, relu, bn, stages, tmem_cols, items, nblocks, halves, bias_smem;
};

__device__ __forceinline__ float lr_bias(const LowrankArgs& a, int n) {
    return a.bias_bf16 ? bf16_bits_to_f32(__ldg(static_cast<const unsigned short*>(a.bias) + n))
                       : __ldg(static_cast<const float*>(a.bias) + n);
}

template <int HALF>
__device__ __forceinline__ void lr_half_barrier() { asm volatile("bar.sync %0, 128;" ::"n"(1 + HALF) : "memory"); }

// the accumulator columns [c, c + 16 * G) of this thread's row, biased, rectified and (residual) added to
template <int G>
__device__ __forceinline__ void lr_finish(const LowrankArgs& a, uint32_t taddr, const float* bias_s, int n, int m, float (&v)[16 * G]) {
#pragma unroll
    for (int q = 0; q < G; ++q) {
        float r[16];
        lr_tmem_ld16(taddr + 16 * q, r);
#pragma unroll
        for (int i = 0; i < 16; ++i) v[16 * q + i] = r[i];
    }
    if (a.bias) {
        if (a.bias_smem) {
#pragma unroll
            for (int i = 0; i < 16 * G; i += 4) {
                const float4 b = *reinterpret_cast<const float4*>(bias_s + n + i);
                v[i] += b.x; v[i + 1] += b.y; v[i + 2] += b.z; v[i + 3] += b.w;
            }
        } else {
#pragma unroll
            for (int i = 0; i < 16 * G; ++i) v[i] += n + i < a.N ? lr_bias(a, n + i) : 0.f;
        }
    }
    if (a.relu) {
#pragma unroll
        for (int i = 0; i < 16 * G; ++i) v[i] = fmaxf(v[i], 0.f);
    }
    if (a.residual && m < a.M) {
#pragma unroll
        for (int q = 0; q < G; ++q) {
            if (n + 16 * q >= a.N) break;
            const uint4* rp = reinterpret_cast<const uint4*>(a.residual + (size_t)m * a.N + n + 16 * q);
            const uint4 r0 = __ldg(rp), r1 = __ldg(rp + 1);
            const uint32_t rw[8] = {r0.x, r0.y, r0.z, r0.w, r1.x, r1.y, r1.z, r1.w};
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                float lo, hi;
                bf16x2_to_f32(rw[i], lo, hi);
                v[16 * q + 2 * i] += lo;
                v[16 * q + 2 * i + 1] += hi;
            }
        }
    }
}

// Drains one accumulator: the 128-byte column chunks of this half, through its two staging tiles.
template <bool F32, int HALF>
__device__ __forceinline__ void lr_store_half(const LowrankArgs& a, const CUtensorMap* tm_out, uint32_t tmem, unsigned char* staging,
                                              const float* bias_s, int n0, int m0, int row, uint32_t lane_addr, bool leader, int& used) {
    constexpr int CW = F32 ? 32 : 64;                     // columns per chunk
    const int chunks = (min(a.bn, a.N - n0) + CW - 1) / CW;
    for (int ch = HALF; ch < chunks; ch += a.halves) {
        unsigned char* tile = staging + (size_t)(HALF * 2 + (used & 1)) * LR_STAGING;
        // the store that used this tile two chunks ago has read it
        if (leader) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
        lr_half_barrier<HALF>();
        unsigned char* dst = tile + row * 128;
#pragma unroll
        for (int c = 0; c < CW; c += 16) {
            if (ch * CW + c >= a.bn) break;               // an accumulator narrower than the chunk
            float v[16];
            lr_finish<1>(a, tmem + lane_addr + (uint32_t)(ch * CW + c), bias_s, n0 + ch * CW + c, m0 + row, v);
            if constexpr (F32) {
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    *reinterpret_cast<float4*>(dst + 16 * ((c / 4 + i) ^ (row & 7))) = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
            } else {
                uint32_t pk[8];
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    pk[i] = (uint32_t)f32_to_bf16_bits(v[2 * i]) | ((uint32_t)f32_to_bf16_bits(v[2 * i + 1]) << 16);
                *reinterpret_cast<uint4*>(dst + 16 * ((c / 8) ^ (row & 7))) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
                *reinterpret_cast<uint4*>(dst + 16 * ((c / 8 + 1) ^ (row & 7))) = make_uint4(pk[4], pk[5], pk[6], pk[7]);
            }
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        lr_half_barrier<HALF>();
        if (leader) {
            lr_tma_store_2d(tm_out, lr_smem_u32(tile), n0 + ch * CW, m0);
            asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        }
        ++used;
    }
}

template <bool F32>
__global__ void __launch_bounds__(LR_THREADS, 1) lowrank_gemm_kernel(const __grid_constant__ CUtensorMap tm_x,
                                                                  const __grid_constant__ CUtensorMap tm_w,
                                                                  const __grid_constant__ CUtensorMap tm_out,
                                                                  LowrankArgs a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    // operand and staging tiles with the 128-byte swizzle must start on a 1024-byte boundary
    unsigned char* smem = smem_raw + ((1024u - (lr_smem_u32(smem_raw) & 1023u)) & 1023u);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int stage_a = LR_BM * LR_BK * 2;
    const int stage_b = a.bn * LR_BK * 2;
    const int stage_bytes = stage_a + stage_b;
    // staging tiles and ring first (1024-byte aligned), then bias, barriers and the tensor-memory address slot
    unsigned char* staging = smem;
    unsigned char* ring_p = staging + (size_t)2 * a.halves * LR_STAGING;
    float* bias_s = reinterpret_cast<float*>(ring_p + (size_t)a.stages * ((stage_bytes + 1023) & ~1023));
    uint64_t* bars = reinterpret_cast<uint64_t*>(bias_s + (a.bias_smem ? ((a.N + 255) & ~255) : 0));
    const uint32_t full0 = lr_smem_u32(bars);
    const uint32_t empty0 = full0 + 8 * a.stages;
    const uint32_t tfull0 = empty0 + 8 * a.stages;
    const uint32_t tempty0 = tfull0 + 16;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * a.stages + 4);
    const uint32_t ring = lr_smem_u32(ring_p);
    const uint32_t stride = (uint32_t)((stage_bytes + 1023) & ~1023);
    const int num_kb = (a.K + LR_BK - 1) / LR_BK;   // a ragged last block is zero-filled by TMA

    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (threadIdx.x == 0) {
        for (int s = 0; s < a.stages; ++s) {
            lr_mbar_init(full0 + 8 * s, 1);
            lr_mbar_init(empty0 + 8 * s, 1);
        }
        for (int s = 0; s < 2; ++s) {
            lr_mbar_init(tfull0 + 8 * s, 1);
            lr_mbar_init(tempty0 + 8 * s, 32 * LR_EPI_WARPS);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        lr_prefetch_tmap(&tm_x);
        lr_prefetch_tmap(&tm_w);
        lr_prefetch_tmap(&tm_out);
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(lr_smem_u32(tmem_slot)), "r"((uint32_t)a.tmem_cols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    // launched as a programmatic dependent: everything above overlaps the end of the kernel before
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (a.bias_smem)
        for (int i = threadIdx.x; i < ((a.N + 255) & ~255); i += LR_THREADS) bias_s[i] = i < a.N ? lr_bias(a, i) : 0.f;
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = *tmem_slot;
    bool failed = false;

    if (warp == 0) {
        LrRing r;
        for (int item = blockIdx.x; item < a.items && !failed; item += gridDim.x) {
            const int m0 = item / a.nblocks * LR_BM, n0 = item % a.nblocks * a.bn;
            for (int kb = 0; kb < num_kb; ++kb, r.next(a.stages)) {
                if (!lr_mbar_wait(empty0 + 8 * r.s, r.ph ^ 1u)) { failed = true; break; }
                if (lr_elect()) {
                    lr_mbar_expect_tx(full0 + 8 * r.s, (uint32_t)stage_bytes);
                    const uint32_t dst = ring + (uint32_t)r.s * stride;
                    lr_tma_load_2d(dst, &tm_x, kb * LR_BK, m0, full0 + 8 * r.s);
                    lr_tma_load_2d(dst + stage_a, &tm_w, kb * LR_BK, n0, full0 + 8 * r.s);
                }
                __syncwarp();
            }
        }
    } else if (warp == 1) {
        const uint32_t idesc = lr_instr_desc(a.bn);
        const uint32_t a_lo = lr_desc_lo(ring), b_lo = lr_desc_lo(ring + stage_a), stage_lo = stride >> 4;
        LrRing r;
        int local = 0;
        for (int item = blockIdx.x; item < a.items && !failed; item += gridDim.x, ++local) {
            const int slot = local & 1;
            if (!lr_mbar_wait(tempty0 + 8 * slot, (((uint32_t)local >> 1) & 1u) ^ 1u)) { failed = true; break; }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t d = tmem_base + (uint32_t)(slot * a.bn);
            for (int kb = 0; kb < num_kb; ++kb, r.next(a.stages)) {
                if (!lr_mbar_wait(full0 + 8 * r.s, r.ph)) { failed = true; break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                if (lr_elect()) {
                    const uint32_t off = (uint32_t)r.s * stage_lo;
#pragma unroll
                    for (int k = 0; k < LR_BK / 16; ++k)
                        lr_mma(d, lr_desc(a_lo + off + 2 * k), lr_desc(b_lo + off + 2 * k), idesc, (kb | k) ? 1u : 0u);
                    lr_commit(empty0 + 8 * r.s);     // frees the stage once these MMAs have read it
                }
                __syncwarp();
            }
            if (lr_elect()) lr_commit(tfull0 + 8 * slot);    // accumulator complete (or as far as it got)
            __syncwarp();
        }
    } else {
        const int lg = warp & 3;                     // tensor-memory lane group of this warp
        const int half = (warp - 2) >> 2;
        const int row = lg * 32 + lane;
        const uint32_t lane_addr = (uint32_t)(lg * 32) << 16;
        const bool leader = (warp == 2 || warp == 6) && lane == 0;
        int local = 0, used = 0;
        for (int item = blockIdx.x; item < a.items; item += gridDim.x, ++local) {
            const int slot = local & 1;
            const int m0 = item / a.nblocks * LR_BM, n0 = item % a.nblocks * a.bn;
            // no way out of the loop on a timeout: the threads of a half meet at its barriers
            if (!failed && !lr_mbar_wait(tfull0 + 8 * slot, ((uint32_t)local >> 1) & 1u)) failed = true;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t tmem = tmem_base + (uint32_t)(slot * a.bn);
            if (half == 0) lr_store_half<F32, 0>(a, &tm_out, tmem, staging, bias_s, n0, m0, row, lane_addr, leader, used);
            else if (a.halves == 2) lr_store_half<F32, 1>(a, &tm_out, tmem, staging, bias_s, n0, m0, row, lane_addr, leader, used);
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            lr_mbar_arrive(tempty0 + 8 * slot);
        }
        if (leader) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    }
    if (failed) atomicOr(&g_lowrank_error, 1u);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)a.tmem_cols) : "memory");
    }
}

}  // namespace pikv

using namespace pikv;

extern "C" int pikv_lowrank_project_bias(const void* x, const void* w, const void* bias, int32_t bias_dtype,
                                         const void* residual, void* out, int32_t out_dtype, int32_t M, int32_t N,
                                         int32_t K, int32_t relu, pikv_stream_t stream) {
    PIKV_REQUIRE(x && w && out, PIKV_EINVAL, "lowrank: null pointer");
    PIKV_REQUIRE(M > 0 && N > 0 && K > 0, PIKV_EINVAL, "lowrank: bad sizes");
    PIKV_REQUIRE(K % 16 == 0, PIKV_EUNSUPPORTED, "lowrank: K=%d must be a multiple of 16", K);
    PIKV_REQUIRE(N % 16 == 0, PIKV_EUNSUPPORTED, "lowrank: N=%d must be a multiple of 16", N);
    PIKV_REQUIRE(bias_dtype == PIKV_BF16 || bias_dtype == PIKV_F32, PIKV_EINVAL, "lowrank: bad bias dtype");
    PIKV_REQUIRE(out_dtype == PIKV_BF16 || out_dtype == PIKV_F32, PIKV_EINVAL, "lowrank: bad out dtype");
    PIKV_REQUIRE(((uintptr_t)x % 16) == 0 && ((uintptr_t)w % 16) == 0 && ((uintptr_t)out % 16) == 0, PIKV_EINVAL,
                 "lowrank: pointers must be 16-byte aligned");
    PIKV_REQUIRE(N <= LR_MAX_BN || N % LR_MAX_BN == 0, PIKV_EUNSUPPORTED, "lowrank: N=%d above %d must be a multiple of %d", N, LR_MAX_BN, LR_MAX_BN);
    LowrankArgs a = {};
    a.bias = bias;
    a.bias_bf16 = bias_dtype == PIKV_BF16;
    a.residual = static_cast<const __nv_bfloat16*>(residual);
    a.M = M; a.N = N; a.K = K; a.relu = relu;
    const bool f32 = out_dtype == PIKV_F32;
    const int tiles = ceil_div(M, LR_BM), sms = sm_count();
    // the widest block re-reads x least; narrower ones when that leaves SMs without an item
    a.bn = min(N, LR_MAX_BN);
    while (a.bn % 128 == 0 && tiles * ceil_div(N, a.bn) < sms) a.bn /= 2;
    a.nblocks = ceil_div(N, a.bn);
    a.items = tiles * a.nblocks;
    CUtensorMap tm_x, tm_w, tm_out;
    int rc = make_tmap(&tm_x, x, M, K, LR_BM);
    if (rc != PIKV_OK) return rc;
    rc = make_tmap(&tm_w, w, N, K, a.bn);
    if (rc != PIKV_OK) return rc;
    rc = f32 ? make_tmap_f32(&tm_out, out, M, N, LR_BM) : make_tmap(&tm_out, out, M, N, LR_BM);
    if (rc != PIKV_OK) return rc;
    a.halves = a.bn > (f32 ? 32 : 64) ? 2 : 1;
    a.bias_smem = bias != nullptr && N <= LR_BIAS_SMEM;
    const int stride = (LR_BM * LR_BK * 2 + a.bn * LR_BK * 2 + 1023) & ~1023;
    const size_t fixed = (size_t)2 * a.halves * LR_STAGING + (a.bias_smem ? ((N + 255) & ~255) * sizeof(float) : 0) +
                         (2 * 8 + 4) * sizeof(uint64_t) + 16 + 1024;
    a.stages = (int)max((size_t)2, min((size_t)8, ((size_t)227 * 1024 - fixed) / stride));
    int cols = 32;
    while (cols < 2 * a.bn) cols <<= 1;
    a.tmem_cols = cols;
    const size_t smem = (size_t)a.stages * stride + fixed;
    auto kern = f32 ? lowrank_gemm_kernel<true> : lowrank_gemm_kernel<false>;
    if (!(f32 ? allow_smem<lowrank_gemm_kernel<true>>() : allow_smem<lowrank_gemm_kernel<false>>())) return check_launch("lowrank smem attribute");
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = min(a.items, sms);
    cfg.blockDim = LR_THREADS;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = static_cast<cudaStream_t>(stream);
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kern, tm_x, tm_w, tm_out, a);
    count_launch(1);
    return check_launch("lowrank_gemm_kernel");
}

extern "C" int pikv_lowrank_project(const void* x, const void* w, const float* bias, const void* residual, void* out,
                                    int32_t out_dtype, int32_t M, int32_t N, int32_t K, int32_t relu,
                                    pikv_stream_t stream) {
    return pikv_lowrank_project_bias(x, w, bias, PIKV_F32, residual, out, out_dtype, M, N, K, relu, stream);
}

namespace pikv {
int lowrank_pair_error_fetch();
int linear_error_fetch();
}  // namespace pikv

// reads and clears the sticky error words of the tcgen05 kernels (synchronises the stream's device)
extern "C" int pikv_lowrank_error_state(void) {
    unsigned v = 0, zero = 0;
    if (cudaMemcpyFromSymbol(&v, g_lowrank_error, sizeof(v)) != cudaSuccess) return -1;
    if (v) cudaMemcpyToSymbol(g_lowrank_error, &zero, sizeof(zero));
    const int pair = pikv::lowrank_pair_error_fetch();
    const int linear = pikv::linear_error_fetch();
    return pair < 0 || linear < 0 ? -1 : (int)v | pair | linear;
}
