// Low-rank round trip of the K and V of one batch in one kernel (SVDCompressor.forward, bf16):
//   out = relu(x[M,K] . w1[R,K]^T + b1) . w2[N,R]^T + b2        R <= 64, the latent rounded to bf16 in between
//
// Persistent grid, one CTA per SM, 12 warps; an item is 128 rows of K or V:
//   warp 0    TMA: a [128 x 64] tile of x and a [R x 64] tile of w1 per ring stage
//   warp 1    first product, tcgen05 M=128 N=R, into one of two accumulators (so the next item's loads and MMAs run
//             while this item is written out)
//   warp 2    TMA: [64 x R] tiles of w2, four in flight
//   warp 3    second product, M=128 N=64 per output chunk, into one of four accumulators
//   warps 4-11  the latent (bias, ReLU, bf16) into the swizzled A operand of the second product, then two groups of
//             four warps take alternate output chunks: bias and a 32-row staging tile per warp that a TMA store writes
//             out in whole lines
// Bound by HBM, and the reason for one kernel is the mix: this part writes at 3.8 TB/s at most but moves 6.4 TB/s when
// it reads as much as it writes, so a projection that only reads followed by a reconstruction that only writes cannot
// reach the copy rate.  K and V of 262144 x 1024 at rank 64 (2.15 GB): four
// launches of the separate products 563 us, this kernel 364 us = 5.9 TB/s; 256 rows per item (half the weight traffic)
// 386 us, as filling and draining the pipeline took twice as long.
// Every mbarrier wait is bounded; on a timeout the CTA sets the projection's error word and drains.
#include "tc_common.cuh"

namespace pikv {

constexpr int LP_THREADS = 384;
constexpr int LP_BUF = 4;                     // w2 tiles and second-product accumulators in flight
constexpr int LP_CHUNK = 64;                  // output columns per second-product tile = one 128-byte line of bf16
constexpr int LP_TILE = LR_BM * LR_BK * 2;    // 16 KB operand tile
constexpr int LP_W2_TILE = LP_CHUNK * LR_BK * 2;
constexpr int LP_STAGE_OUT = 32 * 128;        // staging tile of one warp
constexpr int LP_MAX_N = 4096;                // output columns whose bias fits in shared memory

struct LowrankPairMaps {
    CUtensorMap x[2], w1[2], w2[2], out[2];
};
struct LowrankPairArgs {
    const void* b1[2];
    const void* b2[2];
    int bias_bf16, M, N, K, R, stages, tiles, items;
};

__device__ unsigned g_lowrank_pair_error = 0;   // sticky: a bounded wait ran out

__device__ __forceinline__ float lp_bias(const void* b, int bf16, int i) {
    return bf16 ? bf16_bits_to_f32(__ldg(static_cast<const unsigned short*>(b) + i)) : __ldg(static_cast<const float*>(b) + i);
}

// a wait of a whole warp: all lanes agree on the outcome
__device__ __forceinline__ bool lp_warp_wait(uint32_t bar, uint32_t parity) {
    return __all_sync(0xffffffffu, lr_mbar_wait(bar, parity));
}

__global__ void __launch_bounds__(LP_THREADS, 1) lowrank_pair_kernel(const __grid_constant__ LowrankPairMaps tm, LowrankPairArgs a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    unsigned char* smem = smem_raw + ((1024u - (lr_smem_u32(smem_raw) & 1023u)) & 1023u);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int stage_bytes = LP_TILE + a.R * LR_BK * 2;
    unsigned char* ring_p = smem;                                      // [stages][x, w1]
    unsigned char* lat_p = ring_p + (size_t)a.stages * stage_bytes;    // [item & 1][128 x 64] latent
    unsigned char* w2_p = lat_p + 2 * LP_TILE;                         // [LP_BUF][64 x 64]
    unsigned char* out_p = w2_p + LP_BUF * LP_W2_TILE;                      // [8 warps][2][32 x 64]
    float* b2_s = reinterpret_cast<float*>(out_p + 16 * LP_STAGE_OUT); // [2][N rounded up]
    const int npad = (a.N + LP_CHUNK - 1) / LP_CHUNK * LP_CHUNK;
    float* b1_s = b2_s + 2 * npad;                                     // [2][64]
    uint64_t* bars = reinterpret_cast<uint64_t*>(b1_s + 2 * 64);
    const uint32_t full0 = lr_smem_u32(bars), empty0 = full0 + 8 * a.stages;
    const uint32_t d1_full = empty0 + 8 * a.stages, d1_empty = d1_full + 16;            // [item & 1]
    const uint32_t lat_full = d1_empty + 16, lat_empty = lat_full + 16;                 // [item & 1]
    const uint32_t w2_full = lat_empty + 16, w2_empty = w2_full + 8 * LP_BUF;           // [LP_BUF]
    const uint32_t d2_full = w2_empty + 8 * LP_BUF, d2_empty = d2_full + 8 * LP_BUF;    // [LP_BUF]
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * a.stages + 8 + 4 * LP_BUF);
    const uint32_t ring = lr_smem_u32(ring_p), lat = lr_smem_u32(lat_p), w2s = lr_smem_u32(w2_p);
    const int num_kb = (a.K + LR_BK - 1) / LR_BK, chunks = npad / LP_CHUNK;

    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (threadIdx.x == 0) {
        for (int s = 0; s < a.stages; ++s) {
            lr_mbar_init(full0 + 8 * s, 1);
            lr_mbar_init(empty0 + 8 * s, 1);
        }
        for (int i = 0; i < 2; ++i) {
            lr_mbar_init(d1_full + 8 * i, 1);
            lr_mbar_init(d1_empty + 8 * i, 256);
            lr_mbar_init(lat_full + 8 * i, 256);
            lr_mbar_init(lat_empty + 8 * i, 1);
        }
        for (int i = 0; i < LP_BUF; ++i) {
            lr_mbar_init(w2_full + 8 * i, 1);
            lr_mbar_init(w2_empty + 8 * i, 1);
            lr_mbar_init(d2_full + 8 * i, 1);
            lr_mbar_init(d2_empty + 8 * i, 128);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(lr_smem_u32(tmem_slot)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");
    for (int i = threadIdx.x; i < 2 * npad; i += LP_THREADS) {
        const int t = i / npad, n = i % npad;
        b2_s[i] = a.b2[t] && n < a.N ? lp_bias(a.b2[t], a.bias_bf16, n) : 0.f;
    }
    if (threadIdx.x < 128) {
        const int t = threadIdx.x >> 6, r = threadIdx.x & 63;
        b1_s[threadIdx.x] = a.b1[t] && r < a.R ? lp_bias(a.b1[t], a.bias_bf16, r) : 0.f;
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot;
    // tensor memory: first product [item & 1] x 64 columns, second product [LP_BUF] x 64 columns
    const uint32_t d1_base = tmem, d2_base = tmem + 128;
    bool failed = false;

    if (warp == 0) {
        LrRing r;
        for (int item = blockIdx.x; item < a.items && !failed; item += gridDim.x) {
            const int t = item / a.tiles, m0 = item % a.tiles * LR_BM;
            for (int kb = 0; kb < num_kb; ++kb, r.next(a.stages)) {
                if (!lr_mbar_wait(empty0 + 8 * r.s, r.ph ^ 1u)) { failed = true; break; }
                if (lr_elect()) {
                    lr_mbar_expect_tx(full0 + 8 * r.s, (uint32_t)stage_bytes);
                    const uint32_t dst = ring + (uint32_t)(r.s * stage_bytes);
                    lr_tma_load_2d(dst, &tm.x[t], kb * LR_BK, m0, full0 + 8 * r.s);
                    lr_tma_load_2d(dst + LP_TILE, &tm.w1[t], kb * LR_BK, 0, full0 + 8 * r.s);
                }
                __syncwarp();
            }
        }
    } else if (warp == 1) {
        const uint32_t idesc = lr_instr_desc(a.R);
        const uint32_t a_lo = lr_desc_lo(ring), b_lo = lr_desc_lo(ring + LP_TILE), stage_lo = (uint32_t)stage_bytes >> 4;
        LrRing r;
        int n = 0;
        for (int item = blockIdx.x; item < a.items && !failed; item += gridDim.x, ++n) {
            const int b = n & 1;
            if (!lr_mbar_wait(d1_empty + 8 * b, (((uint32_t)n >> 1) & 1u) ^ 1u)) { failed = true; break; }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            for (int kb = 0; kb < num_kb; ++kb, r.next(a.stages)) {
                if (!lr_mbar_wait(full0 + 8 * r.s, r.ph)) { failed = true; break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                if (lr_elect()) {
                    const uint32_t off = (uint32_t)r.s * stage_lo;
#pragma unroll
                    for (int k = 0; k < LR_BK / 16; ++k)
                        lr_mma(d1_base + (uint32_t)(64 * b), lr_desc(a_lo + off + 2 * k), lr_desc(b_lo + off + 2 * k), idesc, (kb | k) ? 1u : 0u);
                    lr_commit(empty0 + 8 * r.s);
                }
                __syncwarp();
            }
            if (lr_elect()) lr_commit(d1_full + 8 * b);
            __syncwarp();
        }
    } else if (warp == 2) {
        LrRing r;
        for (int item = blockIdx.x; item < a.items && !failed; item += gridDim.x) {
            const int t = item / a.tiles;
            for (int c = 0; c < chunks; ++c, r.next(LP_BUF)) {
                if (!lr_mbar_wait(w2_empty + 8 * r.s, r.ph ^ 1u)) { failed = true; break; }
                if (lr_elect()) {
                    lr_mbar_expect_tx(w2_full + 8 * r.s, (uint32_t)LP_W2_TILE);
                    lr_tma_load_2d(w2s + (uint32_t)(r.s * LP_W2_TILE), &tm.w2[t], 0, c * LP_CHUNK, w2_full + 8 * r.s);
                }
                __syncwarp();
            }
        }
    } else if (warp == 3) {
        const uint32_t idesc = lr_instr_desc(LP_CHUNK);
        const uint32_t a_lo = lr_desc_lo(lat), b_lo = lr_desc_lo(w2s);
        const int steps = a.R / 16;
        LrRing r;
        int n = 0;
        for (int item = blockIdx.x; item < a.items && !failed; item += gridDim.x, ++n) {
            const int b = n & 1;
            if (!lr_mbar_wait(lat_full + 8 * b, ((uint32_t)n >> 1) & 1u)) { failed = true; break; }
            for (int c = 0; c < chunks; ++c, r.next(LP_BUF)) {
                if (!lr_mbar_wait(w2_full + 8 * r.s, r.ph) || !lr_mbar_wait(d2_empty + 8 * r.s, r.ph ^ 1u)) { failed = true; break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                if (lr_elect()) {
                    const uint32_t alo = a_lo + (uint32_t)b * (LP_TILE >> 4), blo = b_lo + (uint32_t)r.s * (LP_W2_TILE >> 4);
#pragma unroll
                    for (int k = 0; k < LR_BK / 16; ++k)
                        if (k < steps) lr_mma(d2_base + (uint32_t)(64 * r.s), lr_desc(alo + 2 * k), lr_desc(blo + 2 * k), idesc, k ? 1u : 0u);
                    lr_commit(d2_full + 8 * r.s);
                    lr_commit(w2_empty + 8 * r.s);
                }
                __syncwarp();
            }
            if (lr_elect()) lr_commit(lat_empty + 8 * b);     // the latent has been read for the last time
            __syncwarp();
        }
    } else {
        const int group = (warp - 4) >> 2, lg = warp & 3;
        const int row = lg * 32 + lane;
        const uint32_t lane_addr = (uint32_t)(lg * 32) << 16;
        unsigned char* stage = out_p + (size_t)(warp - 4) * 2 * LP_STAGE_OUT;
        int it = 0, n = 0, used = 0;
        for (int item = blockIdx.x; item < a.items && !failed; item += gridDim.x, ++n) {
            const int t = item / a.tiles, m0 = item % a.tiles * LR_BM, b = n & 1;
            // ---- latent: accumulator -> bias, ReLU, bf16 -> A operand of the second product ----
            if (!lp_warp_wait(d1_full + 8 * b, ((uint32_t)n >> 1) & 1u) || !lp_warp_wait(lat_empty + 8 * b, (((uint32_t)n >> 1) & 1u) ^ 1u)) {
                failed = true;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            unsigned char* lrow = lat_p + b * LP_TILE + row * 128;
            for (int c = 16 * group; c < a.R; c += 32) {
                float v[16];
                lr_tmem_ld16(d1_base + lane_addr + (uint32_t)(64 * b + c), v);
                uint32_t pk[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const float2 bias = *reinterpret_cast<const float2*>(b1_s + 64 * t + c + 2 * i);
                    pk[i] = (uint32_t)f32_to_bf16_bits(fmaxf(v[2 * i] + bias.x, 0.f)) |
                            ((uint32_t)f32_to_bf16_bits(fmaxf(v[2 * i + 1] + bias.y, 0.f)) << 16);
                }
                *reinterpret_cast<uint4*>(lrow + 16 * ((c / 8) ^ (row & 7))) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
                *reinterpret_cast<uint4*>(lrow + 16 * ((c / 8 + 1) ^ (row & 7))) = make_uint4(pk[4], pk[5], pk[6], pk[7]);
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            lr_mbar_arrive(d1_empty + 8 * b);
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            lr_mbar_arrive(lat_full + 8 * b);
            // ---- output chunks ----
            for (int c = 0; c < chunks; ++c, ++it) {
                if ((it & 1) != group) continue;
                const int s = it % LP_BUF;
                if (!lp_warp_wait(d2_full + 8 * s, (uint32_t)(it / LP_BUF) & 1u)) { failed = true; break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                float v[4][16];
                lr_tmem_ld32(d2_base + lane_addr + (uint32_t)(64 * s), v[0]);
                lr_tmem_ld32(d2_base + lane_addr + (uint32_t)(64 * s + 32), v[2]);
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                lr_mbar_arrive(d2_empty + 8 * s);
                // the store that used this staging tile two chunks ago has read it
                if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
                __syncwarp();
                unsigned char* tile = stage + (used++ & 1) * LP_STAGE_OUT;
                const float* b2 = b2_s + t * npad + c * LP_CHUNK;
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    uint32_t pk[8];
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const float4 b = *reinterpret_cast<const float4*>(b2 + 16 * q + 4 * i);
                        pk[2 * i] = (uint32_t)f32_to_bf16_bits(v[q][4 * i] + b.x) | ((uint32_t)f32_to_bf16_bits(v[q][4 * i + 1] + b.y) << 16);
                        pk[2 * i + 1] = (uint32_t)f32_to_bf16_bits(v[q][4 * i + 2] + b.z) | ((uint32_t)f32_to_bf16_bits(v[q][4 * i + 3] + b.w) << 16);
                    }
                    *reinterpret_cast<uint4*>(tile + lane * 128 + 16 * ((2 * q) ^ (lane & 7))) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
                    *reinterpret_cast<uint4*>(tile + lane * 128 + 16 * ((2 * q + 1) ^ (lane & 7))) = make_uint4(pk[4], pk[5], pk[6], pk[7]);
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) {
                    if (m0 + lg * 32 < a.M) lr_tma_store_2d(&tm.out[t], lr_smem_u32(tile), c * LP_CHUNK, m0 + lg * 32);
                    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                }
            }
        }
        if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    }
    if (failed) atomicOr(&g_lowrank_pair_error, 1u);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
    }
}

// reads and clears this kernel's sticky error word (called by pikv_lowrank_error_state)
int lowrank_pair_error_fetch() {
    unsigned v = 0, zero = 0;
    if (cudaMemcpyFromSymbol(&v, g_lowrank_pair_error, sizeof(v)) != cudaSuccess) return -1;
    if (v) cudaMemcpyToSymbol(g_lowrank_pair_error, &zero, sizeof(zero));
    return (int)v;
}

}  // namespace pikv

using namespace pikv;

extern "C" int pikv_lowrank_pair(const void* const* x, const void* const* w1, const void* const* b1, const void* const* w2,
                                 const void* const* b2, int32_t bias_dtype, void* const* out, int32_t M, int32_t K,
                                 int32_t R, int32_t N, pikv_stream_t stream) {
    PIKV_REQUIRE(x && w1 && b1 && w2 && b2 && out, PIKV_EINVAL, "lowrank_pair: null pointer");
    PIKV_REQUIRE(M > 0 && N > 0 && K > 0 && R > 0, PIKV_EINVAL, "lowrank_pair: bad sizes");
    PIKV_REQUIRE(R % 16 == 0 && R <= 64, PIKV_EUNSUPPORTED, "lowrank_pair: rank %d must be a multiple of 16 up to 64", R);
    PIKV_REQUIRE(K % 8 == 0 && N % 8 == 0 && N <= LP_MAX_N, PIKV_EUNSUPPORTED, "lowrank_pair: K=%d and N=%d must be multiples of 8, N <= %d", K, N, LP_MAX_N);
    PIKV_REQUIRE(bias_dtype == PIKV_BF16 || bias_dtype == PIKV_F32, PIKV_EINVAL, "lowrank_pair: bad bias dtype");
    LowrankPairMaps tm;
    LowrankPairArgs a = {};
    for (int t = 0; t < 2; ++t) {
        PIKV_REQUIRE(x[t] && w1[t] && w2[t] && out[t], PIKV_EINVAL, "lowrank_pair: null pointer");
        PIKV_REQUIRE((((uintptr_t)x[t] | (uintptr_t)w1[t] | (uintptr_t)w2[t] | (uintptr_t)out[t]) & 15) == 0, PIKV_EINVAL,
                     "lowrank_pair: pointers must be 16-byte aligned");
        int rc = make_tmap(&tm.x[t], x[t], M, K, LR_BM);
        if (rc == PIKV_OK) rc = make_tmap(&tm.w1[t], w1[t], R, K, R);
        if (rc == PIKV_OK) rc = make_tmap(&tm.w2[t], w2[t], N, R, LP_CHUNK);
        if (rc == PIKV_OK) rc = make_tmap(&tm.out[t], out[t], M, N, 32);
        if (rc != PIKV_OK) return rc;
        a.b1[t] = b1[t];
        a.b2[t] = b2[t];
    }
    a.bias_bf16 = bias_dtype == PIKV_BF16;
    a.M = M; a.N = N; a.K = K; a.R = R;
    a.tiles = ceil_div(M, LR_BM);
    a.items = 2 * a.tiles;
    const int stage = LP_TILE + R * LR_BK * 2, npad = ceil_div(N, LP_CHUNK) * LP_CHUNK;
    const size_t fixed = 2 * LP_TILE + LP_BUF * LP_W2_TILE + 16 * LP_STAGE_OUT + sizeof(float) * (2 * npad + 128) +
                         (2 * 8 + 8 + 4 * LP_BUF) * sizeof(uint64_t) + 16 + 1024;
    a.stages = (int)min((size_t)8, ((size_t)227 * 1024 - fixed) / stage);
    PIKV_REQUIRE(a.stages >= 2, PIKV_EUNSUPPORTED, "lowrank_pair: not enough shared memory for N=%d", N);
    if (!allow_smem<lowrank_pair_kernel>()) return check_launch("lowrank_pair smem attribute");
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = min(a.items, sm_count());
    cfg.blockDim = LP_THREADS;
    cfg.dynamicSmemBytes = (size_t)a.stages * stage + fixed;
    cfg.stream = static_cast<cudaStream_t>(stream);
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, lowrank_pair_kernel, tm, a);
    count_launch(1);
    return check_launch("lowrank_pair_kernel");
}
