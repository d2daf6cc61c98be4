// The whole gate net of the router on tcgen05 tensor cores:
//   logits[T,E] = relu(x[T,K] . w1[H,K]^T + b1) . w2[E,H]^T + b2      (core/single/pikv_routing.py:34-38)
// followed by the per-token tail of the gate (softmax, top-k, renormalisation, ranks).  The hidden activations [T,H]
// never exist in HBM.
//
//   gate_mlp_kernel      persistent CTA pairs (cta_group::2), an item is 256 tokens times a block of bn hidden units:
//     warp 0     TMA: this CTA's [128 x 64] tile of x and its half, [bn/2 x 64], of the tile of w1, through a ring; the
//                pair's tiles count on the even CTA's barrier
//     warp 1     (even CTA) tcgen05.mma M=256 N=bn over both CTAs' shared memory into one of two accumulators, 128
//                token rows of it in each CTA's tensor memory
//     warps 2-9  drain the previous item (two warps per 32 rows, half the columns each): + b1, ReLU, round to bf16, and
//                the second product of the block's units in registers (packed fp32 FMAs, w2's block in shared memory);
//                the block's partial logits go to the workspace
//     warp 10    writes zeros over the caller's dense dispatch / combine tensors with bulk stores, while the tensor
//                cores run and HBM has nothing else to do
//   gate_cluster_kernel, or for long batches gate_partial_kernel and gate_finalize_kernel (gate.cu): sums a token's
//                        partial logits in block order, adds b2, runs the tail
//
// Bound by the tensor cores and by what L2 delivers to an SM: a pair shares each operand tile, 32 KB per SM for
// 128 x 256 x 64 multiply-adds.  bn is 256, or narrower while that leaves pairs without an item.
// 4096 -> 4096 -> 8: 2048 tokens 632 us with one CTA per 128 tokens walking all hidden units (16 CTAs), 52 us now = 1.32
// PFLOP/s; 16384 tokens 783 us, now 442 us with the tail in a short burst = 1.25 PFLOP/s and 546 us back to back for seconds
// under the power cap.  The library is ahead there: its GEMM with bias and ReLU in the epilogue and the gate behind it take 382
// and 442 us (with a separate ReLU 413 and 484).
// Of the 52, 13 us came from keeping the operands of the issuing instructions warp-uniform (lr_elect).
// Every mbarrier wait is bounded; on a timeout the CTA raises the gate's sticky error word and drains.
#include "gate_common.cuh"
#include "tc_common.cuh"

namespace pikv {

constexpr int GM_THREADS = 352;
constexpr int GM_EPI_WARPS = 8;
constexpr int GM_MAX_BN = 256;
constexpr int GM_ZERO_BYTES = 16 * 1024;

__device__ unsigned g_gate_mlp_error = 0;   // sticky: a bounded wait of gate_mlp_kernel ran out

struct GateMlpArgs {
    const __nv_bfloat16* w2;   // [E,H]
    const void* b1;            // [H] or null
    float* part;               // [groups][T][E] partial logits
    unsigned char* zero[2];    // regions to fill with zeros (16-byte aligned), or null
    size_t zero_bytes;         // of each, a multiple of 16
    int b1_bf16, T, H, K, E, bn, stages, mtiles, groups, per_group, items;
};

__device__ __forceinline__ void gm_epi_barrier() { asm volatile("bar.sync 1, 256;" ::: "memory"); }
__device__ __forceinline__ uint32_t gm_cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void gm_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// the same shared-memory address in the even CTA of the pair
__device__ __forceinline__ uint32_t gm_even(uint32_t addr) { return addr & 0xFEFFFFFFu; }
__device__ __forceinline__ void gm_tma_load(uint32_t dst, const CUtensorMap* tm, int c0, int c1, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
        ::"r"(dst), "l"(tm), "r"(c0), "r"(c1), "r"(bar) : "memory");
}
__device__ __forceinline__ void gm_mma(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accum) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accum) : "memory");
}
// arrives on the barrier at this offset in both CTAs once the pair's MMAs so far are done
__device__ __forceinline__ void gm_commit_both(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                 ::"r"(bar), "h"((uint16_t)3) : "memory");
}
__device__ __forceinline__ void gm_arrive_even(uint32_t bar) {
    asm volatile("{\n\t.reg .b32 a;\n\tmapa.shared::cluster.u32 a, %0, 0;\n\tmbarrier.arrive.release.cluster.shared::cluster.b64 _, [a];\n\t}"
                 ::"r"(bar) : "memory");
}
// a wait on a barrier that the other CTA arrives on
__device__ __forceinline__ bool gm_wait_cluster(uint32_t bar, uint32_t parity) {
    for (unsigned i = 0; i < LR_WAIT_LIMIT; ++i) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
        if (ok) return true;
    }
    return false;
}
// (a0, a1) += (x, x) * (w0, w1), each product rounded into its sum once
__device__ __forceinline__ void gm_fma2(unsigned long long& a, unsigned long long x2, unsigned long long w2) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(a) : "l"(x2), "l"(w2));
}
__device__ __forceinline__ unsigned long long gm_pack2(float lo, float hi) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}

// EC: experts padded to 8, 16, 32 or 64
template <int EC>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(GM_THREADS, 1)
gate_mlp_kernel(const __grid_constant__ CUtensorMap tm_x, const __grid_constant__ CUtensorMap tm_w1, GateMlpArgs a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    unsigned char* smem = smem_raw + ((1024u - (lr_smem_u32(smem_raw) & 1023u)) & 1023u);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = gm_cluster_rank();
    const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
    constexpr int STAGE_A = LR_BM * LR_BK * 2;
    const int stage_bytes = STAGE_A + a.bn / 2 * LR_BK * 2;
    unsigned char* zero_s = smem + (size_t)a.stages * stage_bytes;             // zeros for the bulk fill
    float* w2_s = reinterpret_cast<float*>(zero_s + (a.zero[0] ? GM_ZERO_BYTES : 0));   // [bn][EC]
    float* b1_s = w2_s + a.bn * EC;                                            // [bn]
    float* xch = b1_s + a.bn;                                                  // [EC][128]
    uint64_t* bars = reinterpret_cast<uint64_t*>(xch + EC * 128);
    const uint32_t full0 = lr_smem_u32(bars), empty0 = full0 + 8 * a.stages;
    const uint32_t tfull0 = empty0 + 8 * a.stages, tempty0 = tfull0 + 16;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * a.stages + 4);
    const uint32_t ring = lr_smem_u32(smem);
    const int num_kb = (a.K + LR_BK - 1) / LR_BK;

    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (threadIdx.x == 0) {
        for (int s = 0; s < a.stages; ++s) {
            lr_mbar_init(full0 + 8 * s, 1);
            lr_mbar_init(empty0 + 8 * s, 1);
        }
        for (int s = 0; s < 2; ++s) {
            lr_mbar_init(tfull0 + 8 * s, 1);
            lr_mbar_init(tempty0 + 8 * s, 2 * GM_EPI_WARPS);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        lr_prefetch_tmap(&tm_x);
        lr_prefetch_tmap(&tm_w1);
    }
    if (a.zero[0])
        for (int i = threadIdx.x; i < GM_ZERO_BYTES / 16; i += GM_THREADS) reinterpret_cast<uint4*>(zero_s)[i] = make_uint4(0, 0, 0, 0);
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(lr_smem_u32(tmem_slot)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");          // the zeros are for bulk stores to read
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    gm_cluster_sync();                                                    // the pair's barriers exist
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const uint32_t tmem = *tmem_slot;
    bool failed = false;

    if (warp == 0) {
        LrRing r;
        for (int item = pair; item < a.items && !failed; item += pairs) {
            const int m0 = item % a.mtiles * 2 * LR_BM + (int)rank * LR_BM;
            for (int j = 0; j < a.per_group && !failed; ++j) {
                const int n0 = (item / a.mtiles * a.per_group + j) * a.bn + (int)rank * (a.bn / 2);
                for (int kb = 0; kb < num_kb; ++kb, r.next(a.stages)) {
                    if (!gm_wait_cluster(empty0 + 8 * r.s, r.ph ^ 1u)) { failed = true; break; }
                    if (lr_elect()) {
                        if (rank == 0) lr_mbar_expect_tx(full0 + 8 * r.s, 2u * (uint32_t)stage_bytes);
                        const uint32_t dst = ring + (uint32_t)(r.s * stage_bytes), bar = gm_even(full0 + 8 * r.s);
                        gm_tma_load(dst, &tm_x, kb * LR_BK, m0, bar);
                        gm_tma_load(dst + STAGE_A, &tm_w1, kb * LR_BK, n0, bar);
                    }
                    __syncwarp();
                }
            }
        }
    } else if (warp == 1) {
        if (rank == 0) {
            // D fp32, A and B bf16 K-major, M = 256 over the pair, N = bn
            const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(a.bn >> 3) << 17) | (16u << 24);
            const uint32_t a_lo = lr_desc_lo(ring), b_lo = lr_desc_lo(ring + STAGE_A), stage_lo = (uint32_t)stage_bytes >> 4;
            LrRing r;
            int n = 0;
            for (int item = pair; item < a.items && !failed; item += pairs) {
                for (int j = 0; j < a.per_group && !failed; ++j, ++n) {
                    const int slot = n & 1;
                    if (!gm_wait_cluster(tempty0 + 8 * slot, (((uint32_t)n >> 1) & 1u) ^ 1u)) { failed = true; break; }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t d = tmem + (uint32_t)(slot * GM_MAX_BN);
                    for (int kb = 0; kb < num_kb; ++kb, r.next(a.stages)) {
                        if (!gm_wait_cluster(full0 + 8 * r.s, r.ph)) { failed = true; break; }
                        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                        if (lr_elect()) {
                            const uint32_t off = (uint32_t)r.s * stage_lo;
#pragma unroll
                            for (int k = 0; k < LR_BK / 16; ++k)
                                gm_mma(d, lr_desc(a_lo + off + 2 * k), lr_desc(b_lo + off + 2 * k), idesc, (kb | k) ? 1u : 0u);
                            gm_commit_both(empty0 + 8 * r.s);
                        }
                        __syncwarp();
                    }
                    if (lr_elect()) gm_commit_both(tfull0 + 8 * slot);
                    __syncwarp();
                }
            }
        }
    } else if (warp < 10) {
        const int et = threadIdx.x - 64, half = (warp - 2) >> 2, lg = warp & 3, row = lg * 32 + lane;
        const int cols = a.bn / 2;                        // this warp's columns of the block
        int n = 0;
        for (int item = pair; item < a.items; item += pairs) {
            const int t = item % a.mtiles * 2 * LR_BM + (int)rank * LR_BM + row;
            const int group = item / a.mtiles;
            unsigned long long acc[EC / 2];
#pragma unroll
            for (int e = 0; e < EC / 2; ++e) acc[e] = 0ull;
            for (int j = 0; j < a.per_group; ++j, ++n) {
                const int slot = n & 1, n0 = (group * a.per_group + j) * a.bn;
                gm_epi_barrier();                         // everyone is done with the previous block's weights
                for (int i = et; i < a.bn * EC; i += 32 * GM_EPI_WARPS) {
                    const int e = i / a.bn, c = i % a.bn;
                    w2_s[c * EC + e] = e < a.E && n0 + c < a.H ? __bfloat162float(a.w2[(size_t)e * a.H + n0 + c]) : 0.f;
                }
                for (int c = et; c < a.bn; c += 32 * GM_EPI_WARPS) {
                    float b = 0.f;
                    if (a.b1 && n0 + c < a.H)
                        b = a.b1_bf16 ? __bfloat162float(static_cast<const __nv_bfloat16*>(a.b1)[n0 + c]) : static_cast<const float*>(a.b1)[n0 + c];
                    b1_s[c] = b;
                }
                gm_epi_barrier();
                if (!failed && !gm_wait_cluster(tfull0 + 8 * slot, ((uint32_t)n >> 1) & 1u)) failed = true;
                failed = __any_sync(0xffffffffu, failed);
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                for (int c = half * cols; c < (half + 1) * cols; c += 32) {
                    float v[32];
                    lr_tmem_ld32(tmem + ((uint32_t)(lg * 32) << 16) + (uint32_t)(slot * GM_MAX_BN + c), v);
#pragma unroll
                    for (int i = 0; i < 32; i += 4) {
                        const float4 b = *reinterpret_cast<const float4*>(b1_s + c + i);
                        const float bb[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            const float h = __bfloat162float(__float2bfloat16_rn(fmaxf(v[i + u] + bb[u], 0.f)));
                            const unsigned long long h2 = gm_pack2(h, h);
                            const ulonglong2* w = reinterpret_cast<const ulonglong2*>(w2_s + (size_t)(c + i + u) * EC);
#pragma unroll
                            for (int e = 0; e < EC / 4; ++e) {
                                const ulonglong2 ww = w[e];
                                gm_fma2(acc[2 * e], h2, ww.x);
                                gm_fma2(acc[2 * e + 1], h2, ww.y);
                            }
                        }
                    }
                }
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) gm_arrive_even(tempty0 + 8 * slot);
            }
            // the two column halves of a row meet in shared memory
            float l[EC];
#pragma unroll
            for (int e = 0; e < EC / 2; ++e) asm("mov.b64 {%0, %1}, %2;" : "=f"(l[2 * e]), "=f"(l[2 * e + 1]) : "l"(acc[e]));
            if (half == 1) {
#pragma unroll
                for (int e = 0; e < EC; ++e) xch[e * 128 + row] = l[e];
            }
            gm_epi_barrier();
            if (half == 0 && t < a.T) {
                float* dst = a.part + ((size_t)group * a.T + t) * a.E;
#pragma unroll
                for (int e = 0; e < EC; ++e) l[e] += xch[e * 128 + row];
                if (a.E == EC) {
#pragma unroll
                    for (int e = 0; e < EC; e += 4) *reinterpret_cast<float4*>(dst + e) = make_float4(l[e], l[e + 1], l[e + 2], l[e + 3]);
                } else {
#pragma unroll
                    for (int e = 0; e < EC; ++e)
                        if (e < a.E) dst[e] = l[e];
                }
            }
        }
    } else if (a.zero[0] && lane == 0) {
        const uint32_t src = lr_smem_u32(zero_s);
        const size_t per = (a.zero_bytes + GM_ZERO_BYTES - 1) / GM_ZERO_BYTES;
        for (size_t i = blockIdx.x; i < 2 * per; i += gridDim.x) {
            unsigned char* dst = a.zero[i / per];
            const size_t at = i % per * GM_ZERO_BYTES;
            const uint32_t bytes = (uint32_t)min((size_t)GM_ZERO_BYTES, a.zero_bytes - at);
            asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst + at), "r"(src), "r"(bytes) : "memory");
            asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        }
        asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    }
    if (failed) atomicOr(&g_gate_mlp_error, 1u);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    gm_cluster_sync();                                    // nobody reads the other CTA's shared memory any more
    if (warp == 1) {
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
    }
}

template <int EC>
static int launch_gate_mlp(GateMlpArgs& a, const void* x, const void* w1, cudaStream_t st) {
    CUtensorMap tm_x, tm_w1;
    int rc = make_tmap(&tm_x, x, a.T, a.K, LR_BM);
    if (rc != PIKV_OK) return rc;
    rc = make_tmap(&tm_w1, w1, a.H, a.K, a.bn / 2);
    if (rc != PIKV_OK) return rc;
    const int stage = LR_BM * LR_BK * 2 + a.bn / 2 * LR_BK * 2;
    const size_t fixed = (a.zero[0] ? GM_ZERO_BYTES : 0) + sizeof(float) * ((size_t)a.bn * EC + a.bn + EC * 128) +
                         (2 * 8 + 4) * sizeof(uint64_t) + 16 + 1024;
    a.stages = (int)min((size_t)8, ((size_t)227 * 1024 - fixed) / stage);
    PIKV_REQUIRE(a.stages >= 2, PIKV_EUNSUPPORTED, "gate_mlp: not enough shared memory for E=%d", a.E);
    if (!allow_smem<gate_mlp_kernel<EC>>()) return check_launch("gate_mlp smem attribute");
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = 2 * min(a.items, sm_count() / 2);
    cfg.blockDim = GM_THREADS;
    cfg.dynamicSmemBytes = (size_t)a.stages * stage + fixed;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, gate_mlp_kernel<EC>, tm_x, tm_w1, a);
    count_launch(1);
    return check_launch("gate_mlp_kernel");
}

// reads and clears this kernel's sticky error word (called by pikv_gate_error_state)
int gate_mlp_error_fetch() {
    unsigned v = 0, zero = 0;
    if (cudaMemcpyFromSymbol(&v, g_gate_mlp_error, sizeof(v)) != cudaSuccess) return -1;
    if (v) cudaMemcpyToSymbol(g_gate_mlp_error, &zero, sizeof(zero));
    return (int)v;
}

}  // namespace pikv

using namespace pikv;

extern "C" int pikv_gate_mlp_fused(const pikv_gate_params* p, const void* x, int32_t K, const void* w1, const float* b1,
                                   pikv_stream_t stream) {
    return pikv_gate_mlp_dense(p, x, K, w1, b1, p ? p->b2 : nullptr, PIKV_F32, nullptr, stream);
}

extern "C" int pikv_gate_mlp_dense(const pikv_gate_params* p, const void* x, int32_t K, const void* w1, const void* b1,
                                   const void* b2, int32_t bias_dtype, const pikv_dense_out* dense, pikv_stream_t stream) {
    PIKV_REQUIRE(p != nullptr && x != nullptr && w1 != nullptr, PIKV_EINVAL, "gate_mlp: null pointer");
    PIKV_REQUIRE(p->dtype == PIKV_BF16, PIKV_EUNSUPPORTED, "gate_mlp: bf16 inputs and weights only");
    PIKV_REQUIRE(p->w2 != nullptr && p->H > 0 && K > 0, PIKV_EINVAL, "gate_mlp: the second layer (w2, H) and K are required");
    PIKV_REQUIRE(K % 8 == 0 && p->H % 8 == 0, PIKV_EUNSUPPORTED, "gate_mlp: K=%d and H=%d must be multiples of 8", K, p->H);
    PIKV_REQUIRE(((uintptr_t)x % 16) == 0 && ((uintptr_t)w1 % 16) == 0 && ((uintptr_t)p->w2 % 16) == 0, PIKV_EINVAL,
                 "gate_mlp: x, w1 and w2 must be 16-byte aligned");
    PIKV_REQUIRE(p->phase == PIKV_GATE_WHOLE, PIKV_EINVAL, "gate_mlp: phase must be PIKV_GATE_WHOLE");
    PIKV_REQUIRE(p->T <= LR_BM * GATE_MAX_CTAS, PIKV_ELIMIT, "gate_mlp: at most %d tokens per call", LR_BM * GATE_MAX_CTAS);
    PIKV_REQUIRE(bias_dtype == PIKV_BF16 || bias_dtype == PIKV_F32, PIKV_EINVAL, "gate_mlp: bad bias dtype");
    size_t zero_bytes = 0;
    if (dense) {
        PIKV_REQUIRE(dense->dispatch && dense->combine && dense->capacity > 0 && p->topk_w && p->slot && p->counts_k && p->prob_sum, PIKV_EINVAL,
                     "gate_mlp: the dense outputs need their tensors, a capacity and all routing outputs");
        PIKV_REQUIRE(dense->balance >= 0 && dense->balance <= 3, PIKV_EINVAL, "gate_mlp: bad balance term %d", dense->balance);
        zero_bytes = (size_t)p->T * p->E * dense->capacity * sizeof(float);
        PIKV_REQUIRE((((uintptr_t)dense->dispatch | (uintptr_t)dense->combine | zero_bytes) & 15) == 0, PIKV_EINVAL,
                     "gate_mlp: the dense tensors must be 16-byte aligned and sized");
    }
    // validation, geometry and the workspace layout are the gate's own
    pikv_gate_params q = *p;
    q.act = x;                      // only so that the shared checks see an activation pointer
    q.phase |= PIKV_GATE_FORCE_SIMT;
    GateDev g;
    int rc = gate_run(&q, nullptr, 0, &g);
    if (rc != PIKV_OK) return rc;
    PIKV_REQUIRE(p->workspace_bytes >= pikv_gate_workspace_bytes(p->T, p->E, p->top_k), PIKV_EINVAL, "gate_mlp: workspace too small");
    GateMlpArgs a = {};
    a.w2 = static_cast<const __nv_bfloat16*>(p->w2);
    a.b1 = b1;
    a.b1_bf16 = bias_dtype == PIKV_BF16;
    a.part = gate_partials(g);
    if (dense) {
        a.zero[0] = reinterpret_cast<unsigned char*>(dense->dispatch);
        a.zero[1] = reinterpret_cast<unsigned char*>(dense->combine);
    }
    a.zero_bytes = zero_bytes;
    a.T = p->T; a.H = p->H; a.K = K; a.E = p->E;
    a.mtiles = ceil_div(a.T, 2 * LR_BM);
    a.bn = GM_MAX_BN;
    while (a.bn > 64 && a.mtiles * ceil_div(a.H, a.bn) < sm_count() / 2) a.bn /= 2;
    const int blocks = ceil_div(a.H, a.bn);
    a.per_group = ceil_div(blocks, gate_max_partials(a.T));
    a.groups = ceil_div(blocks, a.per_group);
    a.items = a.mtiles * a.groups;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (a.E <= 8) rc = launch_gate_mlp<8>(a, x, w1, st);
    else if (a.E <= 16) rc = launch_gate_mlp<16>(a, x, w1, st);
    else if (a.E <= 32) rc = launch_gate_mlp<32>(a, x, w1, st);
    else rc = launch_gate_mlp<64>(a, x, w1, st);
    if (rc != PIKV_OK) return rc;
    g.act = nullptr;
    return gate_from_partials(g, a.part, a.groups, b2, a.b1_bf16, dense, st);
}
