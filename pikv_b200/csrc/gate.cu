// Router gate: last-layer logits + softmax + top-k + load-balance counts + slot scan.
//
// Two launches, no atomics on floats, no inter-CTA waiting:
//   gate_*_kernel   each CTA owns a contiguous chunk of tokens; per token it forms the
//                   logits, softmax, top-k and renormalised weights, then ranks its own
//                   (token, k) pairs per expert in order and publishes per-CTA counts;
//   gate_finalize   each CTA turns its local ranks into global slots from the exclusive
//                   prefix of the per-CTA counts; CTA 0 also reduces the totals.
// Results are therefore run-to-run bit-identical.
#include "gate_common.cuh"
#include <stdlib.h>
#include <cooperative_groups.h>

namespace pikv {

// ---- per-CTA ranking of its (token, k) pairs, in order ----------------------------
// sel[0..npairs) holds the expert of every pair of this CTA's chunk.  Writes the local
// rank (number of earlier pairs of the chunk with the same expert) to slot[] and the
// per-CTA counts to the workspace.
template <int EP>
__device__ __forceinline__ void cta_rank_tail(const GateDev& g, const uint8_t* sel, int chunk_start, int ntok,
                                              int* warp_cnt /*[WARPS][EP]*/, int* run /*[EP]*/,
                                              int* cnt_k /*[K][EP]*/) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int npairs = ntok * g.k;
    for (int i = tid; i < EP; i += GATE_THREADS) run[i] = 0;
    for (int i = tid; i < GATE_MAX_K * EP; i += GATE_THREADS) cnt_k[i] = 0;
    __syncthreads();
    for (int base = 0; base < npairs; base += GATE_THREADS) {
        for (int i = tid; i < GATE_WARPS * EP; i += GATE_THREADS) warp_cnt[i] = 0;
        __syncthreads();
        const int p = base + tid;
        const bool valid = p < npairs;
        const int e = valid ? (int)sel[p] : 255;
        const unsigned peers = __match_any_sync(0xffffffffu, e);
        const int rank_in_warp = __popc(peers & ((1u << lane) - 1u));
        if (valid && rank_in_warp == 0) warp_cnt[warp * EP + e] = __popc(peers);
        if (valid) atomicAdd(&cnt_k[(p % g.k) * EP + e], 1);   // integer: order-independent
        __syncthreads();
        if (valid) {
            int r = run[e] + rank_in_warp;
            for (int w = 0; w < warp; ++w) r += warp_cnt[w * EP + e];
            if (g.slot) g.slot[(size_t)chunk_start * g.k + p] = r;
        }
        __syncthreads();
        if (tid < EP) {
            int add = 0;
#pragma unroll
            for (int w = 0; w < GATE_WARPS; ++w) add += warp_cnt[w * EP + tid];
            run[tid] += add;
        }
        __syncthreads();
    }
    const int cta = blockIdx.x;
    for (int e = tid; e < g.E; e += GATE_THREADS) g.cta_cnt[(size_t)cta * g.E + e] = run[e];
    for (int i = tid; i < g.k * g.E; i += GATE_THREADS) {
        int j = i / g.E, e = i % g.E;
        g.cta_cnt_k[((size_t)cta * g.k + j) * g.E + e] = cnt_k[j * EP + e];
    }
}

// ---- gate from activations: SIMT fp32 dot products --------------------------------
// One warp forms the logits of TPW tokens at a time: lanes split the hidden dimension in
// 8-element vectors, every w2 vector is reused for the TPW tokens, partial sums meet in
// an xor butterfly (fixed order), then lane i < TPW runs the tail of token i.
template <typename TIn> struct Vec8;
template <> struct Vec8<__nv_bfloat16> {
    static __device__ __forceinline__ void load(const __nv_bfloat16* p, float (&v)[8]) {
        uint4 r = __ldg(reinterpret_cast<const uint4*>(p));
        bf16x2_to_f32(r.x, v[0], v[1]);
        bf16x2_to_f32(r.y, v[2], v[3]);
        bf16x2_to_f32(r.z, v[4], v[5]);
        bf16x2_to_f32(r.w, v[6], v[7]);
    }
};
template <> struct Vec8<float> {
    static __device__ __forceinline__ void load(const float* p, float (&v)[8]) {
        float4 a = __ldg(reinterpret_cast<const float4*>(p));
        float4 b = __ldg(reinterpret_cast<const float4*>(p) + 1);
        v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
        v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
    }
};

template <typename TIn, int EP, int TPW>
__global__ void __launch_bounds__(GATE_THREADS) gate_act_kernel(GateDev g) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    int* warp_cnt = reinterpret_cast<int*>(smem_raw);                 // [WARPS][EP]
    int* run = warp_cnt + GATE_WARPS * EP;                            // [EP]
    int* cnt_k = run + EP;                                            // [K][EP]
    float* psum_rows = reinterpret_cast<float*>(cnt_k + GATE_MAX_K * EP);  // [WARPS][TPW][EP]
    uint8_t* sel = reinterpret_cast<uint8_t*>(psum_rows + GATE_WARPS * TPW * EP);  // [chunk*k]

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int chunk_start = blockIdx.x * g.chunk;
    const int ntok = min(g.chunk, g.T - chunk_start);
    const TIn* act = static_cast<const TIn*>(g.act);
    const TIn* w2 = static_cast<const TIn*>(g.w2);
    const int H = g.H, E = g.E;

    for (int i = tid; i < GATE_WARPS * TPW * EP; i += GATE_THREADS) psum_rows[i] = 0.f;
    __syncthreads();

    for (int tile = warp * TPW; tile < ntok; tile += GATE_WARPS * TPW) {
        float acc[TPW][EP];
#pragma unroll
        for (int i = 0; i < TPW; ++i)
#pragma unroll
            for (int e = 0; e < EP; ++e) acc[i][e] = 0.f;
        const TIn* rows[TPW];
        bool ok[TPW];
#pragma unroll
        for (int i = 0; i < TPW; ++i) {
            ok[i] = (tile + i) < ntok;
            rows[i] = act + (size_t)(chunk_start + (ok[i] ? tile + i : tile)) * H;
        }
        for (int c = lane * 8; c < H; c += 32 * 8) {
            float a[TPW][8];
#pragma unroll
            for (int i = 0; i < TPW; ++i) Vec8<TIn>::load(rows[i] + c, a[i]);
#pragma unroll
            for (int e = 0; e < EP; ++e) {
                if (e < E) {
                    float w[8];
                    Vec8<TIn>::load(w2 + (size_t)e * H + c, w);
#pragma unroll
                    for (int i = 0; i < TPW; ++i)
#pragma unroll
                        for (int j = 0; j < 8; ++j) acc[i][e] = fmaf(a[i][j], w[j], acc[i][e]);
                }
            }
        }
#pragma unroll
        for (int i = 0; i < TPW; ++i)
#pragma unroll
            for (int e = 0; e < EP; ++e) acc[i][e] = warp_sum(acc[i][e]);
        float l[EP];
#pragma unroll
        for (int e = 0; e < EP; ++e) {
            l[e] = 0.f;
#pragma unroll
            for (int i = 0; i < TPW; ++i)
                if (lane == i) l[e] = acc[i][e];
            if (g.b2 && e < E) l[e] += g.b2[e];
        }
        if (lane < TPW && (tile + lane) < ntok) {
            token_tail<EP>(l, g, chunk_start + tile + lane, sel + (size_t)(tile + lane) * g.k);
            float* row = psum_rows + (warp * TPW + lane) * EP;
#pragma unroll
            for (int e = 0; e < EP; ++e) row[e] += l[e];
        }
    }
    __syncthreads();
    if (tid < E) {
        float s = 0.f;
        for (int r = 0; r < GATE_WARPS * TPW; ++r) s += psum_rows[r * EP + tid];
        g.cta_psum[(size_t)blockIdx.x * E + tid] = s;
    }
    cta_rank_tail<EP>(g, sel, chunk_start, ntok, warp_cnt, run, cnt_k);
}

// ---- gate from precomputed logits: one thread per token ---------------------------
template <int EP>
__device__ __forceinline__ void gate_logits_tokens(const GateDev& g) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    int* warp_cnt = reinterpret_cast<int*>(smem_raw);
    int* run = warp_cnt + GATE_WARPS * EP;
    int* cnt_k = run + EP;
    float* psum_w = reinterpret_cast<float*>(cnt_k + GATE_MAX_K * EP);   // [WARPS][EP]
    uint8_t* sel = reinterpret_cast<uint8_t*>(psum_w + GATE_WARPS * EP);

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int chunk_start = blockIdx.x * g.chunk;
    const int ntok = min(g.chunk, g.T - chunk_start);
    const int E = g.E;
    for (int i = tid; i < GATE_WARPS * EP; i += GATE_THREADS) psum_w[i] = 0.f;
    __syncthreads();
    for (int base = 0; base < ntok; base += GATE_THREADS) {
        const int lt = base + tid;
        float l[EP];
        const bool valid = lt < ntok;
#pragma unroll
        for (int e = 0; e < EP; ++e)
            l[e] = (valid && e < E) ? g.logits_in[(size_t)(chunk_start + lt) * E + e] : 0.f;
        if (valid) token_tail<EP>(l, g, chunk_start + lt, sel + (size_t)lt * g.k);
#pragma unroll
        for (int e = 0; e < EP; ++e) {
            float s = warp_sum(valid ? l[e] : 0.f);
            if (lane == 0 && e < E) psum_w[warp * EP + e] += s;
        }
    }
    __syncthreads();
    if (tid < E) {
        float s = 0.f;
        for (int w = 0; w < GATE_WARPS; ++w) s += psum_w[w * EP + tid];
        g.cta_psum[(size_t)blockIdx.x * E + tid] = s;
    }
    cta_rank_tail<EP>(g, sel, chunk_start, ntok, warp_cnt, run, cnt_k);
}

// sum of p[c * stride] for c = first, first + step, ... < end, eight loads in flight per round trip and
// added in index order (with 64 experts a thread walks a quarter of the CTAs)
template <typename V>
__device__ __forceinline__ V strided_sum(const V* p, size_t stride, int first, int end, int step) {
    V s = V(0);
    int c = first;
    for (; c + 7 * step < end; c += 8 * step) {
        V v[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) v[u] = __ldg(p + (size_t)(c + u * step) * stride);
#pragma unroll
        for (int u = 0; u < 8; ++u) s += v[u];
    }
    for (; c < end; c += step) s += __ldg(p + (size_t)c * stride);
    return s;
}

// ---- gate from the partial logits of gate_mlp.cu ------------------------------------
// A CTA's tokens are a contiguous piece of every [T][E] block, so all threads sum it over the blocks (in block order,
// eight loads in flight) into shared memory; then one thread per token runs the tail.
constexpr int GP_TOKENS = 128;         // tokens per pass
template <int EP>
__global__ void __launch_bounds__(GATE_THREADS) gate_partial_kernel(GateDev g, const float* part, int groups, const void* b2, bool b2_bf16) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    int* warp_cnt = reinterpret_cast<int*>(smem_raw);
    int* run = warp_cnt + GATE_WARPS * EP;
    int* cnt_k = run + EP;
    float* psum_w = reinterpret_cast<float*>(cnt_k + GATE_MAX_K * EP);   // [WARPS][EP]
    float* logit = psum_w + GATE_WARPS * EP;                             // [GP_TOKENS][E + 1]
    uint8_t* sel = reinterpret_cast<uint8_t*>(logit + GP_TOKENS * (EP + 1));

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int chunk_start = blockIdx.x * g.chunk;
    const int ntok = min(g.chunk, g.T - chunk_start);
    const int E = g.E;
    const size_t block = (size_t)g.T * E;
    for (int i = tid; i < GATE_WARPS * EP; i += GATE_THREADS) psum_w[i] = 0.f;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    for (int base = 0; base < ntok; base += GP_TOKENS) {
        const int n = min(GP_TOKENS, ntok - base);
        __syncthreads();
        for (int i = tid; i < n * E; i += GATE_THREADS) {
            const float* p = part + (size_t)(chunk_start + base) * E + i;
            const int e = i % E;
            float s = 0.f;
            int q = 0;
            for (; q + 8 <= groups; q += 8) {
                float v[8];
#pragma unroll
                for (int u = 0; u < 8; ++u) v[u] = __ldg(p + (q + u) * block);
#pragma unroll
                for (int u = 0; u < 8; ++u) s += v[u];
            }
            for (; q < groups; ++q) s += __ldg(p + q * block);
            if (b2) s += b2_bf16 ? __bfloat162float(static_cast<const __nv_bfloat16*>(b2)[e]) : static_cast<const float*>(b2)[e];
            logit[i / E * (EP + 1) + e] = s;
        }
        __syncthreads();
        if (warp < GP_TOKENS / 32) {
            float l[EP];
            const bool valid = tid < n;
#pragma unroll
            for (int e = 0; e < EP; ++e) l[e] = valid && e < E ? logit[tid * (EP + 1) + e] : 0.f;
            if (valid) token_tail<EP>(l, g, chunk_start + base + tid, sel + (size_t)(base + tid) * g.k);
#pragma unroll
            for (int e = 0; e < EP; ++e) {
                const float s = warp_sum(valid ? l[e] : 0.f);
                if (lane == 0 && e < E) psum_w[warp * EP + e] += s;
            }
        }
    }
    __syncthreads();
    if (tid < E) {
        float s = 0.f;
        for (int w = 0; w < GATE_WARPS; ++w) s += psum_w[w * EP + tid];
        g.cta_psum[(size_t)blockIdx.x * E + tid] = s;
    }
    cta_rank_tail<EP>(g, sel, chunk_start, ntok, warp_cnt, run, cnt_k);
}

// the router's auxiliary loss from the probability sums, by one warp (E <= 64: two experts per lane)
__device__ __forceinline__ void router_aux_loss(const float* prob_sum, int T, int E, int balance, float coefficient, float* aux) {
    const int lane = threadIdx.x & 31;
    float p[2], base = 0.f, ent = 0.f, sum = 0.f, l2 = 0.f;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int e = lane + 32 * i;
        p[i] = e < E ? prob_sum[e] / (float)T : 0.f;
        if (e < E) {
            base += p[i] * logf(p[i] * (float)E + 1e-9f);
            ent += p[i] * logf(p[i] + 1e-9f);
            sum += p[i];
            const float d = p[i] - 1.0f / (float)E;
            l2 += d * d;
        }
    }
    base = warp_sum(base);
    const float mean = warp_sum(sum) / (float)E;
    float var = 0.f;
#pragma unroll
    for (int i = 0; i < 2; ++i)
        if (lane + 32 * i < E) var += (p[i] - mean) * (p[i] - mean);
    var = warp_sum(var);
    ent = warp_sum(ent);
    l2 = warp_sum(l2);
    if (lane == 0) {
        float term = 0.f;
        if (balance == 1) term = ent / logf((float)E);                                     // minus the normalised entropy
        else if (balance == 2) term = sqrtf(var / (float)(E - 1)) / (mean + 1e-9f);
        else if (balance == 3) term = l2;
        *aux = base + (balance ? coefficient * term : 0.f);
    }
}

// core/single/pikv_routing.py:107-128: the position in pass j is the number of earlier passes in which this expert
// received at least one token
__device__ __forceinline__ int dense_position(const int* counts_k, int E, int e, int j) {
    int pos = 0;
    for (int i = 0; i < j; ++i) pos += counts_k[i * E + e] > 0 ? 1 : 0;
    return pos;
}
__device__ __forceinline__ void dense_store(const pikv_dense_out& d, int t, int e, int E, int pos, float w) {
    if (pos < 0 || pos >= d.capacity) return;
    const size_t o = ((size_t)t * E + e) * d.capacity + pos;
    d.dispatch[o] = 1.0f;
    d.combine[o] = w;
}

// ---- the whole tail of a short batch in one cluster ---------------------------------
// Up to GC_MAX_TOKENS tokens are cut over the CTAs of one cluster, which exchange their counters through distributed
// shared memory: logits (summed over `groups` blocks of partial logits), softmax, top-k, slots, totals and dense outputs
// in one launch.  Bound by latency: 64 tokens of a 4096-wide net, 64 blocks, took 26 us as three launches
// (gate_partial_kernel, gate_finalize_kernel, dispatch_scatter_kernel), each a chain of dependent loads; this kernel
// takes 13 us by itself with cold caches (2048 tokens: 16 us), in a router call of 26 us (71 us).
// W floats at a 4-byte boundary (rows of EP + 1 floats)
template <int W> struct GatePiece { float v[W]; };
__device__ __forceinline__ void add_to(float& a, float b) { a += b; }
__device__ __forceinline__ void add_to(float4& a, const float4& b) { a.x += b.x; a.y += b.y; a.z += b.z; a.w += b.w; }
// logit[token][expert] = sum over the blocks, for the n tokens from element `first` of every block on; V holds 1 or 4
// experts.  sub: GATE_THREADS values of V for the partial sums of a split.
template <int EP, typename V>
__device__ __forceinline__ void gate_block_sums(const float* part, int groups, size_t block, int first, int n, int E, float* logit, V* sub) {
    constexpr int W = sizeof(V) / 4;
    const int tid = threadIdx.x, cnt = n * E / W;
    int split = 1;
    while (split < 16 && 2 * split * cnt <= GATE_THREADS && 4 * split <= groups) split *= 2;
    const int per = (groups + split - 1) / split;
    for (int i0 = tid; i0 < split * cnt; i0 += GATE_THREADS) {
        const int i = i0 % cnt, q0 = i0 / cnt * per, q1 = min(groups, q0 + per);
        const float* p = part + first + (size_t)i * W;
        V s = {};
        int q = q0;
        for (; q + 8 <= q1; q += 8) {
            V v[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) v[u] = __ldg(reinterpret_cast<const V*>(p + (q + u) * block));
#pragma unroll
            for (int u = 0; u < 8; ++u) add_to(s, v[u]);
        }
        for (; q < q1; ++q) add_to(s, __ldg(reinterpret_cast<const V*>(p + q * block)));
        if (split > 1) sub[i0] = s;
        else *reinterpret_cast<GatePiece<W>*>(logit + i * W / E * (EP + 1) + i * W % E) = *reinterpret_cast<GatePiece<W>*>(&s);
    }
    if (split > 1) {
        __syncthreads();
        if (tid < cnt) {
            V s = sub[tid];
            for (int q = 1; q < split; ++q) add_to(s, sub[q * cnt + tid]);
            *reinterpret_cast<GatePiece<W>*>(logit + tid * W / E * (EP + 1) + tid * W % E) = *reinterpret_cast<GatePiece<W>*>(&s);
        }
    }
    __syncthreads();
}

constexpr int GC_CTAS = 8;
constexpr int GC_MAX_TOKENS = GC_CTAS * GATE_THREADS;
template <int EP>
__global__ void __cluster_dims__(GC_CTAS, 1, 1) __launch_bounds__(GATE_THREADS, 1)
gate_cluster_kernel(GateDev g, const float* part, int groups, const void* b2, bool b2_bf16, pikv_dense_out d) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float* logit = reinterpret_cast<float*>(smem_raw);                   // [GATE_THREADS][EP + 1]
    int* rank_s = reinterpret_cast<int*>(logit + GATE_THREADS * (EP + 1));   // [chunk * k], before that the sums of a split
    uint8_t* sel = reinterpret_cast<uint8_t*>(rank_s + GATE_THREADS * max(4, g.k));  // [chunk * k]
    __shared__ int warp_cnt[GATE_WARPS * EP], run[EP], cnt_k[GATE_MAX_K * EP], base_s[EP], tot_k[GATE_MAX_K * EP];
    __shared__ float psum_w[GATE_WARPS * EP], psum[EP], ptot[EP];
    cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, cta = blockIdx.x, E = g.E, k = g.k;
    const int start = cta * g.chunk, n = max(0, min(g.chunk, g.T - start));
    for (int i = tid; i < EP; i += GATE_THREADS) run[i] = 0;
    for (int i = tid; i < GATE_MAX_K * EP; i += GATE_THREADS) cnt_k[i] = 0;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");

    // logits, four experts per load where the rows allow it; few values and many blocks are split over more threads (a
    // fixed cut, added in order)
    if ((E & 3) == 0) gate_block_sums<EP, float4>(part, groups, (size_t)g.T * E, start * E, n, E, logit, reinterpret_cast<float4*>(rank_s));
    else gate_block_sums<EP, float>(part, groups, (size_t)g.T * E, start * E, n, E, logit, reinterpret_cast<float*>(rank_s));
    float l[EP];
#pragma unroll
    for (int e = 0; e < EP; ++e) {
        l[e] = 0.f;
        if (tid < n && e < E) {
            l[e] = logit[tid * (EP + 1) + e];
            if (b2) l[e] += b2_bf16 ? __bfloat162float(static_cast<const __nv_bfloat16*>(b2)[e]) : static_cast<const float*>(b2)[e];
        }
    }
    if (tid < n) token_tail<EP>(l, g, start + tid, sel + tid * k);
#pragma unroll
    for (int e = 0; e < EP; ++e) {
        const float s = warp_sum(tid < n && e < E ? l[e] : 0.f);
        if (lane == 0) psum_w[warp * EP + e] = s;
    }
    __syncthreads();
    if (tid < EP) {
        float s = 0.f;
        for (int w = 0; w < GATE_WARPS; ++w) s += psum_w[w * EP + tid];
        psum[tid] = s;
    }
    // ranks of the CTA's (token, k) pairs per expert, in order
    for (int base = 0; base < n * k; base += GATE_THREADS) {
        for (int i = tid; i < GATE_WARPS * EP; i += GATE_THREADS) warp_cnt[i] = 0;
        __syncthreads();
        const int p = base + tid;
        const bool valid = p < n * k;
        const int e = valid ? (int)sel[p] : 255;
        const unsigned peers = __match_any_sync(0xffffffffu, e);
        const int in_warp = __popc(peers & ((1u << lane) - 1u));
        if (valid && in_warp == 0) warp_cnt[warp * EP + e] = __popc(peers);
        if (valid) atomicAdd(&cnt_k[(p % k) * EP + e], 1);
        __syncthreads();
        if (valid) {
            int r = run[e] + in_warp;
            for (int w = 0; w < warp; ++w) r += warp_cnt[w * EP + e];
            rank_s[p] = r;
        }
        __syncthreads();
        if (tid < EP) {
            int add = 0;
#pragma unroll
            for (int w = 0; w < GATE_WARPS; ++w) add += warp_cnt[w * EP + tid];
            run[tid] += add;
        }
        __syncthreads();
    }
    cluster.sync();
    for (int i = tid; i < (k + 2) * E; i += GATE_THREADS) {
        const int j = i / E, e = i % E;
        if (j < k) {
            int s = 0;
#pragma unroll
            for (int r = 0; r < GC_CTAS; ++r) s += *cluster.map_shared_rank(&cnt_k[j * EP + e], r);
            tot_k[j * EP + e] = s;
        } else if (j == k) {
            int s = g.slot_base ? g.slot_base[e] : 0;
#pragma unroll
            for (int r = 0; r < GC_CTAS; ++r) {
                const int c = *cluster.map_shared_rank(&run[e], r);
                s += r < cta ? c : 0;
            }
            base_s[e] = s;
        } else if (cta == 0) {
            float s = 0.f;
#pragma unroll
            for (int r = 0; r < GC_CTAS; ++r) s += *cluster.map_shared_rank(&psum[e], r);
            ptot[e] = s;
        }
    }
    __syncthreads();
    for (int p = tid; p < n * k; p += GATE_THREADS) {
        const int e = sel[p], j = p % k, t = start + p / k;
        int s = base_s[e] + rank_s[p];
        if (g.capacity > 0 && s >= g.capacity) s = -1;
        if (g.slot) g.slot[(size_t)start * k + p] = s;
        if (d.dispatch)
            dense_store(d, t, e, E, d.position_mode == 0 ? s : dense_position(tot_k, EP, e, j), g.topk_w[(size_t)start * k + p]);
    }
    if (cta == 0) {
        if (tid < E) {
            int tot = 0;
            for (int j = 0; j < k; ++j) {
                if (g.counts_k) g.counts_k[j * E + tid] = tot_k[j * EP + tid];
                tot += tot_k[j * EP + tid];
            }
            if (g.prob_sum) g.prob_sum[tid] = ptot[tid];
            if (g.new_len) {
                const int len = (g.slot_base ? g.slot_base[tid] : 0) + tot;
                g.new_len[tid] = g.capacity > 0 && len > g.capacity ? g.capacity : len;
            }
        }
        if (d.aux && tid < 32) router_aux_loss(ptot, g.T, E, d.balance, d.coefficient, d.aux);
    }
    cluster.sync();                                   // nobody reads this CTA's counters any more
}
template <int EP>
__global__ void __launch_bounds__(GATE_THREADS) gate_logits_kernel(GateDev g) { gate_logits_tokens<EP>(g); }

// Several gates of one batch: a kernel of a few microseconds each, in one launch (grid y = gate).
struct GateDevs {
    GateDev g[GATE_MAX_BATCH];
};
template <int EP>
__global__ void __launch_bounds__(GATE_THREADS) gate_logits_batch_kernel(const __grid_constant__ GateDevs b) {
    dependency_wait();
    gate_logits_tokens<EP>(b.g[blockIdx.y]);
}

// ---- finalize: local ranks -> global slots; totals --------------------------------
// Threads are laid out as (expert e, part): part p sums the per-CTA counters of CTAs p, p+parts, ...
// so the reads of one prefix are spread over 256/EP2 threads and overlap; parts are combined in a
// fixed order (the float sums stay run-to-run identical).
__device__ __forceinline__ void gate_finalize(const GateDev& g) {
    __shared__ int base_s[GATE_MAX_E];
    __shared__ int part_i[GATE_THREADS];
    __shared__ float part_f[GATE_THREADS];
    const int tid = threadIdx.x, cta = blockIdx.x, E = g.E;
    int ep2 = 8;
    while (ep2 < E) ep2 <<= 1;
    const int parts = GATE_THREADS / ep2;
    const int e = tid & (ep2 - 1), part = tid / ep2;
    asm volatile("griddepcontrol.wait;" ::: "memory");
    {
        part_i[tid] = e < E ? strided_sum(g.cta_cnt + e, (size_t)E, part, cta, parts) : 0;
    }
    __syncthreads();
    if (tid < E) {
        int b = g.slot_base ? g.slot_base[tid] : 0;
        for (int p = 0; p < parts; ++p) b += part_i[p * ep2 + tid];
        base_s[tid] = b;
    }
    __syncthreads();
    const int chunk_start = cta * g.chunk;
    const int ntok = min(g.chunk, g.T - chunk_start);
    if (g.slot) {
        const size_t off = (size_t)chunk_start * g.k;
        for (int p = tid; p < ntok * g.k; p += GATE_THREADS) {
            int ee = g.topk_idx[off + p];
            int s = base_s[ee] + g.slot[off + p];
            g.slot[off + p] = (g.capacity <= 0 || s < g.capacity) ? s : -1;
        }
    }
    if (cta != 0) return;
    // totals over all CTAs: per-column counts, probability sums, new lengths
    int tot = 0;
    for (int j = 0; j < g.k; ++j) {
        const int s = e < E ? strided_sum(g.cta_cnt_k + (size_t)j * E + e, (size_t)g.k * E, part, g.G, parts) : 0;
        __syncthreads();
        part_i[tid] = s;
        __syncthreads();
        if (tid < E) {
            int cnt = 0;
            for (int p = 0; p < parts; ++p) cnt += part_i[p * ep2 + tid];
            if (g.counts_k) g.counts_k[j * E + tid] = cnt;
            tot += cnt;
        }
    }
    part_f[tid] = e < E ? strided_sum(g.cta_psum + e, (size_t)E, part, g.G, parts) : 0.f;
    __syncthreads();
    if (tid < E) {
        float sum = 0.f;
        for (int p = 0; p < parts; ++p) sum += part_f[p * ep2 + tid];
        if (g.prob_sum) g.prob_sum[tid] = sum;
        if (g.new_len) {
            int n = (g.slot_base ? g.slot_base[tid] : 0) + tot;
            g.new_len[tid] = (g.capacity > 0 && n > g.capacity) ? g.capacity : n;
        }
    }
}

__global__ void __launch_bounds__(GATE_THREADS) gate_finalize_kernel(GateDev g) { gate_finalize(g); }
__global__ void __launch_bounds__(GATE_THREADS) gate_finalize_batch_kernel(const __grid_constant__ GateDevs b) { gate_finalize(b.g[blockIdx.y]); }

// ---- dense dispatch / combine ------------------------------------------------------
__global__ void dispatch_scatter_kernel(const int* topk_idx, const float* topk_w, const int* slot, const int* counts_k,
                                        const float* prob_sum, int T, int E, int k, pikv_dense_out d) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (d.aux && blockIdx.x == 0 && threadIdx.x < 32) router_aux_loss(prob_sum, T, E, d.balance, d.coefficient, d.aux);
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= T * k) return;
    const int t = p / k, j = p % k;
    const int e = topk_idx[p];
    dense_store(d, t, e, E, d.position_mode == 0 ? slot[p] : dense_position(counts_k, E, e, j), topk_w[p]);
}

static int gate_geometry(int T, int* chunk_out, int* G_out) {
    int sms = sm_count();
    int G = min(GATE_MAX_CTAS, max(1, min(2 * sms, ceil_div(T, 32))));
    int chunk = ceil_div(T, G);
    if (chunk > GATE_MAX_CHUNK) chunk = GATE_MAX_CHUNK;
    G = ceil_div(T, chunk);
    if (G > GATE_MAX_CTAS) return -1;
    *chunk_out = chunk;
    *G_out = G;
    return 0;
}

template <typename TIn, int EP, int TPW>
static int launch_act(const GateDev& g, cudaStream_t st) {
    size_t smem = sizeof(int) * (GATE_WARPS * EP + EP + GATE_MAX_K * EP) + sizeof(float) * GATE_WARPS * TPW * EP +
                  (size_t)g.chunk * g.k;
    auto kern = gate_act_kernel<TIn, EP, TPW>;
    if (smem > 48 * 1024) cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    kern<<<g.G, GATE_THREADS, smem, st>>>(g);
    return check_launch("gate_act_kernel");
}
template <int EP>
static int launch_logits(const GateDev& g, cudaStream_t st) {
    size_t smem = sizeof(int) * (GATE_WARPS * EP + EP + GATE_MAX_K * EP) + sizeof(float) * GATE_WARPS * EP +
                  (size_t)g.chunk * g.k;
    auto kern = gate_logits_kernel<EP>;
    if (smem > 48 * 1024) cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    kern<<<g.G, GATE_THREADS, smem, st>>>(g);
    return check_launch("gate_logits_kernel");
}

template <typename... KArgs, typename... Args>
static int launch_tail(const char* what, void (*kern)(KArgs...), int grid, size_t smem, cudaStream_t st, const Args&... args) {
    launch_dependent(kern, grid, GATE_THREADS, smem, st, args...);
    return check_launch(what);
}

static int dispatch_launch(const int* topk_idx, const float* topk_w, const int* slot, const int* counts_k, const float* prob_sum,
                           int T, int E, int k, const pikv_dense_out& d, cudaStream_t st) {
    count_launch(1);
    return launch_tail("dispatch_scatter_kernel", dispatch_scatter_kernel, ceil_div(T * k, GATE_THREADS), 0, st, topk_idx, topk_w,
                            slot, counts_k, prob_sum, T, E, k, d);
}

template <int EP>
static int launch_batch(const GateDevs& b, int n, int k, cudaStream_t st) {
    const size_t smem = sizeof(int) * (GATE_WARPS * EP + EP + GATE_MAX_K * EP) + sizeof(float) * GATE_WARPS * EP + (size_t)b.g[0].chunk * k;
    if (smem > 48 * 1024 && !allow_smem<gate_logits_batch_kernel<EP>>()) return check_launch("gate_logits smem attribute");
    const dim3 grid((unsigned)b.g[0].G, (unsigned)n);
    launch_dependent(gate_logits_batch_kernel<EP>, grid, GATE_THREADS, smem, st, b);
    launch_dependent(gate_finalize_batch_kernel, grid, GATE_THREADS, 0, st, b);
    count_launch(2);
    return check_launch("gate_logits_batch_kernel");
}

template <int EP>
static int launch_partial(GateDev& g, const float* part, int groups, const void* b2, bool b2_bf16, const pikv_dense_out* dense, cudaStream_t st) {
    if (g.T <= GC_MAX_TOKENS && (dense == nullptr || g.topk_w != nullptr)) {
        g.chunk = ceil_div(g.T, GC_CTAS);
        g.G = GC_CTAS;
        const size_t smem = sizeof(float) * GATE_THREADS * (EP + 1) + (size_t)GATE_THREADS * max(4, g.k) * (sizeof(int) + 1);
        if (smem > 48 * 1024 && !allow_smem<gate_cluster_kernel<EP>>(200 * 1024)) return check_launch("gate_cluster smem attribute");
        count_launch(1);
        return launch_tail("gate_cluster_kernel", gate_cluster_kernel<EP>, GC_CTAS, smem, st, g, part, groups, b2, b2_bf16,
                                dense ? *dense : pikv_dense_out{});
    }
    const size_t smem = sizeof(int) * (GATE_WARPS * EP + EP + GATE_MAX_K * EP) + sizeof(float) * (GATE_WARPS * EP + GP_TOKENS * (EP + 1)) +
                        (size_t)g.chunk * g.k;
    if (smem > 48 * 1024 && !allow_smem<gate_partial_kernel<EP>>()) return check_launch("gate_partial smem attribute");
    int rc = launch_tail("gate_partial_kernel", gate_partial_kernel<EP>, g.G, smem, st, g, part, groups, b2, b2_bf16);
    if (rc == PIKV_OK) rc = launch_tail("gate_finalize_kernel", gate_finalize_kernel, g.G, 0, st, g);
    count_launch(2);
    return rc != PIKV_OK || !dense ? rc : dispatch_launch(g.topk_idx, g.topk_w, g.slot, g.counts_k, g.prob_sum, g.T, g.E, g.k, *dense, st);
}
int gate_from_partials(GateDev& g, const float* part, int groups, const void* b2, bool b2_bf16, const pikv_dense_out* dense,
                       cudaStream_t st) {
    if (g.E <= 4) return launch_partial<4>(g, part, groups, b2, b2_bf16, dense, st);
    if (g.E <= 8) return launch_partial<8>(g, part, groups, b2, b2_bf16, dense, st);
    if (g.E <= 16) return launch_partial<16>(g, part, groups, b2, b2_bf16, dense, st);
    if (g.E <= 32) return launch_partial<32>(g, part, groups, b2, b2_bf16, dense, st);
    return launch_partial<64>(g, part, groups, b2, b2_bf16, dense, st);
}

// per-CTA counters, then T*top_k chunk-local ranks (used when a consumer finishes the slot scan)
static size_t gate_tail_workspace(int T, int E, int top_k) {
    return (size_t)GATE_MAX_CTAS * (size_t)E * (size_t)(top_k + 2) * 4 + (size_t)T * (size_t)top_k * 4;
}
float* gate_partials(const GateDev& g) {
    return reinterpret_cast<float*>(reinterpret_cast<unsigned char*>(g.cta_cnt) + ((gate_tail_workspace(g.T, g.E, g.k) + 15) & ~(size_t)15));
}

}  // namespace pikv

using namespace pikv;

extern "C" size_t pikv_gate_tail_workspace_bytes(int32_t T, int32_t E, int32_t top_k) {
    return T <= 0 || E <= 0 || top_k <= 0 ? 0 : gate_tail_workspace(T, E, top_k);
}

extern "C" size_t pikv_gate_workspace_bytes(int32_t T, int32_t E, int32_t top_k) {
    if (T <= 0 || E <= 0 || top_k <= 0) return 0;
    return gate_tail_workspace(T, E, top_k) + 16 + (size_t)gate_max_partials(T) * T * E * sizeof(float);
}

namespace pikv {
int gate_run(const pikv_gate_params* p, cudaStream_t st, int what, GateDev* out) {
    PIKV_REQUIRE(p != nullptr, PIKV_EINVAL, "gate: null params");
    PIKV_REQUIRE(p->T > 0 && p->E > 0 && p->top_k > 0, PIKV_EINVAL, "gate: T, E, top_k must be positive");
    PIKV_REQUIRE(p->E <= GATE_MAX_E, PIKV_ELIMIT, "gate: E=%d exceeds %d", p->E, GATE_MAX_E);
    PIKV_REQUIRE(p->top_k <= GATE_MAX_K && p->top_k <= p->E, PIKV_ELIMIT, "gate: top_k=%d must be <= min(E, %d)",
                 p->top_k, GATE_MAX_K);
    PIKV_REQUIRE(p->topk_idx != nullptr, PIKV_EINVAL, "gate: topk_idx output is required");
    PIKV_REQUIRE(p->act != nullptr || p->logits_in != nullptr, PIKV_EINVAL, "gate: give act+w2 or logits_in");
    PIKV_REQUIRE(p->mask_mode == PIKV_MASK_NONE || p->expert_mask != nullptr, PIKV_EINVAL,
                 "gate: mask_mode set without expert_mask");
    PIKV_REQUIRE(p->mask_mode >= 0 && p->mask_mode <= 3, PIKV_EINVAL, "gate: bad mask_mode %d", p->mask_mode);
    PIKV_REQUIRE(p->workspace != nullptr && p->workspace_bytes >= gate_tail_workspace(p->T, p->E, p->top_k),
                 PIKV_EINVAL, "gate: workspace too small");
    GateDev g;
    g.act = p->act; g.w2 = p->w2; g.b2 = p->b2; g.logits_in = p->logits_in;
    g.T = p->T; g.H = p->H; g.E = p->E; g.k = p->top_k;
    g.mask = p->expert_mask; g.mask_mode = p->expert_mask ? p->mask_mode : PIKV_MASK_NONE;
    g.corr = p->correction; g.temperature = p->temperature == 0.f ? 1.f : p->temperature; g.eps = p->renorm_eps;
    g.capacity = p->capacity; g.slot_base = p->slot_base;
    g.probs = p->probs; g.topk_idx = p->topk_idx; g.topk_w = p->topk_w; g.slot = p->slot;
    g.counts_k = p->counts_k; g.prob_sum = p->prob_sum; g.new_len = p->new_len;
    PIKV_REQUIRE(gate_geometry(p->T, &g.chunk, &g.G) == 0, PIKV_ELIMIT, "gate: T=%d too large for one call", p->T);
    int* ws = static_cast<int*>(p->workspace);
    g.cta_cnt = ws;
    g.cta_cnt_k = ws + (size_t)GATE_MAX_CTAS * g.E;
    g.cta_psum = reinterpret_cast<float*>(ws + (size_t)GATE_MAX_CTAS * g.E * (g.k + 1));
    if (what & GATE_RANKS_TO_WS) g.slot = ws + (size_t)GATE_MAX_CTAS * g.E * (g.k + 2);
    int rc;
    const int E = g.E;
    const bool use_tc = g.act != nullptr && g.w2 != nullptr && gate_tc_supported(g, p->dtype) && !(p->phase & PIKV_GATE_FORCE_SIMT);
    if (!(what & GATE_DO_SCORE)) {
        if (use_tc) gate_tc_geometry(g);
        if (out) *out = g;
        if (!(what & GATE_DO_SLOTS)) return PIKV_OK;
        count_launch(1);
        gate_finalize_kernel<<<g.G, GATE_THREADS, 0, st>>>(g);
        return check_launch("gate_finalize_kernel");
    }
    if (use_tc) {
        rc = gate_tc_launch(g, st);
    } else if (g.act != nullptr) {
        PIKV_REQUIRE(g.w2 != nullptr, PIKV_EINVAL, "gate: w2 is required with act");
        PIKV_REQUIRE(g.H > 0 && g.H % 8 == 0, PIKV_EUNSUPPORTED, "gate: H=%d must be a positive multiple of 8", g.H);
        PIKV_REQUIRE(p->dtype == PIKV_F32 || p->dtype == PIKV_BF16, PIKV_EINVAL, "gate: bad dtype %d", p->dtype);
#define PIKV_GATE_DISPATCH(TIn)                                                     \
        if (E <= 4) rc = launch_act<TIn, 4, 4>(g, st);                              \
        else if (E <= 8) rc = launch_act<TIn, 8, 4>(g, st);                         \
        else if (E <= 16) rc = launch_act<TIn, 16, 4>(g, st);                       \
        else if (E <= 32) rc = launch_act<TIn, 32, 2>(g, st);                       \
        else rc = launch_act<TIn, 64, 1>(g, st);
        if (p->dtype == PIKV_BF16) { PIKV_GATE_DISPATCH(__nv_bfloat16) } else { PIKV_GATE_DISPATCH(float) }
#undef PIKV_GATE_DISPATCH
    } else {
        if (E <= 4) rc = launch_logits<4>(g, st);
        else if (E <= 8) rc = launch_logits<8>(g, st);
        else if (E <= 16) rc = launch_logits<16>(g, st);
        else if (E <= 32) rc = launch_logits<32>(g, st);
        else rc = launch_logits<64>(g, st);
    }
    if (rc != PIKV_OK) return rc;
    if (out) *out = g;
    if (!(what & GATE_DO_SLOTS)) {
        count_launch(1);
        return PIKV_OK;
    }
    gate_finalize_kernel<<<g.G, GATE_THREADS, 0, st>>>(g);
    count_launch(2);
    return check_launch("gate_finalize_kernel");
}
}  // namespace pikv

extern "C" int pikv_gate_fused(const pikv_gate_params* p, pikv_stream_t stream) {
    PIKV_REQUIRE(p != nullptr, PIKV_EINVAL, "gate: null params");
    const int phase = p->phase & ~PIKV_GATE_FORCE_SIMT;
    PIKV_REQUIRE(phase >= PIKV_GATE_WHOLE && phase <= PIKV_GATE_SLOTS, PIKV_EINVAL, "gate: bad phase %d", p->phase);
    const int what = phase == PIKV_GATE_SCORE ? GATE_DO_SCORE : phase == PIKV_GATE_SLOTS ? GATE_DO_SLOTS
                                                                                        : (GATE_DO_SCORE | GATE_DO_SLOTS);
    return gate_run(p, static_cast<cudaStream_t>(stream), what, nullptr);
}

extern "C" int pikv_gate_logits(const pikv_gate_params* const* p, int32_t n, pikv_stream_t stream) {
    PIKV_REQUIRE(p != nullptr && n > 0 && n <= GATE_MAX_BATCH, PIKV_EINVAL, "gate_logits: %d gates (1 to %d)", n, GATE_MAX_BATCH);
    GateDevs b = {};
    int k = 0;
    for (int i = 0; i < n; ++i) {
        PIKV_REQUIRE(p[i] && p[i]->logits_in && p[i]->T == p[0]->T && p[i]->E == p[0]->E, PIKV_EINVAL, "gate_logits: the gates share T and E");
        const int rc = gate_run(p[i], nullptr, 0, &b.g[i]);
        if (rc != PIKV_OK) return rc;
        k = max(k, p[i]->top_k);
    }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int E = p[0]->E;
    if (E <= 4) return launch_batch<4>(b, n, k, st);
    if (E <= 8) return launch_batch<8>(b, n, k, st);
    if (E <= 16) return launch_batch<16>(b, n, k, st);
    if (E <= 32) return launch_batch<32>(b, n, k, st);
    return launch_batch<64>(b, n, k, st);
}

extern "C" int pikv_dispatch_loss(const int32_t* topk_idx, const float* topk_w, const int32_t* slot,
                                  const int32_t* counts_k, const float* prob_sum, int32_t T, int32_t E, int32_t top_k,
                                  const pikv_dense_out* d, pikv_stream_t stream) {
    PIKV_REQUIRE(topk_idx && topk_w && d && d->dispatch && d->combine, PIKV_EINVAL, "dispatch_scatter: null pointer");
    PIKV_REQUIRE(T > 0 && E > 0 && top_k > 0 && d->capacity > 0, PIKV_EINVAL, "dispatch_scatter: bad sizes");
    PIKV_REQUIRE(d->position_mode == 0 ? slot != nullptr : counts_k != nullptr, PIKV_EINVAL,
                 "dispatch_scatter: slot (mode 0) or counts_k (mode 1) required");
    PIKV_REQUIRE(d->aux == nullptr || (prob_sum != nullptr && E <= GATE_MAX_E && d->balance >= 0 && d->balance <= 3), PIKV_EINVAL,
                 "dispatch_loss: the loss needs prob_sum, at most %d experts and a balance term from 0 to 3", GATE_MAX_E);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const size_t bytes = (size_t)T * E * d->capacity * sizeof(float);
    if (cudaMemsetAsync(d->dispatch, 0, bytes, st) != cudaSuccess || cudaMemsetAsync(d->combine, 0, bytes, st) != cudaSuccess)
        return check_launch("dispatch_scatter memset");
    return dispatch_launch(topk_idx, topk_w, slot, counts_k, prob_sum, T, E, top_k, *d, st);
}

extern "C" int pikv_dispatch_scatter(const int32_t* topk_idx, const float* topk_w, const int32_t* slot,
                                     const int32_t* counts_k, int32_t T, int32_t E, int32_t top_k,
                                     int32_t capacity, int32_t position_mode, float* dispatch, float* combine,
                                     pikv_stream_t stream) {
    const pikv_dense_out d = {dispatch, combine, capacity, position_mode, 0, 0.f, nullptr};
    return pikv_dispatch_loss(topk_idx, topk_w, slot, counts_k, nullptr, T, E, top_k, &d, stream);
}
