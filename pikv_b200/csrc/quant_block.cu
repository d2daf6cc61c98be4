// Block-wide fake quantisation (the drop-in arithmetic of QuantizedCompressor.forward):
// every column group is one block whose min/max run over ALL rows.
//
//   stats   CTA per (32 * VEC columns, row block, tensor): 16-byte loads, the min/max of every group segment of the
//           tile reduced over the CTA's rows to one partial per (row block, segment)
//   apply   same tiles: the CTA reduces its groups' partials over the row blocks, forms scale / zero point with the
//           reference's formulas, then codes, dequantised values and squared-error partials
//   err     warp per group: reduces the squared-error partials (only when all groups' errors are asked for; the mean
//           of one group, which is what a forward keeps, is finished by the last apply CTA)
// K and V of a forward are one launch of each (grid.z = tensor).  All reductions have a fixed order, so results are
// run-to-run identical.
//
// Bound by the bytes: x is read twice (the second time mostly from L2) and written once.  A segment is the largest
// power of two of 16-byte chunks that divides a group (at most a warp's row), so a group of 128 leaves one partial per
// row block and the apply CTAs read a few dozen of them.  K and V of 8192 x 1024 fp32, groups of 128 (134 MB): 1147 us
// when one thread per group walked the partials of all its columns (params 338 us, err 190 us per tensor) over 4-byte
// loads; 35 us now, the statistics at 4.9 TB/s.
#include "common.cuh"
#include <float.h>

namespace pikv {

constexpr int QB_THREADS = 256;
constexpr int QB_WARPS = QB_THREADS / 32;
constexpr int QB_MAX_RB = 128;
constexpr int QB_UNROLL = 4;           // rows in flight per thread

struct QbTensor {
    const void* x;
    void* dq;            // TOut [N,H] or null
    float* q;            // [N,H] or null
    float* params_out;   // [G][2] or null
};

struct QbArgs {
    QbTensor t[2];
    const float* params_in;   // [G][2]: static mode
    int N, H, rows_per, RB, gs, G, sub, nsub, qmin, qmax, symmetric, tensors;
    float2* mm;               // [tensors][RB][nsub] (min, max)
    float* err;               // [tensors][RB][nsub], or null when nobody asked for errors
    unsigned* ticket;         // CTAs of the last tensor that have stored their errors
    float* mse;               // mean squared error of the last tensor's last group, or null
    float* count;             // sample counter of the module, or null
    float count_add;
};

// VEC consecutive elements of a row as floats; the vector forms are one 16-byte load
template <typename TIn, int VEC>
__device__ __forceinline__ void qb_load(const TIn* p, float (&v)[VEC]) {
    if constexpr (VEC == 4) {
        const float4 f = __ldg(reinterpret_cast<const float4*>(p));
        v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w;
    } else if constexpr (VEC == 8) {
        const uint4 u = __ldg(reinterpret_cast<const uint4*>(p));
        bf16x2_to_f32(u.x, v[0], v[1]);
        bf16x2_to_f32(u.y, v[2], v[3]);
        bf16x2_to_f32(u.z, v[4], v[5]);
        bf16x2_to_f32(u.w, v[6], v[7]);
    } else if constexpr (sizeof(TIn) == 4) {
        v[0] = __ldg(reinterpret_cast<const float*>(p));
    } else {
        v[0] = bf16_bits_to_f32(__ldg(reinterpret_cast<const unsigned short*>(p)));
    }
}
// streamed past L2's useful contents: the second tensor's input is still to be read from there
template <typename TOut, int VEC>
__device__ __forceinline__ void qb_store(TOut* p, const float (&v)[VEC]) {
    if constexpr (sizeof(TOut) == 4) {
        if constexpr (VEC == 1) {
            __stcs(reinterpret_cast<float*>(p), v[0]);
        } else {
#pragma unroll
            for (int i = 0; i < VEC; i += 4) __stcs(reinterpret_cast<float4*>(p + i), make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]));
        }
    } else {
        if constexpr (VEC == 1) {
            *reinterpret_cast<unsigned short*>(p) = f32_to_bf16_bits(v[0]);
        } else {
            uint32_t w[VEC / 2];
#pragma unroll
            for (int i = 0; i < VEC; i += 2) w[i / 2] = (uint32_t)f32_to_bf16_bits(v[i]) | ((uint32_t)f32_to_bf16_bits(v[i + 1]) << 16);
            if constexpr (VEC == 4) __stcs(reinterpret_cast<uint2*>(p), make_uint2(w[0], w[1]));
            else __stcs(reinterpret_cast<uint4*>(p), make_uint4(w[0], w[1], w[2], w[3]));
        }
    }
}

template <typename TIn, int VEC>
__global__ void __launch_bounds__(QB_THREADS) qb_stats_kernel(QbArgs a) {
    __shared__ float2 part[QB_WARPS][32];
    // the apply kernel may be scheduled as CTAs of this one leave; it waits for all of them before it reads partials
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int col = (blockIdx.x * 32 + lane) * VEC;
    const int rb = blockIdx.y;
    if (threadIdx.x == 0 && blockIdx.x == 0 && rb == 0 && blockIdx.z == 0) *a.ticket = 0u;
    const int r1 = min(a.N, (rb + 1) * a.rows_per);
    float mn = FLT_MAX, mx = -FLT_MAX;
    if (col < a.H) {
        const TIn* x = static_cast<const TIn*>(a.t[blockIdx.z].x) + col;
        for (int r = rb * a.rows_per + warp; r < r1; r += QB_UNROLL * QB_WARPS) {
            float v[QB_UNROLL][VEC];
#pragma unroll
            for (int u = 0; u < QB_UNROLL; ++u)     // rows past the end read the last one again: no effect on min / max
                qb_load<TIn, VEC>(x + (size_t)min(r + u * QB_WARPS, r1 - 1) * a.H, v[u]);
#pragma unroll
            for (int u = 0; u < QB_UNROLL; ++u)
#pragma unroll
                for (int i = 0; i < VEC; ++i) {
                    mn = fminf(mn, v[u][i]);
                    mx = fmaxf(mx, v[u][i]);
                }
        }
    }
    part[warp][lane] = make_float2(mn, mx);
    __syncthreads();
    if (warp == 0) {
#pragma unroll
        for (int w = 1; w < QB_WARPS; ++w) {
            mn = fminf(mn, part[w][lane].x);
            mx = fmaxf(mx, part[w][lane].y);
        }
        for (int o = 1; o < a.sub; o <<= 1) {
            mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, o));
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        }
        const int seg = (blockIdx.x * 32 + lane) / a.sub;
        if (lane % a.sub == 0 && seg < a.nsub)
            a.mm[((size_t)blockIdx.z * a.RB + rb) * a.nsub + seg] = make_float2(mn, mx);
    }
}

// segments [s0, s1) of group g: group starts are multiples of a segment
template <int VEC>
__device__ __forceinline__ void qb_group_segments(const QbArgs& a, int g, int& s0, int& s1) {
    const int w = VEC * a.sub;
    s0 = g * a.gs / w;
    s1 = min(a.nsub, (min(a.H, (g + 1) * a.gs) + w - 1) / w);
}

template <typename TIn, typename TOut, int VEC>
__global__ void __launch_bounds__(QB_THREADS) qb_apply_kernel(QbArgs a) {
    __shared__ float2 prm[32 * VEC + 1];
    __shared__ float part[QB_WARPS][32];
    __shared__ bool last;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int z = blockIdx.z, rb = blockIdx.y;
    const int col0 = blockIdx.x * 32 * VEC, col = col0 + lane * VEC;
    const QbTensor& t = a.t[z];
    const int g0 = col0 / a.gs, g1 = (min(a.H, col0 + 32 * VEC) - 1) / a.gs;
    // scale and zero point of the tile's groups
    asm volatile("griddepcontrol.wait;" ::: "memory");
    for (int g = g0 + warp; g <= g1; g += QB_WARPS) {
        QParams p;
        if (a.params_in) {
            p.scale = __ldg(a.params_in + 2 * g);
            p.zp = __ldg(a.params_in + 2 * g + 1);
        } else {
            int s0, s1;
            qb_group_segments<VEC>(a, g, s0, s1);
            const int n = s1 - s0;
            float mn = FLT_MAX, mx = -FLT_MAX;
            for (int i = lane; i < a.RB * n; i += 32) {
                const float2 v = a.mm[((size_t)z * a.RB + i / n) * a.nsub + s0 + i % n];
                mn = fminf(mn, v.x);
                mx = fmaxf(mx, v.y);
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, o));
                mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
            }
            p = quant_params(mn, mx, a.qmin, a.qmax, a.symmetric != 0);
        }
        if (lane == 0) {
            prm[g - g0] = make_float2(p.scale, p.zp);
            if (t.params_out && rb == 0) {
                t.params_out[2 * g] = p.scale;
                t.params_out[2 * g + 1] = p.zp;
            }
        }
    }
    __syncthreads();
    const int r1 = min(a.N, (rb + 1) * a.rows_per);
    float err = 0.f;
    if (col < a.H && (t.dq || t.q || a.err)) {
        const TIn* x = static_cast<const TIn*>(t.x) + col;
        TOut* dq_out = t.dq ? static_cast<TOut*>(t.dq) + col : nullptr;
        float* q_out = t.q ? t.q + col : nullptr;
        const float2 pp = prm[col / a.gs - g0];
        QParams p;
        p.scale = pp.x;
        p.zp = pp.y;
        const float inv = __frcp_rn(p.scale), qmin = (float)a.qmin, qmax = (float)a.qmax;
        auto one = [&](int r, const float (&v)[VEC]) {
            float q[VEC], dq[VEC];
#pragma unroll
            for (int i = 0; i < VEC; ++i) {
                q[i] = quant_code_fast(v[i], p, inv, qmin, qmax);
                dq[i] = dequant_code(q[i], p);
                const float d = __fsub_rn(v[i], dq[i]);
                err = __fadd_rn(err, __fmul_rn(d, d));
            }
            if (dq_out) qb_store<TOut, VEC>(dq_out + (size_t)r * a.H, dq);
            if (q_out) qb_store<float, VEC>(q_out + (size_t)r * a.H, q);
        };
        for (int r = rb * a.rows_per + warp; r < r1; r += QB_UNROLL * QB_WARPS) {
            float v[QB_UNROLL][VEC];
#pragma unroll
            for (int u = 0; u < QB_UNROLL; ++u) qb_load<TIn, VEC>(x + (size_t)min(r + u * QB_WARPS, r1 - 1) * a.H, v[u]);
#pragma unroll
            for (int u = 0; u < QB_UNROLL; ++u)
                if (r + u * QB_WARPS < r1) one(r + u * QB_WARPS, v[u]);
        }
    }
    if (!a.err) return;
    part[warp][lane] = err;
    __syncthreads();
    if (warp == 0) {
#pragma unroll
        for (int w = 1; w < QB_WARPS; ++w) err += part[w][lane];
        for (int o = 1; o < a.sub; o <<= 1) err += __shfl_xor_sync(0xffffffffu, err, o);
        const int seg = (blockIdx.x * 32 + lane) / a.sub;
        if (lane % a.sub == 0 && seg < a.nsub) a.err[((size_t)z * a.RB + rb) * a.nsub + seg] = err;
    }
    if (!a.mse || z != a.tensors - 1) return;
    // the last CTA of the last tensor adds up that tensor's last group
    if (threadIdx.x < 32) {
        __threadfence();
        __syncwarp();
        if (lane == 0) last = atomicAdd(a.ticket, 1u) == gridDim.x * gridDim.y - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    int s0, s1;
    qb_group_segments<VEC>(a, a.G - 1, s0, s1);
    const int n = s1 - s0;
    float s = 0.f;
    for (int i = threadIdx.x; i < a.RB * n; i += QB_THREADS)
        s += __ldcg(a.err + ((size_t)z * a.RB + i / n) * a.nsub + s0 + i % n);
    s = warp_sum(s);
    if (lane == 0) part[warp][0] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        float total = 0.f;
        for (int w = 0; w < QB_WARPS; ++w) total += part[w][0];
        *a.mse = total / ((float)a.N * (float)(a.H - (a.G - 1) * a.gs));
        if (a.count) *a.count += a.count_add;
    }
}

template <int VEC>
__global__ void __launch_bounds__(QB_THREADS) qb_err_kernel(QbArgs a, float* sq_err) {
    const int lane = threadIdx.x & 31;
    const int g = blockIdx.x * QB_WARPS + (threadIdx.x >> 5);
    if (g >= a.G) return;
    int s0, s1;
    qb_group_segments<VEC>(a, g, s0, s1);
    const int n = s1 - s0;
    float s = 0.f;
    for (int i = lane; i < a.RB * n; i += 32) s += a.err[(size_t)(i / n) * a.nsub + s0 + i % n];
    s = warp_sum(s);
    if (lane == 0) sq_err[g] = s;
}

template <typename TIn, typename TOut, int VEC>
static int qb_launch(QbArgs& a, float* sq_err, cudaStream_t st) {
    const int tiles = ceil_div(a.H, 32 * VEC);
    // enough CTAs for four per SM, at least 32 rows each (four loads in flight per thread)
    a.RB = max(1, min(min(ceil_div(4 * sm_count(), tiles * a.tensors), QB_MAX_RB), ceil_div(a.N, QB_WARPS * QB_UNROLL)));
    a.rows_per = ceil_div(ceil_div(a.N, a.RB), QB_WARPS * QB_UNROLL) * QB_WARPS * QB_UNROLL;   // whole steps but for the last block
    a.RB = ceil_div(a.N, a.rows_per);
    a.sub = 1;
    while (a.sub < 32 && a.gs % (2 * a.sub * VEC) == 0) a.sub *= 2;
    a.nsub = ceil_div(a.H, VEC * a.sub);
    const dim3 grid(tiles, a.RB, a.tensors);
    if (!a.params_in) {
        qb_stats_kernel<TIn, VEC><<<grid, QB_THREADS, 0, st>>>(a);
        count_launch(1);
    } else if (a.mse) {
        if (cudaMemsetAsync(a.ticket, 0, sizeof(unsigned), st) != cudaSuccess) return check_launch("quant_block ticket");
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = QB_THREADS;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = a.params_in ? 0 : 1;
    cudaLaunchKernelEx(&cfg, qb_apply_kernel<TIn, TOut, VEC>, a);
    count_launch(1);
    if (sq_err) {
        qb_err_kernel<VEC><<<ceil_div(a.G, QB_WARPS), QB_THREADS, 0, st>>>(a, sq_err);
        count_launch(1);
    }
    return check_launch("quant_block");
}

// 16-byte accesses where rows, groups and every pointer allow them, one element per thread otherwise
static int qb_run(QbArgs& a, int dtype, bool dq_bf16, float* sq_err, void* workspace, cudaStream_t st) {
    float* ws = static_cast<float*>(workspace);
    a.mm = reinterpret_cast<float2*>(ws);
    float* err = ws + (size_t)2 * a.tensors * QB_MAX_RB * a.H;
    a.ticket = reinterpret_cast<unsigned*>(err + (size_t)a.tensors * QB_MAX_RB * a.H);
    a.err = (sq_err || a.mse) ? err : nullptr;
    const int vec = dtype == PIKV_F32 ? 4 : 8;
    bool wide = a.H % vec == 0 && a.gs % vec == 0;
    for (int i = 0; i < a.tensors; ++i)
        wide = wide && (((uintptr_t)a.t[i].x | (uintptr_t)a.t[i].dq | (uintptr_t)a.t[i].q) & 15) == 0;
    if (dtype == PIKV_F32) return wide ? qb_launch<float, float, 4>(a, sq_err, st) : qb_launch<float, float, 1>(a, sq_err, st);
    if (dq_bf16)
        return wide ? qb_launch<__nv_bfloat16, __nv_bfloat16, 8>(a, sq_err, st)
                    : qb_launch<__nv_bfloat16, __nv_bfloat16, 1>(a, sq_err, st);
    return wide ? qb_launch<__nv_bfloat16, float, 8>(a, sq_err, st) : qb_launch<__nv_bfloat16, float, 1>(a, sq_err, st);
}

}  // namespace pikv

using namespace pikv;

static size_t qb_workspace(int tensors, int H) { return ((size_t)3 * tensors * QB_MAX_RB * H + 4) * sizeof(float); }

extern "C" size_t pikv_quant_block_workspace_bytes(int32_t N, int32_t H, int32_t group_size) {
    (void)N;
    return H <= 0 || group_size <= 0 ? 0 : qb_workspace(1, H);
}

extern "C" size_t pikv_quant_block_pair_workspace_bytes(int32_t N, int32_t H, int32_t group_size) {
    (void)N;
    return H <= 0 || group_size <= 0 ? 0 : qb_workspace(2, H);
}

static int qb_check(int32_t dtype, int32_t N, int32_t H, int32_t group_size, int32_t qmin, int32_t qmax) {
    PIKV_REQUIRE(N > 0 && H > 0 && group_size > 0, PIKV_EINVAL, "quant_block: bad sizes");
    PIKV_REQUIRE(qmax > qmin, PIKV_EINVAL, "quant_block: qmax must exceed qmin");
    PIKV_REQUIRE(dtype == PIKV_F32 || dtype == PIKV_BF16, PIKV_EINVAL, "quant_block: bad dtype %d", dtype);
    return PIKV_OK;
}

static void qb_fill(QbArgs& a, int N, int H, int gs, int qmin, int qmax, int symmetric, const float* params_in) {
    a.params_in = params_in;
    a.N = N; a.H = H;
    a.gs = gs;
    a.G = ceil_div(H, gs);
    a.qmin = qmin; a.qmax = qmax; a.symmetric = symmetric;
}

extern "C" int pikv_quant_block(const void* x, int32_t dtype, int32_t N, int32_t H, int32_t group_size, int32_t qmin,
                                int32_t qmax, int32_t symmetric, const float* params_in, float* params_out,
                                float* dq_out, float* q_out, float* sq_err, void* workspace, size_t workspace_bytes,
                                pikv_stream_t stream) {
    PIKV_REQUIRE(x != nullptr, PIKV_EINVAL, "quant_block: null input");
    int rc = qb_check(dtype, N, H, group_size, qmin, qmax);
    if (rc != PIKV_OK) return rc;
    PIKV_REQUIRE(workspace && workspace_bytes >= qb_workspace(1, H), PIKV_EINVAL, "quant_block: workspace too small");
    QbArgs a = {};
    qb_fill(a, N, H, group_size, qmin, qmax, symmetric, params_in);
    a.tensors = 1;
    a.t[0] = {x, dq_out, q_out, params_out};
    return qb_run(a, dtype, false, sq_err, workspace, static_cast<cudaStream_t>(stream));
}

extern "C" int pikv_quant_block_pair(const void* k, const void* v, int32_t dtype, int32_t N, int32_t H,
                                     int32_t group_size, int32_t qmin, int32_t qmax, int32_t symmetric,
                                     const float* params_in, void* dq_k, void* dq_v, float* mse, float* sample_count,
                                     float count_add, void* workspace, size_t workspace_bytes, pikv_stream_t stream) {
    PIKV_REQUIRE(k && v && dq_k && dq_v && mse, PIKV_EINVAL, "quant_block_pair: null pointer");
    int rc = qb_check(dtype, N, H, group_size, qmin, qmax);
    if (rc != PIKV_OK) return rc;
    PIKV_REQUIRE(workspace && workspace_bytes >= qb_workspace(2, H), PIKV_EINVAL, "quant_block_pair: workspace too small");
    QbArgs a = {};
    qb_fill(a, N, H, group_size, qmin, qmax, symmetric, params_in);
    a.tensors = 2;
    a.t[0] = {k, dq_k, nullptr, nullptr};
    a.t[1] = {v, dq_v, nullptr, nullptr};
    a.mse = mse;
    a.count = sample_count;
    a.count_add = count_add;
    return qb_run(a, dtype, dtype == PIKV_BF16, nullptr, workspace, static_cast<cudaStream_t>(stream));
}
