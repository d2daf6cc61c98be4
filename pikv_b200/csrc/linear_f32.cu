// fp32 linear layer on the tensor cores: out[M,N] = x[M,K] . w[N,K]^T + bias, every operand as two f16 limbs.
//
// A row is scaled by a power of two so that its largest magnitude lies in [2^14, 2^15) and split into hi = f16(v) and
// lo = f16(2^11 (v - hi)): hi + 2^-11 lo meets v to 2^-23 of itself down to 2^-27 of the row's largest.  (With lo at v's own
// scale an entry of 2^-18 of the largest lost bits and one of 2^-39 vanished, which shows where the large entry meets a zero:
// relative error 1.3e-5 at a spread of 2^24, 0.7 at 2^40, against 2.9e-7 of fp32 sums.)  The product is
// hi.hi + 2^-11 (hi.lo + lo.hi), what is left out, lo.lo, is at most 2^-22 of each term.  The tensor cores' sums truncate, so
// each bracket has an fp32 accumulator of its own and each half of K another pair; the epilogue adds the four.
// Rows with an entry that the limbs miss by more than 2^-23 of itself (one entry in 60 million of normal inputs), an infinity,
// a NaN or a largest magnitude outside 2^-60 .. 2^60 are marked (scale 0) and their outputs formed by fp32 sums.
//
//   lin_split_kernel   one warp per row of w and x: limbs [rows, hi K | lo K], the inverse scales and whether
//                      each CTA marked a row
//   lin_gemm_kernel    persistent, one CTA per SM.  Items are 128 x 128 outputs, row tiles innermost, contiguous per CTA:
//                      w's tile stays in shared memory (hi and lo of a 64-wide k block next to each other: one MMA of
//                      N = 256 takes both products of an x hi block), x blocks stream through a ring.  Two accumulator
//                      pairs of 256 columns, one per half of K: sixteen epilogue warps, 32 x 32 outputs each, keep the
//                      first half's sums in registers while the second is computed, turn their patches in shared
//                      memory and store whole rows (N is odd in earnest, so neither TMA nor vector stores apply).
//                      At its end all CTAs share out the outputs of marked rows, if there are any (lin_fix).
//
// 1024 x 256 -> 50257: 137 us a call, about 28 of them the splits (134 with the low limb unscaled and entries lost; cuBLAS's fp32
// kernel and its bias pass 715), relative error 2.0e-7 against 64 bits (cuBLAS 2.9e-7; one accumulator for all of K 3.5e-7).
// A marked row of w adds 6 us, one of x 45, all 1024 of x 3.2 ms.  The 79 GFLOP of the three products would take 48 us at the
// measured bf16 rate and the output 32 us of HBM.
#include "tc_common.cuh"

namespace pikv {

constexpr int LIN_BN = 128, LIN_BLOCK = 128 * 128;       // outputs per tile; bytes of a [128 x 64] f16 block
constexpr int LIN_MAX_KB = 4, LIN_STAGES = 4;
constexpr int LIN_EPI_WARPS = 16, LIN_THREADS = 64 + 32 * LIN_EPI_WARPS;
constexpr int LIN_PATCH = 16 * 33 * 4;
constexpr float LIN_LO_SCALE = 2048.f;
constexpr int LIN_FIX_LIST = 2048, LIN_FIX_GROUP = 8;
static_assert(LIN_FIX_GROUP * 64 * LIN_MAX_KB * 4 + (LIN_FIX_LIST + LIN_THREADS + 2) * 4 <= LIN_STAGES * LIN_BLOCK, "linear_f32: marked rows");
constexpr int LIN_SMEM = 2 * LIN_MAX_KB * LIN_BLOCK + LIN_STAGES * LIN_BLOCK + LIN_EPI_WARPS * LIN_PATCH + 256 + 1024;
static_assert(LIN_SMEM <= 227 * 1024, "linear_f32: shared memory");

__device__ unsigned g_linear_error = 0;                  // sticky: set when a bounded wait ran out

struct LinArgs {
    const float *x, *w, *bias, *sx, *sw;
    const int *mx, *mw;                                  // whether a CTA of the split marked a row
    int ctas_x, ctas_w;
    float* out;
    int M, N, K, mtiles;
    long long items;
};

__global__ void __launch_bounds__(256, 8) lin_split_kernel(const float* __restrict__ src, int rows, int K, __half* __restrict__ limbs, float* __restrict__ inv,
                                                         int* __restrict__ marked) {
    dependency_release();
    dependency_wait();
    const int lane = threadIdx.x & 31;
    const int words = K / 4;                             // at most 64: two per lane
    bool marked_any = false;
    for (int r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < rows; r += gridDim.x * blockDim.x / 32) {
        float4 v[2] = {};
        float m = 0.f;
        uint32_t least = 0xffffffffu;                    // bits of the smallest magnitude but zero, less one
        bool bad = false;
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int i = lane + 32 * q;
            if (i < words) v[q] = *reinterpret_cast<const float4*>(src + (size_t)r * K + 4 * i);
            const float a[4] = {fabsf(v[q].x), fabsf(v[q].y), fabsf(v[q].z), fabsf(v[q].w)};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                m = fmaxf(m, a[j]);
                least = min(least, __float_as_uint(a[j]) - 1u);
                bad |= !(a[j] <= 3.402823466e38f);
            }
        }
        m = warp_max(m);
        const int e = (int)(__float_as_uint(m) >> 23) - 127;           // 2^e <= m < 2^(e+1)
        bad = __any_sync(0xffffffffu, bad) || e > 60 || (e < -60 && m != 0.f);
        const float up = bad ? 0.f : m == 0.f ? 1.f : __uint_as_float((uint32_t)(127 + 14 - e) << 23);
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int i = lane + 32 * q;
            if (i >= words) continue;
            const float a[4] = {v[q].x, v[q].y, v[q].z, v[q].w};
            __align__(8) __half h[4], l[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float s = bad ? 0.f : a[j] * up;
                h[j] = __float2half_rn(s);
                l[j] = __float2half_rn((s - __half2float(h[j])) * LIN_LO_SCALE);            // exact before it is rounded
            }
            __half* to = limbs + (size_t)r * 2 * K + 4 * i;
            *reinterpret_cast<uint2*>(to) = *reinterpret_cast<const uint2*>(h);
            *reinterpret_cast<uint2*>(to + K) = *reinterpret_cast<const uint2*>(l);
        }
        // at and above 2^-13 both limbs are normal f16 numbers and the entry is met; below (2^-27 of the largest) it is looked at
        if (!bad && __any_sync(0xffffffffu, least < (uint32_t)max(0, 127 + e - 27) << 23)) {
            bool missed = false;
#pragma unroll 1
            for (int i = lane; i < K; i += 32) {
                const float a = src[(size_t)r * K + i], s = a * up, rest = s - __half2float(__float2half_rn(s));
                // met to 2^-23, and with a low limb of 2^-11 at most, as the products of two are left out; a scaled entry below
                // 2^-126 was rounded itself, perhaps to zero
                missed |= fabsf(s) < 1.f / 8192.f && (fabsf(rest - __half2float(__float2half_rn(rest * LIN_LO_SCALE)) / LIN_LO_SCALE) > fabsf(s) / 8388608.f ||
                                                      fabsf(rest) > fabsf(s) / LIN_LO_SCALE || (s == 0.f && a != 0.f));
            }
            bad = __any_sync(0xffffffffu, missed);
        }
        marked_any |= bad;
        if (lane == 0) inv[r] = bad ? 0.f : m == 0.f ? 1.f : __uint_as_float((uint32_t)(127 - 14 + e) << 23);
    }
    const int marks = __syncthreads_or(marked_any);
    if (threadIdx.x == 0) marked[blockIdx.x] = marks;
}

// ---- outputs of marked rows ----
// The lane's share of eight sums over a warp: the sum of v[i] ends in the lanes with (lane >> 2) == the bits of i reversed
__device__ __forceinline__ float lin_sum8(float (&v)[8], int lane) {
#pragma unroll
    for (int half = 4; half > 0; half >>= 1) {
        const bool upper = lane & (4 * half);
#pragma unroll
        for (int i = 0; i < half; ++i) {
            const float send = upper ? v[i] : v[half + i];
            v[i] = (upper ? v[half + i] : v[i]) + __shfl_xor_sync(0xffffffffu, send, 4 * half);
        }
    }
    float s = v[0];
    s += __shfl_xor_sync(0xffffffffu, s, 2);
    return s + __shfl_xor_sync(0xffffffffu, s, 1);
}

// The outputs of the marked rows of x and of w, by all CTAs: eight marked rows in shared memory, a warp per row of the other operand
__device__ __noinline__ void lin_fix(const LinArgs& a, unsigned char* smem) {
    float (*group)[64 * LIN_MAX_KB] = reinterpret_cast<float (*)[64 * LIN_MAX_KB]>(smem);
    int* list = reinterpret_cast<int*>(group + LIN_FIX_GROUP);             // rows, at most LIN_FIX_LIST
    int* slots = list + LIN_FIX_LIST;                                      // CTAs of the split, at most LIN_THREADS
    int &listed = slots[LIN_THREADS], &found = slots[LIN_THREADS + 1];
    const int tid = threadIdx.x, lane = tid & 31, K = a.K;
    const long long worker = (long long)blockIdx.x * (LIN_THREADS / 32) + (tid >> 5), workers = (long long)gridDim.x * (LIN_THREADS / 32);
    for (int side = 0; side < 2; ++side) {
        const float *own = side == 0 ? a.x : a.w, *other = side == 0 ? a.w : a.x, *inv = side == 0 ? a.sx : a.sw;
        const int* marked = side == 0 ? a.mx : a.mw;
        const int count = side == 0 ? a.M : a.N, others = side == 0 ? a.N : a.M, ctas = side == 0 ? a.ctas_x : a.ctas_w, stride = ctas * 8;
        auto flush = [&]() {
            for (int g0 = 0; g0 < listed; g0 += LIN_FIX_GROUP) {
                const int n = min(LIN_FIX_GROUP, listed - g0);
                __syncthreads();
                for (int i = tid; i < LIN_FIX_GROUP * K; i += LIN_THREADS) group[i / K][i % K] = i / K < n ? own[(size_t)list[g0 + i / K] * K + i % K] : 0.f;
                __syncthreads();
                for (long long o = worker; o < others; o += workers) {
                    float v[LIN_FIX_GROUP] = {};
#pragma unroll
                    for (int c = 0; c < LIN_MAX_KB; ++c) {
                        if (64 * c >= K) break;
                        const float2 u = __ldg(reinterpret_cast<const float2*>(other + (size_t)o * K + 64 * c) + lane);
#pragma unroll
                        for (int q = 0; q < LIN_FIX_GROUP; ++q) {
                            const float2 t = *(reinterpret_cast<const float2*>(&group[q][64 * c]) + lane);
                            v[q] = fmaf(u.x, t.x, fmaf(u.y, t.y, v[q]));
                        }
                    }
                    const float s = lin_sum8(v, lane);
                    const int q = (lane >> 4 & 1) * 4 + (lane >> 3 & 1) * 2 + (lane >> 2 & 1);
                    if ((lane & 3) == 0 && q < n) {
                        const int mine = list[g0 + q];
                        const size_t m = side == 0 ? (size_t)mine : (size_t)o;
                        const int col = side == 0 ? (int)o : mine;
                        a.out[m * a.N + col] = s + (a.bias ? __ldg(a.bias + col) : 0.f);
                    }
                }
            }
            __syncthreads();
            if (tid == 0) listed = 0;
            __syncthreads();
        };
        if (tid == 0) listed = 0;
        __syncthreads();
        for (int c0 = 0; c0 < ctas; c0 += LIN_THREADS) {
            const bool has = c0 + tid < ctas && marked[c0 + tid] != 0;
            if (tid == 0) found = 0;
            if (!__syncthreads_or(has)) continue;
            if (has) slots[atomicAdd(&found, 1)] = c0 + tid;
            __syncthreads();
            for (int q = 0; q < found; ++q) {
                // this CTA of the split had the rows c * 8 + (0 .. 7), and again every `stride` rows
                const long long c = slots[q], mine = (count - c * 8 + stride - 1) / stride * 8;
                for (long long i0 = 0; i0 < mine; i0 += LIN_THREADS) {
                    const long long i = i0 + tid, r = c * 8 + (i & 7) + (i >> 3) * stride;
                    if (i < mine && r < count && inv[r] == 0.f) list[atomicAdd(&listed, 1)] = (int)r;
                    __syncthreads();
                    const int have = listed;
                    __syncthreads();                     // before the next row is listed
                    if (have > LIN_FIX_LIST - LIN_THREADS) flush();
                }
            }
            __syncthreads();                             // `found` and `slots` have been read
        }
        if (listed) flush();
    }
}

__global__ void __launch_bounds__(LIN_THREADS, 1) lin_gemm_kernel(const __grid_constant__ CUtensorMap tm_x, const __grid_constant__ CUtensorMap tm_w,
                                                                  const __grid_constant__ LinArgs a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    unsigned char* smem = smem_raw + ((1024u - (lr_smem_u32(smem_raw) & 1023u)) & 1023u);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, kbs = a.K / 64;
    unsigned char* ring_p = smem + 2 * LIN_MAX_KB * LIN_BLOCK;
    float* patches = reinterpret_cast<float*>(ring_p + LIN_STAGES * LIN_BLOCK);
    uint64_t* bars = reinterpret_cast<uint64_t*>(patches + LIN_EPI_WARPS * LIN_PATCH / 4);
    const uint32_t wt = lr_smem_u32(smem), ring = lr_smem_u32(ring_p);
    const uint32_t full0 = lr_smem_u32(bars), empty0 = full0 + 8 * LIN_STAGES, wfull0 = empty0 + 8 * LIN_STAGES, wempty0 = wfull0 + 8 * LIN_MAX_KB,
                   tfull0 = wempty0 + 8 * LIN_MAX_KB, tempty0 = tfull0 + 16;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * LIN_STAGES + 2 * LIN_MAX_KB + 4);
    if (threadIdx.x == 0) {
        for (int s = 0; s < 2 * LIN_STAGES + 2 * LIN_MAX_KB + 2; ++s) lr_mbar_init(full0 + 8 * s, 1);
        for (int s = 0; s < 2; ++s) lr_mbar_init(tempty0 + 8 * s, 32 * LIN_EPI_WARPS);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        lr_prefetch_tmap(&tm_x);
        lr_prefetch_tmap(&tm_w);
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(lr_smem_u32(tmem_slot)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = *tmem_slot;
    dependency_wait();
    const long long first = a.items * blockIdx.x / gridDim.x, last = a.items * (blockIdx.x + 1) / gridDim.x;
    const int first_kbs = (kbs + 1) / 2;                 // k blocks of the first half
    bool failed = false, marks = false;

    if (warp == 0) {
        LrRing r;
        uint32_t wph = 1;                                // parity of w's free barriers: the first tile finds them free
        int held = -1;
        for (long long item = first; item < last && !failed; ++item) {
            const int nt = (int)(item / a.mtiles), mt = (int)(item % a.mtiles);
            const bool load_w = nt != held;
            for (int kb = 0; kb < kbs && !failed; ++kb) {
                if (load_w) {
                    if (!lr_mbar_wait(wempty0 + 8 * kb, wph)) { failed = true; break; }
                    if (lr_elect()) {
                        lr_mbar_expect_tx(wfull0 + 8 * kb, 2 * LIN_BLOCK);
                        lr_tma_load_2d(wt + (uint32_t)(2 * kb) * LIN_BLOCK, &tm_w, kb * 64, nt * LIN_BN, wfull0 + 8 * kb);
                        lr_tma_load_2d(wt + (uint32_t)(2 * kb + 1) * LIN_BLOCK, &tm_w, a.K + kb * 64, nt * LIN_BN, wfull0 + 8 * kb);
                    }
                    __syncwarp();
                }
                for (int limb = 0; limb < 2; ++limb, r.next(LIN_STAGES)) {
                    if (!lr_mbar_wait(empty0 + 8 * r.s, r.ph ^ 1u)) { failed = true; break; }
                    if (lr_elect()) {
                        lr_mbar_expect_tx(full0 + 8 * r.s, LIN_BLOCK);
                        lr_tma_load_2d(ring + (uint32_t)r.s * LIN_BLOCK, &tm_x, limb * a.K + kb * 64, mt * 128, full0 + 8 * r.s);
                    }
                    __syncwarp();
                }
            }
            if (load_w) {
                held = nt;
                wph ^= 1u;
            }
        }
    } else if (warp == 1) {
        // f16 operands: the instruction descriptor without the bf16 format bits
        constexpr uint32_t id = (1u << 4) | (8u << 24), wide = id | (256u >> 3) << 17, narrow = id | (128u >> 3) << 17;
        LrRing r;
        uint32_t wph = 0;
        int held = -1, local = 0;
        for (long long item = first; item < last && !failed; ++item, ++local) {
            const int nt = (int)(item / a.mtiles);
            const bool fresh = nt != held, leaves = item + 1 == last || (int)((item + 1) / a.mtiles) != nt;
            for (int kb = 0; kb < kbs && !failed; ++kb) {
                const int half = kb >= first_kbs;
                const uint32_t d = tmem_base + (uint32_t)(half * 256);
                const bool opens = kb == 0 || kb == first_kbs;
                if (opens && !lr_mbar_wait(tempty0 + 8 * half, ((uint32_t)local & 1u) ^ 1u)) { failed = true; break; }
                if (fresh && !lr_mbar_wait(wfull0 + 8 * kb, wph)) { failed = true; break; }
                const uint32_t b_lo = lr_desc_lo(wt) + (uint32_t)(2 * kb) * (LIN_BLOCK >> 4);
                for (int limb = 0; limb < 2; ++limb, r.next(LIN_STAGES)) {
                    if (!lr_mbar_wait(full0 + 8 * r.s, r.ph)) { failed = true; break; }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    if (lr_elect()) {
                        const uint32_t a_lo = lr_desc_lo(ring) + (uint32_t)r.s * (LIN_BLOCK >> 4);
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            if (limb == 0) lr_mma(d, lr_desc(a_lo + 2 * k), lr_desc(b_lo + 2 * k), wide, opens && k == 0 ? 0u : 1u);
                            else lr_mma(d + 128, lr_desc(a_lo + 2 * k), lr_desc(b_lo + 2 * k), narrow, 1u);
                        }
                        lr_commit(empty0 + 8 * r.s);
                        if (leaves && limb) lr_commit(wempty0 + 8 * kb);
                        if (limb && (kb + 1 == first_kbs || kb + 1 == kbs)) lr_commit(tfull0 + 8 * half);
                    }
                    __syncwarp();
                }
            }
            if (fresh) {
                held = nt;
                wph ^= 1u;
            }
        }
    } else {
        const int lg = warp & 3, side = (warp - 2) >> 2; // tensor-memory lane group, and which 32 of the 128 columns
        float* patch = patches + (size_t)(warp - 2) * (LIN_PATCH / 4);
        int local = 0;
        // marked rows anywhere, read while the first sums are computed
        for (int i = threadIdx.x - 64; i < a.ctas_x; i += 32 * LIN_EPI_WARPS) marks |= a.mx[i] != 0;
        for (int i = threadIdx.x - 64; i < a.ctas_w; i += 32 * LIN_EPI_WARPS) marks |= a.mw[i] != 0;
        for (long long item = first; item < last && !failed; ++item, ++local) {
            const int nt = (int)(item / a.mtiles), mt = (int)(item % a.mtiles);
            const int m0 = mt * 128 + lg * 32, n0 = nt * LIN_BN + side * 32;
            const float sx = m0 + lane < a.M ? a.sx[m0 + lane] : 1.f;
            const int rows = min(32, a.M - m0);
            const uint32_t taddr = tmem_base + ((uint32_t)(lg * 32) << 16) + (uint32_t)(side * 32);
            // this item's column factors, in flight while its sums are computed
            const int n = n0 + lane;
            const bool in = n < a.N;
            const float sw = in ? __ldg(a.sw + n) : 1.f, bias = in && a.bias ? __ldg(a.bias + n) : 0.f;
            float acc[32] = {};
            for (int half = kbs > first_kbs ? 0 : 1; half < 2; ++half) {
                const int pair = kbs > first_kbs ? half : 0;         // a single k block has one half
                if (!lr_mbar_wait(tfull0 + 8 * pair, (uint32_t)local & 1u)) { failed = true; break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                float v[32];
                lr_tmem_ld32(taddr + pair * 256 + 128, v);
#pragma unroll
                for (int i = 0; i < 32; ++i) acc[i] = fmaf(v[i], 1.f / LIN_LO_SCALE, acc[i]);
                lr_tmem_ld32(taddr + pair * 256, v);
#pragma unroll
                for (int i = 0; i < 32; ++i) acc[i] += v[i];
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                lr_mbar_arrive(tempty0 + 8 * pair);
            }
            if (failed) break;
            const bool marked = __any_sync(0xffffffffu, sx == 0.f || sw == 0.f);
            float* to = a.out + (size_t)m0 * a.N + n;
#pragma unroll
            for (int h = 0; h < 32; h += 16) {           // half the warp's rows at a time: all 32 would cost two ring stages
                if ((lane & 16) == h) {
#pragma unroll
                    for (int i = 0; i < 32; ++i) patch[(lane & 15) * 33 + i] = acc[i];
                }
                __syncwarp();
                if (!marked && rows == 32) {
#pragma unroll
                    for (int r = 0; r < 16; ++r) {
                        const float o = patch[r * 33 + lane] * __shfl_sync(0xffffffffu, sx, h + r) * sw + bias;
                        if (in) to[(size_t)(h + r) * a.N] = o;
                    }
                } else {
                    for (int r = h; r < min(rows, h + 16); ++r) {
                        const float s = __shfl_sync(0xffffffffu, sx, r), o = patch[(r - h) * 33 + lane] * s * sw + bias;
                        if (in && s != 0.f && sw != 0.f) to[(size_t)r * a.N] = o;
                    }
                }
                __syncwarp();
            }
        }
    }
    if (failed) atomicOr(&g_linear_error, 1u);
    const bool whole = !__syncthreads_or(failed);        // after a timeout copies may still land in the ring
    if (__syncthreads_or(marks) && whole) lin_fix(a, ring_p);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
}

int linear_error_fetch() {
    unsigned v = 0, zero = 0;
    if (cudaMemcpyFromSymbol(&v, g_linear_error, sizeof(v)) != cudaSuccess) return -1;
    if (v) cudaMemcpyToSymbol(g_linear_error, &zero, sizeof(zero));
    return (int)v;
}

// workspace: limbs, inverse scales and mark counts of w, then those of x
static size_t lin_limbs(int64_t rows, int K) { return (size_t)rows * 2 * K * 2; }
static size_t lin_scales(int64_t rows) { return ((size_t)rows * 4 + 255) & ~size_t(255); }
static int lin_split_ctas(int rows) { return (int)min((int64_t)8 * sm_count(), ((int64_t)rows + 7) / 8); }
struct LinPart {
    __half* limbs;
    float* inv;
    int* marked;
};
static LinPart lin_part(char*& at, int rows, int K) {
    LinPart p;
    p.limbs = reinterpret_cast<__half*>(at);
    p.inv = reinterpret_cast<float*>(at += lin_limbs(rows, K));
    p.marked = reinterpret_cast<int*>(at += lin_scales(rows));
    at += lin_scales(lin_split_ctas(rows));
    return p;
}

bool linear_f32_supported(int K) { return K > 0 && K % 64 == 0 && K <= 64 * LIN_MAX_KB; }

// w's half of the work, which needs nothing but w; the next kernel may start beside it
int linear_f32_weights(const float* w, int N, int K, void* workspace, cudaStream_t st) {
    char* at = static_cast<char*>(workspace);
    const LinPart p = lin_part(at, N, K);
    lin_split_kernel<<<lin_split_ctas(N), 256, 0, st>>>(w, N, K, p.limbs, p.inv, p.marked);
    count_launch(1);
    return check_launch("lin_split_kernel");
}

// the rest, behind a kernel that itself has waited for linear_f32_weights
int linear_f32_rows(const float* x, const float* w, const float* bias, float* out, int M, int N, int K, void* workspace, cudaStream_t st) {
    char* at = static_cast<char*>(workspace);
    const LinPart pw = lin_part(at, N, K), px = lin_part(at, M, K);
    CUtensorMap tm_x, tm_w;
    int rc = make_tmap_of(&tm_x, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, px.limbs, M, 2 * K, 128);
    if (rc == PIKV_OK) rc = make_tmap_of(&tm_w, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, pw.limbs, N, 2 * K, 128);
    if (rc != PIKV_OK) return rc;
    if (!allow_smem<lin_gemm_kernel>()) return check_launch("linear_f32 smem attribute");
    LinArgs a = {x, w, bias, px.inv, pw.inv, px.marked, pw.marked, lin_split_ctas(M), lin_split_ctas(N), out, M, N, K, ceil_div(M, 128), 0};
    a.items = (long long)ceil_div(N, LIN_BN) * a.mtiles;
    const int sms = sm_count();
    launch_dependent(lin_split_kernel, dim3((unsigned)lin_split_ctas(M)), 256, 0, st, x, M, K, px.limbs, px.inv, px.marked);
    launch_dependent(lin_gemm_kernel, dim3((unsigned)min((long long)sms, a.items)), LIN_THREADS, LIN_SMEM, st, tm_x, tm_w, a);
    count_launch(2);
    return check_launch("linear_f32");
}

}  // namespace pikv

using namespace pikv;

extern "C" {

size_t pikv_linear_f32_workspace_bytes(int32_t M, int32_t N, int32_t K) {
    if (M <= 0 || N <= 0 || K <= 0) return 0;
    return lin_limbs((int64_t)M + N, K) + lin_scales(M) + lin_scales(N) + lin_scales(lin_split_ctas(M)) + lin_scales(lin_split_ctas(N));
}

int pikv_linear_f32(const float* x, const float* w, const float* bias, float* out, int32_t M, int32_t N, int32_t K, void* workspace,
                    size_t workspace_bytes, pikv_stream_t stream) {
    PIKV_REQUIRE(x && w && out && workspace, PIKV_EINVAL, "linear_f32: null pointer");
    PIKV_REQUIRE(M > 0 && N > 0 && K > 0, PIKV_EINVAL, "linear_f32: bad sizes");
    PIKV_REQUIRE(linear_f32_supported(K), PIKV_EUNSUPPORTED, "linear_f32: K=%d must be a multiple of 64 up to %d", K, 64 * LIN_MAX_KB);
    PIKV_REQUIRE((uintptr_t)x % 16 == 0 && (uintptr_t)w % 16 == 0 && (uintptr_t)workspace % 256 == 0 && (uintptr_t)out % 4 == 0, PIKV_EINVAL,
                 "linear_f32: misaligned pointer");
    PIKV_REQUIRE(workspace_bytes >= pikv_linear_f32_workspace_bytes(M, N, K), PIKV_EINVAL, "linear_f32: workspace of %zu bytes", workspace_bytes);
    PIKV_REQUIRE(M <= INT32_MAX - 128 && N <= INT32_MAX - 128, PIKV_ELIMIT, "linear_f32: too many rows");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int rc = linear_f32_weights(w, N, K, workspace, st);
    return rc != PIKV_OK ? rc : linear_f32_rows(x, w, bias, out, M, N, K, workspace, st);
}

}  // extern "C"
