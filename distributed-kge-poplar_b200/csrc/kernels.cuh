// Device kernels of the BESS training step for sm_100a.
//
// Naming follows the reference's step (src/poplar_kge.cpp:664-707): rows of the stacked
// shard table are gathered by `remote`, turned into hidden vectors, looked up by `head`
// and `a2a`, exchanged, scored against the batch-shared tails, and the gradients flow
// back the same way into a row-wise Adam update.  All arithmetic is fp32.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <atomic>

#include "adam.cuh"
#include "exchange.cuh"
#include "pdl.cuh"

namespace kge {

enum ScoreFn : int { SCORE_TRANSE = 0, SCORE_DISTMULT = 1, SCORE_COMPLEX = 2, SCORE_ROTATE = 3, SCORE_TRANSH = 4 };
// TransE, RotatE and TransH score by gamma - distance (src/poplar_kge.cpp:492-499, 532-537, 552-565); the others by the raw product.
__host__ __device__ inline bool score_is_gamma_minus_distance(int score_fn) { return score_fn == SCORE_TRANSE || score_fn == SCORE_ROTATE || score_fn == SCORE_TRANSH; }

// RotatE's relation row holds one angle per complex pair.  The reference casts the angles to
// float16 and takes sine and cosine in float16 (src/poplar_kge.cpp:522-525): restated as the
// correctly rounded float16 of the exact value (double-precision sin / cos of the rounded angle).
__device__ __forceinline__ void rotate_sin_cos(float angle, float& s, float& c) {
    const double theta = (double)__half2float(__float2half_rn(angle));
    s = __half2float(__double2half(sin(theta)));
    c = __half2float(__double2half(cos(theta)));
}
__device__ __forceinline__ float round_to_half(float x) { return __half2float(__float2half_rn(x)); }
enum DistFn : int { DIST_L1 = 0, DIST_L2 = 1, DIST_DOT = 2 };
enum LossFn : int { LOSS_LOGSIGMOID = 0, LOSS_SOFTMAX = 1 };

// What belongs to each of the shards of one process that a launch works on, one per blockIdx.y (.z where y is taken).  The
// kernels of a step are short and mostly far too small to fill 148 SMs, so the shards of a process share every launch.
// More shards go in groups of so many, side by side on streams (Engine::shards_fork).  Four: a contraction's parameters are 8 KB
// with that many, which every launch copies; larger groups have not been measured.
constexpr int kShardBatch = 4;
template <class A>
struct ShardArgs {
    A s[kShardBatch];
};

// Byte layout of one table row: value | adam_m | sqrt(adam_v) | feature
// (src/poplar_kge.cpp:405-417).  Every segment starts on a 16-byte boundary and
// row_bytes is a multiple of 16, so 128-bit accesses are always aligned.
struct RowLayout {
    uint32_t row_bytes;
    uint32_t off_m;
    uint32_t off_q;
    uint32_t off_feat;
    uint32_t d;
    uint32_t f;
    // 1: the value segment holds bfloat16 while adam_m and sqrt(adam_v) keep the state type (bf16
    // embeddings with fp32 optimiser state; the reference has one type per row, src/poplar_kge.cpp:405-417)
    uint32_t value_bf16;
};

__device__ __forceinline__ float load_as_float(const float* p) { return *p; }
__device__ __forceinline__ float load_as_float(const __half* p) { return __half2float(*p); }
__device__ __forceinline__ void store_from_float(float* p, float v) { *p = v; }
__device__ __forceinline__ void store_from_float(__half* p, float v) { *p = __float2half_rn(v); }

__device__ __forceinline__ float load_as_float(const __nv_bfloat16* p) { return __bfloat162float(*p); }
__device__ __forceinline__ void store_from_float(__nv_bfloat16* p, float v) { *p = __float2bfloat16_rn(v); }
__device__ __forceinline__ float4 load4(const __nv_bfloat16* p) {
    const uint2 raw = *reinterpret_cast<const uint2*>(p);
    const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.x));
    const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.y));
    return make_float4(a.x, a.y, b.x, b.y);
}
__device__ __forceinline__ void store4(__nv_bfloat16* p, float4 v) {
    const __nv_bfloat162 lo = __floats2bfloat162_rn(v.x, v.y), hi = __floats2bfloat162_rn(v.z, v.w);
    uint2 raw;
    raw.x = *reinterpret_cast<const uint32_t*>(&lo);
    raw.y = *reinterpret_cast<const uint32_t*>(&hi);
    *reinterpret_cast<uint2*>(p) = raw;
}
// Element c of a row's value segment, whose type the layout names.
template <class ST>
__device__ __forceinline__ float load_value(const RowLayout& L, const uint8_t* row, int c) {
    return L.value_bf16 ? load_as_float(reinterpret_cast<const __nv_bfloat16*>(row) + c) : load_as_float(reinterpret_cast<const ST*>(row) + c);
}
template <class ST>
__device__ __forceinline__ void store_value(const RowLayout& L, uint8_t* row, int c, float v) {
    if (L.value_bf16) store_from_float(reinterpret_cast<__nv_bfloat16*>(row) + c, v);
    else store_from_float(reinterpret_cast<ST*>(row) + c, v);
}

// Four consecutive elements starting at an element index that is a multiple of 4.
__device__ __forceinline__ float4 load4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 load4(const __half* p) {
    uint2 raw = *reinterpret_cast<const uint2*>(p);
    __half2 lo = *reinterpret_cast<__half2*>(&raw.x);
    __half2 hi = *reinterpret_cast<__half2*>(&raw.y);
    float2 a = __half22float2(lo), b = __half22float2(hi);
    return make_float4(a.x, a.y, b.x, b.y);
}
__device__ __forceinline__ void store4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
__device__ __forceinline__ void store4(__half* p, float4 v) {
    __half2 lo = __floats2half2_rn(v.x, v.y), hi = __floats2half2_rn(v.z, v.w);
    uint2 raw;
    raw.x = *reinterpret_cast<uint32_t*>(&lo);
    raw.y = *reinterpret_cast<uint32_t*>(&hi);
    *reinterpret_cast<uint2*>(p) = raw;
}

// Block-wide reductions with a fixed tree, so results do not depend on scheduling.
template <int THREADS>
__device__ __forceinline__ float block_sum(float v, float* scratch) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    __syncthreads();
    if (lane == 0) scratch[warp] = v;
    __syncthreads();
    float total = 0.f;
#pragma unroll
    for (int w = 0; w < THREADS / 32; ++w) total += scratch[w];
    return total;
}
template <int THREADS>
__device__ __forceinline__ float block_max(float v, float* scratch) {
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    __syncthreads();
    if (lane == 0) scratch[warp] = v;
    __syncthreads();
    float total = scratch[0];
#pragma unroll
    for (int w = 1; w < THREADS / 32; ++w) total = fmaxf(total, scratch[w]);
    return total;
}

// Holds the stream for about `cycles` clock ticks (bounded by the argument), so that the host can
// queue the launches that follow before the first of them starts: per-kernel event timing then
// measures kernels, not the host's launch rate.
static __global__ void k_delay(long long cycles) {
    const long long start = clock64();
    while (clock64() - start < cycles) {
    }
}

// ---------------------------------------------------------------------------
// The step's row gather (fr::Buffer::read through getEntityData, src/fructose/fructose.cpp:790-798,
// src/poplar_kge.cpp:405-410): the R rows named by `remote` are copied whole, with 128-bit
// accesses, from the shard table (tens of gigabytes, so every row is a DRAM and TLB miss) into a
// compact buffer with the same row layout.  One warp per row with all of its loads in flight
// before the first store; everything after this kernel in the step reads the compact,
// L2-resident copy.
// What the tensor-core contractions read of a gathered row's features: fp16 features are widened
// to fp32 (exact, one TF32 plane) into feat_wide [R, feat_stride]; fp32 features are read in place
// (the compact copy is their upper plane) and only their lower plane feat_lo is written.  Both null:
// nothing extra.
struct FeaturePlanes {
    float* wide;   // fp16 features as fp32
    float* lo;     // lower TF32 plane of fp32 features
    uint32_t stride;    // floats per row of either
    uint32_t off_feat;  // byte offset of the features in a table row (multiple of 16)
};

__device__ __forceinline__ float tf32_upper(float x) { return __uint_as_float(__float_as_uint(x) & 0xFFFFE000u); }
__device__ __forceinline__ float tf32_lower(float x) { return tf32_upper(x - tf32_upper(x)); }
__device__ __forceinline__ float4 tf32_lower4(float4 v) { return make_float4(tf32_lower(v.x), tf32_lower(v.y), tf32_lower(v.z), tf32_lower(v.w)); }

struct GatherArgs {
    const uint8_t* table;
    const uint32_t* remote;
    uint8_t* rows_c;
    FeaturePlanes fp;
};

static __global__ void __launch_bounds__(256) k_gather_step_rows(const __grid_constant__ ShardArgs<GatherArgs> shards, uint32_t row_bytes, int R) {
    grid_dependency_sync();
    const GatherArgs& g = shards.s[blockIdx.y];
    const FeaturePlanes& fp = g.fp;
    const uint8_t* __restrict__ table = g.table;
    const uint32_t* __restrict__ remote = g.remote;
    uint8_t* __restrict__ rows_c = g.rows_c;
    const int r = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (r >= R) return;
    const uint4* __restrict__ src = reinterpret_cast<const uint4*>(table + (size_t)remote[r] * row_bytes);
    uint4* __restrict__ dst = reinterpret_cast<uint4*>(rows_c + (size_t)r * row_bytes);
    const int chunks = (int)(row_bytes >> 4), feat_chunk0 = (int)(fp.off_feat >> 4);
    for (int c0 = lane; c0 < chunks; c0 += 32 * 8) {
        uint4 v[8];
#pragma unroll
        for (int u = 0; u < 8; ++u)
            if (c0 + 32 * u < chunks) v[u] = src[c0 + 32 * u];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const int c = c0 + 32 * u;
            if (c >= chunks) continue;
            dst[c] = v[u];
            if (c < feat_chunk0) continue;
            if (fp.wide) {  // 8 fp16 values
                const int f = (c - feat_chunk0) * 8;
                const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&v[u].x)), b = __half22float2(*reinterpret_cast<const __half2*>(&v[u].y));
                const float2 cc = __half22float2(*reinterpret_cast<const __half2*>(&v[u].z)), d = __half22float2(*reinterpret_cast<const __half2*>(&v[u].w));
                float* o = fp.wide + (size_t)r * fp.stride + f;
                if (f < (int)fp.stride) *reinterpret_cast<float4*>(o) = make_float4(a.x, a.y, b.x, b.y);
                if (f + 4 < (int)fp.stride) *reinterpret_cast<float4*>(o + 4) = make_float4(cc.x, cc.y, d.x, d.y);
            } else if (fp.lo) {  // 4 fp32 values
                const int f = (c - feat_chunk0) * 4;
                if (f < (int)fp.stride)
                    *reinterpret_cast<float4*>(fp.lo + (size_t)r * fp.stride + f) =
                        tf32_lower4(make_float4(__uint_as_float(v[u].x), __uint_as_float(v[u].y), __uint_as_float(v[u].z), __uint_as_float(v[u].w)));
            }
        }
    }
}

// ---------------------------------------------------------------------------
// hidden = value + feature . W   (src/poplar_kge.cpp:439-467 with the gather of :405-410
// folded in).  A [R, F] is read straight from the gathered table rows; W is [F, D].
// Rows are table[remote[m]], or the consecutive rows row_base + m when `remote` is null
// (the tail batches of predict, src/poplar_kge.cpp:836-839).
// blockIdx.z picks the feature network (head / tail) when they are not shared.
// 64x64 output tile, 16-deep k slices, 256 threads with a 4x4 register tile each.
template <class ST, class FT>
__global__ void __launch_bounds__(256)
k_hidden(const uint8_t* __restrict__ table, RowLayout L, const uint32_t* __restrict__ remote,
         uint32_t row_base, int R, const float* __restrict__ W0, const float* __restrict__ W1,
         float* __restrict__ out0, float* __restrict__ out1) {
    grid_dependency_sync();
    constexpr int BM = 64, BN = 64, BK = 16;
    __shared__ __align__(16) float As[BK][BM + 4];
    __shared__ __align__(16) float Bs[BK][BN];
    const float* __restrict__ W = blockIdx.z ? W1 : W0;
    float* __restrict__ out = blockIdx.z ? out1 : out0;
    const int D = L.d, F = L.f;
    const int t = threadIdx.x, tx = t & 15, ty = t >> 4;
    const int m0 = blockIdx.x * BM, n0 = blockIdx.y * BN;

    const int a_row = t >> 2, a_k = (t & 3) * 4;
    const bool a_ok = m0 + a_row < R;
    const FT* __restrict__ a_ptr = nullptr;
    if (a_ok) {
        const size_t row = remote ? remote[m0 + a_row] : row_base + (uint32_t)(m0 + a_row);
        a_ptr = reinterpret_cast<const FT*>(table + row * L.row_bytes + L.off_feat);
    }
    const int b_k = t >> 4, b_n = (t & 15) * 4;
    const bool d_vec = (D & 3) == 0;

    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;

    for (int k0 = 0; k0 < F; k0 += BK) {
        float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
        const int ka = k0 + a_k;
        if (a_ok) {
            if (ka + 3 < F) {
                a = load4(a_ptr + ka);
            } else {
                if (ka + 0 < F) a.x = load_as_float(a_ptr + ka + 0);
                if (ka + 1 < F) a.y = load_as_float(a_ptr + ka + 1);
                if (ka + 2 < F) a.z = load_as_float(a_ptr + ka + 2);
            }
        }
        float4 b = make_float4(0.f, 0.f, 0.f, 0.f);
        const int kb = k0 + b_k, nb = n0 + b_n;
        if (kb < F) {
            const float* wp = W + (size_t)kb * D + nb;
            if (d_vec && nb + 3 < D) {
                b = load4(wp);
            } else {
                if (nb + 0 < D) b.x = wp[0];
                if (nb + 1 < D) b.y = wp[1];
                if (nb + 2 < D) b.z = wp[2];
                if (nb + 3 < D) b.w = wp[3];
            }
        }
        __syncthreads();
        As[a_k + 0][a_row] = a.x;
        As[a_k + 1][a_row] = a.y;
        As[a_k + 2][a_row] = a.z;
        As[a_k + 3][a_row] = a.w;
        store4(&Bs[b_k][b_n], b);
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < BK; ++kk) {
            const float4 av = load4(&As[kk][ty * 4]);
            const float4 bv = load4(&Bs[kk][tx * 4]);
            const float ar[4] = {av.x, av.y, av.z, av.w};
            const float br[4] = {bv.x, bv.y, bv.z, bv.w};
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(ar[i], br[j], acc[i][j]);
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int m = m0 + ty * 4 + i;
        if (m >= R) continue;
        const size_t row = remote ? remote[m] : row_base + (uint32_t)m;
        const uint8_t* vp = table + row * L.row_bytes;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int n = n0 + tx * 4 + j;
            if (n < D) out[(size_t)m * D + n] = load_value<ST>(L, vp, n) + acc[i][j];
        }
    }
}

// ---------------------------------------------------------------------------
// The lookups of the rows with many lookups (the parts k_prepare_segments cut them into for the
// entity update): block p copies hidden row parts[p].x to the lookups perm[parts[p].y .. parts[p].z),
// heads (+ or * their relation row) into `pred`, tails into the owning shards' buffers, each with
// its companion plane.  The hidden kernel's routing epilogue leaves these rows out, so that no
// single block stores hundreds of copies of one row; this kernel then publishes the tails hand-over.
// TransE and DistMult (the score functions whose routing is fused).
static __global__ void __launch_bounds__(256)
k_route_heavy(const float* __restrict__ hid_h, const float* __restrict__ hid_t, const uint4* __restrict__ parts,
              const uint32_t* __restrict__ count, const uint32_t* __restrict__ perm, const uint32_t* __restrict__ relation,
              const float* __restrict__ rel_table, float* const* __restrict__ send_dst, float* const* __restrict__ send_lo_dst,
              float* __restrict__ pred, float* __restrict__ pred_lo, int B, int a2a, int D, int score_fn, int lo_bf16, ExchangeSync sync) {
    grid_dependency_sync();
    if (blockIdx.x < *count) {
        // every (lookup, 4 columns) pair is one unit of work: all of a part's copies are in flight at once
        const uint4 part = parts[blockIdx.x];
        const int quads = D / 4, n_units = (int)(part.z - part.y) * quads;
        for (int u = threadIdx.x; u < n_units; u += blockDim.x) {
            const uint32_t q = part.y + (uint32_t)(u / quads), e = perm[q];
            const int c = (u % quads) * 4;
            const bool head = e < (uint32_t)B;
            float4 o = load4((head ? hid_h : hid_t) + (size_t)part.x * D + c);
            float *dst, *dst_lo;
            if (head) {
                const float4 r = load4(rel_table + (size_t)relation[e] * D + c);
                o = score_fn == SCORE_TRANSE ? make_float4(o.x + r.x, o.y + r.y, o.z + r.z, o.w + r.w)
                                             : make_float4(o.x * r.x, o.y * r.y, o.z * r.z, o.w * r.w);
                dst = pred + (size_t)e * D;
                dst_lo = lo_bf16 ? pred_lo + (size_t)e * D / 2 : pred_lo + (size_t)e * D;
            } else {
                const uint32_t j = e - (uint32_t)B, shard = j / (uint32_t)a2a, slot = j - shard * (uint32_t)a2a;
                dst = send_dst[shard] + (size_t)slot * D;
                dst_lo = lo_bf16 ? send_lo_dst[shard] + (size_t)slot * D / 2 : send_lo_dst[shard] + (size_t)slot * D;
            }
            store4(dst + c, o);
            if (lo_bf16) store4(reinterpret_cast<__nv_bfloat16*>(dst_lo) + c, o);
            else store4(dst_lo + c, tf32_lower4(o));
        }
    }
    exchange_signal(sync, XCHG_TAILS, gridDim.x);  // the tail rows are in their consumers' memory
}

// ---------------------------------------------------------------------------
// raw[i, j] = sum_k |p_ik - t_jk|  (L1),  sqrt(sum_k (p_ik - t_jk)^2)  (L2),  sum_k p_ik t_jk (dot)
// src/poplar_extensions/distance.cpp:70-104,151-185 and the codelets' l1dist / l2dist;
// the dot form is matMul(a, b^T) of src/poplar_kge.cpp:478-479.
// 32x64 output tile, 32-deep k slices staged in shared memory k-major, 128 threads, 4x4 each.
struct ScoreArgs {
    const float *P, *Tl;
    float* raw;
};

template <int FN>
__global__ void __launch_bounds__(128) k_score(const __grid_constant__ ShardArgs<ScoreArgs> shards, int B, int T, int D, int ld) {
    grid_dependency_sync();
    const float* __restrict__ P = shards.s[blockIdx.z].P;
    const float* __restrict__ Tl = shards.s[blockIdx.z].Tl;
    float* __restrict__ raw = shards.s[blockIdx.z].raw;
    constexpr int BM = 32, BN = 64, BK = 32;
    __shared__ __align__(16) float Ps[BK][BM];
    __shared__ __align__(16) float Ts[BK][BN];
    const int t = threadIdx.x, tx = t & 15, ty = t >> 4;
    const int i0 = blockIdx.y * BM, j0 = blockIdx.x * BN;
    const bool vec = (D & 3) == 0;
    float acc[4][4];
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) acc[a][b] = 0.f;

    for (int k0 = 0; k0 < D; k0 += BK) {
        __syncthreads();
#pragma unroll
        for (int it = 0; it < 2; ++it) {
            const int idx = t + it * 128, row = idx & 31, k4 = (idx >> 5) * 4;
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            const int gi = i0 + row, gk = k0 + k4;
            if (gi < B) {
                const float* src = P + (size_t)gi * D + gk;
                if (vec && gk + 3 < D) {
                    v = load4(src);
                } else {
                    if (gk + 0 < D) v.x = src[0];
                    if (gk + 1 < D) v.y = src[1];
                    if (gk + 2 < D) v.z = src[2];
                    if (gk + 3 < D) v.w = src[3];
                }
            }
            Ps[k4 + 0][row] = v.x;
            Ps[k4 + 1][row] = v.y;
            Ps[k4 + 2][row] = v.z;
            Ps[k4 + 3][row] = v.w;
        }
#pragma unroll
        for (int it = 0; it < 4; ++it) {
            const int idx = t + it * 128, row = idx & 63, k4 = (idx >> 6) * 4;
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            const int gj = j0 + row, gk = k0 + k4;
            if (gj < T) {
                const float* src = Tl + (size_t)gj * D + gk;
                if (vec && gk + 3 < D) {
                    v = load4(src);
                } else {
                    if (gk + 0 < D) v.x = src[0];
                    if (gk + 1 < D) v.y = src[1];
                    if (gk + 2 < D) v.z = src[2];
                    if (gk + 3 < D) v.w = src[3];
                }
            }
            Ts[k4 + 0][row] = v.x;
            Ts[k4 + 1][row] = v.y;
            Ts[k4 + 2][row] = v.z;
            Ts[k4 + 3][row] = v.w;
        }
        __syncthreads();
#pragma unroll 8
        for (int kk = 0; kk < BK; ++kk) {
            const float4 pv = load4(&Ps[kk][ty * 4]);
            const float4 tv = load4(&Ts[kk][tx * 4]);
            const float pr[4] = {pv.x, pv.y, pv.z, pv.w};
            const float tr[4] = {tv.x, tv.y, tv.z, tv.w};
#pragma unroll
            for (int a = 0; a < 4; ++a)
#pragma unroll
                for (int b = 0; b < 4; ++b) {
                    if (FN == DIST_L1) {
                        acc[a][b] += fabsf(pr[a] - tr[b]);
                    } else if (FN == DIST_L2) {
                        const float d = pr[a] - tr[b];
                        acc[a][b] = fmaf(d, d, acc[a][b]);
                    } else {
                        acc[a][b] = fmaf(pr[a], tr[b], acc[a][b]);
                    }
                }
        }
    }
#pragma unroll
    for (int a = 0; a < 4; ++a) {
        const int i = i0 + ty * 4 + a;
        if (i >= B) continue;
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            const int j = j0 + tx * 4 + b;
            if (j < T) raw[(size_t)i * ld + j] = FN == DIST_L2 ? sqrtf(acc[a][b]) : acc[a][b];
        }
    }
}

// The same scores for rows that allow 16-byte copies (D a multiple of 4, 16-byte aligned bases).  A block owns 64 x 4 NB
// outputs and its 8 warps take 32 rows each in four groups that divide k in chunks of 32: a group copies its chunks of both
// operands into its own part of shared memory (asynchronous 16-byte copies, row-major with a stride of 36 floats, which
// keeps the 128-bit reads below free of bank conflicts), one ahead of the one it adds up in register tiles of 4 x NB per lane.
// A chunk is summed by itself (with the chunk eight further on, and so on), and the chunks' sums are added in order at the
// end: the order is part of an L1 model's result (see k_pair_bwd).  Bound by FP32 issue, two instructions per pair of
// elements (66 % of the slots of the SMs that have a block), and by the operands' way from L2, of which wider tiles need less; the width is chosen so that the blocks come to
// whole waves of 148.  512 x 768 x 256 L2 scores: 13.8 us back to back with 48 columns a block, 16.4 with 64, 17.9 with 32.
// With 32 x 32 outputs per block, its 8 warps dividing k and no chunk ahead, steps took (us, before -> after) TransE-L2 at that
// size 72.6 -> 71.3, two shards of it 113.2 -> 109.6, RotatE-L2 256 x 1536 x 256 86.1 -> 82.9, four shards of 256 x 512 x 100
// L1 scores 63.4 -> 59.0.  (Two blocks per SM, and two or four steps of k unrolled, were no faster.)
constexpr int kScoreStride = 36, kScoreRows = 64, kScoreGroups = 4;
__device__ __forceinline__ void score_copy16(float* dst_smem, const float* src) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst_smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src));
}
template <int FN>
__device__ __forceinline__ void score_add(float& sum, float4 p, float4 t) {
    const float pr[4] = {p.x, p.y, p.z, p.w}, tr[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        if (FN == DIST_L1) {
            sum += fabsf(pr[c] - tr[c]);
        } else if (FN == DIST_L2) {
            const float d = pr[c] - tr[c];
            sum = fmaf(d, d, sum);
        } else {
            sum = fmaf(pr[c], tr[c], sum);
        }
    }
}
template <int NB>
constexpr int kScoreStage = (kScoreRows + 4 * NB) * kScoreStride;  // floats of a group's chunk
template <int NB>
constexpr size_t kScoreBlockSmem = (size_t)kScoreGroups * 2 * kScoreStage<NB> * sizeof(float);

// WIDE: more than four chunks of k.
template <int FN, int NB, bool WIDE>
__global__ void __launch_bounds__(256, 1)
k_score_block(const __grid_constant__ ShardArgs<ScoreArgs> shards, int B, int T, int D, int ld, ExchangeSync sync) {
    const float* __restrict__ P = shards.s[blockIdx.z].P;
    const float* __restrict__ Tl = shards.s[blockIdx.z].Tl;
    float* __restrict__ raw = shards.s[blockIdx.z].raw;
    grid_dependency_sync();
    exchange_wait(sync, XCHG_TAILS);  // the tail rows come from the other processes
    extern __shared__ __align__(16) float score_smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, group = warp >> 1, in_group = threadIdx.x & 63;
    const int i0 = blockIdx.y * kScoreRows, j0 = blockIdx.x * 4 * NB, n_chunks = (D + 31) / 32;
    float* const mine = score_smem + group * 2 * kScoreStage<NB>;
    auto stage = [&](int chunk, float* to) {
        const int k0 = chunk * 32, k4 = (in_group & 7) * 4;
#pragma unroll 4
        for (int row = in_group >> 3; row < kScoreRows + 4 * NB; row += 8) {
            const bool is_p = row < kScoreRows;
            const int g = is_p ? i0 + row : j0 + row - kScoreRows;
            float* d = to + row * kScoreStride + k4;
            if (g < (is_p ? B : T) && k0 + k4 < D) score_copy16(d, (is_p ? P : Tl) + (size_t)g * D + k0 + k4);
            else *reinterpret_cast<float4*>(d) = make_float4(0.f, 0.f, 0.f, 0.f);
        }
    };
    auto group_sync = [&] { asm volatile("bar.sync %0, 64;" ::"r"(group + 1) : "memory"); };
    auto commit = [&] { asm volatile("cp.async.commit_group;" ::: "memory"); };
    constexpr int kSets = WIDE ? 2 : 1;  // the sums of the group's chunks that are even and odd among its own
    float acc[kSets][4][NB];
#pragma unroll
    for (int s = 0; s < kSets; ++s)
#pragma unroll
        for (int a = 0; a < 4; ++a)
#pragma unroll
            for (int b = 0; b < NB; ++b) acc[s][a][b] = 0.f;
    const int ty = lane >> 2, tx = lane & 3;  // rows ty + 8a of the warp's 32, columns tx + 4b
    auto add_chunk = [&](int chunk, const float* from, float (&sums)[4][NB]) {
        const float* Ps = from + ((warp & 1) * 32 + ty) * kScoreStride;
        const float* Ts = from + (kScoreRows + tx) * kScoreStride;
        const int k_end = min(32, D - chunk * 32);
#pragma unroll 1
        for (int k4 = 0; k4 < k_end; k4 += 4) {
            float4 pv[4];
#pragma unroll
            for (int a = 0; a < 4; ++a) pv[a] = load4(Ps + 8 * a * kScoreStride + k4);
#pragma unroll
            for (int b = 0; b < NB; ++b) {
                const float4 tv = load4(Ts + 4 * b * kScoreStride + k4);
#pragma unroll
                for (int a = 0; a < 4; ++a) score_add<FN>(sums[a][b], pv[a], tv);
            }
        }
    };
    if (group < n_chunks) stage(group, mine);
    commit();
    if (WIDE && group + kScoreGroups < n_chunks) stage(group + kScoreGroups, mine + kScoreStage<NB>);
    commit();
    for (int chunk = group; chunk < n_chunks; chunk += 2 * kScoreGroups) {
#pragma unroll
        for (int s = 0; s < kSets; ++s) {
            const int c = chunk + s * kScoreGroups;
            if (c >= n_chunks) break;
            asm volatile("cp.async.wait_group 1;" ::: "memory");
            group_sync();
            add_chunk(c, mine + s * kScoreStage<NB>, acc[s]);
            if (WIDE && c + 2 * kScoreGroups < n_chunks) {
                group_sync();
                stage(c + 2 * kScoreGroups, mine + s * kScoreStage<NB>);
            }
            commit();
        }
    }
    // add the chunks' sums: red[chunk modulo 8][row][column]
    __syncthreads();
    constexpr int kPitch = 4 * NB + 4;
    static_assert((WIDE ? 8 : 4) * kScoreRows * kPitch <= kScoreGroups * 2 * kScoreStage<NB>, "the sums fit where the operands were");
#pragma unroll
    for (int s = 0; s < kSets; ++s)
        if (group + s * kScoreGroups < n_chunks) {
            float* red = score_smem + ((group + s * kScoreGroups) * kScoreRows + (warp & 1) * 32 + ty) * kPitch + tx;
#pragma unroll
            for (int a = 0; a < 4; ++a)
#pragma unroll
                for (int b = 0; b < NB; ++b) red[8 * a * kPitch + 4 * b] = acc[s][a][b];
        }
    __syncthreads();
    const int n_sums = min(n_chunks, 8);
    const bool vec = (ld & 3) == 0;
#pragma unroll
    for (int it = 0; it < kScoreRows * NB / 256; ++it) {
        const int q = threadIdx.x + it * 256, row = q / NB, col = q % NB * 4, i = i0 + row, j = j0 + col;
        float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int w = 0; w < (WIDE ? 8 : 4); ++w) {
            if (w >= n_sums) break;
            const float4 v = load4(score_smem + (w * kScoreRows + row) * kPitch + col);
            sum[0] += v.x; sum[1] += v.y; sum[2] += v.z; sum[3] += v.w;
        }
        if (i >= B || j >= T) continue;
        float* dst = raw + (size_t)i * ld + j;
#pragma unroll
        for (int u = 0; u < 4; ++u) sum[u] = FN == DIST_L2 ? sqrtf(sum[u]) : sum[u];
        if (vec && j + 3 < T) {
            store4(dst, make_float4(sum[0], sum[1], sum[2], sum[3]));
        } else {
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (j + u < T) dst[u] = sum[u];
        }
    }
}

template <int FN, int NB, bool WIDE>
inline cudaError_t launch_score_block(const ShardArgs<ScoreArgs>& shards, int n_shards, int B, int T, int D, int ld, cudaStream_t stream, const ExchangeSync& sync) {
    static std::atomic<bool> configured[kMaxDeviceOrdinals] = {};  // one attribute call per instantiation and device is enough
    const int slot = current_device_slot();
    if (slot < 0 || !configured[slot]) {
        const cudaError_t err = cudaFuncSetAttribute(k_score_block<FN, NB, WIDE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kScoreBlockSmem<NB>);
        if (err != cudaSuccess) return err;
        if (slot >= 0) configured[slot] = true;
    }
    const dim3 grid((T + 4 * NB - 1) / (4 * NB), (B + kScoreRows - 1) / kScoreRows, (unsigned)n_shards);
    return launch_dependent(k_score_block<FN, NB, WIDE>, grid, dim3(256), kScoreBlockSmem<NB>, stream, shards, B, T, D, ld, sync);
}
template <int FN, int NB>
inline cudaError_t launch_score_block(const ShardArgs<ScoreArgs>& shards, int n_shards, int B, int T, int D, int ld, cudaStream_t stream, const ExchangeSync& sync) {
    if (D > 32 * kScoreGroups) return launch_score_block<FN, NB, true>(shards, n_shards, B, T, D, ld, stream, sync);
    return launch_score_block<FN, NB, false>(shards, n_shards, B, T, D, ld, stream, sync);
}

// The same scores where there are enough of them to fill the GPU with tiles (ranking): a block owns 64 x 128 outputs, its
// 8 warps 32 x 32 each (or 64 x 96 and 32 x 24, where that ends sooner); all of them walk all of k in chunks of 32 staged one
// ahead.  Each chunk is summed by itself and added to the total, as k_score_block adds its groups' chunks.  Bound by the FP32
// pipe.  (With k_score_block's division of k half the warps have nothing to do at 100 columns, and 1024 outputs a block pay
// for a reduction.)
constexpr int kScoreTileP = 64;
template <int NB>
constexpr int kScoreTileStage = (kScoreTileP + 16 * NB) * kScoreStride;
template <int NB>
constexpr size_t kScoreTileSmem = 2 * kScoreTileStage<NB> * sizeof(float);

template <int FN, int NB>
__global__ void __launch_bounds__(256, 2)
k_score_tile(const __grid_constant__ ShardArgs<ScoreArgs> shards, int B, int T, int D, int ld) {
    const float* __restrict__ P = shards.s[blockIdx.z].P;
    const float* __restrict__ Tl = shards.s[blockIdx.z].Tl;
    float* __restrict__ raw = shards.s[blockIdx.z].raw;
    grid_dependency_sync();
    constexpr int kScoreTileT = 16 * NB;
    extern __shared__ __align__(16) float score_smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, ty = lane >> 2, tx = lane & 3;
    const int i0 = blockIdx.y * kScoreTileP, j0 = blockIdx.x * kScoreTileT;
    auto stage = [&](int k0, float* to) {
#pragma unroll
        for (int it = 0; it < (kScoreTileP + kScoreTileT) * 8 / 256; ++it) {
            const int q = threadIdx.x + it * 256, row = q >> 3, k4 = (q & 7) * 4;
            const bool is_p = row < kScoreTileP;
            const int g = is_p ? i0 + row : j0 + row - kScoreTileP;
            float* d = to + row * kScoreStride + k4;
            if (g < (is_p ? B : T) && k0 + k4 < D) score_copy16(d, (is_p ? P : Tl) + (size_t)g * D + k0 + k4);
            else *reinterpret_cast<float4*>(d) = make_float4(0.f, 0.f, 0.f, 0.f);
        }
    };
    float total[4][NB];
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < NB; ++b) total[a][b] = 0.f;
    const int row_p = (warp >> 2) * 32 + ty, row_t = kScoreTileP + (warp & 3) * 4 * NB + tx;
    stage(0, score_smem);
    asm volatile("cp.async.commit_group;" ::: "memory");
    for (int k0 = 0, half = 0; k0 < D; k0 += 32, half ^= 1) {
        if (k0 + 32 < D) stage(k0 + 32, score_smem + (half ^ 1) * kScoreTileStage<NB>);
        asm volatile("cp.async.commit_group;" ::: "memory");
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();
        const float* Ps = score_smem + half * kScoreTileStage<NB> + row_p * kScoreStride;
        const float* Ts = score_smem + half * kScoreTileStage<NB> + row_t * kScoreStride;
        float acc[4][NB];
#pragma unroll
        for (int a = 0; a < 4; ++a)
#pragma unroll
            for (int b = 0; b < NB; ++b) acc[a][b] = 0.f;
#pragma unroll 1
        for (int k4 = 0; k4 < min(32, D - k0); k4 += 4) {
            float4 pv[4];
#pragma unroll
            for (int a = 0; a < 4; ++a) pv[a] = load4(Ps + 8 * a * kScoreStride + k4);
#pragma unroll
            for (int b = 0; b < NB; ++b) {
                const float4 tv = load4(Ts + 4 * b * kScoreStride + k4);
                const float tr[4] = {tv.x, tv.y, tv.z, tv.w};
#pragma unroll
                for (int a = 0; a < 4; ++a) {
                    const float pr[4] = {pv[a].x, pv[a].y, pv[a].z, pv[a].w};
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        if (FN == DIST_L1) {
                            acc[a][b] += fabsf(pr[c] - tr[c]);
                        } else if (FN == DIST_L2) {
                            const float d = pr[c] - tr[c];
                            acc[a][b] = fmaf(d, d, acc[a][b]);
                        } else {
                            acc[a][b] = fmaf(pr[c], tr[c], acc[a][b]);
                        }
                    }
                }
            }
        }
#pragma unroll
        for (int a = 0; a < 4; ++a)
#pragma unroll
            for (int b = 0; b < NB; ++b) total[a][b] += acc[a][b];
        __syncthreads();
    }
    // through shared memory, so that whole rows are stored
    constexpr int kOut = kScoreTileT + 4;
    static_assert(kScoreTileP * kOut <= 2 * kScoreTileStage<NB>, "the outputs fit");
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < NB; ++b)
            score_smem[(row_p + 8 * a) * kOut + row_t - kScoreTileP + 4 * b] = FN == DIST_L2 ? sqrtf(total[a][b]) : total[a][b];
    __syncthreads();
    const bool vec = (ld & 3) == 0;
    for (int q = threadIdx.x; q < kScoreTileP * kScoreTileT / 4; q += 256) {
        const int row = q / (kScoreTileT / 4), col = q % (kScoreTileT / 4) * 4, i = i0 + row, j = j0 + col;
        if (i >= B || j >= T) continue;
        const float4 v = load4(score_smem + row * kOut + col);
        float* dst = raw + (size_t)i * ld + j;
        if (vec && j + 3 < T) {
            store4(dst, v);
        } else {
            const float t[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (j + u < T) dst[u] = t[u];
        }
    }
}

template <int FN, int NB>
inline cudaError_t launch_score_tile(const ShardArgs<ScoreArgs>& shards, dim3 tiles, int B, int T, int D, int ld, cudaStream_t stream) {
    static std::atomic<bool> configured[kMaxDeviceOrdinals] = {};  // one attribute call per instantiation and device is enough
    const int slot = current_device_slot();
    if (slot < 0 || !configured[slot]) {
        const cudaError_t err = cudaFuncSetAttribute(k_score_tile<FN, NB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kScoreTileSmem<NB>);
        if (err != cudaSuccess) return err;
        if (slot >= 0) configured[slot] = true;
    }
    return launch_dependent(k_score_tile<FN, NB>, tiles, dim3(256), kScoreTileSmem<NB>, stream, shards, B, T, D, ld);
}

// Picks the kernel: the 16-byte-copy form when the rows allow it, the general form otherwise.  Rows of the scores begin
// `ld` floats apart.  `sync` with world > 1: the kernel waits for the tail rows of the other processes (only the
// 16-byte-copy form can; returns cudaErrorNotSupported otherwise so that the caller waits first).
inline bool score_rows_aligned(const float* P, const float* Tl, int D) {
    return (D % 4) == 0 && reinterpret_cast<uintptr_t>(P) % 16 == 0 && reinterpret_cast<uintptr_t>(Tl) % 16 == 0;
}

template <int FN>
inline cudaError_t launch_score(const ShardArgs<ScoreArgs>& shards, int n_shards, int B, int T, int D, int ld, cudaStream_t stream, const ExchangeSync& sync) {
    bool aligned = true;
    for (int s = 0; s < n_shards; ++s) aligned = aligned && score_rows_aligned(shards.s[s].P, shards.s[s].Tl, D);
    const unsigned n = (unsigned)n_shards;
    if (!aligned) {
        if (sync.world > 1) return cudaErrorNotSupported;
        return launch_dependent(k_score<FN>, dim3((T + 63) / 64, (B + 31) / 32, n), dim3(128), 0, stream, shards, B, T, D, ld);
    }
    // Whole tiles from two blocks per SM on; below that, and where tails are waited for, the k range is divided too.  96
    // columns a tile where its waves of 296 blocks end before those of 128 (128 x 40 000 x 100: 834 tiles in three waves, not
    // 626 in three, 62 -> 60 us with its timing).
    auto tiles = [&](int width) { return dim3((T + width - 1) / width, (B + kScoreTileP - 1) / kScoreTileP, n); };
    const dim3 wide = tiles(128), narrow = tiles(96);
    if (sync.world <= 1 && (size_t)wide.x * wide.y * n >= 2 * kSmCount) {
        auto waves = [&](const dim3& t) { return ((size_t)t.x * t.y * n + 2 * kSmCount - 1) / (2 * kSmCount); };
        if (waves(narrow) * 96 < waves(wide) * 128) return launch_score_tile<FN, 6>(shards, narrow, B, T, D, ld, stream);
        return launch_score_tile<FN, 8>(shards, wide, B, T, D, ld, stream);
    }
    // The width whose waves of 148 blocks end first: 4 NB D clocks for a block's sums, about 4 us for what does not depend
    // on its width.
    auto clocks = [&](int nb) {
        const long long blocks = (long long)((T + 4 * nb - 1) / (4 * nb)) * ((B + kScoreRows - 1) / kScoreRows) * n_shards;
        return (blocks + kSmCount - 1) / kSmCount * (4ll * nb * D + 7600);
    };
    if (clocks(16) <= clocks(12) && clocks(16) <= clocks(8)) return launch_score_block<FN, 16>(shards, n_shards, B, T, D, ld, stream, sync);
    if (clocks(12) <= clocks(8)) return launch_score_block<FN, 12>(shards, n_shards, B, T, D, ld, stream, sync);
    return launch_score_block<FN, 8>(shards, n_shards, B, T, D, ld, stream, sync);
}
inline cudaError_t launch_score(int dist_fn, const ShardArgs<ScoreArgs>& shards, int n_shards, int B, int T, int D, int ld, cudaStream_t stream,
                                const ExchangeSync& sync = ExchangeSync{}) {
    switch (dist_fn) {
        case DIST_L1: return launch_score<DIST_L1>(shards, n_shards, B, T, D, ld, stream, sync);
        case DIST_L2: return launch_score<DIST_L2>(shards, n_shards, B, T, D, ld, stream, sync);
        default: return launch_score<DIST_DOT>(shards, n_shards, B, T, D, ld, stream, sync);
    }
}
// One set of rows, the scores without gaps.
inline cudaError_t launch_score(int dist_fn, const float* P, const float* Tl, float* raw, int B, int T, int D, cudaStream_t stream,
                                const ExchangeSync& sync = ExchangeSync{}) {
    ShardArgs<ScoreArgs> shards{};
    shards.s[0] = ScoreArgs{P, Tl, raw};
    return launch_score(dist_fn, shards, 1, B, T, D, T, stream, sync);
}

// ---------------------------------------------------------------------------
// Loss forward and backward for one row of scores per block
// (src/poplar_kge.cpp:615-660; guarded log-sigmoid src/pag/pag.cpp:888-910; log-softmax
// backward :851-860).  Reads raw distances / dot products, writes
//   loss_rows[i] = the row's un-normalised loss term, and
//   coeff[i, j]  = loss_scale * dloss/draw_ij, already divided by the distance for L2
//                  (0 where the distance is 0: l2distance.codelet.cpp:149-158),
// which is the only thing the score backward needs.
struct LossParams {
    int loss_fn;
    int score_fn;
    int dist_fn;
    int n_tail;
    int ld;                  // floats between rows of the scores and of the coefficients, whose last ld - n_tail become zeros
    float gamma;
    float softmax_shift;     // correction_weight * (log(n_entity*n_shard-1) - log(n_tail-1)), or 0
    float adversarial_scale; // 0 = off
    float w_pos, w_neg;      // log-sigmoid weights of the label / of the other columns
    float grad_scale;        // loss_scale / normaliser
};

struct LossArgs {
    const float* raw;        // [B, ld]
    const uint32_t* label;   // [B]
    float *coeff, *coeff_lo; // [B, ld]; coeff_lo: companion plane, null: none
    float* loss_rows;        // [B]
    float *loss_total, *loss_last;  // null: a later kernel adds the rows' terms
    unsigned* counter;
    const float* extra_loss;
};

// After its row, the block that finishes last adds the rows' loss terms in row order (a fixed
// tree: the result does not depend on which block that is) and adds the step's loss to the running
// total of the program run (src/poplar_kge.cpp:735-736).
// `extra` (may be null): a term of the step's loss that another kernel has already summed (the regularisers).
template <int THREADS>
__device__ __forceinline__ void finish_step_loss(const float* loss_rows, int B, float inv_normaliser, float* loss_total,
                                                 float* loss_last, unsigned* counter, float* scratch, const float* extra) {
    __shared__ int is_last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) is_last = atomicAdd(counter, 1u) + 1u == gridDim.x ? 1 : 0;
    __syncthreads();
    if (!is_last) return;
    __threadfence();
    float part = 0.f;
    for (int i = threadIdx.x; i < B; i += THREADS) part += __ldcg(loss_rows + i);
    part = block_sum<THREADS>(part, scratch);
    if (threadIdx.x == 0) {
        const float step_loss = part * inv_normaliser + (extra ? *extra : 0.f);
        *loss_total += step_loss;
        *loss_last = step_loss;
        *counter = 0u;
    }
}

// One block per row.  A thread keeps its PER columns (j, j + THREADS, ...) in registers, read once and all at the same time;
// the sums take them in that order, which is part of an L1 model's result (see k_pair_bwd).  Bound by latency: a row's
// read, two reductions over the block, a chain of exponentials.  With the row read again for the maximum, the sum and the
// coefficients, one column after the other, steps took (us, before -> after) 70.6 -> 68.9 for 512 x 768 softmax scores, 110.0
// -> 106.5 for two such shards, 64.8 -> 62.7 for 1024 x 2048 log-sigmoids, 59.0 -> 57.4 for four shards of 256 x 512.
template <int THREADS, int PER>
__global__ void __launch_bounds__(THREADS)
k_loss(const __grid_constant__ ShardArgs<LossArgs> shards, LossParams lp, float inv_normaliser, int lo_bf16) {
    __shared__ float scratch[2][THREADS / 32];
    const LossArgs& a = shards.s[blockIdx.y];
    const int i = blockIdx.x, T = lp.n_tail;
    const int lab = (int)a.label[i];  // (staged before the kernel in front began)
    grid_dependency_sync();
    float* __restrict__ loss_rows = a.loss_rows;
    const float* __restrict__ r = a.raw + (size_t)i * lp.ld;
    float* __restrict__ c = a.coeff + (size_t)i * lp.ld;
    // the companion plane for the tensor-core gradients: lower TF32 part, or the bf16 rounding
    float* __restrict__ c_lo = a.coeff_lo && !lo_bf16 ? a.coeff_lo + (size_t)i * lp.ld : nullptr;
    __nv_bfloat16* __restrict__ c16 = a.coeff_lo && lo_bf16 ? reinterpret_cast<__nv_bfloat16*>(a.coeff_lo) + (size_t)i * lp.ld : nullptr;
    auto store = [&](int j, float cj) {
        c[j] = cj;
        if (c_lo) c_lo[j] = tf32_lower(cj);
        if (c16) c16[j] = __float2bfloat16_rn(cj);
    };
    float dist[PER];  // distances or dot products
#pragma unroll
    for (int u = 0; u < PER; ++u) {
        const int j = threadIdx.x + u * THREADS;
        dist[u] = j < T ? r[j] : 0.f;
    }
    for (int j = T + (int)threadIdx.x; j < lp.ld; j += THREADS) store(j, 0.f);
    const bool transe = score_is_gamma_minus_distance(lp.score_fn);
    auto score_of = [&](int u) { return transe ? lp.gamma - dist[u] : dist[u]; };
    auto to_coeff = [&](int u, float g_score) {
        float g = transe ? -g_score : g_score;  // d score / d raw
        if (lp.dist_fn == DIST_L2) g = dist[u] == 0.f ? 0.f : g / dist[u];
        return g;
    };
    if (lp.loss_fn == LOSS_SOFTMAX) {
        float mx = -INFINITY;
#pragma unroll
        for (int u = 0; u < PER; ++u) {
            const int j = threadIdx.x + u * THREADS;
            if (j < T) mx = fmaxf(mx, score_of(u) + (j == lab ? 0.f : lp.softmax_shift));
        }
        mx = block_max<THREADS>(mx, scratch[0]);
        float sum = 0.f;
#pragma unroll
        for (int u = 0; u < PER; ++u) {
            const int j = threadIdx.x + u * THREADS;
            if (j < T) sum += expf(score_of(u) + (j == lab ? 0.f : lp.softmax_shift) - mx);
        }
        sum = block_sum<THREADS>(sum, scratch[1]);
        const float log_z = logf(sum);
#pragma unroll
        for (int u = 0; u < PER; ++u) {
            const int j = threadIdx.x + u * THREADS;
            if (j >= T) continue;
            const float logp = score_of(u) + (j == lab ? 0.f : lp.softmax_shift) - mx - log_z;
            const float g = lp.grad_scale * (expf(logp) - (j == lab ? 1.f : 0.f));
            store(j, to_coeff(u, g));
            if (j == lab) loss_rows[i] = -logp;
        }
        if (a.loss_total) finish_step_loss<THREADS>(loss_rows, (int)gridDim.x, inv_normaliser, a.loss_total, a.loss_last, a.counter, scratch[0], a.extra_loss);
        return;
    }
    // log-sigmoid, optionally with self-adversarial weights from a detached softmax
    float adv_max = 0.f, adv_sum = 1.f;
    const bool adv = lp.adversarial_scale > 0.f;
    if (adv) {
        float mx = -INFINITY;
#pragma unroll
        for (int u = 0; u < PER; ++u) {
            const int j = threadIdx.x + u * THREADS;
            if (j < T) mx = fmaxf(mx, lp.adversarial_scale * score_of(u) + (j == lab ? -10000.f : 0.f));
        }
        adv_max = block_max<THREADS>(mx, scratch[0]);
        float sum = 0.f;
#pragma unroll
        for (int u = 0; u < PER; ++u) {
            const int j = threadIdx.x + u * THREADS;
            if (j < T) sum += expf(lp.adversarial_scale * score_of(u) + (j == lab ? -10000.f : 0.f) - adv_max);
        }
        adv_sum = block_sum<THREADS>(sum, scratch[1]);
    }
    float part = 0.f;
#pragma unroll
    for (int u = 0; u < PER; ++u) {
        const int j = threadIdx.x + u * THREADS;
        if (j >= T) continue;
        const float s = score_of(u);
        const bool pos = j == lab;
        float w = pos ? lp.w_pos : lp.w_neg;
        if (adv) {
            const float soft =
                expf(lp.adversarial_scale * s + (pos ? -10000.f : 0.f) - adv_max) / adv_sum;
            w *= (pos ? 1.f : 0.f) + (float)(T - 1) * soft;
        }
        const float x = pos ? s : -s;
        const float ls = x > -11.f ? -log1pf(expf(-fmaxf(x, -11.f))) : x;
        part += w * ls;
        const float dx = (-w * lp.grad_scale) / (1.f + expf(fminf(x, 11.f)));
        store(j, to_coeff(u, pos ? dx : -dx));
    }
    part = block_sum<THREADS>(part, scratch[0]);
    if (threadIdx.x == 0) loss_rows[i] = -part;
    // (null loss_total: a later kernel of the step adds the rows' terms, off the step's critical chain)
    if (a.loss_total) finish_step_loss<THREADS>(loss_rows, (int)gridDim.x, inv_normaliser, a.loss_total, a.loss_last, a.counter, scratch[0], a.extra_loss);
}

template <int THREADS>
inline cudaError_t launch_loss(const ShardArgs<LossArgs>& shards, int n_shards, const LossParams& lp, float inv_normaliser, int lo_bf16, int B,
                               cudaStream_t stream, bool spread) {
    const dim3 grid((unsigned)B, (unsigned)n_shards);
    // columns per thread: as few as the row needs (a batch has at most kMaxSortItems tails)
    const int per = (lp.n_tail + THREADS - 1) / THREADS;
    if (per <= 1) return launch_spread_if<k_loss<THREADS, 1>>(spread, grid, dim3(THREADS), stream, shards, lp, inv_normaliser, lo_bf16);
    if (per <= 2) return launch_spread_if<k_loss<THREADS, 2>>(spread, grid, dim3(THREADS), stream, shards, lp, inv_normaliser, lo_bf16);
    if (per <= 3) return launch_spread_if<k_loss<THREADS, 3>>(spread, grid, dim3(THREADS), stream, shards, lp, inv_normaliser, lo_bf16);
    if (per <= 4) return launch_spread_if<k_loss<THREADS, 4>>(spread, grid, dim3(THREADS), stream, shards, lp, inv_normaliser, lo_bf16);
    if (per <= 6) return launch_spread_if<k_loss<THREADS, 6>>(spread, grid, dim3(THREADS), stream, shards, lp, inv_normaliser, lo_bf16);
    if (per <= 8) return launch_spread_if<k_loss<THREADS, 8>>(spread, grid, dim3(THREADS), stream, shards, lp, inv_normaliser, lo_bf16);
    if (per <= 16) return launch_spread_if<k_loss<THREADS, 16>>(spread, grid, dim3(THREADS), stream, shards, lp, inv_normaliser, lo_bf16);
    return cudaErrorInvalidValue;
}
inline cudaError_t launch_loss(const ShardArgs<LossArgs>& shards, int n_shards, const LossParams& lp, float inv_normaliser, int lo_bf16, int B,
                               cudaStream_t stream, bool spread) {
    // A warp per row, with a serial chain of exponentials, measured 4 us slower for 512 x 768 scores.  A long row of
    // log-sigmoids, whose chains are longest, gets twice the threads: 256 x 1536 self-adversarial scores 12.7 to 9.5 us
    // (a softmax row of that length was 1 us slower with them).
    if (lp.loss_fn == LOSS_LOGSIGMOID && lp.n_tail >= 1024) return launch_loss<512>(shards, n_shards, lp, inv_normaliser, lo_bf16, B, stream, spread);
    return launch_loss<256>(shards, n_shards, lp, inv_normaliser, lo_bf16, B, stream, spread);
}

// ---------------------------------------------------------------------------
// Score backward: out[m, k] = sum_n C(m, n) * f(x[m, k], y[n, k]) with
//   f = sign(x - y)  (L1, sign(0) = 0: l1distance.codelet.cpp:76-79,138-145)
//   f = x - y        (L2; C already holds grad / dist)
//   f = y            (dot: src/pag/pag.cpp:685-701)
// Problem 0 is the gradient of the predicted tails (x = pred, y = tails, C = coeff);
// problem 1 the gradient of the tails (x = tails, y = pred, C = coeff transposed), whose
// rows go straight to the shard that owns them: the return half of the exchange
// (src/pag/pag.cpp:925-932).
struct PairBwdProblem {
    const float* X;
    const float* Y;
    const float* C;
    int M, N;
    int c_stride_m, c_stride_n;
    float* out;               // [M, D] when out_blocks is null
    float* const* out_blocks; // per block of `block_rows` rows, the base pointer of that block
    int block_rows;
};
struct PairBwdArgs {
    PairBwdProblem p[2];
    int D;
    int longest;   // the problem with the longer sums, whose blocks start first; set by launch_pair_bwd
};

// Two neighbouring fp32 values in one 64-bit register pair.  An instruction issues both and holds the FP32 pipe as long as
// two would: half the issue slots, the same pipe time.  The pair gradients and TransH's scores are faster with it, TransH's
// gradients slower (k_transh_bwd).
using f32x2 = unsigned long long;
__device__ __forceinline__ f32x2 pack2(float lo, float hi) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ float2 unpack2(f32x2 v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
// a - b, rounded once.
__device__ __forceinline__ f32x2 sub2(f32x2 a, f32x2 b) { return fma2(b, 0xbf800000bf800000ull, a); }
// 1 where x > 0, else 0 (0 and NaN included): x times infinity, clamped to [0, 1], where a NaN becomes 0.
__device__ __forceinline__ float positive(float x, float infinity) {
    float r;
    asm("mul.rn.sat.f32 %0, %1, %2;" : "=f"(r) : "f"(x), "f"(infinity));
    return r;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
// c with its sign flipped where e is negative: c * sign(e) unless e is 0 or NaN.
__device__ __forceinline__ float flip_by(float c, float e) { return __uint_as_float(__float_as_uint(c) ^ (__float_as_uint(e) & 0x80000000u)); }
// The smallest magnitude so far; NaN once one was.
__device__ __forceinline__ float least_magnitude(float so_far, float a, float b) {
    float r;
    asm("min.NaN.abs.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(so_far), "f"(a), "f"(b));
    return r;
}
// sign(e) of either value: 1, 0 or -1.  Comparisons run at half the FP32 pipe's rate; these products run at the full one.
__device__ __forceinline__ f32x2 sign2(f32x2 e) {
    const float inf = __int_as_float(0x7f800000);
    const float2 v = unpack2(e);
    return sub2(pack2(positive(v.x, inf), positive(v.y, inf)), pack2(positive(v.x, -inf), positive(v.y, -inf)));
}
constexpr int kPairCols = 64, kPairWarps = 8;  // columns and warps of a block of the two backward kernels below

// dst[r][c] = src[r * stride + c] for r < rows, c < cols of a ROWS x COLS array, zeros elsewhere; asynchronous where vec.
template <int ROWS, int COLS>
__device__ __forceinline__ void stage_rows(float* dst, const float* __restrict__ src, size_t stride, int rows, int cols, bool vec) {
    constexpr int kQuads = COLS / 4;
    for (int q = threadIdx.x; q < ROWS * kQuads; q += 32 * kPairWarps) {
        const int r = q / kQuads, c = q % kQuads * 4;
        float* to = dst + q * 4;
        const float* from = src + (size_t)r * stride + c;
        if (vec && r < rows && c < cols) {
            score_copy16(to, from);
        } else {
            float v[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) v[u] = r < rows && c + u < cols ? from[u] : 0.f;
            *reinterpret_cast<float4*>(to) = make_float4(v[0], v[1], v[2], v[3]);
        }
    }
}
__device__ __forceinline__ void stage_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void stage_wait_previous() { asm volatile("cp.async.wait_group 1;" ::: "memory"); }
// Columns k and k + 1 of a row, ones past its end.
__device__ __forceinline__ f32x2 load_pair(const float* __restrict__ row, int k, int D) { return pack2(k < D ? row[k] : 1.f, k + 1 < D ? row[k + 1] : 1.f); }
__device__ __forceinline__ void store_pair(float* __restrict__ row, int k, int D, f32x2 v) {
    const float2 f = unpack2(v);
    if (k + 1 < D && (D & 1) == 0) {
        *reinterpret_cast<float2*>(row + k) = f;
    } else {
        if (k < D) row[k] = f.x;
        if (k + 1 < D) row[k + 1] = f.y;
    }
}

// A warp takes ROWS rows of 64 columns (a lane two of them) and adds the terms up in the order of n, which is part of the
// result: the coefficients of a softmax row add up to zero, so where (nearly) all differences of a column have one sign
// the L1 gradient is the rounding left over from that sum, and Adam's first steps of a parameter do not depend on a
// gradient's size.  (Dividing n over warps was no faster and moved relations by 1e-3.)  The block walks n in chunks of
// 64, both operands staged in shared memory one chunk ahead; two rows share a warp's reads of Y where the problem has
// blocks enough for it.  Two L1 terms are a packed difference, two coefficients with the sign flipped by it, the smallest
// magnitude so far and a packed sum: five instructions, where clamped products for the signs took eight.  A chunk in which
// a difference was 0 or NaN, whose sign is 0 (a few per million terms of float32 values: too few to matter, and some in every
// launch), is added up again with those products.  Bound by instruction issue (four shards of 256 x 512 x 100: 68 % of the slots,
// the FP32 pipe 41 % and shared memory's wavefronts 45 % of the time) and by what is left uneven: blocks with the longer sums start first, and two blocks per SM, not three or four, because a dependent launch's blocks pile up where
// the kernel in front ends first (four shards of 256 x 512 x 100: 31 us, 43 and 56 with three and four blocks; 48 before
// the three changes, when the blocks of a shard's two problems followed each other).  Four rows per warp: 51 us, too few
// warps.  Tried and slower: threads dealt out over (rows, pairs of columns) without gaps, bulk copies of row pieces for
// the staging (about 100 copies a chunk from one warp), and both operands read through L1 without any staging.
constexpr int kPairChunk = 64;

template <int FN, int ROWS>
__global__ void __launch_bounds__(32 * kPairWarps, 2) k_pair_bwd(const __grid_constant__ ShardArgs<PairBwdArgs> shards) {
    grid_dependency_sync();
    const PairBwdArgs& args = shards.s[blockIdx.y];
    const int which = blockIdx.z == 0 ? args.longest : 1 - args.longest;
    constexpr int kRows = ROWS * kPairWarps, kCs = kRows * kPairChunk, kStage = kCs + kPairChunk * kPairCols;
    __shared__ __align__(16) float smem[2][kStage];  // C [kRows][chunk] or [chunk][kRows] | Y [chunk][cols]
    const int D = args.D, col_tiles = (D + kPairCols - 1) / kPairCols, tile_m = (int)blockIdx.x / col_tiles;
    const PairBwdProblem& pr = args.p[which];
    const int M = pr.M, N = pr.N, m0 = tile_m * kRows, k0 = (int)blockIdx.x % col_tiles * kPairCols;
    if (m0 >= M) return;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, m = m0 + warp * ROWS, k = k0 + lane * 2;
    const bool n_fast = pr.c_stride_n == 1, y_vec = (D & 3) == 0;  // else c_stride_m is 1
    const int c_stride = n_fast ? pr.c_stride_m : pr.c_stride_n;
    const bool c_vec = (c_stride & 3) == 0;  // columns of C between its size and its stride are zero
    auto stage = [&](int n0, float* to) {
        if (n_fast) stage_rows<kRows, kPairChunk>(to, pr.C + (size_t)m0 * c_stride + n0, c_stride, M - m0, N - n0, c_vec);
        else stage_rows<kPairChunk, kRows>(to, pr.C + (size_t)n0 * c_stride + m0, c_stride, N - n0, M - m0, c_vec);
        stage_rows<kPairChunk, kPairCols>(to + kCs, pr.Y + (size_t)n0 * D + k0, D, N - n0, D - k0, y_vec);
    };
    f32x2 x[ROWS], acc[ROWS];
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
        // (1 where there is no value, the second of an odd row's last lane too: its difference to the zeros staged there is not 0)
        x[r] = m + r < M ? load_pair(pr.X + (size_t)(m + r) * D, k, D) : 0x3f8000003f800000ull;
        acc[r] = 0ull;
    }
    stage(0, smem[0]);
    stage_commit();
    for (int n0 = 0, half = 0; n0 < N; n0 += kPairChunk, half ^= 1) {
        if (n0 + kPairChunk < N) stage(n0 + kPairChunk, smem[half ^ 1]);
        stage_commit();
        stage_wait_previous();
        __syncthreads();
        const float* cs = smem[half] + (n_fast ? warp * ROWS * kPairChunk : warp * ROWS);
        const float* ys = smem[half] + kCs + lane * 2;
        f32x2 before[ROWS];
        float least[ROWS];
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
            before[r] = acc[r];
            least[r] = 1.f;
        }
#pragma unroll 4
        for (int n = 0; n < kPairChunk; n += 4) {
            float c[ROWS][4];
            if (n_fast) {
#pragma unroll
                for (int r = 0; r < ROWS; ++r) {
                    const float4 q = load4(cs + r * kPairChunk + n);
                    c[r][0] = q.x; c[r][1] = q.y; c[r][2] = q.z; c[r][3] = q.w;
                }
            } else {
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    if (ROWS == 2) {
                        const float2 q = *reinterpret_cast<const float2*>(cs + (n + u) * kRows);
                        c[0][u] = q.x; c[1 % ROWS][u] = q.y;
                    } else {
                        c[0][u] = cs[(n + u) * kRows];
                    }
                }
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const f32x2 y = *reinterpret_cast<const f32x2*>(ys + (n + u) * kPairCols);
#pragma unroll
                for (int r = 0; r < ROWS; ++r) {
                    if (FN == DIST_L1) {
                        const float2 d = unpack2(sub2(x[r], y));
                        least[r] = least_magnitude(least[r], d.x, d.y);
                        acc[r] = add2(acc[r], pack2(flip_by(c[r][u], d.x), flip_by(c[r][u], d.y)));
                    } else {
                        acc[r] = fma2(pack2(c[r][u], c[r][u]), FN == DIST_DOT ? y : sub2(x[r], y), acc[r]);
                    }
                }
            }
        }
        if (FN == DIST_L1) {
#pragma unroll
            for (int r = 0; r < ROWS; ++r) {
                if (least[r] > 0.f) continue;
                acc[r] = before[r];
#pragma unroll 4
                for (int n = 0; n < kPairChunk; ++n) {
                    const float c = n_fast ? cs[r * kPairChunk + n] : cs[n * kRows + r];
                    acc[r] = fma2(pack2(c, c), sign2(sub2(x[r], *reinterpret_cast<const f32x2*>(ys + n * kPairCols))), acc[r]);
                }
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
        if (m + r >= M) continue;
        float* dst;
        if (pr.out_blocks) {
            const int blk = (m + r) / pr.block_rows;
            dst = pr.out_blocks[blk] + (size_t)(m + r - blk * pr.block_rows) * D;
        } else {
            dst = pr.out + (size_t)(m + r) * D;
        }
        store_pair(dst, k, D, acc[r]);
    }
}

template <int FN>
inline cudaError_t launch_pair_bwd(ShardArgs<PairBwdArgs> shards, int n_shards, cudaStream_t stream) {
    const PairBwdArgs& first = shards.s[0];  // the shards' sizes are alike
    const int col_tiles = (first.D + kPairCols - 1) / kPairCols;
    auto tiles = [&](int which, int rows) { return (first.p[which].M + rows * kPairWarps - 1) / (rows * kPairWarps); };
    // two rows per warp where that still leaves two blocks per SM
    const int rows = (tiles(0, 2) + tiles(1, 2)) * col_tiles * n_shards >= 2 * 148 ? 2 : 1;
    for (int s = 0; s < n_shards; ++s) shards.s[s].longest = first.p[0].N >= first.p[1].N ? 0 : 1;
    const dim3 grid(std::max(tiles(0, rows), tiles(1, rows)) * col_tiles, (unsigned)n_shards, 2), block(32 * kPairWarps);
    if (rows == 2) return launch_dependent(k_pair_bwd<FN, 2>, grid, block, 0, stream, shards);
    return launch_dependent(k_pair_bwd<FN, 1>, grid, block, 0, stream, shards);
}
inline cudaError_t launch_pair_bwd(int fn, const ShardArgs<PairBwdArgs>& shards, int n_shards, cudaStream_t stream) {
    if (fn == DIST_L1) return launch_pair_bwd<DIST_L1>(shards, n_shards, stream);
    if (fn == DIST_L2) return launch_pair_bwd<DIST_L2>(shards, n_shards, stream);
    return launch_pair_bwd<DIST_DOT>(shards, n_shards, stream);
}
inline cudaError_t launch_pair_bwd(int fn, const PairBwdArgs& args, cudaStream_t stream) {
    ShardArgs<PairBwdArgs> shards{};
    shards.s[0] = args;
    return launch_pair_bwd(fn, shards, 1, stream);
}

// ---------------------------------------------------------------------------
// Sort-and-segment preparation, once per staged step and shard: orders the B head
// lookups and the T tail lookups by the hidden row they read (ties by position, so the
// order is unique) and records where each row's segment starts; the same for the B
// relation lookups.  The scatter-add of src/pag/pag.cpp:721-743 then becomes one
// sequential sum per row in a fixed order: no float atomics.
// One block per (shard-step).
constexpr int kMaxSortItems = 4096;
constexpr int kSortThreads = 512, kSortWarps = kSortThreads / 32;

// A stable sort of up to kMaxSortItems positions by their keys, one block, in passes over six bits of the key.  A warp
// owns a contiguous part of the positions and ranks them 32 at a time among the warp's equal digits (six ballots); the
// 64 x 16 counts are scanned digit by digit, so equal keys stay in position order.  As many passes as the largest key
// has bits for: two for the 4096 rows of a step, where a bitonic network in shared memory ran 78 stages (two sorts
// of 1280 keys and one of 512 took 80 us, 160 us at 3072, a third of that with the launch this way).
struct BlockSort {
    uint32_t key[kMaxSortItems];
    uint16_t idx[2][kMaxSortItems];
    uint32_t count[64 * kSortWarps];  // [digit][warp]
    uint32_t warp_total[kSortWarps];

    // Sorts the positions 0 .. n - 1 by key (filled by the caller, who has synchronised); all keys are below 2^bits.
    // Returns the sorted positions.
    __device__ const uint16_t* sort(int n, int bits) {
        const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
        const int per_warp = (n + kSortThreads - 1) / kSortThreads * 32, begin = warp * per_warp;
        uint16_t *in = idx[0], *out = idx[1];
        for (int i = threadIdx.x; i < n; i += kSortThreads) in[i] = (uint16_t)i;
        for (int shift = 0; shift < bits; shift += 6) {
            for (int i = threadIdx.x; i < 64 * kSortWarps; i += kSortThreads) count[i] = 0u;
            __syncthreads();
            uint32_t place[kMaxSortItems / kSortThreads], pos[kMaxSortItems / kSortThreads];
#pragma unroll
            for (int it = 0; it < kMaxSortItems / kSortThreads; ++it) {
                const int i = begin + it * 32 + lane;
                const bool live = it * 32 < per_warp && i < n;
                if (!__any_sync(0xffffffffu, live)) break;
                pos[it] = live ? in[i] : 0u;
                const uint32_t digit = (key[pos[it]] >> shift) & 63u;
                uint32_t same = __ballot_sync(0xffffffffu, live);
                if (!live) same = ~same;
#pragma unroll
                for (int b = 0; b < 6; ++b) {
                    const uint32_t ones = __ballot_sync(0xffffffffu, (digit >> b) & 1u);
                    same &= (digit >> b) & 1u ? ones : ~ones;
                }
                uint32_t* const cell = count + digit * kSortWarps + warp;
                const uint32_t before = *cell;
                __syncwarp();
                if (live && lane == __ffs(same) - 1) *cell = before + __popc(same);
                __syncwarp();
                place[it] = before + __popc(same & ((1u << lane) - 1u));
            }
            __syncthreads();
            // exclusive scan over (digit, warp), two neighbours per thread
            const uint2 mine = *reinterpret_cast<const uint2*>(count + 2 * threadIdx.x);
            uint32_t sum = mine.x + mine.y;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t left = __shfl_up_sync(0xffffffffu, sum, o);
                if (lane >= o) sum += left;
            }
            if (lane == 31) warp_total[warp] = sum;
            __syncthreads();
            uint32_t base = 0;
            for (int w = 0; w < warp; ++w) base += warp_total[w];
            base += sum - mine.x - mine.y;
            *reinterpret_cast<uint2*>(count + 2 * threadIdx.x) = make_uint2(base, base + mine.x);
            __syncthreads();
#pragma unroll
            for (int it = 0; it < kMaxSortItems / kSortThreads; ++it) {
                const int i = begin + it * 32 + lane;
                if (it * 32 < per_warp && i < n) out[count[((key[pos[it]] >> shift) & 63u) * kSortWarps + warp] + place[it]] = (uint16_t)pos[it];
            }
            __syncthreads();
            uint16_t* const t = in;
            in = out;
            out = t;
        }
        __syncthreads();
        return in;
    }
    // The first of the n sorted positions whose key is not below `target`.
    __device__ int lower_bound(const uint16_t* sorted, int n, uint32_t target) const {
        int lo = 0, hi = n;
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (key[sorted[mid]] < target) lo = mid + 1; else hi = mid;
        }
        return lo;
    }
};
static_assert(kMaxSortItems <= 65536 && 2 * kSortThreads == 64 * kSortWarps, "positions in 16 bits, two counts per thread");
__device__ __forceinline__ int bits_below(uint32_t limit) { return limit <= 1u ? 0 : 32 - __clz(limit - 1u); }

// Rows with more than kHeavyMin lookups are cut into parts of kHeavyPart lookups, at most kHeavySlots
// parts per shard and step (see k_entity_update).
constexpr int kHeavySlots = 112;
constexpr int kHeavyMin = 12;
constexpr int kHeavyPart = 16;

static __global__ void __launch_bounds__(kSortThreads)
k_prepare_segments(const uint32_t* __restrict__ head, const uint32_t* __restrict__ a2a_idx,
                   const uint32_t* __restrict__ relation, const uint32_t* __restrict__ remote, int B,
                   int T, int R, int n_rel, uint32_t* __restrict__ ent_perm,
                   uint32_t* __restrict__ ent_off, uint32_t* __restrict__ rel_perm,
                   uint32_t* __restrict__ rel_off, uint32_t* __restrict__ first_slot,
                   uint4* __restrict__ heavy_parts, uint32_t* __restrict__ heavy_count, uint4* __restrict__ row_info,
                   uint32_t* __restrict__ lookup_row) {
    __shared__ BlockSort bs;
    const int s = blockIdx.x;
    head += (size_t)s * B;
    relation += (size_t)s * B;
    a2a_idx += (size_t)s * T;
    ent_perm += (size_t)s * (B + T);
    ent_off += (size_t)s * (R + 1);
    rel_perm += (size_t)s * B;
    rel_off += (size_t)s * (n_rel + 1);

    const int n = B + T;
    if (lookup_row)  // the table row of every lookup, for a step whose lookups read the table
        for (int i = threadIdx.x; i < n; i += blockDim.x) lookup_row[(size_t)s * n + i] = remote[(size_t)s * R + (i < B ? head[i] : a2a_idx[i - B])];
    for (int i = threadIdx.x; i < n; i += blockDim.x) bs.key[i] = min(i < B ? head[i] : a2a_idx[i - B], (uint32_t)R);  // lookups past the rows (an operator's caller may pass some): behind them
    __syncthreads();
    const uint16_t* sorted = bs.sort(n, bits_below((uint32_t)R + 1u));
    for (int i = threadIdx.x; i < n; i += blockDim.x) ent_perm[i] = sorted[i];
    for (int r = threadIdx.x; r <= R; r += blockDim.x) ent_off[r] = (uint32_t)bs.lower_bound(sorted, n, (uint32_t)r);
    __syncthreads();

    if (rel_perm) {  // null: the caller has no relation lookups (the operator form of the scatter-add)
        for (int i = threadIdx.x; i < B; i += blockDim.x) bs.key[i] = relation[i];
        __syncthreads();
        sorted = bs.sort(B, bits_below((uint32_t)n_rel));
        for (int i = threadIdx.x; i < B; i += blockDim.x) rel_perm[i] = sorted[i];
        for (int r = threadIdx.x; r <= n_rel; r += blockDim.x) rel_off[r] = (uint32_t)bs.lower_bound(sorted, B, (uint32_t)r);
    }
    if (!remote) return;
    __syncthreads();

    // Which gathered slot is the first to name its table row: only that slot writes the row
    // back.  `remote` is unique apart from the zero padding at its end, whose slots all name
    // row 0; the reference computes every slot from the same gathered copy, so its duplicate
    // writes are identical, and one write reproduces them.
    remote += (size_t)s * R;
    first_slot += (size_t)s * R;
    // The sampler's order (ascending, the padding last) needs no sort.
    bool in_order = true;
    for (int i = threadIdx.x; i < R; i += blockDim.x) {
        const uint32_t row = remote[i], before = i ? remote[i - 1] : 0u;
        in_order = in_order && (row > before ? i == 0 || before != 0u : row == 0u);  // nothing but padding after padding
    }
    if (__syncthreads_and(in_order)) {
        for (int i = threadIdx.x; i < R; i += blockDim.x) first_slot[i] = remote[i] != 0u || i == 0 || remote[i - 1] != 0u ? 1u : 0u;
    } else {
        __shared__ uint32_t s_highest;
        if (threadIdx.x == 0) s_highest = 0u;
        __syncthreads();
        uint32_t highest = 0;
        for (int i = threadIdx.x; i < R; i += blockDim.x) {
            bs.key[i] = remote[i];
            highest = max(highest, remote[i]);
        }
        atomicMax(&s_highest, highest);
        __syncthreads();
        sorted = bs.sort(R, 32 - __clz(s_highest));
        for (int i = threadIdx.x; i < R; i += blockDim.x)
            first_slot[sorted[i]] = i == 0 || bs.key[sorted[i - 1]] != bs.key[sorted[i]] ? 1u : 0u;
    }
    if (heavy_parts) {
    // Rows with many lookups are cut into parts for k_entity_update (bit 1 of first_slot marks them).
    // All threads look for such rows (there are at most (B + T) / kHeavyMin of them); one thread
    // then orders them by row, so that the slots do not depend on the timing, and hands out the parts.
    constexpr int kMaxHeavyRows = 128;
    __shared__ int s_heavy_rows[kMaxHeavyRows];
    __shared__ int s_heavy_n;
    if (threadIdx.x == 0) s_heavy_n = 0;
    __syncthreads();
    for (int r = threadIdx.x; r < R; r += blockDim.x)
        if (ent_off[r + 1] - ent_off[r] > (uint32_t)kHeavyMin) {
            const int i = atomicAdd(&s_heavy_n, 1);
            if (i < kMaxHeavyRows) s_heavy_rows[i] = r;
        }
    __syncthreads();
    if (threadIdx.x == 0) {
        heavy_parts += (size_t)s * kHeavySlots;
        const int n_rows = min(s_heavy_n, kMaxHeavyRows);
        for (int i = 1; i < n_rows; ++i) {  // insertion sort, a handful of entries
            const int r = s_heavy_rows[i];
            int j = i - 1;
            for (; j >= 0 && s_heavy_rows[j] > r; --j) s_heavy_rows[j + 1] = s_heavy_rows[j];
            s_heavy_rows[j + 1] = r;
        }
        int used = 0;
        for (int i = 0; i < n_rows; ++i) {
            const int r = s_heavy_rows[i];
            const uint32_t q0 = ent_off[r], q1 = ent_off[r + 1];
            const int parts = (int)((q1 - q0 + kHeavyPart - 1) / kHeavyPart);
            if (used + parts > kHeavySlots || parts > 255) continue;  // stays with its own block
            for (int p = 0; p < parts; ++p)
                heavy_parts[used + p] = make_uint4((uint32_t)r, q0 + (uint32_t)(p * kHeavyPart),
                                                   min(q1, q0 + (uint32_t)((p + 1) * kHeavyPart)),
                                                   ((uint32_t)used << 16) | ((uint32_t)parts << 8) | (uint32_t)p);
            first_slot[r] |= 2u;
            used += parts;
        }
        heavy_count[s] = (uint32_t)used;
    }
    }
    if (!row_info) return;
    // A row's descriptor for k_entity_update: one sector holds what four scattered loads would fetch.
    __syncthreads();
    row_info += (size_t)s * 2 * R;
    for (int r = threadIdx.x; r < R; r += blockDim.x) {
        const uint32_t q0 = ent_off[r], count = ent_off[r + 1] - q0;
        uint32_t e[4];
        for (int u = 0; u < 4; ++u) e[u] = (uint32_t)u < count ? ent_perm[q0 + u] : 0xffffffffu;
        row_info[2 * r] = make_uint4(q0, count, first_slot[r], remote[r]);
        row_info[2 * r + 1] = make_uint4(e[0], e[1], e[2], e[3]);
    }
}

// ---------------------------------------------------------------------------
// Segment-sum of the lookup gradients into the hidden rows, fused with the row-wise Adam
// update and the write-back (src/pag/pag.cpp:721-743; src/poplar_kge.cpp:695-704;
// src/fructose/frnn.cpp:61-90).  One block per gathered row.  Every gathered row is
// updated, rows with a zero gradient and the padding row included, as in the reference.
// d_hid_h / d_hid_t keep the hidden-row gradients for the projection backward (null: there is none).
//
// Entity popularity is skewed: the shard that holds a step's most popular entity sees one row
// with hundreds of lookups, and a single block would add them sixteen at a time while the rest of
// the GPU idles.  k_prepare_segments therefore cuts every row with more than kHeavyMin lookups
// into parts of kHeavyPart lookups (at most kHeavySlots parts per shard and step).  The first
// kHeavySlots blocks of the grid take one part each, leave its sums in `heavy_partial`, and the
// block that arrives last at the row's counter adds the parts in part order and finishes the
// row; the row's own block skips it.  Nothing waits, and the order of the additions is fixed.
constexpr int kSegmentLanes = 4;  // threads groups that share the lookups of one part of a popular row
constexpr int kRowsPerBlock = 8;  // gathered rows per block of k_entity_update: one warp each

// Dropout of the feature network's output (src/poplar_kge.cpp:459-461; frnn::dropout,
// src/pag/pag.cpp:596-617): an element is kept with probability 1 - p and scaled by 1 / (1 - p);
// the backward passes g / (1 - p) through the kept elements.  (The reference tests output != 0
// instead of the mask; the two differ only where a kept element is exactly zero, which is a row
// without features, whose gradient reaches no parameter.)  The reference draws from the IPU's
// generator; here the mask is a pure function of (seed, training step, shard, call, row, column):
// Philox-4x32-10 keyed by (seed, step), one word per element, kept when word >> 8 is below
// `threshold` = round((1 - p) * 2^24).  Forward and backward recompute it, nothing is stored.
struct DropoutParams {
    uint32_t threshold;        // 0: no dropout
    uint32_t seed;
    const uint32_t* step_key;  // the training step's number, on the device (a graph replays with fixed arguments)
    uint32_t shard;            // global shard index
    float scale;               // 1 / (1 - p)
};

__device__ __forceinline__ void philox_round(uint32_t (&c)[4], uint32_t k0, uint32_t k1);

// Keep bits of columns 4 * col4 .. 4 * col4 + 3 of gathered row r in call `part` (0 head, 1 tail).
__device__ __forceinline__ uint32_t dropout_keep4(const DropoutParams& dp, uint32_t part, uint32_t r, uint32_t col4) {
    uint32_t c[4] = {r, col4, (dp.shard << 1) | part, 0x64726f70u};
    uint32_t k0 = dp.seed, k1 = *dp.step_key;
#pragma unroll
    for (int i = 0; i < 10; ++i) {
        philox_round(c, k0, k1);
        k0 += 0x9E3779B9u;
        k1 += 0xBB67AE85u;
    }
    uint32_t bits = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) bits |= ((c[i] >> 8) < dp.threshold ? 1u : 0u) << i;
    return bits;
}

// hidden = value + dropout(hidden - value), in place on the hidden rows of each call.  With one
// feature network both calls start from the same rows (hid_t_in == hid_h) and get their own masks.
struct DropoutArgs {
    const uint8_t* rows_c;
    float* hid_h;
    const float* hid_t_in;
    float* hid_t;
    DropoutParams dp;
};

template <class ST>
__global__ void __launch_bounds__(256) k_dropout_hidden(const __grid_constant__ ShardArgs<DropoutArgs> shards, RowLayout L, int R) {
    grid_dependency_sync();
    const DropoutArgs& a = shards.s[blockIdx.y];
    const uint8_t* __restrict__ rows_c = a.rows_c;
    float* hid_h = a.hid_h;
    const float* hid_t_in = a.hid_t_in;
    float* hid_t = a.hid_t;
    const DropoutParams& dp = a.dp;
    const int D = (int)L.d, quads = (D + 3) / 4;
    const int i = (int)(blockIdx.x * blockDim.x + threadIdx.x);
    if (i >= R * quads) return;
    const int r = i / quads, q = i - r * quads;
    const uint8_t* __restrict__ row = rows_c + (size_t)r * L.row_bytes;
    const uint32_t keep_h = dropout_keep4(dp, 0u, (uint32_t)r, (uint32_t)q), keep_t = dropout_keep4(dp, 1u, (uint32_t)r, (uint32_t)q);
    for (int u = 0; u < 4; ++u) {
        const int c = 4 * q + u;
        if (c >= D) break;
        const size_t o = (size_t)r * D + c;
        const float v = load_value<ST>(L, row, c);
        const float fh_h = hid_h[o] - v, fh_t = hid_t_in[o] - v;
        hid_h[o] = (keep_h >> u) & 1u ? v + fh_h * dp.scale : v;
        hid_t[o] = (keep_t >> u) & 1u ? v + fh_t * dp.scale : v;
    }
}

// Norm regularisers of the gathered rows (src/poplar_kge.cpp:430-437, 463-465): each of the two
// entityHidden calls of a step (head part, tail part) adds
//   w_e * sum_r N(value_r) + w_f * sum_r N(feature_hidden_r) + w_h * sum_r N(hidden_r),
// N(a) = (sum_k |a_k^p|)^(1/p) per row (lpnorm, :389-391), over all R gathered rows, to the shard's
// loss, not normalised.  The backward is the reference's tape: pow gives g * p * out / a with 0 where
// a is 0 (src/pag/pag.cpp:493-503), abs gives sign (:449-456), so
//   dN/da_k = N / s * |a_k|^p / a_k   (s = sum_k |a_k|^p; 0 where a_k or s is 0),
// times the weight and the loss scale (the root gradient, :691).  |a|^p stands for |a^p|: the same
// wherever a^p is defined.  The feature network's output is taken as hidden - value.
// One warp per row; writes the three gradient terms k_entity_update adds and the row's loss term;
// the last block adds the rows' terms in row order into *loss_out.
struct RegParams {
    float power[3], weight[3];  // embedding, feature, hidden
    float loss_scale;
    int shared;                 // one feature network: both calls see the same rows
};

__device__ __forceinline__ float abs_pow(float a, float p) {
    a = fabsf(a);
    return p == 2.f ? a * a : (p == 1.f ? a : powf(a, p));
}

__device__ __forceinline__ float warp_sum(float v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

struct RegArgs {
    const uint8_t* rows_c;
    const float *hid_h, *hid_t;
    float *reg_val, *reg_h, *reg_t, *loss_rows, *loss_out, *loss_sink;
    unsigned* counter;
};

template <class ST>
__global__ void __launch_bounds__(256) k_regularise(const __grid_constant__ ShardArgs<RegArgs> shards, RowLayout L, int R, RegParams rp) {
    grid_dependency_sync();
    const RegArgs& a = shards.s[blockIdx.y];
    const uint8_t* __restrict__ rows_c = a.rows_c;
    const float* __restrict__ hid_h = a.hid_h;
    const float* __restrict__ hid_t = a.hid_t;
    float* __restrict__ reg_val = a.reg_val;
    float* __restrict__ reg_h = a.reg_h;
    float* __restrict__ reg_t = a.reg_t;
    __shared__ float scratch[8];
    const int lane = threadIdx.x & 31, r = (int)blockIdx.x * 8 + (int)(threadIdx.x >> 5), D = (int)L.d;
    if (r < R) {
        const uint8_t* __restrict__ row = rows_c + (size_t)r * L.row_bytes;
        const float* __restrict__ hid[2] = {hid_h + (size_t)r * D, hid_t + (size_t)r * D};
        float* __restrict__ out[2] = {reg_h + (size_t)r * D, rp.shared ? nullptr : reg_t + (size_t)r * D};
        const int parts = rp.shared ? 1 : 2;
        const float calls = rp.shared ? 2.f : 1.f;  // how many of the two calls a part stands for
        float s_e = 0.f, s_f[2] = {0.f, 0.f}, s_h[2] = {0.f, 0.f};
        for (int c = lane; c < D; c += 32) {
            const float v = load_value<ST>(L, row, c);
            s_e += abs_pow(v, rp.power[0]);
            for (int q = 0; q < parts; ++q) {
                const float h = hid[q][c];
                s_f[q] += abs_pow(h - v, rp.power[1]);
                s_h[q] += abs_pow(h, rp.power[2]);
            }
        }
        // norm and the factor weight * loss_scale * N / s of a row's gradient
        auto norm = [&](float s, int which, float& fac) {
            s = warp_sum(s);
            const float n = s > 0.f ? powf(s, 1.f / rp.power[which]) : 0.f;
            fac = s > 0.f && rp.weight[which] > 0.f ? rp.weight[which] * rp.loss_scale * n / s : 0.f;
            return rp.weight[which] > 0.f ? rp.weight[which] * n : 0.f;
        };
        auto term = [&](float a, int which, float fac) { return a == 0.f || fac == 0.f ? 0.f : fac * abs_pow(a, rp.power[which]) / a; };
        float fac_e, fac_f[2] = {0.f, 0.f}, fac_h[2] = {0.f, 0.f};
        float loss = 2.f * norm(s_e, 0, fac_e);
        for (int q = 0; q < parts; ++q) loss += calls * (norm(s_f[q], 1, fac_f[q]) + norm(s_h[q], 2, fac_h[q]));
        for (int c = lane; c < D; c += 32) {
            const float v = load_value<ST>(L, row, c);
            float gv = 2.f * term(v, 0, fac_e);
            for (int q = 0; q < parts; ++q) {
                const float h = hid[q][c];
                const float g_h = calls * term(h, 2, fac_h[q]);
                gv += g_h;
                out[q][c] = g_h + calls * term(h - v, 1, fac_f[q]);
            }
            reg_val[(size_t)r * D + c] = gv;
        }
        if (lane == 0) a.loss_rows[r] = loss;
    }
    finish_step_loss<256>(a.loss_rows, R, 1.f, a.loss_sink, a.loss_out, a.counter, scratch, nullptr);
}

struct HeavyRows {
    const uint4* parts;      // [kHeavySlots] {gathered row, first lookup, end lookup, (first part's slot << 16) | (parts << 8) | part}
    const uint32_t* count;   // parts in use
    float* partial;          // [kHeavySlots][2][D] sums of a part: head lookups | tail lookups
    unsigned* counter;       // [kHeavySlots] parts of a row that have arrived (indexed by the row's first slot)
    // Optional, [R][2]: everything a row's warp needs before it can load gradient rows, in one 32-byte
    // sector: {first lookup's position, lookups, first_slot word, table row} and the row's first four
    // lookups (k_prepare_segments writes it); null: the warp reads off / first_slot / remote / perm.
    const uint4* row_info;
};

// What k_entity_update reads and writes of one shard.
struct EntityShard {
    uint8_t* table;
    const uint8_t* rows_c;            // the step's gathered rows; null with DIRECT
    const uint32_t *remote, *perm, *off, *first_slot;
    const float *d_head, *grad_recv;
    float *d_hid_h, *d_hid_t;         // gradients of the hidden rows (null: nothing reads them; d_hid_t null: one network)
    float *d_hid_h_lo, *d_hid_t_lo;   // their lower TF32 planes (null: not needed)
    HeavyRows heavy;
    // Gradients of the norm regularisers (k_regularise), [R, D] each, null when all weights are 0:
    // reg_val joins the value's gradient, reg_h / reg_t the gradient of the feature network's output
    // (reg_t null with a shared network, whose reg_h then holds both calls' terms).
    const float *reg_val, *reg_h, *reg_t;
    DropoutParams drop;  // threshold 0: none.  Masks the gradients of the feature network's outputs.
    // Non-null: the value's gradient is left here ([R, D]) and the rows are not updated; k_row_adam
    // does that once the rest of the gradient is known (the feature MLP reads the value too).
    float* defer_grad;
    const float* d_relrow[2];         // [B, D] per-triple gradients of the relation tables' rows (the second one: TransH's normals)
    const uint32_t *rel_perm, *rel_off;  // triples ordered by relation, [n_rel + 1]
    float* const* dense_dst;          // [n_owner] this shard's slot in each owner's receive buffer
    const float* loss_rows;           // [B] loss terms left by k_loss; null: k_loss has added them up
    float *loss_total, *loss_last;
    const float* extra_loss;
};

// The relation rows of the dense gradient are summed by blocks appended to the grid (they too depend only on the score
// gradients): a row's gradient is the sum of the per-triple gradients of its relation's triples, in position order
// (backward of the gather at src/poplar_kge.cpp:489).  Where all shards are in the launch and in this process, a block
// adds the shards' sums in shard order and applies the row's Adam step; else each shard's sum is stored into the memory
// of the process that owns that row of the dense vector (row r to process r % n_owner as its row r / n_owner), which
// k_dense_update waits for.
struct EntityStep {
    RowLayout L;
    int B, R, n_shards;
    const float* step_size;
    float lr_modifier;
    AdamParams ap;
    ExchangeSync sync;
    int n_rel, n_tables, n_owner;     // relation rows per table; tables (0: another kernel sums them)
    int rel_blocks;                   // blocks of a shard that sum relation rows
    int dense_row0[2];                // a table's first row in the dense vector
    float *rel_w[2], *rel_m[2], *rel_v[2];  // null: sums go to dense_dst
    float rel_lr_modifier[2];
    float inv_normaliser;
};

// A thread adds up PER strands of a relation's triples: strand s of LANES * PER takes the triples s, s + LANES * PER, ...
template <int V, int LANES, int PER>
__device__ __forceinline__ void relation_row_sum(const ShardArgs<EntityShard>& shards, const EntityStep& g, int unit, float (*part)[64 * V], uint32_t* s_perm) {
    const int D = (int)g.L.d, col = threadIdx.x & 63, lane = threadIdx.x >> 6;
    const int table = unit >= g.n_rel ? 1 : 0, rho = unit - table * g.n_rel;
    const bool here = g.rel_w[table] != nullptr;
    const int first = here ? 0 : (int)blockIdx.y, last = here ? g.n_shards : first + 1;
    const AdamParams& ap = g.ap;
    // where the row's gradient goes: into its owner's receive buffer, or straight into the row's Adam step
    auto deliver = [&](int c, float total) {
        if (!here) {
            const int row = rho + g.dense_row0[table];
            shards.s[first].dense_dst[row % g.n_owner][(size_t)(row / g.n_owner) * D + c] = total;
            return;
        }
        const size_t e = (size_t)rho * D + c;
        const float alpha = *g.step_size * g.rel_lr_modifier[table];
        const float mo = weighted_sum(ap.beta_m, g.rel_m[table][e], ap.one_minus_beta_m, total);
        const float ve = weighted_sum(ap.beta_v, g.rel_v[table][e], __fmul_rn(ap.one_minus_beta_v, total), total);
        const float x = g.rel_w[table][e];
        g.rel_w[table][e] = x - alpha * (mo / (sqrtf(ve) + ap.epsilon) + ap.weight_decay * x);
        g.rel_m[table][e] = mo;
        g.rel_v[table][e] = ve;
    };
    // four neighbouring columns at once where the rows allow 16-byte accesses
    auto deliver4 = [&](int c, const float (&total)[4]) {
        if (!here) {
            const int row = rho + g.dense_row0[table];
            store4(shards.s[first].dense_dst[row % g.n_owner] + (size_t)(row / g.n_owner) * D + c, make_float4(total[0], total[1], total[2], total[3]));
            return;
        }
        const size_t e = (size_t)rho * D + c;
        const float alpha = *g.step_size * g.rel_lr_modifier[table];
        const float4 m4 = load4(g.rel_m[table] + e), v4 = load4(g.rel_v[table] + e), x4 = load4(g.rel_w[table] + e);
        float mo[4] = {m4.x, m4.y, m4.z, m4.w}, ve[4] = {v4.x, v4.y, v4.z, v4.w}, x[4] = {x4.x, x4.y, x4.z, x4.w};
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            mo[u] = weighted_sum(ap.beta_m, mo[u], ap.one_minus_beta_m, total[u]);
            ve[u] = weighted_sum(ap.beta_v, ve[u], __fmul_rn(ap.one_minus_beta_v, total[u]), total[u]);
            x[u] = x[u] - alpha * (mo[u] / (sqrtf(ve[u]) + ap.epsilon) + ap.weight_decay * x[u]);
        }
        store4(g.rel_w[table] + e, make_float4(x[0], x[1], x[2], x[3]));
        store4(g.rel_m[table] + e, make_float4(mo[0], mo[1], mo[2], mo[3]));
        store4(g.rel_v[table] + e, make_float4(ve[0], ve[1], ve[2], ve[3]));
    };
    bool any = false;
    for (int s = first; s < last; ++s) any = any || shards.s[s].rel_off[rho] != shards.s[s].rel_off[rho + 1];
    if (!any) {
        if (V == 4) {
            const float zero[4] = {0.f, 0.f, 0.f, 0.f};
            for (int c = threadIdx.x * 4; c < D; c += blockDim.x * 4) deliver4(c, zero);
        } else {
            for (int c = threadIdx.x; c < D; c += blockDim.x) deliver(c, 0.f);
        }
        return;
    }
    for (int c0 = 0; c0 < D; c0 += 64 * V) {
        const int c = c0 + col * V;
        float totals[4] = {0.f, 0.f, 0.f, 0.f};
        for (int s = first; s < last; ++s) {
            const EntityShard& a = shards.s[s];
            const float* __restrict__ rows = a.d_relrow[table];
            const uint32_t q0 = a.rel_off[rho], q1 = a.rel_off[rho + 1];
            if (q0 == q1) continue;
            float sum[PER][V];
#pragma unroll
            for (int p = 0; p < PER; ++p)
#pragma unroll
                for (int u = 0; u < V; ++u) sum[p][u] = 0.f;
            for (uint32_t base = q0; base < q1; base += 64 * LANES) {
                const int count = (int)min((uint32_t)(64 * LANES), q1 - base);
                __syncthreads();
                if ((int)threadIdx.x < count) s_perm[threadIdx.x] = a.rel_perm[base + threadIdx.x];
                __syncthreads();
                if (c >= D) continue;
                for (int i = lane; i < count; i += 4 * LANES) {
                    float4 v[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const int ii = i + u * LANES;
                        v[u] = make_float4(0.f, 0.f, 0.f, 0.f);
                        if (ii < count) {
                            const float* src = rows + (size_t)s_perm[ii] * D + c;
                            if (V == 4) v[u] = load4(src); else v[u].x = src[0];
                        }
                    }
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        if (i + u * LANES >= count) continue;
                        float (&strand)[V] = sum[u % PER];
                        strand[0] += v[u].x;
                        if (V == 4) { strand[1 % V] += v[u].y; strand[2 % V] += v[u].z; strand[3 % V] += v[u].w; }
                    }
                }
            }
            __syncthreads();
#pragma unroll
            for (int p = 0; p < PER; ++p)
#pragma unroll
                for (int u = 0; u < V; ++u) part[p * LANES + lane][col * V + u] = sum[p][u];
            __syncthreads();
            if (lane == 0 && c < D) {
#pragma unroll
                for (int u = 0; u < V; ++u) {
                    float total = part[0][col * V + u];
#pragma unroll
                    for (int l = 1; l < LANES * PER; ++l) total += part[l][col * V + u];
                    totals[u] += total;
                }
            }
        }
        if (lane == 0 && c < D) {
            if (V == 4) deliver4(c, totals);
            else deliver(c, totals[0]);
        }
    }
}

// EXTRAS: the regularisers' terms, the dropout masks and the deferred row update are compiled in
// (they cost 20 registers, a third of the resident blocks, which the plain step does not pay).
// DIRECT: the step makes no gathered copy; the state before the update is the table row, which only its first slot touches.
template <class ST, int V, bool EXTRAS = false, bool DIRECT = false>
__global__ void __launch_bounds__(64 * kSegmentLanes, EXTRAS ? 2 : 4)
k_entity_update(const __grid_constant__ ShardArgs<EntityShard> shards, const __grid_constant__ EntityStep g) {
    grid_dependency_sync();
    const EntityShard& rr = shards.s[blockIdx.y];
    const RowLayout& L = g.L;
    const AdamParams& ap = g.ap;
    const int R = g.R, B = g.B, row_blocks = (R + kRowsPerBlock - 1) / kRowsPerBlock;
    if ((int)blockIdx.x >= kHeavySlots + row_blocks) {  // a relation row: needs nothing from the other processes
        __shared__ float rel_part[2 * kSegmentLanes][64 * V];
        __shared__ uint32_t rel_perm[64 * kSegmentLanes];
        const int block = (int)blockIdx.x - kHeavySlots - row_blocks;
        if (block >= g.rel_blocks) {  // the loss block
            float part = 0.f;
            for (int i = threadIdx.x; i < B; i += 64 * kSegmentLanes) part += rr.loss_rows[i];
            part = block_sum<64 * kSegmentLanes>(part, &rel_part[0][0]);
            if (threadIdx.x == 0) {
                const float step_loss = part * g.inv_normaliser + (rr.extra_loss ? *rr.extra_loss : 0.f);
                *rr.loss_total += step_loss;
                *rr.loss_last = step_loss;
            }
            return;
        }
        // rows whose shards are added up here are dealt out over the shards' blocks
        const int unit = g.rel_w[0] ? block * g.n_shards + (int)blockIdx.y : block;
        if (unit >= g.n_rel * g.n_tables) return;
        // (the order of a sum is part of an L1 model's result, see k_pair_bwd: TransH's have eight strands, the others four)
        if (g.n_tables > 1) relation_row_sum<V, kSegmentLanes, 2>(shards, g, unit, rel_part, rel_perm);
        else relation_row_sum<V, kSegmentLanes, 1>(shards, g, unit, rel_part, rel_perm);
        return;
    }
    uint8_t* __restrict__ table = rr.table;
    const uint8_t* __restrict__ rows_c = rr.rows_c;
    const uint32_t* __restrict__ remote = rr.remote;
    const uint32_t* __restrict__ perm = rr.perm;
    const uint32_t* __restrict__ off = rr.off;
    const uint32_t* __restrict__ first_slot = rr.first_slot;
    const float* __restrict__ d_head = rr.d_head;
    const float* __restrict__ grad_recv = rr.grad_recv;
    float* __restrict__ d_hid_h = rr.d_hid_h;
    float* __restrict__ d_hid_t = rr.d_hid_t;
    const HeavyRows& heavy = rr.heavy;
    exchange_wait(g.sync, XCHG_TAIL_GRADS);  // grad_recv is written by the other processes
    // partial sums of the item lanes, [lane][head | tail][64 column threads][V]
    __shared__ float part[kSegmentLanes][2][64 * V];
    __shared__ uint32_t s_perm[64 * kSegmentLanes];
    __shared__ int s_last;
    const int D = L.d;
    const int col = threadIdx.x & 63, lane = threadIdx.x >> 6;
    const bool helper = (int)blockIdx.x < kHeavySlots;
    int r;
    uint32_t q0, q1, info = 0, slot_word;
    size_t row;
    uint4 first4 = make_uint4(0u, 0u, 0u, 0u);
    if (helper) {
        if (blockIdx.x >= *heavy.count) return;
        const uint4 h = heavy.parts[blockIdx.x];
        r = (int)h.x; q0 = h.y; q1 = h.z; info = h.w;
        slot_word = first_slot[r]; row = remote[r];
    } else {
        // one warp per gathered row: nothing in a row's update needs more than a warp, and a block of
        // eight independent warps keeps eight rows' loads in flight
        r = ((int)blockIdx.x - kHeavySlots) * kRowsPerBlock + (int)(threadIdx.x >> 5);
        if (r >= R) return;
        if (heavy.row_info) {
            const uint4 a = heavy.row_info[2 * r];
            first4 = heavy.row_info[2 * r + 1];
            q0 = a.x; q1 = a.x + a.y; slot_word = a.z; row = a.w;
        } else {
            slot_word = first_slot[r]; q0 = off[r]; q1 = off[r + 1]; row = remote[r];
        }
        if (slot_word & 2u) return;  // its lookups are summed part by part by the first blocks
        if (!d_hid_h && !(slot_word & 1u)) return;  // a padding slot behind the first one, and nobody reads its gradient
    }
    ST* xv = reinterpret_cast<ST*>(table + row * L.row_bytes);
    ST* mv = reinterpret_cast<ST*>(table + row * L.row_bytes + L.off_m);
    ST* qv = reinterpret_cast<ST*>(table + row * L.row_bytes + L.off_q);
    // the state before the update comes from the step's gathered copy (slot r), not from the table
    const uint8_t* const state = DIRECT ? table + row * L.row_bytes : rows_c + (size_t)r * L.row_bytes;
    const ST* xs = reinterpret_cast<const ST*>(state);
    const ST* ms = reinterpret_cast<const ST*>(state + L.off_m);
    const ST* qs = reinterpret_cast<const ST*>(state + L.off_q);
    const float alpha = *g.step_size * g.lr_modifier;
    const bool writes_row = (slot_word & 1u) != 0;

    // Sums of the lookups [q0, q1) for the columns c .. c+V-1, separately for head and tail lookups;
    // complete in the threads of lane 0.  Lane l sums the lookups q0 + l, q0 + l + lanes, ... in
    // that order, four loads in flight; the lanes' partial sums are then added in lane order: a
    // fixed tree, whatever the timing.  Called by all threads of the block.
    auto segment_sums = [&](int c, float (&gh)[V], float (&gt)[V]) {
#pragma unroll
        for (int u = 0; u < V; ++u) gh[u] = gt[u] = 0.f;
        for (uint32_t base = q0; base < q1; base += 64 * kSegmentLanes) {
            // the segment's lookups go through shared memory, so the row loads do not wait on them
            const int count = (int)min((uint32_t)(64 * kSegmentLanes), q1 - base);
            __syncthreads();
            if ((int)threadIdx.x < count) s_perm[threadIdx.x] = perm[base + threadIdx.x];
            __syncthreads();
            if (c >= D) continue;
            for (int q = lane; q < count; q += 4 * kSegmentLanes) {
                uint32_t e[4];
                float4 v[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) e[u] = q + u * kSegmentLanes < count ? s_perm[q + u * kSegmentLanes] : 0xffffffffu;
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    v[u] = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (e[u] == 0xffffffffu) continue;
                    const float* src = e[u] < (uint32_t)B ? d_head + (size_t)e[u] * D + c
                                                          : grad_recv + (size_t)(e[u] - B) * D + c;
                    if (V == 4) v[u] = load4(src); else v[u].x = src[0];
                }
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    if (e[u] == 0xffffffffu) continue;
                    if (e[u] < (uint32_t)B) {
                        gh[0] += v[u].x;
                        if (V == 4) { gh[1 % V] += v[u].y; gh[2 % V] += v[u].z; gh[3 % V] += v[u].w; }
                    } else {
                        gt[0] += v[u].x;
                        if (V == 4) { gt[1 % V] += v[u].y; gt[2 % V] += v[u].z; gt[3 % V] += v[u].w; }
                    }
                }
            }
        }
        __syncthreads();  // the previous column block's partials have been consumed
#pragma unroll
        for (int u = 0; u < V; ++u) {
            part[lane][0][col * V + u] = gh[u];
            part[lane][1][col * V + u] = gt[u];
        }
        __syncthreads();
        if (lane != 0) return;
#pragma unroll
        for (int u = 0; u < V; ++u) {
            gh[u] = part[0][0][col * V + u];
            gt[u] = part[0][1][col * V + u];
#pragma unroll
            for (int l = 1; l < kSegmentLanes; ++l) {
                gh[u] += part[l][0][col * V + u];
                gt[u] += part[l][1][col * V + u];
            }
        }
    };

    // The row's hidden gradients and its Adam step for the columns c .. c+V-1 (one thread).
    auto finish = [&](int c, float (&gh)[V], float (&gt)[V]) {
        const size_t o = (size_t)r * D + c;
        float gv[V];  // the value's gradient: the lookups' sums (+ the regularisers' terms for the value)
#pragma unroll
        for (int u = 0; u < V; ++u) gv[u] = gh[u] + gt[u];
        if (EXTRAS && rr.reg_val) {
            // gh / gt become the gradients of the feature network's output
#pragma unroll
            for (int u = 0; u < V; ++u) {
                gv[u] += rr.reg_val[o + u];
                gh[u] += rr.reg_h[o + u];
                if (rr.reg_t) gt[u] += rr.reg_t[o + u];
            }
        }
        if (EXTRAS && rr.drop.threshold) {
            // through the dropout of each call: kept elements pass g / (1 - p)
            const uint32_t keep_h = dropout_keep4(rr.drop, 0u, (uint32_t)r, (uint32_t)c >> 2), keep_t = dropout_keep4(rr.drop, 1u, (uint32_t)r, (uint32_t)c >> 2);
#pragma unroll
            for (int u = 0; u < V; ++u) {
                const int bit = (c & 3) + u;
                gh[u] = (keep_h >> bit) & 1u ? gh[u] * rr.drop.scale : 0.f;
                gt[u] = (keep_t >> bit) & 1u ? gt[u] * rr.drop.scale : 0.f;
            }
        }
        if (!d_hid_h) {
            // no features: nothing reads the hidden rows' gradients
        } else if (V == 4) {
            if (d_hid_t) {
                const float4 a = make_float4(gh[0], gh[1 % V], gh[2 % V], gh[3 % V]), b = make_float4(gt[0], gt[1 % V], gt[2 % V], gt[3 % V]);
                store4(d_hid_h + o, a);
                store4(d_hid_t + o, b);
                if (rr.d_hid_h_lo) store4(rr.d_hid_h_lo + o, tf32_lower4(a));
                if (rr.d_hid_t_lo) store4(rr.d_hid_t_lo + o, tf32_lower4(b));
            } else {
                const float4 a = make_float4(gh[0] + gt[0], gh[1 % V] + gt[1 % V], gh[2 % V] + gt[2 % V], gh[3 % V] + gt[3 % V]);
                store4(d_hid_h + o, a);
                if (rr.d_hid_h_lo) store4(rr.d_hid_h_lo + o, tf32_lower4(a));  // lower plane for the projection gradient
            }
        } else {
            d_hid_h[o] = d_hid_t ? gh[0] : gh[0] + gt[0];
            if (d_hid_t) d_hid_t[o] = gt[0];
        }
        if (EXTRAS && rr.defer_grad) {
#pragma unroll
            for (int u = 0; u < V; ++u) rr.defer_grad[o + u] = gv[u];
            return;
        }
        if (!writes_row) return;
        float x[V], m[V], qq[V];
        if (V == 4) {
            const float4 a = L.value_bf16 ? load4(reinterpret_cast<const __nv_bfloat16*>(xs) + c) : load4(xs + c), b = load4(ms + c), d = load4(qs + c);
            x[0] = a.x; x[1 % V] = a.y; x[2 % V] = a.z; x[3 % V] = a.w;
            m[0] = b.x; m[1 % V] = b.y; m[2 % V] = b.z; m[3 % V] = b.w;
            qq[0] = d.x; qq[1 % V] = d.y; qq[2 % V] = d.z; qq[3 % V] = d.w;
        } else {
            x[0] = load_value<ST>(L, reinterpret_cast<const uint8_t*>(xs), c); m[0] = load_as_float(ms + c); qq[0] = load_as_float(qs + c);
        }
#pragma unroll
        for (int u = 0; u < V; ++u) {
            const float v = weighted_sum(__fmul_rn(ap.one_minus_beta_v, gv[u]), gv[u], ap.beta_v, __fmul_rn(qq[u], qq[u]));
            m[u] = weighted_sum(ap.one_minus_beta_m, gv[u], ap.beta_m, m[u]);
            x[u] = x[u] - alpha * (m[u] / (sqrtf(v) + ap.epsilon) + ap.weight_decay * x[u]);
            qq[u] = sqrtf(v);
        }
        if (V == 4) {
            if (L.value_bf16) store4(reinterpret_cast<__nv_bfloat16*>(xv) + c, make_float4(x[0], x[1 % V], x[2 % V], x[3 % V]));
            else store4(xv + c, make_float4(x[0], x[1 % V], x[2 % V], x[3 % V]));
            store4(mv + c, make_float4(m[0], m[1 % V], m[2 % V], m[3 % V]));
            store4(qv + c, make_float4(qq[0], qq[1 % V], qq[2 % V], qq[3 % V]));
        } else {
            store_value<ST>(L, reinterpret_cast<uint8_t*>(xv), c, x[0]);
            store_from_float(mv + c, m[0]);
            store_from_float(qv + c, qq[0]);
        }
    };

    float gh[V], gt[V];
    if (!helper) {
        // the row's lookups in position order, four lookups and two column chunks (eight loads) in
        // flight; head and tail lookups apart
        const int wl = threadIdx.x & 31;
        if (writes_row && (wl & 7) == 0) {
            // The row's state is needed only after its gradient rows have been summed, but its address is
            // known now: ask L2 for it (one request per 128-byte line, no registers held).
            for (int c = wl * V; c < D; c += 32 * V) {
                asm volatile("prefetch.global.L2 [%0];" ::"l"(L.value_bf16 ? reinterpret_cast<const void*>(reinterpret_cast<const __nv_bfloat16*>(xs) + c)
                                                                             : reinterpret_cast<const void*>(xs + c)));
                asm volatile("prefetch.global.L2 [%0];" ::"l"(ms + c));
                asm volatile("prefetch.global.L2 [%0];" ::"l"(qs + c));
            }
        }
        for (int c0 = 0; c0 < D; c0 += 64 * V) {
            const int ca = c0 + wl * V, cb = ca + 32 * V;
            if (ca >= D) continue;
            const bool two = cb < D;
            float hb[V], tb[V];
#pragma unroll
            for (int u = 0; u < V; ++u) gh[u] = gt[u] = hb[u] = tb[u] = 0.f;
            for (uint32_t q = q0; q < q1; q += 4) {
                uint32_t e[4];
                float4 ga[4], gb[4];
                if (heavy.row_info && q == q0) {  // the first four lookups came with the row's descriptor
                    e[0] = first4.x; e[1] = first4.y; e[2] = first4.z; e[3] = first4.w;
                } else {
#pragma unroll
                    for (int u = 0; u < 4; ++u) e[u] = q + u < q1 ? perm[q + u] : 0xffffffffu;
                }
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    ga[u] = gb[u] = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (e[u] == 0xffffffffu) continue;
                    const float* src = e[u] < (uint32_t)B ? d_head + (size_t)e[u] * D : grad_recv + (size_t)(e[u] - B) * D;
                    if (V == 4) {
                        ga[u] = load4(src + ca);
                        if (two) gb[u] = load4(src + cb);
                    } else {
                        ga[u].x = src[ca];
                        if (two) gb[u].x = src[cb];
                    }
                }
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    if (e[u] == 0xffffffffu) continue;
                    if (e[u] < (uint32_t)B) {
                        gh[0] += ga[u].x; hb[0] += gb[u].x;
                        if (V == 4) {
                            gh[1 % V] += ga[u].y; gh[2 % V] += ga[u].z; gh[3 % V] += ga[u].w;
                            hb[1 % V] += gb[u].y; hb[2 % V] += gb[u].z; hb[3 % V] += gb[u].w;
                        }
                    } else {
                        gt[0] += ga[u].x; tb[0] += gb[u].x;
                        if (V == 4) {
                            gt[1 % V] += ga[u].y; gt[2 % V] += ga[u].z; gt[3 % V] += ga[u].w;
                            tb[1 % V] += gb[u].y; tb[2 % V] += gb[u].z; tb[3 % V] += gb[u].w;
                        }
                    }
                }
            }
            finish(ca, gh, gt);
            if (two) finish(cb, hb, tb);
        }
        return;
    }
    // one part of a popular row: leave its sums; the part that arrives last adds all of them
    const int first = (int)(info >> 16), parts = (int)((info >> 8) & 255u), me = (int)(info & 255u);
    for (int c0 = 0; c0 < D; c0 += 64 * V) {
        const int c = c0 + col * V;
        segment_sums(c, gh, gt);
        if (lane == 0 && c < D) {
            float* mine = heavy.partial + (size_t)(first + me) * 2 * D;
#pragma unroll
            for (int u = 0; u < V; ++u) {
                mine[c + u] = gh[u];
                mine[D + c + u] = gt[u];
            }
        }
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        const unsigned arrived = atomicAdd(&heavy.counter[first], 1u) + 1u;
        s_last = arrived == (unsigned)parts;
        if (s_last) heavy.counter[first] = 0;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    if (lane != 0) return;
    for (int c = col * V; c < D; c += 64 * V) {
#pragma unroll
        for (int u = 0; u < V; ++u) gh[u] = gt[u] = 0.f;
        for (int p = 0; p < parts; ++p) {
            const float* theirs = heavy.partial + (size_t)(first + p) * 2 * D;
#pragma unroll
            for (int u = 0; u < V; ++u) {
                gh[u] += __ldcg(theirs + c + u);
                gt[u] += __ldcg(theirs + D + c + u);
            }
        }
        finish(c, gh, gt);
    }
}

template <class ST, int V, bool EXTRAS = false, bool DIRECT = false>
inline cudaError_t launch_entity_update(const ShardArgs<EntityShard>& shards, const EntityStep& g, cudaStream_t stream) {
    const int loss_blocks = shards.s[0].loss_rows ? 1 : 0;
    const dim3 grid((unsigned)(kHeavySlots + (g.R + kRowsPerBlock - 1) / kRowsPerBlock + g.rel_blocks + loss_blocks), (unsigned)g.n_shards);
    return launch_dependent(k_entity_update<ST, V, EXTRAS, DIRECT>, grid, dim3(64 * kSegmentLanes), 0, stream, shards, g);
}

// ---------------------------------------------------------------------------
// Projection backward: dW[f, d] (+)= sum_r feature[remote[r], f] * d_hidden[r, d]
// (src/pag/pag.cpp:695-700).  A = feature^T is read from the gathered table rows; the r
// range is split over blockIdx.z and each split writes its own partial, summed later in
// a fixed order.  Same 64x64x16 tiling as k_hidden.  gridDim.z = n_net * splits.
template <class FT>
__global__ void __launch_bounds__(256)
k_projection_bwd(const uint8_t* __restrict__ table, RowLayout L, const uint32_t* __restrict__ remote,
                 int R, const float* __restrict__ dh0, const float* __restrict__ dh1, int splits,
                 int rows_per_split, float* __restrict__ partial) {
    grid_dependency_sync();
    constexpr int BM = 64, BN = 64, BK = 16;
    __shared__ __align__(16) float As[BK][BM];
    __shared__ __align__(16) float Bs[BK][BN];
    const int D = L.d, F = L.f;
    const int net = blockIdx.z / splits, split = blockIdx.z - net * splits;
    const float* __restrict__ dh = net ? dh1 : dh0;
    float* __restrict__ out = partial + ((size_t)net * splits + split) * (size_t)F * D;
    const int t = threadIdx.x, tx = t & 15, ty = t >> 4;
    const int m0 = blockIdx.x * BM, n0 = blockIdx.y * BN;
    const int r_lo = split * rows_per_split, r_hi = min(R, r_lo + rows_per_split);
    const int ld_k = t >> 4, ld_c = (t & 15) * 4;
    const bool d_vec = (D & 3) == 0;

    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;

    for (int r0 = r_lo; r0 < r_hi; r0 += BK) {
        const int r = r0 + ld_k;
        float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a;
        if (r < r_hi) {
            const size_t row = remote ? remote[r] : (size_t)r;
            const FT* fp = reinterpret_cast<const FT*>(table + row * L.row_bytes + L.off_feat);
            const int f = m0 + ld_c;
            if (f + 3 < F) {
                a = load4(fp + f);
            } else {
                if (f + 0 < F) a.x = load_as_float(fp + f + 0);
                if (f + 1 < F) a.y = load_as_float(fp + f + 1);
                if (f + 2 < F) a.z = load_as_float(fp + f + 2);
            }
            const int n = n0 + ld_c;
            const float* gp = dh + (size_t)r * D + n;
            if (d_vec && n + 3 < D) {
                b = load4(gp);
            } else {
                if (n + 0 < D) b.x = gp[0];
                if (n + 1 < D) b.y = gp[1];
                if (n + 2 < D) b.z = gp[2];
                if (n + 3 < D) b.w = gp[3];
            }
        }
        __syncthreads();
        store4(&As[ld_k][ld_c], a);
        store4(&Bs[ld_k][ld_c], b);
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < BK; ++kk) {
            const float4 av = load4(&As[kk][ty * 4]);
            const float4 bv = load4(&Bs[kk][tx * 4]);
            const float ar[4] = {av.x, av.y, av.z, av.w};
            const float br[4] = {bv.x, bv.y, bv.z, bv.w};
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(ar[i], br[j], acc[i][j]);
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int f = m0 + ty * 4 + i;
        if (f >= F) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int n = n0 + tx * 4 + j;
            if (n < D) out[(size_t)f * D + n] = acc[i][j];
        }
    }
}

// This shard's contribution to the dense gradients, laid out like the dense parameter
// vector: relation table | projection(s), and written slice by slice into the memory of the
// process that owns (reduces and updates) each row: the rows are dealt out in turn, row r to
// process r % n_owner as its row r / n_owner, so that every process receives and updates an
// equal share of every parameter; dense_dst[owner] is this shard's slot in that process's
// receive buffer.  Relation rows are the segment sums of the
// per-triple relation gradients (backward of the gather at src/poplar_kge.cpp:489);
// projection entries sum the split partials of k_projection_bwd in split order.
constexpr int kRelationLanes = 8;

template <int V>
__global__ void __launch_bounds__(64 * kRelationLanes)
k_dense_partial(const float* __restrict__ d_relrow, const uint32_t* __restrict__ rel_perm,
                const uint32_t* __restrict__ rel_off, int n_rel, int D,
                const float* __restrict__ proj_partial, int n_net, int splits, size_t proj_elems,
                float* const* __restrict__ dense_dst, int n_owner, ExchangeSync sync, int signal_kind, int row_offset) {
    grid_dependency_sync();
    __shared__ float part[kRelationLanes][64 * V];
    __shared__ uint32_t s_perm[64 * kRelationLanes];
    if ((int)blockIdx.x < n_rel) {
        // One relation row.  Relation popularity is skewed, so a few rows own most of the batch's
        // triples: the row's lookups are staged in shared memory, lane l sums triples l, l + lanes,
        // ... (four loads in flight) and the lanes' partial sums are added in lane order.
        const int rho = blockIdx.x, col = threadIdx.x & 63, lane = threadIdx.x >> 6;
        const uint32_t q0 = rel_off[rho], q1 = rel_off[rho + 1];
        // the row goes to the process that owns this slice of the dense vector
        // (row_offset: where these rows begin in the dense vector; 0 for the relation table)
        const int owner = (rho + row_offset) % n_owner;
        float* __restrict__ dst_row = dense_dst[owner] + (size_t)((rho + row_offset) / n_owner) * D;
        if (q0 == q1) {
            for (int c = threadIdx.x; c < D; c += blockDim.x) dst_row[c] = 0.f;
            exchange_signal(sync, signal_kind, gridDim.x);
            return;
        }
        for (int c0 = 0; c0 < D; c0 += 64 * V) {
            const int c = c0 + col * V;
            float g[V];
#pragma unroll
            for (int u = 0; u < V; ++u) g[u] = 0.f;
            for (uint32_t base = q0; base < q1; base += 64 * kRelationLanes) {
                const int count = (int)min((uint32_t)(64 * kRelationLanes), q1 - base);
                __syncthreads();
                if ((int)threadIdx.x < count) s_perm[threadIdx.x] = rel_perm[base + threadIdx.x];
                __syncthreads();
                if (c >= D) continue;
                for (int i = lane; i < count; i += 4 * kRelationLanes) {
                    float4 v[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const int ii = i + u * kRelationLanes;
                        v[u] = make_float4(0.f, 0.f, 0.f, 0.f);
                        if (ii < count) {
                            const float* src = d_relrow + (size_t)s_perm[ii] * D + c;
                            if (V == 4) v[u] = load4(src); else v[u].x = src[0];
                        }
                    }
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        if (i + u * kRelationLanes >= count) continue;
                        g[0] += v[u].x;
                        if (V == 4) { g[1 % V] += v[u].y; g[2 % V] += v[u].z; g[3 % V] += v[u].w; }
                    }
                }
            }
            __syncthreads();
#pragma unroll
            for (int u = 0; u < V; ++u) part[lane][col * V + u] = g[u];
            __syncthreads();
            if (lane == 0 && c < D) {
#pragma unroll
                for (int u = 0; u < V; ++u) {
                    float total = part[0][col * V + u];
#pragma unroll
                    for (int l = 1; l < kRelationLanes; ++l) total += part[l][col * V + u];
                    dst_row[c + u] = total;
                }
            }
        }
        exchange_signal(sync, signal_kind, gridDim.x);
        return;
    }
    const size_t rel_elems = (size_t)n_rel * D;
    const size_t total = (size_t)n_net * proj_elems;
    const size_t first = ((size_t)blockIdx.x - n_rel) * blockDim.x + threadIdx.x;
    const size_t stride = ((size_t)gridDim.x - n_rel) * blockDim.x;
    for (size_t pe = first; pe < total; pe += stride) {
        const size_t net = pe / proj_elems, idx = pe - net * proj_elems;
        float g = 0.f;
        for (int z = 0; z < splits; ++z) g += proj_partial[(net * splits + z) * proj_elems + idx];
        const size_t e = rel_elems + pe, row = e / D;
        dense_dst[row % n_owner][(row / n_owner) * D + (e - row * D)] = g;
    }
    exchange_signal(sync, signal_kind, gridDim.x);
}

// Sum of the shards' dense contributions in shard order (the reduce-scatter of
// src/pag/pag.cpp:980-994), Adam on the slice of the dense vector this process owns
// (src/poplar_kge.cpp:329-339) and the write of the new values into every replica
// (the all-gather on next use, :341-348).  Pointer tables live in device memory; entries
// may point into peers' memory.
constexpr int kDenseParams = 8;
struct DenseUpdateArgs {
    const float* const* partials;  // [n_partial] the shards' slots in this process's receive buffer
    int n_partial;
    float* const* replicas;  // [n_replica] dense parameter vectors
    float* const* replicas_lo;  // [n_replica] their lower TF32 planes (the projections are tensor-core operands); null: none
    int n_replica;
    float* adam_m;
    float* adam_v;
    // This process owns the rows self, self + n_replica, ... of the dense vector: n_own of them,
    // row_width elements each; its j-th row is row j of every slot.
    size_t n_own, row_width;
    // parameter p covers the elements [bounds[p], bounds[p+1]): relation table, projection(s), TransH
    // normals, the feature MLP's up / down projections per network; absent ones are empty
    size_t bounds[kDenseParams + 1];
    float lr_modifier[kDenseParams];
    const float* step_size;
    AdamParams ap;
    ExchangeSync sync;
};

__device__ __forceinline__ int dense_param_of(const DenseUpdateArgs& a, size_t e) {
    int p = 0;
    while (p + 1 < kDenseParams && e >= a.bounds[p + 1]) ++p;
    return p;
}

__device__ __forceinline__ float dense_adam(float x, float g, float& m, float& v, float alpha, const AdamParams& ap) {
    m = weighted_sum(ap.beta_m, m, ap.one_minus_beta_m, g);
    v = weighted_sum(ap.beta_v, v, __fmul_rn(ap.one_minus_beta_v, g), g);
    return x - alpha * (m / (sqrtf(v) + ap.epsilon) + ap.weight_decay * x);
}

// The shards' partial gradients of the owned slice have been written into this process's
// receive buffer by their producers; the new values are written to every process's copy of the
// parameters (posted stores over NVLink).  Four elements per access.
static __global__ void __launch_bounds__(256) k_dense_update(DenseUpdateArgs a, int self) {
    grid_dependency_sync();
    exchange_wait(a.sync, XCHG_DENSE_PARTIALS);  // every process's partial gradients are complete
    const float base_alpha = *a.step_size;
    const size_t W = a.row_width, total = a.n_own * W;
    size_t all_bounds = W;
    for (int p = 1; p <= kDenseParams; ++p) all_bounds |= a.bounds[p];
    const bool vec = (all_bounds & 3) == 0;
    if (vec) {
        for (size_t le = 4 * ((size_t)blockIdx.x * blockDim.x + threadIdx.x); le < total; le += 4 * (size_t)gridDim.x * blockDim.x) {
            const size_t j = le / W, e = (j * a.n_replica + self) * W + (le - j * W);  // slot index -> dense index
            float4 g = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
            for (int s = 0; s < a.n_partial; ++s) {
                const float4 t = *reinterpret_cast<const float4*>(a.partials[s] + le);
                g.x += t.x; g.y += t.y; g.z += t.z; g.w += t.w;
            }
            const int p = dense_param_of(a, e);
            const float alpha = base_alpha * a.lr_modifier[p];
            float4 x = *reinterpret_cast<const float4*>(a.replicas[self] + e);
            float4 m = *reinterpret_cast<const float4*>(a.adam_m + e), v = *reinterpret_cast<const float4*>(a.adam_v + e);
            x.x = dense_adam(x.x, g.x, m.x, v.x, alpha, a.ap);
            x.y = dense_adam(x.y, g.y, m.y, v.y, alpha, a.ap);
            x.z = dense_adam(x.z, g.z, m.z, v.z, alpha, a.ap);
            x.w = dense_adam(x.w, g.w, m.w, v.w, alpha, a.ap);
            *reinterpret_cast<float4*>(a.adam_m + e) = m;
            *reinterpret_cast<float4*>(a.adam_v + e) = v;
            for (int rep = 0; rep < a.n_replica; ++rep) *reinterpret_cast<float4*>(a.replicas[rep] + e) = x;
            if (a.replicas_lo && p > 0) {
                const float4 lo = tf32_lower4(x);
                for (int rep = 0; rep < a.n_replica; ++rep) *reinterpret_cast<float4*>(a.replicas_lo[rep] + e) = lo;
            }
        }
    } else {
        for (size_t le = (size_t)blockIdx.x * blockDim.x + threadIdx.x; le < total; le += (size_t)gridDim.x * blockDim.x) {
            const size_t j = le / W, e = (j * a.n_replica + self) * W + (le - j * W);
            float g = 0.f;
            for (int s = 0; s < a.n_partial; ++s) g += a.partials[s][le];
            const int p = dense_param_of(a, e);
            const float alpha = base_alpha * a.lr_modifier[p];
            float m = a.adam_m[e], v = a.adam_v[e];
            const float x = dense_adam(a.replicas[self][e], g, m, v, alpha, a.ap);
            a.adam_m[e] = m;
            a.adam_v[e] = v;
            for (int rep = 0; rep < a.n_replica; ++rep) a.replicas[rep][e] = x;
            if (a.replicas_lo && p > 0)
                for (int rep = 0; rep < a.n_replica; ++rep) a.replicas_lo[rep][e] = tf32_lower(x);
        }
    }
    exchange_signal(a.sync, XCHG_DENSE_PARAMS, gridDim.x);  // the new values are in every process's copy
}

// ---------------------------------------------------------------------------
// Cross-process barrier on flags in peer-visible memory.  Thread r publishes this
// process's new epoch into peer r's flag array, then waits until peer r's epoch has
// reached it.  The wait is bounded: on expiry the kernel records an error and returns.
struct BarrierArgs {
    unsigned* const* peer_flags;  // [world] base of each process's flag array
    unsigned* my_epoch;           // device counter, incremented once per barrier
    unsigned* status;             // device error word: non-zero = a wait gave up
    int rank, world;
    unsigned long long max_spins;
};

static __global__ void k_barrier(BarrierArgs a) {
    grid_dependency_sync();
    __shared__ unsigned epoch;
    if (threadIdx.x == 0) {
        epoch = *a.my_epoch + 1;
        *a.my_epoch = epoch;
        __threadfence_system();
    }
    __syncthreads();
    const int r = threadIdx.x;
    if (r >= a.world) return;
    volatile unsigned* remote_flag = a.peer_flags[r] + a.rank;
    __threadfence_system();
    *remote_flag = epoch;
    volatile unsigned* mine = a.peer_flags[a.rank] + r;
    // Once a wait has given up, the run is lost: later barriers of the same run do not wait again.
    if (*reinterpret_cast<volatile unsigned*>(a.status) != 0) return;
    unsigned long long spins = 0;
    while ((int)(*mine - epoch) < 0) {
        if (++spins > a.max_spins) {
            atomicExch(a.status, 1u + (unsigned)r);
            break;
        }
        __nanosleep(64);
    }
    __threadfence_system();
}

// ---------------------------------------------------------------------------
// Streaming top-k of predict (src/poplar_kge.cpp:743-810): every query keeps its n_best
// highest-scoring candidates so far; a batch of scores is merged by one warp per query.
// Candidates that beat the query's current cut-off are appended to a per-warp buffer in
// shared memory (warp ballot: the order is fixed) and the buffer is sorted down to n_best
// when it fills.  Order: higher score first, ties by lower row index, so the result does not
// depend on the batch size.  The reference leaves the tie order undefined.
constexpr int kTopkCapacity = 256;  // entries per query buffer; n_best <= capacity / 2

__device__ __forceinline__ unsigned long long topk_key(float score, uint32_t index) {
    uint32_t bits = __float_as_uint(score);
    bits = (bits & 0x80000000u) ? ~bits : (bits | 0x80000000u);  // monotone in the float order
    return ((unsigned long long)bits << 32) | (uint32_t)(~index);
}
__device__ __forceinline__ float topk_score(unsigned long long key) {
    uint32_t bits = (uint32_t)(key >> 32);
    bits = (bits & 0x80000000u) ? (bits & 0x7fffffffu) : ~bits;
    return __uint_as_float(bits);
}
__device__ __forceinline__ uint32_t topk_index(unsigned long long key) { return ~(uint32_t)key; }

// Sorts the warp's buffer in descending key order (empty slots hold key 0, which sorts last): a bitonic network on eight
// keys per lane, key p of the network in lane p / 8, so that 21 of its 36 stages stay inside a lane and the other 15
// exchange through shuffles.  The outer stages are rolled: a sort is run by few warps, now and then, and 40 KB of
// straight-line code took longer to fetch than to run.  (In shared memory, one compare-exchange per visit: 10 us.)
__device__ __forceinline__ void order_desc(unsigned long long& a, unsigned long long& b, bool descending) {
    const bool swap = (a < b) == descending;
    const unsigned long long t = swap ? b : a;
    b = swap ? a : b;
    a = t;
}
__device__ __forceinline__ void warp_sort_desc(unsigned long long* buf) {
    constexpr int kPerLane = kTopkCapacity / 32;
    static_assert(kPerLane == 8, "stages of 4, 2 and 1 inside a lane");
    const int lane = threadIdx.x & 31;
    unsigned long long v[kPerLane];
    __syncwarp();
#pragma unroll
    for (int r = 0; r < kPerLane; ++r) v[r] = buf[r * 32 + lane];  // in any order: they are about to be sorted
    __syncwarp();
    auto inside = [&](bool descending) {
#pragma unroll
        for (int j = 4; j > 0; j >>= 1)
#pragma unroll
            for (int r = 0; r < kPerLane; ++r)
                if (!(r & j)) order_desc(v[r], v[r | j], descending);
    };
#pragma unroll
    for (int r = 0; r < kPerLane; r += 2) order_desc(v[r], v[r + 1], (r & 2) == 0);
#pragma unroll
    for (int j = 2; j > 0; j >>= 1)
#pragma unroll
        for (int r = 0; r < kPerLane; ++r)
            if (!(r & j)) order_desc(v[r], v[r | j], (r & 4) == 0);
    inside((lane & 1) == 0);
#pragma unroll 1
    for (int k = 2; k <= 32; k <<= 1) {  // in lanes
        const bool descending = (lane & k) == 0;
#pragma unroll 1
        for (int j = k >> 1; j > 0; j >>= 1) {
            const bool keep_larger = ((lane & j) == 0) == descending;
#pragma unroll
            for (int r = 0; r < kPerLane; ++r) {
                const unsigned long long other = __shfl_xor_sync(0xffffffffu, v[r], j);
                v[r] = (v[r] > other) == keep_larger ? v[r] : other;
            }
        }
        inside(descending);
    }
#pragma unroll
    for (int r = 0; r < kPerLane; r += 2) *reinterpret_cast<ulonglong2*>(buf + lane * kPerLane + r) = make_ulonglong2(v[r], v[r + 1]);
    __syncwarp();
}

struct TopkParams {
    int n_query, n_best;
    int score_is_gamma_minus;  // TransE: score = gamma - raw
    float gamma;
};

// A batch of scores is merged in two kernels.  k_topk_filter reads all of it at full bandwidth
// (four scores per thread) and leaves, per query, the keys that beat the query's cut-off as it
// stands before the batch in `cand` (at most kTopkCandidates; the count goes on past that).
// k_topk_update, one warp per query, then merges those few keys; a query whose candidates did not
// fit scans its row of scores itself.  In a ranking's first batch, before a cut-off exists, k_topk_seed
// takes the filter's place.  The candidates' order in `cand` depends on timing, the merged result does
// not: it is the n_best largest keys of the old list and the candidates, and keys are unique.
constexpr int kTopkCandidates = 1024;

static __global__ void __launch_bounds__(256)
k_topk_filter(const float* __restrict__ raw, int n_cols, uint32_t first_row, uint32_t last_valid_row,
              const unsigned long long* __restrict__ state, const int* __restrict__ counts,
              unsigned long long* __restrict__ cand, int* __restrict__ cand_count, TopkParams tp) {
    const int q = blockIdx.y, lane = threadIdx.x & 31;
    const unsigned long long cutoff = counts[q] >= tp.n_best ? state[(size_t)q * kTopkCapacity + tp.n_best - 1] : 0ull;
    if (cutoff == 0ull) {  // no cut-off yet: every score is a candidate, the query scans its row itself
        if (blockIdx.x == 0 && threadIdx.x == 0) cand_count[q] = kTopkCandidates + 1;
        return;
    }
    const float* __restrict__ row = raw + (size_t)q * n_cols;
    const bool vec = (n_cols & 3) == 0;
    // a warp walks 128 consecutive scores at a time; its lanes stay together for the ballots
    for (int w0 = 4 * (blockIdx.x * 256 + (threadIdx.x & ~31)); w0 < n_cols; w0 += 4 * 256 * gridDim.x) {
        const int j0 = w0 + 4 * lane;
        float v[4] = {0.f, 0.f, 0.f, 0.f};
        if (j0 < n_cols) {
            if (vec) {
                const float4 x = *reinterpret_cast<const float4*>(row + j0);
                v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
            } else {
                for (int u = 0; u < 4 && j0 + u < n_cols; ++u) v[u] = row[j0 + u];
            }
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int j = j0 + u;
            unsigned long long key = 0ull;
            if (j < n_cols && first_row + (uint32_t)j <= last_valid_row)
                key = topk_key(tp.score_is_gamma_minus ? tp.gamma - v[u] : v[u], first_row + (uint32_t)j);
            const bool pass = key > cutoff;
            const unsigned mask = __ballot_sync(0xffffffffu, pass);
            if (mask == 0) continue;
            int base = 0;
            if (lane == __ffs(mask) - 1) base = atomicAdd(cand_count + q, __popc(mask));  // one addition per warp
            base = __shfl_sync(0xffffffffu, base, __ffs(mask) - 1);
            const int slot = base + __popc(mask & ((1u << lane) - 1));
            if (pass && slot < kTopkCandidates) cand[(size_t)q * kTopkCandidates + slot] = key;
        }
    }
}

// The lanes' keys in descending order.
__device__ __forceinline__ unsigned long long lanes_sort_desc(unsigned long long key) {
    const int lane = threadIdx.x & 31;
#pragma unroll 1
    for (int k = 2; k <= 32; k <<= 1)
#pragma unroll 1
        for (int j = k >> 1; j > 0; j >>= 1) {
            const unsigned long long other = __shfl_xor_sync(0xffffffffu, key, j);
            const bool keep_larger = ((lane & j) == 0) == ((lane & k) == 0);
            key = (key > other) == keep_larger ? key : other;
        }
    return key;
}

// The first `count` of kTopkCapacity keys in descending order, zeros behind them.
static __device__ __noinline__ void topk_sort(unsigned long long* buf, int count) {
    for (int i = count + (threadIdx.x & 31); i < kTopkCapacity; i += 32) buf[i] = 0ull;
    __syncwarp();
    warp_sort_desc(buf);
}

// One warp's list: up to kTopkCapacity keys in shared memory, sorted down to the n_best largest when it fills.
struct TopkList {
    unsigned long long* buf;
    int count, n_best;
    unsigned long long cutoff;  // keys up to it cannot be among the n_best

    // A list of up to 32 keys, as a first scan with a cut-off leaves, is sorted a key per lane (15 exchanges); the register
    // sort of 256 keys takes 36, of eight keys per lane each.
    __device__ __noinline__ void sort() {
        const int lane = threadIdx.x & 31;
        if (count <= 32) {
            const unsigned long long key = lanes_sort_desc(lane < count ? buf[lane] : 0ull);
            count = min(count, n_best);
            buf[lane] = lane < count ? key : 0ull;
            __syncwarp();
            cutoff = count >= n_best ? buf[n_best - 1] : 0ull;
            return;
        }
        warp_sort_desc(buf);
        count = min(count, n_best);
        for (int i = count + lane; i < kTopkCapacity; i += 32) buf[i] = 0ull;
        __syncwarp();
        cutoff = count >= n_best ? buf[n_best - 1] : 0ull;
    }
    // One key per lane (0: none).
    __device__ __forceinline__ void add(unsigned long long key) {
        if (__ballot_sync(0xffffffffu, key > cutoff) != 0) insert(key);
    }
    __device__ __noinline__ void insert(unsigned long long key) {
        const int lane = threadIdx.x & 31;
        if (count + 32 > kTopkCapacity) sort();
        const bool pass = key > cutoff;
        const unsigned mask = __ballot_sync(0xffffffffu, pass);
        if (pass) buf[count + __popc(mask & ((1u << lane) - 1))] = key;
        count += __popc(mask);
        __syncwarp();
    }
    // A lower bound of the n_best-th largest of n keys, before any of them is in the list: among the 32 lanes' largest (n_best
    // up to 32) or four largest keys there are n_best that reach it.  Most keys then never enter the list, which is
    // sorted once instead of every time that 256 keys have come together.
    template <class Key>
    __device__ __forceinline__ void raise_cutoff(int n, Key&& key_of) {
        const int lane = threadIdx.x & 31;
        const bool few = n_best <= 32;
        unsigned long long top[4] = {0ull, 0ull, 0ull, 0ull};
        constexpr int kAhead = 5;  // keys fetched before the first of them is looked at
        for (int i0 = lane; i0 < n; i0 += 32 * kAhead) {
            unsigned long long ahead[kAhead];
#pragma unroll
            for (int u = 0; u < kAhead; ++u) ahead[u] = i0 + 32 * u < n ? key_of(i0 + 32 * u) : 0ull;
#pragma unroll
            for (int u = 0; u < kAhead; ++u) {
                unsigned long long key = ahead[u];
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    if (r > 0 && few) break;
                    const unsigned long long less = key < top[r] ? key : top[r];
                    top[r] = key < top[r] ? top[r] : key;
                    key = less;
                }
            }
        }
        if (few) {
            top[0] = __shfl_sync(0xffffffffu, lanes_sort_desc(top[0]), n_best - 1);
        } else {
#pragma unroll
            for (int r = 0; r < 4; ++r) buf[r * 32 + lane] = top[r];
            for (int i = 128 + lane; i < kTopkCapacity; i += 32) buf[i] = 0ull;
            warp_sort_desc(buf);
            top[0] = buf[n_best - 1];
            __syncwarp();
            for (int i = lane; i < 128; i += 32) buf[i] = 0ull;
            __syncwarp();
        }
        if (top[0] > 0ull && top[0] - 1 > cutoff) cutoff = top[0] - 1;  // the bound itself passes
    }
    // The scores of columns [begin, end) of a query's row.
    __device__ __forceinline__ void scan(const float* __restrict__ row, int begin, int end, uint32_t first_row, uint32_t last_valid_row, const TopkParams& tp) {
        const int lane = threadIdx.x & 31;
        constexpr int kAhead = 8;  // scores fetched before the first of them is looked at: the loads overlap
        for (int base0 = begin; base0 < end; base0 += 32 * kAhead) {
            float ahead[kAhead];
#pragma unroll
            for (int u = 0; u < kAhead; ++u) {
                const int j = base0 + 32 * u + lane;
                ahead[u] = j < end ? row[j] : 0.f;
            }
#pragma unroll
            for (int u = 0; u < kAhead; ++u) {
                const int j = base0 + 32 * u + lane;
                unsigned long long key = 0ull;
                if (j < end && first_row + (uint32_t)j <= last_valid_row)
                    key = topk_key(tp.score_is_gamma_minus ? tp.gamma - ahead[u] : ahead[u], first_row + (uint32_t)j);
                add(key);
            }
        }
    }
};

// The first batch of a ranking, when no query has a cut-off: gridDim.y warps per query each scan a part of its row and
// leave their n_best keys (0 for missing ones) as candidates, which k_topk_update merges like any other.  One warp per
// query took 25 us for every 4096 scores, on as many SMs as there are groups of four queries.
// FEW: up to 32 keys per query.
template <bool FEW>
__global__ void __launch_bounds__(128, FEW ? 8 : 4)
k_topk_seed(const float* __restrict__ raw, int n_cols, uint32_t first_row, uint32_t last_valid_row, unsigned long long* __restrict__ cand,
            int* __restrict__ cand_count, TopkParams tp) {
    __shared__ __align__(16) unsigned long long buffers[4][kTopkCapacity];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, q = blockIdx.x * 4 + warp;
    if (q >= tp.n_query) return;
    unsigned long long* const buf = buffers[warp];
    const int part = ((n_cols + (int)gridDim.y - 1) / (int)gridDim.y + 31) / 32 * 32, begin = (int)blockIdx.y * part;
    const float* __restrict__ row = raw + (size_t)q * n_cols;
    const int end = min(n_cols, begin + part);
    auto score_at = [&](int j) { return tp.score_is_gamma_minus ? tp.gamma - row[j] : row[j]; };
    unsigned long long* __restrict__ out = cand + (size_t)q * kTopkCandidates + (size_t)blockIdx.y * tp.n_best;
    if (blockIdx.y == 0 && lane == 0) cand_count[q] = (int)gridDim.y * tp.n_best;
    if constexpr (FEW) {
        // Scores are held in registers, all of a tile read at the same time, and compared as floats: only what reaches the
        // cut-off's score becomes a key, and the few keys that do are sorted a key per lane.  128 queries x 40 000 scores: 24 us.
        // (58 with every score made a key twice, its reads waiting for a few at a time, and a 256-key sort at the end; 36 with
        // 20 scores held instead of ten, which do not fit 64 registers.)
        constexpr int kHold = 10;
        const int valid = (int)min((long long)end, (long long)last_valid_row - (long long)first_row + 1);
        int count = 0;
        unsigned long long cutoff = 0ull;
        for (int tile = begin; tile < end; tile += 32 * kHold) {
            float score[kHold];
#pragma unroll
            for (int u = 0; u < kHold; ++u) {
                const int j = tile + 32 * u + lane;
                score[u] = j < valid ? score_at(j) : 0.f;
            }
            if (tile == begin) {
                // the n_best-th of the lanes' largest keys: so many keys reach it
                float best = -INFINITY;
                int at = -1;
#pragma unroll
                for (int u = 0; u < kHold; ++u) {
                    const int j = tile + 32 * u + lane;
                    if (j < valid && (at < 0 || score[u] > best)) best = score[u], at = j;
                }
                const unsigned long long bound =
                    __shfl_sync(0xffffffffu, lanes_sort_desc(at >= 0 ? topk_key(best, first_row + (uint32_t)at) : 0ull), tp.n_best - 1);
                if (bound > 0ull) cutoff = bound - 1;
            }
#pragma unroll
            for (int u = 0; u < kHold; ++u) {
                const int j = tile + 32 * u + lane;
                bool pass = j < valid && (cutoff == 0ull || !(score[u] < topk_score(cutoff)));
                if (__ballot_sync(0xffffffffu, pass) == 0) continue;
                const unsigned long long key = topk_key(score[u], first_row + (uint32_t)j);
                pass = pass && key > cutoff;
                const unsigned mask = __ballot_sync(0xffffffffu, pass);
                if (pass) buf[count + __popc(mask & ((1u << lane) - 1))] = key;
                count += __popc(mask);
                __syncwarp();
                if (count + 32 > kTopkCapacity) {
                    topk_sort(buf, count);
                    count = tp.n_best;
                    cutoff = buf[tp.n_best - 1];
                }
            }
        }
        if (count <= 32) {
            const unsigned long long key = lanes_sort_desc(lane < count ? buf[lane] : 0ull);
            if (lane < tp.n_best) out[lane] = key;
        } else {
            topk_sort(buf, count);
            if (lane < tp.n_best) out[lane] = buf[lane];
        }
        return;
    } else {
        TopkList list{buf, 0, tp.n_best, 0ull};
        for (int i = lane; i < kTopkCapacity; i += 32) list.buf[i] = 0ull;
        __syncwarp();
        list.raise_cutoff(end - begin, [&](int i) {
            const uint32_t table_row = first_row + (uint32_t)(begin + i);
            return table_row <= last_valid_row ? topk_key(score_at(begin + i), table_row) : 0ull;
        });
        list.scan(row, begin, end, first_row, last_valid_row, tp);
        list.sort();
        for (int i = lane; i < tp.n_best; i += 32) out[i] = list.buf[i];
    }
}

// raw [n_query, n_cols] holds distances / dot products against rows first_row .. first_row+n_cols-1;
// rows above last_valid_row are padding of the shard and are skipped (src/poplar_kge.cpp:836-842).
// state [n_query, kTopkCapacity] keys, counts [n_query]: the first n_best (or fewer) sorted, what came later behind them.
// 4 warps per block, one query each.  cand / cand_count: the filter's or the seed's output for this batch; the counts are cleared for the next.
static __global__ void __launch_bounds__(128)
k_topk_update(const float* __restrict__ raw, int n_cols, uint32_t first_row, uint32_t last_valid_row,
              unsigned long long* __restrict__ state, int* __restrict__ counts, TopkParams tp,
              const unsigned long long* __restrict__ cand, int* __restrict__ cand_count) {
    __shared__ __align__(16) unsigned long long buffers[4][kTopkCapacity];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int q = blockIdx.x * 4 + warp;
    if (q >= tp.n_query) return;
    const int n_cand = cand_count[q];
    if (n_cand == 0) return;  // nothing in this batch beats the cut-off: the list stands
    unsigned long long* mine = state + (size_t)q * kTopkCapacity;
    const unsigned long long* __restrict__ keys = cand + (size_t)q * kTopkCandidates;
    const int old_count = counts[q];
    if (old_count >= tp.n_best && old_count + n_cand <= kTopkCapacity) {
        // room behind the sorted n_best: a later merge or k_topk_finish sorts; the cut-off stays the older, lower one
        for (int i = lane; i < n_cand; i += 32) mine[old_count + i] = keys[i];
        if (lane == 0) {
            cand_count[q] = 0;
            counts[q] = old_count + n_cand;
        }
        return;
    }
    TopkList list{buffers[warp], old_count, tp.n_best, 0ull};
    for (int i = lane; i < kTopkCapacity; i += 32) list.buf[i] = i < list.count ? mine[i] : 0ull;
    __syncwarp();
    const bool ranked = list.count >= tp.n_best;
    if (ranked) list.sort();
    if (lane == 0) cand_count[q] = 0;
    if (n_cand <= kTopkCandidates) {
        // (a bound first, where what passes it is likely to be sorted a key per lane)
        if (list.count == 0 && n_cand > (tp.n_best <= 16 ? 32 : kTopkCapacity)) list.raise_cutoff(n_cand, [&](int i) { return keys[i]; });
        constexpr int kAhead = 8;  // keys fetched before the first of them is looked at
        for (int base = 0; base < n_cand; base += 32 * kAhead) {
            unsigned long long ahead[kAhead];
#pragma unroll
            for (int u = 0; u < kAhead; ++u) ahead[u] = base + 32 * u + lane < n_cand ? keys[base + 32 * u + lane] : 0ull;
#pragma unroll
            for (int u = 0; u < kAhead; ++u) list.add(ahead[u]);
        }
    } else {  // more than the candidate list holds
        list.scan(raw + (size_t)q * n_cols, 0, n_cols, first_row, last_valid_row, tp);
    }
    if (!ranked) list.sort();
    for (int i = lane; i < list.count; i += 32) mine[i] = list.buf[i];
    if (lane == 0) counts[q] = list.count;
}

// Writes each query's sorted candidates to the shard that asked: query q = (asking shard, slot)
// goes to out_blocks[asking shard] + slot * n_best (the return all-to-all of
// src/poplar_kge.cpp:847-850).  Missing candidates get the reference's BadScore and row 0.
static __global__ void __launch_bounds__(128)
k_topk_finish(const unsigned long long* __restrict__ state, const int* __restrict__ counts, int n_query,
              int queries_per_shard, int n_best, float* const* __restrict__ score_blocks,
              uint32_t* const* __restrict__ index_blocks) {
    __shared__ __align__(16) unsigned long long keys[kTopkCapacity];
    const int q = blockIdx.x;
    if (q >= n_query) return;
    const int shard = q / queries_per_shard, slot = q - shard * queries_per_shard;
    float* __restrict__ so = score_blocks[shard] + (size_t)slot * n_best;
    uint32_t* __restrict__ io = index_blocks[shard] + (size_t)slot * n_best;
    const int count = counts[q];
    for (int i = threadIdx.x; i < kTopkCapacity; i += blockDim.x) keys[i] = i < count ? state[(size_t)q * kTopkCapacity + i] : 0ull;
    __syncthreads();
    if (count > n_best && threadIdx.x < 32) warp_sort_desc(keys);
    __syncthreads();
    for (int i = threadIdx.x; i < n_best; i += blockDim.x) {
        so[i] = i < count ? topk_score(keys[i]) : -1e6f;
        io[i] = i < count ? topk_index(keys[i]) : 0u;
    }
}

// ---------------------------------------------------------------------------
// The BESS batch sampler on the device (src/python/poplar_kge_dataset.py:310-393, `sample_batch`,
// with its uniform strategy; `unique_pad` :161-164).  The training triples lie in device memory
// sorted by (head shard, tail shard) bucket, as local rows: triples[0] head rows, [1] relations,
// [2] tail rows (:199-241).  One block draws everything shard s needs for step i:
//   positions [0, B)       its own positives, B / n per tail shard: head rows (and the relations);
//   positions [B, 2B)      the positives of every head shard whose tail lives on s: tail rows;
//   positions [2B, 2B + n * neg)  the negatives every head shard asks s for: uniform rows of s;
// then sorts them, keeps each row once (`remote`, zero-padded) and gives every position the slot
// of its row (`head`, `a2a`).  Draws are counter-based (Philox keyed by seed and run, counted by
// head shard, step, tail shard and slot), so the block of shard s and the block of the head
// shard that owns a positive compute the same triple without talking to each other, on any GPU.
struct SamplerData {
    const uint32_t* triples;        // [3][n_triples]
    size_t n_triples;
    const uint32_t* bucket_offset;  // [n_shard][n_shard]
    const uint32_t* bucket_count;   // [n_shard][n_shard], none empty
    const uint32_t* shard_count;    // [n_shard] real rows per shard (rows 1 .. count)
};

__device__ __forceinline__ void philox_round(uint32_t (&c)[4], uint32_t k0, uint32_t k1);

__device__ __forceinline__ unsigned long long sampler_draw(uint32_t seed, uint32_t run, uint32_t head_shard, uint32_t step,
                                                           uint32_t tail_shard, uint32_t slot) {
    uint32_t c[4] = {head_shard, step, tail_shard, slot};
    uint32_t k0 = seed, k1 = run ^ 0x243F6A88u;
#pragma unroll
    for (int i = 0; i < 10; ++i) {
        philox_round(c, k0, k1);
        k0 += 0x9E3779B9u;
        k1 += 0xBB67AE85u;
    }
    return ((unsigned long long)c[0] << 32) | c[1];
}

constexpr uint32_t kNegativeSlot = 0x80000000u;  // slot numbers of negatives, apart from those of positives

static __global__ void __launch_bounds__(kSortThreads)
k_sample_batch(SamplerData sd, uint32_t seed, uint32_t run, int n_shard, int shard0, int n_step, int B, int a2a,
               uint32_t* __restrict__ remote, uint32_t* __restrict__ a2a_out, uint32_t* __restrict__ head,
               uint32_t* __restrict__ relation, uint32_t* __restrict__ tail, uint32_t highest_row) {
    __shared__ BlockSort bs;
    __shared__ uint32_t s_scan[kSortThreads];
    const int l = blockIdx.x / n_step, step = blockIdx.x % n_step, s = shard0 + l;
    const int pos = B / n_shard, neg = a2a - pos, T = n_shard * a2a, R = B + T;
    const size_t sidx = (size_t)l * n_step + step;
    remote += sidx * R;
    a2a_out += sidx * T;
    head += sidx * B;
    relation += sidx * B;
    tail += sidx * B;
    for (int p = threadIdx.x; p < R; p += blockDim.x) {
        uint32_t row;
        if (p < B) {
            const int ts = p / pos, k = p - ts * pos;
            const uint32_t bucket = (uint32_t)(s * n_shard + ts);
            const size_t idx = sd.bucket_offset[bucket] + sampler_draw(seed, run, (uint32_t)s, (uint32_t)step, (uint32_t)ts, (uint32_t)k) % sd.bucket_count[bucket];
            row = sd.triples[idx];
            relation[p] = sd.triples[sd.n_triples + idx];
            tail[p] = (uint32_t)(ts * a2a + k);  // where the exchange puts this positive's tail (:257-263)
        } else if (p < 2 * B) {
            const int q = p - B, hs = q / pos, k = q - hs * pos;
            const uint32_t bucket = (uint32_t)(hs * n_shard + s);
            const size_t idx = sd.bucket_offset[bucket] + sampler_draw(seed, run, (uint32_t)hs, (uint32_t)step, (uint32_t)s, (uint32_t)k) % sd.bucket_count[bucket];
            row = sd.triples[2 * sd.n_triples + idx];
        } else {
            const int q = p - 2 * B, hs = q / neg, k = q - hs * neg;
            row = 1u + (uint32_t)(sampler_draw(seed, run, (uint32_t)hs, (uint32_t)step, (uint32_t)s, kNegativeSlot | (uint32_t)k) % sd.shard_count[s]);
        }
        bs.key[p] = row;
    }
    __syncthreads();
    const uint16_t* const sorted = bs.sort(R, 32 - __clz(highest_row));
    // rank of every sorted entry among the distinct rows: an exclusive scan of "starts a new row"
    const int per_thread = (R + (int)blockDim.x - 1) / (int)blockDim.x, first = threadIdx.x * per_thread;
    uint32_t mine = 0;
    for (int i = first; i < first + per_thread && i < R; ++i) mine += i == 0 || bs.key[sorted[i]] != bs.key[sorted[i - 1]] ? 1u : 0u;
    s_scan[threadIdx.x] = mine;
    __syncthreads();
    for (int o = 1; o < (int)blockDim.x; o <<= 1) {  // Hillis-Steele inclusive scan over the threads' counts
        const uint32_t v = (int)threadIdx.x >= o ? s_scan[threadIdx.x - o] : 0u;
        __syncthreads();
        s_scan[threadIdx.x] += v;
        __syncthreads();
    }
    uint32_t rank = s_scan[threadIdx.x] - mine;  // distinct rows before this thread's first entry
    const uint32_t n_unique = s_scan[blockDim.x - 1];
    for (int i = first; i < first + per_thread && i < R; ++i) {
        const uint32_t p = sorted[i];
        const bool starts = i == 0 || bs.key[p] != bs.key[sorted[i - 1]];
        if (starts) remote[rank++] = bs.key[p];
        const uint32_t slot = rank - 1;
        if (p < (uint32_t)B) {
            head[p] = slot;
        } else if (p < (uint32_t)(2 * B)) {
            const uint32_t q = p - (uint32_t)B, hs = q / (uint32_t)pos;
            a2a_out[hs * a2a + (q - hs * pos)] = slot;
        } else {
            const uint32_t q = p - (uint32_t)(2 * B), hs = q / (uint32_t)neg;
            a2a_out[hs * a2a + pos + (q - hs * neg)] = slot;
        }
    }
    for (int i = (int)n_unique + (int)threadIdx.x; i < R; i += blockDim.x) remote[i] = 0u;  // unique_pad's zeros
}

// ---------------------------------------------------------------------------
// Table I/O (src/poplar_kge.cpp:857-871).

// Counter-based normal numbers (Philox-4x32-10 + Box-Muller), keyed by (seed, shard) and
// counted by (row, column / 4): the initial embedding of a row depends only on its
// address, not on which call wrote it.
__device__ __forceinline__ void philox_round(uint32_t (&c)[4], uint32_t k0, uint32_t k1) {
    const uint32_t hi0 = __umulhi(0xD2511F53u, c[0]), lo0 = 0xD2511F53u * c[0];
    const uint32_t hi1 = __umulhi(0xCD9E8D57u, c[2]), lo1 = 0xCD9E8D57u * c[2];
    const uint32_t n0 = hi1 ^ c[1] ^ k0, n2 = hi0 ^ c[3] ^ k1;
    c[0] = n0; c[1] = lo1; c[2] = n2; c[3] = lo0;
}
__device__ __forceinline__ float4 philox_normal4(uint32_t seed, uint32_t stream, uint32_t row,
                                                 uint32_t col4) {
    uint32_t c[4] = {row, col4, stream, 0x6b676562u};
    uint32_t k0 = seed, k1 = 0x9E3779B9u ^ stream;
#pragma unroll
    for (int i = 0; i < 10; ++i) {
        philox_round(c, k0, k1);
        k0 += 0x9E3779B9u;
        k1 += 0xBB67AE85u;
    }
    const float u0 = ((float)(c[0] >> 8) + 0.5f) * (1.0f / 16777216.0f);
    const float u1 = ((float)(c[1] >> 8) + 0.5f) * (1.0f / 16777216.0f);
    const float u2 = ((float)(c[2] >> 8) + 0.5f) * (1.0f / 16777216.0f);
    const float u3 = ((float)(c[3] >> 8) + 0.5f) * (1.0f / 16777216.0f);
    const float r0 = sqrtf(-2.f * logf(u0)), r1 = sqrtf(-2.f * logf(u2));
    float s0, c0, s1, c1;
    sincospif(2.f * u1, &s0, &c0);
    sincospif(2.f * u3, &s1, &c1);
    return make_float4(r0 * c0, r0 * s0, r1 * c1, r1 * s1);
}

// Which table row slot j of a piece of a transfer stands for: the slots at, at + 1, ... of n_local x per_shard, with
// their rows in idx[j] or (null) counted up from `first` in every shard.
struct RowSource {
    uint8_t* tables;  // the local shards' tables, `stride` bytes apart
    size_t stride;
    const uint32_t* idx;
    uint32_t first;
    size_t at, per_shard;
};
struct RowSlot {
    uint32_t row, shard, slot;  // slot: within the shard
};
__device__ __forceinline__ RowSlot row_slot(const RowSource& s, unsigned j) {
    const size_t g = s.at + j, l = g / s.per_shard;
    RowSlot r;
    r.shard = (uint32_t)l;
    r.slot = (uint32_t)(g - l * s.per_shard);
    r.row = s.idx ? s.idx[j] : s.first + r.slot;
    return r;
}

// A slot writes only if no later slot of its shard names the same row, so duplicate indices (the
// overflow slots that the host redirects to row 0, src/python/poplar_kge.py:546-552)
// resolve to the last one in order, deterministically.  All threads of the block look.
__device__ __forceinline__ bool is_last_writer(const RowSource& s, unsigned j, const RowSlot& r) {
    if (!s.idx) return true;
    const uint32_t left = (uint32_t)s.per_shard - r.slot;
    bool later = false;
    for (uint32_t k = 1 + threadIdx.x; k < left; k += blockDim.x) later |= s.idx[j + k] == r.row;
    return !__syncthreads_or(later);
}

// write_entity: fresh embedding ~ N(0, std), zero moments, features from the host array's piece (in pinned memory up to 64 KB,
// else in device memory).
template <class ST, class FT, class IT>
__global__ void __launch_bounds__(128)
k_write_entity(RowSource rows, RowLayout L, const IT* __restrict__ features, uint32_t seed, uint32_t shard0, float stddev) {
    const int j = blockIdx.x;
    const RowSlot s = row_slot(rows, j);
    if (!is_last_writer(rows, j, s)) return;
    uint8_t* base = rows.tables + s.shard * rows.stride + (size_t)s.row * L.row_bytes;
    ST* mv = reinterpret_cast<ST*>(base + L.off_m);
    ST* qv = reinterpret_cast<ST*>(base + L.off_q);
    FT* fv = reinterpret_cast<FT*>(base + L.off_feat);
    const int D = L.d, F = L.f;
    const IT* __restrict__ src = features + (size_t)j * F;
    const bool vec = (F & 3) == 0;
    if (vec)
        for (int c = threadIdx.x * 4; c < F; c += blockDim.x * 4) store4(fv + c, load4(src + c));
    else
        for (int c = threadIdx.x; c < F; c += blockDim.x) store_from_float(fv + c, load_as_float(src + c));
    for (int c4 = threadIdx.x; c4 * 4 < D; c4 += blockDim.x) {
        const float4 z = philox_normal4(seed, shard0 + s.shard, s.row, (uint32_t)c4);
        const float zz[4] = {z.x, z.y, z.z, z.w};
        for (int u = 0; u < 4 && c4 * 4 + u < D; ++u) {
            store_value<ST>(L, base, c4 * 4 + u, stddev * zz[u]);
            store_from_float(mv + c4 * 4 + u, 0.f);
            store_from_float(qv + c4 * 4 + u, 0.f);
        }
    }
}

// initialise_entities: every row of the shard on the device, no host data.  Embeddings as
// write_entity would draw them; features ~ N(0, 1) from a second stream (row 0, the padding
// row, keeps zero features); optimiser state zero.  Stands in for streaming a dataset's
// features through write_entity when the table is tens of gigabytes of synthetic data.
template <class ST, class FT>
__global__ void __launch_bounds__(256)
k_init_table(uint8_t* __restrict__ table, RowLayout L, size_t n_rows, uint32_t seed, uint32_t shard,
             float stddev) {
    const int D = L.d, F = L.f;
    const int d4 = (D + 3) / 4, f4 = (F + 3) / 4, per_row = d4 + f4;
    const size_t total = n_rows * (size_t)per_row;
    for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < total;
         e += (size_t)gridDim.x * blockDim.x) {
        const size_t row = e / per_row;
        const int q = (int)(e - row * per_row);
        uint8_t* base = table + row * L.row_bytes;
        if (q < d4) {
            const float4 z = philox_normal4(seed, shard, (uint32_t)row, (uint32_t)q);
            const float zz[4] = {z.x, z.y, z.z, z.w};
            for (int u = 0; u < 4 && q * 4 + u < D; ++u) {
                store_value<ST>(L, base, q * 4 + u, stddev * zz[u]);
                store_from_float(reinterpret_cast<ST*>(base + L.off_m) + q * 4 + u, 0.f);
                store_from_float(reinterpret_cast<ST*>(base + L.off_q) + q * 4 + u, 0.f);
            }
        } else {
            const int c4 = q - d4;
            const float4 z = philox_normal4(seed ^ 0x5bd1e995u, shard, (uint32_t)row, (uint32_t)c4);
            const float zz[4] = {z.x, z.y, z.z, z.w};
            for (int u = 0; u < 4 && c4 * 4 + u < F; ++u)
                store_from_float(reinterpret_cast<FT*>(base + L.off_feat) + c4 * 4 + u, row == 0 ? 0.f : zz[u]);
        }
    }
}

// write_entity_rows: whole rows [value | m | sqrt(v) | feature] from the host array's piece (as write_entity's).
template <class ST, class FT, class IT>
__global__ void __launch_bounds__(128)
k_write_rows(RowSource rows, RowLayout L, const IT* __restrict__ data) {
    const int j = blockIdx.x;
    const RowSlot s = row_slot(rows, j);
    if (!is_last_writer(rows, j, s)) return;
    const int D = L.d, F = L.f, W = 3 * D + F;
    const IT* __restrict__ src = data + (size_t)j * W;
    uint8_t* base = rows.tables + s.shard * rows.stride + (size_t)s.row * L.row_bytes;
    for (int c = threadIdx.x; c < W; c += blockDim.x) {
        const float v = load_as_float(src + c);
        if (c < D) store_value<ST>(L, base, c, v);
        else if (c < 2 * D) store_from_float(reinterpret_cast<ST*>(base + L.off_m) + (c - D), v);
        else if (c < 3 * D) store_from_float(reinterpret_cast<ST*>(base + L.off_q) + (c - 2 * D), v);
        else store_from_float(reinterpret_cast<FT*>(base + L.off_feat) + (c - 3 * D), v);
    }
}

// read_entity: whole rows out, in the host array's element type, into a piece in pinned memory (up to 64 KB) or device memory:
// four elements per store where the segments allow it, so that a warp's stores make whole 128-byte writes, on the link too.
template <class ST, class FT, class OT>
__global__ void __launch_bounds__(128)
k_read_rows(RowSource rows, RowLayout L, OT* __restrict__ out) {
    const int j = blockIdx.x;
    const RowSlot s = row_slot(rows, j);
    const int D = L.d, F = L.f, W = 3 * D + F;
    const uint8_t* base = rows.tables + s.shard * rows.stride + (size_t)s.row * L.row_bytes;
    OT* __restrict__ dst = out + (size_t)j * W;
    if (((D | F) & 3) == 0) {
        for (int c = threadIdx.x * 4; c < W; c += blockDim.x * 4) {
            float4 v;
            if (c < D) v = L.value_bf16 ? load4(reinterpret_cast<const __nv_bfloat16*>(base) + c) : load4(reinterpret_cast<const ST*>(base) + c);
            else if (c < 2 * D) v = load4(reinterpret_cast<const ST*>(base + L.off_m) + (c - D));
            else if (c < 3 * D) v = load4(reinterpret_cast<const ST*>(base + L.off_q) + (c - 2 * D));
            else v = load4(reinterpret_cast<const FT*>(base + L.off_feat) + (c - 3 * D));
            store4(dst + c, v);
        }
        return;
    }
    for (int c = threadIdx.x; c < W; c += blockDim.x) {
        float v;
        if (c < D) v = load_value<ST>(L, base, c);
        else if (c < 2 * D) v = load_as_float(reinterpret_cast<const ST*>(base + L.off_m) + (c - D));
        else if (c < 3 * D) v = load_as_float(reinterpret_cast<const ST*>(base + L.off_q) + (c - 2 * D));
        else v = load_as_float(reinterpret_cast<const FT*>(base + L.off_feat) + (c - 3 * D));
        store_from_float(dst + c, v);
    }
}

// Plain fp32 row gather with 128-bit accesses (the operator form of fr::Buffer::read,
// src/fructose/fructose.cpp:790-798), used by the operator entry point and the microbench.
template <int V>
__global__ void __launch_bounds__(128)
k_gather_rows(const float* __restrict__ table, size_t width, const uint32_t* __restrict__ idx,
              float* __restrict__ out) {
    const size_t j = blockIdx.x;
    const float* __restrict__ src = table + (size_t)idx[j] * width;
    float* __restrict__ dst = out + j * width;
    if (V == 4) {
        for (size_t c = threadIdx.x * 4; c < width; c += blockDim.x * 4) store4(dst + c, load4(src + c));
    } else {
        for (size_t c = threadIdx.x; c < width; c += blockDim.x) dst[c] = src[c];
    }
}

// y[e] = x[e] rounded to bfloat16 (operands of the bf16 contractions that the host provides).
static __global__ void __launch_bounds__(256) k_to_bf16(const float* __restrict__ x, size_t n, __nv_bfloat16* __restrict__ y) {
    for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < n; e += (size_t)gridDim.x * blockDim.x) y[e] = __float2bfloat16_rn(x[e]);
}

// The feature planes of `count` consecutive table rows from `first_row` on (a pass of predict over
// the table), as k_gather_step_rows makes them for the gathered rows of a training step: fp16
// features widened to fp32 into planes.wide, or the lower TF32 plane of fp32 features into planes.lo.
static __global__ void __launch_bounds__(256)
k_table_feature_planes(const uint8_t* __restrict__ table, RowLayout L, uint32_t first_row, int count, FeaturePlanes planes) {
    const int per_row = (int)((L.row_bytes - L.off_feat) >> 4);  // 16-byte chunks of a row's feature segment
    for (size_t u = (size_t)blockIdx.x * blockDim.x + threadIdx.x; u < (size_t)count * per_row; u += (size_t)gridDim.x * blockDim.x) {
        const int r = (int)(u / per_row), c = (int)(u - (size_t)r * per_row);
        const uint4 v = *reinterpret_cast<const uint4*>(table + ((size_t)first_row + r) * L.row_bytes + L.off_feat + (size_t)c * 16);
        if (planes.wide) {
            const int f = c * 8;
            const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&v.x)), b = __half22float2(*reinterpret_cast<const __half2*>(&v.y));
            const float2 cc = __half22float2(*reinterpret_cast<const __half2*>(&v.z)), d = __half22float2(*reinterpret_cast<const __half2*>(&v.w));
            float* o = planes.wide + (size_t)r * planes.stride + f;
            if (f < (int)planes.stride) *reinterpret_cast<float4*>(o) = make_float4(a.x, a.y, b.x, b.y);
            if (f + 4 < (int)planes.stride) *reinterpret_cast<float4*>(o + 4) = make_float4(cc.x, cc.y, d.x, d.y);
        } else if (planes.lo) {
            const int f = c * 4;
            if (f < (int)planes.stride)
                *reinterpret_cast<float4*>(planes.lo + (size_t)r * planes.stride + f) =
                    tf32_lower4(make_float4(__uint_as_float(v.x), __uint_as_float(v.y), __uint_as_float(v.z), __uint_as_float(v.w)));
        }
    }
}

// lo[e] = the lower TF32 plane of x[e] (for parameters that the host writes).
static __global__ void __launch_bounds__(256) k_lower_plane(const float* __restrict__ x, size_t n, float* __restrict__ lo) {
    for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < n; e += (size_t)gridDim.x * blockDim.x) lo[e] = tf32_lower(x[e]);
}

// Operator form of the duplicate-combining scatter-add: one block per table row, summing
// the rows of its segment in position order.
static __global__ void __launch_bounds__(128)
k_segment_sum_rows(const float* __restrict__ rows, const uint32_t* __restrict__ perm,
                   const uint32_t* __restrict__ off, size_t width, float* __restrict__ out) {
    const size_t r = blockIdx.x;
    for (size_t c = threadIdx.x; c < width; c += blockDim.x) {
        float g = 0.f;
        for (uint32_t q = off[r]; q < off[r + 1]; ++q) g += rows[(size_t)perm[q] * width + c];
        out[r * width + c] = g;
    }
}

// Operator forms of the two activations with their backward (src/pag/pag.cpp:841-864, 888-910).
static __global__ void __launch_bounds__(256)
k_log_sigmoid(const float* __restrict__ x, const float* __restrict__ grad_out, size_t n,
              float* __restrict__ y, float* __restrict__ grad_x) {
    for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < n;
         e += (size_t)gridDim.x * blockDim.x) {
        const float v = x[e];
        y[e] = v > -11.f ? -log1pf(expf(-fmaxf(v, -11.f))) : v;
        grad_x[e] = grad_out[e] / (1.f + expf(fminf(v, 11.f)));
    }
}
static __global__ void __launch_bounds__(256)
k_log_softmax(const float* __restrict__ x, const float* __restrict__ grad_out, int cols,
              float* __restrict__ y, float* __restrict__ grad_x) {
    __shared__ float scratch[8];
    const size_t base = (size_t)blockIdx.x * cols;
    float mx = -INFINITY;
    for (int j = threadIdx.x; j < cols; j += 256) mx = fmaxf(mx, x[base + j]);
    mx = block_max<256>(mx, scratch);
    float sum = 0.f, gsum = 0.f;
    for (int j = threadIdx.x; j < cols; j += 256) {
        sum += expf(x[base + j] - mx);
        gsum += grad_out[base + j];
    }
    sum = block_sum<256>(sum, scratch);
    gsum = block_sum<256>(gsum, scratch);
    const float log_z = logf(sum);
    for (int j = threadIdx.x; j < cols; j += 256) {
        const float logp = x[base + j] - mx - log_z;
        y[base + j] = logp;
        grad_x[base + j] = grad_out[base + j] - gsum * expf(logp);
    }
}

}  // namespace kge
