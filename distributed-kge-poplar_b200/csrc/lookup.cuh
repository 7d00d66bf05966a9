// The lookups of a step: rows named by `head` and `a2a` become the predicted tails and the tail rows that the shards
// exchange (src/poplar_kge.cpp:489-567, 676-684), and the predicted tails' gradients become those of the head rows and of
// the relation rows (the backward of the same lines).
#pragma once

#include <type_traits>

#include "kernels.cuh"

namespace kge {

// Where the rows that lookups name lie: hidden rows in fp32, or, in a model without features, whose hidden rows are the
// stored values, the table itself.
struct LookupRows {
    const uint8_t *head, *tail;           // bases of the rows that head and tail lookups read
    const uint32_t *head_row, *tail_row;  // [B], [T] rows by lookup
    size_t stride;                        // bytes
};

struct LookupArgs {
    LookupRows rows;
    const uint32_t* relation;      // [B]
    float* const* send_dst;        // [n_shard] this shard's slot in every shard's tail buffer
    float* const* send_lo_dst;     // the same in the companion plane; null: none
    float *pred, *pred_lo, *nrm;   // [B, D] predicted tails, their companion plane (or null), TransH's unit normals
    const uint32_t* remote;        // not null: every gathered row also goes to `hid` as fp32, [R, D]
    float* hid;
};
struct LookupSizes {
    const float *rel_table, *normal_table;
    int B, T, a2a, D, R;
    int lo_bf16;    // the companion planes hold the bfloat16 rounding instead of the lower TF32 part
    int prefetch;   // the index streams were complete before the kernel in front of this one began
    ExchangeSync sync;
};

// Four columns at c of a row and of its companion plane.
__device__ __forceinline__ void store_with_plane(float* out, float* lo, int lo_bf16, size_t row, int D, int c, float4 v) {
    store4(out + row * D + c, v);
    if (!lo) return;
    if (lo_bf16) store4(reinterpret_cast<__nv_bfloat16*>(lo) + row * D + c, v);
    else store4(lo + row * D + c, tf32_lower4(v));
}
__device__ __forceinline__ void store_with_plane(float* out, float* lo, int lo_bf16, size_t row, int D, int c, float v) {
    out[row * D + c] = v;
    if (!lo) return;
    if (lo_bf16) reinterpret_cast<__nv_bfloat16*>(lo)[row * D + c] = __float2bfloat16_rn(v);
    else lo[row * D + c] = tf32_lower(v);
}

// A warp per row of D columns and the same columns of N float rows beside it: f(c, value, beside) with float4s where rows allow
// 16-byte accesses, four pieces of every row in flight a lane.
template <int N, class VT, class F>
__device__ __forceinline__ void for_row(const VT* __restrict__ src, const float* const (&rows)[N], int D, F f) {
    const int lane = threadIdx.x & 31;
    auto pieces = [&](auto zero, int stride, auto load_value, auto load_beside) {
        using T = decltype(zero);
        const int step = stride * 32;
        for (int c0 = lane * stride; c0 < D; c0 += 4 * step) {
            T v[4], beside[4][N];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                if (c0 + u * step >= D) continue;
                v[u] = load_value(src + c0 + u * step);
#pragma unroll
                for (int i = 0; i < N; ++i)
                    if (rows[i]) beside[u][i] = load_beside(rows[i] + c0 + u * step);
            }
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (c0 + u * step < D) f(c0 + u * step, v[u], beside[u]);
        }
    };
    if ((D & 3) == 0) pieces(float4{}, 4, [](const VT* p) { return load4(p); }, [](const float* p) { return load4(p); });
    else pieces(0.f, 1, [](const VT* p) { return load_as_float(p); }, [](const float* p) { return *p; });
}
template <class VT, class F>
__device__ __forceinline__ void for_row(const VT* __restrict__ src, int D, F f) {
    const float* const none[1] = {nullptr};
    for_row<1>(src, none, D, [&](int c, auto v, const auto&) { f(c, v); });
}

// Sums over a row's columns for a whole warp: add(c, sums) for the columns lane, lane + 64, ... into one set of sums and for
// lane + 32, lane + 96, ... into another, each then added up over the lanes.  (The order is part of TransH's result, whose
// L1 gradients turn on the last bit of a score: see k_pair_bwd.)
template <int N, class F>
__device__ __forceinline__ void two_strands(int D, float (&sums)[2][N], F add) {
    const int lane = threadIdx.x & 31;
#pragma unroll 2
    for (int c = lane; c < D; c += 64) {
        add(c, sums[0]);
        if (c + 32 < D) add(c + 32, sums[1]);
    }
#pragma unroll
    for (int i = 0; i < N; ++i) {
        sums[0][i] = warp_sum(sums[0][i]);
        sums[1][i] = warp_sum(sums[1][i]);
    }
}

// Warps per head lookup: a RotatE row of 256 is 128 sines and cosines in double precision, four in a row for each lane of one
// warp (event pairs for 256 heads: 10.7 us, 8.5 with four warps).
template <int FN>
constexpr int kHeadWarps = FN == SCORE_ROTATE ? 4 : 1;

// One warp per lookup: a tail lookup's row goes straight into the receive buffer of the destination shard (a peer's
// memory when that shard lives in another process), a head lookup's becomes its predicted tail.  Bound by latency: an
// index, then the row, which without features comes from the table in DRAM; the lines of those rows are asked into L2
// before the kernel in front has ended (`prefetch`: rows that it still updates are read after it).  As three kernels (rows
// copied whole into a compact buffer, widened into hidden rows, routed by blocks of 64 threads) a step took 78.9 us for
// 1024 triples x 2048 tails of 512 bf16 values and 90 us for ComplEx at 768 x 1536 x 400; this way 64.1 and 75.
template <class VT, int FN>
__global__ void __launch_bounds__(256) k_lookup(const __grid_constant__ ShardArgs<LookupArgs> shards, const __grid_constant__ LookupSizes g) {
    const LookupArgs& a = shards.s[blockIdx.y];
    const int warp = (int)blockIdx.x * 8 + (int)(threadIdx.x >> 5), lane = threadIdx.x & 31, D = g.D;
    const int n_head = g.B * kHeadWarps<FN>, part = warp < n_head ? warp % kHeadWarps<FN> : 0;
    const int unit = warp < n_head ? warp / kHeadWarps<FN> : warp - n_head + g.B;  // lookup, or behind them gathered row
    const bool is_head = unit < g.B, is_tail = !is_head && unit < g.B + g.T;
    if (g.prefetch && (is_head || is_tail)) {
        const uint8_t* row = is_head ? a.rows.head + (size_t)a.rows.head_row[unit] * a.rows.stride
                                     : a.rows.tail + (size_t)a.rows.tail_row[unit - g.B] * a.rows.stride;
        const int bytes = D * (int)sizeof(VT);
        for (int o = lane * 128; o < bytes + 128; o += 32 * 128)
            asm volatile("prefetch.global.L2 [%0];" ::"l"(row + min(o, bytes - 1)));
    }
    grid_dependency_sync();
    if (is_tail) {
        const int b = unit - g.B, dst = b / g.a2a, j = b - dst * g.a2a;
        float* out = a.send_dst[dst];
        float* lo = a.send_lo_dst ? a.send_lo_dst[dst] : nullptr;
        for_row(reinterpret_cast<const VT*>(a.rows.tail + (size_t)a.rows.tail_row[b] * a.rows.stride), D,
                [&](int c, auto v) { store_with_plane(out, lo, g.lo_bf16, (size_t)j, D, c, v); });
    } else if (is_head) {
        const int i = unit;
        const VT* __restrict__ h = reinterpret_cast<const VT*>(a.rows.head + (size_t)a.rows.head_row[i] * a.rows.stride);
        const float* __restrict__ r = g.rel_table + (size_t)a.relation[i] * D;
        if (FN == SCORE_COMPLEX || FN == SCORE_ROTATE) {
            const int half = D / 2;
#pragma unroll 4
            for (int c = part * 32 + lane; c < half; c += 32 * kHeadWarps<FN>) {
                const float hr = load_as_float(h + c), hi = load_as_float(h + c + half);
                float rr, ri;  // the relation as a complex number: stored (ComplEx) or the unit rotation by the stored angle (RotatE)
                if (FN == SCORE_ROTATE) rotate_sin_cos(r[c], ri, rr);
                else { rr = r[c]; ri = r[c + half]; }
                store_with_plane(a.pred, a.pred_lo, g.lo_bf16, (size_t)i, D, c, hr * rr - hi * ri);
                store_with_plane(a.pred, a.pred_lo, g.lo_bf16, (size_t)i, D, c + half, hr * ri + hi * rr);
            }
        } else if (FN == SCORE_TRANSH) {
            // n_i = w_i / |w_i|,  pt_i = h_i - n_i (n_i . h_i) + r_i
            const float* __restrict__ w = g.normal_table + (size_t)a.relation[i] * D;
            float sums[2][2] = {};
            two_strands(D, sums, [&](int c, float (&sum)[2]) {
                sum[0] += w[c] * w[c];
                sum[1] += w[c] * load_as_float(h + c);
            });
            const float ww = sums[0][0] + sums[1][0], wh = sums[0][1] + sums[1][1];
            const float inv = 1.f / sqrtf(ww), nh = wh * inv;  // n . h
#pragma unroll 4
            for (int c = lane; c < D; c += 32) {
                const float n = w[c] * inv;
                a.nrm[(size_t)i * D + c] = n;
                a.pred[(size_t)i * D + c] = load_as_float(h + c) - n * nh + r[c];
            }
        } else {
            const float* const beside[1] = {r};
            for_row<1>(h, beside, D, [&](int c, auto v, const auto& q) {
                auto with = [&](float x, float y) { return FN == SCORE_TRANSE ? x + y : x * y; };
                if constexpr (sizeof(v) == sizeof(float4))
                    store_with_plane(a.pred, a.pred_lo, g.lo_bf16, (size_t)i, D, c, make_float4(with(v.x, q[0].x), with(v.y, q[0].y), with(v.z, q[0].z), with(v.w, q[0].w)));
                else
                    store_with_plane(a.pred, a.pred_lo, g.lo_bf16, (size_t)i, D, c, with(v, q[0]));
            });
        }
    } else if (a.remote && unit - g.B - g.T < g.R) {
        const int r = unit - g.B - g.T;
        for_row(reinterpret_cast<const VT*>(a.rows.head + (size_t)a.remote[r] * a.rows.stride), D,
                [&](int c, auto v) { store_with_plane(a.hid, nullptr, 0, (size_t)r, D, c, v); });
    }
    exchange_signal(g.sync, XCHG_TAILS, gridDim.x * gridDim.y);  // the tail rows are in their consumers' memory
}

// `value_type` of the rows: 0 fp32, 1 fp16, 2 bf16.
inline cudaError_t launch_lookup(const ShardArgs<LookupArgs>& shards, int n_shards, const LookupSizes& g, int score_fn, int value_type, cudaStream_t stream,
                                 bool spread = true) {
    auto with_type = [&](auto fn) {
        constexpr int FN = decltype(fn)::value;
        const int warps = g.B * kHeadWarps<FN> + g.T + (shards.s[0].remote ? g.R : 0);
        const dim3 grid((unsigned)((warps + 7) / 8), (unsigned)n_shards);
        if (value_type == 2) return launch_spread_if<k_lookup<__nv_bfloat16, FN>>(spread, grid, dim3(256), stream, shards, g);
        if (value_type == 1) return launch_spread_if<k_lookup<__half, FN>>(spread, grid, dim3(256), stream, shards, g);
        return launch_spread_if<k_lookup<float, FN>>(spread, grid, dim3(256), stream, shards, g);
    };
    switch (score_fn) {
        case SCORE_DISTMULT: return with_type(std::integral_constant<int, SCORE_DISTMULT>{});
        case SCORE_COMPLEX: return with_type(std::integral_constant<int, SCORE_COMPLEX>{});
        case SCORE_ROTATE: return with_type(std::integral_constant<int, SCORE_ROTATE>{});
        case SCORE_TRANSH: return with_type(std::integral_constant<int, SCORE_TRANSH>{});
        default: return with_type(std::integral_constant<int, SCORE_TRANSE>{});
    }
}

// Gradients of the head vector and of the relation row (backward of src/poplar_kge.cpp:501-530, 539-569).  TransE needs no
// kernel: both equal d_pred.
struct LookupBwdArgs {
    LookupRows rows;
    const uint32_t* relation;
    const float* d_pred;
    float *d_head, *d_relrow;
    const float *nrm, *d_nrm;  // TransH: unit normals and their gradients from the scores
    float* d_normrow;          // TransH: per-triple gradients of the raw normals
};

template <class VT, int FN>
__global__ void __launch_bounds__(256)
k_lookup_bwd(const __grid_constant__ ShardArgs<LookupBwdArgs> shards, const float* __restrict__ rel_table, const float* __restrict__ normal_table, int B, int D) {
    grid_dependency_sync();
    const LookupBwdArgs& a = shards.s[blockIdx.y];
    const int warp = (int)blockIdx.x * 8 + (int)(threadIdx.x >> 5), lane = threadIdx.x & 31, part = warp % kHeadWarps<FN>;
    const int i = warp / kHeadWarps<FN>;
    if (i >= B) return;
    const VT* __restrict__ h = reinterpret_cast<const VT*>(a.rows.head + (size_t)a.rows.head_row[i] * a.rows.stride);
    const float* __restrict__ dp = a.d_pred + (size_t)i * D;
    const float* __restrict__ r = rel_table + (size_t)a.relation[i] * D;
    float* __restrict__ dh = a.d_head + (size_t)i * D;
    float* __restrict__ dr = a.d_relrow + (size_t)i * D;
    if (FN == SCORE_DISTMULT) {
        const float* const beside[2] = {r, dp};
        for_row<2>(h, beside, D, [&](int c, auto v, const auto& o) {
            const auto &q = o[0], &g = o[1];
            if constexpr (sizeof(v) == sizeof(float4)) {
                store4(dh + c, make_float4(g.x * q.x, g.y * q.y, g.z * q.z, g.w * q.w));
                store4(dr + c, make_float4(g.x * v.x, g.y * v.y, g.z * v.z, g.w * v.w));
            } else {
                dh[c] = g * q;
                dr[c] = g * v;
            }
        });
    } else if (FN == SCORE_ROTATE) {
        // The gradients of sine and cosine pass back through the float16 casts and the float16 sin / cos
        // (src/pag/pag.cpp:552-595, 619-633): rounded to float16 at each of those points, the angle's gradient is their
        // float16 sum.
        const int half = D / 2;
        for (int c = part * 32 + lane; c < half; c += 32 * kHeadWarps<FN>) {
            const float hr = load_as_float(h + c), hi = load_as_float(h + c + half), gr = dp[c], gi = dp[c + half];
            float s, co;
            rotate_sin_cos(r[c], s, co);
            dh[c] = gr * co + gi * s;
            dh[c + half] = -gr * s + gi * co;
            const float d_sin = round_to_half(-gr * hi + gi * hr), d_cos = round_to_half(gr * hr + gi * hi);
            const float via_sin = round_to_half(d_sin * co), via_cos = round_to_half(-d_cos * s);
            dr[c] = round_to_half(via_sin + via_cos);
            dr[c + half] = 0.f;  // the table keeps rows of D floats; the upper half of an angle row is unused
        }
    } else if (FN == SCORE_COMPLEX) {
        const int half = D / 2;
#pragma unroll 4
        for (int c = lane; c < half; c += 32) {
            const float hr = load_as_float(h + c), hi = load_as_float(h + c + half), rr = r[c], ri = r[c + half], gr = dp[c], gi = dp[c + half];
            dh[c] = gr * rr + gi * ri;
            dh[c + half] = -gr * ri + gi * rr;
            dr[c] = gr * hr + gi * hi;
            dr[c + half] = -gr * hi + gi * hr;
        }
    } else {
        //   d_head = d_pt - n (n . d_pt),   d_relrow = d_pt,
        //   d_n (total) = d_n - (n . h) d_pt - h (n . d_pt),   d_normrow = (d_n - n (n . d_n)) / |w|
        const float* __restrict__ w = normal_table + (size_t)a.relation[i] * D;
        const float* __restrict__ n = a.nrm + (size_t)i * D;
        const float* __restrict__ dn = a.d_nrm + (size_t)i * D;
        float sums[2][3] = {}, last[2][1] = {};
        two_strands(D, sums, [&](int c, float (&sum)[3]) {
            sum[0] += w[c] * w[c];
            sum[1] += n[c] * load_as_float(h + c);
            sum[2] += n[c] * dp[c];
        });
        const float ww = sums[0][0] + sums[1][0], nh = sums[0][1] + sums[1][1], ndp = sums[0][2] + sums[1][2];
        two_strands(D, last, [&](int c, float (&sum)[1]) { sum[0] += n[c] * (dn[c] - nh * dp[c] - load_as_float(h + c) * ndp); });
        const float ndn = last[0][0] + last[1][0];  // n . (total d_n)
        const float inv = 1.f / sqrtf(ww);
#pragma unroll 4
        for (int c = lane; c < D; c += 32) {
            dh[c] = dp[c] - n[c] * ndp;
            dr[c] = dp[c];
            a.d_normrow[(size_t)i * D + c] = (dn[c] - nh * dp[c] - load_as_float(h + c) * ndp - n[c] * ndn) * inv;
        }
    }
}

inline cudaError_t launch_lookup_bwd(const ShardArgs<LookupBwdArgs>& shards, int n_shards, const float* rel_table, const float* normal_table, int B, int D,
                                     int score_fn, int value_type, cudaStream_t stream, bool spread = true) {
    auto with_type = [&](auto fn) {
        constexpr int FN = decltype(fn)::value;
        const dim3 grid((unsigned)((B * kHeadWarps<FN> + 7) / 8), (unsigned)n_shards);
        if (value_type == 2) return launch_spread_if<k_lookup_bwd<__nv_bfloat16, FN>>(spread, grid, dim3(256), stream, shards, rel_table, normal_table, B, D);
        if (value_type == 1) return launch_spread_if<k_lookup_bwd<__half, FN>>(spread, grid, dim3(256), stream, shards, rel_table, normal_table, B, D);
        return launch_spread_if<k_lookup_bwd<float, FN>>(spread, grid, dim3(256), stream, shards, rel_table, normal_table, B, D);
    };
    switch (score_fn) {
        case SCORE_COMPLEX: return with_type(std::integral_constant<int, SCORE_COMPLEX>{});
        case SCORE_ROTATE: return with_type(std::integral_constant<int, SCORE_ROTATE>{});
        case SCORE_TRANSH: return with_type(std::integral_constant<int, SCORE_TRANSH>{});
        default: return with_type(std::integral_constant<int, SCORE_DISTMULT>{});
    }
}

}  // namespace kge
