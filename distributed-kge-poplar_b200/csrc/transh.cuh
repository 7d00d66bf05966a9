// TransH (src/poplar_kge.cpp:539-565): every relation has a translation row and a hyperplane
// normal; heads and tails are projected onto the hyperplane before the translation is compared,
//   n_i  = w_i / |w_i|                                  (w = relation_normal[relation_i])
//   pt_i = h_i - n_i (n_i . h_i) + r_i                  (the predicted tail)
//   e_ijk = pt_ik - (t_jk - n_ik (n_i . t_j))
//   score_ij = gamma - sum_k |e_ijk|                     (always the L1 form, whatever model.distance_fn says).
// Here are the pairwise distances with the two [B, T] matrices the backward needs (s_ij = n_i . t_j and
// u_ij = sum_k sign(e_ijk) n_ik) and the gradients of the distance with respect to pt, n and the tails; the prediction and its
// backward down to the head rows, the translation rows and the raw normals are k_lookup and k_lookup_bwd.  FP32-pipe kernels;
// every sum has a fixed order.
#pragma once

#include <algorithm>

#include "kernels.cuh"

namespace kge {

// raw[i, j] = sum_k |e_ijk|, and (BACKWARD) S[i, j] = n_i . t_j, U[i, j] = sum_k sign(e_ijk) n_ik.
// A warp owns 4 x 8 outputs with its lanes along k (lane l has k = l, l + 32, ...), so that a row is read in whole
// 128-byte lines and held by the lanes for all outputs of the tile; the 32 sums of a quantity are then reduced over the
// lanes by halving: a step exchanges half of a lane's sums with its partner and adds, 31 exchanges for 32 sums instead
// of 160, and leaves lane l with output l.  Bound by the FP32 pipe and the latency of the rows' loads (a lane's sums
// fill the registers of two blocks per SM).  512 x 768 x 128: 316 us with a warp per tail, a query after the other and
// three full reductions each; 39 us this way.
constexpr int kTranshRows = 4, kTranshCols = 8, kTranshWarps = 8;
constexpr int kTranshMaxTails = 65535 * kTranshCols * kTranshWarps;  // per launch

// sums[o] of all lanes added up for o = 0 .. 31; lane l returns the total of sums[l].
__device__ __forceinline__ float reduce_to_lanes(float (&sums)[32]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int half = 16; half > 0; half >>= 1) {
        const bool upper = (lane & half) != 0;
#pragma unroll
        for (int o = 0; o < half; ++o) {
            const float give = upper ? sums[o] : sums[o + half], keep = upper ? sums[o + half] : sums[o];
            sums[o] = keep + __shfl_xor_sync(0xffffffffu, give, half);
        }
    }
    return sums[0];
}

struct TranshScoreArgs {
    const float *pt, *nrm, *tails;
    float *raw, *S, *U;  // [B, ld]
};

template <bool BACKWARD>
__global__ void __launch_bounds__(32 * kTranshWarps, 2)
k_transh_score(const __grid_constant__ ShardArgs<TranshScoreArgs> shards, int B, int T, int D, int ld, ExchangeSync sync) {
    const TranshScoreArgs& args = shards.s[blockIdx.z];
    const float* __restrict__ pt = args.pt;
    const float* __restrict__ nrm = args.nrm;
    const float* __restrict__ tails = args.tails;
    float* __restrict__ raw = args.raw;
    float* __restrict__ S = args.S;
    float* __restrict__ U = args.U;
    grid_dependency_sync();
    exchange_wait(sync, XCHG_TAILS);  // the tails come from the other processes
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int i0 = blockIdx.x * kTranshRows, j0 = (blockIdx.y * kTranshWarps + warp) * kTranshCols;
    if (j0 >= T) return;
    // Rows as 32-bit offsets, past the end the last one.  A training step's rows (4096 of 2^20 columns at most) lie within
    // 2^32 of the first; those of a ranking pass, which may be any number, are counted from the block's own first rows.
    int from_i = 0, from_j = 0;
    if constexpr (!BACKWARD) {
        from_i = i0;
        from_j = (int)blockIdx.y * kTranshWarps * kTranshCols;
        pt += (size_t)from_i * D;
        nrm += (size_t)from_i * D;
        tails += (size_t)from_j * D;
    }
    uint32_t row_i[kTranshRows], row_j[kTranshCols];
#pragma unroll
    for (int a = 0; a < kTranshRows; ++a) row_i[a] = (uint32_t)(min(i0 + a, B - 1) - from_i) * (uint32_t)D;
#pragma unroll
    for (int b = 0; b < kTranshCols; ++b) row_j[b] = (uint32_t)(min(j0 + b, T - 1) - from_j) * (uint32_t)D;
    const int i = i0 + lane / kTranshCols, j = j0 + lane % kTranshCols;  // the output whose totals this lane ends up with
    const bool live = i < B && j < T;
    const size_t out = (size_t)i * ld + j;

    // two neighbouring tails at a time
    constexpr int kPairs = kTranshCols / 2;
    f32x2 s2[kTranshRows][kPairs];
#pragma unroll
    for (int a = 0; a < kTranshRows; ++a)
#pragma unroll
        for (int b = 0; b < kPairs; ++b) s2[a][b] = 0ull;
    for (int k = lane; k < D; k += 32) {
        f32x2 t[kPairs];
#pragma unroll
        for (int b = 0; b < kPairs; ++b) t[b] = pack2(tails[row_j[2 * b] + k], tails[row_j[2 * b + 1] + k]);
#pragma unroll
        for (int a = 0; a < kTranshRows; ++a) {
            const float n = nrm[row_i[a] + k];
#pragma unroll
            for (int b = 0; b < kPairs; ++b) s2[a][b] = fma2(pack2(n, n), t[b], s2[a][b]);
        }
    }
    float sums[32];
    auto spread = [&](const f32x2 (&v)[kTranshRows][kPairs]) {
#pragma unroll
        for (int a = 0; a < kTranshRows; ++a)
#pragma unroll
            for (int b = 0; b < kPairs; ++b) {
                const float2 f = unpack2(v[a][b]);
                sums[a * kTranshCols + 2 * b] = f.x;
                sums[a * kTranshCols + 2 * b + 1] = f.y;
            }
    };
    spread(s2);
    const float s_mine = reduce_to_lanes(sums);
    if (BACKWARD && live) S[out] = s_mine;
    f32x2 u2[kTranshRows][kPairs];
#pragma unroll
    for (int a = 0; a < kTranshRows; ++a)
#pragma unroll
        for (int b = 0; b < kPairs; ++b) {
            const int o = a * kTranshCols + 2 * b;
            s2[a][b] = pack2(__shfl_sync(0xffffffffu, s_mine, o), __shfl_sync(0xffffffffu, s_mine, o + 1));
            sums[o] = sums[o + 1] = 0.f;
            u2[a][b] = 0ull;
        }
    for (int k = lane; k < D; k += 32) {
        f32x2 t[kPairs];
#pragma unroll
        for (int b = 0; b < kPairs; ++b) t[b] = pack2(tails[row_j[2 * b] + k], tails[row_j[2 * b + 1] + k]);
#pragma unroll
        for (int a = 0; a < kTranshRows; ++a) {
            const float p = pt[row_i[a] + k], n = nrm[row_i[a] + k];
            const f32x2 pp = pack2(p, p), nn = pack2(n, n);
#pragma unroll
            for (int b = 0; b < kPairs; ++b) {
                const int o = a * kTranshCols + 2 * b;
                const f32x2 e = fma2(nn, s2[a][b], sub2(pp, t[b]));
                const float2 f = unpack2(e);
                sums[o] += fabsf(f.x);
                sums[o + 1] += fabsf(f.y);
                if (BACKWARD) u2[a][b] = fma2(nn, sign2(e), u2[a][b]);
            }
        }
    }
    const float dist = reduce_to_lanes(sums);
    if (live) raw[out] = dist;
    if (BACKWARD) {
        spread(u2);
        const float total = reduce_to_lanes(sums);
        if (live) U[out] = total;
    }
}

// S and U null: the distances alone (predict).
inline cudaError_t launch_transh_score(const ShardArgs<TranshScoreArgs>& shards, int n_shards, int B, int T, int D, int ld, const ExchangeSync& sync,
                                       cudaStream_t stream) {
    constexpr int kCols = kTranshCols * kTranshWarps;
    const dim3 grid((B + kTranshRows - 1) / kTranshRows, (T + kCols - 1) / kCols, (unsigned)n_shards), block(32 * kTranshWarps);
    const bool backward = shards.s[0].S != nullptr;
    if (backward && (uint64_t)std::max(B, T) * D > UINT32_MAX) return cudaErrorInvalidValue;
    if (T > kTranshMaxTails) return cudaErrorInvalidValue;
    if (backward) return launch_dependent(k_transh_score<true>, grid, block, 0, stream, shards, B, T, D, ld, sync);
    return launch_dependent(k_transh_score<false>, grid, block, 0, stream, shards, B, T, D, ld, sync);
}
inline cudaError_t launch_transh_score(const float* pt, const float* nrm, const float* tails, float* raw, int B, int T, int D, cudaStream_t stream) {
    ShardArgs<TranshScoreArgs> shards{};
    shards.s[0] = TranshScoreArgs{pt, nrm, tails, raw, nullptr, nullptr};
    return launch_transh_score(shards, 1, B, T, D, T, ExchangeSync{}, stream);
}

// Gradients of the distances times C [B, T] (C = d loss / d raw), with sg_ijk = sign(pt_ik - t_jk + n_ik S_ij):
//   rows i:  d_pt_ik = sum_j C_ij sg_ijk,   d_n_ik = sum_j C_ij (sg_ijk S_ij + U_ij t_jk)
//   rows j:  d_t_jk  = sum_i C_ij (U_ij n_ik - sg_ijk), stored to the shard that owns tail j
// In k_pair_bwd's form (sums in order, the operands staged one chunk ahead) but with one column per lane, 32 per block:
// a packed instruction holds the FP32 pipe twice as long, so pairs only halve the warps that hide latency.  The first blocks
// take the rows i (one per warp, chunks of 64 tails), the others the rows j (two per warp, which share the reads of pt and
// n; chunks of 32 triples).  512 x 768 x 128: 153 us with a block per output row and a thread per column, 87 us with pairs,
// 61 us this way.
struct TranshBwdArgs {
    const float *pt, *nrm, *tails, *C, *S, *U;
    float *d_pt, *d_n;
    float* const* d_tail_blocks;
    int block_rows, B, T, D, ld, blocks_i;  // ld: floats between rows of C, S and U; what lies between T and ld is zero
};
constexpr int kTranshBwdCols = 32, kTranshChunkI = 64, kTranshChunkJ = 32;
constexpr int kTranshStage = 3 * kPairWarps * kTranshChunkI + kTranshChunkI * kTranshBwdCols;  // floats of one chunk
static_assert(3 * 2 * kPairWarps * kTranshChunkJ + 2 * kTranshChunkJ * kTranshBwdCols <= kTranshStage, "both kinds of rows use the same memory");

__device__ __forceinline__ float sign_of(float e) {
    const float inf = __int_as_float(0x7f800000);
    return positive(e, inf) - positive(e, -inf);
}

__device__ __forceinline__ void transh_bwd_triples(const TranshBwdArgs& g, int block, float (*smem)[kTranshStage]) {
    constexpr int kChunk = kTranshChunkI, kPlane = kPairWarps * kChunk, kCols = kTranshBwdCols;
    const int D = g.D, T = g.T, col_tiles = (D + kCols - 1) / kCols;
    const int i0 = block / col_tiles * kPairWarps, k0 = block % col_tiles * kCols;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, i = i0 + warp, k = k0 + lane;
    const bool t_vec = (D & 3) == 0, c_vec = (g.ld & 3) == 0, live = i < g.B && k < D;
    auto stage = [&](int j0, float* to) {
        const float* planes[3] = {g.C, g.S, g.U};
#pragma unroll
        for (int q = 0; q < 3; ++q) stage_rows<kPairWarps, kChunk>(to + q * kPlane, planes[q] + (size_t)i0 * g.ld + j0, g.ld, g.B - i0, T - j0, c_vec);
        stage_rows<kChunk, kCols>(to + 3 * kPlane, g.tails + (size_t)j0 * D + k0, D, T - j0, D - k0, t_vec);
    };
    const float p = live ? g.pt[(size_t)i * D + k] : 0.f, n = live ? g.nrm[(size_t)i * D + k] : 0.f;
    float acc_p = 0.f, acc_n = 0.f;
    stage(0, smem[0]);
    stage_commit();
    for (int j0 = 0, half = 0; j0 < T; j0 += kChunk, half ^= 1) {
        if (j0 + kChunk < T) stage(j0 + kChunk, smem[half ^ 1]);
        stage_commit();
        stage_wait_previous();
        __syncthreads();
        const float* c = smem[half] + warp * kChunk;
        const float* t = smem[half] + 3 * kPlane + lane;
#pragma unroll 2
        for (int j = 0; j < kChunk; j += 4) {
            const float4 qc = load4(c + j), qs = load4(c + kPlane + j), qu = load4(c + 2 * kPlane + j);
            const float cj[4] = {qc.x, qc.y, qc.z, qc.w}, sj[4] = {qs.x, qs.y, qs.z, qs.w}, uj[4] = {qu.x, qu.y, qu.z, qu.w};
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const float tj = t[(j + u) * kCols], sg = sign_of(fmaf(n, sj[u], p - tj));
                acc_p = fmaf(cj[u], sg, acc_p);
                acc_n = fmaf(cj[u], fmaf(sg, sj[u], uj[u] * tj), acc_n);
            }
        }
        __syncthreads();
    }
    if (!live) return;
    g.d_pt[(size_t)i * D + k] = acc_p;
    g.d_n[(size_t)i * D + k] = acc_n;
}

__device__ __forceinline__ void transh_bwd_tails(const TranshBwdArgs& g, int block, float (*smem)[kTranshStage]) {
    constexpr int kChunk = kTranshChunkJ, kRows = 2 * kPairWarps, kPlane = kRows * kChunk, kCols = kTranshBwdCols, kWide = kChunk * kCols;
    const int D = g.D, T = g.T, B = g.B, col_tiles = (D + kCols - 1) / kCols;
    const int j0 = block / col_tiles * kRows, k0 = block % col_tiles * kCols;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, j = j0 + 2 * warp, k = k0 + lane;
    const bool vec = (D & 3) == 0, c_vec = (g.ld & 3) == 0;
    auto stage = [&](int i0, float* to) {
        const float* planes[3] = {g.C, g.S, g.U};
#pragma unroll
        for (int q = 0; q < 3; ++q) stage_rows<kChunk, kRows>(to + q * kPlane, planes[q] + (size_t)i0 * g.ld + j0, g.ld, B - i0, T - j0, c_vec);
        stage_rows<kChunk, kCols>(to + 3 * kPlane, g.pt + (size_t)i0 * D + k0, D, B - i0, D - k0, vec);
        stage_rows<kChunk, kCols>(to + 3 * kPlane + kWide, g.nrm + (size_t)i0 * D + k0, D, B - i0, D - k0, vec);
    };
    float t[2], acc[2] = {0.f, 0.f};
#pragma unroll
    for (int r = 0; r < 2; ++r) t[r] = j + r < T && k < D ? g.tails[(size_t)(j + r) * D + k] : 0.f;
    stage(0, smem[0]);
    stage_commit();
    for (int i0 = 0, half = 0; i0 < B; i0 += kChunk, half ^= 1) {
        if (i0 + kChunk < B) stage(i0 + kChunk, smem[half ^ 1]);
        stage_commit();
        stage_wait_previous();
        __syncthreads();
        const float* c = smem[half] + 2 * warp;
        const float* p = smem[half] + 3 * kPlane + lane;
#pragma unroll 8
        for (int i = 0; i < kChunk; ++i) {
            const float pi = p[i * kCols], ni = p[kWide + i * kCols];
            const float2 qc = *reinterpret_cast<const float2*>(c + i * kRows), qs = *reinterpret_cast<const float2*>(c + kPlane + i * kRows),
                         qu = *reinterpret_cast<const float2*>(c + 2 * kPlane + i * kRows);
            const float cj[2] = {qc.x, qc.y}, sj[2] = {qs.x, qs.y}, uj[2] = {qu.x, qu.y};
#pragma unroll
            for (int r = 0; r < 2; ++r) acc[r] = fmaf(cj[r], fmaf(uj[r], ni, -sign_of(fmaf(ni, sj[r], pi - t[r]))), acc[r]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int r = 0; r < 2; ++r)
        if (j + r < T && k < D) g.d_tail_blocks[(j + r) / g.block_rows][(size_t)((j + r) % g.block_rows) * D + k] = acc[r];
}

static __global__ void __launch_bounds__(32 * kPairWarps, 4) k_transh_bwd(const __grid_constant__ ShardArgs<TranshBwdArgs> shards) {
    grid_dependency_sync();
    const TranshBwdArgs& g = shards.s[blockIdx.y];
    __shared__ __align__(16) float smem[2][kTranshStage];
    if ((int)blockIdx.x < g.blocks_i) transh_bwd_triples(g, blockIdx.x, smem);
    else transh_bwd_tails(g, (int)blockIdx.x - g.blocks_i, smem);
}

inline cudaError_t launch_transh_bwd(ShardArgs<TranshBwdArgs> shards, int n_shards, cudaStream_t stream) {
    const TranshBwdArgs& g = shards.s[0];
    const int col_tiles = (g.D + kTranshBwdCols - 1) / kTranshBwdCols;
    const int blocks_i = (g.B + kPairWarps - 1) / kPairWarps * col_tiles, blocks_j = (g.T + 2 * kPairWarps - 1) / (2 * kPairWarps) * col_tiles;
    for (int s = 0; s < n_shards; ++s) shards.s[s].blocks_i = blocks_i;
    return launch_dependent(k_transh_bwd, dim3(blocks_i + blocks_j, (unsigned)n_shards), dim3(32 * kPairWarps), 0, stream, shards);
}

}  // namespace kge
