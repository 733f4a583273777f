// The float32 product of up to 16 rows in bfloat16 parts (gemm_f32_split.cuh): the weights are read once
// and split in registers, a warp multiplies 16 features by a block of 64 terms at a time with `mma.sync` m16n8k16, the
// tokens on its N side; the warps of a CTA (and CTAs of a cluster) share the blocks of the same features.
//
// What bounds it: reading the weights, if they arrive all the time and the splitting (about 260 instructions for a block's
// 4 KB) runs under it.  Hence the walking kernel for few rows by many features, and parts of the rows kept in
// registers.  In chains of products over weights that are not in L2, FMA kernel before / now, us: 1 row by 151,936 x 896
// 95.9 / 86.4 (6.3 TB/s), 5 rows 114 / 86.8; 9,728 x 896, 1, 4, 8 and 16 rows 7.4, 8.9, 12.1, 16.3 / 8.6, 8.9, 9.4, 16.7;
// 896 x 4,864 8.5, 10.1, 14.3, 14.6 / 7.6, 8.0, 8.1, 11.2; 1,152 x 896 4.0, 4.4, 5.3, 5.7 / 3.8, 4.2, 4.4, 5.3.
#include <cooperative_groups.h>

#include "gemm_f32_split.cuh"

namespace somi {

constexpr int kFrFeatures = 16, kFrWarps = 8, kFrThreads = 32 * kFrWarps;
constexpr int kFrMostSmem = 227 * 1024;
constexpr int kFrPitch = 20;              // floats between tokens of a partial tile (no bank twice in a store)

// A warp's blocks of the weights arrive in shared memory by cp.async, all of them or STAGES ahead, before the
// dependency wait where they are constants.  A block there is [16 rows][64 floats] with its 16-byte quads permuted
// so that the eight lanes of an access (two rows, four quads) meet eight different bank groups: quad q of row r stands at
// (q & 8) + ((q ^ (q / 8 * 2) ^ (r % 2 * 4)) & 7).

// The terms of a step (gemm_f32_split.cuh) are four quads of a row, one a lane; the two numbers of each half of its quad
// are neighbours in the MMA on both sides.
// The sums of a block in shared memory with 8 MT rows whose parts `parts` gives, a lane's share of a step at a time.
template <int MT, typename F>
__device__ __forceinline__ void fr_multiply(float (&acc)[MT][4], const float* block, F parts) {
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const float* wr = block + g * kFsBK + (t & 2) * 16;
    const int low = (t & 1) ^ (t & 2) ^ ((g & 1) << 2);
    uint32_t a0[4][4];
    uint2 c0[MT][4];
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[m][e] = 0.f;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int q = 4 * (low ^ (2 * j));
        const float4 u = *reinterpret_cast<const float4*>(wr + q), v = *reinterpret_cast<const float4*>(wr + 8 * kFsBK + q);
        uint32_t a1[4], a2[4];
        uint2 c1[MT], c2[MT];
        fs_split(u.x, u.y, a0[j][0], a1[0], a2[0]);
        fs_split(v.x, v.y, a0[j][1], a1[1], a2[1]);
        fs_split(u.z, u.w, a0[j][2], a1[2], a2[2]);
        fs_split(v.z, v.w, a0[j][3], a1[3], a2[3]);
#pragma unroll
        for (int m = 0; m < MT; ++m) parts(m, j, c0[m][j], c1[m], c2[m]);
#pragma unroll
        for (int m = 0; m < MT; ++m) mma_bf16_16816(acc[m], a0[j], c2[m].x, c2[m].y);
#pragma unroll
        for (int m = 0; m < MT; ++m) mma_bf16_16816(acc[m], a2, c0[m][j].x, c0[m][j].y);
#pragma unroll
        for (int m = 0; m < MT; ++m) mma_bf16_16816(acc[m], a1, c1[m].x, c1[m].y);
#pragma unroll
        for (int m = 0; m < MT; ++m) mma_bf16_16816(acc[m], a0[j], c1[m].x, c1[m].y);
#pragma unroll
        for (int m = 0; m < MT; ++m) mma_bf16_16816(acc[m], a1, c0[m][j].x, c0[m][j].y);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int m = 0; m < MT; ++m) mma_bf16_16816(acc[m], a0[j], c0[m][j].x, c0[m][j].y);
}

// own_blocks: blocks of a CTA (whole ranges); warp i takes every eighth of them, from the i-th on.  IN_PLACE: a warp has no more of
// them than stages, and a block's sums overwrite the block.
template <int MT, int STAGES, bool IN_PLACE, bool CLUSTER>
__global__ void __launch_bounds__(kFrThreads, MT > 1 || STAGES > 2 ? 2 : 3)
f32_rows_kernel(const float* __restrict__ x, const float* __restrict__ w, const float* __restrict__ bias,
                float* __restrict__ y, int M, int N, int K, int blocks, int range_blocks, int own_blocks, int cluster_size,
                long long ldx, long long ldy, long long bsx, long long bsw, long long bsy, int w_constant) {
    constexpr int OUT = kFrFeatures * 8 * MT, TILE = 8 * MT * kFrPitch, BLOCK = kFrFeatures * kFsBK;
    extern __shared__ __align__(128) float fr_buf[];     // [warp][stage][BLOCK], [block of this CTA][TILE], [range][OUT]
    pdl_launch_dependents();
    x += blockIdx.z * bsx;
    w += blockIdx.z * bsw;
    y += blockIdx.z * bsy;
    const int rank = CLUSTER ? blockIdx.x % cluster_size : 0;
    const int n0 = (CLUSTER ? blockIdx.x / cluster_size : blockIdx.x) * kFrFeatures;
    const int b0 = min(blocks, rank * own_blocks), b1 = min(blocks, b0 + own_blocks);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    const int first = b0 + warp;
    float* ring = fr_buf + warp * STAGES * BLOCK;
    float* sums = fr_buf + kFrWarps * STAGES * BLOCK;

    // a lane copies quad `lane % 16` of every second row of a block; rows behind the last are not read
    const int q16 = lane & 15, row0 = lane >> 4, live_rows = N - n0 - row0;
    const float* w_src = w + static_cast<long long>(n0 + row0) * K + 4 * q16;
    const uint32_t w_dst = smem_u32(ring + row0 * kFsBK + 4 * ((q16 & 8) | ((q16 ^ (q16 >> 3 << 1) ^ (row0 << 2)) & 7)));
    auto fetch = [&](int b, int stage) {
        if (b < b1) {
            const float* src = w_src + b * kFsBK;
            const uint32_t dst = w_dst + stage * (BLOCK * 4);
            if ((b + 1) * kFsBK <= K && n0 + kFrFeatures <= N) {
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst + i * 2 * kFsBK * 4), "l"(src + i * 2 * K));
            } else {
                const bool in = b * kFsBK + 4 * q16 < K;
                for (int i = 0; i < 8; ++i) {
                    const bool live = in && 2 * i < live_rows;
                    cp_async_16(dst + i * 2 * kFsBK * 4, live ? src + i * 2 * K : w, live ? 16 : 0);
                }
            }
        }
        cp_async_commit();
    };
    float4 xq[MT][4];
    const int quad = t < 2 ? 4 * t : 24 + 4 * t;         // of step 0; eight terms further on in each
    const float* x_src[MT];                              // (rows behind the last repeat it: what they give is not stored)
#pragma unroll
    for (int m = 0; m < MT; ++m) x_src[m] = x + min(8 * m + g, M - 1) * ldx + quad;
    auto load_x = [&](int b) {
        if ((b + 1) * kFsBK <= K) {
#pragma unroll
            for (int m = 0; m < MT; ++m)
#pragma unroll
                for (int j = 0; j < 4; ++j) xq[m][j] = *reinterpret_cast<const float4*>(x_src[m] + b * kFsBK + 8 * j);
        } else {
#pragma unroll
            for (int m = 0; m < MT; ++m)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int k = b * kFsBK + 8 * j;
                    xq[m][j] = k + quad < K ? *reinterpret_cast<const float4*>(x_src[m] + k) : make_float4(0.f, 0.f, 0.f, 0.f);
                }
        }
    };
    if (!w_constant) pdl_wait();
#pragma unroll
    for (int i = 0; i < STAGES; ++i) fetch(first + i * kFrWarps, i);            // [constant], or behind the wait
    pdl_wait();
    if (first < b1) load_x(first);
    int stage = 0;
#pragma unroll 1
    for (int b = first; b < b1; b += kFrWarps) {
        cp_async_wait<STAGES - 1>();
        __syncwarp();
        float acc[MT][4];
        fr_multiply<MT>(acc, ring + stage * BLOCK, [&](int m, int j, uint2& c0, uint2& c1, uint2& c2) {
            fs_split(xq[m][j].x, xq[m][j].y, c0.x, c1.x, c2.x);
            fs_split(xq[m][j].z, xq[m][j].w, c0.y, c1.y, c2.y);
        });
        if (b + kFrWarps < b1) load_x(b + kFrWarps);
        __syncwarp();                                    // the stage has been read
        float* block_sums = IN_PLACE ? ring + stage * BLOCK : sums + (b - b0) * TILE;
        if (!IN_PLACE) fetch(b + STAGES * kFrWarps, stage);
        else cp_async_commit();
        stage = stage + 1 == STAGES ? 0 : stage + 1;
        float* dst = block_sums + 2 * t * kFrPitch + g;
#pragma unroll
        for (int m = 0; m < MT; ++m)
#pragma unroll
            for (int e = 0; e < 4; ++e) dst[(8 * m + (e & 1)) * kFrPitch + 8 * (e >> 1)] = acc[m][e];
    }
    __syncthreads();
    // a thread adds the blocks of its outputs' ranges, and (alone, or from all CTAs of the cluster) the ranges
    auto range_sum = [&](int r, int o) {
        const int i0 = r * range_blocks - b0, i1 = min(blocks - b0, i0 + range_blocks), at = o / kFrFeatures * kFrPitch + o % kFrFeatures;
        auto one = [&](int i) {
            return IN_PLACE ? fr_buf[((i % kFrWarps) * STAGES + i / kFrWarps) * BLOCK + at] : sums[i * TILE + at];
        };
        float s = one(i0);
#pragma unroll 4
        for (int i = i0 + 1; i < i1; ++i) s = __fadd_rn(s, one(i));
        return s;
    };
    auto store = [&](int o, float v) {
        const int m = o / kFrFeatures, n = n0 + o % kFrFeatures;
        if (m >= M || n >= N) return;
        if (!fs_finite(v)) v = fs_plain_sum(x + m * ldx, w + static_cast<long long>(n) * K, K);
        y[m * ldy + n] = bias ? __fadd_rn(v, bias[n]) : v;
    };
    const int ranges = (blocks + range_blocks - 1) / range_blocks;
    if (!CLUSTER) {
        for (int o = threadIdx.x; o < OUT; o += kFrThreads) {
            float v = range_sum(0, o);
            for (int r = 1; r < ranges; ++r) v = __fadd_rn(v, range_sum(r, o));
            store(o, v);
        }
        return;
    }
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    const int own_ranges = own_blocks / range_blocks, r0 = rank * own_ranges, r1 = min(ranges, r0 + own_ranges);
    float* totals = sums + (IN_PLACE ? 0 : own_blocks * TILE);
    for (int i = threadIdx.x; i < (r1 - r0) * OUT; i += kFrThreads) totals[i] = range_sum(r0 + i / OUT, i % OUT);
    cluster.sync();
    for (int o = rank * kFrThreads + threadIdx.x; o < OUT; o += cluster_size * kFrThreads) {
        float v = cluster.map_shared_rank(totals, 0)[o];
        for (int r = 1; r < ranges; ++r)
            v = __fadd_rn(v, cluster.map_shared_rank(totals, r / own_ranges)[r % own_ranges * OUT + o]);
        store(o, v);
    }
    cluster.sync();                                      // no CTA leaves while its sums are read
}

// Up to 8 rows and 16 blocks by many features: the CTAs that fill the chip walk through the tiles.  A warp keeps its (one
// or two) blocks' parts of the rows in registers for good, and each of its stages is filled again, with the next tile's weights, as
// soon as it has been read: weights arrive all the time.  (With a CTA a tile, those of an SM wait for their weights
// together and multiply together.)
__global__ void __launch_bounds__(kFrThreads, 2)
f32_rows_walk_kernel(const float* __restrict__ x, const float* __restrict__ w, const float* __restrict__ bias,
                     float* __restrict__ y, int M, int N, int K, int blocks, int range_blocks, int tiles, long long ldx,
                     long long ldy, long long bsx, long long bsw, long long bsy, int w_constant) {
    constexpr int OUT = kFrFeatures * 8, TILE = 8 * kFrPitch, BLOCK = kFrFeatures * kFsBK;
    extern __shared__ __align__(128) float fr_buf[];     // [warp][stage][BLOCK], twice [block][TILE]
    pdl_launch_dependents();
    x += blockIdx.z * bsx;
    w += blockIdx.z * bsw;
    y += blockIdx.z * bsy;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    float* ring = fr_buf + warp * 2 * BLOCK;
    float* sums = fr_buf + kFrWarps * 2 * BLOCK;
    const int q16 = lane & 15, row0 = lane >> 4;
    const float* w_src = w + static_cast<long long>(row0) * K + 4 * q16;
    const uint32_t w_dst = smem_u32(ring + row0 * kFsBK + 4 * ((q16 & 8) | ((q16 ^ (q16 >> 3 << 1) ^ (row0 << 2)) & 7)));
    auto fetch = [&](int tile, int i) {                  // this warp's block i of a tile into stage i
        const int b = warp + i * kFrWarps, n0 = tile * kFrFeatures;
        if (b < blocks && tile < tiles) {
            const float* src = w_src + static_cast<long long>(n0) * K + b * kFsBK;
            const uint32_t dst = w_dst + i * (BLOCK * 4);
            if ((b + 1) * kFsBK <= K && n0 + kFrFeatures <= N) {
#pragma unroll
                for (int r = 0; r < 8; ++r)
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst + r * 2 * kFsBK * 4), "l"(src + r * 2 * K));
            } else {
                const bool in = b * kFsBK + 4 * q16 < K;
                for (int r = 0; r < 8; ++r) {
                    const bool live = in && n0 + row0 + 2 * r < N;
                    cp_async_16(dst + r * 2 * kFsBK * 4, live ? src + r * 2 * K : w, live ? 16 : 0);
                }
            }
        }
        cp_async_commit();
    };
    int tile = blockIdx.x;
    if (!w_constant) pdl_wait();
    fetch(tile, 0);                                      // [constant], or behind the wait
    fetch(tile, 1);
    pdl_wait();
    uint2 parts[2][4][3];
    const float* x_src = x + min(g, M - 1) * ldx + (t < 2 ? 4 * t : 24 + 4 * t);   // (rows behind the last repeat it)
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int k = (warp + i * kFrWarps) * kFsBK + 8 * j;
            const float4 q = k + (t < 2 ? 4 * t : 24 + 4 * t) < K ? *reinterpret_cast<const float4*>(x_src + k)
                                                                  : make_float4(0.f, 0.f, 0.f, 0.f);
            fs_split(q.x, q.y, parts[i][j][0].x, parts[i][j][1].x, parts[i][j][2].x);
            fs_split(q.z, q.w, parts[i][j][0].y, parts[i][j][1].y, parts[i][j][2].y);
        }
    const int ranges = (blocks + range_blocks - 1) / range_blocks;
    for (int odd = 0; tile < tiles; tile += gridDim.x, odd ^= 1) {
        float* tile_sums = sums + odd * blocks * TILE;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int b = warp + i * kFrWarps;
            cp_async_wait<1>();                          // (the other stage's copies may be under way)
            __syncwarp();
            if (b < blocks) {
                float acc[1][4];
                fr_multiply<1>(acc, ring + i * BLOCK, [&](int, int j, uint2& c0, uint2& c1, uint2& c2) {
                    c0 = parts[i][j][0];
                    c1 = parts[i][j][1];
                    c2 = parts[i][j][2];
                });
                float* dst = tile_sums + b * TILE + 2 * t * kFrPitch + g;
#pragma unroll
                for (int e = 0; e < 4; ++e) dst[(e & 1) * kFrPitch + 8 * (e >> 1)] = acc[0][e];
            }
            __syncwarp();                                // the stage has been read
            fetch(tile + gridDim.x, i);
        }
        __syncthreads();
        const int m = threadIdx.x / kFrFeatures, n = tile * kFrFeatures + threadIdx.x % kFrFeatures;
        if (m < M && n < N) {
            const float* src = tile_sums + m * kFrPitch + threadIdx.x % kFrFeatures;
            float v = 0.f;
            for (int r = 0, i = 0; r < ranges; ++r) {
                float s = src[i++ * TILE];
                for (const int end = min(blocks, (r + 1) * range_blocks); i < end; ++i) s = __fadd_rn(s, src[i * TILE]);
                v = r == 0 ? s : __fadd_rn(v, s);
            }
            if (!fs_finite(v)) v = fs_plain_sum(x + m * ldx, w + static_cast<long long>(n) * K, K);
            y[m * ldy + n] = bias ? __fadd_rn(v, bias[n]) : v;
        }
    }
}

template <int MT, int STAGES, bool IN_PLACE, bool CLUSTER>
int fr_launch_one(const FsArgs& a, int cluster, int blocks, int range_blocks, int own, cudaStream_t stream) {
    const int smem = 4 * (kFrWarps * STAGES * kFrFeatures * kFsBK + (IN_PLACE ? 0 : own * 8 * MT * kFrPitch) +
                          (CLUSTER ? own / range_blocks * kFrFeatures * 8 * MT : 0));
    constexpr auto kernel = f32_rows_kernel<MT, STAGES, IN_PLACE, CLUSTER>;
    allow_smem<kernel>(kFrMostSmem);
    launch_pdl_cluster(kernel, dim3((a.N + kFrFeatures - 1) / kFrFeatures * cluster, 1, a.batch), dim3(kFrThreads), smem,
                       cluster, stream, a.x, a.w, a.bias, a.y, a.M, a.N, a.K, blocks, range_blocks, own, cluster, a.ldx, a.ldy,
                       a.bsx, a.bsw, a.bsy, a.w_constant);
    return launch_status();
}

template <int MT>
int fr_launch(const FsArgs& a, cudaStream_t stream) {
    const int blocks = (a.K + kFsBK - 1) / kFsBK, range_blocks = fs_range_blocks(blocks);
    const int ranges = (blocks + range_blocks - 1) / range_blocks;
    const long long tiles = static_cast<long long>((a.N + kFrFeatures - 1) / kFrFeatures) * a.batch;
    // more tiles than the chip holds CTAs, and registers for the rows' parts (151,936 x 896, 1 row: a CTA a tile 103 us,
    // walking 86; 9,728 x 896, 8 rows: 12.1 and 9.4)
    if (MT == 1 && blocks <= 2 * kFrWarps && tiles > 148 * 2) {
        const int smem = 4 * (kFrWarps * 2 * kFrFeatures * kFsBK + 2 * blocks * 8 * kFrPitch);
        allow_smem<f32_rows_walk_kernel>(kFrMostSmem);
        const int all = (a.N + kFrFeatures - 1) / kFrFeatures, ctas = (148 * 2 + a.batch - 1) / a.batch;
        launch_pdl(f32_rows_walk_kernel, dim3(all < ctas ? all : ctas, 1, a.batch), dim3(kFrThreads), smem, stream, a.x, a.w,
                   a.bias, a.y, a.M, a.N, a.K, blocks, range_blocks, all, a.ldx, a.ldy, a.bsx, a.bsw, a.bsy, a.w_constant);
        return launch_status();
    }
    // at most 40 blocks a CTA, five a warp, whose sums stand in shared memory; fewer while the chip has room for more CTAs
    // (896 x 4,864, 8 rows: 112 CTAs of a cluster of two 10.9 us, 224 of four 8.0)
    int cluster = 1;
    while (blocks > 40 * cluster || (blocks > 20 * cluster && cluster < 8 && 2 * cluster * tiles <= 148 * 2)) cluster *= 2;
    const int own = (ranges + cluster - 1) / cluster * range_blocks, most = own < blocks ? own : blocks;
#define SOMI_FR(STAGES, IN_PLACE) \
    return cluster > 1 ? fr_launch_one<MT, STAGES, IN_PLACE, true>(a, cluster, blocks, range_blocks, own, stream) \
                       : fr_launch_one<MT, STAGES, IN_PLACE, false>(a, 1, blocks, range_blocks, own, stream)
    if (most <= 2 * kFrWarps) SOMI_FR(2, true);
    if (most <= 3 * kFrWarps) SOMI_FR(3, true);
    SOMI_FR(3, false);
#undef SOMI_FR
}

int fs_launch_rows(const FsArgs& a, cudaStream_t stream) { return a.M <= 8 ? fr_launch<1>(a, stream) : fr_launch<2>(a, stream); }

}  // namespace somi
