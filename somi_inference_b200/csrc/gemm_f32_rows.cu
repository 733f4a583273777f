// The float32 product of up to 16 rows in bfloat16 parts (gemm_f32_split.cuh): the weights are read once
// and split in registers, a warp multiplies 16 features by a block of 64 terms at a time with `mma.sync` m16n8k16, the
// tokens on its N side; the warps of a CTA (and CTAs of a cluster) share the blocks of the same features.
//
// What bounds it: reading the weights, if they arrive all the time and the splitting (about 260 instructions for a block's
// 4 KB) runs under it.  Hence the stream, whose CTAs stay, and deep stages where the chip is not full.  In chains of products
// over weights that are not in L2, FMA kernel before / now, us (what `fr_launch` measured between kernels stands there):
//     151,936 x 896, 1, 4, 8, 16 rows   96, 104, 116, 150   / 82, 85, 85, 129   (6.6 TB/s)
//     152,064 x 3,584                   379, 398, 441, 584  / 309, 315, 330, 496 (7.1 TB/s)
//     22,016 x 2,048                    39, 48, 69, 81      / 29, 29, 30, 48
//     9,728 x 896                       7.4, 8.7, 12.1, 17  / 8.0, 8.2, 8.3, 15.6
//     896 x 4,864                       8.4, 9.7, 13.4, 14  / 7.5, 7.9, 8.1, 11.1
//     2,048 x 2,048                     5.9, 7.3, 11.9, 12  / 5.4, 5.7, 5.8, 7.8
//     1,152 x 896                       3.9, 4.4, 5.3, 5.6  / 3.2, 3.6, 3.5, 4.9
// One or two rows are up to 10 % slower than as FMAs where the tiles fill the chip little more than once (9,728 x 896, 5,120 x 5,120,
// 2,560 x 2,048): there the FMA kernel's smaller CTAs let more of the next product's weights be under way; and for few features of many
// terms (256 x 3,584, 768 x 8,960), where a warp's range is a chain.
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

// The same by CTAs that fill the chip and walk through the tiles: a warp takes a whole range of a tile, adds its blocks in registers, and
// each of its stages is filled again as soon as it has been read, with a later block or the next tile's first: weights arrive all the time.
// RANGES warps a CTA, `CTAS` of them an SM.
template <int MT, int STAGES, int RANGES, int CTAS>
__global__ void __launch_bounds__(32 * RANGES, CTAS)
f32_rows_stream_kernel(const float* __restrict__ x, const float* __restrict__ w, const float* __restrict__ bias,
                       float* __restrict__ y, int M, int N, int K, int blocks, int range_blocks, int tiles, long long ldx,
                       long long ldy, long long bsx, long long bsw, long long bsy, int w_constant) {
    constexpr int OUT = kFrFeatures * 8 * MT, TILE = 8 * MT * kFrPitch, BLOCK = kFrFeatures * kFsBK;
    extern __shared__ __align__(128) float fr_buf[];     // [warp][stage][BLOCK], twice [warp][TILE]
    pdl_launch_dependents();
    x += blockIdx.z * bsx;
    w += blockIdx.z * bsw;
    y += blockIdx.z * bsy;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    const int b0 = min(blocks, warp * range_blocks), b1 = min(blocks, b0 + range_blocks);
    float* ring = fr_buf + warp * STAGES * BLOCK;
    float* sums = fr_buf + RANGES * STAGES * BLOCK;
    const int q16 = lane & 15, row0 = lane >> 4;
    const float* w_src = w + static_cast<long long>(row0) * K + 4 * q16;
    const uint32_t w_dst = smem_u32(ring + row0 * kFsBK + 4 * ((q16 & 8) | ((q16 ^ (q16 >> 3 << 1) ^ (row0 << 2)) & 7)));
    // the next block to fetch: blocks b0 .. of a tile, then of the CTA's next one
    int next_tile = blockIdx.x, next = b0;
    auto fetch = [&](int stage) {
        if (next_tile < tiles && next < b1) {
            const int n0 = next_tile * kFrFeatures;
            const float* src = w_src + static_cast<long long>(n0) * K + next * kFsBK;
            const uint32_t dst = w_dst + stage * (BLOCK * 4);
            if ((next + 1) * kFsBK <= K && n0 + kFrFeatures <= N) {
#pragma unroll
                for (int r = 0; r < 8; ++r)
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst + r * 2 * kFsBK * 4), "l"(src + r * 2 * K));
            } else {
                const bool in = next * kFsBK + 4 * q16 < K;
                for (int r = 0; r < 8; ++r) {
                    const bool live = in && n0 + row0 + 2 * r < N;
                    cp_async_16(dst + r * 2 * kFsBK * 4, live ? src + r * 2 * K : w, live ? 16 : 0);
                }
            }
            if (++next == b1) {
                next = b0;
                next_tile += gridDim.x;
            }
        }
        cp_async_commit();
    };
    float4 xq[MT][4];
    const int quad = t < 2 ? 4 * t : 24 + 4 * t;
    const float* x_src[MT];
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
    for (int i = 0; i < STAGES; ++i) fetch(i);           // [constant], or behind the wait
    pdl_wait();
    if (b0 < b1) load_x(b0);
    int stage = 0, odd = 0;
    const int ranges = (blocks + range_blocks - 1) / range_blocks;
#pragma unroll 1
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x, odd ^= 1) {
        float* own = sums + (odd * RANGES + warp) * TILE;
        if (b0 < b1) {
            float sum[MT][4];
#pragma unroll 1
            for (int b = b0; b < b1; ++b) {
                cp_async_wait<STAGES - 1>();
                __syncwarp();
                float acc[MT][4];
                fr_multiply<MT>(acc, ring + stage * BLOCK, [&](int m, int j, uint2& c0, uint2& c1, uint2& c2) {
                    fs_split(xq[m][j].x, xq[m][j].y, c0.x, c1.x, c2.x);
                    fs_split(xq[m][j].z, xq[m][j].w, c0.y, c1.y, c2.y);
                });
                load_x(b + 1 < b1 ? b + 1 : b0);
                __syncwarp();                            // the stage has been read
                fetch(stage);
                stage = stage + 1 == STAGES ? 0 : stage + 1;
#pragma unroll
                for (int m = 0; m < MT; ++m)
#pragma unroll
                    for (int e = 0; e < 4; ++e) sum[m][e] = b == b0 ? acc[m][e] : __fadd_rn(sum[m][e], acc[m][e]);
            }
            float* dst = own + 2 * t * kFrPitch + g;
#pragma unroll
            for (int m = 0; m < MT; ++m)
#pragma unroll
                for (int e = 0; e < 4; ++e) dst[(8 * m + (e & 1)) * kFrPitch + 8 * (e >> 1)] = sum[m][e];
        }
        __syncthreads();
        for (int o = threadIdx.x; o < OUT; o += 32 * RANGES) {
            const int m = o / kFrFeatures, n = tile * kFrFeatures + o % kFrFeatures;
            if (m >= M || n >= N) continue;
            const float* src = sums + odd * RANGES * TILE + m * kFrPitch + o % kFrFeatures;
            float v = src[0];
            for (int r = 1; r < ranges; ++r) v = __fadd_rn(v, src[r * TILE]);
            if (!fs_finite(v)) v = fs_plain_sum(x + m * ldx, w + static_cast<long long>(n) * K, K);
            y[m * ldy + n] = bias ? __fadd_rn(v, bias[n]) : v;
        }
    }
}

template <int MT, int STAGES, int RANGES, int CTAS>
int fr_launch_stream(const FsArgs& a, int blocks, int range_blocks, cudaStream_t stream) {
    constexpr auto kernel = f32_rows_stream_kernel<MT, STAGES, RANGES, CTAS>;
    constexpr int smem = 4 * (RANGES * STAGES * kFrFeatures * kFsBK + 2 * RANGES * 8 * MT * kFrPitch);
    static_assert(CTAS * (smem + 1024) <= 228 * 1024, "the CTAs of an SM share its 228 KB");
    allow_smem<kernel>(smem);
    const int tiles = (a.N + kFrFeatures - 1) / kFrFeatures, ctas = (148 * CTAS + a.batch - 1) / a.batch;
    launch_pdl(kernel, dim3(tiles < ctas ? tiles : ctas, 1, a.batch), dim3(32 * RANGES), smem, stream, a.x, a.w, a.bias, a.y, a.M, a.N,
               a.K, blocks, range_blocks, tiles, a.ldx, a.ldy, a.bsx, a.bsw, a.bsy, a.w_constant);
    return launch_status();
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

// Which kernel.  A tile's ranges are the warps of a CTA of the stream, so it wants as many tiles as CTAs fill the chip, and where
// they fill it little more than once, so many an SM that one round takes them all (1 row, 5,120 x 5,120, 320 tiles: two an SM 24.0 us,
// three 20.9; 9,728 x 896, 608: four 9.6, five 8.0; more tiles: 152,064 x 3,584 306 and 321, 17,920 x 1,536 19.0 and 21.5).  With fewer
// tiles than SMs deeper stages (2,048 x 11,008, 128: two 27.4, four 19.2; 1,152 x 896, 72: two 3.8, six 3.2).  A cluster shares a tile's
// blocks out where that leaves each of its CTAs few of many (896 x 4,864, 56 tiles: 7.5 us and 8.5; 512 x 8,960 7.9 and 14.1; but 896 x 2,048
// 5.6 and 4.0, 896 x 8,960, 36 blocks a CTA, 15.1 and 14.4), and for 9 to 16 rows from fewer blocks on (960 x 3,584 8.8 and 10.0; 2,048 x
// 1,536 7.6 and 8.7).
template <int MT>
int fr_launch(const FsArgs& a, cudaStream_t stream) {
    const int blocks = (a.K + kFsBK - 1) / kFsBK, range_blocks = fs_range_blocks(blocks);
    const int ranges = (blocks + range_blocks - 1) / range_blocks;
    const long long tiles = static_cast<long long>((a.N + kFrFeatures - 1) / kFrFeatures) * a.batch;
    // at most 40 blocks a CTA of a cluster, five a warp, whose sums stand in shared memory; fewer while the chip has room for more CTAs
    // (896 x 4,864, 8 rows: 112 CTAs of a cluster of two 10.9 us, 224 of four 8.0)
    int cluster = 1;
    while (blocks > 40 * cluster || (blocks > 20 * cluster && cluster < 8 && 2 * cluster * tiles <= 148 * 2)) cluster *= 2;
    const int own = (ranges + cluster - 1) / cluster * range_blocks, most = own < blocks ? own : blocks;
    if (blocks >= 32) {                                  // (eight ranges)
        const bool shared = cluster * tiles <= 148 * 2 && (MT == 1 ? blocks >= 64 && (own <= 24 || cluster == 8) : blocks >= 48);
        if (!shared && tiles <= 148) return fr_launch_stream<MT, 4, 8, 1>(a, blocks, range_blocks, stream);
        if constexpr (MT == 1)
            if (tiles > 148 * 2 && tiles <= 148 * 3) return fr_launch_stream<MT, 2, 8, 3>(a, blocks, range_blocks, stream);
        if (!shared) return fr_launch_stream<MT, 2, 8, 2>(a, blocks, range_blocks, stream);
    } else {
        if constexpr (MT == 1) {
            if (tiles > 148 * 4 && tiles <= 148 * 5) return fr_launch_stream<MT, 2, 4, 5>(a, blocks, range_blocks, stream);
            if (tiles <= 148 * 2) return fr_launch_stream<MT, 6, 4, 2>(a, blocks, range_blocks, stream);
        }
        if (MT == 1 || tiles > 148 * 2) return fr_launch_stream<MT, 2, 4, 4>(a, blocks, range_blocks, stream);
    }
#define SOMI_FR(STAGES, IN_PLACE) \
    if (cluster > 1) return fr_launch_one<MT, STAGES, IN_PLACE, true>(a, cluster, blocks, range_blocks, own, stream); \
    if constexpr (MT == 2) return fr_launch_one<MT, STAGES, IN_PLACE, false>(a, 1, blocks, range_blocks, own, stream)
    if (most <= 2 * kFrWarps) { SOMI_FR(2, true); }
    else if (most <= 3 * kFrWarps) { SOMI_FR(3, true); }
    else { SOMI_FR(3, false); }
#undef SOMI_FR
    return SOMI_ERR_UNSUPPORTED;                          // (64 blocks and more are at least two CTAs')
}

int fs_launch_rows(const FsArgs& a, cudaStream_t stream) { return a.M <= 8 ? fr_launch<1>(a, stream) : fr_launch<2>(a, stream); }

}  // namespace somi
