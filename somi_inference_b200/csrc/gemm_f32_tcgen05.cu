// The float32 product of more than 16 rows in bfloat16 parts (gemm_f32_split.cuh) on `tcgen05.mma`.
//
// A CTA owns 128 rows of one operand by NB of the other.  Eight warps read blocks of 64 terms of both into registers (a
// block ahead), split them and write the parts as six swizzled tiles, two blocks deep; two threads issue the blocks'
// 24 MMA steps in turn, each into an accumulator of its own in tensor memory; eight warps read the accumulators and
// add them to their sums in registers (a thread has one row and half of the columns).
//
// What bounds it: shared memory. At 128 x 144 a block's MMAs read 206 KB of it and the split parts are 104 KB, 2,430 cycles at 128
// bytes; timelines show a block every 2,600 to 2,900 (splitting 2,100 to 2,500, MMAs 1,600 to 1,850, adding 500, side by
// side), 2,400 cycles in front of the first and 4,000 behind the last.  Twelve splitting and four adding warps were no
// faster (207 rows by 9,728 features 31.8 us, 64 rows 23.1).  Issuing the next block's loads one by one between the splits took 4,500 cycles a block, with
// every load behind all splits the loads' latency was added to them; so they go in two groups, a and b.
// In chains of products, FMA kernel before / now, us: 9,728 x 896, 17, 64, 207, 1,024 and 4,096 rows 22, 37, 115, 424, 1,623 /
// 17.7, 19.7, 30.0, 111, 398 (179 TFLOP/s of float32 products); 896 x 4,864 21, 39, 65, 255, 950 / 14.8, 15.0, 20.1, 72, 225;
// 1,152 x 896 7.9, 11.0, 17.7, 66, 230 / 7.7, 7.8, 11.4, 20.2, 50.
#include <cooperative_groups.h>

#include "gemm_f32_split.cuh"
#include "tcgen05.cuh"

namespace somi {

// Warps 0-7 split operands, 8-15 add up accumulators, 16 and 17 issue MMAs (two idle ones complete their group).
constexpr int kFtGroup = 256, kFtThreads = 2 * kFtGroup + 128;
// Registers: the launch gives 96 a thread, and the groups share them out.
constexpr int kFtSplitRegs = 104, kFtSumRegs = 104, kFtIssueRegs = 64;
static_assert(8 * kFtSplitRegs + 8 * kFtSumRegs + 4 * kFtIssueRegs == 20 * 96,
              "setmaxnreg waits for ever for registers that the launch did not take");
constexpr int kFtTile = 128 * kFsBK * 2;              // bytes of one part of the 128 rows

__device__ int g_gemm_f32_error = 0;

// Eight, sixteen or 24 columns of this thread's row as pairs, arrived.
__device__ __forceinline__ void ft_ld8(uint32_t taddr, uint64_t* v) {
    float r[8];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n"
                 "tcgen05.wait::ld.sync.aligned;\n"
                 : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3]), "=f"(r[4]), "=f"(r[5]), "=f"(r[6]), "=f"(r[7])
                 : "r"(taddr)
                 : "memory");
#pragma unroll
    for (int e = 0; e < 4; ++e) v[e] = pair_f32(r[2 * e], r[2 * e + 1]);
}
__device__ __forceinline__ void ft_ld16(uint32_t taddr, uint64_t* v) {
    float r[16];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
                 "tcgen05.wait::ld.sync.aligned;\n"
                 : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3]), "=f"(r[4]), "=f"(r[5]), "=f"(r[6]), "=f"(r[7]),
                   "=f"(r[8]), "=f"(r[9]), "=f"(r[10]), "=f"(r[11]), "=f"(r[12]), "=f"(r[13]), "=f"(r[14]), "=f"(r[15])
                 : "r"(taddr)
                 : "memory");
#pragma unroll
    for (int e = 0; e < 8; ++e) v[e] = pair_f32(r[2 * e], r[2 * e + 1]);
}
__device__ __forceinline__ void ft_ld24(uint32_t taddr, uint64_t* v) {
    float r[24];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%24];\n"
                 "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%16,%17,%18,%19,%20,%21,%22,%23}, [%25];\n"
                 "tcgen05.wait::ld.sync.aligned;\n"
                 : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3]), "=f"(r[4]), "=f"(r[5]), "=f"(r[6]), "=f"(r[7]),
                   "=f"(r[8]), "=f"(r[9]), "=f"(r[10]), "=f"(r[11]), "=f"(r[12]), "=f"(r[13]), "=f"(r[14]), "=f"(r[15]),
                   "=f"(r[16]), "=f"(r[17]), "=f"(r[18]), "=f"(r[19]), "=f"(r[20]), "=f"(r[21]), "=f"(r[22]), "=f"(r[23])
                 : "r"(taddr), "r"(taddr + 16)
                 : "memory");
#pragma unroll
    for (int e = 0; e < 12; ++e) v[e] = pair_f32(r[2 * e], r[2 * e + 1]);
}
// acc += columns taddr .. of the thread's row.
template <int COLS, int C = 0, int SIZE>
__device__ __forceinline__ void ft_add(uint32_t taddr, uint64_t (&acc2)[SIZE]) {
    if constexpr (C < COLS) {
        constexpr int N = COLS - C < 24 ? COLS - C : 24;
        static_assert(N % 8 == 0 && 2 * SIZE >= COLS, "a load of 8, 16 or 24 columns");
        uint64_t v[12];
        if constexpr (N == 24) ft_ld24(taddr + C, v);
        else if constexpr (N == 16) ft_ld16(taddr + C, v);
        else ft_ld8(taddr + C, v);
#pragma unroll
        for (int e = 0; e < N / 2; ++e) acc2[C / 2 + e] = add_f32x2(acc2[C / 2 + e], v[e]);
        ft_add<COLS, C + 24>(taddr, acc2);
    }
}
__device__ __forceinline__ void ft_st8(uint32_t taddr, const uint64_t* v) {
    float r[8];
#pragma unroll
    for (int e = 0; e < 4; ++e) unpair_f32(v[e], r[2 * e], r[2 * e + 1]);
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};\n" ::"r"(taddr),
                 "f"(r[0]), "f"(r[1]), "f"(r[2]), "f"(r[3]), "f"(r[4]), "f"(r[5]), "f"(r[6]), "f"(r[7])
                 : "memory");
}

template <int NB>
constexpr int ft_smem() { return 2 * 3 * (kFtTile + NB * kFsBK * 2) + 1024; }
template <int NB>
__host__ __device__ constexpr int ft_columns() { return 3 * NB <= 128 ? 128 : (3 * NB <= 256 ? 256 : 512); }

// The 128 rows are features and the NB columns tokens, or (TOKENS) the other way round.  A cluster of
// `cluster_size` CTAs shares a tile's ranges, `own_ranges` (one or two) each; else the CTA walks through all of them.
template <int NB, bool TOKENS>
__global__ void __launch_bounds__(kFtThreads, 1)
f32_tiles_kernel(const float* __restrict__ x, const float* __restrict__ w, const float* __restrict__ bias,
                 float* __restrict__ y, int M, int N, int K, int blocks, int range_blocks, int cluster_size, int own_ranges,
                 long long ldx, long long ldy, long long bsx, long long bsw, long long bsy, int w_constant) {
    constexpr int PLANE_B = NB * kFsBK * 2, STAGE = 3 * (kFtTile + PLANE_B);
    constexpr int LB = (NB + 31) / 32, HALF = NB / 2;    // rows of the NB side a thread loads; columns it sums
    extern __shared__ unsigned char ft_raw[];
    unsigned char* stages = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(ft_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    __shared__ __align__(8) unsigned long long full_bar[2], done_bar[2], free_bar[2];
    __shared__ uint32_t tmem_s;
    __shared__ int failed_s;
    pdl_launch_dependents();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid == 0) {
        for (int s = 0; s < 2; ++s) {
            mbar_init(smem_u32(&full_bar[s]), kFtGroup / 32);
            mbar_init(smem_u32(&done_bar[s]), 1);
            mbar_init(smem_u32(&free_bar[s]), kFtGroup / 32);
        }
        mbar_fence_init();
        failed_s = 0;
    }
    if (warp == 16) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&tmem_s)),
                     "r"(ft_columns<NB>())
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    t5::fence_before();
    __syncthreads();
    t5::fence_after();
    const uint32_t tmem = tmem_s;
    x += blockIdx.z * bsx;
    w += blockIdx.z * bsw;
    y += blockIdx.z * bsy;
    const int rank = blockIdx.x % cluster_size;
    const int n0 = blockIdx.x / cluster_size * (TOKENS ? NB : 128), m0 = blockIdx.y * (TOKENS ? 128 : NB);
    const int b0 = cluster_size > 1 ? min(blocks, rank * own_ranges * range_blocks) : 0;
    const int n_blocks = (cluster_size > 1 ? min(blocks, b0 + own_ranges * range_blocks) : blocks) - b0;
    namespace cg = cooperative_groups;
    const cg::cluster_group cluster = cg::this_cluster();

    if (warp >= 16) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;\n" ::"n"(kFtIssueRegs));
        pdl_wait();
        if (warp < 18 && lane == 0) {
            // ---- two issuing threads take the blocks in turn, each with a stage and an accumulator of its own, so that
            // one's tests of barriers run under the other's MMAs
            constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(NB >> 3) << 17) | (8u << 24);
            const int s = warp - 16;
            const uint32_t d = tmem + s * NB, a = smem_u32(stages) + s * STAGE, c = a + 3 * kFtTile;
            const uint64_t a_desc = t5::desc_kmajor(a), c_desc = t5::desc_kmajor(c);
#pragma unroll 1
            for (int i = s; i < n_blocks; i += 2) {
                if (!mbar_wait(smem_u32(&full_bar[s]), i >> 1 & 1, 2000000) ||
                    (i > 1 && !mbar_wait(smem_u32(&free_bar[s]), (i >> 1 & 1) ^ 1, 2000000))) {
                    failed_s = 1;
                    break;
                }
                t5::fence_after();
                auto step = [&](int px, int pw, int j, uint32_t accumulate) {
                    const int pa = TOKENS ? px : pw, pc = TOKENS ? pw : px;
                    t5::mma_ss(d, a_desc + ((pa * kFtTile + j * 32) >> 4), c_desc + ((pc * PLANE_B + j * 32) >> 4), idesc, accumulate);
                };
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    step(2, 0, j, j > 0);
                    step(0, 2, j, 1);
                    step(1, 1, j, 1);
                    step(1, 0, j, 1);
                    step(0, 1, j, 1);
                }
#pragma unroll
                for (int j = 0; j < 4; ++j) step(0, 0, j, 1);
                t5::commit(smem_u32(&done_bar[s]));
            }
        }
        __syncwarp();
        if (cluster_size > 1) {                          // (the two meetings of the summing warps are everyone's)
            cluster.sync();
            cluster.sync();
        }
    } else if (warp < 8) {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;\n" ::"n"(kFtSplitRegs));
        // ---- splits terms 4 c8 .. and 32 + 4 c8 .. of rows r, r + 32, .. (rows behind the last one repeat it: what they
        // give is not stored)
        constexpr int PASSES = 4 + LB;
        const int r = tid >> 3, c8 = tid & 7;
        const float* a_src = (TOKENS ? x + m0 * ldx : w + static_cast<long long>(n0) * K) + 4 * c8;
        const float* b_src = (TOKENS ? w + static_cast<long long>(n0) * K : x + m0 * ldx) + 4 * c8;
        const int a_ld = static_cast<int>(TOKENS ? ldx : K), b_ld = static_cast<int>(TOKENS ? K : ldx);
        const int a_last = (TOKENS ? M - m0 : N - n0) - 1, b_last = (TOKENS ? N - n0 : M - m0) - 1;
        int off[PASSES];
#pragma unroll
        for (int i = 0; i < PASSES; ++i)
            off[i] = i < 4 ? min(r + 32 * i, a_last) * a_ld : min(r + 32 * (i - 4), b_last) * b_ld;
        float4 q[PASSES][2];
        auto load = [&](int from, int to, int b) {
            if ((b + 1) * kFsBK <= K) {
#pragma unroll
                for (int i = 0; i < PASSES; ++i)
                    if (i >= from && i < to) {
                        const float* p = (i < 4 ? a_src : b_src) + off[i] + b * kFsBK;
                        q[i][0] = *reinterpret_cast<const float4*>(p);
                        q[i][1] = *reinterpret_cast<const float4*>(p + 32);
                    }
            } else {
                const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                for (int i = 0; i < PASSES; ++i)
                    if (i >= from && i < to) {
                        const float* p = (i < 4 ? a_src : b_src) + off[i] + b * kFsBK;
                        q[i][0] = b * kFsBK + 4 * c8 < K ? *reinterpret_cast<const float4*>(p) : zero;
                        q[i][1] = b * kFsBK + 32 + 4 * c8 < K ? *reinterpret_cast<const float4*>(p + 32) : zero;
                    }
            }
        };
        if (!w_constant) pdl_wait();
        load(TOKENS ? 4 : 0, TOKENS ? PASSES : 4, b0);          // w: [constant], or behind the wait
        pdl_wait();
        load(TOKENS ? 0 : 4, TOKENS ? 4 : PASSES, b0);
        bool ok = true;
#pragma unroll 1
        for (int i = 0; i < n_blocks; ++i) {
            if (ok && i > 1 && !mbar_wait(smem_u32(&done_bar[i & 1]), (i >> 1 & 1) ^ 1, 2000000)) { ok = false; failed_s = 1; }
            unsigned char* st = stages + (i & 1) * STAGE + r * 128 + ((c8 ^ (r & 7)) << 4);
            auto put = [&](int from, int to) {
#pragma unroll
                for (int p = 0; p < PASSES; ++p) {
                    if (p < from || p >= to) continue;
                    uint4 part[3];
                    fs_split(q[p][0].x, q[p][0].y, part[0].x, part[1].x, part[2].x);
                    fs_split(q[p][0].z, q[p][0].w, part[0].y, part[1].y, part[2].y);
                    fs_split(q[p][1].x, q[p][1].y, part[0].z, part[1].z, part[2].z);
                    fs_split(q[p][1].z, q[p][1].w, part[0].w, part[1].w, part[2].w);
                    if (NB % 32 != 0 && p == PASSES - 1 && r + 32 * (LB - 1) >= NB) continue;
                    unsigned char* dst = st + (p < 4 ? p * 32 * 128 : 3 * kFtTile + (p - 4) * 32 * 128);
#pragma unroll
                    for (int e = 0; e < 3; ++e) *reinterpret_cast<uint4*>(dst + e * (p < 4 ? kFtTile : PLANE_B)) = part[e];
                }
            };
            // (the next block's loads go into registers as they become free)
            put(0, 4);
            if (i + 1 < n_blocks) load(0, 4, b0 + i + 1);
            put(4, PASSES);
            if (i + 1 < n_blocks) load(4, PASSES, b0 + i + 1);
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&full_bar[i & 1]));
        }
        __syncwarp();
        if (cluster_size > 1) {
            cluster.sync();
            cluster.sync();
        }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;\n" ::"n"(kFtSumRegs));
        // ---- row 32 (warp % 4) + lane of the tile, one half of its columns
        pdl_wait();
        uint64_t acc2[HALF / 2];
#pragma unroll
        for (int c = 0; c < HALF / 2; ++c) acc2[c] = 0ull;
        bool ok = true;
        const int half = warp >> 2 & 1;
        const uint32_t own = tmem + (static_cast<uint32_t>(warp & 3) << 21) + half * HALF;
        int left = range_blocks, closed = 0;
#pragma unroll 1
        for (int i = 0; i < n_blocks; ++i) {
            const int s = i & 1;
            if (ok && !mbar_wait(smem_u32(&done_bar[s]), i >> 1 & 1, 2000000)) { ok = false; failed_s = 1; }
            __syncwarp();                                // (the loads below are the whole warp's)
            t5::fence_after();
            ft_add<HALF>(own + s * NB, acc2);
            t5::fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&free_bar[s]));
            if (--left == 0 || i + 1 == n_blocks) {      // the range is complete: onto the sum of those before (or beside it)
                const bool last = i + 1 == n_blocks;
                if (closed > 0 && cluster_size == 1) ft_add<HALF>(own + 2 * NB, acc2);
                if (!last) {
#pragma unroll
                    for (int c = 0; c < HALF; c += 8) {
                        ft_st8(own + 2 * NB + c, acc2 + c / 2);
#pragma unroll
                        for (int e = 0; e < 4; ++e) acc2[c / 2 + e] = 0ull;
                    }
                    t5::wait_st();
                }
                ++closed;
                left = range_blocks;
            }
        }
        float acc[HALF];
#pragma unroll
        for (int c = 0; c < HALF; c += 2) unpair_f32(acc2[c / 2], acc[c], acc[c + 1]);

        const int row = (warp & 3) * 32 + lane, col0 = half * HALF;
        if (cluster_size > 1) {                          // (the last MMA has read the stages)
            float* tile = reinterpret_cast<float*>(stages);
            if (closed > 1) {
#pragma unroll
                for (int c = 0; c < HALF; c += 8) {
                    uint64_t v[4];
                    ft_ld8(own + 2 * NB + c, v);
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        unpair_f32(v[e], tile[(col0 + c + 2 * e) * 128 + row], tile[(col0 + c + 2 * e + 1) * 128 + row]);
                }
                tile += NB * 128;
            }
#pragma unroll
            for (int c = 0; c < HALF; ++c) tile[(col0 + c) * 128 + row] = acc[c];
            // the ranges' tiles [column][128 rows], one or two in a CTA's shared memory: every CTA adds up a share of the
            // elements in the order of the ranges
            cluster.sync();
            const int ranges = (blocks + range_blocks - 1) / range_blocks;
            const int step = cluster_size * kFtGroup;
            for (int i0 = rank * kFtGroup + tid - kFtGroup; i0 < NB * 32; i0 += 2 * step) {
                float4 part[2][8];                       // two elements' loads in flight
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const int i = i0 + u * step;
                    if (i >= NB * 32 || m0 + (i >> 5) >= M || n0 + (i & 31) * 4 >= N) continue;
                    const float4* mine = reinterpret_cast<const float4*>(stages) + i;
#pragma unroll
                    for (int k = 0; k < 8; ++k)
                        if (k < ranges)
                            part[u][k] = own_ranges == 1 ? *cluster.map_shared_rank(mine, k)
                                                         : *cluster.map_shared_rank(mine + k % 2 * NB * 32, k / 2);
                }
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const int i = i0 + u * step, m = m0 + (i >> 5), n = n0 + (i & 31) * 4;       // a column, four of its rows
                    if (i >= NB * 32 || m >= M || n >= N) continue;
                    float v[4] = {part[u][0].x, part[u][0].y, part[u][0].z, part[u][0].w};
#pragma unroll
                    for (int k = 1; k < 8; ++k)
                        if (k < ranges) {
                            v[0] = __fadd_rn(v[0], part[u][k].x);
                            v[1] = __fadd_rn(v[1], part[u][k].y);
                            v[2] = __fadd_rn(v[2], part[u][k].z);
                            v[3] = __fadd_rn(v[3], part[u][k].w);
                        }
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        if (n + e < N) {
                            if (!fs_finite(v[e])) v[e] = fs_plain_sum(x + m * ldx, w + static_cast<long long>(n + e) * K, K);
                            y[m * ldy + n + e] = bias ? __fadd_rn(v[e], bias[n + e]) : v[e];
                        }
                }
            }
            // no CTA leaves while its tile is read: the stores above have taken what was read, and nobody waits for them here
            __syncwarp();
            asm volatile("barrier.cluster.arrive.relaxed.aligned;\nbarrier.cluster.wait.aligned;\n" ::: "memory");
        } else if (ok && !TOKENS) {
            const int n = n0 + row, count = n < N ? min(HALF, M - m0 - col0) : 0;
            float* dst = y + (m0 + col0) * ldy + n;
            const float b = bias != nullptr && n < N ? bias[n] : 0.f;
            bool fine = true;
#pragma unroll
            for (int c = 0; c < HALF; ++c)
                if (c < count) {
                    fine &= fs_finite(acc[c]);
                    dst[c * ldy] = bias ? __fadd_rn(acc[c], b) : acc[c];
                }
            if (!fine)
                for (int c = 0; c < count; ++c)
                    if (!fs_finite(dst[c * ldy])) {
                        const float v = fs_plain_sum(x + (m0 + col0 + c) * ldx, w + static_cast<long long>(n) * K, K);
                        dst[c * ldy] = bias ? __fadd_rn(v, b) : v;
                    }
        } else if (ok) {
            // a thread's row is a token's: through shared memory (the last MMA has read the stages), so that a
            // warp stores whole rows (a store of 16 bytes a row and lane took 6 us a tile)
            constexpr int PITCH = HALF + 4;
            float* own_rows = reinterpret_cast<float*>(stages) + (warp - 8) * 32 * PITCH;
#pragma unroll
            for (int c = 0; c < HALF; c += 4)
                *reinterpret_cast<float4*>(own_rows + lane * PITCH + c) = make_float4(acc[c], acc[c + 1], acc[c + 2], acc[c + 3]);
            __syncwarp();
            const bool wide = ((ldy | bsy) & 3) == 0 && (reinterpret_cast<uintptr_t>(y) & 15) == 0;
            bool fine = true;
#pragma unroll
            for (int c = 0; c < HALF; ++c) fine &= fs_finite(acc[c]);
            // (uniform: whole quads of finite numbers, or element by element)
            const int live = M - m0 - (warp & 3) * 32, cols = N - n0 - col0;
            if (wide && (N & 3) == 0 && __all_sync(0xffffffffu, fine)) {
                float* dst = y + (m0 + (warp & 3) * 32) * ldy + n0 + col0;
                constexpr int ACROSS = HALF / 4;
#pragma unroll 6
                for (int k = 0; k < ACROSS; ++k) {
                    const int i = k * 32 + lane, rr = i / ACROSS, c = i % ACROSS * 4;
                    if (rr >= live || c >= cols) continue;
                    float4 v = *reinterpret_cast<const float4*>(own_rows + rr * PITCH + c);
                    if (bias != nullptr) {
                        const float* b = bias + n0 + col0 + c;
                        v = make_float4(__fadd_rn(v.x, b[0]), __fadd_rn(v.y, b[1]), __fadd_rn(v.z, b[2]), __fadd_rn(v.w, b[3]));
                    }
                    *reinterpret_cast<float4*>(dst + rr * ldy + c) = v;
                }
            } else {
#pragma unroll 1
                for (int i = lane; i < 32 * HALF; i += 32) {
                    const int m = m0 + (warp & 3) * 32 + i / HALF, n = n0 + col0 + i % HALF;
                    if (i / HALF >= live || n >= N) continue;
                    float v = own_rows[i / HALF * PITCH + i % HALF];
                    if (!fs_finite(v)) v = fs_plain_sum(x + m * ldx, w + static_cast<long long>(n) * K, K);
                    y[m * ldy + n] = bias ? __fadd_rn(v, bias[n]) : v;
                }
            }
        }
    }
    t5::fence_before();
    __syncthreads();
    if (warp == 16)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(ft_columns<NB>()) : "memory");
    if (tid == 0 && failed_s) atomicExch(&g_gemm_f32_error, 1);
}

// A form of the launch and what it is expected to take, in cycles: waves of CTAs times (24 MMA steps a block and a fixed part; the
// tensor pipe takes 51 cycles for a step of up to 64 columns and one for two columns from there on).  It need not be exact, only
// tell a nearly empty last wave: 207 rows by 9,728 features are 152 tiles of 128 features by 112 rows, two waves, or 136 of
// 144 features by 128 rows, one wave (41 and 31 us).
// With eight ranges a CTA may take two: 32 rows by 4,096 x 2,048 are three waves of clusters of eight or one of clusters of four (26.4 and
// 13.9 us; FMAs 20.0), 203 by 2,048 x 11,008 108 and 68; one a CTA stays ahead where it saves no wave (48 by 5,120 x 2,048 28.4 and 30.0).
struct FtForm {
    int nb, tokens, cluster, own;
    long long cost;
};

template <int NB, bool TOKENS>
int ft_launch_one(const FsArgs& a, int cluster, int own, int blocks, int range_blocks, cudaStream_t stream) {
    constexpr auto kernel = f32_tiles_kernel<NB, TOKENS>;
    allow_smem<kernel>(ft_smem<NB>());
    constexpr int TN = TOKENS ? NB : 128, TM = TOKENS ? 128 : NB;
    for (int m = 0; m < a.M;) {                          // (a grid has at most 65,535 tiles of rows)
        const int rows = a.M - m < 65535 * TM ? a.M - m : 65535 * TM;
        launch_pdl_cluster(kernel, dim3((a.N + TN - 1) / TN * cluster, (rows + TM - 1) / TM, a.batch), dim3(kFtThreads),
                           ft_smem<NB>(), cluster, stream, a.x + m * a.ldx, a.w, a.bias, a.y + m * a.ldy, rows, a.N, a.K,
                           blocks, range_blocks, cluster, own, a.ldx, a.ldy, a.bsx, a.bsw, a.bsy, a.w_constant);
        m += rows;
    }
    return launch_status();
}

int fs_launch_tiles(const FsArgs& a, cudaStream_t stream) {
    const int blocks = (a.K + kFsBK - 1) / kFsBK, range_blocks = fs_range_blocks(blocks);
    const int ranges = (blocks + range_blocks - 1) / range_blocks;
    FtForm best{0, 0, 0, 0, 0};
    auto consider = [&](int nb, int tokens, int own) {   // (own: ranges of a CTA, 0 for all)
        const int cluster = own == 0 ? 1 : (ranges + own - 1) / own;
        const long long tiles = static_cast<long long>(tokens ? (a.N + nb - 1) / nb : (a.N + 127) / 128) *
                                (tokens ? (a.M + 127) / 128 : (a.M + nb - 1) / nb) * a.batch;
        const int step = nb / 2 > 51 ? nb / 2 : 51;
        // (clusters of seven or eight leave a few SMs of every GPC idle)
        const int slots = cluster == 1 ? 148 : (cluster <= 4 ? 132 : 112) / cluster;
        const long long waves = (tiles + slots - 1) / slots;
        const long long cost = waves * (24ll * step * (cluster == 1 ? blocks : own * range_blocks) + (cluster == 1 ? 4000 : 4000 + 2000 * own));
        if (best.nb == 0 || cost < best.cost) best = FtForm{nb, tokens, cluster, own, cost};
    };
    constexpr int kTokenTiles[] = {32, 64, 96, 112, 128}, kFeatureTiles[] = {96, 112, 128, 144};
    for (int nb : kTokenTiles) {
        consider(nb, 0, 0);
        if (ranges > 1) consider(nb, 0, 1);
        if (ranges > 4) consider(nb, 0, 2);
    }
    for (int nb : kFeatureTiles) consider(nb, 1, 0);
#define SOMI_FT(NB, T) \
    if (best.nb == NB && best.tokens == T) return ft_launch_one<NB, T>(a, best.cluster, best.own, blocks, range_blocks, stream)
    SOMI_FT(32, 0);
    SOMI_FT(64, 0);
    SOMI_FT(96, 0);
    SOMI_FT(112, 0);
    SOMI_FT(128, 0);
    SOMI_FT(96, 1);
    SOMI_FT(112, 1);
    SOMI_FT(128, 1);
    SOMI_FT(144, 1);
#undef SOMI_FT
    return SOMI_ERR_UNSUPPORTED;
}

}  // namespace somi

using namespace somi;

SOMI_API int somi_gemm_f32_error() {
    int v = 0, zero = 0;
    if (cudaMemcpyFromSymbol(&v, g_gemm_f32_error, sizeof(int)) != cudaSuccess) return -1;
    if (v) cudaMemcpyToSymbol(g_gemm_f32_error, &zero, sizeof(int));
    return v;
}
