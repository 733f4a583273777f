// The float32 path's matrix product: y[M, N] = x[M, K] w[N, K]^T (+ bias[N]).  From 512 terms on, where rows can be
// read 16 bytes at a time, the product goes to tensor cores in exact bfloat16 parts (gemm_f32_split.cuh, gemm_f32_rows.cu,
// gemm_f32_tcgen05.cu); this file takes the others, every product and sum a float32 FMA on the CUDA cores.
// Neither uses a reduced-precision mode of any kind.
//
// The reference's engine uses the library product here (nn.Linear,
// somi_inference/models/qwen2.py:221-222,268-271).  This engine does not, for two reasons.  The
// float32 path exists to show faults that bfloat16 hides, so its arithmetic must be beyond doubt:
// on the software stack this engine was developed on (cuBLAS 12.8, B200) the library's float32
// product with TF32 switched off returned, in some processes, pairs of wrong output columns for
// products of a few rows (16 x 320 x 192 and the like).  And an output element here is summed in
// an order that K alone fixes: the same token gives the same bits in a step of one token and in a
// step of a thousand, which the library does not promise.
//
// The order: K is cut into 1, 2, 4 or 8 ranges (`sg_ranges`); inside a range the even and the odd
// terms are two chains of FMAs in ascending order (one `fma.rn.f32x2` advances both), whose sum is
// the range's; the ranges are added in ascending order, the bias last.  So a step whose outputs are
// too few to fill the chip gives every range a CTA of its own (a thread-block cluster; the ranges'
// tiles are added over distributed shared memory), a step with enough tiles lets one CTA walk
// through all ranges, and both give the same bits.
//
// What bounds it: a few rows stream the weights, so the tile is 64 weight rows by the rows rounded up
// to 2, 4, 8, 16 or 32, with four 32-deep stages of cp.async in flight per CTA and the first ones
// issued before the dependency wait (a model's weights are constants).  More rows are bound by shared memory and the FMA
// pipe in turn: a 64 x 64 tile, 8 x 4 outputs a thread, operands read from shared memory four k at a time as one
// 16-byte access (rows 36 floats apart, so eight neighbouring rows lie in different banks).  Up to 384 rows
// a 32-row tile, of which there are twice as many, is the faster.  Measured with 896 terms, when those came here too:
// 32 / 64 rows a tile, 9,728 x 896, 257, 384 and 448 rows 144.3 / 156.4, 185.8 / 188.4, 212.5 / 217.7 us, 512 rows
// 239.9 / 229.6; 1,024 rows 425 us (42 TFLOP/s; the tensor cores take 113).
#include <cooperative_groups.h>

#include "gemm_f32_split.cuh"

namespace somi {

constexpr int kSgBK = 32;             // k per stage
constexpr int kSgPitch = kSgBK + 4;   // floats between rows of a stage
constexpr int kSgBN = 64;
constexpr int kSgStages = 4;

// Tiles from which on one CTA walks through all ranges.  Tiles of few rows stream weights, and two an SM
// are enough to do so; taller ones need the FMA pipe filled to the end of the last wave: 9,728 x 896 at 64
// rows takes 60 us with 304 walking CTAs and 38 us with four times as many short ones.
constexpr long long sg_fill_tiles(int rows) { return rows < 32 ? 148 * 2 : 148 * 8; }

// Into how many ranges K is cut: a function of K alone (see above), for ranges of at least 64 terms
// and of about 224 to 608 at the model sizes this path runs.
inline int sg_ranges(int K) { return K >= 2048 ? 8 : (K >= 512 ? 4 : (K >= 128 ? 2 : 1)); }
inline int sg_range_length(int K, int ranges) {
    return (K + ranges * kSgBK - 1) / (ranges * kSgBK) * kSgBK;
}

__device__ __forceinline__ void sg_fma2(unsigned long long& d, unsigned long long a, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
__device__ __forceinline__ float sg_sum2(unsigned long long d) {
    float lo, hi;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(d));
    return __fadd_rn(lo, hi);
}
template <int BYTES>
__device__ __forceinline__ void sg_copy(uint32_t dst, const float* src, bool in) {
    // (a source size of 0 writes zeros and reads nothing)
    if (BYTES == 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(in ? 16 : 0) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(dst), "l"(src), "r"(in ? 4 : 0) : "memory");
}

// What a thread copies of rows [row0, row0 + ROWS) of a matrix, 32 columns at a time: the same
// columns of every row it visits, so a stage costs it one pointer addition a copy.
template <int ROWS, int THREADS, bool VEC>
struct SgLoader {
    static constexpr int PER = VEC ? 4 : 1, ACROSS = kSgBK / PER;      // copies a row
    static constexpr int APART = THREADS / ACROSS;                     // rows between a thread's copies
    static constexpr int COPIES = (ROWS + APART - 1) / APART;
    static_assert(THREADS % ACROSS == 0 && COPIES <= 32, "a thread stays in its columns");
    const float* src;
    const float* safe;
    long long step;
    uint32_t dst, live;
    int k;

    __device__ __forceinline__ SgLoader(float* stage, const float* m, long long ld, int row0, int n_rows, int k0) {
        const int r = threadIdx.x / ACROSS;
        k = k0 + threadIdx.x % ACROSS * PER;
        safe = m;
        src = m + static_cast<long long>(row0 + r) * ld + k;
        step = ld * APART;
        dst = static_cast<uint32_t>(__cvta_generic_to_shared(stage + r * kSgPitch + threadIdx.x % ACROSS * PER));
        live = 0;
#pragma unroll
        for (int c = 0; c < COPIES; ++c)
            if (r + c * APART < ROWS && row0 + r + c * APART < n_rows) live |= 1u << c;
    }
    // columns k0 + 32 s .. of the range that ends at k_end, into the stage `at` bytes further on
    __device__ __forceinline__ void copy(int s, int k_end, uint32_t at) const {
        const float* p = src + s * kSgBK;
        const uint32_t mask = k + s * kSgBK < k_end ? live : 0u;
#pragma unroll
        for (int c = 0; c < COPIES; ++c) {
            const bool in = (mask >> c) & 1u;
            if (ROWS % APART == 0 || threadIdx.x / ACROSS + c * APART < ROWS)
                sg_copy<4 * PER>(dst + at + c * APART * kSgPitch * 4, in ? p : safe, in);
            p += step;
        }
    }
};

template <int BM, int TM, int TN>
__host__ __device__ constexpr int sg_threads() { return (BM / TM) * (kSgBN / TN); }
template <int BM>
constexpr int sg_smem() { return kSgStages * (BM + kSgBN) * kSgPitch * 4; }

// CLUSTER: the CTA computes one range, blockIdx.x % ranges; else all of them.
template <int BM, int TM, int TN, bool VEC, bool CLUSTER>
__global__ void __launch_bounds__(sg_threads<BM, TM, TN>())
sgemm_nt_kernel(const float* __restrict__ x, const float* __restrict__ w, const float* __restrict__ bias,
                float* __restrict__ y, int M, int N, int K, int ranges, int range_length, long long ldx,
                long long ldy, long long bsx, long long bsw, long long bsy, int w_constant) {
    constexpr int THREADS = sg_threads<BM, TM, TN>();
    constexpr int ROWS_APART = BM / TM, COLS_APART = kSgBN / TN;
    extern __shared__ __align__(16) float sg_buf[];      // [stage][x rows | w rows][pitch]
    constexpr int STAGE = (BM + kSgBN) * kSgPitch;
    pdl_launch_dependents();
    // blockIdx.z is the product's index in a batch: operands of product b start b * bs{x,w,y}
    // elements further on; rows of x and y lie ldx and ldy elements apart (w's rows K)
    x += blockIdx.z * bsx;
    w += blockIdx.z * bsw;
    y += blockIdx.z * bsy;
    const int n0 = (CLUSTER ? blockIdx.x / ranges : blockIdx.x) * kSgBN, m0 = blockIdx.y * BM;
    const int first = CLUSTER ? blockIdx.x % ranges : 0;
    const int k_begin = min(K, first * range_length);
    const int k_end = CLUSTER ? min(K, k_begin + range_length) : K;
    const int steps = (k_end - k_begin + kSgBK - 1) / kSgBK;
    // a warp's lanes share as few rows of either operand as they can: 4 x 8 outputs apart
    constexpr bool SQUARE = ROWS_APART % 4 == 0;
    constexpr int WARP_COLS = COLS_APART / 8;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int tr = SQUARE ? warp / WARP_COLS * 4 + lane / 8 : threadIdx.x / COLS_APART;
    const int tc = SQUARE ? warp % WARP_COLS * 8 + lane % 8 : threadIdx.x % COLS_APART;

    const SgLoader<kSgBN, THREADS, VEC> w_rows(sg_buf + BM * kSgPitch, w, K, n0, N, k_begin);
    const SgLoader<BM, THREADS, VEC> x_rows(sg_buf, x, ldx, m0, M, k_begin);
    auto load_w = [&](int s) { w_rows.copy(s, k_end, s % kSgStages * (STAGE * 4)); };
    auto load_x = [&](int s) { x_rows.copy(s, k_end, s % kSgStages * (STAGE * 4)); };
    if (!w_constant) pdl_wait();
#pragma unroll
    for (int s = 0; s < kSgStages - 1; ++s)
        if (s < steps) load_w(s);                        // [constant], or behind the wait
    pdl_wait();
#pragma unroll
    for (int s = 0; s < kSgStages - 1; ++s) {
        if (s < steps) load_x(s);
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    }
    unsigned long long acc[TM][TN];
    float total[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) { acc[i][j] = 0ull; total[i][j] = 0.f; }
    const int steps_per_range = range_length / kSgBK;
    int left = steps_per_range;
    bool started = false;
    auto close_range = [&]() {
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TN; ++j) {
                const float r = sg_sum2(acc[i][j]);
                total[i][j] = started ? __fadd_rn(total[i][j], r) : r;
                acc[i][j] = 0ull;
            }
        started = true;
    };
    for (int s = 0; s < steps; ++s) {
        asm volatile("cp.async.wait_group %0;\n" ::"n"(kSgStages - 2) : "memory");
        __syncthreads();                                 // stage s is here; stage s - 1 has been read
        if (s + kSgStages - 1 < steps) {
            load_w(s + kSgStages - 1);
            load_x(s + kSgStages - 1);
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
        const float* xs = sg_buf + (s % kSgStages) * STAGE + tr * kSgPitch;
        const float* ws = sg_buf + (s % kSgStages) * STAGE + (BM + tc) * kSgPitch;
#pragma unroll(TM * TN >= 32 ? 4 : 8)
        for (int k = 0; k < kSgBK; k += 4) {
            ulonglong2 b[TN];
#pragma unroll
            for (int j = 0; j < TN; ++j)
                b[j] = *reinterpret_cast<const ulonglong2*>(ws + j * COLS_APART * kSgPitch + k);
#pragma unroll
            for (int i = 0; i < TM; ++i) {
                const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(xs + i * ROWS_APART * kSgPitch + k);
#pragma unroll
                for (int j = 0; j < TN; ++j) sg_fma2(acc[i][j], a.x, b[j].x);
#pragma unroll
                for (int j = 0; j < TN; ++j) sg_fma2(acc[i][j], a.y, b[j].y);
            }
        }
        if (!CLUSTER && --left == 0) {
            close_range();
            left = steps_per_range;
        }
    }
    if (CLUSTER || left != steps_per_range) close_range();
    if (!CLUSTER) {
#pragma unroll
        for (int i = 0; i < TM; ++i) {
            const int gm = m0 + tr + i * ROWS_APART;
            if (gm >= M) continue;
#pragma unroll
            for (int j = 0; j < TN; ++j) {
                const int gn = n0 + tc + j * COLS_APART;
                if (gn < N) y[gm * ldy + gn] = bias ? __fadd_rn(total[i][j], bias[gn]) : total[i][j];
            }
        }
        return;
    }
    // the ranges' tiles, each in its CTA's shared memory; every CTA of the cluster adds up a share of
    // the elements in the order of the ranges (no K leaves one empty)
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    __syncthreads();                                     // the stages are free
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j)
            sg_buf[(tr + i * ROWS_APART) * kSgBN + tc + j * COLS_APART] = total[i][j];
    cluster.sync();
    constexpr int QUADS = BM * kSgBN / 4;
    const bool wide = (ldy & 3) == 0 && (bsy & 3) == 0 && (reinterpret_cast<uintptr_t>(y) & 15) == 0;
    for (int idx = first * THREADS + threadIdx.x; idx < QUADS; idx += ranges * THREADS) {
        const int gm = m0 + idx / (kSgBN / 4), gn = n0 + idx % (kSgBN / 4) * 4;
        float4 part[8];
#pragma unroll
        for (int r = 0; r < 8; ++r)
            if (r < ranges) part[r] = *cluster.map_shared_rank(reinterpret_cast<const float4*>(sg_buf) + idx, r);
        float4 sum = part[0];
#pragma unroll
        for (int r = 1; r < 8; ++r)
            if (r < ranges)
                sum = make_float4(__fadd_rn(sum.x, part[r].x), __fadd_rn(sum.y, part[r].y),
                                  __fadd_rn(sum.z, part[r].z), __fadd_rn(sum.w, part[r].w));
        if (gm >= M) continue;
        float out[4] = {sum.x, sum.y, sum.z, sum.w};
#pragma unroll
        for (int e = 0; e < 4; ++e)
            if (bias != nullptr && gn + e < N) out[e] = __fadd_rn(out[e], bias[gn + e]);
        float* dst = y + gm * ldy + gn;
        if (wide && gn + 3 < N) {
            *reinterpret_cast<float4*>(dst) = make_float4(out[0], out[1], out[2], out[3]);
        } else {
#pragma unroll
            for (int e = 0; e < 4; ++e)
                if (gn + e < N) dst[e] = out[e];
        }
    }
    cluster.sync();                                      // no CTA leaves while its tile is read
}

template <int BM, int TM, int TN, bool VEC, bool CLUSTER>
int sg_launch_one(const FsArgs& a, int ranges, cudaStream_t stream) {
    auto kernel = sgemm_nt_kernel<BM, TM, TN, VEC, CLUSTER>;
    constexpr int smem = sg_smem<BM>();
    if (smem > 48 * 1024)
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    const unsigned tiles_n = static_cast<unsigned>((a.N + kSgBN - 1) / kSgBN);
    // (a grid has at most 65,535 tiles of rows: 4.19 M rows go in one launch)
    for (int m = 0; m < a.M;) {
        const int rows = a.M - m < 65535 * BM ? a.M - m : 65535 * BM;
        launch_pdl_cluster(kernel, dim3(tiles_n * (CLUSTER ? ranges : 1), (rows + BM - 1) / BM, a.batch),
                           dim3(sg_threads<BM, TM, TN>()), smem, CLUSTER ? ranges : 1, stream, a.x + m * a.ldx, a.w,
                           a.bias, a.y + m * a.ldy, rows, a.N, a.K, ranges, sg_range_length(a.K, ranges), a.ldx,
                           a.ldy, a.bsx, a.bsw, a.bsy, a.w_constant);
        m += rows;
    }
    return launch_status();
}

template <int BM, int TM, int TN>
int sg_launch(const FsArgs& a, cudaStream_t stream) {
    const int ranges = sg_ranges(a.K);
    const long long tiles = static_cast<long long>((a.N + kSgBN - 1) / kSgBN) * ((a.M + BM - 1) / BM) * a.batch;
    const bool cluster = ranges > 1 && tiles < sg_fill_tiles(BM);
    const bool vec = ((a.K | a.ldx | a.bsx | a.bsw) & 3) == 0 &&
                     ((reinterpret_cast<uintptr_t>(a.x) | reinterpret_cast<uintptr_t>(a.w)) & 15) == 0;
    if (vec) return cluster ? sg_launch_one<BM, TM, TN, true, true>(a, ranges, stream)
                            : sg_launch_one<BM, TM, TN, true, false>(a, ranges, stream);
    return cluster ? sg_launch_one<BM, TM, TN, false, true>(a, ranges, stream)
                   : sg_launch_one<BM, TM, TN, false, false>(a, ranges, stream);
}

}  // namespace somi

using namespace somi;

// y_b[M, N] = x_b[M, K] w_b[N, K]^T (+ bias) for b in [0, batch), all float32.  Rows of x_b and y_b lie
// ldx and ldy elements apart, rows of w_b K; product b's operands start b * bs{x,w,y} elements
// after product 0's (so the heads of a [tokens, heads, width] tensor are a batch without a copy).
// w_constant: no kernel of the same step writes w (a model's weights), so it is read before the
// dependency wait.
SOMI_API int somi_gemm_f32_batched(const float* x, const float* w, const float* bias, float* y, int M,
                                   int N, int K, int batch, long long ldx, long long ldy,
                                   long long bsx, long long bsw, long long bsy, int w_constant,
                                   cudaStream_t stream) {
    if (M <= 0 || N <= 0 || batch <= 0) return 0;
    if (K <= 0 || batch > 65535 || ldx < K || ldy < N) return SOMI_ERR_UNSUPPORTED;
    const FsArgs a{x, w, bias, y, M, N, K, batch, w_constant, ldx, ldy, bsx, bsw, bsy};
    if (fs_takes(a)) return M <= 16 ? fs_launch_rows(a, stream) : fs_launch_tiles(a, stream);
    if (M <= 2) return sg_launch<2, 2, 1>(a, stream);
    if (M <= 4) return sg_launch<4, 4, 1>(a, stream);
    if (M <= 8) return sg_launch<8, 2, 2>(a, stream);
    if (M <= 16) return sg_launch<16, 4, 2>(a, stream);
    if (M <= 384) return sg_launch<32, 8, 2>(a, stream);
    return sg_launch<64, 8, 4>(a, stream);
}

// y[M, N] = x[M, K] w[N, K]^T (+ bias), all float32, row-major.
SOMI_API int somi_gemm_f32(const float* x, const float* w, const float* bias, float* y, int M, int N,
                           int K, int w_constant, cudaStream_t stream) {
    return somi_gemm_f32_batched(x, w, bias, y, M, N, K, 1, K, N, 0, 0, 0, w_constant, stream);
}
