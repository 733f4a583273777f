// The matrix-state recurrence with a constant decay per head, S <- g S + k v^T, y = S^T q, for prompt portions
// in chunks of 64 rows (bfloat16 inputs; the step by step form in recurrent_parts.cu serves single
// tokens, short portions, float32 inputs, decays per channel and the delta rule).  With S_0 the state in
// front of a chunk, t and s rows of it counted from 0, and n rows:
//     y_t = g^(t + 1) S_0^T q_t + sum over s <= t of g^(t - s) (q_t . k_s) v_s
//     S_n = g^n S_0 + U,   U = sum over s of g^(n - 1 - s) k_s v_s^T
// Three kernels: U of every chunk and head; the states in front of every chunk, from U in place and in
// order (and the last one to the request's slot); y.  Everything is float32: the products are FMAs on the
// CUDA cores, the powers of g are powf, q and k are activated and rotated in float32 as they are read.
//
// Why: step by step, a portion is one chain of rows per (head, 16 columns) with two sums over a warp each:
// 224 CTAs for 28 heads of 128, 522 us for 2,048 rows behind 43 us of preparation.  In chunks a row
// costs a third more FMAs (64 x 2 x (5/8) + 128 x 2 per column against 128 x 2 and the sums over warps), but nothing
// waits for anything but the second kernel, and the FMA pipe is the bound: thread tiles of 8 x 8 and 4 x 8 from
// shared memory, the upper triangle left out in blocks of 16.  The same rows: angles 5, U 70, states 36,
// y 123 us (0.92 and 1.5 G FMAs at 26 and 24 TFLOP/s; scalar and paired FMAs take the same time).  The layer
// with it, step by step / in chunks, 28 heads of 128: 128 rows 98 / 99 us, 256 132 / 115, 2,048 796 / 446, 8,192
// 3,053 / 1,669; 14 heads of 64: 32 rows 33 / 37, 64 40 / 37, 2,048 467 / 92.
#include "common.cuh"
#include "rotation.cuh"
#include "vec4.cuh"

namespace somi {

constexpr int kChRows = 64;           // rows per chunk (the tile list's query tiles of 64)
constexpr int kChThreads = 256;
constexpr int kChBK = 32;             // key channels of the state staged at a time

__device__ __forceinline__ float ch_silu(float z) { return z / (1.0f + expf(-z)); }
__device__ __forceinline__ void ch_fma2(unsigned long long& d, unsigned long long a, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
__device__ __forceinline__ float ch_sum2(unsigned long long d) {
    float lo, hi;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(d));
    return lo + hi;
}

// Cosine and sine of every pair of the portions' rows, once for all heads.
__global__ void chunk_angles_kernel(const int* __restrict__ positions, const double* __restrict__ freq, int half,
                                    int n, float2* __restrict__ cs) {
    pdl_launch_dependents();
    pdl_wait();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) cs[i] = turn_by(static_cast<double>(positions[i / half]), freq[i % half]);
}

struct ChRows {                       // rows of q, k or v of one head
    const __nv_bfloat16* p;           // row 0 of the step, the head's first element
    long long stride;
    int silu;
    const float2* cs;                 // [T, half], or null
    int half;
};

// Rows [row0, row0 + rows) into shared memory as float32 times `factor(row)`, zeros up to 64 rows.  A thread
// takes two quads of a row at a time, the two that turn together where the row turns; all its loads are
// under way before the first value is used (one after the other they took longer than the products).
template <int D, typename F>
__device__ __forceinline__ void ch_load(float* dst, int pitch, const ChRows& m, int row0, int rows, F factor) {
    constexpr int ACROSS = D / 8, APART = kChThreads / ACROSS, N = kChRows / APART;
    const int r0 = threadIdx.x / ACROSS, p = threadIdx.x % ACROSS, turning = m.cs != nullptr ? m.half / 4 : 0;
    const bool turn = p < turning;
    const int c = turn ? 4 * p : 8 * turning + 8 * (p - turning), c2 = turn ? c + m.half : c + 4;
    uint2 x[N], o[N];
    float4 a[N], b[N];
#pragma unroll
    for (int i = 0; i < N; ++i) {
        const int r = r0 + i * APART;
        x[i] = o[i] = make_uint2(0, 0);
        a[i] = b[i] = make_float4(1.f, 0.f, 1.f, 0.f);
        if (r < rows) {
            const __nv_bfloat16* row = m.p + static_cast<size_t>(row0 + r) * m.stride;
            x[i] = __ldg(reinterpret_cast<const uint2*>(row + c));
            o[i] = __ldg(reinterpret_cast<const uint2*>(row + c2));
            if (turn) {
                const float4* cs = reinterpret_cast<const float4*>(m.cs + static_cast<size_t>(row0 + r) * m.half + c);
                a[i] = cs[0];
                b[i] = cs[1];
            }
        }
    }
#pragma unroll
    for (int i = 0; i < N; ++i) {
        const int r = r0 + i * APART;
        F4 u = load4(reinterpret_cast<const __nv_bfloat16*>(&x[i])), v = load4(reinterpret_cast<const __nv_bfloat16*>(&o[i]));
        if (m.silu) {
#pragma unroll
            for (int e = 0; e < 4; ++e) { u.v[e] = ch_silu(u.v[e]); v.v[e] = ch_silu(v.v[e]); }
        }
        if (turn) {
            const float cs[4] = {a[i].x, a[i].z, b[i].x, b[i].z}, sn[4] = {a[i].y, a[i].w, b[i].y, b[i].w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float lo = fmaf(u.v[e], cs[e], -(v.v[e] * sn[e]));
                v.v[e] = fmaf(v.v[e], cs[e], u.v[e] * sn[e]);
                u.v[e] = lo;
            }
        }
        const float f = r < rows ? factor(r) : 0.f;
#pragma unroll
        for (int e = 0; e < 4; ++e) { u.v[e] *= f; v.v[e] *= f; }
        store4(dst + r * pitch + c, u);
        store4(dst + r * pitch + c2, v);
    }
}

// U [tile][head][value channel][key channel].  A CTA per (tile, head); a thread owns C x C elements.
template <int D>
__global__ void __launch_bounds__(kChThreads)
chunk_update_kernel(ChRows k, ChRows v, const float* __restrict__ decay, const int* __restrict__ tiles, int heads,
                    int group, float* __restrict__ u) {
    constexpr int C = D / 16;
    extern __shared__ __align__(16) float ch_smem[];
    float* ks = ch_smem;                                  // [64][D]
    float* vs = ks + kChRows * D;                         // [64][D]
    pdl_launch_dependents();
    pdl_wait();
    const int* tile = tiles + 3 * blockIdx.x;
    const int row0 = tile[1], rows = tile[2], h = blockIdx.y;
    __shared__ float pow_s[kChRows];
    if (threadIdx.x < kChRows) pow_s[threadIdx.x] = powf(decay[h], static_cast<float>(threadIdx.x));
    __syncthreads();
    k.p += static_cast<size_t>(h / group) * D;
    v.p += static_cast<size_t>(h) * D;
    ch_load<D>(ks, D, k, row0, rows, [&](int r) { return pow_s[rows - 1 - r]; });
    ch_load<D>(vs, D, v, row0, rows, [](int) { return 1.f; });
    __syncthreads();
    // key channels 4 ti .. (and 64 further on), value channels 4 tj .. likewise; a warp 4 x 8 of them
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int ti = warp / 2 * 4 + lane / 8, tj = warp % 2 * 8 + lane % 8;
    float acc[C][C];                                      // [value channel][key channel]
#pragma unroll
    for (int j = 0; j < C; ++j)
#pragma unroll
        for (int i = 0; i < C; ++i) acc[j][i] = 0.f;
#pragma unroll 4
    for (int s = 0; s < kChRows; ++s) {
        float a[C], b[C];
#pragma unroll
        for (int e = 0; e < C; e += 4) {
            const F4 x = load4(ks + s * D + 4 * ti + 16 * e), y = load4(vs + s * D + 4 * tj + 16 * e);
#pragma unroll
            for (int i = 0; i < 4; ++i) { a[e + i] = x.v[i]; b[e + i] = y.v[i]; }
        }
#pragma unroll
        for (int j = 0; j < C; ++j)
#pragma unroll
            for (int i = 0; i < C; ++i) acc[j][i] = fmaf(a[i], b[j], acc[j][i]);
    }
    float* dst = u + (static_cast<size_t>(blockIdx.x) * heads + h) * D * D;
#pragma unroll
    for (int j = 0; j < C; ++j)
#pragma unroll
        for (int i = 0; i < C; i += 4)
            store4(dst + (4 * tj + j % 4 + 64 * (j / 4)) * D + 4 * ti + 16 * i,
                   F4{{acc[j][i], acc[j][i + 1], acc[j][i + 2], acc[j][i + 3]}});
}

// U of a request's chunks -> the states in front of them, in place; the state behind the last to its slot.
// grid (D * D / 4 / 256, heads, portions).
template <int D>
__global__ void __launch_bounds__(kChThreads)
chunk_states_kernel(float* __restrict__ u, const float* __restrict__ decay, const int* __restrict__ cu_q,
                    const int* __restrict__ state_slot, float* __restrict__ state, int heads) {
    pdl_launch_dependents();
    pdl_wait();
    const int h = blockIdx.y, r = blockIdx.z;
    int tile = 0;                                         // the request's first
    for (int i = 0; i < r; ++i) tile += (cu_q[i + 1] - cu_q[i] + kChRows - 1) / kChRows;
    const int rows = cu_q[r + 1] - cu_q[r], n = (rows + kChRows - 1) / kChRows;
    const float g = decay[h], full = powf(g, static_cast<float>(kChRows));
    const float tail = powf(g, static_cast<float>(rows - (n - 1) * kChRows));
    const int at = (blockIdx.x * kChThreads + threadIdx.x) * 4;
    float* own = state + (static_cast<size_t>(state_slot[r]) * heads + h) * D * D + at;
    float* p = u + (static_cast<size_t>(tile) * heads + h) * D * D + at;
    const size_t step = static_cast<size_t>(heads) * D * D;
    F4 s = load4(own);
    constexpr int AHEAD = 8;                              // loads in flight
    for (int c0 = 0; c0 < n; c0 += AHEAD) {
        F4 x[AHEAD];
#pragma unroll
        for (int c = 0; c < AHEAD; ++c)
            if (c0 + c < n) x[c] = load4(p + (c0 + c) * step);
#pragma unroll
        for (int c = 0; c < AHEAD; ++c) {
            if (c0 + c >= n) break;
            store4(p + (c0 + c) * step, s);
            const float f = c0 + c == n - 1 ? tail : full;
#pragma unroll
            for (int e = 0; e < 4; ++e) s.v[e] = fmaf(s.v[e], f, x[c].v[e]);
        }
    }
    store4(own, s);
}

// y of a chunk.  A CTA per (tile, head): rows tr + 16 i; the products q . k_s for keys tc + 16 j; outputs
// of value channels tc + 16 j (from the state) and then, with P in shared memory, the same.
template <int D>
__global__ void __launch_bounds__(kChThreads, 2)
chunk_outputs_kernel(ChRows q, ChRows k, ChRows v, float q_scale, const float* __restrict__ decay,
                     const int* __restrict__ tiles, const float* __restrict__ states, int heads, int group,
                     float* __restrict__ y) {
    constexpr int C = D / 16, P = D + 4, PP = kChRows + 4, SP = kChBK + 4, STAGES = 2;
    extern __shared__ __align__(16) float ch_smem[];
    float* qs = ch_smem;                                  // [64][P]
    float* ps = qs + kChRows * P;                         // [64][PP]
    float* xs = ps + kChRows * PP;                        // k [64][P], then stages of the state [D][SP], then v [64][D]
    __shared__ float pow_s[kChRows + 1];
    pdl_launch_dependents();
    pdl_wait();
    const int* tile = tiles + 3 * blockIdx.x;
    const int row0 = tile[1], rows = tile[2], h = blockIdx.y;
    q.p += static_cast<size_t>(h / group) * D;
    k.p += static_cast<size_t>(h / group) * D;
    v.p += static_cast<size_t>(h) * D;
    if (threadIdx.x <= kChRows) pow_s[threadIdx.x] = powf(decay[h], static_cast<float>(threadIdx.x));
    ch_load<D>(qs, P, q, row0, rows, [&](int) { return q_scale; });
    ch_load<D>(xs, P, k, row0, rows, [](int) { return 1.f; });
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int tr = warp / 2 * 4 + lane / 8, tc = warp % 2 * 8 + lane % 8;
    {
        unsigned long long acc[4][4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[i][j] = 0ull;
#pragma unroll 4
        for (int d = 0; d < D; d += 4) {
            ulonglong2 b[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) b[j] = *reinterpret_cast<const ulonglong2*>(xs + (tc + 16 * j) * P + d);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(qs + (tr + 16 * i) * P + d);
#pragma unroll
                for (int j = 0; j <= i; ++j) ch_fma2(acc[i][j], a.x, b[j].x);
#pragma unroll
                for (int j = 0; j <= i; ++j) ch_fma2(acc[i][j], a.y, b[j].y);
            }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j <= i; ++j) {
                const int t = tr + 16 * i, s = tc + 16 * j;
                ps[t * PP + s] = s <= t ? ch_sum2(acc[i][j]) * pow_s[t - s] : 0.f;
            }
    }
    __syncthreads();                                      // k has been read
    const float* st = states + (static_cast<size_t>(blockIdx.x) * heads + h) * D * D;
    auto stage = [&](int c) {                             // key channels 32 c .. of all value channels
        float* dst = xs + c % STAGES * (D * SP);
        for (int i = threadIdx.x; i < D * (kChBK / 4); i += kChThreads) {
            const int j = i / (kChBK / 4), e = i % (kChBK / 4) * 4;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(
                             static_cast<uint32_t>(__cvta_generic_to_shared(dst + j * SP + e))),
                         "l"(st + j * D + c * kChBK + e)
                         : "memory");
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    // even and odd terms of every output's product with the state
    unsigned long long acc[4][C];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < C; ++j) acc[i][j] = 0ull;
    stage(0);
    for (int c = 0; c < D / kChBK; ++c) {
        if (c + 1 < D / kChBK) {
            stage(c + 1);
            asm volatile("cp.async.wait_group 1;\n" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        }
        __syncthreads();
        const float* ss = xs + c % STAGES * (D * SP);
#pragma unroll 2
        for (int d = 0; d < kChBK; d += 4) {
            ulonglong2 a[4];
#pragma unroll
            for (int i = 0; i < 4; ++i)
                a[i] = *reinterpret_cast<const ulonglong2*>(qs + (tr + 16 * i) * P + c * kChBK + d);
#pragma unroll
            for (int j = 0; j < C; ++j) {
                const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(ss + (tc + 16 * j) * SP + d);
#pragma unroll
                for (int i = 0; i < 4; ++i) ch_fma2(acc[i][j], a[i].x, b.x);
#pragma unroll
                for (int i = 0; i < 4; ++i) ch_fma2(acc[i][j], a[i].y, b.y);
            }
        }
        __syncthreads();                                  // the stage has been read
    }
    float o[4][C];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < C; ++j) o[i][j] = ch_sum2(acc[i][j]) * pow_s[tr + 16 * i + 1];
    ch_load<D>(xs, D, v, row0, rows, [](int) { return 1.f; });
    __syncthreads();
#pragma unroll
    for (int b = 0; b < 4; ++b) {                         // 16 keys that the rows of blocks b .. 3 see
#pragma unroll 2
        for (int s = 16 * b; s < 16 * b + 16; s += 4) {
            F4 p[4];
#pragma unroll
            for (int i = b; i < 4; ++i) p[i] = load4(ps + (tr + 16 * i) * PP + s);
#pragma unroll
            for (int m = 0; m < 4; ++m)
#pragma unroll
                for (int j = 0; j < C; ++j) {
                    const float x = xs[(s + m) * D + tc + 16 * j];
                    // (on the diagonal a later row's infinity must not meet a probability of zero)
                    if (s + m <= tr + 16 * b) o[b][j] = fmaf(p[b].v[m], x, o[b][j]);
#pragma unroll
                    for (int i = b + 1; i < 4; ++i) o[i][j] = fmaf(p[i].v[m], x, o[i][j]);
                }
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int t = tr + 16 * i;
        if (t >= rows) continue;
        float* dst = y + static_cast<size_t>(row0 + t) * heads * D + static_cast<size_t>(h) * D + tc;
#pragma unroll
        for (int j = 0; j < C; ++j) dst[16 * j] = o[i][j];
    }
}

template <int D>
constexpr int ch_update_smem() { return 4 * 2 * kChRows * D; }
template <int D>
constexpr int ch_outputs_smem() {
    constexpr int k = kChRows * (D + 4), s = 2 * D * (kChBK + 4);
    return 4 * (kChRows * (D + 4) + kChRows * (kChRows + 4) + (k > s ? k : s));
}

template <int D>
int launch_chunks(const ChRows& q, const ChRows& k, const ChRows& v, float q_scale, const float* decay, float* state,
                  const int* cu_q, const int* state_slot, const int* tiles, int n_tiles, int n_req, int heads,
                  int group, float* u, float* y, cudaStream_t stream) {
    cudaFuncSetAttribute(chunk_update_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, ch_update_smem<D>());
    cudaFuncSetAttribute(chunk_outputs_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, ch_outputs_smem<D>());
    const dim3 grid(n_tiles, heads);
    launch_pdl(chunk_update_kernel<D>, grid, dim3(kChThreads), ch_update_smem<D>(), stream, k, v, decay, tiles, heads,
               group, u);
    launch_pdl(chunk_states_kernel<D>, dim3(D * D / 4 / kChThreads, heads, n_req), dim3(kChThreads), 0, stream, u, decay,
               cu_q, state_slot, state, heads);
    launch_pdl(chunk_outputs_kernel<D>, grid, dim3(kChThreads), ch_outputs_smem<D>(), stream, q, k, v, q_scale, decay,
               tiles, u, heads, group, y);
    return launch_status();
}

}  // namespace somi

using namespace somi;

// q, k: bfloat16 rows of heads / group heads of D elements, `stride` apart; v: of `heads` heads; D = 64 or 128.
// `silu`: q and k (bit 0) and v (bit 1) pass SiLU.  rot > 0: the pairs (i, i + rot / 2) of q and k turn by
// positions * rot_freq; angles: float32 scratch [portions' rows, rot].  `tiles`: int32 [n_tiles, 3] = (request,
// first row, rows <= 64) over the n_req multi-token requests, in order.  u: float32 scratch [n_tiles, heads, D, D].
// state: float32 [slots, heads, D, D] (value channel, key channel); y: float32 rows of heads * D.
SOMI_API int somi_matrix_state_chunks(const void* q, const void* k, const void* v, long long q_stride,
                                      long long k_stride, long long v_stride, int silu, float q_scale,
                                      const float* decay, float* state, const int* cu_q, const int* state_slot,
                                      const int* tiles, int n_tiles, int n_req, int n_rows, int heads, int group, int D,
                                      const int* positions, const double* rot_freq, int rot, float* angles, float* u,
                                      float* y, cudaStream_t stream) {
    if (n_tiles <= 0 || n_req <= 0) return 0;
    const uintptr_t bits = reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(v);
    if (decay == nullptr || (rot > 0 && (positions == nullptr || rot_freq == nullptr || angles == nullptr)))
        return SOMI_ERR_UNSUPPORTED;
    if ((D != 64 && D != 128) || heads <= 0 || heads > 65535 || n_req > 65535 || group <= 0 || heads % group ||
        ((q_stride | k_stride | v_stride) & 3) || (bits & 7) || rot < 0 || rot > D || rot % 8 || (rot > 0 && (silu & 1)) ||
        ((reinterpret_cast<uintptr_t>(state) | reinterpret_cast<uintptr_t>(u)) & 15) || (reinterpret_cast<uintptr_t>(angles) & 15))
        return SOMI_ERR_UNSUPPORTED;
    float2* cs = rot > 0 ? reinterpret_cast<float2*>(angles) : nullptr;
    const int half = rot / 2, n = n_rows * half;
    if (rot > 0) launch_pdl(chunk_angles_kernel, dim3((n + 255) / 256), dim3(256), 0, stream, positions, rot_freq, half, n, cs);
    const ChRows qr{static_cast<const __nv_bfloat16*>(q), q_stride, silu & 1, cs, half};
    const ChRows kr{static_cast<const __nv_bfloat16*>(k), k_stride, silu & 1, cs, half};
    const ChRows vr{static_cast<const __nv_bfloat16*>(v), v_stride, silu >> 1 & 1, nullptr, 0};
    return D == 64 ? launch_chunks<64>(qr, kr, vr, q_scale, decay, state, cu_q, state_slot, tiles, n_tiles, n_req, heads,
                                       group, u, y, stream)
                   : launch_chunks<128>(qr, kr, vr, q_scale, decay, state, cu_q, state_slot, tiles, n_tiles, n_req, heads,
                                        group, u, y, stream);
}
