// The matrix-state recurrence with a constant decay per head, S <- g S + k v^T, y = S^T q, for prompt portions
// in chunks of 128 rows (bfloat16 inputs; the step by step form in recurrent_parts.cu serves single
// tokens, short portions, float32 inputs, decays per channel and the delta rule).  With S_0 the state in
// front of a chunk, t and s rows of it counted from 0, and n rows:
//     y_t = g^(t + 1) S_0^T q_t + sum over s <= t of g^(t - s) (q_t . k_s) v_s
//     S_n = g^n S_0 + U,   U = sum over s of g^(n - 1 - s) k_s v_s^T
// Three kernels: U of every chunk and head; the states in front of every chunk, from U in place and in
// order (and the last one to the request's slot); y.  Everything is float32: q and k are activated and rotated in float32 as they
// are read, the powers of g are powf, and the products take every float32 operand as three bfloat16 numbers whose sum it
// is (gemm_f32_split.cuh; v as it is, where it is not activated), summed in float32 by `tcgen05.mma`, 64 terms at a time.
//
// Why: step by step, a portion is one chain of rows per (head, 16 columns) with two sums over a warp each:
// 224 CTAs for 28 heads of 128, 522 us for 2,048 rows behind 43 us of preparation.  In chunks nothing
// waits for anything but the second kernel.  As FMAs on the CUDA cores, in chunks of 64 rows, the products took U 70 and y 123 us
// (25 TFLOP/s); on tensor cores, with half as many states in between, the same rows take: angles 3, U 29, states 18 (36), y 88 us,
// each with nothing in L2 (y 65 with 128 terms in an accumulator, whose error was 2.7 times the FMAs').  What bounds y: a CTA's phases (load
// and split, multiply, load and split, ..) one behind the other, two CTAs to an SM, 448 CTAs in two rounds of 296: 41 % of a warp's
// time is waiting for loads, 16 % for instructions, the tensor pipe is busy 14 % of the cycles.  In 128 registers y spills 16 to 150 bytes;
// fetching a phase ahead did not shorten it, U by 1 us.
// The layer with it, 28 heads of 128, 2,048 rows: step by step 796, FMAs 462, now 385 us.
#include "gemm_f32_split.cuh"
#include "rotation.cuh"
#include "tcgen05.cuh"
#include "vec4.cuh"

namespace somi {

constexpr int kChRows = 128;          // rows per chunk: two tiles of the tile list, the MMA's M
constexpr int kChTile = 64;
constexpr int kChThreads = 256;

__device__ int g_chunks_error = 0;

__device__ __forceinline__ float ch_silu(float z) { return z / (1.0f + expf(-z)); }

// Cosine and sine of every pair of the portions' rows, once for all heads.
__global__ void chunk_angles_kernel(const int* __restrict__ positions, const double* __restrict__ freq, int half,
                                    int n, float2* __restrict__ cs) {
    pdl_launch_dependents();
    pdl_wait();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) cs[i] = turn_by(static_cast<double>(positions[i / half]), freq[i % half]);
}

// The place in u of the first chunk of request r of a run, which begins `row` rows behind the run's first: its n rows' chunks end in
// front of the next request's place, (row + n + 127 + 127 r) / 128, and nobody sums over the requests in front.
__device__ __forceinline__ int ch_place(int row, int r) { return (row + (kChRows - 1) * r) / kChRows; }

// The chunks of a run of requests, as its tiles of 64 rows give them: each pair of a request's tiles, at the pair's first.
struct ChTiles {
    const int *tiles, *cu_q;          // (request, first row, rows); the run's requests' first rows
    int first;                        // the run's first request
    // The chunk that begins with tile i: its first row, its place in u, and how many rows it has (0: the tile is another chunk's second).
    __device__ __forceinline__ int rows_of(int i, int& row0, int& place) const {
        const int r = ld_step(tiles + 3 * i) - first;     // [descriptor]
        row0 = ld_step(tiles + 3 * i + 1);
        const int begin = ld_step(cu_q + r);
        place = ch_place(begin - ld_step(cu_q), r) + (row0 - begin) / kChRows;
        return (row0 - begin) / kChTile & 1 ? 0 : min(kChRows, ld_step(cu_q + r + 1) - row0);
    }
};

struct ChRows {                       // rows of q, k or v of one head
    const __nv_bfloat16* p;           // row 0 of the step, the head's first element
    long long stride;
    int silu;
    const float2* cs;                 // [T, half], or null
    int half;
};

// Two quads of a row, activated, turned against each other where the row turns, times f.
__device__ __forceinline__ void ch_values(const uint2& x, const uint2& o, bool turn, const float4& a, const float4& b, int silu,
                                          float f, F4& u, F4& v) {
    u = load4(reinterpret_cast<const __nv_bfloat16*>(&x));
    v = load4(reinterpret_cast<const __nv_bfloat16*>(&o));
    if (silu) {
#pragma unroll
        for (int e = 0; e < 4; ++e) { u.v[e] = ch_silu(u.v[e]); v.v[e] = ch_silu(v.v[e]); }
    }
    if (turn) {
        const float cs[4] = {a.x, a.z, b.x, b.z}, sn[4] = {a.y, a.w, b.y, b.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float lo = fmaf(u.v[e], cs[e], -(v.v[e] * sn[e]));
            v.v[e] = fmaf(v.v[e], cs[e], u.v[e] * sn[e]);
            u.v[e] = lo;
        }
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) { u.v[e] *= f; v.v[e] *= f; }
}
// A row's channels in pairs of quads: pair p is the quads at c and c2, which turn against each other or are neighbours.
__device__ __forceinline__ void ch_pair(const ChRows& m, int p, bool& turn, int& c, int& c2) {
    const int turning = m.cs != nullptr ? m.half / 4 : 0;
    turn = p < turning;
    c = turn ? 4 * p : 8 * turning + 8 * (p - turning);
    c2 = turn ? c + m.half : c + 4;
}
// The three parts of a quad (gemm_f32_split.cuh), as 8 bytes each.
__device__ __forceinline__ void ch_split(const F4& u, uint2 (&part)[3]) {
    fs_split(u.v[0], u.v[1], part[0].x, part[1].x, part[2].x);
    fs_split(u.v[2], u.v[3], part[0].y, part[1].y, part[2].y);
}

// Numbers of row r that have no parts (an MMA would carry what they are to rows that do not see them): 0 in their place, and
// the row noted.
__device__ __forceinline__ void ch_leave_out(F4& u, F4& v, int r, uint32_t* odd) {
    float most = 0.f;
#pragma unroll
    for (int e = 0; e < 4; ++e) most = fs_largest(fs_largest(most, u.v[e]), v.v[e]);
    if (fs_has_parts(most)) return;
    atomicOr(odd + (r >> 5), 1u << (r & 31));
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        if (!fs_has_parts(u.v[e])) u.v[e] = 0.f;
        if (!fs_has_parts(v.v[e])) v.v[e] = 0.f;
    }
}

// What a thread reads of ROWS rows of one or two matrices (q and k turn by the same angles): pair `pl` of every APART-th row.
// Fetched a phase before it is used, so that the loads run under the MMAs of the phase before.
template <int ROWS, int PAIRS, int MATS>
struct ChFetch {
    static constexpr int APART = kChThreads / PAIRS, N = ROWS / APART;
    static_assert(ROWS % APART == 0, "whole passes");
    uint2 x[MATS][N], o[MATS][N];
    float4 a[N], b[N];
    int c, c2;
    bool turn;
    __device__ __forceinline__ void fetch(const ChRows* const (&m)[MATS], int row0, int at, int rows, int p0) {
        ch_pair(*m[0], p0 + static_cast<int>(threadIdx.x) % PAIRS, turn, c, c2);
#pragma unroll
        for (int i = 0; i < N; ++i) {
            const int r = at + threadIdx.x / PAIRS + i * APART;
            a[i] = b[i] = make_float4(1.f, 0.f, 1.f, 0.f);
#pragma unroll
            for (int k = 0; k < MATS; ++k) x[k][i] = o[k][i] = make_uint2(0, 0);
            if (r < rows) {
#pragma unroll
                for (int k = 0; k < MATS; ++k) {
                    const __nv_bfloat16* row = m[k]->p + static_cast<size_t>(row0 + r) * m[k]->stride;
                    x[k][i] = __ldg(reinterpret_cast<const uint2*>(row + c));
                    o[k][i] = __ldg(reinterpret_cast<const uint2*>(row + c2));
                }
                if (turn) {
                    const float4* cs = reinterpret_cast<const float4*>(m[0]->cs + static_cast<size_t>(row0 + r) * m[0]->half + c);
                    a[i] = cs[0];
                    b[i] = cs[1];
                }
            }
        }
    }
    // The parts of matrix K times factor(row).  FLAT: tiles of [ROWS][8 pairs], a pair's eight numbers together: 64 channels in
    // an order that q, k and the state share, for products over channels.  Else tiles of [ROWS][64 channels] in the rows'
    // order, a block of 64 channels behind the other, and numbers that have no parts are left out, their rows noted in `odd`.
    template <int K, bool FLAT, typename F>
    __device__ __forceinline__ void put(unsigned char* dst, int plane, int silu, int at, F factor, uint32_t* odd = nullptr) const {
        static_assert(!FLAT || PAIRS == 8, "64 channels");
        const int pl = threadIdx.x % PAIRS;
#pragma unroll
        for (int i = 0; i < N; ++i) {
            const int rl = threadIdx.x / PAIRS + i * APART;
            F4 u, v;
            ch_values(x[K][i], o[K][i], turn, a[i], b[i], silu, factor(at + rl), u, v);
            if (!FLAT) ch_leave_out(u, v, at + rl, odd);
            uint2 pu[3], pv[3];
            ch_split(u, pu);
            ch_split(v, pv);
            auto place = [&](int channel) {
                return dst + channel / 64 * (ROWS * 128) + rl * 128 + (((channel & 63) >> 3 ^ (rl & 7)) << 4) + (channel & 4) * 2;
            };
#pragma unroll
            for (int e = 0; e < 3; ++e) {
                if (FLAT) {
                    *reinterpret_cast<uint4*>(dst + e * plane + rl * 128 + ((pl ^ (rl & 7)) << 4)) =
                        make_uint4(pu[e].x, pu[e].y, pv[e].x, pv[e].y);
                } else {
                    *reinterpret_cast<uint2*>(place(c) + e * plane) = pu[e];
                    *reinterpret_cast<uint2*>(place(c2) + e * plane) = pv[e];
                }
            }
        }
    }
};
// 64 rows of v from row `at` on, to tiles of [64][64 channels]: as they are, or (SILU) three parts.  Numbers that have no
// parts are left out and their rows noted in `odd`.
template <int D, bool SILU>
struct ChFetchV {
    static constexpr int ACROSS = D / 4, APART = kChThreads / ACROSS, N = 64 / APART;
    uint2 x[N];
    __device__ __forceinline__ void fetch(const ChRows& m, int row0, int at, int rows) {
        const int c = threadIdx.x % ACROSS * 4;
#pragma unroll
        for (int i = 0; i < N; ++i) {
            const int r = at + threadIdx.x / ACROSS + i * APART;
            x[i] = r < rows ? __ldg(reinterpret_cast<const uint2*>(m.p + static_cast<size_t>(row0 + r) * m.stride + c)) : make_uint2(0, 0);
        }
    }
    __device__ __forceinline__ void put(unsigned char* dst, int plane, int at, uint32_t* odd) const {
        const int c = threadIdx.x % ACROSS * 4;
#pragma unroll
        for (int i = 0; i < N; ++i) {
            const int rl = threadIdx.x / ACROSS + i * APART;
            F4 u = load4(reinterpret_cast<const __nv_bfloat16*>(&x[i])), none{{0.f, 0.f, 0.f, 0.f}};
            if (SILU) {
#pragma unroll
                for (int e = 0; e < 4; ++e) u.v[e] = ch_silu(u.v[e]);
            }
            ch_leave_out(u, none, at + rl, odd);
            uint2 part[3];
            ch_split(u, part);
            unsigned char* to = dst + c / 64 * (64 * 128) + rl * 128 + (((c & 63) >> 3 ^ (rl & 7)) << 4) + (c & 4) * 2;
#pragma unroll
            for (int e = 0; e < (SILU ? 3 : 1); ++e) *reinterpret_cast<uint2*>(to + e * plane) = part[e];
        }
    }
};

// Products of parts, the small ones first, in groups of K steps: `f(a's part, b's part, step, accumulate)`, the first into an empty
// accumulator.  PB: 3, or 1 where b is bfloat16.
template <int PB, typename F>
__device__ __forceinline__ void ch_products(int steps, F f) {
    for (int j = 0; j < steps; ++j) {
        f(2, 0, j, j > 0);
        if (PB == 3) {
            f(0, 2, j, true);
            f(1, 1, j, true);
        }
        f(1, 0, j, true);
        if (PB == 3) f(0, 1, j, true);
    }
    for (int j = 0; j < steps; ++j) f(0, 0, j, true);
}
__host__ __device__ constexpr uint32_t ch_idesc(int n, bool a_mn, bool b_mn) {
    return (1u << 4) | (1u << 7) | (1u << 10) | (a_mn ? 1u << 15 : 0u) | (b_mn ? 1u << 16 : 0u) |
           (static_cast<uint32_t>(n >> 3) << 17) | (8u << 24);
}

// What both MMA kernels set up: one barrier, 256 columns of tensor memory.
struct ChMma {
    uint32_t bar, tmem, phase;
    bool ok;
    __device__ __forceinline__ void start(unsigned long long* bar_s, uint32_t* tmem_s) {
        bar = smem_u32(bar_s);
        phase = 0;
        ok = true;
        if (threadIdx.x == 0) {
            mbar_init(bar, 1);
            mbar_fence_init();
        }
        if (threadIdx.x < 32) {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(tmem_s)), "r"(256) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
        }
        t5::fence_before();
        __syncthreads();
        t5::fence_after();
        tmem = *tmem_s;
    }
    // shared memory that all threads have written is the MMAs' operand from here on
    __device__ __forceinline__ void operands_ready() {
        fence_proxy_async();
        t5::fence_before();
        __syncthreads();
        t5::fence_after();
    }
    __device__ __forceinline__ void wait() {              // for what thread 0 has committed
        if (ok && !mbar_wait(bar, phase, 2000000)) {
            ok = false;
            atomicExch(&g_chunks_error, 1);
        }
        phase ^= 1;
        __syncwarp();
        t5::fence_after();
    }
    __device__ __forceinline__ void end() {
        t5::fence_before();
        __syncthreads();
        if (threadIdx.x < 32) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(256) : "memory");
    }
};

// The way of numbers without parts, as FMAs: one channel of a row, activated and turned; q_row k_row or q_row S.
__device__ __forceinline__ float ch_value(const ChRows& m, int row, int c) {
    const __nv_bfloat16* p = m.p + static_cast<size_t>(row) * m.stride;
    float x = __bfloat162float(p[c]);
    if (m.silu) x = ch_silu(x);
    if (m.cs == nullptr || c >= 2 * m.half) return x;
    const bool low = c < m.half;
    const float other = __bfloat162float(p[low ? c + m.half : c - m.half]);
    const float2 t = m.cs[static_cast<size_t>(row) * m.half + (low ? c : c - m.half)];
    return low ? fmaf(x, t.x, -(other * t.y)) : fmaf(x, t.x, other * t.y);
}
__device__ __forceinline__ float ch_dot(const ChRows& q, int row, float q_scale, const ChRows& k, int k_row, int channels) {
    float dot = 0.f;
#pragma unroll 1
    for (int c = 0; c < channels; ++c) dot = fmaf(ch_value(q, row, c) * q_scale, ch_value(k, k_row, c), dot);
    return dot;
}
__device__ __forceinline__ float ch_dot(const ChRows& q, int row, float q_scale, const float* state, int channels) {
    float dot = 0.f;
#pragma unroll 1
    for (int c = 0; c < channels; ++c) dot = fmaf(ch_value(q, row, c) * q_scale, state[c], dot);
    return dot;
}

// U [chunk][head][value channel][key channel].  A CTA per (tile, head), two on an SM: 64 rows at a time, k in parts and v; D = V^T K with
// the rows as the products' K, both operands as the rows lie; the halves' sums in two accumulators.
template <int D, bool SILU>
__global__ void __launch_bounds__(kChThreads, 2)
chunk_update_kernel(ChRows k, ChRows v, const float* __restrict__ decay, ChTiles tiles, int heads,
                    int group, float* __restrict__ u) {
    constexpr int PLANE = 64 * D * 2, PV = SILU ? 3 : 1;
    extern __shared__ unsigned char ch_raw[];
    unsigned char* vs = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(ch_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    unsigned char* ks = vs + PV * PLANE;                  // (with 64 channels an MMA reads 64 more of v: into k, and not used)
    __shared__ float pow_s[kChRows];
    __shared__ uint32_t odd_s[kChRows / 32];
    __shared__ __align__(8) unsigned long long bar_s;
    __shared__ uint32_t tmem_s;
    pdl_launch_dependents();
    int row0, place;
    const int rows = tiles.rows_of(blockIdx.x, row0, place), h = blockIdx.y;
    if (rows == 0) {
        pdl_wait();
        return;
    }
    ChMma mma;
    if (threadIdx.x < kChRows / 32) odd_s[threadIdx.x] = 0;
    mma.start(&bar_s, &tmem_s);
    pdl_wait();
    if (threadIdx.x < kChRows) pow_s[threadIdx.x] = powf(decay[h], static_cast<float>(threadIdx.x));
    __syncthreads();
    k.p += static_cast<size_t>(h / group) * D;
    v.p += static_cast<size_t>(h) * D;
    const int halves = rows > 64 ? 2 : 1;
    ChFetch<64, D / 8, 1> fk;
    ChFetchV<D, SILU> fv;
    fk.fetch({&k}, row0, 0, rows, 0);
    fv.fetch(v, row0, 0, rows);
    for (int i = 0; i < halves; ++i) {
        if (i > 0) mma.wait();                            // the first half's operands have been read
        fv.put(vs, PLANE, 64 * i, odd_s);
        fk.template put<0, false>(ks, PLANE, k.silu, 64 * i, [&](int r) { return pow_s[max(rows - 1 - r, 0)]; }, odd_s);
        if (i + 1 < halves) {
            fk.fetch({&k}, row0, 64, rows, 0);
            fv.fetch(v, row0, 64, rows);
        }
        mma.operands_ready();
        if (threadIdx.x == 0) {
            const uint64_t kd = t5::desc_mnmajor(smem_u32(ks), 64 * 128), vd = t5::desc_mnmajor(smem_u32(vs), 64 * 128);
            ch_products<PV>(4, [&](int pk, int pv, int j, bool more) {
                t5::mma_ss(mma.tmem + i * D, vd + ((pv * PLANE + j * 16 * 128) >> 4), kd + ((pk * PLANE + j * 16 * 128) >> 4),
                           ch_idesc(D, true, true), more);
            });
            t5::commit(mma.bar);
        }
    }
    mma.wait();
    // row 32 (warp % 4) + lane, one half of its columns, through shared memory to whole rows
    constexpr int COLS = D / 2, PITCH = COLS + 4;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if ((warp & 3) * 32 < D) {
        float* own = reinterpret_cast<float*>(vs) + warp * 32 * PITCH;
        const uint32_t at = mma.tmem + (static_cast<uint32_t>(warp & 3) << 21) + (warp >> 2) * COLS;
#pragma unroll
        for (int c = 0; c < COLS; c += 32) {
            float x[32];
            t5::ld32(at + c, x);
            if (halves > 1) {
                float z[32];
                t5::ld32(at + D + c, z);
#pragma unroll
                for (int e = 0; e < 32; ++e) x[e] += z[e];
            }
#pragma unroll
            for (int e = 0; e < 32; e += 4)
                *reinterpret_cast<float4*>(own + lane * PITCH + c + e) = make_float4(x[e], x[e + 1], x[e + 2], x[e + 3]);
        }
        if (odd_s[0] | odd_s[1] | odd_s[2] | odd_s[3]) {
            const int c_v = (warp & 3) * 32 + lane;
#pragma unroll 1
            for (int s = 0; s < rows; ++s) {
                if (!(odd_s[s >> 5] >> (s & 31) & 1)) continue;
                const float x = ch_value(v, row0 + s, c_v);
#pragma unroll 1
                for (int c = 0; c < COLS; ++c) {
                    const float z = ch_value(k, row0 + s, (warp >> 2) * COLS + c) * pow_s[rows - 1 - s];
                    if (!fs_has_parts(x) || !fs_has_parts(z)) own[lane * PITCH + c] = fmaf(z, x, own[lane * PITCH + c]);
                }
            }
        }
        __syncwarp();
        float* dst = u + (static_cast<size_t>(place) * heads + h) * D * D + (warp & 3) * 32 * D + (warp >> 2) * COLS;
#pragma unroll 4
        for (int i = lane; i < 32 * (COLS / 4); i += 32) {
            const int r = i / (COLS / 4), c = i % (COLS / 4) * 4;
            *reinterpret_cast<float4*>(dst + r * D + c) = *reinterpret_cast<const float4*>(own + r * PITCH + c);
        }
    }
    mma.end();
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
    const int place = ch_place(cu_q[r] - cu_q[0], r);
    const int rows = cu_q[r + 1] - cu_q[r], n = (rows + kChRows - 1) / kChRows;
    const float g = decay[h], full = powf(g, static_cast<float>(kChRows));
    const float tail = powf(g, static_cast<float>(rows - (n - 1) * kChRows));
    const int at = (blockIdx.x * kChThreads + threadIdx.x) * 4;
    float* own = state + (static_cast<size_t>(state_slot[r]) * heads + h) * D * D + at;
    float* p = u + (static_cast<size_t>(place) * heads + h) * D * D + at;
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

// y of a chunk.  A CTA per (tile, head), two on an SM.  q S and scores q k^T, for 64 channels at a time; then a thread takes half
// a row of scores, masks and decays them and writes them as parts for their product with v, 64 keys at a time.  Every sum
// of 64 terms has an accumulator of its own and they are added in registers (gemm_f32_split.cuh says why: with 128 terms
// in one, y of 28 heads of 128 was off by 6.6e-7, with 64 by 1.7e-7, as FMAs by 2.4e-7).  With 128 channels two of them fill
// the CTA's half of tensor memory: so q S comes first, its two sums wait in y, and q's first 64 channels are split once more for the scores.
template <int D, bool SILU>
__global__ void __launch_bounds__(kChThreads, 2)
chunk_outputs_kernel(ChRows q, ChRows k, ChRows v, float q_scale, const float* __restrict__ decay,
                     ChTiles tiles, const float* __restrict__ states, int heads, int group,
                     float* __restrict__ y) {
    constexpr int PLANE = kChRows * 128, VPLANE = 64 * D * 2, PV = SILU ? 3 : 1, PARTS = D / 64;
    extern __shared__ unsigned char ch_raw[];
    unsigned char* xs = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(ch_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    unsigned char* ys = xs + 3 * PLANE;
    __shared__ float pow_s[kChRows + 1];
    __shared__ uint32_t odd_s[kChRows / 32];
    __shared__ __align__(8) unsigned long long bar_s;
    __shared__ uint32_t tmem_s;
    pdl_launch_dependents();
    int row0, place;
    const int rows = tiles.rows_of(blockIdx.x, row0, place), h = blockIdx.y;
    if (rows == 0) {
        pdl_wait();
        return;
    }
    ChMma mma;
    if (threadIdx.x < kChRows / 32) odd_s[threadIdx.x] = 0;
    mma.start(&bar_s, &tmem_s);
    pdl_wait();
    q.p += static_cast<size_t>(h / group) * D;
    k.p += static_cast<size_t>(h / group) * D;
    v.p += static_cast<size_t>(h) * D;
    if (threadIdx.x <= kChRows) pow_s[threadIdx.x] = powf(decay[h], static_cast<float>(threadIdx.x));
    const float* st = states + (static_cast<size_t>(place) * heads + h) * D * D;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, halves = rows > 64 ? 2 : 1;
    const uint32_t first = mma.tmem, second = mma.tmem + 128;
    const uint64_t xd = t5::desc_kmajor(smem_u32(xs)), yd = t5::desc_kmajor(smem_u32(ys));
    // xs (64 channels of q) by ys (of k or the state) into columns `to` on
    auto multiply = [&](uint32_t to, int n) {
        mma.operands_ready();
        if (threadIdx.x == 0) {
            ch_products<3>(4, [&](int pa, int pb, int j, bool more) {
                t5::mma_ss(to, xd + ((pa * PLANE + j * 32) >> 4), yd + ((pb * PLANE + j * 32) >> 4), ch_idesc(n, false, false), more);
            });
            t5::commit(mma.bar);
        }
    };
    // the state's key channels 64 i .., in the order of q's; `ready` runs between the loads and the writes
    auto put_state = [&](int i, auto ready) {
        constexpr int N = D / (kChThreads / 8);
        const int r0 = threadIdx.x / 8, pl = threadIdx.x % 8;
        bool turn;
        int c, c2;
        ch_pair(q, 8 * i + pl, turn, c, c2);
        F4 a[N], b[N];
#pragma unroll
        for (int n = 0; n < N; ++n) {
            const float* p = st + (r0 + n * (kChThreads / 8)) * D;
            a[n] = load4(p + c);
            b[n] = load4(p + c2);
        }
        ready();
#pragma unroll
        for (int n = 0; n < N; ++n) {
            const int r = r0 + n * (kChThreads / 8);
            uint2 pa[3], pb[3];
            ch_split(a[n], pa);
            ch_split(b[n], pb);
#pragma unroll
            for (int e = 0; e < 3; ++e)
                *reinterpret_cast<uint4*>(ys + e * PLANE + r * 128 + ((pl ^ (r & 7)) << 4)) = make_uint4(pa[e].x, pa[e].y, pb[e].x, pb[e].y);
        }
    };
    const int t = (warp & 3) * 32 + lane, s0 = (warp >> 2) * 64;         // the thread's row, its scores' first key
    const uint32_t lanes = static_cast<uint32_t>(warp & 3) << 21;
    constexpr int COLS = D / 2, PITCH = COLS + 4;
    const int col0 = (warp >> 2) * COLS, live = rows - (warp & 3) * 32;  // (of the warp's 32 rows)
    float* dst = y + static_cast<size_t>(row0 + (warp & 3) * 32) * heads * D + static_cast<size_t>(h) * D + col0;
    bool fine = true;
    ChFetch<kChRows, 8, 2> f;
    float p[64];
    if constexpr (PARTS == 1) {
        f.fetch({&q, &k}, row0, 0, rows, 0);
        f.template put<0, true>(xs, PLANE, q.silu, 0, [&](int) { return q_scale; });
        f.template put<1, true>(ys, PLANE, k.silu, 0, [](int) { return 1.f; });
        multiply(first, kChRows);
        put_state(0, [&]() { mma.wait(); });
        multiply(second, D);
        t5::ld32(first + lanes + s0, p);
        t5::ld32(first + lanes + s0 + 32, p + 32);
    } else {
        for (int i = 0; i < PARTS; ++i) {
            ChFetch<kChRows, 8, 1> fq;
            fq.fetch({&q}, row0, 0, rows, 8 * i);
            put_state(i, [&]() { if (i > 0) mma.wait(); });
            fq.template put<0, true>(xs, PLANE, q.silu, 0, [&](int) { return q_scale; });
            multiply(i == 0 ? second : first, D);
        }
        mma.wait();
        constexpr int WIDE = 32 + 4;
        float* turn_s = reinterpret_cast<float*>(ys) + warp * 32 * WIDE;
#pragma unroll
        for (int c = 0; c < COLS; c += 32) {             // g^(t + 1) q S of this thread's row and half, to y
            float a[32], b[32], most = 0.f;
            t5::ld32(second + lanes + col0 + c, a);
            t5::ld32(first + lanes + col0 + c, b);
#pragma unroll
            for (int e = 0; e < 32; ++e) {
                a[e] = (a[e] + b[e]) * pow_s[t + 1];
                most = fs_largest(most, a[e]);
            }
            fine &= fs_finite(most);
#pragma unroll
            for (int e = 0; e < 32; e += 4)
                *reinterpret_cast<float4*>(turn_s + lane * WIDE + e) = make_float4(a[e], a[e + 1], a[e + 2], a[e + 3]);
            __syncwarp();
#pragma unroll
            for (int i = lane; i < 32 * 8; i += 32)
                if (i / 8 < live)
                    *reinterpret_cast<float4*>(dst + static_cast<size_t>(i / 8) * heads * D + c + i % 8 * 4) =
                        *reinterpret_cast<const float4*>(turn_s + i / 8 * WIDE + i % 8 * 4);
            __syncwarp();
        }
        ChFetch<kChRows, 8, 1> fk;
        fk.fetch({&k}, row0, 0, rows, 8);                // (q's second half is there)
        __syncthreads();
        fk.template put<0, true>(ys, PLANE, k.silu, 0, [](int) { return 1.f; });
        multiply(first, kChRows);
        f.fetch({&q, &k}, row0, 0, rows, 0);
        mma.wait();
        f.template put<0, true>(xs, PLANE, q.silu, 0, [&](int) { return q_scale; });
        f.template put<1, true>(ys, PLANE, k.silu, 0, [](int) { return 1.f; });
        multiply(second, kChRows);
    }
    ChFetchV<D, SILU> fv;
    fv.fetch(v, row0, 0, rows);
    mma.wait();                                           // q and the state or keys have been read
    if constexpr (PARTS == 2) {
#pragma unroll
        for (int c = 0; c < 64; c += 32) {
            float b[32];
            t5::ld32(second + lanes + s0 + c, p + c);
            t5::ld32(first + lanes + s0 + c, b);
#pragma unroll
            for (int e = 0; e < 32; ++e) p[c + e] += b[e];
        }
    }
#pragma unroll
    for (int s = 0; s < 64; ++s) p[s] = s0 + s <= t ? p[s] * pow_s[max(t - s0 - s, 0)] : 0.f;
    constexpr uint32_t NEXT = D;                          // columns from the first keys' accumulator to the others'
    for (int i = 0; i < halves; ++i) {
        if (i > 0) mma.wait();
        if (warp >> 2 == i) {
#pragma unroll
            for (int c = 0; c < 64; c += 8) {
                uint4 part[3];
                fs_split(p[c], p[c + 1], part[0].x, part[1].x, part[2].x);
                fs_split(p[c + 2], p[c + 3], part[0].y, part[1].y, part[2].y);
                fs_split(p[c + 4], p[c + 5], part[0].z, part[1].z, part[2].z);
                fs_split(p[c + 6], p[c + 7], part[0].w, part[1].w, part[2].w);
#pragma unroll
                for (int e = 0; e < 3; ++e)
                    *reinterpret_cast<uint4*>(xs + e * PLANE + t * 128 + ((c / 8 ^ (t & 7)) << 4)) = part[e];
            }
        }
        fv.put(ys, VPLANE, 64 * i, odd_s);
        if (i + 1 < halves) fv.fetch(v, row0, 64, rows);
        mma.operands_ready();
        if (threadIdx.x == 0) {
            const uint64_t vd = t5::desc_mnmajor(smem_u32(ys), 64 * 128);
            ch_products<PV>(4, [&](int pa, int pb, int j, bool more) {
                t5::mma_ss(first + i * NEXT, xd + ((pa * PLANE + j * 32) >> 4), vd + ((pb * VPLANE + j * 16 * 128) >> 4), ch_idesc(D, false, true), more);
            });
            t5::commit(mma.bar);
        }
    }
    mma.wait();
    // y = g^(t + 1) q S + P v: half of a row's columns a thread, through shared memory to whole rows
    float* own = reinterpret_cast<float*>(xs) + warp * 32 * PITCH;
    const uint32_t odd = odd_s[0] | odd_s[1] | odd_s[2] | odd_s[3];
    float most = 0.f;
#pragma unroll
    for (int c = 0; c < COLS; c += 32) {
        float o[32];
        t5::ld32(first + lanes + col0 + c, o);
        if (halves > 1) {
            float z[32];
            t5::ld32(first + NEXT + lanes + col0 + c, z);
#pragma unroll
            for (int e = 0; e < 32; ++e) o[e] += z[e];
        }
        if constexpr (PARTS == 1) {
            float z[32];
            t5::ld32(second + lanes + col0 + c, z);
#pragma unroll
            for (int e = 0; e < 32; ++e) o[e] = fmaf(z[e], pow_s[t + 1], o[e]);
        }
#pragma unroll
        for (int e = 0; e < 32; ++e) most = fs_largest(most, o[e]);
#pragma unroll
        for (int e = 0; e < 32; e += 4)
            *reinterpret_cast<float4*>(own + lane * PITCH + c + e) = make_float4(o[e], o[e + 1], o[e + 2], o[e + 3]);
    }
    fine &= fs_finite(most);
    // what v left out goes to the rows that see it; what came out infinite or NaN is summed again, as FMAs
    if ((odd != 0 || !fine) && t < rows) {
        float* mine = own + lane * PITCH;
        float* carried = dst + static_cast<size_t>(lane) * heads * D;
        unsigned long long again = 0;
#pragma unroll 1
        for (int c = 0; c < COLS; ++c) {
            if (fs_finite(mine[c]) && (PARTS == 1 || fs_finite(carried[c]))) continue;
            again |= 1ull << c;
            const float z = ch_dot(q, row0 + t, q_scale, st + (col0 + c) * D, D) * pow_s[t + 1];
            mine[c] = PARTS == 1 ? z : 0.f;
            if (PARTS == 2) carried[c] = z;
        }
#pragma unroll 1
        for (int s = 0; s <= t; ++s) {
            const bool left_out = odd_s[s >> 5] >> (s & 31) & 1;
            if (again == 0 && !left_out) continue;
            const float score = ch_dot(q, row0 + t, q_scale, k, row0 + s, D) * pow_s[t - s];
#pragma unroll 1
            for (int c = 0; c < COLS; ++c) {
                const float x = ch_value(v, row0 + s, col0 + c);
                if ((again >> c & 1) || (left_out && !fs_has_parts(x))) mine[c] = fmaf(score, x, mine[c]);
            }
        }
    }
    __syncwarp();
#pragma unroll 4
    for (int i = lane; i < 32 * (COLS / 4); i += 32) {
        const int r = i / (COLS / 4), c = i % (COLS / 4) * 4;
        if (r >= live) continue;
        float4 o = *reinterpret_cast<const float4*>(own + r * PITCH + c);
        float4* to = reinterpret_cast<float4*>(dst + static_cast<size_t>(r) * heads * D + c);
        if (PARTS == 2) o = make_float4(o.x + to->x, o.y + to->y, o.z + to->z, o.w + to->w);
        *to = o;
    }
    mma.end();
}

template <int D, bool SILU>
constexpr int ch_update_smem() {
    constexpr int parts = ((SILU ? 3 : 1) + 3) * 64 * D * 2, out = 8 * 32 * (D / 2 + 4) * 4;
    return (parts > out ? parts : out) + 1024;
}
constexpr int kChOutputsSmem = 6 * kChRows * 128 + 1024;

template <int D, bool SILU>
int launch_chunks(const ChRows& q, const ChRows& k, const ChRows& v, float q_scale, const float* decay, float* state,
                  const int* cu_q, const int* state_slot, const int* tile_list, int n_tiles, int n_req, int first, int heads,
                  int group, float* u, float* y, cudaStream_t stream) {
    const ChTiles tiles{tile_list, cu_q, first};
    allow_smem<chunk_update_kernel<D, SILU>>(ch_update_smem<D, SILU>());
    allow_smem<chunk_outputs_kernel<D, SILU>>(kChOutputsSmem);
    const dim3 grid(n_tiles, heads);
    launch_pdl(chunk_update_kernel<D, SILU>, grid, dim3(kChThreads), ch_update_smem<D, SILU>(), stream, k, v, decay, tiles, heads,
               group, u);
    launch_pdl(chunk_states_kernel<D>, dim3(D * D / 4 / kChThreads, heads, n_req), dim3(kChThreads), 0, stream, u, decay,
               cu_q, state_slot, state, heads);
    launch_pdl(chunk_outputs_kernel<D, SILU>, grid, dim3(kChThreads), kChOutputsSmem, stream, q, k, v, q_scale, decay,
               tiles, u, heads, group, y);
    return launch_status();
}

}  // namespace somi

using namespace somi;

// q, k: bfloat16 rows of heads / group heads of D elements, `stride` apart; v: of `heads` heads; D = 64 or 128.
// `silu`: q and k (bit 0) and v (bit 1) pass SiLU.  rot > 0: the pairs (i, i + rot / 2) of q and k turn by
// positions * rot_freq; angles: float32 scratch [portions' rows, rot].  `tiles`: int32 [n_tiles, 3] = (request,
// first row, rows <= 64) over the n_req multi-token requests, in order, request numbers from `first` on.  u: float32 scratch
// [(64 n_tiles + 127 n_req) / 128, heads, D, D].
// state: float32 [slots, heads, D, D] (value channel, key channel); y: float32 rows of heads * D.
SOMI_API int somi_matrix_state_chunks(const void* q, const void* k, const void* v, long long q_stride,
                                      long long k_stride, long long v_stride, int silu, float q_scale,
                                      const float* decay, float* state, const int* cu_q, const int* state_slot,
                                      const int* tiles, int n_tiles, int n_req, int n_rows, int heads, int group, int D,
                                      const int* positions, const double* rot_freq, int rot, float* angles, float* u,
                                      float* y, int first, cudaStream_t stream) {
    if (n_tiles <= 0 || n_req <= 0) return 0;
    const uintptr_t bits = reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(v);
    if (decay == nullptr || (rot > 0 && (positions == nullptr || rot_freq == nullptr || angles == nullptr)))
        return SOMI_ERR_UNSUPPORTED;
    if ((D != 64 && D != 128) || heads <= 0 || heads > 65535 || n_req > 65535 || group <= 0 || heads % group ||
        ((q_stride | k_stride | v_stride) & 3) || (bits & 7) || rot < 0 || rot > D || rot % 8 || (rot > 0 && (silu & 1)) ||
        ((reinterpret_cast<uintptr_t>(state) | reinterpret_cast<uintptr_t>(u) | reinterpret_cast<uintptr_t>(y)) & 15) || (reinterpret_cast<uintptr_t>(angles) & 15))
        return SOMI_ERR_UNSUPPORTED;
    float2* cs = rot > 0 ? reinterpret_cast<float2*>(angles) : nullptr;
    const int half = rot / 2, n = n_rows * half;
    if (rot > 0) launch_pdl(chunk_angles_kernel, dim3((n + 255) / 256), dim3(256), 0, stream, positions, rot_freq, half, n, cs);
    const ChRows qr{static_cast<const __nv_bfloat16*>(q), q_stride, silu & 1, cs, half};
    const ChRows kr{static_cast<const __nv_bfloat16*>(k), k_stride, silu & 1, cs, half};
    const ChRows vr{static_cast<const __nv_bfloat16*>(v), v_stride, silu >> 1 & 1, nullptr, 0};
#define SOMI_CHUNKS(D_, SILU_) \
    launch_chunks<D_, SILU_>(qr, kr, vr, q_scale, decay, state, cu_q, state_slot, tiles, n_tiles, n_req, first, heads, group, u, y, stream)
    if (D == 64) return silu & 2 ? SOMI_CHUNKS(64, true) : SOMI_CHUNKS(64, false);
    return silu & 2 ? SOMI_CHUNKS(128, true) : SOMI_CHUNKS(128, false);
#undef SOMI_CHUNKS
}

SOMI_API int somi_chunks_error() {
    int v = 0, zero = 0;
    if (cudaMemcpyFromSymbol(&v, g_chunks_error, sizeof(int)) != cudaSuccess) return -1;
    if (v) cudaMemcpyToSymbol(g_chunks_error, &zero, sizeof(int));
    return v;
}
