// Causal grouped-query attention of the float32 path over the paged cache, head sizes 64 and 128, with
// or without a window: a kernel for prompt portions and one for single-token requests, which cut the
// keys the same way and so give a row the same bits.  (Other sizes, other masks, capped scores, sinks
// and gates run the kernel in attention_generic.cu.)  The softmax is float32.
//
// A row's arithmetic: keys come in chunks of 64 aligned to position 0.  Scores and outputs of a chunk are
// products of exact bfloat16 parts with float32 sums (gemm_f32_split.cuh), 64 terms a chain of `mma.sync` steps: a score
// is the sum over a head of 64, or two such sums added, the chunk's maximum m_c and sum l_c are its own, and o_c is the sum of p v
// over its keys.  Chunks are merged in
// ascending order: with M the larger maximum, L <- L e^(M_old - M) + l_c e^(m_c - M), O likewise.  The
// prompt kernel merges in registers; the split kernel writes (m_c, l_c, o_c) and the merge kernel
// goes through them.  So how a request was cut into steps, or what else is in a step, changes no bit.  A score that comes out
// infinite or NaN is summed again as FMAs; a value that is not finite, or so large that bfloat16 rounds it to infinity, stays out of
// the products and is added to the rows that see it.
//
// Why these two shapes.  Single tokens are bound by latency and by the cache's bytes: one CTA per
// (request, key/value head, chunk) reads keys and values once for all query heads of the group, with every
// copy of the chunk in flight at once and those of older positions issued before the dependency wait.
// Portions: keys and values are split once a chunk for all rows of a CTA.  With many tiles a warp keeps 16 rows' scores,
// probabilities (which are the second product's operand as they stand) and outputs in registers; with few, 8, 4 or 2 warps share 16
// rows, so that a chunk takes less time.  What bounds the first: two warps a scheduler, about 2,200 instructions for 16 rows and
// a chunk, of which 384 are MMAs of 8 cycles each (the tensor pipe is busy a third of the time).  Layers of 14 heads of 64 with
// their products in us, 64-row tiles of FMAs before / now: 203 rows 76 / 47, 512 155 / 83, 1,024 312 / 164, 2,048 745 / 365,
// 5,000 2,864 / 1,508, 64 rows behind 2,000 positions 195 / 170; 4 single tokens behind 1,000 22.7 / 20.6.
#include "gemm_f32_split.cuh"

namespace somi {

constexpr int kF32Chunk = 64;         // keys per chunk
constexpr int kF32Rows = 64;          // query rows of a tile of the list
constexpr int kF32Heads = 8;          // query heads a split CTA takes at a time

__device__ __forceinline__ void f32_copy(float* dst, const float* src, bool in) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n"
                 ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(dst))), "l"(src), "r"(in ? 16 : 0) : "memory");
}
__device__ __forceinline__ void f32_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void f32_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// The 64 probabilities of a row from its scores, maximum and sum over the chunk: a row is four lanes', of which lane t has
// keys 8 i + 2 t and the one behind (as an MMA leaves them); a lane adds its keys in ascending order, then the lanes'
// sums meet in pairs.  A hidden key's score is -infinity.  The maximum passes over a score that is not a number, so what a key adds
// is decided by its own score: a NaN among hidden keys (m = -infinity) makes p and the sum NaN.
__device__ __forceinline__ float2 f32_chunk_softmax(float (&s)[8][2]) {
    float m = -INFINITY, l = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) m = fmaxf(m, fmaxf(s[i][0], s[i][1]));
    m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 1));
    m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 2));
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            s[i][e] = s[i][e] == -INFINITY ? 0.f : expf(s[i][e] - m);
            l = __fadd_rn(l, s[i][e]);
        }
    l = __fadd_rn(l, __shfl_xor_sync(0xffffffffu, l, 1));
    l = __fadd_rn(l, __shfl_xor_sync(0xffffffffu, l, 2));
    return make_float2(m, l);
}
// (M, L) <- (M, L) merged with a chunk's; returns the factors of the old output and of the chunk's.
__device__ __forceinline__ float2 f32_merge(float& M, float& L, float m, float l) {
    if (m == -INFINITY && l == 0.f) return make_float2(1.f, 0.f);     // the row sees nothing of the chunk
    const float top = fmaxf(M, m);
    const float2 f = make_float2(expf(M - top), expf(m - top));  // (M = -inf before the first chunk: 0)
    L = __fmaf_rn(l, f.y, __fmul_rn(L, f.x));
    M = top;
    return f;
}
__device__ __forceinline__ float f32_merge_out(float o, float oc, float2 f) {
    return __fmaf_rn(oc, f.y, __fmul_rn(o, f.x));
}

// The small products of a step, then (`f32_main`) the large one: d += a b in parts, for T tiles in turn (one tile's steps wait for
// each other; volatile asm keeps the order that is written).
template <int T>
__device__ __forceinline__ void f32_small(float (*d)[4], const uint32_t (&a)[3][4], const uint2 (&b)[T][3]) {
#pragma unroll
    for (int i = 0; i < T; ++i) mma_bf16_16816(d[i], a[2], b[i][0].x, b[i][0].y);
#pragma unroll
    for (int i = 0; i < T; ++i) mma_bf16_16816(d[i], a[0], b[i][2].x, b[i][2].y);
#pragma unroll
    for (int i = 0; i < T; ++i) mma_bf16_16816(d[i], a[1], b[i][1].x, b[i][1].y);
#pragma unroll
    for (int i = 0; i < T; ++i) mma_bf16_16816(d[i], a[1], b[i][0].x, b[i][0].y);
#pragma unroll
    for (int i = 0; i < T; ++i) mma_bf16_16816(d[i], a[0], b[i][1].x, b[i][1].y);
}
__device__ __forceinline__ void f32_main(float (&d)[4], const uint32_t (&a)[4], const uint2& b) { mma_bf16_16816(d, a, b.x, b.y); }

// A score as plain FMAs (only where the product of parts is not finite).
static __device__ __noinline__ float f32_plain_score(const float* q, float scale, const float* k, int hd) {
    float s0 = 0.f, s1 = 0.f;
    for (int d = 0; d < hd; d += 2) {
        s0 = fmaf(q[d] * scale, k[d], s0);
        s1 = fmaf(q[d + 1] * scale, k[d + 1], s1);
    }
    return s0 + s1;
}

__device__ __forceinline__ void f32_ldmatrix_pair(uint2& b, uint2& next, uint32_t addr) {
    uint32_t r[4];
    ldmatrix_x4(r, addr);
    b = make_uint2(r[0], r[1]);
    next = make_uint2(r[2], r[3]);
}
__device__ __forceinline__ void f32_ldmatrix_pair_trans(uint2& b, uint2& next, uint32_t addr) {
    uint32_t r[4];
    ldmatrix_x4_trans(r, addr);
    b = make_uint2(r[0], r[1]);
    next = make_uint2(r[2], r[3]);
}
// c ? a : b of registers (not of addresses: an array that is indexed by a variable moves to memory).
__device__ __forceinline__ float f32_select(bool c, float a, float b) {
    float d;
    asm("{\n.reg .pred p;\nsetp.ne.s32 p, %3, 0;\nselp.f32 %0, %1, %2, p;\n}\n" : "=f"(d) : "f"(a), "f"(b), "r"(static_cast<int>(c)));
    return d;
}
// Eight numbers' parts, 16 bytes each, `plane` bytes apart.
__device__ __forceinline__ void f32_put8(unsigned char* dst, int plane, const float4& u, const float4& v) {
    uint4 part[3];
    fs_split(u.x, u.y, part[0].x, part[1].x, part[2].x);
    fs_split(u.z, u.w, part[0].y, part[1].y, part[2].y);
    fs_split(v.x, v.y, part[0].z, part[1].z, part[2].z);
    fs_split(v.z, v.w, part[0].w, part[1].w, part[2].w);
#pragma unroll
    for (int e = 0; e < 3; ++e) *reinterpret_cast<uint4*>(dst + e * plane) = part[e];
}

// ------------------------------------------------------------------------- prompt portions
// Head size 64, many tiles: a CTA of four warps takes a tile of 64 rows of one head.  A warp owns 16 rows: their scores,
// probabilities and outputs stay in registers.
__global__ void __launch_bounds__(128, 2)
attention_f32_rows_kernel(const float* __restrict__ qkv, int row_stride, const float* __restrict__ kcache,
                          const float* __restrict__ vcache, const int* __restrict__ block_table,
                          int bt_stride, const int* __restrict__ cu_q, const int* __restrict__ ctx_len,
                          const int* __restrict__ tiles, int n_tiles, int nq, int nkv, int page_size,
                          float scale, int window, float* __restrict__ out) {
    constexpr int HD = 64, ROWS = kF32Rows, THREADS = 128;
    constexpr int QPLANE = ROWS * HD * 2, KPLANE = kF32Chunk * HD * 2;
    constexpr int ITEMS = kF32Chunk * HD / 8 / THREADS;                  // eights of a chunk's rows a thread
    extern __shared__ __align__(128) unsigned char f32_raw[];
    unsigned char* Qs = f32_raw;                                         // parts [3][ROWS][HD], in swizzled rows like all of them
    unsigned char* Ks = Qs + 3 * QPLANE;                                 // [3][64][HD]
    unsigned char* Vs = Ks + 3 * KPLANE;                                 // [3][64][HD]
    __shared__ unsigned wild_s[2][2];                                    // keys of a chunk with a value that has no parts
    __shared__ long long at_s[2][kF32Chunk];                             // where a chunk's keys lie, or -1
    pdl_launch_dependents();
    pdl_wait();
    const int* tile = tiles + 3 * (n_tiles - 1 - static_cast<int>(blockIdx.x));   // a prompt's last rows first
    const int req = tile[0], row0 = tile[1], rows = tile[2], head = blockIdx.y;
    const int kvh = head / (nq / nkv);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const int pos0 = ctx_len[req] + (row0 - cu_q[req]);
    const int first_key = window > 0 ? max(0, pos0 - window + 1) : 0, end_key = pos0 + rows;
    const int* bt = block_table + static_cast<size_t>(req) * bt_stride;
    auto row_of = [&](const float* cache, int j) {
        return cache + ((static_cast<size_t>(bt[j / page_size]) * nkv + kvh) * page_size + j % page_size) * HD;
    };
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    // (a row's place takes two divisions and a look into the table: once a chunk, two chunks ahead)
    auto find = [&](int c, int n) {
        const int j = c * kF32Chunk + n;
        at_s[c & 1][n] = j >= first_key && j < end_key
                             ? ((static_cast<long long>(bt[j / page_size]) * nkv + kvh) * page_size + j % page_size) * HD : -1;
    };
    auto fetch = [&](float4 (&q)[ITEMS][2], const float* cache, int c) {
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) {
            const int idx = tid + THREADS * i;
            const long long at = at_s[c & 1][idx / (HD / 8)];
            const float* src = cache + (at < 0 ? 0 : at) + idx % (HD / 8) * 8;
            q[i][0] = at < 0 ? zero : *reinterpret_cast<const float4*>(src);
            q[i][1] = at < 0 ? zero : *reinterpret_cast<const float4*>(src + 4);
        }
    };
    auto put_k = [&](const float4 (&q)[ITEMS][2]) {
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) {
            const int idx = tid + THREADS * i;
            f32_put8(Ks + swizzled_offset<HD>(idx / (HD / 8), idx % (HD / 8)), KPLANE, q[i][0], q[i][1]);
        }
    };
    auto put_v = [&](const float4 (&q)[ITEMS][2], int c) {
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) {
            const int idx = tid + THREADS * i, n = idx / (HD / 8);
            float x[8] = {q[i][0].x, q[i][0].y, q[i][0].z, q[i][0].w, q[i][1].x, q[i][1].y, q[i][1].z, q[i][1].w};
            float most = 0.f;
#pragma unroll
            for (int e = 0; e < 8; ++e) most = fs_largest(most, x[e]);
            if (!fs_has_parts(most)) {
                atomicOr(&wild_s[c & 1][n >> 5], 1u << (n & 31));
#pragma unroll
                for (int e = 0; e < 8; ++e)
                    if (!fs_has_parts(x[e])) x[e] = 0.f;
            }
            f32_put8(Vs + swizzled_offset<HD>(n, idx % (HD / 8)), KPLANE, make_float4(x[0], x[1], x[2], x[3]), make_float4(x[4], x[5], x[6], x[7]));
        }
    };
    const int c_first = first_key / kF32Chunk, c_end = (end_key + kF32Chunk - 1) / kF32Chunk;
    float4 kq[ITEMS][2], vq[ITEMS][2];
    if (tid < 2 * kF32Chunk) find(c_first + tid / kF32Chunk, tid % kF32Chunk);
    __syncthreads();
    fetch(kq, kcache, c_first);
    fetch(vq, vcache, c_first);
    for (int idx = tid; idx < ROWS * (HD / 8); idx += THREADS) {
        const int r = idx / (HD / 8), ch = idx % (HD / 8);
        float4 u = zero, v = zero;
        if (r < rows) {
            const float* src = qkv + static_cast<size_t>(row0 + r) * row_stride + head * HD + ch * 8;
            u = *reinterpret_cast<const float4*>(src);
            v = *reinterpret_cast<const float4*>(src + 4);
        }
        f32_put8(Qs + swizzled_offset<HD>(r, ch), QPLANE, make_float4(u.x * scale, u.y * scale, u.z * scale, u.w * scale),
                 make_float4(v.x * scale, v.y * scale, v.z * scale, v.w * scale));
    }
    if (tid < 4) wild_s[tid >> 1][tid & 1] = 0;
    const int r_lo = warp * 16;
    const uint32_t q_at = smem_u32(Qs), k_at = smem_u32(Ks), v_at = smem_u32(Vs);
    // (a row's chunks of 16 bytes are permuted by its last three bits: those of the lane's row)
    auto chunk_of = [](int row, int ch) { return (ch ^ (row & 7)) << 4; };
    auto q_frag = [&](uint32_t (&a)[4], int plane, int j) {              // this warp's rows, terms 16 j ..
        ldmatrix_x4(a, q_at + plane * QPLANE + (r_lo + (lane & 15)) * HD * 2 + chunk_of(lane & 7, 2 * j + (lane >> 4)));
    };
    auto k_frag = [&](uint2& b, uint2& next, int plane, int i, int j) {  // keys of tiles i and i + 1, terms 16 j ..
        const int n = i * 8 + (lane >> 4) * 8 + (lane & 7);
        f32_ldmatrix_pair(b, next, k_at + plane * KPLANE + n * HD * 2 + chunk_of(lane & 7, 2 * j + (lane >> 3 & 1)));
    };
    auto v_frag = [&](uint2& b, uint2& next, int plane, int i, int j) {  // keys 16 j .., columns of tiles i and i + 1
        f32_ldmatrix_pair_trans(b, next, v_at + plane * KPLANE + (16 * j + (lane & 15)) * HD * 2 + chunk_of(lane & 7, i + (lane >> 4)));
    };
    float O[HD / 8][4], M[2] = {-INFINITY, -INFINITY}, L[2] = {0.f, 0.f};
#pragma unroll
    for (int i = 0; i < HD / 8; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) O[i][e] = 0.f;

#pragma unroll 1
    for (int c = c_first; c < c_end; ++c) {
        __syncthreads();                                 // the chunk before has been read
        put_k(kq);
        put_v(vq, c);
        __syncthreads();
        if (c + 1 < c_end) {
            fetch(kq, kcache, c + 1);
            fetch(vq, vcache, c + 1);
        }
        if (tid < 2) wild_s[(c + 1) & 1][tid] = 0;
        if (tid < kF32Chunk) find(c + 2, tid);
        if (r_lo >= rows) continue;
        // ---- scores
        float s[8][4];
#pragma unroll
        for (int half = 0; half < HD / 64; ++half) {
            float d[8][4];
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int e = 0; e < 4; ++e) d[i][e] = 0.f;
#pragma unroll 1
            for (int j = 0; j < 4; ++j) {
                uint32_t a[3][4];
#pragma unroll
                for (int e = 0; e < 3; ++e) q_frag(a[e], e, 4 * half + j);
#pragma unroll
                for (int i = 0; i < 8; i += 4) {
                    uint2 b[4][3];
#pragma unroll
                    for (int e = 0; e < 3; ++e) {
                        k_frag(b[0][e], b[1][e], e, i, 4 * half + j);
                        k_frag(b[2][e], b[3][e], e, i + 2, 4 * half + j);
                    }
                    f32_small<4>(d + i, a, b);
                }
            }
#pragma unroll 1
            for (int j = 0; j < 4; ++j) {
                uint32_t a[4];
                q_frag(a, 0, 4 * half + j);
#pragma unroll
                for (int i = 0; i < 8; i += 2) {
                    uint2 b, b2;
                    k_frag(b, b2, 0, i, 4 * half + j);
                    f32_main(d[i], a, b);
                    f32_main(d[i + 1], a, b2);
                }
            }
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int e = 0; e < 4; ++e) s[i][e] = half == 0 ? d[i][e] : __fadd_rn(s[i][e], d[i][e]);
        }
        const int k_lo = c * kF32Chunk, p_lo = pos0 + r_lo;              // the first key's and the warp's first row's position
        const bool all_seen = k_lo + kF32Chunk - 1 <= p_lo && (window <= 0 || k_lo > p_lo + 15 - window);
        float none = 0.f;
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int e = 0; e < 4; ++e) none = fmaf(s[i][e], 0.f, none);
        if (!all_seen || none != 0.f) {
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int r = r_lo + g + 8 * (e >> 1), key = k_lo + 8 * i + 2 * t + (e & 1), pos = pos0 + r;
                    const bool seen = r < rows && key <= pos && (window <= 0 || key > pos - window);
                    if (seen && !fs_finite(s[i][e]))
                        s[i][e] = f32_plain_score(qkv + static_cast<size_t>(row0 + r) * row_stride + head * HD, scale, row_of(kcache, key), HD);
                    if (!seen) s[i][e] = -INFINITY;
                }
        }
        // ---- probabilities of rows g and g + 8
        float2 f[2];
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            float row[8][2];
#pragma unroll
            for (int i = 0; i < 8; ++i) { row[i][0] = s[i][2 * k]; row[i][1] = s[i][2 * k + 1]; }
            const float2 ml = f32_chunk_softmax(row);
#pragma unroll
            for (int i = 0; i < 8; ++i) { s[i][2 * k] = row[i][0]; s[i][2 * k + 1] = row[i][1]; }
            f[k] = f32_merge(M[k], L[k], ml.x, ml.y);
        }
        const unsigned wild0 = wild_s[c & 1][0], wild1 = wild_s[c & 1][1];
        // ---- outputs, 64 columns at a time: the probabilities are the MMA's A as they stand
#pragma unroll
        for (int part = 0; part < HD / 64; ++part) {
            float oc[8][4];
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int e = 0; e < 4; ++e) oc[i][e] = 0.f;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                uint32_t a[3][4];
                fs_split(s[2 * j][0], s[2 * j][1], a[0][0], a[1][0], a[2][0]);
                fs_split(s[2 * j][2], s[2 * j][3], a[0][1], a[1][1], a[2][1]);
                fs_split(s[2 * j + 1][0], s[2 * j + 1][1], a[0][2], a[1][2], a[2][2]);
                fs_split(s[2 * j + 1][2], s[2 * j + 1][3], a[0][3], a[1][3], a[2][3]);
#pragma unroll
                for (int i = 0; i < 8; i += 4) {
                    uint2 b[4][3];
#pragma unroll
                    for (int e = 0; e < 3; ++e) {
                        v_frag(b[0][e], b[1][e], e, 8 * part + i, j);
                        v_frag(b[2][e], b[3][e], e, 8 * part + i + 2, j);
                    }
                    f32_small<4>(oc + i, a, b);
                }
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const uint32_t a[4] = {pack_bf16(s[2 * j][0], s[2 * j][1]), pack_bf16(s[2 * j][2], s[2 * j][3]),
                                       pack_bf16(s[2 * j + 1][0], s[2 * j + 1][1]), pack_bf16(s[2 * j + 1][2], s[2 * j + 1][3])};
#pragma unroll
                for (int i = 0; i < 8; i += 2) {
                    uint2 b, b2;
                    v_frag(b, b2, 0, 8 * part + i, j);
                    f32_main(oc[i], a, b);
                    f32_main(oc[i + 1], a, b2);
                }
            }
            if (wild0 | wild1) {                         // values without parts, to the rows that see them
#pragma unroll 1
                for (int n = 0; n < kF32Chunk; ++n) {
                    if (!((n < 32 ? wild0 : wild1) >> (n & 31) & 1)) continue;
                    const int key = k_lo + n;
                    float p0 = 0.f, p1 = 0.f;
#pragma unroll
                    for (int i = 0; i < 8; ++i)
                        {
                            p0 = f32_select(n == 8 * i + (n & 6), s[i][0], f32_select(n == 8 * i + (n & 6) + 1, s[i][1], p0));
                            p1 = f32_select(n == 8 * i + (n & 6), s[i][2], f32_select(n == 8 * i + (n & 6) + 1, s[i][3], p1));
                        }
                    p0 = __shfl_sync(0xffffffffu, p0, (lane & ~3) | (n & 7) >> 1);
                    p1 = __shfl_sync(0xffffffffu, p1, (lane & ~3) | (n & 7) >> 1);
                    const float* v = row_of(vcache, key) + 64 * part + 2 * t;
#pragma unroll 1
                    for (int e = 0; e < 4; ++e) {
                        const int r = r_lo + g + 8 * (e >> 1), pos = pos0 + r;
                        if (r >= rows || key > pos || (window > 0 && key <= pos - window)) continue;
#pragma unroll
                        for (int i = 0; i < 8; ++i) {
                            const float x = v[8 * i + (e & 1)];
                            if (fs_has_parts(x)) continue;
#pragma unroll
                            for (int k = 0; k < 4; ++k) oc[i][k] = f32_select(k == e, __fmaf_rn(e < 2 ? p0 : p1, x, oc[i][k]), oc[i][k]);
                        }
                    }
                }
            }
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int e = 0; e < 4; ++e) O[8 * part + i][e] = f32_merge_out(O[8 * part + i][e], oc[i][e], f[e >> 1]);
        }
    }
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const int r = r_lo + g + 8 * k;
        if (r >= rows) continue;
        float* dst = out + static_cast<size_t>(row0 + r) * (nq * HD) + head * HD + 2 * t;
#pragma unroll
        for (int i = 0; i < HD / 8; ++i)
            *reinterpret_cast<float2*>(dst + 8 * i) = make_float2(O[i][2 * k] / L[k], O[i][2 * k + 1] / L[k]);
    }
}

// The same for few tiles: a CTA takes 16 RI rows of a tile of 64 (a share of it), and 8 / RI warps share 16 rows, a
// part of the keys each, then of the columns; scores and probabilities pass through shared memory.
template <int HD, int RI>
__device__ __forceinline__ void
f32_shares(int tile_at, int head, int part, const float* __restrict__ qkv, int row_stride, const float* __restrict__ kcache,
           const float* __restrict__ vcache, const int* __restrict__ block_table, int bt_stride, const int* __restrict__ cu_q,
           const int* __restrict__ ctx_len, const int* __restrict__ tiles, int nq, int nkv, int page_size, float scale,
           int window, float* __restrict__ out) {
    constexpr int ROWS = 16 * RI, PP = kF32Chunk + 4;
    constexpr int ACROSS = 8 / RI, KT = 8 / ACROSS, OT = HD / 8 / ACROSS;          // n8 tiles of keys and columns for a warp
    constexpr int QPLANE = ROWS * HD * 2, KPLANE = kF32Chunk * HD * 2, PPLANE = ROWS * 128;
    constexpr int ITEMS = kF32Chunk * HD / 8 / 256;                      // eights of a chunk's rows a thread
    extern __shared__ __align__(128) unsigned char f32_raw[];
    unsigned char* Qs = f32_raw;                                         // parts [3][ROWS][HD], in swizzled rows like all of them
    unsigned char* Ks = Qs + 3 * QPLANE;                                 // [3][64][HD]
    unsigned char* Vs = Ks + 3 * KPLANE;                                 // [3][64][HD]
    unsigned char* Ps = Vs + 3 * KPLANE;                                 // [3][ROWS][64]
    float* Ss = reinterpret_cast<float*>(Ps + 3 * PPLANE);               // [ROWS][PP]
    __shared__ float M_s[ROWS], L_s[ROWS];
    __shared__ float2 f_s[ROWS];
    __shared__ unsigned wild_s[2][2];
    __shared__ long long at_s[2][kF32Chunk];
    pdl_launch_dependents();
    pdl_wait();
    const int* tile = tiles + 3 * tile_at;
    const int req = tile[0], row0 = tile[1] + part * ROWS;
    const int rows = min(ROWS, tile[2] - part * ROWS);
    if (rows <= 0) return;
    const int kvh = head / (nq / nkv);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const int pos0 = ctx_len[req] + (row0 - cu_q[req]);
    const int first_key = window > 0 ? max(0, pos0 - window + 1) : 0, end_key = pos0 + rows;
    const int* bt = block_table + static_cast<size_t>(req) * bt_stride;
    auto row_of = [&](const float* cache, int j) {
        return cache + ((static_cast<size_t>(bt[j / page_size]) * nkv + kvh) * page_size + j % page_size) * HD;
    };
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    auto find = [&](int c, int n) {
        const int j = c * kF32Chunk + n;
        at_s[c & 1][n] = j >= first_key && j < end_key
                             ? ((static_cast<long long>(bt[j / page_size]) * nkv + kvh) * page_size + j % page_size) * HD : -1;
    };
    // a thread's eights of a chunk: in registers a chunk ahead, then in parts to shared memory
    float4 kq[ITEMS][2], vq[ITEMS][2];
    auto fetch = [&](float4 (&q)[ITEMS][2], const float* cache, int c) {
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) {
            const int idx = tid + 256 * i;
            const long long at = at_s[c & 1][idx / (HD / 8)];
            const float* src = cache + (at < 0 ? 0 : at) + idx % (HD / 8) * 8;
            q[i][0] = at < 0 ? zero : *reinterpret_cast<const float4*>(src);
            q[i][1] = at < 0 ? zero : *reinterpret_cast<const float4*>(src + 4);
        }
    };
    auto put_k = [&]() {
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) {
            const int idx = tid + 256 * i;
            f32_put8(Ks + swizzled_offset<HD>(idx / (HD / 8), idx % (HD / 8)), KPLANE, kq[i][0], kq[i][1]);
        }
    };
    auto put_v = [&](int c) {
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) {
            const int idx = tid + 256 * i, n = idx / (HD / 8);
            float x[8] = {vq[i][0].x, vq[i][0].y, vq[i][0].z, vq[i][0].w, vq[i][1].x, vq[i][1].y, vq[i][1].z, vq[i][1].w};
            float most = 0.f;
#pragma unroll
            for (int e = 0; e < 8; ++e) most = fs_largest(most, x[e]);
            if (!fs_has_parts(most)) {
                atomicOr(&wild_s[c & 1][n >> 5], 1u << (n & 31));
#pragma unroll
                for (int e = 0; e < 8; ++e)
                    if (!fs_has_parts(x[e])) x[e] = 0.f;
            }
            f32_put8(Vs + swizzled_offset<HD>(n, idx % (HD / 8)), KPLANE, make_float4(x[0], x[1], x[2], x[3]), make_float4(x[4], x[5], x[6], x[7]));
        }
    };
    const int c_first = first_key / kF32Chunk, c_end = (end_key + kF32Chunk - 1) / kF32Chunk;
    if (tid < 2 * kF32Chunk) find(c_first + tid / kF32Chunk, tid % kF32Chunk);
    if (tid < 4) wild_s[tid >> 1][tid & 1] = 0;
    if (tid < ROWS) { M_s[tid] = -INFINITY; L_s[tid] = 0.f; }
    __syncthreads();
    fetch(kq, kcache, c_first);
    fetch(vq, vcache, c_first);
    for (int idx = tid; idx < ROWS * (HD / 8); idx += 256) {
        const int r = idx / (HD / 8), ch = idx % (HD / 8);
        float4 u = zero, v = zero;
        if (r < rows) {
            const float* src = qkv + static_cast<size_t>(row0 + r) * row_stride + head * HD + ch * 8;
            u = *reinterpret_cast<const float4*>(src);
            v = *reinterpret_cast<const float4*>(src + 4);
        }
        f32_put8(Qs + swizzled_offset<HD>(r, ch), QPLANE, make_float4(u.x * scale, u.y * scale, u.z * scale, u.w * scale),
                 make_float4(v.x * scale, v.y * scale, v.z * scale, v.w * scale));
    }
    put_k();
    if (c_first + 1 < c_end) fetch(kq, kcache, c_first + 1);
    // this warp's 16 rows; its keys from 8 KT (warp % ACROSS) on, its columns from 8 OT (warp % ACROSS) on
    const int r_lo = warp / ACROSS * 16, share = warp % ACROSS;
    const uint32_t q_at = smem_u32(Qs), k_at = smem_u32(Ks), v_at = smem_u32(Vs), p_at = smem_u32(Ps);
    float O[OT][4];
#pragma unroll
    for (int i = 0; i < OT; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) O[i][e] = 0.f;
    __syncthreads();

    for (int c = c_first; c < c_end; ++c) {
        // ---- scores
        float s[KT][4];
        auto q_frag = [&](uint32_t (&a)[4], int plane, int j) {          // rows r_lo .., terms 16 j ..
            ldmatrix_x4(a, q_at + plane * QPLANE + swizzled_offset<HD>(r_lo + (lane & 15), 2 * j + (lane >> 4)));
        };
        auto k_frag = [&](uint2& b, int plane, int i, int j) {           // keys of tile i, terms 16 j ..
            const int n = (share * KT + i) * 8 + (lane & 7);
            asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0,%1}, [%2];\n"
                         : "=r"(b.x), "=r"(b.y)
                         : "r"(k_at + plane * KPLANE + swizzled_offset<HD>(n, 2 * j + (lane >> 3 & 1))));
        };
#pragma unroll
        for (int half = 0; half < HD / 64; ++half) {
            float d[KT][4];
#pragma unroll
            for (int i = 0; i < KT; ++i)
#pragma unroll
                for (int e = 0; e < 4; ++e) d[i][e] = 0.f;
            uint32_t a0[4][4];
            uint2 b0[4][KT];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                uint32_t a[3][4];
                uint2 b[KT][3];
#pragma unroll
                for (int e = 0; e < 3; ++e) {
                    q_frag(a[e], e, 4 * half + j);
#pragma unroll
                    for (int i = 0; i < KT; ++i) k_frag(b[i][e], e, i, 4 * half + j);
                }
                f32_small<KT>(d, a, b);
#pragma unroll
                for (int i = 0; i < KT; ++i) b0[j][i] = b[i][0];
#pragma unroll
                for (int e = 0; e < 4; ++e) a0[j][e] = a[0][e];
            }
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int i = 0; i < KT; ++i) f32_main(d[i], a0[j], b0[j][i]);
#pragma unroll
            for (int i = 0; i < KT; ++i)
#pragma unroll
                for (int e = 0; e < 4; ++e) s[i][e] = half == 0 ? d[i][e] : __fadd_rn(s[i][e], d[i][e]);
        }
#pragma unroll
        for (int i = 0; i < KT; ++i)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int r = r_lo + g + 8 * (e >> 1), n = (share * KT + i) * 8 + 2 * t + (e & 1), key = c * kF32Chunk + n, pos = pos0 + r;
                const bool seen = r < rows && key <= pos && (window <= 0 || key > pos - window);
                float x = s[i][e];
                if (seen && !fs_finite(x))
                    x = f32_plain_score(qkv + static_cast<size_t>(row0 + r) * row_stride + head * HD, scale, row_of(kcache, key), HD);
                Ss[r * PP + n] = seen ? x : -INFINITY;
            }
        __syncthreads();                                 // (the values and probabilities before have been read, too)
        put_v(c);
        if (c + 1 < c_end) {
            put_k();
            fetch(vq, vcache, c + 1);
        }
        {   // 2 RI rows a warp, four lanes each (with fewer than eight some lanes repeat the others)
            const int r = warp * 2 * RI + g % (2 * RI);
            float row[8][2];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const float2 x = *reinterpret_cast<const float2*>(Ss + r * PP + 8 * i + 2 * t);
                row[i][0] = x.x;
                row[i][1] = x.y;
            }
            const float2 ml = f32_chunk_softmax(row);
            if (g < 2 * RI) {
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    uint32_t part[3];
                    fs_split(row[i][0], row[i][1], part[0], part[1], part[2]);
#pragma unroll
                    for (int e = 0; e < 3; ++e) *reinterpret_cast<uint32_t*>(Ps + e * PPLANE + swizzled_offset<64>(r, i) + 4 * t) = part[e];
                }
                if (t == 0) {
                    float M = M_s[r], L = L_s[r];
                    f_s[r] = f32_merge(M, L, ml.x, ml.y);
                    M_s[r] = M;
                    L_s[r] = L;
                }
            }
        }
        if (tid < 2) wild_s[(c + 1) & 1][tid] = 0;
        if (tid < kF32Chunk) find(c + 2, tid);           // (chunk c's places have been read)
        __syncthreads();
        if (c + 2 < c_end) fetch(kq, kcache, c + 2);
        // ---- outputs
        float oc[OT][4];
#pragma unroll
        for (int i = 0; i < OT; ++i)
#pragma unroll
            for (int e = 0; e < 4; ++e) oc[i][e] = 0.f;
        {
            auto p_frag = [&](uint32_t (&a)[4], int plane, int j) {
                ldmatrix_x4(a, p_at + plane * PPLANE + swizzled_offset<64>(r_lo + (lane & 15), 2 * j + (lane >> 4)));
            };
            auto v_frag = [&](uint2& b, int plane, int i, int j) {       // keys 16 j .., columns of tile i
                asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0,%1}, [%2];\n"
                             : "=r"(b.x), "=r"(b.y)
                             : "r"(v_at + plane * KPLANE + swizzled_offset<HD>(16 * j + (lane & 15), share * OT + i)));
            };
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                uint32_t a[3][4];
                uint2 b[OT][3];
#pragma unroll
                for (int e = 0; e < 3; ++e) {
                    p_frag(a[e], e, j);
#pragma unroll
                    for (int i = 0; i < OT; ++i) v_frag(b[i][e], e, i, j);
                }
                f32_small<OT>(oc, a, b);
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                uint32_t a[4];
                p_frag(a, 0, j);
#pragma unroll
                for (int i = 0; i < OT; ++i) {
                    uint2 b;
                    v_frag(b, 0, i, j);
                    f32_main(oc[i], a, b);
                }
            }
        }
        if (wild_s[c & 1][0] | wild_s[c & 1][1]) {
#pragma unroll 1
            for (int n = 0; n < kF32Chunk; ++n) {
                if (!(wild_s[c & 1][n >> 5] >> (n & 31) & 1)) continue;
                const int key = c * kF32Chunk + n;
                const float* v = row_of(vcache, key);
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int r = r_lo + g + 8 * (e >> 1), pos = pos0 + r;
                    if (r >= rows || key > pos || (window > 0 && key <= pos - window)) continue;
                    float p = 0.f;
#pragma unroll
                    for (int k = 2; k >= 0; --k)
                        p += __bfloat162float(*reinterpret_cast<const __nv_bfloat16*>(Ps + k * PPLANE + swizzled_offset<64>(r, n >> 3) + (n & 7) * 2));
#pragma unroll
                    for (int i = 0; i < OT; ++i) {
                        const float x = v[(share * OT + i) * 8 + 2 * t + (e & 1)];
                        if (!fs_has_parts(x)) oc[i][e] = __fmaf_rn(p, x, oc[i][e]);
                    }
                }
            }
        }
        const float2 f0 = f_s[r_lo + g], f1 = f_s[r_lo + g + 8];
#pragma unroll
        for (int i = 0; i < OT; ++i)
#pragma unroll
            for (int e = 0; e < 4; ++e) O[i][e] = f32_merge_out(O[i][e], oc[i][e], e < 2 ? f0 : f1);
    }
#pragma unroll
    for (int e = 0; e < 4; e += 2) {
        const int r = r_lo + g + 4 * e;
        if (r >= rows) continue;
        const float L = L_s[r];
        float* dst = out + static_cast<size_t>(row0 + r) * (nq * HD) + head * HD + share * OT * 8 + 2 * t;
#pragma unroll
        for (int i = 0; i < OT; ++i) *reinterpret_cast<float2*>(dst + 8 * i) = make_float2(O[i][e] / L, O[i][e + 1] / L);
    }
}

template <int HD, int RI>
__global__ void __launch_bounds__(256, HD == 64 ? 2 : 1)
attention_f32_shares_kernel(const float* __restrict__ qkv, int row_stride, const float* __restrict__ kcache,
                            const float* __restrict__ vcache, const int* __restrict__ block_table,
                            int bt_stride, const int* __restrict__ cu_q, const int* __restrict__ ctx_len,
                            const int* __restrict__ tiles, int n_tiles, int nq, int nkv, int page_size,
                            float scale, int window, float* __restrict__ out) {
    f32_shares<HD, RI>(n_tiles - 1 - static_cast<int>(blockIdx.x), blockIdx.y, blockIdx.z, qkv, row_stride, kcache, vcache,
                       block_table, bt_stride, cu_q, ctx_len, tiles, nq, nkv, page_size, scale, window, out);   // a prompt's last rows first
}

// ------------------------------------------------------------------- single-token requests
// part_o [request][query head][chunk][HD], part_ml likewise with (m, l); a request's chunks are counted from the
// one of its first visible key, so that a window needs no more of them than it reaches.
template <int HD>
__device__ __forceinline__ void
f32_single(int at, int kvh, int i, const float* __restrict__ qkv, int row_stride, int row_base, int req_base,
           const float* __restrict__ kcache, const float* __restrict__ vcache, const int* __restrict__ block_table, int bt_stride,
           const int* __restrict__ ctx_len, int nq, int nkv, int page_size, float scale, int window, int max_chunks,
           float* __restrict__ part_o, float2* __restrict__ part_ml) {
    constexpr int P = HD + 4, PP = kF32Chunk + 4;
    constexpr int QUADS = HD / 4, OT = HD / 32;          // n8 tiles of columns a warp
    extern __shared__ __align__(16) float f32_smem[];
    float* Vs = f32_smem;                // [64][P]
    float* Ps = Vs + kF32Chunk * P;      // [8][PP]
    pdl_launch_dependents();
    const int req = req_base + i;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const int pos = ld_step(ctx_len + req);              // [descriptor]
    const int first_key = window > 0 ? max(0, pos - window + 1) : 0;
    const int c = first_key / kF32Chunk + at;
    if (c * kF32Chunk > pos) {
        pdl_wait();
        return;
    }
    const int* bt = block_table + static_cast<size_t>(req) * bt_stride;
    auto row_of = [&](const float* cache, int j) {
        return cache + ((static_cast<size_t>(ld_step(bt + j / page_size)) * nkv + kvh) * page_size + j % page_size) * HD;
    };
    // every position but the step's own is there already: keys to registers (two tiles of eight a warp, four terms of a step
    // a lane; a step's terms may stand in any order), values to shared memory
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    float4 kq[2][HD / 16];
    const int own = pos - c * kF32Chunk;                 // where the step's own key stands, if in this chunk
    auto fetch_k = [&](bool late) {
#pragma unroll
        for (int n8 = 0; n8 < 2; ++n8) {
            const int n = warp * 16 + n8 * 8 + g, j = c * kF32Chunk + n;
            if ((n == own) != late) continue;
            const bool in = j >= first_key && j <= pos;
            const float* src = in ? row_of(kcache, j) + 4 * t : kcache;
#pragma unroll
            for (int d = 0; d < HD / 16; ++d) kq[n8][d] = in ? __ldcg(reinterpret_cast<const float4*>(src + 16 * d)) : zero;
        }
    };
    auto load_v = [&](int from, int to) {
        for (int idx = tid; idx < kF32Chunk * QUADS; idx += 128) {
            const int n = idx / QUADS, d = idx % QUADS * 4, j = c * kF32Chunk + n;
            if (n < from || n >= to) continue;
            const bool in = j >= first_key && j <= pos;
            f32_copy(Vs + n * P + d, in ? row_of(vcache, j) + d : vcache, in);
        }
    };
    fetch_k(false);                                      // [descriptor], [old-cache]
    load_v(0, min(kF32Chunk, own));
    pdl_wait();
    fetch_k(true);
    load_v(min(kF32Chunk, own), kF32Chunk);
    f32_commit();
    const int group = nq / nkv;
    const float* q_row = qkv + static_cast<size_t>(row_base + i) * row_stride + static_cast<size_t>(kvh) * group * HD;
    for (int h0 = 0; h0 < group; h0 += kF32Heads) {
        const int heads = min(kF32Heads, group - h0);
        if (h0) __syncthreads();
        // ---- scores of head g (rows 8 .. 15 of the MMA are zero) and this warp's 16 keys
        float4 qq[HD / 16];
#pragma unroll
        for (int d = 0; d < HD / 16; ++d) {
            const float4 q = g < heads ? *reinterpret_cast<const float4*>(q_row + (h0 + g) * HD + 16 * d + 4 * t) : zero;
            qq[d] = make_float4(q.x * scale, q.y * scale, q.z * scale, q.w * scale);
        }
        float s[2][4];
#pragma unroll
        for (int half = 0; half < HD / 64; ++half) {
            float d[2][4] = {};
            uint32_t a0[4][4];
            uint2 b0[4][2];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float4 q = qq[4 * half + j];
                uint32_t a[3][4] = {};
                fs_split(q.x, q.y, a[0][0], a[1][0], a[2][0]);
                fs_split(q.z, q.w, a[0][2], a[1][2], a[2][2]);
                uint2 b[2][3];
#pragma unroll
                for (int n8 = 0; n8 < 2; ++n8) {
                    const float4 k = kq[n8][4 * half + j];
                    fs_split(k.x, k.y, b[n8][0].x, b[n8][1].x, b[n8][2].x);
                    fs_split(k.z, k.w, b[n8][0].y, b[n8][1].y, b[n8][2].y);
                    b0[j][n8] = b[n8][0];
                }
                f32_small<2>(d, a, b);
#pragma unroll
                for (int e = 0; e < 4; ++e) a0[j][e] = a[0][e];
            }
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int n8 = 0; n8 < 2; ++n8) f32_main(d[n8], a0[j], b0[j][n8]);
#pragma unroll
            for (int n8 = 0; n8 < 2; ++n8)
#pragma unroll
                for (int e = 0; e < 2; ++e) s[n8][e] = half == 0 ? d[n8][e] : __fadd_rn(s[n8][e], d[n8][e]);
        }
#pragma unroll
        for (int n8 = 0; n8 < 2; ++n8)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int n = warp * 16 + n8 * 8 + 2 * t + e, key = c * kF32Chunk + n;
                const bool seen = key >= first_key && key <= pos;
                float x = s[n8][e];
                if (seen && g < heads && !fs_finite(x)) x = f32_plain_score(q_row + (h0 + g) * HD, scale, row_of(kcache, key), HD);
                Ps[g * PP + n] = seen ? x : -INFINITY;
            }
        f32_wait<0>();
        __syncthreads();
        {   // two rows a warp, four lanes each (the other lanes repeat them)
            const int r = warp * 2 + (g & 1);
            float row[8][2];
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const float2 x = *reinterpret_cast<const float2*>(Ps + r * PP + 8 * k + 2 * t);
                row[k][0] = x.x;
                row[k][1] = x.y;
            }
            const float2 ml = f32_chunk_softmax(row);
            __syncwarp();
            if (g < 2) {
#pragma unroll
                for (int k = 0; k < 8; ++k) *reinterpret_cast<float2*>(Ps + r * PP + 8 * k + 2 * t) = make_float2(row[k][0], row[k][1]);
                if (t == 0 && r < heads)
                    part_ml[(static_cast<size_t>(i) * nq + kvh * group + h0 + r) * max_chunks + at] = ml;
            }
        }
        __syncthreads();
        // ---- outputs of head g and this warp's columns; keys 16 j + 4 t .. of a step a lane
        float o[OT][4];
#pragma unroll
        for (int n8 = 0; n8 < OT; ++n8)
#pragma unroll
            for (int e = 0; e < 4; ++e) o[n8][e] = 0.f;
        uint32_t a0[4][4];
        uint2 b0[4][OT];
        bool wild = false;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float4 p = *reinterpret_cast<const float4*>(Ps + g * PP + 16 * j + 4 * t);
            uint32_t a[3][4] = {};
            fs_split(p.x, p.y, a[0][0], a[1][0], a[2][0]);
            fs_split(p.z, p.w, a[0][2], a[1][2], a[2][2]);
            uint2 b[OT][3];
#pragma unroll
            for (int n8 = 0; n8 < OT; ++n8) {
                const float* src = Vs + (16 * j + 4 * t) * P + (warp * OT + n8) * 8 + g;
                float v[4];
#pragma unroll
                for (int m = 0; m < 4; ++m) {
                    v[m] = src[m * P];
                    if (!fs_has_parts(v[m])) {
                        wild = true;
                        v[m] = 0.f;
                    }
                }
                fs_split(v[0], v[1], b[n8][0].x, b[n8][1].x, b[n8][2].x);
                fs_split(v[2], v[3], b[n8][0].y, b[n8][1].y, b[n8][2].y);
                b0[j][n8] = b[n8][0];
            }
            f32_small<OT>(o, a, b);
#pragma unroll
            for (int e = 0; e < 4; ++e) a0[j][e] = a[0][e];
        }
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int n8 = 0; n8 < OT; ++n8) f32_main(o[n8], a0[j], b0[j][n8]);
        if (__any_sync(0xffffffffu, wild)) {             // values without parts, one by one
#pragma unroll 1
            for (int n = 0; n < kF32Chunk; ++n) {
                const int key = c * kF32Chunk + n;
                if (key < first_key || key > pos) continue;
#pragma unroll
                for (int n8 = 0; n8 < OT; ++n8)
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        const float x = Vs[n * P + (warp * OT + n8) * 8 + 2 * t + e];
                        if (!fs_has_parts(x)) o[n8][e] = __fmaf_rn(Ps[g * PP + n], x, o[n8][e]);
                    }
            }
        }
        if (g < heads) {
            float* dst = part_o + ((static_cast<size_t>(i) * nq + kvh * group + h0 + g) * max_chunks + at) * HD + warp * OT * 8 + 2 * t;
#pragma unroll
            for (int n8 = 0; n8 < OT; ++n8) *reinterpret_cast<float2*>(dst + 8 * n8) = make_float2(o[n8][0], o[n8][1]);
        }
    }
}

// A CTA's work is a chain of loads and small products, so CTAs beside each other hide it, and five an SM in 96 registers (which cost
// 120 bytes of spills), three with 128 columns, are faster than the three and two that take what registers they like.  Layers in us, as
// FMAs / three or two an SM / now: 14 heads over 2 of 64, 1 token behind 8,000 30.9 / 39.0 / 32.7, 16 behind 4,000 57.9 / 59.8 / 51.7, 64 behind 2,000
// 95.1 / 102.6 / 85.1; 28 over 4 of 128, 8 behind 2,048 98.8 / 85.2 / 78.4.
template <int HD>
__global__ void __launch_bounds__(128, HD == 64 ? 5 : 3)
attention_f32_split_kernel(const float* __restrict__ qkv, int row_stride, int row_base, int req_base,
                           const float* __restrict__ kcache, const float* __restrict__ vcache,
                           const int* __restrict__ block_table, int bt_stride, const int* __restrict__ ctx_len,
                           int nq, int nkv, int page_size, float scale, int window, int max_chunks,
                           float* __restrict__ part_o, float2* __restrict__ part_ml) {
    f32_single<HD>(blockIdx.x, blockIdx.y, blockIdx.z, qkv, row_stride, row_base, req_base, kcache, vcache, block_table, bt_stride,
                   ctx_len, nq, nkv, page_size, scale, window, max_chunks, part_o, part_ml);
}

// Portions and single tokens of a step in one launch (head size 64): the portions' CTAs first, then one per (chunk, kv head, request), whose
// upper four warps have nothing to do.  Both parts' registers are more than 128: 72 to 92 bytes are spilled.
template <int RI>
__global__ void __launch_bounds__(256, 2)
attention_f32_mixed_kernel(const float* __restrict__ qkv, int row_stride, const float* __restrict__ kcache,
                           const float* __restrict__ vcache, const int* __restrict__ block_table, int bt_stride,
                           const int* __restrict__ cu_q, const int* __restrict__ ctx_len, const int* __restrict__ tiles,
                           int n_tiles, int nq, int nkv, int page_size, float scale, int window, float* __restrict__ out,
                           int row_base, int req_base, int max_chunks, float* __restrict__ part_o,
                           float2* __restrict__ part_ml) {
    const int portion = n_tiles * nq * (4 / RI);
    int b = blockIdx.x;
    if (b < portion) {
        f32_shares<64, RI>(n_tiles - 1 - b % n_tiles, b / n_tiles % nq, b / (n_tiles * nq), qkv, row_stride, kcache, vcache,
                           block_table, bt_stride, cu_q, ctx_len, tiles, nq, nkv, page_size, scale, window, out);
        return;
    }
    if (threadIdx.x >= 128) return;                      // (whole warps: barriers count the threads that are left)
    b -= portion;
    f32_single<64>(b % max_chunks, b / max_chunks % nkv, b / (max_chunks * nkv), qkv, row_stride, row_base, req_base, kcache,
                   vcache, block_table, bt_stride, ctx_len, nq, nkv, page_size, scale, window, max_chunks, part_o, part_ml);
}

template <int HD>
__global__ void __launch_bounds__(HD)
attention_f32_merge_kernel(const float* __restrict__ part_o, const float2* __restrict__ part_ml, int max_chunks,
                           const int* __restrict__ ctx_len, int row_base, int req_base, int nq, int window,
                           float* __restrict__ out) {
    const int i = blockIdx.x, head = blockIdx.y, d = threadIdx.x;
    pdl_launch_dependents();
    pdl_wait();
    const int pos = ctx_len[req_base + i];
    const int end = pos / kF32Chunk + 1 - (window > 0 ? max(0, pos - window + 1) : 0) / kF32Chunk;
    const size_t base = (static_cast<size_t>(i) * nq + head) * max_chunks;
    float M = -INFINITY, L = 0.f, O = 0.f;
    for (int c0 = 0; c0 < end; c0 += 8) {            // eight chunks' loads in flight
        float2 ml[8];
        float o[8];
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            const bool in = c0 + c < end;
            ml[c] = in ? part_ml[base + c0 + c] : make_float2(-INFINITY, 0.f);
            o[c] = in ? part_o[(base + c0 + c) * HD + d] : 0.f;
        }
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            const float2 f = f32_merge(M, L, ml[c].x, ml[c].y);
            O = f32_merge_out(O, o[c], f);
        }
    }
    out[static_cast<size_t>(row_base + i) * nq * HD + head * HD + d] = O / L;
}

template <int HD>
constexpr int f32_rows_smem(int rows) { return 3 * 2 * HD * (rows + 2 * kF32Chunk); }
template <int HD>
constexpr int f32_shares_smem(int rows) { return f32_rows_smem<HD>(rows) + 3 * 2 * rows * kF32Chunk + 4 * rows * (kF32Chunk + 4); }
template <int HD>
constexpr int f32_split_smem() { return 4 * (kF32Chunk * (HD + 4) + kF32Heads * (kF32Chunk + 4)); }

static_assert(f32_split_smem<64>() <= f32_shares_smem<64>(16), "a launch of both has the portions' shared memory");

}  // namespace somi

using namespace somi;

SOMI_API int somi_attention_f32_chunk() { return kF32Chunk; }

// Whether these sizes and addresses are this file's (16-byte rows of queries, keys and values).
SOMI_API int somi_attention_f32_supported(const float* qkv, const float* kcache, const float* vcache,
                                          const float* out, int row_stride, int nq, int nkv, int hd) {
    const uintptr_t bits = reinterpret_cast<uintptr_t>(qkv) | reinterpret_cast<uintptr_t>(kcache) |
                           reinterpret_cast<uintptr_t>(vcache) | reinterpret_cast<uintptr_t>(out);
    return (hd == 64 || hd == 128) && nkv > 0 && nq % nkv == 0 && nq <= 65535 && row_stride % 4 == 0 && (bits & 15) == 0;
}

// Few tiles: two or four CTAs share one, each with a part of its rows; many: a warp keeps 16 rows to itself (the same
// bits).  Layer of 14 heads over 2 of 64, 4 / 2 shares / rows in us: 203 rows (56 tiles and heads) 47 / 51 / 62, 64 rows behind
// 2,000 positions (14) 170 / 197 / 266, 300 behind 100 (70) 66 / 71 / 91, 512 (112) 92 / 83 / 103, 1,024 (224) 205 / 164 /
// 171, 2,048 (448) 585 / 413 / 365, 5,000 (1,106) 2,924 / 1,892 / 1,508.
static int f32_shares_of(int n_tiles, int nq) {
    const long long ctas = static_cast<long long>(n_tiles) * nq;
    return ctas <= 100 ? 4 : (ctas <= 148 * 2 ? 2 : 1);
}

// Prompt portions: the tile list's query tiles are at most 64 rows.
SOMI_API int somi_attention_f32_portion(const float* qkv, int row_stride, const float* kcache, const float* vcache,
                                        const int* block_table, int bt_stride, const int* cu_q, const int* ctx_len,
                                        const int* tiles, int n_tiles, int nq, int nkv, int hd, int page_size,
                                        float scale, int window, float* out, cudaStream_t stream) {
    if (n_tiles <= 0) return 0;
    if (!somi_attention_f32_supported(qkv, kcache, vcache, out, row_stride, nq, nkv, hd) || page_size <= 0)
        return SOMI_ERR_UNSUPPORTED;
    const int shares = f32_shares_of(n_tiles, nq);
#define SOMI_F32_PORTION(KERNEL, THREADS, SHARES, SMEM) \
    (allow_smem<KERNEL>(SMEM), launch_pdl(KERNEL, dim3(n_tiles, nq, SHARES), dim3(THREADS), SMEM, stream, qkv, row_stride, kcache, \
                                          vcache, block_table, bt_stride, cu_q, ctx_len, tiles, n_tiles, nq, nkv, page_size, \
                                          scale, window, out))
#define SOMI_F32_SHARES(HD, RI) SOMI_F32_PORTION((attention_f32_shares_kernel<HD, RI>), 256, 4 / RI, f32_shares_smem<HD>(16 * RI))
    if (hd == 64) {
        if (shares == 1) SOMI_F32_PORTION(attention_f32_rows_kernel, 128, 1, f32_rows_smem<64>(kF32Rows));
        else if (shares == 2) SOMI_F32_SHARES(64, 2);
        else SOMI_F32_SHARES(64, 1);
    } else {
        if (shares == 1) SOMI_F32_SHARES(128, 4);
        else if (shares == 2) SOMI_F32_SHARES(128, 2);
        else SOMI_F32_SHARES(128, 1);
    }
#undef SOMI_F32_SHARES
#undef SOMI_F32_PORTION
    return launch_status();
}

// Single-token requests: request req_base + i, row row_base + i.  part: n_decode * nq * max_chunks * (hd + 2)
// floats, max_chunks at least the chunks that the longest request's token sees keys of.
SOMI_API int somi_attention_f32_single(const float* qkv, int row_stride, int row_base, int req_base, int n_decode,
                                       const float* kcache, const float* vcache, const int* block_table,
                                       int bt_stride, const int* ctx_len, int nq, int nkv, int hd, int page_size,
                                       float scale, int window, float* part, int max_chunks, float* out,
                                       cudaStream_t stream) {
    if (n_decode <= 0) return 0;
    if (!somi_attention_f32_supported(qkv, kcache, vcache, out, row_stride, nq, nkv, hd) || page_size <= 0 ||
        max_chunks <= 0 || n_decode > 65535 || nkv > 65535 || (reinterpret_cast<uintptr_t>(part) & 7))
        return SOMI_ERR_UNSUPPORTED;
    float2* part_ml = reinterpret_cast<float2*>(part);
    float* part_o = part + 2 * static_cast<size_t>(n_decode) * nq * max_chunks;
    auto go = [&](auto split, auto merge, int smem) {
        launch_pdl(split, dim3(max_chunks, nkv, n_decode), dim3(128), smem, stream, qkv, row_stride, row_base, req_base,
                   kcache, vcache, block_table, bt_stride, ctx_len, nq, nkv, page_size, scale, window, max_chunks,
                   part_o, part_ml);
        launch_pdl(merge, dim3(n_decode, nq), dim3(hd), 0, stream, part_o, part_ml, max_chunks, ctx_len, row_base,
                   req_base, nq, window, out);
        return launch_status();
    };
    return hd == 64 ? go(attention_f32_split_kernel<64>, attention_f32_merge_kernel<64>, f32_split_smem<64>())
                    : go(attention_f32_split_kernel<128>, attention_f32_merge_kernel<128>, f32_split_smem<128>());
}

// Whether a step's portions and single tokens go in one launch: head size 64, where few tiles share their rows out and the single tokens
// are at most four waves of CTAs as large as the portions', two an SM.  A captured layer of 14 heads over 2 of 64, one launch / apart, us:
// 203 rows and 4 tokens behind 1,000 (136 CTAs of single tokens) 51.2 / 57.8, 16 (544) 55.1 / 61.1, 32 (1,088) 66.0 / 68.1, 64
// (2,176) 91.0 / 85.7; 16 behind 2,000 (1,088) 67.7 / 69.7; 64 rows behind 2,000 and 8 tokens 174 / 181; 1,024 rows and 16 tokens 171 / 180.
// At 128 a CTA fills an SM and the single tokens wait for the portions: 28 heads over 4, 203 rows and 4 tokens 201 / 192, 8 tokens 218 / 204.
SOMI_API int somi_attention_f32_mixed_takes(int n_tiles, int nq, int nkv, int hd, int n_decode, int max_chunks) {
    return hd == 64 && n_tiles > 0 && n_decode > 0 && nq > 0 && f32_shares_of(n_tiles, nq) > 1 &&
           static_cast<long long>(n_decode) * max_chunks * nkv <= 4 * 2 * 148;
}

// Both, where the rule above takes them: arguments as of the two functions in front of it.
SOMI_API int somi_attention_f32_mixed(const float* qkv, int row_stride, const float* kcache, const float* vcache,
                                      const int* block_table, int bt_stride, const int* cu_q, const int* ctx_len,
                                      const int* tiles, int n_tiles, int nq, int nkv, int hd, int page_size, float scale,
                                      int window, float* out, int row_base, int req_base, int n_decode, float* part,
                                      int max_chunks, cudaStream_t stream) {
    if (!somi_attention_f32_supported(qkv, kcache, vcache, out, row_stride, nq, nkv, hd) || page_size <= 0 || max_chunks <= 0 ||
        n_decode > 65535 || (reinterpret_cast<uintptr_t>(part) & 7) ||
        !somi_attention_f32_mixed_takes(n_tiles, nq, nkv, hd, n_decode, max_chunks))
        return SOMI_ERR_UNSUPPORTED;
    float2* part_ml = reinterpret_cast<float2*>(part);
    float* part_o = part + 2 * static_cast<size_t>(n_decode) * nq * max_chunks;
    const int shares = f32_shares_of(n_tiles, nq), singles = n_decode * max_chunks * nkv;
    auto go = [&](auto kernel, int smem, int ctas) {
        launch_pdl(kernel, dim3(ctas + singles), dim3(256), smem, stream, qkv, row_stride, kcache, vcache, block_table, bt_stride,
                   cu_q, ctx_len, tiles, n_tiles, nq, nkv, page_size, scale, window, out, row_base, req_base, max_chunks, part_o,
                   part_ml);
        launch_pdl(attention_f32_merge_kernel<64>, dim3(n_decode, nq), dim3(64), 0, stream, part_o, part_ml, max_chunks, ctx_len,
                   row_base, req_base, nq, window, out);
        return launch_status();
    };
    allow_smem<attention_f32_mixed_kernel<1>>(f32_shares_smem<64>(16));
    allow_smem<attention_f32_mixed_kernel<2>>(f32_shares_smem<64>(32));
    return shares == 2 ? go(attention_f32_mixed_kernel<2>, f32_shares_smem<64>(32), n_tiles * nq * 2)
                       : go(attention_f32_mixed_kernel<1>, f32_shares_smem<64>(16), n_tiles * nq * 4);
}
