// Causal grouped-query attention of the float32 path over the paged cache, head sizes 64 and 128, with
// or without a window: a kernel for prompt portions and one for single-token requests, which cut the
// keys the same way and so give a row the same bits.  (Other sizes, other masks, capped scores, sinks
// and gates run the kernel in attention_generic.cu.)  All products are float32 FMAs, the softmax is
// float32.
//
// A row's arithmetic: keys come in chunks of 64 aligned to position 0.  In a chunk a score is two
// chains of FMAs (even and odd elements of the head) and their sum, the chunk's maximum m_c and
// sum l_c are its own, and o_c sums p v over its keys in ascending order.  Chunks are merged in
// ascending order: with M the larger maximum, L <- L e^(M_old - M) + l_c e^(m_c - M), O likewise.  The
// prompt kernel merges in registers; the split kernel writes (m_c, l_c, o_c) and the merge kernel
// goes through them.  So how a request was cut into steps, or what else is in a step, changes no bit.
//
// Why these two shapes.  Single tokens are bound by latency and by the cache's bytes: one CTA per
// (request, key/value head, chunk) reads keys and values once for all query heads of the group, with every
// copy of the chunk in flight at once and those of older positions issued before the dependency wait.
// A portion is bound by the FMA pipe: 64 rows of one head per CTA, 4 x 4 scores a thread from shared
// memory four elements at a time, the next keys fetched under the softmax and the next values under
// the scores.
#include "common.cuh"

namespace somi {

constexpr int kF32Chunk = 64;         // keys per chunk
constexpr int kF32Rows = 64;          // query rows of a tile of the list
constexpr int kF32Heads = 8;          // query heads a split CTA takes at a time

__device__ __forceinline__ void f32_fma2(unsigned long long& d, unsigned long long a, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
__device__ __forceinline__ float f32_sum2(unsigned long long d) {
    float lo, hi;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(d));
    return __fadd_rn(lo, hi);
}
__device__ __forceinline__ void f32_copy(float* dst, const float* src, bool in) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n"
                 ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(dst))), "l"(src), "r"(in ? 16 : 0) : "memory");
}
__device__ __forceinline__ void f32_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void f32_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// The 64 probabilities of a row, two a lane, from its scores: maximum and sum over the chunk.  A hidden key's
// score is -infinity.  The maximum passes over a score that is not a number, so what a key adds is decided
// by its own score: a NaN among hidden keys (m = -infinity) makes p and the sum NaN.
__device__ __forceinline__ float2 f32_chunk_softmax(float& s0, float& s1) {
    const float m = warp_max(fmaxf(s0, s1));
    s0 = s0 == -INFINITY ? 0.f : expf(s0 - m);
    s1 = s1 == -INFINITY ? 0.f : expf(s1 - m);
    return make_float2(m, warp_sum(__fadd_rn(s0, s1)));
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

// ------------------------------------------------------------------------- prompt portions
// A CTA takes 16 RI rows of a tile of 64: share blockIdx.z of it.
template <int HD, int RI>
__global__ void __launch_bounds__(256)
attention_f32_portion_kernel(const float* __restrict__ qkv, int row_stride, const float* __restrict__ kcache,
                             const float* __restrict__ vcache, const int* __restrict__ block_table,
                             int bt_stride, const int* __restrict__ cu_q, const int* __restrict__ ctx_len,
                             const int* __restrict__ tiles, int n_tiles, int nq, int nkv, int page_size,
                             float scale, int window, float* __restrict__ out) {
    constexpr int ROWS = 16 * RI;
    constexpr int P = HD + 4;            // floats between rows of Q and K: neighbours in different banks
    constexpr int PP = kF32Chunk + 4;
    constexpr int COLS = HD / 16;        // output columns a thread
    extern __shared__ __align__(16) float f32_smem[];
    float* Qs = f32_smem;                // [ROWS][P]
    float* Ks = Qs + ROWS * P;       // [64][P]
    float* Vs = Ks + kF32Chunk * P;      // [64][HD]
    float* Ps = Vs + kF32Chunk * HD;     // [ROWS][PP]
    __shared__ float M_s[ROWS], L_s[ROWS];
    __shared__ float2 f_s[ROWS];
    pdl_launch_dependents();
    pdl_wait();
    const int* tile = tiles + 3 * (n_tiles - 1 - static_cast<int>(blockIdx.x));   // a prompt's last rows first
    const int req = tile[0], row0 = tile[1] + blockIdx.z * ROWS, head = blockIdx.y;
    const int rows = min(ROWS, tile[2] - static_cast<int>(blockIdx.z) * ROWS);
    if (rows <= 0) return;
    const int kvh = head / (nq / nkv);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int pos0 = ctx_len[req] + (row0 - cu_q[req]);
    const int first_key = window > 0 ? max(0, pos0 - window + 1) : 0, end_key = pos0 + rows;
    const int* bt = block_table + static_cast<size_t>(req) * bt_stride;

    auto load = [&](float* dst, int pitch, const float* cache, int c) {
        for (int idx = tid; idx < kF32Chunk * (HD / 4); idx += 256) {
            const int n = idx / (HD / 4), d = idx % (HD / 4) * 4, j = c * kF32Chunk + n;
            const bool in = j >= first_key && j < end_key;
            const float* src = cache;
            if (in) src += ((static_cast<size_t>(bt[j / page_size]) * nkv + kvh) * page_size + j % page_size) * HD + d;
            f32_copy(dst + n * pitch + d, src, in);
        }
        f32_commit();
    };
    const int c_first = first_key / kF32Chunk, c_end = (end_key + kF32Chunk - 1) / kF32Chunk;
    load(Ks, P, kcache, c_first);
    load(Vs, HD, vcache, c_first);
    for (int idx = tid; idx < ROWS * (HD / 4); idx += 256) {
        const int r = idx / (HD / 4), d = idx % (HD / 4) * 4;
        float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
        if (r < rows)
            q = *reinterpret_cast<const float4*>(qkv + static_cast<size_t>(row0 + r) * row_stride + head * HD + d);
        *reinterpret_cast<float4*>(Qs + r * P + d) = make_float4(q.x * scale, q.y * scale, q.z * scale, q.w * scale);
    }
    if (tid < ROWS) { M_s[tid] = -INFINITY; L_s[tid] = 0.f; }
    // scores: rows tr + 16 i, keys tc + 16 j, the lanes of a warp 4 x 8 of them; outputs: rows
    // tr + 16 i, columns four neighbours from 4 tc (and 64 further on)
    const int tr = warp / 2 * 4 + lane / 8, tc = warp % 2 * 8 + lane % 8;
    float O[RI][COLS];
#pragma unroll
    for (int i = 0; i < RI; ++i)
#pragma unroll
        for (int e = 0; e < COLS; ++e) O[i][e] = 0.f;

    for (int c = c_first; c < c_end; ++c) {
        f32_wait<1>();                                   // the keys; the values may be under way
        __syncthreads();
        {
            unsigned long long acc[RI][4];
#pragma unroll
            for (int i = 0; i < RI; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = 0ull;
#pragma unroll 4
            for (int d = 0; d < HD; d += 4) {
                ulonglong2 k[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) k[j] = *reinterpret_cast<const ulonglong2*>(Ks + (tc + 16 * j) * P + d);
#pragma unroll
                for (int i = 0; i < RI; ++i) {
                    const ulonglong2 q = *reinterpret_cast<const ulonglong2*>(Qs + (tr + 16 * i) * P + d);
#pragma unroll
                    for (int j = 0; j < 4; ++j) f32_fma2(acc[i][j], q.x, k[j].x);
#pragma unroll
                    for (int j = 0; j < 4; ++j) f32_fma2(acc[i][j], q.y, k[j].y);
                }
            }
#pragma unroll
            for (int i = 0; i < RI; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int r = tr + 16 * i, n = tc + 16 * j, key = c * kF32Chunk + n, pos = pos0 + r;
                    const bool seen = r < rows && key <= pos && (window <= 0 || key > pos - window);
                    Ps[r * PP + n] = seen ? f32_sum2(acc[i][j]) : -INFINITY;
                }
        }
        __syncthreads();
        const bool more = c + 1 < c_end;
        if (more) load(Ks, P, kcache, c + 1);
        for (int r = warp * 2 * RI; r < (warp + 1) * 2 * RI; ++r) {
            float s0 = Ps[r * PP + lane], s1 = Ps[r * PP + lane + 32];
            const float2 ml = f32_chunk_softmax(s0, s1);
            Ps[r * PP + lane] = s0;
            Ps[r * PP + lane + 32] = s1;
            if (lane == 0) {
                float M = M_s[r], L = L_s[r];
                f_s[r] = f32_merge(M, L, ml.x, ml.y);
                M_s[r] = M;
                L_s[r] = L;
            }
        }
        if (more) f32_wait<1>(); else f32_wait<0>();     // the values
        __syncthreads();
        // A hidden key's infinity must not meet a probability of zero: where some row does not see all of the
        // chunk, its values are looked through first, and only if one is not finite do the sums leave out what
        // is hidden (that way in full, unrolled as the other, made a 1,024-row layer 337 instead of 309 us by its
        // registers alone).
        const int k_lo = c * kF32Chunk, k_hi = k_lo + kF32Chunk - 1;
        bool plain = k_hi <= pos0 && (window <= 0 || k_lo > pos0 + ROWS - 1 - window);
        if (!plain) {
            bool wild = false;
            for (int idx = tid; idx < kF32Chunk * (HD / 4); idx += 256) {
                const float4 t = *reinterpret_cast<const float4*>(Vs + idx * 4);
                wild = wild || !(fabsf(t.x) < INFINITY && fabsf(t.y) < INFINITY && fabsf(t.z) < INFINITY && fabsf(t.w) < INFINITY);
            }
            plain = !__syncthreads_or(wild);
        }
        float oc[RI][COLS];
#pragma unroll
        for (int i = 0; i < RI; ++i)
#pragma unroll
            for (int e = 0; e < COLS; ++e) oc[i][e] = 0.f;
        if (plain) {
#pragma unroll 4
            for (int n = 0; n < kF32Chunk; n += 4) {
                float4 p[RI];
#pragma unroll
                for (int i = 0; i < RI; ++i) p[i] = *reinterpret_cast<const float4*>(Ps + (tr + 16 * i) * PP + n);
#pragma unroll
                for (int m = 0; m < 4; ++m) {
                    float v[COLS];
#pragma unroll
                    for (int e = 0; e < COLS; e += 4) {
                        const float4 t = *reinterpret_cast<const float4*>(Vs + (n + m) * HD + tc * 4 + e * 16);
                        v[e] = t.x; v[e + 1] = t.y; v[e + 2] = t.z; v[e + 3] = t.w;
                    }
#pragma unroll
                    for (int i = 0; i < RI; ++i) {
                        const float w = m == 0 ? p[i].x : (m == 1 ? p[i].y : (m == 2 ? p[i].z : p[i].w));
#pragma unroll
                        for (int e = 0; e < COLS; ++e) oc[i][e] = __fmaf_rn(w, v[e], oc[i][e]);
                    }
                }
            }
        } else {
#pragma unroll 1
            for (int n = 0; n < kF32Chunk; ++n) {
#pragma unroll
                for (int i = 0; i < RI; ++i) {
                    const int key = k_lo + n, pos = pos0 + tr + 16 * i;
                    if (key > pos || (window > 0 && key <= pos - window)) continue;
                    const float w = Ps[(tr + 16 * i) * PP + n];
#pragma unroll
                    for (int e = 0; e < COLS; ++e)
                        oc[i][e] = __fmaf_rn(w, Vs[n * HD + tc * 4 + e % 4 + e / 4 * 64], oc[i][e]);
                }
            }
        }
#pragma unroll
        for (int i = 0; i < RI; ++i) {
            const float2 f = f_s[tr + 16 * i];
#pragma unroll
            for (int e = 0; e < COLS; ++e) O[i][e] = f32_merge_out(O[i][e], oc[i][e], f);
        }
        __syncthreads();                                 // the values and probabilities have been read
        if (more) load(Vs, HD, vcache, c + 1);
    }
#pragma unroll
    for (int i = 0; i < RI; ++i) {
        const int r = tr + 16 * i;
        if (r >= rows) continue;
        const float L = L_s[r];
        float* dst = out + static_cast<size_t>(row0 + r) * (nq * HD) + head * HD + tc * 4;
#pragma unroll
        for (int e = 0; e < COLS; e += 4)
            *reinterpret_cast<float4*>(dst + e * 16) = make_float4(O[i][e] / L, O[i][e + 1] / L, O[i][e + 2] / L, O[i][e + 3] / L);
    }
}

// ------------------------------------------------------------------- single-token requests
// part_o [request][query head][chunk][HD], part_ml likewise with (m, l); a request's chunks are counted from the
// one of its first visible key, so that a window needs no more of them than it reaches.
template <int HD>
__global__ void __launch_bounds__(128)
attention_f32_split_kernel(const float* __restrict__ qkv, int row_stride, int row_base, int req_base,
                           const float* __restrict__ kcache, const float* __restrict__ vcache,
                           const int* __restrict__ block_table, int bt_stride, const int* __restrict__ ctx_len,
                           int nq, int nkv, int page_size, float scale, int window, int max_chunks,
                           float* __restrict__ part_o, float2* __restrict__ part_ml) {
    constexpr int P = HD + 4, PP = kF32Chunk + 4;
    constexpr int QUADS = HD / 4, OUT_ROWS = kF32Heads * HD / 128;   // output rows a thread
    extern __shared__ __align__(16) float f32_smem[];
    float* Ks = f32_smem;                // [64][P]
    float* Vs = Ks + kF32Chunk * P;      // [64][HD]
    float* Qs = Vs + kF32Chunk * HD;     // [8][P]
    float* Ps = Qs + kF32Heads * P;      // [8][PP]
    pdl_launch_dependents();
    const int kvh = blockIdx.y, i = blockIdx.z, req = req_base + i;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int pos = ld_step(ctx_len + req);              // [descriptor]
    const int first_key = window > 0 ? max(0, pos - window + 1) : 0;
    const int at = blockIdx.x, c = first_key / kF32Chunk + at;
    if (c * kF32Chunk > pos) {
        pdl_wait();
        return;
    }
    const int* bt = block_table + static_cast<size_t>(req) * bt_stride;
    auto load = [&](float* dst, int pitch, const float* cache, int from, int to) {
        for (int idx = tid; idx < kF32Chunk * QUADS; idx += 128) {
            const int n = idx / QUADS, d = idx % QUADS * 4, j = c * kF32Chunk + n;
            if (n < from || n >= to) continue;
            const bool in = j >= first_key && j <= pos;
            const float* src = cache;
            if (in) src += ((static_cast<size_t>(ld_step(bt + j / page_size)) * nkv + kvh) * page_size + j % page_size) * HD + d;
            f32_copy(dst + n * pitch + d, src, in);
        }
    };
    // every position but the step's own is there already
    const int own = min(kF32Chunk, pos - c * kF32Chunk);
    load(Ks, P, kcache, 0, own);                         // [descriptor], [old-cache]
    load(Vs, HD, vcache, 0, own);
    pdl_wait();
    load(Ks, P, kcache, own, kF32Chunk);
    load(Vs, HD, vcache, own, kF32Chunk);
    f32_commit();
    const int group = nq / nkv;
    const float* q_row = qkv + static_cast<size_t>(row_base + i) * row_stride + static_cast<size_t>(kvh) * group * HD;
    for (int h0 = 0; h0 < group; h0 += kF32Heads) {
        const int heads = min(kF32Heads, group - h0);
        if (h0) __syncthreads();
        for (int idx = tid; idx < kF32Heads * QUADS; idx += 128) {
            const int r = idx / QUADS, d = idx % QUADS * 4;
            float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
            if (r < heads) q = *reinterpret_cast<const float4*>(q_row + (h0 + r) * HD + d);
            *reinterpret_cast<float4*>(Qs + r * P + d) = make_float4(q.x * scale, q.y * scale, q.z * scale, q.w * scale);
        }
        f32_wait<0>();
        __syncthreads();
        {   // a key and four heads a thread
            const int n = tid & 63, r0 = tid / 64 * 4, key = c * kF32Chunk + n;
            unsigned long long acc[4] = {0ull, 0ull, 0ull, 0ull};
#pragma unroll 8
            for (int d = 0; d < HD; d += 4) {
                const ulonglong2 k = *reinterpret_cast<const ulonglong2*>(Ks + n * P + d);
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    const ulonglong2 q = *reinterpret_cast<const ulonglong2*>(Qs + (r0 + r) * P + d);
                    f32_fma2(acc[r], q.x, k.x);
                    f32_fma2(acc[r], q.y, k.y);
                }
            }
            const bool seen = key >= first_key && key <= pos;
#pragma unroll
            for (int r = 0; r < 4; ++r) Ps[(r0 + r) * PP + n] = seen ? f32_sum2(acc[r]) : -INFINITY;
        }
        __syncthreads();
        for (int r = warp * 2; r < warp * 2 + 2; ++r) {
            float s0 = Ps[r * PP + lane], s1 = Ps[r * PP + lane + 32];
            const float2 ml = f32_chunk_softmax(s0, s1);
            Ps[r * PP + lane] = s0;
            Ps[r * PP + lane + 32] = s1;
            if (lane == 0 && r < heads)
                part_ml[(static_cast<size_t>(i) * nq + kvh * group + h0 + r) * max_chunks + at] = ml;
        }
        __syncthreads();
        const int d = tid % HD, r0 = tid / HD * OUT_ROWS;
        float o[OUT_ROWS];
#pragma unroll
        for (int r = 0; r < OUT_ROWS; ++r) o[r] = 0.f;
#pragma unroll 4
        for (int n = 0; n < kF32Chunk; n += 4) {
            float v[4];
#pragma unroll
            for (int m = 0; m < 4; ++m) v[m] = Vs[(n + m) * HD + d];
#pragma unroll
            for (int r = 0; r < OUT_ROWS; ++r) {
                const float4 p = *reinterpret_cast<const float4*>(Ps + (r0 + r) * PP + n);
                o[r] = __fmaf_rn(p.x, v[0], o[r]);
                o[r] = __fmaf_rn(p.y, v[1], o[r]);
                o[r] = __fmaf_rn(p.z, v[2], o[r]);
                o[r] = __fmaf_rn(p.w, v[3], o[r]);
            }
        }
#pragma unroll
        for (int r = 0; r < OUT_ROWS; ++r)
            if (r0 + r < heads)
                part_o[((static_cast<size_t>(i) * nq + kvh * group + h0 + r0 + r) * max_chunks + at) * HD + d] = o[r];
    }
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
constexpr int f32_portion_smem(int rows) { return 4 * ((rows + 64) * (HD + 4) + 64 * HD + rows * (kF32Chunk + 4)); }
template <int HD>
constexpr int f32_split_smem() { return 4 * (64 * (HD + 4) + 64 * HD + kF32Heads * (HD + 4 + kF32Chunk + 4)); }

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

// Prompt portions: the tile list's query tiles are at most 64 rows.
SOMI_API int somi_attention_f32_portion(const float* qkv, int row_stride, const float* kcache, const float* vcache,
                                        const int* block_table, int bt_stride, const int* cu_q, const int* ctx_len,
                                        const int* tiles, int n_tiles, int nq, int nkv, int hd, int page_size,
                                        float scale, int window, float* out, cudaStream_t stream) {
    if (n_tiles <= 0) return 0;
    if (!somi_attention_f32_supported(qkv, kcache, vcache, out, row_stride, nq, nkv, hd) || page_size <= 0)
        return SOMI_ERR_UNSUPPORTED;
    // Few tiles: two or four CTAs share one, each with a part of its rows (the same bits).  Layer of 14 heads over 2
    // of 64 with 1 / 2 / 4 shares: 64 rows behind 2,000 positions (14 CTAs of 64 rows) 312 / 222 / 189 us, 203 rows
    // (56) 79 / 76 / 79, 1,024 (224) 333 / 311 / 351, 2,048 (448) 737 / 781 / 935.
    const long long ctas = static_cast<long long>(n_tiles) * nq;
    const int shares = ctas <= 148 / 4 ? 4 : (ctas <= 148 * 2 ? 2 : 1);
    auto go = [&](auto kernel, int smem) {
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        launch_pdl(kernel, dim3(n_tiles, nq, shares), dim3(256), smem, stream, qkv, row_stride, kcache, vcache, block_table,
                   bt_stride, cu_q, ctx_len, tiles, n_tiles, nq, nkv, page_size, scale, window, out);
        return launch_status();
    };
    const int rows = kF32Rows / shares;
    if (hd == 64)
        return shares == 1 ? go(attention_f32_portion_kernel<64, 4>, f32_portion_smem<64>(rows))
             : shares == 2 ? go(attention_f32_portion_kernel<64, 2>, f32_portion_smem<64>(rows))
                           : go(attention_f32_portion_kernel<64, 1>, f32_portion_smem<64>(rows));
    return shares == 1 ? go(attention_f32_portion_kernel<128, 4>, f32_portion_smem<128>(rows))
         : shares == 2 ? go(attention_f32_portion_kernel<128, 2>, f32_portion_smem<128>(rows))
                       : go(attention_f32_portion_kernel<128, 1>, f32_portion_smem<128>(rows));
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
        cudaFuncSetAttribute(split, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
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
