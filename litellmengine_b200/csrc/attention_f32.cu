// Paged causal attention of the 32-bit mode for head sizes 64 and 128: float32 queries, keys, values and results, every
// product a float32 multiply-add (no tensor cores: nothing may be rounded below 32 bits).  The general kernel
// (attention_generic.cu) stays for other head sizes, biases, sinks and kept keys.
//
//   decode   single tokens, keys cut into splits.  What bounds it: the bytes of the cache.  A block serves ONE kv head for
//            all query heads of its group (the general kernel reads every key once per query head), eight warps with eight
//            keys in flight each: a lane holds 1/32 of a key and of a value (16 bytes at head size 128), so a warp's load
//            is one row.  The 8 x group partial scores of a lane are added across lanes by halving exchanges (31 shuffles
//            for 32 sums instead of 160), which leaves lane i with the score of (key i / group, head i % group).
//   prefill  portions of several tokens.  What bounds it: multiply-adds.  A block takes 64 query rows of one head, tiles of
//            64 keys; a thread makes 4 x 4 scores and 4 rows x 8 output columns, 8 and 10.7 multiply-adds per shared
//            16-byte load, where the general kernel made one dot product a lane and one value column a load.
// Measured, 32 query heads over 8 of 128, against the general kernel: a prompt of 500 tokens 888 -> 129 us (167 with 8 rows a
// thread in blocks of 128 threads and the list of tiles outermost in the grid); 8 single tokens at contexts of 1,125 to 1,500
// 190 -> 29 us (85 MB of keys and values: 2.9 TB/s; the exchanges, not the bytes, are what is left).
#include "common.cuh"
#include <math_constants.h>
#include <type_traits>

#define FA_WARPS 8

template <int VW> struct FaVec;
template <> struct FaVec<4> { typedef float4 T; };
template <> struct FaVec<2> { typedef float2 T; };

template <int VW> __device__ __forceinline__ void fa_load(float (&o)[VW], const float* p) {
    const typename FaVec<VW>::T v = *reinterpret_cast<const typename FaVec<VW>::T*>(p);
    const float* f = reinterpret_cast<const float*>(&v);
#pragma unroll
    for (int i = 0; i < VW; ++i) o[i] = f[i];
}

// D = 32 VW entries a head, G query heads a kv head, KT keys a warp takes at a time (KT x G <= 32).  grid (splits, nkv, rows).
// One split: the result goes to `out`; several: unnormalised sums, maximum and weight sum to the scratch.
template <int VW, int G, int KT>
__global__ void __launch_bounds__(FA_WARPS * 32, 2) attention_f32_decode_kernel(
    const float* __restrict__ q, float* __restrict__ out, float* __restrict__ part_acc, float* __restrict__ part_ml,
    const float* __restrict__ cache, const int32_t* __restrict__ rows, const int32_t* __restrict__ positions,
    const int32_t* __restrict__ token_entry, const int32_t* __restrict__ entry_slot, const int32_t* __restrict__ block_table,
    int table_stride, int nq, int nkv, int page_size, int window, float scale, int num_pages, int32_t* __restrict__ status) {
    pdl_begin();
    constexpr int D = 32 * VW, V = KT * G;
    constexpr int SHIFT = V == 32 ? 0 : V == 16 ? 1 : 2;                   // log2 of the lanes that hold the same score
    __shared__ float merge_acc[FA_WARPS][G][D];
    __shared__ float merge_ml[FA_WARPS][G][2];
    const int r = blockIdx.z, kvh = blockIdx.y, split = blockIdx.x, splits = gridDim.x;
    const int t = rows ? rows[r] : r;
    if (t < 0) return;                                                     // a padding entry of the row list
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int pos = positions[t];
    const int32_t* table = block_table + static_cast<size_t>(entry_slot[token_entry[t]]) * table_stride;
    const int lo = first_visible(pos, window);
    const int tiles = (pos - lo) / KT + 1, per = (tiles + splits - 1) / splits;
    const int first = split * per, last = min(first + per, tiles);
    const size_t khead = static_cast<size_t>(page_size) * D, kpage = 2 * static_cast<size_t>(nkv) * khead;
    float qv[G][VW], acc[G][VW];
#pragma unroll
    for (int g = 0; g < G; ++g) {
        fa_load<VW>(qv[g], q + (static_cast<size_t>(t) * nq + kvh * G + g) * D + lane * VW);
#pragma unroll
        for (int i = 0; i < VW; ++i) { qv[g][i] *= scale; acc[g][i] = 0.0f; }
    }
    const int my_key = (lane >> SHIFT) / G;                                // of the score this lane ends up with
    float m = -CUDART_INF_F, l = 0.0f;                                     // of head (lane >> SHIFT) % G
    for (int tile = first + warp; tile < last; tile += FA_WARPS) {
        const int j0 = lo + tile * KT;
        long long row = -1;                                                // lane k: where key j0 + k lies
        if (lane < KT && j0 + lane <= pos) {
            const int j = j0 + lane, logical = j / page_size;
            const int page = logical < table_stride ? table[logical] : -1;
            if (page < 0 || page >= num_pages) {
                if (atomicCAS(status, 0, 4) == 0) status[1] = t;
            } else {
                row = static_cast<long long>(page * kpage + kvh * khead + static_cast<size_t>(j - logical * page_size) * D);
            }
        }
        float kx[KT][VW], vx[KT][VW];
#pragma unroll
        for (int k = 0; k < KT; ++k) {
            const long long at = __shfl_sync(0xffffffffu, row, k);
            if (at >= 0) {
                fa_load<VW>(kx[k], cache + at + lane * VW);
                fa_load<VW>(vx[k], cache + at + nkv * khead + lane * VW);
            } else {
#pragma unroll
                for (int i = 0; i < VW; ++i) kx[k][i] = vx[k][i] = 0.0f;
            }
        }
        float s[V];
#pragma unroll
        for (int k = 0; k < KT; ++k)
#pragma unroll
            for (int g = 0; g < G; ++g) {
                float d = 0.0f;
#pragma unroll
                for (int i = 0; i < VW; ++i) d = fmaf(qv[g][i], kx[k][i], d);
                s[k * G + g] = d;
            }
        int n = V;
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            if (n > 1) {
                n >>= 1;
#pragma unroll
                for (int i = 0; i < V / 2; ++i)
                    if (i < n) {
                        const bool up = (lane & off) != 0;
                        const float send = up ? s[i] : s[i + n], keep = up ? s[i + n] : s[i];
                        s[i] = keep + __shfl_xor_sync(0xffffffffu, send, off);
                    }
            } else {
                s[0] += __shfl_xor_sync(0xffffffffu, s[0], off);
            }
        }
        const bool seen = __shfl_sync(0xffffffffu, row, my_key) >= 0;
        const float score = seen ? s[0] : -CUDART_INF_F;
        float top = score;
#pragma unroll
        for (int off = G << SHIFT; off < 32; off <<= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, off));
        const float m_new = fmaxf(m, top);
        const float alpha = (m == -CUDART_INF_F) ? 0.0f : expf(m - m_new);
        const float base = m_new == -CUDART_INF_F ? 0.0f : m_new;         // only scores of minus infinity so far: weights of zero
        const float p = seen ? expf(score - base) : 0.0f;
        l = l * alpha + p;
        if (__any_sync(0xffffffffu, m_new != m)) {
#pragma unroll
            for (int g = 0; g < G; ++g) {
                const float a = __shfl_sync(0xffffffffu, alpha, g << SHIFT);
#pragma unroll
                for (int i = 0; i < VW; ++i) acc[g][i] *= a;
            }
        }
        m = m_new;
#pragma unroll
        for (int k = 0; k < KT; ++k)
#pragma unroll
            for (int g = 0; g < G; ++g) {
                const float pk = __shfl_sync(0xffffffffu, p, (k * G + g) << SHIFT);
#pragma unroll
                for (int i = 0; i < VW; ++i) acc[g][i] = fmaf(pk, vx[k][i], acc[g][i]);
            }
    }
    // a lane's l counts its own keys only; lanes that hold the same score count it once
    if (lane & ((1 << SHIFT) - 1)) l = 0.0f;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1)
        if (off < (1 << SHIFT) || off >= (G << SHIFT)) l += __shfl_xor_sync(0xffffffffu, l, off);
#pragma unroll
    for (int g = 0; g < G; ++g)
#pragma unroll
        for (int i = 0; i < VW; ++i) merge_acc[warp][g][lane * VW + i] = acc[g][i];
    if (lane < (G << SHIFT) && (lane & ((1 << SHIFT) - 1)) == 0) {
        merge_ml[warp][lane >> SHIFT][0] = m;
        merge_ml[warp][lane >> SHIFT][1] = l;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < G * D; i += FA_WARPS * 32) {             // the warps' results, in warp order
        const int g = i / D, d = i - g * D;
        float M = -CUDART_INF_F;
#pragma unroll
        for (int w = 0; w < FA_WARPS; ++w) M = fmaxf(M, merge_ml[w][g][0]);
        float a = 0.0f, L = 0.0f;
#pragma unroll
        for (int w = 0; w < FA_WARPS; ++w) {
            const float f = merge_ml[w][g][0] == -CUDART_INF_F ? 0.0f : expf(merge_ml[w][g][0] - M);
            a = fmaf(merge_acc[w][g][d], f, a);
            L = fmaf(merge_ml[w][g][1], f, L);
        }
        const int h = kvh * G + g;
        if (splits == 1) {
            out[(static_cast<size_t>(t) * nq + h) * D + d] = a / L;
        } else {
            const size_t at = (static_cast<size_t>(r) * nq + h) * splits + split;
            part_acc[at * D + d] = a;
            if (d == 0) { part_ml[at * 2] = M; part_ml[at * 2 + 1] = L; }
        }
    }
}

// grid (rows, nq), D threads: the splits of a row's head, in order
__global__ void attention_f32_combine_kernel(const float* __restrict__ part_acc, const float* __restrict__ part_ml,
                                             const int32_t* __restrict__ rows, float* __restrict__ out, int nq, int splits) {
    pdl_begin();
    const int r = blockIdx.x, h = blockIdx.y, D = blockDim.x;
    const int t = rows ? rows[r] : r;
    if (t < 0) return;
    const size_t at = (static_cast<size_t>(r) * nq + h) * splits;
    float M = -CUDART_INF_F;
    for (int s = 0; s < splits; ++s) M = fmaxf(M, part_ml[(at + s) * 2]);
    float a = 0.0f, L = 0.0f;
    for (int s = 0; s < splits; ++s) {
        const float ms = part_ml[(at + s) * 2];
        const float f = ms == -CUDART_INF_F ? 0.0f : expf(ms - M);
        a = fmaf(part_acc[(at + s) * D + threadIdx.x], f, a);
        L = fmaf(part_ml[(at + s) * 2 + 1], f, L);
    }
    out[(static_cast<size_t>(t) * nq + h) * D + threadIdx.x] = a / L;
}

extern "C" int llm_attention_f32_decode_supported(int d, int group) {
    return (d == 64 || d == 128) && (group == 1 || group == 2 || group == 4 || group == 8);
}

// q, out: float32 [T, nq * d]; cache: float32 [pages, 2, nkv, page_size, d]; rows: int32 [n_rows] (null: rows 0 .. n_rows - 1;
// -1: padding); scratch: float32, n_rows * nq * splits * (d + 2) of them when splits > 1.
extern "C" int llm_attention_f32_decode(
    const float* q, float* out, const float* cache, const int32_t* rows, int n_rows, const int32_t* positions,
    const int32_t* token_entry, const int32_t* entry_slot, const int32_t* block_table, int table_stride, int nq, int nkv, int d,
    int page_size, int window, float scale, int num_pages, int splits, float* scratch, int32_t* status, uintptr_t stream) {
    if (n_rows <= 0) return LLM_OK;
    if (nq <= 0 || nkv <= 0 || nq % nkv != 0 || page_size <= 0 || splits < 1 || splits > 65535 || nkv > 65535 || n_rows > 65535 ||
        nq > 65535 || !llm_attention_f32_decode_supported(d, nq / nkv))
        return LLM_REFUSED_SIZE;
    if (!aligned16(q) || !aligned16(out) || !aligned16(cache) || (splits > 1 && (!scratch || !aligned16(scratch))))
        return LLM_REFUSED_ALIGN;
    float* part_acc = scratch;
    float* part_ml = scratch ? scratch + static_cast<size_t>(n_rows) * nq * splits * d : nullptr;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    const dim3 grid(splits, nkv, n_rows), block(FA_WARPS * 32);
#define GO(VW, G, KT)                                                                                                     \
    launch_pdl((attention_f32_decode_kernel<VW, G, KT>), grid, block, 0, s, q, out, part_acc, part_ml, cache, rows,       \
               positions, token_entry, entry_slot, block_table, table_stride, nq, nkv, page_size, window, scale,          \
               num_pages, status)
    const int group = nq / nkv;
    if (d == 128) {
        if (group == 1) GO(4, 1, 8); else if (group == 2) GO(4, 2, 8); else if (group == 4) GO(4, 4, 8); else GO(4, 8, 4);
    } else {
        if (group == 1) GO(2, 1, 8); else if (group == 2) GO(2, 2, 8); else if (group == 4) GO(2, 4, 8); else GO(2, 8, 4);
    }
#undef GO
    if (splits > 1)
        launch_pdl(attention_f32_combine_kernel, dim3(n_rows, nq), dim3(d), 0, s, part_acc, part_ml, rows, out, nq, splits);
    return launch_status();
}

// ---- portions of several tokens ---------------------------------------------------------------------------------
#define FP_ROWS 64
#define FP_KEYS 64
#define FP_THREADS 256
#define FP_RPT (FP_ROWS * 16 / FP_THREADS)      // query rows a thread takes

template <int D>
__global__ void __launch_bounds__(FP_THREADS, 2) attention_f32_prefill_kernel(
    const float* __restrict__ q, float* __restrict__ out, const float* __restrict__ cache, const int32_t* __restrict__ tiles,
    const int32_t* __restrict__ entry_slot, const int32_t* __restrict__ entry_q_start, const int32_t* __restrict__ entry_q_len,
    const int32_t* __restrict__ entry_kv_len, const int32_t* __restrict__ block_table, int table_stride, int nq, int nkv,
    int page_size, int window, float scale, int num_pages, int tile_rows, int32_t* __restrict__ status) {
    pdl_begin();
    constexpr int KLD = D + 4, PLD = FP_KEYS + 4, C4 = D / 4, OC = D / 64;      // OC: groups of 64 output columns
    extern __shared__ __align__(16) float fp_smem[];
    float* qs = fp_smem;                                     // [64][D], scaled
    float* ks = qs + FP_ROWS * D;                            // [64][D + 4]; the weights [64][68] lie over it once the scores are made
    float* vs = ks + FP_KEYS * KLD;                          // [64][D]
    float* ps = ks;
    const int h = blockIdx.x, kvh = h / (nq / nkv);
    const int e = tiles[2 * blockIdx.z], part = gridDim.y - 1 - blockIdx.y;      // the part that walks more keys first
    if (e < 0) return;                                       // a padding entry of the tile list
    const int q0 = tiles[2 * blockIdx.z + 1] + FP_ROWS * part;
    const int q_len = entry_q_len[e], past = entry_kv_len[e] - q_len;
    const int rows_here = min(min(FP_ROWS, tile_rows - FP_ROWS * part), q_len - q0);
    if (rows_here <= 0) return;
    const int row_base = entry_q_start[e] + q0;
    const int32_t* table = block_table + static_cast<size_t>(entry_slot[e]) * table_stride;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, tx = tid & 15, ty = tid >> 4;
    const int pos_first = past + q0, pos_last = pos_first + rows_here - 1, lo_last = first_visible(pos_last, window);
    const size_t khead = static_cast<size_t>(page_size) * D, kpage = 2 * static_cast<size_t>(nkv) * khead;
    for (int i = tid; i < FP_ROWS * C4; i += FP_THREADS) {
        const int r = i / C4, c = i - r * C4;
        float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (r < rows_here) v = *reinterpret_cast<const float4*>(q + (static_cast<size_t>(row_base + r) * nq + h) * D + 4 * c);
        v.x *= scale; v.y *= scale; v.z *= scale; v.w *= scale;
        *reinterpret_cast<float4*>(qs + r * D + 4 * c) = v;
    }
    float o[FP_RPT][4 * OC], m[FP_RPT], l[FP_RPT];
#pragma unroll
    for (int r = 0; r < FP_RPT; ++r) {
        m[r] = -CUDART_INF_F; l[r] = 0.0f;
#pragma unroll
        for (int c = 0; c < 4 * OC; ++c) o[r][c] = 0.0f;
    }
    auto stage = [&](float* dst, int ld, int kt, size_t off) {                  // a warp brings whole rows
        for (int r = warp; r < FP_KEYS; r += FP_THREADS / 32) {
            const int j = kt + r;
            const float* src = nullptr;
            if (j <= pos_last) {
                const int logical = j / page_size;
                const int page = logical < table_stride ? table[logical] : -1;
                if (page < 0 || page >= num_pages) {
                    if (lane == 0 && atomicCAS(status, 0, 4) == 0) status[1] = row_base;
                } else {
                    src = cache + page * kpage + off + kvh * khead + static_cast<size_t>(j - logical * page_size) * D;
                }
            }
            for (int c = lane; c < C4; c += 32) {
                float* d = dst + r * ld + 4 * c;
                if (src) {
                    const unsigned a = static_cast<unsigned>(__cvta_generic_to_shared(d));
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(a), "l"(src + 4 * c));
                } else {
                    *reinterpret_cast<float4*>(d) = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                }
            }
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    for (int kt = first_visible(pos_first, window); kt <= pos_last; kt += FP_KEYS) {
        stage(ks, KLD, kt, 0);
        stage(vs, D, kt, nkv * khead);
        asm volatile("cp.async.wait_group 1;\n" ::: "memory");
        __syncthreads();                                     // the keys (and at first the queries) are in place
        float s[FP_RPT][4];
#pragma unroll
        for (int r = 0; r < FP_RPT; ++r) s[r][0] = s[r][1] = s[r][2] = s[r][3] = 0.0f;
#pragma unroll 2
        for (int k = 0; k < D; k += 4) {
            float4 kb[4];
#pragma unroll
            for (int c = 0; c < 4; ++c) kb[c] = *reinterpret_cast<const float4*>(ks + (tx + 16 * c) * KLD + k);
#pragma unroll
            for (int r = 0; r < FP_RPT; ++r) {
                const float4 a = *reinterpret_cast<const float4*>(qs + (ty * FP_RPT + r) * D + k);
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    s[r][c] = fmaf(a.x, kb[c].x, s[r][c]);
                    s[r][c] = fmaf(a.y, kb[c].y, s[r][c]);
                    s[r][c] = fmaf(a.z, kb[c].z, s[r][c]);
                    s[r][c] = fmaf(a.w, kb[c].w, s[r][c]);
                }
            }
        }
        __syncthreads();                                     // the keys are read: the weights may take their place
#pragma unroll
        for (int r = 0; r < FP_RPT; ++r) {
            const int pos = pos_first + ty * FP_RPT + r, lo = first_visible(pos, window);
            float top = -CUDART_INF_F;
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const int j = kt + tx + 16 * c;
                if (j > pos || j < lo) s[r][c] = -CUDART_INF_F;
                top = fmaxf(top, s[r][c]);
            }
#pragma unroll
            for (int off = 1; off < 16; off <<= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, off));
            const float m_new = fmaxf(m[r], top);
            const float base = m_new == -CUDART_INF_F ? 0.0f : m_new;         // a row that has seen no key yet
            const float alpha = expf(m[r] - base);
            float sum = 0.0f;
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const float p = expf(s[r][c] - base);
                const int j = kt + tx + 16 * c;
                ps[(ty * FP_RPT + r) * PLD + tx + 16 * c] = (j > pos || j < lo) ? -1.0f : p;
                sum += p;
            }
            l[r] = l[r] * alpha + sum;
            m[r] = m_new;
#pragma unroll
            for (int c = 0; c < 4 * OC; ++c) o[r][c] *= alpha;
        }
        asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        __syncthreads();                                     // weights and values are in place
        // Zero times a value that is not finite is NaN: where some row of the block does not see some key of the tile, each product
        // is made only for the rows that see its key (weight -1: it does not).
        auto values = [&](auto hidden) {
#pragma unroll 1
            for (int k = 0; k < FP_KEYS; k += 4) {
                float4 p[FP_RPT];
#pragma unroll
                for (int r = 0; r < FP_RPT; ++r) p[r] = *reinterpret_cast<const float4*>(ps + (ty * FP_RPT + r) * PLD + k);
#pragma unroll
                for (int u = 0; u < 4; ++u)
#pragma unroll
                    for (int c = 0; c < OC; ++c) {
                        const float4 v = *reinterpret_cast<const float4*>(vs + (k + u) * D + c * 64 + tx * 4);
#pragma unroll
                        for (int r = 0; r < FP_RPT; ++r) {
                            const float w = u == 0 ? p[r].x : u == 1 ? p[r].y : u == 2 ? p[r].z : p[r].w;
                            if (decltype(hidden)::value && w < 0.0f) continue;
                            o[r][4 * c] = fmaf(w, v.x, o[r][4 * c]);
                            o[r][4 * c + 1] = fmaf(w, v.y, o[r][4 * c + 1]);
                            o[r][4 * c + 2] = fmaf(w, v.z, o[r][4 * c + 2]);
                            o[r][4 * c + 3] = fmaf(w, v.w, o[r][4 * c + 3]);
                        }
                    }
            }
        };
        if (kt + FP_KEYS - 1 > pos_first || kt < lo_last) values(std::true_type());
        else values(std::false_type());
        __syncthreads();                                     // before the next tile overwrites them
    }
#pragma unroll
    for (int r = 0; r < FP_RPT; ++r) {
#pragma unroll
        for (int off = 1; off < 16; off <<= 1) l[r] += __shfl_xor_sync(0xffffffffu, l[r], off);
        if (ty * FP_RPT + r >= rows_here) continue;
        const float inv = 1.0f / l[r];
        float* orow = out + (static_cast<size_t>(row_base + ty * FP_RPT + r) * nq + h) * D;
#pragma unroll
        for (int c = 0; c < OC; ++c)
            *reinterpret_cast<float4*>(orow + c * 64 + tx * 4) =
                make_float4(o[r][4 * c] * inv, o[r][4 * c + 1] * inv, o[r][4 * c + 2] * inv, o[r][4 * c + 3] * inv);
    }
}

extern "C" int llm_attention_f32_prefill_supported(int d) { return d == 64 || d == 128; }

// q, out: float32 [T, nq * d]; cache as above; tiles: int32 [n_tiles][2] = (entry, first query row inside it), `tile_rows` rows
// each, -1 for padding.
extern "C" int llm_attention_f32_prefill(
    const float* q, float* out, const float* cache, const int32_t* tiles, int n_tiles, int tile_rows, const int32_t* entry_slot,
    const int32_t* entry_q_start, const int32_t* entry_q_len, const int32_t* entry_kv_len, const int32_t* block_table,
    int table_stride, int nq, int nkv, int d, int page_size, int window, float scale, int num_pages, int32_t* status,
    uintptr_t stream) {
    if (n_tiles <= 0) return LLM_OK;
    if (nq <= 0 || nkv <= 0 || nq % nkv != 0 || page_size <= 0 || n_tiles > 65535 || tile_rows <= 0 ||
        !llm_attention_f32_prefill_supported(d))
        return LLM_REFUSED_SIZE;
    if (!aligned16(q) || !aligned16(out) || !aligned16(cache)) return LLM_REFUSED_ALIGN;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    const size_t smem = static_cast<size_t>(FP_ROWS * d + FP_KEYS * (d + 4) + FP_KEYS * d) * sizeof(float);
    // blocks start in this order: tiles come longest walk first, and the heads of one before the next
    const dim3 grid(nq, (tile_rows + FP_ROWS - 1) / FP_ROWS, n_tiles);
#define GO(D)                                                                                                              \
    {                                                                                                                      \
        const cudaError_t e = cudaFuncSetAttribute(attention_f32_prefill_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, \
                                                   static_cast<int>(smem));                                                \
        if (e != cudaSuccess) return static_cast<int>(e);                                                                  \
        launch_pdl((attention_f32_prefill_kernel<D>), grid, dim3(FP_THREADS), smem, s, q, out, cache, tiles, entry_slot,   \
                   entry_q_start, entry_q_len, entry_kv_len, block_table, table_stride, nq, nkv, page_size, window, scale, \
                   num_pages, tile_rows, status);                                                                          \
    }
    if (d == 128) GO(128) else GO(64)
#undef GO
    return launch_status();
}
