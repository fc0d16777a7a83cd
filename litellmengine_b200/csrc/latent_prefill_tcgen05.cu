// Prompt portions of latent attention on the 5th-generation tensor cores, bfloat16: heads of 128 key entries and 64 rotated
// ones, values of 128.
//
// The kernels in latent_attention.cu attend over the cached rows [c | kr] themselves, which is right for a few queries: per
// query, key and head that costs 2 (2 R + P) flops (2,176 at R 512, P 64).  A portion of many queries meets every row with
// every query, so here the rows are mapped ONCE to per-head keys and values, [k | v][h] = W_ukv[h] c, and attention costs
// 2 (128 + 64 + 128) = 640.  The map is 2 R 256 flops a row and head, i.e. as much as 170 queries save.  Steps:
//   latent_gather    the rows of every portion, from their pages, to consecutive rows of one tensor, each request's padded
//                    with zero rows to whole tiles (so that a tile never shows another request's rows)
//   (a product)      [k | v] of all rows and heads
//   queries          [qn | rotated qr] per head in bfloat16: in the epilogue of their product (linear_pair_latent_q in
//                    gemm_pair_tcgen05.cu) where that takes them, else by latent_q_pack (12 us of 2,000 tokens and 32 heads)
//   attention        below
// Measured, 32 heads over rows of 512 + 64, a prompt of 2,000 tokens: attention over the cached rows 1,275 us; here rows 5,
// map 18, attention 62 us (0.69 PFLOP/s of what it cannot do without, 43 GFLOP; with two threads a row that exchanged
// their maxima before the weights, and products issued in a branch for one lane, 85).  The layer 1,480 -> 237 us, and 224 with packed
// queries (and a step's table of angles, which all layers share: 2 us to make, not in the layer's figure).
//
// Attention.  The structure of the one-pass kernel in attention_prefill_tcgen05.cu (a reference maximum that trails the
// running one, two rows of work in turns on the tensor pipe, P over S in TMEM, a softmax thread a row, weights of half a tile made
// beside their maximum), with two changes.
// Every head has keys of its own, so the two pieces of work that share a key/value tile are two tiles of 128 QUERY rows of
// one head.  And a tile is 96 keys: queries are 2 x 128 x 192 (96 KB), a tile of 128 keys with its values 80 KB, and two of
// those would not fit beside them; two of 96 keys (60 KB each) do, and a product of N 96 is as efficient as one of 128.
// The rotated key part is the same for all heads and comes straight from the gathered rows.
#include "tcgen05_attention.cuh"
#include <math_constants.h>

#define LP_BM 128
#define LP_BN 96
#define LP_QB (LP_BM * 64)                   // elements of one 64-column block of a query tile
#define LP_KB (LP_BN * 64)                   // and of a key or value tile
#define LP_DK 192
#define LP_DV 128
#define LP_STAGES 2
#define LP_JUMP 8.0f
#define LP_THREADS (128 + 2 * 128)            // producer, issuer, two without work, four softmax warps a query tile

__device__ __forceinline__ void lp_ld16(unsigned taddr, unsigned (&r)[48], int at) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
                 : "=r"(r[at]), "=r"(r[at + 1]), "=r"(r[at + 2]), "=r"(r[at + 3]), "=r"(r[at + 4]), "=r"(r[at + 5]), "=r"(r[at + 6]),
                   "=r"(r[at + 7]), "=r"(r[at + 8]), "=r"(r[at + 9]), "=r"(r[at + 10]), "=r"(r[at + 11]), "=r"(r[at + 12]),
                   "=r"(r[at + 13]), "=r"(r[at + 14]), "=r"(r[at + 15])
                 : "r"(taddr) : "memory");
}
__device__ __forceinline__ void lp_st8(unsigned taddr, const unsigned (&r)[24], int at) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};\n" ::
                     "r"(taddr), "r"(r[at]), "r"(r[at + 1]), "r"(r[at + 2]), "r"(r[at + 3]), "r"(r[at + 4]), "r"(r[at + 5]),
                 "r"(r[at + 6]), "r"(r[at + 7]) : "memory");
}

// A row's attention again, without the tensor cores, over the keys it sees and no others (half of its columns, gated): what a
// row takes whose sums are not finite.  Weights of hidden keys are zero, and zero times a value that is not finite is NaN; a
// token of a portion must not spoil the rows before it, nor one behind their window those after it.  q: the row's head; k: the
// head's [k | v] of the first of `keys` keys; r: their rotated parts.
__device__ __noinline__ void lp_row_again(const bf16* __restrict__ q, const bf16* __restrict__ k, size_t k_stride, const bf16* __restrict__ r,
                                          size_t r_stride, int keys, int half, float scale_log2e, float gate, bf16* __restrict__ out) {
    float m = -CUDART_INF_F, l = 0.0f, acc[64];
#pragma unroll
    for (int c = 0; c < 64; ++c) acc[c] = 0.0f;
#pragma unroll 1
    for (int j = 0; j < keys; ++j, k += k_stride, r += r_stride) {
        float s = 0.0f;
#pragma unroll 1
        for (int c = 0; c < LP_DK; c += 8) {
            float a[8], b[8];
            load8(q + c, a);
            load8(c < 128 ? k + c : r + c - 128, b);
#pragma unroll
            for (int i = 0; i < 8; ++i) s = fmaf(a[i], b[i], s);
        }
        s *= scale_log2e;
        if (s != s) {                                             // a key that the row sees is NaN: so is the row
            l = s;
            break;
        }
        const float top = fmaxf(m, s), base = top == -CUDART_INF_F ? 0.0f : top;
        const float alpha = t5_ex2(m - base), p = t5_ex2(s - base);
        l = fmaf(l, alpha, p);
        m = top;
#pragma unroll
        for (int c = 0; c < 64; c += 8) {
            float v[8];
            load8(k + 128 + half * 64 + c, v);
#pragma unroll
            for (int i = 0; i < 8; ++i) acc[c + i] = fmaf(p, v[i], acc[c + i] * alpha);
        }
    }
    const float inv = l == 0.0f ? 0.0f : gate / l;
#pragma unroll
    for (int c = 0; c < 64; c += 8) {
        float v[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = acc[c + i] * inv;
        store8(out + c, v);
    }
}

// grid (H, work items).  tiles: int32 [n][2] = (segment, first query row inside the portion), 256 rows each, longest walk
// first; segs: int32 [segments][4] = (entry, first position gathered, first gathered row, rows).
__global__ void __launch_bounds__(LP_THREADS, 1) latent_prefill_tcgen05_kernel(
    const __grid_constant__ CUtensorMap q_map, const __grid_constant__ CUtensorMap kv_map, const __grid_constant__ CUtensorMap r_map,
    bf16* __restrict__ out, const int32_t* __restrict__ tiles, const int32_t* __restrict__ segs,
    const int32_t* __restrict__ entry_q_start, const int32_t* __restrict__ entry_q_len, const int32_t* __restrict__ entry_kv_len,
    int H, int R, int window, float scale_log2e, const float* __restrict__ gate, long long gate_stride, int32_t* __restrict__ status,
    const bf16* __restrict__ q, const bf16* __restrict__ kv, const bf16* __restrict__ gathered) {
    pdl_begin();
    extern __shared__ unsigned char smem_dyn[];
    unsigned char* smem_al = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_dyn) + 1023) & ~uintptr_t(1023));
    bf16* q_s = reinterpret_cast<bf16*>(smem_al);                 // [2 query tiles][3 blocks][128][64]
    bf16* k_s = q_s + 2 * 3 * LP_QB;                              // [stages][3][96][64]
    bf16* v_s = k_s + LP_STAGES * 3 * LP_KB;                      // [stages][2][96][64]
    __shared__ __align__(8) unsigned long long q_full, k_full[LP_STAGES], k_empty[LP_STAGES], v_full[LP_STAGES], v_empty[LP_STAGES],
        s_full[2], p_full[2][2], pv_half[2], pv_done[2];
    __shared__ unsigned tmem_base_s;
    __shared__ int abort_flag;

    const int h = blockIdx.x;
    const int seg = tiles[2 * blockIdx.y], q0 = tiles[2 * blockIdx.y + 1];
    const int e = segs[4 * seg], first_pos = segs[4 * seg + 1], kv_row0 = segs[4 * seg + 2];
    const int q_len = entry_q_len[e];
    const int past = entry_kv_len[e] - q_len - first_pos;         // positions are counted from the first gathered row
    const int row_base = entry_q_start[e] + q0;
    const int rows_all = min(2 * LP_BM, q_len - q0);
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    auto rows_of = [&](int g) { return max(0, min(LP_BM, rows_all - g * LP_BM)); };
    const int k_lo = first_visible(past + q0, window) / LP_BN * LP_BN;      // the earliest key of the earliest row
    auto tiles_of = [&](int g) {                                  // key tiles that query tile g walks, all from k_lo
        const int rows = rows_of(g);
        return rows > 0 ? (past + q0 + g * LP_BM + rows - 1 - k_lo) / LP_BN + 1 : 0;
    };
    const int n0 = tiles_of(0), n1 = tiles_of(1), n_tiles = max(n0, n1);

    if (tid == 0) {
        abort_flag = 0;
        t5_mbar_init(&q_full, 1);
        for (int s = 0; s < LP_STAGES; ++s) {
            t5_mbar_init(&k_full[s], 1); t5_mbar_init(&k_empty[s], 1);
            t5_mbar_init(&v_full[s], 1); t5_mbar_init(&v_empty[s], 1);
        }
        for (int g = 0; g < 2; ++g) {
            t5_mbar_init(&s_full[g], 1);
            for (int hf = 0; hf < 2; ++hf) t5_mbar_init(&p_full[g][hf], 4);      // a softmax warp each
            t5_mbar_init(&pv_half[g], 1);
            t5_mbar_init(&pv_done[g], 1);
        }
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(t5_smem(&tmem_base_s)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    t5_fence_before();
    __syncthreads();
    t5_fence_after();
    const unsigned tmem = __shfl_sync(0xffffffffu, tmem_base_s, 0);
    auto s_col = [](int g) { return static_cast<unsigned>(g * 128); };           // 96 columns used
    auto o_col = [](int g) { return static_cast<unsigned>(256 + g * 128); };

    if (warp == 0) {
        // ---- producer: one thread, eleven boxes at most a tile ----
        if (lane == 0) {
            t5_expect_tx(&q_full, 2 * 3 * LP_QB * sizeof(bf16));
#pragma unroll
            for (int g = 0; g < 2; ++g)
#pragma unroll
                for (int b = 0; b < 3; ++b)
                    t5_tma_2d(q_s + (g * 3 + b) * LP_QB, &q_map, h * LP_DK + 64 * b, row_base + g * LP_BM, &q_full);
            int issued = 0;
            bool ok = true;
            for (int j = 0; j < n_tiles; ++j) {
                const int st = j % LP_STAGES, y = kv_row0 + k_lo + j * LP_BN;
                if (j >= LP_STAGES && !t5_wait(&k_empty[st], ((j / LP_STAGES) - 1) & 1, &abort_flag, status, row_base)) { ok = false; break; }
                t5_expect_tx(&k_full[st], 3 * LP_KB * sizeof(bf16));
                bf16* kd = k_s + st * 3 * LP_KB;
                t5_tma_2d(kd, &kv_map, h * 256, y, &k_full[st]);
                t5_tma_2d(kd + LP_KB, &kv_map, h * 256 + 64, y, &k_full[st]);
                t5_tma_2d(kd + 2 * LP_KB, &r_map, R, y, &k_full[st]);
                issued = 2 * j + 1;
                if (j >= LP_STAGES && !t5_wait(&v_empty[st], ((j / LP_STAGES) - 1) & 1, &abort_flag, status, row_base)) { ok = false; break; }
                t5_expect_tx(&v_full[st], 2 * LP_KB * sizeof(bf16));
                bf16* vd = v_s + st * 2 * LP_KB;
                t5_tma_2d(vd, &kv_map, h * 256 + 128, y, &v_full[st]);
                t5_tma_2d(vd + LP_KB, &kv_map, h * 256 + 192, y, &v_full[st]);
                issued = 2 * j + 2;
            }
            if (!ok || abort_flag) {                              // let what is in flight land before the CTA goes away
                for (int i = 0; i < T5_WAIT_LIMIT && !t5_try_wait(&q_full, 0); ++i) {}
                const int nk = (issued + 1) / 2, nv = issued / 2;
                for (int j = max(0, nk - LP_STAGES); j < nk; ++j)
                    for (int i = 0; i < T5_WAIT_LIMIT && !t5_try_wait(&k_full[j % LP_STAGES], (j / LP_STAGES) & 1); ++i) {}
                for (int j = max(0, nv - LP_STAGES); j < nv; ++j)
                    for (int i = 0; i < T5_WAIT_LIMIT && !t5_try_wait(&v_full[j % LP_STAGES], (j / LP_STAGES) & 1); ++i) {}
            }
        }
    } else if (warp == 1) {
        // ---- MMA issuer: S0(j), O1 += P1 V(j-1), S1(j), O0 += P0 V(j); a query tile takes part while it has keys ----
        // All lanes walk the loop, one of them issues.
        constexpr unsigned IDESC_QK = t5_idesc(LP_BM, LP_BN, 0);
        constexpr unsigned IDESC_PV = t5_idesc(LP_BM, LP_DV, 1);
        const unsigned lead = elect_one();
        const unsigned long long qd0 = t5_desc(q_s, 16, 1024), kd0 = t5_desc(k_s, 16, 1024);
        const unsigned long long vd0 = t5_desc(v_s, LP_KB * sizeof(bf16), 1024);
        constexpr unsigned long long K_STEP = (3 * LP_KB * sizeof(bf16)) >> 4, V_STEP = (2 * LP_KB * sizeof(bf16)) >> 4;
        auto qk = [&](int g, int st) {
#pragma unroll
            for (int k = 0; k < 12; ++k)
                t5_mma_ss_lead(lead, tmem + s_col(g), qd0 + g * ((3 * LP_QB * sizeof(bf16)) >> 4) + (((k >> 2) * LP_QB + (k & 3) * 16) * sizeof(bf16) >> 4),
                               kd0 + st * K_STEP + (((k >> 2) * LP_KB + (k & 3) * 16) * sizeof(bf16) >> 4), IDESC_QK, k > 0);
            t5_commit_lead(lead, &s_full[g]);
        };
        auto pv = [&](int g, int j, int st) -> bool {             // in two halves, each as soon as its weights are there
#pragma unroll
            for (int hf = 0; hf < 2; ++hf) {
                if (!t5_wait_warp(&p_full[g][hf], j & 1, &abort_flag, status, row_base)) return false;
                t5_fence_after();
#pragma unroll
                for (int k = 3 * hf; k < 3 * hf + 3; ++k)
                    t5_mma_ts_lead(lead, tmem + o_col(g), tmem + s_col(g) + k * 8, vd0 + st * V_STEP + ((k * 16 * 64) * sizeof(bf16) >> 4),
                                   IDESC_PV, (j > 0 || k > 0) ? 1u : 0u);
                t5_commit_lead(lead, hf ? &pv_done[g] : &pv_half[g]);
            }
            return true;
        };
        bool ok = t5_wait_warp(&q_full, 0, &abort_flag, status, row_base);
#pragma unroll 1
        for (int j = 0; ok && j < n_tiles; ++j) {
            const int st = j & 1;
            ok = t5_wait_warp(&k_full[st], (j >> 1) & 1, &abort_flag, status, row_base);
            if (!ok) break;
            t5_fence_after();
            if (j < n0) qk(0, st);
            if (j > 0) {
                if (j - 1 < n1) {
                    ok = pv(1, j - 1, 1 - st);
                    if (!ok) break;
                }
                t5_commit_lead(lead, &v_empty[1 - st]);           // the last reader of the values of tile j - 1
            }
            if (j < n1) qk(1, st);
            t5_commit_lead(lead, &k_empty[st]);
            ok = t5_wait_warp(&v_full[st], (j >> 1) & 1, &abort_flag, status, row_base);
            if (ok && j < n0) ok = pv(0, j, st);
        }
        static_assert(LP_STAGES == 2, "a tile's stage is its parity");
        if (ok && n1 == n_tiles) pv(1, n1 - 1, (n1 - 1) & 1);
    } else if (warp >= 4) {
        // ---- softmax: a thread owns one query row = one TMEM lane, all 96 columns of a tile ----
        const int g = (warp - 4) >> 2;                            // warps 4..7: the first query tile, 8..11: the second
        const int quarter = warp & 3;
        const int row = quarter * 32 + lane;
        const unsigned lane_addr = static_cast<unsigned>(quarter * 32) << 16;
        const unsigned my_s = tmem + lane_addr + s_col(g);
        const unsigned my_o = tmem + lane_addr + o_col(g);
        const int rows_here = rows_of(g), mine = g ? n1 : n0;
        // rows behind the portion's last are other tokens' or zeros: they are worked like the rest and not stored
        const int pos_first = past + q0 + g * LP_BM, pos = pos_first + row;
        const int lo = first_visible(pos, window), lo_last = first_visible(pos_first + rows_here - 1, window);
        float m = -CUDART_INF_F, l = 0.0f;                        // m: the reference maximum, in units of log2
        bool ok = true;
        for (int j = 0; j < mine; ++j) {
            const int kt = k_lo + j * LP_BN;
            // after a wait has run out (ok false, for whole warps) a thread touches nothing else
            if (ok) ok = __all_sync(0xffffffffu, t5_wait(&s_full[g], j & 1, &abort_flag, status, row_base));
            if (!ok) break;
            t5_fence_after();
            const bool full_tile = (kt + LP_BN - 1 <= pos_first) && (kt >= lo_last);
            unsigned r[48];
            auto fetch = [&](int hf) {                            // 48 scores of the row, what it does not see at -inf
                lp_ld16(my_s + 48 * hf, r, 0);
                lp_ld16(my_s + 48 * hf + 16, r, 16);
                lp_ld16(my_s + 48 * hf + 32, r, 32);
                t5_wait_ld();
                if (!full_tile) {
                    const int k0 = kt + 48 * hf;
                    auto first = [&](int n) { return n <= 0 ? 0ull : n >= 48 ? (1ull << 48) - 1ull : (1ull << n) - 1ull; };
                    const unsigned long long seen = first(pos + 1 - k0) & ~first(lo - k0);
#pragma unroll
                    for (int i = 0; i < 48; ++i) r[i] = seen & (1ull << i) ? r[i] : 0xff800000u;
                }
            };
            auto max_of = [&] {
                float a = __uint_as_float(r[0]), b = __uint_as_float(r[1]);
#pragma unroll
                for (int i = 2; i < 48; i += 2) { a = fmaxf(a, __uint_as_float(r[i])); b = fmaxf(b, __uint_as_float(r[i + 1])); }
                return fmaxf(a, b);
            };
            auto weights = [&](unsigned (&pk)[24]) {              // rounded to bfloat16, and their sum
                const float ref = m == -CUDART_INF_F ? 0.0f : m;
                const unsigned long long e2 = t5_two(scale_log2e, scale_log2e), m2 = t5_two(-ref, -ref);
                float s0 = 0.0f, s1 = 0.0f;
#pragma unroll
                for (int i = 0; i < 48; i += 2) {
                    float x0, x1;
                    t5_untwo(t5_fma2(t5_two(__uint_as_float(r[i]), __uint_as_float(r[i + 1])), e2, m2), x0, x1);
                    const float p0 = t5_ex2(x0), p1 = t5_ex2(x1);
                    pk[i >> 1] = t5_pack(p0, p1);
                    s0 += p0;
                    s1 += p1;
                }
                return s0 + s1;
            };
            // The row's reference moves up to mx when that has run away from it; O and l move too, once the products under way
            // have joined O.
            auto move_to = [&](float mx, unsigned long long* done, int parity) {
                const bool adopt = (m == -CUDART_INF_F) && (mx > m), jump = (m != -CUDART_INF_F) && (mx > m + LP_JUMP);
                if (__any_sync(0xffffffffu, jump)) {
                    ok = __all_sync(0xffffffffu, t5_wait(done, parity, &abort_flag, status, row_base));
                    if (!ok) return;
                    t5_fence_after();
                    const float alpha = jump ? t5_ex2(m - mx) : 1.0f;
                    l *= alpha;
#pragma unroll 1
                    for (int c = 0; c < LP_DV; c += 32) {
                        unsigned o[32];
                        t5_ld32(my_o + c, o);
                        t5_wait_ld();
#pragma unroll
                        for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
                        t5_st32(my_o + c, o);
                    }
                }
                if (adopt || jump) m = mx;
            };
            if (j == 0) {                                         // the first tile's maximum before its weights
                fetch(0);
                const float mx = max_of();
                fetch(1);
                move_to(fmaxf(mx, max_of()) * scale_log2e, nullptr, 0);       // scale > 0; -inf stays -inf; nothing to wait for
            }
#pragma unroll 1
            for (int hf = 0; hf < 2; ++hf) {
                unsigned pk[24];
                fetch(hf);
                // after that the weights are made at the reference that is there, beside their maximum, and again if it has to move
                const float mx = j == 0 ? m : max_of() * scale_log2e;
                float sum = weights(pk);
                if (__any_sync(0xffffffffu, mx > (m == -CUDART_INF_F ? m : m + LP_JUMP))) {
                    move_to(mx, hf ? &pv_half[g] : &pv_done[g], (hf ? j : j - 1) & 1);
                    if (!ok) break;
                    fetch(hf);
                    sum = weights(pk);
                }
                l += sum;
                lp_st8(my_s + 24 * hf, pk, 0);                    // over columns of S that have been read
                lp_st8(my_s + 24 * hf + 8, pk, 8);
                lp_st8(my_s + 24 * hf + 16, pk, 16);
                t5_wait_st();
                t5_fence_before();
                __syncwarp();
                if (lane == 0) t5_arrive(&p_full[g][hf]);
            }
        }
        if (ok && mine > 0 && __all_sync(0xffffffffu, t5_wait(&pv_done[g], (mine - 1) & 1, &abort_flag, status, row_base))) {
            t5_fence_after();
            float inv = (l > 0.0f) ? 1.0f / l : 0.0f;
            if (gate && row < rows_here)                          // a sigmoid gate per token and head, on the result as it leaves
                inv /= 1.0f + expf(-gate[static_cast<size_t>(row_base + g * LP_BM + row) * gate_stride + h]);
            bool finite = l <= 3.402823466e38f;                   // not infinite, not NaN
            bf16* orow = out + (static_cast<size_t>(row_base + g * LP_BM + row) * H + h) * LP_DV;
#pragma unroll 1
            for (int c = 0; c < LP_DV; c += 32) {
                unsigned o[32];
                t5_ld32(my_o + c, o);
                t5_wait_ld();
#pragma unroll
                for (int i = 0; i < 32; ++i) finite = finite && fabsf(__uint_as_float(o[i])) <= 3.402823466e38f;
                if (row < rows_here) {
#pragma unroll
                    for (int i = 0; i < 32; i += 8) {
                        uint4 w;
                        w.x = t5_pack(__uint_as_float(o[i]) * inv, __uint_as_float(o[i + 1]) * inv);
                        w.y = t5_pack(__uint_as_float(o[i + 2]) * inv, __uint_as_float(o[i + 3]) * inv);
                        w.z = t5_pack(__uint_as_float(o[i + 4]) * inv, __uint_as_float(o[i + 5]) * inv);
                        w.w = t5_pack(__uint_as_float(o[i + 6]) * inv, __uint_as_float(o[i + 7]) * inv);
                        *reinterpret_cast<uint4*>(orow + c + i) = w;
                    }
                }
            }
            if (row < rows_here && !finite) {
                const size_t token = static_cast<size_t>(row_base + g * LP_BM + row), at = static_cast<size_t>(kv_row0 + max(lo, 0));
                const float share = gate ? 1.0f / (1.0f + expf(-gate[token * gate_stride + h])) : 1.0f;
#pragma unroll 1
                for (int half = 0; half < 2; ++half)
                    lp_row_again(q + (token * H + h) * LP_DK, kv + (at * H + h) * 256, static_cast<size_t>(H) * 256,
                                 gathered + at * (R + 64) + R, R + 64, pos - max(lo, 0) + 1, half, scale_log2e, share, orow + half * 64);
            }
        }
    }
    t5_fence_before();
    __syncthreads();
    if (warp == 1) {
        t5_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(512u) : "memory");
    }
}

// ---- the rows of the portions, and the queries --------------------------------------------------------------------
// grid (row groups of 8, segments), a warp a row: position first + i of the segment's request, zeros beyond its last one.
__global__ void latent_gather_kernel(const bf16* __restrict__ rows_cache, long long page_stride, bf16* __restrict__ out,
                                     const int32_t* __restrict__ segs, const int32_t* __restrict__ entry_slot,
                                     const int32_t* __restrict__ entry_kv_len, const int32_t* __restrict__ block_table,
                                     int table_stride, int DK, int page_size, int num_pages, int32_t* __restrict__ status) {
    pdl_begin();
    const int* s = segs + 4 * blockIdx.y;
    const int i = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (i >= s[3]) return;
    const int e = s[0], pos = s[1] + i;
    const bf16* src = nullptr;
    if (pos < entry_kv_len[e]) {
        const int logical = pos / page_size;
        const int page = logical < table_stride ? block_table[static_cast<size_t>(entry_slot[e]) * table_stride + logical] : -1;
        if (page < 0 || page >= num_pages) {
            if (lane == 0 && atomicCAS(status, 0, 4) == 0) status[1] = s[2] + i;
        } else {
            src = rows_cache + static_cast<long long>(page) * page_stride + static_cast<size_t>(pos - logical * page_size) * DK;
        }
    }
    bf16* dst = out + static_cast<size_t>(s[2] + i) * DK;
    for (int c = lane; c < DK / 8; c += 32)
        *reinterpret_cast<uint4*>(dst + 8 * c) = src ? *reinterpret_cast<const uint4*>(src + 8 * c) : make_uint4(0u, 0u, 0u, 0u);
}

// One block a token: q float32 [T, H * (D + P)] -> bfloat16 of the same layout, the first `dims` entries of every head's
// P-part rotated (pairs as in latent_attention.cu).  The angles of a token are made once for all heads.  2,000 tokens of 32 heads of
// 128 + 64: 20 -> 16 us with four heads of a thread on their way before the angles are made.
#define LQ_HELD 4
template <bool WIDE>          // heads of more eights than a block has threads: a row of blocks
__global__ void __launch_bounds__(1024) latent_q_pack_kernel(const float* __restrict__ q, bf16* __restrict__ out, const int32_t* __restrict__ positions,
                                     const float* __restrict__ inv_freq, int H, int D, int P, int dims, int rot_pairs, float rot_mag) {
    pdl_begin();
    extern __shared__ float2 turn[];                              // (cos, sin) of the token's angles, times the magnitude
    const int t = blockIdx.x, half = dims / 2, W = D + P;
    const float* src = q + static_cast<size_t>(t) * H * W;
    bf16* dst = out + static_cast<size_t>(t) * H * W;
    // a thread keeps its place in the head and goes from head to head, LQ_HELD heads on their way at once
    const int per = WIDE ? 1 : blockDim.x / (W / 8), c = static_cast<int>(WIDE ? blockIdx.y * blockDim.x + threadIdx.x : threadIdx.x % (W / 8)) * 8;
    const int k0 = c - D, h0 = WIDE ? 0 : threadIdx.x / (W / 8);
    const int heads = WIDE && c >= W ? 0 : H;
    const bool whole = k0 >= 0 && k0 + 8 <= dims && (rot_pairs || half % 8 == 0);      // all eight turn, with neighbours or with eight others
    const bool first = k0 < half;
    const int f0 = rot_pairs ? k0 >> 1 : first ? k0 : k0 - half;
    for (int hb = h0; hb < heads || hb == h0; hb += LQ_HELD * per) {
        float v[LQ_HELD][8];
#pragma unroll
        for (int j = 0; j < LQ_HELD; ++j)
            if (hb + j * per < heads) load8(src + (hb + j * per) * W + c, v[j]);
        if (hb == h0) {
            const float pos = static_cast<float>(positions[t]);
            for (int f = threadIdx.x; f < half; f += blockDim.x) {
                float sn, cs;
                sincosf(pos * inv_freq[f], &sn, &cs);
                turn[f] = make_float2(cs * rot_mag, sn * rot_mag);
            }
            __syncthreads();
        }
#pragma unroll
        for (int j = 0; j < LQ_HELD; ++j) {
            const int h = hb + j * per;
            if (h >= heads) break;
            const float* hd = src + h * W;
            if (whole && rot_pairs) {
#pragma unroll
                for (int u = 0; u < 8; u += 2) {
                    const float2 cs = turn[f0 + (u >> 1)];
                    const float x = v[j][u], y = v[j][u + 1];
                    v[j][u] = x * cs.x - y * cs.y;
                    v[j][u + 1] = y * cs.x + x * cs.y;
                }
            } else if (whole) {
                float other[8];
                load8(hd + c + (first ? half : -half), other);
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    const float2 cs = turn[f0 + u];
                    v[j][u] = first ? v[j][u] * cs.x - other[u] * cs.y : v[j][u] * cs.x + other[u] * cs.y;
                }
            } else if (k0 >= 0) {
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    const int k = k0 + u;
                    if (k < dims) {
                        const bool low = rot_pairs ? (k & 1) == 0 : k < half;
                        const int f = rot_pairs ? k >> 1 : (low ? k : k - half);
                        const float other = hd[D + (rot_pairs ? k ^ 1 : (low ? k + half : k - half))];
                        const float2 cs = turn[f];
                        v[j][u] = low ? v[j][u] * cs.x - other * cs.y : v[j][u] * cs.x + other * cs.y;
                    }
                }
            }
            store8(dst + h * W + c, v[j]);
        }
    }
}

extern "C" int llm_latent_prefill_supported(int D, int V, int R, int P) {
    return D == 128 && V == LP_DV && P == 64 && R > 0 && R % 8 == 0;
}

// rows_cache: bfloat16 [pages, 1, page, DK] with `page_stride`; out: bfloat16 [total rows, DK]; segs as above, every first
// gathered row and row count a multiple of the key tile; most_rows: the largest count.
extern "C" int llm_latent_gather(const void* rows_cache, long long page_stride, void* out, const int32_t* segs, int n_segs,
                                 int most_rows, const int32_t* entry_slot, const int32_t* entry_kv_len,
                                 const int32_t* block_table, int table_stride, int DK, int page_size, int num_pages,
                                 int32_t* status, uintptr_t stream) {
    if (n_segs <= 0 || most_rows <= 0) return LLM_OK;
    if (n_segs > 65535 || DK <= 0 || DK % 8 || page_size <= 0) return LLM_REFUSED_SIZE;
    if (!aligned16(rows_cache) || !aligned16(out) || page_stride % 8) return LLM_REFUSED_ALIGN;
    launch_pdl(latent_gather_kernel, dim3((most_rows + 7) / 8, n_segs), dim3(256), 0, reinterpret_cast<cudaStream_t>(stream),
               static_cast<const bf16*>(rows_cache), page_stride, static_cast<bf16*>(out), segs, entry_slot, entry_kv_len,
               block_table, table_stride, DK, page_size, num_pages, status);
    return launch_status();
}

extern "C" int llm_latent_q_pack(const float* q, void* out, const int32_t* positions, const float* inv_freq, int num_tokens, int H,
                                 int D, int P, int dims, int rot_pairs, float rot_mag, uintptr_t stream) {
    if (num_tokens <= 0) return LLM_OK;
    if (H <= 0 || D <= 0 || P < 0 || D % 8 || P % 8 || dims < 0 || dims > P || dims % 2 || (dims > 0 && !inv_freq)) return LLM_REFUSED_SIZE;
    if (!aligned16(q) || !aligned16(out)) return LLM_REFUSED_ALIGN;
    const int eights = (D + P) / 8;                               // threads: as many whole heads as 256 of them hold, or one, or a part of it
    const int threads = eights > 1024 ? 1024 : eights > 256 ? eights : 256 / eights * eights, parts = (eights + 1023) / 1024;
    if (parts > 65535) return LLM_REFUSED_SIZE;
    launch_pdl(parts > 1 ? latent_q_pack_kernel<true> : latent_q_pack_kernel<false>, dim3(num_tokens, parts), dim3(threads),
               sizeof(float2) * (dims / 2), reinterpret_cast<cudaStream_t>(stream), q, static_cast<bf16*>(out), positions, inv_freq, H, D, P,
               dims, rot_pairs, rot_mag);
    return launch_status();
}

// q: bfloat16 [num_tokens, H * 192]; kv: bfloat16 [rows, H * 256] = per head [k | v]; gathered: bfloat16 [rows, R + 64];
// out: bfloat16 [num_tokens, H * 128]; tile_rows, tile_keys: what the caller cut its tiles to and padded its segments to,
// which have to be this kernel's; gate: null, or float32, token t's and head h's at t * gate_stride + h, the result is
// multiplied by its sigmoid.
extern "C" int llm_latent_prefill(const void* q, const void* kv, const void* gathered, void* out, int num_tokens, int rows,
                                  const int32_t* tiles, int n_tiles, int tile_rows, int tile_keys, const int32_t* segs,
                                  const int32_t* entry_q_start, const int32_t* entry_q_len, const int32_t* entry_kv_len, int H, int R,
                                  int window, float scale, const float* gate, long long gate_stride, int32_t* status, uintptr_t stream) {
    if (n_tiles <= 0) return LLM_OK;
    if (H <= 0 || n_tiles > 65535 || tile_rows != 2 * LP_BM || tile_keys != LP_BN || !llm_latent_prefill_supported(128, LP_DV, R, 64) ||
        rows <= 0 || rows % LP_BN || !(scale > 0.0f) || window < 0)
        return LLM_REFUSED_SIZE;
    if (!aligned16(q) || !aligned16(kv) || !aligned16(gathered) || !aligned16(out)) return LLM_REFUSED_ALIGN;
    CUtensorMap q_map, kv_map, r_map;
    if (!t5_encode_2d(&q_map, q, static_cast<long long>(H) * LP_DK, num_tokens, 64, LP_BM) ||
        !t5_encode_2d(&kv_map, kv, static_cast<long long>(H) * 256, rows, 64, LP_BN) ||
        !t5_encode_2d(&r_map, gathered, R + 64, rows, 64, LP_BN))
        return LLM_REFUSED_SIZE;
    const size_t smem = static_cast<size_t>(2 * 3 * LP_QB + LP_STAGES * 5 * LP_KB) * sizeof(bf16) + 1024;
    const cudaError_t e = cudaFuncSetAttribute(latent_prefill_tcgen05_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    if (e != cudaSuccess) return static_cast<int>(e);
    launch_pdl(latent_prefill_tcgen05_kernel, dim3(H, n_tiles), dim3(LP_THREADS), smem, reinterpret_cast<cudaStream_t>(stream), q_map,
               kv_map, r_map, static_cast<bf16*>(out), tiles, segs, entry_q_start, entry_q_len, entry_kv_len, H, R, window,
               scale * 1.4426950408889634f, gate, gate_stride, status, static_cast<const bf16*>(q), static_cast<const bf16*>(kv),
               static_cast<const bf16*>(gathered));
    return launch_status();
}
