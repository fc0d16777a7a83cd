// Paged causal attention for prompt portions on the 5th-generation tensor cores: tcgen05.mma with
// accumulators in tensor memory (TMEM), operands fetched by TMA, bfloat16, head size 128.
//
// A CTA takes 128 consecutive query rows of one request for one query head (a tile of the same
// host-built list the mma.sync kernel uses) and walks the request's keys in tiles of 64, TWICE:
//   pass A:  S = Q K^T (tcgen05.mma, M 128 x N 64 x K 128 -> TMEM), row maxima m over visible keys;
//   pass B:  S again, P = exp2(S*scale*log2e - m) (exact softmax numerators: m is final, so the
//            output accumulator never has to be rescaled), l += row sums, P rounded to bfloat16
//            goes back into TMEM, O += P V (tcgen05.mma with A from TMEM, V as an MN-major
//            shared-memory operand), and at the end out = O / l.
// Running S twice costs half as much again in tensor work and removes the correction step of
// the running-maximum form (src/ops/attention.cu:204-249) from the critical path; the numbers
// are those of a two-pass softmax (src/ops/paged_attention.cpp:159-217).
//
// A CTA serves TWO query heads of the same kv head when the group size is even (one otherwise):
// they share every key/value tile in shared memory, which halves the L2 traffic and the number
// of copy-engine operations per unit of tensor work (with 16-token pages a tile is 4 pages x 2
// halves x K and V = 16 boxes of 2 KB, and the copy engine's time per box is what the first
// version of this kernel waited for).
// Roles: warp 0 feeds the copy engine (Q once, then K or K+V tiles, four stages); one lane of
// warp 1 issues the MMAs and owns the TMEM allocation; then four softmax warps per head: a
// thread owns one query row = one TMEM lane (a warp can only reach the 32 lanes of its quarter).
// Per head S is double-buffered in TMEM and P overwrites the first half of its own S in place
// (S0 S1 O = 64+64+128 = 256 columns per head), so the S of the next tile is computed while the
// softmax of this one runs.
// Every mbarrier wait is bounded; on a timeout the CTA raises an abort flag, records status
// code 6, lets its copies land (bounded) and frees its TMEM before it returns.
#include "tcgen05_attention.cuh"
#include <math_constants.h>

#define T5_BM 128
#define T5_BN 64
#define T5_D 128
#define T5_QHALF (T5_BM * 64)                 // elements of one 64-column half of the 128-row query tile
#define T5_HALF (T5_BN * 64)                  // elements of one 64-column half of a key or value tile
#define T5_TILE (2 * T5_HALF)

// HEADS query heads of one kv head share every key/value tile (HEADS = 2 when the group size is
// even, else 1); STAGES key/value tiles sit in shared memory.
template <int HEADS, int STAGES>
__global__ void __launch_bounds__(64 + 128 * HEADS, 1) paged_prefill_attention_tcgen05_kernel(
    const __grid_constant__ CUtensorMap q_map, const __grid_constant__ CUtensorMap kv_map, bf16* __restrict__ out,
    const int32_t* __restrict__ tiles, const int32_t* __restrict__ entry_slot, const int32_t* __restrict__ entry_q_start,
    const int32_t* __restrict__ entry_q_len, const int32_t* __restrict__ entry_kv_len,
    const int32_t* __restrict__ block_table, int table_stride, int nq, int nkv, int page_size, int window,
    float scale_log2e, int num_pages, int32_t* __restrict__ status) {
    pdl_begin();
    constexpr int SOFTMAX_THREADS = 128 * HEADS;
    constexpr unsigned TMEM_COLS = 256 * HEADS;                   // per head: S0 S1 (64 each) and O (128)
    extern __shared__ unsigned char smem_dyn[];
    unsigned char* smem_al = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_dyn) + 1023) & ~uintptr_t(1023));
    bf16* q_s = reinterpret_cast<bf16*>(smem_al);                 // [HEADS][2][128][64]
    bf16* k_s = q_s + HEADS * 2 * T5_QHALF;                       // [STAGES][2][BN][64]
    bf16* v_s = k_s + STAGES * T5_TILE;                           // [STAGES][2][BN][64]
    __shared__ __align__(8) unsigned long long q_full, kv_full[STAGES], kv_empty[STAGES], s_full[2], s_read[2],
        p_full[2], s_used[2], o_done;
    __shared__ unsigned tmem_base_s;
    __shared__ int abort_flag;

    // Heads vary fastest: CTAs are handed to SMs in this order, and the tile list has the most
    // expensive tiles first, so those start first whatever the number of heads.
    const int tile = blockIdx.y;
    const int h0 = blockIdx.x * HEADS;                            // first query head of this CTA
    const int kvh = h0 / (nq / nkv);
    const int e = tiles[2 * tile], q0 = tiles[2 * tile + 1];
    if (e < 0) return;                                            // a padding entry of the tile list: no work
    const int q_len = entry_q_len[e], kv_len = entry_kv_len[e];
    const int past = kv_len - q_len;
    const int row_base = entry_q_start[e] + q0;
    const int rows_here = min(T5_BM, q_len - q0);
    const int32_t* table = block_table + static_cast<size_t>(entry_slot[e]) * table_stride;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int pos_first = past + q0, pos_last = past + q0 + rows_here - 1;
    const int k_lo = first_visible(pos_first, window) / T5_BN * T5_BN;
    const int n_tiles = (pos_last - k_lo) / T5_BN + 1;
    const int total = 2 * n_tiles;                                // pass A then pass B over the same tiles

    if (tid == 0) {
        abort_flag = 0;
        t5_mbar_init(&q_full, 1);
        for (int s = 0; s < STAGES; ++s) { t5_mbar_init(&kv_full[s], 1); t5_mbar_init(&kv_empty[s], 1); }
        for (int s = 0; s < 2; ++s) {
            t5_mbar_init(&s_full[s], 1);
            t5_mbar_init(&s_read[s], SOFTMAX_THREADS);   // pass A: every softmax thread has read its row of S
            t5_mbar_init(&p_full[s], SOFTMAX_THREADS);   // pass B: every softmax thread has put its row of P over S
            t5_mbar_init(&s_used[s], 1);                 // pass B: the P V products that read this buffer have finished
        }
        t5_mbar_init(&o_done, 1);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == 1) {                                              // one warp allocates this CTA's TMEM columns
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(t5_smem(&tmem_base_s)), "r"(TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    t5_fence_before();
    __syncthreads();
    t5_fence_after();
    const unsigned tmem = tmem_base_s;
    // columns of head g: S buffer b at g*256 + b*64, O at g*256 + 128; P lives in the first 32 columns of its S
    auto s_col = [](int g, int b) { return static_cast<unsigned>(g * 256 + b * 64); };
    auto o_col = [](int g) { return static_cast<unsigned>(g * 256 + 128); };

    if (warp == 0) {
        // ---- producer ----
        if (lane == 0) {
            t5_expect_tx(&q_full, HEADS * 2 * T5_QHALF * sizeof(bf16));
#pragma unroll
            for (int g = 0; g < HEADS; ++g) {
                t5_tma_2d(q_s + g * 2 * T5_QHALF, &q_map, (h0 + g) * T5_D, row_base, &q_full);
                t5_tma_2d(q_s + g * 2 * T5_QHALF + T5_QHALF, &q_map, (h0 + g) * T5_D + 64, row_base, &q_full);
            }
            const int boxes = T5_BN / page_size;
            const int last_logical = pos_last / page_size;
            int issued = 0;
            for (int u = 0; u < total; ++u) {
                const int st = u % STAGES, it = u % n_tiles;
                const bool with_v = u >= n_tiles;
                if (u >= STAGES && !t5_wait(&kv_empty[st], ((u / STAGES) - 1) & 1, &abort_flag, status, row_base)) break;
                t5_expect_tx(&kv_full[st], (with_v ? 2u : 1u) * T5_TILE * sizeof(bf16));
                const int first_logical = (k_lo + it * T5_BN) / page_size;
                for (int j = 0; j < boxes; ++j) {
                    const int logical = min(first_logical + j, last_logical);
                    int page = logical < table_stride ? __ldg(table + logical) : -1;
                    if (page < 0 || page >= num_pages) {
                        if (atomicCAS(status, 0, 4) == 0) status[1] = row_base;
                        page = 0;
                    }
                    const int k_row = ((page * 2) * nkv + kvh) * page_size;
                    const int v_row = ((page * 2 + 1) * nkv + kvh) * page_size;
#pragma unroll
                    for (int half = 0; half < 2; ++half) {
                        t5_tma_2d(k_s + st * T5_TILE + half * T5_HALF + j * page_size * 64, &kv_map, half * 64, k_row, &kv_full[st]);
                        if (with_v)
                            t5_tma_2d(v_s + st * T5_TILE + half * T5_HALF + j * page_size * 64, &kv_map, half * 64, v_row, &kv_full[st]);
                    }
                }
                issued = u + 1;
            }
            if (abort_flag)
                for (int u = max(0, issued - STAGES); u < issued; ++u)
                    for (int i = 0; i < T5_WAIT_LIMIT && !t5_try_wait(&kv_full[u % STAGES], (u / STAGES) & 1); ++i) {}
        }
    } else if (warp == 1) {
        // ---- MMA issuer ----
        if (lane == 0) {
            constexpr unsigned IDESC_QK = t5_idesc(T5_BM, T5_BN, 0);
            constexpr unsigned IDESC_PV = t5_idesc(T5_BM, T5_D, 1);
            bool ok = t5_wait(&q_full, 0, &abort_flag, status, row_base);
            // Descriptors are built once: a tile further on in shared memory is the same descriptor
            // plus its byte offset / 16 in the address field (one thread issues every product, so
            // what it computes per instruction is what limits the rate of issue).
            const unsigned long long qd0 = t5_desc(q_s, 16, 1024), kd0 = t5_desc(k_s, 16, 1024);
            const unsigned long long vd0 = t5_desc(v_s, T5_HALF * sizeof(bf16), 1024);
            constexpr unsigned long long STAGE_STEP = (T5_TILE * sizeof(bf16)) >> 4;
            auto issue_qk = [&](int u) -> bool {
                const int st = u % STAGES, sb = u & 1;
                if (!t5_wait(&kv_full[st], (u / STAGES) & 1, &abort_flag, status, row_base)) return false;
                if (u >= 2) {                                     // the buffer's previous tile must be done with it
                    const int prev = u - 2;
                    const bool a = prev < n_tiles;
                    if (!t5_wait(a ? &s_read[sb] : &s_used[sb], ((a ? prev : prev - n_tiles) >> 1) & 1, &abort_flag, status,
                                 row_base))
                        return false;
                }
                t5_fence_after();
#pragma unroll
                for (int g = 0; g < HEADS; ++g)
#pragma unroll
                    for (int k = 0; k < T5_D / 16; ++k) {
                        const unsigned long long qoff = ((g * 2 + (k >> 2)) * T5_QHALF + (k & 3) * 16) * sizeof(bf16) >> 4;
                        const unsigned long long koff = ((k >> 2) * T5_HALF + (k & 3) * 16) * sizeof(bf16) >> 4;
                        t5_mma_ss(tmem + s_col(g, sb), qd0 + qoff, kd0 + st * STAGE_STEP + koff, IDESC_QK, k > 0);
                    }
                t5_commit(&s_full[sb]);
                if (u < n_tiles) t5_commit(&kv_empty[st]);        // pass A: the keys are all this stage held
                return true;
            };
            if (ok && total > 0) ok = issue_qk(0);
            for (int u = 0; ok && u < total; ++u) {
                if (u + 1 < total) ok = issue_qk(u + 1);          // the next S while this tile's softmax runs
                if (!ok || u < n_tiles) continue;
                const int st = u % STAGES, sb = u & 1, v = u - n_tiles;
                if (!t5_wait(&p_full[sb], (v >> 1) & 1, &abort_flag, status, row_base)) { ok = false; break; }
                t5_fence_after();
#pragma unroll
                for (int g = 0; g < HEADS; ++g)
#pragma unroll
                    for (int k = 0; k < T5_BN / 16; ++k) {
                        const unsigned long long voff = (k * 16 * 64) * sizeof(bf16) >> 4;   // 16 keys further, both 64-column halves
                        t5_mma_ts(tmem + o_col(g), tmem + s_col(g, sb) + k * 8, vd0 + st * STAGE_STEP + voff,
                                  IDESC_PV, (v > 0 || k > 0) ? 1u : 0u);
                    }
                t5_commit(&kv_empty[st]);
                t5_commit(&s_used[sb]);
                if (u == total - 1) t5_commit(&o_done);
            }
        }
    } else {
        // ---- softmax: a thread owns one query row of one head = one TMEM lane, all 64 columns of a tile ----
        const int sw = warp - 2;
        const int g = sw >> 2;                                    // warps 2..5: head h0, warps 6..9: head h0 + 1
        const int quarter = warp & 3;                             // the TMEM lanes this warp may touch
        const int row = quarter * 32 + lane;
        const unsigned lane_addr = static_cast<unsigned>(quarter * 32) << 16;
        const int pos = (row < rows_here) ? past + q0 + row : -1;
        const int lo = first_visible(pos, window), lo_last = first_visible(pos_last, window);
        float m = -CUDART_INF_F, l = 0.0f;
        bool ok = true;
        for (int u = 0; ok && u < n_tiles; ++u) {                 // pass A: maxima
            const int sb = u & 1, kt = k_lo + u * T5_BN;
            if (!t5_wait(&s_full[sb], (u >> 1) & 1, &abort_flag, status, row_base)) { ok = false; break; }
            t5_fence_after();
            const bool full_tile = (kt + T5_BN - 1 <= pos_first) && (kt >= lo_last) && (rows_here == T5_BM);
            unsigned r[2][32];                                    // both halves of the row are requested at once
            t5_ld32(tmem + lane_addr + s_col(g, sb), r[0]);
            t5_ld32(tmem + lane_addr + s_col(g, sb) + 32, r[1]);
            t5_wait_ld();
            t5_fence_before();
            t5_arrive(&s_read[sb]);                               // S is in registers: the buffer may be overwritten
#pragma unroll
            for (int cc = 0; cc < 2; ++cc) {
                if (full_tile) {                                  // every row of the CTA sees every key of the tile
#pragma unroll
                    for (int i = 0; i < 32; ++i) m = fmaxf(m, __uint_as_float(r[cc][i]));
                } else {
#pragma unroll
                    for (int i = 0; i < 32; ++i) {
                        const int key = kt + cc * 32 + i;
                        if (key <= pos && key >= lo) m = fmaxf(m, __uint_as_float(r[cc][i]));
                    }
                }
            }
        }
        const float msub = (m == -CUDART_INF_F) ? 0.0f : m * scale_log2e;
        for (int u = n_tiles; ok && u < total; ++u) {             // pass B: numerators with the final maximum
            const int sb = u & 1, v = u - n_tiles, kt = k_lo + v * T5_BN;
            if (!t5_wait(&s_full[sb], (u >> 1) & 1, &abort_flag, status, row_base)) { ok = false; break; }
            t5_fence_after();
            const bool full_tile = (kt + T5_BN - 1 <= pos_first) && (kt >= lo_last) && (rows_here == T5_BM);
            unsigned pk[32], r[2][32];
            t5_ld32(tmem + lane_addr + s_col(g, sb), r[0]);
            t5_ld32(tmem + lane_addr + s_col(g, sb) + 32, r[1]);
            t5_wait_ld();
#pragma unroll
            for (int cc = 0; cc < 2; ++cc) {
                if (full_tile) {
#pragma unroll
                    for (int i = 0; i < 32; i += 2) {
                        const float p0 = t5_ex2(fmaf(__uint_as_float(r[cc][i]), scale_log2e, -msub));
                        const float p1 = t5_ex2(fmaf(__uint_as_float(r[cc][i + 1]), scale_log2e, -msub));
                        l += p0 + p1;
                        pk[(cc * 32 + i) >> 1] = t5_pack(p0, p1);
                    }
                } else {
#pragma unroll
                    for (int i = 0; i < 32; i += 2) {
                        const int key = kt + cc * 32 + i;
                        const float p0 = (key <= pos && key >= lo) ? t5_ex2(fmaf(__uint_as_float(r[cc][i]), scale_log2e, -msub)) : 0.0f;
                        const float p1 = (key + 1 <= pos && key + 1 >= lo) ? t5_ex2(fmaf(__uint_as_float(r[cc][i + 1]), scale_log2e, -msub)) : 0.0f;
                        l += p0 + p1;
                        pk[(cc * 32 + i) >> 1] = t5_pack(p0, p1);
                    }
                }
            }
            // the whole row of S is in registers: P goes over its first 32 columns
            {
                unsigned a[16], b[16];
#pragma unroll
                for (int i = 0; i < 16; ++i) { a[i] = pk[i]; b[i] = pk[16 + i]; }
                t5_st16(tmem + lane_addr + s_col(g, sb), a);
                t5_st16(tmem + lane_addr + s_col(g, sb) + 16, b);
            }
            t5_wait_st();
            t5_fence_before();
            t5_arrive(&p_full[sb]);
        }
        if (ok && t5_wait(&o_done, 0, &abort_flag, status, row_base)) {
            t5_fence_after();
            const float inv = (l > 0.0f) ? 1.0f / l : 0.0f;
            bf16* orow = out + (static_cast<size_t>(row_base + row) * nq + h0 + g) * T5_D;
#pragma unroll 1
            for (int c = 0; c < T5_D; c += 32) {
                unsigned r[32];
                t5_ld32(tmem + lane_addr + o_col(g) + c, r);
                t5_wait_ld();
                if (row < rows_here) {
#pragma unroll
                    for (int i = 0; i < 32; i += 8) {
                        uint4 w;
                        w.x = t5_pack(__uint_as_float(r[i]) * inv, __uint_as_float(r[i + 1]) * inv);
                        w.y = t5_pack(__uint_as_float(r[i + 2]) * inv, __uint_as_float(r[i + 3]) * inv);
                        w.z = t5_pack(__uint_as_float(r[i + 4]) * inv, __uint_as_float(r[i + 5]) * inv);
                        w.w = t5_pack(__uint_as_float(r[i + 6]) * inv, __uint_as_float(r[i + 7]) * inv);
                        *reinterpret_cast<uint4*>(orow + c + i) = w;
                    }
                }
            }
        }
    }
    t5_fence_before();
    __syncthreads();
    if (warp == 1) {
        t5_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(TMEM_COLS) : "memory");
    }
}

// ---- one pass with a running reference maximum, two heads in turns -------------------------------
// The same work in ONE pass over the keys, for the two query heads of a group that share a key/value
// tile (the kernel above stays for groups of odd size): 128 keys a tile, S = Q K^T of head 0 while
// the softmax threads of head 1 work and the other way round, so the tensor pipe has a product of
// one head to run while the other head's weights are being made.  Per head TMEM holds S (128
// columns of float32) and O (128 columns); P (bfloat16) lies over S, 64 columns from column 0 on, each over columns
// that its thread has read.
// The weights are P = exp2(S*scale*log2e - m) with a reference m per row that trails the running
// maximum: m moves up only when the maximum has passed it by more than 8 (a factor 256, far
// inside what bfloat16 and the float32 sums hold), and only then O and the row sum l are
// multiplied by exp2(m_old - m_new) (the running-maximum form of src/ops/attention.cu:204-249 with
// the correction made rare).  The result sum(P V) / sum(P) does not depend on which m was used.
// After a portion's first tile the weights of 64 keys are made at the reference that is there, beside these keys' maximum, and
// made again in the rare case that it has to move: neither waits for the other.
// Roles: warp 0 looks up pages and asks the copy engine for keys and values (rings of two tiles
// each); warp 1 issues every product; warps 2 and 3 have no work (tensor memory gives a warp the 32 lanes of its index mod 4); then
// four softmax warps per head, a thread a query row.
// What bounds it, read from the SM clock inside the kernel: a tile takes 3,900 clocks, of which the tensor pipe works 2,048
// and the exponentials of both heads (8 clocks a warp and value) 2,048.  A head's chain is 2,100 to 2,500 clocks from S to the
// last weight, as the other head's exponentials get in its way, and 1,300 from there to the next S: half of P V (the other half runs
// under the second half's weights), Q K^T, and the commit's way.  Against the form before (two threads a row that exchanged their
// maxima before the weights, one lane alone in the issuing loop), us: 967 + 1,933 tokens behind 700 and 613 118 -> 95, 2,500 tokens
// 98 -> 76, 8,192 tokens 605 -> 510, 300 + 600 tokens 31 -> 20; windowed with sinks, 2,500 tokens, 88 -> 73.  A step of that: rows behind a
// portion's last used to send the whole of its last tile, the longest, through the masked form (98 -> 81).  Two threads a row in this
// form, with a vote of two warps in the place of the exchange: 2.2 us a tile against 2.05; a share of the exponentials as
// polynomials on the multiply-add pipe: 15.0 clocks a value and warp against 12.0 (an exponential keeps its warp from issuing for its 8 clocks).
#define T5O_BN 128
#define T5O_HALF (T5O_BN * 64)                // elements of one 64-column half of a 128-key tile
#define T5O_TILE (2 * T5O_HALF)
#define T5O_STAGES 2
#define T5O_JUMP 8.0f
#define T5O_THREADS (128 + 2 * 128)            // producer warp, issuing warp, two without work, then 4 softmax warps per head

// BIAS: the scores carry more than the scale.  `head_bias` is float32 [nq][3] = (t, r1, r2) per query head and the
// weight of key j for the query at position i is exp(S * scale * t - r1 * ln(1 + r2 * (i - j))).  The bias depends on
// the head and on i - j only, and a tile of 128 rows by 128 keys meets 255 distances: the 128 softmax threads of a
// head work out two each (two logarithms a thread a tile instead of 128) into a table in shared memory for the NEXT tile,
// behind the barrier that they all pass once a tile in this mode.  Two tables take turns.
// EXT: a window that keeps the sequence's first `keep_first` keys (the tiles that hold them and lie wholly below the
// window's first tile are walked first; kept keys inside the window's tiles are a matter of the mask), one more term
// exp(sinks[head]) in the softmax's denominator, a sigmoid gate per head (column gate_off + head of a float32 row per
// token), a factor, and a result that is a column range of a wider buffer.  Measured, 32 heads over 8, window 1,024, four
// kept keys, learned sinks, 2,500 tokens: 216 us on mma.sync (attention_prefill.cu), 73 us here.  In this mode the reference
// is the running maximum itself, so that the largest weight so far is exactly one in bfloat16, as on mma.sync, and the
// weights are summed as rounded.  With a reference that trails and a sum of unrounded weights it takes 10 us less, and the error against
// 64 bits is 3, 13 and 20 % above that of mma.sync at spreads of the scores of 1, 2 and 4 (now 0.2 % below, level, 0.1 % below).
struct T5Ext {
    int keep_first;
    const float* sinks;
    const float* gate;
    long long gate_stride;
    int gate_off;
    float out_scale;
    long long out_stride;
    int out_off;
};
enum { T5_PLAIN, T5_BIAS, T5_EXT };
template <int MODE>
__global__ void __launch_bounds__(T5O_THREADS, 1) paged_prefill_attention_tcgen05_online_kernel(
    const __grid_constant__ CUtensorMap q_map, const __grid_constant__ CUtensorMap kv_map, bf16* __restrict__ out,
    const int32_t* __restrict__ tiles, const int32_t* __restrict__ entry_slot, const int32_t* __restrict__ entry_q_start,
    const int32_t* __restrict__ entry_q_len, const int32_t* __restrict__ entry_kv_len,
    const int32_t* __restrict__ block_table, int table_stride, int nq, int nkv, int page_size, int window,
    float scale_log2e, int num_pages, int32_t* __restrict__ status, const float* __restrict__ head_bias, const T5Ext ext) {
    pdl_begin();
    constexpr bool BIAS = MODE == T5_BIAS, EXT = MODE == T5_EXT;
    constexpr int STAGES = T5O_STAGES;
    constexpr unsigned TMEM_COLS = 512;                           // S0 S1 O0 O1, 128 columns each
    extern __shared__ unsigned char smem_dyn[];
    unsigned char* smem_al = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_dyn) + 1023) & ~uintptr_t(1023));
    bf16* q_s = reinterpret_cast<bf16*>(smem_al);                 // [2 heads][2 halves][128][64]
    bf16* k_s = q_s + 2 * 2 * T5_QHALF;                           // [STAGES][2][128][64]
    bf16* v_s = k_s + STAGES * T5O_TILE;                          // [STAGES][2][128][64]
    // keys and values have rings of their own: a key tile is free once both heads' S are made, a
    // value tile only after both heads' P V, half a tile's work later
    __shared__ __align__(8) unsigned long long q_full, k_full[STAGES], k_empty[STAGES], v_full[STAGES], v_empty[STAGES],
        s_full[2], p_full[2][2], pv_half[2], pv_done[2];
    __shared__ unsigned tmem_base_s;
    __shared__ int abort_flag;
    __shared__ float bias_tbl[BIAS ? 2 : 1][2][BIAS ? 256 : 1];   // [tile parity][head][i - j - (first row - first key of the tile) + 127]

    const int tile = blockIdx.y;
    const int h0 = blockIdx.x * 2;                                // first of this CTA's two query heads
    const int kvh = h0 / (nq / nkv);
    const int e = tiles[2 * tile], q0 = tiles[2 * tile + 1];
    if (e < 0) return;                                            // a padding entry of the tile list: no work
    const int q_len = entry_q_len[e], kv_len = entry_kv_len[e];
    const int past = kv_len - q_len;
    const int row_base = entry_q_start[e] + q0;
    const int rows_here = min(T5_BM, q_len - q0);
    const int32_t* table = block_table + static_cast<size_t>(entry_slot[e]) * table_stride;
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int pos_first = past + q0, pos_last = past + q0 + rows_here - 1;
    const int k_lo = first_visible(pos_first, window) / T5O_BN * T5O_BN;
    const int keep = EXT && window > 0 ? ext.keep_first : 0;
    const int head_tiles = EXT ? min((keep + T5O_BN - 1) / T5O_BN, k_lo / T5O_BN) : 0;
    const int n_tiles = head_tiles + (pos_last - k_lo) / T5O_BN + 1;
    auto tile_key = [&](int j) { return EXT && j < head_tiles ? j * T5O_BN : k_lo + (j - head_tiles) * T5O_BN; };

    if (tid == 0) {
        abort_flag = 0;
        t5_mbar_init(&q_full, 1);
        for (int s = 0; s < STAGES; ++s) {
            t5_mbar_init(&k_full[s], 1); t5_mbar_init(&k_empty[s], 1);
            t5_mbar_init(&v_full[s], 1); t5_mbar_init(&v_empty[s], 1);
        }
        for (int g = 0; g < 2; ++g) {
            t5_mbar_init(&s_full[g], 1);                 // the head's S of a tile is in TMEM
            for (int hf = 0; hf < 2; ++hf) t5_mbar_init(&p_full[g][hf], 4);      // every softmax warp of the head has put its rows of half of P over S
            t5_mbar_init(&pv_half[g], 1);                // the head's O holds P V of the tile's first 64 keys
            t5_mbar_init(&pv_done[g], 1);                // the head's O holds the tile's P V
        }
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(t5_smem(&tmem_base_s)), "r"(TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    t5_fence_before();
    __syncthreads();
    t5_fence_after();
    const unsigned tmem = __shfl_sync(0xffffffffu, tmem_base_s, 0);
    auto s_col = [](int g) { return static_cast<unsigned>(g * 128); };
    auto o_col = [](int g) { return static_cast<unsigned>(256 + g * 128); };

    if (warp == 0) {
        // ---- producer: lane b looks up the page of box b of a tile, one tile ahead, and asks the copy
        // engine for it ----
        // (One thread doing this box by box spent 140 clocks a copy, 4,500 a tile: longer than the
        // tile's products take.  A warp-wide copy instruction makes all boxes' requests at once.)
        if (lane == 0) {
            t5_expect_tx(&q_full, 2 * 2 * T5_QHALF * sizeof(bf16));
#pragma unroll
            for (int g = 0; g < 2; ++g) {
                t5_tma_2d(q_s + g * 2 * T5_QHALF, &q_map, (h0 + g) * T5_D, row_base, &q_full);
                t5_tma_2d(q_s + g * 2 * T5_QHALF + T5_QHALF, &q_map, (h0 + g) * T5_D + 64, row_base, &q_full);
            }
        }
        const int boxes = T5O_BN / page_size;                     // at most 16
        const int last_logical = pos_last / page_size;
        auto page_of = [&](int j) {                               // lane b: the page of box b of tile j (checked)
            if (j >= n_tiles || lane >= boxes) return 0;
            int logical = min(tile_key(j) / page_size + lane, last_logical);
            if (EXT) {                                            // pages that hold no key anybody sees may be gone: read a held one
                if (j < head_tiles) logical = min(logical, (keep - 1) / page_size);
                else if (logical * page_size >= keep) logical = max(logical, first_visible(pos_first, window) / page_size);
            }
            int page = logical < table_stride ? __ldg(table + logical) : -1;
            if (page < 0 || page >= num_pages) {
                if (atomicCAS(status, 0, 4) == 0) status[1] = row_base;
                page = 0;
            }
            return page;
        };
        int issued_k = 0, issued_v = 0;
        int next_page = page_of(0);
        bool ok = true;
        for (int j = 0; j < n_tiles; ++j) {
            const int st = j % STAGES;
            const int my_page = next_page;
            next_page = page_of(j + 1);
#pragma unroll 1
            for (int values = 0; values < 2; ++values) {
                unsigned long long* full = values ? &v_full[st] : &k_full[st];
                if (lane == 0) {
                    if (j >= STAGES && !t5_wait(values ? &v_empty[st] : &k_empty[st], ((j / STAGES) - 1) & 1, &abort_flag, status, row_base))
                        ok = false;
                    if (ok) t5_expect_tx(full, T5O_TILE * sizeof(bf16));
                }
                ok = __shfl_sync(0xffffffffu, ok, 0);
                if (!ok) break;
                bf16* dst = (values ? v_s : k_s) + st * T5O_TILE;
                if (lane < boxes) {                               // every lane asks for its own box: one instruction, `boxes` copies
                    const int row0 = ((my_page * 2 + values) * nkv + kvh) * page_size;
                    t5_tma_2d(dst + lane * page_size * 64, &kv_map, 0, row0, full);
                    t5_tma_2d(dst + T5O_HALF + lane * page_size * 64, &kv_map, 64, row0, full);
                }
                if (values) issued_v = j + 1; else issued_k = j + 1;
            }
            if (!ok) break;
        }
        if (lane == 0 && abort_flag) {                            // let what is in flight land before the CTA goes away
            for (int j = max(0, issued_k - STAGES); j < issued_k; ++j)
                for (int i = 0; i < T5_WAIT_LIMIT && !t5_try_wait(&k_full[j % STAGES], (j / STAGES) & 1); ++i) {}
            for (int j = max(0, issued_v - STAGES); j < issued_v; ++j)
                for (int i = 0; i < T5_WAIT_LIMIT && !t5_try_wait(&v_full[j % STAGES], (j / STAGES) & 1); ++i) {}
        }
    } else if (warp == 1) {
        // ---- MMA issuer: S0(j), O1 += P1 V(j-1), S1(j), O0 += P0 V(j), ... ----
        // All lanes walk the loop, one of them issues.  Descriptors are made of what all lanes hold alike; a tile further on in
        // shared memory is the same descriptor plus its byte offset / 16 in the address field.
        constexpr unsigned IDESC_QK = t5_idesc(T5_BM, T5O_BN, 0);
        constexpr unsigned IDESC_PV = t5_idesc(T5_BM, T5_D, 1);
        const unsigned lead = elect_one();
        const unsigned long long qd0 = t5_desc(q_s, 16, 1024), kd0 = t5_desc(k_s, 16, 1024);
        const unsigned long long vd0 = t5_desc(v_s, T5O_HALF * sizeof(bf16), 1024);
        constexpr unsigned long long STAGE_STEP = (T5O_TILE * sizeof(bf16)) >> 4, VSTEP = (16 * 64 * sizeof(bf16)) >> 4;   // 16 keys further, both 64-column halves
        auto qk = [&](int g, int st) {
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const unsigned long long qo = (((k >> 2) * T5_QHALF + (k & 3) * 16) * sizeof(bf16)) >> 4;
                const unsigned long long ko = (((k >> 2) * T5O_HALF + (k & 3) * 16) * sizeof(bf16)) >> 4;
                t5_mma_ss_lead(lead, tmem + s_col(g), qd0 + g * ((2 * T5_QHALF * sizeof(bf16)) >> 4) + qo, kd0 + st * STAGE_STEP + ko, IDESC_QK, k > 0);
            }
            t5_commit_lead(lead, &s_full[g]);
        };
        auto pv = [&](int g, int j, int st) -> bool {
#pragma unroll
            for (int hf = 0; hf < 2; ++hf) {
                if (!t5_wait_warp(&p_full[g][hf], j & 1, &abort_flag, status, row_base)) return false;
                t5_fence_after();
#pragma unroll
                for (int k = 4 * hf; k < 4 * hf + 4; ++k)
                    t5_mma_ts_lead(lead, tmem + o_col(g), tmem + s_col(g) + k * 8, vd0 + st * STAGE_STEP + k * VSTEP, IDESC_PV, (j > 0 || k > 0) ? 1u : 0u);
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
            qk(0, st);
            if (j > 0) {
                ok = pv(1, j - 1, 1 - st);
                if (!ok) break;
                t5_commit_lead(lead, &v_empty[1 - st]);                // the last reader of the values of tile j-1
            }
            qk(1, st);
            t5_commit_lead(lead, &k_empty[st]);                        // the last reader of the keys of tile j
            ok = t5_wait_warp(&v_full[st], (j >> 1) & 1, &abort_flag, status, row_base) && pv(0, j, st);
        }
        static_assert(T5O_STAGES == 2, "a tile's stage is its parity");
        if (ok && pv(1, n_tiles - 1, (n_tiles - 1) & 1)) t5_commit_lead(lead, &v_empty[(n_tiles - 1) & 1]);
    } else if (warp >= 4) {
        // ---- softmax: a thread owns one query row of one head = one TMEM lane, all 128 columns of a tile ----
        const int g = (warp - 4) >> 2;                            // warps 4..7: head h0, warps 8..11: head h0 + 1
        const int quarter = warp & 3;                             // the TMEM lanes this warp may touch
        const int row = quarter * 32 + lane;
        const unsigned lane_addr = static_cast<unsigned>(quarter * 32) << 16;
        const unsigned my_s = tmem + lane_addr + s_col(g);
        const unsigned my_o = tmem + lane_addr + o_col(g);
        // Rows behind the portion's last are other tokens' or zeros: they are worked like the rest (nothing of a row reaches another
        // one) and not stored.
        const int pos = past + q0 + row;
        const int lo = first_visible(pos, window), lo_last = first_visible(pos_last, window);
        float m = -CUDART_INF_F, l = 0.0f;                        // m: the reference maximum, in units of log2
        bool ok = true;
        // with BIAS the scores are turned into their final form (units of log2) as they arrive, and `eff` is 1
        float sc = scale_log2e, r1 = 0.0f, r2 = 0.0f;
        if constexpr (BIAS) {
            const float* hb = head_bias + static_cast<size_t>(h0 + g) * 3;
            sc *= hb[0]; r1 = hb[1]; r2 = hb[2];
        }
        const float eff = BIAS ? 1.0f : scale_log2e;
        auto fill_table = [&](int jt, int which) {                // the distances of tile jt: first row - first key - 127 + (0 .. 255)
#pragma unroll
            for (int i = row; i < 256; i += 128) {
                const int dist = pos_first - (k_lo + jt * T5O_BN) - 127 + i;
                bias_tbl[which][g][i] = dist > 0 ? r1 * __log2f(fmaf(r2, static_cast<float>(dist), 1.0f)) : 0.0f;
            }
        };
        if constexpr (BIAS) fill_table(0, 0);
        for (int j = 0; j < n_tiles; ++j) {
            const int kt = tile_key(j);
            if constexpr (BIAS) {
                asm volatile("bar.sync %0, 128;\n" ::"r"(1 + g) : "memory");      // the table of this tile is there
                if (j + 1 < n_tiles) fill_table(j + 1, (j + 1) & 1);
            }
            const bool full_tile = (kt + T5O_BN - 1 <= pos_first) && (kt >= lo_last || (EXT && kt + T5O_BN - 1 < keep));
            // columns 32 c .. 32 c + 31 of the scores: S -> S * scale * t - bias(i - j), and what the row does not see to -inf
            auto settle = [&](unsigned (&r)[32], int c) {
                if constexpr (BIAS) {
                    const float* tb = &bias_tbl[j & 1][g][row - c * 32 + 127];
#pragma unroll
                    for (int i = 0; i < 32; ++i) r[i] = __float_as_uint(fmaf(__uint_as_float(r[i]), sc, -tb[-i]));
                }
                if (!full_tile) {
                    auto first = [&](int n) { return n <= 0 ? 0u : n >= 32 ? ~0u : (1u << n) - 1u; };
                    const int k0 = kt + 32 * c;
                    const unsigned seen = first(pos + 1 - k0) & (~first(lo - k0) | (EXT ? first(keep - k0) : 0u));
#pragma unroll
                    for (int i = 0; i < 32; ++i) r[i] = seen & (1u << i) ? r[i] : 0xff800000u;
                }
            };
            auto max_of = [](const unsigned (&r)[32], float mx) {
                float a = __uint_as_float(r[0]), b = __uint_as_float(r[1]);
#pragma unroll
                for (int i = 2; i < 32; i += 2) { a = fmaxf(a, __uint_as_float(r[i])); b = fmaxf(b, __uint_as_float(r[i + 1])); }
                return fmaxf(mx, fmaxf(a, b));
            };
            // the weights of 32 columns, rounded to bfloat16, and their sum (EXT: of the rounded ones)
            auto weights = [&](const unsigned (&r)[32], unsigned (&pk)[16], float ref, float sum) {
                const unsigned long long e2 = t5_two(eff, eff), m2 = t5_two(-ref, -ref);
                float s0 = 0.0f, s1 = 0.0f;
#pragma unroll
                for (int i = 0; i < 32; i += 2) {
                    float x0, x1;
                    t5_untwo(t5_fma2(t5_two(__uint_as_float(r[i]), __uint_as_float(r[i + 1])), e2, m2), x0, x1);
                    const float p0 = t5_ex2(x0), p1 = t5_ex2(x1);
                    pk[i >> 1] = t5_pack(p0, p1);
                    if (EXT) {
                        s0 += __uint_as_float(pk[i >> 1] << 16);
                        s1 += __uint_as_float(pk[i >> 1] & 0xffff0000u);
                    } else {
                        s0 += p0;
                        s1 += p1;
                    }
                }
                return sum + (s0 + s1);
            };
            // After a wait has run out (ok false, for whole warps) a thread still passes every barrier above and touches nothing else.
            if (ok) ok = __all_sync(0xffffffffu, t5_wait(&s_full[g], j & 1, &abort_flag, status, row_base));
            if (!ok) continue;
            t5_fence_after();
            unsigned r[2][32];
            // the row's O and l on to another reference, once the products that are under way have joined O
            auto move_to = [&](float mx, bool jump, unsigned long long* done, int parity) {
                if (__any_sync(0xffffffffu, jump)) {
                    ok = __all_sync(0xffffffffu, t5_wait(done, parity, &abort_flag, status, row_base));
                    if (!ok) return;
                    t5_fence_after();
                    const float alpha = jump ? t5_ex2(m - mx) : 1.0f;
                    l *= alpha;
                    t5_ld32(my_o, r[0]);
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        t5_wait_ld();
                        if (c < 3) t5_ld32(my_o + 32 * (c + 1), r[(c + 1) & 1]);
#pragma unroll
                        for (int i = 0; i < 32; ++i) r[c & 1][i] = __float_as_uint(__uint_as_float(r[c & 1][i]) * alpha);
                        t5_st32(my_o + 32 * c, r[c & 1]);
                    }
                }
            };
            const bool first_max = EXT || j == 0;                     // the tile's maximum before its weights
            if (first_max) {                                          // (EXT: the reference is the running maximum itself)
                float mx = -CUDART_INF_F;
                t5_ld32(my_s, r[0]);
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    t5_wait_ld();
                    if (c < 3) t5_ld32(my_s + 32 * (c + 1), r[(c + 1) & 1]);
                    settle(r[c & 1], c);
                    mx = max_of(r[c & 1], mx);
                }
                mx *= eff;                                            // scale > 0; -inf stays -inf
                move_to(mx, m != -CUDART_INF_F && mx > m, &pv_done[g], (j - 1) & 1);
                if (!ok) continue;
                m = fmaxf(m, mx);
            }
            // The tile in two halves of 64 keys: the products over the first run while the weights of the second are made.
#pragma unroll 1
            for (int hf = 0; hf < 2; ++hf) {
                const unsigned s_at = my_s + 64 * hf, p_at = my_s + 32 * hf;
                unsigned pk[2][16];
                float ref = m == -CUDART_INF_F ? 0.0f : m;
                float sum = 0.0f, mx = -CUDART_INF_F;
                // The weights at the reference that the keys before have left, beside these keys' maximum: the reference hardly ever
                // moves, and then neither has waited for the other.
                t5_ld32(s_at, r[0]);
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    t5_wait_ld();
                    if (c < 1) t5_ld32(s_at + 32, r[1]);
                    settle(r[c], 2 * hf + c);
                    if (!first_max) mx = max_of(r[c], mx);
                    sum = weights(r[c], pk[c], ref, sum);
                }
                if (!first_max) {
                    mx *= eff;                                        // scale > 0; -inf stays -inf
                    // move the reference up only when the maximum has run away from it
                    const bool adopt = (m == -CUDART_INF_F) && (mx > m);      // nothing accumulated under the old reference
                    const bool jump = (m != -CUDART_INF_F) && (mx > m + T5O_JUMP);
                    if (__any_sync(0xffffffffu, adopt || jump)) {
                        move_to(mx, jump, hf ? &pv_half[g] : &pv_done[g], (hf ? j : j - 1) & 1);
                        if (!ok) break;
                        if (adopt || jump) m = mx;
                        ref = m == -CUDART_INF_F ? 0.0f : m;
                        sum = 0.0f;
                        t5_ld32(s_at, r[0]);
#pragma unroll
                        for (int c = 0; c < 2; ++c) {
                            t5_wait_ld();
                            if (c < 1) t5_ld32(s_at + 32, r[1]);
                            settle(r[c], 2 * hf + c);
                            sum = weights(r[c], pk[c], ref, sum);
                        }
                    }
                }
                l += sum;
                t5_st16(p_at, pk[0]);                                 // over columns of S that have been read
                t5_st16(p_at + 16, pk[1]);
                t5_wait_st();
                t5_fence_before();
                if constexpr (EXT) {
                    // Keys of the tile that no row of the block sees (behind its last one, below the window, behind the kept ones) have
                    // weights of zero, but what lies there may be anything (a request that had the page before, a held page's copy), and
                    // zero times a value that is not finite is NaN: their values are set to zero before the products, a row of 256 bytes a
                    // thread.
                    const int key = kt + row, lo_first = first_visible(pos_first, window);
                    if (hf == 0 && g == 0 && (kt + T5O_BN - 1 > pos_last || (kt < lo_first && kt + T5O_BN > keep))) {
                        ok = __all_sync(0xffffffffu, t5_wait(&v_full[j % STAGES], (j / STAGES) & 1, &abort_flag, status, row_base));
                        if (!ok) break;
                        if (key > pos_last || (key < lo_first && key >= keep)) {
                            uint4* v = reinterpret_cast<uint4*>(v_s + (j % STAGES) * T5O_TILE + row * 64);
#pragma unroll
                            for (int c = 0; c < 16; ++c) v[(c >> 3) * (T5O_HALF / 8) + ((c + lane) & 7)] = make_uint4(0u, 0u, 0u, 0u);      // a quarter-warp: all banks
                        }
                        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
                    }
                }
                __syncwarp();
                if (lane == 0) t5_arrive(&p_full[g][hf]);
            }
        }
        if (ok && __all_sync(0xffffffffu, t5_wait(&pv_done[g], (n_tiles - 1) & 1, &abort_flag, status, row_base))) {
            t5_fence_after();
            if (EXT && ext.sinks) l += t5_ex2(fmaf(ext.sinks[h0 + g], 1.4426950408889634f, -m));   // a term without a value
            float inv = (l > 0.0f) ? 1.0f / l : 0.0f;
            bf16* orow = out + (static_cast<size_t>(row_base + row) * nq + h0 + g) * T5_D;
            if constexpr (EXT) {
                orow = out + static_cast<size_t>(row_base + row) * ext.out_stride + ext.out_off + (h0 + g) * T5_D;
                inv *= ext.out_scale;
                if (ext.gate && row < rows_here)
                    inv /= 1.0f + expf(-ext.gate[static_cast<size_t>(row_base + row) * ext.gate_stride + ext.gate_off + h0 + g]);
            }
            unsigned r[2][32];
            t5_ld32(my_o, r[0]);
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                t5_wait_ld();
                if (c < 3) t5_ld32(my_o + 32 * (c + 1), r[(c + 1) & 1]);
                if (row < rows_here) {
                    const unsigned (&v)[32] = r[c & 1];
#pragma unroll
                    for (int i = 0; i < 32; i += 8) {
                        uint4 w;
                        w.x = t5_pack(__uint_as_float(v[i]) * inv, __uint_as_float(v[i + 1]) * inv);
                        w.y = t5_pack(__uint_as_float(v[i + 2]) * inv, __uint_as_float(v[i + 3]) * inv);
                        w.z = t5_pack(__uint_as_float(v[i + 4]) * inv, __uint_as_float(v[i + 5]) * inv);
                        w.w = t5_pack(__uint_as_float(v[i + 6]) * inv, __uint_as_float(v[i + 7]) * inv);
                        *reinterpret_cast<uint4*>(orow + c * 32 + i) = w;
                    }
                }
            }
        }
    }
    t5_fence_before();
    __syncthreads();
    if (warp == 1) {
        t5_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(TMEM_COLS) : "memory");
    }
}

// ---- host side ---------------------------------------------------------------------------------------
extern "C" int llm_paged_prefill_tcgen05_supported(int d, int page_size) {
    return d == T5_D && (page_size == 8 || page_size == 16 || page_size == 32 || page_size == 64);
}
extern "C" int llm_paged_prefill_tcgen05_tile_rows() { return T5_BM; }

// The scores' additions (a temperature per head, a logarithmic distance bias) are built into the kernel that serves
// two heads of a group at once.
extern "C" int llm_paged_prefill_tcgen05_biased_supported(int d, int page_size, int group) {
    return llm_paged_prefill_tcgen05_supported(d, page_size) && group > 0 && group % 2 == 0;
}

// q, out: bfloat16 [num_tokens, nq*128]; cache: bfloat16 [pages, 2, nkv, page_size, 128];
// tiles: int32 [n_tiles][2] = (entry, first query row of the tile inside the entry), 128 rows each.
// head_bias: null, or float32 [nq][3] = (temperature, r1, r2) per query head (even groups only).
static int t5_launch(
    const void* q, void* out, const void* cache, int num_tokens, const int32_t* tiles, int n_tiles,
    const int32_t* entry_slot, const int32_t* entry_q_start, const int32_t* entry_q_len, const int32_t* entry_kv_len,
    const int32_t* block_table, int table_stride, int nq, int nkv, int d, int page_size, int window, float scale,
    int num_pages, int32_t* status, const float* head_bias, const T5Ext* ext, uintptr_t stream) {
    if (n_tiles <= 0) return LLM_OK;
    if (nq <= 0 || nkv <= 0 || nq % nkv != 0 || !llm_paged_prefill_tcgen05_supported(d, page_size) || nq > 65535 ||
        n_tiles > 65535)
        return LLM_REFUSED_SIZE;
    if (!aligned16(q) || !aligned16(out) || !aligned16(cache)) return LLM_REFUSED_ALIGN;
    CUtensorMap q_map, kv_map;
    if (!t5_encode_2d(&q_map, q, static_cast<long long>(nq) * d, num_tokens, 64, T5_BM)) return LLM_REFUSED_SIZE;
    if (!t5_encode_2d(&kv_map, cache, d, static_cast<long long>(num_pages) * 2 * nkv * page_size, 64, page_size))
        return LLM_REFUSED_SIZE;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    const float sl2 = scale * 1.4426950408889634f;
    const int group = nq / nkv;
    if ((head_bias || ext) && (group % 2 != 0 || (head_bias && ext))) return LLM_REFUSED_SIZE;
#define T5_GO(HEADS, STAGES)                                                                                         \
    {                                                                                                                \
        const size_t smem = static_cast<size_t>(HEADS * 2 * T5_QHALF + 2 * STAGES * T5_TILE) * sizeof(bf16) + 1024;  \
        auto kern = paged_prefill_attention_tcgen05_kernel<HEADS, STAGES>;                                           \
        const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,                \
                                                   static_cast<int>(smem));                                          \
        if (e != cudaSuccess) return static_cast<int>(e);                                                            \
        launch_pdl(kern, dim3(nq / HEADS, n_tiles), dim3(64 + 128 * HEADS), smem, s, q_map, kv_map,                  \
                   static_cast<bf16*>(out), tiles, entry_slot, entry_q_start, entry_q_len, entry_kv_len,             \
                   block_table, table_stride, nq, nkv, page_size, window, sl2, num_pages, status);                   \
    }
    if (group % 2 == 0) {                                           // two heads of a group share a CTA: the one-pass kernel
        const size_t smem = static_cast<size_t>(2 * 2 * T5_QHALF + 2 * T5O_STAGES * T5O_TILE) * sizeof(bf16) + 1024;
        auto kern = head_bias ? paged_prefill_attention_tcgen05_online_kernel<T5_BIAS>
                    : ext     ? paged_prefill_attention_tcgen05_online_kernel<T5_EXT>
                              : paged_prefill_attention_tcgen05_online_kernel<T5_PLAIN>;
        const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
        if (e != cudaSuccess) return static_cast<int>(e);
        launch_pdl(kern, dim3(nq / 2, n_tiles), dim3(T5O_THREADS), smem, s, q_map, kv_map, static_cast<bf16*>(out), tiles,
                   entry_slot, entry_q_start, entry_q_len, entry_kv_len, block_table, table_stride, nq, nkv, page_size,
                   window, sl2, num_pages, status, head_bias, ext ? *ext : T5Ext{});
        return launch_status();
    }
    T5_GO(1, 4)                                                     // odd groups: the two-pass kernel, one head per CTA
#undef T5_GO
    return launch_status();
}

extern "C" int llm_paged_attention_prefill_tcgen05(
    const void* q, void* out, const void* cache, int num_tokens, const int32_t* tiles, int n_tiles,
    const int32_t* entry_slot, const int32_t* entry_q_start, const int32_t* entry_q_len, const int32_t* entry_kv_len,
    const int32_t* block_table, int table_stride, int nq, int nkv, int d, int page_size, int window, float scale,
    int num_pages, int32_t* status, uintptr_t stream) {
    return t5_launch(q, out, cache, num_tokens, tiles, n_tiles, entry_slot, entry_q_start, entry_q_len, entry_kv_len,
                     block_table, table_stride, nq, nkv, d, page_size, window, scale, num_pages, status, nullptr, nullptr, stream);
}

extern "C" int llm_paged_attention_prefill_tcgen05_biased(
    const void* q, void* out, const void* cache, int num_tokens, const int32_t* tiles, int n_tiles,
    const int32_t* entry_slot, const int32_t* entry_q_start, const int32_t* entry_q_len, const int32_t* entry_kv_len,
    const int32_t* block_table, int table_stride, int nq, int nkv, int d, int page_size, int window, float scale,
    int num_pages, int32_t* status, const float* head_bias, uintptr_t stream) {
    if (!head_bias) return LLM_REFUSED_SIZE;
    return t5_launch(q, out, cache, num_tokens, tiles, n_tiles, entry_slot, entry_q_start, entry_q_len, entry_kv_len,
                     block_table, table_stride, nq, nkv, d, page_size, window, scale, num_pages, status, head_bias, nullptr, stream);
}

// out: bfloat16, row t and head h at t * out_stride + out_off + h * 128.  keep_first: with a window, the first so many keys stay
// visible; sinks: null, or float32 [nq]; gate: null, or float32 rows of gate_stride with one value a head from gate_off on.
extern "C" int llm_paged_attention_prefill_tcgen05_ext(
    const void* q, void* out, const void* cache, int num_tokens, const int32_t* tiles, int n_tiles,
    const int32_t* entry_slot, const int32_t* entry_q_start, const int32_t* entry_q_len, const int32_t* entry_kv_len,
    const int32_t* block_table, int table_stride, int nq, int nkv, int d, int page_size, int window, float scale,
    int num_pages, int32_t* status, int keep_first, const float* sinks, const float* gate, long long gate_stride, int gate_off,
    float out_scale, long long out_stride, int out_off, uintptr_t stream) {
    if (keep_first < 0 || !(scale > 0.0f)) return LLM_REFUSED_SIZE;
    if (out_stride % 8 || out_off % 8) return LLM_REFUSED_ALIGN;
    const T5Ext ext = {keep_first, sinks, gate, gate_stride, gate_off, out_scale, out_stride, out_off};
    return t5_launch(q, out, cache, num_tokens, tiles, n_tiles, entry_slot, entry_q_start, entry_q_len, entry_kv_len,
                     block_table, table_stride, nq, nkv, d, page_size, window, scale, num_pages, status, nullptr, &ext, stream);
}
