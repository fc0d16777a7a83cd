// y[M, N] = x[M, K] . W[N, K]^T for float32 operands and more rows than a decode step, on the 5th-generation tensor cores.
//
// A float32 value is the sum of three bfloat16 values, h + m + l: h and m are what is left, rounded to nearest, so every
// remainder is exact and signed, |m| <= 2^-8 and |l| <= 2^-17 of the value, and l takes the rest exactly (down to bfloat16's
// smallest numbers: values below 2^-110 lose their last bits).  A product is then hh + (hm + mh) + (mm + hl + lh) plus ml + lm
// + ll, which are left out: at most 2^-24 of the product, what rounding it once may cost, and of either sign (pieces that are
// cut instead of rounded all have the value's sign, and what they leave out reaches 2^-21, always towards zero).  Six bfloat16
// products with float32 accumulation take the place of one float32 product, at 6 / 31 of the tensor cores' time against the
// multiply-add units' (4,096 against 128 products a clock and SM).
//
// What makes the sums as good as float32's: the tensor cores cut, rather than round, what they add to an accumulator, and
// 256 steps in a row along K = 4096 would show that.  So an accumulator lives for 64 k-values only, smallest terms first,
// and is then added, rounded, to sums kept in registers by the warps that drain it.  Error against 64 bits (relative, 2-norm,
// K = 4096, values of either sign and of one): 1.1e-7 and 1.0e-7; the library's float32 product 4.3e-7 to 1.2e-6 and 1.5e-7 to
// 9.9e-7.
// A result that is not finite is computed again with plain multiply-adds (a split infinity times zero is NaN, and a value
// above bfloat16's largest rounds to infinity), so infinities and NaN come out as a float32 product has them.
//
// A CTA makes 128 weight rows x NT tokens (the MMA's M side is the weights, so that 17 tokens cost a tile of 32).  Roles: warp
// 0 feeds the copy engine: 128 x 64 weights as float32, and NT x 64 of the three planes of x, which a small kernel has
// split; warps 2 to 9 split the weights in shared memory, half a row a thread (11 instructions for two values; storing the split
// weights instead would double their memory and their bytes); warp 1 issues 6 x 4 products a block of 64;
// warps 10 to 17 drain.  Planes are double-buffered (96 KB of weights' planes, 96 KB of x at NT 128).
// The weights' planes go to tensor memory, from where the tensor cores take their left operand: kept in shared memory, their
// stores and the operand reads of 24 products a block (8 KB each) filled the shared-memory path (500 tokens of 4096 x 12288:
// 323 us, 291 in tensor memory).  The issuing warp walks the blocks with all its lanes: in a branch for one lane each of the three
// waits in front of a block kept the tensor pipe idle for 250 clocks of the 2,500 to 2,900 that a block took (its 24 products are
// 1,536); the table has both.
// The loop that makes sums again which are not finite stays rolled: unrolled into each of a drain thread's sums it cost
// finite ones up to 20 % (500 tokens of 6144 x 4096: 209 us, now 167).
// Tiles that fill the SMs badly are cut along K (`splits`), the parts added in order by a second kernel.
//
// Measured (us; products issued in a branch for one lane, in turns on one GPU; the library's float32 product in brackets), everything cold:
//   N x K              17 rows            64 rows            128 rows           500 rows           2,048 rows
//   6144 x 4096        36; 46 (106)       40; 48 (129)       46; 56 (170)       148; 180 (542)     513; 597 (1,773)
//   4096 x 4096        30; 38 (105)       32; 38 (106)       40; 46 (126)       95; 112 (311)      347; 409 (1,132)
//   24576 x 4096       112; 148 (199)     123; 155 (283)     150; 182 (551)     509; 591 (1,779)   1,850; 2,100 (6,686)
//   4096 x 12288       63; 80 (250)       69; 83 (321)       81; 97 (373)       251; 296 (925)     985; 1,100 (3,353)
//   2048 x 2048        22; 28 (54)        24; 28 (53)        30; 34 (52)        44; 51 (87)        118; 136 (308)
// (4096 x 12288 from 500 rows on depends on the clocks: behind a second of such products 292 to 304 and 1,050, and 337 and 1,210 before.)
// Matrices of fewer than 2^21 values stay with the library: of 1024 x 1024, 17 rows take 23 us against 18 (and 64 to 2,048 rows 23
// to 34 against 29 to 86: for many rows the line could lie lower).
#include "tcgen05_attention.cuh"
#include <math_constants.h>

#define LT_ROWS 128                              // weight rows of a tile
#define LT_K 64                                  // k-values of a block: a 128-byte row of bfloat16
#define LT_SPLITTERS 256                          // threads that split the weights
#define LT_THREADS (18 * 32)
#define LT_BOX (LT_ROWS * 32 * 4)                // bytes of a box of float32 weights: 32 k-values, half a block
#define LT_STATUS 9

__device__ __forceinline__ bool lt_wait(unsigned long long* bar, unsigned parity, volatile int* abort_flag, int32_t* status) {
    for (int i = 0; i < T5_WAIT_LIMIT; ++i) {
        if (t5_try_wait(bar, parity)) return true;
        if (*abort_flag) return false;
    }
    *abort_flag = 1;
    if (atomicCAS(status, 0, LT_STATUS) == 0) status[1] = blockIdx.y;
    return false;
}

// The same for a whole warp, which goes on or stops together (tensor-memory accesses are a warp's).
__device__ __forceinline__ bool lt_wait_warp(unsigned long long* bar, unsigned parity, volatile int* abort_flag, int32_t* status) {
    return __all_sync(0xffffffffu, lt_wait(bar, parity, abort_flag, status));
}

// Two floats as a pair of bfloat16 (a in the lower half), rounded to nearest; a and b become what is left of them.
__device__ __forceinline__ unsigned lt_piece(float& a, float& b) {
    unsigned r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;\n" : "=r"(r) : "f"(b), "f"(a));
    a -= __uint_as_float(r << 16);
    b -= __uint_as_float(r & 0xffff0000u);
    return r;
}
// Eight floats as three planes of eight bfloat16.
__device__ __forceinline__ void lt_split8(const float4 a, const float4 b, unsigned* h, unsigned* m, unsigned* l) {
    float v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        h[i] = lt_piece(v[2 * i], v[2 * i + 1]);
        m[i] = lt_piece(v[2 * i], v[2 * i + 1]);
        l[i] = lt_piece(v[2 * i], v[2 * i + 1]);
    }
}

__device__ __forceinline__ void lt_st8(unsigned taddr, const unsigned (&r)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};\n" ::
                     "r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]) : "memory");
}
__global__ void linear_f32_split_kernel(const float* __restrict__ x, uint4* __restrict__ planes, long long pieces) {
    pdl_begin();
    const long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= pieces) return;
    const float4* p = reinterpret_cast<const float4*>(x) + 2 * i;
    unsigned h[4], m[4], l[4];
    lt_split8(p[0], p[1], h, m, l);
    planes[i] = make_uint4(h[0], h[1], h[2], h[3]);
    planes[pieces + i] = make_uint4(m[0], m[1], m[2], m[3]);
    planes[2 * pieces + i] = make_uint4(l[0], l[1], l[2], l[3]);
}

// grid (token tiles, row tiles, splits of K): tiles that share weights are neighbours.  NT: tokens of a tile (32, 64 or 128);
// WB: boxes of float32 weights in flight; XS: blocks of x;
// PS: blocks of the weights' planes (2 or 4; as many as fit beside the accumulators).  y: [M, N], or [splits, M, N] parts.
template <int NT, int WB, int XS, int PS>
__global__ void __launch_bounds__(LT_THREADS, 1) linear_f32_tcgen05_kernel(
    const __grid_constant__ CUtensorMap w_map, const __grid_constant__ CUtensorMap x_map, const float* __restrict__ x,
    const float* __restrict__ w, float* __restrict__ y, int M, int N, int K, int blocks_per_split, int32_t* __restrict__ status) {
    pdl_invite();
    constexpr int X_PLANE = NT * LT_K, DRAIN = NT >= 64 ? 256 : 128, COLS = NT >= 64 ? NT / 2 : NT;
    // tensor memory: two accumulators of NT columns, then PS stages of three planes of 32 columns (64 k-values as pairs)
    constexpr unsigned TMEM_COLS = 512, PLANE_COL = 2 * NT;
    static_assert(2 * NT + PS * 96 <= 512, "tensor memory");
    extern __shared__ unsigned char smem_dyn[];
    unsigned char* smem_al = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_dyn) + 1023) & ~uintptr_t(1023));
    unsigned char* w_s = smem_al;                                 // [WB][128 rows][32 floats], 128-byte swizzle
    bf16* x_s = reinterpret_cast<bf16*>(w_s + WB * LT_BOX);       // [XS][3 planes][NT][64]
    __shared__ __align__(8) unsigned long long w_full[WB], w_empty[WB], p_full[PS], p_empty[PS], x_full[XS], x_empty[XS],
        acc_full[2], acc_empty[2];
    __shared__ unsigned tmem_base_s;
    __shared__ int abort_flag;

    const int m0 = blockIdx.x * NT, n0 = blockIdx.y * LT_ROWS;
    const int kb0 = blockIdx.z * blocks_per_split, kb_all = (K + LT_K - 1) / LT_K;
    const int kbs = min(blocks_per_split, kb_all - kb0);          // at least one: the host sees to that
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    if (tid == 0) {
        abort_flag = 0;
        for (int s = 0; s < WB; ++s) { t5_mbar_init(&w_full[s], 1); t5_mbar_init(&w_empty[s], LT_SPLITTERS); }
        for (int s = 0; s < XS; ++s) { t5_mbar_init(&x_full[s], 1); t5_mbar_init(&x_empty[s], 1); }
        for (int s = 0; s < PS; ++s) {
            t5_mbar_init(&p_full[s], LT_SPLITTERS);               // every splitting thread has written its part of a row
            t5_mbar_init(&p_empty[s], 1);                         // the products that read these planes have finished
        }
        for (int s = 0; s < 2; ++s) { t5_mbar_init(&acc_full[s], 1); t5_mbar_init(&acc_empty[s], DRAIN); }
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

    if (warp == 0) {
        if (lane == 0) {
            int nw = 0, nx = 0;
            bool ok = true;
            const int boxes = 2 * kbs;
            auto fetch_w = [&]() {                                // the next box
                const int st = nw % WB;
                if (nw >= WB && !lt_wait(&w_empty[st], ((nw / WB) - 1) & 1, &abort_flag, status)) return false;
                t5_expect_tx(&w_full[st], LT_BOX);
                t5_tma_2d(w_s + st * LT_BOX, &w_map, kb0 * LT_K + nw * 32, n0, &w_full[st]);
                ++nw;
                return true;
            };
            pdl_wait();                                           // before the weights too: the kernel in front may have made them
            while (ok && nw < min(WB, boxes)) ok = fetch_w();
            auto fetch_x = [&]() {                                // the next block
                const int st = nx % XS;
                if (nx >= XS && !lt_wait(&x_empty[st], ((nx / XS) - 1) & 1, &abort_flag, status)) return false;
                t5_expect_tx(&x_full[st], 3 * X_PLANE * sizeof(bf16));
#pragma unroll
                for (int p = 0; p < 3; ++p)
                    t5_tma_2d(x_s + (st * 3 + p) * X_PLANE, &x_map, (kb0 + nx) * LT_K, p * M + m0, &x_full[st]);
                ++nx;
                return true;
            };
            // x runs a block ahead of the weights: its stage is free when the one of the planes being written is
            if (ok) ok = fetch_x();
            for (int kb = 0; ok && kb < kbs; ++kb) {
                if (nx < kbs) ok = fetch_x();
                while (ok && nw < min(boxes, 2 * kb + 2 + WB)) ok = fetch_w();
            }
            if (!ok || abort_flag) {                              // let what is in flight land before the CTA goes away
                for (int n = max(0, nw - WB); n < nw; ++n)
                    for (int i = 0; i < T5_WAIT_LIMIT && !t5_try_wait(&w_full[n % WB], (n / WB) & 1); ++i) {}
                for (int kb = max(0, nx - XS); kb < nx; ++kb)
                    for (int i = 0; i < T5_WAIT_LIMIT && !t5_try_wait(&x_full[kb % XS], (kb / XS) & 1); ++i) {}
            }
        }
    } else if (warp == 1) {
        pdl_wait();                                               // before any bounded wait: the kernel in front may take its time
        constexpr unsigned IDESC = t5_idesc(LT_ROWS, NT, 0);
        const unsigned lead = elect_one();                         // all lanes walk the blocks, one issues
        const unsigned long long xd = t5_desc(x_s, 16, 1024);
        constexpr unsigned long long X_STEP = X_PLANE * sizeof(bf16) >> 4;
        // the smallest terms first: l h, h l, m m, m h, h m, h h
        constexpr int WP[6] = {2, 0, 1, 1, 0, 0}, XP[6] = {0, 2, 1, 0, 1, 0};
#pragma unroll 1
        for (int kb = 0; kb < kbs; ++kb) {
            const int st = kb & 1, xs = kb % XS, ps = kb % PS;
            if (kb >= 2 && !lt_wait_warp(&acc_empty[st], ((kb >> 1) - 1) & 1, &abort_flag, status)) break;
            if (!lt_wait_warp(&x_full[xs], (kb / XS) & 1, &abort_flag, status)) break;
            if (!lt_wait_warp(&p_full[ps], (kb / PS) & 1, &abort_flag, status)) break;
            t5_fence_after();
            const unsigned long long xb = xd + xs * 3 * X_STEP;
            const unsigned pl = tmem + PLANE_COL + ps * 96;
#pragma unroll
            for (int t = 0; t < 6; ++t)
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    t5_mma_ts_lead(lead, tmem + st * NT, pl + WP[t] * 32 + k * 8, xb + XP[t] * X_STEP + 2 * k, IDESC, t > 0 || k > 0);
            t5_commit_lead(lead, &p_empty[ps]);
            t5_commit_lead(lead, &x_empty[xs]);
            t5_commit_lead(lead, &acc_full[st]);
        }
    } else if (warp < 10) {
        // ---- split the weights: two threads a row, each 16 k-values of every box ----
        pdl_wait();
        const int quarter = warp & 3, part = (warp - 2) >> 2, r = quarter * 32 + lane, sw = r & 7;
        const unsigned planes = tmem + (static_cast<unsigned>(quarter * 32) << 16) + PLANE_COL + 8 * part;
        bool ok = true;
        for (int kb = 0; ok && kb < kbs; ++kb) {
            const int st = kb % PS;
            if (kb >= PS && !lt_wait_warp(&p_empty[st], ((kb / PS) - 1) & 1, &abort_flag, status)) break;
            t5_fence_after();
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const int box = 2 * kb + half, ws = box % WB;
                if (!lt_wait_warp(&w_full[ws], (box / WB) & 1, &abort_flag, status)) { ok = false; break; }
                const unsigned char* src = w_s + ws * LT_BOX + r * 128;
                float4 a[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) a[i] = *reinterpret_cast<const float4*>(src + ((4 * part + i) ^ sw) * 16);
                unsigned h[8], m[8], l[8];
                lt_split8(a[0], a[1], h, m, l);
                lt_split8(a[2], a[3], h + 4, m + 4, l + 4);
                lt_st8(planes + st * 96 + 16 * half, h);
                lt_st8(planes + st * 96 + 32 + 16 * half, m);
                lt_st8(planes + st * 96 + 64 + 16 * half, l);
                t5_arrive(&w_empty[ws]);
            }
            if (!ok) break;
            t5_wait_st();
            t5_fence_before();
            t5_arrive(&p_full[st]);
        }
    } else if (NT >= 64 || warp < 14) {
        // ---- drain: a thread owns weight row n0 + its TMEM lane, COLS tokens ----
        pdl_wait();
        const int quarter = warp & 3, part = (warp - 10) >> 2;
        const unsigned addr = tmem + (static_cast<unsigned>(quarter * 32) << 16) + part * COLS;
        float acc[COLS];
#pragma unroll
        for (int i = 0; i < COLS; ++i) acc[i] = 0.0f;
        bool ok = true;
        for (int kb = 0; kb < kbs; ++kb) {
            const int st = kb & 1;
            if (!lt_wait_warp(&acc_full[st], (kb >> 1) & 1, &abort_flag, status)) { ok = false; break; }
            t5_fence_after();
#pragma unroll
            for (int c = 0; c < COLS; c += 16) {
                unsigned r[16];
                t5_ld16(addr + st * NT + c, r);
                t5_wait_ld();
#pragma unroll
                for (int i = 0; i < 16; ++i) acc[c + i] += __uint_as_float(r[i]);
            }
            t5_fence_before();
            t5_arrive(&acc_empty[st]);
        }
        const int n = n0 + quarter * 32 + lane;
        if (ok && n < N) {
            float* out = y + static_cast<size_t>(blockIdx.z) * M * N;
            const int k_from = kb0 * LT_K, k_to = min(K, (kb0 + kbs) * LT_K);
#pragma unroll
            for (int i = 0; i < COLS; ++i) {
                const int m = m0 + part * COLS + i;
                if (m >= M) continue;
                float v = acc[i];
                if (!(fabsf(v) <= 3.402823466e38f)) {             // infinite or NaN: what plain multiply-adds make of it
                    v = 0.0f;
                    const float *xr = x + static_cast<size_t>(m) * K, *wr = w + static_cast<size_t>(n) * K;
#pragma unroll 1
                    for (int k = k_from; k < k_to && v == v; k += 4) {      // a sum that is NaN stays it
                        const float4 a = *reinterpret_cast<const float4*>(xr + k), b = *reinterpret_cast<const float4*>(wr + k);
                        v = fmaf(a.w, b.w, fmaf(a.z, b.z, fmaf(a.y, b.y, fmaf(a.x, b.x, v))));
                    }
                }
                out[static_cast<size_t>(m) * N + n] = v;
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

// Four neighbours a thread, one where the length is no multiple of four (the parts then start anywhere).  The same sums in the
// same order; three parts of 500 x 6,144: 17 us with one value a thread, now 11.
template <typename V>
__global__ void linear_f32_sum_kernel(const V* __restrict__ parts, V* __restrict__ y, long long n, int splits) {
    pdl_begin();
    const long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) return;
    V v = parts[i];
    for (int s = 1; s < splits; ++s) {
        const V p = parts[s * n + i];
        if constexpr (sizeof(V) == 16) { v.x += p.x; v.y += p.y; v.z += p.z; v.w += p.w; }
        else v += p;
    }
    y[i] = v;
}

static bool lt_encode_f32(CUtensorMap* map, const void* base, long long cols, long long rows, int box_rows) {
    CUtensorMap probe;
    if (g_t5_state == 0 && !t5_encode_2d(&probe, base, 64, 128, 64, 8)) return false;      // looks the encoder up
    if (g_t5_state < 0 || rows >= (1LL << 31)) return false;
    const cuuint64_t dims[2] = {static_cast<cuuint64_t>(cols), static_cast<cuuint64_t>(rows)};
    const cuuint64_t strides[1] = {static_cast<cuuint64_t>(cols) * sizeof(float)};
    const cuuint32_t box[2] = {32u, static_cast<cuuint32_t>(box_rows)};
    const cuuint32_t estr[2] = {1u, 1u};
    return g_t5_encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<void*>(base), dims, strides, box, estr,
                       CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                       CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

static int lt_tile(int M) { return M <= 32 ? 32 : M <= 64 ? 64 : 128; }

// Into how many parts K is cut: the least of waves of 148 CTAs x (blocks of 64 x BLK + 4 us) + the parts' way through memory,
// with a block's time (1.5 us at 128 tokens, 1.0 below: a fifth more than it takes, and fewer parts of equal time
// would sum longer runs).  In 1, 2, 3, 4, 6, 8 parts (us, cold): 500 tokens of 6144 x 4096 169, 151, 146, 173, 183, 206 (takes 3), of 4096 x
// 4096 93, 103, 110, 120, 134, 144 (1), of 4096 x 12288 247, 261, then at lower clocks 319, 328, 336, 328 (1); 17 tokens of 4096 x 12288 239,
// 128, 85, 65, 83, 71 (4), of 24576 x 4096 149, 120, 114, 126, 124, 130 (3).
extern "C" int llm_linear_f32_tcgen05_splits(int M, int N, int K) {
    if (M <= 0 || N <= 0 || K <= 0) return 1;
    const int nt = lt_tile(M);
    const long long tiles = static_cast<long long>((M + nt - 1) / nt) * ((N + LT_ROWS - 1) / LT_ROWS);
    const int kb = (K + LT_K - 1) / LT_K;
    const double block = nt == 128 ? 1.5 : 1.0;
    int best = 1;
    double least = 0.0;
    for (int s = 1; s <= 8 && (s == 1 || kb / s >= 8); ++s) {        // a part is at least eight blocks
        const int per = (kb + s - 1) / s;
        if (s > 1 && ((kb + per - 1) / per != s || 4LL * s * M * N > (64 << 20))) continue;
        const double us = static_cast<double>((tiles * s + 147) / 148) * (per * block + 4.0) + (s > 1 ? 3.0 + 8e-6 * s * M * N / 4.0 : 0.0);
        if (s == 1 || us < least) { least = us; best = s; }
    }
    return best;
}

// x: float32 [M, K]; w: float32 [N, K]; y: float32 [M, N]; planes: room for 3 * M * K bfloat16; parts: room for splits * M * N
// floats when splits > 1.  K a multiple of 8.
extern "C" int llm_linear_f32_tcgen05(const float* x, const float* w, float* y, void* planes, float* parts, int splits, int M, int N,
                                      int K, int32_t* status, uintptr_t stream) {
    if (M <= 0 || N <= 0) return LLM_OK;
    if (K <= 0 || (K & 7) || splits < 1 || (splits > 1 && !parts) || 3LL * M >= (1LL << 31)) return LLM_REFUSED_SIZE;
    if (!aligned16(x) || !aligned16(w) || !aligned16(planes)) return LLM_REFUSED_ALIGN;
    const int nt = lt_tile(M), kb = (K + LT_K - 1) / LT_K, per = (kb + splits - 1) / splits;
    if ((kb + per - 1) / per != splits || (N + LT_ROWS - 1) / LT_ROWS > 65535) return LLM_REFUSED_SIZE;
    CUtensorMap w_map, x_map;
    if (!lt_encode_f32(&w_map, w, K, N, LT_ROWS) || !t5_encode_2d(&x_map, planes, K, 3LL * M, LT_K, nt)) return LLM_REFUSED_SIZE;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    const long long pieces = static_cast<long long>(M) * K / 8;
    launch_pdl(linear_f32_split_kernel, dim3(static_cast<unsigned>((pieces + 255) / 256)), dim3(256), 0, s, x, static_cast<uint4*>(planes), pieces);
    const dim3 grid((M + nt - 1) / nt, (N + LT_ROWS - 1) / LT_ROWS, splits);
    float* to = splits > 1 ? parts : y;
#define GO(NT, WB, XS, PS)                                                                                                    \
    {                                                                                                                   \
        auto kern = linear_f32_tcgen05_kernel<NT, WB, XS, PS>;                                                                 \
        const size_t smem = WB * LT_BOX + XS * 3 * NT * LT_K * sizeof(bf16) + 1024;                    \
        const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)); \
        if (e != cudaSuccess) return static_cast<int>(e);                                                               \
        launch_pdl(kern, grid, dim3(LT_THREADS), smem, s, w_map, x_map, x, w, to, M, N, K, per, status);                \
    }
    if (nt == 32) GO(32, 8, 5, 4) else if (nt == 64) GO(64, 6, 5, 4) else GO(128, 4, 3, 2)
#undef GO
    if (splits > 1) {
        const long long n = static_cast<long long>(M) * N, n4 = n / 4;
        if (n % 4 == 0 && aligned16(parts) && aligned16(y))
            launch_pdl((linear_f32_sum_kernel<float4>), dim3(static_cast<unsigned>((n4 + 255) / 256)), dim3(256), 0, s,
                       reinterpret_cast<const float4*>(parts), reinterpret_cast<float4*>(y), n4, splits);
        else
            launch_pdl((linear_f32_sum_kernel<float>), dim3(static_cast<unsigned>((n + 255) / 256)), dim3(256), 0, s, static_cast<const float*>(parts), y, n, splits);
    }
    return launch_status();
}
