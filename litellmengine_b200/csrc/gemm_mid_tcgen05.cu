// y[M, N] = x[M, K] . w[N, K]^T for 17 to 48 rows (decode steps of a few dozen requests): the weights stream once through the
// 5th-generation tensor cores.
//
// Bytes bound such a product: every weight is read once, for 2 M flops.  The weights are the tensor cores' left operand (128 features
// a tile) and the tokens the right one (N 32 or 48), so that no lane of a product is spent on tokens that are not there.
//   * The SMs are filled by cutting K: the CTAs of a tile are one cluster, each takes an even part of K, and they add their
//     sums up in each other's shared memory, in the parts' order.  Nothing is left for another kernel, no result depends on timing.
//   * Gate and up: a tile is 64 gate features and the 64 up features beside them, and the cluster writes act(gate) * up.
//   * Weights do not depend on the kernel in front: a CTA's first stages are on their way before it waits for that kernel, and two
//     CTAs an SM hold up to 200 KB of them.
//   * The issuing warp walks its stages with all lanes (a wait inside a branch for one lane keeps the tensor pipe idle for 250 clocks).
//   * Weights come as boxes of the matrix as it is: the stored blocks of gemm_skinny.cu instead were -1.0 to +5 us of 5 to 52.
// Roles: warp 0 feeds the copy engine, warp 1 issues, warps 2 to 5 take the sums (a thread a feature); all six add the parts.
// Waits are bounded: one that runs out, in whichever warp, sets status code 8 (the result is then flagged), and the feeding thread waits
// for its last copies before the CTA ends.
//
// Against the library product (gated: and the activation kernel), cold weights, us at 17 / 40 rows; [floor by bytes]:
//   1,024 x 3,072   3.8, 7.1 / 4.4, 6.6  [1.0]      5,120 x 13,824  25.4, 31.1 / 26.6, 32.5  [21.6]
//   4,096 x 4,096   8.2, 9.8 / 9.3, 9.9  [5.1]      2,048 x 26,112  21.6, 25.4 / 22.6, 25.7  [16.3]
//   6,144 x 4,096   10.9, 11.7 / 11.7, 11.8  [7.7]  151,936 x 2,048  98.7, 105 / 103, 108  [95]
//   4,096 x 12,288  18.8, 21.9 / 20.1, 21.9  [15.4] gated 2 x 12,288 x 4,096  36.6, 38.0 / 37.7, 38.9  [30.7]
// At 64 rows it was level or slower (4,096 x 2,048: 7.6 against 6.3; 5,120 x 5,120: 13.4, 11.9): the sums of the parts grow with the
// rows.  Adding them with one load in flight a thread instead of eight cost 20 us at 24,576 x 4,096 in three parts.
#include "tcgen05_attention.cuh"

#define GD_ROWS 128          // features of a tile (gated: 64 of both)
#define GD_K 64              // k-values of a stage: 128-byte rows
#define GD_PIECE (64 * GD_K) // weights of one copy
#define GD_THREADS 192
#define GD_MAX_TOKENS 48
#define GD_STATUS 8

__device__ __forceinline__ bool gd_wait(unsigned long long* bar, unsigned parity, int waits, volatile int* abort_flag, int32_t* status) {
    for (int i = 0; i < waits; ++i) {
        if (t5_try_wait(bar, parity)) return true;
        if (*abort_flag) return false;
    }
    *abort_flag = 1;
    if (atomicCAS(status, 0, GD_STATUS) == 0) status[1] = blockIdx.y;
    return false;
}

// grid (parts of K, tiles), a cluster the parts of a tile.  N: features of the result.
template <int NT, int STAGES, bool GATED, typename TO>
__global__ void __launch_bounds__(GD_THREADS, 2) linear_mid_kernel(
    const __grid_constant__ CUtensorMap w_map, const __grid_constant__ CUtensorMap x_map, TO* __restrict__ y,
    int M, int N, int K, int act, float limit, int waits, int32_t* __restrict__ status) {
    constexpr int X_PIECE = NT * GD_K;
    constexpr unsigned W_BYTES = 2 * GD_PIECE * sizeof(bf16), X_BYTES = X_PIECE * sizeof(bf16);
    extern __shared__ unsigned char smem_dyn[];
    unsigned char* smem_al = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_dyn) + 1023) & ~uintptr_t(1023));
    bf16* w_s = reinterpret_cast<bf16*>(smem_al);                 // [STAGES][2][64][64], 128-byte swizzle
    bf16* x_s = w_s + STAGES * 2 * GD_PIECE;                      // [STAGES][NT][64]
    float* sums = reinterpret_cast<float*>(smem_al);              // [NT][128], when the stages have been read
    __shared__ __align__(8) unsigned long long full[STAGES], empty[STAGES], acc_full;
    __shared__ unsigned tmem_base_s;
    __shared__ int abort_flag;
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int part = blockIdx.x, parts = gridDim.x, tile = blockIdx.y;
    const int kb_all = (K + GD_K - 1) / GD_K, kb0 = part * kb_all / parts, kbs = (part + 1) * kb_all / parts - kb0;
    const int row0 = GATED ? tile * 64 : tile * GD_ROWS, row1 = GATED ? N + tile * 64 : row0 + 64;      // the tile's two pieces of 64 rows
    if (tid == 0) {
        abort_flag = 0;
        for (int s = 0; s < STAGES; ++s) { t5_mbar_init(&full[s], 1); t5_mbar_init(&empty[s], 1); }
        t5_mbar_init(&acc_full, 1);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(t5_smem(&tmem_base_s)), "r"(64u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    t5_fence_before();
    __syncthreads();
    t5_fence_after();
    pdl_invite();                                                 // not before: this CTA's tensor memory is taken
    const unsigned tmem = __shfl_sync(0xffffffffu, tmem_base_s, 0);

    int issued = 0;                                               // stages that were asked for, in the thread that asks
    if (warp == 0) {
        if (lane == 0) {
            auto weights = [&](int kb) {                          // both pieces of a stage; the stage is free
                const int st = kb % STAGES, k = (kb0 + kb) * GD_K;
                t5_expect_tx(&full[st], W_BYTES + X_BYTES);
#pragma unroll
                for (int p = 0; p < 2; ++p) t5_tma_2d(w_s + (st * 2 + p) * GD_PIECE, &w_map, k, p ? row1 : row0, &full[st]);
            };
            auto tokens = [&](int kb) { t5_tma_2d(x_s + (kb % STAGES) * X_PIECE, &x_map, (kb0 + kb) * GD_K, 0, &full[kb % STAGES]); };
            const int first = min(STAGES, kbs);
            for (int kb = 0; kb < first; ++kb) weights(kb);       // nobody's output
            pdl_wait();
            for (int kb = 0; kb < first; ++kb) tokens(kb);
            issued = first;
            for (int kb = STAGES; kb < kbs; ++kb) {
                if (!gd_wait(&empty[kb % STAGES], (kb / STAGES - 1) & 1, waits, &abort_flag, status)) break;
                weights(kb);
                tokens(kb);
                issued = kb + 1;
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        pdl_wait();
        constexpr unsigned IDESC = t5_idesc(GD_ROWS, NT, 0);
        const unsigned lead = elect_one();
        const unsigned long long wd = t5_desc(w_s, 16, 1024), xd = t5_desc(x_s, 16, 1024);
        bool ok = true;
#pragma unroll 1
        for (int kb = 0; kb < kbs; ++kb) {
            const int st = kb % STAGES;
            ok = __all_sync(0xffffffffu, gd_wait(&full[st], (kb / STAGES) & 1, waits, &abort_flag, status));
            if (!ok) break;
#pragma unroll
            for (int k = 0; k < GD_K / 16; ++k)
                t5_mma_ss_lead(lead, tmem, wd + st * (W_BYTES >> 4) + 2 * k, xd + st * (X_BYTES >> 4) + 2 * k, IDESC, (kb | k) ? 1u : 0u);
            t5_commit_lead(lead, &empty[st]);
        }
        if (ok) t5_commit_lead(lead, &acc_full);
    } else {
        pdl_wait();
        const int quarter = warp & 3, row = quarter * 32 + lane;
        const bool ok = __all_sync(0xffffffffu, gd_wait(&acc_full, 0, waits, &abort_flag, status));
        t5_fence_after();
        unsigned r[NT / 16][16];
#pragma unroll
        for (int c = 0; c < NT / 16; ++c) t5_ld16(tmem + (static_cast<unsigned>(quarter * 32) << 16) + 16 * c, r[c]);
        t5_wait_ld();
        if (ok)
#pragma unroll
            for (int c = 0; c < NT / 16; ++c)
#pragma unroll
                for (int i = 0; i < 16; ++i) sums[(16 * c + i) * GD_ROWS + row] = __uint_as_float(r[c][i]);
    }
    t5_fence_before();
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");      // every part's sums are there
    {
        // The parts' sums in order, four features a thread, all parts' loads in flight at once.
        const unsigned base = t5_smem(sums);
        auto total = [&](int at) {
            float4 f[8];
#pragma unroll
            for (int p = 0; p < 8; ++p)
                if (p < parts) {
                    unsigned addr;
                    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(addr) : "r"(base + 4u * at), "r"(p));
                    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];\n" : "=f"(f[p].x), "=f"(f[p].y), "=f"(f[p].z), "=f"(f[p].w) : "r"(addr));
                }
            float4 v = f[0];
#pragma unroll
            for (int p = 1; p < 8; ++p)
                if (p < parts) v.x += f[p].x, v.y += f[p].y, v.z += f[p].z, v.w += f[p].w;
            return v;
        };
        if constexpr (GATED) {
            const int f = 4 * (tid & 15);
#pragma unroll 2
            for (int tok = part + (tid >> 4) * parts; tok < M; tok += GD_THREADS / 16 * parts) {
                const float4 g = total(tok * GD_ROWS + f), u = total(tok * GD_ROWS + 64 + f);
                const float gs[4] = {g.x, g.y, g.z, g.w}, us[4] = {u.x, u.y, u.z, u.w};
                __align__(8) bf16 out[4];
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    out[i] = from_f32<bf16>(gated(to_f32(from_f32<bf16>(gs[i])), to_f32(from_f32<bf16>(us[i])), act, limit));
                *reinterpret_cast<uint2*>(y + static_cast<size_t>(tok) * N + tile * 64 + f) = *reinterpret_cast<const uint2*>(out);
            }
        } else {
            const int f = 4 * lane;
#pragma unroll 2
            for (int tok = part + warp * parts; tok < M; tok += GD_THREADS / 32 * parts) {
                const float4 t = total(tok * GD_ROWS + f);
                const float ts[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    if (row0 + f + i < N) y[static_cast<size_t>(tok) * N + row0 + f + i] = from_f32<TO>(ts[i]);
            }
        }
    }
    if (tid == 0 && abort_flag)                                   // whoever gave up: what is in flight lands before the CTA goes away
        for (int kb = max(0, issued - STAGES); kb < issued; ++kb)
            for (int i = 0; i < T5_WAIT_LIMIT && !t5_try_wait(&full[kb % STAGES], (kb / STAGES) & 1); ++i) {}
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");      // nobody leaves while its sums are read
    if (warp == 1) {
        t5_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(64u) : "memory");
    }
}

// ---- host side ------------------------------------------------------------------------------------------------------
static int g_gd_sms = 0;
static bool gd_device() {
    if (g_gd_sms) return true;
    int dev = 0;
    return cudaGetDevice(&dev) == cudaSuccess && cudaDeviceGetAttribute(&g_gd_sms, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess && g_gd_sms > 0;
}

// Sizes this kernel takes: rows of whole 16-byte pieces and, gated, features that fill their tiles.
extern "C" int llm_linear_mid_supported(int M, int N, int K, int gated) {
    return M >= 1 && M <= GD_MAX_TOKENS && N >= 1 && N <= (1 << 22) && K >= GD_K && K % 8 == 0 && K <= (1 << 20) && (!gated || N % 64 == 0) && gd_device();
}

// Into how many parts K is cut: the most, up to 8 (a cluster), with which all clusters run at once.  Two CTAs an SM, less an eighth,
// because clusters do not fill a group of SMs to the last slot: 9,216 x 4,096 in two parts (144 CTAs) took 15.6 us, in three (216)
// 14.9, in four (288) 20.9; 6,144 x 4,096 in four (192) 11.6, five (240) 10.9, six (288) 15.7; 24,576 x 4,096 (192 tiles) in one 36,
// two 40.9, three 43.
extern "C" int llm_linear_mid_parts(int N, int K, int gated) {
    if (!gd_device()) return 1;
    const long long tiles = gated ? (N + 63) / 64 : (N + GD_ROWS - 1) / GD_ROWS, slots = 2LL * g_gd_sms * 7 / 8;
    const int kb = (K + GD_K - 1) / GD_K;
    int best = 1;
    while (best < 8 && (best + 1) * tiles <= slots && kb / (best + 1) >= 4) ++best;
    return best;
}

template <int NT, int STAGES, bool GATED, typename TO>
static int gd_launch(const void* x, const void* w, void* y, int M, int N, int K, int act, float limit, int parts, int waits, int32_t* status, cudaStream_t s) {
    CUtensorMap w_map, x_map;
    if (!t5_encode_2d(&x_map, x, K, M, GD_K, NT)) return LLM_REFUSED_SIZE;
    if (!t5_encode_2d(&w_map, w, K, static_cast<long long>(N) * (GATED ? 2 : 1), GD_K, 64)) return LLM_REFUSED_SIZE;
    const size_t smem = static_cast<size_t>(STAGES) * (2 * GD_PIECE + NT * GD_K) * sizeof(bf16) + 1024;
    auto kern = linear_mid_kernel<NT, STAGES, GATED, TO>;
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    if (e != cudaSuccess) return static_cast<int>(e);
    const int tiles = GATED ? N / 64 : (N + GD_ROWS - 1) / GD_ROWS;
    if (tiles > 65535) return LLM_REFUSED_SIZE;
    launch_pdl_cluster(kern, dim3(parts, tiles), dim3(GD_THREADS), smem, s, parts, w_map, x_map, static_cast<TO*>(y), M, N, K,
                       act, limit, waits, status);
    return launch_status();
}

// x: bfloat16 [M, K]; w: bfloat16 [N, K] (gated: [2 N, K] = [gate; up]);
// y: [M, N] float32 or bfloat16; gated: bfloat16, act 0 silu, 1 the tanh form of gelu, 2 the clamped form with `limit`, gate and up
// rounded to bfloat16 first.  waits: tries of a wait (each suspends for a while) before it gives up.
extern "C" int llm_linear_mid(const void* x, const void* w, void* y, int out_dtype, int gated, int act, float limit, int M, int N, int K,
                              int waits, int32_t* status, uintptr_t stream) {
    if (!llm_linear_mid_supported(M, N, K, gated)) return LLM_REFUSED_SIZE;
    if (gated && (act < 0 || act > 2 || (act == 2 && !(limit > 0.0f)))) return LLM_REFUSED_SIZE;
    if ((out_dtype != LLM_DT_F32 && out_dtype != LLM_DT_BF16) || (gated && out_dtype != LLM_DT_BF16)) return LLM_REFUSED_DTYPE;
    if (!aligned16(x) || !aligned16(w) || status == nullptr) return LLM_REFUSED_ALIGN;
    const int parts = llm_linear_mid_parts(N, K, gated);
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
#define GO_M(GATED, TO)                                                                                \
    return M <= 32 ? gd_launch<32, 5, GATED, TO>(x, w, y, M, N, K, act, limit, parts, waits, status, s)      \
                   : gd_launch<48, 5, GATED, TO>(x, w, y, M, N, K, act, limit, parts, waits, status, s)
    if (gated) GO_M(true, bf16);
    if (out_dtype == LLM_DT_F32) GO_M(false, float);
    GO_M(false, bf16);
#undef GO_M
}
