// y[M, N] = x[M, K] . w[N, K]^T for up to 16 rows and weights that the SMs' shared memory holds all at once: the products of a
// small model's decode step.
//
// Such a step is a chain of kernels that wait for one another, and what it takes is their number times the way from one to the
// next; bytes do not bound it (the 0.6B layer's products are 4 to 13 MB).  So a product here leaves nothing for another kernel:
//   * A CTA takes 16 output features and ALL of K (its eight warps share K and add their sums up in shared memory), so there
//     are no partial sums.  gemm_skinny.cu gives a CTA 64 features by 512 k-values, which moves large weights faster, but its 4
//     to 6 sums an output are read again by the next kernel.
//   * Its weights (16 x K, pieces of 2 KB) are asked for before the wait for the kernel in front.  The rule that sends a product
//     here (llm_linear_small_supported) is that every CTA is on an SM at once: then all of the weights are on their way while that
//     kernel still runs.
//   * The rows may be made on the way (`normed`): rmsnorm of the residual stream plus what is pending, a warp a row, every CTA for
//     itself (2 x M x K floats from L2).  Row r of the sum is written to another buffer by CTA r: the stream itself is still
//     being read by the rest of the grid.
//   * Gate and up (`gated`): a CTA takes 16 features of both and writes act(gate) * up, both rounded to bfloat16 first.
// The norm's and the activation's numbers are those of norm.cu and activation.cu, added in their order.
// A decode step of 8 layers of width 1,024 at a context of 320, us, before (streaming product, norm and activation kernels) and now: 1
// request 268, 233; 5 287, 252; 8 303, 278; 9 334, 311; 16 347, 330.  Rows made by every CTA pay up to 8 of them: with more
// the stream is read too often (16 requests 354; and with 16 features a CTA instead of 32, 374).  It is better where the next kernel's
// CTAs find room while this one's still run: with 8 eights of a row held where 4 do, 267 us for 5 requests instead of 247; rows of more
// than 1,024 values, whose CTAs take 110 to 170 KB, are not left to a product by a block (`rows_worth_leaving` in ops.py).
// Products run on mma.sync m16n8k16 with the weights as the 16-row operand and the tokens as the 8 columns; sums are float32.
// The wait for the weights is bounded: a thread whose tries run out records status code 8 and goes on (the result is then flagged), but
// does not end before the copies have landed, for which it waits, bounded again: the block's memory may be another one's next.
#include "common.cuh"
#include <cuda.h>

#define GM_ROWS 16          // output features of a CTA
#define GM_THREADS 256
#define GM_WARPS 8
#define GM_SUB 64           // k-values of a piece of weights: 16 rows of 128 bytes, chunks of 16 bytes XOR-swizzled by the row
#define GM_DRAIN_LIMIT 8000000
#define GM_HELD 8           // eights of a row that a lane of a norming warp holds at most: rows of up to 2,048

__device__ __forceinline__ unsigned gm_smem(const void* p) { return static_cast<unsigned>(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ bool gm_try_wait(unsigned long long* bar, unsigned parity) {
    unsigned ok;
    asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
                 : "=r"(ok) : "r"(gm_smem(bar)), "r"(parity) : "memory");
    return ok != 0;
}
__device__ __forceinline__ void gm_ldmatrix_x4(unsigned (&r)[4], const void* smem) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(gm_smem(smem)));
}
__device__ __forceinline__ void gm_mma(float (&c)[4], const unsigned (&a)[4], unsigned b0, unsigned b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// 16-byte chunk `chunk` (of 8) of row `row` in a [rows][64] piece
__device__ __forceinline__ bf16* gm_at(bf16* base, int row, int chunk) { return base + row * GM_SUB + ((chunk ^ (row & 7)) << 3); }


// Where the rows come from: x (bfloat16 [M, K]), or h, pending and the norm's weight g.
struct GmRows {
    const bf16* x;
    const float *h, *pending, *g;
    float* h_out;
    long long pending_stride;
    int pending_parts;
    float eps;
};

// Shared memory of the weights, and after them of the warps' sums.
__host__ __device__ constexpr int gm_first_bytes(int mt, int slabs, int subs) {
    const int w = slabs * subs * GM_ROWS * GM_SUB * 2, sums = GM_WARPS * slabs * GM_ROWS * mt * 4;
    return w > sums ? w : sums;
}

// Slabs of 16 weight rows a CTA takes: gate and up, or two neighbours where each CTA makes its rows (a CTA for every 32 features
// then reads half as much of the stream in all).
#define GM_SLABS(GATED, HELD) ((GATED) || (HELD) > 0 ? 2 : 1)

// HELD: eights of a row that a lane of a norming warp holds (4 or 8; 0: the rows are there).
template <int MT, int HELD, bool GATED, typename TO, bool BOXES>
__global__ void __launch_bounds__(GM_THREADS, HELD == 8 ? 2 : 3) linear_small_kernel(const GmRows in, const bf16* __restrict__ w_tiled, TO* __restrict__ y,
                                                                  int M, int N, int K, int act, float limit, int waits, int32_t* __restrict__ status,
                                                                  const __grid_constant__ CUtensorMap w_map) {
    constexpr int SLABS = GM_SLABS(GATED, HELD), PIECE = GM_ROWS * GM_SUB, SUMS = GM_ROWS * MT;
    extern __shared__ __align__(1024) unsigned char smem_raw[];          // the swizzle's pattern repeats every 1024 bytes
    const int subs = (K + GM_SUB - 1) / GM_SUB;
    bf16* w_s = reinterpret_cast<bf16*>(smem_raw);                       // [slabs][subs][16][64]
    float* sum_s = reinterpret_cast<float*>(smem_raw);                   // [warps][slabs][MT][16], where the weights have been
    bf16* x_s = reinterpret_cast<bf16*>(smem_raw + gm_first_bytes(MT, SLABS, subs));      // [subs][MT][64]
    __shared__ __align__(8) unsigned long long full;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int n0 = blockIdx.x * GM_ROWS * (GATED ? 1 : SLABS);

    pdl_invite();
    if (warp == 0) {
        if (lane == 0) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(gm_smem(&full)));
            asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(gm_smem(&full)),
                         "r"(static_cast<unsigned>(SLABS * subs * PIECE * sizeof(bf16))) : "memory");
        }
        __syncwarp();
        for (int i = lane; i < SLABS * subs; i += 32) {                  // the weights do not depend on the kernel before this one
            const int slab = i / subs, sub = i % subs;
            const int row = n0 + slab * (GATED ? N : GM_ROWS);           // gated: the up rows lie N rows behind the gate rows
            bf16* dst = w_s + i * PIECE;
            if constexpr (BOXES) {
                asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];\n" ::
                                 "r"(gm_smem(dst)), "l"(&w_map), "r"(sub * GM_SUB), "r"(row), "r"(gm_smem(&full)) : "memory");
            } else {                                                     // stored blocks of 64 rows x 256 k-values, four pieces of 64 each
                const size_t block = static_cast<size_t>(row / 64) * ((K + 255) / 256) + sub / 4;
                asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::
                                 "r"(gm_smem(dst)), "l"(w_tiled + (block * 4 + sub % 4) * (64 * GM_SUB) + (row % 64) * GM_SUB),
                             "r"(static_cast<unsigned>(PIECE * sizeof(bf16))), "r"(gm_smem(&full)) : "memory");
            }
        }
    }
    float* g_s = reinterpret_cast<float*>(x_s + subs * MT * GM_SUB);     // HELD: [K], the norm's weight
    if constexpr (HELD > 0)
        for (int k = tid * 4; k < K; k += GM_THREADS * 4) *reinterpret_cast<float4*>(g_s + k) = *reinterpret_cast<const float4*>(in.g + k);
    __syncthreads();
    pdl_wait();
    if constexpr (HELD > 0) {
        for (int r = warp; r < MT; r += GM_WARPS) {
            float v[HELD][8];
            const bool there = r < M;
            const size_t at = static_cast<size_t>(r) * K;
            float total = 0.0f, inv = 0.0f;
            if (there) {
#pragma unroll
                for (int j = 0; j < HELD; ++j) {
                    const int k = (j * 32 + lane) * 8;
                    if (k < K) load8(in.h + at + k, v[j]);
                }
                if (in.pending) {
                    for (int part = 0; part < in.pending_parts; ++part) {
                        const float* p = in.pending + part * in.pending_stride + at;
#pragma unroll
                        for (int j = 0; j < HELD; ++j) {
                            const int k = (j * 32 + lane) * 8;
                            if (k < K) {
                                float b[8];
                                load8(p + k, b);
#pragma unroll
                                for (int u = 0; u < 8; ++u) v[j][u] += b[u];
                            }
                        }
                    }
                }
                // the sum of squares as norm.cu adds it: a thread's eight values one after the other, the threads of a warp by
                // halves, then the warps by halves
                float s[HELD];
#pragma unroll
                for (int j = 0; j < HELD; ++j) {
                    s[j] = 0.0f;
                    if ((j * 32 + lane) * 8 < K) {
#pragma unroll
                        for (int u = 0; u < 8; ++u) s[j] += v[j][u] * v[j][u];
                    }
                }
#pragma unroll
                for (int j = 0; j < HELD; ++j) s[j] = warp_sum(s[j]);
                // (sums of warps that have no values are zero)
                if constexpr (HELD == 8) total = ((s[0] + s[4]) + (s[2] + s[6])) + ((s[1] + s[5]) + (s[3] + s[7]));
                else total = (s[0] + s[2]) + (s[1] + s[3]);
                inv = 1.0f / sqrtf(total / static_cast<float>(K) + in.eps);
            }
#pragma unroll
            for (int j = 0; j < HELD; ++j) {
                const int k = (j * 32 + lane) * 8;
                if (k >= subs * GM_SUB) continue;
                float a[8] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
                if (there && k < K) {
                    float g[8];
                    load8(g_s + k, g);
#pragma unroll
                    for (int u = 0; u < 8; ++u) a[u] = v[j][u] * inv * g[u];
                    if (in.h_out && blockIdx.x == r % gridDim.x) store8(in.h_out + at + k, v[j]);
                }
                store8(gm_at(x_s + (k / GM_SUB) * MT * GM_SUB, r, (k % GM_SUB) / 8), a);
            }
        }
    } else {
        const int chunks = subs * 8;                                     // 16-byte chunks of a row
        for (int c = tid; c < MT * chunks; c += GM_THREADS) {
            const int r = c / chunks, ch = c % chunks;
            const bool there = r < M && ch * 8 < K;
            const unsigned dst = gm_smem(gm_at(x_s + (ch >> 3) * MT * GM_SUB, r, ch & 7));
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(in.x + (there ? static_cast<size_t>(r) * K + ch * 8 : 0)),
                         "r"(there ? 16 : 0));
        }
        asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
    }
    __syncthreads();                                                     // the rows are there, and the barrier exists for everyone
    bool landed = false;
    for (int n = 0; n < waits && !landed; ++n) landed = gm_try_wait(&full, 0);
    float acc[SLABS][MT / 8][4], acc2[SLABS][MT / 8][4];                 // over the even and the odd steps of 16 k-values
#pragma unroll
    for (int z = 0; z < SLABS; ++z)
#pragma unroll
        for (int j = 0; j < MT / 8; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[z][j][e] = acc2[z][j][e] = 0.0f;
    for (int sub = warp; sub < subs; sub += GM_WARPS) {
        bf16* xs = x_s + sub * MT * GM_SUB;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            unsigned b[MT / 8][4];                                       // tokens 8j..8j+7, two steps of 16 k-values
#pragma unroll
            for (int j = 0; j < MT / 8; ++j) gm_ldmatrix_x4(b[j], gm_at(xs, j * 8 + (lane & 7), h * 4 + (lane >> 3)));
#pragma unroll
            for (int z = 0; z < SLABS; ++z) {
                bf16* ws = w_s + (z * subs + sub) * PIECE;
                unsigned a0[4], a1[4];
                gm_ldmatrix_x4(a0, gm_at(ws, (lane & 7) + ((lane >> 3) & 1) * 8, h * 4 + (lane >> 4)));
                gm_ldmatrix_x4(a1, gm_at(ws, (lane & 7) + ((lane >> 3) & 1) * 8, h * 4 + 2 + (lane >> 4)));
#pragma unroll
                for (int j = 0; j < MT / 8; ++j) gm_mma(acc[z][j], a0, b[j][0], b[j][1]);
#pragma unroll
                for (int j = 0; j < MT / 8; ++j) gm_mma(acc2[z][j], a1, b[j][2], b[j][3]);
            }
        }
    }
    __syncthreads();                                                     // everyone has read the weights
#pragma unroll
    for (int z = 0; z < SLABS; ++z)
#pragma unroll
        for (int j = 0; j < MT / 8; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e)
                sum_s[(warp * SLABS + z) * SUMS + (j * 8 + (lane & 3) * 2 + (e & 1)) * GM_ROWS + (lane >> 2) + (e >> 1) * 8] = acc[z][j][e] + acc2[z][j][e];
    __syncthreads();
    for (int o = tid; o < (GATED ? 1 : SLABS) * SUMS; o += GM_THREADS) {  // a thread an output, the warps' sums in order
        const int tok = o % SUMS / GM_ROWS, f = n0 + o / SUMS * GM_ROWS + o % GM_ROWS;
        if (tok >= M || f >= N) continue;
        auto sum_of = [&](int at) {
            float v = sum_s[at];
#pragma unroll
            for (int p = 1; p < GM_WARPS; ++p) v += sum_s[p * SLABS * SUMS + at];
            return v;
        };
        float out = sum_of(o);
        if constexpr (GATED) out = gated(to_f32(from_f32<bf16>(out)), to_f32(from_f32<bf16>(sum_of(SUMS + o))), act, limit);
        y[static_cast<size_t>(tok) * N + f] = from_f32<TO>(out);
    }
    if (!landed) {
        if (atomicCAS(status, 0, 8) == 0) status[1] = blockIdx.x;
        for (int n = 0; n < GM_DRAIN_LIMIT && !gm_try_wait(&full, 0); ++n) {}
    }
}

// ---- host side ------------------------------------------------------------------------------------------------------
static int g_gm_sms = 0;
static bool gm_device() {
    if (g_gm_sms) return true;
    int dev = 0;
    return cudaGetDevice(&dev) == cudaSuccess && cudaDeviceGetAttribute(&g_gm_sms, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess && g_gm_sms > 0;
}
static long long gm_bytes(int mt, int K, bool normed, bool gated) {
    const int subs = (K + GM_SUB - 1) / GM_SUB;
    return gm_first_bytes(mt, GM_SLABS(gated, normed), subs) + static_cast<long long>(subs) * GM_SUB * mt * 2 + (normed ? 4LL * K : 0);
}

static int gm_ctas(int N, bool normed, bool gated) {
    const int each = GM_ROWS * (gated ? 1 : GM_SLABS(false, normed));
    return (N + each - 1) / each;
}

// CTAs of a form that an SM holds by their registers: four for up to eight rows that are there, three otherwise, two for wide made rows.
template <int MT, int HELD, bool GATED>
static int gm_resident() {
    static int n = 0;
    if (n == 0 && cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, linear_small_kernel<MT, HELD, GATED, bf16, true>, GM_THREADS, 0) != cudaSuccess) {
        (void)cudaGetLastError();
        n = 0;
    }
    return n;
}
static int gm_resident_of(int M, int K, int normed, int gated) {
    if (normed && K <= 1024) return gated ? gm_resident<8, 4, true>() : gm_resident<8, 4, false>();
    if (normed) return gated ? gm_resident<8, 8, true>() : gm_resident<8, 8, false>();
    if (M <= 8) return gated ? gm_resident<8, 0, true>() : gm_resident<8, 0, false>();
    return gated ? gm_resident<16, 0, true>() : gm_resident<16, 0, false>();
}

// Whether a product of M rows, N features (gated: the activation's, with 2 N rows of weights) over K values comes here: all CTAs on the
// SMs at once, by their registers and in 220 KB of shared memory an SM.  normed: at most eight rows, which a warp's registers hold.
// A second wave of CTAs asks for its weights when the first one is done.  Chains of products, us, this kernel and the streaming product, 8
// rows: K 512, N 11,840 (five CTAs an SM where four fit) 4.8, 3.2; K 256, N 18,944 (eight) 4.4, 3.1; 16 rows, K 256, N 9,472 (four where
// three fit) 4.2, 3.1; gated, K 256, N 9,472 4.4, 4.3.  With a K of up to 512 the streaming product leaves whole sums as well, and is
// faster from 385 on with many features: 8 rows, K 512, N 4,096 2.70, 2.56; 6,144 2.90, 2.64; 9,472 3.16, 2.65; K 448, N 9,472 3.07, 2.66; K
// 384, N 8,192 2.81, 2.90; K 576, N 9,472 3.49, 3.67 and then a kernel that adds the slices.
extern "C" int llm_linear_small_supported(int M, int N, int K, int normed, int gated) {
    if (M < 1 || M > (normed ? 8 : 16) || N < 1 || K < 64 || K % 8 || (normed && K > 256 * GM_HELD) || (gated && N % GM_ROWS) || N > (1 << 20) || K > (1 << 16)) return 0;
    if (!normed && !gated && K > 384 && K <= 512 && N > 4096) return 0;
    if (!gm_device()) return 0;
    const long long each = gm_bytes(M <= 8 ? 8 : 16, K, normed, gated) + 1024, ctas = gm_ctas(N, normed, gated);
    const long long per_sm = (ctas + g_gm_sms - 1) / g_gm_sms;
    return per_sm <= gm_resident_of(M, K, normed, gated) && per_sm * each <= 220 * 1024 ? 1 : 0;
}

typedef CUresult (*GmEncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                               const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static GmEncodeFn g_gm_encode = nullptr;
static int g_gm_encode_state = 0;

// Plain weights [rows, K] in boxes of 16 rows x 64 k-values, 128-byte swizzle: what the stored blocks hold.
static bool gm_weight_map(CUtensorMap* map, const void* w, long long rows, int K) {
    if (g_gm_encode_state == 0) {
        void* fn = nullptr;
        cudaDriverEntryPointQueryResult qres;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qres) == cudaSuccess &&
            qres == cudaDriverEntryPointSuccess && fn != nullptr) {
            g_gm_encode = reinterpret_cast<GmEncodeFn>(fn);
            g_gm_encode_state = 1;
        } else {
            (void)cudaGetLastError();
            g_gm_encode_state = -1;
        }
    }
    if (g_gm_encode_state < 0) return false;
    const cuuint64_t dims[2] = {static_cast<cuuint64_t>(K), static_cast<cuuint64_t>(rows)};
    const cuuint64_t strides[1] = {static_cast<cuuint64_t>(K) * sizeof(bf16)};
    const cuuint32_t box[2] = {GM_SUB, GM_ROWS};
    const cuuint32_t estr[2] = {1u, 1u};
    return g_gm_encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(w), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                       CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int MT, int HELD, bool GATED, typename TO, bool BOXES>
static int gm_launch(const GmRows& in, const void* w, void* y, int M, int N, int K, int act, float limit, int waits, int32_t* status, cudaStream_t s) {
    CUtensorMap map = {};
    if (BOXES && !gm_weight_map(&map, w, static_cast<long long>(N) * (GATED ? 2 : 1), K)) return LLM_REFUSED_ALIGN;
    const size_t smem = static_cast<size_t>(gm_bytes(MT, K, HELD > 0, GATED));
    auto kern = linear_small_kernel<MT, HELD, GATED, TO, BOXES>;
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    if (e != cudaSuccess) return static_cast<int>(e);
    launch_pdl(kern, dim3(gm_ctas(N, HELD > 0, GATED)), dim3(GM_THREADS), smem, s, in, static_cast<const bf16*>(w), static_cast<TO*>(y), M, N, K,
               act, limit, waits, status, map);
    return launch_status();
}

template <int HELD, bool GATED, typename TO>
static int gm_pick(const GmRows& in, const void* w, int tiled, void* y, int M, int N, int K, int act, float limit, int waits, int32_t* status, cudaStream_t s) {
    if (HELD > 0 || M <= 8)
        return tiled ? gm_launch<8, HELD, GATED, TO, false>(in, w, y, M, N, K, act, limit, waits, status, s)
                     : gm_launch<8, HELD, GATED, TO, true>(in, w, y, M, N, K, act, limit, waits, status, s);
    return tiled ? gm_launch<16, 0, GATED, TO, false>(in, w, y, M, N, K, act, limit, waits, status, s)
                 : gm_launch<16, 0, GATED, TO, true>(in, w, y, M, N, K, act, limit, waits, status, s);
}

// x: bfloat16 [M, K], or null: then the rows are rmsnorm(h + pending) * g with h, pending float32 [M, K] (pending: null, or
// pending_parts of them pending_stride apart) and h_out (null, or another buffer than h) = h + pending.  w: bfloat16 [N, K] (gated:
// [2 N, K] = [gate; up]) as it is, or (`tiled`) in the stored blocks of gemm_skinny.cu.  y: [M, N] float32 or bfloat16; gated:
// bfloat16, act 0 silu, 1 the tanh form of gelu, 2 the clamped form with `limit`.  waits: tries of the wait for the weights (each suspends
// for a while) before a block gives up.
extern "C" int llm_linear_small(const void* x, const float* h, const float* pending, int pending_parts, long long pending_stride, const float* g,
                                float eps, float* h_out, const void* w, int tiled, void* y, int out_dtype, int gated, int act, float limit,
                                int M, int N, int K, int waits, int32_t* status, uintptr_t stream) {
    const int normed = x == nullptr;
    if (!llm_linear_small_supported(M, N, K, normed, gated) || (normed && (!h || !g || (pending && pending_parts < 1) || h_out == h)))
        return LLM_REFUSED_SIZE;
    if (gated && (act < 0 || act > 2 || (act == 2 && !(limit > 0.0f)))) return LLM_REFUSED_SIZE;
    if ((out_dtype != LLM_DT_F32 && out_dtype != LLM_DT_BF16) || (gated && out_dtype != LLM_DT_BF16)) return LLM_REFUSED_DTYPE;
    if (!aligned16(x) || !aligned16(h) || !aligned16(pending) || !aligned16(g) || !aligned16(h_out) || pending_stride % 4 ||
        (reinterpret_cast<uintptr_t>(w) & (tiled ? 127u : 15u)) || status == nullptr)
        return LLM_REFUSED_ALIGN;
    GmRows in = {};
    in.x = static_cast<const bf16*>(x);
    in.h = h; in.pending = pending; in.pending_parts = pending_parts; in.pending_stride = pending_stride;
    in.g = g; in.eps = eps; in.h_out = h_out;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
#define GO(GATED, TO)                                                                                     \
    return !normed    ? gm_pick<0, GATED, TO>(in, w, tiled, y, M, N, K, act, limit, waits, status, s)            \
           : K <= 1024 ? gm_pick<4, GATED, TO>(in, w, tiled, y, M, N, K, act, limit, waits, status, s)           \
                       : gm_pick<8, GATED, TO>(in, w, tiled, y, M, N, K, act, limit, waits, status, s)
    if (gated) GO(true, bf16);
    if (out_dtype == LLM_DT_F32) GO(false, float);
    GO(false, bf16);
#undef GO
}
