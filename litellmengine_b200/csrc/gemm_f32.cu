// y[M, N] = x[M, K] . W[N, K]^T in float32 for the few rows of a decode step: the weights stream through once.
//
// What bounds it: the bytes of W.  A warp owns LF_ROWS = 4 weight rows and 1 / KS of their length; a lane reads 16 bytes
// of each row a step (512 contiguous bytes a row and warp), two steps ahead of the arithmetic, so that an SM keeps
// 16 warps x 2 x 2 KB of loads in flight (6.5 TB/s at 0.8 us of latency wants 35 KB).  The token rows come through the
// first-level cache, which all warps of an SM share; W passes it by without being kept.  Per 2 KB of weights a warp
// spends M x 4 multiply-add instructions and M + 4 sixteen-byte loads: at M = 8 both pipes are at a third of their rate
// when W arrives at 6.5 TB/s, at M = 16 at two thirds; above that the arithmetic would bound it.
// A lane's sums are over K / (32 KS) products in order, then lanes and slices are added as a tree: shorter chains, and a
// smaller error, than one running sum over K.
// KS warps of a block share the same rows and cut K, so that matrices of few rows fill the chip too (`lf_fill`).
//
// Measured (us, a chain of products whose weights exceed L2; the library's float32 product in brackets):
//   N x K              1 row          8 rows         16 rows
//   6144 x 4096        17 (34)        24 (62)        39 (79)
//   4096 x 4096        12 (17)        16 (51)        28 (66)
//   24576 x 4096       59 (71)        76 (134)       131 (196)
//   4096 x 12288       33 (44)        41 (136)       70 (142)
//   152000 x 1024      89 (94)        111 (200)      191 (240)
// i.e. 0.9 to 1.0 of the measured copy bandwidth at a row, 0.65 to 0.86 at 8, where the token rows' loads from the
// first-level cache (4 KB per 2 KB of weights) are what is left.  Its error against 64 bits is 1.1e-7 (relative, 2-norm)
// at K = 4096 where the library's is 1.4e-7 to 1.1e-6.  From 17 rows on the arithmetic bounds it (N = 152000, 24 rows:
// 277 against the library's 243): large matrices go to the tensor cores (gemm_f32_tcgen05.cu), small ones to the library.
#include "common.cuh"

#define LF_ROWS 4
#define LF_WARPS 8

__device__ __forceinline__ float4 lf_stream(const float* p) {       // a weight: read once, not kept in the first-level cache
    float4 v;
    asm volatile("ld.global.nc.L1::no_allocate.L2::128B.v4.f32 {%0,%1,%2,%3}, [%4];\n"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
    return v;
}

// grid (groups of MT token rows, groups of weight rows): the blocks that share weight rows are neighbours in launch order,
// so all but one of them find those rows in the second-level cache
template <int MT, int KS>
__global__ void __launch_bounds__(LF_WARPS * 32, MT <= 4 ? 3 : 2) linear_f32_stream_kernel(
    const float* __restrict__ x, const float* __restrict__ w, float* __restrict__ y, int M, int N, int K) {
    pdl_invite();
    const int m0 = blockIdx.x * MT;
    x += static_cast<size_t>(m0) * K;
    y += static_cast<size_t>(m0) * N;
    M = min(M - m0, MT);
    constexpr int V = LF_ROWS * MT;                     // sums a warp makes
    __shared__ float red[KS > 1 ? LF_WARPS * V : 1];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int group = warp / KS, slice = warp % KS;
    const int n0 = (blockIdx.y * (LF_WARPS / KS) + group) * LF_ROWS;
    const int k4 = K >> 2;
    constexpr int STEP = 32 * KS;                       // in units of four k-values
    const float* wr[LF_ROWS];
#pragma unroll
    for (int r = 0; r < LF_ROWS; ++r) wr[r] = w + static_cast<size_t>(min(n0 + r, N - 1)) * K;
    float acc[LF_ROWS][MT];
#pragma unroll
    for (int r = 0; r < LF_ROWS; ++r)
#pragma unroll
        for (int m = 0; m < MT; ++m) acc[r][m] = 0.0f;
    const float4 zero = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    auto fetch = [&](float4 (&b)[LF_ROWS], int c) {
#pragma unroll
        for (int r = 0; r < LF_ROWS; ++r) b[r] = c < k4 ? lf_stream(wr[r] + 4 * c) : zero;
    };
    int c = slice * 32 + lane;
    float4 b0[LF_ROWS], b1[LF_ROWS];
    pdl_wait();                                         // before the weights too: the kernel in front may have made them
    fetch(b0, c);
    fetch(b1, c + STEP);
    auto multiply = [&](const float4 (&b)[LF_ROWS], int at) {
        const float* xp = x + 4 * at;
#pragma unroll
        for (int m = 0; m < MT; ++m) {
            float4 a = *reinterpret_cast<const float4*>(xp + static_cast<size_t>(min(m, M - 1)) * K);
#pragma unroll
            for (int r = 0; r < LF_ROWS; ++r) {
                acc[r][m] = fmaf(a.x, b[r].x, acc[r][m]);
                acc[r][m] = fmaf(a.y, b[r].y, acc[r][m]);
                acc[r][m] = fmaf(a.z, b[r].z, acc[r][m]);
                acc[r][m] = fmaf(a.w, b[r].w, acc[r][m]);
            }
        }
    };
    while (c < k4) {                                    // a lane past the end stops: 0 x infinity must not join its sums
        multiply(b0, c);
        fetch(b0, c + 2 * STEP);
        if (c + STEP < k4) {
            multiply(b1, c + STEP);
            fetch(b1, c + 3 * STEP);
        }
        c += 2 * STEP;
    }
    __syncwarp();
    // the lanes' sums: halves exchanged until a lane holds one total (value `lane` of 32), the rest by plain exchanges
    float* v = &acc[0][0];
    constexpr int SETS = V > 32 ? V / 32 : 1, SV = V > 32 ? 32 : V;
    float total[SETS];
#pragma unroll
    for (int s = 0; s < SETS; ++s) {
        float t[SV];
#pragma unroll
        for (int i = 0; i < SV; ++i) t[i] = v[s * SV + i];
        int n = SV;
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            if (n > 1) {
                n >>= 1;
#pragma unroll
                for (int i = 0; i < SV / 2; ++i)
                    if (i < n) {
                        const bool up = (lane & off) != 0;
                        const float send = up ? t[i] : t[i + n], keep = up ? t[i + n] : t[i];
                        t[i] = keep + __shfl_xor_sync(0xffffffffu, send, off);
                    }
            } else {
                t[0] += __shfl_xor_sync(0xffffffffu, t[0], off);
            }
        }
        total[s] = t[0];
    }
    constexpr int SHIFT = SV == 32 ? 0 : SV == 16 ? 1 : SV == 8 ? 2 : 3;      // lanes that hold the same total: 1 << SHIFT
    const int held = lane >> SHIFT;
    const bool first = (lane & ((1 << SHIFT) - 1)) == 0;
    if (KS > 1) {
#pragma unroll
        for (int s = 0; s < SETS; ++s)
            if (first) red[warp * V + s * SV + held] = total[s];
        __syncthreads();
        if (slice != 0) return;
#pragma unroll
        for (int s = 0; s < SETS; ++s) {
            float t = 0.0f;
#pragma unroll
            for (int k = 0; k < KS; ++k) t += red[(warp + k) * V + s * SV + held];
            total[s] = t;
        }
    }
#pragma unroll
    for (int s = 0; s < SETS; ++s) {
        const int i = s * SV + held, r = i / MT, m = i % MT;
        if (first && m < M && n0 + r < N) y[static_cast<size_t>(m) * N + n0 + r] = total[s];
    }
}

// The share of the block slots' time that a grid with `ks` slices keeps busy: blocks over whole waves of resident blocks.
// Measured at 8 rows (us for 1, 2, 4, 8 slices): 4096 x 4096: 24.6 15.6 17.2 18.1, 6144 x 4096: 25.7 28.4 23.6 24.4,
// 32768 x 4096: 98 93 96 106, 152000 x 1024: 111 122 153 224; the fill picks 2, 4, 2 and 1.
static double lf_fill(long long groups, long long tokens, int ks, int mt) {
    const long long per = LF_WARPS / ks, blocks = (groups + per - 1) / per * tokens, slots = 148LL * (mt <= 4 ? 3 : 2);
    return static_cast<double>(blocks) / static_cast<double>((blocks + slots - 1) / slots * slots);
}

// x: float32 [M, K]; w: float32 [N, K]; y: float32 [M, N].  K a multiple of 4.
extern "C" int llm_linear_f32(const float* x, const float* w, float* y, int M, int N, int K, uintptr_t stream) {
    if (M <= 0 || N <= 0) return LLM_OK;
    if (K <= 0 || (K & 3)) return LLM_REFUSED_SIZE;
    if (!aligned16(x) || !aligned16(w)) return LLM_REFUSED_ALIGN;
    const int mt = M == 1 ? 1 : M == 2 ? 2 : M <= 4 ? 4 : 8;
    const int groups = (N + LF_ROWS - 1) / LF_ROWS, tokens = (M + mt - 1) / mt;
    double best = 0.0;                                  // the fewest slices that fill the last wave about as well as any
    for (int c = 1; c <= 8; c *= 2) best = lf_fill(groups, tokens, c, mt) > best ? lf_fill(groups, tokens, c, mt) : best;
    int ks = 1;
    while (ks < 8 && lf_fill(groups, tokens, ks, mt) < best - 0.07) ks *= 2;
    while (ks > 1 && groups / (LF_WARPS / ks) >= 65535) ks /= 2;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    const int per_block = LF_WARPS / ks;
    const int row_blocks = (groups + per_block - 1) / per_block;
    if (row_blocks > 65535) return LLM_REFUSED_SIZE;
    const dim3 grid(tokens, row_blocks), block(LF_WARPS * 32);
#define GO(MT, KS) launch_pdl((linear_f32_stream_kernel<MT, KS>), grid, block, 0, s, x, w, y, M, N, K)
#define GO_M(MT)                                                                                     \
    { if (ks == 1) GO(MT, 1); else if (ks == 2) GO(MT, 2); else if (ks == 4) GO(MT, 4); else GO(MT, 8); }
    if (mt == 1) GO_M(1)
    else if (mt == 2) GO_M(2)
    else if (mt == 4) GO_M(4)
    else GO_M(8)
#undef GO_M
#undef GO
    return launch_status();
}
