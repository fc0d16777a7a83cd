// The gated delta rule with a decay per key channel: per head a state S [D, V] that every token decays row by
// row, corrects towards its value and reads,
//
//     S <- diag(g_t) S        u = beta_t (v_t - S^T k_t)        S <- S + k_t u^T        o_t = S^T q_t
//
// with q and k unit vectors per head (q times D^-1/2), q, k and v behind a short causal convolution over time and
// silu, beta = sigmoid of one projection per head, g = exp(-exp(A_h) softplus(z)) with z a low-rank projection plus
// a bias, and afterwards per head o / rms(o) * w * sigmoid(a low-rank gate).  The state, the decays, the step sizes,
// the unit norms and every product of the recurrence are 32-bit arithmetic: multiply-adds, or, for long portions of heads of 128,
// sums of bfloat16 products on the tensor cores that are as near (delta_scan_mma_kernel).
//
// The columns of S do not touch one another: column v needs k, q, g of the head and its own v_t.  So blocks take any
// number of columns of any head, and a long prompt of one request spreads over as many SMs as it has columns without
// being cut in time.  C columns (1, 2 or 4) are L lanes of a warp, each holding R = DP / L rows of all of them (rows
// 4 l + 4 L j .. + 3 of lane l), so that a vector read from shared memory serves C columns.  Along time eight tokens go
// together: a chunk's chain of loads, products, exchanges and dependent u is what a long portion waits for (2,048 tokens
// of one request, 16 heads of 128 x 128, 361 us with four tokens a chunk, 272 with eight).  With p_i the product of the
// decays of the chunk's tokens up
// to i, s_j that of the tokens behind j, and S the state that enters the chunk,
//
//     r_i = S^T (p_i k_i)     x_i = S^T (p_i q_i)                            sixteen products with S, one exchange of sums
//     u_i = beta_i (v_i - r_i - sum_{j<i} A_ij u_j)                           A_ij = sum_d k_i k_j (decays from j to i)
//     o_i = x_i + sum_{j<=i} B_ij u_j                                         B_ij = sum_d q_i k_j (decays from j to i)
//     S  <- p_7 S + sum_j (s_j k_j) u_j
//
// which is the recurrence with its sums regrouped: every factor is a product of decays, none is divided by one.  The
// vectors p k, p q, s k and the numbers A, B are the same for all columns of a head.
//
//   delta_prepare_kernel   (or ..._fours_kernel) a warp per (four tokens, head of q, k or v): convolution, silu, unit norm of q and k; beta
//   delta_lowrank_kernel   the second halves of both low-rank projections: decays and gates (delta_lowrank_mma_kernel: bfloat16
//                          weights and ranks above 32, on the tensor cores)
//   delta_chunk_kernel     a warp per (eight tokens, head): p k, p q, s k, p_7, A and B
//   delta_scan_kernel      one block per (entry, head, columns): the recurrence over the entry's tokens, staged sixteen
//                          at a time with cp.async into two buffers; o in 32-bit; keeps the convolutions' last inputs
//                          (delta_batch_kernel and delta_scan_mma_kernel take the places of these two for long portions)
//   delta_output_kernel    a warp per (token, head): norm, weight, gate, scale, store in the compute dtype
//   delta_step_kernel      all of it for entries of ONE token (decode steps): one block per (entry, head) copies the head's
//                          state and its slice of the low-rank weights into shared memory before it waits for the kernel
//                          in front of it, makes q, k, v, decays and gates, and writes the new state as it goes
//
// Per request slot the mixer keeps one row of floats: S of every head transposed, [H][V][DP] (DP = D rounded up to
// 32, 64, 128 or 256; rows from D on stay zero), then a ring of `taps` rows of the C = 2 G D + H V convolved
// projections; the row of the token at position p sits at ring row p mod taps.  A token reads the rows of positions
// p - 1 .. p - taps + 1 and writes row p mod taps, which is none of those, so in a decode step blocks that share a
// key head may read the ring while one of them writes it.
#include "common.cuh"
#include "split_mma.cuh"
#include "tcgen05_attention.cuh"

#define DR_TB 16            // tokens staged at a time
#define DR_CHUNK 8          // tokens that go through the state together
#define DR_LANES 8          // lanes a column of the state is spread over in the decode kernel

__device__ __forceinline__ void dr_cp16(float* smem_dst, const float* src) {
    const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(smem_dst));
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src));
}

__device__ __forceinline__ void dr_prefetch(const void* p) { asm volatile("prefetch.global.L2 [%0];\n" ::"l"(p)); }

__device__ __forceinline__ float dr_silu(float x) { return __fdividef(x, 1.0f + expf(-x)); }
__device__ __forceinline__ float dr_sigmoid(float x) { return __fdividef(1.0f, 1.0f + expf(-x)); }
// ln(1 + e^x); rounding 1 + e to a float costs at most half a unit in the last place of a decay
__device__ __forceinline__ float dr_softplus(float x) { return fmaxf(x, 0.0f) + logf(1.0f + expf(-fabsf(x))); }
// the decay of one key channel: exp(-exp(A) softplus(z)); `ea` is exp(A)
__device__ __forceinline__ float dr_decay(float z, float ea) { return expf(-ea * dr_softplus(z)); }

// What the kernels know of a head's shape and of where things are.
struct DeltaShape {
    int H, G, D, V, DP, VP, taps;
    int q_off, k_off, v_off, b_off, a_off, ra, g_off, rg;      // columns of the projection; ranks of decay and gate
    long long stride;                                          // of the projection's rows
    long long slot_stride, ring_off;                           // floats of a slot; where its ring starts
};

// The convolved value of channel c (an index into q | k | v side by side, as they stand in the projection's columns
// from q_off on) for the token in batch row t: the rows of this step, then the request's ring, zeros before the start.
__device__ __forceinline__ float dr_conv(const DeltaShape& s, const float* __restrict__ proj, const float* __restrict__ w,
                                         const float* __restrict__ ring, long long t, long long row0, int pos, int c) {
    const int C = 2 * s.G * s.D + s.H * s.V;
    float acc = 0.0f;
    for (int j = 0; j < s.taps; ++j) {                          // oldest first
        const int back = s.taps - 1 - j;
        float x = 0.0f;
        if (t - back >= row0) x = proj[(t - back) * s.stride + s.q_off + c];
        else if (pos - back >= 0) x = ring[static_cast<long long>((pos - back) % s.taps) * C + c];
        acc += w[static_cast<size_t>(c) * s.taps + j] * x;
    }
    return acc;
}

#define DP_WARPS 8
#define DP_TOKENS 4
// grid: (ceil(tokens / DP_TOKENS), ceil((2 G + H) / DP_WARPS)): a warp takes four tokens of one head of q, k or v.  PER:
// channels a lane holds at a time (q and k need a whole head at once, v is taken 32 PER channels at a time).
template <int PER>
__global__ void delta_prepare_kernel(const DeltaShape s, const float* __restrict__ proj, const float* __restrict__ conv_w,
                                     const float* __restrict__ state, const int32_t* __restrict__ positions,
                                     const int32_t* __restrict__ token_entry, const int32_t* __restrict__ entry_slot,
                                     const int32_t* __restrict__ entry_q_start, float* __restrict__ qn, float* __restrict__ kn,
                                     float* __restrict__ vn, float* __restrict__ beta, int num_tokens) {
    pdl_begin();
    const int t0 = blockIdx.x * DP_TOKENS, nt = min(DP_TOKENS, num_tokens - t0);
    const int item = blockIdx.y * DP_WARPS + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (item >= 2 * s.G + s.H) return;
    const bool is_v = item >= 2 * s.G, is_q = item < s.G;
    const int head = is_v ? item - 2 * s.G : is_q ? item : item - s.G;
    const int width = is_v ? s.V : s.D, padded = is_v ? s.VP : s.DP;
    const int ch0 = is_v ? 2 * s.G * s.D + head * s.V : item * s.D;        // the head's first channel in q | k | v
    float* dst = (is_v ? vn : is_q ? qn : kn) + (static_cast<size_t>(t0) * (is_v ? s.H : s.G) + head) * padded;
    const int dst_stride = (is_v ? s.H : s.G) * padded;
    const int e0 = token_entry[t0], e3 = token_entry[t0 + nt - 1];
    // four tokens of one portion with three more of it in front of them: every input is a row of this step
    const bool plain = s.taps <= 4 && nt == DP_TOKENS && e0 == e3 && t0 - 3 >= entry_q_start[e0];
    for (int c0 = 0; c0 < padded; c0 += 32 * PER) {
        float y[DP_TOKENS][PER];
        if (plain) {
            const float* pr = proj + static_cast<long long>(t0 - 3) * s.stride + s.q_off + ch0 + c0 + lane;
#pragma unroll
            for (int i = 0; i < PER; ++i) {
                const int c = c0 + lane + 32 * i;
                if (c < width) {
                    const float* w = conv_w + static_cast<size_t>(ch0 + c) * s.taps + s.taps - 1;      // the last tap
                    const float w3 = w[0], w2 = s.taps > 1 ? w[-1] : 0.0f, w1 = s.taps > 2 ? w[-2] : 0.0f, w0 = s.taps > 3 ? w[-3] : 0.0f;
                    float x[DP_TOKENS + 3];
#pragma unroll
                    for (int j = 0; j < DP_TOKENS + 3; ++j) x[j] = pr[j * s.stride + 32 * i];
#pragma unroll
                    for (int j = 0; j < DP_TOKENS; ++j) y[j][i] = dr_silu(w0 * x[j] + w1 * x[j + 1] + w2 * x[j + 2] + w3 * x[j + 3]);
                } else {
#pragma unroll
                    for (int j = 0; j < DP_TOKENS; ++j) y[j][i] = 0.0f;
                }
            }
        } else {
#pragma unroll
            for (int j = 0; j < DP_TOKENS; ++j) {
                const int t = min(t0 + j, num_tokens - 1), e = token_entry[t];
                const float* ring = state + entry_slot[e] * s.slot_stride + s.ring_off;
#pragma unroll
                for (int i = 0; i < PER; ++i) {
                    const int c = c0 + lane + 32 * i;
                    y[j][i] = c < width ? dr_silu(dr_conv(s, proj, conv_w, ring, t, entry_q_start[e], positions[t], ch0 + c)) : 0.0f;
                }
            }
        }
        if (!is_v) {                               // unit vectors; q also times D^-1/2 (the whole head is here: D <= 32 PER)
            float n[DP_TOKENS];
#pragma unroll
            for (int j = 0; j < DP_TOKENS; ++j) {
                n[j] = 0.0f;
#pragma unroll
                for (int i = 0; i < PER; ++i) n[j] += y[j][i] * y[j][i];
            }
#pragma unroll
            for (int m = 16; m > 0; m >>= 1)
#pragma unroll
                for (int j = 0; j < DP_TOKENS; ++j) n[j] += __shfl_xor_sync(0xffffffffu, n[j], m);
#pragma unroll
            for (int j = 0; j < DP_TOKENS; ++j) {
                const float inv = 1.0f / sqrtf((n[j] + 1e-6f) * (is_q ? static_cast<float>(s.D) : 1.0f));
#pragma unroll
                for (int i = 0; i < PER; ++i) y[j][i] *= inv;
            }
        }
#pragma unroll
        for (int j = 0; j < DP_TOKENS; ++j)
#pragma unroll
            for (int i = 0; i < PER; ++i) {
                const int c = c0 + lane + 32 * i;
                if (j < nt && c < padded) dst[j * dst_stride + c] = y[j][i];      // behind a head's end: zeros
            }
    }
    if (is_v && lane < nt) beta[static_cast<size_t>(t0 + lane) * s.H + head] = dr_sigmoid(proj[(t0 + lane) * s.stride + s.b_off + head]);
}

// The same for heads of up to 128 channels, up to four taps and rows that can be read sixteen bytes at a time.  A lane takes four
// neighbouring channels, and all it reads (seven rows, the taps) is on its way before the first use: the kernel above waits for
// its loads four times in a row, and a block at a portion's start reads the ring or zeros one value after another.  Here rows come from
// wherever they are: a block whose tokens belong to several portions passes once for each.
// Latency bounds it (a warp has seven rows to wait for; three blocks of 80 registers an SM).  1,700 tokens of three portions, 16 heads of
// 128, everything cold: 43 -> 33 us; layers with eight tokens a chunk: 2 x 1,000 tokens 402 -> 392, 4 x 500 363 -> 354, 4 x 260 215 -> 205, 8 heads
// 2 x 1,000 248 -> 235, 8 x 1,000 621 -> 605, 9 x 900 594 -> 578.  Two blocks of 96 registers 38; four 38; rows fetched before the portion is known 37 (spills).
__global__ void __launch_bounds__(DP_WARPS * 32, 3) delta_prepare_fours_kernel(
    const DeltaShape s, const float* __restrict__ proj, const float* __restrict__ conv_w, const float* __restrict__ state,
    const int32_t* __restrict__ positions, const int32_t* __restrict__ token_entry, const int32_t* __restrict__ entry_slot,
    const int32_t* __restrict__ entry_q_start, float* __restrict__ qn, float* __restrict__ kn, float* __restrict__ vn,
    float* __restrict__ beta, int num_tokens) {
    pdl_begin();
    const int t0 = blockIdx.x * DP_TOKENS, nt = min(DP_TOKENS, num_tokens - t0);
    const int item = blockIdx.y * DP_WARPS + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (item >= 2 * s.G + s.H) return;
    const bool is_v = item >= 2 * s.G, is_q = item < s.G;
    const int head = is_v ? item - 2 * s.G : is_q ? item : item - s.G;
    const int width = is_v ? s.V : s.D, padded = is_v ? s.VP : s.DP;
    const int ch0 = is_v ? 2 * s.G * s.D + head * s.V : item * s.D;        // the head's first channel in q | k | v
    const int C = 2 * s.G * s.D + s.H * s.V;
    float* dst = (is_v ? vn : is_q ? qn : kn) + (static_cast<size_t>(t0) * (is_v ? s.H : s.G) + head) * padded;
    const int dst_stride = (is_v ? s.H : s.G) * padded;
    int last;
    for (int first = 0; first < nt; first = last) {                         // the block's tokens of one portion
        const int e = token_entry[t0 + first], begin = entry_q_start[e];
        for (last = first + 1; last < nt && token_entry[t0 + last] == e;) ++last;
        const bool within = begin <= t0 - 3 && nt == DP_TOKENS;             // every row is one of this step
        const int pos0 = within ? 0 : positions[t0 + first] - first - 3;    // the position of row 0, if it is the portion's
        const float* ring = within ? nullptr : state + entry_slot[e] * s.slot_stride + s.ring_off;
        for (int c0 = 0; c0 < padded; c0 += 128) {
            const int c = c0 + 4 * lane, cc = ch0 + min(c, width - 4);      // lanes behind the head's end read its last channels
            const float4 zero = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            float4 x[DP_TOKENS + 3], w[4];
#pragma unroll
            for (int j = 0; j < DP_TOKENS + 3; ++j) {
                const int t = t0 - 3 + j;
                if (within || (t >= begin && t < t0 + nt))
                    x[j] = *reinterpret_cast<const float4*>(proj + t * s.stride + s.q_off + cc);
                else if (j >= 4 - s.taps && t < begin && pos0 + j >= 0)
                    x[j] = *reinterpret_cast<const float4*>(ring + static_cast<long long>((pos0 + j) % s.taps) * C + cc);
                else
                    x[j] = zero;
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float* tap = conv_w + static_cast<size_t>(cc + i) * s.taps;
                if (s.taps == 4) w[i] = *reinterpret_cast<const float4*>(tap);
                else w[i] = make_float4(0.0f, s.taps > 2 ? tap[s.taps - 3] : 0.0f, s.taps > 1 ? tap[s.taps - 2] : 0.0f, tap[s.taps - 1]);
            }
            float y[DP_TOKENS][4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                auto part = [&](int j) { return i == 0 ? x[j].x : i == 1 ? x[j].y : i == 2 ? x[j].z : x[j].w; };
#pragma unroll
                for (int j = 0; j < DP_TOKENS; ++j) {
                    float acc = 0.0f;               // only taps there are: none times a row that is not finite
                    if (s.taps > 3) acc = w[i].x * part(j);
                    if (s.taps > 2) acc = fmaf(w[i].y, part(j + 1), acc);
                    if (s.taps > 1) acc = fmaf(w[i].z, part(j + 2), acc);
                    y[j][i] = c < width ? dr_silu(fmaf(w[i].w, part(j + 3), acc)) : 0.0f;
                }
            }
            if (!is_v) {                            // unit vectors; q also times D^-1/2 (the whole head is here)
                float n[DP_TOKENS];
#pragma unroll
                for (int j = 0; j < DP_TOKENS; ++j) n[j] = y[j][0] * y[j][0] + y[j][1] * y[j][1] + y[j][2] * y[j][2] + y[j][3] * y[j][3];
#pragma unroll
                for (int m = 16; m > 0; m >>= 1)
#pragma unroll
                    for (int j = 0; j < DP_TOKENS; ++j) n[j] += __shfl_xor_sync(0xffffffffu, n[j], m);
#pragma unroll
                for (int j = 0; j < DP_TOKENS; ++j) {
                    const float inv = 1.0f / sqrtf((n[j] + 1e-6f) * (is_q ? static_cast<float>(s.D) : 1.0f));
#pragma unroll
                    for (int i = 0; i < 4; ++i) y[j][i] *= inv;
                }
            }
#pragma unroll
            for (int j = 0; j < DP_TOKENS; ++j)
                if (j >= first && j < last && c < padded)                   // behind a head's end: zeros
                    *reinterpret_cast<float4*>(dst + j * dst_stride + c) = make_float4(y[j][0], y[j][1], y[j][2], y[j][3]);
        }
    }
    if (is_v && lane < nt) beta[static_cast<size_t>(t0 + lane) * s.H + head] = dr_sigmoid(proj[(t0 + lane) * s.stride + s.b_off + head]);
}

// Second halves of the low-rank projections.  A block takes DL_TOKENS tokens and DL_CHANNELS channels (two a thread) of
// either the decays or the gates; the tokens' first halves sit in shared memory as [rank][tokens], so that a thread
// reads four tokens' values at a time and each weight serves all of the block's tokens.  Weights are transposed,
// [rank][channels].
#define DL_TOKENS 16
#define DL_PITCH 20               // floats from rank to rank in shared memory
#define DL_THREADS 128
#define DL_CHANNELS (2 * DL_THREADS)
template <typename TW>
__global__ void __launch_bounds__(DL_THREADS) delta_lowrank_kernel(
    const DeltaShape s, const float* __restrict__ proj, const TW* __restrict__ wa, const float* __restrict__ dt_bias,
    const float* __restrict__ a_log, const TW* __restrict__ wg, float* __restrict__ decay, float* __restrict__ gate, int num_tokens,
    int decay_blocks) {
    pdl_begin();
    extern __shared__ __align__(16) float a[];
    const bool is_decay = static_cast<int>(blockIdx.y) < decay_blocks;
    const int rank = is_decay ? s.ra : s.rg, off = is_decay ? s.a_off : s.g_off;
    const int channels = is_decay ? s.H * s.D : s.H * s.V;
    const TW* w = is_decay ? wa : wg;
    const int t0 = blockIdx.x * DL_TOKENS;
    const int nt = min(DL_TOKENS, num_tokens - t0);
    for (int idx = threadIdx.x; idx < DL_TOKENS * rank; idx += blockDim.x) {
        const int t = idx / rank, j = idx - t * rank;
        a[j * DL_PITCH + t] = t < nt ? proj[static_cast<size_t>(t0 + t) * s.stride + off + j] : 0.0f;
    }
    __syncthreads();
    const int c0 = (is_decay ? blockIdx.y : blockIdx.y - decay_blocks) * DL_CHANNELS + threadIdx.x;
    const bool there[2] = {c0 < channels, c0 + DL_THREADS < channels};
    if (!there[0]) return;
    float z[2][DL_TOKENS];
#pragma unroll
    for (int n = 0; n < 2; ++n) {
        const float bias = is_decay && there[n] ? dt_bias[c0 + n * DL_THREADS] : 0.0f;
#pragma unroll
        for (int t = 0; t < DL_TOKENS; ++t) z[n][t] = bias;
    }
    for (int j0 = 0; j0 < rank; j0 += 4) {                      // eight weights in flight
        float wv[2][4];
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
            for (int u = 0; u < 4; ++u)
                wv[n][u] = j0 + u < rank && there[n] ? to_f32(w[static_cast<size_t>(j0 + u) * channels + c0 + n * DL_THREADS]) : 0.0f;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const float4* ar = reinterpret_cast<const float4*>(a + min(j0 + u, rank - 1) * DL_PITCH);
#pragma unroll
            for (int t = 0; t < DL_TOKENS; t += 4) {
                const float4 v = ar[t >> 2];
#pragma unroll
                for (int n = 0; n < 2; ++n) {
                    z[n][t] += wv[n][u] * v.x;
                    z[n][t + 1] += wv[n][u] * v.y;
                    z[n][t + 2] += wv[n][u] * v.z;
                    z[n][t + 3] += wv[n][u] * v.w;
                }
            }
        }
    }
#pragma unroll
    for (int n = 0; n < 2; ++n) {
        if (!there[n]) continue;
        const int c = c0 + n * DL_THREADS;
        if (is_decay) {
            const int h = c / s.D, d = c - h * s.D;
            const float ea = expf(a_log[h]);
#pragma unroll
            for (int t = 0; t < DL_TOKENS; ++t)
                if (t < nt) decay[(static_cast<size_t>(t0 + t) * s.H + h) * s.DP + d] = dr_decay(z[n][t], ea);
        } else {
#pragma unroll
            for (int t = 0; t < DL_TOKENS; ++t)
                if (t < nt) gate[static_cast<size_t>(t0 + t) * channels + c] = dr_sigmoid(z[n][t]);
        }
    }
}

// The same for prompt portions with bfloat16 weights, on the tensor cores.  A float32 input is exactly the sum of three
// bfloat16 values (each the next eight bits of its significand), and its product with a bfloat16 weight is exact, so three
// products with 32-bit sums take the place of one 32-bit product.  The tensor cores cut what they add: each sixteen ranks
// are therefore summed from zero, smallest values first, and added, rounded, to the running sums.  What bounded the kernel
// above is its multiply-adds and the loads that feed them (one weight a lane for sixteen).  A block makes 64 tokens x 128 channels, a warp 32 x 32.
// 1,700 tokens, rank 64, 4,096 channels: 62.7 -> 33.7 us (blocks of 10 us, two an SM: waiting for the inputs, splitting them and
// the exponentials follow one another).  Error of a gate against 64 bits (root mean square, relative): 6.0e-8 -> 4.6e-8, at
// rank 200 1.2e-7 -> 5.5e-8.
#define DM_TOKENS 64
#define DM_CHANNELS 128
#define DM_RANKS 64               // at a time in shared memory
#define DM_XP (DM_RANKS + 8)      // pitches: an odd number of 16-byte chunks
#define DM_WP (DM_CHANNELS + 8)
__global__ void __launch_bounds__(256, 2) delta_lowrank_mma_kernel(
    const DeltaShape s, const float* __restrict__ proj, const bf16* __restrict__ wa, const float* __restrict__ dt_bias,
    const float* __restrict__ a_log, const bf16* __restrict__ wg, float* __restrict__ decay, float* __restrict__ gate, int num_tokens,
    int decay_blocks) {
    __shared__ __align__(16) bf16 xs[3][DM_TOKENS][DM_XP];
    __shared__ __align__(16) bf16 ws[DM_RANKS][DM_WP];
    pdl_begin();
    const bool is_decay = static_cast<int>(blockIdx.y) < decay_blocks;
    const int rank = is_decay ? s.ra : s.rg, off = is_decay ? s.a_off : s.g_off;
    const int width = is_decay ? s.D : s.V, channels = s.H * width;
    const bf16* w = is_decay ? wa : wg;
    const int t0 = blockIdx.x * DM_TOKENS, nt = min(DM_TOKENS, num_tokens - t0);
    const int ch0 = (is_decay ? blockIdx.y : blockIdx.y - decay_blocks) * DM_CHANNELS;
    const int tid = threadIdx.x, lane = tid & 31, wt = (tid >> 5 & 1) * 32, wc = (tid >> 6) * 32;      // the warp's tokens, channels
    const bool wide = channels % 8 == 0 && (reinterpret_cast<uintptr_t>(w) & 15) == 0;
    float z[2][4][4];
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int n = 0; n < 4; ++n)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int c = ch0 + wc + 8 * n + 2 * (lane & 3) + (i & 1);
                z[m][n][i] = is_decay && c < channels ? dt_bias[c] : 0.0f;
            }
    for (int k0 = 0; k0 < rank; k0 += DM_RANKS) {
        if (k0) __syncthreads();
        if (wide) {
            for (int idx = tid; idx < DM_RANKS * (DM_CHANNELS / 8); idx += 256) {
                const int j = idx / (DM_CHANNELS / 8), c = idx % (DM_CHANNELS / 8) * 8;
                const bool there = k0 + j < rank && ch0 + c < channels;
                cp_async16(&ws[j][c], there ? w + static_cast<size_t>(k0 + j) * channels + ch0 + c : w, there);
            }
            cp_async_commit();
        } else {
            for (int idx = tid; idx < DM_RANKS * DM_CHANNELS; idx += 256) {
                const int j = idx / DM_CHANNELS, c = idx % DM_CHANNELS;
                ws[j][c] = k0 + j < rank && ch0 + c < channels ? w[static_cast<size_t>(k0 + j) * channels + ch0 + c] : from_f32<bf16>(0.0f);
            }
        }
        float x[DM_TOKENS / 8][2];                              // a warp's row a time, two ranks a lane: all loads at once
        const int j = 2 * lane;
#pragma unroll
        for (int i = 0; i < DM_TOKENS / 8; ++i) {
            const int t = (tid >> 5) + 8 * i;
            const float* row = proj + static_cast<size_t>(t0 + t) * s.stride + off + k0 + j;
            x[i][0] = t < nt && k0 + j < rank ? row[0] : 0.0f;
            x[i][1] = t < nt && k0 + j + 1 < rank ? row[1] : 0.0f;
        }
#pragma unroll
        for (int i = 0; i < DM_TOKENS / 8; ++i)
#pragma unroll
            for (int p = 0; p < 3; ++p) {
                unsigned bits[2];
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    bits[e] = x[i][e] == x[i][e] ? __float_as_uint(x[i][e]) & 0xffff0000u : 0x7fc00000u;
                    x[i][e] = (bits[e] & 0x7f800000u) == 0x7f800000u ? 0.0f : x[i][e] - __uint_as_float(bits[e]);      // nothing behind an infinity
                }
                *reinterpret_cast<unsigned*>(&xs[p][(tid >> 5) + 8 * i][j]) = bits[1] | bits[0] >> 16;
            }
        cp_async_wait_all();
        __syncthreads();
        const int steps = (min(DM_RANKS, rank - k0) + 15) / 16;
        for (int k = 0; k < steps; ++k) {
            unsigned b[2][4];
#pragma unroll
            for (int n = 0; n < 2; ++n) ldmatrix_x4_trans(b[n], &ws[16 * k + (lane & 15)][wc + 16 * n + (lane >> 4) * 8]);
#pragma unroll
            for (int m = 0; m < 2; ++m) {
                unsigned x[3][4];
#pragma unroll
                for (int p = 0; p < 3; ++p) ldmatrix_x4(x[p], &xs[p][wt + 16 * m + (lane & 15)][16 * k + (lane >> 4) * 8]);
#pragma unroll
                for (int n = 0; n < 4; ++n) {
                    float sum[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
                    for (int p = 2; p >= 0; --p) mma_bf16(sum, x[p], b[n >> 1][2 * (n & 1)], b[n >> 1][2 * (n & 1) + 1]);
#pragma unroll
                    for (int i = 0; i < 4; ++i) z[m][n][i] += sum[i];
                }
            }
        }
    }
#pragma unroll
    for (int n = 0; n < 4; ++n) {
        const int c = ch0 + wc + 8 * n + 2 * (lane & 3);
#pragma unroll
        for (int i = 0; i < 2; ++i) {                           // neighbouring channels: a quad's stores are one sector
            if (c + i >= channels) continue;
            const int h = (c + i) / width;
            const float ea = is_decay ? expf(a_log[h]) : 0.0f;
            float* dst = is_decay ? decay + static_cast<size_t>(h) * s.DP + (c + i - h * width) : gate + c + i;
            const size_t row = is_decay ? static_cast<size_t>(s.H) * s.DP : channels;
#pragma unroll
            for (int m = 0; m < 2; ++m)
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    const int t = wt + 16 * m + 8 * r + (lane >> 2);
                    const float v = z[m][n][2 * r + i];
                    if (t < nt) dst[(t0 + t) * row] = is_decay ? dr_decay(v, ea) : dr_sigmoid(v);
                }
        }
    }
}

// Sum over the eight lanes of a column.
__device__ __forceinline__ float dr_lane_sum(float v) {
    v += __shfl_xor_sync(0xffffffffu, v, 1);
    v += __shfl_xor_sync(0xffffffffu, v, 2);
    v += __shfl_xor_sync(0xffffffffu, v, 4);
    return v;
}

// One token against the R rows (R / 4 groups of four) that a lane holds of a column: decays S, returns o and writes.
template <int R>
__device__ __forceinline__ float dr_token(float (&S)[R], const float* __restrict__ k, const float* __restrict__ q,
                                          const float* __restrict__ g, int l, float v, float beta, float kq) {
    float4 kk[R / 4];
    float r0 = 0.0f, r1 = 0.0f, o0 = 0.0f, o1 = 0.0f;
#pragma unroll
    for (int j = 0; j < R / 4; ++j) {
        const float4 gg = *reinterpret_cast<const float4*>(g + 4 * l + 32 * j);
        const float4 qq = *reinterpret_cast<const float4*>(q + 4 * l + 32 * j);
        kk[j] = *reinterpret_cast<const float4*>(k + 4 * l + 32 * j);
        S[4 * j] *= gg.x;
        S[4 * j + 1] *= gg.y;
        S[4 * j + 2] *= gg.z;
        S[4 * j + 3] *= gg.w;
        r0 += S[4 * j] * kk[j].x;
        r1 += S[4 * j + 1] * kk[j].y;
        r0 += S[4 * j + 2] * kk[j].z;
        r1 += S[4 * j + 3] * kk[j].w;
        o0 += S[4 * j] * qq.x;
        o1 += S[4 * j + 1] * qq.y;
        o0 += S[4 * j + 2] * qq.z;
        o1 += S[4 * j + 3] * qq.w;
    }
    const float r = dr_lane_sum(r0 + r1), o = dr_lane_sum(o0 + o1);
    const float u = beta * (v - r);
#pragma unroll
    for (int j = 0; j < R / 4; ++j) {
        S[4 * j] += kk[j].x * u;
        S[4 * j + 1] += kk[j].y * u;
        S[4 * j + 2] += kk[j].z * u;
        S[4 * j + 3] += kk[j].w * u;
    }
    return o + kq * u;
}

// One level of a sum over lanes that also deals the values out: of N values each lane keeps the N / 2 that its bit
// `MASK` says, summed with its partner's.
template <int N, int MASK>
__device__ __forceinline__ void dr_deal(float* v, int lane) {
    const bool up = lane & MASK;
#pragma unroll
    for (int n = 0; n < N / 2; ++n) {
        const float send = up ? v[n] : v[n + N / 2], keep = up ? v[n + N / 2] : v[n];
        v[n] = keep + __shfl_xor_sync(0xffffffffu, send, MASK);
    }
}

// Sums of NV values over the L lanes of a group, left in sums[0 .. NV - 1] (in shared memory).
template <int NV, int L>
__device__ __forceinline__ void dr_sums(float (&v)[NV], int lane, int l, float* sums) {
    if constexpr (NV > 1 && L >= 2) dr_deal<NV, L / 2>(v, lane);
    if constexpr (NV > 2 && L >= 4) dr_deal<NV / 2, L / 4>(v, lane);
    if constexpr (NV > 4 && L >= 8) dr_deal<NV / 4, L / 8>(v, lane);
    if constexpr (NV > 8 && L >= 16) dr_deal<NV / 8, L / 16>(v, lane);
    if constexpr (NV > 16 && L >= 32) dr_deal<NV / 16, L / 32>(v, lane);
    constexpr int REST = NV >= L ? 1 : L / NV, K = NV >= L ? NV / L : 1;       // lanes that share a value; values a lane holds
#pragma unroll
    for (int m = REST / 2; m > 0; m >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], m);
    if (NV >= L || (l & (REST - 1)) == 0) {
#pragma unroll
        for (int n = 0; n < K; ++n) sums[(l / REST) * K + n] = v[n];
    }
}

#define DR_NUM (2 * DR_CHUNK * DR_CHUNK)      // numbers a chunk: A [8][8], zero from its diagonal on, then B [8][8], zero above it

// Where a chunk's shared vectors and numbers are: chunks start at every eighth row of an entry, so row / 8 + entry is a
// number of its own for each of them.
__device__ __forceinline__ long long dr_chunk_place(long long row, int entry) { return row / DR_CHUNK + entry; }

// What a chunk's eight tokens share over all columns of a head: a warp per (first token of a chunk, head); tokens that
// begin no chunk have no work.  pk = p k, pq = p q, and in place of the decays s k; total = p_7; num = A and B.
#define DC_WARPS 4
template <int DP>
__global__ void __launch_bounds__(DC_WARPS * 32) delta_chunk_kernel(
    const DeltaShape s, const float* __restrict__ qn, const float* __restrict__ kn, float* decay, float* __restrict__ pk,
    float* __restrict__ pq, float* __restrict__ total, float* __restrict__ num, const int32_t* __restrict__ token_entry,
    const int32_t* __restrict__ entry_q_start, const int32_t* __restrict__ entry_q_len, int num_tokens) {
    // no early invitation: the blocks of the scan behind this kernel would be dealt to whichever SMs have room while
    // this one drains, several to one SM, and the scan takes as long as its fullest SM
    pdl_wait();
    const long long t = blockIdx.x;
    const int h = blockIdx.y * DC_WARPS + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (h >= s.H) return;
    const int entry = token_entry[t];
    const long long row0 = entry_q_start[entry];
    if ((t - row0) % DR_CHUNK) return;
    const int nt = static_cast<int>(min(static_cast<long long>(DR_CHUNK), row0 + entry_q_len[entry] - t));
    const int kvh = h / (s.H / s.G);
    const size_t place = static_cast<size_t>(dr_chunk_place(t, entry)) * s.H + h;
    constexpr int CH = DR_CHUNK, NA = CH * (CH - 1) / 2;                    // A's pairs (i, j < i), then B's (i, j <= i)
    __shared__ float nums[DC_WARPS][DR_NUM];
    float* mine = nums[threadIdx.x >> 5];
    float acc[CH * CH];
#pragma unroll
    for (int n = 0; n < CH * CH; ++n) acc[n] = 0.0f;
    for (int x = lane * 4; x < DP; x += 128) {
        float kk[CH][4], qq[CH][4], gg[CH][4];
#pragma unroll
        for (int i = 0; i < CH; ++i) {
            float4 a = make_float4(0, 0, 0, 0), b = a, c = make_float4(1, 1, 1, 1);      // a missing token
            if (i < nt) {
                const size_t at = (static_cast<size_t>(t + i) * s.G + kvh) * DP + x;
                a = *reinterpret_cast<const float4*>(kn + at);
                b = *reinterpret_cast<const float4*>(qn + at);
                c = *reinterpret_cast<const float4*>(decay + (static_cast<size_t>(t + i) * s.H + h) * DP + x);
            }
            kk[i][0] = a.x; kk[i][1] = a.y; kk[i][2] = a.z; kk[i][3] = a.w;
            qq[i][0] = b.x; qq[i][1] = b.y; qq[i][2] = b.z; qq[i][3] = b.w;
            gg[i][0] = c.x; gg[i][1] = c.y; gg[i][2] = c.z; gg[i][3] = c.w;
        }
        float p[4] = {1.0f, 1.0f, 1.0f, 1.0f};
#pragma unroll
        for (int j = 0; j < CH; ++j) {
            float w[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                w[e] = kk[j][e];
                acc[NA + j * (j + 1) / 2 + j] += qq[j][e] * w[e];
#pragma unroll
                for (int i = j + 1; i < CH; ++i) {
                    w[e] *= gg[i][e];
                    acc[i * (i - 1) / 2 + j] += kk[i][e] * w[e];
                    acc[NA + i * (i + 1) / 2 + j] += qq[i][e] * w[e];
                }
                p[e] *= gg[j][e];
            }
            if (j < nt) {
                const size_t at = (static_cast<size_t>(t + j) * s.H + h) * DP + x;
                *reinterpret_cast<float4*>(pk + at) = make_float4(p[0] * kk[j][0], p[1] * kk[j][1], p[2] * kk[j][2], p[3] * kk[j][3]);
                *reinterpret_cast<float4*>(pq + at) = make_float4(p[0] * qq[j][0], p[1] * qq[j][1], p[2] * qq[j][2], p[3] * qq[j][3]);
                *reinterpret_cast<float4*>(decay + at) = make_float4(w[0], w[1], w[2], w[3]);
            }
        }
        *reinterpret_cast<float4*>(total + place * DP + x) = make_float4(p[0], p[1], p[2], p[3]);
    }
    dr_deal<64, 16>(acc, lane);
    dr_deal<32, 8>(acc, lane);
    dr_deal<16, 4>(acc, lane);
    dr_deal<8, 2>(acc, lane);
    dr_deal<4, 1>(acc, lane);                 // lane l holds values 2 l and 2 l + 1
    for (int n = lane; n < DR_NUM; n += 32) mine[n] = 0.0f;
    __syncwarp();
#pragma unroll
    for (int n = 0; n < 2; ++n) {
        const int v = 2 * lane + n;
        const bool is_a = v < NA;
        const int m = is_a ? v : v - NA;
        int i = is_a ? 1 : 0, at = 0;         // row i of the triangle starts at value `at` and has i (A) or i + 1 (B) of them
        while (at + (is_a ? i : i + 1) <= m) { at += is_a ? i : i + 1; ++i; }
        mine[(is_a ? 0 : CH * CH) + CH * i + (m - at)] = acc[n];
    }
    __syncwarp();
    float* out = num + place * DR_NUM;
    *reinterpret_cast<float4*>(out + 4 * lane) = *reinterpret_cast<const float4*>(mine + 4 * lane);
}

// C neighbouring floats from shared memory.
template <int C> __device__ __forceinline__ void dr_row(float (&v)[C], const float* p) {
    if constexpr (C == 4) {
        const float4 x = *reinterpret_cast<const float4*>(p);
        v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
    } else {
#pragma unroll
        for (int m = 0; m < C; ++m) v[m] = p[m];
    }
}

// The convolutions' inputs of a portion's last tokens go into the request's ring (the kernels before the scan have read it): by each
// block of a scan its columns' values, and the head's queries and keys by one.  THREADS: of the block, 0: as it was launched.
template <int THREADS>
__device__ __forceinline__ void dr_keep_inputs(const DeltaShape& s, const float* __restrict__ proj, float* slot, const int32_t* __restrict__ positions,
                                               long long row0, int count, int h, int c0, int cols, bool first) {
    const int channels = 2 * s.G * s.D + s.H * s.V, keep = min(count, s.taps - 1), kvh = h / (s.H / s.G);
    const auto threads = [] { if constexpr (THREADS > 0) return THREADS; else return blockDim.x; }();
    float* ring = slot + s.ring_off;
    const bool with_qk = first && h % (s.H / s.G) == 0;
    for (int i = 0; i < keep; ++i) {
        const long long t = row0 + count - keep + i;
        float* dst = ring + static_cast<long long>(positions[t] % s.taps) * channels;
        const float* src = proj + t * s.stride + s.q_off;
        if (with_qk)
            for (int d = threadIdx.x; d < s.D; d += threads) {
                dst[kvh * s.D + d] = src[kvh * s.D + d];
                dst[(s.G + kvh) * s.D + d] = src[(s.G + kvh) * s.D + d];
            }
        for (int x = threadIdx.x; x < cols && c0 + x < s.V; x += threads) {
            const int ch = 2 * s.G * s.D + h * s.V + c0 + x;
            dst[ch] = src[ch];
        }
    }
}

// grid: entries (longest portion first) x H x column tiles, the tiles fastest: WARPS warps a block, each 32 / L groups of C columns.
template <int DP, int C, int WARPS, int L>
__global__ void __launch_bounds__(WARPS * 32) delta_scan_kernel(
    const DeltaShape s, const float* __restrict__ proj, const float* __restrict__ pq, const float* __restrict__ pk,
    const float* __restrict__ vn, const float* __restrict__ beta, const float* __restrict__ sk, const float* __restrict__ total,
    const float* __restrict__ num, float* __restrict__ o, float* __restrict__ state, const int32_t* __restrict__ positions,
    const int32_t* __restrict__ entry_slot, const int32_t* __restrict__ entry_q_start, const int32_t* __restrict__ entry_q_len,
    int num_entries, int tiles) {
    pdl_begin();
    constexpr int R = DP / L, THREADS = WARPS * 32, CH = DR_CHUNK, CHUNKS = DR_TB / CH;
    constexpr int COLS = WARPS * (32 / L) * C, NV = 2 * CH * C;
    // a buffer: q, k, s k, v of a batch of tokens, then beta; then p_7 and the numbers of its chunks
    constexpr int BUF = DR_TB * (3 * DP + COLS + 1) + CHUNKS * (DP + DR_NUM);
    extern __shared__ __align__(16) float smem[];
    const int tid = threadIdx.x, lane = tid & 31, tile = blockIdx.x % tiles, c0 = tile * COLS;
    const int h = blockIdx.x / tiles % s.H;
    int entry = blockIdx.x / (tiles * s.H);
    if (num_entries <= 32) {                                    // longest portions first: the entry with `entry` ones before it
        const int mine = lane < num_entries ? entry_q_len[lane] : -1;
        int before = 0;
        for (int e = 0; e < num_entries; ++e) {
            const int len = __shfl_sync(0xffffffffu, mine, e);
            before += len > mine || (len == mine && e < lane);
        }
        entry = __ffs(__ballot_sync(0xffffffffu, before == entry && lane < num_entries)) - 1;
    }
    const int l = lane & (L - 1), group = tid / L, cb = group * C;          // the group's first column in the block
    float* sums = smem + 2 * BUF + group * NV;                  // [16][C]: the group's sums, by value and column
    const long long row0 = entry_q_start[entry];
    const int count = entry_q_len[entry];
    float* slot = state + entry_slot[entry] * s.slot_stride;
    float* col_state = slot + (static_cast<long long>(h) * s.V + c0 + cb) * DP + 4 * l;
    const int cols_here = s.V - c0 - cb;                        // columns of the group that exist, if fewer than C
    float S[C][R];
#pragma unroll
    for (int m = 0; m < C; ++m)
#pragma unroll
        for (int j = 0; j < R / 4; ++j) {
            const float4 x = m < cols_here ? *reinterpret_cast<const float4*>(col_state + m * DP + 4 * L * j) : make_float4(0, 0, 0, 0);
            S[m][4 * j] = x.x; S[m][4 * j + 1] = x.y; S[m][4 * j + 2] = x.z; S[m][4 * j + 3] = x.w;
        }
    const size_t first = (static_cast<size_t>(row0) * s.H + h) * DP;
    const int row_stride = s.H * DP;
    const size_t place = static_cast<size_t>(dr_chunk_place(row0, entry)) * s.H + h;
    auto stage = [&](int done, int buf) {
        constexpr int PIECES = DP / 4, STEP = THREADS / PIECES > 0 ? THREADS / PIECES : 1;
        const int nb = min(DR_TB, count - done);
        float* bq = smem + buf * BUF;
        float* bk = bq + DR_TB * DP;
        float* bs = bk + DR_TB * DP;
        float* bv = bs + DR_TB * DP;
        float* bb = bv + DR_TB * COLS;
        float* bt = bb + DR_TB;
        float* bn = bt + CHUNKS * DP;
        const size_t at = first + static_cast<size_t>(done) * row_stride;
        for (int x = (tid % PIECES) * 4; x < DP; x += THREADS * 4)
            for (int tok = tid / PIECES; tok < nb; tok += STEP) {
                const size_t from = at + static_cast<size_t>(tok) * row_stride + x;
                dr_cp16(bq + tok * DP + x, pq + from);
                dr_cp16(bk + tok * DP + x, pk + from);
                dr_cp16(bs + tok * DP + x, sk + from);
            }
        const int chunks = (nb + DR_CHUNK - 1) / DR_CHUNK;
        const size_t first_chunk = place + static_cast<size_t>(done / DR_CHUNK) * s.H;
        for (int idx = tid; idx < chunks * PIECES; idx += THREADS) {
            const int ch = idx / PIECES, x = (idx - ch * PIECES) * 4;
            dr_cp16(bt + ch * DP + x, total + (first_chunk + static_cast<size_t>(ch) * s.H) * DP + x);
        }
        for (int idx = tid; idx < chunks * (DR_NUM / 4); idx += THREADS) {
            const int ch = idx / (DR_NUM / 4), x = (idx - ch * (DR_NUM / 4)) * 4;
            dr_cp16(bn + ch * DR_NUM + x, num + (first_chunk + static_cast<size_t>(ch) * s.H) * DR_NUM + x);
        }
        for (int idx = tid; idx < nb * (COLS / 4); idx += THREADS) {
            const int tok = idx / (COLS / 4), x = (idx - tok * (COLS / 4)) * 4;
            if (c0 + x < s.VP) dr_cp16(bv + tok * COLS + x, vn + (static_cast<size_t>(row0 + done + tok) * s.H + h) * s.VP + c0 + x);
        }
        if (tid < nb) {
            const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(bb + tid));
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(d), "l"(beta + static_cast<size_t>(row0 + done + tid) * s.H + h));
        }
        for (int idx = nb * DP + tid; idx < chunks * DR_CHUNK * DP; idx += THREADS) bs[idx] = 0.0f;      // missing tokens write nothing
        asm volatile("cp.async.commit_group;\n" ::);
    };
    stage(0, 0);
    for (int done = 0, b = 0; done < count; done += DR_TB, ++b) {
        const int nb = min(DR_TB, count - done);
        if (done + DR_TB < count) {
            stage(done + DR_TB, (b + 1) & 1);
            asm volatile("cp.async.wait_group 1;\n" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        }
        __syncthreads();
        const float* bq = smem + (b & 1) * BUF;
        const float* bk = bq + DR_TB * DP;
        const float* bs = bk + DR_TB * DP;
        const float* bv = bs + DR_TB * DP;
        const float* bb = bv + DR_TB * COLS;
        const float* bt = bb + DR_TB;
        const float* bn = bt + CHUNKS * DP;
        const int chunks = (nb + DR_CHUNK - 1) / DR_CHUNK;
        for (int ch = 0; ch < chunks; ++ch) {
            const float* k = bk + ch * CH * DP + 4 * l;
            const float* q = bq + ch * CH * DP + 4 * l;
            const float* w = bs + ch * CH * DP + 4 * l;
            float v[NV];                      // value n of column m at n C + m: r_0 .. r_7, x_0 .. x_7
#pragma unroll
            for (int n = 0; n < NV; ++n) v[n] = 0.0f;
#pragma unroll
            for (int j = 0; j < R / 4; ++j)
#pragma unroll
                for (int i = 0; i < CH; ++i) {
                    const float4 a = *reinterpret_cast<const float4*>(k + i * DP + 4 * L * j);
                    const float4 e = *reinterpret_cast<const float4*>(q + i * DP + 4 * L * j);
#pragma unroll
                    for (int m = 0; m < C; ++m) {
                        v[i * C + m] += S[m][4 * j] * a.x;
                        v[(CH + i) * C + m] += S[m][4 * j] * e.x;
                        v[i * C + m] += S[m][4 * j + 1] * a.y;
                        v[(CH + i) * C + m] += S[m][4 * j + 1] * e.y;
                        v[i * C + m] += S[m][4 * j + 2] * a.z;
                        v[(CH + i) * C + m] += S[m][4 * j + 2] * e.z;
                        v[i * C + m] += S[m][4 * j + 3] * a.w;
                        v[(CH + i) * C + m] += S[m][4 * j + 3] * e.w;
                    }
                }
            dr_sums<NV, L>(v, lane, l, sums);
            __syncwarp();
            const float* nu = bn + ch * DR_NUM;
            const int left = nb - ch * CH;                     // tokens of the chunk; the missing ones write nothing
            float u[CH][C];
#pragma unroll
            for (int i = 0; i < CH; ++i) {
                const float be = bb[ch * CH + i];
                const float4 a0 = *reinterpret_cast<const float4*>(nu + CH * i), a1 = *reinterpret_cast<const float4*>(nu + CH * i + 4);
                const float a[CH] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
                float vt[C], r[C];
                dr_row<C>(vt, bv + (ch * CH + i) * COLS + cb);
                dr_row<C>(r, sums + i * C);
#pragma unroll
                for (int m = 0; m < C; ++m) {
                    float x = vt[m] - r[m];
#pragma unroll
                    for (int j = 0; j < i; ++j) x -= a[j] * u[j][m];
                    u[i][m] = i < left ? be * x : 0.0f;
                }
            }
#pragma unroll
            for (int n = l; n < CH * C; n += L) {               // token n / C of column n % C
                const int i = n / C, m = n % C;
                const float4 b0 = *reinterpret_cast<const float4*>(nu + CH * CH + CH * i), b1 = *reinterpret_cast<const float4*>(nu + CH * CH + CH * i + 4);
                const float bi[CH] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
                float out = sums[(CH + i) * C + m];
#pragma unroll
                for (int t = 0; t < CH; ++t) {
                    const float um = C == 1 ? u[t][0] : C == 2 ? ((m & 1) ? u[t][C - 1] : u[t][0])
                                            : (m & 2) ? ((m & 1) ? u[t][C - 1] : u[t][C >= 4 ? 2 : 0]) : ((m & 1) ? u[t][C >= 2 ? 1 : 0] : u[t][0]);
                    if (t <= i) out += bi[t] * um;              // a later token's u may be NaN, and zero times it too
                }
                if (i < left && m < cols_here)
                    o[(static_cast<size_t>(row0 + done + ch * CH + i) * s.H + h) * s.V + c0 + cb + m] = out;
            }
#pragma unroll
            for (int j = 0; j < R / 4; ++j) {
                const float4 p = *reinterpret_cast<const float4*>(bt + ch * DP + 4 * l + 4 * L * j);
#pragma unroll
                for (int m = 0; m < C; ++m) {
                    S[m][4 * j] *= p.x;
                    S[m][4 * j + 1] *= p.y;
                    S[m][4 * j + 2] *= p.z;
                    S[m][4 * j + 3] *= p.w;
                }
#pragma unroll
                for (int t = 0; t < CH; ++t) {
                    const float4 x = *reinterpret_cast<const float4*>(w + t * DP + 4 * L * j);
#pragma unroll
                    for (int m = 0; m < C; ++m) {
                        S[m][4 * j] += x.x * u[t][m];
                        S[m][4 * j + 1] += x.y * u[t][m];
                        S[m][4 * j + 2] += x.z * u[t][m];
                        S[m][4 * j + 3] += x.w * u[t][m];
                    }
                }
            }
            __syncwarp();                                       // `sums` is written again
        }
        __syncthreads();                      // this buffer is filled again two batches on
    }
#pragma unroll
    for (int m = 0; m < C; ++m)
        if (m < cols_here)
#pragma unroll
            for (int j = 0; j < R / 4; ++j)
                *reinterpret_cast<float4*>(col_state + m * DP + 4 * L * j) = make_float4(S[m][4 * j], S[m][4 * j + 1], S[m][4 * j + 2], S[m][4 * j + 3]);
    // The block's size as a constant moves the registers of the walk above (us, launch's size and constant): one column a warp 172 and
    // 181 (1,000 tokens, 4 heads); two 190 and 184 (8 heads); four 643 and 636 (2,500 tokens beside 16 single ones, 16 heads).
    dr_keep_inputs<C == 1 ? 0 : THREADS>(s, proj, slot, positions, row0, count, h, c0, COLS, tile == 0);
}

// ---- states of 128 rows on the tensor cores -------------------------------------------------------------------------
// The same recurrence, sixteen tokens at a time, as products: with X = V - (p k) S (tokens by columns),
//
//     U = T X       O = (p q) S + B U       S <- p_15 S + (s k)^T U              T = (1 + diag(beta) A)^-1 diag(beta)
//
// All factors are products of decays, none is divided by one, whatever the decays are: A and B are made of dot products whose
// decays from j to i are cut in the middle of the smallest of the batch's halves, quarters, eighths and pairs that holds both,
// what lies before the cut with k_j, what lies behind with k_i or q_i.  Products of float32 values are sums of six bfloat16 products
// (split_mma.cuh); the state stays in float32 accumulators, transposed, and takes a batch's contribution with rounded
// additions.
//
//   delta_batch_kernel   a block per (sixteen tokens, head): an image of what all columns of the head share, just as the scan
//                        wants it in shared memory: planes of p k, p q, s k, of T and B, then p_15 and the mark
//   delta_scan_mma_kernel  a block per (entry, head, 16 columns), four warps: 32 rows of the state each.  The
//                        shares of X and O over the rows go through shared memory; every warp then makes the U of its columns itself.
//
// A batch that holds something not finite or very large is marked with its first such token.  The scan makes what is before it as
// always, with nothing in the place of what follows (a weight of zero times an infinity is NaN), and then walks through the batch
// token by token for the outputs from the mark on and the state.
// What bounds it: a batch's chain, 1.5 us alone on an SM: 48 small products a warp over the state, shares and X, U, the state, the
// outputs of two warps and the waits in between.  With 32 columns and eight warps a block, two warps a scheduler, it was 2.2 us
// (3,700 clocks, 1,000 of them the products over the state, 600 the update, the tensor pipe busy for 40 %); blocks of 16 columns fetch
// the images twice as often and two of them share an SM without waiting for one another.  Portions of 284,
// 567 and 849 tokens, 16 heads of 128 x 128: the layer 335 -> 319 us; one portion of 1,000 and one of 1,000 tokens 419 -> 383; the
// kernels of eight tokens before (us): the scan 160, what it shares 24 (here 44: dot products and the writing of 76 MB).
// Error against 64 bits (2-norm, outputs and states) from the same unit norms, decays and step sizes: 7.7e-8 and 6.0e-8, the kernels of
// eight tokens 8.6e-8 and 7.9e-8.  With sums as the tensor cores cut them (split_mma_whole) and dot products in four chains it was
// 10.4e-8 and 8.6e-8, and the layer 320 us instead of 326.
#define DX_T 16
#define DX_PITCH 136                 // of a row of a plane: eight rows of 16 bytes fall into all banks
#define DX_PLANE (DX_T * DX_PITCH)
#define DX_NP 24                     // of a row of T or B
#define DX_NPLANE (DX_T * DX_NP)
#define DX_IMAGE (2 * (9 * DX_PLANE + 6 * DX_NPLANE) + 4 * 128 + 16)       // bytes
#define DX_MOST 1.0737418e9f         // 2^30
#define DX_LP 132                    // of a row of a level's vectors
#define DX_ROWS (4 * 4 * 24 * DX_LP) // bytes of the four levels' vectors
#define DX_BATCH_SMEM (DX_ROWS + 4 * (512 + 32))
#define DX_STATUS 11

// Where a batch's image is: batches start at every sixteenth row of an entry.
__device__ __forceinline__ long long dx_place(long long row, int entry) { return row / DX_T + entry; }

__global__ void __launch_bounds__(128) delta_batch_kernel(
    const DeltaShape s, const float* __restrict__ qn, const float* __restrict__ kn, const float* __restrict__ vn, const float* __restrict__ beta,
    const float* __restrict__ decay, unsigned char* __restrict__ images, const int32_t* __restrict__ entry_q_start,
    const int32_t* __restrict__ entry_q_len, int num_entries) {
    pdl_wait();                      // no early invitation: see delta_chunk_kernel
    constexpr int D = 128;
    const int h = blockIdx.y, tid = threadIdx.x, kvh = h / (s.H / s.G);
    int entry = -1, first = 0, nt = 0;                                      // the entry that has a batch in this place, if any
    for (int e0 = 0; e0 < num_entries && entry < 0; e0 += 32) {
        const int e = e0 + (tid & 31);
        int m = -1, left = 0;
        if (e < num_entries) {
            m = static_cast<int>(blockIdx.x) - static_cast<int>(dx_place(entry_q_start[e], e));
            left = entry_q_len[e] - DX_T * m;
        }
        const unsigned found = __ballot_sync(0xffffffffu, m >= 0 && left > 0);
        if (found) {
            const int at = __ffs(found) - 1;
            entry = e0 + at;
            first = __shfl_sync(0xffffffffu, m, at) * DX_T;
            nt = min(DX_T, __shfl_sync(0xffffffffu, left, at));
        }
    }
    if (entry < 0) return;
    const long long t = entry_q_start[entry] + first;
    extern __shared__ __align__(16) unsigned char dx_smem[];
    bf16* planes = reinterpret_cast<bf16*>(dx_smem);                        // [p k, p q, s k][3][16][136]
    bf16* small = planes + 9 * DX_PLANE;                                    // [T, B][3][16][24]
    float* total = reinterpret_cast<float*>(small + 6 * DX_NPLANE);         // [128], then the mark
    float* rows = reinterpret_cast<float*>(dx_smem);                        // before the planes: [4 levels][24][132], k_i, q_i, then k_j
    float* nums = reinterpret_cast<float*>(dx_smem + DX_ROWS);              // A [16][16], then B [16][16]
    float* shares = nums + 512;                                             // [4 warps][8 tokens]: q_i k_i
    __shared__ unsigned marks[4];
    // a thread: channels c and c + 1 of tokens 8 hf .. 8 hf + 7 (and the decays of all)
    const int c = 2 * (tid & 63), hf = tid >> 6, lane = tid & 31;
    {
        float2 k[8], q[8], g[DX_T];
        const float2 zero = make_float2(0.0f, 0.0f), one = make_float2(1.0f, 1.0f);
        const float* gp = decay + (static_cast<size_t>(t) * s.H + h) * D + c;
        const size_t at = (static_cast<size_t>(t + 8 * hf) * s.G + kvh) * D + c;
#pragma unroll
        for (int i = 0; i < DX_T; ++i) g[i] = i < nt ? *reinterpret_cast<const float2*>(gp + static_cast<size_t>(i) * s.H * D) : one;      // a missing token
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            k[i] = 8 * hf + i < nt ? *reinterpret_cast<const float2*>(kn + at + static_cast<size_t>(i) * s.G * D) : zero;
            q[i] = 8 * hf + i < nt ? *reinterpret_cast<const float2*>(qn + at + static_cast<size_t>(i) * s.G * D) : zero;
        }
        unsigned bad = 0;                                                   // tokens that are not finite or very large
        for (int x = 4 * lane; x < s.V; x += 128)                           // a warp four tokens' values
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int tok = 4 * (tid >> 5) + i;
                if (tok < nt) {
                    const float4 v = *reinterpret_cast<const float4*>(vn + (static_cast<size_t>(t + tok) * s.H + h) * s.VP + x);
                    if (!(fabsf(v.x) <= DX_MOST && fabsf(v.y) <= DX_MOST && fabsf(v.z) <= DX_MOST && fabsf(v.w) <= DX_MOST)) bad |= 1u << tok;
                }
            }
        if (tid < nt && !(fabsf(beta[static_cast<size_t>(t + tid) * s.H + h]) <= 1.0f)) bad |= 1u << tid;
#pragma unroll
        for (int i = 0; i < DX_T; ++i)
            if (!(g[i].x >= 0.0f && g[i].x <= 1.0f && g[i].y >= 0.0f && g[i].y <= 1.0f)) bad |= 1u << i;
#pragma unroll
        for (int i = 0; i < 8; ++i)
            if (!(fabsf(k[i].x) <= 2.0f && fabsf(k[i].y) <= 2.0f && fabsf(q[i].x) <= 2.0f && fabsf(q[i].y) <= 2.0f)) bad |= 1u << (8 * hf + i);
        bad = __reduce_or_sync(0xffffffffu, bad);
        if (lane == 0) marks[tid >> 5] = bad;
        for (int i = tid; i < 512; i += 128) nums[i] = 0.0f;
        // halves of 16, 8, 4 and 2 tokens: `half` tokens either side of a cut
        auto row = [&](int level, int r) -> float2& { return *reinterpret_cast<float2*>(rows + (24 * level + r) * DX_LP + c); };
        auto times = [](float2 a, float2 b) { return make_float2(a.x * b.x, a.y * b.y); };
        if (hf) {
            float2 f = one;
#pragma unroll
            for (int m = 0; m < 8; ++m) {
                f = times(f, g[8 + m]);
                row(0, m) = times(f, k[m]);
                row(0, 8 + m) = times(f, q[m]);
            }
        } else {
            float2 b = one;
#pragma unroll
            for (int m = 7; m >= 0; --m) {
                row(0, 16 + m) = times(b, k[m]);
                b = times(b, g[m]);
            }
        }
#pragma unroll
        for (int level = 1; level < 4; ++level) {
            const int half = 8 >> level;
#pragma unroll
            for (int cut = half; cut < 8; cut += 2 * half) {                // of this thread's eight tokens
                const int base = 4 * hf + (cut - half) / 2;
                float2 f = one, b = one;
#pragma unroll
                for (int m = 0; m < half; ++m) {
                    f = times(f, hf ? g[8 + cut + m] : g[cut + m]);
                    row(level, base + m) = times(f, k[cut + m]);
                    row(level, 8 + base + m) = times(f, q[cut + m]);
                    row(level, 16 + base + half - 1 - m) = times(b, k[cut - 1 - m]);
                    b = times(b, hf ? g[8 + cut - 1 - m] : g[cut - 1 - m]);
                }
            }
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const float x = warp_sum(q[i].x * k[i].x + q[i].y * k[i].y);
            if (lane == 0) shares[(tid >> 5) * 8 + i] = x;
        }
        __syncthreads();
        // A's and B's dot products of a pair of tokens share its k_j: 64, 32, 16 and 8 pairs a level
        if (tid < 120) {
            const int level = tid < 64 ? 0 : tid < 96 ? 1 : tid < 112 ? 2 : 3, half = 8 >> level, n = tid - (128 - (128 >> level));
            const int i = n / half, j = n % half, base = i / half * half;       // i: row of all eight
            const float* ka = rows + (24 * level + i) * DX_LP;
            const float* qa = ka + 8 * DX_LP;
            const float* b = rows + (24 * level + 16 + base + j) * DX_LP;
            float x[16], z[16];                      // sixteen chains of eight: four of 32 had twice the error
#pragma unroll
            for (int n = 0; n < 16; ++n) x[n] = z[n] = 0.0f;
#pragma unroll 2
            for (int d = 0; d < D; d += 16)
#pragma unroll
                for (int n = 0; n < 16; n += 4) {
                    const float4 u = *reinterpret_cast<const float4*>(ka + d + n), w = *reinterpret_cast<const float4*>(qa + d + n), v = *reinterpret_cast<const float4*>(b + d + n);
                    x[n] = fmaf(u.x, v.x, x[n]); x[n + 1] = fmaf(u.y, v.y, x[n + 1]); x[n + 2] = fmaf(u.z, v.z, x[n + 2]); x[n + 3] = fmaf(u.w, v.w, x[n + 3]);
                    z[n] = fmaf(w.x, v.x, z[n]); z[n + 1] = fmaf(w.y, v.y, z[n + 1]); z[n + 2] = fmaf(w.z, v.z, z[n + 2]); z[n + 3] = fmaf(w.w, v.w, z[n + 3]);
                }
#pragma unroll
            for (int n = 8; n > 0; n >>= 1)
#pragma unroll
                for (int m = 0; m < n; ++m) { x[m] += x[m + n]; z[m] += z[m + n]; }
            const int to = 16 * (2 * base + half + i % half) + 2 * base + j;
            nums[to] = x[0];
            nums[256 + to] = z[0];
        }
        if (tid < DX_T) nums[256 + 17 * tid] = shares[2 * (tid >> 3) * 8 + (tid & 7)] + shares[(2 * (tid >> 3) + 1) * 8 + (tid & 7)];
        __syncthreads();                                                    // the planes take the rows' place
        auto put = [&](int which, int i, float2 v) {
#pragma unroll
            for (int p = 0; p < 3; ++p) *reinterpret_cast<unsigned*>(planes + (which * 3 + p) * DX_PLANE + i * DX_PITCH + c) = split_piece(v.x, v.y);
        };
        float2 p = one, e = one;
        if (hf) {
#pragma unroll
            for (int i = 0; i < 8; ++i) p = times(p, g[i]);
        } else {
#pragma unroll
            for (int i = 15; i >= 8; --i) e = times(e, g[i]);
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            p = times(p, hf ? g[8 + i] : g[i]);
            put(0, 8 * hf + i, times(p, k[i]));
            put(1, 8 * hf + i, times(p, q[i]));
        }
        if (hf) *reinterpret_cast<float2*>(total + c) = p;
#pragma unroll
        for (int i = 7; i >= 0; --i) {
            put(2, 8 * hf + i, times(e, k[i]));
            e = times(e, hf ? g[8 + i] : g[i]);
        }
        const unsigned any = marks[0] | marks[1] | marks[2] | marks[3];
        if (tid < 4) reinterpret_cast<int*>(total + D)[tid] = any ? __ffs(any) - 1 : DX_T;
    }
    auto put_small = [&](int which, int i, int j, float v) {
        float rest = 0.0f;
#pragma unroll
        for (int p = 0; p < 3; ++p) reinterpret_cast<unsigned short*>(small)[(which * 3 + p) * DX_NPLANE + i * DX_NP + j] = static_cast<unsigned short>(split_piece(v, rest));
    };
    if (tid < DX_T) {                                // column `tid` of T: rows in order
        float x[DX_T];
#pragma unroll
        for (int i = 0; i < DX_T; ++i) {
            const float be = i < nt ? beta[static_cast<size_t>(t + i) * s.H + h] : 0.0f;
            float v = i == tid ? 1.0f : 0.0f, w = 0.0f;
#pragma unroll
            for (int m = 0; m < i; ++m) (m & 1 ? w : v) -= nums[16 * i + m] * x[m];
            x[i] = i < tid ? 0.0f : be * (v + w);
            put_small(0, i, tid, x[i]);
        }
    } else if (tid >= 32) {
        for (int idx = tid - 32; idx < 256; idx += 96) put_small(1, idx >> 4, idx & 15, nums[256 + idx]);
    }
    __syncthreads();
    uint4* to = reinterpret_cast<uint4*>(images + (static_cast<size_t>(blockIdx.x) * s.H + h) * DX_IMAGE);
    for (int i = tid; i < DX_IMAGE / 16; i += 128) to[i] = reinterpret_cast<const uint4*>(dx_smem)[i];
}

// grid: entries (longest portion first) x H x column tiles of DX_COLS, the tiles fastest.
#define DX_COLS 16
#define DX_SMEM (2 * DX_IMAGE + 4 * 4 * 32 * 16)
__global__ void __launch_bounds__(128, 2) delta_scan_mma_kernel(
    const DeltaShape s, const float* __restrict__ proj, const unsigned char* __restrict__ images, const float* __restrict__ qn,
    const float* __restrict__ kn, const float* __restrict__ vn, const float* __restrict__ beta, const float* __restrict__ decay,
    float* __restrict__ o, float* __restrict__ state, const int32_t* __restrict__ positions, const int32_t* __restrict__ entry_slot,
    const int32_t* __restrict__ entry_q_start, const int32_t* __restrict__ entry_q_len, int num_entries, int tiles, int32_t* __restrict__ status) {
    pdl_begin();
    constexpr int D = 128;
    extern __shared__ __align__(16) unsigned char dx_smem[];
    float4* shares = reinterpret_cast<float4*>(dx_smem + 2 * DX_IMAGE);      // [4 warps][X 2, O 2][32 lanes]
    __shared__ __align__(8) unsigned long long full[2];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, lg = lane >> 2, lt = lane & 3;
    const int tile = blockIdx.x % tiles, c0 = tile * DX_COLS, h = blockIdx.x / tiles % s.H, kvh = h / (s.H / s.G);
    int entry = blockIdx.x / (tiles * s.H);
    if (num_entries <= 32) {                                    // longest portions first: the entry with `entry` ones before it
        const int mine = lane < num_entries ? entry_q_len[lane] : -1;
        int before = 0;
        for (int e = 0; e < num_entries; ++e) {
            const int len = __shfl_sync(0xffffffffu, mine, e);
            before += len > mine || (len == mine && e < lane);
        }
        entry = __ffs(__ballot_sync(0xffffffffu, before == entry && lane < num_entries)) - 1;
    }
    const long long row0 = entry_q_start[entry];
    const int count = entry_q_len[entry];
    if (count <= 0) return;                                     // no copy may be on its way when the block ends
    float* slot = state + entry_slot[entry] * s.slot_stride;
    // a warp: all columns, rows 32 warp .. + 31; tile n, element i: column v0 + 8 (i >> 1), row d0 + 8 n + (i & 1)
    const int v0 = c0 + lg, dw = 32 * warp, d0 = dw + 2 * lt;
    float* my_state = slot + (static_cast<long long>(h) * s.V + v0) * D + d0;
    float S[4][4];
    bool bad_state = false;
    auto look = [&]() {
        bad_state = false;
#pragma unroll
        for (int n = 0; n < 4; ++n)
#pragma unroll
            for (int i = 0; i < 4; ++i) bad_state |= !(fabsf(S[n][i]) < 1.1529215e18f);      // 2^60
    };
#pragma unroll
    for (int n = 0; n < 4; ++n) {
        const float2 lo = *reinterpret_cast<const float2*>(my_state + 8 * n), hi = *reinterpret_cast<const float2*>(my_state + 8 * D + 8 * n);
        S[n][0] = lo.x; S[n][1] = lo.y; S[n][2] = hi.x; S[n][3] = hi.y;
    }
    look();
    if (tid == 0) {
        t5_mbar_init(&full[0], 1);
        t5_mbar_init(&full[1], 1);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    bool bad = __syncthreads_or(bad_state);
    const unsigned char* image = images + (static_cast<size_t>(dx_place(row0, entry)) * s.H + h) * DX_IMAGE;
    const size_t image_step = static_cast<size_t>(s.H) * DX_IMAGE;
    auto stage = [&](int b) {                                   // one copy for the whole image: by sixteen bytes a thread it took 1,800 clocks to issue
        if (tid == 0) {
            t5_expect_tx(&full[b], DX_IMAGE);
            asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::
                             "r"(t5_smem(dx_smem + b * DX_IMAGE)), "l"(image), "r"(DX_IMAGE), "r"(t5_smem(&full[b])) : "memory");
        }
        image += image_step;
    };
    auto landed = [&](int b, unsigned parity) {
        for (int i = 0; i < T5_WAIT_LIMIT; ++i)
            if (t5_try_wait(&full[b], parity)) return true;
        return false;
    };
    // values of (column v0 + 8 (i >> 1), token 8 u + 2 lt + (i & 1))
    const float* my_v = vn + (static_cast<size_t>(row0) * s.H + h) * s.VP + v0;
    const int v_step = s.H * s.VP;
    const float* next_v = my_v + static_cast<size_t>(2 * lt) * v_step;
    float v[2][4];
    auto fetch = [&](int done) {
#pragma unroll
        for (int u = 0; u < 2; ++u)
#pragma unroll
            for (int i = 0; i < 4; ++i) v[u][i] = done + 8 * u + 2 * lt + (i & 1) < count ? next_v[(8 * u + (i & 1)) * v_step + 8 * (i >> 1)] : 0.0f;
        next_v += static_cast<size_t>(DX_T) * v_step;
    };
    const int frow = (lane >> 4) * 8 + (lane & 7), fcol = ((lane >> 3) & 1) * 8;
    const int grow = fcol + (lane & 7), gcol = (lane >> 4) * 8;
    constexpr int A[6] = {2, 0, 1, 1, 0, 0}, B[6] = {0, 2, 1, 0, 1, 0};          // planes of the six products, the smallest first
    stage(0);
    fetch(0);
    for (int done = 0, b = 0; done < count; done += DX_T, b ^= 1) {
        const int nb = min(DX_T, count - done);
        if (__syncthreads_or(!landed(b, (done / (2 * DX_T)) & 1))) {         // (never: the copy did not land in time)
            if (tid == 0 && atomicCAS(status, 0, DX_STATUS) == 0) status[1] = blockIdx.x;
            return;
        }
        if (done + DX_T < count) stage(b ^ 1);
        const bf16* planes = reinterpret_cast<const bf16*>(dx_smem + b * DX_IMAGE);
        const bf16* small = planes + 9 * DX_PLANE;
        const float* total = reinterpret_cast<const float*>(small + 6 * DX_NPLANE);
        float* oo = o + (static_cast<size_t>(row0 + done) * s.H + h) * s.V + v0;
        const size_t o_step = static_cast<size_t>(s.H) * s.V;
        const int good = bad ? 0 : *reinterpret_cast<const int*>(total + D);      // tokens in front of the mark
        // shares of (p k) S and (p q) S over this warp's rows
        float rm[2][4], rs[2][4], xm[2][4], xs[2][4];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            unsigned a[3][4], yk[3][4], yq[3][4];
#pragma unroll
            for (int p = 0; p < 3; ++p) {
                ldmatrix_x4(yk[p], planes + p * DX_PLANE + frow * DX_PITCH + dw + 16 * j + fcol);
                ldmatrix_x4(yq[p], planes + (3 + p) * DX_PLANE + frow * DX_PITCH + dw + 16 * j + fcol);
            }
            split_tiles(S[2 * j], S[2 * j + 1], a);
#pragma unroll
            for (int i = 0; i < 6; ++i)              // four sums side by side
#pragma unroll
                for (int w = 0; w < 4; ++w) {
                    const int u = w & 1;
                    float (&c)[4] = w < 2 ? (i < 5 ? rs[u] : rm[u]) : (i < 5 ? xs[u] : xm[u]);
                    const unsigned b0 = w < 2 ? yk[B[i]][2 * u] : yq[B[i]][2 * u], b1 = w < 2 ? yk[B[i]][2 * u + 1] : yq[B[i]][2 * u + 1];
                    if (j == 0 && (i == 0 || i == 5)) mma_bf16_first(c, a[A[i]], b0, b1);
                    else mma_bf16(c, a[A[i]], b0, b1);
                }
        }
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            shares[(warp * 4 + u) * 32 + lane] = make_float4(rm[u][0] + rs[u][0], rm[u][1] + rs[u][1], rm[u][2] + rs[u][2], rm[u][3] + rs[u][3]);
            shares[(warp * 4 + 2 + u) * 32 + lane] = make_float4(xm[u][0] + xs[u][0], xm[u][1] + xs[u][1], xm[u][2] + xs[u][2], xm[u][3] + xs[u][3]);
        }
        __syncthreads();
        auto over_rows = [&](int which) {            // the four warps' shares, in the same order whoever adds them
            float4 x[4];
#pragma unroll
            for (int w = 0; w < 4; ++w) x[w] = shares[(w * 4 + which) * 32 + lane];
            return make_float4((x[0].x + x[1].x) + (x[2].x + x[3].x), (x[0].y + x[1].y) + (x[2].y + x[3].y),
                               (x[0].z + x[1].z) + (x[2].z + x[3].z), (x[0].w + x[1].w) + (x[2].w + x[3].w));
        };
        auto before_mark = [&](float (&c)[2][4]) {
            if (good < DX_T)
#pragma unroll
                for (int u = 0; u < 2; ++u)
#pragma unroll
                    for (int i = 0; i < 4; ++i) c[u][i] = 8 * u + 2 * lt + (i & 1) < good ? c[u][i] : 0.0f;
        };
        float x[2][4];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const float4 r = over_rows(u);
            x[u][0] = v[u][0] - r.x; x[u][1] = v[u][1] - r.y; x[u][2] = v[u][2] - r.z; x[u][3] = v[u][3] - r.w;
        }
        before_mark(x);
        if (done + DX_T < count) fetch(done + DX_T);
        unsigned a[3][4], y[3][4];
        float um[2][4], us[2][4];
        split_tiles(x[0], x[1], a);
#pragma unroll
        for (int p = 0; p < 3; ++p) ldmatrix_x4(y[p], small + p * DX_NPLANE + frow * DX_NP + fcol);
        split_mma_whole(um, us, a, y);
#pragma unroll
        for (int u = 0; u < 2; ++u)
#pragma unroll
            for (int i = 0; i < 4; ++i) um[u][i] += us[u][i];
        before_mark(um);
        split_tiles(um[0], um[1], a);
        if (good == DX_T) {
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                float c[2][4], cs[2][4];
#pragma unroll
                for (int p = 0; p < 3; ++p) ldmatrix_x4_trans(y[p], planes + (6 + p) * DX_PLANE + grow * DX_PITCH + dw + 16 * j + gcol);
                split_mma_whole(c, cs, a, y);
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const float2 f = *reinterpret_cast<const float2*>(total + dw + 16 * j + 8 * u + 2 * lt);
#pragma unroll
                    for (int i = 0; i < 4; ++i) S[2 * j + u][i] = fmaf(S[2 * j + u][i], i & 1 ? f.y : f.x, cs[u][i]) + c[u][i];
                }
            }
        }
        if (warp >= 2) {                             // two warps of the four make the outputs, eight tokens each
            const int u = warp & 1;
            float om[4], os[4];
#pragma unroll
            for (int p = 0; p < 3; ++p) ldmatrix_x4(y[p], small + (3 + p) * DX_NPLANE + frow * DX_NP + fcol);
            const unsigned b0[3] = {u ? y[0][2] : y[0][0], u ? y[1][2] : y[1][0], u ? y[2][2] : y[2][0]};
            const unsigned b1[3] = {u ? y[0][3] : y[0][1], u ? y[1][3] : y[1][1], u ? y[2][3] : y[2][1]};
            split_mma_whole(om, os, a, b0, b1);
            const float4 r = over_rows(2 + u);
            const float out[4] = {r.x + (om[0] + os[0]), r.y + (om[1] + os[1]), r.z + (om[2] + os[2]), r.w + (om[3] + os[3])};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int t = 8 * u + 2 * lt + (i & 1);
                if (t < min(nb, good)) oo[t * o_step + 8 * (i >> 1)] = out[i];
            }
        }
        if (good < DX_T) {                           // token by token
            __syncthreads();                         // the shares have been read
            float* sums = reinterpret_cast<float*>(shares);                   // [2][4 row quarters][16 columns]
            for (int t = 0; t < nb; ++t) {
                const size_t row = row0 + done + t;
                const float be = beta[row * s.H + h];
                float2 kk[4], qq[4];
                float r0 = 0.0f, r1 = 0.0f;
#pragma unroll
                for (int n = 0; n < 4; ++n) {
                    const float2 g = *reinterpret_cast<const float2*>(decay + (row * s.H + h) * D + d0 + 8 * n);
                    kk[n] = *reinterpret_cast<const float2*>(kn + (row * s.G + kvh) * D + d0 + 8 * n);
                    qq[n] = *reinterpret_cast<const float2*>(qn + (row * s.G + kvh) * D + d0 + 8 * n);
                    S[n][0] *= g.x; S[n][1] *= g.y; S[n][2] *= g.x; S[n][3] *= g.y;
                    r0 += S[n][0] * kk[n].x + S[n][1] * kk[n].y;
                    r1 += S[n][2] * kk[n].x + S[n][3] * kk[n].y;
                }
                auto all_rows = [&](float& x0, float& x1, float* to) {        // sums over the state's rows, in every warp
#pragma unroll
                    for (int off = 1; off <= 2; off <<= 1) {
                        x0 += __shfl_xor_sync(0xffffffffu, x0, off);
                        x1 += __shfl_xor_sync(0xffffffffu, x1, off);
                    }
                    if (lt == 0) {
                        to[warp * DX_COLS + v0 - c0] = x0;
                        to[warp * DX_COLS + v0 - c0 + 8] = x1;
                    }
                    __syncthreads();
                    x0 = x1 = 0.0f;
#pragma unroll
                    for (int w = 0; w < 4; ++w) {
                        x0 += to[w * DX_COLS + v0 - c0];
                        x1 += to[w * DX_COLS + v0 - c0 + 8];
                    }
                };
                all_rows(r0, r1, sums);
                const float u0 = be * (my_v[static_cast<size_t>(done + t) * v_step] - r0), u1 = be * (my_v[static_cast<size_t>(done + t) * v_step + 8] - r1);
                float x0 = 0.0f, x1 = 0.0f;
#pragma unroll
                for (int n = 0; n < 4; ++n) {
                    S[n][0] += kk[n].x * u0; S[n][1] += kk[n].y * u0; S[n][2] += kk[n].x * u1; S[n][3] += kk[n].y * u1;
                    x0 += S[n][0] * qq[n].x + S[n][1] * qq[n].y;
                    x1 += S[n][2] * qq[n].x + S[n][3] * qq[n].y;
                }
                all_rows(x0, x1, sums + 4 * DX_COLS);
                if (lt == 0 && warp == 0 && t >= good) {
                    oo[t * o_step] = x0;
                    oo[t * o_step + 8] = x1;
                }
            }
            look();
            bad = __syncthreads_or(bad_state);
        }
    }
#pragma unroll
    for (int n = 0; n < 4; ++n) {
        *reinterpret_cast<float2*>(my_state + 8 * n) = make_float2(S[n][0], S[n][1]);
        *reinterpret_cast<float2*>(my_state + 8 * D + 8 * n) = make_float2(S[n][2], S[n][3]);
    }
    dr_keep_inputs<128>(s, proj, slot, positions, row0, count, h, c0, DX_COLS, tile == 0);
}

// A warp per (token, head): o / rms(o) * w * gate * scale.
template <typename TO>
__global__ void delta_output_kernel(const float* __restrict__ o, const float* __restrict__ gate, const float* __restrict__ norm_w,
                                    float eps, float out_scale, TO* __restrict__ out, long long out_stride, int out_off, int H,
                                    int V, long long items) {
    pdl_begin();
    const long long item = static_cast<long long>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (item >= items) return;
    const int lane = threadIdx.x & 31;
    const long long t = item / H;
    const int h = static_cast<int>(item - t * H);
    const float* row = o + item * V;
    const float* gr = gate + item * V;
    float ss = 0.0f;
    for (int c = lane; c < V; c += 32) ss += row[c] * row[c];
    ss = warp_sum(ss);
    const float inv = 1.0f / sqrtf(ss / static_cast<float>(V) + eps);
    TO* orow = out + t * out_stride + out_off + h * V;
    for (int c = lane; c < V; c += 32) orow[c] = from_f32<TO>(row[c] * inv * norm_w[c] * gr[c] * out_scale);
}

// Entries that bring one token: one block per (entry, head).  STAGED: the head's state (V columns of DP floats) and, with
// `low_staged`, its slices of the low-rank weights are copied into shared memory before the block waits for the kernel in
// front of it (nothing else in a step writes this stage's states, and the weights never change); otherwise they are read
// as they are needed.
template <int R, typename TW, typename TO, bool STAGED>
__global__ void __launch_bounds__(512) delta_step_kernel(
    const DeltaShape s, const float* __restrict__ proj, const float* __restrict__ conv_w, const TW* __restrict__ wa,
    const float* __restrict__ dt_bias, const float* __restrict__ a_log, const TW* __restrict__ wg,
    const float* __restrict__ norm_w, float eps, float out_scale, TO* __restrict__ out, long long out_stride, int out_off,
    float* __restrict__ state, const int32_t* __restrict__ positions, const int32_t* __restrict__ entry_slot,
    const int32_t* __restrict__ entry_q_start, int low_staged) {
    pdl_invite();
    constexpr int DP = DR_LANES * R;
    extern __shared__ __align__(16) float smem[];
    float* sq = smem;                         // [DP] each
    float* sk = sq + DP;
    float* sg = sk + DP;
    float* red = sg + DP;                     // 36
    float* sv = red + 36;                     // [V] each
    float* so = sv + s.V;
    float* sgate = so + s.V;
    float* first = sgate + s.V;               // [ra + rg]: the first halves of the low-rank projections
    const int chans = s.D + s.V, tid = threadIdx.x, nthreads = blockDim.x;
    int parts = nthreads / chans;             // threads that share a channel's low-rank sum
    parts = parts < 1 ? 1 : parts > 8 ? 8 : parts;
    float* split = first + s.ra + s.rg;       // [parts][D + V]
    float* held = smem + ((3 * DP + 36 + 3 * s.V + s.ra + s.rg + parts * chans + 3) & ~3);     // STAGED: [V][DP]
    TW* low = reinterpret_cast<TW*>(held + (STAGED ? static_cast<size_t>(s.V) * DP : 0));      // STAGED: [ra][D], [rg][V]
    const int entry = blockIdx.x, h = blockIdx.y;
    const int kvh = h / (s.H / s.G);
    const long long t = entry_q_start[entry];
    const int pos = positions[t];
    float* slot = state + entry_slot[entry] * s.slot_stride;
    float* head_state = slot + static_cast<long long>(h) * s.V * DP;
    float* ring = slot + s.ring_off;
    const int C = 2 * s.G * s.D + s.H * s.V;
    // what the block will read of weights and of earlier steps' inputs, on its way to the cache before the wait
    const int cq = kvh * s.D, ck = (s.G + kvh) * s.D, cv = 2 * s.G * s.D + h * s.V;
    for (int i = tid * 32; i < s.D * s.taps; i += nthreads * 32) {
        dr_prefetch(conv_w + static_cast<size_t>(cq) * s.taps + i);
        dr_prefetch(conv_w + static_cast<size_t>(ck) * s.taps + i);
    }
    for (int i = tid * 32; i < s.V * s.taps; i += nthreads * 32) dr_prefetch(conv_w + static_cast<size_t>(cv) * s.taps + i);
    for (int i = tid; i < s.taps * 32; i += nthreads) {         // a ring row's three pieces in lines of 32 floats
        const float* row = ring + static_cast<long long>(i >> 5) * C;
        for (int x = (i & 31) * 32; x < s.D; x += 1024) {
            dr_prefetch(row + cq + x);
            dr_prefetch(row + ck + x);
        }
        for (int x = (i & 31) * 32; x < s.V; x += 1024) dr_prefetch(row + cv + x);
    }
    for (int i = tid * 32; i < s.D; i += nthreads * 32) dr_prefetch(dt_bias + h * s.D + i);
    for (int i = tid * 32; i < s.V; i += nthreads * 32) dr_prefetch(norm_w + i);
    if (!(STAGED && low_staged)) {
        for (int i = tid; i < s.ra; i += nthreads)
            for (int x = 0; x < s.D; x += 128 / static_cast<int>(sizeof(TW))) dr_prefetch(wa + static_cast<size_t>(i) * s.H * s.D + h * s.D + x);
        for (int i = tid; i < s.rg; i += nthreads)
            for (int x = 0; x < s.V; x += 128 / static_cast<int>(sizeof(TW))) dr_prefetch(wg + static_cast<size_t>(i) * s.H * s.V + h * s.V + x);
    }
    const float ea = expf(a_log[h]);
    if (STAGED) {
        constexpr int PER = 16 / sizeof(TW);
        const int na = low_staged ? s.ra * (s.D / PER) : 0, ng = low_staged ? s.rg * (s.V / PER) : 0;
        for (int i = tid; i < na + ng; i += nthreads) {
            const bool is_decay = i < na;
            const int n = is_decay ? i : i - na, w = is_decay ? s.D : s.V, j = n / (w / PER), x = (n - j * (w / PER)) * PER;
            const TW* src = is_decay ? wa + static_cast<size_t>(j) * s.H * s.D + h * s.D + x : wg + static_cast<size_t>(j) * s.H * s.V + h * s.V + x;
            dr_cp16(reinterpret_cast<float*>(low + (is_decay ? 0 : s.ra * s.D) + j * w + x), reinterpret_cast<const float*>(src));
        }
        for (int i = tid * 4; i < s.V * DP; i += nthreads * 4) dr_cp16(held + i, head_state + i);
        asm volatile("cp.async.commit_group;\n" ::);
    }
    pdl_wait();
    const float* pr = proj + t * s.stride;
    const float beta = dr_sigmoid(pr[s.b_off + h]);
    for (int j = tid; j < s.ra + s.rg; j += nthreads) first[j] = j < s.ra ? pr[s.a_off + j] : pr[s.g_off + j - s.ra];
    // convolutions; the row's own place in the ring is none that any block reads in this step
    float* mine = ring + static_cast<long long>(pos % s.taps) * C;
    const bool with_qk = h % (s.H / s.G) == 0;
    for (int i = tid; i < 2 * DP + s.V; i += nthreads) {
        if (i < 2 * DP) {
            const int d = i < DP ? i : i - DP;
            float x = 0.0f;
            if (d < s.D) {
                const int ch = (i < DP ? kvh : s.G + kvh) * s.D + d;
                x = dr_silu(dr_conv(s, proj, conv_w, ring, t, t, pos, ch));
                if (with_qk && s.taps > 1) mine[ch] = pr[s.q_off + ch];
            }
            sq[i] = x;                        // q, then k behind it
        } else {
            const int ch = 2 * s.G * s.D + h * s.V + (i - 2 * DP);
            sv[i - 2 * DP] = dr_silu(dr_conv(s, proj, conv_w, ring, t, t, pos, ch));
            if (s.taps > 1) mine[ch] = pr[s.q_off + ch];
        }
    }
    if (STAGED) asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();
    for (int i = tid; i < parts * chans; i += nthreads) {       // low-rank second halves
        const int p = i / chans, ch = i - p * chans;
        const bool is_decay = ch < s.D;
        const int rank = is_decay ? s.ra : s.rg, x = is_decay ? ch : ch - s.D;
        const bool here = STAGED && low_staged;
        const int width = here ? (is_decay ? s.D : s.V) : (is_decay ? s.H * s.D : s.H * s.V);
        const TW* w = here ? low + (is_decay ? 0 : s.ra * s.D) + x : is_decay ? wa + h * s.D + x : wg + h * s.V + x;
        const float* a = is_decay ? first : first + s.ra;
        const int per = (rank + parts - 1) / parts, j1 = min(rank, (p + 1) * per);
        float z = 0.0f;
        int j = p * per;
        for (; j + 16 <= j1; j += 16) {
            float wv[16];
#pragma unroll
            for (int u = 0; u < 16; ++u) wv[u] = to_f32(w[(j + u) * width]);
#pragma unroll
            for (int u = 0; u < 16; ++u) z += wv[u] * a[j + u];
        }
        for (; j < j1; ++j) z += to_f32(w[j * width]) * a[j];
        split[i] = z;
    }
    const int warp = tid >> 5, lane = tid & 31;
    if (warp == 0) {                          // unit norms and k . q
        float qq = 0.0f, kk = 0.0f, qk = 0.0f;
        for (int d = lane; d < DP; d += 32) {
            qq += sq[d] * sq[d];
            kk += sk[d] * sk[d];
            qk += sq[d] * sk[d];
        }
        qq = warp_sum(qq);
        kk = warp_sum(kk);
        qk = warp_sum(qk);
        const float iq = 1.0f / sqrtf(qq + 1e-6f) / sqrtf(static_cast<float>(s.D)), ik = 1.0f / sqrtf(kk + 1e-6f);
        for (int d = lane; d < DP; d += 32) {
            sq[d] *= iq;
            sk[d] *= ik;
        }
        if (lane == 0) red[33] = qk * iq * ik;
    }
    __syncthreads();
    for (int i = tid; i < DP + s.V; i += nthreads) {
        if (i < DP) {
            float g = 0.0f;
            if (i < s.D) {
                float z = dt_bias[h * s.D + i];
                for (int p = 0; p < parts; ++p) z += split[p * chans + i];
                g = dr_decay(z, ea);
            }
            sg[i] = g;
        } else {
            float z = 0.0f;
            for (int p = 0; p < parts; ++p) z += split[p * chans + s.D + (i - DP)];
            sgate[i - DP] = dr_sigmoid(z);
        }
    }
    __syncthreads();
    const float kq = red[33];
    const int l = tid & (DR_LANES - 1), cols = nthreads / DR_LANES;
    for (int c0 = 0; c0 < s.V; c0 += cols) {
        const int c = c0 + tid / DR_LANES;
        const bool there = c < s.V;
        const float* from = (STAGED ? held : head_state) + static_cast<size_t>(there ? c : 0) * DP;
        float* to = head_state + static_cast<size_t>(there ? c : 0) * DP;
        float S[R];
#pragma unroll
        for (int j = 0; j < R / 4; ++j) {
            const float4 x = *reinterpret_cast<const float4*>(from + 4 * l + 32 * j);
            S[4 * j] = x.x; S[4 * j + 1] = x.y; S[4 * j + 2] = x.z; S[4 * j + 3] = x.w;
        }
        const float o = dr_token<R>(S, sk, sq, sg, l, there ? sv[c] : 0.0f, beta, kq);
        if (there) {
#pragma unroll
            for (int j = 0; j < R / 4; ++j)
                *reinterpret_cast<float4*>(to + 4 * l + 32 * j) = make_float4(S[4 * j], S[4 * j + 1], S[4 * j + 2], S[4 * j + 3]);
            if (l == 0) so[c] = o;
        }
    }
    __syncthreads();
    float ss = 0.0f;
    for (int c = tid; c < s.V; c += nthreads) ss += so[c] * so[c];
    const float total = block_sum(ss, red);
    const float inv = 1.0f / sqrtf(total / static_cast<float>(s.V) + eps);
    TO* orow = out + t * out_stride + out_off + h * s.V;
    for (int c = tid; c < s.V; c += nthreads) orow[c] = from_f32<TO>(so[c] * inv * norm_w[c] * sgate[c] * out_scale);
}

// D rounded up to what the kernels are instantiated for: 32, 64, 128, 256; 0: larger.
extern "C" int llm_delta_padded(int D) { return D <= 0 ? 0 : D <= 32 ? 32 : D <= 64 ? 64 : D <= 128 ? 128 : D <= 256 ? 256 : 0; }

extern "C" int llm_delta_supported(int D, int V) { return llm_delta_padded(D) > 0 && V > 0 && V <= 1024; }

static int delta_shape(DeltaShape& s, int H, int G, int D, int V, int taps, int q_off, int b_off, int a_off, int ra, int g_off,
                       int rg, long long stride, long long slot_stride) {
    const int DP = llm_delta_padded(D);
    if (H <= 0 || G <= 0 || H % G || !llm_delta_supported(D, V) || taps < 1 || ra <= 0 || rg <= 0 || ra > 1024 || rg > 1024 || H > 65535)
        return LLM_REFUSED_SIZE;
    const long long ring_off = static_cast<long long>(H) * V * DP;
    if (slot_stride < ring_off + static_cast<long long>(taps) * (2LL * G * D + static_cast<long long>(H) * V) || slot_stride % 4)
        return LLM_REFUSED_SIZE;
    s = {H, G, D, V, DP, (V + 3) / 4 * 4, taps, q_off, q_off + G * D, q_off + 2 * G * D, b_off, a_off, ra, g_off, rg,
         stride, slot_stride, ring_off};
    return LLM_OK;
}

#define DR_SMS 148
#define DR_ALONE_SMEM (116 * 1024)

// Whether llm_delta_scan takes the tensor-core kernels: it is then given room for llm_delta_image_bytes() a batch of sixteen tokens and
// head (T / 16 + entries + 1 places) instead of pk, pq, total and num.  Their fixed part is larger, and few columns spread thinner over
// the SMs than with a warp to one to four of them; single tokens of other requests count, since the kernels of eight tokens give each
// warp more columns for them.  Whole calls (us, eight tokens a chunk and this; portions + single tokens, heads of 128 columns):
//   1,536 and 2,048 columns: 300, 16: 108, 114; 1,000, 16: 219, 219; 2,500, 16: 481, 500; 300 + 1, 8: 119, 125; but 1,000 + 1, 8: 201, 200;
//   2,500 + 1, 8: 428, 424; 2,500 + 1, 6: 410, 398; 2,500 + 3, 4: 420, 393; 2,500 + 8, 2: 404, 383
//   more: 300 + 1, 16: 123, 117; 1,000 + 1, 16: 266, 225; 1,000 + 2, 8: 250, 198; 1,000, 24: 287, 254; 2,500, 32: 726, 652; 300 + 300, 16:
//   129, 123; 284 + 567, 16: 182, 165; 260 + 5, 4: 127, 117
//   portions below 256: 100, 16: 60, 64; 4 x 200, 16: 123, 128; 32 x 64, 16: 259, 276
// (with blocks of 32 columns; with 16 the layer of one request takes 1,000, 16: 263, 231; 2,500, 16: 605, 524; 2,000, 8: 344, 297; 2,000,
// 4: 306, 275, and below 256 tokens both are level: the line could lie lower, and one request come here too)
// So: 256 tokens and more; more than 2,048 columns, or 1,500 where several requests share a step with a portion of 1,000 tokens; up to
// 9,472 columns, the two blocks of 32 columns an SM for which the line was measured first.  With blocks of 16 columns that are four, two of
// which an SM holds (97 KB each); a second wave of equal portions does not double the walk, because a block alone on its SM has half the
// columns and nothing in its way.  Layers, us, eight tokens a chunk, blocks of 32 columns and these: portions of 16 heads: 2 x 1,000 392, 378, 354; 3 x
// 1,000 591, 577, 572; 4 x 1,000 (8,192 columns) 681, 679, 672; 4 x 500 354, 361, 358; 4 x 260 205, 213, 209; 400, 800, 1,200 and 1,600
// 765, 707, 664; 3 x 300 and 2,000 650, 581, 546; 8 heads: 6 x 1,000 532, 517, 513; 8 x 1,000 605, 606, 598; 9 x 900 578, 584, 577; 8 from 200
// to 900 400, 377, 337.  (Equal short portions near the end of the range would be 1 to 2 % faster with eight tokens a chunk.)
extern "C" int llm_delta_image_bytes() { return DX_IMAGE; }
static bool dx_takes(int H, int D, int V) { return D == 128 && V > 0 && V % 32 == 0 && H > 0 && H <= 65535; }
extern "C" int llm_delta_batched(int H, int D, int V, int num_entries, int max_len) {
    const long long columns = static_cast<long long>(num_entries) * H * V;
    const bool enough = columns > 2048 || (columns >= 1500 && num_entries > 1 && max_len >= 1000);
    return dx_takes(H, D, V) && max_len >= 256 && enough && columns <= 64 * DR_SMS;
}

// Everything of a step that is not all single tokens.  Scratch (float32): qn, kn [T, G, DP], vn [T, H, VP], beta [T, H],
// decay [T, H, DP] (whose places from D on must be finite), gate and o [T, H, V], pk and pq [T, H, DP], and for P =
// T / 8 + entries + 1 chunks total [P, H, DP] and num [P, H, 128]; or, in place of the last four, images (see llm_delta_batched).
// `conv_w` [C, taps]: the rows of q, k and v one after another.  max_len: tokens of the longest entry, 0: not known.
extern "C" int llm_delta_scan(
    const float* proj, long long stride, int q_off, int b_off, int a_off, int ra, int g_off, int rg, const float* conv_w, int taps,
    const void* wa, const void* wg, int w_dtype, const float* dt_bias, const float* a_log, const float* norm_w, float eps,
    float out_scale, void* out, int out_dtype, long long out_stride, int out_off, float* state, long long slot_stride,
    const int32_t* positions, const int32_t* token_entry, const int32_t* entry_slot, const int32_t* entry_q_start,
    const int32_t* entry_q_len, int num_tokens, int num_entries, int max_len, int H, int G, int D, int V, float* qn, float* kn,
    float* vn, float* beta, float* decay, float* gate, float* o, float* pk, float* pq, float* total, float* num, void* images, int32_t* status,
    uintptr_t stream) {
    if (num_tokens <= 0 || num_entries <= 0) return LLM_OK;
    DeltaShape s;
    const int rc = delta_shape(s, H, G, D, V, taps, q_off, b_off, a_off, ra, g_off, rg, stride, slot_stride);
    if (rc != LLM_OK) return rc;
    if (!aligned16(state) || !aligned16(qn) || !aligned16(kn) || !aligned16(vn) || !aligned16(decay) || !aligned16(pk) || !aligned16(pq) ||
        !aligned16(total) || !aligned16(num))
        return LLM_REFUSED_ALIGN;
    if (w_dtype != LLM_DT_F32 && w_dtype != LLM_DT_BF16) return LLM_REFUSED_DTYPE;
    if (out_dtype != LLM_DT_F32 && out_dtype != LLM_DT_BF16) return LLM_REFUSED_DTYPE;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    const dim3 pgrid((num_tokens + DP_TOKENS - 1) / DP_TOKENS, (2 * G + H + DP_WARPS - 1) / DP_WARPS);
    const bool fours = s.DP == 128 && taps <= 4 && D % 4 == 0 && V % 4 == 0 && stride % 4 == 0 && q_off % 4 == 0 && slot_stride % 4 == 0 &&
                       s.ring_off % 4 == 0 && aligned16(proj) && aligned16(conv_w);
    if (fours) {
        launch_pdl(delta_prepare_fours_kernel, pgrid, dim3(DP_WARPS * 32), 0, st, s, proj, conv_w, state, positions, token_entry, entry_slot,
                   entry_q_start, qn, kn, vn, beta, num_tokens);
    } else {
#define PREPARE(PER)                                                                                                  \
    launch_pdl((delta_prepare_kernel<PER>), pgrid, dim3(DP_WARPS * 32), 0, st, s, proj, conv_w, state, positions,      \
               token_entry, entry_slot, entry_q_start, qn, kn, vn, beta, num_tokens)
    switch (s.DP) {
        case 32: PREPARE(1); break;
        case 64: PREPARE(2); break;
        case 128: PREPARE(4); break;
        default: PREPARE(8); break;
    }
#undef PREPARE
    }
    const int da = (H * D + DL_CHANNELS - 1) / DL_CHANNELS, ga = (H * V + DL_CHANNELS - 1) / DL_CHANNELS;
    const dim3 lgrid((num_tokens + DL_TOKENS - 1) / DL_TOKENS, da + ga);
    const size_t lsmem = static_cast<size_t>(DL_PITCH) * (ra > rg ? ra : rg) * sizeof(float);
    if (lgrid.y > 65535) return LLM_REFUSED_SIZE;
#define LOWRANK(TW)                                                                                                   \
    do {                                                                                                              \
        auto kern = delta_lowrank_kernel<TW>;                                                                         \
        if (lsmem > 48 * 1024) {                                                                                      \
            const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,             \
                                                       static_cast<int>(lsmem));                                      \
            if (e != cudaSuccess) return static_cast<int>(e);                                                         \
        }                                                                                                             \
        launch_pdl(kern, lgrid, dim3(DL_THREADS), lsmem, st, s, proj, static_cast<const TW*>(wa), dt_bias, a_log,    \
                   static_cast<const TW*>(wg), decay, gate, num_tokens, da);                                          \
    } while (0)
    const int dm = (H * D + DM_CHANNELS - 1) / DM_CHANNELS, gm = (H * V + DM_CHANNELS - 1) / DM_CHANNELS;
    // Both at 4,096 channels (us, this one first): rank 64, 8 tokens 6.8, 11.8; 64: 10.1, 13.9; 512: 12.0, 18.6; 1,700: 33.7, 62.7;
    // rank 200, 512 tokens 18.7, 37.8; rank 16, 512 tokens 10.8, 10.1.  32-bit weights would need the exact split too.
    if (w_dtype == LLM_DT_BF16 && (ra > 32 || rg > 32) && dm + gm <= 65535)
        launch_pdl(delta_lowrank_mma_kernel, dim3((num_tokens + DM_TOKENS - 1) / DM_TOKENS, dm + gm), dim3(256), 0, st, s, proj,
                   static_cast<const bf16*>(wa), dt_bias, a_log, static_cast<const bf16*>(wg), decay, gate, num_tokens, dm);
    else if (w_dtype == LLM_DT_F32) LOWRANK(float);
    else LOWRANK(bf16);
#undef LOWRANK
    const long long walks = static_cast<long long>(num_tokens) * H;
    if (images) {
        if (!dx_takes(H, D, V) || !aligned16(images)) return LLM_REFUSED_SIZE;
        static_assert(DX_IMAGE <= DX_ROWS && DX_IMAGE % 16 == 0, "the image takes the vectors' place");
        cudaError_t e = cudaFuncSetAttribute(delta_batch_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, DX_BATCH_SMEM);
        if (e != cudaSuccess) return static_cast<int>(e);
        launch_pdl(delta_batch_kernel, dim3(num_tokens / DX_T + num_entries, H), dim3(128), DX_BATCH_SMEM, st, s, qn, kn, vn, beta, decay,
                   static_cast<unsigned char*>(images), entry_q_start, entry_q_len, num_entries);
        constexpr int most = DX_SMEM > DR_ALONE_SMEM ? DX_SMEM : DR_ALONE_SMEM;
        e = cudaFuncSetAttribute(delta_scan_mma_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
        if (e != cudaSuccess) return static_cast<int>(e);
        const int tiles = V / DX_COLS;
        const long long blocks = static_cast<long long>(num_entries) * H * tiles;
        const bool alone = blocks <= DR_SMS || (blocks <= 2 * DR_SMS && walks * tiles <= static_cast<long long>(DR_SMS) * max_len);
        launch_pdl(delta_scan_mma_kernel, dim3(static_cast<unsigned>(blocks)), dim3(128), alone ? most : DX_SMEM, st, s, proj,
                   static_cast<const unsigned char*>(images), qn, kn, vn, beta, decay, o, state, positions, entry_slot, entry_q_start,
                   entry_q_len, num_entries, tiles, status);
    } else {
    const dim3 cgrid(num_tokens, (H + DC_WARPS - 1) / DC_WARPS);
#define CHUNKS_OF(DP)                                                                                                 \
    launch_pdl((delta_chunk_kernel<DP>), cgrid, dim3(DC_WARPS * 32), 0, st, s, qn, kn, decay, pk, pq, total, num,      \
               token_entry, entry_q_start, entry_q_len, num_tokens)
    switch (s.DP) {
        case 32: CHUNKS_OF(32); break;
        case 64: CHUNKS_OF(64); break;
        case 128: CHUNKS_OF(128); break;
        default: CHUNKS_OF(256); break;
    }
#undef CHUNKS_OF
// A portion is as long as its blocks' walk, and a block beside another on its SM walks at a little over half the pace.  So
// portions start longest first, and the blocks ask for more than half of an SM's shared memory, each to have an SM of its own,
// while the device's SMs can do all walks in the time of the longest one: the last blocks begin where short portions have ended.
// Up to two blocks an SM, and by the longest portion (`max_len`; not known, 0: while no SM gets two).  Measured (us; portions
// of 284, 567 and 849 tokens, 192 blocks): as the hardware deals them 241, longest first 188, and alone 160; eight of 55 to 445
// tokens, 256 blocks: longest first 106, and alone 89; 512 blocks: side by side 179, alone 208.  Equal portions of 256 tokens, the
// whole layer's kernels: 156 blocks side by side 128, alone 148; 192: 138, 157; 256: 151, 172; 288: 154, 176.
#define SCAN(DP, C, WARPS, L)                                                                                         \
    do {                                                                                                              \
        auto kern = delta_scan_kernel<DP, C, WARPS, L>;                                                               \
        constexpr int COLS = WARPS * (32 / L) * C, CH = DR_TB / DR_CHUNK;                                             \
        constexpr size_t need = (2 * (DR_TB * (3 * DP + COLS + 1) + CH * (DP + DR_NUM)) + COLS * 2 * DR_CHUNK) * sizeof(float); \
        constexpr size_t most = need > DR_ALONE_SMEM ? need : DR_ALONE_SMEM;                                          \
        const int tiles = (V + COLS - 1) / COLS;                                                                      \
        const long long blocks = static_cast<long long>(num_entries) * H * tiles;                                     \
        if (blocks > 0x7fffffffLL) return LLM_REFUSED_SIZE;                                                           \
        const bool alone = blocks <= DR_SMS || (blocks <= 2 * DR_SMS && walks * tiles <= static_cast<long long>(DR_SMS) * max_len); \
        const size_t smem = alone ? most : need;                                                                      \
        /* the limit is the same for every launch: another thread may be between the two calls */                     \
        const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(most)); \
        if (e != cudaSuccess) return static_cast<int>(e);                                                             \
        launch_pdl(kern, dim3(static_cast<unsigned>(blocks)), dim3(WARPS * 32), smem, st, s, proj, pq, pk, vn, beta, decay, \
                   total, num, o, state, positions, entry_slot, entry_q_start, entry_q_len, num_entries, tiles);      \
    } while (0)
    // few columns: fewer a warp, so that more schedulers have one; many: more a warp, which costs fewer instructions a column.
    // Measured at 128 rows (us; one, two, four columns on 32 lanes, four on 16): 512 columns (1,000 tokens) 106 111 133 177,
    // 1,024: 141 112 134 181, 2,048: 213 159 136 182, 4,096 (1,500 tokens of 4 requests): 203 154 131 113.
    const long long columns = static_cast<long long>(num_entries) * H * V;
    const int plan = columns <= 640 ? 0 : columns <= 1300 ? 1 : columns <= 3000 ? 2 : 3;
    switch (s.DP) {
        case 32: SCAN(32, 2, 2, 8); break;
        case 64: SCAN(64, 2, 4, 16); break;
        case 128:
            if (plan == 0) SCAN(128, 1, 4, 32);
            else if (plan == 1) SCAN(128, 2, 4, 32);
            else if (plan == 2) SCAN(128, 4, 4, 32);
            else SCAN(128, 4, 4, 16);
            break;
        default:
            if (plan == 0) SCAN(256, 1, 4, 32);
            else SCAN(256, 2, 4, 32);
            break;
    }
#undef SCAN
    }
    const long long items = static_cast<long long>(num_tokens) * H;
    const long long oblocks = (items + 3) / 4;
    if (oblocks > 0x7fffffffLL) return LLM_REFUSED_SIZE;
    if (out_dtype == LLM_DT_F32)
        launch_pdl((delta_output_kernel<float>), dim3(static_cast<unsigned>(oblocks)), dim3(128), 0, st, o, gate, norm_w, eps, out_scale,
                   static_cast<float*>(out), out_stride, out_off, H, V, items);
    else
        launch_pdl((delta_output_kernel<bf16>), dim3(static_cast<unsigned>(oblocks)), dim3(128), 0, st, o, gate, norm_w, eps, out_scale,
                   static_cast<bf16*>(out), out_stride, out_off, H, V, items);
    return launch_status();
}

// A step whose entries all bring one token.
extern "C" int llm_delta_step(
    const float* proj, long long stride, int q_off, int b_off, int a_off, int ra, int g_off, int rg, const float* conv_w, int taps,
    const void* wa, const void* wg, int w_dtype, const float* dt_bias, const float* a_log, const float* norm_w, float eps,
    float out_scale, void* out, int out_dtype, long long out_stride, int out_off, float* state, long long slot_stride,
    const int32_t* positions, const int32_t* entry_slot, const int32_t* entry_q_start, int num_entries, int H, int G, int D, int V,
    uintptr_t stream) {
    if (num_entries <= 0) return LLM_OK;
    DeltaShape s;
    const int rc = delta_shape(s, H, G, D, V, taps, q_off, b_off, a_off, ra, g_off, rg, stride, slot_stride);
    if (rc != LLM_OK) return rc;
    if (!aligned16(state)) return LLM_REFUSED_ALIGN;
    int threads = V * DR_LANES;
    // few blocks: as fast as one can be; many: small ones, three to an SM, that overlap
    const bool few = static_cast<long long>(num_entries) * H <= 2 * 148;
    const int most = few ? 512 : 256;
    threads = threads > most ? most : (threads + 31) / 32 * 32;
    if (threads < 128) threads = 128;
    int parts = threads / (D + V);
    parts = parts < 1 ? 1 : parts > 8 ? 8 : parts;
    const size_t base = (3 * static_cast<size_t>(s.DP) + 36 + 3 * V + ra + rg + static_cast<size_t>(parts) * (D + V) + 3) / 4 * 4 * sizeof(float);
    const int esz = w_dtype == LLM_DT_F32 ? 4 : 2, per = 16 / esz;
    const size_t held = static_cast<size_t>(V) * s.DP * sizeof(float), low = (static_cast<size_t>(ra) * D + static_cast<size_t>(rg) * V) * esz;
    const bool vec = D % per == 0 && V % per == 0 && aligned16(wa) && aligned16(wg);
    const bool staged = base + held <= 200 * 1024;
    const int low_staged = staged && vec && base + held + low <= 200 * 1024 && few;
    const size_t smem = base + (staged ? held : 0) + (low_staged ? low : 0);
    if (smem > 200 * 1024) return LLM_REFUSED_SIZE;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    const dim3 grid(num_entries, H);
#define STEP(R, TW, TO)                                                                                               \
    do {                                                                                                              \
        auto kern = staged ? delta_step_kernel<R, TW, TO, true> : delta_step_kernel<R, TW, TO, false>;                \
        if (smem > 48 * 1024) {                                                                                       \
            const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,             \
                                                       static_cast<int>(smem));                                       \
            if (e != cudaSuccess) return static_cast<int>(e);                                                         \
        }                                                                                                             \
        launch_pdl(kern, grid, dim3(threads), smem, st, s, proj, conv_w, static_cast<const TW*>(wa), dt_bias, a_log,  \
                   static_cast<const TW*>(wg), norm_w, eps, out_scale, static_cast<TO*>(out), out_stride, out_off,    \
                   state, positions, entry_slot, entry_q_start, low_staged);                                          \
    } while (0)
#define BY_R(TW, TO)                                                                                                  \
    switch (s.DP) {                                                                                                   \
        case 32: STEP(4, TW, TO); break;                                                                              \
        case 64: STEP(8, TW, TO); break;                                                                              \
        case 128: STEP(16, TW, TO); break;                                                                            \
        default: STEP(32, TW, TO); break;                                                                             \
    }
    if (w_dtype == LLM_DT_F32 && out_dtype == LLM_DT_F32) { BY_R(float, float) }
    else if (w_dtype == LLM_DT_F32 && out_dtype == LLM_DT_BF16) { BY_R(float, bf16) }
    else if (w_dtype == LLM_DT_BF16 && out_dtype == LLM_DT_BF16) { BY_R(bf16, bf16) }
    else if (w_dtype == LLM_DT_BF16 && out_dtype == LLM_DT_F32) { BY_R(bf16, float) }
    else return LLM_REFUSED_DTYPE;
#undef BY_R
#undef STEP
    return launch_status();
}
