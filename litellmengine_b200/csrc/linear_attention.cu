// Gated linear attention: a per-head state S [D, V] that every token decays per key channel and
// adds an outer product to,
//
//     S_t = diag(alpha_t) S_(t-1) + k_t v_t^T          o_t = S_t^T q_t
//
// with the state, the decays and every product of the recurrence in 32-bit arithmetic: multiply-adds, or, for states of 128 x 128
// and a decay per key channel, sums of bfloat16 products on the tensor cores that are as near (gla_scan_mma_kernel).
//
// gla_decay_kernel   alpha[t, c] = exp(ln(sigmoid(z)) / tau),  z = w2[c, :] . a[t, :] + b2[c]: the second
//                    half of a low-rank decay projection, kept out of the matrix-product path so that its
//                    input is never rounded.  A block takes 32 tokens x 128 channels and reads its slice
//                    of the (transposed) weights once.
// gla_scan_kernel    one block per (work item, head) walks the item's tokens in order.  Thread (dg, v)
//                    keeps rows dg*R .. dg*R+R-1 of column v of the state in registers; tokens are
//                    staged through shared memory sixteen at a time (no barrier between the tokens of a
//                    batch: each row group leaves its share of o in shared memory).  Epilogue per staged
//                    batch, a warp per token: the row groups' shares are added, then RMS norm of o over V,
//                    weight, output gate silu(g), scale, store in the compute dtype into a column range
//                    of the layer's output buffer.
//                    Three modes make long prompt portions parallel over chunks of tokens:
//                      FULL   state in from the request's slot, outputs, state out to the slot
//                             (single decoded tokens and short portions: one pass)
//                      LOCAL  state in = 0, no outputs; the chunk's own contribution L and its total
//                             decay A = prod alpha go to scratch
//                      OUT    state in from scratch (what gla_chain_kernel put there), outputs only
// gla_step_kernel    the same for entries of ONE token (decode steps): the state streams through, see there.
// gla_chain_kernel   per (long entry, head), over its chunks in order: scratch[c] <- S (the state that
//                    enters chunk c), S <- diag(A_c) S + L_c; at the end the slot's state <- S.
//
//
// The same kernels run every recurrence of that shape whose decay is one number per (token, head) or a
// constant per head (template SCALAR of the scan kernel; strides of `alpha` in the step kernel):
//
//     S_t = a_t S_(t-1) + e_t k_t v_t^T     [ n_t = a_t n_(t-1) + e_t k_t ]      o_t = S_t^T q_t [ / den_t ]
//
// with an optional input scale e per (token, head) and an optional normaliser vector n kept beside S (an
// extra column of the state whose "value" is 1): den_t = max(|n_t . q_t|, floor_t) + 1e-6 with a floor per
// (token, head).  Retention: a = a constant per head, no e, no n.  A matrix memory with exponential
// gates: a, e and floor come from recur_gates_kernel (prompt portions) or are made inside the step
// kernel (decode steps).  The epilogue's output norm takes a weight [V] shared by the heads, a weight
// per head, or none, and its gate is silu or a sigmoid.  A head's state in a slot is S [D, V], then
// n [D] when there is one, then whatever else the mixer keeps there (`state_head_stride`).
//
// A position's output depends on how a prompt is cut only through the order of 32-bit additions.
#include "split_mma.cuh"
#include <type_traits>

#define GLA_TB 16          // tokens staged at a time
#define GLA_FULL 0
#define GLA_LOCAL 1
#define GLA_OUT 2

#define GLA_DECAY_TOKENS 32       // tokens a block of the decay kernel takes
#define GLA_DECAY_CHANNELS 128    // and channels (one a thread)

// w2t is the second half of the decay projection TRANSPOSED, [rank, channels]: thread c of a block reads
// w2t[j][c] for every j once (neighbouring threads read neighbouring words) and applies it to all of the
// block's tokens, whose inputs a[t][:] sit in shared memory.
__global__ void gla_decay_kernel(const float* __restrict__ proj, long long stride, int a_off, int rank,
                                 const float* __restrict__ w2t, const float* __restrict__ b2, float inv_tau,
                                 float* __restrict__ la, int channels, int num_tokens) {
    pdl_begin();
    extern __shared__ float a[];                    // [GLA_DECAY_TOKENS][rank]
    const int t0 = blockIdx.x * GLA_DECAY_TOKENS;
    const int nt = min(GLA_DECAY_TOKENS, num_tokens - t0);
    for (int idx = threadIdx.x; idx < nt * rank; idx += blockDim.x) {
        const int t = idx / rank, j = idx - t * rank;
        a[idx] = proj[static_cast<size_t>(t0 + t) * stride + a_off + j];
    }
    __syncthreads();
    const int c = blockIdx.y * GLA_DECAY_CHANNELS + threadIdx.x;
    if (c >= channels) return;
    float z[GLA_DECAY_TOKENS];
    const float bias = b2 ? b2[c] : 0.0f;
#pragma unroll
    for (int t = 0; t < GLA_DECAY_TOKENS; ++t) z[t] = bias;
    int j = 0;
    for (; j + 16 <= rank; j += 16) {              // sixteen weights in flight: a decode step's few blocks are bound by
        float w[16];                                // the latency of these loads, not by their bytes
#pragma unroll
        for (int u = 0; u < 16; ++u) w[u] = w2t[static_cast<size_t>(j + u) * channels + c];
#pragma unroll
        for (int u = 0; u < 16; ++u)
#pragma unroll
            for (int t = 0; t < GLA_DECAY_TOKENS; ++t)
                if (t < nt) z[t] += w[u] * a[t * rank + j + u];
    }
    for (; j < rank; ++j) {
        const float w = w2t[static_cast<size_t>(j) * channels + c];
#pragma unroll
        for (int t = 0; t < GLA_DECAY_TOKENS; ++t)
            if (t < nt) z[t] += w * a[t * rank + j];
    }
#pragma unroll
    for (int t = 0; t < GLA_DECAY_TOKENS; ++t)
        if (t < nt) {
            // ln(sigmoid(z)) without overflow on either side
            const float ls = fminf(z[t], 0.0f) - log1pf(expf(-fabsf(z[t])));
            la[static_cast<size_t>(t0 + t) * channels + c] = expf(ls * inv_tau);      // alpha = sigmoid(z)^(1/tau)
        }
}

typedef unsigned long long gla_pair;
__device__ __forceinline__ gla_pair gla_mul2(gla_pair a, gla_pair b) {
    gla_pair r;
    asm("mul.rn.f32x2 %0, %1, %2;\n" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ gla_pair gla_fma2(gla_pair a, gla_pair b, gla_pair c) {
    gla_pair r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;\n" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ gla_pair gla_both(float lo, float hi) {
    gla_pair r;
    asm("mov.b64 %0, {%1, %2};\n" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ float2 gla_split(gla_pair a) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;\n" : "=f"(r.x), "=f"(r.y) : "l"(a));
    return r;
}

// The same where channels come in fours: a thread makes 4 channels x 8 tokens, so that a weight load and two loads of four
// inputs (kept token-minor in shared memory) feed 32 multiply-adds; one thread a channel needed a shared load for every
// multiply-add.  The sums run over the rank in the same order.  2,048 tokens x 2,048 channels of rank 64: 71 -> 36 us,
// 29 with one form of ln(sigmoid(z)) for either sign (the two sides of a branch were both walked), 21 with the inputs laid out so that
// storing them token-minor meets every bank once (32 lanes had met one), without a division per input, and two tokens an instruction;
// 700 tokens 24 -> 11.  Issue bounds it, and half of what is issued are the exponentials and logarithms of a 2,048 x 2,048 result.
// Six to eight blocks an SM (fewer registers, weights four at a time) 22 to 26.
__global__ void __launch_bounds__(128, 5) gla_decay_tiled_kernel(const float* __restrict__ proj, long long stride, int a_off, int rank,
                                                              const float* __restrict__ w2t, const float* __restrict__ b2,
                                                              float inv_tau, float* __restrict__ la, int channels, int num_tokens) {
    pdl_begin();
    extern __shared__ __align__(16) float a[];      // [rank][GLA_DECAY_TOKENS], a row's eights of tokens exchanged by its index
    const int t0 = blockIdx.x * GLA_DECAY_TOKENS;
    const int nt = min(GLA_DECAY_TOKENS, num_tokens - t0);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, tg = warp * 8;
    {   // a warp brings eight tokens, four inputs of each at a time: every bank once
        const int t = tg + (lane >> 2);
        const float* row = proj + static_cast<size_t>(t0 + min(t, nt - 1)) * stride + a_off;
#pragma unroll 8
        for (int j = lane & 3; j < rank; j += 4)
            a[j * GLA_DECAY_TOKENS + ((warp ^ (j & 3)) << 3) + (lane >> 2)] = t < nt ? row[j] : 0.0f;
    }
    __syncthreads();
    const int c = blockIdx.y * GLA_DECAY_CHANNELS + lane * 4;
    if (c >= channels) return;
    gla_pair z[4][4];                               // [tokens in twos][channel]
    const float4 bias = b2 ? *reinterpret_cast<const float4*>(b2 + c) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
    for (int t = 0; t < 4; ++t) {
        z[t][0] = gla_both(bias.x, bias.x);
        z[t][1] = gla_both(bias.y, bias.y);
        z[t][2] = gla_both(bias.z, bias.z);
        z[t][3] = gla_both(bias.w, bias.w);
    }
    auto add = [&](const float4 w, int j) {
        const ulonglong2* at = reinterpret_cast<const ulonglong2*>(a + j * GLA_DECAY_TOKENS + ((warp ^ (j & 3)) << 3));
        const ulonglong2 lo = at[0], hi = at[1];
        const gla_pair x[4] = {lo.x, lo.y, hi.x, hi.y}, w2[4] = {gla_both(w.x, w.x), gla_both(w.y, w.y), gla_both(w.z, w.z), gla_both(w.w, w.w)};
#pragma unroll
        for (int t = 0; t < 4; ++t)
#pragma unroll
            for (int i = 0; i < 4; ++i) z[t][i] = gla_fma2(w2[i], x[t], z[t][i]);
    };
    int j = 0;
    for (; j + 8 <= rank; j += 8) {
        float4 w[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) w[u] = *reinterpret_cast<const float4*>(w2t + static_cast<size_t>(j + u) * channels + c);
#pragma unroll
        for (int u = 0; u < 8; ++u) add(w[u], j + u);
    }
    for (; j < rank; ++j) add(*reinterpret_cast<const float4*>(w2t + static_cast<size_t>(j) * channels + c), j);
    auto decay = [&](float v) { return expf((fminf(v, 0.0f) - log1pf(expf(-fabsf(v)))) * inv_tau); };
#pragma unroll
    for (int t = 0; t < 8; ++t)
        if (tg + t < nt) {
            float r[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float2 two = gla_split(z[t / 2][i]);
                r[i] = decay(t & 1 ? two.y : two.x);
            }
            *reinterpret_cast<float4*>(la + static_cast<size_t>(t0 + tg + t) * channels + c) = make_float4(r[0], r[1], r[2], r[3]);
        }
}

extern "C" int llm_gla_decay(const float* proj, long long stride, int a_off, int rank, const float* w2t, const float* b2,
                             float tau, float* la, int num_tokens, int channels, uintptr_t stream) {
    if (num_tokens <= 0) return LLM_OK;
    if (rank <= 0 || channels <= 0 || !(tau > 0.0f) || rank > 1024) return LLM_REFUSED_SIZE;
    const dim3 grid((num_tokens + GLA_DECAY_TOKENS - 1) / GLA_DECAY_TOKENS,
                    (channels + GLA_DECAY_CHANNELS - 1) / GLA_DECAY_CHANNELS);
    if (grid.y > 65535) return LLM_REFUSED_SIZE;
    // From 16 rows on (fewer leave most of a thread's eight idle), and while the inputs fit 48 KB.  Both (us, this one first), at
    // 2,048 channels of rank 64: 8 tokens 15.0, 14.3; 16: 15.3, 16.2; 32: 16.6, 21.1; 256: 17.5, 23.1; 2,048: 39.6, 64.6; at 512
    // channels 14.7, 13.7; 15.1, 16.0; 16.4, 20.8; 16.7, 21.2; 20.0, 33.9.
    if (num_tokens >= 16 && channels % 4 == 0 && rank <= 384 && aligned16(w2t) && aligned16(la) && (!b2 || aligned16(b2))) {
        launch_pdl(gla_decay_tiled_kernel, grid, dim3(128), GLA_DECAY_TOKENS * rank * sizeof(float), reinterpret_cast<cudaStream_t>(stream),
                   proj, stride, a_off, rank, w2t, b2, 1.0f / tau, la, channels, num_tokens);
        return launch_status();
    }
    launch_pdl(gla_decay_kernel, grid, dim3(GLA_DECAY_CHANNELS), GLA_DECAY_TOKENS * rank * sizeof(float),
               reinterpret_cast<cudaStream_t>(stream), proj, stride, a_off, rank, w2t, b2, 1.0f / tau, la, channels,
               num_tokens);
    return launch_status();
}

__device__ __forceinline__ void gla_cp16(float* smem_dst, const float* src) {
    const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(smem_dst));
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src));
}

// items: int32 [n, 4] = (entry, first row in the batch, tokens, index of the item's scratch) or null: item i
// is entry i, all of it.  `alpha` [T, H*D] are the decays themselves (what gla_decay_kernel writes).
// What varies between the recurrences that share these kernels (see the top of the file).
struct RecurOpts {
    long long a_tok, a_head;          // SCALAR: alpha index = token * a_tok + head * a_head
    const float* kscale;              // SCALAR: e per (token, head) at token * H + head, or null
    const float* nfloor;              // floor per (token, head): non-null means the state has a normaliser column
    int norm_stride;                  // output norm weight index = head * norm_stride + channel (0: shared by the heads)
    int gate_kind;                    // 0 none, 1 sigmoid, 2 silu
    long long state_head_stride, state_slot_stride;
};

__device__ __forceinline__ float recur_gate(float g, int kind) {
    if (kind == 0) return 1.0f;
    const float sg = 1.0f / (1.0f + expf(-g));
    return kind == 1 ? sg : g * sg;
}

template <int R, int MAX_THREADS, typename TO, bool SCALAR>
__global__ void __launch_bounds__(MAX_THREADS) gla_scan_kernel(
    const float* __restrict__ proj, long long stride, int q_off, int k_off, int v_off, int g_off,
    const float* __restrict__ alpha, const float* __restrict__ norm_w, float eps, float q_scale, float out_scale,
    TO* __restrict__ out, long long out_stride, int out_off, float* __restrict__ state,
    const int32_t* __restrict__ entry_slot, const int32_t* __restrict__ entry_q_start,
    const int32_t* __restrict__ entry_q_len, const int32_t* __restrict__ items, int mode,
    float* __restrict__ scratch_s, float* __restrict__ scratch_a, int H, int D, int V, int DG, int vec,
    const RecurOpts opt) {
    pdl_begin();
    extern __shared__ __align__(16) float smem[];
    const int h = blockIdx.y;
    int entry, row0, count, sidx;
    if (items) {
        entry = items[4 * blockIdx.x];
        if (entry < 0) return;                       // padding of a work list
        row0 = items[4 * blockIdx.x + 1];
        count = items[4 * blockIdx.x + 2];
        sidx = items[4 * blockIdx.x + 3];
    } else {
        entry = blockIdx.x;
        row0 = entry_q_start[entry];
        count = entry_q_len[entry];
        sidx = entry;
    }
    const int tid = threadIdx.x, nthreads = blockDim.x;
    // thread (dg, v) for tid < VC * DG; the block is rounded up to whole warps and the rest only help to stage.
    // Column V (when there is one) is the normaliser n, whose "value" is 1.
    // (what only the SCALAR recurrences use folds away in the per-channel instantiation, whose register budget is tight)
    const float* nfloor = SCALAR ? opt.nfloor : nullptr;
    const int norm_stride = SCALAR ? opt.norm_stride : 0;
    const int gate_kind = SCALAR ? opt.gate_kind : 2;
    const long long head_stride = SCALAR ? opt.state_head_stride : static_cast<long long>(D) * V;
    const long long slot_stride = SCALAR ? opt.state_slot_stride : static_cast<long long>(H) * D * V;
    const int VC = V + (nfloor ? 1 : 0);
    const bool active = tid < VC * DG;
    const int v = active ? tid % VC : 0, dg = active ? tid / VC : 0;
    // two staging buffers of [TB][D] queries, keys, decays and [TB][V] values ([TB] decays and [TB] input
    // scales instead of [TB][D] decays when SCALAR): batch b+1 is copied in (cp.async, sixteen bytes at a
    // time) while batch b is worked on
    const int buf_floats = SCALAR ? GLA_TB * (2 * D + V + 2) : GLA_TB * (3 * D + V);
    float* part = smem + 2 * buf_floats;            // [TB][DG][VC]: each row group's share of o, added up in the epilogue
    const size_t HD = static_cast<size_t>(H) * D;
    const bool outputs = mode != GLA_LOCAL;
    // a thread whose R rows all exist reads its decays, keys and queries sixteen bytes at a time
    const bool whole = active && dg * R + R <= D && (D & 3) == 0;

    float S[R];
    float* slot_state = state + static_cast<size_t>(entry_slot[entry]) * slot_stride + h * head_stride;
    const size_t chunk_state = static_cast<size_t>(D) * VC;     // a chunk's scratch holds S and n, nothing else
    const float* s_in = mode == GLA_FULL ? slot_state
                        : (mode == GLA_OUT ? scratch_s + (static_cast<size_t>(sidx) * H + h) * chunk_state : nullptr);
    // element (d, v) of a head's state: S[d][v] for v < V, then n[d]
    auto at = [&](int d) { return v < V ? static_cast<size_t>(d) * V + v : static_cast<size_t>(D) * V + d; };
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int d = dg * R + r;
        S[r] = (s_in && active && d < D) ? s_in[at(d)] : 0.0f;
    }

    auto stage = [&](int done, int buf) {
        const int nb = min(GLA_TB, count - done);
        const size_t base = static_cast<size_t>(row0 + done);
        float* bq = smem + buf * buf_floats;
        float* bk = bq + GLA_TB * D;
        float* ba = bk + GLA_TB * D;
        float* bv = SCALAR ? ba : ba + GLA_TB * D;
        if (SCALAR) {                                // the batch's decays and input scales: two numbers a token
            float* bs = bv + GLA_TB * V;
            if (tid < nb) {
                bs[tid] = alpha[(base + tid) * opt.a_tok + h * opt.a_head];
                bs[GLA_TB + tid] = opt.kscale ? opt.kscale[(base + tid) * H + h] : 1.0f;
            }
        }
        if (vec) {
            const int d4 = D >> 2, v4 = V >> 2;
            for (int idx = tid; idx < nb * d4; idx += nthreads) {
                const int tok = idx / d4, c = (idx - tok * d4) << 2;
                const float* pr = proj + (base + tok) * stride + h * D + c;
                gla_cp16(bk + tok * D + c, pr + k_off);
                if (!SCALAR) gla_cp16(ba + tok * D + c, alpha + (base + tok) * HD + h * D + c);
                if (outputs) gla_cp16(bq + tok * D + c, pr + q_off);
            }
            for (int idx = tid; idx < nb * v4; idx += nthreads) {
                const int tok = idx / v4, c = (idx - tok * v4) << 2;
                gla_cp16(bv + tok * V + c, proj + (base + tok) * stride + v_off + h * V + c);
            }
            asm volatile("cp.async.commit_group;\n" ::);
        } else {
            for (int idx = tid; idx < nb * D; idx += nthreads) {
                const int tok = idx / D, d = idx - tok * D;
                const float* pr = proj + (base + tok) * stride + h * D + d;
                bk[idx] = pr[k_off];
                if (!SCALAR) ba[idx] = alpha[(base + tok) * HD + h * D + d];
                if (outputs) bq[idx] = pr[q_off];
            }
            for (int idx = tid; idx < nb * V; idx += nthreads) {
                const int tok = idx / V, c = idx - tok * V;
                bv[idx] = proj[(base + tok) * stride + v_off + h * V + c];
            }
        }
    };

    stage(0, 0);
    for (int done = 0, b = 0; done < count; done += GLA_TB, ++b) {
        const int nb = min(GLA_TB, count - done);
        const size_t base = static_cast<size_t>(row0 + done);
        const bool more = done + GLA_TB < count;
        if (more) stage(done + GLA_TB, (b + 1) & 1);
        if (vec) {
            if (more) asm volatile("cp.async.wait_group 1;\n" ::: "memory");
            else asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        }
        __syncthreads();
        const float* sq = smem + (b & 1) * buf_floats;
        const float* sk = sq + GLA_TB * D;
        const float* sa = sk + GLA_TB * D;
        const float* sv = SCALAR ? sa : sa + GLA_TB * D;
        const float* ss2 = sv + GLA_TB * V;         // SCALAR: [TB] decays, [TB] input scales
        for (int tok = 0; tok < nb; ++tok) {
            float vt = v < V ? sv[tok * V + v] : 1.0f;
            const float* a = sa + tok * D + dg * R;
            const float* k = sk + tok * D + dg * R;
            const float* q = sq + tok * D + dg * R;
            float p0 = 0.0f, p1 = 0.0f;
            if (SCALAR) {
                const float a1 = ss2[tok];
                vt *= ss2[GLA_TB + tok];
                if (whole) {
                    const float4* k4 = reinterpret_cast<const float4*>(k);
                    const float4* q4 = reinterpret_cast<const float4*>(q);
#pragma unroll
                    for (int r = 0; r < R; r += 4) {
                        const float4 kv = k4[r >> 2];
                        S[r] = a1 * S[r] + kv.x * vt;
                        S[r + 1] = a1 * S[r + 1] + kv.y * vt;
                        S[r + 2] = a1 * S[r + 2] + kv.z * vt;
                        S[r + 3] = a1 * S[r + 3] + kv.w * vt;
                        if (outputs) {
                            const float4 qv = q4[r >> 2];
                            p0 += S[r] * qv.x;
                            p1 += S[r + 1] * qv.y;
                            p0 += S[r + 2] * qv.z;
                            p1 += S[r + 3] * qv.w;
                        }
                    }
                } else if (active) {
#pragma unroll
                    for (int r = 0; r < R; ++r)
                        if (dg * R + r < D) {
                            S[r] = a1 * S[r] + k[r] * vt;
                            if (outputs) p0 += S[r] * q[r];
                        }
                }
            } else if (whole) {
                const float4* a4 = reinterpret_cast<const float4*>(a);
                const float4* k4 = reinterpret_cast<const float4*>(k);
                const float4* q4 = reinterpret_cast<const float4*>(q);
                if (outputs) {
#pragma unroll
                    for (int r = 0; r < R; r += 4) {
                        const float4 av = a4[r >> 2], kv = k4[r >> 2], qv = q4[r >> 2];
                        S[r] = av.x * S[r] + kv.x * vt;             p0 += S[r] * qv.x;
                        S[r + 1] = av.y * S[r + 1] + kv.y * vt;     p1 += S[r + 1] * qv.y;
                        S[r + 2] = av.z * S[r + 2] + kv.z * vt;     p0 += S[r + 2] * qv.z;
                        S[r + 3] = av.w * S[r + 3] + kv.w * vt;     p1 += S[r + 3] * qv.w;
                    }
                } else {
#pragma unroll
                    for (int r = 0; r < R; r += 4) {
                        const float4 av = a4[r >> 2], kv = k4[r >> 2];
                        S[r] = av.x * S[r] + kv.x * vt;
                        S[r + 1] = av.y * S[r + 1] + kv.y * vt;
                        S[r + 2] = av.z * S[r + 2] + kv.z * vt;
                        S[r + 3] = av.w * S[r + 3] + kv.w * vt;
                    }
                }
            } else if (active) {
#pragma unroll
                for (int r = 0; r < R; r += 2) {
                    if (dg * R + r < D) {
                        S[r] = a[r] * S[r] + k[r] * vt;
                        if (outputs) p0 += S[r] * q[r];
                    }
                    if (dg * R + r + 1 < D) {
                        S[r + 1] = a[r + 1] * S[r + 1] + k[r + 1] * vt;
                        if (outputs) p1 += S[r + 1] * q[r + 1];
                    }
                }
            }
            if (outputs && active) part[(tok * DG + dg) * VC + v] = p0 + p1;
        }
        __syncthreads();
        if (outputs) {                              // a warp per token: add the row groups, norm over V, weight, gate, scale
            const int warp = tid >> 5, lane = tid & 31, nwarps = nthreads >> 5;
            for (int tok = warp; tok < nb; tok += nwarps) {
                float* o = part + tok * DG * VC;
                float mul = q_scale;                // q = W_q x * q_scale, applied to the finished sum
                if (nfloor) {                       // the normaliser: n . q, floored, divides the output
                    float nq = o[V];
                    for (int g2 = 1; g2 < DG; ++g2) nq += o[g2 * VC + V];
                    nq *= q_scale;
                    mul = q_scale / (fmaxf(fabsf(nq), nfloor[(base + tok) * H + h]) + 1e-6f);
                }
                __syncwarp();
                float ss = 0.0f;
                for (int c = lane; c < V; c += 32) {
                    float sum = o[c];
                    for (int g2 = 1; g2 < DG; ++g2) sum += o[g2 * VC + c];
                    sum *= mul;
                    o[c] = sum;
                    ss += sum * sum;
                }
                ss = warp_sum(ss);
                const float inv = 1.0f / sqrtf(ss / static_cast<float>(V) + eps);
                const float* gr = proj + (base + tok) * stride + g_off + h * V;
                const float* nw = norm_w + h * norm_stride;
                TO* orow = out + (base + tok) * out_stride + out_off + h * V;
                for (int c = lane; c < V; c += 32)
                    orow[c] = from_f32<TO>(o[c] * inv * ((SCALAR && !norm_w) ? 1.0f : nw[c]) * recur_gate(gr[c], gate_kind) * out_scale);
            }
        }
        __syncthreads();                            // this buffer is filled again two batches on
    }
    if (mode == GLA_OUT) return;
    float* s_out = mode == GLA_FULL ? slot_state : scratch_s + (static_cast<size_t>(sidx) * H + h) * chunk_state;
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int d = dg * R + r;
        if (active && d < D) s_out[at(d)] = S[r];
    }
    if (mode == GLA_LOCAL) {                        // the chunk's total decay per key channel
        for (int d = tid; d < D; d += nthreads) {
            float prod = 1.0f;
            for (int tok = 0; tok < count; ++tok)
                prod *= SCALAR ? alpha[(static_cast<size_t>(row0) + tok) * opt.a_tok + h * opt.a_head]
                               : alpha[(static_cast<size_t>(row0) + tok) * HD + h * D + d];
            scratch_a[(static_cast<size_t>(sidx) * H + h) * D + d] = prod;
        }
    }
}

// ---- the per-channel scan for states of 64 or 128 rows, register-tiled --------------------------------------------
// In the kernel above a thread owns one column, so every product of the recurrence needs its share of a 16-byte shared load
// of decays, keys and queries that serves that column only: 24 loads (96 clocks of the 128-byte shared-memory path) for 96
// multiply-adds a token and thread at R = 32.  Here a thread owns RR rows x 8 columns: one load of four decays, keys or
// queries serves eight columns, 3 RR / 4 + 2 loads for 24 RR multiply-adds, and packed two-wide arithmetic (two rows an
// instruction) halves what has to be issued.  Sixteen lanes hold the rows of a column (a lane's rows are 4 rg .. + 3 and, at
// 128 rows, 64 + 4 rg .. + 3, so that a quarter-warp's loads are contiguous); their shares of o are added by halving
// exchanges, two tokens at a time: fifteen shuffles for sixteen sums, one of which each lane leaves in shared memory.  A block is 2 V
// threads, two blocks an SM.  Same modes, staging and epilogue as above; every state element is updated by the same
// operations in the same order (k v, then decay times state plus that), only o's sum runs over the rows in another order.
// 2,048 tokens, 16 heads of 128 x 128: local pass and output pass 133 and 217 us -> 66 and 113 us
// (161 with one token's sums at a time and the gates read from global memory in the epilogue).  Other states, 16 heads (us, the
// kernel above and this one): one pass over 64 tokens; local and output pass over 2,048:
//   64 x 32    29, 30;  42, 17;  53, 40        128 x 32    28, 40;  59, 25;  68, 73
//   64 x 64    30, 24;  50, 25;  63, 41        128 x 64    34, 34;  87, 37;  108, 72
//   64 x 128   37, 27;  86, 45;  117, 71       128 x 128   50, 41;  133, 66; 217, 113
// so 32 columns (blocks of 64 threads) stay with the kernel above, but for the local pass and, at 64 rows, the
// output pass.

template <int RR, int MODE, typename TO>
__global__ void __launch_bounds__(256, 2) gla_scan_tiled_kernel(
    const float* __restrict__ proj, long long stride, int q_off, int k_off, int v_off, int g_off,
    const float* __restrict__ alpha, const float* __restrict__ norm_w, float eps, float q_scale, float out_scale,
    TO* __restrict__ out, long long out_stride, int out_off, float* __restrict__ state,
    const int32_t* __restrict__ entry_slot, const int32_t* __restrict__ entry_q_start,
    const int32_t* __restrict__ entry_q_len, const int32_t* __restrict__ items,
    float* __restrict__ scratch_s, float* __restrict__ scratch_a, int H, int V) {
    pdl_begin();
    constexpr int D = 16 * RR, Q4 = RR / 4;          // Q4: groups of four rows a lane holds
    constexpr bool OUTPUTS = MODE != GLA_LOCAL;
    extern __shared__ __align__(16) float smem[];
    const int h = blockIdx.y;
    int entry, row0, count, sidx;
    if (items) {
        entry = items[4 * blockIdx.x];
        if (entry < 0) return;                       // padding of a work list
        row0 = items[4 * blockIdx.x + 1];
        count = items[4 * blockIdx.x + 2];
        sidx = items[4 * blockIdx.x + 3];
    } else {
        entry = blockIdx.x;
        row0 = entry_q_start[entry];
        count = entry_q_len[entry];
        sidx = entry;
    }
    const int tid = threadIdx.x, nthreads = blockDim.x, warp = tid >> 5, lane = tid & 31;
    const int rg = lane & 15, col0 = (tid >> 4) * 8;
    const int buf_floats = GLA_TB * (3 * D + 2 * V);
    float* part = smem + 2 * buf_floats;             // [TB][V]
    const size_t HD = static_cast<size_t>(H) * D, per = static_cast<size_t>(D) * V;
    float* slot_state = state + (static_cast<size_t>(entry_slot[entry]) * H + h) * per;
    const float* s_in = MODE == GLA_FULL ? slot_state : MODE == GLA_OUT ? scratch_s + (static_cast<size_t>(sidx) * H + h) * per : nullptr;
    gla_pair S[RR / 2][8], A[RR / 2];
    auto row_of = [&](int p) { return 64 * (p >> 1) + 4 * rg + 2 * (p & 1); };       // the first of a pair's two rows
#pragma unroll
    for (int p = 0; p < RR / 2; ++p) {
        A[p] = gla_both(1.0f, 1.0f);
        float lo[8], hi[8];
        if (MODE == GLA_LOCAL) {
#pragma unroll
            for (int c = 0; c < 8; ++c) lo[c] = hi[c] = 0.0f;
        } else {
            load8(s_in + static_cast<size_t>(row_of(p)) * V + col0, lo);
            load8(s_in + static_cast<size_t>(row_of(p) + 1) * V + col0, hi);
        }
#pragma unroll
        for (int c = 0; c < 8; ++c) S[p][c] = gla_both(lo[c], hi[c]);
    }
    auto stage = [&](int done, int buf) {
        const int nb = min(GLA_TB, count - done);
        const size_t base = static_cast<size_t>(row0 + done);
        float* bq = smem + buf * buf_floats;
        float* bk = bq + GLA_TB * D;
        float* ba = bk + GLA_TB * D;
        float* bv = ba + GLA_TB * D;
        for (int idx = tid; idx < nb * (D / 4); idx += nthreads) {
            const int tok = idx / (D / 4), c = (idx % (D / 4)) << 2;
            const float* pr = proj + (base + tok) * stride + h * D + c;
            gla_cp16(bk + tok * D + c, pr + k_off);
            gla_cp16(ba + tok * D + c, alpha + (base + tok) * HD + h * D + c);
            if (OUTPUTS) gla_cp16(bq + tok * D + c, pr + q_off);
        }
        const int v4 = V >> 2;
        for (int idx = tid; idx < nb * v4; idx += nthreads) {
            const int tok = idx / v4, c = (idx - tok * v4) << 2;
            gla_cp16(bv + tok * V + c, proj + (base + tok) * stride + v_off + h * V + c);
            if (OUTPUTS) gla_cp16(bv + (GLA_TB + tok) * V + c, proj + (base + tok) * stride + g_off + h * V + c);      // the gates
        }
        asm volatile("cp.async.commit_group;\n" ::);
    };
    stage(0, 0);
    for (int done = 0, b = 0; done < count; done += GLA_TB, ++b) {
        const int nb = min(GLA_TB, count - done);
        const size_t base = static_cast<size_t>(row0 + done);
        if (done + GLA_TB < count) {
            stage(done + GLA_TB, (b + 1) & 1);
            asm volatile("cp.async.wait_group 1;\n" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        }
        __syncthreads();
        const float* sq = smem + (b & 1) * buf_floats;
        const float* sk = sq + GLA_TB * D;
        const float* sa = sk + GLA_TB * D;
        const float* sv = sa + GLA_TB * D;
        // two tokens at a time: their sixteen sums over the rows go through one chain of exchanges
        for (int tok0 = 0; tok0 < nb; tok0 += 2) {
            float o[16];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int tok = tok0 + u;
                if (u == 1 && tok >= nb) {
#pragma unroll
                    for (int c = 0; c < 8; ++c) o[8 + c] = 0.0f;
                    break;
                }
                gla_pair k[RR / 2], a[RR / 2], q[RR / 2];
#pragma unroll
                for (int g = 0; g < Q4; ++g) {
                    const ulonglong2 kk = *reinterpret_cast<const ulonglong2*>(sk + tok * D + 64 * g + 4 * rg);
                    const ulonglong2 aa = *reinterpret_cast<const ulonglong2*>(sa + tok * D + 64 * g + 4 * rg);
                    k[2 * g] = kk.x; k[2 * g + 1] = kk.y;
                    a[2 * g] = aa.x; a[2 * g + 1] = aa.y;
                    if (OUTPUTS) {
                        const ulonglong2 qq = *reinterpret_cast<const ulonglong2*>(sq + tok * D + 64 * g + 4 * rg);
                        q[2 * g] = qq.x; q[2 * g + 1] = qq.y;
                    }
                }
                float v[8];
                load8(sv + tok * V + col0, v);
#pragma unroll
                for (int c = 0; c < 8; ++c) {
                    const gla_pair vv = gla_both(v[c], v[c]);
                    gla_pair share = 0;
#pragma unroll
                    for (int p = 0; p < RR / 2; ++p) {
                        S[p][c] = gla_fma2(a[p], S[p][c], gla_mul2(k[p], vv));
                        if (OUTPUTS) share = p == 0 ? gla_mul2(S[p][c], q[p]) : gla_fma2(S[p][c], q[p], share);
                    }
                    if (OUTPUTS) {
                        const float2 t = gla_split(share);
                        o[8 * u + c] = t.x + t.y;
                    }
                }
                if (MODE == GLA_LOCAL) {             // the chunk's total decay per key channel
#pragma unroll
                    for (int p = 0; p < RR / 2; ++p) A[p] = gla_mul2(A[p], a[p]);
                }
            }
            if (OUTPUTS) {
#pragma unroll
                for (int off = 8, n = 8; n >= 1; off >>= 1, n >>= 1)
#pragma unroll
                    for (int i = 0; i < 8; ++i)
                        if (i < n) {
                            const bool up = (lane & off) != 0;
                            const float send = up ? o[i] : o[i + n], keep = up ? o[i + n] : o[i];
                            o[i] = keep + __shfl_xor_sync(0xffffffffu, send, off);
                        }
                const int tok = tok0 + (rg >> 3);     // lane rg holds column rg % 8 of token rg / 8
                if (tok < nb) part[tok * V + col0 + (rg & 7)] = o[0];
            }
        }
        __syncthreads();
        if (OUTPUTS) {                               // a warp per token: norm over V, weight, gate, scale
            for (int tok = warp; tok < nb; tok += nthreads >> 5) {
                float* o = part + tok * V;
                float ss = 0.0f;
                for (int c = lane; c < V; c += 32) {
                    const float x = o[c] * q_scale;
                    ss += x * x;
                }
                const float inv = q_scale / sqrtf(warp_sum(ss) / static_cast<float>(V) + eps) * out_scale;
                const float* gr = sv + (GLA_TB + tok) * V;
                TO* orow = out + (base + tok) * out_stride + out_off + h * V;
                for (int c = lane; c < V; c += 32) orow[c] = from_f32<TO>(o[c] * inv * norm_w[c] * recur_gate(gr[c], 2));
            }
            // the next batch's shares are written after its first barrier; this buffer, whose gates were just read, is filled
            // again by the next batch's staging: every warp must be done with it
            __syncthreads();
        }
    }
    if (MODE == GLA_OUT) return;
    float* s_out = MODE == GLA_FULL ? slot_state : scratch_s + (static_cast<size_t>(sidx) * H + h) * per;
#pragma unroll
    for (int p = 0; p < RR / 2; ++p) {
        float lo[8], hi[8];
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            const float2 t = gla_split(S[p][c]);
            lo[c] = t.x; hi[c] = t.y;
        }
        store8(s_out + static_cast<size_t>(row_of(p)) * V + col0, lo);
        store8(s_out + static_cast<size_t>(row_of(p) + 1) * V + col0, hi);
        if (MODE == GLA_LOCAL && col0 == 0) {
            const float2 t = gla_split(A[p]);
            float* to = scratch_a + (static_cast<size_t>(sidx) * H + h) * D + row_of(p);
            to[0] = t.x; to[1] = t.y;
        }
    }
}

// A block is alone on its SM while there are no more of them than SMs: two walk side by side at half the pace, and the
// hardware doubles them up where blocks of the kernel in front still sit on the others.  128 x 128, 128 blocks: one pass over eight
// requests of 64 tokens 65 -> 42 us, the output pass over 512 tokens 56 -> 36.
#define GLA_ALONE_BLOCKS 148
#define GLA_ALONE_SMEM (116 * 1024)
static bool gla_tiled_takes(int D, int V, int mode) {
    static int rows_forced = -1;                   // LLM_GLA_ROWS asks for the kernel above
    if (rows_forced < 0) rows_forced = getenv("LLM_GLA_ROWS") != nullptr;
    if (rows_forced || (D != 64 && D != 128)) return false;
    return V == 64 || V == 128 || (V == 32 && (mode == GLA_LOCAL || (mode == GLA_OUT && D == 64)));
}

// ---- the per-channel scan for states of 128 x 128, on the tensor cores ---------------------------------------------
// Thirty-two tokens at a time (64 without outputs) the recurrence is four products.  With f_t the product of the decays behind token t up to the
// batch's end, b the product of all of them, k'_t = f_t k_t, q'_t = q_t / f_t:
//
//     o_t = (diag(b) S)^T q'_t + sum over s <= t of (q'_t . k'_s) v_s          S <- diag(b) S + sum over s of k'_s v_s^T
//
// (b / f_t is the decays up to t; q'_t . k'_s is q_t . k_s with the decays between them.)  Every product is of float32 values as
// sums of three bfloat16 values, six products with float32 accumulation (split_mma.cuh): what is left out is 2^-24 of a
// product, and the terms that are not the largest have accumulators of their own, since the tensor cores cut what they add.
// Two blocks of eight warps an SM, so that one's loads and preparations hide behind the other's products.  A thread loads four
// channels of four tokens of everything at once; the products of the decays of every four tokens go through shared memory, then
// k', q' and v stay there as planes of bfloat16.  A warp makes sixteen columns of the outputs and of the state, whose values come
// from memory as they are needed, transposed, as left operands.
// A batch whose decays multiply to less than 2^-60 in some channel (q' would leave float32's range in the end), or that holds values
// beyond 2^30, infinities or NaN (a masked weight of zero times one of them is NaN), walks token by token as the kernels above do.
// What bounds it: latency.  2,048 tokens of 16 heads, 512 items of 64 tokens, everything cold: local pass 72 -> 43 us, output pass
// 121 -> 94 (the register-tiled kernel above before); of the output pass's time the tensor pipe is busy for 29 %, two blocks an SM hide
// some of each other's waits for rows, state and shared memory, and at 128 registers a thread spills 184 bytes (88 in the local pass).
// Tried: 16 tokens a batch with the state kept in accumulators 92 for 82 back to back; 64 tokens a batch, one block of 16 warps an SM 87.
// Error against 64 bits (2-norm, 2,048 tokens, decays
// sigmoid(z)^(1/tau), tau 2, 8, 64): states 3.2, 4.0 and 6.1e-8, the kernel above 4.7, 7.4 and 17.3; outputs 10.2, 10.6 and 12.4e-8,
// and 13.0, 13.1 and 20.2.  With all sums of the states as the tensor cores cut them the states were 5.5, 6.0 and 7.2.
#define GM_D 128
#define GM_PITCH 136                 // of a row of a plane: eight rows of 16 bytes fall into all banks
#define GM_WP 40                     // of a row of weights
#define GM_OP 132                    // of a row of outputs
#define GM_LEAST 8.6736174e-19f      // 2^-60
#define GM_MOST 1.0737418e9f         // 2^30
#define GM_AHEAD 296                 // blocks that run at a time
// Tokens of a batch and bytes of shared memory, with outputs (three tensors of planes, the weights' planes and shares) and without
#define GM_TOKENS(outputs) ((outputs) ? 32 : 64)
#define GM_SMEM(outputs) ((outputs) ? 2 * (9 * 32 * GM_PITCH + 3 * 32 * GM_WP) + 4 * (32 * GM_D + GM_D) : 2 * 6 * 64 * GM_PITCH + 4 * GM_D)

// g sigmoid(g) by CUDA's division within 2 ulp, which gives 0 for divisors from 2^126 on: silu is below 1e-36 there, and stays NaN for
// minus infinity.  (The correctly rounded division: 2 us more of 94.)
__device__ __forceinline__ float gm_silu(float g) { return __fdividef(g, 1.0f + expf(-g)); }
__device__ __forceinline__ float4 gm_mul(float4 a, float4 b) { return make_float4(a.x * b.x, a.y * b.y, a.z * b.z, a.w * b.w); }
__device__ __forceinline__ float4 gm_fma(float4 a, float4 b, float4 c) {
    return make_float4(fmaf(a.x, b.x, c.x), fmaf(a.y, b.y, c.y), fmaf(a.z, b.z, c.z), fmaf(a.w, b.w, c.w));
}
// 1 / f by CUDA's division within 2 ulp; who needs it nearer has gm_rest1
__device__ __forceinline__ float4 gm_inverse(float4 f) {
    return make_float4(__fdividef(1.0f, f.x), __fdividef(1.0f, f.y), __fdividef(1.0f, f.z), __fdividef(1.0f, f.w));
}
// a b - p, exactly, where p is a b rounded
__device__ __forceinline__ float4 gm_rest(float4 a, float4 b, float4 p) {
    return make_float4(fmaf(a.x, b.x, -p.x), fmaf(a.y, b.y, -p.y), fmaf(a.z, b.z, -p.z), fmaf(a.w, b.w, -p.w));
}
// A product of many decays and what its roundings left out: f_t has up to 63 of them, which alone would be a larger error than a
// state that is decayed token by token has.
struct GmPair { float4 hi, lo; };
__device__ __forceinline__ GmPair gm_times(GmPair f, float4 a) {
    const float4 hi = gm_mul(f.hi, a);
    return {hi, gm_fma(f.lo, a, gm_rest(f.hi, a, hi))};
}
__device__ __forceinline__ GmPair gm_times(GmPair f, GmPair a) {
    const float4 hi = gm_mul(f.hi, a.hi);
    return {hi, gm_fma(f.hi, a.lo, gm_fma(f.lo, a.hi, gm_rest(f.hi, a.hi, hi)))};
}
// (1 - r hi) - r lo
__device__ __forceinline__ float4 gm_rest1(float4 r, GmPair f) {
    return make_float4(fmaf(-r.x, f.lo.x, fmaf(-r.x, f.hi.x, 1.0f)), fmaf(-r.y, f.lo.y, fmaf(-r.y, f.hi.y, 1.0f)),
                       fmaf(-r.z, f.lo.z, fmaf(-r.z, f.hi.z, 1.0f)), fmaf(-r.w, f.lo.w, fmaf(-r.w, f.hi.w, 1.0f)));
}
__device__ __forceinline__ bool gm_fits(float4 x) {
    return fabsf(x.x) <= GM_MOST && fabsf(x.y) <= GM_MOST && fabsf(x.z) <= GM_MOST && fabsf(x.w) <= GM_MOST;
}

template <int MODE, typename TO>
__global__ void __launch_bounds__(256, 2) gla_scan_mma_kernel(
    const float* __restrict__ proj, long long stride, int q_off, int k_off, int v_off, int g_off,
    const float* __restrict__ alpha, const float* __restrict__ norm_w, float eps, float q_scale, float out_scale,
    TO* __restrict__ out, long long out_stride, int out_off, float* __restrict__ state,
    const int32_t* __restrict__ entry_slot, const int32_t* __restrict__ entry_q_start,
    const int32_t* __restrict__ entry_q_len, const int32_t* __restrict__ items,
    float* __restrict__ scratch_s, float* __restrict__ scratch_a, int H) {
    pdl_begin();
    constexpr bool OUTPUTS = MODE != GLA_LOCAL;
    constexpr int D = GM_D, V = GM_D, T = GM_TOKENS(OUTPUTS), PLANE = T * GM_PITCH, GROUPS = T / 4, PER_WARP = GROUPS / 8;
    extern __shared__ __align__(16) unsigned char gm_smem[];
    const int h = blockIdx.y;
    int entry, row0, count, sidx;
    if (items) {
        entry = items[4 * blockIdx.x];
        if (entry < 0) return;                       // padding of a work list
        row0 = items[4 * blockIdx.x + 1];
        count = items[4 * blockIdx.x + 2];
        sidx = items[4 * blockIdx.x + 3];
    } else {
        entry = blockIdx.x;
        row0 = entry_q_start[entry];
        count = entry_q_len[entry];
        sidx = entry;
    }
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, lg = lane >> 2, lt = lane & 3;
    bf16* pq = reinterpret_cast<bf16*>(gm_smem);     // [3][T][136] each; queries with outputs only
    bf16* pk = pq + (OUTPUTS ? 3 * PLANE : 0);
    bf16* pv = pk + 3 * PLANE;
    bf16* pp = pv + 3 * PLANE;                       // with outputs: [3][32][40]
    float* part = reinterpret_cast<float*>(pp + (OUTPUTS ? 3 * T * GM_WP : 0));      // with outputs: [24][16][8] shares, then [32][128] gates
    float* bend = part + (OUTPUTS ? T * V : 0);      // [128], and the end: GM_SMEM
    float* prod4 = reinterpret_cast<float*>(pk);     // two of [T / 4][128], before the keys
    float* os = reinterpret_cast<float*>(pq);        // [32][132] outputs, where the queries were
    float* gates = part;
    float* walk_k = reinterpret_cast<float*>(gm_smem);                   // token by token: [T][128] keys, decays, values, queries,
    float *walk_a = walk_k + T * D, *walk_v = walk_a + T * D, *walk_q = walk_v + T * V;
    float* walk_o = walk_q + T * D;                  // [32][132] of outputs
    static_assert(4 * (OUTPUTS ? 4 * T * D + T * GM_OP : 3 * T * D) <= GM_SMEM(OUTPUTS) - 4 * D, "shared memory");
    const size_t HD = static_cast<size_t>(H) * D, per = static_cast<size_t>(D) * V;
    float* slot_state = state + (static_cast<size_t>(entry_slot[entry]) * H + h) * per;
    float* chunk_state = scratch_s + (static_cast<size_t>(sidx) * H + h) * per;
    const float* s_in = MODE == GLA_FULL ? slot_state : chunk_state;
    float* s_out = MODE == GLA_FULL ? slot_state : chunk_state;
    // fragments: rows of 8 x 8 matrices that this lane points at
    const int frow = (lane >> 4) * 8 + (lane & 7), fcol = ((lane >> 3) & 1) * 8;
    const int grow = fcol + (lane & 7), gcol = (lane >> 4) * 8;
    const int v0 = 16 * warp + lg;                   // a warp has columns 16 warp .. + 15 of the state
    for (int done = 0; done < count; done += T) {
        const int nb = min(T, count - done);
        const size_t base = static_cast<size_t>(row0 + done);
        const bool none = MODE == GLA_LOCAL && done == 0, more = done + T < count;      // no state in; a state out, if only for the next batch
        bool bad = false;
        {
            const int c = lane << 2;                 // four channels of four tokens, groups warp and, of 64 tokens, warp + 8
            const float4 zero = make_float4(0.0f, 0.0f, 0.0f, 0.0f), one = make_float4(1.0f, 1.0f, 1.0f, 1.0f);
            const float* rows = proj + base * stride + h * D + c;
            auto load = [&](int t, int off) { return t < nb ? *reinterpret_cast<const float4*>(rows + t * stride + off) : zero; };
            float4 a[PER_WARP][4], k[PER_WARP][4], v[4], q[4];
#pragma unroll
            for (int n = 0; n < PER_WARP; ++n)
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int t = 4 * (warp + 8 * n) + i;
                    a[n][i] = t < nb ? *reinterpret_cast<const float4*>(alpha + (base + t) * HD + h * D + c) : one;
                    k[n][i] = load(t, k_off);
                }
#pragma unroll
            for (int n = 0; n < PER_WARP; ++n) {
#pragma unroll
                for (int i = 0; i < 4; ++i) v[i] = load(4 * (warp + 8 * n) + i, v_off);
                GmPair f = {a[n][3], zero};
#pragma unroll
                for (int i = 2; i >= 0; --i) f = gm_times(f, a[n][i]);
                *reinterpret_cast<float4*>(prod4 + (warp + 8 * n) * D + c) = f.hi;
                *reinterpret_cast<float4*>(prod4 + (GROUPS + warp + 8 * n) * D + c) = f.lo;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    bad |= !gm_fits(v[i]);
                    split_store4(pv + (4 * (warp + 8 * n) + i) * GM_PITCH + c, PLANE, v[i]);
                }
            }
            if (OUTPUTS)
#pragma unroll
                for (int i = 0; i < 4; ++i) q[i] = load(4 * warp + i, q_off);
            __syncthreads();
            GmPair behind[PER_WARP];                 // decays behind the thread's four tokens
            {
                GmPair f = {one, zero};
                int g = GROUPS - 1;
#pragma unroll
                for (int n = PER_WARP - 1; n >= 0; --n) {
                    for (; g > warp + 8 * n; --g)
                        f = gm_times(f, GmPair{*reinterpret_cast<const float4*>(prod4 + g * D + c), *reinterpret_cast<const float4*>(prod4 + (GROUPS + g) * D + c)});
                    behind[n] = f;
                }
            }
            __syncthreads();                         // the keys' planes take the products' place
            float4 f;
#pragma unroll
            for (int n = PER_WARP - 1; n >= 0; --n) {
#pragma unroll
                for (int i = 3; i >= 0; --i) {
                    const int at = (4 * (warp + 8 * n) + i) * GM_PITCH + c;
                    const float4 x = k[n][i], kh = gm_mul(x, behind[n].hi);
                    bad |= !gm_fits(x);
                    split_store4(pk + at, PLANE, kh, gm_fma(x, behind[n].lo, gm_rest(x, behind[n].hi, kh)));
                    if (OUTPUTS) {
                        const float4 r = gm_inverse(behind[n].hi), qh = gm_mul(q[i], r);
                        bad |= !gm_fits(q[i]);
                        // 1 / (hi + lo) = r (1 + (1 - r hi) - r lo), as near as matters: r's own error too is in the bracket
                        split_store4(pq + at, PLANE, qh, gm_fma(qh, gm_rest1(r, behind[n]), gm_rest(q[i], r, qh)));
                    }
                    behind[n] = gm_times(behind[n], a[n][i]);
                }
            }
            f = make_float4(behind[0].hi.x + behind[0].lo.x, behind[0].hi.y + behind[0].lo.y, behind[0].hi.z + behind[0].lo.z, behind[0].hi.w + behind[0].lo.w);
            if (warp == 0) {
                *reinterpret_cast<float4*>(bend + c) = f;
                const float least = OUTPUTS ? GM_LEAST : 0.0f;
                bad |= !gm_fits(f) || !(f.x >= least && f.y >= least && f.z >= least && f.w >= least);
                if (MODE == GLA_LOCAL) {
                    float4* to = reinterpret_cast<float4*>(scratch_a + (static_cast<size_t>(sidx) * H + h) * D + c);
                    *to = done == 0 ? f : gm_mul(*to, f);
                }
            }
        }
        if (items && done == 0 && warp < 4 + OUTPUTS) {                // the rows of the block that an SM takes up next, on their way into the second-level cache
            const int at = blockIdx.y * gridDim.x + blockIdx.x + GM_AHEAD, later = at % gridDim.x, hh = at / gridDim.x;
            if (hh < H && items[4 * later] >= 0) {
                const size_t first = items[4 * later + 1];
                const int n = items[4 * later + 2];
                const float* from = (warp == 0 ? alpha : proj) + first * (warp == 0 ? HD : stride) + hh * D +
                                    (warp == 0 ? 0 : warp == 1 ? k_off : warp == 2 ? v_off : warp == 3 ? (OUTPUTS ? q_off : v_off) : g_off);
                for (int t = lane; t < n; t += 32)
                    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;\n" ::"l"(from + t * (warp == 0 ? HD : stride)), "r"(D * 4));
            }
        }
        const float* o0 = os;
        bool walk = __syncthreads_or(bad);
        if (!walk) {
            float ahead[2][4];                   // the state's next sixteen rows
            auto fetch = [&](int j) {
#pragma unroll
                for (int u = 0; u < 2; ++u)
#pragma unroll
                        for (int i = 0; i < 4; ++i) ahead[u][i] = s_in[static_cast<size_t>(16 * j + 8 * u + 2 * lt + (i & 1)) * V + v0 + 8 * (i >> 1)];
            };
            if (OUTPUTS) {
                fetch(0);
                // the weights q' . k' of the three pairs of token blocks, 8 keys a tile, a quarter of the channels a unit
                for (int unit = warp; unit < 24; unit += 8) {
                    const int tile = unit >> 2, i = tile < 2 ? 0 : 1, s0 = 8 * (tile - 2 * i), d = 32 * (unit & 3);
                    float w[4] = {}, ws[2][4] = {};
                    unsigned y[3][4];                // 8 keys, 32 channels
#pragma unroll
                    for (int p = 0; p < 3; ++p) ldmatrix_x4(y[p], pk + p * PLANE + (s0 + (lane & 7)) * GM_PITCH + d + 8 * (lane >> 3));
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        unsigned x[3][4];
#pragma unroll
                        for (int p = 0; p < 3; ++p) ldmatrix_x4(x[p], pq + p * PLANE + (16 * i + grow) * GM_PITCH + d + 16 * j + gcol);
                        constexpr int A[5] = {2, 0, 1, 1, 0}, B[5] = {0, 2, 1, 0, 1};
#pragma unroll
                        for (int m = 0; m < 5; ++m) mma_bf16(ws[j], x[A[m]], y[B[m]][2 * j], y[B[m]][2 * j + 1]);
                        mma_bf16(w, x[0], y[0][2 * j], y[0][2 * j + 1]);
                    }
                    float* to = part + unit * 128 + lg * 8 + 2 * lt;
                    *reinterpret_cast<float2*>(to) = make_float2(w[0] + (ws[0][0] + ws[1][0]), w[1] + (ws[0][1] + ws[1][1]));
                    *reinterpret_cast<float2*>(to + 64) = make_float2(w[2] + (ws[0][2] + ws[1][2]), w[3] + (ws[0][3] + ws[1][3]));
                }
                float o[2][2][4] = {}, om[2][2][4] = {};
#pragma unroll
                for (int j = 0; j < D / 16; ++j) {
                    float s[2][4];
#pragma unroll
                    for (int u = 0; u < 2; ++u) {
                        const float2 f = *reinterpret_cast<const float2*>(bend + 16 * j + 8 * u + 2 * lt);
#pragma unroll
                        for (int i = 0; i < 4; ++i) s[u][i] = ahead[u][i] * (i & 1 ? f.y : f.x);
                    }
                    if (j + 1 < D / 16) fetch(j + 1);
                    unsigned x[3][4], y[3][4];
                    split_tiles(s[0], s[1], x);
#pragma unroll
                    for (int b = 0; b < 2; ++b) {
#pragma unroll
                        for (int p = 0; p < 3; ++p) ldmatrix_x4(y[p], pq + p * PLANE + (16 * b + frow) * GM_PITCH + 16 * j + fcol);
                        split_mma(o[b], om[b], x, y);
                    }
                }
                // A state that is infinite, NaN or beyond bfloat16's range has pieces that are NaN, and these are in the smaller products:
                // multiply-adds say what becomes of which column.
                float sum = 0.0f;
#pragma unroll
                for (int i = 0; i < 4; ++i) sum += (om[0][0][i] + om[0][1][i]) + (om[1][0][i] + om[1][1][i]);
                walk = __syncthreads_or(!(fabsf(sum) <= 3.4028235e38f));
                if (!walk) {
                    for (int idx = tid; idx < 6 * 64; idx += 256) {          // the shares; what lies ahead of a token weighs nothing
                        const int tile = idx >> 6, i = tile < 2 ? 0 : 1, at = 2 * (idx & 63);
                        const int t = 16 * i + (at >> 3), s = 8 * (tile - 2 * i) + (at & 7);
                        float2 x[4];
#pragma unroll
                        for (int u = 0; u < 4; ++u) x[u] = *reinterpret_cast<const float2*>(part + (4 * tile + u) * 128 + at);
                        float w0 = s <= t ? (x[0].x + x[1].x) + (x[2].x + x[3].x) : 0.0f, w1 = s + 1 <= t ? (x[0].y + x[1].y) + (x[2].y + x[3].y) : 0.0f;
#pragma unroll
                        for (int p = 0; p < 3; ++p) *reinterpret_cast<unsigned*>(pp + (p * T + t) * GM_WP + s) = split_piece(w0, w1);
                    }
                    __syncthreads();
                    for (int idx = tid; idx < T * (V / 4); idx += 256) {
                        const int t = idx / (V / 4), c = (idx % (V / 4)) << 2;
                        cp_async16(gates + t * V + c, proj + (base + min(t, nb - 1)) * stride + g_off + h * V + c, t < nb);
                    }
                    cp_async_commit();
#pragma unroll
                    for (int sb = 0; sb < 2; ++sb) {
                        unsigned x[3][4], y[3][4];
#pragma unroll
                        for (int p = 0; p < 3; ++p) ldmatrix_x4_trans(x[p], pv + p * PLANE + (16 * sb + frow) * GM_PITCH + 16 * warp + fcol);
#pragma unroll
                        for (int b = sb; b < 2; ++b) {
#pragma unroll
                            for (int p = 0; p < 3; ++p) ldmatrix_x4(y[p], pp + (p * T + 16 * b + frow) * GM_WP + 16 * sb + fcol);
                            split_mma(o[b], om[b], x, y);
                        }
                    }
                    // the queries' planes were last read in front of a barrier
#pragma unroll
                    for (int b = 0; b < 2; ++b)
#pragma unroll
                        for (int u = 0; u < 2; ++u)
#pragma unroll
                            for (int i = 0; i < 4; ++i)
                                os[(16 * b + 8 * u + 2 * lt + (i & 1)) * GM_OP + v0 + 8 * (i >> 1)] = o[b][u][i] + om[b][u][i];
                }
            }
            if (!walk && (MODE != GLA_OUT || more)) {
                unsigned x[T / 16][3][4];
#pragma unroll
                for (int sb = 0; sb < T / 16; ++sb)
#pragma unroll
                    for (int p = 0; p < 3; ++p) ldmatrix_x4_trans(x[sb][p], pv + p * PLANE + (16 * sb + frow) * GM_PITCH + 16 * warp + fcol);
                if (!none) fetch(0);
#pragma unroll
                for (int j = 0; j < D / 16; ++j) {
                    float c[2][4] = {}, cm[2][4] = {}, n[2][4];      // n: the last sixteen tokens, which strong decays leave little but
#pragma unroll
                    for (int sb = 0; sb < T / 16; ++sb) {
                        unsigned y[3][4];
#pragma unroll
                        for (int p = 0; p < 3; ++p) ldmatrix_x4_trans(y[p], pk + p * PLANE + (16 * sb + grow) * GM_PITCH + 16 * j + gcol);
                        if (sb + 1 < T / 16) split_mma(c, cm, x[sb], y);
                        else split_mma_whole<false>(n, cm, x[sb], y);
                    }
                    float old[2][4];
#pragma unroll
                    for (int u = 0; u < 2; ++u)
#pragma unroll
                        for (int i = 0; i < 4; ++i) old[u][i] = none ? 0.0f : ahead[u][i];
                    if (!none && j + 1 < D / 16) fetch(j + 1);
#pragma unroll
                    for (int u = 0; u < 2; ++u) {
                        const int row = 16 * j + 8 * u + 2 * lt;
                        const float2 f = *reinterpret_cast<const float2*>(bend + row);
#pragma unroll
                        for (int i = 0; i < 4; ++i)
                            s_out[static_cast<size_t>(row + (i & 1)) * V + v0 + 8 * (i >> 1)] = (fmaf(old[u][i], i & 1 ? f.y : f.x, cm[u][i]) + c[u][i]) + n[u][i];
                    }
                }
            }
        }
        if (walk) {                                  // token by token, the state in registers
            for (int idx = tid; idx < nb * (D / 4); idx += 256) {
                const int t = idx / (D / 4), c = (idx % (D / 4)) << 2;
                const float* pr = proj + (base + t) * stride + h * D + c;
                *reinterpret_cast<float4*>(walk_k + t * D + c) = *reinterpret_cast<const float4*>(pr + k_off);
                *reinterpret_cast<float4*>(walk_v + t * V + c) = *reinterpret_cast<const float4*>(pr + v_off);
                *reinterpret_cast<float4*>(walk_a + t * D + c) = *reinterpret_cast<const float4*>(alpha + (base + t) * HD + h * D + c);
                if (OUTPUTS) *reinterpret_cast<float4*>(walk_q + t * D + c) = *reinterpret_cast<const float4*>(pr + q_off);
            }
            __syncthreads();
            const int d0 = 2 * lt;                   // tile n, element i: row d0 + 8 n + (i & 1), column v0 + 8 (i >> 1)
            float S[16][4];
#pragma unroll
            for (int n = 0; n < 16; ++n)
#pragma unroll
                for (int i = 0; i < 4; ++i) S[n][i] = none ? 0.0f : s_in[static_cast<size_t>(d0 + 8 * n + (i & 1)) * V + v0 + 8 * (i >> 1)];
            for (int t = 0; t < nb; ++t) {
                const float w0 = walk_v[t * V + v0], w1 = walk_v[t * V + v0 + 8];
                float x0[2] = {}, x1[2] = {}, y0[2] = {}, y1[2] = {};
#pragma unroll
                for (int n = 0; n < 16; ++n) {
                    const float2 a = *reinterpret_cast<const float2*>(walk_a + t * D + d0 + 8 * n);
                    const float2 k = *reinterpret_cast<const float2*>(walk_k + t * D + d0 + 8 * n);
                    S[n][0] = a.x * S[n][0] + k.x * w0;
                    S[n][1] = a.y * S[n][1] + k.y * w0;
                    S[n][2] = a.x * S[n][2] + k.x * w1;
                    S[n][3] = a.y * S[n][3] + k.y * w1;
                    if (OUTPUTS) {
                        const float2 q = *reinterpret_cast<const float2*>(walk_q + t * D + d0 + 8 * n);
                        x0[n & 1] += S[n][0] * q.x;
                        y0[n & 1] += S[n][1] * q.y;
                        x1[n & 1] += S[n][2] * q.x;
                        y1[n & 1] += S[n][3] * q.y;
                    }
                }
                if (OUTPUTS) {
                    float z0 = (x0[0] + x0[1]) + (y0[0] + y0[1]), z1 = (x1[0] + x1[1]) + (y1[0] + y1[1]);
#pragma unroll
                    for (int off = 1; off <= 2; off <<= 1) {
                        z0 += __shfl_xor_sync(0xffffffffu, z0, off);
                        z1 += __shfl_xor_sync(0xffffffffu, z1, off);
                    }
                    if (lt == 0) {
                        walk_o[t * GM_OP + v0] = z0;
                        walk_o[t * GM_OP + v0 + 8] = z1;
                    }
                }
            }
            if (MODE != GLA_OUT || more)
#pragma unroll
                for (int n = 0; n < 16; ++n)
#pragma unroll
                    for (int i = 0; i < 4; ++i) s_out[static_cast<size_t>(d0 + 8 * n + (i & 1)) * V + v0 + 8 * (i >> 1)] = S[n][i];
            __syncthreads();
            o0 = walk_o;
        }
        if (OUTPUTS) {                               // a warp per token: norm over V, weight, gate, scale
            const float4 nw = *reinterpret_cast<const float4*>(norm_w + 4 * lane);
            cp_async_wait_all();
            __syncthreads();
            const bool staged = o0 == os;
#pragma unroll
            for (int i = 0; i < T / 8; ++i) {     // (four tokens' chains side by side)
                const int tok = min(warp + 8 * i, nb - 1);
                const float4 g = *reinterpret_cast<const float4*>(staged ? gates + tok * V + 4 * lane : proj + (base + tok) * stride + g_off + h * V + 4 * lane);
                const float4 o = *reinterpret_cast<const float4*>(o0 + tok * GM_OP + 4 * lane);
                const float4 x = make_float4(o.x * q_scale, o.y * q_scale, o.z * q_scale, o.w * q_scale);
                const float ss = warp_sum(x.x * x.x + x.y * x.y + x.z * x.z + x.w * x.w);
                const float inv = q_scale / sqrtf(ss / static_cast<float>(V) + eps) * out_scale;
                if (warp + 8 * i < nb) {
                    TO* orow = out + (base + tok) * out_stride + out_off + h * V + 4 * lane;
                    orow[0] = from_f32<TO>(o.x * inv * nw.x * gm_silu(g.x));
                    orow[1] = from_f32<TO>(o.y * inv * nw.y * gm_silu(g.y));
                    orow[2] = from_f32<TO>(o.z * inv * nw.z * gm_silu(g.z));
                    orow[3] = from_f32<TO>(o.w * inv * nw.w * gm_silu(g.w));
                }
            }
        }
        if (more) __syncthreads();                   // shared memory and the state in memory are about to be used again
    }
}

// Rows of a state column that one thread keeps (R), the row groups DG = ceil(D / R), and the block size the
// kernel is compiled for: 16, else 32, else 64, else 8 rows, whichever block of V * DG threads fits first
// within 512 threads (64 x 64 a head: 110 us with 16 rows, 134 with 8, 173 with 32 for 2,048 tokens of 16
// heads; 128 x 128: 32 rows, 185 us for 8 heads), then within what the kernel's registers allow at that R (a block's registers are threads x registers
// per thread, at most 65,536).  States too large for that (128 x 256 a head and more) take R = 64 compiled
// for 512 or 1,024 threads: the compiler then keeps part of the state in local memory, which is slow and
// correct.
// `wide32`: a block of up to 544 threads at 32 rows a thread is allowed (17 warps: a state of 128 x 128 with one
// more column, the normaliser of a matrix memory, is 4 row groups x 129 columns = 516 threads; at 64 rows a
// thread it would run half as fast).
static int gla_rows_per_thread(int D, int V, int* dg_out, int* max_threads, bool wide32 = false) {
    const int cands[4] = {8, 16, 32, 64};
    const int limits[2][4] = {{512, 512, 512, 384}, {1024, 1024, 512, 384}};
    const int compiled_for[4] = {1024, 1024, 512, 384};
    static int forced = -1;                        // LLM_GLA_ROWS=8|16|32|64: take that R when its block fits (for measurements)
    if (forced < 0) {
        const char* e = getenv("LLM_GLA_ROWS");
        forced = e ? atoi(e) : 0;
    }
    for (int c = 0; c < 4; ++c)
        if (forced == cands[c] && static_cast<long long>(V) * ((D + forced - 1) / forced) <= limits[1][c]) {
            *dg_out = (D + forced - 1) / forced;
            *max_threads = compiled_for[c];
            return forced;
        }
    const int order[4] = {1, 2, 3, 0};             // 16 rows a thread first: measured best wherever its block fits 512 threads
    for (int pass = 0; pass < 2; ++pass)
        for (int o = 0; o < 4; ++o) {
            const int c = order[o];
            const int dg = (D + cands[c] - 1) / cands[c];
            if (static_cast<long long>(V) * dg <= limits[pass][c]) {
                *dg_out = dg;
                *max_threads = compiled_for[c];
                return cands[c];
            }
            if (wide32 && cands[c] == 32 && static_cast<long long>(V) * dg <= 544) {
                *dg_out = dg;
                *max_threads = 544;
                return 32;
            }
        }
    const int dg = (D + 63) / 64;
    for (int limit = 512; limit <= 1024; limit *= 2)
        if (static_cast<long long>(V) * dg <= limit) {
            *dg_out = dg;
            *max_threads = limit;
            return 64;
        }
    return 0;
}

extern "C" int llm_gla_supported(int D, int V) {
    int dg, mt;
    return (D > 0 && V > 0 && gla_rows_per_thread(D, V, &dg, &mt) > 0) ? 1 : 0;
}

// The general entry point.  decay_kind 0: a decay per (token, head, key channel), `alpha` [T, H*D]; 1: a decay
// per (token, head) at alpha[token * a_tok + head * a_head] (a_tok 0: a constant per head), with `kscale` and
// `nfloor` as in RecurOpts.  norm_w null: a weightless output norm.
extern "C" int llm_recur_scan(
    const float* proj, long long stride, int q_off, int k_off, int v_off, int g_off, const float* la,
    const float* norm_w, float eps, float q_scale, float out_scale, void* out, int out_dtype, long long out_stride,
    int out_off, float* state, const int32_t* entry_slot, const int32_t* entry_q_start, const int32_t* entry_q_len,
    const int32_t* items, int num_items, int mode, float* scratch_s, float* scratch_a, int H, int D, int V,
    int decay_kind, long long a_tok, long long a_head, const float* kscale, const float* nfloor, int norm_stride,
    int gate_kind, long long state_head_stride, long long state_slot_stride, uintptr_t stream) {
    if (num_items <= 0) return LLM_OK;
    if (H <= 0 || D <= 0 || V <= 0 || mode < 0 || mode > 2 || H > 65535) return LLM_REFUSED_SIZE;
    if (mode != GLA_FULL && (!items || !scratch_s || !scratch_a)) return LLM_REFUSED_SIZE;
    if (decay_kind < 0 || decay_kind > 1 || gate_kind < 0 || gate_kind > 2) return LLM_REFUSED_SIZE;
    // the per-channel instantiation is gated linear attention as it was: its options are fixed
    if (decay_kind == 0 && (kscale || nfloor || !norm_w || norm_stride != 0 || gate_kind != 2 ||
                            state_head_stride != static_cast<long long>(D) * V ||
                            state_slot_stride != static_cast<long long>(H) * D * V))
        return LLM_REFUSED_SIZE;
    const int VC = V + (nfloor ? 1 : 0);
    if (state_head_stride < static_cast<long long>(D) * VC) return LLM_REFUSED_SIZE;
    int DG = 0, MT = 0;
    const int R = gla_rows_per_thread(D, VC, &DG, &MT, decay_kind == 1);
    if (R == 0) return LLM_REFUSED_SIZE;
    const size_t per_buf = decay_kind ? (2 * static_cast<size_t>(D) + V + 2) : (3 * static_cast<size_t>(D) + V);
    const size_t smem = static_cast<size_t>(GLA_TB) * (2 * per_buf + static_cast<size_t>(DG) * VC) * sizeof(float);
    // sixteen-byte copies into the staging buffers want every row piece on a sixteen-byte boundary
    const int vec = D % 4 == 0 && V % 4 == 0 && stride % 4 == 0 && q_off % 4 == 0 && k_off % 4 == 0 && v_off % 4 == 0 &&
                    aligned16(proj) && (decay_kind || aligned16(la));
    if (smem > 220 * 1024) return LLM_REFUSED_SIZE;
    if (out_dtype != LLM_DT_F32 && out_dtype != LLM_DT_BF16) return LLM_REFUSED_DTYPE;
    if (decay_kind == 0 && vec && g_off % 4 == 0 && gla_tiled_takes(D, V, mode) && aligned16(state) && (mode == GLA_FULL || aligned16(scratch_s))) {
        const size_t need = static_cast<size_t>(GLA_TB) * (2 * (3 * D + 2 * V) + V) * sizeof(float);      // 88 KB at most
        const size_t bytes = static_cast<long long>(num_items) * H <= GLA_ALONE_BLOCKS ? GLA_ALONE_SMEM : need;
#define TILED(RR, MODE, TO)                                                                                          \
        do {                                                                                                          \
            auto kern = gla_scan_tiled_kernel<RR, MODE, TO>;                                                          \
            /* the limit is the same for every launch: another thread may be between the two calls */                 \
            const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, GLA_ALONE_SMEM); \
            if (e != cudaSuccess) return static_cast<int>(e);                                                         \
            launch_pdl(kern, dim3(num_items, H), dim3(2 * V), bytes, reinterpret_cast<cudaStream_t>(stream), proj,     \
                       stride, q_off, k_off, v_off, g_off, la, norm_w, eps, q_scale, out_scale,                       \
                       static_cast<TO*>(out), out_stride, out_off, state, entry_slot, entry_q_start, entry_q_len,     \
                       items, scratch_s, scratch_a, H, V);                                                            \
            return launch_status();                                                                                   \
        } while (0)
#define TILED_MODES(RR, TO)                                                                                           \
        do { if (mode == GLA_FULL) TILED(RR, GLA_FULL, TO); else if (mode == GLA_LOCAL) TILED(RR, GLA_LOCAL, TO); else TILED(RR, GLA_OUT, TO); } while (0)
        if (D == 128) { if (out_dtype == LLM_DT_F32) TILED_MODES(8, float); else TILED_MODES(8, bf16); }
        else { if (out_dtype == LLM_DT_F32) TILED_MODES(4, float); else TILED_MODES(4, bf16); }
#undef TILED_MODES
#undef TILED
    }
    const RecurOpts opt = {a_tok, a_head, kscale, nfloor, norm_stride, gate_kind, state_head_stride, state_slot_stride};
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    const dim3 grid(num_items, H), block((VC * DG + 31) / 32 * 32);
#define LAUNCH(RR, MM, TO, SC)                                                                                    \
    do {                                                                                                          \
        auto kern = gla_scan_kernel<RR, MM, TO, SC>;                                                                \
        if (smem > 48 * 1024) {                                                                                   \
            const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,         \
                                                       static_cast<int>(smem));                                   \
            if (e != cudaSuccess) return static_cast<int>(e);                                                     \
        }                                                                                                         \
        launch_pdl(kern, grid, block, smem, s, proj, stride, q_off, k_off, v_off, g_off, la, norm_w, eps, q_scale, \
                   out_scale, static_cast<TO*>(out), out_stride, out_off, state, entry_slot, entry_q_start,       \
                   entry_q_len, items, mode, scratch_s, scratch_a, H, D, V, DG, vec, opt);                        \
    } while (0)
#define BY_R(TO, SC)                                                                                              \
    switch (R) {                                                                                                  \
        case 8: LAUNCH(8, 1024, TO, SC); break;                                                                   \
        case 16: LAUNCH(16, 1024, TO, SC); break;                                                                 \
        case 32: LAUNCH(32, 512, TO, SC); break;                                                                  \
        default:                                                                                                  \
            if (MT == 384) LAUNCH(64, 384, TO, SC);                                                               \
            else if (MT == 512) LAUNCH(64, 512, TO, SC);                                                          \
            else LAUNCH(64, 1024, TO, SC);                                                                        \
            break;                                                                                                \
    }
    if (R == 32 && MT == 544) {
        if (out_dtype == LLM_DT_F32) LAUNCH(32, 544, float, true);
        else LAUNCH(32, 544, bf16, true);
    } else if (out_dtype == LLM_DT_F32) { if (decay_kind) { BY_R(float, true) } else { BY_R(float, false) } }
    else { if (decay_kind) { BY_R(bf16, true) } else { BY_R(bf16, false) } }
#undef BY_R
#undef LAUNCH
    return launch_status();
}

// Gated linear attention: a decay per key channel, a norm weight [V] shared by the heads, a silu gate, the
// states [slots, H, D, V] alone in their slots.  `longest`: tokens of the longest item, 0 if not known.
// Items that bring fewer than eight tokens each stay with the register-tiled kernel: a batch costs the tensor-core kernel the same
// for one token as for 32.  One pass over items of 128 x 128, 16 heads (us, tiled and tensor cores): 32 items of 3 tokens 28
// and 40, of 16 47 and 41, of 64 130 and 91; one item of 16 tokens 16 and 13, of 64 41 and 25, of 128 74 and 49; 8 of 100 61 and 49.
// `tau`: decays are sigmoid(z)^(1/tau), 0 if not known.  Below 2 every batch of 32 tokens has a channel that decays to less than 2^-60
// for a z around zero, so that the passes with outputs would prepare their batches and then walk: they stay with the register-tiled
// kernel.  2,048 tokens of 16 heads, output pass (us, tiled and tensor cores): tau 1 121 and 176, tau 2 121 and 94 (176 when z is
// around -2); 8 items of 100 in one pass 70 and 92, 70 and 61.  The local pass takes any decays: 72 and 43.
#define GM_FROM 8
#define GM_TAU 2.0f
extern "C" int llm_gla_scan(
    const float* proj, long long stride, int q_off, int k_off, int v_off, int g_off, const float* la,
    const float* norm_w, float eps, float q_scale, float out_scale, void* out, int out_dtype, long long out_stride,
    int out_off, float* state, const int32_t* entry_slot, const int32_t* entry_q_start, const int32_t* entry_q_len,
    const int32_t* items, int num_items, int mode, float* scratch_s, float* scratch_a, int H, int D, int V, int longest, float tau,
    uintptr_t stream) {
    static const bool rows_forced = getenv("LLM_GLA_ROWS") != nullptr;
    const bool taken = D == GM_D && V == GM_D && (longest <= 0 || longest >= GM_FROM) && (mode == GLA_LOCAL || tau <= 0.0f || tau >= GM_TAU) && !rows_forced && stride % 4 == 0 && q_off % 4 == 0 &&
                       k_off % 4 == 0 && v_off % 4 == 0 && g_off % 4 == 0 && aligned16(proj) && aligned16(la) && norm_w && aligned16(norm_w);
    if (num_items <= 0 || !taken || H <= 0 || H > 65535 || mode < 0 || mode > 2 || (mode != GLA_FULL && (!items || !scratch_s || !scratch_a)) ||
        (mode != GLA_FULL && !aligned16(scratch_a)) || (out_dtype != LLM_DT_F32 && out_dtype != LLM_DT_BF16))
        return llm_recur_scan(proj, stride, q_off, k_off, v_off, g_off, la, norm_w, eps, q_scale, out_scale, out, out_dtype,
                              out_stride, out_off, state, entry_slot, entry_q_start, entry_q_len, items, num_items, mode,
                              scratch_s, scratch_a, H, D, V, 0, 0, 0, nullptr, nullptr, 0, 2,
                              static_cast<long long>(D) * V, static_cast<long long>(H) * D * V, stream);
    auto launch = [&](auto kern, auto* to) {
        constexpr int with = GM_SMEM(true), without = GM_SMEM(false);
        static_assert(with <= GLA_ALONE_SMEM && without <= GLA_ALONE_SMEM, "shared memory");
        const int bytes = static_cast<long long>(num_items) * H <= GLA_ALONE_BLOCKS ? GLA_ALONE_SMEM : mode == GLA_LOCAL ? without : with;
        const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, GLA_ALONE_SMEM);
        if (e != cudaSuccess) return static_cast<int>(e);
        launch_pdl(kern, dim3(num_items, H), dim3(256), bytes, reinterpret_cast<cudaStream_t>(stream), proj, stride, q_off, k_off,
                   v_off, g_off, la, norm_w, eps, q_scale, out_scale, to, out_stride, out_off, state, entry_slot, entry_q_start,
                   entry_q_len, items, scratch_s, scratch_a, H);
        return launch_status();
    };
    auto by_mode = [&](auto* to) {
        using TO = std::remove_pointer_t<decltype(to)>;
        return mode == GLA_FULL    ? launch(gla_scan_mma_kernel<GLA_FULL, TO>, to)
               : mode == GLA_LOCAL ? launch(gla_scan_mma_kernel<GLA_LOCAL, TO>, to)
                                   : launch(gla_scan_mma_kernel<GLA_OUT, TO>, to);
    };
    return out_dtype == LLM_DT_F32 ? by_mode(static_cast<float*>(out)) : by_mode(static_cast<bf16*>(out));
}

// The recurrence for entries that bring ONE token (decode steps): the state is streamed, not held: thread
// (row group, column) walks its rows of the column once, eight loads in flight, S <- alpha S + k v written
// back as it goes, its share of o left in shared memory; then a warp per 32 columns adds the shares and
// applies norm, weight, gate and scale.  Few registers, so several blocks share an SM and the state's
// bytes bound the kernel, as keys and values bound decode attention.  Entry i is row q_start[i].
// What the step kernel can make itself instead of reading it: a rotation of q and k (retention), and the
// gates of a matrix memory with exponential gating (its decay, input scale and floor).
struct StepExtras {
    const float* rot_inv_freq;        // float32 [rot_dims / 2] or null: rotate pairs (i, i + rot_dims/2) of q and k
    int rot_dims;                     // by the angle float(position) * inv_freq[i]
    const int32_t* positions;
    float gate_cap;                   // > 0: a = exp(f + m - m'), e = exp(i - m'), floor = exp(-m') from the raw gates
    int i_off, f_off;                 // columns of the projection that hold them, one per head
    const float* i_bias;
    const float* f_bias;
    long long m_off;                  // where the running maximum m sits inside a head's state
};

// The log gates of a matrix memory: i = cap * tanh(z_i / cap), f = logsigmoid(cap * tanh(z_f / cap)).
__device__ __forceinline__ void recur_log_gates(float zi, float zf, float cap, float& ig, float& fg) {
    ig = cap * tanhf(zi / cap);
    const float c = cap * tanhf(zf / cap);
    fg = c < 0.0f ? c - log1pf(expf(c)) : -log1pf(expf(-c));
}

template <typename TO>
__global__ void gla_step_kernel(
    const float* __restrict__ proj, long long stride, int q_off, int k_off, int v_off, int g_off,
    const float* __restrict__ la, const float* __restrict__ norm_w, float eps, float q_scale, float out_scale,
    TO* __restrict__ out, long long out_stride, int out_off, float* __restrict__ state,
    const int32_t* __restrict__ entry_slot, const int32_t* __restrict__ entry_q_start, int H, int D, int V, int DG,
    int a_off, int rank, const float* __restrict__ w2t, const float* __restrict__ b2, float inv_tau,
    long long a_tok, long long a_head, long long a_chan, int normaliser, const RecurOpts opt, const StepExtras ex) {
    pdl_begin();
    extern __shared__ __align__(16) float smem[];
    const int VC = V + (normaliser ? 1 : 0);
    float* sq = smem;                 // [D]
    float* sk = sq + D;
    float* sa = sk + D;
    float* sv = sa + D;               // [V]
    float* part = sv + V;             // [DG][VC]
    float* red = part + DG * VC;      // 33, then 3 scalars of the gates
    float* a1 = red + 36;             // [rank]: the decay projection's first half, when the decays are made here
    const int entry = blockIdx.x, h = blockIdx.y, tid = threadIdx.x;
    const size_t row = static_cast<size_t>(entry_q_start[entry]);
    const float* pr = proj + row * stride;
    float* head_state = state + static_cast<size_t>(entry_slot[entry]) * opt.state_slot_stride + h * opt.state_head_stride;
    if (!la && rank > 0) {
        for (int j = tid; j < rank; j += blockDim.x) a1[j] = pr[a_off + j];
        __syncthreads();
    }
    if (ex.gate_cap > 0.0f && tid == 0) {
        float ig, fg;
        recur_log_gates(pr[ex.i_off + h] + ex.i_bias[h], pr[ex.f_off + h] + ex.f_bias[h], ex.gate_cap, ig, fg);
        const float m_old = head_state[ex.m_off];
        const float m_new = fmaxf(fg + m_old, ig);
        red[33] = expf(fg + m_old - m_new);
        red[34] = expf(ig - m_new);
        red[35] = expf(-m_new);
        head_state[ex.m_off] = m_new;
    }
    for (int d = tid; d < D; d += blockDim.x) {
        sq[d] = pr[q_off + h * D + d];
        sk[d] = pr[k_off + h * D + d];
        if (la) {
            sa[d] = la[row * a_tok + h * a_head + d * a_chan];       // the decay itself
        } else if (rank > 0) {                         // alpha = sigmoid(w2[c, :] . a1 + b2[c]) ^ (1 / tau), as gla_decay_kernel
            const int c = h * D + d, C = H * D;
            float z = b2 ? b2[c] : 0.0f;
            int j = 0;
            for (; j + 16 <= rank; j += 16) {
                float w[16];
#pragma unroll
                for (int u = 0; u < 16; ++u) w[u] = w2t[static_cast<size_t>(j + u) * C + c];
#pragma unroll
                for (int u = 0; u < 16; ++u) z += w[u] * a1[j + u];
            }
            for (; j < rank; ++j) z += w2t[static_cast<size_t>(j) * C + c] * a1[j];
            const float ls = z < 0.0f ? z - log1pf(expf(z)) : -log1pf(expf(-z));
            sa[d] = expf(ls * inv_tau);
        }
    }
    for (int c = tid; c < V; c += blockDim.x) sv[c] = pr[v_off + h * V + c];
    __syncthreads();
    if (ex.rot_inv_freq) {                             // pairs (i, i + half) of q and k turn by position * inv_freq[i]
        const int half = ex.rot_dims >> 1;
        const float p = static_cast<float>(ex.positions[row]);
        for (int i = tid; i < half; i += blockDim.x) {
            float sn, cs;
            sincosf(p * ex.rot_inv_freq[i], &sn, &cs);
            const float qu = sq[i], qv = sq[i + half], ku = sk[i], kv = sk[i + half];
            sq[i] = qu * cs - qv * sn;
            sq[i + half] = qv * cs + qu * sn;
            sk[i] = ku * cs - kv * sn;
            sk[i + half] = kv * cs + ku * sn;
        }
    }
    float floor_t = 0.0f;
    if (ex.gate_cap > 0.0f) {
        const float keep = red[33], put = red[34];
        floor_t = red[35];
        __syncthreads();                               // the rotation (if any) and red[] are settled
        for (int d = tid; d < D; d += blockDim.x) {
            sa[d] = keep;
            sk[d] *= put;
        }
    }
    __syncthreads();
    const bool active = tid < VC * DG;
    const int c = active ? tid % VC : 0, dg = active ? tid / VC : 0;
    const int rows = (D + DG - 1) / DG, d0 = dg * rows, d1 = min(D, d0 + rows);
    // column c < V of S has stride V; the normaliser column is contiguous after S
    float* S = c < V ? head_state + c : head_state + static_cast<size_t>(D) * V;
    const size_t ss = c < V ? V : 1;
    if (active) {
        const float vt = c < V ? sv[c] : 1.0f;
        float p = 0.0f;
        int d = d0;
        for (; d + 8 <= d1; d += 8) {
            float x[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) x[u] = S[static_cast<size_t>(d + u) * ss];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                x[u] = sa[d + u] * x[u] + sk[d + u] * vt;
                S[static_cast<size_t>(d + u) * ss] = x[u];
                p += x[u] * sq[d + u];
            }
        }
        for (; d < d1; ++d) {
            const float x = sa[d] * S[static_cast<size_t>(d) * ss] + sk[d] * vt;
            S[static_cast<size_t>(d) * ss] = x;
            p += x * sq[d];
        }
        part[dg * VC + c] = p;
    }
    __syncthreads();
    float mul = q_scale;                               // q = W_q x * q_scale, applied to the finished sums
    if (normaliser) {
        float nq = part[V];
        for (int g2 = 1; g2 < DG; ++g2) nq += part[g2 * VC + V];
        mul = q_scale / (fmaxf(fabsf(nq * q_scale), floor_t) + 1e-6f);
    }
    __syncthreads();
    float sq2 = 0.0f;
    for (int i = tid; i < V; i += blockDim.x) {
        float o = part[i];
        for (int g2 = 1; g2 < DG; ++g2) o += part[g2 * VC + i];
        o *= mul;
        part[i] = o;
        sq2 += o * o;
    }
    const float total = block_sum(sq2, red);
    const float inv = 1.0f / sqrtf(total / static_cast<float>(V) + eps);
    TO* orow = out + row * out_stride + out_off + h * V;
    const float* nw = norm_w ? norm_w + h * opt.norm_stride : nullptr;
    for (int i = tid; i < V; i += blockDim.x)
        orow[i] = from_f32<TO>(part[i] * inv * (nw ? nw[i] : 1.0f) * recur_gate(pr[g_off + h * V + i], opt.gate_kind) * out_scale);
}

// The general entry point of the step kernel.  `la` with strides (a_tok, a_head, a_chan): the decays as they
// are (a constant per head: 0, 1, 0).  la null and rank > 0: the low-rank decay projection is applied here.
// gate_cap > 0: the gates of a matrix memory are made here (a normaliser column is then kept, and m at m_off).
extern "C" int llm_recur_step(
    const float* proj, long long stride, int q_off, int k_off, int v_off, int g_off, const float* la,
    const float* norm_w, float eps, float q_scale, float out_scale, void* out, int out_dtype, long long out_stride,
    int out_off, float* state, const int32_t* entry_slot, const int32_t* entry_q_start, int num_entries, int H, int D,
    int V, int a_off, int rank, const float* w2t, const float* b2, float tau, long long a_tok, long long a_head,
    long long a_chan, int norm_stride, int gate_kind, long long state_head_stride, long long state_slot_stride,
    const float* rot_inv_freq, int rot_dims, const int32_t* positions, float gate_cap, int i_off, int f_off,
    const float* i_bias, const float* f_bias, uintptr_t stream) {
    if (num_entries <= 0) return LLM_OK;
    if (H <= 0 || D <= 0 || V <= 0 || H > 65535 || V > 1023) return LLM_REFUSED_SIZE;
    const int normaliser = gate_cap > 0.0f ? 1 : 0;
    if (!la && !normaliser && (!w2t || rank <= 0 || rank > 4096 || !(tau > 0.0f))) return LLM_REFUSED_SIZE;
    if (la || normaliser) rank = 0;
    if (normaliser && (!i_bias || !f_bias)) return LLM_REFUSED_SIZE;
    if (rot_inv_freq && (rot_dims <= 0 || rot_dims % 2 || rot_dims > D || !positions)) return LLM_REFUSED_SIZE;
    if (gate_kind < 0 || gate_kind > 2) return LLM_REFUSED_SIZE;
    const int VC = V + normaliser;
    if (state_head_stride < static_cast<long long>(D) * VC + normaliser) return LLM_REFUSED_SIZE;
    int DG = 256 / VC;
    if (DG < 1) DG = 1;
    if (DG > D) DG = D;
    const int threads = (VC * DG + 31) / 32 * 32;
    const size_t smem = (3 * static_cast<size_t>(D) + V + static_cast<size_t>(DG) * VC + 36 + rank) * sizeof(float);
    if (smem > 48 * 1024) return LLM_REFUSED_SIZE;
    const float inv_tau = rank > 0 ? 1.0f / tau : 0.0f;
    const RecurOpts opt = {0, 0, nullptr, nullptr, norm_stride, gate_kind, state_head_stride, state_slot_stride};
    const StepExtras ex = {rot_inv_freq, rot_dims, positions, gate_cap, i_off, f_off, i_bias, f_bias,
                           static_cast<long long>(D) * V + D};
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    const dim3 grid(num_entries, H);
    if (out_dtype == LLM_DT_F32)
        launch_pdl((gla_step_kernel<float>), grid, dim3(threads), smem, s, proj, stride, q_off, k_off, v_off, g_off, la, norm_w,
                   eps, q_scale, out_scale, static_cast<float*>(out), out_stride, out_off, state, entry_slot, entry_q_start,
                   H, D, V, DG, a_off, rank, w2t, b2, inv_tau, a_tok, a_head, a_chan, normaliser, opt, ex);
    else if (out_dtype == LLM_DT_BF16)
        launch_pdl((gla_step_kernel<bf16>), grid, dim3(threads), smem, s, proj, stride, q_off, k_off, v_off, g_off, la, norm_w,
                   eps, q_scale, out_scale, static_cast<bf16*>(out), out_stride, out_off, state, entry_slot, entry_q_start,
                   H, D, V, DG, a_off, rank, w2t, b2, inv_tau, a_tok, a_head, a_chan, normaliser, opt, ex);
    else
        return LLM_REFUSED_DTYPE;
    return launch_status();
}

extern "C" int llm_gla_step(
    const float* proj, long long stride, int q_off, int k_off, int v_off, int g_off, const float* la,
    const float* norm_w, float eps, float q_scale, float out_scale, void* out, int out_dtype, long long out_stride,
    int out_off, float* state, const int32_t* entry_slot, const int32_t* entry_q_start, int num_entries, int H, int D,
    int V, int a_off, int rank, const float* w2t, const float* b2, float tau, uintptr_t stream) {
    // la null: the decays are computed here from the projection's columns a_off .. a_off + rank (w2t, b2, tau as
    // for llm_gla_decay), which saves a decode step one launch a layer
    if (!la && (!w2t || rank <= 0)) return LLM_REFUSED_SIZE;
    return llm_recur_step(proj, stride, q_off, k_off, v_off, g_off, la, norm_w, eps, q_scale, out_scale, out, out_dtype,
                          out_stride, out_off, state, entry_slot, entry_q_start, num_entries, H, D, V, a_off, rank, w2t,
                          b2, tau, static_cast<long long>(H) * D, D, 1, 0, 2, static_cast<long long>(D) * V,
                          static_cast<long long>(H) * D * V, nullptr, 0, nullptr, 0.0f, 0, 0, nullptr, nullptr, stream);
}

// chains: int32 [n, 3] = (entry, first scratch index, number of chunks); chunk c of the entry is scratch
// index first + c.  grid (n, H, blocks over D*V).  E elements a thread: four where the sizes and addresses allow (V a multiple of 4:
// they share a row), which keeps 128 bytes of a thread's loads in flight: 32 chunks of 16 heads of 128 x 128, 22 -> 10 us.
template <int E>
__global__ void __launch_bounds__(256) gla_chain_kernel(float* __restrict__ state, float* __restrict__ scratch_s,
                                 const float* __restrict__ scratch_a, const int32_t* __restrict__ chains,
                                 const int32_t* __restrict__ entry_slot, int H, int D, int V, int VC,
                                 long long state_head_stride, long long state_slot_stride) {
    pdl_begin();
    typedef typename std::conditional<E == 4, float4, float>::type T;
    const int entry = chains[3 * blockIdx.x];
    if (entry < 0) return;
    const int first = chains[3 * blockIdx.x + 1], n = chains[3 * blockIdx.x + 2];
    const int h = blockIdx.y;
    const int e = E * (blockIdx.z * blockDim.x + threadIdx.x);
    if (e >= D * VC) return;
    const int d = e < D * V ? e / V : e - D * V;         // S [D, V], then the normaliser n [D] when VC = V + 1
    const size_t per = static_cast<size_t>(D) * VC;
    T* st = reinterpret_cast<T*>(state + static_cast<size_t>(entry_slot[entry]) * state_slot_stride + h * state_head_stride + e);
    T S = *st;
    for (int c0 = 0; c0 < n; c0 += 8) {              // eight chunks' loads in flight, then the chain through them
        T L[8];
        float A[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const size_t at = static_cast<size_t>(first + min(c0 + i, n - 1)) * H + h;
            L[i] = *reinterpret_cast<const T*>(scratch_s + at * per + e);
            A[i] = scratch_a[at * D + d];
        }
#pragma unroll
        for (int i = 0; i < 8; ++i)
            if (c0 + i < n) {
                *reinterpret_cast<T*>(scratch_s + (static_cast<size_t>(first + c0 + i) * H + h) * per + e) = S;
                if constexpr (E == 4)
                    S = make_float4(A[i] * S.x + L[i].x, A[i] * S.y + L[i].y, A[i] * S.z + L[i].z, A[i] * S.w + L[i].w);
                else
                    S = A[i] * S + L[i];
            }
    }
    *st = S;
}

// `normaliser` 1: a head's state is S [D, V] followed by n [D], and both are chained.
extern "C" int llm_recur_chain(float* state, float* scratch_s, const float* scratch_a, const int32_t* chains,
                               int num_chains, const int32_t* entry_slot, int H, int D, int V, int normaliser,
                               long long state_head_stride, long long state_slot_stride, uintptr_t stream) {
    if (num_chains <= 0) return LLM_OK;
    if (H <= 0 || D <= 0 || V <= 0 || H > 65535) return LLM_REFUSED_SIZE;
    const int VC = V + (normaliser ? 1 : 0);
    const bool four = !normaliser && V % 4 == 0 && aligned16(state) && aligned16(scratch_s) && state_head_stride % 4 == 0 && state_slot_stride % 4 == 0;
    const int threads = four ? 128 : 256, elements = four ? (D * VC + 3) / 4 : D * VC;
    const int bz = (elements + threads - 1) / threads;
    if (bz > 65535) return LLM_REFUSED_SIZE;
    launch_pdl(four ? gla_chain_kernel<4> : gla_chain_kernel<1>, dim3(num_chains, H, bz), dim3(threads), 0, reinterpret_cast<cudaStream_t>(stream),
               state, scratch_s, scratch_a, chains, entry_slot, H, D, V, VC, state_head_stride, state_slot_stride);
    return launch_status();
}

extern "C" int llm_gla_chain(float* state, float* scratch_s, const float* scratch_a, const int32_t* chains,
                             int num_chains, const int32_t* entry_slot, int H, int D, int V, uintptr_t stream) {
    return llm_recur_chain(state, scratch_s, scratch_a, chains, num_chains, entry_slot, H, D, V, 0,
                           static_cast<long long>(D) * V, static_cast<long long>(H) * D * V, stream);
}

// ---- what a recurrence with gates or a rotation needs before the scan over a prompt portion ------------
// recur_gates_kernel: per (entry, head), over the entry's tokens in order, from the raw gate columns of the
// projection: i = cap * tanh((z_i + b_i) / cap), f = logsigmoid(cap * tanh((z_f + b_f) / cap)), the running
// maximum m' = max(f + m, i) (m from the head's state, written back at the end), and per token
//     keep = exp(f + m - m'),   put = exp(i - m'),   floor = exp(-m')
// into three float32 [T, H] arrays (`gates` [3, T, H]).  Tokens are taken 128 at a time: every thread makes
// one token's log gates, one thread walks the maxima (an add and a max a token), every thread makes its token's
// exponentials and stores.
#define RG_TOKENS 128
__global__ void recur_gates_kernel(const float* __restrict__ proj, long long stride, int i_off, int f_off,
                                   const float* __restrict__ i_bias, const float* __restrict__ f_bias, float cap,
                                   float* __restrict__ gates, long long num_tokens, float* __restrict__ state,
                                   long long m_off, long long state_head_stride, long long state_slot_stride,
                                   const int32_t* __restrict__ entry_slot, const int32_t* __restrict__ entry_q_start,
                                   const int32_t* __restrict__ entry_q_len, int H) {
    pdl_begin();
    __shared__ float ig[RG_TOKENS], fg[RG_TOKENS], fl[RG_TOKENS], mx[RG_TOKENS];
    __shared__ float carry;
    const int entry = blockIdx.x, h = blockIdx.y, tid = threadIdx.x;
    const long long row0 = entry_q_start[entry];
    const int count = entry_q_len[entry];
    float* mp = state + static_cast<size_t>(entry_slot[entry]) * state_slot_stride + h * state_head_stride + m_off;
    if (tid == 0) carry = *mp;
    const float bi = i_bias[h], bf = f_bias[h];
    for (int done = 0; done < count; done += RG_TOKENS) {
        const int nb = min(RG_TOKENS, count - done);
        __syncthreads();
        if (tid < nb) {
            const float* pr = proj + (row0 + done + tid) * stride;
            recur_log_gates(pr[i_off + h] + bi, pr[f_off + h] + bf, cap, ig[tid], fg[tid]);
        }
        __syncthreads();
        if (tid == 0) {                                    // the chain itself is an add and a max a token
            float m = carry;
            for (int t = 0; t < nb; ++t) {
                const float m_new = fmaxf(fg[t] + m, ig[t]);
                fl[t] = m;                                 // the maximum that entered the token
                mx[t] = m_new;
                m = m_new;
            }
            carry = m;
        }
        __syncthreads();
        if (tid < nb) {                                    // the exponentials, a token a thread
            const long long at = (row0 + done + tid) * H + h;
            const float m_old = fl[tid], m_new = mx[tid];
            gates[at] = expf(fg[tid] + m_old - m_new);                        // keep
            gates[num_tokens * H + at] = expf(ig[tid] - m_new);               // put
            gates[2 * num_tokens * H + at] = expf(-m_new);                    // floor
        }
    }
    __syncthreads();
    if (tid == 0) *mp = carry;
}

extern "C" int llm_recur_gates(const float* proj, long long stride, int i_off, int f_off, const float* i_bias,
                               const float* f_bias, float cap, float* gates, long long num_tokens, float* state,
                               long long m_off, long long state_head_stride, long long state_slot_stride,
                               const int32_t* entry_slot, const int32_t* entry_q_start, const int32_t* entry_q_len,
                               int num_entries, int H, uintptr_t stream) {
    if (num_entries <= 0 || num_tokens <= 0) return LLM_OK;
    if (H <= 0 || H > 65535 || !(cap > 0.0f) || !i_bias || !f_bias) return LLM_REFUSED_SIZE;
    launch_pdl(recur_gates_kernel, dim3(num_entries, H), dim3(RG_TOKENS), 0, reinterpret_cast<cudaStream_t>(stream),
               proj, stride, i_off, f_off, i_bias, f_bias, cap, gates, num_tokens, state, m_off, state_head_stride,
               state_slot_stride, entry_slot, entry_q_start, entry_q_len, H);
    return launch_status();
}

// rotate_qk_kernel: in place on the float32 projection, pairs (i, i + dims/2) of every head of q and of k turn by
// the angle float(position) * inv_freq[i]; entries from `dims` on pass unchanged.  One block a token.
__global__ void rotate_qk_kernel(float* __restrict__ proj, long long stride, int q_off, int k_off, int heads_q,
                                 int heads_k, int D, int dims, const float* __restrict__ inv_freq,
                                 const int32_t* __restrict__ positions) {
    pdl_begin();
    const long long t = blockIdx.x;
    const int half = dims >> 1;
    const float p = static_cast<float>(positions[t]);
    float* row = proj + t * stride;
    const int pairs = (heads_q + heads_k) * half;
    for (int idx = threadIdx.x; idx < pairs; idx += blockDim.x) {
        const int head = idx / half, i = idx - head * half;
        float* x = head < heads_q ? row + q_off + head * D : row + k_off + (head - heads_q) * D;
        float sn, cs;
        sincosf(p * inv_freq[i], &sn, &cs);
        const float u = x[i], v = x[i + half];
        x[i] = u * cs - v * sn;
        x[i + half] = v * cs + u * sn;
    }
}

extern "C" int llm_rotate_qk(float* proj, long long stride, int q_off, int k_off, int heads_q, int heads_k, int D,
                             int dims, const float* inv_freq, const int32_t* positions, int num_tokens,
                             uintptr_t stream) {
    if (num_tokens <= 0) return LLM_OK;
    if (D <= 0 || dims <= 0 || dims % 2 || dims > D || heads_q < 0 || heads_k < 0) return LLM_REFUSED_SIZE;
    launch_pdl(rotate_qk_kernel, dim3(num_tokens), dim3(128), 0, reinterpret_cast<cudaStream_t>(stream), proj, stride,
               q_off, k_off, heads_q, heads_k, D, dims, inv_freq, positions);
    return launch_status();
}
