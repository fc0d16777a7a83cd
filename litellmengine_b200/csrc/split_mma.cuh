// Products of float32 values on the warp-wide tensor-core instructions: a float32 value is the sum of three bfloat16 values, each
// what is left, rounded to nearest (every remainder is exact), and a product is the six products of them that matter: what is left
// out is at most 2^-24 of it.  Holds for magnitudes up to 2^127 and, without losing last bits, down to 2^-110.
#pragma once

#include "mma_tiles.cuh"

// Two floats as a pair of bfloat16 (a in the lower half), rounded to nearest; a and b become what is left of them.
__device__ __forceinline__ unsigned split_piece(float& a, float& b) {
    unsigned r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;\n" : "=r"(r) : "f"(b), "f"(a));
    a -= __uint_as_float(r << 16);
    b -= __uint_as_float(r & 0xffff0000u);
    return r;
}
// The accumulators of two neighbouring 16 x 8 tiles (columns k .. k + 7, k + 8 .. k + 15) as the three planes of a 16 x 16 left operand.
__device__ __forceinline__ void split_tiles(const float (&lo)[4], const float (&hi)[4], unsigned (&planes)[3][4]) {
    float v[8] = {lo[0], lo[1], lo[2], lo[3], hi[0], hi[1], hi[2], hi[3]};
#pragma unroll
    for (int p = 0; p < 3; ++p)
#pragma unroll
        for (int i = 0; i < 4; ++i) planes[p][i] = split_piece(v[2 * i], v[2 * i + 1]);
}
__device__ __forceinline__ void mma_bf16_first(float (&c)[4], const unsigned (&a)[4], unsigned b0, unsigned b1) {      // from zero
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};\n"
                 : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.0f));
}
// Two tiles of 8 columns side by side, a [16 x 16] by b [16 x 16]: the five smaller of the six products, smallest first, onto `small`,
// the largest onto `main`.
__device__ __forceinline__ void split_mma(float (&main)[2][4], float (&small)[2][4], const unsigned (&a)[3][4], const unsigned (&b)[3][4]) {
    constexpr int A[5] = {2, 0, 1, 1, 0}, B[5] = {0, 2, 1, 0, 1};
#pragma unroll
    for (int i = 0; i < 5; ++i)
#pragma unroll
        for (int u = 0; u < 2; ++u) mma_bf16(small[u], a[A[i]], b[B[i]][2 * u], b[B[i]][2 * u + 1]);
#pragma unroll
    for (int u = 0; u < 2; ++u) mma_bf16(main[u], a[0], b[0][2 * u], b[0][2 * u + 1]);
}
// The same from zero, and nearer.  The tensor cores cut a sum to 24 bits where an addition rounds, which is twice the error (5.8e-8 of a
// sum of sixteen, 2-norm); but they have what they cut: the largest product once more, less what came out of it, goes to `small`.
// One tile here; two below, where FRESH false leaves `small` its sums so far.
__device__ __forceinline__ void split_mma_whole(float (&main)[4], float (&small)[4], const unsigned (&a)[3][4], const unsigned (&b0)[3], const unsigned (&b1)[3]) {
    constexpr int A[5] = {2, 0, 1, 1, 0}, B[5] = {0, 2, 1, 0, 1};
    float rest[4];
    mma_bf16_first(main, a[0], b0[0], b1[0]);
    mma_bf16_first(small, a[A[0]], b0[B[0]], b1[B[0]]);
#pragma unroll
    for (int i = 0; i < 4; ++i) rest[i] = -main[i];
    mma_bf16(rest, a[0], b0[0], b1[0]);
#pragma unroll
    for (int i = 1; i < 5; ++i) mma_bf16(small, a[A[i]], b0[B[i]], b1[B[i]]);
#pragma unroll
    for (int i = 0; i < 4; ++i) small[i] += rest[i];
}
template <bool FRESH = true>
__device__ __forceinline__ void split_mma_whole(float (&main)[2][4], float (&small)[2][4], const unsigned (&a)[3][4], const unsigned (&b)[3][4]) {
    constexpr int A[5] = {2, 0, 1, 1, 0}, B[5] = {0, 2, 1, 0, 1};
    float rest[2][4];
#pragma unroll
    for (int u = 0; u < 2; ++u) mma_bf16_first(main[u], a[0], b[0][2 * u], b[0][2 * u + 1]);
#pragma unroll
    for (int i = 0; i < 5; ++i)
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            if (FRESH && i == 0) mma_bf16_first(small[u], a[A[0]], b[B[0]][2 * u], b[B[0]][2 * u + 1]);
            else mma_bf16(small[u], a[A[i]], b[B[i]][2 * u], b[B[i]][2 * u + 1]);
            if (i == 2) {
#pragma unroll
                for (int m = 0; m < 4; ++m) rest[u][m] = -main[u][m];
                mma_bf16(rest[u], a[0], b[0][2 * u], b[0][2 * u + 1]);
            }
        }
#pragma unroll
    for (int u = 0; u < 2; ++u)
#pragma unroll
        for (int i = 0; i < 4; ++i) small[u][i] += rest[u][i];
}
// Four floats into the three planes, four neighbours of a row; `rest`, what their roundings left out, goes with the second pieces.
__device__ __forceinline__ void split_store4(bf16* to, int plane, float4 v, float4 rest = make_float4(0.0f, 0.0f, 0.0f, 0.0f)) {
#pragma unroll
    for (int p = 0; p < 3; ++p) {
        uint2 r;
        r.x = split_piece(v.x, v.y);
        r.y = split_piece(v.z, v.w);
        *reinterpret_cast<uint2*>(to + p * plane) = r;
        if (p == 0) v = make_float4(v.x + rest.x, v.y + rest.y, v.z + rest.z, v.w + rest.w);
    }
}
