// mlp.cuh -- the learned eddy-viscosity closure: a 6 -> 64 -> 64 -> 1 MLP (SiLU,
// SiLU, softplus) with BF16 weights and activations on the tensor cores
// (mma.sync m16n8k16, FP32 accumulation).  One warp evaluates a tile of 16 samples.
//
// Arithmetic (the CPU oracle oracle/les_oracle.py restates it, roundings included):
//   xb = bf16(x)                       x: 6 features, padded with zeros to 16
//   z1 = W1^T xb + b1,  h1 = silu(z1),  h1b = bf16(h1)
//   z2 = W2^T h1b + b2, h2 = silu(z2),  h2b = bf16(h2)
//   z3 = w3 . h2b + b3 (FP32),          out = softplus(z3)      (nu_t / nu)
// Backward for the loss L = mean((out - y)^2):
//   gz3 = 2 (out - y) / B * sigmoid(z3)
//   gw3 = sum gz3 h2b, gb3 = sum gz3;   gh2 = gz3 w3b
//   gz2 = gh2 * silu'(z2), gz2b = bf16(gz2)
//   gW2 = sum h1b gz2b^T, gb2 = sum gz2b; gh1 = W2 gz2b
//   gz1 = gh1 * silu'(z1), gz1b = bf16(gz1)
//   gW1 = sum xb gz1b^T,  gb1 = sum gz1b
// Weights live in shared memory in the layouts the B operand wants: W1T[n][k]
// (64 x 16, k >= 6 zero), W2T[n][k] = W2[k][n] (forward), W2R[n][k] = W2[n][k]
// (backward, where the roles of the two indices swap).
#pragma once
#include <cuda_bf16.h>

#include "tc_common.cuh"

namespace tc {

constexpr int MLP_IN = 6, MLP_H = 64, MLP_K1 = 16;
// packed FP32 parameter vector: W1[6][64], b1[64], W2[64][64], b2[64], w3[64], b3
constexpr int MLP_OW1 = 0, MLP_OB1 = MLP_OW1 + MLP_IN * MLP_H, MLP_OW2 = MLP_OB1 + MLP_H,
              MLP_OB2 = MLP_OW2 + MLP_H * MLP_H, MLP_OW3 = MLP_OB2 + MLP_H, MLP_OB3 = MLP_OW3 + MLP_H,
              MLP_NPAR = MLP_OB3 + 1;

// Shared-memory image of the network (bf16 matrices, fp32 vectors).
// row strides padded (24, 72 elements) so that the 8 rows a B-fragment load touches
// fall in different shared-memory banks
constexpr int MLP_LD1 = MLP_K1 + 8, MLP_LD2 = MLP_H + 8;
struct alignas(16) MlpSmem {
    alignas(16) __nv_bfloat16 W1T[MLP_H][MLP_LD1];
    alignas(16) __nv_bfloat16 W2T[MLP_H][MLP_LD2];
    alignas(16) __nv_bfloat16 W2R[MLP_H][MLP_LD2];
    float b1[MLP_H], b2[MLP_H], w3[MLP_H];  // w3 already rounded to bf16
    float b3;
};

// Fill from the packed FP32 parameters (cooperatively by the CTA; caller syncs).
__device__ __forceinline__ void mlp_load_smem(MlpSmem& S, const float* P) {
    for (int e = threadIdx.x; e < MLP_H * MLP_K1; e += blockDim.x) {
        const int k = e / MLP_H, n = e - k * MLP_H;
        S.W1T[n][k] = __float2bfloat16_rn(k < MLP_IN ? P[MLP_OW1 + k * MLP_H + n] : 0.f);
    }
    // W2 is read once, row by row, and stored in both layouts: reading it once per layout, the
    // transposed one with a stride of 64 floats, was most of a small batch's gradient pass
    // (4096 samples: 11.1 -> 9.4 us)
#pragma unroll 8
    for (int e = 2 * threadIdx.x; e < MLP_H * MLP_H; e += 2 * blockDim.x) {
        const int k = e / MLP_H, n = e - k * MLP_H;
        const float w0 = P[MLP_OW2 + e], w1 = P[MLP_OW2 + e + 1];
        const __nv_bfloat162 w = __floats2bfloat162_rn(w0, w1);
        S.W2T[n][k] = w.x;
        S.W2T[n + 1][k] = w.y;
        *reinterpret_cast<__nv_bfloat162*>(&S.W2R[k][n]) = w;
    }
    for (int e = threadIdx.x; e < MLP_H; e += blockDim.x) {
        S.b1[e] = P[MLP_OB1 + e];
        S.b2[e] = P[MLP_OB2 + e];
        S.w3[e] = __bfloat162float(__float2bfloat16_rn(P[MLP_OW3 + e]));
    }
    if (threadIdx.x == 0) S.b3 = P[MLP_OB3];
}

__device__ __forceinline__ unsigned pack_bf16(float lo, float hi) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);  // .x = lo (low half)
    return *reinterpret_cast<const unsigned*>(&v);
}
__device__ __forceinline__ float bf16r(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }

// D = A(16x16 bf16, row) * B(16x8 bf16, col) + D (fp32)
__device__ __forceinline__ void mma_bf16(float d[4], const unsigned a[4], unsigned b0, unsigned b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// B fragment (16 x 8, col layout) of the k-step kk, n-tile nt, from a [n][k] bf16 array.
template <int LD>
__device__ __forceinline__ void ldb(const __nv_bfloat16 (*M)[LD], int kk, int nt, unsigned& b0, unsigned& b1) {
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const __nv_bfloat16* row = &M[nt * 8 + g][kk * 16 + 2 * t];
    b0 = *reinterpret_cast<const unsigned*>(row);
    b1 = *reinterpret_cast<const unsigned*>(row + 8);
}

// sigmoid with the fast exponential and division intrinsics (a few float ulps, far
// below the BF16 rounding that follows every activation)
__device__ __forceinline__ float sigm(float z) { return __fdividef(1.f, 1.f + __expf(-z)); }
__device__ __forceinline__ float silu(float z) { return z * sigm(z); }
__device__ __forceinline__ float dsilu(float z) {
    const float s = sigm(z);
    return s * (1.f + z * (1.f - s));
}
__device__ __forceinline__ float softplus(float z) { return z > 20.f ? z : log1pf(expf(z)); }

// Accumulator tile 16 x 64: 8 n-tiles of m16n8, element (row g or g+8, col 8 nt + 2t (+1)).
struct Acc64 {
    float c[8][4];
};

// Rows of a C tile -> A fragments (16 x 64 bf16 = 4 k-steps) of the next product.
__device__ __forceinline__ void c_to_a(const Acc64& C, unsigned A[4][4]) {
#pragma unroll
    for (int kk = 0; kk < 4; kk++) {
        A[kk][0] = pack_bf16(C.c[2 * kk][0], C.c[2 * kk][1]);
        A[kk][1] = pack_bf16(C.c[2 * kk][2], C.c[2 * kk][3]);
        A[kk][2] = pack_bf16(C.c[2 * kk + 1][0], C.c[2 * kk + 1][1]);
        A[kk][3] = pack_bf16(C.c[2 * kk + 1][2], C.c[2 * kk + 1][3]);
    }
}

// ---- inference of 32 samples ----
__device__ __forceinline__ float ex2_fast(float x) {
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float rcp_fast(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
// silu of two values, each with its own exponential and reciprocal as in silu (the training
// pass), the rest in packed arithmetic.  One reciprocal of the product of both denominators put
// two more roundings into each value, and a bound on the exponentials in place of the values
// below z = -44.
__device__ __forceinline__ float2 silu2(float z0, float z1) {
    const float L2E = 1.44269504088896340736f;
    const float2 t = __fmul2_rn(make_float2(z0, z1), make_float2(-L2E, -L2E));
    const float2 d = __fadd2_rn(make_float2(ex2_fast(t.x), ex2_fast(t.y)), make_float2(1.f, 1.f));
    return __fmul2_rn(make_float2(z0, z1), make_float2(rcp_fast(d.x), rcp_fast(d.y)));
}
// B fragments of two k-steps (kk, kk+1) of n-tile nt from a [n][k] bf16 array in one ldmatrix.
template <int LD>
__device__ __forceinline__ void ldb2(const __nv_bfloat16 (*M)[LD], int kk, int nt, unsigned b[4]) {
    const int lane = threadIdx.x & 31;
    const unsigned a = smem_u32(&M[nt * 8 + (lane & 7)][kk * 16 + 8 * (lane >> 3)]);
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(b[0]), "=r"(b[1]), "=r"(b[2]), "=r"(b[3])
                 : "r"(a));
}

// Forward pass of 32 samples (two 16-row tiles sharing every weight fragment) whose features
// lie in xb as bf16 [sample][8] (6 features, 2 zeros).  Returns z3 of the sample this lane
// stands for: 16 (t >> 1) + 8 (t & 1) + g with g = lane / 4, t = lane % 4.
__device__ __forceinline__ float mlp_infer32(const MlpSmem& S, const __nv_bfloat16 (*xb)[8]) {
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    unsigned ax[2][2];
#pragma unroll
    for (int m = 0; m < 2; m++)
#pragma unroll
        for (int h = 0; h < 2; h++) ax[m][h] = *reinterpret_cast<const unsigned*>(&xb[16 * m + 8 * h + g][2 * t]);
    unsigned h1[2][4][4];
#pragma unroll
    for (int nt = 0; nt < 8; nt++) {
        const float2 b = *reinterpret_cast<const float2*>(&S.b1[8 * nt + 2 * t]);
        const unsigned w0 = *reinterpret_cast<const unsigned*>(&S.W1T[nt * 8 + g][2 * t]);
#pragma unroll
        for (int m = 0; m < 2; m++) {
            float z[4] = {b.x, b.y, b.x, b.y};
            const unsigned a[4] = {ax[m][0], ax[m][1], 0u, 0u};  // features k >= 8 are zero, and so is their weight row
            mma_bf16(z, a, w0, 0u);
            const float2 lo = silu2(z[0], z[1]), hi = silu2(z[2], z[3]);
            h1[m][nt >> 1][2 * (nt & 1)] = pack_bf16(lo.x, lo.y);
            h1[m][nt >> 1][2 * (nt & 1) + 1] = pack_bf16(hi.x, hi.y);
        }
    }
    float p[2][2] = {};
#pragma unroll
    for (int nt = 0; nt < 8; nt++) {
        unsigned w[2][4];
        ldb2<MLP_LD2>(S.W2T, 0, nt, w[0]);
        ldb2<MLP_LD2>(S.W2T, 2, nt, w[1]);
        const float2 b = *reinterpret_cast<const float2*>(&S.b2[8 * nt + 2 * t]);
        const float2 w3 = *reinterpret_cast<const float2*>(&S.w3[8 * nt + 2 * t]);
#pragma unroll
        for (int m = 0; m < 2; m++) {
            float z[4] = {b.x, b.y, b.x, b.y};
#pragma unroll
            for (int kk = 0; kk < 4; kk++) mma_bf16(z, h1[m][kk], w[kk >> 1][2 * (kk & 1)], w[kk >> 1][2 * (kk & 1) + 1]);
            const float2 lo = silu2(z[0], z[1]), hi = silu2(z[2], z[3]);
            const __nv_bfloat162 l = __floats2bfloat162_rn(lo.x, lo.y), h = __floats2bfloat162_rn(hi.x, hi.y);
            p[m][0] += w3.x * __low2float(l);
            p[m][0] += w3.y * __high2float(l);
            p[m][1] += w3.x * __low2float(h);
            p[m][1] += w3.y * __high2float(h);
        }
    }
#pragma unroll
    for (int m = 0; m < 2; m++)
#pragma unroll
        for (int h = 0; h < 2; h++) {
            p[m][h] += __shfl_xor_sync(0xffffffffu, p[m][h], 1);
            p[m][h] += __shfl_xor_sync(0xffffffffu, p[m][h], 2);
        }
    const float q0 = (t & 1) ? p[0][1] : p[0][0], q1 = (t & 1) ? p[1][1] : p[1][0];
    return ((t & 2) ? q1 : q0) + S.b3;
}

// The closure's inputs in float (the run's inference path; the training samples use
// les_features in double), as the network's BF16 inputs: the five invariants of S and O from
// the unique entries of the symmetric S and the antisymmetric O = {O01, O02, O12} (sc: the
// wall-unit scale), and the plane's y+ input.
__device__ __forceinline__ void les_features_bf16(const float G[3][3], float sc, float yp, __nv_bfloat16* out) {
    const float h = 0.5f * sc;
    const float s00 = G[0][0] * sc, s11 = G[1][1] * sc, s22 = G[2][2] * sc;
    const float s01 = (G[0][1] + G[1][0]) * h, s02 = (G[0][2] + G[2][0]) * h, s12 = (G[1][2] + G[2][1]) * h;
    const float a = (G[0][1] - G[1][0]) * h, b = (G[0][2] - G[2][0]) * h, c = (G[1][2] - G[2][1]) * h;
    // S^2 and O^2 (both symmetric)
    const float t00 = s00 * s00 + s01 * s01 + s02 * s02, t11 = s01 * s01 + s11 * s11 + s12 * s12,
                t22 = s02 * s02 + s12 * s12 + s22 * s22;
    const float t01 = s00 * s01 + s01 * s11 + s02 * s12, t02 = s00 * s02 + s01 * s12 + s02 * s22,
                t12 = s01 * s02 + s11 * s12 + s12 * s22;
    const float o00 = -(a * a + b * b), o11 = -(a * a + c * c), o22 = -(b * b + c * c);
    const float o01 = -b * c, o02 = a * c, o12 = -a * b;
    const float l1 = t00 + t11 + t22, l2 = o00 + o11 + o22;
    const float l3 = t00 * s00 + t11 * s11 + t22 * s22 + 2.f * (t01 * s01 + t02 * s02 + t12 * s12);
    const float l4 = o00 * s00 + o11 * s11 + o22 * s22 + 2.f * (o01 * s01 + o02 * s02 + o12 * s12);
    const float l5 = o00 * t00 + o11 * t11 + o22 * t22 + 2.f * (o01 * t01 + o02 * t02 + o12 * t12);
    uint4 v;
    v.x = pack_bf16(asinhf(l1), asinhf(l2));
    v.y = pack_bf16(asinhf(l3), asinhf(l4));
    v.z = pack_bf16(asinhf(l5), yp);
    v.w = 0u;
    *reinterpret_cast<uint4*>(out) = v;
}

// Forward pass of one 16-sample tile.  ax: A fragment of the features (16 x 16).
// Returns z1, z2 (pre-activations, for the backward pass), the h1b A fragments and
// z3 for the two rows (g, g+8) this lane holds.
__device__ __forceinline__ void mlp_forward_tile(const MlpSmem& S, const unsigned ax[4], Acc64& z1, Acc64& z2,
                                                 unsigned h1a[4][4], float z3[2]) {
    const int lane = threadIdx.x & 31, t = lane & 3;
#pragma unroll
    for (int nt = 0; nt < 8; nt++) {
        const float b0 = S.b1[8 * nt + 2 * t], b1 = S.b1[8 * nt + 2 * t + 1];
        z1.c[nt][0] = b0;
        z1.c[nt][1] = b1;
        z1.c[nt][2] = b0;
        z1.c[nt][3] = b1;
        unsigned w0, w1;
        ldb<MLP_LD1>(S.W1T, 0, nt, w0, w1);
        mma_bf16(z1.c[nt], ax, w0, w1);
    }
    Acc64 h1;
#pragma unroll
    for (int nt = 0; nt < 8; nt++)
#pragma unroll
        for (int e = 0; e < 4; e++) h1.c[nt][e] = silu(z1.c[nt][e]);
    c_to_a(h1, h1a);
#pragma unroll
    for (int nt = 0; nt < 8; nt++) {
        const float b0 = S.b2[8 * nt + 2 * t], b1 = S.b2[8 * nt + 2 * t + 1];
        z2.c[nt][0] = b0;
        z2.c[nt][1] = b1;
        z2.c[nt][2] = b0;
        z2.c[nt][3] = b1;
#pragma unroll
        for (int kk = 0; kk < 4; kk++) {
            unsigned w0, w1;
            ldb<MLP_LD2>(S.W2T, kk, nt, w0, w1);
            mma_bf16(z2.c[nt], h1a[kk], w0, w1);
        }
    }
    // z3 = w3 . bf16(silu(z2)) + b3: partial over this lane's columns, then the quad
    float p0 = 0.f, p1 = 0.f;
#pragma unroll
    for (int nt = 0; nt < 8; nt++)
#pragma unroll
        for (int e = 0; e < 2; e++) {
            const float w = S.w3[8 * nt + 2 * t + e];
            p0 += w * bf16r(silu(z2.c[nt][e]));
            p1 += w * bf16r(silu(z2.c[nt][2 + e]));
        }
    p0 += __shfl_xor_sync(0xffffffffu, p0, 1);
    p0 += __shfl_xor_sync(0xffffffffu, p0, 2);
    p1 += __shfl_xor_sync(0xffffffffu, p1, 1);
    p1 += __shfl_xor_sync(0xffffffffu, p1, 2);
    z3[0] = p0 + S.b3;
    z3[1] = p1 + S.b3;
}

// A fragment of a 16 x 16 feature tile from 16 rows of 6 floats (row r at X + r*ldx;
// rows >= nrow are zero).
__device__ __forceinline__ void feature_fragment(const float* X, int ldx, int nrow, unsigned ax[4]) {
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    float v[2][4];
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const int r = g + 8 * h;
#pragma unroll
        for (int j = 0; j < 2; j++) {
            const int k = 2 * t + j;
            v[h][j] = (r < nrow && k < MLP_IN) ? X[(size_t)r * ldx + k] : 0.f;
            v[h][2 + j] = 0.f;  // k = 2t+8+j >= 8 > 6
        }
    }
    ax[0] = pack_bf16(v[0][0], v[0][1]);
    ax[1] = pack_bf16(v[1][0], v[1][1]);
    ax[2] = 0u;
    ax[3] = 0u;
}

}  // namespace tc
