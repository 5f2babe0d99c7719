// k_srk.cu -- the pointwise passes of the collocated segregated Runge-Kutta step
// (collocated_SRK/func_global.h:317-408), fused around the one stencil each needs, the
// gradient.  A stage is: explicit term K_i of the stage velocity (k_flux_coll), the pressure
// right-hand side K_i - G buf + alpha v - d_i nu1 (one pass of this kernel), the pressure
// solve, and one pass that forms p_i = mu + buf, mu_i, q_i, K_i - G p_i, the next stage's
// velocity and the next stage's buf and p-hat.
// Bound by DRAM: the passes of a four-stage ARS step move about 120 words per node (3.1 ms at
// 384x384x257 mixed, 90% of the copy bandwidth).  As separate gradient, linear-combination
// and scalar kernels they moved 173 (4.4 ms) and took 17 launches more; the step with its
// diagnostics went from 7.28 to 5.84 ms, at 128x64x49 FP64 from 0.354 to 0.21 ms.
#include <algorithm>

#include "kernels.cuh"

namespace tc {

// Explicit roundings: the results of separate kernels, each storing its own, whatever the
// compiler would contract here (dp/dt, a difference of pressures over tau, shows every change
// of rounding of the float form 1e-4 of itself large).
__device__ __forceinline__ float r_add(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double r_add(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float r_mul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double r_mul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float r_fma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double r_fma(double a, double b, double c) { return __fma_rn(a, b, c); }

// W x-adjacent values as one access: 16 bytes, or 8 for float where NX is no multiple of 4
template <typename T, int W>
struct alignas(W * sizeof(T)) Vw {
    T v[W];
};
template <typename T, int W>
__device__ __forceinline__ Vw<T, W> ldw(const T* p) {
    return *reinterpret_cast<const Vw<T, W>*>(p);
}
template <typename T, int W>
__device__ __forceinline__ void stw(T* p, const Vw<T, W>& a) {
    *reinterpret_cast<Vw<T, W>*>(p) = a;
}

constexpr int SRX = 32, SRY = 8;  // threads along x (W nodes each) and rows per CTA

// SUM: the gradient's field is ga + gb (rounded), else ga.  Every load of a part is issued
// before its arithmetic: with one load per trip of a run-time loop the pass waited for
// memory (384x384x257 mixed: 0.98 / 0.49 ms per pass with / without SUM against 0.80 / 0.32).
// CTAs per SM: what still waits is hidden by more warps.  Three in place of two take 80
// registers a thread: 0.67 / 0.27 ms mixed, and FP64 256x192x128 1.86 to 1.67 ms per step;
// four, at 64, give the pass without SUM another 6% and spill 26 words of the one with it.
template <typename T, int W, bool SUM>
__global__ void __launch_bounds__(SRX* SRY, sizeof(T) == 4 && !SUM ? 4 : 3) k_srk_stage(SrkStage<T> a) {
    constexpr int MT = TC_SRK_MAX_STAGES;  // terms besides the first
    using V = Vw<T, W>;
    const Geom& g = a.g;
    pdl_launch();
    pdl_wait();
    const int NX = g.NX, NY = g.NY, NZ = g.NZ;
    const size_t NXY = (size_t)NX * NY, N = (size_t)g.N;
    const int x = W * (blockIdx.x * SRX + threadIdx.x % SRX), iy = blockIdx.y * SRY + threadIdx.x / SRX, z = blockIdx.z;
    if (x >= NX || iy >= NY) return;
    const size_t pl = (size_t)z * NXY, row = pl + (size_t)iy * NX, id = row + x;
    auto field = [&](size_t i) { return SUM ? r_add(a.ga[i], a.gb[i]) : a.ga[i]; };
    auto fieldw = [&](size_t i) {
        V r = ldw<T, W>(a.ga + i);
        if constexpr (SUM) {
            const V s = ldw<T, W>(a.gb + i);
#pragma unroll
            for (int j = 0; j < W; j++) r.v[j] = r_add(r.v[j], s.v[j]);
        }
        return r;
    };
    const bool wall = z == 0 || z == NZ - 1;
    V p0, xv;
    if (a.xs) xv = ldw<T, W>(a.xs + id);
    if (SUM || a.ga) {
        p0 = fieldw(id);
        V K[3], x0[3];
#pragma unroll
        for (int c = 0; c < 3; c++) {
            K[c] = ldw<T, W>(a.rhs + c * N + id);
            x0[c] = ldw<T, W>(a.x[0] + c * N + id);
        }
        if (!wall) {
            const T pl0 = field(row + (x == 0 ? NX - 1 : x - 1)), pr0 = field(row + (x + W == NX ? 0 : x + W));
            const V pym = fieldw(pl + (size_t)(iy == 0 ? NY - 1 : iy - 1) * NX + x),
                    pyp = fieldw(pl + (size_t)(iy + 1 == NY ? 0 : iy + 1) * NX + x), pzm = fieldw(id - NXY),
                    pzp = fieldw(id + NXY);
            const T hx = T(0.5) * (T)g.inv_hx, hy = T(0.5) * (T)g.inv_hy, ch = a.m.cellh[z];
            T e[W + 2];
            e[0] = pl0;
            e[W + 1] = pr0;
#pragma unroll
            for (int j = 0; j < W; j++) e[j + 1] = p0.v[j];
#pragma unroll
            for (int j = 0; j < W; j++) {
                K[0].v[j] = r_add(K[0].v[j], -r_mul(hx, r_add(e[j + 2], -e[j])));
                K[1].v[j] = r_add(K[1].v[j], -r_mul(hy, r_add(pyp.v[j], -pym.v[j])));
                K[2].v[j] = r_add(K[2].v[j], -(r_mul(T(0.5), r_add(pzp.v[j], -pzm.v[j])) / ch));
            }
        }
#pragma unroll
        for (int c = 0; c < 3; c++) {
            V q[MT];
#pragma unroll
            for (int k = 0; k < MT; k++)
                if (k + 1 < a.nt) q[k] = ldw<T, W>(a.x[k + 1] + c * N + id);
            if (a.kout) stw<T, W>(a.kout + c * N + id, K[c]);
            V acc;
            if (a.own_first) {  // K + c_0 x_0 + ...
#pragma unroll
                for (int j = 0; j < W; j++) acc.v[j] = r_fma(a.c[0], x0[c].v[j], K[c].v[j]);
            } else {
                acc = x0[c];
            }
#pragma unroll
            for (int k = 0; k < MT; k++)
                if (k + 1 < a.nt) {
#pragma unroll
                    for (int j = 0; j < W; j++) acc.v[j] = r_fma(a.c[k + 1], q[k].v[j], acc.v[j]);
                }
            if (!a.own_first) {  // ... then K
#pragma unroll
                for (int j = 0; j < W; j++) acc.v[j] = r_fma(a.c_own, K[c].v[j], acc.v[j]);
            }
            if (a.nu1) {
                V n;
#pragma unroll
                for (int j = 0; j < W; j++) n.v[j] = r_fma(a.alpha, x0[c].v[j], K[c].v[j]);
                stw<T, W>(a.nu1 + c * N + id, n);
            }
            stw<T, W>(a.vout + c * N + id, acc);
        }
    }
    if (!a.xs) return;
    V mu, qi, q[MT], r[MT], ph;  // this stage's mu and q; the earlier stages'
    if constexpr (SUM) mu = ldw<T, W>(a.ga + id);
#pragma unroll
    for (int k = 0; k < MT; k++)
        if (k < a.nj) {
            q[k] = ldw<T, W>(a.mujt[k] + id);
            if (a.stab) r[k] = ldw<T, W>(a.qj[k] + id);
        }
    if (a.stab && a.buf_out) ph = ldw<T, W>(a.p + id);
    if constexpr (SUM) {
        if (a.stab) {
            const V h = ldw<T, W>(a.pjhat + id);
#pragma unroll
            for (int j = 0; j < W; j++) qi.v[j] = r_mul(a.inv, r_add(p0.v[j], -h.v[j]));
            stw<T, W>(a.q_out + id, qi);
        }
#pragma unroll
        for (int j = 0; j < W; j++) mu.v[j] = r_fma(-a.cb, xv.v[j], mu.v[j]);
        if (a.mu_out) stw<T, W>(a.mu_out + id, mu);
        if (a.p_out) stw<T, W>(a.p_out + id, p0);
    }
    if (!a.buf_out) return;
    // the next stage's buf and p-hat
    V muj;
#pragma unroll
    for (int j = 0; j < W; j++) muj.v[j] = r_mul(a.c0, xv.v[j]);
#pragma unroll
    for (int k = 0; k < MT; k++)
        if (k < a.nj) {
#pragma unroll
            for (int j = 0; j < W; j++) {
                muj.v[j] = r_fma(a.cm[k], q[k].v[j], muj.v[j]);
            }
        }
    if constexpr (SUM) {
#pragma unroll
        for (int j = 0; j < W; j++) muj.v[j] = r_fma(a.cm[a.nj], mu.v[j], muj.v[j]);
    }
    if (a.stab) {
        if (a.use_cpd) {
#pragma unroll
            for (int j = 0; j < W; j++) ph.v[j] = r_fma(a.cpd, xv.v[j], ph.v[j]);
        }
#pragma unroll
        for (int k = 0; k < MT; k++)
            if (k < a.nj) {
#pragma unroll
                for (int j = 0; j < W; j++) ph.v[j] = r_fma(a.cq[k], r[k].v[j], ph.v[j]);
            }
        if constexpr (SUM) {
#pragma unroll
            for (int j = 0; j < W; j++) ph.v[j] = r_fma(a.cq[a.nj], qi.v[j], ph.v[j]);
        }
        stw<T, W>(a.pjhat + id, ph);
#pragma unroll
        for (int j = 0; j < W; j++)  // without stages before, c0 x + p-hat is one operation
            muj.v[j] = SUM ? r_add(muj.v[j], ph.v[j]) : r_fma(a.c0, xv.v[j], ph.v[j]);
    }
#pragma unroll
    for (int j = 0; j < W; j++) muj.v[j] = r_fma(-a.cb, xv.v[j], muj.v[j]);
    stw<T, W>(a.buf_out + id, muj);
}

template <typename T, int W>
static void srk_stage_w(const SrkStage<T>& a, cudaStream_t s) {
    const int nq = (a.g.NX + W - 1) / W;
    const dim3 grid((nq + SRX - 1) / SRX, (a.g.NY + SRY - 1) / SRY, a.g.NZ);
    if (a.gb) launch_pdl(a.g.pdl, k_srk_stage<T, W, true>, grid, SRX * SRY, 0, s, a);
    else launch_pdl(a.g.pdl, k_srk_stage<T, W, false>, grid, SRX * SRY, 0, s, a);
}

template <typename T>
void launch_srk_stage(const SrkStage<T>& a, cudaStream_t s) {
    // NX is even; every array of the step starts at a multiple of N values from an allocation
    if constexpr (sizeof(T) == 4) {
        if (a.g.NX % 4 == 0) return srk_stage_w<T, 4>(a, s);
    }
    srk_stage_w<T, 2>(a, s);
}
template void launch_srk_stage<double>(const SrkStage<double>&, cudaStream_t);
template void launch_srk_stage<float>(const SrkStage<float>&, cudaStream_t);

}  // namespace tc
