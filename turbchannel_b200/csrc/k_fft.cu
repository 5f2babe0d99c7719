// k_fft.cu -- the divergence kernel and the dispatch of the pressure solve's register FFTs
// (k_fft.cuh) by transform length; lengths without one keep the Stockham kernels of
// k_poisson.cu.  Same data layouts and results.
//   k_div_quad_z   : divergence of the vector RHS (streaming, 16-byte row loads)
//                    into a scratch real field.
#include "k_fft.cuh"
#include "stencil_div.cuh"

namespace tc {

// ---------------------------------------------------------------------------
// divergence of the vector RHS (streaming, 4 cells of a row per thread) and the
// forward x-FFT of a real field
// ---------------------------------------------------------------------------
// Same expressions as div_at (stencil_div.cuh), evaluated for x..x+3 from 16-byte row
// loads (NX % 4 == 0: the periodic wrap then moves whole 4-cell chunks), each thread
// marching over ZC consecutive planes of its 4-cell row: the w planes z-1 .. z+2 of the
// stencils stay in registers from one plane to the next (one new w load per plane
// instead of four; measured at 384x384x256, float: 0.188 ms with the x-FFT against 0.223
// ms for one plane per thread).
// Bounded for four CTAs per SM in float (64 registers) and three in double (80 registers;
// 0.351 against 0.359 ms with the x-FFT at 384x256x384; float with one CTA as the bound
// takes 79 registers and 0.193 against 0.184 ms)
template <typename T, int SCHEME, int ZC>
__global__ void __launch_bounds__(256, sizeof(T) == 8 ? 3 : 4) k_div_quad_z(DivFftArgs<T> a, T* __restrict__ out) {
    const Geom& g = a.g;
    pdl_launch();
    pdl_wait();
    const int NX = g.NX, NY = g.NY, NZ = g.NZ, NQ = NX >> 2, NZB = (NZ + ZC - 1) / ZC;
    const long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= (long long)NQ * NY * NZB) return;
    const int row = (int)(q / NQ), x = (int)(q - (long long)row * NQ) * 4;
    // float: plane chunks in descending z, the float flux kernel's last-written planes (high
    // z) being the ones still in L2 (divergence + x-FFT 0.177 against 0.179 ms at
    // 384x256x384); double keeps ascending chunks (the FP64 flux kernel writes in z-chunks,
    // and descending took 0.377 against 0.353 ms)
    const int y = row % NY, z0 = (sizeof(T) == 4 ? NZB - 1 - row / NY : row / NY) * ZC;
    const size_t NXY = (size_t)NX * NY, col = (size_t)y * NX + x;
    const T *u = a.v.c[0], *v = a.v.c[1], *w = a.v.c[2];
    const T ihx = (T)g.inv_hx, ihy = (T)g.inv_hy;
    const int xq = x + 4 == NX ? 0 : x + 4, xm = x == 0 ? NX - 1 : x - 1;
    const int yp = y + 1 == NY ? 0 : y + 1, ym = y == 0 ? NY - 1 : y - 1;
    const int ypp = yp + 1 == NY ? 0 : yp + 1;
    auto ldw = [&](int zz) {
        Acc4<T> r;
        if (zz >= 0 && zz < NZ) r = ld4(w + (size_t)zz * NXY + col);
        else
#pragma unroll
            for (int k = 0; k < 4; k++) r.v[k] = T(0);
        return r;
    };
    Acc4<T> Wz[4];  // w at the planes z-1, z, z+1, z+2
    Wz[0] = ldw(z0 - 1);
    Wz[1] = ldw(z0);
    Wz[2] = ldw(z0 + 1);
    Wz[3] = ldw(z0 + 2);
#pragma unroll
    for (int kz = 0; kz < ZC; kz++) {
        const int z = z0 + kz;
        if (z >= NZ) break;
        if (kz > 0) {
            Wz[0] = Wz[1];
            Wz[1] = Wz[2];
            Wz[2] = Wz[3];
            Wz[3] = ldw(z + 2);
        }
        const size_t pl = (size_t)z * NXY, rb = pl + (size_t)y * NX, id = rb + x;
        T e[9];  // u at x-1 .. x+7
        {
            const Acc4<T> U0 = ld4(u + id), U1 = ld4(u + rb + xq);
            e[0] = u[rb + xm];
#pragma unroll
            for (int k = 0; k < 4; k++) {
                e[1 + k] = U0.v[k];
                e[5 + k] = U1.v[k];
            }
        }
        T d[4];
        if constexpr (SCHEME == TC_SCHEME_VV4) {
            const T C27 = T(0.03703703703703703703);
            const T dz = a.m.DZ[z], dzw = a.m.DZW[z];
            const Acc4<T> V0 = ld4(v + id), Vp = ld4(v + pl + (size_t)yp * NX + x),
                          Vpp = ld4(v + pl + (size_t)ypp * NX + x), Vm = ld4(v + pl + (size_t)ym * NX + x);
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const T W0 = Wz[1].v[k];
                const T Wr = z == NZ - 1 ? T(0) : Wz[2].v[k];
                const T Wrr = z == NZ - 1 ? W0 : (z == NZ - 2 ? T(0) : Wz[3].v[k]);
                const T Wll = z == 0 ? Wz[2].v[k] : (z == 1 ? T(0) : Wz[0].v[k]);
                const T dudx = ihx * (dz * (e[k + 2] - e[k + 1]) - C27 * dzw * (e[k + 3] - e[k]));
                const T dvdy = ihy * (dz * (Vp.v[k] - V0.v[k]) - C27 * dzw * (Vpp.v[k] - Vm.v[k]));
                d[k] = dudx + dvdy + (Wr - W0) - C27 * (Wrr - Wll);
            }
        } else if constexpr (SCHEME == TC_SCHEME_HW2) {
            const T hz = a.m.DZ[z];
            const Acc4<T> V0 = ld4(v + id), Vp = ld4(v + pl + (size_t)yp * NX + x);
#pragma unroll
            for (int k = 0; k < 4; k++)
                d[k] = (e[k + 2] - e[k + 1]) * ihx * hz + (Vp.v[k] - V0.v[k]) * ihy * hz +
                       ((z < NZ - 1) ? (Wz[2].v[k] - Wz[1].v[k]) : (-Wz[1].v[k]));
        } else {
            const T hz = a.m.cellh[z], hx = (T)g.hx, hy = (T)g.hy;
            const Acc4<T> Vp = ld4(v + pl + (size_t)yp * NX + x), Vm = ld4(v + pl + (size_t)ym * NX + x);
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const T Wa = z == 0 ? Wz[2].v[k] : (z == NZ - 1 ? Wz[1].v[k] : Wz[2].v[k]);
                const T Wb = z == 0 ? Wz[1].v[k] : Wz[0].v[k];
                T dd = 0;
                dd += T(0.5) * (e[k + 2] - e[k]) * hy * hz;
                dd += T(0.5) * (Vp.v[k] - Vm.v[k]) * hx * hz;
                dd += T(0.5) * (Wa - Wb) * hx * hy;
                d[k] = dd;
            }
        }
        if constexpr (sizeof(T) == 4) {
            *reinterpret_cast<float4*>(out + id) = make_float4(d[0], d[1], d[2], d[3]);
        } else {
            reinterpret_cast<double2*>(out + id)[0] = make_double2(d[0], d[1]);
            reinterpret_cast<double2*>(out + id)[1] = make_double2(d[2], d[3]);
        }
    }
}

constexpr int DIV_ZC = 4;  // planes per thread of k_div_quad_z
template <typename T>
static void div_quad_launch(const DivFftArgs<T>& a, T* out, cudaStream_t s) {
    const long long nq = (long long)(a.g.NX / 4) * a.g.NY * ((a.g.NZ + DIV_ZC - 1) / DIV_ZC);
    const unsigned nb = (unsigned)((nq + 255) / 256);
    if (a.g.scheme == TC_SCHEME_VV4) launch_pdl(a.g.pdl, k_div_quad_z<T, TC_SCHEME_VV4, DIV_ZC>, nb, 256, 0, s, a, out);
    else if (a.g.scheme == TC_SCHEME_HW2) launch_pdl(a.g.pdl, k_div_quad_z<T, TC_SCHEME_HW2, DIV_ZC>, nb, 256, 0, s, a, out);
    else launch_pdl(a.g.pdl, k_div_quad_z<T, TC_SCHEME_COLLOC, DIV_ZC>, nb, 256, 0, s, a, out);
}

// ---------------------------------------------------------------------------
// dispatch on the transform length
// ---------------------------------------------------------------------------
#define TC_FFT_SIZES(X) X(16) X(24) X(32) X(48) X(64) X(96) X(128) X(192) X(256) X(384) X(512) X(768) X(1024)
TC_FFT_LENGTHS(s, TC_FFT_SIZES)

// The register transforms of the other 2^a 3^b (k_fft_m.cu, k_fft_l.cu), and of y-counts that
// no power-of-two tile of rows divides, are not used by the mixed SRK step: its dp/dt is a
// difference of pressures over tau, which any other rounding of a float transform moves by
// 1e-4 of itself (k_zsolve.cu keeps its z-solve for the same reason).
template <typename T>
static bool fft_keep(const Geom& g) {
    return sizeof(T) == 4 && g.norm_srk != 0;
}

template <typename T>
bool launch_yfft_reg(const YFftArgs<T>& a, cudaStream_t s) {
    if (yfft_s<T>(a, s)) return true;
    return !fft_keep<T>(a.g) && (yfft_m<T>(a, s) || yfft_l<T>(a, s));
}

template <typename T>
static bool xfft_any(const DivFftArgs<T>& a, const T* src, cudaStream_t s) {
    if (fft_keep<T>(a.g)) return a.g.NY % 8 == 0 && xfft_s<T>(a, src, s);
    return xfft_s<T>(a, src, s) || xfft_m<T>(a, src, s) || xfft_l<T>(a, src, s);
}

// Whether an x-FFT kernel takes these lines (the vector RHS is put through the divergence
// only then).
static bool xfft_has(const Geom& g, bool keep) {
    if (g.NX > 1024 || g.NY % 6 * (g.NY % 8) != 0) return false;
    switch (g.NX) {
#define TC_HAS(n) case n:
        TC_FFT_SIZES(TC_HAS)
#undef TC_HAS
        return !keep || g.NY % 8 == 0;
        default: return !keep;
    }
}

// The vector RHS first goes through the divergence into a.dtmp (a scratch field), then the
// real field is transformed.
template <typename T>
int launch_div_xfft_reg(const DivFftArgs<T>& a, cudaStream_t s) {
    const bool vec = a.src_scalar == nullptr, keep = fft_keep<T>(a.g);
    if (vec && (a.dtmp == nullptr || (keep && a.g.NX % 4 != 0))) return 0;
    if (!vec) return xfft_any<T>(a, a.src_scalar, s) ? 1 : 0;
    if (!xfft_has(a.g, keep)) return 0;
    if (a.g.NX % 4 == 0) {
        div_quad_launch<T>(a, a.dtmp, s);
    } else {
        const DivArgs<T> d{a.g, a.m, a.v, a.dtmp};
        launch_divergence<T>(d, s);
    }
    return xfft_any<T>(a, a.dtmp, s) ? 2 : 0;
}

template <typename T>
bool launch_ixfft_reg(const IxFftArgs<T>& a, cudaStream_t s) {
    if (fft_keep<T>(a.g)) return a.g.NY % 8 == 0 && ixfft_s<T>(a, s);
    return ixfft_s<T>(a, s) || ixfft_m<T>(a, s) || ixfft_l<T>(a, s);
}

// The divergence pass alone (for the plane transforms of k_fft_plane.cu): false when the
// vector RHS has no scratch or NX % 4 != 0.
template <typename T>
bool launch_div_quad(const DivFftArgs<T>& a, cudaStream_t s) {
    if (a.dtmp == nullptr || a.g.NX % 4 != 0) return false;
    div_quad_launch<T>(a, a.dtmp, s);
    return true;
}

template bool launch_div_quad<double>(const DivFftArgs<double>&, cudaStream_t);
template bool launch_div_quad<float>(const DivFftArgs<float>&, cudaStream_t);
template bool launch_yfft_reg<double>(const YFftArgs<double>&, cudaStream_t);
template bool launch_yfft_reg<float>(const YFftArgs<float>&, cudaStream_t);
template int launch_div_xfft_reg<double>(const DivFftArgs<double>&, cudaStream_t);
template int launch_div_xfft_reg<float>(const DivFftArgs<float>&, cudaStream_t);
template bool launch_ixfft_reg<double>(const IxFftArgs<double>&, cudaStream_t);
template bool launch_ixfft_reg<float>(const IxFftArgs<float>&, cudaStream_t);

}  // namespace tc
