// k_fft.cuh -- the pressure solve's line transforms for the lengths that have a compiled
// two-pass register transform (fft_reg.cuh); k_fft.cu, k_fft_m.cu and k_fft_l.cu instantiate
// them for their lengths.
//   k_xfft_reg     : forward x-FFT of `rows` y-rows of a real field (the divergence
//                    or the scalar RHS), two rows packed as one complex line,
//                    unpacked to spec[z][kx][y] (kx = 0..NX/2);
//   k_yfft_reg     : complex FFT of contiguous y-lines of spec, in place, straight
//                    from and back to global memory;
//   k_ixfft_reg    : Hermitian-extended half spectrum of two rows packed as one
//                    complex line, inverse x-FFT, scaled real rows into p.
#pragma once
#include <algorithm>

#include "fft_reg.cuh"
#include "kernels.cuh"

namespace tc {

// ---------------------------------------------------------------------------
// y-FFT
// ---------------------------------------------------------------------------
constexpr int YFFT_LINE_BUDGET = 128;  // lines x N1 per CTA
// Lines per CTA: few (8 at N = 384: 26 KB of shared memory in float, 51 KB in double),
// so that many CTAs share an SM and hide each other's global-memory latency (measured
// at 384 x 384 x 256: 32 float lines per CTA 0.082 ms, 16 lines 0.074, 8 lines 0.058).
template <typename T, int N>
constexpr int yfft_reg_lines() {
    const int l = YFFT_LINE_BUDGET / FftSplit<N>::N1;
    return l < 1 ? 1 : l;
}

template <typename T, int N, int SIGN>
__global__ void __launch_bounds__(256) k_yfft_reg(cplx<T>* spec, long long nlines, const cplx<T>* __restrict__ tw) {
    constexpr int N1 = FftSplit<N>::N1, N2 = FftSplit<N>::N2, YL = FftSplit<N>::YL;
    constexpr int LINES = yfft_reg_lines<T, N>();
    extern __shared__ __align__(16) unsigned char smraw[];
    cplx<T>* Y = reinterpret_cast<cplx<T>*>(smraw);
    pdl_launch();
    pdl_wait();
    // the forward transform takes the lines in descending z, the reverse of the x-FFT that
    // wrote them (its last planes are still in L2), and leaves the low planes, which the
    // z-solve's forward sweep reads first, written last (384x256x384 float: y-FFT 0.052
    // against 0.059 ms, z-solve 0.144 against 0.152; double 0.097 / 0.283 against 0.101 / 0.292)
    const long long blk = SIGN < 0 ? (long long)gridDim.x - 1 - blockIdx.x : (long long)blockIdx.x;
    const long long L0 = blk * LINES;
    const int nl = (int)min((long long)LINES, nlines - L0);
    cplx<T>* base = spec + L0 * N;
    for (int it = threadIdx.x; it < nl * N2; it += blockDim.x) {
        const int l = it / N2, n2 = it - l * N2;
        const cplx<T>* src = base + (size_t)l * N + n2;
        cplx<T> v[N1];
#pragma unroll
        for (int n1 = 0; n1 < N1; n1++) v[n1] = src[n1 * N2];
        fft_pass_a<T, N, SIGN>(v, n2, tw, Y + l * YL);
    }
    __syncthreads();
    for (int it = threadIdx.x; it < nl * N1; it += blockDim.x) {
        const int l = it / N1, k1 = it - l * N1;
        cplx<T> v[N2];
        fft_pass_b<T, N, SIGN>(v, k1, Y + l * YL);
        cplx<T>* dst = base + (size_t)l * N + k1;
#pragma unroll
        for (int k2 = 0; k2 < N2; k2++) dst[k2 * N1] = v[k2];
    }
}

template <typename T, int N>
static void yfft_reg_launch(const YFftArgs<T>& a, cudaStream_t s) {
    constexpr int LINES = yfft_reg_lines<T, N>();
    const long long total = (long long)a.g.NZ * a.g.NXH;
    const size_t smem = (size_t)LINES * FftSplit<N>::YL * sizeof(cplx<T>);
    auto k = a.sign < 0 ? k_yfft_reg<T, N, -1> : k_yfft_reg<T, N, +1>;
    smem_limit(k, smem);
    launch_pdl(a.g.pdl, k, (unsigned)((total + LINES - 1) / LINES), 256, smem, s, a.spec, total, a.twy);
}

// ---------------------------------------------------------------------------
// forward x-FFT of a real field
// ---------------------------------------------------------------------------
// ceil(2^32 / n): __umulhi(e, fft_magic(n)) = e / n for e n < 2^32 (n = 1: see the caller).
static inline unsigned fft_magic(int n) { return 0xffffffffu / (unsigned)n + 1u; }

// Whether the forward x-FFT of `rows` rows (256 threads) keeps its transformed lines in
// the first pass's buffer: one second-pass line segment per thread at most.
template <int N>
__host__ __device__ constexpr bool xfft_alias(int rows) {
    return (rows / 2) * FftSplit<N>::N1 <= 256;
}

// Three CTAs per SM in float (79 registers at N = 384, no spill), two in double.
template <typename T, int N>
__global__ void __launch_bounds__(256, sizeof(T) == 4 ? 3 : 2) k_xfft_reg(DivFftArgs<T> a, const T* src, int rows, unsigned mrows) {
    constexpr int N1 = FftSplit<N>::N1, N2 = FftSplit<N>::N2, YL = FftSplit<N>::YL, ZS = N + 1;
    extern __shared__ __align__(16) unsigned char smraw[];
    const Geom& g = a.g;
    pdl_launch();
    pdl_wait();
    const int NY = g.NY, NXH = N / 2 + 1, nl = rows >> 1;
    cplx<T>* Y = reinterpret_cast<cplx<T>*>(smraw);
    // transformed lines, stride N+1: over Y itself when every thread holds at most one
    // line segment of the second pass (read all, barrier, write), else after Y
    const bool alias = xfft_alias<N>(rows);
    cplx<T>* Zs = alias ? Y : Y + nl * YL;
    const int z = blockIdx.y, y0 = blockIdx.x * rows;
    const T* plane = src + ((size_t)z * NY + y0) * N;
    for (int it = threadIdx.x; it < nl * N2; it += blockDim.x) {
        const int l = it / N2, n2 = it - l * N2;
        const T* d0 = plane + (size_t)(2 * l) * N + n2;
        cplx<T> v[N1];
#pragma unroll
        for (int n1 = 0; n1 < N1; n1++) v[n1] = {d0[n1 * N2], d0[N + n1 * N2]};
        fft_pass_a<T, N, -1>(v, n2, a.twx, Y + l * YL);
    }
    __syncthreads();
    if (alias) {
        const bool mine = (int)threadIdx.x < nl * N1;
        const int l = threadIdx.x / N1, k1 = threadIdx.x - l * N1;
        cplx<T> v[N2];
        if (mine) fft_pass_b<T, N, -1>(v, k1, Y + l * YL);
        __syncthreads();
        if (mine) {
            cplx<T>* zl = Zs + l * ZS + k1;
#pragma unroll
            for (int k2 = 0; k2 < N2; k2++) zl[k2 * N1] = v[k2];
        }
    } else {
        for (int it = threadIdx.x; it < nl * N1; it += blockDim.x) {
            const int l = it / N1, k1 = it - l * N1;
            cplx<T> v[N2];
            fft_pass_b<T, N, -1>(v, k1, Y + l * YL);
            cplx<T>* zl = Zs + l * ZS + k1;
#pragma unroll
            for (int k2 = 0; k2 < N2; k2++) zl[k2 * N1] = v[k2];
        }
    }
    __syncthreads();
    // unpack the two real rows of each line: X_a = (Z_k + conj Z_{N-k}) / 2, X_b = (Z_k - conj Z_{N-k}) / 2i
    for (int e = threadIdx.x; e < NXH * rows; e += blockDim.x) {
        const int kx = (int)__umulhi((unsigned)e, mrows), r = e - kx * rows, l = r >> 1;
        const cplx<T> Zk = Zs[l * ZS + kx], Zm = Zs[l * ZS + (kx == 0 ? 0 : N - kx)];
        cplx<T> val;
        if ((r & 1) == 0) val = {T(0.5) * (Zk.x + Zm.x), T(0.5) * (Zk.y - Zm.y)};
        else val = {T(0.5) * (Zk.y + Zm.y), -T(0.5) * (Zk.x - Zm.x)};
        a.spec[((size_t)z * NXH + kx) * NY + y0 + r] = val;
    }
}

template <typename T, int N>
static size_t div_xfft_reg_smem(int rows) {
    return (size_t)(rows / 2) * (FftSplit<N>::YL + (xfft_alias<N>(rows) ? 0 : N + 1)) * sizeof(cplx<T>);
}

template <typename T, int N>
static void xfft_reg_launch(const DivFftArgs<T>& a, const T* src, int rows, cudaStream_t s) {
    const size_t smem = div_xfft_reg_smem<T, N>(rows);
    auto k = k_xfft_reg<T, N>;
    smem_limit(k, smem);
    launch_pdl(a.g.pdl, k, dim3(a.g.NY / rows, a.g.NZ), 256, smem, s, a, src, rows, fft_magic(rows));
}

// ---------------------------------------------------------------------------
// inverse x-FFT, persistent and double-buffered (float)
// ---------------------------------------------------------------------------
constexpr int XP_NT = 256;
// Shared memory of an SM's CTAs, at most: the rest is the L1 that the twiddle factors stay in
// (512x512x256 float: 145 us with two CTAs of 107 KB, 114 with two of 74 KB).
constexpr size_t XP_SMEM = 204 * 1024;
// Row stride of a tile of half spectra, tile[kx * stride + row]: neighbouring lanes gather
// the 16 bytes of two rows (float; one row in double) of neighbouring kx, which this stride
// spreads over all banks.
template <typename T>
__host__ __device__ constexpr int ixfft_stride(int rows) {
    return sizeof(T) == 4 ? (rows / 2 | 1) * 2 : rows | 1;
}
// rows r, r + 1 of a tile row (r even)
template <typename T>
__device__ __forceinline__ void ld_rows(const cplx<T>* t, cplx<T>& a, cplx<T>& b) {
    if constexpr (sizeof(T) == 4) {
        const float4 q = *reinterpret_cast<const float4*>(t);
        a = {q.x, q.y};
        b = {q.z, q.w};
    } else {
        a = t[0];
        b = t[1];
    }
}

// As k_ixfft_reg (the Hermitian-extended half spectrum of two rows per complex line, inverse
// transform, scaled rows into p), with each CTA walking tiles of RB (16) y-values of one plane
// and copying the next tile's half spectrum (NX/2+1 rows of RB contiguous values) into its
// second buffer while it transforms the current one.  Bound by DRAM, 4.8 TB/s at 512x512x256
// float (0.114 ms) and 4.5 at 384x384x256 (0.068).
template <typename T, int N>
struct IPipe {
    static constexpr int RB = sizeof(T) == 4 ? 16 : 8, NL = RB / 2, TS = ixfft_stride<T>(RB), NXH = N / 2 + 1;
    static constexpr int PC = 16 / sizeof(cplx<T>), CPK = RB / PC;  // 16-byte chunks per kx row
    static constexpr size_t tile = (size_t)NXH * TS * sizeof(cplx<T>), y = (size_t)NL * FftSplit<N>::YL * sizeof(cplx<T>);
    static constexpr size_t shared = 2 * (tile > y ? tile : y), own = 2 * tile + y;
    // alias: the first pass is written over the tile it was gathered from (every thread holds
    // at most one line segment), else to a buffer of its own after the two tiles.  It costs a
    // barrier, and is worth it for the shared memory: not where that still gives one CTA per
    // SM either way (NX = 768: 82 us with a buffer, 104 without at 768x384x128).
    static constexpr bool alias = NL * FftSplit<N>::N2 <= XP_NT && (2 * shared <= XP_SMEM || own > XP_SMEM);
    static constexpr size_t buf = ((alias ? shared / 2 : tile) + 15) / 16 * 16;
    static constexpr size_t smem = 2 * buf + (alias ? 0 : y);
};

template <typename T, int N>
__global__ void __launch_bounds__(XP_NT) k_ixfft_pipe(IxFftArgs<T> a) {
    using P = IPipe<T, N>;
    constexpr int RB = P::RB, NL = P::NL, TS = P::TS, NXH = P::NXH, PC = P::PC, CPK = P::CPK;
    constexpr int N1 = FftSplit<N>::N1, N2 = FftSplit<N>::N2, YL = FftSplit<N>::YL, NH = N / 2;
    extern __shared__ __align__(16) unsigned char smraw[];
    const Geom& g = a.g;
    const int NY = g.NY, YB = NY / RB;
    const long long ntile = (long long)YB * g.NZ;
    pdl_launch();
    pdl_wait();
    // tiles in ascending z: the correction that reads p next walks the planes downwards,
    // so that the next step's flux kernel, which starts at z = 0, finds the low planes of
    // the new velocity in L2 (at 384x256x384 the flux kernel gains more, 7 us, than this
    // kernel loses against descending tiles, 1.5 us)
    auto fetch = [&](long long t, int b) {
        const int z = (int)(t / YB), y0 = (int)(t - (long long)z * YB) * RB;
        cplx<T>* tile = reinterpret_cast<cplx<T>*>(smraw + b * P::buf);
        for (int e = threadIdx.x; e < NXH * CPK; e += XP_NT) {
            const int kx = e / CPK, c = e - kx * CPK;
            cp_async<16>(tile + kx * TS + c * PC, a.spec + ((size_t)z * NXH + kx) * NY + y0 + c * PC);
        }
    };
    long long t = blockIdx.x;
    if (t < ntile) fetch(t, 0);
    cp_async_commit();
    const T sc = a.scale;
    for (int b = 0; t < ntile; t += gridDim.x, b ^= 1) {
        if (t + gridDim.x < ntile) fetch(t + gridDim.x, b ^ 1);
        cp_async_commit();
        cp_async_wait<1>();
        __syncthreads();  // tile t is in buffer b
        const int z = (int)(t / YB), y0 = (int)(t - (long long)z * YB) * RB;
        cplx<T>* tile = reinterpret_cast<cplx<T>*>(smraw + b * P::buf);
        cplx<T>* Y = P::alias ? tile : reinterpret_cast<cplx<T>*>(smraw + 2 * P::buf);
        // the Hermitian-extended line of rows 2l, 2l+1 at the first pass's positions
        auto gather = [&](int l, int n2, cplx<T>(&v)[N1]) {
#pragma unroll
            for (int n1 = 0; n1 < N1; n1++) {
                const int k = N2 * n1 + n2;
                const bool up = k > NH;
                cplx<T> av, bv;
                ld_rows(tile + (up ? N - k : k) * TS + 2 * l, av, bv);
                if (up) {
                    av.y = -av.y;
                    bv.y = -bv.y;
                }
                if (k == 0 || k == NH) {
                    av.y = 0;
                    bv.y = 0;
                }
                v[n1] = {av.x - bv.y, av.y + bv.x};
            }
        };
        if constexpr (P::alias) {
            const bool mine = (int)threadIdx.x < NL * N2;
            const int l = threadIdx.x / N2, n2 = threadIdx.x - l * N2;
            cplx<T> v[N1];
            if (mine) gather(l, n2, v);
            __syncthreads();
            if (mine) fft_pass_a<T, N, +1>(v, n2, a.twx, Y + l * YL);
        } else {
            for (int it = threadIdx.x; it < NL * N2; it += XP_NT) {
                const int l = it / N2, n2 = it - l * N2;
                cplx<T> v[N1];
                gather(l, n2, v);
                fft_pass_a<T, N, +1>(v, n2, a.twx, Y + l * YL);
            }
        }
        __syncthreads();
        for (int it = threadIdx.x; it < NL * N1; it += XP_NT) {
            const int l = it / N1, k1 = it - l * N1;
            cplx<T> v[N2];
            fft_pass_b<T, N, +1>(v, k1, Y + l * YL);
            T* pa = a.p + ((size_t)z * NY + y0 + 2 * l) * N + k1;
            T* pb = pa + N;
#pragma unroll
            for (int k2 = 0; k2 < N2; k2++) {
                pa[k2 * N1] = v[k2].x * sc;
                pb[k2 * N1] = v[k2].y * sc;
            }
        }
        __syncthreads();  // buffer b (and Y) are refilled by the next iterations
    }
}

template <typename T, int N>
static bool ixfft_pipe_launch(const IxFftArgs<T>& a, cudaStream_t s) {
    // float only: in double the tiles halve and the k_ixfft_reg form measured faster
    if constexpr (sizeof(T) != 4) {
        return false;
    } else {
        using P = IPipe<T, N>;
        if (a.g.NY % P::RB != 0) return false;
        auto k = k_ixfft_pipe<T, N>;
        // per size and device (function attributes are per device), resolved at the first launch
        constexpr int MAXDEV = 64;
        static int sms_of[MAXDEV] = {}, occ_of[MAXDEV] = {};  // occ 0: not resolved yet, -1: does not fit
        int dev = 0;
        cudaGetDevice(&dev);
        if (dev < 0 || dev >= MAXDEV) return false;
        if (occ_of[dev] == 0) {
            int optin = 0, o = 0, n = 0;
            cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
            cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
            if (P::smem <= (size_t)optin) {
                cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)P::smem);
                cudaOccupancyMaxActiveBlocksPerMultiprocessor(&o, k, XP_NT, P::smem);
                o = std::min(o, std::max(1, (int)(XP_SMEM / P::smem)));
            }
            sms_of[dev] = n;
            occ_of[dev] = o > 0 ? o : -1;
        }
        const int occ = occ_of[dev], sms = sms_of[dev];
        if (occ < 1) return false;
        const long long ntile = (long long)(a.g.NY / P::RB) * a.g.NZ;
        const int grid = (int)std::min<long long>(ntile, (long long)sms * occ);
        launch_pdl(a.g.pdl, k, grid, XP_NT, P::smem, s, a);
        return true;
    }
}

// ---------------------------------------------------------------------------
// inverse x-FFT
// ---------------------------------------------------------------------------
template <typename T, int N>
__global__ void __launch_bounds__(512) k_ixfft_reg(IxFftArgs<T> a, int rows, unsigned mchunks, int alias) {
    constexpr int N1 = FftSplit<N>::N1, N2 = FftSplit<N>::N2, YL = FftSplit<N>::YL, NH = N / 2, NXH = NH + 1;
    constexpr int PC = 16 / sizeof(cplx<T>);  // complex values per 16-byte chunk
    extern __shared__ __align__(16) unsigned char smraw[];
    const Geom& g = a.g;
    pdl_launch();
    pdl_wait();
    const int NY = g.NY, nl = rows >> 1, TS = ixfft_stride<T>(rows);
    cplx<T>* tile = reinterpret_cast<cplx<T>*>(smraw);  // tile[kx * TS + r]
    // alias: the first pass's output over the tile itself, every thread holding at most
    // one line segment (gather all, barrier, transform and write); else after the tile
    cplx<T>* Y = alias ? tile : tile + NXH * TS;
    // planes in descending z, the reverse of the inverse y-FFT that wrote them
    const int z = gridDim.y - 1 - blockIdx.y, y0 = blockIdx.x * rows;
    {
        const int cpr = rows / PC;
        for (int e = threadIdx.x; e < NXH * cpr; e += blockDim.x) {
            const int kx = (int)__umulhi((unsigned)e, mchunks), c = e - kx * cpr;
            cp_async<16>(tile + kx * TS + c * PC, a.spec + ((size_t)z * NXH + kx) * NY + y0 + c * PC);
        }
        cp_async_commit();
        cp_async_wait<0>();
    }
    __syncthreads();
    // the Hermitian-extended line of two packed rows at the first pass's positions
    auto gather = [&](int l, int n2, cplx<T>(&v)[N1]) {
#pragma unroll
        for (int n1 = 0; n1 < N1; n1++) {
            const int k = N2 * n1 + n2;
            const bool up = k > NH;
            const cplx<T>* t = tile + (up ? N - k : k) * TS + 2 * l;
            cplx<T> av, bv;
            ld_rows(t, av, bv);
            if (up) {
                av.y = -av.y;
                bv.y = -bv.y;
            }
            if (k == 0 || k == NH) {
                av.y = 0;
                bv.y = 0;
            }
            v[n1] = {av.x - bv.y, av.y + bv.x};
        }
    };
    if (alias) {
        const bool mine = (int)threadIdx.x < nl * N2;
        const int l = threadIdx.x / N2, n2 = threadIdx.x - l * N2;
        cplx<T> v[N1];
        if (mine) gather(l, n2, v);
        __syncthreads();
        if (mine) fft_pass_a<T, N, +1>(v, n2, a.twx, Y + l * YL);
    } else {
        for (int it = threadIdx.x; it < nl * N2; it += blockDim.x) {
            const int l = it / N2, n2 = it - l * N2;
            cplx<T> v[N1];
            gather(l, n2, v);
            fft_pass_a<T, N, +1>(v, n2, a.twx, Y + l * YL);
        }
    }
    __syncthreads();
    const T sc = a.scale;
    for (int it = threadIdx.x; it < nl * N1; it += blockDim.x) {
        const int l = it / N1, k1 = it - l * N1;
        cplx<T> v[N2];
        fft_pass_b<T, N, +1>(v, k1, Y + l * YL);
        T* pa = a.p + ((size_t)z * NY + y0 + 2 * l) * N + k1;
        T* pb = pa + N;
#pragma unroll
        for (int k2 = 0; k2 < N2; k2++) {
            pa[k2 * N1] = v[k2].x * sc;
            pb[k2 * N1] = v[k2].y * sc;
        }
    }
}

// Double: one thread per first-pass line segment when that takes at most 512 threads, and
// the tile and the first pass's output share their buffer, which doubles the rows that
// fit the shared-memory budget (measured at 384x384x256: 0.139 ms against 0.164 ms).
// Float keeps 256 threads and separate buffers (0.083 ms against 0.087 ms aliased).
template <typename T, int N>
static bool ixfft_alias(int rows) {
    return sizeof(T) == 8 && (rows / 2) * FftSplit<N>::N2 <= 512;
}
template <typename T, int N>
static int ixfft_threads(int rows) {
    const int items = (rows / 2) * FftSplit<N>::N2;
    return ixfft_alias<T, N>(rows) ? std::max(256, (items + 31) / 32 * 32) : 256;
}

template <typename T, int N>
static size_t ixfft_reg_smem(int rows) {
    const size_t tile = (size_t)(N / 2 + 1) * ixfft_stride<T>(rows), y = (size_t)(rows / 2) * FftSplit<N>::YL;
    return (ixfft_alias<T, N>(rows) ? std::max(tile, y) : tile + y) * sizeof(cplx<T>);
}

template <typename T, int N>
static void ixfft_reg_launch(const IxFftArgs<T>& a, int rows, cudaStream_t s) {
    const size_t smem = ixfft_reg_smem<T, N>(rows);
    auto k = k_ixfft_reg<T, N>;
    smem_limit(k, smem);
    launch_pdl(a.g.pdl, k, dim3(a.g.NY / rows, a.g.NZ), ixfft_threads<T, N>(rows), smem, s, a, rows, fft_magic(rows / (16 / (int)sizeof(cplx<T>))), ixfft_alias<T, N>(rows) ? 1 : 0);
}

// Rows per CTA of the x-FFT kernels: the largest of 32, 16, 8 (NY = 2 or 4 times a power of
// 3: 36, 18, 12, 6) that divides NY and whose shared memory stays within XFFT_SMEM_PREF (four CTAs per SM: measured faster
// than two), else within 110 KB (two CTAs per SM); 0 if none.
constexpr size_t XFFT_SMEM_PREF = 56 * 1024;
template <typename T, int N>
static int xfft_reg_rows(int NY, bool inverse) {
    for (size_t cap : {XFFT_SMEM_PREF, (size_t)110 * 1024})
        for (int r : {36, 32, 18, 16, 12, 8, 6}) {
            if (NY % r || (NY % 8 == 0) != (r % 8 == 0)) continue;
            const size_t sm = inverse ? ixfft_reg_smem<T, N>(r) : div_xfft_reg_smem<T, N>(r);
            if (sm <= cap) return r;
        }
    return 0;
}


// The transforms of the lengths of one translation unit: 0 / false when the length is not
// among them or no tile of rows fits.
#define TC_FFT_LENGTHS(NAME, SIZES)                                                             \
    template <typename T>                                                                       \
    bool yfft_##NAME(const YFftArgs<T>& a, cudaStream_t s) {                                    \
        switch (a.g.NY) {                                                                       \
            SIZES(TC_YCASE)                                                                     \
            default: return false;                                                              \
        }                                                                                       \
    }                                                                                           \
    template <typename T>                                                                       \
    bool xfft_##NAME(const DivFftArgs<T>& a, const T* src, cudaStream_t s) {                    \
        switch (a.g.NX) {                                                                       \
            SIZES(TC_XCASE)                                                                     \
            default: return false;                                                              \
        }                                                                                       \
    }                                                                                           \
    template <typename T>                                                                       \
    bool ixfft_##NAME(const IxFftArgs<T>& a, cudaStream_t s) {                                  \
        switch (a.g.NX) {                                                                       \
            SIZES(TC_IXCASE)                                                                    \
            default: return false;                                                              \
        }                                                                                       \
    }                                                                                           \
    template bool yfft_##NAME<double>(const YFftArgs<double>&, cudaStream_t);                   \
    template bool yfft_##NAME<float>(const YFftArgs<float>&, cudaStream_t);                     \
    template bool xfft_##NAME<double>(const DivFftArgs<double>&, const double*, cudaStream_t);  \
    template bool xfft_##NAME<float>(const DivFftArgs<float>&, const float*, cudaStream_t);     \
    template bool ixfft_##NAME<double>(const IxFftArgs<double>&, cudaStream_t);                 \
    template bool ixfft_##NAME<float>(const IxFftArgs<float>&, cudaStream_t);
#define TC_YCASE(n)                  \
    case n:                          \
        yfft_reg_launch<T, n>(a, s); \
        return true;
#define TC_XCASE(n)                                          \
    case n: {                                                \
        const int rows = xfft_reg_rows<T, n>(a.g.NY, false); \
        if (rows) xfft_reg_launch<T, n>(a, src, rows, s);    \
        return rows != 0;                                    \
    }
#define TC_IXCASE(n)                                                                          \
    case n: {                                                                                 \
        const int rows = xfft_reg_rows<T, n>(a.g.NY, true);                                   \
        if (rows && !ixfft_pipe_launch<T, n>(a, s)) ixfft_reg_launch<T, n>(a, rows, s);       \
        return rows != 0;                                                                     \
    }

// k_fft.cu: 16 ... 1024 = 2^a, 3 2^a; k_fft_m.cu, k_fft_l.cu: the other even 2^a 3^b
#define TC_FFT_DECL(NAME)                                                             \
    template <typename T> bool yfft_##NAME(const YFftArgs<T>& a, cudaStream_t s);     \
    template <typename T> bool xfft_##NAME(const DivFftArgs<T>& a, const T* src, cudaStream_t s); \
    template <typename T> bool ixfft_##NAME(const IxFftArgs<T>& a, cudaStream_t s);
TC_FFT_DECL(m)
TC_FFT_DECL(l)
#undef TC_FFT_DECL

}  // namespace tc
