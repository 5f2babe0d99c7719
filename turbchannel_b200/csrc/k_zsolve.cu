// k_zsolve.cu -- the step's banded solve along z, one matrix per Fourier mode, from factors
// computed once at solver creation.
//
// The z-matrix of a mode depends on the mesh and the mode only, so k_zfactor eliminates it
// once in double (the matrices of staggered/func_global.h:71-189 and
// collocated_AB3/func_global.h:21-70).  They are symmetric (the upper band of row i is the
// lower band of the rows below it), and they are eliminated from both walls towards the
// middle: rows 0 .. H-1 downwards, rows NZ-1 .. H+nm upwards, then the nm middle rows (3 of
// the 7-diagonal VV4 matrices, 1 of the tridiagonal ones) as a small dense block.  The two
// halves are independent, which halves the serial chain of a column, and by symmetry the
// lower factors are the upper ones of the rows before:
//   7-diagonal, per row {1/d, b1, b2, b3}, b_k its coupling to the k-th row further inwards
//   (t counts rows from the wall):
//     y_t = r_t - b1_{t-1} y_{t-1} - b2_{t-2} y_{t-2} - b3_{t-3} y_{t-3}
//     x_t = y_t / d_t - b1_t x_{t+1} - b2_t x_{t+2} - b3_t x_{t+3}
//   tridiagonal, per row {1/d, b1}: the same without b2, b3.
// Mode (kx, NY - ky) has the matrix of (kx, ky): factors are stored for ky <= NY/2.
//
// A CTA takes KP such pairs of modes, copies their whole columns and factors into shared
// memory (every load of the tile in flight at once), runs both sweeps there, one warp per
// half and one lane per real component of a mode, and writes the columns back from the
// second sweep.  The half next to the far wall is stored mirrored and both are padded to
// whole batches of rows, so that the two warps run the same straight code without
// remainders (a cold instruction cache is a large part of a small grid's time).
// The spectrum crosses DRAM once in each direction and the factors once: per mode and row
// 16 B of data and 8 B (VV4) or 4 B of factors in float.  The form before it kept one
// thread per mode sweeping global memory from one wall to the other: its forward result
// went out to L2/DRAM and came back (16 B more), each sweep read factors of its own (16 B
// or 6 B), and small grids had too few threads to hide the load latency of each row batch.
// before -> now, us (before: the sweep, its double low modes next to it on a side stream):
//   HW2 64x64x64 FP64 17.1 (+ 5.6) -> 5.5      HW2 128x128x128 FP64 34.0 (+ 8.8) -> 11.3
//   coll 256x256x192 FP64 98 (+ 16) -> 61-65   VV4 216x108x95 mixed 17-24 (+ 9) -> 11.6
//   VV4 128x96x256 mixed 43 (+ 19) -> 19       VV4 256x256x256 mixed 75 (+ 23) -> 64
//   VV4 384x384x256 mixed 134 (+ 25) -> 143    VV4 512x512x256 mixed 246 (+ 31) -> 247
// Two tiles of 8 pairs per SM beat three or six of 4 or 2 pairs (384x384x256 HW2 FP64: 219
// against 262 and 343 us), the sweeping lanes being what a small tile leaves idle.
// In the mixed mode the modes with kx < low_modes and min(ky, NY-ky) < low_modes are tiles
// of their own in double (the first blocks of the same launch); the tile of mode (0, 0)
// also applies the pressure normalisation.
#include <algorithm>
#include <type_traits>

#include "kernels.cuh"

namespace tc {

// ---------------------------------------------------------------------------
// tiles
// ---------------------------------------------------------------------------
// Middle rows; rows of the half next to wall 0 (the other half has the remaining ones).
__host__ __device__ constexpr int zs_mid(bool vv) { return vv ? 3 : 1; }
__host__ __device__ constexpr int zs_top(int NZ, bool vv) { return (NZ - zs_mid(vv)) / 2; }
// Rows per register batch, and a half's rows rounded up to whole batches (rows of zeros
// before the wall row): row t of half h is stored at h * zs_half + zs_half - cnt + t, the
// middle rows after both halves.
__host__ __device__ constexpr int zs_batch(bool vv, int eb) { return vv && eb == 8 ? 4 : 8; }
__host__ __device__ constexpr int zs_half(int NZ, bool vv) {
    return (NZ - zs_mid(vv) - zs_top(NZ, vv) + 7) / 8 * 8;
}
__host__ __device__ constexpr int zs_rows(int NZ, bool vv) { return 2 * zs_half(NZ, vv) + zs_mid(vv); }

static bool zs_vv(const Geom& g) { return g.scheme == TC_SCHEME_VV4; }
static int zs_values(const Geom& g) { return zs_vv(g) ? 4 : 2; }
// shared memory of a tile: per row and pair two complex values and the pair's factors
static size_t zs_smem(const Geom& g, int kp, int eb, bool staged = true) {
    return (size_t)zs_rows(g.NZ, zs_vv(g)) * kp * (4 + (staged ? zs_values(g) : 0)) * eb;
}
static int zs_ktiles(const Geom& g, int kp) { return (g.NY / 2 + kp) / kp; }  // tiles of the NY/2+1 pairs of one kx
constexpr size_t ZS_SMEM = 110 * 1024;  // at most, while a tile has two pairs or more: two CTAs per SM
constexpr size_t ZS_SMEM_MAX = SMEM_MOST;  // beyond (NZ of several thousand): factors stay in global memory
constexpr int ZS_CTAS = 148 * 2;

// Pairs per tile: 8 (64-byte rows in float), fewer where the columns are long (shared
// memory) or the grid would leave SMs without a CTA.
static int zs_pairs(const Geom& g, int eb) {
    for (int kp : {8, 4, 2})
        if (zs_smem(g, kp, eb) <= ZS_SMEM && (kp == 2 || zs_ktiles(g, kp) * g.NXH >= ZS_CTAS)) return kp;
    return 1;
}
static int zs_pairs_low(const Geom& g) { return std::max(1, zs_pairs(g, 4) / 2); }  // double tiles of the mixed mode

// Pairs of modes whose columns an SM holds at a time: 1 KB of the system's and the kernel's own
// shared memory next to each tile.
static int zs_resident_pairs(const Geom& g, int eb) {
    const int kp = zs_pairs(g, eb);
    return kp * (int)std::min<size_t>(32, 228 * 1024 / (zs_smem(g, kp, eb) + 2592));
}

// One thread per mode sweeping global memory (k_zsolve_stream) in place of tiles:
// VV4 grids in double with many modes (288x288 and larger), where a tile's columns and factors
// take 64 KB per 4 pairs, half the lanes of each sweeping warp are idle and three tiles fit an SM,
// while the streaming form has enough modes in flight to run at its DRAM traffic: streaming /
// tiles 0.187 / 0.192 ms at 288x288x256 (equal at 96 and 192 planes), 0.211 / 0.244 at
// 324x324x256, 0.264 / 0.335 at 384x384x256, 0.089 / 0.093 at 384x384x96; below, the tiles win
// (192x192x256: 0.088 against 0.120) or are equal (256x256x256).
// And columns so long that an SM holds few pairs, in grids with the modes to fill the chip
// another way (a spectrum beyond the L2, 150 MB): whole solves, streaming / tiles in us, HW2 FP64
// 256x256x1024 (4 pairs per SM) 1300 / 1720, VV4 FP64 256x256x1024 (3) 1520 / 2570, mixed (6)
// 790 / 1090, HW2 mixed 128x128x2800 (3) 780 / 1290; but HW2 FP64 128x128x700 (93 MB) 318 / 273
// (4 rows per batch), and 256x256x384 (12 pairs) 513 / 529.  The mixed form streams from 100 MB on
// where an SM holds 3 pairs or fewer: VV4 128x128x2048 (136 MB) 580 / 1081, HW2 96x96x2800 (104 MB)
// 640 / 771.
constexpr long long ZS_STREAM_MODES = 41000, ZS_STREAM_BYTES = 150000000, ZS_STREAM_BYTES_FEW = 100000000;
constexpr int ZS_STREAM_PAIRS = 8;
static bool zs_stream(const Geom& g, int eb) {
    if (eb == 4 && g.norm_srk != 0) return false;
    const long long modes = (long long)g.NXH * g.NY;
    if (eb == 8 && zs_vv(g) && modes >= ZS_STREAM_MODES) return true;
    const long long bytes = modes * g.NZ * 2 * eb;
    const int pairs = zs_resident_pairs(g, eb);
    return (bytes >= ZS_STREAM_BYTES && pairs <= ZS_STREAM_PAIRS) || (eb == 4 && bytes >= ZS_STREAM_BYTES_FEW && pairs <= 3);
}

// The mixed SRK step keeps the one-sided solve of one thread per mode (k_zsolve_srk): its
// dp/dt is a difference of pressures over tau, which any other rounding of the float solve
// moves by 1e-4 of itself once the start-up transient is over, and large SRK grids are a
// little faster this way (384x384x257: 0.110 against 0.119 ms).
static bool zs_srk(const Geom& g, int eb) { return eb == 4 && g.norm_srk != 0; }

size_t zfactor_bytes(const Geom& g, int eb) {
    if (zs_srk(g, eb)) return (size_t)g.NXH * (g.NY / 2 + 1) * g.NZ * 3 * eb;
    if (zs_stream(g, eb)) return (size_t)g.NXH * (g.NY / 2 + 1) * g.NZ * zs_values(g) * eb;
    const int kp = zs_pairs(g, eb);
    return (size_t)g.NXH * zs_ktiles(g, kp) * kp * zs_rows(g.NZ, zs_vv(g)) * zs_values(g) * eb;
}
size_t zfactor_low_bytes(const Geom& g) {
    if (zs_srk(g, 4)) return (size_t)g.low_modes * g.low_modes * g.NZ * 3 * sizeof(double);
    const int kp = zs_pairs_low(g);
    return (size_t)g.low_modes * ((g.low_modes + kp - 1) / kp) * kp * zs_rows(g.NZ, zs_vv(g)) * zs_values(g) * sizeof(double);
}

// ---------------------------------------------------------------------------
// factors: tile-major [tile][stored row][pair of the tile][value]; rows of padding stay zero
// ---------------------------------------------------------------------------
template <typename T, int SCHEME>
__global__ void __launch_bounds__(128) k_zfactor(ZSolveArgs<T> a, int kp, int kpl, bool stream) {
    // tiles: a.fac and (the mixed mode) a.fac_low; stream: a.fac alone; a.fac null: a.fac_low alone
    constexpr bool VV = SCHEME == TC_SCHEME_VV4;
    constexpr int NV = VV ? 4 : 2;
    const Geom& g = a.g;
    const int NYH1 = g.NY / 2 + 1, NZ = g.NZ;
    const size_t m = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= (size_t)g.NXH * NYH1) return;
    const int kx = (int)(m / NYH1), ky = (int)(m - (size_t)kx * NYH1);
    const bool pin = (kx == 0 && ky == 0);
    const int LM = g.low_modes;
    const bool low = a.fac_low != nullptr && kx < LM && ky < LM;
    if (a.fac == nullptr && !low) return;
    const int nkt = (NYH1 + kp - 1) / kp, nkl = (LM + kpl - 1) / kpl;
    // stream: eliminated from wall 0 to the far wall, [row][pair][value]
    const int top = stream ? NZ : zs_top(NZ, VV), half = zs_half(NZ, VV), rows = zs_rows(NZ, VV);
    T* F = reinterpret_cast<T*>(a.fac) + ((size_t)(kx * (size_t)nkt + ky / kp) * rows * kp + ky % kp) * NV;
    double* FL = low ? reinterpret_cast<double*>(a.fac_low) + ((size_t)(kx * nkl + ky / kpl) * rows * kpl + ky % kpl) * NV
                     : nullptr;
    const double* MA = a.m.dMAT_A;
    const double* DZ = a.m.dDZ;
    const double* DZW = a.m.dDZW;
    auto put = [&](int row, int v, double x) {
        if (stream) {
            reinterpret_cast<T*>(a.fac)[((size_t)row * g.NXH * NYH1 + m) * NV + v] = (T)x;
            return;
        }
        const int i = row < top ? half - top + row
                                : (row < top + zs_mid(VV) ? 2 * half + row - top
                                                         : 2 * half - (NZ - zs_mid(VV) - top) + NZ - 1 - row);
        if (a.fac) F[(size_t)i * kp * NV + v] = (T)x;
        if (low) FL[(size_t)i * kpl * NV + v] = x;
    };
    // the row's diagonal and its coupling to row i + k
    double MM = 0, s3x = 0, s3y = 0, sx = 0, sy = 0;
    if constexpr (SCHEME == TC_SCHEME_HW2) {
        MM = 2 * ((1 - a.tabs.cosx[kx]) * g.inv_hx * g.inv_hx + (1 - a.tabs.cosy[ky]) * g.inv_hy * g.inv_hy);
    } else if constexpr (SCHEME == TC_SCHEME_COLLOC) {
        MM = (1 - a.tabs.cosx[kx]) * g.hy / g.hx + (1 - a.tabs.cosy[ky]) * g.hx / g.hy;
    } else {
        sx = a.tabs.sinx[kx];
        sy = a.tabs.siny[ky];
        s3x = 3 * sx - 4 * sx * sx * sx;
        s3y = 3 * sy - 4 * sy * sy * sy;
    }
    auto diag = [&](int i) -> double {
        double d;
        if constexpr (SCHEME == TC_SCHEME_HW2) {
            d = -DZ[i] * MM - (i > 0 ? MA[i] : 0.0);
            if (i != NZ - 1) d -= MA[i + 1];
        } else if constexpr (SCHEME == TC_SCHEME_COLLOC) {
            if (i == 0) {
                d = -MA[1];
                if (!g.fd_mode) d += DZ[0] * MM;
            } else {
                const double mm = (g.fd_mode && (i == NZ - 1)) ? 0.0 : MM;
                d = 0;
                d -= MA[i] + DZ[i - 1] * mm;
                if (i != NZ - 1) d -= MA[i + 1] + DZ[i] * mm;
            }
        } else {
            const double C27 = 0.03703703703703703703, C9 = 0.11111111111111111111;
            if (i <= 2) d = a.m.MAT_D[i];
            else if (i >= NZ - 3) d = a.m.MAT_D[i - (NZ - 3) + 3];
            else {
                double sum = 0;
                for (int k = 0; k < 3; k++) sum += MA[i * 3 + k];
                for (int k = 1; k <= 3; k++) sum += MA[(i + k) * 3 + 3 - k];
                d = -sum;
            }
            if (pin && i == 0) d *= 2;
            double ci = DZ[i] * sx - C27 * DZW[i] * s3x;
            d -= 4 * g.inv_hx * g.inv_hx * ci * ci / (DZ[i] - C9 * DZW[i]);
            ci = DZ[i] * sy - C27 * DZW[i] * s3y;
            d -= 4 * g.inv_hy * g.inv_hy * ci * ci / (DZ[i] - C9 * DZW[i]);
            return d;
        }
        return pin && i == 0 ? 2 * d : d;
    };
    auto off = [&](int i, int k) -> double {  // 0 beyond the far wall
        if (i + k >= NZ) return 0.0;
        return VV ? MA[(i + k) * 3 + 3 - k] : MA[i + 1];
    };
    constexpr int NB = VV ? 3 : 1, NMID = zs_mid(VV);
    double S[NMID][NMID];  // the middle block, less what both halves eliminate from it
    for (int p = 0; p < NMID && !stream; p++)
        for (int q = p; q < NMID; q++) S[p][q] = p == q ? diag(top + p) : off(top + p, q - p);
    for (int dir = 0; dir < (stream ? 1 : 2); dir++) {
        const int cnt = dir ? NZ - NMID - top : top;
        double b[NB][NB + 1] = {}, D[NB] = {};  // the last NB rows' b_1.. and pivots, newest first
        for (int t = 0; t < cnt; t++) {
            const int i = dir ? NZ - 1 - t : t;
            double d = diag(i), u[NB + 1];
            for (int j = 1; j <= NB; j++) d -= b[j - 1][j] * b[j - 1][j] * D[j - 1];
            if (fabs(d) < 1e-30) {
                if (a.err_flag) atomicExch(a.err_flag, 1);
                return;
            }
            const double inv = 1.0 / d;
            for (int k = 1; k <= NB; k++) {
                u[k] = dir ? (i - k >= 0 ? off(i - k, k) : 0.0) : off(i, k);
                for (int j = 1; j + k <= NB; j++) u[k] -= b[j - 1][j] * b[j - 1][j + k] * D[j - 1];
            }
            for (int j = NB - 1; j > 0; j--) {
                D[j] = D[j - 1];
                for (int k = 1; k <= NB; k++) b[j][k] = b[j - 1][k];
            }
            D[0] = d;
            put(i, 0, inv);
            for (int k = 1; k <= NB; k++) {
                b[0][k] = u[k] * inv;
                put(i, k, b[0][k]);
            }
        }
        if (stream) return;
        for (int p = 0; p < NMID; p++)  // p, q count middle rows from this half
            for (int q = p; q < NMID; q++)
                for (int j = 1; j + q <= NB; j++) {
                    const double c = b[j - 1][j + p] * b[j - 1][j + q] * D[j - 1];
                    if (dir) S[NMID - 1 - q][NMID - 1 - p] -= c;
                    else S[p][q] -= c;
                }
    }
    if constexpr (VV) {  // inverse of the symmetric 3 x 3 block
        const double c00 = S[1][1] * S[2][2] - S[1][2] * S[1][2], c01 = S[0][2] * S[1][2] - S[0][1] * S[2][2],
                     c02 = S[0][1] * S[1][2] - S[0][2] * S[1][1];
        const double det = S[0][0] * c00 + S[0][1] * c01 + S[0][2] * c02;
        if (fabs(det) < 1e-90) {
            if (a.err_flag) atomicExch(a.err_flag, 1);
            return;
        }
        const double v = 1.0 / det, c11 = S[0][0] * S[2][2] - S[0][2] * S[0][2], c12 = S[0][1] * S[0][2] - S[0][0] * S[1][2],
                     c22 = S[0][0] * S[1][1] - S[0][1] * S[0][1];
        put(top, 0, c00 * v); put(top, 1, c01 * v); put(top, 2, c02 * v); put(top, 3, 0.0);
        put(top + 1, 0, c01 * v); put(top + 1, 1, c11 * v); put(top + 1, 2, c12 * v); put(top + 1, 3, 0.0);
        put(top + 2, 0, c02 * v); put(top + 2, 1, c12 * v); put(top + 2, 2, c22 * v); put(top + 2, 3, 0.0);
    } else {
        if (fabs(S[0][0]) < 1e-30) {
            if (a.err_flag) atomicExch(a.err_flag, 1);
            return;
        }
        put(top, 0, 1.0 / S[0][0]);
        put(top, 1, 0.0);
    }
}

// Factors of the mixed SRK step: per mode (kx, ky <= NY/2) F[row][mode] = {1/d, A/d}, then
// B[row][mode] = the elimination's upper entry; the low modes also in double, mode-major.
__global__ void __launch_bounds__(128) k_zfactor_srk(ZSolveArgs<float> a) {
    const Geom& g = a.g;
    const int NYH1 = g.NY / 2 + 1, NZ = g.NZ, LM = g.low_modes;
    const size_t M = (size_t)g.NXH * NYH1, m = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= M) return;
    const int kx = (int)(m / NYH1), ky = (int)(m - (size_t)kx * NYH1);
    const bool low = kx < LM && ky < LM;
    const size_t jl = (size_t)kx * LM + ky;
    const double* MA = a.m.dMAT_A;
    const double* DZ = a.m.dDZ;
    Q2<float>* F = reinterpret_cast<Q2<float>*>(a.fac);
    float* B = reinterpret_cast<float*>(F + (size_t)NZ * M);
    Q2<double>* FL = reinterpret_cast<Q2<double>*>(a.fac_low) + jl * NZ;
    double* BL = reinterpret_cast<double*>(reinterpret_cast<Q2<double>*>(a.fac_low) + (size_t)LM * LM * NZ) + jl * NZ;
    const double MM = (1 - a.tabs.cosx[kx]) * g.hy / g.hx + (1 - a.tabs.cosy[ky]) * g.hx / g.hy;
    double pp = 0;
    for (int i = 0; i < NZ; i++) {
        double d;
        if (i == 0) {
            d = -MA[1];
            if (!g.fd_mode) d += DZ[0] * MM;
            if (kx == 0 && ky == 0) d *= 2;
        } else {
            const double mm = (g.fd_mode && (i == NZ - 1)) ? 0.0 : MM;
            d = 0;
            d -= MA[i] + DZ[i - 1] * mm;
            if (i != NZ - 1) d -= MA[i + 1] + DZ[i] * mm;
            d -= MA[i] * pp;
        }
        d = 1 / d;
        const double f1 = i ? MA[i] * d : 0.0;
        pp = i != NZ - 1 ? MA[i + 1] * d : 0.0;
        F[(size_t)i * M + m] = {(float)d, (float)f1};
        B[(size_t)i * M + m] = (float)pp;
        if (low) {
            FL[i] = {d, f1};
            BL[i] = pp;
        }
    }
}

template <typename T>
void launch_zfactor(const ZSolveArgs<T>& a, cudaStream_t s) {
    const size_t M = (size_t)a.g.NXH * (a.g.NY / 2 + 1);
    const unsigned nb = (unsigned)((M + 127) / 128);
    if constexpr (sizeof(T) == 4) {
        if (zs_srk(a.g, 4)) {
            k_zfactor_srk<<<nb, 128, 0, s>>>(a);
            return;
        }
    }
    const int kp = zs_pairs(a.g, sizeof(T)), kpl = zs_pairs_low(a.g);
    ZSolveArgs<T> b = a;
    if (sizeof(T) == 8) b.fac_low = nullptr;  // FP64: the low modes are modes like any other
    const auto k = a.g.scheme == TC_SCHEME_VV4   ? k_zfactor<T, TC_SCHEME_VV4>
                   : a.g.scheme == TC_SCHEME_HW2 ? k_zfactor<T, TC_SCHEME_HW2>
                                                 : k_zfactor<T, TC_SCHEME_COLLOC>;
    if (zs_stream(a.g, sizeof(T))) {
        b.fac_low = nullptr;
        k<<<nb, 128, 0, s>>>(b, kp, kpl, true);
        if (sizeof(T) == 8) return;
        b.fac_low = a.fac_low;
        b.fac = nullptr;
    }
    k<<<nb, 128, 0, s>>>(b, kp, kpl, false);
}

// ---------------------------------------------------------------------------
// solve
// ---------------------------------------------------------------------------
constexpr int ZS_NT = 64;

// Mean-mode normalisation of a column in shared memory (stride `st` complex values, row i at stored(i)), every
// thread of the CTA taking part: the shift NormalizePressure applies after the inverse FFT
// (staggered/func_global.h:657-675; collocated_AB3/func_global.h:163-170 or, for the SRK
// step, collocated_SRK/func_global.h:130-137), which only touches the mean mode.
template <typename C, typename MD, typename ROW>
__device__ void normalize_mean_column(const Geom& g, const MD& m, cplx<C>* xs, int st, ROW&& stored, double* red) {
    const int NZ = g.NZ;
    double part = 0;
    for (int i = threadIdx.x; i < NZ; i += blockDim.x) {
        double wgt;
        if (g.scheme == TC_SCHEME_VV4) wgt = m.dKERG[i] * m.dDZ[i];
        else if (g.scheme == TC_SCHEME_HW2) wgt = m.dDZ[i];
        else wgt = m.dcellh[i] * g.hx * g.hy;
        part += (double)xs[(size_t)stored(i) * st].x * wgt;
    }
    part = warp_sum(part);
    const int nw = (int)(blockDim.x >> 5);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = part;
    __syncthreads();
    double psum = 0;
    for (int w = 0; w < nw; w++) psum += red[w];
    double c;
    if (g.scheme == TC_SCHEME_VV4) c = psum / m.KERG_norm2;
    else if (g.scheme == TC_SCHEME_HW2) c = psum / (m.dZZ[NZ] - m.dZZ[0]);
    else c = (double)g.NXY * (g.norm_srk ? psum / g.area : psum * g.hx * g.hy / g.area);
    for (int i = threadIdx.x; i < NZ; i += blockDim.x)
        xs[(size_t)stored(i) * st].x = (C)((double)xs[(size_t)stored(i) * st].x - (g.scheme == TC_SCHEME_VV4 ? c * m.dKERG[i] : c));
    __syncthreads();
}

// Barrier of the two halves' warps, which reach it from their own copies of the sweep.
__device__ __forceinline__ void zs_halves_sync() { asm volatile("bar.sync 1, 64;\n" ::: "memory"); }

// One half of a column in shared memory: nb batches of R rows from x towards the middle (x,
// f: this lane's component and its pair's factors of the half's first stored row; xm, fm: of
// the first middle row).  The halves' contributions to the NB middle rows meet in mid.  A
// batch's shared loads are issued before the recurrence of the batch before it.
// store(where, value, row): the solution, from the second sweep; row counts down to 0 at the
// wall (negative: padding), the middle rows (half 0 only) come first as row >= cnt.
template <typename C, int NB, int KP, typename ST>
__device__ __forceinline__ void zs_half_solve(C* x, const C* fv, C* xm, const C* fmv, int nb, int cnt, int half, C* mid,
                                              bool own, ST&& store) {
    using Q = typename std::conditional<NB == 3, Q4<C>, Q2<C>>::type;
    constexpr int R = zs_batch(NB == 3, sizeof(C)), NL = 4 * KP;
    const Q* f = reinterpret_cast<const Q*>(fv);
    const Q* fm = reinterpret_cast<const Q*>(fmv);
    C xa[2][R];
    Q fa[2][R];
    C y1 = 0, y2 = 0, y3 = 0, b1 = 0, b2 = 0, b2p = 0, b3 = 0, b3p = 0, b3q = 0;
    {
        auto load = [&](int b) {
#pragma unroll
            for (int k = 0; k < R; k++) {
                xa[b][k] = x[k * NL];
                fa[b][k] = f[k * KP];
            }
            x += R * NL;
            f += R * KP;
        };
        auto run = [&](int b, C* p) {
#pragma unroll
            for (int k = 0; k < R; k++) {
                C y = xa[b][k];
                const Q q = fa[b][k];
                if constexpr (NB == 3) {
                    y = y - b3q * y3 - b2p * y2;
                    y3 = y2;
                    y2 = y1;
                }
                y -= b1 * y1;
                y1 = y;
                if (own) p[k * NL] = y;
                b1 = q.y;
                if constexpr (NB == 3) {
                    b3q = b3p; b3p = b3; b3 = q.w;
                    b2p = b2; b2 = q.z;
                }
            }
        };
        load(0);
#pragma unroll 1
        for (int b = 0; b < nb; b += 2) {
            if (b + 1 < nb) load(1);
            run(0, b + 1 < nb ? x - 2 * R * NL : x - R * NL);
            if (b + 1 >= nb) break;
            if (b + 2 < nb) load(0);
            run(1, b + 2 < nb ? x - 2 * R * NL : x - R * NL);
        }
    }
    // contributions to the middle rows, nearest first; row q of half 1 is middle row NB-1-q
    const int lane = threadIdx.x & 31;
    {
        C m[NB];
        m[0] = b1 * y1;
        if constexpr (NB == 3) {
            m[0] += b2p * y2 + b3q * y3;
            m[1] = b2 * y1 + b3p * y2;
            m[2] = b3 * y1;
        }
#pragma unroll
        for (int k = 0; k < NB; k++) mid[(half * NB + (half ? NB - 1 - k : k)) * 32 + lane] = m[k];
    }
    zs_halves_sync();
    C v[NB];
    {
        C r[NB];
#pragma unroll
        for (int k = 0; k < NB; k++) r[k] = xm[k * NL] - (mid[k * 32 + lane] + mid[(NB + k) * 32 + lane]);
        if constexpr (NB == 3) {
#pragma unroll
            for (int k = 0; k < 3; k++) {
                const Q q = fm[k * KP];
                v[k] = q.x * r[0] + q.y * r[1] + q.z * r[2];
            }
        } else {
            v[0] = r[0] * fm->x;
        }
    }
    zs_halves_sync();  // both halves have read the middle rows
    if (half == 0) {
#pragma unroll
        for (int k = NB - 1; k >= 0; k--) store(xm + k * NL, v[k], cnt + k);
    }
    C x1 = half ? v[NB - 1] : v[0], x2 = 0, x3 = 0;
    if constexpr (NB == 3) {
        x2 = v[1];
        x3 = half ? v[0] : v[2];
    }
    {
        auto load = [&](int b) {
            x -= R * NL;
            f -= R * KP;
#pragma unroll
            for (int k = 0; k < R; k++) {
                xa[b][k] = x[k * NL];
                fa[b][k] = f[k * KP];
            }
        };
        int row = cnt - 1;
        auto run = [&](int b, C* p) {
#pragma unroll
            for (int k = R - 1; k >= 0; k--) {
                const Q q = fa[b][k];
                C w = xa[b][k] * q.x;
                if constexpr (NB == 3) {
                    w = w - q.w * x3 - q.z * x2;
                    x3 = x2;
                    x2 = x1;
                }
                w -= q.y * x1;
                x1 = w;
                store(p + k * NL, w, row - (R - 1 - k));
            }
            row -= R;
        };
        load(0);
#pragma unroll 1
        for (int b = 0; b < nb; b += 2) {
            if (b + 1 < nb) load(1);
            run(0, b + 1 < nb ? x + R * NL : x);
            if (b + 1 >= nb) break;
            if (b + 2 < nb) load(0);
            run(1, b + 2 < nb ? x + R * NL : x);
        }
    }
}

// One tile: the pairs kh0 .. kh0+KP-1 (below khlim; those with kx, kh < skip left out) of
// kx, in the arithmetic type C.  Shared memory: [stored row][pair][ky = kh, NY - kh]
// complex, then the factors [stored row][pair][NV].  NORM: the tile holds mode (0, 0), whose
// solution goes through shared memory for the normalisation.  FS: factors staged in shared
// memory; false (columns too long for both): read from global memory.
template <typename C, typename T, bool VV, int KP, bool FS, bool NORM>
__device__ __forceinline__ void zsolve_tile(const ZSolveArgs<T>& a, unsigned char* sm, int kx, int kh0, int khlim, int skip,
                                            const C* __restrict__ fac, C* mid) {
    constexpr int NM = 2 * KP, NL = 4 * KP, NB = VV ? 3 : 1, NV = NB + 1, RSTEP = ZS_NT / NM;
    static_assert(ZS_NT % NM == 0 && NL <= 32 && ZS_NT == 64, "one warp per half");
    const Geom& g = a.g;
    const int NY = g.NY, NZ = g.NZ;
    const int top = zs_top(NZ, VV), bot = NZ - NB - top, hr = zs_half(NZ, VV), rows = 2 * hr + NB;
    const size_t M = (size_t)g.NXH * NY;
    cplx<T>* spec = a.spec + (size_t)kx * NY;
    cplx<C>* X = reinterpret_cast<cplx<C>*>(sm);
    C* F = reinterpret_cast<C*>(X + (size_t)rows * NM);
    const int j = threadIdx.x % NM, r0 = threadIdx.x / NM, kh = kh0 + j % KP;
    const bool valid = kh < khlim && !(kx < skip && kh < skip) && (j < KP || (kh != 0 && 2 * kh != NY));
    cplx<T>* col = spec + (j < KP ? kh : NY - kh);  // used where valid only
    cplx<C>* xs = X + 2 * (j % KP) + j / KP;
    auto stored = [&](int i) {  // stored row of row i
        return i < top ? hr - top + i : (i < top + NB ? 2 * hr + i - top : 2 * hr - bot + (NZ - 1 - i));
    };
    if constexpr (FS) {  // factors: one contiguous block, no kernel's output
        constexpr int RB = KP * NV * (int)sizeof(C), W = RB % 16 == 0 ? 16 : 8;
        const unsigned char* src = reinterpret_cast<const unsigned char*>(fac);
        unsigned char* dst = reinterpret_cast<unsigned char*>(F);
        const int n = rows * RB;
#pragma unroll 4
        for (int e = threadIdx.x * W; e < n; e += ZS_NT * W) cp_async<W>(dst + e, src + e);
    }
    for (int i = r0; i < 2 * hr - top - bot; i += RSTEP)  // rows of padding
        xs[(i < hr - top ? i : hr + i - (hr - top)) * NM] = {C(0), C(0)};
    pdl_wait();
    if (valid) {
        const cplx<T>* src = col + (size_t)r0 * M;
#pragma unroll 4
        for (int i = r0; i < NZ; i += RSTEP, src += (size_t)RSTEP * M) {
            if constexpr (sizeof(C) == sizeof(T)) {
                cp_async<sizeof(cplx<T>)>(xs + stored(i) * NM, src);
            } else {
                const cplx<T> v = *src;
                xs[stored(i) * NM] = {(C)v.x, (C)v.y};
            }
        }
    }
    cp_async_commit();
    cp_async_wait<0>();
    __syncthreads();
    {
        // warp h sweeps half h; lanes beyond the tile follow another lane's column without
        // writing, so that whole warps reach the halves' barriers
        const int lane = threadIdx.x & 31, l = lane % NL, p = l >> 2, k = kh0 + p, h = threadIdx.x >> 5;
        const bool own = lane < NL, mirror = (l >> 1) & 1;
        const bool in = own && k < khlim && !(kx < skip && k < skip) && (!mirror || (k != 0 && 2 * k != NY));
        C* x = reinterpret_cast<C*>(X) + l;
        const C* f = (FS ? F : fac) + p * NV;
        const int cnt = h ? bot : top;
        // solution rows leave in the order of the second sweep
        T* d = reinterpret_cast<T*>(spec + (mirror ? NY - k : k) + (size_t)(h ? NZ - bot : top + NB - 1) * M) + (l & 1);
        const long long step = (h ? 2 : -2) * (long long)M;
        zs_half_solve<C, NB, KP>(x + h * hr * NL, f + h * hr * KP * NV, x + 2 * hr * NL, f + 2 * hr * KP * NV,
                                 hr / zs_batch(VV, sizeof(C)), cnt, h, mid, own, [&](C* ps, C v, int row) {
                                     if constexpr (NORM) {
                                         if (own) *ps = v;
                                     } else {
                                         if (in && row >= 0) *d = (T)v;
                                         d += step;
                                     }
                                 });
    }
    if constexpr (NORM) {
        __shared__ double red[ZS_NT / 32];
        __syncthreads();
        normalize_mean_column(g, a.m, X, NM, stored, red);
        if (valid)
            for (int i = r0; i < NZ; i += RSTEP) {
                const cplx<C> v = xs[stored(i) * NM];
                col[(size_t)i * M] = {(T)v.x, (T)v.y};
            }
    }
}

// Blocks 0 .. nlow-1: the low modes' double tiles (KPL pairs; mixed mode only); then the
// NXH x nkt tiles of KP pairs.
template <typename T, bool VV, int KP, bool FS>
__global__ void __launch_bounds__(ZS_NT) k_zsolve_col(ZSolveArgs<T> a, int nlow, int nkl, int nkt) {
    constexpr int KPL = KP > 1 ? KP / 2 : 1, NV = VV ? 4 : 2;
    extern __shared__ __align__(32) unsigned char smz[];
    __shared__ __align__(16) double mid[2 * 3 * 32];
    const Geom& g = a.g;
    pdl_launch();
    const int LM = g.low_modes, NZ = g.NZ, NYH1 = g.NY / 2 + 1;
    if constexpr (sizeof(T) == 4) {
        if ((int)blockIdx.x < nlow) {
            const int t = blockIdx.x, kx = t / nkl, k0 = (t - kx * nkl) * KPL;
            const double* fac = reinterpret_cast<const double*>(a.fac_low) + (size_t)t * zs_rows(NZ, VV) * KPL * NV;
            if (t == 0) zsolve_tile<double, T, VV, KPL, FS, true>(a, smz, 0, 0, LM, 0, fac, mid);
            else zsolve_tile<double, T, VV, KPL, FS, false>(a, smz, kx, k0, LM, 0, fac, mid);
            return;
        }
    }
    const int t = (int)blockIdx.x - nlow, kx = t / nkt, k0 = (t - kx * nkt) * KP;
    const T* fac = reinterpret_cast<const T*>(a.fac) + (size_t)t * zs_rows(NZ, VV) * KP * NV;
    if constexpr (sizeof(T) == 8) {
        if (t == 0) {
            zsolve_tile<T, T, VV, KP, FS, true>(a, smz, 0, 0, NYH1, 0, fac, reinterpret_cast<T*>(mid));
            return;
        }
    }
    zsolve_tile<T, T, VV, KP, FS, false>(a, smz, kx, k0, NYH1, sizeof(T) == 4 ? LM : 0, fac, reinterpret_cast<T*>(mid));
}

// low_only: the low modes' tiles of a mixed solve whose other modes stream
template <typename T, bool VV, int KP, bool FS = true>
static void zsolve_kp(const ZSolveArgs<T>& a, cudaStream_t s, bool low_only) {
    constexpr int KPL = KP > 1 ? KP / 2 : 1;
    const Geom& g = a.g;
    const int nkt = zs_ktiles(g, KP);
    const int nkl = (g.low_modes + KPL - 1) / KPL, nlow = sizeof(T) == 4 ? g.low_modes * nkl : 0;
    size_t smem = low_only ? 0 : zs_smem(g, KP, sizeof(T), FS);
    if (nlow) smem = std::max(smem, zs_smem(g, KPL, 8, FS));
    if constexpr (KP == 1 && FS) {
        if (smem > ZS_SMEM_MAX) return zsolve_kp<T, VV, 1, false>(a, s, low_only);
    }
    auto k = k_zsolve_col<T, VV, KP, FS>;
    smem_limit(k, smem, FS ? SMEM_MOST : SMEM_MOST + 2048);
    const size_t n = low_only ? 0 : (size_t)g.NXH * nkt;
    launch_pdl(a.g.pdl && !low_only, k, (unsigned)(nlow + n), ZS_NT, smem, s, a, nlow, nkl, nkt);
}

// ---------------------------------------------------------------------------
// one thread per mode (zs_stream)
// ---------------------------------------------------------------------------
// Adjacent lanes take the modes (kx, kh), (kx, NY-kh), which share their factors.  Rows are
// moved R at a time through two register batches, the next batch's loads in flight.  FP64 VV4:
// R = 2 keeps 5 CTAs of 128 threads per SM, so that the ~74 k modes of a 384 x 384 plane run in
// one wave (384x384x256: 4 rows 0.318 ms, 3 rows 0.296, 2 rows 0.27-0.29).  The others wait for
// memory with few modes: whole solves in us, VV4 mixed 128x128x2800 1055 with 4 rows, 975 with 6,
// 791 with 8; HW2 mixed 853 with 6, 781 with 8, 870 with 12; HW2 FP64 256x256x1024 1355 with 4,
// 1297 with 6, 1291 with 8, and 288x288x700 1263, 1252, 1348.
template <typename T, bool VV>
__global__ void __launch_bounds__(128) k_zsolve_stream(ZSolveArgs<T> a) {
    constexpr int R = sizeof(T) == 8 ? (VV ? 2 : 6) : 8;
    using C = cplx<T>;
    using Q = typename std::conditional<VV, Q4<T>, Q2<T>>::type;
    const Geom& g = a.g;
    pdl_launch();
    pdl_wait();
    const int NY = g.NY, NYH1 = NY / 2 + 1, NZ = g.NZ;
    const size_t M = (size_t)g.NXH * NY, MH = (size_t)g.NXH * NYH1;
    const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const size_t mh = t >> 1;
    const int kx = (int)(mh / NYH1), kh = (int)(mh - (size_t)kx * NYH1);
    bool act = mh < MH && !((t & 1) && (kh == 0 || 2 * kh == NY));  // odd lanes: no partner mode
    if (sizeof(T) == 4 && kx < g.low_modes && kh < g.low_modes) act = false;
    if (!act && (sizeof(T) == 4 || blockIdx.x != 0)) return;
    const Q* F = reinterpret_cast<const Q*>(a.fac) + mh;
    C* x = a.spec + (size_t)kx * NY + ((t & 1) ? NY - kh : kh);
    C ra[R], rb[R];
    Q fa[R], fb[R];
    if (act) {
        C y1 = {0, 0}, y2 = {0, 0}, y3 = {0, 0};
        T b1 = 0, b2 = 0, b2p = 0, b3 = 0, b3p = 0, b3q = 0;
        auto load = [&](int i0, C(&r)[R], Q(&f)[R]) {
#pragma unroll
            for (int k = 0; k < R; k++)
                if (i0 + k < NZ) {
                    r[k] = x[(size_t)(i0 + k) * M];
                    f[k] = F[(size_t)(i0 + k) * MH];
                }
        };
        auto run = [&](int i0, const C(&r)[R], const Q(&f)[R]) {
#pragma unroll
            for (int k = 0; k < R; k++) {
                if (i0 + k >= NZ) break;
                C y = r[k];
                if constexpr (VV) {
                    y.x = y.x - b3q * y3.x - b2p * y2.x;
                    y.y = y.y - b3q * y3.y - b2p * y2.y;
                    y3 = y2; y2 = y1;
                }
                y.x -= b1 * y1.x;
                y.y -= b1 * y1.y;
                x[(size_t)(i0 + k) * M] = y;
                y1 = y;
                if constexpr (VV) {
                    b3q = b3p; b3p = b3; b3 = f[k].w;
                    b2p = b2; b2 = f[k].z;
                }
                b1 = f[k].y;
            }
        };
        load(0, ra, fa);
        for (int i0 = 0; i0 < NZ; i0 += 2 * R) {
            load(i0 + R, rb, fb);
            run(i0, ra, fa);
            load(i0 + 2 * R, ra, fa);
            run(i0 + R, rb, fb);
        }
    }
    if (act) {
        C x1 = {0, 0}, x2 = {0, 0}, x3 = {0, 0};
        auto load = [&](int i0, C(&r)[R], Q(&f)[R]) {
#pragma unroll
            for (int k = 0; k < R; k++)
                if (i0 - k >= 0) {
                    r[k] = x[(size_t)(i0 - k) * M];
                    f[k] = F[(size_t)(i0 - k) * MH];
                }
        };
        auto run = [&](int i0, const C(&r)[R], const Q(&f)[R]) {
#pragma unroll
            for (int k = 0; k < R; k++) {
                if (i0 - k < 0) break;
                C v;
                v.x = r[k].x * f[k].x;
                v.y = r[k].y * f[k].x;
                if constexpr (VV) {
                    v.x = v.x - f[k].w * x3.x - f[k].z * x2.x;
                    v.y = v.y - f[k].w * x3.y - f[k].z * x2.y;
                    x3 = x2; x2 = x1;
                }
                v.x -= f[k].y * x1.x;
                v.y -= f[k].y * x1.y;
                x[(size_t)(i0 - k) * M] = v;
                x1 = v;
            }
        };
        load(NZ - 1, ra, fa);
        for (int i0 = NZ - 1; i0 >= 0; i0 -= 2 * R) {
            load(i0 - R, rb, fb);
            run(i0, ra, fa);
            load(i0 - 2 * R, ra, fa);
            run(i0 - R, rb, fb);
        }
    }
    if (sizeof(T) == 8 && blockIdx.x == 0) {  // mode (0, 0) is thread 0's
        __shared__ double red[4];
        __syncthreads();
        auto row = [&](int i) { return (size_t)i * M; };
        normalize_mean_column(g, a.m, a.spec, 1, row, red);
    }
}

// ---------------------------------------------------------------------------
// tridiagonal solve of the mixed SRK step (zs_srk)
// ---------------------------------------------------------------------------
// One thread per mode outside the low set, adjacent lanes taking the modes (kx, kh),
// (kx, NY-kh) that share their factors; rows are moved R at a time through two register
// batches, the loads of batch b+1 issued before batch b is consumed (6 rows: 4 CTAs of 128
// threads per SM, one wave of the modes of a 384 x 384 plane).
__global__ void __launch_bounds__(128) k_zsolve_srk(ZSolveArgs<float> a) {
    constexpr int R = 6;
    using C = cplx<float>;
    const Geom& g = a.g;
    const int NY = g.NY, NYH1 = NY / 2 + 1, NZ = g.NZ, LM = g.low_modes;
    const size_t M = (size_t)g.NXH * NY, MH = (size_t)g.NXH * NYH1;
    const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const size_t mh = t >> 1;
    if (mh >= MH) return;
    const int kx = (int)(mh / NYH1), kh = (int)(mh - (size_t)kx * NYH1);
    if ((t & 1) && (kh == 0 || 2 * kh == NY)) return;  // no partner mode
    if (kx < LM && kh < LM) return;
    const Q2<float>* F = reinterpret_cast<const Q2<float>*>(a.fac) + mh;
    const float* B = reinterpret_cast<const float*>(reinterpret_cast<const Q2<float>*>(a.fac) + (size_t)NZ * MH) + mh;
    C* x = a.spec + (size_t)kx * NY + ((t & 1) ? NY - kh : kh);
    {
        C z1 = {0, 0};
        C ra[R], rb[R];
        Q2<float> fa[R], fb[R];
        auto load = [&](int i0, C(&r)[R], Q2<float>(&f)[R]) {
#pragma unroll
            for (int k = 0; k < R; k++)
                if (i0 + k < NZ) {
                    r[k] = x[(size_t)(i0 + k) * M];
                    f[k] = F[(size_t)(i0 + k) * MH];
                }
        };
        auto run = [&](int i0, const C(&r)[R], const Q2<float>(&f)[R]) {
#pragma unroll
            for (int k = 0; k < R; k++) {
                if (i0 + k >= NZ) break;
                C z;
                z.x = r[k].x * f[k].x;
                z.y = r[k].y * f[k].x;
                z.x -= f[k].y * z1.x;
                z.y -= f[k].y * z1.y;
                x[(size_t)(i0 + k) * M] = z;
                z1 = z;
            }
        };
        load(0, ra, fa);
        for (int i0 = 0; i0 < NZ; i0 += 2 * R) {
            load(i0 + R, rb, fb);
            run(i0, ra, fa);
            load(i0 + 2 * R, ra, fa);
            run(i0 + R, rb, fb);
        }
    }
    {
        C x1 = {0, 0};
        C za[R], zb[R];
        float ba[R], bb[R];
        auto load = [&](int i0, C(&zz)[R], float(&bq)[R]) {
#pragma unroll
            for (int k = 0; k < R; k++)
                if (i0 - k >= 0) {
                    zz[k] = x[(size_t)(i0 - k) * M];
                    bq[k] = B[(size_t)(i0 - k) * MH];
                }
        };
        auto run = [&](int i0, const C(&zz)[R], const float(&bq)[R]) {
#pragma unroll
            for (int k = 0; k < R; k++) {
                if (i0 - k < 0) break;
                C v;
                v.x = zz[k].x - bq[k] * x1.x;
                v.y = zz[k].y - bq[k] * x1.y;
                x[(size_t)(i0 - k) * M] = v;
                x1 = v;
            }
        };
        load(NZ - 1, za, ba);
        for (int i0 = NZ - 1; i0 >= 0; i0 -= 2 * R) {
            load(i0 - R, zb, bb);
            run(i0, za, ba);
            load(i0 - 2 * R, za, ba);
            run(i0 - R, zb, bb);
        }
    }
}

// Its low modes in double: one CTA per mode, the column and its factors staged in shared
// memory, one thread running the two sweeps 8 rows at a time; mode (0,0) also normalised.
__global__ void __launch_bounds__(128) k_zsolve_srk_low(ZSolveArgs<float> a) {
    constexpr int LOWB = 8;
    using C = cplx<double>;
    extern __shared__ __align__(32) unsigned char smraw[];
    __shared__ double red[4];
    const Geom& g = a.g;
    const int LM = g.low_modes, nky = 2 * LM - 1;
    const int idx = blockIdx.x;
    const int kx = idx / nky, j = idx - kx * nky;
    const int ky = j < LM ? j : g.NY - (j - LM + 1);
    if (kx >= g.NXH || ky < 0 || ky >= g.NY) return;
    const int kh = j < LM ? j : j - LM + 1;  // min(ky, NY - ky)
    const int NZ = g.NZ;
    const size_t M = (size_t)g.NXH * g.NY, m = (size_t)kx * g.NY + ky, jl = (size_t)kx * LM + kh;
    Q2<double>* sF = reinterpret_cast<Q2<double>*>(smraw);
    double* sB = reinterpret_cast<double*>(sF + NZ);
    const size_t xo = ((size_t)NZ * 24 + 31) & ~(size_t)31;
    C* xs = reinterpret_cast<C*>(smraw + xo);
    const Q2<double>* F = reinterpret_cast<const Q2<double>*>(a.fac_low) + jl * NZ;
    const double* B =
        reinterpret_cast<const double*>(reinterpret_cast<const Q2<double>*>(a.fac_low) + (size_t)LM * LM * NZ) + jl * NZ;
    for (int i = threadIdx.x; i < NZ; i += blockDim.x) {
        const cplx<float> v = a.spec[(size_t)i * M + m];
        xs[i] = {(double)v.x, (double)v.y};
        sF[i] = F[i];
        sB[i] = B[i];
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        C z1 = {0, 0};
        for (int i0 = 0; i0 < NZ; i0 += LOWB) {
            Q2<double> f[LOWB];
            C r[LOWB];
#pragma unroll
            for (int k = 0; k < LOWB; k++)
                if (i0 + k < NZ) {
                    f[k] = sF[i0 + k];
                    r[k] = xs[i0 + k];
                }
#pragma unroll
            for (int k = 0; k < LOWB; k++) {
                if (i0 + k >= NZ) break;
                C z;
                z.x = r[k].x * f[k].x;
                z.y = r[k].y * f[k].x;
                z.x -= f[k].y * z1.x;
                z.y -= f[k].y * z1.y;
                xs[i0 + k] = z;
                z1 = z;
            }
        }
        C x1 = {0, 0};
        for (int i0 = NZ - 1; i0 >= 0; i0 -= LOWB) {
            double bq[LOWB];
            C zz[LOWB];
#pragma unroll
            for (int k = 0; k < LOWB; k++)
                if (i0 - k >= 0) {
                    bq[k] = sB[i0 - k];
                    zz[k] = xs[i0 - k];
                }
#pragma unroll
            for (int k = 0; k < LOWB; k++) {
                if (i0 - k < 0) break;
                C v;
                v.x = zz[k].x - bq[k] * x1.x;
                v.y = zz[k].y - bq[k] * x1.y;
                xs[i0 - k] = v;
                x1 = v;
            }
        }
    }
    __syncthreads();
    if (m == 0) {
        auto row = [](int i) { return i; };
        normalize_mean_column(g, a.m, xs, 1, row, red);
    }
    for (int i = threadIdx.x; i < NZ; i += blockDim.x) {
        const C v = xs[i];
        a.spec[(size_t)i * M + m] = {(float)v.x, (float)v.y};
    }
}

static void zsolve_srk(const ZSolveArgs<float>& a, cudaStream_t s, cudaStream_t side, cudaEvent_t fork, cudaEvent_t join) {
    // the two sets of modes are disjoint: the low modes on a side stream
    cudaEventRecord(fork, s);
    cudaStreamWaitEvent(side, fork, 0);
    const size_t smem = (((size_t)a.g.NZ * 24 + 31) & ~(size_t)31) + (size_t)a.g.NZ * sizeof(cplx<double>);
    smem_limit(k_zsolve_srk_low, smem);
    k_zsolve_srk_low<<<a.g.low_modes * (2 * a.g.low_modes - 1), 128, smem, side>>>(a);
    cudaEventRecord(join, side);
    const size_t MH = (size_t)a.g.NXH * (a.g.NY / 2 + 1);
    k_zsolve_srk<<<(unsigned)((2 * MH + 127) / 128), 128, 0, s>>>(a);
    cudaStreamWaitEvent(s, join, 0);
}

template <typename T, bool VV>
static void zsolve_tiles(const ZSolveArgs<T>& a, cudaStream_t s, bool low_only) {
    switch (zs_pairs(a.g, sizeof(T))) {
        case 8: zsolve_kp<T, VV, 8>(a, s, low_only); break;
        case 4: zsolve_kp<T, VV, 4>(a, s, low_only); break;
        case 2: zsolve_kp<T, VV, 2>(a, s, low_only); break;
        default: zsolve_kp<T, VV, 1>(a, s, low_only); break;
    }
}

// returns launches
template <typename T, bool VV>
static int zsolve_vv(const ZSolveArgs<T>& a, cudaStream_t s, cudaStream_t side, cudaEvent_t fork, cudaEvent_t join) {
    if (!zs_stream(a.g, sizeof(T))) {
        zsolve_tiles<T, VV>(a, s, false);
        return 1;
    }
    const size_t n = (size_t)2 * a.g.NXH * (a.g.NY / 2 + 1);
    if (sizeof(T) == 8) {
        launch_pdl(a.g.pdl, k_zsolve_stream<T, VV>, (unsigned)((n + 127) / 128), 128, 0, s, a);
        return 1;
    }
    // the two sets of modes are disjoint: the low modes' tiles on the side stream
    cudaEventRecord(fork, s);
    cudaStreamWaitEvent(side, fork, 0);
    zsolve_tiles<T, VV>(a, side, true);
    cudaEventRecord(join, side);
    launch_pdl(false, k_zsolve_stream<T, VV>, (unsigned)((n + 127) / 128), 128, 0, s, a);
    cudaStreamWaitEvent(s, join, 0);
    return 2;
}

template <typename T>
int launch_zsolve_fac(const ZSolveArgs<T>& a, cudaStream_t s, cudaStream_t side, cudaEvent_t fork, cudaEvent_t join) {
    if constexpr (sizeof(T) == 4) {
        if (zs_srk(a.g, 4)) {
            zsolve_srk(a, s, side, fork, join);
            return 2;
        }
    }
    return a.g.scheme == TC_SCHEME_VV4 ? zsolve_vv<T, true>(a, s, side, fork, join) : zsolve_vv<T, false>(a, s, side, fork, join);
}

template int launch_zsolve_fac<double>(const ZSolveArgs<double>&, cudaStream_t, cudaStream_t, cudaEvent_t, cudaEvent_t);
template int launch_zsolve_fac<float>(const ZSolveArgs<float>&, cudaStream_t, cudaStream_t, cudaEvent_t, cudaEvent_t);
template void launch_zfactor<double>(const ZSolveArgs<double>&, cudaStream_t);
template void launch_zfactor<float>(const ZSolveArgs<float>&, cudaStream_t);

}  // namespace tc
