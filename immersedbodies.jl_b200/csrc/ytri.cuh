// ytri.cuh -- the y direction of the DST-diagonalised solves, solved directly.
//
// After the X pass every column kx of the field is an independent system in y:
// with t = 2 - 2 cos(pi kx / nx) and T = tridiag(-1, 2, -1) (rows 1..M-1,
// M = ny, zero beyond both ends)
//   Laplacian inverse           (T + t) x = b
//   implicit diffusion          (1 + c (T + t)) x = b,  i.e. (T + t + 1/c) x = b / c
// which is what a DST along y, the multiplier and a second DST along y compute.
// With r + 1/r = 2 + t, r < 1, the solution is a sum of two first-order
// recurrences and two homogeneous terms:
//   P_j = b_j + r P_(j-1),  Q_j = b_j + r Q_(j+1),
//   x_j = r / (1 - r^2) (P_j + Q_j - b_j) - A r^j - B r^(M-j),
// A and B from x_0 = x_M = 0; the homogeneous terms enter as starting values of
// the recurrences (P_0, Q_M).
//
// A block owns W columns, 64 threads each; a thread holds MR consecutive rows
// of one column in registers.  Local recurrences give each chunk's total, one
// warp per column and direction scans the 64 totals with shuffles, and the
// recurrences run again from the scanned starts.  The field is read once and
// written once (in place if wanted), about 14 FP64 operations a row, two
// barriers: the two transforms it replaces are 60 operations a row each through
// seven shared-memory round trips.  Measured, back to back in a graph: one
// 1024^2 FP64 field 6.5 us with the correction of the low modes described below, 5.2
// without (20.6 as transforms; 2.6 TB/s read and written with it), five
// in one launch 20.3 us (78), one 512^2 field 4.7 us.  Bound by latency for one
// field (load, scan, store in one wave), by memory for many.  1 - r is kept to full relative accuracy
// (r as a two-part sum), so small t loses nothing.
//
// The reference's eigenvalues -2 ((cx + cy) - 2) carry the rounding of the
// cosines, up to 2.4e-12 of the smallest one at 1024 x 1024.  So that results
// keep that spectrum, the columns kx <= 16 add the difference of the two
// inverses in the modes ky <= 16 (beyond, it is below 3e-14); the modes'
// coefficients come from each chunk's zeroth and first moments, exact enough
// for a correction of that size.  Fields of at most 32 rows take the modes'
// exact sum for those columns instead (the homogeneous terms cancel badly when
// nx >> ny).
#pragma once
#include "common.cuh"

namespace ibpm {

// 1/d: the hardware reciprocal approximation refined by two Newton-Raphson
// steps (e = 1 - d y, y += y e); within an ulp or two of the correctly rounded
// quotient, for the positive, normal d of the spectral multipliers.
__device__ __forceinline__ double recip(double d) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
    double e = fma(-d, y, 1.0);
    y = fma(y, e, y);
    e = fma(-d, y, 1.0);
    return fma(y, e, y);
}

// Spectral multipliers scale / Lambda (src/fluid.jl:117-134)
enum { MULT_LAPINV = 0, MULT_AEXPL = 1, MULT_AIMPL = 2 };
struct Mult {
    int mode;
    const double *cx;   // cos(pi i / nx), i = 0..nx
    const double *cy;   // cos(pi j / ny), j = 0..ny
    double scale;       // 1 / (4 nx ny)
    double c;           // dt / (2 Re hc^2) of the level; the reference's (lam dt) / (2 Re hc^2)
                        // becomes lam c (within one rounding)
    __device__ __forceinline__ double operator()(int i, int j) const {
        const double lam = -2 * ((cx[i] + cy[j]) - 2);
        if (mode == MULT_LAPINV) return scale * recip(lam);
        if (mode == MULT_AEXPL) return scale * (1 - lam * c);  // scale / (1 / (1 - lam c))
        return scale * recip(1 + lam * c);
    }
};

constexpr int kYChunks = 64;   // threads (chunks of rows) per column
constexpr int kYMaxW = 8;      // columns per block, at most
constexpr int kYModes = 16;    // modes of the spectrum correction in each direction
constexpr int kYFull = 32;     // rows up to which the corrected columns take the full mode sum
constexpr int kYDiff = kYModes * kYFull + 8;  // doubles of one correction table (the last: in use or not)

// One column's constants, written once per (size, coefficient) by ycols_kernel:
// computed in the solve, their exponentials and square root were two thirds of
// its instructions (1405 a warp at 16 rows a thread).
struct __align__(16) YCol {
    double rh, rl;  // r = rh + rl
    double R;       // r^MR
    double kap;     // r / (1 - r^2), and the scales of the X passes and of c
    double eM;      // r^M
    double det;     // 1 / (1 - r^2M)
    double ek;      // r^k, k = rows up to M in the chunk that holds row M
    double ek1;     // r^(k - 1)
    double sx;      // 2 sin(pi kx / nx): what a unit source on the first column adds
    double pad;
};
// Boundary values from the coarser level (RingOut in kernels.cuh): batch b at
// lines + b stride
struct YRing {
    const double *lines = nullptr;
    long long stride = 0;
    int nx = 0, ny = 0;
};
// The y solve of one launch: batch b takes cols + b cstride and diff + b dstride.
struct YSolve {
    const YCol *cols;
    const double *diff;   // [kYModes][kYFull]: what mode (kx, ky) adds
    const double2 *phase; // [kYChunks + 1][kYFull]: sin and cos of pi ky j / M at the chunk's centre row j,
                          // then at j = 4 MR
    long long cstride, dstride;
};

// In place; leading dimension ld, batch stride bs.  blockDim.x = 64 << wshift,
// 64 MR >= M.
// RING: the field's sources on its outer rows and columns are added to b.
template <int MR, bool RING>
__global__ void __launch_bounds__(kYChunks *kYMaxW)
    ytri_kernel(double *f, long long bs, int ld, int ncols, int M, int wshift, YSolve ys, YRing yr) {
    overlap_begin();
    constexpr int kPad = kYMaxW * (kYChunks + 2);
    // chunk totals, then starts of P and Q; r^(row) of the homogeneous terms.  Row
    // stride 64 + 16 / W: the threads' stores and the scan's 16-byte loads are free
    // of bank conflicts
    __shared__ __align__(16) double sP[kPad], sQ[kPad], sA[kPad], sB[kPad];
    __shared__ double sPM[kYMaxW], sQ1[kYMaxW];
    __shared__ double2 mom[kYMaxW * kYChunks];
    __shared__ double modes[kYMaxW][kYFull];
    const int W = 1 << wshift, tid = threadIdx.x, S = kYChunks + (16 >> wshift);
    const int w = tid & (W - 1), p = tid >> wshift;
    const int c0 = blockIdx.x << wshift, col = c0 + w;  // 0-based column: kx = col + 1
    const int b = blockIdx.y, n = M - 1, j0 = p * MR;   // rows j0+1 .. j0+MR
    const bool valid = col < ncols;
    double *src = f + b * bs + col + (long long)ld * j0;
    double v[MR];
#pragma unroll
    for (int k = 0; k < MR; ++k) v[k] = valid && j0 + k < n ? src[ld * k] : 0.0;
    const YCol *cols = ys.cols + b * ys.cstride;
    const double2 rr = *reinterpret_cast<const double2 *>(&cols[valid ? col : 0].rh);
    const double rh = rr.x, rl = rr.y;
    // every constant is fetched with the rows, so that no later phase waits for one
    const int lane = tid & 31, cw = tid >> 6;  // the column this warp scans
    const YCol &yc = cols[min(c0 + cw, ncols - 1)];
    const double R = yc.R, ekx = (tid & 32) ? yc.ek1 : yc.ek;
    const double2 ce = *reinterpret_cast<const double2 *>(&cols[valid ? col : 0].eM);
    const double kap = cols[valid ? col : 0].kap;
    const bool full = n <= kYFull;
    const int nmode = full ? n : min(kYModes, n);
    double2 ph_p = make_double2(0.0, 0.0), ph_t = ph_p, ph_r = ph_p;
    const bool correct = c0 < kYModes && __ldg(ys.diff + b * ys.dstride + kYDiff - 1) != 0.0;
    if (correct) {
        const int ky = min(tid >> (2 + wshift), kYFull - 1);
        ph_p = __ldg(&ys.phase[p * kYFull]);
        ph_t = __ldg(&ys.phase[(tid & 3) * kYFull + ky]);
        ph_r = __ldg(&ys.phase[kYChunks * kYFull + ky]);
    }
    if constexpr (RING) {
        // the coarse columns' values, interpolated to this chunk's rows: the odd rows
        // are means of two; the last column's sign alternates with kx
        const double *hat = yr.lines + b * yr.stride;
        const double *cl = hat + 2 * yr.nx + M / 4 - 1, *cr = cl + yr.ny;
        const double sx = cols[valid ? col : 0].sx, sg = (col & 1) ? -sx : sx;
        if constexpr (MR % 2 == 0) {
            double q[MR / 2 + 1];
#pragma unroll
            for (int m = 0; m <= MR / 2; ++m) {
                const int at = j0 / 2 + m;
                q[m] = at <= M / 2 ? fma(sx, cl[at], sg * cr[at]) : 0.0;
            }
#pragma unroll
            for (int k = 0; k < MR; ++k)
                if (j0 + k < n) v[k] += (k & 1) ? q[(k + 1) / 2] : 0.5 * (q[k / 2] + q[k / 2 + 1]);
        } else {
#pragma unroll
            for (int k = 0; k < MR; ++k) {
                const int j = j0 + k + 1;
                if (j > n) continue;
                const double hi = fma(sx, cl[(j + 1) / 2], sg * cr[(j + 1) / 2]);
                v[k] += (j & 1) ? 0.5 * (hi + fma(sx, cl[j / 2], sg * cr[j / 2])) : hi;
            }
        }
        if (valid) {
            if (p == 0) v[0] += hat[col];
#pragma unroll
            for (int k = 0; k < MR; ++k)
                if (j0 + k == n - 1) v[k] += hat[yr.nx + col];
        }
    }

    // local recurrences; the owner of row M stops there
    double lp = 0.0, lq = 0.0;
#pragma unroll
    for (int k = 0; k < MR; ++k) {
        if (j0 + k < M) lp = fma(rh, lp, fma(rl, lp, v[k]));
        lq = fma(rh, lq, fma(rl, lq, v[MR - 1 - k]));
    }
    sP[w * S + p] = lp;
    sQ[w * S + p] = lq;
    constexpr int KC = (MR - 1) / 2;  // the chunk's centre row is j0 + 1 + KC
    if (correct) {
        double m0 = 0.0, m1 = 0.0;
#pragma unroll
        for (int k = 0; k < MR; ++k) {
            m0 += v[k];
            m1 = fma((double)(k - KC), v[k], m1);
        }
        mom[p * W + w] = make_double2(m0, m1);
    }
    __syncthreads();

    // one warp per column and direction scans the chunk totals (two a lane) and
    // forms the powers of r the homogeneous terms start with
    {
        const int pown = (M - 1) / MR;  // holds row M
        if (tid & 32) {
            double2 *slot = reinterpret_cast<double2 *>(sQ + cw * S) + lane;
            const double2 a = *slot;
            const int e1 = pown - 2 - 2 * lane;  // chunks between chunk 2 lane + 1 and the last one below row M
            double acc = fma(R, a.y, a.x), f = R, g = ekx;
            if (e1 > 0 && (e1 & 1)) g *= f;
            f *= f;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const double u = __shfl_down_sync(0xffffffffu, acc, o);
                if (lane + o < 32) acc = fma(f, u, acc);
                if (e1 > 0 && (e1 & (2 * o))) g *= f;
                f *= f;
            }
            double e = __shfl_down_sync(0xffffffffu, acc, 1);
            if (lane == 31) e = 0.0;
            *slot = make_double2(fma(R, e, a.y), e);
            // chunk 2 lane: one chunk more; the chunk below row M's starts from row M - 1's own power
            const double b1 = e1 >= 0 ? g : 1.0;
            const double b0 = e1 >= 0 ? g * R : e1 == -1 ? ekx : 1.0;
            reinterpret_cast<double2 *>(sB + cw * S)[lane] = make_double2(b0, b1);
            if (lane == 0) sQ1[cw] = acc;
        } else {
            double2 *slot = reinterpret_cast<double2 *>(sP + cw * S) + lane;
            const double2 a = *slot;
            double acc = fma(R, a.x, a.y), f = R * R, g = 1.0;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const double u = __shfl_up_sync(0xffffffffu, acc, o);
                if (lane >= o) acc = fma(f, u, acc);
                if (lane & o) g *= f;
                f *= f;
            }
            double e = __shfl_up_sync(0xffffffffu, acc, 1);
            if (lane == 0) e = 0.0;
            const double e1 = fma(R, e, a.x);
            *slot = make_double2(e, e1);
            reinterpret_cast<double2 *>(sA + cw * S)[lane] = make_double2(g, g * R);
            if (pown >> 1 == lane) sPM[cw] = (pown & 1) ? fma(ekx, e1, a.y) : fma(ekx, e, a.x);
        }
    }
    if (correct) {  // mode coefficients of the block's columns: four threads a mode, 16 chunks each
        const int part = tid & 3;
        double2 ph = ph_t;
        for (int task = tid >> 2; task < W * nmode; task += blockDim.x >> 2) {
            const int mw = task & (W - 1), ky = task >> wshift;  // mode ky + 1
            if (task >= (int)blockDim.x >> 2) {
                ph = __ldg(&ys.phase[part * kYFull + ky]);
                ph_r = __ldg(&ys.phase[kYChunks * kYFull + ky]);
            }
            const double om = 3.14159265358979323846 / M * (ky + 1);
            double s0 = 0.0, s1 = 0.0;
#pragma unroll
            for (int q = 0; q < kYChunks / 4; ++q) {
                const double2 mm = mom[(q * 4 + part) * W + mw];
                s0 = fma(mm.x, ph.x, s0);
                s1 = fma(mm.y, ph.y, s1);
                ph = make_double2(fma(ph.x, ph_r.y, ph.y * ph_r.x), fma(ph.y, ph_r.y, -ph.x * ph_r.x));  // 4 chunks on
            }
            double acc = fma(om, s1, s0);
            const unsigned quad = 0xfu << (tid & 28);  // the task's four threads
            acc += __shfl_xor_sync(quad, acc, 1);
            acc += __shfl_xor_sync(quad, acc, 2);
            if (part == 0)
                modes[mw][ky] = c0 + mw < kYModes ? acc * __ldg(ys.diff + b * ys.dstride + (c0 + mw) * kYFull + ky) : 0.0;
        }
    }
    __syncthreads();

    const double Q0 = fma(rh, sQ1[w], rl * sQ1[w]), PM = sPM[w];
    const double A = fma(-ce.x, PM, Q0) * ce.y, B = fma(-ce.x, Q0, PM) * ce.y;
    double P = fma(-A, sA[w * S + p], sP[w * S + p]);
    double Q = j0 + MR < M ? fma(-B, sB[w * S + p], sQ[w * S + p]) : -B;
    double x[MR];
#pragma unroll
    for (int k = 0; k < MR; ++k) {
        x[k] = fma(rh, P, rl * P);
        P = x[k] + v[k];
    }
#pragma unroll
    for (int k = MR - 1; k >= 0; --k) {
        if (j0 + k < n) {
            Q = fma(rh, Q, fma(rl, Q, v[k]));
            x[k] = (x[k] + Q) * kap;
        }
    }
    if (correct && col < kYModes) {
        double e0 = 0.0, e1 = 0.0;
        double2 ph = ph_p;
        for (int ky = 0; ky < nmode; ++ky) {
            const double a = modes[w][ky];
            e0 = fma(a, ph.x, e0);
            e1 = fma(a * (ky + 1), ph.y, e1);
            ph = make_double2(fma(ph.x, ph_p.y, ph.y * ph_p.x), fma(ph.y, ph_p.y, -ph.x * ph_p.x));  // next mode
        }
        e1 *= 3.14159265358979323846 / M;
#pragma unroll
        for (int k = 0; k < MR; ++k) x[k] = full ? e0 : x[k] + fma((double)(k - KC), e1, e0);
    }
    if (valid) {
#pragma unroll
        for (int k = 0; k < MR; ++k)
            if (j0 + k < n) src[ld * k] = x[k];
    }
}

// The column constants and correction tables of the solves of gridDim.y
// coefficients coef[b] (null: the Laplacian inverse), and the modes' phases.
// gridDim.x * blockDim.x >= max(nx - 1, (kYChunks + 1) kYFull).
static __global__ void ycols_kernel(YCol *cols, double *diff, double2 *phase, const double *cx, const double *cy, int nx,
                                    int M, int MR, const double *coef) {
    const int b = blockIdx.y, q = blockIdx.x * blockDim.x + threadIdx.x, n = M - 1;
    const bool lap = coef == nullptr;
    const double c = lap ? 0.0 : coef[b];
    const double ic = lap ? 1.0 : fmin(1 / c, 1e150);  // t^2 stays finite
    if (q < nx - 1) {
        const double t0 = 2 - 2 * cx[q + 1], t = lap ? t0 : t0 + ic;
        const double root = sqrt(t * t + 4 * t), s = 2 * t / (t + root);  // s = 1 - r
        YCol y;
        y.rh = 2 / (2 + t + root);
        y.rl = y.rh >= 0.5 ? (1 - y.rh) - s : 0.0;
        const double lr = y.rh >= 0.5 ? log1p(-s) : log(y.rh);
        const int k = M - (M - 1) / MR * MR;
        y.R = exp(MR * lr);
        y.kap = y.rh / (s * (1 + y.rh)) * (ic / (2.0 * nx));
        y.eM = exp(M * lr);
        y.det = -1 / expm1(2 * M * lr);
        y.ek = exp(k * lr);
        y.ek1 = exp((k - 1) * lr);
        y.sx = 2 * sinpi((double)(q + 1) / nx);
        y.pad = 0.0;
        cols[(long long)b * (nx - 1) + q] = y;
    }
    const bool full = n <= kYFull;
    double *d = diff + (long long)b * kYDiff;
    if (q < kYModes * kYFull) {
        const int kx = q / kYFull + 1, ky = q % kYFull + 1;
        double a = 0.0;
        if (kx < nx && ky <= (full ? n : min(kYModes, n))) {
            const double h = sinpi(0.5 * ky / M);
            const double lref = -2 * ((cx[kx] + cy[ky]) - 2), lam = (2 - 2 * cx[kx]) + 4 * h * h;
            const double dref = lap ? lref : 1 + c * lref, dl = lap ? lam : 1 + c * lam;
            a = full ? 1 / dref : (lap ? 1.0 : c) * (lam - lref) / (dl * dref);
            a /= (double)nx * M;  // 1 / (2 nx) of the X passes, 2 / M of the mode's norm
        }
        d[q] = a;
    }
    if (q == 0) {
        // in use where the cosines' rounding is above 1e-14 of the eigenvalue
        double off = full ? 1.0 : 0.0;
        for (int k = 1; k <= min(4, min(nx - 1, n)) * 4; ++k) {
            const int kx = (k - 1) / 4 + 1, ky = (k - 1) % 4 + 1;
            if (ky > n) continue;
            const double h = sinpi(0.5 * ky / M), lref = -2 * ((cx[kx] + cy[ky]) - 2);
            const double lam = (2 - 2 * cx[kx]) + 4 * h * h;
            off = fmax(off, fabs(lam - lref) / (lam + (lap ? 0.0 : ic)));
        }
        d[kYDiff - 1] = off > 1e-14 ? 1.0 : 0.0;
    }
    if (b == 0 && q < (kYChunks + 1) * kYFull) {
        const int ky = q % kYFull + 1, p = q / kYFull;
        const int jc = p < kYChunks ? p * MR + 1 + (MR - 1) / 2 : 4 * MR;
        double sn, cs;
        sincospi((double)((ky * jc) % (2 * M)) / M, &sn, &cs);
        phase[q] = make_double2(sn, cs);
    }
}

// Explicit diffusion (1 - c (T + t)) b of the columns after the X pass, not in place.
template <class T>
__global__ void yexpl_kernel(const T *__restrict__ in, T *__restrict__ out, int ld, int nx, int M, double c,
                             const double *__restrict__ cx) {
    const int col = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y * blockDim.y + threadIdx.y + 1;
    if (col >= nx - 1 || j > M - 1) return;
    const T *src = in + col + (long long)ld * (j - 1);
    const double t = 2 - 2 * cx[col + 1];
    const double v = (double)src[0], lo = j > 1 ? (double)src[-ld] : 0.0, hi = j < M - 1 ? (double)src[ld] : 0.0;
    out[col + (long long)ld * (j - 1)] = (T)((fma(-c, fma(t, v, 2 * v - lo - hi), v)) / (2.0 * nx));
}

// Columns per block, as log2, for nbatch fields of ncols columns (measured,
// 2 / 4 / 8 columns: one 1024^2 field 8.3 / 6.5 / 10.0 us, five 31.8 / 20.3 /
// 22.7 us; one 256^2 field 3.7 / 4.3 / 8.0 us, where few blocks leave the
// correcting ones as the kernel's length).
inline int ytri_wshift(int ncols, int nbatch) { return (long long)ncols * nbatch < 300 ? 1 : 2; }

// Rows per thread of a transform length M: the smallest compiled chunk that covers it.
inline int ytri_rows(int M) {
    const int need = (M + kYChunks - 1) / kYChunks;
    for (int r : {1, 2, 3, 4, 5, 6, 8, 10, 12, 14, 16})
        if (r >= need) return r;
    return 0;
}

// Writes the tables of nb coefficients (coef device, or null with nb = 1); the
// return code is the launch's own.
inline cudaError_t launch_ycols(YCol *cols, double *diff, double2 *phase, const double *cx, const double *cy, int nx, int M,
                                const double *coef, int nb, cudaStream_t st) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(((kYChunks + 1) * kYFull + 127) / 128, nb);  // more than 1023 threads, so every column too
    cfg.blockDim = dim3(128);
    cfg.stream = st;
    return cudaLaunchKernelEx(&cfg, ycols_kernel, cols, diff, phase, cx, cy, nx, M, ytri_rows(M), coef);
}

// Enqueues the Y solve, in place, of nbatch fields with 1 << wshift columns a block; the
// return code is the launch's own.
inline cudaError_t launch_ytri(double *f, long long bs, int ld, int ncols, int M, int nbatch, int wshift,
                               const YSolve &ys, cudaStream_t st, const YRing &yr = {}, bool overlap = false) {
    auto go = [&](auto *k) {
        return launch_overlapped(overlap, k, dim3((ncols + (1 << wshift) - 1) >> wshift, nbatch), dim3(kYChunks << wshift), 0,
                                 st, f, bs, ld, ncols, M, wshift, ys, yr);
    };
    switch (ytri_rows(M)) {
        case 1: return yr.lines ? go(ytri_kernel<1, true>) : go(ytri_kernel<1, false>);
        case 2: return yr.lines ? go(ytri_kernel<2, true>) : go(ytri_kernel<2, false>);
        case 3: return yr.lines ? go(ytri_kernel<3, true>) : go(ytri_kernel<3, false>);
        case 4: return yr.lines ? go(ytri_kernel<4, true>) : go(ytri_kernel<4, false>);
        case 5: return yr.lines ? go(ytri_kernel<5, true>) : go(ytri_kernel<5, false>);
        case 6: return yr.lines ? go(ytri_kernel<6, true>) : go(ytri_kernel<6, false>);
        case 8: return yr.lines ? go(ytri_kernel<8, true>) : go(ytri_kernel<8, false>);
        case 10: return yr.lines ? go(ytri_kernel<10, true>) : go(ytri_kernel<10, false>);
        case 12: return yr.lines ? go(ytri_kernel<12, true>) : go(ytri_kernel<12, false>);
        case 14: return yr.lines ? go(ytri_kernel<14, true>) : go(ytri_kernel<14, false>);
        case 16: return yr.lines ? go(ytri_kernel<16, true>) : go(ytri_kernel<16, false>);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace ibpm
