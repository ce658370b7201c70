// kernels.cuh -- device kernels of the IBPM time step (line passes, stencils,
// B^-1 algebra).  Field element type T is double (plain FP64 path) or float
// (mixed-precision path); arithmetic on boundary values, multipliers and
// coupling sums is done in double.  Included by ibpm.cu only.
#pragma once
#include <type_traits>
#include "common.cuh"
#include "fft_pow2.cuh"
#include "tc_dst.h"
#include "ytri.cuh"

namespace ibpm {

// ---------------------------------------------------------------------------
// Line-pass kernels
// ---------------------------------------------------------------------------

// Shared-memory layout of a pass kernel: nbuf line buffers of D::C, then the
// double2 scan scratch at a 16-byte boundary.
template <class D>
__host__ __device__ constexpr size_t scratch_offset(int M, int nbuf) {
    return ((size_t)nbuf * D::smem_len(M) * sizeof(typename D::C) + 15) / 16 * 16;
}
template <class D>
__host__ __device__ constexpr size_t pass_smem(int M, int nbuf, int ngroups) {
    return scratch_offset<D>(M, nbuf) + (size_t)D::NWARP * ngroups * sizeof(double2);
}

// Prologue: plain field
template <class T>
struct InPlain {
    const T *p;
    long long bs;
    int ld;
    __device__ __forceinline__ double operator()(int b, int i, int j) const {
        return (double)p[b * bs + (long long)(i - 1) + (long long)ld * (j - 1)];
    }
};

// Prologue: levels of several fields, batch b level b % nl (ls apart) of field b / nl.
// at(b) is the one level as a plain field: the X pass resolves it once per block
// (the division, left in the load, cost a 1024^2 pass 4 of its 12.7 us).
template <class T>
struct InLevels {
    const T *p;
    long long bs;
    int ld, nl;
    long long ls;
    __device__ __forceinline__ InPlain<T> at(int b) const { return InPlain<T>{p + (b / nl) * bs + (b % nl) * ls, 0, ld}; }
};
template <class In>
__device__ __forceinline__ const In &resolve(const In &in, int) { return in; }
template <class T>
__device__ __forceinline__ InPlain<T> resolve(const InLevels<T> &in, int b) { return in.at(b); }

// Prologue of the telescoping solves that add the boundary values to the field
// (FP32 levels, tensor-core transforms; src/fluid.jl:194-197):
// Gamma_tmp = Gamma[:, lev]; apply_bc!(Gamma_tmp, get_bc(psi[:, lev+1]); fac=1)
// (the coarser level's psi may be of another element type TC)
template <class T, class TC = T>
struct InBC {
    const T *gam;
    const TC *coarse;
    long long bs, cbs;
    Grid g;
    __device__ __forceinline__ double operator()(int b, int i, int j) const {
        const T *G = gam + b * bs;
        double v = (double)G[GI(i, j)];
        if (on_ring(g, i, j)) v = apply_bc_at(v, coarse + b * cbs, g, i, j, 1.0);
        return v;
    }
    // The compile-time X pass loads the field alone (plain()) and then adds the
    // boundary values to the ring elements (ring()), so the loads of a line are
    // not held up behind the boundary reads; the sum is the one operator() forms.
    static constexpr bool kSplitRing = true;
    __device__ __forceinline__ double plain(int b, int i, int j) const { return (double)gam[b * bs + GI(i, j)]; }
    __device__ __forceinline__ bool ring_row(int j) const { return j == 1 || j == g.ny - 1; }
    __device__ __forceinline__ double ring(double v, int b, int i, int j) const {
        return apply_bc_at(v, coarse + b * cbs, g, i, j, 1.0);
    }
};

// detects the split prologue of InBC
template <class In, class = void>
struct SplitRing {
    static constexpr bool value = false;
};
template <class In>
struct SplitRing<In, std::void_t<decltype(In::kSplitRing)>> {
    static constexpr bool value = In::kSplitRing;
};

// A prologue over a field that is zero outside the block i0..i1 x j0..j1: there
// the field reads as zero without a load (the boundary values on the ring are
// still added).  The coarse levels of a B application are such fields: their
// vorticity is the finer level's coarsified into the central block
// (coarsify!, src/fluid.jl:208-228), and zero elsewhere.
template <class In>
struct InCentral {
    In in;
    int i0, i1, j0, j1;
    static constexpr bool kSplitRing = SplitRing<In>::value;
    __device__ __forceinline__ bool inside(int i, int j) const { return i >= i0 && i <= i1 && j >= j0 && j <= j1; }
    __device__ __forceinline__ double operator()(int b, int i, int j) const {
        if constexpr (kSplitRing)
            return inside(i, j) ? in(b, i, j) : in.ring(0.0, b, i, j);
        else
            return inside(i, j) ? in(b, i, j) : 0.0;
    }
    __device__ __forceinline__ double plain(int b, int i, int j) const { return inside(i, j) ? in.plain(b, i, j) : 0.0; }
    __device__ __forceinline__ bool ring_row(int j) const { return in.ring_row(j); }
    __device__ __forceinline__ double ring(double v, int b, int i, int j) const { return in.ring(v, b, i, j); }
};

// Prologue rot!(Gamma, reg!(q, f)) (src/fluid.jl:101-111 after src/coupling.jl:72-85),
// evaluated from the regularised patch.
template <class T>
struct InRegRot {
    Patch<T> pt;
    __device__ __forceinline__ double operator()(int b, int I, int J) const {
        return (pt.get(b, 0, I + 1, J) - pt.get(b, 0, I + 1, J + 1)) + (pt.get(b, 1, I + 1, J + 1) - pt.get(b, 1, I, J + 1));
    }
};

// Prologue rot!(Gamma, reg!(q, f)) of the cases of a batched ensemble group:
// batch b reads case b's patch (zero outside its bounding box).
template <class T>
struct InRegRotTab {
    const CaseView *tab;
    __device__ __forceinline__ double operator()(int b, int I, int J) const {
        const CaseView &cv = tab[b];
        const Patch<T> pt{static_cast<const T *>(cv.patch), cv.P.bbox, 0};
        return (pt.get(0, 0, I + 1, J) - pt.get(0, 0, I + 1, J + 1)) + (pt.get(0, 1, I + 1, J + 1) - pt.get(0, 1, I, J + 1));
    }
};

// Epilogue: plain store
template <class T>
struct OutPlain {
    T *p;
    long long bs;
    int ld;
    __device__ __forceinline__ void operator()(int b, int i, int j, double v) const {
        p[b * bs + (long long)(i - 1) + (long long)ld * (j - 1)] = (T)v;
    }
};

// Epilogue of project_circ (src/coupling.jl:227): Gamma[:, 1] .-= x
template <class T>
struct OutSub {
    T *p;
    long long bs;
    int ld;
    // The X pass fetches the targets eight at a time and then stores: read between
    // the stores, one after another, they cost a 1024^2 pass 15 of its 24 us.
    static constexpr bool kReads = true;
    __device__ __forceinline__ T load(int b, int i, int j) const { return p[b * bs + (long long)(i - 1) + (long long)ld * (j - 1)]; }
    __device__ __forceinline__ void store(int b, int i, int j, T old, double v) const {
        p[b * bs + (long long)(i - 1) + (long long)ld * (j - 1)] = (T)((double)old - v);
    }
    __device__ __forceinline__ void operator()(int b, int i, int j, double v) const {
        T *q = p + b * bs + (long long)(i - 1) + (long long)ld * (j - 1);
        *q = (T)((double)*q - v);
    }
};

// Boundary values of the next finer level (get_bc! of a solved level's psi,
// src/fluid.jl:278-306) as the finer level's Y solve takes them.  Per batch:
// 2 nx doubles, the DST along x of the interpolated rows ny/4 and 3 ny/4 (at
// their kx - 1), then 2 ny doubles, the columns nx/4 and 3 nx/4 by row.
// A source on the field's outer rows enters its column systems as those two
// transformed rows, one on its outer columns as two sine-weighted vectors, so
// the X passes need no boundary values and run for all levels at once.
//
// The rows' way from the solved scratch field (kx, y) to there is linear:
// back along x, the centre part interpolated, and along x again.  Q is that
// operator as a matrix (ring_matrix_kernel), so a few warps form both rows as dot
// products.  As two transforms in one block, one after the other, they were the
// length of every kernel that held them: 11 us of a 17 us one at 1024 points.
struct RingOut {
    double *lines = nullptr;
    long long stride = 0;
    int nx = 0, ny = 0;
    const double *Q = nullptr;  // row kx - 1, qld entries
    int qld = 0, step = 1;      // step 2: only modes of kx's parity couple (nx a multiple of 4)
};

// One output mode per call: kx - 1 = k of both rows of batches b .. b + F - 1, by
// the calling warp: an entry of Q is read once for all of them.
template <int F, class In>
__device__ __forceinline__ void ring_mode_f(const In &in, int b, const RingOut &ro, int k) {
    const int lane = threadIdx.x & 31, jb = ro.ny / 4, jt = 3 * ro.ny / 4;
    const int m0 = ro.step == 2 ? (k & 1) + 1 : 1;  // first input mode
    const int nm = ro.step == 2 ? (ro.nx - m0 + 1) / 2 : ro.nx - 1;
    const double *__restrict__ row = ro.Q + (long long)ro.qld * k;
    double sb[F] = {}, st[F] = {};
#pragma unroll(8 / F)
    for (int q = lane; q < nm; q += 32) {
        const int m = m0 + q * ro.step;
        const double w = __ldg(&row[q]);
#pragma unroll
        for (int f = 0; f < F; ++f) {
            sb[f] = fma(w, in(b + f, m, jb), sb[f]);
            st[f] = fma(w, in(b + f, m, jt), st[f]);
        }
    }
#pragma unroll
    for (int f = 0; f < F; ++f) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            sb[f] += __shfl_xor_sync(0xffffffffu, sb[f], o);
            st[f] += __shfl_xor_sync(0xffffffffu, st[f], o);
        }
        if (lane == 0) {
            double *dst = ro.lines + (b + f) * ro.stride + k;
            dst[0] = sb[f];
            dst[ro.nx] = st[f];
        }
    }
}
// the batches b .. b + kRingF - 1 of nb, for b a multiple of kRingF
constexpr int kRingF = 4;
template <class In>
__device__ __forceinline__ void ring_mode(const In &in, int b, int nb, const RingOut &ro, int k) {
    if (b % kRingF != 0) return;
    if (b + kRingF <= nb) {
        ring_mode_f<kRingF>(in, b, ro, k);
    } else {
        for (; b < nb; ++b) ring_mode_f<1>(in, b, ro, k);
    }
}
// Q[k][q] = sum_i 2 sin(pi kx i / nx) ring_i(m), ring_i(m) the mode m interpolated
// to the finer level's boundary point i (sn: sin(pi j / nx), j <= nx).
static __global__ void ring_matrix_kernel(double *Q, int qld, int step, int nx, const double *__restrict__ sn) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x, k = blockIdx.y, kx = k + 1;
    const int m = step == 2 ? (k & 1) + 1 + 2 * q : q + 1;
    if (q >= qld) return;
    double acc = 0.0;
    if (m < nx) {
        auto sine = [&](int a) {  // sin(pi a / nx), a >= 0
            a %= 2 * nx;
            return a <= nx ? __ldg(&sn[a]) : -__ldg(&sn[2 * nx - a]);
        };
        double lo = 2 * sine(m * (nx / 4));
        for (int c = 1; c <= nx / 2; ++c) {  // coarse point nx/4 + c: boundary points 2c - 1 and 2c
            const double hi = 2 * sine(m * (nx / 4 + c));
            acc = fma(2 * sine(kx * (2 * c - 1)), 0.5 * (hi + lo), acc);
            if (2 * c < nx) acc = fma(2 * sine(kx * (2 * c)), hi, acc);
            lo = hi;
        }
    }
    Q[(long long)qld * k + q] = acc;
}

// A solved coarse level reduced to what the finer level reads: one warp per row j
// in ny/4 .. ny/4 + ny/2 for the columns psi(nx/4, j) and psi(3 nx/4, j) as
// weighted sums over kx (wl, wr: 2 sin(pi kx i / nx), RODFT00's factor), one per
// mode of the rows.  The chain from level to level waits for this (4.5 us for one
// 1024^2 FP64 level) and not for the level's last X pass (8.7 us), which runs for
// all levels at once after it, or not at all where only the level-1 flux is
// wanted.  psi (may be null; batch stride pbs): where a window
// (win + win_stride b, or everywhere if null) reaches the domain's boundary, whose
// faces a curl takes from the coarser level, the first block also stores those two
// rows and the others the two columns of psi.
template <class D>
__global__ void __launch_bounds__(64)
    xlines_kernel(InPlain<typename D::Real> in, RingOut ro, PlanT<typename D::Real> pl, const double *__restrict__ wl,
                  const double *__restrict__ wr, typename D::Real *psi, long long pbs, const int *__restrict__ win,
                  int win_stride) {
    overlap_begin();
    using T = typename D::Real;
    using C = typename D::C;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int b = blockIdx.y, t = threadIdx.x, bx = (int)blockIdx.x - 1;
    if (psi != nullptr && win != nullptr) {
        const int *w = win + b * win_stride;
        if (w[0] > 1 && w[1] < ro.nx && w[2] > 1 && w[3] < ro.ny) psi = nullptr;
    }
    if (bx < 0) {
        if (psi == nullptr) return;
        psi += b * pbs;
        C *buf = reinterpret_cast<C *>(smem_raw) + (t / D::TPF) * D::smem_len(pl.M);
        double2 *wt = reinterpret_cast<double2 *>(smem_raw + scratch_offset<D>(pl.M, 64 / D::TPF)) + D::NWARP * (t / D::TPF);
        const int jb = ro.ny / 4, jt = 3 * ro.ny / 4, tt = t % D::TPF;  // every group holds the same line
        for (int i = tt; i <= pl.M; i += D::TPF)
            buf[D::idx(i)] = i >= 1 && i < pl.M ? Cx<T>::make((T)in(b, i, jb), (T)in(b, i, jt)) : Cx<T>::make(0, 0);
        __syncthreads();
        D::dst(buf, pl, tt, wt);
        if (t < D::TPF)
            for (int i = 1 + tt; i < pl.M; i += D::TPF) {
                const C y = buf[D::idx(i)];
                psi[(i - 1) + (long long)(pl.M - 1) * (jb - 1)] = y.x;
                psi[(i - 1) + (long long)(pl.M - 1) * (jt - 1)] = y.y;
            }
        return;
    }
    const int task = bx * 2 + (t >> 5), ncol = ro.ny / 2 + 1;
    if (task >= ncol) {
        if (task - ncol < ro.nx - 1) ring_mode(in, b, (int)gridDim.y, ro, task - ncol);
        return;
    }
    const int j = ro.ny / 4 + task;
    double sl = 0.0, sr = 0.0;
#pragma unroll 8
    for (int i = 1 + (t & 31); i < ro.nx; i += 32) {
        const double v = in(b, i, j);
        sl = fma(v, __ldg(&wl[i - 1]), sl);
        sr = fma(v, __ldg(&wr[i - 1]), sr);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        sl += __shfl_xor_sync(0xffffffffu, sl, o);
        sr += __shfl_xor_sync(0xffffffffu, sr, o);
    }
    if ((t & 31) == 0) {
        double *col = ro.lines + b * ro.stride + 2 * ro.nx + (j - 1);
        col[0] = (double)(T)sl;
        col[ro.ny] = (double)(T)sr;
        if (psi != nullptr && j != ro.ny / 4 && j != 3 * ro.ny / 4) {  // those rows are the first block's
            T *row = psi + b * pbs + (long long)(ro.nx - 1) * (j - 1) - 1;
            row[ro.nx / 4] = (T)sl;
            row[3 * ro.nx / 4] = (T)sr;
        }
    }
}

// an epilogue that reads its target
template <class Out, class = void>
struct ReadsTarget {
    static constexpr bool value = false;
};
template <class Out>
struct ReadsTarget<Out, std::void_t<decltype(Out::kReads)>> {
    static constexpr bool value = Out::kReads;
};

// X pass: DST along x of rows (ja, jb) = (2p+1, 2p+2) of each batch field.
// D is the line transform (Pow2Dst<M> or GenericDst); NG line pairs per block.
// rows (device, may be null): a face window i0, i1, j0, j1 (batch b's at rows +
// (b % rows_mod) rows_stride).  A block
// none of whose rows lies in j0-1 .. j1 returns at once: with zero_outside = 0
// its output rows stay unwritten (the rows a curl of those faces reads lie
// inside), with zero_outside = 1 it writes them as zeros (the transform of the
// input's zero rows: rot of a patch inside the window is zero outside them).
template <class D, int NG, class In, class Out>
__global__ void __launch_bounds__(D::TPF *NG, D::OCC / (D::TPF * NG))
    xpass_kernel(In inp, Out out, PlanT<typename D::Real> pl, int nrows, const int *__restrict__ rows = nullptr,
                 int zero_outside = 0, int rows_stride = 0, int rows_mod = 1) {
    overlap_begin();
    const int bx = blockIdx.x;
    if (rows != nullptr) {  // uniform over the block: before any barrier
        rows += (long long)rows_stride * (blockIdx.y % rows_mod);
        const int r0 = 2 * NG * bx + 1, r1 = r0 + 2 * NG - 1;
        if (r1 < rows[2] - 1 || r0 > rows[3]) {
            if (zero_outside) {
                const int t = threadIdx.x % D::TPF, ja = r0 + 2 * (int)(threadIdx.x / D::TPF);
                for (int jj = ja; jj <= ja + 1 && jj <= nrows; ++jj)
                    for (int i = 1 + t; i < pl.M; i += D::TPF) out((int)blockIdx.y, i, jj, 0.0);
            }
            return;
        }
    }
    using T = typename D::Real;
    using C = typename D::C;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    C *smem = reinterpret_cast<C *>(smem_raw);
    constexpr int TPF = D::TPF;
    const int M = pl.M;
    const int G = D::smem_len(M);
    const int g = threadIdx.x / TPF, t = threadIdx.x % TPF;
    C *buf = smem + g * G;
    double2 *wt = reinterpret_cast<double2 *>(smem_raw + scratch_offset<D>(M, NG)) + D::NWARP * g;
    const int b = blockIdx.y;
    const auto in = resolve(inp, b);
    const int pair = bx * NG + g;
    const int ja = 2 * pair + 1, jb = 2 * pair + 2;
    const bool va = ja <= nrows, vb = jb <= nrows;
    if constexpr (D::MC > 0) {
        // compile-time trip count: every global load of the thread is in flight
        // before the first shared-memory store
        constexpr int NIT = (D::MC + 1 + TPF - 1) / TPF;
        T za[NIT], zb[NIT];
        if constexpr (SplitRing<In>::value) {
#pragma unroll
            for (int k = 0; k < NIT; ++k) {
                const int i = t + k * TPF;
                const bool in_line = i >= 1 && i < D::MC;
                za[k] = (in_line && va) ? (T)in.plain(b, i, ja) : (T)0;
                zb[k] = (in_line && vb) ? (T)in.plain(b, i, jb) : (T)0;
            }
            // boundary values on the ring: whole rows 1 and ny-1, the ends of the others
            const bool ra = va && in.ring_row(ja), rb = vb && in.ring_row(jb);
#pragma unroll
            for (int k = 0; k < NIT; ++k) {
                const int i = t + k * TPF;
                if (i < 1 || i >= D::MC) continue;
                const bool end = i == 1 || i == D::MC - 1;
                // za[k] holds the field value exactly ((T)(double)x == x), so no reload
                if (va && (ra || end)) za[k] = (T)in.ring((double)za[k], b, i, ja);
                if (vb && (rb || end)) zb[k] = (T)in.ring((double)zb[k], b, i, jb);
            }
        } else {
#pragma unroll
            for (int k = 0; k < NIT; ++k) {
                const int i = t + k * TPF;
                const bool in_line = i >= 1 && i < D::MC;
                za[k] = (in_line && va) ? (T)in(b, i, ja) : (T)0;
                zb[k] = (in_line && vb) ? (T)in(b, i, jb) : (T)0;
            }
        }
#pragma unroll
        for (int k = 0; k < NIT; ++k) {
            const int i = t + k * TPF;
            if (i <= D::MC) buf[D::idx(i)] = Cx<T>::make(za[k], zb[k]);
        }
    } else {
        // loads of eight elements of both rows in flight before their stores
        constexpr int CH = 8;
        for (int i0 = t; i0 <= M; i0 += CH * TPF) {
            T za[CH], zb[CH];
#pragma unroll
            for (int k = 0; k < CH; ++k) {
                const int i = i0 + k * TPF;
                const bool in_line = i >= 1 && i < M;
                za[k] = (in_line && va) ? (T)in(b, i, ja) : (T)0;
                zb[k] = (in_line && vb) ? (T)in(b, i, jb) : (T)0;
            }
#pragma unroll
            for (int k = 0; k < CH; ++k)
                if (i0 + k * TPF <= M) buf[D::idx(i0 + k * TPF)] = Cx<T>::make(za[k], zb[k]);
        }
    }
    __syncthreads();
    D::dst(buf, pl, t, wt);
    if constexpr (ReadsTarget<Out>::value) {
        constexpr int CH = 8;
        for (int i0 = 1 + t; i0 < M; i0 += CH * TPF) {
            T oa[CH], ob[CH];
#pragma unroll
            for (int k = 0; k < CH; ++k) {
                const int i = i0 + k * TPF;
                oa[k] = i < M && va ? out.load(b, i, ja) : (T)0;
                ob[k] = i < M && vb ? out.load(b, i, jb) : (T)0;
            }
#pragma unroll
            for (int k = 0; k < CH; ++k) {
                const int i = i0 + k * TPF;
                if (i >= M) break;
                const C y = buf[D::idx(i)];
                if (va) out.store(b, i, ja, oa[k], y.x);
                if (vb) out.store(b, i, jb, ob[k], y.y);
            }
        }
    } else {
        for (int i = 1 + t; i < M; i += TPF) {
            const C y = buf[D::idx(i)];
            if (va) out(b, i, ja, y.x);
            if (vb) out(b, i, jb, y.y);
        }
    }
}

// Y pass by transforms: for each column i, x[i, :] = DST_y(mult(i, :) * DST_y(in[i, :])),
// Laplacian inverse (coef null) or implicit diffusion of coefficients coef[b coef_stride].
// A block owns 2*NG adjacent columns; loads and stores are row-coalesced; in
// place or not.  The FP32 engine's solves: the direct solve (ytri.cuh) is faster
// and closer to 64 bits for them too, but an FP32 run is reproducible only bit for
// bit (one changed rounding draws the transforms' noise anew, 1e-5 of the
// vorticity in ten steps and 1e-4..1e-3 of the forces), so that engine keeps its
// order of operations, its FP64 level-1 solves and B^-1 included.
template <class D, int NG>
__global__ void __launch_bounds__(D::TPF *NG, D::OCC / (D::TPF * NG))
    ypass_kernel(const typename D::Real *in, typename D::Real *out, long long bs, int ld, int ncols,
                 PlanT<typename D::Real> pl, const double *__restrict__ coef, int coef_stride,
                 const double *__restrict__ cx, const double *__restrict__ cy, double scale) {
    using T = typename D::Real;
    using C = typename D::C;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    C *smem = reinterpret_cast<C *>(smem_raw);
    constexpr int TPF = D::TPF;
    const int M = pl.M;
    const int G = D::smem_len(M);
    const int g = threadIdx.x / TPF, t = threadIdx.x % TPF;
    C *buf = smem + g * G;
    double2 *wt = reinterpret_cast<double2 *>(smem_raw + scratch_offset<D>(M, NG)) + D::NWARP * g;
    const int b = blockIdx.y;
    const int c0 = blockIdx.x * 2 * NG;  // 0-based first column of the block
    const T *src = in + b * bs;
    T *dst = out + b * bs;
    constexpr int W = 2 * NG;
    if constexpr (D::MC > 0) {
        // compile-time trip count, loads issued in chunks of CH before their stores
        constexpr int NT = NG * TPF;
        constexpr int NIT = (W * (D::MC + 1) + NT - 1) / NT;
        constexpr int CH = 12;
#pragma unroll
        for (int k0 = 0; k0 < NIT; k0 += CH) {
            T v[CH];
#pragma unroll
            for (int k = 0; k < CH; ++k) {
                const int e = threadIdx.x + (k0 + k) * NT;
                const int c = e % W, jj = e / W;
                const int col = c0 + c;
                v[k] = (k0 + k < NIT && jj >= 1 && jj < D::MC && col < ncols) ? src[col + (long long)ld * (jj - 1)]
                                                                               : (T)0;
            }
#pragma unroll
            for (int k = 0; k < CH; ++k) {
                const int e = threadIdx.x + (k0 + k) * NT;
                const int c = e % W, jj = e / W;
                if (k0 + k < NIT && jj <= D::MC) *(reinterpret_cast<T *>(smem + (c >> 1) * G + D::idx(jj)) + (c & 1)) = v[k];
            }
        }
    } else {
        for (int e = threadIdx.x; e < W * (M + 1); e += blockDim.x) {
            const int c = e % W, jj = e / W;
            const int col = c0 + c;
            T v = 0;
            if (jj >= 1 && jj < M && col < ncols) v = src[col + (long long)ld * (jj - 1)];
            T *slot = reinterpret_cast<T *>(smem + (c >> 1) * G + D::idx(jj)) + (c & 1);
            *slot = v;
        }
    }
    __syncthreads();
    // DST, spectral multiply, DST; one loop body so the transform is emitted once
#pragma unroll 1
    for (int pass = 0; pass < 2; ++pass) {
        D::dst(buf, pl, t, wt);
        if (pass == 1) break;
        const int ia = c0 + 2 * g + 1, ib = c0 + 2 * g + 2;  // 1-based columns
        const double cb = coef ? coef[b * coef_stride] : 0.0;
        auto factor = [&](double cxi, double cyj) -> double {
            const double lam = -2 * ((cxi + cyj) - 2);
            return scale * recip(coef ? 1 + lam * cb : lam);
        };
        if constexpr (D::MC > 0) {
            constexpr int NIT = (D::MC - 1 + TPF - 1) / TPF;
            const double cxa = ia <= ncols ? __ldg(&cx[ia]) : 0.0, cxb = ib <= ncols ? __ldg(&cx[ib]) : 0.0;
            double cyv[NIT];
#pragma unroll
            for (int k = 0; k < NIT; ++k) {
                const int jj = 1 + t + k * TPF;
                cyv[k] = jj < D::MC ? __ldg(&cy[jj]) : 0.0;
            }
#pragma unroll
            for (int k = 0; k < NIT; ++k) {
                const int jj = 1 + t + k * TPF;
                if (jj >= D::MC) break;
                C y = buf[D::idx(jj)];
                y.x = (T)(y.x * ((ia <= ncols) ? factor(cxa, cyv[k]) : 0.0));
                y.y = (T)(y.y * ((ib <= ncols) ? factor(cxb, cyv[k]) : 0.0));
                buf[D::idx(jj)] = y;
            }
        } else {
            for (int jj = 1 + t; jj < M; jj += TPF) {
                C y = buf[D::idx(jj)];
                y.x = (T)(y.x * ((ia <= ncols) ? factor(__ldg(&cx[ia]), __ldg(&cy[jj])) : 0.0));
                y.y = (T)(y.y * ((ib <= ncols) ? factor(__ldg(&cx[ib]), __ldg(&cy[jj])) : 0.0));
                buf[D::idx(jj)] = y;
            }
        }
        __syncthreads();
    }
    for (int e = threadIdx.x; e < W * (M + 1); e += blockDim.x) {
        const int c = e % W, jj = e / W;
        const int col = c0 + c;
        if (jj >= 1 && jj < M && col < ncols) {
            const T *slot = reinterpret_cast<const T *>(smem + (c >> 1) * G + D::idx(jj)) + (c & 1);
            dst[col + (long long)ld * (jj - 1)] = *slot;
        }
    }
}

// ---------------------------------------------------------------------------
// Merged trial solve of get_trial_state (src/fluid.jl:485-496) by transforms:
//   Gamma_s = Ainv (A Gamma + rest),  rest = dt (1.5 N1 - 0.5 N2) + rhsbc.
// With S the 2D DST-I and S S = 1/scale:  S(A Gamma) = S(Gamma) / Lambda_e, so
//   Gamma_s = S( scale / Lambda_i * ( S(Gamma) / Lambda_e + S(rest) ) ),
// three passes instead of the reference's four transforms in six passes.  The FP32
// engine's; the FP64 engine takes A Gamma from the nonlinear kernel's stencil and
// one field through the general passes (84 against 220 us at 1024^2 x 5).
// ---------------------------------------------------------------------------

// X pass: row j of level b as one complex line z = Gamma + i rest.
template <class D, int NG>
__global__ void __launch_bounds__(D::TPF *NG, D::OCC / (D::TPF * NG))
    xpass_trial_kernel(const typename D::Real *__restrict__ gam, const typename D::Real *__restrict__ rest,
                       typename D::Real *__restrict__ t1, typename D::Real *__restrict__ t2, long long bs, int ld,
                       PlanT<typename D::Real> pl, int nrows) {
    using T = typename D::Real;
    using C = typename D::C;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    C *smem = reinterpret_cast<C *>(smem_raw);
    constexpr int TPF = D::TPF;
    const int M = pl.M;
    const int G = D::smem_len(M);
    const int g = threadIdx.x / TPF, t = threadIdx.x % TPF;
    C *buf = smem + g * G;
    double2 *wt = reinterpret_cast<double2 *>(smem_raw + scratch_offset<D>(M, NG)) + D::NWARP * g;
    const int b = blockIdx.y;
    const int j = blockIdx.x * NG + g + 1;
    const bool valid = j <= nrows;
    const long long row = b * bs + (long long)ld * (j - 1);
    if constexpr (D::MC > 0) {
        constexpr int NIT = (D::MC + 1 + TPF - 1) / TPF;
        T za[NIT], zb[NIT];
#pragma unroll
        for (int k = 0; k < NIT; ++k) {
            const int i = t + k * TPF;
            const bool ok = valid && i >= 1 && i < D::MC;
            za[k] = ok ? gam[row + i - 1] : (T)0;
            zb[k] = ok ? rest[row + i - 1] : (T)0;
        }
#pragma unroll
        for (int k = 0; k < NIT; ++k) {
            const int i = t + k * TPF;
            if (i <= D::MC) buf[D::idx(i)] = Cx<T>::make(za[k], zb[k]);
        }
    } else {
        for (int i = t; i <= M; i += TPF) {
            C z = Cx<T>::make(0, 0);
            if (valid && i >= 1 && i < M) z = Cx<T>::make(gam[row + i - 1], rest[row + i - 1]);
            buf[D::idx(i)] = z;
        }
    }
    __syncthreads();
    D::dst(buf, pl, t, wt);
    if (valid)
        for (int i = 1 + t; i < M; i += TPF) {
            const C y = buf[D::idx(i)];
            t1[row + i - 1] = y.x;
            t2[row + i - 1] = y.y;
        }
}

// Y pass: a block owns 2NG adjacent columns.  Phase 1 transforms each column's
// (S_x Gamma, S_x rest) pair as one complex line and combines
//   v = scale / Lambda_i * (S Gamma / Lambda_e + S rest)
//     = (S Gamma (1 - lam c) + S rest) * scale / (1 + lam c),   c = dt / (2 Re hc^2);
// phase 2 transforms the real v of two columns packed as one complex line (out may
// be t1: a block reads its columns whole before it stores them).
// Resident threads per SM the kernel is compiled for: 512 for FP32 lines of up to
// 512 points (at most 128 registers a thread), 256 otherwise.
template <class D>
constexpr int trial_occ() {
    return (sizeof(typename D::Real) == 4 && D::MC > 0 && D::MC <= 512) ? 512 : 256;
}
template <class D, int NG>
__global__ void __launch_bounds__(D::TPF *NG, trial_occ<D>() / (D::TPF * NG))
    ypass_trial_kernel(const typename D::Real *t1, const typename D::Real *__restrict__ t2, typename D::Real *out,
                       long long bs, int ncols, PlanT<typename D::Real> pl, const double *__restrict__ coef,
                       const double *__restrict__ cx, const double *__restrict__ cy, double scale) {
    using T = typename D::Real;
    using C = typename D::C;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    C *smem = reinterpret_cast<C *>(smem_raw);
    constexpr int TPF = D::TPF;
    constexpr int W = 2 * NG;
    const int M = pl.M;
    const int G = D::smem_len(M);
    const int g = threadIdx.x / TPF, t = threadIdx.x % TPF;
    double2 *wt = reinterpret_cast<double2 *>(smem_raw + scratch_offset<D>(M, W)) + D::NWARP * g;
    const int b = blockIdx.y;
    const int c0 = blockIdx.x * W;  // 0-based first column
    const T *s1 = t1 + b * bs, *s2 = t2 + b * bs;
    T *dst = out + b * bs;
    if constexpr (D::MC > 0) {
        constexpr int NT = NG * TPF;
        constexpr int NIT = (W * (D::MC + 1) + NT - 1) / NT;
        constexpr int CH = 8;
#pragma unroll
        for (int k0 = 0; k0 < NIT; k0 += CH) {
            T va[CH], vb[CH];
#pragma unroll
            for (int k = 0; k < CH; ++k) {
                const int e = threadIdx.x + (k0 + k) * NT;
                const int c = e % W, jj = e / W;
                const int col = c0 + c;
                const bool ok = k0 + k < NIT && jj >= 1 && jj < D::MC && col < ncols;
                const long long o = col + (long long)ncols * (jj - 1);
                va[k] = ok ? s1[o] : (T)0;
                vb[k] = ok ? s2[o] : (T)0;
            }
#pragma unroll
            for (int k = 0; k < CH; ++k) {
                const int e = threadIdx.x + (k0 + k) * NT;
                const int c = e % W, jj = e / W;
                if (k0 + k < NIT && jj <= D::MC) smem[c * G + D::idx(jj)] = Cx<T>::make(va[k], vb[k]);
            }
        }
    } else
    for (int e = threadIdx.x; e < W * (M + 1); e += blockDim.x) {
        const int c = e % W, jj = e / W;
        const int col = c0 + c;
        C z = Cx<T>::make(0, 0);
        if (jj >= 1 && jj < M && col < ncols) {
            const long long o = col + (long long)ncols * (jj - 1);
            z = Cx<T>::make(s1[o], s2[o]);
        }
        smem[c * G + D::idx(jj)] = z;
    }
    __syncthreads();
    const double cb = coef[b];
#pragma unroll 1
    for (int r = 0; r < 2; ++r) {
        const int c = r * NG + g;
        C *buf = smem + c * G;
        D::dst(buf, pl, t, wt);
        const int col1 = c0 + c + 1;  // 1-based column
        const bool ok = col1 <= ncols;
        const double cxv = ok ? __ldg(&cx[col1]) : 0.0;
        auto combine = [&](int jj, double cyj) {
            const C y = buf[D::idx(jj)];
            double v = 0.0;
            if (ok) {
                const double lam = -2 * ((cxv + cyj) - 2);
                v = ((double)y.x * (1 - lam * cb) + (double)y.y) * (scale * recip(1 + lam * cb));
            }
            buf[D::idx(jj)] = Cx<T>::make((T)v, 0);
        };
        if constexpr (D::MC > 0) {
            constexpr int NIT = (D::MC - 1 + TPF - 1) / TPF;
            double cyv[NIT];
#pragma unroll
            for (int k = 0; k < NIT; ++k) {
                const int jj = 1 + t + k * TPF;
                cyv[k] = jj < D::MC ? __ldg(&cy[jj]) : 0.0;
            }
#pragma unroll
            for (int k = 0; k < NIT; ++k) {
                const int jj = 1 + t + k * TPF;
                if (jj < D::MC) combine(jj, cyv[k]);
            }
        } else {
            for (int jj = 1 + t; jj < M; jj += TPF) combine(jj, __ldg(&cy[jj]));
        }
        __syncthreads();
    }
    // phase 2: pack columns (2g, 2g+1) into buffer 2g
    {
        C *ba = smem + (2 * g) * G;
        const C *bb = smem + (2 * g + 1) * G;
        for (int jj = 1 + t; jj < M; jj += TPF) ba[D::idx(jj)].y = bb[D::idx(jj)].x;
        __syncthreads();
        D::dst(ba, pl, t, wt);
    }
    for (int e = threadIdx.x; e < W * (M + 1); e += blockDim.x) {
        const int c = e % W, jj = e / W;
        const int col = c0 + c;
        if (jj >= 1 && jj < M && col < ncols) {
            const C y = smem[(c & ~1) * G + D::idx(jj)];
            dst[col + (long long)ncols * (jj - 1)] = (c & 1) ? y.y : y.x;
        }
    }
}

// ---------------------------------------------------------------------------
// Stencil kernels
// ---------------------------------------------------------------------------

// nonlinear (src/fluid.jl:441-455) = rot(direct_product(avg_flux(q + q0), Gamma, Gamma_bc)) / hc^2,
// with Gamma_bc = 0.25 get_bc(Gamma[:, lev+1]) (src/fluid.jl:473-483).  Batch b = level - 1.
template <class T, class TC = T>
struct NonlinArgs {
    const T *psi;         // ng x L: the flux q is its curl (with the coarser level's psi around it)
    const T *q;           // nq x L, read instead of psi by the FROMQ form
    const T *gam;         // ng x L
    T *out;               // ng x L (state.nonlin[1])
    const T *n2;          // ng x L (state.nonlin[2]); with rest != nullptr
    T *rest;              // ng x L: dt (1.5 N1 - 0.5 N2) + rhsbc, in the FP64 engine plus A Gamma, or nullptr
    const StepDev *prm;
    Grid g;
    // Ensembles of cases of one shape, stacked case-major (batch b = case L + level - 1):
    // per-case Reynolds numbers (null: g.Re) and callback values (prm[case] when set)
    const double *re_tab = nullptr;
    int prm_per_case = 0;
    // Fields that start at level lev0 (batch b is level lev0 + b % (L - lev0 + 1));
    // coarse (element type TC), when set, is the Gamma of level lev0 + 1 (a field
    // of another precision); otherwise a field's coarser level is the next batch.
    int lev0 = 1;
    const TC *coarse = nullptr;
    const TC *psi_coarse = nullptr;  // likewise psi of level lev0 + 1
};

// Tile of the nonlinear kernel: kNlTX x kNlTY circulation points per block of
// kNlTX x kNlBY threads (two rows of outputs per thread).
constexpr int kNlTX = 32, kNlTY = 16, kNlBY = 8;

// nonlinear (src/fluid.jl:340-455) fused with the rhs assembly of
// get_trial_state (src/fluid.jl:487-493), all levels (blockIdx.z) at once.
// The tile's faces, Gamma (with a one-point halo) and N2 are copied to shared
// memory with cp.async, all in flight at once; every face average Q = (q + q0)
// pair sum / 2 (avg_flux!) is then formed once per tile, and each flux product
// (direct_product_loops!) and the rot! difference from there, with the
// reference's expressions, so each value rounds exactly as in a direct
// evaluation.
// EXT: the ensemble / mixed-precision features of NonlinArgs (levels from lev0,
// per-case tables, a coarse field of another type); without them the kernel
// keeps the single-case code (fewer live registers, more resident blocks).
// The flux is formed from psi's tile, each face the difference curl! stores: one
// tile instead of two, and the steps keep no flux of their own (its curl, five 1024^2
// FP64 levels: 42 us and 84 MB written and read again).  The kernel is bound by
// instructions, 520 an output with an index division and bounds tests for every
// element of its tiles; inner tiles do without: five 1024^2 levels 86.6 us reading q,
// 75.8 psi, 53.0 with inner tiles by rows.  FROMQ reads q itself, for the
// first step after a caller set a q that is not psi's curl.
template <class T, class TC = T, bool EXT = false, bool FROMQ = false>
__global__ void __launch_bounds__(kNlTX *kNlBY, EXT ? 4 : 5) nonlinear_kernel(NonlinArgs<T, TC> a) {
    const Grid &g = a.g;
    const int nx = g.nx, ny = g.ny;
    const int b = blockIdx.z;
    int lev = b + 1, cs = 0;
    if constexpr (EXT) {
        const int nlev = g.L - a.lev0 + 1;
        lev = a.lev0 + b % nlev;
        cs = b / nlev;
    }
    // per-case values, formed where they are used (no register held across the kernel)
    auto prm_of = [&]() -> const StepDev * { return EXT ? a.prm + (a.prm_per_case ? cs : 0) : a.prm; };
    auto re_of = [&]() -> double { return (EXT && a.re_tab) ? a.re_tab[cs] : g.Re; };
    const int I0 = blockIdx.x * kNlTX, J0 = blockIdx.y * kNlTY;  // outputs I0+1..I0+TX, J0+1..J0+TY
    const long long nq = (long long)(nx + 1) * ny + (long long)nx * (ny + 1), ng = (long long)(nx - 1) * (ny - 1);
    const long long nu = (long long)(nx + 1) * ny;
    const T *q = FROMQ ? a.q + b * nq : a.psi + b * ng;
    const T *Gt = a.gam + b * ng;
    const TC *C = nullptr, *CP = nullptr;  // the coarser level's Gamma and psi
    if (lev < g.L) {
        if (EXT && a.coarse != nullptr) {
            C = a.coarse + cs * ng;
            if (!FROMQ) CP = a.psi_coarse + cs * ng;
        } else if constexpr (std::is_same<T, TC>::value) {
            C = a.gam + (b + 1) * ng;
            if (!FROMQ) CP = a.psi + (b + 1) * ng;
        }
    }
    __shared__ double aqy[kNlTY + 2][kNlTX];      // avg_qy(i, j), i = I0+2+x, j = J0+1+y
    __shared__ double aqx[kNlTY][kNlTX + 2];      // avg_qx(i, j), i = I0+1+x, j = J0+2+y
    __shared__ T gm[kNlTY + 2][kNlTX + 2];        // Gamma(i, j),  i = I0+x,   j = J0+y
    __shared__ T ru[FROMQ ? kNlTY + 1 : 1][FROMQ ? kNlTX + 2 : 1];  // q_u(i, j), i = I0+1+x, j = J0+1+y
    __shared__ T rv[FROMQ ? kNlTY + 2 : 1][FROMQ ? kNlTX + 1 : 1];  // q_v(i, j), i = I0+1+x, j = J0+1+y
    __shared__ T pm[FROMQ ? 1 : kNlTY + 2][FROMQ ? 1 : kNlTX + 2];  // psi(i, j), i = I0+x, j = J0+y
    __shared__ T rn[kNlTY][kNlTX];                // N2(i, j),     i = I0+1+x, j = J0+1+y
    const int tid = threadIdx.y * kNlTX + threadIdx.x;
    constexpr int NT = kNlTX * kNlBY;
    const double hc = gridstep(g, lev);
    // base_flux! of a static grid is U hc on every face (fluid.jl:22-32)
    const double sbx = prm_of()->fs[0] * hc, sby = prm_of()->fs[1] * hc;
    const bool moving = g.grid_moving;
    auto around = [&](int i, int j) -> double {  // psi on the domain's boundary, from the coarser level
        if (j == 0 || j == ny) return getbc(CP, g, j == 0 ? SIDE_B : SIDE_T, i + 1);
        return getbc(CP, g, i == 0 ? SIDE_L : SIDE_R, j + 1);
    };
    // A tile whose vertices all lie inside the grid (most of a large one) takes its
    // rows by warps, without an index division or a bounds test per element, and
    // two neighbouring output rows per thread, which share a flux product
    const bool inner = !FROMQ && I0 > 0 && J0 > 0 && I0 + kNlTX + 1 < nx && J0 + kNlTY + 1 < ny;
    const int tx = threadIdx.x, ty = threadIdx.y;
    if (inner) {
        const int at = (nx - 1) * (J0 - 1 + ty) + I0 - 1 + tx;  // Gamma(I0 + tx, J0 + ty)
#pragma unroll
        for (int k = 0; k < (kNlTY + 2 + kNlBY - 1) / kNlBY; ++k) {
            const int y = ty + k * kNlBY;
            if (y < kNlTY + 2) {
                cp_async_elem(&gm[y][tx], Gt + at + (nx - 1) * (k * kNlBY));
                cp_async_elem(&pm[FROMQ ? 0 : y][FROMQ ? 0 : tx], q + at + (nx - 1) * (k * kNlBY));
            }
        }
        if (tid < 2 * (kNlTY + 2)) {  // the two columns beyond the warp's width
            const int y = tid >> 1, x = kNlTX + (tid & 1), o = (nx - 1) * (J0 - 1 + y) + I0 - 1 + x;
            cp_async_elem(&gm[y][x], Gt + o);
            cp_async_elem(&pm[FROMQ ? 0 : y][FROMQ ? 0 : x], q + o);
        }
        if (a.rest) {
            const T *n2 = a.n2 + b * ng + at + nx;  // one row and one column on
#pragma unroll
            for (int k = 0; k < kNlTY / kNlBY; ++k)
                cp_async_elem(&rn[ty + k * kNlBY][tx], n2 + (nx - 1) * (k * kNlBY));
        }
    } else {
    // the tile's raw faces, Gamma and N2, all in flight at once (zeros outside the grid)
    if constexpr (FROMQ) {
#pragma unroll
        for (int e = tid; e < (kNlTY + 1) * (kNlTX + 2); e += NT) {
            const int x = e % (kNlTX + 2), y = e / (kNlTX + 2);
            const int i = I0 + 1 + x, j = J0 + 1 + y;
            if (i <= nx + 1 && j <= ny)
                cp_async_elem(&ru[y][x], q + UI(i, j));
            else
                ru[y][x] = T(0);
        }
#pragma unroll
        for (int e = tid; e < (kNlTY + 2) * (kNlTX + 1); e += NT) {
            const int x = e % (kNlTX + 1), y = e / (kNlTX + 1);
            const int i = I0 + 1 + x, j = J0 + 1 + y;
            if (i <= nx && j <= ny + 1)
                cp_async_elem(&rv[y][x], q + VI(i, j));
            else
                rv[y][x] = T(0);
        }
    }
#pragma unroll
    for (int e = tid; e < (kNlTY + 2) * (kNlTX + 2); e += NT) {
        const int x = e % (kNlTX + 2), y = e / (kNlTX + 2);
        const int i = I0 + x, j = J0 + y;
        if (i >= 1 && i <= nx - 1 && j >= 1 && j <= ny - 1) {
            cp_async_elem(&gm[y][x], Gt + GI(i, j));
            if constexpr (!FROMQ) cp_async_elem(&pm[y][x], q + GI(i, j));
        } else {
            gm[y][x] = T(0);
            // FP64: the coarser level's values around the field go into the tile; they
            // are not FP32 numbers, so FP32's edge tiles form them where they are used
            if constexpr (!FROMQ) pm[y][x] = sizeof(T) == 8 && i <= nx && j <= ny ? (T)around(i, j) : T(0);
        }
    }
    if (a.rest) {
#pragma unroll
        for (int e = tid; e < kNlTY * kNlTX; e += NT) {
            const int x = e % kNlTX, y = e / kNlTX;
            const int i = I0 + 1 + x, j = J0 + 1 + y;
            if (i <= nx - 1 && j <= ny - 1)
                cp_async_elem(&rn[y][x], a.n2 + b * ng + GI(i, j));
            else
                rn[y][x] = T(0);
        }
    }
    }
    cp_async_wait_all();
    __syncthreads();
    // the faces of the tile, i = I0+1+x, j = J0+1+y: read, or psi's differences
    // (curl!, fluid.jl:230-276; FP32's own subtraction rounds as the FP64 one cast)
    const bool edge = sizeof(T) == 4 && !inner;
    auto vertex = [&](int x, int y) -> double {  // psi(I0 + x, J0 + y)
        const int i = I0 + x, j = J0 + y;
        return i >= 1 && i <= nx - 1 && j >= 1 && j <= ny - 1 ? (double)pm[y][x] : around(i, j);
    };
    auto face_u = [&](int y, int x) -> double {
        if constexpr (FROMQ) return (double)ru[y][x];
        if (edge) return (double)(T)(vertex(x, y + 1) - vertex(x, y));
        return (double)(pm[y + 1][x] - pm[y][x]);
    };
    auto face_v = [&](int y, int x) -> double {
        if constexpr (FROMQ) return (double)rv[y][x];
        if (edge) return (double)(T)(vertex(x, y) - vertex(x + 1, y));
        return (double)(pm[y][x] - pm[y][x + 1]);
    };
    // face averages Q = (q + q0) pair sums / 2 (avg_flux!), each formed once per tile
    if (inner && !moving) {
        auto ay = [&](int y, int x) {
            aqy[y][x] = ((double)(pm[y][x + 1] - pm[y][x + 2]) + (double)(pm[y][x] - pm[y][x + 1]) + sby + sby) / 2;
        };
        auto ax = [&](int y, int x) {
            aqx[y][x] = ((double)(pm[y + 2][x] - pm[y + 1][x]) + (double)(pm[y + 1][x] - pm[y][x]) + sbx + sbx) / 2;
        };
        if constexpr (!FROMQ) {
#pragma unroll
            for (int k = 0; k < (kNlTY + 2 + kNlBY - 1) / kNlBY; ++k)
                if (ty + k * kNlBY < kNlTY + 2) ay(ty + k * kNlBY, tx);
#pragma unroll
            for (int k = 0; k < kNlTY / kNlBY; ++k) ax(ty + k * kNlBY, tx);
            if (tid < 2 * kNlTY) ax(tid >> 1, kNlTX + (tid & 1));
        }
    } else {
#pragma unroll
    for (int e = tid; e < (kNlTY + 2) * kNlTX; e += NT) {
        const int x = e % kNlTX, y = e / kNlTX;
        const int i = I0 + 2 + x, j = J0 + 1 + y;
        double v = 0.0;
        if (i <= nx && j <= ny + 1) {
            // q_v(i, j) and q_v(i - 1, j)
            if (moving)
                v = (face_v(y, x + 1) + face_v(y, x) + base_flux_y(g, prm_of(), lev, i, j) +
                     base_flux_y(g, prm_of(), lev, i - 1, j)) / 2;
            else
                v = (face_v(y, x + 1) + face_v(y, x) + sby + sby) / 2;
        }
        aqy[y][x] = v;
    }
#pragma unroll
    for (int e = tid; e < kNlTY * (kNlTX + 2); e += NT) {
        const int x = e % (kNlTX + 2), y = e / (kNlTX + 2);
        const int i = I0 + 1 + x, j = J0 + 2 + y;
        double v = 0.0;
        if (i <= nx + 1 && j <= ny) {
            // q_u(i, j) and q_u(i, j - 1)
            if (moving)
                v = (face_u(y + 1, x) + face_u(y, x) + base_flux_x(g, prm_of(), lev, i, j) +
                     base_flux_x(g, prm_of(), lev, i, j - 1)) / 2;
            else
                v = (face_u(y + 1, x) + face_u(y, x) + sbx + sbx) / 2;
        }
        aqx[y][x] = v;
    }
    }
    __syncthreads();
    // the FP64 engine's results of an inner tile; the FP32 one keeps the general form
    // below, whose multiply-adds are contracted in one fixed way (its results are
    // reproducible bit for bit)
    if constexpr (sizeof(T) == 8 && std::is_same<T, TC>::value && !FROMQ) {
        if (inner) {
            auto fx = [&](int yj) { return (aqy[yj][tx] * gm[yj][tx + 1] + aqy[yj - 1][tx] * gm[yj - 1][tx + 1]) / 2; };
            auto fy = [&](int xi, int y) { return -(aqx[y][xi] * gm[y + 1][xi] + aqx[y][xi - 1] * gm[y + 1][xi - 1]) / 2; };
            const double ih2 = 1 / (hc * hc);
            const double cg = a.rest ? 0.5 * (g.dt / (re_of() * (hc * hc))) : 0.0;
            static_assert(kNlTY == 2 * kNlBY, "two output rows a thread");
            const int y0 = 2 * ty;
            const long long o = b * ng + GI(I0 + 1 + tx, J0 + 1 + y0);
            double f0 = fx(y0 + 1);
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                const int y = y0 + k;
                const double f1 = fx(y + 2);
                const double r = (f0 - f1) + (fy(tx + 2, y) - fy(tx + 1, y));
                f0 = f1;
                const double n1 = r * ih2;
                a.out[o + k * (nx - 1)] = (T)n1;
                if (a.rest) {
                    double v = (g.dt * 1.5) * n1 + (g.dt * -0.5) * (double)rn[y][tx];
                    const double gc = gm[y + 1][tx + 1];  // + A Gamma, see below
                    const double lap = (gm[y + 1][tx] + gm[y + 1][tx + 2] - 2 * gc) + (gm[y][tx + 1] + gm[y + 2][tx + 1] - 2 * gc);
                    v += gc + cg * lap;
                    a.rest[o + k * (nx - 1)] = (T)v;
                }
            }
            return;
        }
    }
    const int x = threadIdx.x, I = I0 + 1 + x;
    if (I > nx - 1) return;
    // x-flux product at (I+1, j) (direct_product_loops!, fluid.jl:396-415)
    auto fqx = [&](int j) -> double {
        const int i = I + 1, yj = j - J0;
        if (j == 1) return (aqy[yj][x] * gm[yj][x + 1] + aqy[yj - 1][x] * (getbc(C, g, SIDE_B, i) * 0.25)) / 2;
        if (j == ny) return (aqy[yj - 1][x] * gm[yj - 1][x + 1] + aqy[yj][x] * (getbc(C, g, SIDE_T, i) * 0.25)) / 2;
        return (aqy[yj][x] * gm[yj][x + 1] + aqy[yj - 1][x] * gm[yj - 1][x + 1]) / 2;
    };
    // y-flux product at (i, J+1), i in {I, I+1} (fluid.jl:417-436)
    auto fqy = [&](int i, int y) -> double {
        const int xi = i - I0;  // aqx column of avg_qx(i, .) is xi - 1, gm column of Gamma(i, .) is xi
        if (i == 1) return -(aqx[y][xi] * gm[y + 1][xi] + aqx[y][xi - 1] * (getbc(C, g, SIDE_L, J0 + 2 + y) * 0.25)) / 2;
        if (i == nx)
            return -(aqx[y][xi - 1] * gm[y + 1][xi - 1] + aqx[y][xi] * (getbc(C, g, SIDE_R, J0 + 2 + y) * 0.25)) / 2;
        return -(aqx[y][xi] * gm[y + 1][xi] + aqx[y][xi - 1] * gm[y + 1][xi - 1]) / 2;
    };
#pragma unroll
    for (int k = 0; k < kNlTY / kNlBY; ++k) {
        const int y = threadIdx.y + k * kNlBY, J = J0 + 1 + y;
        if (J > ny - 1) break;
        // rot! at Gamma(I, J) with i = I+1, j = J+1 (fluid.jl:106-108)
        const double r = (fqx(J) - fqx(J + 1)) + (fqy(I + 1, y) - fqy(I, y));
        const double n1 = r * (1 / (hc * hc));
        a.out[b * ng + GI(I, J)] = (T)n1;
        if (a.rest) {
            // rest = dt b1 N1 + dt b2 N2 + rhsbc (fluid.jl:487-493), rhsbc = apply_bc!(0, get_bc(..); fac)
            double v = (g.dt * 1.5) * n1 + (g.dt * -0.5) * (double)rn[y][x];
            if constexpr (sizeof(T) == 8 && std::is_same<T, TC>::value) {
                // + A Gamma.  A = 1 - c (-Laplacian), diagonal under the 2D DST, is this
                // five-point stencil with zeros beyond the field: taking it here spares
                // the trial solve a second field through its passes
                const double gc = gm[y + 1][x + 1];
                const double lap = (gm[y + 1][x] + gm[y + 1][x + 2] - 2 * gc) + (gm[y][x + 1] + gm[y + 2][x + 1] - 2 * gc);
                v += gc + 0.5 * (g.dt / (re_of() * (hc * hc))) * lap;
            }
            if (lev < g.L && on_ring(g, I, J)) {
                const double fac = 0.25 * g.dt / (re_of() * (hc * hc));
                v = v + apply_bc_at(0.0, C, g, I, J, fac);
            }
            a.rest[b * ng + GI(I, J)] = (T)v;
        }
    }
}

// 4-argument curl! (src/fluid.jl:230-276) with psi_bc = get_bc(psi_coarse) (zero if null).
// One thread per (i, j) writes both faces there: the x face u(i, j) (i <= nx+1,
// j <= ny) and the y face v(i, j) (i <= nx, j <= ny+1); inside the ring they share
// psi(i-1, j-1).  Batch b (blockIdx.z) uses psi + b*bs, q + b*qbs, coarse + b*cbs;
// with nl > 1 batch b is level b % nl + 1 of nl levels, whose coarsest has no
// coarser field.
// win (device, may be null): only the faces in i0..i1 x j0..j1 are written, by a
// grid of any size sweeping the window.
// differs (CHECK form): set to 1 if q holds anything else than those faces.
template <class T, class TP, class TC, bool CHECK = false>
__global__ void curl_kernel(T *__restrict__ qout, long long qbs, const TP *__restrict__ psi, long long bs,
                            const TC *__restrict__ coarse, long long cbs, Grid g, const int *__restrict__ win = nullptr,
                            int nl = 1, int *differs = nullptr) {
    overlap_begin();
    const int nx = g.nx, ny = g.ny;
    const long long nu = (long long)(nx + 1) * ny;
    const int b = blockIdx.z;
    const TP *Pt = psi + b * bs;
    const TC *C = coarse && (nl == 1 || (b + 1) % nl != 0) ? coarse + b * cbs : nullptr;
    T *q = qout + b * qbs;
    auto P = [&](long long k) -> double { return (double)Pt[k]; };
    auto put = [&](long long k, double v) {
        if constexpr (CHECK) {
            if (!(q[k] == (T)v)) *differs = 1;
        } else {
            q[k] = (T)v;
        }
    };
    auto face = [&](int i, int j) {
        if (i >= 2 && i <= nx - 1 && j >= 2 && j <= ny - 1) {
            const double pc = P(GI(i - 1, j - 1));
            put(UI(i, j), P(GI(i - 1, j)) - pc);
            put(VI(i, j), pc - P(GI(i, j - 1)));
            return;
        }
        if (j <= ny) {
            double v;
            if (i == 1)
                v = getbc(C, g, SIDE_L, j + 1) - getbc(C, g, SIDE_L, j);
            else if (i == nx + 1)
                v = getbc(C, g, SIDE_R, j + 1) - getbc(C, g, SIDE_R, j);
            else if (j == 1)
                v = P(GI(i - 1, 1)) - getbc(C, g, SIDE_B, i);
            else if (j == ny)
                v = getbc(C, g, SIDE_T, i) - P(GI(i - 1, ny - 1));
            else
                v = P(GI(i - 1, j)) - P(GI(i - 1, j - 1));
            put(UI(i, j), v);
        }
        if (i <= nx) {
            double v;
            if (j == 1)
                v = getbc(C, g, SIDE_B, i) - getbc(C, g, SIDE_B, i + 1);
            else if (j == ny + 1)
                v = getbc(C, g, SIDE_T, i) - getbc(C, g, SIDE_T, i + 1);
            else if (i == 1)
                v = getbc(C, g, SIDE_L, j) - P(GI(1, j - 1));
            else if (i == nx)
                v = P(GI(nx - 1, j - 1)) - getbc(C, g, SIDE_R, j);
            else
                v = P(GI(i - 1, j - 1)) - P(GI(i, j - 1));
            put(VI(i, j), v);
        }
    };
    const int ti = blockIdx.x * blockDim.x + threadIdx.x, tj = blockIdx.y * blockDim.y + threadIdx.y;
    if (win == nullptr) {
        if (ti + 1 <= nx + 1 && tj + 1 <= ny + 1) face(ti + 1, tj + 1);
        return;
    }
    // the window (known on the device only) in grid-strided sweeps of a smaller grid
    const int i1 = min(win[1], nx + 1), j1 = min(win[3], ny + 1);
    for (int j = max(win[2], 1) + tj; j <= j1; j += gridDim.y * blockDim.y)
        for (int i = max(win[0], 1) + ti; i <= i1; i += gridDim.x * blockDim.x) face(i, j);
}

// coarsify! (src/fluid.jl:208-228): fine level -> central block of the next coarser level
// (the fine level may be of another element type TF).
// fine_central: the fine level is zero outside its own central block (faces
// nx/4+1 .. 3nx/4-1 by ny/4+1 .. 3ny/4-1); stencils wholly outside it give zero
// without a load.
template <class T, class TF = T>
__global__ void coarsify_kernel(T *__restrict__ coarse, const TF *__restrict__ fine, long long bs, Grid g,
                                int fine_central = 0) {
    overlap_begin();
    const int nx = g.nx, ny = g.ny;
    const int ni = (nx / 2 - 2 - (-nx / 2 + 2)) / 2 + 1, nic = (nx / 4 - 1) - (-nx / 4 + 1) + 1;
    const int nj = (ny / 2 - 2 - (-ny / 2 + 2)) / 2 + 1, njc = (ny / 4 - 1) - (-ny / 4 + 1) + 1;
    const int ci = ni < nic ? ni : nic, cj = nj < njc ? nj : njc;
    const int a = blockIdx.x * blockDim.x + threadIdx.x, bb = blockIdx.y * blockDim.y + threadIdx.y;
    if (a >= ci || bb >= cj) return;
    const TF *Gf = fine + blockIdx.z * bs;
    T *Gc = coarse + blockIdx.z * bs;
    auto G = [&](long long k) -> double { return (double)Gf[k]; };
    const int i = nx / 2 + (-nx / 2 + 2) + 2 * a, ic = nx / 2 + (-nx / 4 + 1) + a;
    const int j = ny / 2 + (-ny / 2 + 2) + 2 * bb, jc = ny / 2 + (-ny / 4 + 1) + bb;
    if (fine_central && (i + 1 < nx / 4 + 1 || i - 1 > 3 * nx / 4 - 1 || j + 1 < ny / 4 + 1 || j - 1 > 3 * ny / 4 - 1)) {
        Gc[GI(ic, jc)] = (T)0.0;
        return;
    }
    Gc[GI(ic, jc)] = (T)(G(GI(i, j)) + 0.5 * (G(GI(i + 1, j)) + G(GI(i, j + 1)) + G(GI(i - 1, j)) + G(GI(i, j - 1))) +
                         0.25 * (G(GI(i + 1, j + 1)) + G(GI(i + 1, j - 1)) + G(GI(i - 1, j - 1)) + G(GI(i - 1, j + 1))));
}

// x = Binv z for the precomputed B^-1 (src/coupling.jl:187-192), column-major n x n.
// Grid (ceil(n/64), ceil(n/64)); partial sums part[chunk * n + row], summed in
// chunk order by binv_reduce_kernel (deterministic).
static __global__ void __launch_bounds__(256) binv_gemv_kernel(const double *__restrict__ A, const double *__restrict__ z,
                                                        double *__restrict__ part, int n) {
    __shared__ double red[4][64];
    const int r = threadIdx.x % 64, s = threadIdx.x / 64;
    const int row = blockIdx.x * 64 + r;
    const int cbeg = blockIdx.y * 64;
    double acc = 0.0;
    if (row < n) {
        if (cbeg + 64 <= n) {
#pragma unroll
            for (int c = cbeg + s; c < cbeg + 64; c += 4) acc += A[row + (long long)n * c] * __ldg(&z[c]);
        } else {
            for (int c = cbeg + s; c < n; c += 4) acc += A[row + (long long)n * c] * __ldg(&z[c]);
        }
    }
    red[s][r] = acc;
    __syncthreads();
    if (s == 0 && row < n) part[(long long)blockIdx.y * n + row] = ((red[0][r] + red[1][r]) + red[2][r]) + red[3][r];
}

// binv_gemv_kernel for the cases of a batched ensemble group (case = blockIdx.z,
// grid sized for the largest case): x = Binv Ftmp of each case into its partials.
static __global__ void __launch_bounds__(256) binv_gemv_multi_kernel(const CaseView *__restrict__ tab) {
    __shared__ double red[4][64];
    const CaseView &cv = tab[blockIdx.z];
    const int n = 2 * cv.P.np;
    const int nchunk = (n + 63) / 64;
    if ((int)blockIdx.x >= nchunk || (int)blockIdx.y >= nchunk) return;  // uniform over the block
    const double *__restrict__ A = cv.Binv;
    const double *__restrict__ z = cv.Ftmp;
    const int r = threadIdx.x % 64, s = threadIdx.x / 64;
    const int row = blockIdx.x * 64 + r;
    const int cbeg = blockIdx.y * 64;
    double acc = 0.0;
    if (row < n) {
        if (cbeg + 64 <= n) {
#pragma unroll
            for (int c = cbeg + s; c < cbeg + 64; c += 4) acc += A[row + (long long)n * c] * __ldg(&z[c]);
        } else {
            for (int c = cbeg + s; c < n; c += 4) acc += A[row + (long long)n * c] * __ldg(&z[c]);
        }
    }
    red[s][r] = acc;
    __syncthreads();
    if (s == 0 && row < n) cv.part[(long long)blockIdx.y * n + row] = ((red[0][r] + red[1][r]) + red[2][r]) + red[3][r];
}

// F~b = sum of the chunk partials; update_vars! fb = F~b h / dt (problem.jl:676-685);
// total force sum over panels (problem.jl:853-856).  One block.
static __global__ void binv_reduce_kernel(const double *__restrict__ part, int nchunk, int n, double *__restrict__ fbt,
                                   double *__restrict__ fb, double *__restrict__ total, double h, double dt,
                                   int from_part) {
    __shared__ double sx[32], sy[32];
    const int np = n / 2;
    double tx = 0.0, ty = 0.0;
    for (int k = threadIdx.x; k < n; k += blockDim.x) {
        double v;
        if (from_part) {
            v = 0.0;
#pragma unroll 8
            for (int c = 0; c < nchunk; ++c) v += part[(long long)c * n + k];
            fbt[k] = v;
        } else {
            v = fbt[k];
        }
        const double f = v * h / dt;
        fb[k] = f;
        if (k < np)
            tx += f;
        else
            ty += f;
    }
    for (int o = 16; o > 0; o >>= 1) {
        tx += __shfl_xor_sync(0xffffffffu, tx, o);
        ty += __shfl_xor_sync(0xffffffffu, ty, o);
    }
    if ((threadIdx.x & 31) == 0) {
        sx[threadIdx.x >> 5] = tx;
        sy[threadIdx.x >> 5] = ty;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double ax = 0.0, ay = 0.0;
        for (int k = 0; k < (int)(blockDim.x >> 5); ++k) {
            ax += sx[k];
            ay += sy[k];
        }
        total[0] = ax;
        total[1] = ay;
    }
}

// binv_reduce_kernel for the cases of a batched ensemble group: one block per case.
static __global__ void binv_reduce_multi_kernel(const CaseView *__restrict__ tab, double h, double dt) {
    __shared__ double sx[32], sy[32];
    const CaseView &cv = tab[blockIdx.x];
    const int n = 2 * cv.P.np, np = n / 2, nchunk = (n + 63) / 64;
    double tx = 0.0, ty = 0.0;
    for (int k = threadIdx.x; k < n; k += blockDim.x) {
        double v = 0.0;
#pragma unroll 8
        for (int c = 0; c < nchunk; ++c) v += cv.part[(long long)c * n + k];
        cv.Fbt[k] = v;
        const double f = v * h / dt;
        cv.fb[k] = f;
        if (k < np)
            tx += f;
        else
            ty += f;
    }
    for (int o = 16; o > 0; o >>= 1) {
        tx += __shfl_xor_sync(0xffffffffu, tx, o);
        ty += __shfl_xor_sync(0xffffffffu, ty, o);
    }
    if ((threadIdx.x & 31) == 0) {
        sx[threadIdx.x >> 5] = tx;
        sy[threadIdx.x >> 5] = ty;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double ax = 0.0, ay = 0.0;
        for (int k = 0; k < (int)(blockDim.x >> 5); ++k) {
            ax += sx[k];
            ay += sy[k];
        }
        cv.total[0] = ax;
        cv.total[1] = ay;
    }
}

// Gauss-Jordan inversion without pivoting of a positive definite matrix (stands
// in for LinearAlgebra.inv at src/coupling.jl:190).  Element (a, b) after step k
// of S: the pivot row scaled by 1/p, the pivot column by -1/p, the pivot by 1/p,
// every other element S[a,b] - S[a,k] (S[k,b] / p).
__device__ __forceinline__ double gj_elem(const double *__restrict__ S, int n, int k, int a, int b) {
    const double p = S[k + (long long)n * k];
    if (a == k && b == k) return 1.0 / p;
    if (a == k) return S[k + (long long)n * b] / p;
    if (b == k) return -S[a + (long long)n * k] / p;
    return S[a + (long long)n * b] - S[a + (long long)n * k] * (S[k + (long long)n * b] / p);
}
// Steps k and k+1 in one launch, from S into D (ping-pong buffers, so no element
// is read after another thread overwrote it): the step-(k+1) expression applied
// to the step-k elements gj_elem forms, the same values bit for bit as two
// one-step launches.  A pivot <= 0 sets *err to its step + 1.
static __global__ void gj_step2_kernel(const double *__restrict__ S, double *__restrict__ D, int n, int k, int *err) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y;
    if (i >= n) return;
    const int k1 = k + 1;
    const double q = gj_elem(S, n, k, k1, k1);
    if (i == 0 && j == 0) {
        if (!(S[k + (long long)n * k] > 0.0))
            atomicCAS(err, 0, k + 1);
        else if (!(q > 0.0))
            atomicCAS(err, 0, k1 + 1);
    }
    const double rk = gj_elem(S, n, k, k1, j) / q;
    const double ck = gj_elem(S, n, k, i, k1);
    double v;
    if (i == k1 && j == k1)
        v = 1.0 / q;
    else if (i == k1)
        v = rk;
    else if (j == k1)
        v = -ck / q;
    else
        v = gj_elem(S, n, k, i, j) - ck * rk;
    D[i + (long long)n * j] = v;
}

// Steps k .. k + b - 1 (b <= kGJB) of the same elimination in one launch, as one
// block pivot: with K = {k .. k + b - 1}, P = S_KK^-1 (formed here by b
// unpivoted steps on the b x b block),
//   D_KK = P, D_KR = P S_KR, D_RK = -S_RK P, D_RR = S_RR - S_RK P S_KR,
// which equals the b single steps in exact arithmetic (not bit for bit).  One
// block per column j, threads over rows i (n <= blockDim.x * gridDim.x).  A
// pivot <= 0 sets *err to its step + 1.
constexpr int kGJB = 16;  // steps per block-pivot launch (blockDim >= kGJB^2)
static __global__ void gj_block_kernel(const double *__restrict__ S, double *__restrict__ D, int n, int k, int b,
                                       int *err) {
    __shared__ double Pm[kGJB][kGJB];
    __shared__ double T[kGJB];  // P S_Kj for this block's column j
    const int j = blockIdx.y, t = threadIdx.x;
    constexpr int kE = kGJB * kGJB;
    if (t < kE) {
        const int a = t / kGJB, c = t % kGJB;
        Pm[a][c] = (a < b && c < b) ? S[(k + a) + (long long)n * (k + c)] : 0.0;
    }
    __syncthreads();
    // in-place unpivoted Gauss-Jordan of the b x b block, thread t < kGJB^2 owning (t / kGJB, t % kGJB)
    const int a = t / kGJB, c = t % kGJB;
    for (int q = 0; q < b; ++q) {
        double p = 0.0, aq = 0.0, qc = 0.0, ac = 0.0;
        if (t < kE) {
            p = Pm[q][q];
            aq = Pm[a][q];
            qc = Pm[q][c];
            ac = Pm[a][c];
        }
        __syncthreads();
        if (t == 0 && blockIdx.x == 0 && j == 0 && !(p > 0.0)) atomicCAS(err, 0, k + q + 1);
        if (t < kE && a < b && c < b) {
            const double ip = 1.0 / p;
            if (a == q && c == q)
                Pm[a][c] = ip;
            else if (a == q)
                Pm[a][c] = qc * ip;
            else if (c == q)
                Pm[a][c] = -aq * ip;
            else
                Pm[a][c] = ac - aq * (qc * ip);
        }
        __syncthreads();
    }
    const bool jk = j >= k && j < k + b;
    if (t < b) {
        double v = 0.0;
        if (!jk)
            for (int e = 0; e < b; ++e) v += Pm[t][e] * S[(k + e) + (long long)n * j];
        T[t] = v;
    }
    __syncthreads();
    const int i = blockIdx.x * blockDim.x + t;
    if (i >= n) return;
    const bool ik = i >= k && i < k + b;
    double v;
    if (ik && jk) {
        v = Pm[i - k][j - k];
    } else if (ik) {
        v = T[i - k];
    } else if (jk) {
        v = 0.0;
        for (int e = 0; e < b; ++e) v -= S[i + (long long)n * (k + e)] * Pm[e][j - k];
    } else {
        v = S[i + (long long)n * j];
        for (int e = 0; e < b; ++e) v -= S[i + (long long)n * (k + e)] * T[e];
    }
    D[i + (long long)n * j] = v;
}

// M <- (M + M^T) / 2 in place (n x n, column-major): thread (i, j) with i < j
// owns both entries of its pair.
static __global__ void symmetrize_kernel(double *__restrict__ M, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y;
    if (i >= j || j >= n) return;
    const double a = M[i + (long long)n * j], b = M[j + (long long)n * i];
    const double v = 0.5 * (a + b);
    M[i + (long long)n * j] = v;
    M[j + (long long)n * i] = v;
}

// Identity columns [c0, c0+nb) of a 2np-length basis, one per batch.
static __global__ void unit_columns_kernel(double *__restrict__ f, int n, int c0, int nb) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n * nb) return;
    const int b = t / n, k = t % n;
    f[t] = (k == c0 + b) ? 1.0 : 0.0;
}

}  // namespace ibpm
