// Geodesic backtraces of the tables (Radiation::UpdateFourierCoefficients,
// src/Radiation.cpp:191-237): one thread per (interior cell, streaming
// direction) runs the reference's backward Fehlberg RK45.  FP64 with
// contracted multiply-adds; the coefficients agree with the reference's to
// rounding (its step-size control calls libm's pow, which is not correctly
// rounded, so they are not bit-identical in any case).
//
// Every stage interpolates 21 metric fields between 4 nodes and evaluates the
// right-hand side.  What bounds it, at 400^2 cells x 16 directions and
// tolerance 1e-10 (35.3 M trials of 6 stages):
//   - arithmetic: the right-hand side is contracted over the velocity before
//     the metric is applied (about 50 FP64 instructions against 277 term by
//     term), and a field takes one product and three multiply-adds with the
//     corner weights;
//   - L1: a block takes a run of cells of one row and keeps the 3 rows of
//     nodes around it in shared memory, where nodes are 22 doubles apart (their
//     16-byte reads hit disjoint banks; in global memory, 256 bytes apart,
//     every distinct node of a warp's read was a cache line of its own).
// A point outside those rows (more than a cell away from its own) reads
// global memory.
#include <algorithm>

#include "device_common.cuh"

namespace grlbm
{
namespace
{
constexpr int kFields = 22; // doubles read per node: the 21 fields and the pad
static_assert(kFields == RF_DG222 + 2 && kFields % 2 == 0, "whole 16-byte pairs");
constexpr int kThreads = 128, kMaxCells = 32;

// The excision test and node coordinates, rounded as everywhere else.
__device__ __forceinline__ bool inside_bh(const GridDev &g, double x, double y)
{
    return g.kind != 0 && __dadd_rn(__dmul_rn(x, x), __dmul_rn(y, y)) <= g.excision2;
}

// num / den, correctly rounded, from r = RN(1 / den) and den in [1, 2): one
// refinement and one Markstein step (P. Markstein, IBM J. Res. Dev. 34(1), 1990).
__device__ __forceinline__ double quotient(double num, double den, double r)
{
    double q = num * r;
    q = __fma_rn(__fma_rn(-q, den, num), r, q);
    return __fma_rn(__fma_rn(-q, den, num), r, q);
}

// What a thread needs of the grid: the spacings scaled into [1, 2) by a power
// of two (exactly), their reciprocals, and the block's staged nodes.
struct Local
{
    int px0, py0, pnx; // nodes [px0, px0 + pnx) x [py0, py0 + 3) in shared memory, kFields doubles each
    double sx, dx, rx, sy, dy, ry; // scale, scaled spacing, its reciprocal
};

// The grid square of a point and its place in it; false outside the domain.
__device__ __forceinline__ bool locate(const GridDev &g, const Local &l, double x, double y, int &i0, int &j0,
                                       double &tx, double &ty)
{
    const double fi = quotient((x - g.startx) * l.sx, l.dx, l.rx), fj = quotient((y - g.starty) * l.sy, l.dy, l.ry);
    i0 = __double2int_rd(fi);
    j0 = __double2int_rd(fj);
    const int nx = (int)g.nx, ny = (int)g.ny;
    if ((unsigned)i0 > (unsigned)(nx - 3) || (unsigned)j0 > (unsigned)(ny - 3))
    {
        if (!(x >= g.startx && x <= g.endx && y >= g.starty && y <= g.endy))
            return false;
        // a point exactly on the boundary keeps its corners on the grid
        i0 = min(max(i0, 0), nx - 2);
        j0 = min(max(j0, 0), ny - 2);
    }
    tx = fi - (double)i0;
    ty = fj - (double)j0;
    return true;
}

// Bilinear interpolation of the packed metric fields, with the flat-space
// values outside the domain (src/Metric.cpp:338-348, 584-780).
__device__ __forceinline__ void fields_at(const GridDev &g, const double *__restrict__ rkf, const Local &l, double x,
                                          double y, double (&v)[kFields])
{
    int i0, j0;
    double tx, ty;
    if (!locate(g, l, x, y, i0, j0, tx, ty))
    {
#pragma unroll
        for (int f = 0; f < kFields; f++)
            v[f] = 0.0;
        v[RF_ALPHA] = v[RF_GU11] = v[RF_GU22] = 1.0;
        return;
    }
    const int ci = i0 - l.px0, cj = j0 - l.py0;
    const bool staged = (unsigned)ci < (unsigned)(l.pnx - 1) && (unsigned)cj < 2u;
    const double sx = 1.0 - tx, sy = 1.0 - ty;
    const double w00 = sx * sy, w10 = tx * sy, w01 = sx * ty, w11 = tx * ty;
    auto gather = [&](const double *p00, int step, int64_t row) {
        const double *p10 = p00 + step, *p01 = p00 + row * step, *p11 = p01 + step;
#pragma unroll
        for (int f = 0; f < kFields; f += 2) // in pairs (16-byte loads)
        {
            const double2 a = *reinterpret_cast<const double2 *>(p00 + f), b = *reinterpret_cast<const double2 *>(p10 + f);
            const double2 c = *reinterpret_cast<const double2 *>(p01 + f), d = *reinterpret_cast<const double2 *>(p11 + f);
            v[f] = fma(d.x, w11, fma(c.x, w01, fma(b.x, w10, a.x * w00)));
            v[f + 1] = fma(d.y, w11, fma(c.y, w01, fma(b.y, w10, a.y * w00)));
        }
    };
    extern __shared__ __align__(16) double patch[];
    if (staged)
        gather(patch + (ci + cj * l.pnx) * kFields, kFields, l.pnx);
    else
        gather(rkf + ((int64_t)i0 + (int64_t)j0 * g.nx) * kRkStride, kRkStride, g.nx);
}

// 2x2 spatial block of the (inverse) tetrad at a coordinate; identity outside.
__device__ __forceinline__ void tetrad_block(const GridDev &g, const double *__restrict__ rkf, const Local &l, double x,
                                             double y, int first, double &a11, double &a12, double &a21, double &a22)
{
    int i0, j0;
    double tx, ty;
    a11 = a22 = 1.0;
    a12 = a21 = 0.0;
    if (!locate(g, l, x, y, i0, j0, tx, ty))
        return;
    const double *p00 = rkf + ((int64_t)i0 + (int64_t)j0 * g.nx) * kRkStride + first;
    const double *p10 = p00 + kRkStride, *p01 = p00 + g.nx * kRkStride, *p11 = p01 + kRkStride;
    double v[4];
#pragma unroll
    for (int f = 0; f < 4; f++)
    {
        const double f0 = __ldg(p00 + f) * (1.0 - tx) + __ldg(p10 + f) * tx;
        const double f1 = __ldg(p01 + f) * (1.0 - tx) + __ldg(p11 + f) * tx;
        v[f] = f0 * (1.0 - ty) + f1 * ty;
    }
    a11 = v[0], a12 = v[1], a21 = v[2], a22 = v[3];
}

struct RkState
{
    double x1, x2, v1, v2, nu;
};

// One stage: the 3+1 geodesic right-hand side of Vincent, Gourgoulhon & Novak
// (2012) as the reference has it (src/GeodesicEquationSolver.cpp:5-55),
//   dx_k = alpha v_k - beta_k,   dnu = nu (alpha K_ij v_i v_j - v_i d_i alpha),
//   dv_k = v_k (v_i d_i alpha - alpha K_ij v_i v_j) - v_i d_i beta_k
//        + gamma^kl (2 alpha K_lj v_j - d_l alpha - alpha T_l / 2),
//   T_l  = (d_i gamma_lj + d_j gamma_il - d_l gamma_ij) v_i v_j
//        = 2 v_i (d_i gamma v)_l - v (d_l gamma v).
__device__ __forceinline__ RkState stage(const GridDev &g, const double *__restrict__ rkf, const Local &l,
                                         const RkState &s)
{
    double f[kFields];
    fields_at(g, rkf, l, s.x1, s.x2, f);
    const double al = f[RF_ALPHA], v1 = s.v1, v2 = s.v2;
    const double kv1 = f[RF_K11] * v1 + f[RF_K12] * v2, kv2 = f[RF_K12] * v1 + f[RF_K22] * v2;
    const double a1 = f[RF_DG111] * v1 + f[RF_DG112] * v2, a2 = f[RF_DG112] * v1 + f[RF_DG122] * v2; // d_1 gamma v
    const double b1 = f[RF_DG211] * v1 + f[RF_DG212] * v2, b2 = f[RF_DG212] * v1 + f[RF_DG222] * v2; // d_2 gamma v
    const double t1 = 2.0 * (v1 * a1 + v2 * b1) - (v1 * a1 + v2 * a2);
    const double t2 = 2.0 * (v1 * a2 + v2 * b2) - (v1 * b1 + v2 * b2);
    const double p = al * (v1 * kv1 + v2 * kv2) - (v1 * f[RF_DA1] + v2 * f[RF_DA2]);
    const double w1 = al * (2.0 * kv1 - 0.5 * t1) - f[RF_DA1], w2 = al * (2.0 * kv2 - 0.5 * t2) - f[RF_DA2];
    RkState k;
    k.x1 = al * v1 - f[RF_B1];
    k.x2 = al * v2 - f[RF_B2];
    k.v1 = f[RF_GU11] * w1 + f[RF_GU12] * w2 - v1 * p - (v1 * f[RF_DB11] + v2 * f[RF_DB21]);
    k.v2 = f[RF_GU12] * w1 + f[RF_GU22] * w2 - v2 * p - (v1 * f[RF_DB12] + v2 * f[RF_DB22]);
    k.nu = p * s.nu;
    return k;
}

// y + s (sum of c_i k_i), component by component
#define GRLBM_EACH(out, expr)                                                                                 \
    do                                                                                                         \
    {                                                                                                          \
        out.x1 = y0.x1 + s * (expr(x1));                                                                       \
        out.x2 = y0.x2 + s * (expr(x2));                                                                       \
        out.v1 = y0.v1 + s * (expr(v1));                                                                       \
        out.v2 = y0.v2 + s * (expr(v2));                                                                       \
        out.nu = y0.nu + s * (expr(nu));                                                                       \
    } while (0)

// Adaptive Runge-Kutta-Fehlberg 4(5) backwards over dt with the reference's
// tableau (including its 11/44 at stage 6), absolute velocity error control
// and step update 0.95 (tol/TE)^(1/4) (src/GeodesicEquationSolver.cpp:80-188).
// trials counts accepted + rejected steps; a backtrace that exceeds max_trials
// stops where it is and sets capped.
__device__ __forceinline__ void rk45_backtrace(const GridDev &g, const double *__restrict__ rkf, const Local &l,
                                               double tol, double dt, RkState &y0, int max_trials, int &trials,
                                               bool &capped)
{
    double total = 0.0, h = dt;
    trials = 0;
    capped = false;
    RkState k1 = stage(g, rkf, l, y0);
    while (total < dt)
    {
        if (trials >= max_trials)
        {
            capped = true;
            break;
        }
        trials++;
        h = fmin(h, dt - total);
        const double s = -h;
        RkState y, k2, k3, k4, k5, k6;
#define GRLBM_C(q) (1.0 / 4.0) * k1.q
        GRLBM_EACH(y, GRLBM_C);
#undef GRLBM_C
        k2 = stage(g, rkf, l, y);
#define GRLBM_C(q) (3.0 / 32.0) * k1.q + (9.0 / 32.0) * k2.q
        GRLBM_EACH(y, GRLBM_C);
#undef GRLBM_C
        k3 = stage(g, rkf, l, y);
#define GRLBM_C(q) (1932.0 / 2197.0) * k1.q - (7200.0 / 2197.0) * k2.q + (7296.0 / 2197.0) * k3.q
        GRLBM_EACH(y, GRLBM_C);
#undef GRLBM_C
        k4 = stage(g, rkf, l, y);
#define GRLBM_C(q) (439.0 / 216.0) * k1.q - (8.0) * k2.q + (3680.0 / 513.0) * k3.q - (845.0 / 4104.0) * k4.q
        GRLBM_EACH(y, GRLBM_C);
#undef GRLBM_C
        k5 = stage(g, rkf, l, y);
#define GRLBM_C(q)                                                                                            \
    -(8.0 / 27.0) * k1.q + (2.0) * k2.q - (3544.0 / 2565.0) * k3.q + (1859.0 / 4104.0) * k4.q - (11.0 / 44.0) * k5.q
        GRLBM_EACH(y, GRLBM_C);
#undef GRLBM_C
        k6 = stage(g, rkf, l, y);
#define GRLBM_TE(q)                                                                                           \
    ((1.0 / 360.0) * k1.q - (128.0 / 4275.0) * k3.q - (2197.0 / 75240.0) * k4.q + (1.0 / 50.0) * k5.q +        \
     (2.0 / 55.0) * k6.q)
        const double e1 = h * GRLBM_TE(v1), e2 = h * GRLBM_TE(v2);
#undef GRLBM_TE
        const double te = sqrt(e1 * e1 + e2 * e2);
        if (te > tol)
        {
            h *= 0.95 * pow(tol / te, 1.0 / 4.0);
            continue; // from the same point: k1 stands
        }
#define GRLBM_C(q)                                                                                            \
    (16.0 / 135.0) * k1.q + (6656.0 / 12825.0) * k3.q + (28561.0 / 56430.0) * k4.q - (9.0 / 50.0) * k5.q +     \
        (2.0 / 55.0) * k6.q
        GRLBM_EACH(y0, GRLBM_C);
#undef GRLBM_C
        total += h;
        h *= 0.95 * pow(tol / (te + 1e-50), 1.0 / 4.0);
        if (inside_bh(g, y0.x1, y0.x2) || dev_outside(g, y0.x1, y0.x2))
            break;
        if (total < dt)
            k1 = stage(g, rkf, l, y0);
    }
}
#undef GRLBM_EACH

// cells of a row per block for nf directions: as many as fit the block
int block_cells(int nf) { return std::max(1, std::min(kMaxCells, kThreads / nf)); }

// UpdateFourierCoefficients (src/Radiation.cpp:204-235): the block's
// trajectories, then their projection (Fourier::GetCoefficients,
// src/FourierHarmonics.cpp:33-45): coef_k = sum_f (data_f w_f) B_k(phi_f),
// accumulated over f in order with each product and sum rounded on its own.
// A block holds whole cells, so the five fields (1/s, x, y, vIF_x, vIF_y) go
// from thread to thread through shared memory: no workspace in HBM and no
// second kernel (0.12 ms at 400^2 x 16, and a 100 MB allocation per build).
// blockIdx.x: the runs of `cells` cells of a row, row after row.
#ifndef GRLBM_GEODESIC_MIN_BLOCKS
#define GRLBM_GEODESIC_MIN_BLOCKS 3
#endif
__global__ void __launch_bounds__(kThreads, GRLBM_GEODESIC_MIN_BLOCKS)
    k_geodesic(const __grid_constant__ GeodesicArgs a, int cells)
{
    extern __shared__ __align__(16) double patch[];
    const int nx_ = (int)a.g.nx_, nf = a.nf;
    __shared__ double data[5][kThreads]; // the block's trajectory ends
    const int runs = (nx_ + cells - 1) / cells;
    const int x0 = (int)(blockIdx.x % (unsigned)runs) * cells;
    const int row = (int)(a.c0 / a.g.nx_) + (int)(blockIdx.x / (unsigned)runs);
    Local l;
    l.px0 = x0; // the node left of the run's first cell
    l.py0 = row;
    l.pnx = min(cells, nx_ - x0) + 2;
    for (int e = threadIdx.x; e < 3 * l.pnx * (kFields / 2); e += kThreads)
    {
        const int n = e / (kFields / 2), f = 2 * (e - n * (kFields / 2));
        const int64_t ij = (int64_t)(x0 + n % l.pnx) + (int64_t)(row + n / l.pnx) * a.g.nx;
        *reinterpret_cast<double2 *>(patch + n * kFields + f) =
            __ldg(reinterpret_cast<const double2 *>(a.rkf + ij * kRkStride + f));
    }
    __syncthreads();
    // scaled spacings (exact: powers of two)
    l.sx = scalbn(1.0, -ilogb(a.g.dx));
    l.sy = scalbn(1.0, -ilogb(a.g.dy));
    l.dx = a.g.dx * l.sx;
    l.dy = a.g.dy * l.sy;
    l.rx = __drcp_rn(l.dx);
    l.ry = __drcp_rn(l.dy);
    int trials = 0;
    bool capped = false;
    const int lx = (int)threadIdx.x / nf, f = (int)threadIdx.x - lx * nf;
    const bool active = lx < cells && x0 + lx < nx_;
    const int64_t i = 1 + x0 + lx, j = 1 + row, ij = i + j * a.g.nx;
    if (active)
    {
        RkState y;
        y.x1 = __dadd_rn(a.g.startx, __dmul_rn((double)i, a.g.dx));
        y.x2 = __dadd_rn(a.g.starty, __dmul_rn((double)j, a.g.dy));
        y.nu = 1.0;
        const double alpha = __ldg(a.rkf + ij * kRkStride + RF_ALPHA);
        // Vec2ObservedByEulObs<IF,LF>(alpha (1, c), xy) (src/SpecialMath.cpp:131-136)
        const double u1 = __ldg(a.ss_cx + f) * alpha, u2 = __ldg(a.ss_cy + f) * alpha;
        double fld[kFields];
        fields_at(a.g, a.rkf, l, y.x1, y.x2, fld);
        const double w1 = u1 / fld[RF_ALPHA], w2 = u2 / fld[RF_ALPHA];
        double t11, t12, t21, t22;
        tetrad_block(a.g, a.rkf, l, y.x1, y.x2, RF_T11, t11, t12, t21, t22);
        y.v1 = t11 * w1 + t12 * w2;
        y.v2 = t21 * w1 + t22 * w2;
        if (!inside_bh(a.g, y.x1, y.x2))
            rk45_backtrace(a.g, a.rkf, l, a.tol, a.g.dt, y, a.max_trials, trials, capped);
        else
            y.v1 = y.v2 = 0.0;
        double i11, i12, i21, i22;
        tetrad_block(a.g, a.rkf, l, y.x1, y.x2, RF_TI11, i11, i12, i21, i22);
        data[0][threadIdx.x] = 1.0 / y.nu;
        data[1][threadIdx.x] = y.x1;
        data[2][threadIdx.x] = y.x2;
        data[3][threadIdx.x] = i11 * y.v1 + i12 * y.v2;
        data[4][threadIdx.x] = i21 * y.v1 + i22 * y.v2;
    }
    // block-aggregated counters
    __shared__ unsigned long long s_trials;
    __shared__ int s_capped;
    if (threadIdx.x == 0)
    {
        s_trials = 0;
        s_capped = 0;
    }
    __syncthreads();
    if (active) // this thread's harmonic f of its cell
    {
        double c[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
        for (int k = 0; k < nf; k++)
        {
            const double w = __ldg(a.ss_w + k), b = __ldg(a.basis + k * nf + f);
#pragma unroll
            for (int q = 0; q < 5; q++)
                c[q] = __dadd_rn(c[q], __dmul_rn(__dmul_rn(data[q][lx * nf + k], w), b));
        }
        double *out = a.coef + ij * nf + f;
#pragma unroll
        for (int q = 0; q < 5; q++)
            out[(int64_t)q * a.g.nxy * nf] = c[q];
    }
    if (trials)
        atomicAdd(&s_trials, (unsigned long long)trials);
    if (capped)
        atomicAdd(&s_capped, 1);
    __syncthreads();
    if (threadIdx.x == 0)
    {
        if (s_trials)
            atomicAdd(a.trials_total, s_trials);
        if (s_capped)
            atomicAdd(a.nonconverged, s_capped);
    }
}
} // namespace

// a.c0 and a.cn are whole rows of interior cells
void launch_geodesic(const GeodesicArgs &a, cudaStream_t s)
{
    const int cells = block_cells(a.nf);
    const unsigned rows = (unsigned)(a.cn / a.g.nx_);
    if (rows == 0)
        return;
    const unsigned grid = (unsigned)((a.g.nx_ + cells - 1) / cells) * rows;
    k_geodesic<<<grid, kThreads, (size_t)(cells + 2) * 3 * kFields * sizeof(double), s>>>(a, cells);
}
} // namespace grlbm
