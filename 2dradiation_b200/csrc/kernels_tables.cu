// The per-(cell, direction) departure records derived from the geodesic
// tables' Fourier coefficients (kernels_geodesic.cu), and the alpha-ratio
// cubes.  FP64 throughout; built with -fmad=false so that each
// expression rounds exactly as the reference's CPU build does.
#include "approx_math.hpp"
#include "device_common.cuh"

namespace grlbm
{
// Departure records from the Fourier series: what StreamCurvedFixed
// evaluates every step (src/Radiation.cpp:478-499) and the angle part of
// IntensityAt (:324-328).  One thread per (interior cell, direction): plain
// records are written direction-major ([d * ncell + c], threads over cells
// fastest), precision records cell-major ([c * nd + d], threads over
// directions fastest).
__global__ void __launch_bounds__(128) k_departure(DepartureArgs a)
{
    const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (tid >= a.cn * a.nd)
        return;
    int d;
    int64_t c, ri; // the cell, and its record's index
    if (a.rec32 || a.recf)
    {
        c = a.c0 + tid / a.nd;
        d = (int)(tid % a.nd);
        ri = c * a.nd + d;
    }
    else
    {
        d = (int)(tid / a.cn);
        c = a.c0 + (tid - (int64_t)d * a.cn);
        ri = (int64_t)d * a.g.ncell + c;
    }
    const int64_t i = 1 + c % a.g.nx_, j = 1 + c / a.g.nx_;
    const int64_t ij = i + j * a.g.nx;
    const int64_t fs = a.g.nxy * a.nf;
    const double *cS = a.coef + ij * a.nf;
    // Fourier::GetValue (src/FourierHarmonics.cpp:56-61), summed in k order
    double s = 0.0, xt = 0.0, yt = 0.0, v1 = 0.0, v2 = 0.0;
    for (int k = 0; k < a.nf; k++)
    {
        const double b = __ldg(a.eval + k * a.nd + d);
        s += cS[k] * b;
        xt += cS[k + fs] * b;
        yt += cS[k + 2 * fs] * b;
        v1 += cS[k + 3 * fs] * b;
        v2 += cS[k + 4 * fs] * b;
    }
    double4 r64;
    float4 r32;
    double4 sf; // the FP64 side record {i_dep - i, j_dep - j, angle coordinate, s^3 alpha_c^3}
    double dd; // angle coordinate of the departure direction
    if (dev_inside_bh(a.g, xt, yt))
    {
        r64 = make_double4((double)i, (double)j, -1.0, 0.0);
        dd = 10.0 * d + 5.0;
        r32 = make_float4(0.f, 0.f, (float)dd, 0.f);
        sf = make_double4(0.0, 0.0, dd, 0.0);
    }
    else
    {
        const double it = (xt - a.g.startx) / a.g.dx;
        const double jt = (yt - a.g.starty) / a.g.dy;
        if (!(it >= 0.0 && it < (double)(a.g.nx - 1) && jt >= 0.0 && jt < (double)(a.g.ny - 1)))
            atomicAdd(a.clamped, 1);
        if (jt == jt)
        {
            // node rows the bilinear gather reads, relative to the cell (a slab's ghost depth)
            const double jf = floor(jt) - (double)j;
            const double ext = fmax(fabs(jf), fabs(jf + 1.0));
            atomicMax(a.row_extent, ext < 1e9 ? (int)ext : 1000000000);
        }
        // RotationMatrix(0).Inverse() * v (src/DataTypes.hh:625-635)
        const double w1 = v1 * a.rot_c - v2 * a.rot_s;
        const double w2 = v1 * a.rot_s + v2 * a.rot_c;
        // InterpolationGrid::d (src/Stencil.cpp:35-38)
        dd = (double)a.ng * approx_phi(w1, w2) / (2.0 * kPi);
        dd = dd < 1e-8 ? 1e-8 : (dd > (double)a.ng - 1e-8 ? (double)a.ng - 1e-8 : dd);
        const double s3 = s * (s * s);
        r64 = make_double4(it, jt, dd, s3);
        // FP32 side record: offsets kept on the grid, alpha_c^3 folded in
        double ox = it - (double)i, oy = jt - (double)j;
        const double lox = -(double)i, hix = (double)(a.g.nx - 2 - i) + 0.999;
        const double loy = -(double)j, hiy = (double)(a.g.ny - 2 - j) + 0.999;
        ox = ox < lox ? lox : (ox > hix ? hix : ox);
        oy = oy < loy ? loy : (oy > hiy ? hiy : oy);
        if (!(ox == ox))
            ox = 0.0;
        if (!(oy == oy))
            oy = 0.0;
        const double al = a.alpha[ij];
        const double s3a3 = s3 * (al * al * al);
        r32 = make_float4((float)ox, (float)oy, (float)dd, (float)s3a3);
        sf = make_double4(ox, oy, dd, s3a3);
    }
    if (a.rec32)
    {
        // packed record (packed32): row type, window start and blend; the
        // corner in the fractions' sign bits, far in the scale's
        const double fxd = floor((double)r32.x), fyd = floor((double)r32.y);
        const bool near = (fxd == -1.0 || fxd == 0.0) && (fyd == -1.0 || fyd == 0.0);
        double ddc = dd == dd ? dd : 0.0;
        int g = (int)floor(ddc);
        g = g < 0 ? 0 : (g > a.ng - 1 ? a.ng - 1 : g);
        double t = ddc - (double)g;
        t = t < 0.0 ? 0.0 : (t > 1.0 ? 1.0 : t);
        const int rt = g % a.q, m = g / a.q;
        const unsigned start = (unsigned)((a.row_base[rt] + a.p * m) % a.nd);
        unsigned tq = (unsigned)(t * (double)(1u << packed32::kTBits) + 0.5);
        tq = tq > (1u << packed32::kTBits) - 1u ? (1u << packed32::kTBits) - 1u : tq;
        const unsigned word = tq | ((unsigned)rt << packed32::kTypeShift) | (start << packed32::kStartShift);
        const float fx = near ? (float)((double)r32.x - fxd) : 0.f, fy = near ? (float)((double)r32.y - fyd) : 0.f;
        const unsigned ux = __float_as_uint(fx) | (near && fxd == 0.0 ? 0x80000000u : 0u);
        const unsigned uy = __float_as_uint(fy) | (near && fyd == 0.0 ? 0x80000000u : 0u);
        const unsigned uw = __float_as_uint(r32.w) | (near ? 0u : 0x80000000u);
        a.rec32[ri] = make_uint4(word, ux, uy, uw);
        if (!near && a.far)
            atomicAdd(a.far, 1ull);
        a.side32[ri] = r32;
    }
    if (a.recf)
    {
        // packed64 record: the fractions, blend and window of the FP64 side
        // record, with the corner, row type, window start and far flag in the
        // spare bits of 1 + f
        const double fxd = floor(sf.x), fyd = floor(sf.y);
        const bool near = (fxd == -1.0 || fxd == 0.0) && (fyd == -1.0 || fyd == 0.0);
        double ddc = dd == dd ? dd : 0.0;
        int g = (int)floor(ddc);
        g = g < 0 ? 0 : (g > a.ng - 1 ? a.ng - 1 : g);
        double t = ddc - (double)g;
        t = t < 0.0 ? 0.0 : (t > 1.0 ? 1.0 : t);
        const int rt = g % a.q, m = g / a.q;
        const unsigned start = (unsigned)((a.row_base[rt] + a.p * m) % a.nd);
        // 1 + f in [1, 2): a value that rounds up to 2 is kept just below it
        auto biased = [](double f, unsigned payload) {
            double v = 1.0 + f;
            if (!(v < 2.0))
                v = 1.9999999999999998;
            const unsigned long long b = (unsigned long long)__double_as_longlong(v);
            const unsigned hi = ((unsigned)(b >> 32) & packed64::kMantHi) | payload;
            return __hiloint2double((int)hi, (int)(unsigned)b);
        };
        const double fx = near ? sf.x - fxd : 0.0, fy = near ? sf.y - fyd : 0.0;
        const unsigned cx = near && fxd == 0.0 ? 0x80000000u : 0u, cy = near && fyd == 0.0 ? 0x80000000u : 0u;
        double4 rf;
        rf.x = biased(fx, cx | ((unsigned)rt << packed64::kExpShift));
        rf.y = biased(fy, cy);
        rf.z = biased(t, start << packed64::kExpShift);
        rf.w = near ? sf.w : __hiloint2double((int)((unsigned)__double2hiint(sf.w) | 0x80000000u), __double2loint(sf.w));
        a.recf[ri] = rf;
        if (!near && a.far)
            atomicAdd(a.far, 1ull);
        a.sidef[ri] = sf;
    }
    if (a.rec64)
        a.rec64[ri] = r64;
}

// (alpha_ij / alpha_n)^3 for the 3x3 neighbours n of each interior node, as
// IntegerPow<3>(alpha / metric.GetAlpha(corner)) (src/Radiation.cpp:502-505).
__global__ void k_alpha_cube(GridDev g, const double *alpha, double *acube)
{
    const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= g.ncell)
        return;
    const int64_t i = 1 + c % g.nx_, j = 1 + c / g.nx_;
    const int64_t ij = i + j * g.nx;
    const double al = alpha[ij];
    for (int dj = -1; dj <= 1; dj++)
        for (int di = -1; di <= 1; di++)
        {
            const double r = al / alpha[ij + di + dj * g.nx];
            acube[ij + (3 * (dj + 1) + (di + 1)) * g.nxy] = r * (r * r);
        }
}

static inline unsigned nblk(int64_t n, int b) { return (unsigned)((n + b - 1) / b); }

void launch_departure(const DepartureArgs &a, cudaStream_t s)
{
    k_departure<<<nblk(a.cn * a.nd, 128), 128, 0, s>>>(a);
}
void launch_alpha_cube(const GridDev &g, const double *alpha, double *acube, cudaStream_t s)
{
    k_alpha_cube<<<nblk(g.ncell, 128), 128, 0, s>>>(g, alpha, acube);
}
} // namespace grlbm
