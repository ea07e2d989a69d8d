// Plain FP64 form of the radiation step, and the FP64 utility kernels.
//
// Built with -fmad=false: every multiply and add rounds on its own, and every
// expression below follows the association order of the reference's C++
// (src/Radiation.cpp), so that -- given the same geodesic tables -- the state
// after each step is bit-identical to the reference's IEEE build.  That is
// what the 1e-12 parity needs: the lambda iteration stops on the relative
// change of all six moments, including ones that are pure rounding noise
// (e.g. Fy of a nearly isotropic cell), so its iteration counts, and through
// them E, follow the last bits of the streamed intensities.
#include <type_traits>

#include "approx_math.hpp"
#include "device_common.cuh"

namespace grlbm
{
namespace
{
// one stream value: StreamFlatFixed (src/Radiation.cpp:394-410) or
// StreamCurvedFixed with IntensityAt (:478-508, 322-343)
// `clamp_mask` receives bit q set where corner q's angular interpolation was
// positive (kept by the clamp at zero); flat streaming keeps every corner.
// Off: the type of the state's element offsets (unsigned when the state has
// fewer than 2^32 elements, int64_t otherwise).
template <bool CURVED, typename Off>
__device__ __forceinline__ double stream_value(const PlainStepArgs &a, int d, const double4 &r, int64_t i, int64_t j,
                                               int64_t ij, unsigned &clamp_mask)
{
    clamp_mask = 0xFu;
    const int64_t nxy = a.g.nxy;
    const int nx = (int)a.g.nx; // node indices fit in 32 bits (nx * ny < 2^31)
    if constexpr (CURVED)
    {
        if (r.z < 0.0) // departure point inside the excision
            return 0.0;
        const double it = r.x, jt = r.y;
        // corners kept on the grid whatever the record holds
        const int i0 = min(max((int)floor(it), 0), nx - 2); // the conversion saturates: same clamp
        const int j0 = min(max((int)floor(jt), 0), (int)a.g.ny - 2);
        // g0 = floor(z) % nGrid, taken without the division when in range
        const int gz = (int)floor(r.z);
        int g0 = (unsigned)gz < (unsigned)a.ng ? gz : gz % a.ng;
        g0 = g0 < 0 ? 0 : g0;
        const int g1 = g0 + 1 == a.ng ? 0 : g0 + 1; // (g0 + 1) % nGrid
        // Each row is 4 consecutive directions, and the next row starts at
        // the same one or one further on (checked for every direction count
        // in tests/test_plain_paths.py): the two rows read 5 directions.
        const double t = r.z - (double)g0, t1 = 1.0 - t;
        const IgRow *r0 = a.ig_rows + g0, *r1 = a.ig_rows + g1;
        const int b0 = __ldg(&r0->idx.x);
        const bool shift = __ldg(&r1->idx.x) != b0;
        const double2 wa = __ldg(&r0->w01), wb = __ldg(&r0->w23), wc = __ldg(&r1->w01), wd = __ldg(&r1->w23);
        const double al = __ldg(a.alpha + ij);
        const int n00 = i0 + j0 * nx;
        Off o[5]; // element offsets of the directions at corner 00
#pragma unroll
        for (int k = 0; k < 5; k++)
        {
            const int dk = b0 + k;
            o[k] = (Off)(dk >= a.nd ? dk - a.nd : dk) * (Off)nxy + (Off)n00;
        }
        const int di0 = i0 - (int)i, dj0 = j0 - (int)j;
        const bool near = di0 >= -1 && di0 <= 0 && dj0 >= -1 && dj0 <= 0;
        const double *cube00 = a.acube + (ij + (int64_t)(3 * (dj0 + 1) + (di0 + 1)) * nxy);
        double Iq[4];
#pragma unroll
        for (int q = 0; q < 4; q++) // corners 00, 01, 10, 11
        {
            const int off = (q >> 1) + (q & 1) * nx;
            const double x0 = __ldg(a.Iin + (o[0] + (Off)off)), x1 = __ldg(a.Iin + (o[1] + (Off)off));
            const double x2 = __ldg(a.Iin + (o[2] + (Off)off)), x3 = __ldg(a.Iin + (o[3] + (Off)off));
            const double x4 = __ldg(a.Iin + (o[4] + (Off)off));
            const double y0 = shift ? x1 : x0, y1 = shift ? x2 : x1, y2 = shift ? x3 : x2, y3 = shift ? x4 : x3;
            const double v0 = wa.x * x0 + wa.y * x1 + wb.x * x2 + wb.y * x3;
            const double v1 = wc.x * y0 + wc.y * y1 + wd.x * y2 + wd.y * y3;
            double v = v0 * t1 + v1 * t;
            if (!(0.0 < v))
                clamp_mask &= ~(1u << q);
            v = (0.0 < v) ? v : 0.0;
            double cube;
            if (near)
                cube = __ldg(cube00 + (int64_t)((q >> 1) + 3 * (q & 1)) * nxy);
            else
            {
                const double rr = al / __ldg(a.alpha + n00 + off);
                cube = rr * (rr * rr);
            }
            Iq[q] = cube * v;
        }
        const double fx = it - (double)i0, fy = jt - (double)j0;
        const double f0 = Iq[0] * (1.0 - fx) + Iq[2] * fx;
        const double f1 = Iq[1] * (1.0 - fx) + Iq[3] * fx;
        return r.w * (f0 * (1.0 - fy) + f1 * fy);
    }
    else
    {
        double xt = a.g.startx + (double)i * a.g.dx;
        double yt = a.g.starty + (double)j * a.g.dy;
        xt -= __ldg(a.cx + d) * a.g.dt;
        yt -= __ldg(a.cy + d) * a.g.dt;
        const double it = (xt - a.g.startx) / a.g.dx, jt = (yt - a.g.starty) / a.g.dy;
        const int i0 = min(max((int)floor(it), 0), nx - 2);
        const int j0 = min(max((int)floor(jt), 0), (int)a.g.ny - 2);
        const double *plane = a.Iin + (int64_t)d * nxy;
        const int c00 = i0 + j0 * nx;
        const double fx = it - (double)i0, fy = jt - (double)j0;
        const double f0 = __ldg(plane + c00) * (1.0 - fx) + __ldg(plane + c00 + 1) * fx;
        const double f1 = __ldg(plane + c00 + nx) * (1.0 - fx) + __ldg(plane + c00 + nx + 1) * fx;
        return f0 * (1.0 - fy) + f1 * fy;
    }
}

struct Moments
{
    double E, Fx, Fy, Pxx, Pxy, Pyy;
    __device__ __forceinline__ void zero() { E = Fx = Fy = Pxx = Pxy = Pyy = 0.0; }
    // ComputeMomentsIF / Collide accumulation order (src/Radiation.cpp:259-266, 706-712)
    __device__ __forceinline__ void add(double w, double v, double n1, double n2)
    {
        const double c = w * v;
        E += c;
        Fx += c * n1;
        Fy += c * n2;
        Pxx += c * n1 * n1;
        Pxy += c * n1 * n2;
        Pyy += c * n2 * n2;
    }
};

// one collided intensity (src/Radiation.cpp:690-703).  Divisions by A, A*A
// and (lorentz + 1) are skipped only where they are exact no-ops (A == 1,
// un == 0), so the result is the reference's bit for bit.
__device__ __forceinline__ double collide_value(double I, double n1, double n2, double u1, double u2, double lor,
                                                double adt, double eta, double k0, double k3, double kak0,
                                                double fE, double fFx, double fFy)
{
    const double un = u1 * n1 + u2 * n2;
    const double A = lor * (1.0 - un);
    const double sc = (un == 0.0) ? lor : (1 - (lor * un) / (lor + 1)) * lor;
    double nF1 = n1 - sc * u1, nF2 = n2 - sc * u2;
    if (A != 1.0)
    {
        nF1 = nF1 / A;
        nF2 = nF2 / A;
    }
    const double nF = nF1 * fFx + nF2 * fFy;
    const double M = k0 * fE + k3 * nF;
    double src = adt * (eta + M);
    const double AA = A * A;
    if (AA != 1.0)
        src = src / AA;
    return (I + src) / (1.0 + adt * kak0 * A);
}

// num / den, correctly rounded, from r = RN(1/den): one refinement brings
// RN(num r) (within 1.5 ulp of the quotient) to within one ulp, then one
// Markstein step (P. Markstein, IBM J. Res. Dev. 34(1), 1990: with r within
// half an ulp of 1/den and q within one ulp of num/den, the remainder
// num - den q is exact in one fma and RN(q + rem r) is the correctly rounded
// quotient) gives the IEEE result.  Used where den is the same for many
// divisions; outside 2^-900 <= |num| < 2^900, where a step could underflow or
// overflow, the ordinary division is taken.  Requires 1 <= den < 2^100.
__device__ __forceinline__ double div_rn(double num, double den, double r)
{
    // exponent field in [123, 1923) or exactly zero, tested on the integer pipe
    const unsigned hi = (unsigned)__double2hiint(num), ex = (hi >> 20) & 0x7ffu;
    if (ex - 123u >= 1800u && ((hi << 1) | (unsigned)__double2loint(num)) != 0u)
        return num / den;
    double q = __dmul_rn(num, r);
    q = __fma_rn(__fma_rn(-q, den, num), r, q);
    return __fma_rn(__fma_rn(-q, den, num), r, q);
}

// Fourier::GetValue (src/FourierHarmonics.cpp:56-61) with Fourier::Basis
// (:5-14) at a run-time angle, for the five series of a node's geodesic
// tables (S, X, Y, Cx, Cy) at once: coefficient k of series q at
// coef[q * fs + k * sk].  Each basis value is computed once and used by all
// five, and every sum keeps its order over k.
__device__ __forceinline__ void fourier_values5(const double *coef, int64_t fs, int64_t sk, int nf, double phi,
                                                double out[5])
{
    const double sqrt2 = 1.4142135623730951; // sqrt(2), correctly rounded
    double r0 = 0, r1 = 0, r2 = 0, r3 = 0, r4 = 0;
    // the argument of term 2m - 1, phi * (2m - 1 + 1.0) / 2.0, and of term 2m,
    // phi * 2m / 2.0, round alike: one sincos serves both
    double sin_m = 0.0, cos_m = 1.0;
    for (int k = 0; k < nf; k++)
    {
        double b;
        if (k == 0)
            b = 1.0;
        else if (k % 2 != 0)
        {
            sincos(phi * (k + 1.0) / 2.0, &sin_m, &cos_m);
            b = sqrt2 * cos_m;
        }
        else
            b = sqrt2 * sin_m;
        const double *c = coef + k * sk;
        r0 += c[0] * b;
        r1 += c[fs] * b;
        r2 += c[2 * fs] * b;
        r3 += c[3 * fs] * b;
        r4 += c[4 * fs] * b;
    }
    out[0] = r0, out[1] = r1, out[2] = r2, out[3] = r3, out[4] = r4;
}

// IntensityAt (src/Radiation.cpp:322-343) of node n for the (unrotated)
// direction (v1, v2): rotated into the node's stencil frame by the inverse of
// its previous rotation angle, then the two cubic rows of the interpolation
// grid, blended and clamped at zero.
__device__ __forceinline__ double intensity_at(const PlainStepArgs &a, int64_t n, double v1, double v2)
{
    const double2 rinv = a.rot_inv[n]; // RotationMatrix(angle).Inverse()
    const double sn = rinv.x, cs = rinv.y;
    const double w1 = v1 * cs - v2 * sn, w2 = v1 * sn + v2 * cs;
    double dd = (double)a.ng * approx_phi(w1, w2) / (2.0 * kPi); // InterpolationGrid::d
    dd = dd < 1e-8 ? 1e-8 : ((double)a.ng - 1e-8 < dd ? (double)a.ng - 1e-8 : dd);
    // g0 = floor(dd) % nGrid, g1 = (g0 + 1) % nGrid, without the divisions
    // on the in-range path (the clamp keeps floor(dd) in [0, nGrid))
    const int gz = (int)floor(dd);
    int g0 = (unsigned)gz < (unsigned)a.ng ? gz : gz % a.ng;
    g0 = g0 < 0 ? 0 : g0;
    const int g1 = g0 + 1 == a.ng ? 0 : g0 + 1;
    const IgRow R0 = a.ig_rows[g0], R1 = a.ig_rows[g1];
    const int idx0[4] = {R0.idx.x, R0.idx.y, R0.idx.z, R0.idx.w};
    const int idx1[4] = {R1.idx.x, R1.idx.y, R1.idx.z, R1.idx.w};
    const double w0[4] = {R0.w01.x, R0.w01.y, R0.w23.x, R0.w23.y};
    const double wr1[4] = {R1.w01.x, R1.w01.y, R1.w23.x, R1.w23.y};
    double value0 = 0, value1 = 0;
#pragma unroll
    for (int k = 0; k < 4; k++)
    {
        value0 += w0[k] * __ldg(a.Iin + (int64_t)idx0[k] * a.g.nxy + n);
        value1 += wr1[k] * __ldg(a.Iin + (int64_t)idx1[k] * a.g.nxy + n);
    }
    const double t = dd - (double)g0;
    const double v = value0 * (1.0 - t) + value1 * t;
    return (0.0 < v) ? v : 0.0;
}

// One stream value of adaptive streaming: StreamFlatAdaptive
// (src/Radiation.cpp:415-452) or StreamCurvedAdaptive (:513-575), for the
// cell's direction d rotated by the cell's new angle (sine sc, cosine cc).
// Curved streaming reads coefficient k of series q of the cell at
// cf[q * qs + k * ks].
template <bool CURVED>
__device__ __forceinline__ double stream_value_adaptive(const PlainStepArgs &a, int d, int64_t i, int64_t j,
                                                        int64_t ij, double sc, double cc, const double *cf,
                                                        int qs, int ks)
{
    const int64_t nx = a.g.nx;
    const double cx = __ldg(a.cx + d), cy = __ldg(a.cy + d);
    const double dir1 = cx * cc - cy * sc, dir2 = cx * sc + cy * cc;
    double it, jt, v1, v2, s3 = 1.0;
    if constexpr (CURVED)
    {
        const double phi = approx_phi(dir1, dir2);
        double fv[5];
        fourier_values5(cf, qs, ks, a.nf, phi, fv);
        const double sh = fv[0], xt = fv[1], yt = fv[2];
        v1 = fv[3];
        v2 = fv[4];
        if (dev_inside_bh(a.g, xt, yt))
            return 0.0;
        it = (xt - a.g.startx) / a.g.dx;
        jt = (yt - a.g.starty) / a.g.dy;
        s3 = sh * (sh * sh);
    }
    else
    {
        double xt = a.g.startx + (double)i * a.g.dx, yt = a.g.starty + (double)j * a.g.dy;
        xt -= dir1 * a.g.dt;
        yt -= dir2 * a.g.dt;
        it = (xt - a.g.startx) / a.g.dx;
        jt = (yt - a.g.starty) / a.g.dy;
        v1 = dir1;
        v2 = dir2;
    }
    // corners kept on the grid whatever the departure
    const int64_t i0 = min(max((int64_t)floor(it), (int64_t)0), nx - 2);
    const int64_t j0 = min(max((int64_t)floor(jt), (int64_t)0), a.g.ny - 2);
    const double al = CURVED ? __ldg(a.alpha + ij) : 1.0;
    double Iq[4];
#pragma unroll
    for (int q = 0; q < 4; q++) // corners 00, 01, 10, 11
    {
        const int64_t n = (i0 + (q >> 1)) + (j0 + (q & 1)) * nx;
        double v = intensity_at(a, n, v1, v2);
        if (CURVED)
        {
            const double rr = al / __ldg(a.alpha + n);
            v = rr * (rr * rr) * v;
        }
        Iq[q] = v;
    }
    const double fx = it - (double)i0, fy = jt - (double)j0;
    const double f0 = Iq[0] * (1.0 - fx) + Iq[2] * fx;
    const double f1 = Iq[1] * (1.0 - fx) + Iq[3] * fx;
    const double bil = f0 * (1.0 - fy) + f1 * fy;
    return CURVED ? s3 * bil : bil;
}

// Template switches of the step's kernels.  RECORD: also write what the
// adjoint needs about this step -- per (d, c) the corner clamp mask, per cell
// the lambda-iteration count and the first iterate's E -- without changing
// any result.  ADAPTIVE: the adaptive streaming types -- each cell's stencil
// is rotated by its new angle (its directions in stream, moments and
// collide) and corners are read in their previous frames.

// The fixed streaming types run the step as two kernels, so that the
// stream's dependent gathers (record, interpolation rows, 32 corner taps)
// of different directions run in different threads instead of one after the
// other in one thread per cell.  Stream: one thread per (cell, direction) of
// the slab rows writes the streamed value to S (and, recording, the corner
// clamp mask).
// Blocks are 32 x 4 tiles of cells (blockIdx.x, blockIdx.y over the slab
// rows) of one direction (blockIdx.z).
// Grid order of the stream kernel: directions fastest for adaptive streaming
// (the blocks of one tile, which read the same Fourier coefficients, run
// together), tiles fastest for fixed streaming (measured: 2% faster and 3%
// slower respectively the other way round).
constexpr bool kDirFastestAdaptive = true, kDirFastestFixed = false;
#ifndef GRLBM_SPLIT_TILE_X
#define GRLBM_SPLIT_TILE_X 16
#endif
constexpr int kSplitTileX = GRLBM_SPLIT_TILE_X, kSplitTileY = kStepBlock / kSplitTileX;
// resident blocks per SM the stream kernel's registers are sized for (6:
// 80 registers, no spills in the curved gather with 32-bit offsets)
#ifndef GRLBM_STREAM_MIN_BLOCKS
#define GRLBM_STREAM_MIN_BLOCKS 6
#endif
template <bool CURVED, bool RECORD, bool ADAPTIVE, bool WIDE = false>
__global__ void __launch_bounds__(kStepBlock, GRLBM_STREAM_MIN_BLOCKS) k_stream_plain(PlainStepArgs a, StepRecord rec)
{
    static_assert(!(CURVED && ADAPTIVE), "curved adaptive streaming runs k_stream_plain_curved_adaptive");
    constexpr bool DFAST = ADAPTIVE ? kDirFastestAdaptive : kDirFastestFixed;
    const int d = DFAST ? blockIdx.x : blockIdx.z;
    const int bx = DFAST ? blockIdx.y : blockIdx.x, by = DFAST ? blockIdx.z : blockIdx.y;
    const int i = 1 + bx * kSplitTileX + (int)(threadIdx.x % kSplitTileX);
    const int j = (int)a.g.jlo + by * kSplitTileY + (int)(threadIdx.x / kSplitTileX);
    if (i > a.g.nx_ || j >= a.g.jhi)
        return;
    const int64_t cc = (int64_t)(i - 1) + (int64_t)(j - 1) * a.g.nx_;
    const int64_t ij = (int64_t)i + (int64_t)j * a.g.nx;
    unsigned cm = 0xFu;
    double val = 0.0;
    if (!(CURVED && (a.flags[ij] & 2)))
    {
        if constexpr (ADAPTIVE)
        {
            // the cell's rotation (RotationMatrix(rotationAngle[ij]), src/DataTypes.hh:630-635)
            const double2 rn = a.rot_new[ij];
            val = stream_value_adaptive<CURVED>(a, d, i, j, ij, rn.x, rn.y, nullptr, 0, 0);
        }
        else
        {
            const double4 r = CURVED ? a.rec[(int64_t)d * a.g.ncell + cc] : make_double4(0, 0, 0, 0);
            val = stream_value<CURVED, std::conditional_t<WIDE, int64_t, unsigned>>(a, d, r, i, j, ij, cm);
        }
    }
    if (RECORD)
        rec.clamp[(int64_t)d * a.g.ncell + cc] = (uint8_t)cm;
    a.S[(int64_t)d * a.g.nxy + ij] = val;
}

// Curved fixed stream from a staged patch: a block takes 16 x 4 cells with
// all their directions.  It first copies the state of the tile's 18 x 6 nodes
// ([direction][row][node], nd * 896 bytes) and its cells' alpha cubes into
// shared memory; its threads (64 cells x 4 directions at a time) then stream
// direction after direction, each thread's next record loaded while the
// current one is worked on.  Same arithmetic, in the same order, as
// stream_value<true>.
//
// What bounds the gather from global memory (stream_value) is latency: record,
// interpolation rows and 20 corner taps one after the other at 24 warps per
// SM (266 us at 400^2 x 64, DRAM 21% and L1 62% busy; fewer tap loads and
// coalesced alpha cubes alone left it at 270 us).  Here a tap is a
// conflict-free 8-byte shared-memory read and only the record still comes
// from DRAM, a direction ahead.
constexpr int kPatchX = 16, kPatchY = 4;
constexpr int kPatchCells = kPatchX * kPatchY;
// (a direction's plane is a multiple of 16 doubles: lanes whose windows start
// at different directions still read the banks of their own nodes)
constexpr int kPatchPitch = kPatchX + 2, kPatchNodes = kPatchPitch * (kPatchY + 2);
constexpr int kPatchPlane = (kPatchNodes + 15) / 16 * 16;
// with more directions the patch and its rows leave one block per SM: those
// gather from global memory
constexpr int kPatchMaxDirs = 88;
// up to this three blocks of 4 directions fit an SM, above it two of 6: 24
// warps of 80 registers either way (200^2 x 32: 21.8 us against 23.7; 400^2 x
// 64: 149 us against 140)
constexpr int kPatchFewDirs = 57;
__host__ __device__ constexpr size_t patch_smem(int nd)
{
    return ((size_t)nd * kPatchPlane + 9 * kPatchCells) * sizeof(double) + (size_t)10 * nd * 36;
}
__device__ __forceinline__ void copy8_async(double *dst, const double *src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ double4 load_once(const double4 *p)
{
    const double2 lo = __ldcs(reinterpret_cast<const double2 *>(p)), hi = __ldcs(reinterpret_cast<const double2 *>(p) + 1);
    return make_double4(lo.x, lo.y, hi.x, hi.y);
}
template <bool RECORD, int DIRS>
__global__ void __launch_bounds__(kPatchCells * DIRS, DIRS == 4 ? 3 : 2)
    k_stream_plain_patch(const __grid_constant__ PlainStepArgs a, const __grid_constant__ StepRecord rec)
{
    // [d][row][node], the cells' 9 alpha cubes [n][cell], the interpolation rows
    extern __shared__ double patch[];
    constexpr int kPatchDirs = DIRS, kPatchThreads = kPatchCells * DIRS;
    const int t = threadIdx.x, lx = t % kPatchX, ly = (t / kPatchX) % kPatchY, dg = t / kPatchCells;
    const int cell = t % kPatchCells;
    const int nx = (int)a.g.nx, nd = a.nd;
    const int x0 = (int)blockIdx.x * kPatchX, y0 = (int)a.g.jlo - 1 + (int)blockIdx.y * kPatchY; // the patch's first node
    const int64_t nxy = a.g.nxy;
    double *cubes = patch + (size_t)nd * kPatchPlane;
    const int i = 1 + x0 + lx, j = 1 + y0 + ly;
    const bool active = i <= (int)a.g.nx_ && j < (int)a.g.jhi;
    const int ij = i + j * nx;
    const int64_t cc = (int64_t)(i - 1) + (int64_t)(j - 1) * a.g.nx_;
    const bool streams = active && !(a.flags[ij] & 2);
    double4 r = make_double4(0, 0, 0, 0);
    if (streams && dg < nd)
        r = load_once(a.rec + (int64_t)dg * a.g.ncell + cc);
    // thread t copies node t mod 128 of the plane (108 nodes) of every second direction
    {
        const int n = t % 128, prow = n / kPatchPitch, pcol = n - prow * kPatchPitch;
        const int ni = x0 + pcol, nj = y0 + prow;
        if (n < kPatchNodes && ni < nx && nj < (int)a.g.ny)
        {
            const double *src = a.Iin + ni + (int64_t)nj * nx;
            for (int d = t / 128; d < nd; d += kPatchThreads / 128)
                copy8_async(patch + d * kPatchPlane + n, src + (int64_t)d * nxy);
        }
    }
    double2 *wrow = reinterpret_cast<double2 *>(cubes + 9 * kPatchCells);
    int *brow = reinterpret_cast<int *>(wrow + 2 * a.ng);
    for (int g = t; g < a.ng; g += kPatchThreads)
    {
        const IgRow *r0 = a.ig_rows + g, *r1 = a.ig_rows + (g + 1 == a.ng ? 0 : g + 1);
        wrow[2 * g] = r0->w01;
        wrow[2 * g + 1] = r0->w23;
        brow[g] = 2 * r0->idx.x + (r1->idx.x != r0->idx.x);
    }
    if (active)
        for (int n = dg; n < 9; n += kPatchDirs)
            copy8_async(cubes + n * kPatchCells + cell, a.acube + ij + (int64_t)n * nxy);
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    __syncthreads();
    if (!active)
        return;
    unsigned far = 0; // this thread's directions (bit d / 4) that depart outside the 3x3 neighbourhood
    static_assert(kPatchMaxDirs <= 32 * kPatchDirs, "one bit per direction of a thread");
    for (int d = dg; d < nd; d += kPatchDirs)
    {
        const double4 rc = r;
        if (streams && d + kPatchDirs < nd)
            r = load_once(a.rec + (int64_t)(d + kPatchDirs) * a.g.ncell + cc);
        unsigned cm = 0xFu;
        double val = 0.0;
        if (streams && !(rc.z < 0.0))
        {
            const int i0 = min(max((int)floor(rc.x), 0), nx - 2);
            const int j0 = min(max((int)floor(rc.y), 0), (int)a.g.ny - 2);
            if ((unsigned)(i0 - i + 1) <= 1u && (unsigned)(j0 - j + 1) <= 1u)
            {
                const int gz = (int)floor(rc.z);
                int g0 = (unsigned)gz < (unsigned)a.ng ? gz : gz % a.ng;
                g0 = g0 < 0 ? 0 : g0;
                const int g1 = g0 + 1 == a.ng ? 0 : g0 + 1;
                const double tt = rc.z - (double)g0, t1 = 1.0 - tt;
                const int bs = brow[g0], b0 = bs >> 1;
                const bool shift = bs & 1;
                const double2 wa = wrow[2 * g0], wb = wrow[2 * g0 + 1], wc = wrow[2 * g1], wd = wrow[2 * g1 + 1];
                const double *p[5];
#pragma unroll
                for (int k = 0; k < 5; k++)
                {
                    const int dk = b0 + k;
                    p[k] = patch + ((dk >= nd ? dk - nd : dk) * kPatchPlane + (i0 - x0) + (j0 - y0) * kPatchPitch);
                }
                const double *cube00 = cubes + (3 * (j0 - j + 1) + (i0 - i + 1)) * kPatchCells + cell;
                double Iq[4];
#pragma unroll
                for (int q = 0; q < 4; q++) // corners 00, 01, 10, 11
                {
                    const int off = (q >> 1) + (q & 1) * kPatchPitch;
                    const double c0 = p[0][off], c1 = p[1][off], c2 = p[2][off], c3 = p[3][off], c4 = p[4][off];
                    const double e0 = shift ? c1 : c0, e1 = shift ? c2 : c1, e2 = shift ? c3 : c2, e3 = shift ? c4 : c3;
                    const double v0 = wa.x * c0 + wa.y * c1 + wb.x * c2 + wb.y * c3;
                    const double v1 = wc.x * e0 + wc.y * e1 + wd.x * e2 + wd.y * e3;
                    double v = v0 * t1 + v1 * tt;
                    if (!(0.0 < v))
                        cm &= ~(1u << q);
                    v = (0.0 < v) ? v : 0.0;
                    Iq[q] = cube00[((q >> 1) + 3 * (q & 1)) * kPatchCells] * v;
                }
                const double fx = rc.x - (double)i0, fy = rc.y - (double)j0;
                const double f0 = Iq[0] * (1.0 - fx) + Iq[2] * fx;
                const double f1 = Iq[1] * (1.0 - fx) + Iq[3] * fx;
                val = rc.w * (f0 * (1.0 - fy) + f1 * fy);
            }
            else
                far |= 1u << (d / kPatchDirs);
        }
        if (RECORD)
            rec.clamp[(int64_t)d * a.g.ncell + cc] = (uint8_t)cm;
        a.S[(int64_t)d * nxy + ij] = val;
    }
    // the rare far departures, from global memory
    for (; far; far &= far - 1)
    {
        const int d = (__ffs((int)far) - 1) * kPatchDirs + dg;
        unsigned cm;
        a.S[(int64_t)d * nxy + ij] =
            stream_value<true, int64_t>(a, d, load_once(a.rec + (int64_t)d * a.g.ncell + cc), i, j, ij, cm);
        if (RECORD)
            rec.clamp[(int64_t)d * a.g.ncell + cc] = (uint8_t)cm;
    }
}

// Curved adaptive stream: a block takes 16 cells of one row for kPDirs
// directions (16: 7% faster than 8, and 32 slower, at 400^2 x 64).  It first
// stages the row's Fourier coefficients (5 nF x 16 doubles, at most 40 KB)
// in shared memory, where its directions share them; each warp then covers
// 16 cells x 2 directions.
constexpr int kPDirs = kAdaptiveBlock / kSplitTileX;
__global__ void __launch_bounds__(kAdaptiveBlock) k_stream_plain_curved_adaptive(PlainStepArgs a)
{
    extern __shared__ double sco[]; // [q * nF + k][cell]
    // blockIdx.x: direction group fastest, then the row; blockIdx.y: the run of 16 cells
    const int ndg = (a.nd + kPDirs - 1) / kPDirs;
    const int t = threadIdx.x, c = t % kSplitTileX;
    const int d = (int)(blockIdx.x % (unsigned)ndg) * kPDirs + t / kSplitTileX;
    const int x0 = 1 + (int)blockIdx.y * kSplitTileX, i = x0 + c;
    const int j = (int)a.g.jlo + (int)(blockIdx.x / (unsigned)ndg);
    const int nrow = min(kSplitTileX, (int)a.g.nx_ + 1 - x0);
    const int64_t row0 = (int64_t)x0 + (int64_t)j * a.g.nx;
    // coefficient k of series q of node ij sits at coef[(q nF + k) nxy + ij]
    for (int e = t; e < 5 * a.nf * kSplitTileX; e += kAdaptiveBlock)
    {
        const int p = e / kSplitTileX, cc = e % kSplitTileX;
        sco[e] = cc < nrow ? a.coef[(int64_t)p * a.g.nxy + row0 + cc] : 0.0;
    }
    __syncthreads();
    if (c >= nrow || d >= a.nd)
        return;
    const int64_t ij = row0 + c;
    double val = 0.0;
    if (!(a.flags[ij] & 2))
    {
        // the cell's rotation (RotationMatrix(rotationAngle[ij]), src/DataTypes.hh:630-635)
        const double2 rn = a.rot_new[ij];
        val = stream_value_adaptive<true>(a, d, i, j, ij, rn.x, rn.y, sco + c, a.nf * kSplitTileX, kSplitTileX);
    }
    a.S[(int64_t)d * a.g.nxy + ij] = val;
}

// The lambda iteration's exit test (src/Radiation.cpp:714-721): whether
// sqrt(sum ((p - m) / m)^2) over the six moments is above 1e-4.  The sum is
// first taken in FP32 (within 1e-5 of itself while every moment is in FP32's
// range); only where that is within 0.1% of the limit, or not in range, are
// the six quotients and the root taken as the reference does.
__device__ __forceinline__ bool still_changing(const double (&p)[6], const double (&m)[6])
{
    float s = 0.f, lo = 1e30f, hi = 0.f;
#pragma unroll
    for (int q = 0; q < 6; q++)
    {
        const float d = (float)(p[q] - m[q]), f = (float)m[q], x = __fdividef(d, f);
        s += x * x;
        lo = fminf(lo, fabsf(f));
        hi = fmaxf(hi, fabsf(f));
        // a difference below FP32's normal range counts as out of range, zero does not
        if (d != 0.f && fabsf(d) < 1e-30f)
            lo = 0.f;
    }
    if (lo > 1e-30f && hi < 1e30f && (s > 1.001e-8f || s < 0.999e-8f) && s < 1e30f)
        return s > 1e-8f;
    double e = 0.0, ee[6];
#pragma unroll
    for (int q = 0; q < 6; q++)
        ee[q] = (p[q] - m[q]) / m[q];
    e = ee[0] * ee[0] + ee[1] * ee[1] + ee[2] * ee[2] + ee[3] * ee[3] + ee[4] * ee[4] + ee[5] * ee[5];
    return fabs(sqrt(e)) > 1e-4;
}

// Moments and collide of the streamed values: one thread per cell sums the
// moments in direction order (ComputeMomentsIF's order), runs the lambda
// iteration (src/Radiation.cpp:641-736) and writes the collided intensities.
// The order of a moment's sum is the reference's, so a cell's passes over the
// directions are serial and the kernel is bound by issuing them: with COLUMN
// (up to kColumnMaxDirs directions) each cell's streamed values wait in a
// column of shared memory, and the passes of a fluid at rest without anisotropic
// scattering are stripped to the 17 FP64 operations per direction that the
// roundings need.  (Two lanes per cell, sharing the quotients and the six
// sums, doubled the warps but took a third more operations: 183 us against
// 134 at 400^2 x 64.)
constexpr int kColumnTileY = 4; // 16 x 4 cells per block with COLUMN
// the column up to 91 directions (100^2 x 91 flat: 39 us a step against 69
// without it), 90 for a moving fluid (400 x 300 x 91: 1125 against 727)
constexpr int kColumnMaxDirs = 91, kColumnMaxDirsMoving = 90;
// Resident blocks the kernel with the column is compiled for.  A fluid at rest
// without anisotropic scattering: 6 (142 registers; 8 blocks are 2% to 5%
// slower).  GENERAL, a fluid that moves or scatters anisotropically somewhere,
// whose passes are chains of divisions: 8 (128 registers; 400 x 300 x 48 moving,
// flat: 381 us a step against 474 with 6, x 33 anisotropic: 90 against 103).
#ifndef GRLBM_COLLIDE_MIN_BLOCKS
#define GRLBM_COLLIDE_MIN_BLOCKS 6
#endif
#ifndef GRLBM_COLLIDE_GENERAL_BLOCKS
#define GRLBM_COLLIDE_GENERAL_BLOCKS 8
#endif
#ifndef GRLBM_COLLIDE_WIDE_BLOCKS
#define GRLBM_COLLIDE_WIDE_BLOCKS 4
#endif
#ifndef GRLBM_COLLIDE_UNROLL
#define GRLBM_COLLIDE_UNROLL 8
#endif
constexpr int kCollideUnroll = GRLBM_COLLIDE_UNROLL;
constexpr size_t collide_smem(int nd, bool column)
{
    return (size_t)nd * (4 + (column ? kSplitTileX * kColumnTileY : 0)) * sizeof(double);
}
template <bool RECORD, bool ADAPTIVE, bool COLUMN, bool GENERAL = false>
__global__ void __launch_bounds__(COLUMN ? kSplitTileX *kColumnTileY : kStepBlock,
                                  !COLUMN ? GRLBM_COLLIDE_WIDE_BLOCKS
                                          : (GENERAL ? GRLBM_COLLIDE_GENERAL_BLOCKS : GRLBM_COLLIDE_MIN_BLOCKS))
    k_collide_plain(const __grid_constant__ PlainStepArgs a, const __grid_constant__ StepRecord rec)
{
    constexpr int TY = COLUMN ? kColumnTileY : kSplitTileY, NT = kSplitTileX * TY;
    extern __shared__ __align__(16) double dyn[]; // {n1, n2, w, 0} per direction, then the values [d][cell]
    const int t = threadIdx.x;
    const int ti = 1 + (int)blockIdx.x * kSplitTileX + t % kSplitTileX;
    const int tj = (int)a.g.jlo + (int)blockIdx.y * TY + t / kSplitTileX;
    const bool active = ti <= a.g.nx_ && tj < a.g.jhi;
    const int64_t i = active ? ti : 1, j = active ? tj : 1;
    const int64_t ij = i + j * a.g.nx;
    const int64_t nxy = a.g.nxy;
    const int nd = a.nd;
    const double *S = a.S + ij;
    double2 *dir = reinterpret_cast<double2 *>(dyn);
    double *col = dyn + 4 * nd + t;
    const double *dn1 = ADAPTIVE ? a.cx : a.n1, *dn2 = ADAPTIVE ? a.cy : a.n2;
    for (int d = t; d < nd; d += NT)
    {
        dir[2 * d] = make_double2(dn1[d], dn2[d]);
        dir[2 * d + 1] = make_double2(a.w[d], 0.0);
    }
    const bool collides = active && !(a.flags[ij] & 1);
    // the cell's rotation (adaptive streaming)
    double rot_s = 0.0, rot_c = 1.0;
    if (ADAPTIVE)
    {
        const double2 rn = a.rot_new[ij];
        rot_s = rn.x;
        rot_c = rn.y;
    }
    __syncthreads();
    auto streamed = [&](int d) { return COLUMN ? col[d * NT] : S[(int64_t)d * nxy]; };
    // direction d of the cell's stencil
    auto direction = [&](int d) {
        const double2 n = dir[2 * d];
        return ADAPTIVE ? make_double2(n.x * rot_c - n.y * rot_s, n.x * rot_s + n.y * rot_c) : n;
    };
    Moments m;
    m.zero();
    // the streamed values' high words: the range of the quotients' shortcut
    unsigned least = 0x7fffffffu, most = 0u;
    if (active)
    {
#pragma unroll 8
        for (int d = 0; d < nd; d++)
        {
            const double v = S[(int64_t)d * nxy];
            if (COLUMN)
                col[d * NT] = v;
            const double2 n = direction(d);
            const unsigned hi = (unsigned)__double2hiint(v);
            most = max(most, hi);
            least = min(least, (hi | (unsigned)__double2loint(v)) == 0u ? 0x7fffffffu : hi);
            m.add(dir[2 * d + 1].x, v, n.x, n.y);
        }
    }
    const int64_t cc = (i - 1) + (j - 1) * a.g.nx_;
    if (RECORD && active)
        rec.e0[cc] = m.E;
    int cycles = 0;
    if (collides)
    {
        const double u1 = a.u1[ij], u2 = a.u2[ij], lor = a.lor[ij], adt = a.adt[ij];
        const double eta = a.eta[ij], k0 = a.k0[ij], k3 = a.k3[ij], kak0 = a.ka[ij] + a.k0[ij];
        // A fluid at rest has u = 0 and lorentz = 1, so in collide_value
        // A = 1, n_ff = n and AA = 1 exactly: the update reduces to
        // (I + adt (eta + (k0 fE + k3 (n1 fFx + n2 fFy)))) / (1 + adt kak0)
        // with the same roundings.
        const bool rest = u1 == 0.0 && u2 == 0.0 && lor == 1.0;
        const double den = 1.0 + adt * kak0;
        const bool fast_div = rest && den >= 1.0 && den < 0x1p+100;
        const double rden = __drcp_rn(den);
        double fE = 0, fFx = 0, fFy = 0;
        // Without anisotropic scattering (3 kappa1 = 0) the source
        // adt (eta + (k0 fE + 0 (n . fF))) of a fluid at rest is the same
        // number for every direction as long as fF is finite: `src`, worked
        // out once per cycle.  `plain`: every S + src is also zero or in the
        // range of div_rn's shortcut (no negative terms, none tiny or huge).
        bool iso = false, plain = false;
        double src = 0.0;
        auto quotient_plain = [&](double num) {
            double q = __dmul_rn(num, rden);
            q = __fma_rn(__fma_rn(-q, den, num), rden, q);
            return __fma_rn(__fma_rn(-q, den, num), rden, q);
        };
        auto value = [&](int d, double2 n) {
            const double num = streamed(d) + (iso ? src : adt * (eta + (k0 * fE + k3 * (n.x * fFx + n.y * fFy))));
            return fast_div ? div_rn(num, den, rden) : num / den;
        };
        bool more = true;
        do
        {
            cycles++;
            const double p[6] = {m.E, m.Fx, m.Fy, m.Pxx, m.Pxy, m.Pyy};
            const bool was_iso = iso;
            if (rest && fabs(p[0]) < 1e300 && fabs(p[1]) < 1e300 && fabs(p[2]) < 1e300 && fabs(p[3]) < 1e300 &&
                fabs(p[4]) < 1e300 && fabs(p[5]) < 1e300)
            {
                // the transform below with u = 0, lorentz = 1 and finite moments
                fE = p[0];
                fFx = p[1];
                fFy = p[2];
                iso = k3 == 0.0;
            }
            else
            {
                // fluid-frame moments of the previous iterate (src/Radiation.cpp:672-678)
                const double uF = u1 * p[1] + u2 * p[2];
                const double uxP = u1 * p[3] + u2 * p[4];
                const double uyP = u1 * p[4] + u2 * p[5];
                const double uuP = u1 * uxP + u2 * uyP;
                fE = lor * lor * (p[0] - 2.0 * uF + uuP);
                fFx = lor * lor * (p[1] - lor * p[0] * u1 - uxP + u1 * lor / (1.0 + lor) * ((2.0 * lor + 1.0) * uF - lor * uuP));
                fFy = lor * lor * (p[2] - lor * p[0] * u2 - uyP + u2 * lor / (1.0 + lor) * ((2.0 * lor + 1.0) * uF - lor * uuP));
                iso = false;
            }
            if (iso)
            {
                const double before = src;
                src = adt * (eta + k0 * fE);
                // The same source as in the cycle before (always so without
                // scattering), or in the first cycle nothing to absorb,
                // scatter or emit: the cycle would find the moments that m
                // already holds, and relative changes of 0 (or 0 / 0), which
                // end the iteration.
                if (cycles > 1 ? was_iso && src == before : src == 0.0 && den == 1.0)
                    break;
                const unsigned hs = (unsigned)__double2hiint(src);
                plain = fast_div && most < 0x70000000u && least > 0x0b000000u &&
                        (src == 0.0 || (hs > 0x0b000000u && hs < 0x70000000u));
            }
            m.zero();
            if (iso && plain)
            {
#pragma unroll kCollideUnroll
                for (int d = 0; d < nd; d++)
                {
                    const double2 n = direction(d);
                    m.add(dir[2 * d + 1].x, quotient_plain(streamed(d) + src), n.x, n.y);
                }
            }
            else if (rest)
            {
#pragma unroll 4
                for (int d = 0; d < nd; d++)
                {
                    const double2 n = direction(d);
                    m.add(dir[2 * d + 1].x, value(d, n), n.x, n.y);
                }
            }
            else
                for (int d = 0; d < nd; d++)
                {
                    const double2 n = direction(d);
                    const double v =
                        collide_value(streamed(d), n.x, n.y, u1, u2, lor, adt, eta, k0, k3, kak0, fE, fFx, fFy);
                    m.add(dir[2 * d + 1].x, v, n.x, n.y);
                }
            const double q[6] = {m.E, m.Fx, m.Fy, m.Pxx, m.Pxy, m.Pyy};
            more = still_changing(p, q);
        } while (more && cycles < 100);
        // the last iterate, recomputed from the same operands
        double *out = a.Iout + ij;
        if (iso && plain)
        {
#pragma unroll kCollideUnroll
            for (int d = 0; d < nd; d++)
                out[(int64_t)d * nxy] = quotient_plain(streamed(d) + src);
        }
        else if (rest)
        {
#pragma unroll 4
            for (int d = 0; d < nd; d++)
                out[(int64_t)d * nxy] = value(d, direction(d));
        }
        else
            for (int d = 0; d < nd; d++)
            {
                const double2 n = direction(d);
                out[(int64_t)d * nxy] =
                    collide_value(streamed(d), n.x, n.y, u1, u2, lor, adt, eta, k0, k3, kak0, fE, fFx, fFy);
            }
    }
    if (RECORD && active)
        rec.cycles[cc] = cycles;
    if (active)
    {
        a.mom[ij] = m.E;
        a.mom[ij + nxy] = m.Fx;
        a.mom[ij + 2 * nxy] = m.Fy;
        a.mom[ij + 3 * nxy] = m.Pxx;
        a.mom[ij + 4 * nxy] = m.Pxy;
        a.mom[ij + 5 * nxy] = m.Pyy;
    }
    // lambda-iteration statistics: warp sums and maxima, one atomic per warp
    unsigned sum = (unsigned)cycles, mx = (unsigned)cycles;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
    {
        sum += __shfl_xor_sync(0xffffffffu, sum, o);
        mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    }
    if ((t & 31) == 0 && sum)
    {
        atomicAdd(a.iter_sum, (unsigned long long)sum);
        atomicMax(a.iter_max, mx);
    }
}

// UpdateRotationMatrizes (src/Radiation.cpp:361-378): for the interior cells
// of the slab, the angle of the flux averaged over the 3x3 neighbourhood
// where at least 1% of the light moves along it, else the previous angle.
template <typename T>
__global__ void k_rotation_update(GridDev g, const T *mom, const double *ang_old, double *ang_new)
{
    const int64_t c0 = (g.jlo - 1) * g.nx_;
    const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= (g.jhi - g.jlo) * g.nx_)
        return;
    const int64_t cc = c0 + c;
    const int64_t i = 1 + cc % g.nx_, j = 1 + cc / g.nx_;
    const int64_t ij = i + j * g.nx, nxy = g.nxy;
    double fx = 0.0, fy = 0.0;
    for (int b = -1; b <= 1; b++)
        for (int a = -1; a <= 1; a++)
        {
            const int64_t n = (i + a) + (j + b) * g.nx;
            fx += (double)mom[n + nxy];
            fy += (double)mom[n + 2 * nxy];
        }
    fx /= 9.0;
    fy /= 9.0;
    const double norm = sqrt(fx * fx + fy * fy);
    const double E = (double)mom[ij];
    ang_new[ij] = (E > 1e-16 && norm / E > 0.01) ? approx_phi(fx, fy) : ang_old[ij];
}

// The rotations an adaptive step reads at every node: the inverse of the
// previous one (RotationMatrix(angle).Inverse(), src/DataTypes.hh:625-635,
// as IntensityAt uses it at each corner) and the new one (the cell's own
// stencil), as {sin, cos}.
// V2: double2, or float2 for the precision form (the FP64 values rounded).
template <typename V2>
__global__ void k_rotation_trig(int64_t nxy, const double *ang_old, const double *ang_new, V2 *rot_inv, V2 *rot_new)
{
    using T = decltype(V2::x);
    const int64_t n = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= nxy)
        return;
    const double th = fmod(-ang_old[n] + 2.0 * kPi, 2.0 * kPi);
    rot_inv[n] = V2{(T)approx_sin(th), (T)approx_cos(th)};
    const double tn = ang_new[n];
    rot_new[n] = V2{(T)approx_sin(tn), (T)approx_cos(tn)};
}

// The moments at the halo nodes, which the reference recomputes after every
// stream from intensities it never writes there (zero).
template <typename T>
__global__ void k_zero_halo_moments(GridDev g, T *mom)
{
    const int64_t ij = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (ij >= g.nxy)
        return;
    const int64_t i = ij % g.nx, j = ij / g.nx;
    if (i == 0 || i == g.nx - 1 || j == 0 || j == g.ny - 1)
        for (int q = 0; q < 6; q++)
            mom[ij + q * g.nxy] = (T)0;
}

// Radiation::ComputeMomentsIF (src/Radiation.cpp:239-269): the six moments
// of the current intensities at every node, halo included, in the
// reference's order.  The precision form's state is converted back to I
// (J / (1 / alpha^3)) first.
// With `ang` (adaptive streaming) the directions are the stencil's rotated
// by each node's angle, n1/n2 then holding the unrotated directions.
template <typename T, typename SC>
__global__ void k_moments_from_I(const T *I, int64_t nxy, StateLayout L, int nd, const double *w,
                                 const double *n1, const double *n2, const SC *scale, const double *ang,
                                 double *mom)
{
    const int64_t ij = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (ij >= nxy)
        return;
    double rs = 0.0, rc = 1.0;
    if (ang)
    {
        rs = approx_sin(ang[ij]);
        rc = approx_cos(ang[ij]);
    }
    Moments m;
    m.zero();
    const int64_t sij = L.at(ij);
    for (int d = 0; d < nd; d++)
    {
        const double wd = __ldg(w + d);
        if (wd == 0.0)
            continue;
        double v = (double)I[sij * L.sp + (int64_t)d * L.plane];
        if (scale)
            v = v / (double)scale[ij];
        const double c1 = __ldg(n1 + d), c2 = __ldg(n2 + d);
        if (ang)
            m.add(wd, v, c1 * rc - c2 * rs, c1 * rs + c2 * rc);
        else
            m.add(wd, v, c1, c2);
    }
    mom[ij] = m.E;
    mom[ij + nxy] = m.Fx;
    mom[ij + 2 * nxy] = m.Fy;
    mom[ij + 3 * nxy] = m.Pxx;
    mom[ij + 4 * nxy] = m.Pxy;
    mom[ij + 5 * nxy] = m.Pyy;
}

// Radiation::LoadInitialData for fixed streaming (src/Radiation.cpp:138-181)
template <typename T>
__global__ void k_sources(T *I, StateLayout L, int nd, const int64_t *nodes, const T *vals, int64_t nsrc)
{
    const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (tid >= nsrc * nd)
        return;
    const int64_t s = tid / nd;
    const int d = (int)(tid - s * nd);
    I[L.elem(nodes[s], d)] = vals[tid];
    if (d < L.mirror) // the cell-major state repeats the first directions after the last
        I[L.elem(nodes[s], nd + d)] = vals[tid];
}

// Radiation::ComputeMomentsLF (src/Radiation.cpp:270-301)
template <typename T>
__global__ void k_moments_lf(int64_t nxy, const T *mom, const double *lfp, const uint8_t *bh, double *out)
{
    const int64_t ij = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (ij >= nxy)
        return;
    double o[7] = {0, 0, 0, 0, 0, 0, 0};
    if (!bh[ij])
    {
        const double E = mom[ij], Fx = mom[ij + nxy], Fy = mom[ij + 2 * nxy];
        const double Pxx = mom[ij + 3 * nxy], Pxy = mom[ij + 4 * nxy], Pyy = mom[ij + 5 * nxy];
        const double Tm[9] = {E, Fx, Fy, Fx, Pxx, Pxy, Fy, Pxy, Pyy};
        const double *e = lfp + ij * 12;
        double L[9];
#pragma unroll
        for (int a_ = 0; a_ < 3; a_++)
#pragma unroll
            for (int b = 0; b < 3; b++)
            {
                double s = 0.0;
#pragma unroll
                for (int A = 0; A < 3; A++)
#pragma unroll
                    for (int B = 0; B < 3; B++)
                        s += Tm[3 * A + B] * e[3 * a_ + A] * e[3 * b + B];
                L[3 * a_ + b] = s;
            }
        o[0] = L[0];
        o[1] = L[1];
        o[2] = L[2];
        o[3] = L[4];
        o[4] = L[5];
        o[5] = L[8];
        const double g11 = e[9], g12 = e[10], g22 = e[11];
        // Norm2 (src/SpecialMath.cpp:20-27): sum_i sum_j gamma_ij v_i v_j
        double n2 = 0.0;
        n2 += g11 * o[1] * o[1];
        n2 += g12 * o[1] * o[2];
        n2 += g12 * o[2] * o[1];
        n2 += g22 * o[2] * o[2];
        o[6] = sqrt(fabs(n2));
    }
#pragma unroll
    for (int q = 0; q < 7; q++)
        out[ij + q * nxy] = o[q];
}

// global energy: fixed-order partial sums of interior E, then one block
template <typename T>
__global__ void __launch_bounds__(256) k_energy_partial(GridDev g, const T *E, double *partial)
{
    __shared__ double s[256];
    const int t = threadIdx.x;
    double acc = 0.0;
    const int64_t c0 = (g.jlo - 1) * g.nx_, c1 = (g.jhi - 1) * g.nx_; // the slab's cells
    for (int64_t c = c0 + (int64_t)blockIdx.x * 256 + t; c < c1; c += (int64_t)gridDim.x * 256)
    {
        const int64_t i = 1 + c % g.nx_, j = 1 + c / g.nx_;
        acc += (double)E[i + j * g.nx];
    }
    s[t] = acc;
    __syncthreads();
    for (int w = 128; w > 0; w >>= 1)
    {
        if (t < w)
            s[t] += s[t + w];
        __syncthreads();
    }
    if (t == 0)
        partial[blockIdx.x] = s[0];
}

__global__ void __launch_bounds__(256) k_energy_final(const double *partial, int n, double *out)
{
    __shared__ double s[256];
    const int t = threadIdx.x;
    double acc = 0.0;
    for (int k = t; k < n; k += 256)
        acc += partial[k];
    s[t] = acc;
    __syncthreads();
    for (int w = 128; w > 0; w >>= 1)
    {
        if (t < w)
            s[t] += s[t + w];
        __syncthreads();
    }
    if (t == 0)
        *out = s[0];
}

// Fourier coefficients [5][nxy][nf] -> [5][nf][nxy]
__global__ void k_coef_k_major(const double *coef, double *coef_k, int64_t nxy, int nf)
{
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t per = nxy * nf;
    if (t >= 5 * per)
        return;
    const int64_t q = t / per, r = t - q * per; // r = k * nxy + ij
    const int64_t k = r / nxy, ij = r - k * nxy;
    coef_k[t] = coef[q * per + ij * nf + k];
}

// the boundary's cell-major double [ij][d] <-> a state buffer of layout L
template <class T, class SC>
__global__ void k_to_dirmajor(const double *in, T *out, int64_t nxy, StateLayout L, int nd, const SC *scale)
{
    __shared__ double tile[32][33];
    const int64_t ij0 = (int64_t)blockIdx.x * 32;
    const int d0 = blockIdx.y * 32;
    for (int r = threadIdx.y; r < 32; r += 8)
    {
        const int64_t ij = ij0 + r;
        const int d = d0 + threadIdx.x;
        if (ij < nxy && d < nd)
            tile[r][threadIdx.x] = in[ij * nd + d];
    }
    __syncthreads();
    for (int r = threadIdx.y; r < 32; r += 8)
    {
        const int d = d0 + r;
        const int64_t ij = ij0 + threadIdx.x;
        if (ij < nxy && d < nd)
        {
            const T v = scale ? (T)tile[threadIdx.x][r] * (T)scale[ij] : (T)tile[threadIdx.x][r];
            out[L.elem(ij, d)] = v;
            if (d < L.mirror) // the cell-major state repeats the first directions after the last
                out[L.elem(ij, nd + d)] = v;
        }
    }
}
template <class T, class SC>
__global__ void k_to_cellmajor(const T *in, double *out, int64_t nxy, StateLayout L, int nd, const SC *scale)
{
    __shared__ double tile[32][33];
    const int64_t ij0 = (int64_t)blockIdx.x * 32;
    const int d0 = blockIdx.y * 32;
    for (int r = threadIdx.y; r < 32; r += 8)
    {
        const int d = d0 + r;
        const int64_t ij = ij0 + threadIdx.x;
        if (ij < nxy && d < nd)
            tile[threadIdx.x][r] = scale ? (double)in[L.elem(ij, d)] / (double)scale[ij] : (double)in[L.elem(ij, d)];
    }
    __syncthreads();
    for (int r = threadIdx.y; r < 32; r += 8)
    {
        const int64_t ij = ij0 + r;
        const int d = d0 + threadIdx.x;
        if (ij < nxy && d < nd)
            out[ij * nd + d] = tile[r][threadIdx.x];
    }
}
__global__ void k_widen(const float *in, double *out, int64_t n)
{
    const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k < n)
        out[k] = (double)in[k];
}

inline unsigned nblk(int64_t n, int b) { return (unsigned)((n + b - 1) / b); }
} // namespace

cudaError_t prepare_step_plain(int smem_bytes)
{
    (void)smem_bytes;
    const int patch = (int)patch_smem(kPatchMaxDirs);
    cudaError_t e = cudaSuccess;
    auto limit = [&](const void *f, int bytes) {
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    };
    limit((const void *)k_stream_plain_patch<false, 4>, patch);
    limit((const void *)k_stream_plain_patch<true, 4>, patch);
    limit((const void *)k_stream_plain_patch<false, 6>, patch);
    limit((const void *)k_stream_plain_patch<true, 6>, patch);
    const int column = (int)collide_smem(kColumnMaxDirs, true);
    limit((const void *)k_collide_plain<false, false, true>, column);
    limit((const void *)k_collide_plain<false, false, true, true>, column);
    limit((const void *)k_collide_plain<false, true, true>, column);
    limit((const void *)k_collide_plain<false, true, true, true>, column);
    limit((const void *)k_collide_plain<true, false, true>, column);
    return e;
}
int launch_step_plain(const PlainStepArgs &a, bool curved, cudaStream_t s, const StepRecord *record)
{
    const int64_t cells = (a.g.jhi - a.g.jlo) * a.g.nx_;
    if (cells <= 0)
        return 0;
    const bool adaptive = a.ang_new != nullptr;
    const StepRecord none{};
    const StepRecord &rec = record && !adaptive ? *record : none;
    const unsigned tx = nblk(a.g.nx_, kSplitTileX), ty = nblk(a.g.jhi - a.g.jlo, kSplitTileY);
    const dim3 sgrid(tx, ty, (unsigned)a.nd), sgrid_df((unsigned)a.nd, tx, ty);
    if (adaptive) // UpdateRotationMatrizes from the previous moments, before the stream
    {
        k_rotation_update<double><<<nblk(cells, 128), 128, 0, s>>>(a.g, a.mom, a.ang_old, const_cast<double *>(a.ang_new));
        launch_rotation_trig(a.g.nxy, a.ang_old, a.ang_new, const_cast<double2 *>(a.rot_inv),
                             const_cast<double2 *>(a.rot_new), s);
    }
    // stream
    const dim3 ga = kDirFastestAdaptive ? sgrid_df : sgrid, gf = kDirFastestFixed ? sgrid_df : sgrid;
    if (adaptive && curved)
        k_stream_plain_curved_adaptive<<<dim3(nblk(a.nd, kPDirs) * (unsigned)(a.g.jhi - a.g.jlo), tx), kAdaptiveBlock,
                                         (size_t)5 * a.nf * kSplitTileX * sizeof(double), s>>>(a);
    else if (adaptive)
        k_stream_plain<false, false, true><<<ga, kStepBlock, 0, s>>>(a, rec);
    else if (curved && a.nd <= kPatchMaxDirs && !a.wide)
    {
        const dim3 pgrid(nblk(a.g.nx_, kPatchX), nblk(a.g.jhi - a.g.jlo, kPatchY));
        const size_t sm = patch_smem(a.nd);
        if (a.nd <= kPatchFewDirs)
            record ? k_stream_plain_patch<true, 4><<<pgrid, 4 * kPatchCells, sm, s>>>(a, rec)
                   : k_stream_plain_patch<false, 4><<<pgrid, 4 * kPatchCells, sm, s>>>(a, rec);
        else
            record ? k_stream_plain_patch<true, 6><<<pgrid, 6 * kPatchCells, sm, s>>>(a, rec)
                   : k_stream_plain_patch<false, 6><<<pgrid, 6 * kPatchCells, sm, s>>>(a, rec);
    }
    else if (curved && a.wide) // 64-bit state offsets
        record ? k_stream_plain<true, true, false, true><<<gf, kStepBlock, 0, s>>>(a, rec)
               : k_stream_plain<true, false, false, true><<<gf, kStepBlock, 0, s>>>(a, rec);
    else if (curved)
        record ? k_stream_plain<true, true, false><<<gf, kStepBlock, 0, s>>>(a, rec)
               : k_stream_plain<true, false, false><<<gf, kStepBlock, 0, s>>>(a, rec);
    else
        record ? k_stream_plain<false, true, false><<<gf, kStepBlock, 0, s>>>(a, rec)
               : k_stream_plain<false, false, false><<<gf, kStepBlock, 0, s>>>(a, rec);
    // moments and collide: with each cell's values in shared memory when they fit
    const bool column = a.nd <= (a.fluid == FLUID_MOVING ? kColumnMaxDirsMoving : kColumnMaxDirs);
    const bool general = column && !record && a.fluid != FLUID_AT_REST;
    const dim3 kgrid(tx, column ? nblk(a.g.jhi - a.g.jlo, kColumnTileY) : ty);
    const unsigned kthreads = column ? kSplitTileX * kColumnTileY : kStepBlock;
    const size_t ksmem = collide_smem(a.nd, column);
    if (record && !adaptive)
        column ? k_collide_plain<true, false, true><<<kgrid, kthreads, ksmem, s>>>(a, rec)
               : k_collide_plain<true, false, false><<<kgrid, kthreads, ksmem, s>>>(a, rec);
    else if (!column)
        adaptive ? k_collide_plain<false, true, false><<<kgrid, kthreads, ksmem, s>>>(a, rec)
                 : k_collide_plain<false, false, false><<<kgrid, kthreads, ksmem, s>>>(a, rec);
    else if (adaptive)
        general ? k_collide_plain<false, true, true, true><<<kgrid, kthreads, ksmem, s>>>(a, rec)
                : k_collide_plain<false, true, true><<<kgrid, kthreads, ksmem, s>>>(a, rec);
    else
        general ? k_collide_plain<false, false, true, true><<<kgrid, kthreads, ksmem, s>>>(a, rec)
                : k_collide_plain<false, false, true><<<kgrid, kthreads, ksmem, s>>>(a, rec);
    if (adaptive) // the halo moments, recomputed by the reference from unwritten (zero) intensities
        k_zero_halo_moments<double><<<nblk(a.g.nxy, 256), 256, 0, s>>>(a.g, a.mom);
    return (column ? kCollideColumn : 0) | (general ? kCollideGeneral : 0);
}
void launch_sources64(double *I, int64_t nxy, int nd, const int64_t *nodes, const double *vals, int64_t nsrc,
                      cudaStream_t s)
{
    k_sources<double><<<nblk(nsrc * nd, 256), 256, 0, s>>>(I, StateLayout{nxy, nxy, nxy}, nd, nodes, vals, nsrc);
}
void launch_sources32(float *I, const StateLayout &L, int nd, const int64_t *nodes, const float *vals, int64_t nsrc,
                      cudaStream_t s)
{
    k_sources<float><<<nblk(nsrc * nd, 256), 256, 0, s>>>(I, L, nd, nodes, vals, nsrc);
}
void launch_coef_k_major(const double *coef, double *coef_k, int64_t nxy, int nf, cudaStream_t s)
{
    k_coef_k_major<<<nblk(5 * nxy * nf, 256), 256, 0, s>>>(coef, coef_k, nxy, nf);
}
void launch_rotation_trig(int64_t nxy, const double *ang_old, const double *ang_new, double2 *rot_inv,
                          double2 *rot_new, cudaStream_t s)
{
    k_rotation_trig<<<nblk(nxy, 256), 256, 0, s>>>(nxy, ang_old, ang_new, rot_inv, rot_new);
}
void launch_rotation_trig32(int64_t nxy, const double *ang_old, const double *ang_new, float2 *rot_inv,
                            float2 *rot_new, cudaStream_t s)
{
    k_rotation_trig<<<nblk(nxy, 256), 256, 0, s>>>(nxy, ang_old, ang_new, rot_inv, rot_new);
}
// UpdateRotationMatrizes before, and the halo moments after, an adaptive
// precision-form step (FP32 moments)
void launch_rotation_update32(const GridDev &g, const float *mom, const double *ang_old, double *ang_new,
                              cudaStream_t s)
{
    const int64_t cells = (g.jhi - g.jlo) * g.nx_;
    if (cells > 0)
        k_rotation_update<float><<<nblk(cells, 128), 128, 0, s>>>(g, mom, ang_old, ang_new);
}
void launch_zero_halo_moments32(const GridDev &g, float *mom, cudaStream_t s)
{
    k_zero_halo_moments<float><<<nblk(g.nxy, 256), 256, 0, s>>>(g, mom);
}
void launch_moments_lf64(int64_t nxy, const double *mom, const double *lfp, const uint8_t *bh, double *out,
                         cudaStream_t s)
{
    k_moments_lf<double><<<nblk(nxy, 256), 256, 0, s>>>(nxy, mom, lfp, bh, out);
}
void launch_moments_lf32(int64_t nxy, const float *mom, const double *lfp, const uint8_t *bh, double *out,
                         cudaStream_t s)
{
    k_moments_lf<float><<<nblk(nxy, 256), 256, 0, s>>>(nxy, mom, lfp, bh, out);
}
void launch_energy64(const GridDev &g, const double *E, double *partial, int nblocks, double *out, cudaStream_t s)
{
    k_energy_partial<double><<<nblocks, 256, 0, s>>>(g, E, partial);
    k_energy_final<<<1, 256, 0, s>>>(partial, nblocks, out);
}
void launch_energy32(const GridDev &g, const float *E, double *partial, int nblocks, double *out, cudaStream_t s)
{
    k_energy_partial<float><<<nblocks, 256, 0, s>>>(g, E, partial);
    k_energy_final<<<1, 256, 0, s>>>(partial, nblocks, out);
}
void launch_to_dirmajor64(const double *in, double *out, int64_t nxy, int nd, cudaStream_t s)
{
    k_to_dirmajor<double, double><<<dim3(nblk(nxy, 32), nblk(nd, 32)), dim3(32, 8), 0, s>>>(
        in, out, nxy, StateLayout{nxy, nxy, nxy}, nd, nullptr);
}
void launch_to_dirmajor32(const double *in, float *out, int64_t nxy, const StateLayout &L, int nd,
                          const float *scale, cudaStream_t s)
{
    k_to_dirmajor<float, float><<<dim3(nblk(nxy, 32), nblk(nd, 32)), dim3(32, 8), 0, s>>>(in, out, nxy, L, nd, scale);
}
void launch_to_cellmajor64(const double *in, double *out, int64_t nxy, int nd, cudaStream_t s)
{
    k_to_cellmajor<double, double><<<dim3(nblk(nxy, 32), nblk(nd, 32)), dim3(32, 8), 0, s>>>(
        in, out, nxy, StateLayout{nxy, nxy, nxy}, nd, nullptr);
}
void launch_to_cellmajor32(const float *in, double *out, int64_t nxy, const StateLayout &L, int nd,
                           const float *scale, cudaStream_t s)
{
    k_to_cellmajor<float, float><<<dim3(nblk(nxy, 32), nblk(nd, 32)), dim3(32, 8), 0, s>>>(in, out, nxy, L, nd, scale);
}
void launch_moments_from_I64(const double *I, int64_t nxy, int nd, const double *w, const double *n1,
                             const double *n2, const double *ang, double *mom, cudaStream_t s)
{
    k_moments_from_I<double, double><<<nblk(nxy, 128), 128, 0, s>>>(I, nxy, StateLayout{nxy, nxy, nxy}, nd, w, n1, n2,
                                                                     nullptr, ang, mom);
}
void launch_moments_from_I32(const float *J, int64_t nxy, const StateLayout &L, int nd, const double *w,
                             const double *n1, const double *n2, const float *scale, const double *ang, double *mom,
                             cudaStream_t s)
{
    k_moments_from_I<float, float><<<nblk(nxy, 128), 128, 0, s>>>(J, nxy, L, nd, w, n1, n2, scale, ang, mom);
}
void launch_widen32(const float *in, double *out, int64_t n, cudaStream_t s)
{
    k_widen<<<nblk(n, 256), 256, 0, s>>>(in, out, n);
}
void launch_sources64L(double *I, const StateLayout &L, int nd, const int64_t *nodes, const double *vals,
                       int64_t nsrc, cudaStream_t s)
{
    k_sources<double><<<nblk(nsrc * nd, 256), 256, 0, s>>>(I, L, nd, nodes, vals, nsrc);
}
void launch_to_state64(const double *in, double *out, int64_t nxy, const StateLayout &L, int nd, const double *scale,
                       cudaStream_t s)
{
    k_to_dirmajor<double, double><<<dim3(nblk(nxy, 32), nblk(nd, 32)), dim3(32, 8), 0, s>>>(in, out, nxy, L, nd, scale);
}
void launch_from_state64(const double *in, double *out, int64_t nxy, const StateLayout &L, int nd, const double *scale,
                         cudaStream_t s)
{
    k_to_cellmajor<double, double><<<dim3(nblk(nxy, 32), nblk(nd, 32)), dim3(32, 8), 0, s>>>(in, out, nxy, L, nd, scale);
}
void launch_moments_from_state64(const double *J, int64_t nxy, const StateLayout &L, int nd, const double *w,
                                 const double *n1, const double *n2, const double *scale, double *mom, cudaStream_t s)
{
    k_moments_from_I<double, double><<<nblk(nxy, 128), 128, 0, s>>>(J, nxy, L, nd, w, n1, n2, scale, nullptr, mom);
}
} // namespace grlbm
