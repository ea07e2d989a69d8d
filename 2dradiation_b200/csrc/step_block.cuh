// The fixed streaming types' step with one patch per block: the precision
// form (kernels_step32.cu) and the fast FP64 form (kernels_step64.cu).
//
// A block takes a tile of RUN x 8 cells (RUN 8 or 4), stages the tile's
// (RUN + 2) x 10 node patch of the whole state with one TMA tensor copy, and
// its 8 warps then work alone, each on a run of RUN cells of one row:
//   1. stream.  Curved: the lanes take the run's (cell, direction) pairs in
//      order, 32 at a time, so that a direction count off 32 leaves no lane
//      idle and the run's records are one contiguous read.  Flat: a lane takes
//      a direction along the run, and a cell's right-hand nodes are the next
//      one's left-hand ones;
//   2. moments and the lambda iteration: four lanes per cell (h: the parity
//      of the directions summed, e: which three of the six moments);
//   3. store the run's new state, 16 bytes a lane where the directions allow.
// Every value is computed with the operations, in the order, of the
// warp-per-tile kernels (phase 2 there: two lanes per cell, h), so the results
// are the same bits.
//
// Why: there every warp stages a patch of its own, so shared memory holds an
// SM to 12 (FP32) or 8 (FP64) warps at 64 directions and the kernels wait on
// their chains; here 24 (80 registers) and 16 (128).  One patch for 64 cells
// has 100 nodes where four of 4 x 4 cells have 144.  Against the warp-per-tile
// kernels, curved: 400^2 x 64 FP32 83.0 to 82.0 us, fast FP64 163 to 154 us;
// 400^2 x 48 87 to 72 and 146 to 126 us; 237 x 181 x 36 with a moving fluid 53
// to 39 and 92 to 67 us; 200^2 x 32 20.4 to 16.3 and 34.7 to 28.1 us; flat 300^2
// x 64 31.1 to 28.8 and 98 to 56 us; 100^2 x 20 9.3 to 7.2 and 15.3 to 10.2 us.
//
// What bounds it at 400^2 x 64: in FP32 instruction issue (67% busy, 66 M warp
// instructions) and shared-memory reads (71% of the wavefronts); in FP64 the
// shared-memory reads (68%) and the chains of 16 warps.  Tried and left out, at that size: a persistent
// grid with the next patch staged during phases 2 and 3 (FP32 96 us: registers
// spill), and a lane per direction along the run in curved streaming too, its
// taps and weights kept for the next cell where the window and corner stay (91
// us: fewer reads, as many instructions).
#pragma once
#include <algorithm>
#include <type_traits>

#include "device_common.cuh"
#include "step_common.cuh"

namespace grlbm
{
namespace block
{
constexpr int kThreads = 32 * kBlockStepWarps;

// V neighbouring values; the streamed values of a cell start at an even
// element only, the directions and the state at V
template <int V, class T>
__device__ __forceinline__ void load_row(T (&v)[V], const T *p)
{
    using T2 = std::conditional_t<sizeof(T) == 4, float2, double2>;
    if constexpr (V == 1)
        v[0] = p[0];
    else
#pragma unroll
        for (int k = 0; k < V; k += 2)
        {
            const T2 x = *reinterpret_cast<const T2 *>(p + k);
            v[k] = x.x, v[k + 1] = x.y;
        }
}
template <int V, class T>
__device__ __forceinline__ void store_row(T *p, const T (&v)[V])
{
    if constexpr (V == 4)
        *reinterpret_cast<float4 *>(p) = make_float4(v[0], v[1], v[2], v[3]);
    else if constexpr (V == 2)
    {
        std::conditional_t<sizeof(T) == 4, float2, double2> x;
        x.x = v[0], x.y = v[1];
        *reinterpret_cast<decltype(x) *>(p) = x;
    }
    else
        p[0] = v[0];
}

// F, a form: its types T, Args, Table and Rec, and its load (of a record),
// curved, far_curved, flat_tables and flat (one streamed value), moments (a
// lane's three sums), coeffs (the collide map's) and changing (whether the
// iteration goes on).
// SHARE: the grid is cut to a share of the GPU (a batch's launch shapes below
// 0): a block takes every gridDim.x-th tile, copies the tables once, and
// stages its next patch as soon as all of its warps have streamed theirs.  A
// batch step of 64 uneven FP32 problems on shares of 4 GPUs: 1174 us against
// 1338 with a block a tile.
template <class F, bool CURVED, int RUN, bool SHARE>
__global__ void __launch_bounds__(kThreads, F::kMinBlocks)
    k_step_block(const __grid_constant__ typename F::Args a, const __grid_constant__ BlockStep b,
                 const typename F::Table *__restrict__ dtp)
{
    using T = typename F::T;
    using T4 = typename F::T4;
    using T2 = typename F::T2;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    unsigned char *smem = step::align128(smem_raw);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nd = a.nd, dp = a.dp, dps = a.dps, ss = b.ss, px = RUN + 2;
    const int nxn = (int)a.g.nx, nx_ = (int)a.g.nx_;
    T *rowtab = reinterpret_cast<T *>(smem + b.off_rows);
    T *momtab = reinterpret_cast<T *>(smem + b.off_mom); // {w, w n1, w n2, n1, w n1^2, w n1 n2, w n2^2, n2}
    T *n1s = reinterpret_cast<T *>(smem + b.off_dir), *n2s = n1s + b.nd4; // the directions
    T *wmom = reinterpret_cast<T *>(smem + b.off_wmom);
    T *patch = reinterpret_cast<T *>(smem + b.off_patch);
    T *S = reinterpret_cast<T *>(smem + b.off_s) + warp * RUN * ss; // the run's streamed values [cell][direction]
    T4 *map = reinterpret_cast<T4 *>(smem + b.off_map) + warp * RUN; // phase 3's map of each cell
    unsigned *stat = reinterpret_cast<unsigned *>(smem + 16);             // cycles, most cycles, warps done
    const unsigned bar = smem_addr(smem);
    auto stage = [&](int x, int y) { // (thread 0)
        mbar_arrive_expect(bar, (unsigned)(px * (kBlockStepWarps + 2) * dps * (int)sizeof(T)));
        tma_load_4d(smem_addr(patch), &b.map, 0, 0, x, y, bar);
    };
    int tile = (int)blockIdx.x; // SHARE: row after row
    int x0 = (SHARE ? tile % b.tiles_x : tile) * RUN;
    int y0 = (int)a.g.jlo - 1 + (SHARE ? tile / b.tiles_x : (int)blockIdx.y) * kBlockStepWarps;
    if (threadIdx.x == 0)
    {
        mbar_init(bar, 1);
        stage(x0, y0);
        stat[0] = stat[1] = stat[2] = 0u;
    }
    unsigned it_sum = 0u, it_max = 0u, parity = 0u;
    for (bool first = true;; first = false)
    {
        // the warp's run: cells (xw + c, yw), c < ncells, of the interior
        // (lanes of a cell: h, e; with runs of 4 the upper lanes idle in phase 2)
        const int c = lane & 7, h = (lane >> 3) & 1, e = lane >> 4;
        const int xw = x0, yw = y0 + warp;
        const int ncells = yw < (int)a.g.jhi - 1 ? max(0, min(RUN, nx_ - xw)) : 0;
        const int total = ncells * nd;
        const bool cact = c < ncells;
        const int cij = (1 + xw + (cact ? c : 0)) + (1 + (ncells ? yw : y0)) * nxn;
        const int cfl = cact ? (int)a.flags[cij] : 3;
        const typename F::Rec *rp = nullptr;
        typename F::Rec r[2];
        const bool tables = !SHARE || first;
        if (CURVED)
        {
            rp = a.rec + ((size_t)(xw + yw * nx_) * (size_t)nd + (size_t)lane);
#pragma unroll
            for (int k = 0; k < 2; k++)
                r[k] = F::load(rp + 32 * k, lane + 32 * k < total);
            for (int k = tables ? threadIdx.x : b.q * 12; k < b.q * 12; k += kThreads)
            {
                const int row = k / 12, col = k - 12 * row;
                if (col < F::kRow)
                    rowtab[row * F::kRow + col] = __ldg(dtp->rowtab + k);
            }
        }
        for (int k = tables ? threadIdx.x : nd; k < nd; k += kThreads)
        {
            const T *cf = dtp->dirc + 8 * k;
            T *m = momtab + 8 * k;
            m[0] = cf[0], m[1] = cf[1], m[2] = cf[2], m[3] = cf[6];
            m[4] = cf[3], m[5] = cf[4], m[6] = cf[5], m[7] = cf[7];
            n1s[k] = cf[6], n2s[k] = cf[7];
        }
        if (tables && threadIdx.x < 18)
            wmom[threadIdx.x] = __ldg(dtp->wmom + threadIdx.x);
        if (!CURVED)
            F::flat_tables(a, b, *dtp, smem + b.off_flat, x0, y0);
        __syncthreads();
        if (!step::wait_tile(bar, parity, a.fault))
            return;

        // ---- phase 1: stream ----
        const unsigned holes = __ballot_sync(0xffffffffu, lane < 8 && cact && (cfl & 2)); // cells that stream zeros
        const T *wpatch = patch + warp * px * dps;
        const int pdp = px * dps;
        if (CURVED)
        {
            // the run's (cell, direction) pairs in order, 32 at a time
            int cell = 0, d = lane;
            while (d >= nd)
                d -= nd, cell++;
            for (int e0 = 0; e0 < total; e0 += 64)
            {
                typename F::Rec n[2];
#pragma unroll
                for (int k = 0; k < 2; k++)
                    n[k] = F::load(rp + (e0 + 64 + 32 * k), e0 + 64 + 32 * k + lane < total);
#pragma unroll
                for (int k = 0; k < 2; k++)
                {
                    if (e0 + 32 * k + lane < total)
                    {
                        bool far;
                        T v = F::curved(r[k], wpatch + cell * dps, dps, pdp, rowtab, far);
                        if ((holes >> cell) & 1u)
                            v = T(0);
                        else if (far)
                            v = F::far_curved(a, *dtp, xw + 1 + cell, yw + 1, xw + cell + yw * nx_, d);
                        S[cell * ss + d] = v;
                    }
                    d += 32;
                    while (d >= nd)
                        d -= nd, cell++;
                    r[k] = n[k];
                }
            }
        }
        else
        {
            // a lane takes one direction through `span` cells of the run: a cell's
            // right-hand nodes are the next one's left-hand ones
            const int ncols = nd * b.parts, span = RUN / b.parts;
            for (int p0 = 0; p0 < ncols; p0 += 32)
            {
                int d = p0 + lane, from = 0;
                while (d >= nd)
                    d -= nd, from += span;
                const int n = min(span, ncells - from);
                if (p0 + lane < ncols && n > 0)
                    F::flat_run(a, b, *dtp, smem + b.off_flat, wpatch + from * dps, S + from * ss + d, n, dps, pdp, ss,
                                from, warp, xw + 1 + from, yw + 1, d);
            }
        }
        if (SHARE)
        {
            __syncthreads();
            tile += (int)gridDim.x;
            x0 = tile % b.tiles_x * RUN;
            y0 = (int)a.g.jlo - 1 + tile / b.tiles_x * kBlockStepWarps;
            if (threadIdx.x == 0 && tile < b.tiles_x * b.tiles_y)
                stage(x0, y0);
        }
        else
            __syncwarp();

        // ---- phase 2: moments and collide, four lanes per cell ----
        if (cact)
        {
            const unsigned quad = 0x01010101u << c; // the cell's lanes
            const T u1 = __ldg(a.u1 + cij), u2 = __ldg(a.u2 + cij), lor = __ldg(a.lor + cij);
            const T adt = __ldg(a.adt + cij), eta = __ldg(a.eta + cij), k0 = __ldg(a.k0 + cij);
            const T k3 = __ldg(a.k3 + cij), kak0 = __ldg(a.ka + cij) + k0;
            const T scale = CURVED ? __ldg(a.ia3 + cij) : T(1);
            T *Sc = S + c * ss;
            T m[6];
            {
                T own[3];
                F::moments(Sc, momtab + 4 * e, nd, h, quad, own);
#pragma unroll
                for (int q = 0; q < 3; q++)
                {
                    const T other = __shfl_xor_sync(quad, own[q], 16);
                    m[q] = e ? other : own[q];
                    m[3 + q] = e ? own[q] : other;
                }
            }
            T og = T(1), oa = T(0), ob1 = T(0), ob2 = T(0);
            if (!(cfl & 1))
            {
                int cycles = 0;
                const bool rest = (u1 == T(0)) && (u2 == T(0));
                // m_new[q] = A[q] + (eta + k0 fE) B[q] + k3 (fFx C[q] + fFy D[q])
                T A6[6], B6[6], C6[6], D6[6];
                T g0 = T(0), h0 = T(0);
                if (rest)
                {
                    g0 = T(1) / (T(1) + adt * kak0);
                    h0 = adt * g0;
#pragma unroll
                    for (int q = 0; q < 6; q++)
                    {
                        A6[q] = g0 * m[q];
                        B6[q] = h0 * wmom[q];
                        C6[q] = h0 * wmom[6 + q];
                        D6[q] = h0 * wmom[12 + q];
                    }
                }
                else
                {
                    // lane e = 0 sums A and B, lane e = 1 C and D; each computes the
                    // map's coefficients of every second of the directions of its
                    // parity h and hands the other lane's share over
                    T X6[6], Y6[6];
#pragma unroll
                    for (int q = 0; q < 6; q++)
                        X6[q] = Y6[q] = T(0);
                    const unsigned pair = 0x00010001u << (lane & 15); // both lanes of this parity
                    for (int d0 = h; d0 < nd; d0 += 4)
                    {
                        const int dd = min(d0 + 2 * e, nd - 1);
                        const T w = momtab[8 * dd];
                        T g, hh, q1, q2;
                        F::coeffs(n1s[dd], n2s[dd], u1, u2, lor, adt, kak0, g, hh, q1, q2);
                        const T gs = w * g * Sc[dd], wh = w * hh;
                        const T whq1 = wh * q1, whq2 = wh * q2;
                        const T ox = __shfl_xor_sync(pair, e ? gs : whq1, 16), oy = __shfl_xor_sync(pair, e ? wh : whq2, 16);
                        const T x[2] = {e ? ox : gs, e ? whq1 : ox}, y[2] = {e ? oy : wh, e ? whq2 : oy};
#pragma unroll
                        for (int s = 0; s < 2; s++)
                            if (d0 + 2 * s < nd)
                            {
                                const T n1 = n1s[d0 + 2 * s], n2 = n2s[d0 + 2 * s];
                                const T mu[6] = {T(1), n1, n2, n1 * n1, n1 * n2, n2 * n2};
#pragma unroll
                                for (int q = 0; q < 6; q++)
                                {
                                    X6[q] = F::fma(x[s], mu[q], X6[q]);
                                    Y6[q] = F::fma(y[s], mu[q], Y6[q]);
                                }
                            }
                    }
#pragma unroll
                    for (int q = 0; q < 6; q++)
                    {
                        X6[q] += __shfl_xor_sync(quad, X6[q], 8);
                        Y6[q] += __shfl_xor_sync(quad, Y6[q], 8);
                        const T ox = __shfl_xor_sync(quad, X6[q], 16), oy = __shfl_xor_sync(quad, Y6[q], 16);
                        A6[q] = e ? ox : X6[q], B6[q] = e ? oy : Y6[q];
                        C6[q] = e ? X6[q] : ox, D6[q] = e ? Y6[q] : oy;
                    }
                }
                bool changing = true;
                T fE = T(0), fFx = T(0), fFy = T(0);
                while (changing && cycles < 100)
                {
                    cycles++;
                    const T pE = m[0], pFx = m[1], pFy = m[2], pPxx = m[3], pPxy = m[4], pPyy = m[5];
                    const T uF = u1 * pFx + u2 * pFy;
                    const T uxP = u1 * pPxx + u2 * pPxy;
                    const T uyP = u1 * pPxy + u2 * pPyy;
                    const T uuP = u1 * uxP + u2 * uyP;
                    fE = lor * lor * (pE - T(2) * uF + uuP);
                    const T rr = lor / (T(1) + lor) * ((T(2) * lor + T(1)) * uF - lor * uuP);
                    fFx = lor * lor * (pFx - lor * pE * u1 - uxP + u1 * rr);
                    fFy = lor * lor * (pFy - lor * pE * u2 - uyP + u2 * rr);
                    const T ee = eta + k0 * fE;
                    const T prev[6] = {pE, pFx, pFy, pPxx, pPxy, pPyy};
#pragma unroll
                    for (int q = 0; q < 6; q++)
                        m[q] = A6[q] + ee * B6[q] + k3 * (fFx * C6[q] + fFy * D6[q]);
                    changing = F::changing(prev, m);
                }
                // the intensities of the last iterate: at rest the affine map phase
                // 3 applies; a moving fluid's here, every fourth direction a lane
                const T ee = eta + k0 * fE;
                if (rest)
                {
                    og = g0 * scale;
                    oa = h0 * ee * scale;
                    ob1 = h0 * k3 * fFx * scale;
                    ob2 = h0 * k3 * fFy * scale;
                }
                else
                {
                    for (int dd = h + 2 * e; dd < nd; dd += 4)
                    {
                        T g, hh, q1, q2;
                        F::coeffs(n1s[dd], n2s[dd], u1, u2, lor, adt, kak0, g, hh, q1, q2);
                        Sc[dd] = (g * Sc[dd] + hh * (ee + k3 * (q1 * fFx + q2 * fFy))) * scale;
                    }
                }
                if (lane < 8)
                {
                    it_sum += (unsigned)cycles;
                    it_max = max(it_max, (unsigned)cycles);
                }
            }
            else
                og = scale;
            if (h == 0)
#pragma unroll
                for (int q = 0; q < 3; q++)
                    a.mom[(size_t)cij + (size_t)(3 * e + q) * (size_t)a.g.nxy] = e ? m[3 + q] : m[q];
            if (lane < 8)
            {
                T4 o;
                o.x = og, o.y = oa, o.z = ob1, o.w = ob2;
                map[c] = o;
            }
        }
        __syncwarp();

        // ---- phase 3: the run's new state, and the mirrored directions 0..3
        // after each cell's last one ----
        T *out = a.Iout + (size_t)(1 + xw + (1 + yw) * nxn) * (size_t)dp;
        // V directions a lane
        auto store = [&](auto vc) {
            constexpr int V = decltype(vc)::value;
            const int nv = nd / V;
            int k = lane, cl = 0;
            while (k >= nv)
                k -= nv, cl++;
            while (cl < ncells)
            {
                const T4 o = map[cl];
                T v[V], n1[V], n2[V];
                load_row<V>(v, S + cl * ss + V * k);
                load_row<V>(n1, n1s + V * k);
                load_row<V>(n2, n2s + V * k);
#pragma unroll
                for (int s = 0; s < V; s++)
                    v[s] = F::fma(o.x, v[s], F::fma(o.z, n1[s], F::fma(o.w, n2[s], o.y)));
                T *p = out + cl * dp + V * k;
                store_row<V>(p, v);
                if (V * k < kStateMirror)
                    store_row<V>(p + nd, v);
                k += 32;
                while (k >= nv)
                    k -= nv, cl++;
            }
        };
        if (F::kWide == 4 && (nd & 3) == 0)
            store(std::integral_constant<int, F::kWide>{});
        else if ((nd & 1) == 0)
            store(std::integral_constant<int, 2>{});
        else
            store(std::integral_constant<int, 1>{});
        if (!SHARE || tile >= b.tiles_x * b.tiles_y)
            break;
    }

    // the lambda iteration's statistics: the block's last warp adds them
    it_sum = __reduce_add_sync(0xffffffffu, it_sum);
    it_max = __reduce_max_sync(0xffffffffu, it_max);
    if (lane == 0)
    {
        atomicAdd(stat, it_sum);
        atomicMax(stat + 1, it_max);
        __threadfence_block();
        if (atomicAdd(stat + 2, 1u) == kBlockStepWarps - 1u)
        {
            __threadfence_block();
            const unsigned sum = atomicAdd(stat, 0u);
            if (sum)
            {
                atomicAdd(a.iter_sum, (unsigned long long)sum);
                atomicMax(a.iter_max, atomicMax(stat + 1, 0u));
            }
        }
    }
}

// Launches the kernel over the step's tiles: `share` on a grid of b.grid
// blocks where that is fewer than the tiles, else one block a tile: rows of
// tiles lie along the grid's y, as many at a time as that may hold.  Returns
// the blocks launched.
template <class Args, class Table>
int launch_tiles(const void *kernel, const void *share, const Args &a, const BlockStep &b, const Table *dt,
                  cudaStream_t s)
{
    if (b.grid > 0 && b.grid < (int64_t)b.tiles_x * b.tiles_y)
    {
        void *args[] = {const_cast<Args *>(&a), const_cast<BlockStep *>(&b), &dt};
        cudaLaunchKernel(share, dim3(b.grid), dim3(kThreads), args, (size_t)b.smem, s);
        return b.grid;
    }
    for (int first = 0; b.tiles_x > 0 && first < b.tiles_y; first += kMaxGridY)
    {
        Args part = a;
        part.g.jlo += (int64_t)first * kBlockStepWarps;
        void *args[] = {&part, const_cast<BlockStep *>(&b), &dt};
        cudaLaunchKernel(kernel, dim3(b.tiles_x, std::min(b.tiles_y - first, kMaxGridY)), dim3(kThreads), args,
                         (size_t)b.smem, s);
    }
    return b.tiles_x * b.tiles_y;
}

// Row stride of the streamed values: 2 modulo the banks (of T), so that the
// 8 cells and two parities phase 2 reads at once fall in different banks, and
// even, for phase 3's pairs.
template <class T>
int s_stride(int nd)
{
    const int m = 128 / (int)sizeof(T);
    return nd + ((2 - nd) % m + m) % m;
}

// Shared-memory offsets of a tile of 8 rows of `run` cells.
template <class F>
void set_layout(BlockStep &b, int nd, int dps, int q, bool curved, int flat_bytes)
{
    using T = typename F::T;
    auto align = [](int v, int to) { return (v + to - 1) / to * to; };
    b.ss = s_stride<T>(nd);
    b.q = q;
    b.nd4 = align(nd, 4);
    b.off_wmom = 64;
    b.off_rows = align(b.off_wmom + 18 * (int)sizeof(T), 32);
    b.off_mom = align(b.off_rows + (curved ? q * F::kRow * (int)sizeof(T) : 0), 32);
    b.off_dir = align(b.off_mom + 8 * nd * (int)sizeof(T), 32);
    b.off_flat = align(b.off_dir + 2 * b.nd4 * (int)sizeof(T), 32);
    b.off_map = align(b.off_flat + (curved ? 0 : flat_bytes), 32);
    b.off_patch = align(b.off_map + kBlockStepWarps * b.run * 4 * (int)sizeof(T), 128);
    b.off_s = align(b.off_patch + (b.run + 2) * (kBlockStepWarps + 2) * dps * (int)sizeof(T), 128);
    // flat streaming splits the run's cells among lanes where whole runs would
    // leave lanes idle: the fewest cell steps a warp takes, a run's first cell
    // costing twice the others' node reads
    double best = 0.0;
    b.parts = 1;
    for (int p = 1; p <= b.run; p *= 2)
    {
        const double cost = ((nd * p + 31) / 32) * (b.run / p + 0.7);
        if (p == 1 || cost < best)
            best = cost, b.parts = p;
    }
    b.smem = 128 + b.off_s + kBlockStepWarps * b.run * b.ss * (int)sizeof(T);
}
} // namespace block
} // namespace grlbm
