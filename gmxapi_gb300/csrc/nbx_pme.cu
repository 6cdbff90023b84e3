// Smooth particle-mesh Ewald: the reciprocal-space half of the Ewald sum whose
// real-space half is the cluster-pair kernel.
//
// Restates, for one rectangular box on one GPU and pme_order 4, the reference's PME path:
//  - grid sizes (calcFftGrid, src/gromacs/fft/calcgrid.cpp:63-160, with
//    minimalPmeGridSize, src/gromacs/ewald/pme.cpp:488-500);
//  - fractional coordinates and gridline indices (calc_interpolation_idx,
//    src/gromacs/ewald/pme_spread.cpp:65-140 with make_gridindex_to_localindex,
//    pme_grid.cpp:779-830 on one rank: t = n (x / L + 2), index = (int)t mod n);
//  - the B-spline weights and derivatives (CALC_SPLINE(4), pme_spread.cpp:220-266);
//  - spreading q theta_x theta_y theta_z onto the points index + 0..3, periodic
//    (spread_coefficients_bsplines_thread + wrap_periodic_pmegrid);
//  - the spline moduli (make_bspline_moduli / make_dft_mod,
//    src/gromacs/ewald/calculate_spline_moduli.cpp:52-122);
//  - the reciprocal solve with energy and virial (solve_pme_yzx,
//    src/gromacs/ewald/pme_solve.cpp:332-587);
//  - the force gather (gather_f_bsplines / do_fspline,
//    src/gromacs/ewald/pme_gather.cpp:78-360).
// The 3-D real<->complex transforms are hand-written (nbx_fft_len.cuh, nbx_fft.cu; unnormalised
// both ways, like the reference's).  Spreading accumulates with float atomics (16-byte vector reductions
// when nz is a multiple of 4); the energy and the virial terms are summed per warp in
// float and across the grid in FP64.
//
// Layouts in device memory: real grid [nx][ny][nz] (z fastest); half-complex grid
// [nx][ny][nz/2+1] of float2 (the usual real-to-complex layout), so the complex index
// (kx, ky, kz) is the reference's (x, y, z) complex-grid cell with z halved.
#include "../../include/nbnxm_gb300.h"
#include "nbx_internal.cuh"

#include "nbx_fft.cuh"
#include "nbx_pme_solve.cuh"

#include <algorithm>
#include <climits>
#include <cmath>
#include <cstdint>
#include <string>
#include <vector>

namespace
{

constexpr int kOrder = 4;  // pme_order (grid points per dimension and atom)

using nbx::PmeDims;
using nbx::PmeTotals;
using nbx::solve_add;
using nbx::solve_finish;
using nbx::solve_point;

// CALC_SPLINE(4) for the fraction dr: weights th[0..3] and derivatives dth[0..3]
__device__ __forceinline__ void bspline4(float dr, float th[4], float dth[4])
{
    float d0 = 1.0f - dr, d1 = dr, d2;
    d2 = __fmul_rn(__fmul_rn(0.5f, dr), d1);
    d1 = __fmul_rn(0.5f, __fadd_rn(__fmul_rn(dr + 1.0f, d0), __fmul_rn(2.0f - dr, d1)));
    d0 = __fmul_rn(__fmul_rn(0.5f, 1.0f - dr), d0);
    dth[0] = -d0;
    dth[1] = d0 - d1;
    dth[2] = d1 - d2;
    dth[3] = d2;
    const float div = 1.0f / 3.0f;
    th[3]           = __fmul_rn(__fmul_rn(div, dr), d2);
    th[2]           = __fmul_rn(div, __fadd_rn(__fmul_rn(dr + 1.0f, d1), __fmul_rn(3.0f - dr, d2)));
    th[1]           = __fmul_rn(div, __fadd_rn(__fmul_rn(dr + 2.0f, d0), __fmul_rn(2.0f - dr, d1)));
    th[0]           = __fmul_rn(__fmul_rn(div, 1.0f - dr), d0);
}

// gridline index ((int)t mod n) and fraction of one coordinate, t = n (x / L + 2)
__device__ __forceinline__ int interp_index(float x, float rec, int n, float* frac)
{
    const float t  = __fmul_rn((float)n, __fadd_rn(__fmul_rn(x, rec), 2.0f));  // c_pmeMaxUnitcellShift = 2
    const int   ti = (int)floorf(t);  // the reference's truncation for t >= 0
    *frac          = t - (float)ti;
    const int i    = ti % n;
    return i < 0 ? i + n : i;
}

struct AtomSplines
{
    int   i0[3];
    float th[3][kOrder];
    float dth[3][kOrder];
};

__device__ __forceinline__ void atom_splines(const PmeDims& d, const float* x, int a, AtomSplines& s)
{
    for (int k = 0; k < 3; k++)
    {
        float fr;
        s.i0[k] = interp_index(x[3 * a + k], d.rec[k], d.n[k], &fr);
        bspline4(fr, s.th[k], s.dth[k]);
    }
}

__device__ __forceinline__ int wrap_once(int i, int n)
{
    return i >= n ? i - n : i;
}

// Spline data in the reference's test layout: idx [N][3], theta/dtheta [3][N][4].
__global__ void k_pme_splines(PmeDims d, int natoms, const float* x, int* idx, float* theta,
                              float* dtheta)
{
    nbx::pdl_begin();
    const int a = blockIdx.x * blockDim.x + threadIdx.x;
    if (a >= natoms)
    {
        return;
    }
    AtomSplines s;
    atom_splines(d, x, a, s);
    for (int k = 0; k < 3; k++)
    {
        idx[3 * a + k] = s.i0[k];
        for (int o = 0; o < kOrder; o++)
        {
            theta[((size_t)k * natoms + a) * kOrder + o]  = s.th[k][o];
            dtheta[((size_t)k * natoms + a) * kOrder + o] = s.dth[k][o];
        }
    }
}

__device__ __forceinline__ void red_add_v4(float* addr, float a, float b, float c, float d)
{
    asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(addr), "f"(a), "f"(b), "f"(c), "f"(d));
}

// The four z points gz0..gz0+3 of one (x, y) grid row as 16-byte vector reductions:
// with nz a multiple of 4 (and a 16-byte aligned grid) they fall in the aligned blocks
// [gz0 & ~3, +4) and the next one (periodic), which receive the weights shifted by gz0 & 3.
__device__ __forceinline__ void spread_row_v4(float* row, int gz0, int nz, const float w[4])
{
    const int a  = gz0 & 3;
    float*    pa = row + (gz0 - a);
    float*    pb = row + (gz0 - a + 4 == nz ? 0 : gz0 - a + 4);
    switch (a)
    {
        case 0: red_add_v4(pa, w[0], w[1], w[2], w[3]); break;
        case 1:
            red_add_v4(pa, 0.0f, w[0], w[1], w[2]);
            red_add_v4(pb, w[3], 0.0f, 0.0f, 0.0f);
            break;
        case 2:
            red_add_v4(pa, 0.0f, 0.0f, w[0], w[1]);
            red_add_v4(pb, w[2], w[3], 0.0f, 0.0f);
            break;
        default:
            red_add_v4(pa, 0.0f, 0.0f, 0.0f, w[0]);
            red_add_v4(pb, w[1], w[2], w[3], 0.0f);
            break;
    }
}

// x point ix of an atom: adds its 4 x 4 (y, z) weights to the grid.
template<bool kVec>
__device__ __forceinline__ void spread_quarter(const PmeDims& d, int a, int ix, const float* x,
                                               const float* q, float* grid)
{
    const float qa = q[a];
    if (qa == 0.0f)
    {
        return;
    }
    AtomSplines s;
    atom_splines(d, x, a, s);
    const int   gx = wrap_once(s.i0[0] + ix, d.n[0]);
    const float vx = qa * s.th[0][ix];
    int         gz[kOrder];
    for (int iz = 0; iz < kOrder; iz++)
    {
        gz[iz] = wrap_once(s.i0[2] + iz, d.n[2]);
    }
    for (int iy = 0; iy < kOrder; iy++)
    {
        const int   gy  = wrap_once(s.i0[1] + iy, d.n[1]);
        const float vxy = vx * s.th[1][iy];
        float*      row = grid + ((size_t)gx * d.n[1] + gy) * d.n[2];
        float       w[kOrder];
        for (int iz = 0; iz < kOrder; iz++)
        {
            w[iz] = vxy * s.th[2][iz];
        }
        if (kVec)
        {
            spread_row_v4(row, s.i0[2], d.n[2], w);
        }
        else
        {
            for (int iz = 0; iz < kOrder; iz++)
            {
                atomicAdd(&row[gz[iz]], w[iz]);
            }
        }
    }
}

// Four threads per atom (one x point each).
template<bool kVec>
__global__ void k_pme_spread(PmeDims d, int natoms, const float* x, const float* q,
                             float* grid)
{
    nbx::pdl_begin();
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if ((t >> 2) < natoms)
    {
        spread_quarter<kVec>(d, t >> 2, t & 3, x, q, grid);
    }
}

// ---- spreading and gathering by bricks of the grid ----
// With many atoms per grid point the spread above is bound by L2 reductions (28 16-byte reductions
// an atom; 288k atoms on 120^3: 46 us) and the gather by uncoalesced loads (17 us).  Here the atoms are
// filed by the 8 x 8 x 8 brick of grid points that holds their first point.  One warp per brick adds its
// atoms one after another to an 11 x 11 x 11 tile in shared memory that only it touches -- lane (x, y,
// z mod 2) adds two of the 64 points, no atomics, since 32-bit float atomics in shared memory are
// compare-and-swap loops -- and flushes the tile with 3 reductions per row; one block per brick gathers
// from a shared-memory copy of the tile.  A brick holds up to `cap` atoms (2 x the mean + 32); atoms of
// fuller bricks go to a list that takes the direct path.
constexpr int kBrick       = 8;
constexpr int kTile        = kBrick + kOrder - 1;  // 11 points per dimension
constexpr int kTileSy      = 14;                   // tile strides: lanes (x, y, z mod 2) of one atom
constexpr int kTileSx      = 168;                  // fall in 32 distinct banks
constexpr int kTileFloats  = kTile * kTileSx;
constexpr int kBrickWarps  = 4;
constexpr int kGatherThreads = 96;

struct Bricks
{
    int     nb[3];  // bricks per dimension
    int     cap;    // atoms a brick holds
    // [bricks] atoms filed (may exceed cap), [1] length of the overflow list, [1] that length for the
    // gather, which clears the others as it reads them: zero between calls
    int*    count;
    float4* frac;   // [bricks][cap] fractions of the three coordinates and the charge
    int2*   ref;    // [bricks][cap] atom, point within the brick (x * 64 + y * 8 + z)
    int*    over;   // overflow list: atoms
};

__device__ __forceinline__ int brick_count(const Bricks& b)
{
    return b.nb[0] * b.nb[1] * b.nb[2];
}

// Files the atoms by brick and clears the grid (no block adds to it before this kernel has ended).
__global__ void __launch_bounds__(256) k_pme_file(PmeDims d, Bricks b, int natoms, const float* x,
                                                  const float* q, float4* grid4, int n4)
{
    nbx::pdl_begin();
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    for (int i = t; i < n4; i += gridDim.x * blockDim.x)
    {
        grid4[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
    const float qa   = t < natoms ? q[t] : 0.0f;
    const bool  on   = qa != 0.0f;
    const int   lane = threadIdx.x & 31;
    int         i0[3] = { 0, 0, 0 };
    float       fr[3] = { 0.0f, 0.0f, 0.0f };
    int         brick = -1 - lane;
    if (on)
    {
#pragma unroll
        for (int k = 0; k < 3; k++)
        {
            i0[k] = interp_index(x[3 * t + k], d.rec[k], d.n[k], &fr[k]);
        }
        brick = ((i0[0] / kBrick) * b.nb[1] + i0[1] / kBrick) * b.nb[2] + i0[2] / kBrick;
    }
    // one atomic per brick of the warp's atoms (consecutive atoms are mostly neighbours)
    const unsigned peers  = __match_any_sync(0xffffffffu, brick);
    const int      leader = __ffs(peers) - 1;
    int            base   = 0;
    if (on && lane == leader)
    {
        base = atomicAdd(&b.count[brick], __popc(peers));
    }
    const int slot = __shfl_sync(0xffffffffu, base, leader) + __popc(peers & ((1u << lane) - 1u));
    if (!on)
    {
        return;
    }
    if (slot < b.cap)
    {
        const size_t at = (size_t)brick * b.cap + slot;
        b.frac[at]      = make_float4(fr[0], fr[1], fr[2], qa);
        b.ref[at] = make_int2(t, ((i0[0] % kBrick) * kBrick + i0[1] % kBrick) * kBrick + i0[2] % kBrick);
    }
    else
    {
        b.over[atomicAdd(&b.count[brick_count(b)], 1)] = t;
    }
}

// Grid offset of point k (0 .. 11) past the start of a brick, wrapped once.
__device__ __forceinline__ int brick_point(int start, int k, int n)
{
    return wrap_once(start + k, n);
}

struct SpreadWarp
{
    float  tile[kTileFloats];
    float2 wx[32][kOrder];  // {q theta_x, tile offset of the atom's first point (int bits)}
    float  wy[32][kOrder];
    float4 wz[32];          // theta_z 0, 2, 1, 3
};

__global__ void __launch_bounds__(32 * kBrickWarps)
        k_pme_spread_bricks(PmeDims d, Bricks b, const float* x, const float* q, float* grid)
{
    nbx::pdl_begin();
    extern __shared__ float4 spread_smem[];
    SpreadWarp& w     = reinterpret_cast<SpreadWarp*>(spread_smem)[threadIdx.x >> 5];
    const int   lane  = threadIdx.x & 31;
    const int   brick = blockIdx.x * kBrickWarps + (threadIdx.x >> 5);
    const int   nbr   = brick_count(b);
    // overflow atoms: four threads each, straight into the grid
    const int nover = b.count[nbr];
    if (blockIdx.x == 0 && threadIdx.x == 0)
    {
        b.count[nbr + 1] = nover;
    }
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < 4 * nover; i += gridDim.x * blockDim.x)
    {
        spread_quarter<true>(d, b.over[i >> 2], i & 3, x, q, grid);
    }
    const int n = brick < nbr ? min(b.count[brick], b.cap) : 0;
    if (n == 0)
    {
        return;
    }
    for (int i = lane; i < kTileFloats / 4; i += 32)
    {
        reinterpret_cast<float4*>(w.tile)[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
    const int ix = lane >> 3, iy = (lane >> 1) & 3, zh = lane & 1;
    float* const mine = w.tile + ix * kTileSx + iy * kTileSy + zh;
    for (int k0 = 0; k0 < n; k0 += 32)
    {
        __syncwarp();
        if (k0 + lane < n)
        {
            const size_t at = (size_t)brick * b.cap + k0 + lane;
            const float4 fr = b.frac[at];
            const int    l  = b.ref[at].y;
            const float  off =
                    __int_as_float((l >> 6) * kTileSx + ((l >> 3) & 7) * kTileSy + (l & 7));
            float th[kOrder], dth[kOrder];
            bspline4(fr.x, th, dth);
#pragma unroll
            for (int o = 0; o < kOrder; o++)
            {
                w.wx[lane][o] = make_float2(fr.w * th[o], off);
            }
            bspline4(fr.y, th, dth);
#pragma unroll
            for (int o = 0; o < kOrder; o++)
            {
                w.wy[lane][o] = th[o];
            }
            bspline4(fr.z, th, dth);
            w.wz[lane] = make_float4(th[0], th[2], th[1], th[3]);
        }
        __syncwarp();
        const int m = min(32, n - k0);
        // the next atom's weights are read before this atom's points are updated
        float2 ax = w.wx[0][ix];
        float  ay = w.wy[0][iy];
        float2 az = reinterpret_cast<const float2*>(&w.wz[0])[zh];
        for (int k = 0; k < m; k++)
        {
            float* const p   = mine + __float_as_int(ax.y);
            const float  wxy = ax.x * ay;
            const float  w0 = wxy * az.x, w1 = wxy * az.y;
            const int    nx = k + 1 < m ? k + 1 : k;
            ax              = w.wx[nx][ix];
            ay              = w.wy[nx][iy];
            az              = reinterpret_cast<const float2*>(&w.wz[nx])[zh];
            const float t0 = p[0], t1 = p[2];
            p[0] = t0 + w0;
            p[2] = t1 + w1;
            __syncwarp();  // other lanes' points of the next atom may be these
        }
    }
    __syncwarp();
    // flush: row (x, y) as 3 aligned blocks of 4 z points
    const int bz = brick % b.nb[2], by = (brick / b.nb[2]) % b.nb[1], bx = brick / (b.nb[2] * b.nb[1]);
    for (int i = lane; i < kTile * kTile * 3; i += 32)
    {
        const int    row = i / 3, z4 = 4 * (i - 3 * row);
        const int    tx = row / kTile, ty = row - tx * kTile;
        const float* t  = w.tile + tx * kTileSx + ty * kTileSy + z4;
        const float  v0 = t[0], v1 = t[1], v2 = t[2], v3 = z4 == 8 ? 0.0f : t[3];
        if (v0 != 0.0f || v1 != 0.0f || v2 != 0.0f || v3 != 0.0f)
        {
            const int gx = brick_point(bx * kBrick, tx, d.n[0]), gy = brick_point(by * kBrick, ty, d.n[1]);
            const int gz = brick_point(bz * kBrick, z4, d.n[2]);
            red_add_v4(grid + ((size_t)gx * d.n[1] + gy) * d.n[2] + gz, v0, v1, v2, v3);
        }
    }
}

constexpr int kSolveThreads   = 256;
constexpr int kSolveMaxBlocks = 4096;  // one point per thread up to 1M points, grid-stride above
// With energies, 4 blocks per SM (grid-stride): each block adds once to the completion
// counter, and thousands of same-address atomics would serialise in L2.
constexpr int kSolveEnergyBlocksPerSm = 4;

// The x transform of the forward FFT, the solve and the x transform of the backward FFT in one
// pass over the half-complex grid (the x lines are the last forward and the first backward
// transform): block (ky, z-tile) loads the tile [nx][T] of x lines, warp c transforms column c,
// solves its points (kx, ky, kz = tile * T + c) and transforms it back; the energy and virial sums are
// totalled by the gather.  Lengths without a compile-time transform (nbx_fft_len.cuh).
template<bool kEnergy>
__global__ void __launch_bounds__(kSolveThreads, 6) k_pme_fft_x_solve(nbx::FftAxis ax, PmeDims d, float2* cgrid,
                                                                   const float* __restrict__ bsp, float elfac,
                                                                   float factor, float pivol, int ntiles, double* partials)
{
    nbx::pdl_begin();
    constexpr int T    = nbx::kFftTile;
    extern __shared__ float2 xsm[];
    const int     n    = ax.n;  // nx
    const int     nzc  = d.n[2] / 2 + 1;
    float2*       W    = xsm;
    float2*       tile = xsm + n;                  // [n][T + 1]
    float2*       scr  = tile + (size_t)n * (T + 1);  // [T][n]
    const int     ky   = blockIdx.x / ntiles;
    const int     t    = blockIdx.x - ky * ntiles;
    const int     warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const size_t  base = (size_t)ky * nzc + (size_t)t * T;
    const size_t  es   = (size_t)d.n[1] * nzc;
    const int     cols = min(T, nzc - t * T);
    for (int k = threadIdx.x; k < n; k += blockDim.x)
    {
        W[k] = ax.roots[k];
    }
    for (int idx = threadIdx.x; idx < n * T; idx += blockDim.x)
    {
        const int i = idx / T, c = idx - i * T;
        tile[i * (T + 1) + c] = c < cols ? cgrid[base + (size_t)i * es + c] : make_float2(0.0f, 0.0f);
    }
    __syncthreads();
    float acc[7] = { 0, 0, 0, 0, 0, 0, 0 };
    if (warp < cols)
    {
        float2*   col = tile + warp;
        float2*   s   = scr + (size_t)warp * n;
        const int kz  = t * T + warp;
        // forward along x, then the solve on the column wherever the transform left it
        const bool in_s = nbx::fft_line<false>(col, T + 1, s, 1, W, ax, lane);
        float2*    v    = in_s ? s : col;
        const int  vs   = in_s ? 1 : T + 1;
        for (int kx = lane; kx < n; kx += 32)
        {
            if (kx != 0 || ky != 0 || kz != 0)
            {
                float2 c = v[kx * vs];
                solve_point(d, bsp, elfac, factor, pivol, kx, ky, kz, kEnergy, c, acc);
                v[kx * vs] = c;
            }
        }
        __syncwarp();
        // backward along x
        float2*    other = in_s ? col : s;
        const int  os    = in_s ? T + 1 : 1;
        const bool moved = nbx::fft_line<true>(v, vs, other, os, W, ax, lane);
        // the result is in `other` when moved; bring it to the tile column
        if (moved != in_s)
        {
            // result in s
            for (int i = lane; i < n; i += 32)
            {
                col[i * (T + 1)] = s[i];
            }
        }
    }
    __syncthreads();
    for (int idx = threadIdx.x; idx < n * T; idx += blockDim.x)
    {
        const int i = idx / T, c = idx - i * T;
        if (c < cols)
        {
            cgrid[base + (size_t)i * es + c] = tile[i * (T + 1) + c];
        }
    }
    if (kEnergy)
    {
        solve_add(acc, partials);
    }
}

// solve_pme_yzx over the half-complex grid: scales each element by eterm and sums the
// energy and virial terms (energy = 0.5 sum, virial = 0.25 sum).  Per-point terms and
// per-thread / per-warp sums are float (the reference sums them in `real`), per block and
// across blocks FP64 (solve_finish).
__global__ void __launch_bounds__(kSolveThreads) k_pme_solve(PmeDims d, float2* cgrid, const float* __restrict__ bsp,
                                                             float elfac, float factor, float pivol, double* partials,
                                                             unsigned int* done, double* energy_out,
                                                             double* virial_out)
{
    nbx::pdl_begin();
    const bool energy = energy_out || virial_out;
    const int  nzc    = d.n[2] / 2 + 1;
    const int  total  = d.n[0] * d.n[1] * nzc;
    float      acc[7] = { 0, 0, 0, 0, 0, 0, 0 };
    // (kx, ky, kz) of t, advanced by the grid stride with carries instead of divisions
    const int t0     = blockIdx.x * blockDim.x + threadIdx.x;
    const int stride = gridDim.x * blockDim.x;
    int       kz = t0 % nzc, ky = (t0 / nzc) % d.n[1], kx = t0 / (nzc * d.n[1]);
    const int sz = stride % nzc, sy = (stride / nzc) % d.n[1], sx = stride / (nzc * d.n[1]);
    for (int t = t0; t < total; t += stride)
    {
        if (kx != 0 || ky != 0 || kz != 0)
        {
            float2 c = cgrid[t];
            solve_point(d, bsp, elfac, factor, pivol, kx, ky, kz, energy, c, acc);
            cgrid[t] = c;
        }
        kz += sz;
        int carry = 0;
        if (kz >= nzc)
        {
            kz -= nzc;
            carry = 1;
        }
        ky += sy + carry;
        carry = 0;
        if (ky >= d.n[1])
        {
            ky -= d.n[1];
            carry = 1;
        }
        kx += sx + carry;
    }
    if (energy)
    {
        solve_finish(acc, partials, done, energy_out, virial_out);
    }
}

// solve_pme_lj_yzx, geometric combination rule (one grid; pme_solve.cpp:588-915): the
// dispersion influence function eterm = -((1 - 2 b) e^-b + 2 b sqrt(pi) sqrt(b) erfc(sqrt(b))) / D,
// b = pi^2 m^2 / beta_lj^2, D = B_x B_y B_z 3 V / (pi^1.5 beta_lj^3); the k = 0 element is
// scaled too.  Energy and virial sums as in k_pme_solve.
__global__ void __launch_bounds__(kSolveThreads) k_pme_solve_lj(PmeDims d, float2* cgrid,
                                                                const float* __restrict__ bsp, float factor,
                                                                float by_pref, double* partials, unsigned int* done,
                                                                double* energy_out, double* virial_out)
{
    nbx::pdl_begin();
    const bool energy = energy_out || virial_out;
    const int  nzc    = d.n[2] / 2 + 1;
    const int  total  = d.n[0] * d.n[1] * nzc;
    float      acc[7] = { 0, 0, 0, 0, 0, 0, 0 };
    const int  t0     = blockIdx.x * blockDim.x + threadIdx.x;
    const int  stride = gridDim.x * blockDim.x;
    int        kz = t0 % nzc, ky = (t0 / nzc) % d.n[1], kx = t0 / (nzc * d.n[1]);
    const int  sz = stride % nzc, sy = (stride / nzc) % d.n[1], sx = stride / (nzc * d.n[1]);
    for (int t = t0; t < total; t += stride)
    {
        const int   mx    = kx < (d.n[0] + 1) / 2 ? kx : kx - d.n[0];
        const int   my    = ky < (d.n[1] + 1) / 2 ? ky : ky - d.n[1];
        const float mhx   = (float)mx * d.rec[0];
        const float mhy   = (float)my * d.rec[1];
        const float mhz   = (float)kz * d.rec[2];
        const float m2    = mhx * mhx + mhy * mhy + mhz * mhz;
        const float den   = bsp[d.n[0] + d.n[1] + kz] * (by_pref * bsp[d.n[0] + ky]) * bsp[kx];
        const float b     = factor * m2;
        const float e1    = expf(-b);
        const float mk    = sqrtf(b);
        const float e2    = 1.7724538509055159f * mk * erfcf(mk);
        const float eterm = -((1.0f - 2.0f * b) * e1 + 2.0f * b * e2) / den;
        float2      c     = cgrid[t];
        if (energy)
        {
            const float vterm   = 3.0f * (-e1 + e2) / den;
            const float corner  = (kz == 0 || kz == (d.n[2] + 1) / 2) ? 0.5f : 1.0f;
            const float struct2 = 2.0f * (c.x * c.x + c.y * c.y);
            const float ets2    = corner * eterm * struct2;
            const float ets2vf  = corner * 2.0f * factor * vterm * struct2;
            acc[0] += ets2;
            acc[1] += ets2vf * mhx * mhx - ets2;
            acc[2] += ets2vf * mhx * mhy;
            acc[3] += ets2vf * mhx * mhz;
            acc[4] += ets2vf * mhy * mhy - ets2;
            acc[5] += ets2vf * mhy * mhz;
            acc[6] += ets2vf * mhz * mhz - ets2;
        }
        c.x *= eterm;
        c.y *= eterm;
        cgrid[t] = c;
        kz += sz;
        int carry = 0;
        if (kz >= nzc)
        {
            kz -= nzc;
            carry = 1;
        }
        ky += sy + carry;
        carry = 0;
        if (ky >= d.n[1])
        {
            ky -= d.n[1];
            carry = 1;
        }
        kx += sx + carry;
    }
    if (energy)
    {
        solve_finish(acc, partials, done, energy_out, virial_out);
    }
}

// Force of one atom of charge qa from the potential grid (do_fspline + gather_f_bsplines), added to f.
__device__ __forceinline__ void gather_atom(const PmeDims& d, int a, float qa, const float* x,
                                            const float* grid, float* f)
{
    AtomSplines s;
    atom_splines(d, x, a, s);
    int gz[kOrder];
    for (int iz = 0; iz < kOrder; iz++)
    {
        gz[iz] = wrap_once(s.i0[2] + iz, d.n[2]);
    }
    float fx = 0.0f, fy = 0.0f, fz = 0.0f;
    for (int ix = 0; ix < kOrder; ix++)
    {
        const int gx = wrap_once(s.i0[0] + ix, d.n[0]);
        for (int iy = 0; iy < kOrder; iy++)
        {
            const int    gy  = wrap_once(s.i0[1] + iy, d.n[1]);
            const float* row = grid + ((size_t)gx * d.n[1] + gy) * d.n[2];
            float        sz = 0.0f, sdz = 0.0f;
            for (int iz = 0; iz < kOrder; iz++)
            {
                const float g = row[gz[iz]];
                sz            = fmaf(s.th[2][iz], g, sz);
                sdz           = fmaf(s.dth[2][iz], g, sdz);
            }
            fx = fmaf(s.dth[0][ix] * s.th[1][iy], sz, fx);
            fy = fmaf(s.th[0][ix] * s.dth[1][iy], sz, fy);
            fz = fmaf(s.th[0][ix] * s.th[1][iy], sdz, fz);
        }
    }
    f[3 * a + 0] -= qa * (fx * (float)d.n[0] * d.rec[0]);
    f[3 * a + 1] -= qa * (fy * (float)d.n[1] * d.rec[1]);
    f[3 * a + 2] -= qa * (fz * (float)d.n[2] * d.rec[2]);
}

// kLanes 4: four threads per atom, one x point each; 1: a thread per atom.
template<int kLanes>
__global__ void k_pme_gather(PmeDims d, int natoms, const float* x, const float* q,
                             const float* grid, float* f, PmeTotals tot)
{
    nbx::pdl_begin();
    if (tot.partials && blockIdx.x == 0 && threadIdx.x < 32)
    {
        nbx::solve_total(tot.partials, tot.energy_out, tot.virial_out);
    }
    const int   t  = blockIdx.x * blockDim.x + threadIdx.x;
    const int   a  = t / kLanes, ix = t % kLanes;
    const float qa = a < natoms ? q[a] : 0.0f;
    if (kLanes == 1)
    {
        if (qa != 0.0f)
        {
            gather_atom(d, a, qa, x, grid, f);
        }
        return;
    }
    float       fx = 0.0f, fy = 0.0f, fz = 0.0f;
    if (qa != 0.0f)
    {
        AtomSplines s;
        atom_splines(d, x, a, s);
        int gz[kOrder];
        for (int iz = 0; iz < kOrder; iz++)
        {
            gz[iz] = wrap_once(s.i0[2] + iz, d.n[2]);
        }
        auto pick = [ix](const float(&w)[kOrder]) { return ix == 0 ? w[0] : ix == 1 ? w[1] : ix == 2 ? w[2] : w[3]; };
        const float thx = pick(s.th[0]), dthx = pick(s.dth[0]);
        const int   gx  = wrap_once(s.i0[0] + ix, d.n[0]);
#pragma unroll
        for (int iy = 0; iy < kOrder; iy++)
        {
            const int    gy  = wrap_once(s.i0[1] + iy, d.n[1]);
            const float* row = grid + ((size_t)gx * d.n[1] + gy) * d.n[2];
            float        sz = 0.0f, sdz = 0.0f;
#pragma unroll
            for (int iz = 0; iz < kOrder; iz++)
            {
                const float g = row[gz[iz]];
                sz            = fmaf(s.th[2][iz], g, sz);
                sdz           = fmaf(s.dth[2][iz], g, sdz);
            }
            fx = fmaf(dthx * s.th[1][iy], sz, fx);
            fy = fmaf(thx * s.dth[1][iy], sz, fy);
            fz = fmaf(thx * s.th[1][iy], sdz, fz);
        }
    }
#pragma unroll
    for (int o = 1; o < 4; o <<= 1)
    {
        fx += __shfl_xor_sync(0xffffffffu, fx, o);
        fy += __shfl_xor_sync(0xffffffffu, fy, o);
        fz += __shfl_xor_sync(0xffffffffu, fz, o);
    }
    if (qa != 0.0f && ix < 3)
    {
        const float fd = ix == 0 ? fx : ix == 1 ? fy : fz;
        const int   n  = ix == 0 ? d.n[0] : ix == 1 ? d.n[1] : d.n[2];
        const float rc = ix == 0 ? d.rec[0] : ix == 1 ? d.rec[1] : d.rec[2];
        f[3 * a + ix] -= qa * (fd * (float)n * rc);
    }
}

// The same by bricks: a block per brick reads the brick's 11 x 11 x 12 points into shared memory and
// takes its filed atoms, one per thread; the counts are cleared for the next call.
__global__ void __launch_bounds__(kGatherThreads, 10)
        k_pme_gather_bricks(PmeDims d, Bricks b, const float* x, const float* q,
                            const float* grid, float* f, PmeTotals tot)
{
    nbx::pdl_begin();
    __shared__ float tile[kTileFloats];
    const int        nbr = brick_count(b), brick = blockIdx.x;
    const int        n     = min(b.count[brick], b.cap);
    const int        nover = b.count[nbr + 1];
    if (tot.partials && blockIdx.x == 0 && threadIdx.x < 32)
    {
        nbx::solve_total(tot.partials, tot.energy_out, tot.virial_out);
    }
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nover; i += gridDim.x * blockDim.x)
    {
        const int a = b.over[i];
        gather_atom(d, a, q[a], x, grid, f);
    }
    // the first atom's data come in beside the tile
    const size_t first = (size_t)brick * b.cap;
    float4       fr    = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    int2         rf    = make_int2(0, 0);
    if ((int)threadIdx.x < n)
    {
        fr = b.frac[first + threadIdx.x];
        rf = b.ref[first + threadIdx.x];
    }
    const int bz = brick % b.nb[2], by = (brick / b.nb[2]) % b.nb[1], bx = brick / (b.nb[2] * b.nb[1]);
    for (int i = threadIdx.x; i < (n > 0 ? kTile * kTile * 3 : 0); i += kGatherThreads)
    {
        const int    row = i / 3, z4 = 4 * (i - 3 * row);
        const int    tx = row / kTile, ty = row - tx * kTile;
        const int    gx = brick_point(bx * kBrick, tx, d.n[0]), gy = brick_point(by * kBrick, ty, d.n[1]);
        const int    gz = brick_point(bz * kBrick, z4, d.n[2]);
        const float4 g  = *reinterpret_cast<const float4*>(grid + ((size_t)gx * d.n[1] + gy) * d.n[2] + gz);
        float2*      t  = reinterpret_cast<float2*>(tile + tx * kTileSx + ty * kTileSy + z4);
        t[0]            = make_float2(g.x, g.y);
        t[1]            = make_float2(g.z, g.w);
    }
    __syncthreads();
    if (threadIdx.x == 0)
    {
        b.count[brick] = 0;
        if (brick == 0)
        {
            b.count[nbr] = 0;
        }
    }
    for (int k = threadIdx.x; k < n; k += kGatherThreads)
    {
        if (k >= kGatherThreads)
        {
            fr = b.frac[first + k];
            rf = b.ref[first + k];
        }
        float*      fa = f + 3 * (size_t)rf.x;
        const float f0 = fa[0], f1 = fa[1], f2 = fa[2];
        float       thx[kOrder], dx[kOrder], thy[kOrder], dy[kOrder], thz[kOrder], dz[kOrder];
        bspline4(fr.x, thx, dx);
        bspline4(fr.y, thy, dy);
        bspline4(fr.z, thz, dz);
        const float* t = tile + (rf.y >> 6) * kTileSx + ((rf.y >> 3) & 7) * kTileSy + (rf.y & 7);
        float        fx = 0.0f, fy = 0.0f, fz = 0.0f;
#pragma unroll
        for (int ix = 0; ix < kOrder; ix++)
        {
#pragma unroll
            for (int iy = 0; iy < kOrder; iy++)
            {
                float sz = 0.0f, sdz = 0.0f;
#pragma unroll
                for (int iz = 0; iz < kOrder; iz++)
                {
                    const float g = t[ix * kTileSx + iy * kTileSy + iz];
                    sz            = fmaf(thz[iz], g, sz);
                    sdz           = fmaf(dz[iz], g, sdz);
                }
                fx = fmaf(dx[ix] * thy[iy], sz, fx);
                fy = fmaf(thx[ix] * dy[iy], sz, fy);
                fz = fmaf(thx[ix] * thy[iy], sdz, fz);
            }
        }
        fa[0] = f0 - fr.w * (fx * (float)d.n[0] * d.rec[0]);
        fa[1] = f1 - fr.w * (fy * (float)d.n[1] * d.rec[1]);
        fa[2] = f2 - fr.w * (fz * (float)d.n[2] * d.rec[2]);
    }
}

// The solve's totals alone (an evaluation without atoms has no gather).
__global__ void k_pme_totals(PmeTotals tot)
{
    nbx::pdl_begin();
    nbx::solve_total(tot.partials, tot.energy_out, tot.virial_out);
}

// calcFftGrid for one dimension: the smallest listed size with spacing <= the target
int fft_grid_size(float length, float spacing)
{
    static const int init[] = { 6, 8, 10, 12, 14, 16, 20, 24, 25, 28, 32, 36, 40, 42, 44 };
    static const int base[] = { 45, 48, 50, 52, 54, 56, 60, 64, 70, 72, 75, 80, 81, 84 };
    const int        ninit  = (int)(sizeof(init) / sizeof(init[0]));
    const int        nbase  = (int)(sizeof(base) / sizeof(base[0]));
    const int        nmin   = std::max((int)((double)(length / spacing) + 0.999), 2 * (kOrder - 1));
    int              i      = ninit - 1;
    if (init[i] >= nmin)
    {
        while (i > 0 && init[i - 1] >= nmin)
        {
            i--;
        }
        return init[i];
    }
    int fac2 = 1;
    i        = nbase - 1;
    while (fac2 * base[i] < nmin)
    {
        fac2 *= 2;
    }
    int n = 0;
    do
    {
        const int attempt = fac2 * base[i];
        if (((attempt % 4 == 0 && attempt != 140) || attempt == 90) && attempt >= nmin)
        {
            n = attempt;
        }
        i--;
    } while (i > 0);
    return n;
}

// make_bspline_moduli + make_dft_mod for pme_order 4 (spline order 3)
void bspline_moduli(int n, float* mod)
{
    const int splineOrder  = kOrder - 1;
    double    data[kOrder] = { 1.0, 0.0, 0.0, 0.0 };
    for (int k = 2; k <= splineOrder; k++)
    {
        const double div = 1.0 / k;
        for (int m = k - 1; m > 0; m--)
        {
            data[m] = div * ((k - m) * data[m - 1] + (m + 1) * data[m]);
        }
        data[0] = div * data[0];
    }
    for (int i = 0; i < n; i++)
    {
        double sc = 0.0, ss = 0.0;
        for (int j = 0; j < splineOrder; j++)
        {
            const double arg = (2.0 * 3.14159265358979323846 * i * (j + 1)) / n;
            sc += data[j] * std::cos(arg);
            ss += data[j] * std::sin(arg);
        }
        mod[i] = (float)(sc * sc + ss * ss);
    }
    if (splineOrder % 2 == 0 && n % 2 == 0)
    {
        mod[n / 2] = (mod[n / 2 - 1] + mod[n / 2 + 1]) * 0.5f;
    }
}

thread_local std::string g_pme_error;

} // namespace

struct nbx_pme
{
    int          device     = 0;
    cudaStream_t stream     = nullptr;
    bool         own_stream = false;
    PmeDims      d{};
    float        box[3]    = { 0, 0, 0 };
    float        beta      = 0.0f;
    float        epsilon_r = 1.0f;
    int          lj        = 0;  // 1: the Lennard-Jones (dispersion) grid, coefficients sqrt(C6)
    float*       grid      = nullptr;  // real grid [nx][ny][nz]
    float2*      cgrid     = nullptr;  // half-complex grid [nx][ny][nz/2+1]
    float*       bsp       = nullptr;  // spline moduli x | y | z
    double*      sums      = nullptr;  // solve sums [kSolveReplicas][8]: energy + 6 virial terms, zero between solves
    bool         summed    = false;    // a solve has added to the sums and no totals were taken yet
    unsigned*    done      = nullptr;  // blocks of the running solve that have written their partials
    int          num_sms   = 1;
    nbx::FftPlan3 fft{};  // the hand-written 3D real <-> half-complex transform (nbx_fft.cu)
    bool          plan = false;
    bool          fused_smem_ok = false;  // the fused x pass + solve has its shared memory
    // filing of the atoms by grid brick (launch_file), allocated when the first call that takes it runs
    Bricks bricks{};
    int    brick_atoms = 0;      // atoms the filing arrays are sized for
    std::vector<void*> old_bricks;  // smaller arrays, which captured graphs may still use
    bool   filed       = false;  // atoms are filed and the counts not yet cleared by a gather
    bool   by_bricks   = false;  // the last pme_potential went by bricks, and so does its gather
    std::string  err;
};

namespace
{

int pme_error(nbx_pme* p, int code, const std::string& msg)
{
    (p ? p->err : g_pme_error) = msg;
    return code;
}

int cuda_status(nbx_pme* p, cudaError_t e)
{
    return e == cudaSuccess ? NBX_OK : pme_error(p, NBX_ERR_CUDA, cudaGetErrorString(e));
}

size_t real_points(const nbx_pme* p)
{
    return (size_t)p->d.n[0] * p->d.n[1] * p->d.n[2];
}

size_t complex_points(const nbx_pme* p)
{
    return (size_t)p->d.n[0] * p->d.n[1] * (p->d.n[2] / 2 + 1);
}

cudaError_t launch_spread(nbx_pme* p, int natoms, const float* d_x, const float* d_q, float* grid)
{
    cudaError_t e = cudaMemsetAsync(grid, 0, sizeof(float) * real_points(p), p->stream);
    if (e != cudaSuccess || natoms == 0)
    {
        return e;
    }
    const int  blocks = (int)((4LL * natoms + 255) / 256);
    const bool vec    = p->d.n[2] % 4 == 0 && (reinterpret_cast<uintptr_t>(grid) & 15) == 0;
    if (vec)
    {
        nbx::launch_pdl(k_pme_spread<true>, blocks, 256, 0, p->stream, p->d, natoms, d_x, d_q, grid);
    }
    else
    {
        nbx::launch_pdl(k_pme_spread<false>, blocks, 256, 0, p->stream, p->d, natoms, d_x, d_q, grid);
    }
    return cudaGetLastError();
}

// Whether nbx_pme_compute_device files the atoms by brick.  The extra pass over the atoms has to pay, and
// a brick's tile has to be worth its flush: at 85 atoms a brick (water at 0.12 nm) file + spread + gather
// take 6.5 + 17.7 + 16.0 us at 288k atoms with cold caches, spread + gather directly 45.9 + 17.2 us.  Whole
// evaluations by bricks and directly: water of 16 500 atoms 21.5 and 25.2 us, of 13 200 22.9 and 23.3, of 7 500 21.1 and
// 16.6; crystals at 44 to 55 atoms a brick 25.1 and 33.5 us (32 000 atoms), 54.5 and 60.2 (131 072), at 22 atoms a
// brick 26.1 and 31.4 (23 328) but 51.0 and 47.2 (55 296), 87.2 and 75.8 (131 072); atoms in random order at 32 a brick
// 124 and 140 us (300 000).  Rows are flushed in aligned blocks of 4 points, and a tile may wrap once per dimension.
bool use_bricks(const nbx_pme* p, int natoms)
{
    const int* n = p->d.n;
    return natoms >= 16384 && n[2] % 4 == 0 && n[0] >= 16 && n[1] >= 16 && n[2] >= 16
           && (double)natoms * (kBrick * kBrick * kBrick) >= 32.0 * (double)real_points(p);
}

void free_bricks(nbx_pme* p)
{
    cudaFree(p->bricks.frac);
    for (void* b : p->old_bricks)
    {
        cudaFree(b);
    }
    p->old_bricks.clear();
    p->bricks      = Bricks{};
    p->brick_atoms = 0;
    p->filed       = false;
}

// The filing arrays (one allocation) for natoms atoms; false when there is no memory for them: then the
// direct path runs and the arrays that were there stay.
bool alloc_bricks(nbx_pme* p, int natoms)
{
    Bricks b{};
    size_t nbr = 1;
    for (int k = 0; k < 3; k++)
    {
        b.nb[k] = (p->d.n[k] + kBrick - 1) / kBrick;
        nbr *= (size_t)b.nb[k];
    }
    b.cap              = ((int)(2.0 * natoms / (double)nbr) + 32 + 31) / 32 * 32;
    const size_t slots = nbr * (size_t)b.cap;
    const size_t bytes = slots * (sizeof(float4) + sizeof(int2)) + sizeof(int) * ((size_t)natoms + nbr + 2);
    cudaError_t  e     = cudaMalloc(&b.frac, bytes);
    if (e == cudaSuccess)
    {
        b.ref   = reinterpret_cast<int2*>(b.frac + slots);
        b.count = reinterpret_cast<int*>(b.ref + slots);
        b.over  = b.count + nbr + 2;
        e       = cudaMemsetAsync(b.count, 0, sizeof(int) * (nbr + 2), p->stream);
    }
    if (e == cudaSuccess)
    {
        e = cudaFuncSetAttribute(k_pme_spread_bricks, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)(sizeof(SpreadWarp) * kBrickWarps));
    }
    // arrays that are replaced go on to serve the graphs that were captured with them: their counts have to be
    // zero, as a gather leaves them
    if (e == cudaSuccess && p->bricks.frac && p->filed)
    {
        e = cudaMemsetAsync(p->bricks.count, 0, sizeof(int) * (nbr + 1), p->stream);
    }
    if (e != cudaSuccess)
    {
        cudaGetLastError();
        cudaFree(b.frac);
        return false;
    }
    if (p->bricks.frac)
    {
        p->old_bricks.push_back(p->bricks.frac);
    }
    p->bricks      = b;
    p->brick_atoms = natoms;
    p->filed       = false;
    return true;
}

// As alloc_bricks, when the arrays there are too small; nothing is allocated while the stream is being
// captured (the direct path runs then).  The arrays grow by at least half, so that all the replaced ones together
// hold at most twice as many atoms as the present ones.
bool ensure_bricks(nbx_pme* p, int natoms)
{
    if (p->brick_atoms >= natoms)
    {
        return true;
    }
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(p->stream, &capture) != cudaSuccess || capture != cudaStreamCaptureStatusNone)
    {
        cudaGetLastError();
        return false;
    }
    return alloc_bricks(p, (int)std::max<long long>(natoms, std::min(3LL * p->brick_atoms / 2, (long long)INT_MAX)));
}

cudaError_t launch_spread_bricks(nbx_pme* p, int natoms, const float* d_x, const float* d_q, float* grid)
{
    const Bricks& b   = p->bricks;
    const int     nbr = b.nb[0] * b.nb[1] * b.nb[2];
    if (p->filed)
    {
        // an earlier call filed its atoms and failed before its gather
        const cudaError_t e = cudaMemsetAsync(b.count, 0, sizeof(int) * (size_t)(nbr + 1), p->stream);
        if (e != cudaSuccess)
        {
            return e;
        }
    }
    p->filed = true;
    nbx::launch_pdl(k_pme_file, (natoms + 255) / 256, 256, 0, p->stream, p->d, b, natoms, d_x, d_q,
                    reinterpret_cast<float4*>(grid), (int)(real_points(p) / 4));
    nbx::launch_pdl(k_pme_spread_bricks, (nbr + kBrickWarps - 1) / kBrickWarps, 32 * kBrickWarps,
                    sizeof(SpreadWarp) * kBrickWarps, p->stream, p->d, b, d_x, d_q, grid);
    return cudaGetLastError();
}

cudaError_t launch_gather_bricks(nbx_pme* p, const float* d_x, const float* d_q, const float* grid, float* d_f,
                                 const PmeTotals& tot)
{
    const Bricks& b   = p->bricks;
    const int     nbr = b.nb[0] * b.nb[1] * b.nb[2];
    nbx::launch_pdl(k_pme_gather_bricks, nbr, kGatherThreads, 0, p->stream, p->d, b, d_x, d_q, grid, d_f, tot);
    const cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess)
    {
        p->filed = false;
    }
    return e;
}

// Before a solve that adds to the sums: clears what an earlier call left there that ended between its solve and
// its gather, which takes the totals and clears them.
cudaError_t begin_sums(nbx_pme* p)
{
    if (!p->summed)
    {
        return cudaSuccess;
    }
    const cudaError_t e = cudaMemsetAsync(p->sums, 0, sizeof(double) * 8 * nbx::kSolveReplicas, p->stream);
    if (e == cudaSuccess)
    {
        p->summed = false;
    }
    return e;
}

cudaError_t launch_solve(nbx_pme* p, float2* cgrid, double* d_energy, double* d_virial)
{
    if (d_energy || d_virial)
    {
        const cudaError_t e = begin_sums(p);
        if (e != cudaSuccess)
        {
            return e;
        }
    }
    const double vol     = (double)p->box[0] * p->box[1] * p->box[2];
    const int    nc      = (int)complex_points(p);
    const int    cap     = (d_energy || d_virial) ? kSolveEnergyBlocksPerSm * p->num_sms : kSolveMaxBlocks;
    const int    nblocks = std::max(1, std::min((nc + kSolveThreads - 1) / kSolveThreads, cap));
    // factor = pi^2 / beta^2 (pme_solve.cpp:341,602), in float like `real`
    const float  factor  = (float)(M_PI * M_PI) / (p->beta * p->beta);
    if (p->lj)
    {
        // by = 3 V B_y / (pi sqrt(pi) beta^3) (pme_solve.cpp:664)
        const float by_pref = (float)(3.0 * vol / (M_PI * std::sqrt(M_PI) * (double)p->beta * p->beta * p->beta));
        nbx::launch_pdl(k_pme_solve_lj, nblocks, kSolveThreads, 0, p->stream, p->d, cgrid, p->bsp, factor, by_pref,
                        p->sums, p->done, d_energy, d_virial);
        return cudaGetLastError();
    }
    // elfac = ONE_4PI_EPS0 / epsilon_r (pme_solve.cpp:354)
    const float elfac = (float)nbx::one_4pi_eps0() / p->epsilon_r;
    const float pivol = (float)M_PI * (float)vol;
    nbx::launch_pdl(k_pme_solve, nblocks, kSolveThreads, 0, p->stream, p->d, cgrid, p->bsp, elfac, factor, pivol,
                    p->sums, p->done, d_energy, d_virial);
    return cudaGetLastError();
}

// The x pass and the Coulomb solve in one kernel (any length whose line fits the shared memory).
bool fused_x_solve(const nbx_pme* p)
{
    return !p->lj && p->d.n[0] > 1 && (p->fft.len[0] || p->fused_smem_ok);
}

cudaError_t launch_x_solve(nbx_pme* p, double* d_energy, double* d_virial)
{
    if (d_energy || d_virial)
    {
        const cudaError_t e = begin_sums(p);
        if (e != cudaSuccess)
        {
            return e;
        }
        p->summed = true;
    }
    const double vol    = (double)p->box[0] * p->box[1] * p->box[2];
    const float  factor = (float)(M_PI * M_PI) / (p->beta * p->beta);
    const float  elfac  = (float)nbx::one_4pi_eps0() / p->epsilon_r;
    const float  pivol  = (float)M_PI * (float)vol;
    if (p->fft.len[0])
    {
        const nbx::PmeSolve ps = { p->d, p->bsp, elfac, factor, pivol, (d_energy || d_virial) ? p->sums : nullptr };
        p->fft.len[0]->x_solve(p->fft.ax[0].roots, p->cgrid, ps, p->stream);
        return cudaGetLastError();
    }
    const int    nzc    = p->d.n[2] / 2 + 1;
    const int    ntiles = (nzc + nbx::kFftTile - 1) / nbx::kFftTile;
    const size_t smem   = nbx::fft_tiled_smem(p->d.n[0]);
    if (d_energy || d_virial)
    {
        nbx::launch_pdl(k_pme_fft_x_solve<true>, p->d.n[1] * ntiles, kSolveThreads, smem, p->stream, p->fft.ax[0],
                        p->d, p->cgrid, p->bsp, elfac, factor, pivol, ntiles, p->sums);
    }
    else
    {
        nbx::launch_pdl(k_pme_fft_x_solve<false>, p->d.n[1] * ntiles, kSolveThreads, smem, p->stream, p->fft.ax[0],
                        p->d, p->cgrid, p->bsp, elfac, factor, pivol, ntiles, p->sums);
    }
    return cudaGetLastError();
}

constexpr int kGatherLanesAtoms = 32768;

cudaError_t launch_gather(nbx_pme* p, int natoms, const float* d_x, const float* d_q, const float* grid, float* d_f,
                          const PmeTotals& tot = PmeTotals{ nullptr, nullptr, nullptr })
{
    if (natoms > 0)
    {
        // four threads per atom while a thread per atom leaves the GPU waiting for its 64 loads: 3 000 atoms 6.8 ->
        // 4.6 us, 32 000 8.7 -> 7.7 us; from then on the splines, computed four times, cost more (20 steps of 32 000 /
        // 42 592 / 55 296 / 62 500 atoms 1508 / 1697 / 1915 / 2144 us with a thread per atom, 1503 / 1697 / 1946 /
        // 2212 us with four)
        if (natoms <= kGatherLanesAtoms)
        {
            nbx::launch_pdl(k_pme_gather<4>, (4 * natoms + 127) / 128, 128, 0, p->stream, p->d, natoms, d_x, d_q, grid,
                            d_f, tot);
        }
        else
        {
            nbx::launch_pdl(k_pme_gather<1>, (natoms + 127) / 128, 128, 0, p->stream, p->d, natoms, d_x, d_q, grid, d_f,
                            tot);
        }
    }
    else if (tot.partials)
    {
        nbx::launch_pdl(k_pme_totals, 1, 32, 0, p->stream, tot);
    }
    return cudaGetLastError();
}

bool atoms_ok(int natoms, const void* a, const void* b)
{
    return natoms >= 0 && (natoms == 0 || (a && b));
}

} // namespace

extern "C" {

float nbx_ewald_coefficient(float rcoulomb, float ewald_rtol)
{
    if (!(rcoulomb > 0.0f))
    {
        return 0.0f;
    }
    return nbx::calc_ewaldcoeff_q(rcoulomb, ewald_rtol > 0.0f ? ewald_rtol : 1e-5f);
}

int nbx_pme_grid_size(const float* box, float spacing, int* n)
{
    if (!box || !n || !(spacing > 0.0f))
    {
        return pme_error(nullptr, NBX_ERR_INVALID_INPUT, "null argument or non-positive spacing");
    }
    for (int k = 0; k < 3; k++)
    {
        if (!(box[k] > 0.0f))
        {
            return pme_error(nullptr, NBX_ERR_INVALID_INPUT, "box edges must be positive");
        }
        n[k] = fft_grid_size(box[k], spacing);
    }
    return NBX_OK;
}

const char* nbx_pme_last_error(const nbx_pme* p)
{
    return p ? p->err.c_str() : g_pme_error.c_str();
}

int nbx_pme_create(const float* box, const int* grid, float ewaldcoeff_q, float epsilon_r, int device, nbx_pme** out)
{
    if (!box || !grid || !out || !(ewaldcoeff_q > 0.0f))
    {
        return pme_error(nullptr, NBX_ERR_INVALID_INPUT, "null argument or non-positive Ewald coefficient");
    }
    *out = nullptr;
    for (int k = 0; k < 3; k++)
    {
        if (!(box[k] > 0.0f) || grid[k] < 2 * (kOrder - 1) || grid[k] > 4096)
        {
            return pme_error(nullptr, NBX_ERR_INVALID_INPUT,
                             "box edges must be positive and grid sizes in [6, 4096] (minimalPmeGridSize)");
        }
    }
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0)
    {
        cudaGetLastError();
        return pme_error(nullptr, NBX_ERR_NO_DEVICE, "no CUDA device");
    }
    if (device < 0 || device >= ndev)
    {
        return pme_error(nullptr, NBX_ERR_INVALID_INPUT, "device index out of range");
    }
    cudaSetDevice(device);
    nbx_pme* p   = new nbx_pme();
    p->device    = device;
    p->beta      = ewaldcoeff_q;
    p->epsilon_r = epsilon_r > 0.0f ? epsilon_r : 1.0f;
    for (int k = 0; k < 3; k++)
    {
        p->box[k]   = box[k];
        p->d.n[k]   = grid[k];
        p->d.rec[k] = 1.0f / box[k];
    }
    cudaError_t e = cudaStreamCreateWithFlags(&p->stream, cudaStreamNonBlocking);
    p->own_stream = e == cudaSuccess;
    if (e == cudaSuccess) e = cudaMalloc(&p->grid, sizeof(float) * real_points(p));
    if (e == cudaSuccess) e = cudaMalloc(&p->cgrid, sizeof(float2) * complex_points(p));
    if (e == cudaSuccess) e = cudaMalloc(&p->bsp, sizeof(float) * (grid[0] + grid[1] + grid[2]));
    if (e == cudaSuccess) e = cudaMalloc(&p->sums, sizeof(double) * 8 * nbx::kSolveReplicas);
    if (e == cudaSuccess) e = cudaMemset(p->sums, 0, sizeof(double) * 8 * nbx::kSolveReplicas);
    if (e == cudaSuccess) e = cudaMalloc(&p->done, sizeof(unsigned));
    if (e == cudaSuccess) e = cudaMemset(p->done, 0, sizeof(unsigned));
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&p->num_sms, cudaDevAttrMultiProcessorCount, device);
    if (e == cudaSuccess)
    {
        std::vector<float> mod(grid[0] + grid[1] + grid[2]);
        bspline_moduli(grid[0], mod.data());
        bspline_moduli(grid[1], mod.data() + grid[0]);
        bspline_moduli(grid[2], mod.data() + grid[0] + grid[1]);
        e = cudaMemcpy(p->bsp, mod.data(), sizeof(float) * mod.size(), cudaMemcpyHostToDevice);
    }
    if (e != cudaSuccess)
    {
        const std::string msg = cudaGetErrorString(e);
        nbx_pme_destroy(p);
        return pme_error(nullptr, NBX_ERR_OUT_OF_MEMORY, "PME allocation: " + msg);
    }
    const cudaError_t fe = nbx::fft_plan_create(&p->fft, grid);
    p->plan              = (fe == cudaSuccess);
    if (p->plan)
    {
        const size_t xs  = nbx::fft_tiled_smem(grid[0]);
        p->fused_smem_ok = xs <= 48 * 1024
                           || (cudaFuncSetAttribute(k_pme_fft_x_solve<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                    (int)xs) == cudaSuccess
                               && cudaFuncSetAttribute(k_pme_fft_x_solve<false>,
                                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)xs) == cudaSuccess);
    }
    if (!p->plan)
    {
        nbx_pme_destroy(p);
        return pme_error(nullptr, fe == cudaErrorInvalidValue ? NBX_ERR_INVALID_INPUT : NBX_ERR_CUDA,
                         fe == cudaErrorInvalidValue
                                 ? "FFT grid size: every dimension must be at most 1024 with prime factors of at most 255"
                                 : std::string("FFT plan: ") + cudaGetErrorString(fe));
    }
    // the filing arrays for a box at the density of a condensed system (110 atoms per nm^3), so that the
    // first call does not allocate; larger calls grow them, boxes above 4M atoms allocate on first use
    const double atoms = 110.0 * box[0] * box[1] * box[2];
    if (atoms <= 4.0e6 && use_bricks(p, (int)atoms))
    {
        alloc_bricks(p, (int)atoms);
    }
    *out = p;
    return NBX_OK;
}

int nbx_pme_create_lj(const float* box, const int* grid, float ewaldcoeff_lj, int device, nbx_pme** out)
{
    const int rc = nbx_pme_create(box, grid, ewaldcoeff_lj, 1.0f, device, out);
    if (rc == NBX_OK)
    {
        (*out)->lj = 1;
    }
    return rc;
}

float nbx_ewald_coefficient_lj(float rvdw, float ewald_rtol_lj)
{
    // calc_ewaldcoeff_lj (ewald/ewald_utils.cpp:76-115): exp(-x^2)(1 + x^2 + x^4/2) = rtol, x = beta rc
    if (!(rvdw > 0.0f))
    {
        return 0.0f;
    }
    const float rtol = ewald_rtol_lj > 0.0f ? ewald_rtol_lj : 1e-3f;
    auto        f    = [rvdw](float beta) {
        const float x2 = (beta * rvdw) * (beta * rvdw);
        return std::exp(-x2) * (1.0f + x2 + x2 * x2 / 2.0f);
    };
    float beta = 5.0f;
    int   i    = 0;
    do
    {
        i++;
        beta *= 2.0f;
    } while (f(beta) > rtol);
    const int n    = i + 60;
    float     low  = 0.0f, high = beta;
    for (i = 0; i < n; i++)
    {
        beta = (low + high) / 2.0f;
        if (f(beta) > rtol)
        {
            low = beta;
        }
        else
        {
            high = beta;
        }
    }
    return beta;
}

int nbx_pme_destroy(nbx_pme* p)
{
    if (!p)
    {
        return NBX_OK;
    }
    cudaSetDevice(p->device);
    if (p->stream)
    {
        cudaStreamSynchronize(p->stream);
    }
    if (p->plan)
    {
        nbx::fft_plan_destroy(&p->fft);
    }
    free_bricks(p);
    cudaFree(p->grid);
    cudaFree(p->cgrid);
    cudaFree(p->bsp);
    cudaFree(p->sums);
    cudaFree(p->done);
    if (p->own_stream)
    {
        cudaStreamDestroy(p->stream);
    }
    delete p;
    return NBX_OK;
}

int nbx_pme_set_stream(nbx_pme* p, void* s)
{
    if (!p)
    {
        return pme_error(nullptr, NBX_ERR_INVALID_INPUT, "null handle");
    }
    if (static_cast<cudaStream_t>(s) == p->stream)
    {
        return NBX_OK;
    }
    cudaSetDevice(p->device);
    cudaStreamSynchronize(p->stream);
    if (p->own_stream)
    {
        cudaStreamDestroy(p->stream);
    }
    p->stream     = static_cast<cudaStream_t>(s);
    p->own_stream = false;
    return NBX_OK;
}

int nbx_pme_get_info(const nbx_pme* p, int* grid, float* ewaldcoeff_q)
{
    if (!p)
    {
        return pme_error(nullptr, NBX_ERR_INVALID_INPUT, "null handle");
    }
    for (int k = 0; k < 3 && grid; k++)
    {
        grid[k] = p->d.n[k];
    }
    if (ewaldcoeff_q)
    {
        *ewaldcoeff_q = p->beta;
    }
    return NBX_OK;
}

int nbx_pme_splines_device(nbx_pme* p, int natoms, const float* d_x, int* d_idx, float* d_theta, float* d_dtheta)
{
    if (!p || !atoms_ok(natoms, d_x, d_idx) || (natoms > 0 && (!d_theta || !d_dtheta)))
    {
        return pme_error(p, NBX_ERR_INVALID_INPUT, "null argument or negative atom count");
    }
    cudaSetDevice(p->device);
    if (natoms == 0)
    {
        return NBX_OK;
    }
    nbx::launch_pdl(k_pme_splines, (natoms + 127) / 128, 128, 0, p->stream, p->d, natoms, d_x, d_idx, d_theta,
                    d_dtheta);
    return cuda_status(p, cudaGetLastError());
}

int nbx_pme_spread_device(nbx_pme* p, int natoms, const float* d_x, const float* d_q, float* d_grid)
{
    if (!p || !atoms_ok(natoms, d_x, d_q) || !d_grid)
    {
        return pme_error(p, NBX_ERR_INVALID_INPUT, "null argument or negative atom count");
    }
    cudaSetDevice(p->device);
    return cuda_status(p, launch_spread(p, natoms, d_x, d_q, d_grid));
}

int nbx_pme_solve_device(nbx_pme* p, void* d_cgrid, double* d_energy, double* d_virial)
{
    if (!p || !d_cgrid)
    {
        return pme_error(p, NBX_ERR_INVALID_INPUT, "null argument");
    }
    cudaSetDevice(p->device);
    return cuda_status(p, launch_solve(p, static_cast<float2*>(d_cgrid), d_energy, d_virial));
}

int nbx_pme_gather_device(nbx_pme* p, int natoms, const float* d_x, const float* d_q, const float* d_grid, float* d_f)
{
    if (!p || !atoms_ok(natoms, d_x, d_q) || !d_grid || (natoms > 0 && !d_f))
    {
        return pme_error(p, NBX_ERR_INVALID_INPUT, "null argument or negative atom count");
    }
    cudaSetDevice(p->device);
    return cuda_status(p, launch_gather(p, natoms, d_x, d_q, d_grid, d_f));
}

struct nbx_fft3d
{
    int           device = 0;
    nbx::FftPlan3 plan{};
};

int nbx_fft3d_create(const int* grid, int device, nbx_fft3d** out)
{
    if (!grid || !out)
    {
        return pme_error(nullptr, NBX_ERR_INVALID_INPUT, "null argument");
    }
    *out = nullptr;
    if (cudaSetDevice(device) != cudaSuccess)
    {
        return pme_error(nullptr, NBX_ERR_NO_DEVICE, "no CUDA device " + std::to_string(device));
    }
    auto*             f = new nbx_fft3d;
    f->device           = device;
    const cudaError_t e = nbx::fft_plan_create(&f->plan, grid);
    if (e != cudaSuccess)
    {
        nbx::fft_plan_destroy(&f->plan);
        delete f;
        return pme_error(nullptr, e == cudaErrorInvalidValue ? NBX_ERR_INVALID_INPUT : NBX_ERR_CUDA,
                         e == cudaErrorInvalidValue
                                 ? "FFT grid size: every dimension must be at most 1024 with prime factors of at most 255"
                                 : std::string("FFT plan: ") + cudaGetErrorString(e));
    }
    *out = f;
    return NBX_OK;
}

int nbx_fft3d_destroy(nbx_fft3d* f)
{
    if (f)
    {
        cudaSetDevice(f->device);
        nbx::fft_plan_destroy(&f->plan);
        delete f;
    }
    return NBX_OK;
}

int nbx_fft3d_execute_device(nbx_fft3d* f, int direction, float* d_real, void* d_cgrid, void* stream)
{
    if (!f || !d_real || !d_cgrid || (direction != 1 && direction != -1))
    {
        return pme_error(nullptr, NBX_ERR_INVALID_INPUT, "null argument or direction other than +1 / -1");
    }
    cudaSetDevice(f->device);
    const auto        s = static_cast<cudaStream_t>(stream);
    const cudaError_t e = direction > 0 ? nbx::fft_r2c(f->plan, d_real, static_cast<float2*>(d_cgrid), s)
                                        : nbx::fft_c2r(f->plan, static_cast<float2*>(d_cgrid), d_real, s);
    return e == cudaSuccess ? NBX_OK : pme_error(nullptr, NBX_ERR_CUDA, cudaGetErrorString(e));
}

int nbx_pme_fft_device(nbx_pme* p, int direction, float* d_real, void* d_cgrid)
{
    if (!p || !d_real || !d_cgrid || (direction != 1 && direction != -1))
    {
        return pme_error(p, NBX_ERR_INVALID_INPUT, "null argument or direction other than +1 / -1");
    }
    cudaSetDevice(p->device);
    const cudaError_t e = direction > 0 ? nbx::fft_r2c(p->fft, d_real, static_cast<float2*>(d_cgrid), p->stream)
                                        : nbx::fft_c2r(p->fft, static_cast<float2*>(d_cgrid), d_real, p->stream);
    return cuda_status(p, e);
}

int nbx_pme_compute_device(nbx_pme* p, int natoms, const float* d_x, const float* d_q, float* d_f, double* d_energy,
                           double* d_virial)
{
    if (!p || !atoms_ok(natoms, d_x, d_q) || (natoms > 0 && !d_f))
    {
        return pme_error(p, NBX_ERR_INVALID_INPUT, "null argument or negative atom count");
    }
    const int rc = nbx::pme_potential(p, natoms, d_x, d_q, d_energy, d_virial, p->stream);
    return rc == NBX_OK ? nbx::pme_forces(p, natoms, d_x, d_q, d_f, d_energy, d_virial) : rc;
}

} // extern "C"

namespace nbx
{

int pme_potential(nbx_pme* p, int natoms, const float* d_x, const float* d_q, double* d_energy, double* d_virial,
                  cudaStream_t s)
{
    cudaSetDevice(p->device);
    const cudaStream_t keep = p->stream;
    p->stream               = s;
    const bool  bricks      = use_bricks(p, natoms) && ensure_bricks(p, natoms);
    cudaError_t e           = bricks ? launch_spread_bricks(p, natoms, d_x, d_q, p->grid)
                                     : launch_spread(p, natoms, d_x, d_q, p->grid);
    p->by_bricks            = bricks;
    if (fused_x_solve(p))
    {
        // z and y forward, then x forward + solve + x backward in one pass, then y and z backward
        if (e == cudaSuccess) e = nbx::fft_r2c_zy(p->fft, p->grid, p->cgrid, p->stream);
        if (e == cudaSuccess) e = launch_x_solve(p, d_energy, d_virial);
        if (e == cudaSuccess) e = nbx::fft_c2r_yz(p->fft, p->cgrid, p->grid, p->stream);
    }
    else
    {
        if (e == cudaSuccess) e = nbx::fft_r2c(p->fft, p->grid, p->cgrid, p->stream);
        if (e == cudaSuccess) e = launch_solve(p, p->cgrid, d_energy, d_virial);
        if (e == cudaSuccess) e = nbx::fft_c2r(p->fft, p->cgrid, p->grid, p->stream);
    }
    p->stream = keep;
    return cuda_status(p, e);
}

int pme_forces(nbx_pme* p, int natoms, const float* d_x, const float* d_q, float* d_f, double* d_energy,
               double* d_virial)
{
    PmeTotals tot = { nullptr, nullptr, nullptr };
    if (fused_x_solve(p) && (d_energy || d_virial))
    {
        tot = { p->sums, d_energy, d_virial };
    }
    const cudaError_t e = p->by_bricks ? launch_gather_bricks(p, d_x, d_q, p->grid, d_f, tot)
                                       : launch_gather(p, natoms, d_x, d_q, p->grid, d_f, tot);
    if (e == cudaSuccess && tot.partials)
    {
        p->summed = false;
    }
    return cuda_status(p, e);
}

} // namespace nbx

extern "C" {

int nbx_pme_synchronize(nbx_pme* p)
{
    if (!p)
    {
        return pme_error(nullptr, NBX_ERR_INVALID_INPUT, "null handle");
    }
    cudaSetDevice(p->device);
    return cuda_status(p, cudaStreamSynchronize(p->stream));
}

} // extern "C"
