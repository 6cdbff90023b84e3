// The reciprocal solve of one PME point and its energy / virial sums, shared by the solve kernels
// (nbx_pme.cu) and the fused x pass (nbx_fft_len.cuh).
#pragma once

#include <cuda_runtime.h>

namespace nbx
{

struct PmeDims
{
    int   n[3];
    float rec[3];  // recipbox diagonal: 1 / box edge (invertBoxMatrix, math/invertmatrix.cpp:62-64)
};

// What the Coulomb solve of the x pass needs besides the grid: spline moduli x | y | z, the three scalars
// of solve_pme_yzx, and the energy and virial sums.
struct PmeSolve
{
    PmeDims      d;
    const float* bsp;
    float        elfac, factor, pivol;
    double*      partials;  // [kSolveReplicas][8], zero between solves; nullptr: no energy or virial
};

// Where the kernel that ends an evaluation (the gather) writes the solve's energy and virial.  Its first
// warp sums the replicas: at 120^3 a completion counter and a last block in the x pass cost 8 us.
struct PmeTotals
{
    double* partials;  // nullptr: nothing to write
    double* energy_out;
    double* virial_out;
};

// Copies of the 7 sums that blocks add to (block b to copy b mod 32): FP64 adds on one address
// serialise in L2.
constexpr int kSolveReplicas = 32;

// The block's energy / virial sums: per warp in float (solve_add_warp), after a block barrier per block in
// FP64 added to one of the replicas (solve_add_block).  Blocks of at most 256 threads, a multiple of 32.
__device__ __forceinline__ void solve_add_warp(const float acc[7], double (*red)[8])
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int k = 0; k < 7; k++)
    {
        float v = acc[k];
        for (int o = 16; o > 0; o >>= 1)
        {
            v += __shfl_xor_sync(0xffffffffu, v, o);
        }
        if (lane == 0)
        {
            red[k][warp] = (double)v;
        }
    }
}

__device__ __forceinline__ void solve_add_block(const double (*red)[8], double* partials)
{
    if (threadIdx.x < 7)
    {
        double v = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); w++)
        {
            v += red[threadIdx.x][w];
        }
        atomicAdd(&partials[(blockIdx.x % kSolveReplicas) * 8 + threadIdx.x], v);
    }
}

__device__ __forceinline__ void solve_add(const float acc[7], double* partials)
{
    __shared__ double red[7][8];
    solve_add_warp(acc, red);
    __syncthreads();
    solve_add_block(red, partials);
}

// One warp: the replicas' sums (complete: of an earlier kernel, or behind a completion counter), which
// are cleared for the next solve; energy = 0.5 sum, virial = 0.25 sum.
__device__ __forceinline__ void solve_total(double* partials, double* energy_out, double* virial_out)
{
    const int lane = threadIdx.x & 31;
    double    tot[7];
    for (int k = 0; k < 7; k++)
    {
        double v               = __ldcg(&partials[lane * 8 + k]);
        partials[lane * 8 + k] = 0.0;
        for (int o = 16; o > 0; o >>= 1)
        {
            v += __shfl_xor_sync(0xffffffffu, v, o);
        }
        tot[k] = v;
    }
    if (lane == 0)
    {
        if (energy_out)
        {
            energy_out[0] = 0.5 * tot[0];
        }
        if (virial_out)
        {
            virial_out[0]                 = 0.25 * tot[1];
            virial_out[1] = virial_out[3] = 0.25 * tot[2];
            virial_out[2] = virial_out[6] = 0.25 * tot[3];
            virial_out[4]                 = 0.25 * tot[4];
            virial_out[5] = virial_out[7] = 0.25 * tot[5];
            virial_out[8]                 = 0.25 * tot[6];
        }
    }
}

// A solve on its own (no gather follows): the last block to finish writes the totals.
__device__ __forceinline__ void solve_finish(const float acc[7], double* partials, unsigned int* done,
                                             double* energy_out, double* virial_out)
{
    __shared__ bool last;
    solve_add(acc, partials);
    if (threadIdx.x < 7)
    {
        __threadfence();
    }
    __syncthreads();
    if (threadIdx.x == 0)
    {
        last = atomicAdd(done, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (last && threadIdx.x < 32)
    {
        __threadfence();
        solve_total(partials, energy_out, virial_out);
        if (threadIdx.x == 0)
        {
            *done = 0u;  // ready for the next solve on this stream
        }
    }
}

// One point (kx, ky, kz) != 0 of solve_pme_yzx (pme_solve.cpp:332-587): scales c by eterm and, with
// energies, adds its energy and virial terms to acc.
__device__ __forceinline__ void solve_point(const PmeDims& d, const float* __restrict__ bsp, float elfac, float factor,
                                            float pivol, int kx, int ky, int kz, bool energy, float2& c, float acc[7])
{
    const int   mx    = kx < (d.n[0] + 1) / 2 ? kx : kx - d.n[0];
    const int   my    = ky < (d.n[1] + 1) / 2 ? ky : ky - d.n[1];
    const float mhx   = (float)mx * d.rec[0];
    const float mhy   = (float)my * d.rec[1];
    const float mhz   = (float)kz * d.rec[2];
    const float m2    = mhx * mhx + mhy * mhy + mhz * mhz;
    const float by    = pivol * bsp[d.n[0] + ky];
    const float den   = m2 * bsp[d.n[0] + d.n[1] + kz] * by * bsp[kx];
    const float eterm = elfac / den * expf(-factor * m2);
    if (energy)
    {
        const float corner  = (kz == 0 || kz == (d.n[2] + 1) / 2) ? 0.5f : 1.0f;
        const float struct2 = 2.0f * (c.x * c.x + c.y * c.y);
        const float ets2    = corner * eterm * struct2;
        const float ets2vf  = ets2 * ((factor * m2 + 1.0f) * 2.0f / m2);
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
}

} // namespace nbx
