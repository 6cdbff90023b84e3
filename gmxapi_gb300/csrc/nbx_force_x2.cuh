// The force / energy kernel with the packed pair core (nbx_pair_x2.cuh), instantiated by nbx_force_x2.cu
// (potential-shift and plain cut-off LJ, all shapes) and nbx_force_x2_lj.cu (switch modifiers and LJ-PME,
// the default shape).
#pragma once

#include "nbx_internal.cuh"
#include "nbx_pair_x2.cuh"

namespace nbx
{
namespace
{

constexpr int kForceThreads = 256;

// kDepth: j-stage buffers per warp; kLj as in pair_phys_x2.
template<bool kEnergy, int kCoul, int kDepth, int kBlocks, int kLj>
__global__ void __launch_bounds__(kForceThreads, kBlocks) k_force_x2(DeviceView v, int* work_counter)
{
    pdl_begin();
    // {-6*C6, 12*C12, LJ energy shift of the pair, LJ-PME grid 6*C6 (geometric)} per type pair
    extern __shared__ float4 smem_x2[];
    float4*   nbfp_s = smem_x2;
    const int nt1    = v.ntypes1;
    for (int k = threadIdx.x; k < nt1 * nt1; k += blockDim.x)
    {
        const float2 p = v.nbfp[k];
        // (12C12 cpot12)/12 - (6C6 cpot6)/6 (kernel_gpu_ref.cpp:327-336)
        // LJ-PME grid: sqrt(6 C6_ii) sqrt(6 C6_jj), the reference's nbfp_comb product (geometric rule)
        float c6grid = 0.0f;
        if (kLj == 3)
        {
            const int ti = k / nt1, tj = k % nt1;
            c6grid       = sqrtf(v.nbfp[ti * nt1 + ti].x) * sqrtf(v.nbfp[tj * nt1 + tj].x);
        }
        nbfp_s[k] = make_float4(-p.x, p.y, p.y * v.cpot12 * (1.0f / 12.0f) - p.x * v.cpot6 * (1.0f / 6.0f), c6grid);
    }
    __syncthreads();
    if (v.hdr->status & (kStatusListOverflow | kStatusExclOverflow | kStatusGridOverflow))
    {
        return;
    }
    const unsigned   full = 0xffffffffu;
    const int        lane = threadIdx.x & 31;
    const int        numSci = v.hdr->num_sci;
    JStageP<kDepth>  js;
    WarpSmemX2       w;
    carve_x2<kDepth>(smem_x2 + nt1 * nt1, threadIdx.x >> 5, js, w);
    stage_init_x2(js, lane);
    const PairConstsX2 k = pair_consts_x2(v);
    const SysPtrsX2 p = { v.xq, v.tgrid, v.xqp, v.fnb, v.cj4, v.excl, v.shiftvec, v.fshift };

    __shared__ double e_acc_s[2][kForceThreads];
    double&           e_lj_acc = e_acc_s[0][threadIdx.x];
    double&           e_el_acc = e_acc_s[1][threadIdx.x];
    e_lj_acc                   = 0.0;
    e_el_acc                   = 0.0;
    // excluded-pair and self energies as work items of this queue (LJ-PME keeps its own kernel)
    const int numChunks = kEnergy && kLj != 3 ? v.excl_chunks : 0;
    // the work item in hand: list entry e with its record s, or exclusion chunk e
    int  t = 0, e = 0;
    bool chunk = false;
    Sci  s{};
    auto claim = [&]() {
        if (lane == 0)
        {
            t = atomicAdd(work_counter, 1);
        }
    };
    auto fetch = [&]() {
        t = __shfl_sync(full, t, 0);
        if (t < numSci + numChunks)
        {
            chunk = item_is_chunk(t, numSci, numChunks, e);
            if (!chunk)
            {
                s = v.sci[e];
            }
        }
    };
    claim();
    fetch();
    while (t < numSci + numChunks)
    {
        if (kEnergy && kLj != 3 && chunk)
        {
            const double beta2  = (double)v.beta * (double)v.beta;
            double       excl_s = 0.0;
            for (int i = e * v.excl_atoms + lane; i < min(v.n, (e + 1) * v.excl_atoms); i += 32)
            {
                double dummy_lj = 0.0;
                excl_atom(v, v, i, false, beta2, e_el_acc, excl_s, dummy_lj);
            }
            e_el_acc = fma(excl_s, -(double)v.beta * 1.1283791670955125739, e_el_acc);
            claim();
            fetch();
            continue;
        }
        const Sci si = s;
        if (!process_entry_x2<kEnergy, kCoul, kDepth, kLj>(k, p, si, reinterpret_cast<const char*>(nbfp_s), js, w, nt1, lane,
                                                       v.wait_test_bytes, e_lj_acc, e_el_acc, claim, fetch))
        {
            stage_timeout_x2(js, &v.hdr->status, lane);
            break;
        }
    }
    if (kEnergy)
    {
        // one add per block and energy: all blocks' adds fall on two addresses, where FP64 adds serialise
        // (an add per warp cost about 4 us at the end of every launch)
        __syncthreads();
        if (threadIdx.x < 64)
        {
            const double* acc = e_acc_s[threadIdx.x >> 5];
            double        sum = 0.0;
            for (int i = lane; i < kForceThreads; i += 32)
            {
                sum += acc[i];
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
            {
                sum += __shfl_xor_sync(full, sum, o);
            }
            if (lane == 0 && sum != 0.0)
            {
                atomicAdd(&v.energy[threadIdx.x >> 5], threadIdx.x < 32 ? sum : sum * v.epsfac_d);
            }
        }
    }
}

template<bool kEnergy, int kCoul, int kDepth, int kBlocks, int kLj>
cudaError_t launch_x2(const DeviceView& v, cudaStream_t s, int num_sms, int* counter)
{
    const size_t smem = sizeof(float4) * ((size_t)v.ntypes1 * v.ntypes1
                                          + (size_t)(kForceThreads / 32) * warp_smem_f4_x2<kDepth>());
    cudaError_t e = smem_optin<k_force_x2<kEnergy, kCoul, kDepth, kBlocks, kLj>>(
            smem + sizeof(double) * 2 * kForceThreads, smem);
    if (e != cudaSuccess)
    {
        return e;
    }
    const int blocks = v.force_share ? num_sms * kBlocks * 3 / 4 : num_sms * kBlocks;
    launch_pdl(k_force_x2<kEnergy, kCoul, kDepth, kBlocks, kLj>, blocks, kForceThreads, smem, s, v, counter);
    return cudaGetLastError();
}

// Coulomb flavour of the packed core: 0 reaction field, 1 Ewald, 2 Ewald with the potential shift
// (energies only; forces do not depend on the shift)
inline int coulomb_flavour(const DeviceView& v, bool energy)
{
    if (v.coulomb != 0)
    {
        return 0;
    }
    return (energy && v.sh_ewald != 0.0f) ? 2 : 1;
}

} // namespace
} // namespace nbx
