// Cluster-pair LJ + Ewald real-space (or reaction-field) force / energy kernel with the packed
// pair core (nbx_pair_x2.cuh): two atom pairs per lane in FP32x2 arithmetic.
//
// Physics of the reference's GPU-layout kernels
// (src/gromacs/nbnxm/kernels_reference/kernel_gpu_ref.cpp:57-379), potential-shift or plain
// cut-off LJ here; the switch modifiers and LJ-PME in nbx_force_x2_lj.cu.
// The launch, work queue, excluded-pair energy items and FP64 energy sums are those of that
// kernel; the shapes (j-stage buffers per warp, blocks per SM) are template parameters chosen at
// run time (nbx_set_force_kernel, the batched autotuner).
#include "nbx_force_x2.cuh"

namespace nbx
{

// potential shift and plain cut-off
cudaError_t launch_force_x2(const DeviceView& v, bool energy, cudaStream_t s, int num_sms, int* counter)
{
    using Launch = cudaError_t (*)(const DeviceView&, cudaStream_t, int, int*);
    // [blocks 2, 3][depth 2, 3][energy][coulomb flavour]
    static const Launch table[2][2][2][3] = {
        { { { launch_x2<false, 0, 2, 2, 0>, launch_x2<false, 1, 2, 2, 0>, launch_x2<false, 1, 2, 2, 0> },
            { launch_x2<true, 0, 2, 2, 0>, launch_x2<true, 1, 2, 2, 0>, launch_x2<true, 2, 2, 2, 0> } },
          { { launch_x2<false, 0, 3, 2, 0>, launch_x2<false, 1, 3, 2, 0>, launch_x2<false, 1, 3, 2, 0> },
            { launch_x2<true, 0, 3, 2, 0>, launch_x2<true, 1, 3, 2, 0>, launch_x2<true, 2, 3, 2, 0> } } },
        { { { launch_x2<false, 0, 2, 3, 0>, launch_x2<false, 1, 2, 3, 0>, launch_x2<false, 1, 2, 3, 0> },
            { launch_x2<true, 0, 2, 3, 0>, launch_x2<true, 1, 2, 3, 0>, launch_x2<true, 2, 2, 3, 0> } },
          { { launch_x2<false, 0, 3, 3, 0>, launch_x2<false, 1, 3, 3, 0>, launch_x2<false, 1, 3, 3, 0> },
            { launch_x2<true, 0, 3, 3, 0>, launch_x2<true, 1, 3, 3, 0>, launch_x2<true, 2, 3, 3, 0> } } },
    };
    return table[v.force_blocks == 3 ? 1 : 0][v.stage_depth == 3 ? 1 : 0][energy ? 1 : 0][coulomb_flavour(v, energy)](
            v, s, num_sms, counter);
}

} // namespace nbx
