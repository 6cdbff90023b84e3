// The packed force kernel (nbx_force_x2.cuh) with the LJ switch modifiers and LJ-PME.  One shape: two stage
// buffers per warp and two blocks per SM, the fastest of the unmodified kernel.
#include "nbx_force_x2.cuh"

namespace nbx
{

// lj: 1 force switch, 2 potential switch, 3 LJ-PME
cudaError_t launch_force_x2_lj(const DeviceView& v, int lj, bool energy, cudaStream_t s, int num_sms, int* counter)
{
    using Launch = cudaError_t (*)(const DeviceView&, cudaStream_t, int, int*);
    // [lj - 1][energy][coulomb flavour]
    static const Launch table[3][2][3] = {
        { { launch_x2<false, 0, 2, 2, 1>, launch_x2<false, 1, 2, 2, 1>, launch_x2<false, 1, 2, 2, 1> },
          { launch_x2<true, 0, 2, 2, 1>, launch_x2<true, 1, 2, 2, 1>, launch_x2<true, 2, 2, 2, 1> } },
        { { launch_x2<false, 0, 2, 2, 2>, launch_x2<false, 1, 2, 2, 2>, launch_x2<false, 1, 2, 2, 2> },
          { launch_x2<true, 0, 2, 2, 2>, launch_x2<true, 1, 2, 2, 2>, launch_x2<true, 2, 2, 2, 2> } },
        { { launch_x2<false, 0, 2, 2, 3>, launch_x2<false, 1, 2, 2, 3>, launch_x2<false, 1, 2, 2, 3> },
          { launch_x2<true, 0, 2, 2, 3>, launch_x2<true, 1, 2, 2, 3>, launch_x2<true, 2, 2, 2, 3> } },
    };
    return table[lj - 1][energy ? 1 : 0][coulomb_flavour(v, energy)](v, s, num_sms, counter);
}

} // namespace nbx
