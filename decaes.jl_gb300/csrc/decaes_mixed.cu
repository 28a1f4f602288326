// decaes_mixed.cu -- the voxel-solve kernel with the mixed-precision method only: single-volume launches
// and batched / served launches whose volumes all use that method run these
// kernels (half the code of the kernels that carry both methods).  A separate
// translation unit, compiled in parallel with the others.  512 threads: one block
// holds up to 16 warps, as many as an SM's registers and shared memory take.
#define DECAES_METHODS 2
#include "voxel_kernels.cuh"

namespace dk {

__global__ void __launch_bounds__(512) k_voxels_mixed(const __grid_constant__ Params P) { voxels_body(P); }
__global__ void __launch_bounds__(512) k_voxels_batch_mixed(const __grid_constant__ BatchParams B) { voxels_batch_body(B); }

}  // namespace dk
