// gb2_split.cu -- split-precision instantiation of the fused pair step.
//
// Same kernel source as the FP64 path (gb2_step.cuh) with SPLIT = true:
// neighbour screening, positions, the overlap of each touching pair, walls,
// gravity and the Velocity-Verlet integration stay FP64; the sphere-sphere
// contact chain runs in FP32 on FP64-differenced relative positions and the
// per-atom pair sums are FP32 with Kahan compensation.  This unit is built
// with FMA contraction and the fast FP32 intrinsics allowed; the FP64 unit
// is not.
#include "gb2_step.cuh"

namespace gb2 {

void launch_pair_split(const Dev &D, cudaStream_t st, int shearupdate, int integrate, int fuse_next, int store_f,
                       size_t smem)
{
    launch_pair_step<true>(D, 1, st, shearupdate, integrate, fuse_next, store_f, smem);
}

void launch_tail_split(const Dev &D, bool long_lists, int nblocks, cudaStream_t st, int shearupdate, int integrate,
                       int fuse_next, int store_f)
{
    launch_pair_tail<true>(D, long_lists, nblocks, st, shearupdate, integrate, fuse_next, store_f);
}

}  // namespace gb2
