// b200_matvec with BF16 / F32 weights and none of the optional parts: slot sums or an embedding row, one RMS norm, stored or gated pairs.
#include "matvec_core.cuh"

int b200_mv::launch_ext_plain(const b200_matvec_args &a, const Geometry &geo, int spt, int rb, int grid, cudaStream_t st)
{
    return launch_typed<FAM_PLAIN>(a, geo, spt, rb, grid, st);
}
