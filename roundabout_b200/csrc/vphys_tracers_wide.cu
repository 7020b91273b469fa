// vphys_tracers_wide.cu -- the exact tracer solve (vphys_tracers.cuh) with six to
// sixteen tracers in one thread, for shallow columns (tracer_groups).  A file of its
// own, so that only a program that runs its kernels loads them: in vphys_tracers.cu
// they made the first call of every program 8 ms longer (5.5 -> 14 ms; nvcc
// compresses device code of that size).
#include <cuda_runtime.h>

#include "vphys_tracers.cuh"

namespace vphys {

void launch_tracers_wide(const Params &p, double dt, bool diffuse, bool nonlocal, bool two, cudaStream_t stream)
{
    if (p.ntr <= 8)
        two ? launch_tracers_n<8, true>(p, dt, diffuse, nonlocal, 1, stream)
            : launch_tracers_n<8, false>(p, dt, diffuse, nonlocal, 1, stream);
    else
        two ? launch_tracers_n<NTR_MAX, true>(p, dt, diffuse, nonlocal, 1, stream)
            : launch_tracers_n<NTR_MAX, false>(p, dt, diffuse, nonlocal, 1, stream);
}

}  // namespace vphys
