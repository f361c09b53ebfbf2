// FP32 instances of the half-length real transform pass (pp_rhalf.cuh): the
// correction solves of the refined mode.
#include "pp_rhalf.cuh"

cudaError_t pp_launch_line_pass_rh_f32(const PPLinePassArgs& a, bool inverse, bool strided, cudaStream_t st)
{
    return pp_rh::launch<float>(a, inverse, strided, st);
}
