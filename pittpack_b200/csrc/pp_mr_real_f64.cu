// F64 instances of the run-time planned transform pass (pp_mr.cuh): the real families.
#include "pp_mr.cuh"

cudaError_t pp_launch_mr_real_f64(const PPLinePassArgs& a, const PPMrPlan& p, bool inverse, bool strided, cudaStream_t st)
{
    return pp_mr::launch_real<double>(a, p, inverse, strided, st);
}
