// F64 instances of the run-time planned transform pass (pp_mr.cuh): complex
// lines and half spectra.
#include "pp_mr.cuh"

cudaError_t pp_launch_mr_periodic_f64(const PPLinePassArgs& a, const PPMrPlan& p, bool inverse, bool strided,
                                     cudaStream_t st)
{
    return pp_mr::launch_periodic<double>(a, p, inverse, strided, st);
}
