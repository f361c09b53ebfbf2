// F64 instances of the transform pass planned at compile time (pp_mr.cuh),
// lengths 800 .. 1536.
#include "pp_mr.cuh"

cudaError_t pp_launch_mr_ct_e_f64(const PPLinePassArgs& a, const PPMrPlan& p, bool inverse, bool strided,
                                    cudaStream_t st)
{
    switch (a.n) {
    case 800: return pp_mr::launch_ct<double, 800>(a, p, inverse, strided, st);
    case 864: return pp_mr::launch_ct<double, 864>(a, p, inverse, strided, st);
    case 900: return pp_mr::launch_ct<double, 900>(a, p, inverse, strided, st);
    case 960: return pp_mr::launch_ct<double, 960>(a, p, inverse, strided, st);
    case 1000: return pp_mr::launch_ct<double, 1000>(a, p, inverse, strided, st);
    case 1152: return pp_mr::launch_ct<double, 1152>(a, p, inverse, strided, st);
    case 1200: return pp_mr::launch_ct<double, 1200>(a, p, inverse, strided, st);
    case 1280: return pp_mr::launch_ct<double, 1280>(a, p, inverse, strided, st);
    case 1536: return pp_mr::launch_ct<double, 1536>(a, p, inverse, strided, st);
    default: return cudaErrorInvalidValue;
    }
}
