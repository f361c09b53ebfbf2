// F64 instances of the transform pass planned at compile time (pp_mr.cuh),
// lengths 270 .. 450.
#include "pp_mr.cuh"

cudaError_t pp_launch_mr_ct_c_f64(const PPLinePassArgs& a, const PPMrPlan& p, bool inverse, bool strided,
                                    cudaStream_t st)
{
    switch (a.n) {
    case 270: return pp_mr::launch_ct<double, 270>(a, p, inverse, strided, st);
    case 288: return pp_mr::launch_ct<double, 288>(a, p, inverse, strided, st);
    case 300: return pp_mr::launch_ct<double, 300>(a, p, inverse, strided, st);
    case 320: return pp_mr::launch_ct<double, 320>(a, p, inverse, strided, st);
    case 324: return pp_mr::launch_ct<double, 324>(a, p, inverse, strided, st);
    case 360: return pp_mr::launch_ct<double, 360>(a, p, inverse, strided, st);
    case 384: return pp_mr::launch_ct<double, 384>(a, p, inverse, strided, st);
    case 400: return pp_mr::launch_ct<double, 400>(a, p, inverse, strided, st);
    case 432: return pp_mr::launch_ct<double, 432>(a, p, inverse, strided, st);
    case 450: return pp_mr::launch_ct<double, 450>(a, p, inverse, strided, st);
    default: return cudaErrorInvalidValue;
    }
}
