// F64 instances of the transform pass planned at compile time (pp_mr.cuh),
// lengths 40 .. 120.
#include "pp_mr.cuh"

cudaError_t pp_launch_mr_ct_a_f64(const PPLinePassArgs& a, const PPMrPlan& p, bool inverse, bool strided,
                                    cudaStream_t st)
{
    switch (a.n) {
    case 40: return pp_mr::launch_ct<double, 40>(a, p, inverse, strided, st);
    case 48: return pp_mr::launch_ct<double, 48>(a, p, inverse, strided, st);
    case 50: return pp_mr::launch_ct<double, 50>(a, p, inverse, strided, st);
    case 54: return pp_mr::launch_ct<double, 54>(a, p, inverse, strided, st);
    case 60: return pp_mr::launch_ct<double, 60>(a, p, inverse, strided, st);
    case 72: return pp_mr::launch_ct<double, 72>(a, p, inverse, strided, st);
    case 80: return pp_mr::launch_ct<double, 80>(a, p, inverse, strided, st);
    case 90: return pp_mr::launch_ct<double, 90>(a, p, inverse, strided, st);
    case 96: return pp_mr::launch_ct<double, 96>(a, p, inverse, strided, st);
    case 100: return pp_mr::launch_ct<double, 100>(a, p, inverse, strided, st);
    case 108: return pp_mr::launch_ct<double, 108>(a, p, inverse, strided, st);
    case 120: return pp_mr::launch_ct<double, 120>(a, p, inverse, strided, st);
    default: return cudaErrorInvalidValue;
    }
}
