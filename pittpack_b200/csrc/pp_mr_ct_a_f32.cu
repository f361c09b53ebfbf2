// F32 instances of the transform pass planned at compile time (pp_mr.cuh),
// lengths 40 .. 120.
#include "pp_mr.cuh"

cudaError_t pp_launch_mr_ct_a_f32(const PPLinePassArgs& a, const PPMrPlan& p, bool inverse, bool strided,
                                    cudaStream_t st)
{
    switch (a.n) {
    case 40: return pp_mr::launch_ct<float, 40>(a, p, inverse, strided, st);
    case 48: return pp_mr::launch_ct<float, 48>(a, p, inverse, strided, st);
    case 50: return pp_mr::launch_ct<float, 50>(a, p, inverse, strided, st);
    case 54: return pp_mr::launch_ct<float, 54>(a, p, inverse, strided, st);
    case 60: return pp_mr::launch_ct<float, 60>(a, p, inverse, strided, st);
    case 72: return pp_mr::launch_ct<float, 72>(a, p, inverse, strided, st);
    case 80: return pp_mr::launch_ct<float, 80>(a, p, inverse, strided, st);
    case 90: return pp_mr::launch_ct<float, 90>(a, p, inverse, strided, st);
    case 96: return pp_mr::launch_ct<float, 96>(a, p, inverse, strided, st);
    case 100: return pp_mr::launch_ct<float, 100>(a, p, inverse, strided, st);
    case 108: return pp_mr::launch_ct<float, 108>(a, p, inverse, strided, st);
    case 120: return pp_mr::launch_ct<float, 120>(a, p, inverse, strided, st);
    default: return cudaErrorInvalidValue;
    }
}
