// F32 instances of the transform pass planned at compile time (pp_mr.cuh),
// lengths 270 .. 450.
#include "pp_mr.cuh"

cudaError_t pp_launch_mr_ct_c_f32(const PPLinePassArgs& a, const PPMrPlan& p, bool inverse, bool strided,
                                    cudaStream_t st)
{
    switch (a.n) {
    case 270: return pp_mr::launch_ct<float, 270>(a, p, inverse, strided, st);
    case 288: return pp_mr::launch_ct<float, 288>(a, p, inverse, strided, st);
    case 300: return pp_mr::launch_ct<float, 300>(a, p, inverse, strided, st);
    case 320: return pp_mr::launch_ct<float, 320>(a, p, inverse, strided, st);
    case 324: return pp_mr::launch_ct<float, 324>(a, p, inverse, strided, st);
    case 360: return pp_mr::launch_ct<float, 360>(a, p, inverse, strided, st);
    case 384: return pp_mr::launch_ct<float, 384>(a, p, inverse, strided, st);
    case 400: return pp_mr::launch_ct<float, 400>(a, p, inverse, strided, st);
    case 432: return pp_mr::launch_ct<float, 432>(a, p, inverse, strided, st);
    case 450: return pp_mr::launch_ct<float, 450>(a, p, inverse, strided, st);
    default: return cudaErrorInvalidValue;
    }
}
