// F64 instances of the transform pass planned at compile time (pp_mr.cuh),
// lengths 480 .. 768.
#include "pp_mr.cuh"

cudaError_t pp_launch_mr_ct_d_f64(const PPLinePassArgs& a, const PPMrPlan& p, bool inverse, bool strided,
                                    cudaStream_t st)
{
    switch (a.n) {
    case 480: return pp_mr::launch_ct<double, 480>(a, p, inverse, strided, st);
    case 500: return pp_mr::launch_ct<double, 500>(a, p, inverse, strided, st);
    case 540: return pp_mr::launch_ct<double, 540>(a, p, inverse, strided, st);
    case 576: return pp_mr::launch_ct<double, 576>(a, p, inverse, strided, st);
    case 600: return pp_mr::launch_ct<double, 600>(a, p, inverse, strided, st);
    case 640: return pp_mr::launch_ct<double, 640>(a, p, inverse, strided, st);
    case 720: return pp_mr::launch_ct<double, 720>(a, p, inverse, strided, st);
    case 750: return pp_mr::launch_ct<double, 750>(a, p, inverse, strided, st);
    case 768: return pp_mr::launch_ct<double, 768>(a, p, inverse, strided, st);
    default: return cudaErrorInvalidValue;
    }
}
