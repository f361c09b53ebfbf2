// F32 instances of the transform pass planned at compile time (pp_mr.cuh),
// lengths 480 .. 768.
#include "pp_mr.cuh"

cudaError_t pp_launch_mr_ct_d_f32(const PPLinePassArgs& a, const PPMrPlan& p, bool inverse, bool strided,
                                    cudaStream_t st)
{
    switch (a.n) {
    case 480: return pp_mr::launch_ct<float, 480>(a, p, inverse, strided, st);
    case 500: return pp_mr::launch_ct<float, 500>(a, p, inverse, strided, st);
    case 540: return pp_mr::launch_ct<float, 540>(a, p, inverse, strided, st);
    case 576: return pp_mr::launch_ct<float, 576>(a, p, inverse, strided, st);
    case 600: return pp_mr::launch_ct<float, 600>(a, p, inverse, strided, st);
    case 640: return pp_mr::launch_ct<float, 640>(a, p, inverse, strided, st);
    case 720: return pp_mr::launch_ct<float, 720>(a, p, inverse, strided, st);
    case 750: return pp_mr::launch_ct<float, 750>(a, p, inverse, strided, st);
    case 768: return pp_mr::launch_ct<float, 768>(a, p, inverse, strided, st);
    default: return cudaErrorInvalidValue;
    }
}
