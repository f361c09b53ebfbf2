// F32 instances of the transform pass planned at compile time (pp_mr.cuh),
// lengths 144 .. 250.
#include "pp_mr.cuh"

cudaError_t pp_launch_mr_ct_b_f32(const PPLinePassArgs& a, const PPMrPlan& p, bool inverse, bool strided,
                                    cudaStream_t st)
{
    switch (a.n) {
    case 144: return pp_mr::launch_ct<float, 144>(a, p, inverse, strided, st);
    case 150: return pp_mr::launch_ct<float, 150>(a, p, inverse, strided, st);
    case 160: return pp_mr::launch_ct<float, 160>(a, p, inverse, strided, st);
    case 162: return pp_mr::launch_ct<float, 162>(a, p, inverse, strided, st);
    case 180: return pp_mr::launch_ct<float, 180>(a, p, inverse, strided, st);
    case 192: return pp_mr::launch_ct<float, 192>(a, p, inverse, strided, st);
    case 200: return pp_mr::launch_ct<float, 200>(a, p, inverse, strided, st);
    case 216: return pp_mr::launch_ct<float, 216>(a, p, inverse, strided, st);
    case 240: return pp_mr::launch_ct<float, 240>(a, p, inverse, strided, st);
    case 250: return pp_mr::launch_ct<float, 250>(a, p, inverse, strided, st);
    default: return cudaErrorInvalidValue;
    }
}
