// F64 instances of the transform pass planned at compile time (pp_mr.cuh),
// lengths 144 .. 250.
#include "pp_mr.cuh"

cudaError_t pp_launch_mr_ct_b_f64(const PPLinePassArgs& a, const PPMrPlan& p, bool inverse, bool strided,
                                    cudaStream_t st)
{
    switch (a.n) {
    case 144: return pp_mr::launch_ct<double, 144>(a, p, inverse, strided, st);
    case 150: return pp_mr::launch_ct<double, 150>(a, p, inverse, strided, st);
    case 160: return pp_mr::launch_ct<double, 160>(a, p, inverse, strided, st);
    case 162: return pp_mr::launch_ct<double, 162>(a, p, inverse, strided, st);
    case 180: return pp_mr::launch_ct<double, 180>(a, p, inverse, strided, st);
    case 192: return pp_mr::launch_ct<double, 192>(a, p, inverse, strided, st);
    case 200: return pp_mr::launch_ct<double, 200>(a, p, inverse, strided, st);
    case 216: return pp_mr::launch_ct<double, 216>(a, p, inverse, strided, st);
    case 240: return pp_mr::launch_ct<double, 240>(a, p, inverse, strided, st);
    case 250: return pp_mr::launch_ct<double, 250>(a, p, inverse, strided, st);
    default: return cudaErrorInvalidValue;
    }
}
