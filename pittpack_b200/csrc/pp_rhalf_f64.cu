// FP64 instances of the half-length real transform pass (pp_rhalf.cuh): the
// plain solve; and the host side of a pass in either precision.
#include "pp_rhalf.cuh"

int pp_rh_lines(int n, bool strided) { return pp_rh::lines(n, strided); }

bool pp_rh_covers(const PPLinePassArgs& a, bool inverse, bool strided, bool out_cplx)
{
    if (pp_rh::lines(a.n, strided) == 0) return false;
    if (a.kind == PP_KIND_FFT) return a.half != 0;
    // a real family writes complex points only as the solution P
    return !out_cplx || (inverse && !strided);
}

cudaError_t pp_rh_line_pass(PPLinePassArgs a, bool inverse, bool strided, bool in_cplx, bool out_cplx, bool fp32,
                            cudaStream_t st)
{
    const size_t es = fp32 ? sizeof(float) : sizeof(double);
    const bool own = a.o_elem_stride != 0;
    a.in_cplx = in_cplx;
    a.out_cplx = out_cplx;
    // the contiguous pass's widest accesses, where every line starts on their
    // boundary: quads of the input (pairs for DCT-IV / DST-IV and the real side
    // of the half spectra), two complex points of P (pairs of reals for the
    // forward DCT-IV / DST-IV)
    const size_t wi = (a.half || pp_kind_is_quarter(a.kind) ? 2 : 4) * es, wo = (inverse ? 4 : 2) * es;
    auto whole = [](const void* p, long s1, long s2, size_t elem, size_t w) {
        return reinterpret_cast<uintptr_t>(p) % w == 0 && ((size_t)s1 * elem) % w == 0 && ((size_t)s2 * elem) % w == 0;
    };
    a.vec16 = !strided && !in_cplx && whole(a.src, a.line_stride, a.plane_stride, es, wi);
    a.vec_out = !strided && whole(a.dst, own ? a.o_line_stride : a.line_stride, own ? a.o_plane_stride : a.plane_stride,
                                  (out_cplx ? 2 : 1) * es, wo);
    a.L = pp_rh::lines(a.n, strided);
    a.tiles_per_plane = (a.nlines + a.L - 1) / a.L;
    return fp32 ? pp_launch_line_pass_rh_f32(a, inverse, strided, st) : pp_rh::launch<double>(a, inverse, strided, st);
}
