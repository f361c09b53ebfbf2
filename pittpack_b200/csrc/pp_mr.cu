// Host side of the run-time planned transform pass (pp_mr.cuh): the radices,
// lines and threads of a length, and one pass in either precision.
#include "pp_mr.cuh"
cudaError_t pp_launch_mr_ct_a_f64(const PPLinePassArgs&, const PPMrPlan&, bool, bool, cudaStream_t);
cudaError_t pp_launch_mr_ct_a_f32(const PPLinePassArgs&, const PPMrPlan&, bool, bool, cudaStream_t);
cudaError_t pp_launch_mr_ct_b_f64(const PPLinePassArgs&, const PPMrPlan&, bool, bool, cudaStream_t);
cudaError_t pp_launch_mr_ct_b_f32(const PPLinePassArgs&, const PPMrPlan&, bool, bool, cudaStream_t);
cudaError_t pp_launch_mr_ct_c_f64(const PPLinePassArgs&, const PPMrPlan&, bool, bool, cudaStream_t);
cudaError_t pp_launch_mr_ct_c_f32(const PPLinePassArgs&, const PPMrPlan&, bool, bool, cudaStream_t);
cudaError_t pp_launch_mr_ct_d_f64(const PPLinePassArgs&, const PPMrPlan&, bool, bool, cudaStream_t);
cudaError_t pp_launch_mr_ct_d_f32(const PPLinePassArgs&, const PPMrPlan&, bool, bool, cudaStream_t);
cudaError_t pp_launch_mr_ct_e_f64(const PPLinePassArgs&, const PPMrPlan&, bool, bool, cudaStream_t);
cudaError_t pp_launch_mr_ct_e_f32(const PPLinePassArgs&, const PPMrPlan&, bool, bool, cudaStream_t);

namespace {

// the instances planned at compile time, by ranges of lengths; within a range
// the lengths without one answer cudaErrorInvalidValue
using CtLaunch = cudaError_t (*)(const PPLinePassArgs&, const PPMrPlan&, bool, bool, cudaStream_t);
struct CtRange {
    int lo, hi;
    CtLaunch f64, f32;
};
const CtRange kCt[] = {
    {40, 120, pp_launch_mr_ct_a_f64, pp_launch_mr_ct_a_f32},
    {144, 250, pp_launch_mr_ct_b_f64, pp_launch_mr_ct_b_f32},
    {270, 450, pp_launch_mr_ct_c_f64, pp_launch_mr_ct_c_f32},
    {480, 768, pp_launch_mr_ct_d_f64, pp_launch_mr_ct_d_f32},
    {800, 1536, pp_launch_mr_ct_e_f64, pp_launch_mr_ct_e_f32},
};

// the lengths of pp_mr_ct_*.cu
bool compiled(int n)
{
    static const short lengths[] = {40,  48,  50,  54,  60,  72,  80,  90,  96,  100, 108, 120, 144,  150,  160,  162,  180,
                                    192, 200, 216, 240, 250, 270, 288, 300, 320, 324, 360, 384, 400,  432,  450,  480,  500,
                                    540, 576, 600, 640, 720, 750, 768, 800, 864, 900, 960, 1000, 1152, 1200, 1280, 1536};
    for (int c : lengths)
        if (c == n) return true;
    return false;
}

// Whether a plan is faster than the generic kernel (pp_linepass.cu).  Known at
// compile time, or with a radix 11 or 13 (p^2 work a butterfly there): always; also
// even DCT-II / DST-II lengths, whose passes are level on the smallest grids and whose
// z solve gains the z-tiled spectrum (50 x 42 x 37 36.9 and 35.3 us).  Read at
// run time, its passes are calls of their own at 128 registers, which a grid waits
// for that fills the GPU only once or twice, and complex lines of three passes longer
// than that.  Two passes of a direction, planned to generic:
//   real, N x 64 x 8, x 24, x 80, x 256:  25 1.67, 1.59, 1.18, 0.81; 45 1.41, 1.40,
//     0.94, 0.67; 105 1.02, 0.98, 0.65, 0.59; 315 1.38, 0.81, 0.99, 0.62; even 42 1.01,
//     1.02, 0.73, 0.51, its DCT-IV 1.13, 1.17, 0.86, 0.62
//   complex y, 64 x N x 8 .. 256:  45 1.37, 1.27, 1.19, 0.88; 315 1.33, 1.14, 1.38,
//     1.28; 448 1.15, 1.00, 1.27, 1.12; x 800: 125 1.50, 135 0.82, 225 0.77, 189 1.03
// Solves with the planned kernel always: 25^2 x 40 N-N 57 us and 37, 45^2 x 40 P-P 47
// and 35, 315 x 64 x 40 P-P 105 and 80, 125 x 128 x 64 P-P 89 and 76.
bool pays(int n, int kind, bool half, const PPMrPlan& p, long points)
{
    if (compiled(n) || n % 11 == 0 || n % 13 == 0) return true;
    if (n % 2 == 0 && (kind == PP_KIND_DCT2 || kind == PP_KIND_DST2)) return true;
    const bool cplx = kind == PP_KIND_FFT && !half;
    return points >= (cplx && p.npass > 2 ? 8000000L : 350000L);
}

}  // namespace

bool pp_mr_plan(int n, int kind, bool half, long points, PPMrPlan* p)
{
    *p = PPMrPlan{};
    const bool odd = n & 1;
    if ((half || pp_kind_is_quarter(kind)) && odd) return false;
    *p = pp_mr::make_plan((half || (kind != PP_KIND_FFT && !odd)) ? n / 2 : n);
    if (p->m > 0 && !pays(n, kind, half, *p, points)) *p = PPMrPlan{};
    return p->m > 0;
}

int pp_mr_lines(int n, int kind, const PPMrPlan& p)
{
    // real lines of odd length go two to an FFT line
    return (kind != PP_KIND_FFT && (n & 1)) ? 2 * p.L : p.L;
}

cudaError_t pp_mr_line_pass(PPLinePassArgs a, const PPMrPlan& p, bool inverse, bool strided, bool in_cplx,
                            bool out_cplx, bool fp32, cudaStream_t st)
{
    const size_t es = fp32 ? sizeof(float) : sizeof(double);
    const bool own = a.o_elem_stride != 0;
    a.in_cplx = in_cplx;
    a.out_cplx = out_cplx;
    // pairs of reals in, pairs of reals or (the solution P) of complex points out
    auto whole = [](const void* q, long s1, long s2, size_t elem, size_t w) {
        return reinterpret_cast<uintptr_t>(q) % w == 0 && ((size_t)s1 * elem) % w == 0 && ((size_t)s2 * elem) % w == 0;
    };
    if (!fp32 && !strided && pp_lpm_takes(a.n, a.kind, a.half, inverse)) {
        // 16-byte runs of its input; lines a CTA as its launches have them, real ones two to an FFT
        const int lpc = a.n >= 960 ? 1 : a.n >= 480 ? 2 : 4;
        a.L = a.kind == PP_KIND_FFT && !a.half ? lpc : 2 * lpc;
        a.tiles_per_plane = (a.nlines + a.L - 1) / a.L;
        a.vec16 = whole(a.src, a.line_stride, a.plane_stride, (in_cplx ? 2 : 1) * es, 16);
        return a.kind == PP_KIND_FFT ? pp_launch_lpm_cplx(a, inverse, st) : pp_launch_lpm_real(a, inverse, st);
    }
    a.vec16 = !strided && !in_cplx && whole(a.src, a.line_stride, a.plane_stride, es, 2 * es);
    a.vec_out = !strided && whole(a.dst, own ? a.o_line_stride : a.line_stride, own ? a.o_plane_stride : a.plane_stride,
                                  (out_cplx ? 2 : 1) * es, (inverse ? 4 : 2) * es);
    a.L = pp_mr_lines(a.n, a.kind, p);
    a.tiles_per_plane = (a.nlines + a.L - 1) / a.L;
    for (const CtRange& c : kCt)
        if (a.n >= c.lo && a.n <= c.hi) {
            const cudaError_t e = (fp32 ? c.f32 : c.f64)(a, p, inverse, strided, st);
            if (e != cudaErrorInvalidValue) return e;
        }
    if (a.kind == PP_KIND_FFT)
        return fp32 ? pp_launch_mr_periodic_f32(a, p, inverse, strided, st)
                    : pp_launch_mr_periodic_f64(a, p, inverse, strided, st);
    return fp32 ? pp_launch_mr_real_f32(a, p, inverse, strided, st) : pp_launch_mr_real_f64(a, p, inverse, strided, st);
}
