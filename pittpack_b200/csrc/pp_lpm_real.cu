// Contiguous FP64 passes of DCT-II/III and DST-II/III, lengths m 2^k
// (pp_lp2.cuh): the lengths that pp_lpm_takes lists.
#include "pp_lp2.cuh"

namespace {

template <int FAM>
cudaError_t launch_family(const PPLinePassArgs& a, bool inverse, cudaStream_t st)
{
    using namespace pp_lp2;
#define PP_LPM(N, LPC) \
    case N: return inverse ? launch_lpm<N, LPC, FAM, true>(a, st) : launch_lpm<N, LPC, FAM, false>(a, st);
#define PP_LPM_INV(N, LPC) \
    case N: return inverse ? launch_lpm<N, LPC, FAM, true>(a, st) : cudaErrorInvalidValue;
    switch (a.n) {
        PP_LPM_INV(576, 2) PP_LPM_INV(768, 2)
        PP_LPM(960, 1) PP_LPM(1152, 1) PP_LPM(1280, 1) PP_LPM(1536, 1)
    default: return cudaErrorInvalidValue;
    }
#undef PP_LPM
#undef PP_LPM_INV
}

}  // namespace

cudaError_t pp_launch_lpm_real(const PPLinePassArgs& a, bool inverse, cudaStream_t st)
{
    return a.kind == PP_KIND_DST2 ? launch_family<pp_lp2::F_DST2>(a, inverse, st)
                                  : launch_family<pp_lp2::F_DCT2>(a, inverse, st);
}
