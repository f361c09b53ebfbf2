// Contiguous FP64 passes of complex lines and half spectra, lengths m 2^k
// (pp_lp2.cuh): the lengths that pp_lpm_takes lists.
#include "pp_lp2.cuh"

cudaError_t pp_launch_lpm_cplx(const PPLinePassArgs& a, bool inverse, cudaStream_t st)
{
    using namespace pp_lp2;
#define PP_LPM(N, LPC) \
    case N: return inverse ? launch_lpm<N, LPC, F_FFT, true>(a, st) : launch_lpm<N, LPC, F_FFT, false>(a, st);
#define PP_LPM_HALF(N, LPC) \
    case N: return inverse ? launch_lpm<N, LPC, F_C2R, true>(a, st) : launch_lpm<N, LPC, F_R2C, false>(a, st);
    if (a.half) {
        switch (a.n) {
            PP_LPM_HALF(960, 1) PP_LPM_HALF(1152, 1) PP_LPM_HALF(1280, 1) PP_LPM_HALF(1536, 1)
        default: return cudaErrorInvalidValue;
        }
    }
    switch (a.n) {
        PP_LPM(320, 4) PP_LPM(480, 2) PP_LPM(576, 2) PP_LPM(640, 2) PP_LPM(768, 2)
        PP_LPM(960, 1) PP_LPM(1152, 1) PP_LPM(1280, 1) PP_LPM(1536, 1)
    default: return cudaErrorInvalidValue;
    }
#undef PP_LPM
#undef PP_LPM_HALF
}
