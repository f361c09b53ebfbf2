// Kernel argument blocks and launchers shared by the solver's host code.
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>

#include "pp_fft.cuh"

#define PP_LINE_THREADS 256
#define PP_Z_THREADS 256

// Dirichlet face corrections subtracted from the dz^2-scaled RHS
// (modifyRhsDirichlet, src/pencilDcmp.cpp:4623-4835); null where a face is
// not Dirichlet.  z faces are [j][i], x faces [k][j], y faces [k][i].
struct PPLift {
    const double* z0;
    const double* z1;
    const double* x0;
    const double* x1;
    const double* y0;
    const double* y1;
    int any;
};

struct PPLinePassArgs {
    const double* src;
    double* dst;
    int n;             // points along the transformed direction
    int kind;          // PPKind
    int nlines;        // lines per plane
    int nplanes;
    long elem_stride;  // strides in elements (complex elements count once)
    long line_stride;
    long plane_stride;
    // every kernel but the generic one: the tile of lines l0.. starts at
    // plane * plane_stride + l0 * tile_stride (0: l0 * line_stride), and the
    // output may use its own strides (o_*; o_elem_stride = 0: the input's).
    // This lets the y passes write / read the z-tiled spectrum layout, and the x
    // passes rows of their own width (half spectra, padded rows).
    long tile_stride;
    long o_elem_stride, o_line_stride, o_plane_stride, o_tile_stride;
    int L;             // lines per CTA tile
    int tiles_per_plane;
    PPFftPlan fft;     // length n, or n/2 for the quarter-wave families
    const double2* cs; // pre/post twiddles of the family (see pp_linepass.cu)
    int rhs_scale;     // forward x-pass: multiply by dz twice and subtract the lift
    double dz;
    PPLift lift;
    int nx, ny, nz;
    double out_scale;  // inverse x-pass: 1 / (nx ny)
    // twiddles in the kernel's precision: used by the tile kernel (pp_lp2.cuh), the
    // half-length and planned ones (pp_rhalf.cuh, pp_mr.cuh) and the FP32 generic one
    const void* tw;    // FFT twiddles (double2 or float2), length n or n/2
    const void* cs2;   // family twiddles in the kernel's precision
    int in_cplx, out_cplx;
    int vec16;          // tile kernel: src and its run starts are 16-byte aligned
                        // (half-length and planned kernels: aligned to the widest load)
    int vec_out;        // half-length and planned kernels: dst and its runs are aligned to the widest store
    int half;           // periodic x pass of a real RHS on half spectra (N/2 + 1 complex per
                        // line): forward real -> half, inverse half -> real (read as reals
                        // where in_cplx is 0, after a non-periodic y)
    // refinement epilogue of the inverse x pass (acc != null): the real part v
    // of each output becomes u = acc + out_scale v + zplane[plane] in FP64;
    // written to acc, or (dst != null) as the final complex-interleaved P
    double* acc;
    const double* zplane;
    double zscale;      // zplane[plane] is multiplied by this
    int acc_read;       // 0: the previous u is zero (first sweep), acc is not read
    // bounded waits (the bulk-copy staging of the contiguous passes): a CTA
    // whose wait runs out adds 1 here (if set) and returns without output
    int* err;
};

// The run-time planned transform pass (pp_mr.cuh): lengths whose FFT factors
// into 2, 3, 5, 7, 11 and 13; passed to the kernel by value
#define PP_MR_MAXPASS 6
struct PPMrPlan {
    int m;                          // FFT points a line (0: no such plan)
    int L, lgl;                     // FFT lines a CTA (a power of two)
    int npass;
    int radix[PP_MR_MAXPASS];
    unsigned magic[PP_MR_MAXPASS];  // division by the span of each pass
    int threads;
};
// the plan of a direction (half: its periodic half spectra) of a grid of so many
// points; false where it has none, or the generic kernel is faster
bool pp_mr_plan(int n, int kind, bool half, long points, PPMrPlan* p);
// data lines per CTA tile
int pp_mr_lines(int n, int kind, const PPMrPlan& p);
// one pass (a.tw and a.cs2 in its precision, strides and output strides set), in
// this kernel or where it is faster in the register kernel below
cudaError_t pp_mr_line_pass(PPLinePassArgs a, const PPMrPlan& p, bool inverse, bool strided, bool in_cplx,
                            bool out_cplx, bool fp32, cudaStream_t st);
// Whether a contiguous FP64 pass of a planned length runs the register kernel of
// the lengths m 2^k instead (lpm_kernel, pp_lp2.cuh).  From 480 FFT points on the
// planned kernel's tiles of up to 4096 points leave a CTA two to four lines (two-way
// bank conflicts below eight) and an SM two or three CTAs.  Planned and register
// kernel, us a pass over 24 M points, 128 rows a plane:
//   complex   480 250 and 195, 576 235 and 170, 640 237 and 208, 768 224 and 210,
//             960 232 and 183, 1152 252 and 195, 1536 281 and 215; 320 (16 M points)
//             125 and 116, but 384 142 and 152
//   half      forward 960 148 and 103, 1280 142 and 118, 1536 130 and 117, but 768
//             105 and 117; inverse 960 156 and 119, 1536 159 and 136
//   N-N       forward 960 144 and 116, 1152 143 and 121, 1536 138 and 132, but 768
//             114 and 117; inverse 576 136 and 122, 768 157 and 132, 960 183 and 134,
//             1536 167 and 144, but 640 120 and 127 (D-D alike)
// Strided, DCT-IV / DST-IV and FP32 passes are faster planned (y at 960^2 x 34 N-N 197
// and 458 us; DST-IV 960 forward 152 and 146, inverse 170 and 201).  One line a CTA
// in the planned kernel, odd radix first, did not reach it (960 N-N 125 and 161 us).
constexpr bool pp_lpm_takes(int n, int kind, bool half, bool inverse)
{
    const bool large = n == 960 || n == 1152 || n == 1280 || n == 1536;
    if (kind == PP_KIND_FFT && !half) return large || n == 320 || n == 480 || n == 576 || n == 640 || n == 768;
    if (kind == PP_KIND_FFT) return large;
    if (kind == PP_KIND_DST2 || kind == PP_KIND_DCT2) return large || (inverse && (n == 576 || n == 768));
    return false;
}
cudaError_t pp_launch_lpm_cplx(const PPLinePassArgs& a, bool inverse, cudaStream_t st);
cudaError_t pp_launch_lpm_real(const PPLinePassArgs& a, bool inverse, cudaStream_t st);
cudaError_t pp_launch_mr_real_f64(const PPLinePassArgs& a, const PPMrPlan& p, bool inverse, bool strided, cudaStream_t st);
cudaError_t pp_launch_mr_real_f32(const PPLinePassArgs& a, const PPMrPlan& p, bool inverse, bool strided, cudaStream_t st);
cudaError_t pp_launch_mr_periodic_f64(const PPLinePassArgs& a, const PPMrPlan& p, bool inverse, bool strided,
                                      cudaStream_t st);
cudaError_t pp_launch_mr_periodic_f32(const PPLinePassArgs& a, const PPMrPlan& p, bool inverse, bool strided,
                                      cudaStream_t st);

// shared memory of the generic kernel: two buffers of L lines of nfft complex
// points in FP64, or in FP32 (fp32)
size_t pp_line_pass_smem(int L, int nfft, bool fp32 = false);

// Lines whose FFT length nf is past one generic-kernel tile (pp_longline.cu):
// the FFT in four steps, nf = n1 n2, through a global scratch array of
// nplanes x nlines x nf complex points; or, where nf has a prime factor past
// one tile, by the chirp z-transform: a cyclic convolution of length
// M = n1 n2 (a power of two >= 2 nf - 1) by two four-step FFTs
struct PPLongPlan {
    int n1, n2;
    PPFftPlan f1, f2;      // plans of n1 and n2 with their FP64 twiddles
    const void* tw1f;      // FP32 twiddles of n1 and n2
    const void* tw2f;
    const double2* twl;    // W_(n1 n2)^j, j < n1 n2, FP64 and FP32
    const void* twlf;
    void* scratch;
    // chirp z-transform (M = n1 n2 > 0): c_k = e^{i pi k^2 / nf}, k < nf, and
    // the FFT of the chirp kernel for the forward and backward transforms, in
    // the four-step output order; FP64 and FP32
    int M;
    int nf;                // the transform's FFT length (n1 n2 without the chirp z-transform)
    const double2* chirp;
    const void* chirpf;
    const double2* bhat[2];
    const void* bhatf[2];
};
// the split nf = n1 n2 (n1 <= n2, nearest the square root, both within one
// generic-kernel tile); false where there is none (a prime beyond that size)
bool pp_long_split(int nf, int* n1, int* n2);
// the chirp z-transform's convolution length for nf (a power of two >= 2 nf - 1)
// and its split; false past the four-step's reach
bool pp_bluestein_split(int nf, int* M, int* n1, int* n2);
size_t pp_long_scratch_bytes(long lines, int nf);
cudaError_t pp_launch_long_line_pass(const PPLinePassArgs& a, const PPLongPlan& lp, bool inverse, bool strided,
                                     bool in_cplx, bool out_cplx, cudaStream_t st, bool fp32);
// power-of-two lengths 16..2048: complex FFT lines per CTA (0 = not covered);
// a tile holds this many data lines for the periodic family and twice as many
// for the real families
int pp_lp2_lpc(int n);
template <typename Real, typename TI, typename TO>
cudaError_t pp_launch_line_pass_pow2(const PPLinePassArgs& a, bool inverse, bool strided, cudaStream_t st);
// the real families and the periodic half spectra through a complex FFT of
// half the length (pp_rhalf.cuh): data lines per CTA tile (0 = not covered),
// whether a pass takes that kernel, and the pass (a.tw and a.cs2 in its
// precision, strides and output strides set; out strides of 0: the input's)
int pp_rh_lines(int n, bool strided);
bool pp_rh_covers(const PPLinePassArgs& a, bool inverse, bool strided, bool out_cplx);
cudaError_t pp_rh_line_pass(PPLinePassArgs a, bool inverse, bool strided, bool in_cplx, bool out_cplx, bool fp32,
                            cudaStream_t st);
cudaError_t pp_launch_line_pass_rh_f32(const PPLinePassArgs& a, bool inverse, bool strided, cudaStream_t st);
// every other length (pp_fft_plan); fp32: the FP32 kernel, twiddles from a.tw and
// a.cs2 (FP64: a.fft.tw and a.cs), with the refinement epilogue when a.acc is set
cudaError_t pp_launch_line_pass(const PPLinePassArgs& a, bool inverse, bool strided, bool in_cplx, bool out_cplx,
                                cudaStream_t st, bool fp32 = false);

// z-boundary kinds of the tridiagonal systems
enum PPZBc : int { PP_Z_DIRICHLET = 0, PP_Z_NEUMANN = 1, PP_Z_PERIODIC = 2 };

struct PPZArgs {
    double* data;       // spectrum [k][ky][kx], real or complex
    int nx, ny, nz;
    int TS;             // systems (adjacent kx) per CTA
    int tiles_x;
    const double* ax;   // -2 + 2 cos((kx + num) f / (nx + den)), per kx
    const double* ay;   // same per ky
    double Cx, Cy;      // (dz/dx)^2, (dz/dy)^2
    int zlo, zhi;       // PPZBc of the two z ends
    int pin_always;     // 1: zero-mode row replacement whatever the z ends (reference)
    int P;              // lanes per system (0: the default for nz)
    int data_fp32;      // spectrum stored as float / float2 (solved in FP64)
    int skip_zero;      // write zeros for the kx = ky = 0 column
    int tiled;          // spectrum in the z-tiled layout: tile (ky, kx / TS) is the
                        // contiguous block [k][kx % TS] at (ky (nx / TS) + kx / TS) nz TS
    int* err;           // counts CTAs whose bounded waits ran out (may be null)
};

// lanes that share one z system (a power of two <= 32) of a grid with that
// many systems
int pp_zsolve_lanes(int nz, bool cplx, long systems);
// systems per CTA and threads per CTA of the z solve
void pp_zsolve_config(int nz, bool cplx, int nx, int* TS, int* threads);
// the same for a chosen lane count (0 or invalid: the default); the launch
// must then carry P = that lane count
void pp_zsolve_config_p(int nz, bool cplx, int nx, int lanes, int* TS, int* threads, int systems = 0, int ny = 0);
int pp_zsolve_valid_lanes(int nz, int P);
size_t pp_zsolve_smem_p(int TS, int nz, bool cplx, int P);
// the longest z systems the z solve takes: a CTA of one system on 32 lanes
// whose column, pivot table and scratch fit the opt-in shared memory of a
// CTA (cplx: complex spectra; g32: the refined solve's FP32 spectra, staged
// beside the tile); about 25,000 rows for real spectra, 13,000 for complex
int pp_zsolve_max_nz(bool cplx, bool g32);

// FP64 residual r = f dz^2 - lift - A u of the refined solve (pp_mixed.cu)
struct PPResidArgs {
    const double* f;   // real RHS, unscaled
    const double* u;   // current solution (real), or null for u = 0
    float* r;          // FP32 residual out
    double* part;      // FP64 sums of r per (plane, xy tile): [nz][pp_resid_tiles], or null
    int nx, ny, nz;
    double dz, Cx, Cy;
    int bc[6];         // face codes: 0 Dirichlet, 1 Neumann, 2 periodic
    PPLift lift;
    double* upart;     // FP64 sums of u, same layout, or null
};
// xy tiles per plane of the residual kernel (the partial sums' row length)
int pp_resid_tiles(int nx, int ny);
cudaError_t pp_launch_resid(const PPResidArgs& a, cudaStream_t st);
// The kx = ky = 0 column of a refined sweep from per-CTA partial sums
// ([plane][tpp] each), added in a fixed order (one block per plane):
// zcol[k] = scale * sum_t part[k tpp + t]; if upart is set, uplane[k] = the
// plane's sum of upart and *usum = the sum of uplane (nz doubles of scratch).
cudaError_t pp_launch_zero_mode_sums(const double* part, const double* upart, int tpp, int nz, double scale,
                                     double* zcol, double* usum, double* uplane, cudaStream_t st);
// zero-mean solution (pp_mean.cu): the mean of the real parts of the n
// complex-interleaved values of P is subtracted from them; scratch holds
// pp_zero_mean_scratch_doubles() doubles
size_t pp_zero_mean_scratch_doubles();
cudaError_t pp_launch_zero_mean(double* P, long n, double* scratch, cudaStream_t st);
// u[i] = P[2 i] for the n complex-interleaved values of P (P 16-byte aligned)
cudaError_t pp_launch_real_part(const double* P, double* u, long n, cudaStream_t st);
// Singular problems: keep the null-space constant of the refined solution at
// the value implied by the pinned FP64 zero-mode solve of b (see pp_mixed.cu).
cudaError_t pp_launch_zero_mode_anchor(double* zcol, int nz, const double* usum, double* mstar, double zscale,
                                       double npts, int first, cudaStream_t st);
cudaError_t pp_launch_zsolve(const PPZArgs& a, bool cplx, cudaStream_t st);

// alternate z solve by multigrid V-cycles (pp_zsolve_mg.cu): the same systems
// as pp_launch_zsolve, FP64 spectra
struct PPZMgArgs {
    double* data;       // spectrum [k][ky][kx], real or complex
    int nx, ny, nz;
    const double* ax;
    const double* ay;
    double Cx, Cy;
    int zlo, zhi;
    int pin_always;
    int max_cycles;     // bound on V-cycles per system
    int* stats;         // [0] max cycles used, [1] systems stopped at the bound; or null
    int G;              // systems per CTA (set by the launcher)
    int tot;            // cells of all levels (set by the launcher)
};
int pp_zsolve_mg_levels_total(int nz);
size_t pp_zsolve_mg_smem(int G, int nz, bool cplx);
// cudaErrorInvalidValue when one system's levels do not fit shared memory
cudaError_t pp_launch_zsolve_mg(PPZMgArgs a, bool cplx, cudaStream_t st);

// the reference's alternate z solvers as its CPU build computes them
// (pp_zsolve_ref.cu): method PP_ZSOLVE_REF_PCR or PP_ZSOLVE_REF_CRP on the
// [k][ky][kx] spectrum (parts = 2: complex-interleaved), in place
struct PPZRefArgs {
    double* data;
    int nx, ny, nz;   // spectrum columns, rows, planes
    int parts;
    const double* ax;
    const double* ay;
    double Cx, Cy;
    int zlo, zhi;     // PP_Z_DIRICHLET / PP_Z_NEUMANN / PP_Z_PERIODIC
    int method;
};
bool pp_zsolve_ref_defined(int method, int nz, int zlo, int zhi);
cudaError_t pp_launch_zsolve_ref(const PPZRefArgs& a, cudaStream_t st);

struct pp_solver_s;
// columns a row of the spectrum may be padded by: up to a multiple of 16, or of
// 8, where that is at most an eighth of it
inline int pp_spare_cols(int nx)
{
    for (int q = 16; q >= 8; q /= 2)
        if ((q - nx % q) % q <= nx / 8) return (q - nx % q) % q;
    return 0;
}
// bytes of each of a handle's two spectrum buffers: the complex points of the
// grid, which hold the padding columns of real spectra too, and where y is
// periodic (its spectrum may be complex) the padding columns beside them
size_t pp_spectrum_bytes(int nx, int ny, int nz, bool y_periodic);
// whether a handle may pad complex spectra (default: yes): pp_assign_boundary
// then enlarges the spectrum buffers where the memory is there
void pp_allow_padding(pp_solver_s* h, bool allow);
// a handle (pp_destroy frees it) that works in its caller's memory: the two
// spectrum buffers of 'bytes' (pp_spectrum_bytes), and for the refined solve a
// quarter as much for the FP32 residual (null otherwise).  The caller binds the
// right-hand side and the solution (pp_bind_device_buffers) before a solve,
// keeps the memory longer than the handle, and runs handles that share it one
// after the other.
int pp_create_lent(int nx, int ny, int nz, void* spec_a, void* spec_b, size_t bytes, void* work, pp_solver_s** out);
