// Transform pass of the real families and of the periodic half spectra for
// power-of-two lengths N = 32 .. 1024: one real line is a complex FFT of
// M = N / 2 points,
//   z_m = v_{2m} + i v_{2m+1},  V_k = E_k + W_N^k O_k,  V_{M-k} = conj(E_k - W_N^k O_k),
//   E_k = (Z_k + conj Z_{M-k}) / 2,  O_k = (Z_k - conj Z_{M-k}) / (2 i)
// (v: the line in Makhoul's order for DCT-II / DST-II, the line itself for the
// real <-> half-spectrum pass; DCT-IV / DST-IV need no separation), with the
// same per-family pre/post-processing as pp_linepass.cu (see the reference
// citations there).
//
// What bounds such a pass is the L1 / shared-memory data pipe, not HBM: every
// point crosses it once per load, store, exchange and separation.  So here
//   * a thread holds E = 16 complex points (8 for N <= 128), T = M / E threads
//     a line: the FFT needs one exchange through shared memory up to N = 512
//     (two at 1024), where 8 points a thread and two lines to one FFT of N
//     need two (pp_lp2.cuh);
//   * the line goes from global memory straight into the registers of the
//     first radix-E pass and from the last pass straight out: no staged tile.
//     The strided (y) pass reads rows in any order for free (a row segment of
//     the tile's L columns is its unit); the contiguous (x) pass reads quads
//     x_{4s} .. x_{4s+3}, of which thread t keeps z_s and hands z_{M-1-s} to
//     thread T-1-t of the same warp by shuffles;
//   * the pair (k, M - k) meets in thread t = k mod T by one shuffle from
//     thread T - t (half the registers cross), which then emits the four
//     outputs k, N - k, M - k, M + k.  The strided pass maps threads so that
//     t and T - t share a warp.
//
// Measured at 512^3 FP64, ms per pass, two lines to one FFT of N with a staged
// tile (pp_lp2.cuh) -> here:
//             x forward       y forward       y inverse       x inverse
//   N-N    0.519 -> 0.373  0.571 -> 0.420  0.576 -> 0.423  0.574 -> 0.498
//   D-D    0.549 -> 0.409  0.591 -> 0.433  0.609 -> 0.446  0.614 -> 0.527
//   N-D    0.557 -> 0.366  0.605 -> 0.452  0.597 -> 0.475  0.683 -> 0.505
//   P-P    0.514 -> 0.337  (complex y lines)               0.573 -> 0.475
// i.e. 5.8, 5.1, 5.1 and 6.5 TB/s for N-N, 79 - 100 % of the measured copy rate.
// The loads of a pass are issued together, from precomputed pointers: with
// each point's index arithmetic between them the inverse passes took 0.60
// and 0.75 ms.
#pragma once

#include <type_traits>

#include "pp_common.cuh"
#include "pp_kernels.h"

namespace pp_rh {

// DST2 / DCT2 / DCT-IV and DST-IV / real -> half spectrum / half spectrum -> real
enum Fam : int { F_DST2 = 0, F_DCT2 = 1, F_Q4 = 2, F_R2C = 3, F_C2R = 4 };

template <typename T>
struct V2;
template <>
struct V2<double> {
    using type = double2;
};
template <>
struct V2<float> {
    using type = float2;
};

// ---- radix plan of M points, E a thread: radices E, E, .., the rest ------------------
constexpr int npass(int m, int e)
{
    int p = 0;
    while (m > 1) {
        m /= m < e ? m : e;
        ++p;
    }
    return p;
}
constexpr int radix(int m, int e, int pass)
{
    int r = m < e ? m : e;
    for (int i = 0; i < pass; ++i) {
        m /= r;
        r = m < e ? m : e;
    }
    return r;
}
constexpr int span(int m, int e, int pass)
{
    int s = 1;
    for (int i = 0; i < pass; ++i) s *= radix(m, e, i);
    return s;
}

// ---- DFTs in registers -----------------------------------------------------------------
template <int SIGN, typename C>
PP_D void d2(C& a, C& b)
{
    const C t = c_sub(a, b);
    a = c_add(a, b);
    b = t;
}
template <int SIGN, typename C>
PP_D void d4(C& v0, C& v1, C& v2, C& v3)
{
    const C a = c_add(v0, v2), b = c_sub(v0, v2), c = c_add(v1, v3), d = c_mul_si<SIGN>(c_sub(v1, v3));
    v0 = c_add(a, c);
    v2 = c_sub(a, c);
    v1 = c_add(b, d);
    v3 = c_sub(b, d);
}
// times e^{SIGN i pi / 4}, e^{SIGN 3 i pi / 4}
template <int SIGN, typename C>
PP_D C w8_1(C a)
{
    using R = typename CReal<C>::type;
    const R h = (R)0.70710678118654752440084436210484904;
    return mkc<C>(h * (a.x - SIGN * a.y), h * (a.y + SIGN * a.x));
}
template <int SIGN, typename C>
PP_D C w8_3(C a)
{
    using R = typename CReal<C>::type;
    const R h = (R)0.70710678118654752440084436210484904;
    return mkc<C>(h * (-a.x - SIGN * a.y), h * (-a.y + SIGN * a.x));
}
template <int SIGN, typename C>
PP_D C cmulc(C a, typename CReal<C>::type c, typename CReal<C>::type s)  // times c + SIGN i s
{
    return mkc<C>(a.x * c - SIGN * (a.y * s), a.y * c + SIGN * (a.x * s));
}
template <int SIGN, int R, typename C>
PP_D void dft(C* v)
{
    using Re = typename CReal<C>::type;
    if constexpr (R == 2) {
        d2<SIGN>(v[0], v[1]);
    } else if constexpr (R == 4) {
        d4<SIGN>(v[0], v[1], v[2], v[3]);
    } else if constexpr (R == 8) {
        d4<SIGN>(v[0], v[2], v[4], v[6]);
        d4<SIGN>(v[1], v[3], v[5], v[7]);
        const C o1 = w8_1<SIGN>(v[3]), o2 = c_mul_si<SIGN>(v[5]), o3 = w8_3<SIGN>(v[7]);
        const C e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6], o0 = v[1];
        v[0] = c_add(e0, o0);
        v[4] = c_sub(e0, o0);
        v[1] = c_add(e1, o1);
        v[5] = c_sub(e1, o1);
        v[2] = c_add(e2, o2);
        v[6] = c_sub(e2, o2);
        v[3] = c_add(e3, o3);
        v[7] = c_sub(e3, o3);
    } else {
        static_assert(R == 16, "radix 2, 4, 8 or 16");
        // 4 x 4: n = n1 + 4 n2, k = 4 k1 + k2 in place, then the digit swap
        const Re c1 = (Re)0.92387953251128675612818318939678829, s1 = (Re)0.38268343236508977172845998403039887;
#pragma unroll
        for (int i = 0; i < 4; ++i) d4<SIGN>(v[i], v[i + 4], v[i + 8], v[i + 12]);
        // v[n1 + 4 k2] times W_16^{n1 k2}
        v[5] = cmulc<SIGN>(v[5], c1, s1);
        v[9] = w8_1<SIGN>(v[9]);
        v[13] = cmulc<SIGN>(v[13], s1, c1);
        v[6] = w8_1<SIGN>(v[6]);
        v[10] = c_mul_si<SIGN>(v[10]);
        v[14] = w8_3<SIGN>(v[14]);
        v[7] = cmulc<SIGN>(v[7], s1, c1);
        v[11] = w8_3<SIGN>(v[11]);
        v[15] = cmulc<SIGN>(v[15], -c1, -s1);
#pragma unroll
        for (int i = 0; i < 4; ++i) d4<SIGN>(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
        // v[4 k2 + k1] = X_{k2 + 4 k1}
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = i + 1; j < 4; ++j) {
                const C x = v[4 * i + j];
                v[4 * i + j] = v[4 * j + i];
                v[4 * j + i] = x;
            }
    }
}

// point q of the R points times W^{q k}, W = e^{SIGN 2 pi i s / TN}, tw[m] =
// e^{-2 pi i m / TN}: the factors with q = 1, 2, 3, 4, 8, 12 from the table, the
// rest as one product of two of them
template <int SIGN, int R, typename C>
PP_D void twiddle(C* u, int ks, const C* __restrict__ tw)
{
    auto ld = [&](int q) -> C {
        C w = __ldg(&tw[q * ks]);
        if (SIGN > 0) w.y = -w.y;
        return w;
    };
    const C w1 = ld(1);
    u[1] = c_mul(u[1], w1);
    if constexpr (R >= 4) {
        const C w2 = ld(2), w3 = ld(3);
        u[2] = c_mul(u[2], w2);
        u[3] = c_mul(u[3], w3);
#pragma unroll
        for (int q = 4; q < R; q += 4) {
            const C wq = ld(q);
            u[q] = c_mul(u[q], wq);
            u[q + 1] = c_mul(u[q + 1], c_mul(w1, wq));
            u[q + 2] = c_mul(u[q + 2], c_mul(w2, wq));
            u[q + 3] = c_mul(u[q + 3], c_mul(w3, wq));
        }
    }
}

// ---- geometry of an instance -----------------------------------------------------------
template <int N, int E, int L, bool STR>
struct Geo {
    static constexpr int M = N / 2, T = M / E, NT = L * T;
    // a line's exchange stays in one warp in the contiguous pass
    static constexpr bool WARP = !STR;
    static_assert(STR || (T <= 32 && 32 % T == 0), "contiguous pass: a line within one warp");
    static_assert(!STR || ((L == 8 || L == 16) && (T % (32 / L) == 0 || NT < 32)), "strided pass: t and T - t in one warp");
    // slot of point i of line l: the strided pass keeps the lines side by side
    // (a phase of 8 lanes reads 8 lines of one point), the contiguous one pads
    // a slot every E points
    static constexpr int LP = M + M / E;
    static PP_D int slot(int l, int i) { return STR ? i * L + l : l * LP + i + i / E; }
    static constexpr int slots = STR ? M * L : L * LP;
};

template <int M, int E, int L, bool STR, int R, int NS, typename G, typename C>
PP_D void exchange(C* v, C* sb, int l, int t, bool again)
{
    constexpr int T = M / E;
    auto sync = [] {
        if constexpr (G::WARP) __syncwarp();
        else __syncthreads();
    };
    if (again) sync();  // the previous exchange has been read
#pragma unroll
    for (int g = 0; g < E / R; ++g) {
        const int b = t + g * T;
        const int base = (b / NS) * NS * R + (b % NS);
#pragma unroll
        for (int q = 0; q < R; ++q) sb[G::slot(l, base + q * NS)] = v[g * R + q];
    }
    sync();
}

// passes P.. of the FFT: exchange, gather, twiddle, butterflies; leaves point
// t + T j in v[j]
template <int SIGN, int M, int E, int L, bool STR, int P, typename G, typename C>
PP_D void passes(C* v, C* sb, int l, int t, const C* __restrict__ tw, int tws)
{
    constexpr int NP = npass(M, E), T = M / E;
    if constexpr (P < NP) {
        constexpr int RP = radix(M, E, P - 1), R = radix(M, E, P), NS = span(M, E, P);
        exchange<M, E, L, STR, RP, span(M, E, P - 1), G>(v, sb, l, t, P > 1);
#pragma unroll
        for (int g = 0; g < E / R; ++g)
#pragma unroll
            for (int q = 0; q < R; ++q) v[g * R + q] = sb[G::slot(l, t + g * T + q * (M / R))];
#pragma unroll
        for (int g = 0; g < E / R; ++g) {
            const int k = (t + g * T) % NS;
            twiddle<SIGN, R>(v + g * R, k * (M / (NS * R)) * tws, tw);
            dft<SIGN, R>(v + g * R);
        }
        if constexpr (P == NP - 1 && E != R) {
            // v[g R + q] holds point t + T (g + q E / R)
            C w[E];
#pragma unroll
            for (int j = 0; j < E; ++j) w[j] = v[j];
#pragma unroll
            for (int g = 0; g < E / R; ++g)
#pragma unroll
                for (int q = 0; q < R; ++q) v[g + q * (E / R)] = w[g * R + q];
        }
        passes<SIGN, M, E, L, STR, P + 1, G>(v, sb, l, t, tw, tws);
    }
}

PP_D double shf(double v, int src) { return __shfl_sync(0xffffffffu, v, src); }
PP_D float shf(float v, int src) { return __shfl_sync(0xffffffffu, v, src); }
template <typename C>
PP_D C shfc(C v, int src) { return mkc<C>(shf(v.x, src), shf(v.y, src)); }

// four adjacent values, 32-byte (FP64) or 16-byte (FP32) aligned
PP_D void ld4(const double* p, double* x)
{
    asm("ld.global.v4.f64 {%0,%1,%2,%3}, [%4];" : "=d"(x[0]), "=d"(x[1]), "=d"(x[2]), "=d"(x[3]) : "l"(p) : "memory");
}
PP_D void ld4(const float* p, float* x)
{
    const float4 v = *reinterpret_cast<const float4*>(p);
    x[0] = v.x;
    x[1] = v.y;
    x[2] = v.z;
    x[3] = v.w;
}
PP_D void st4(double* p, double a, double b, double c, double d)
{
    asm volatile("st.global.v4.f64 [%0], {%1,%2,%3,%4};" ::"l"(p), "d"(a), "d"(b), "d"(c), "d"(d) : "memory");
}

// the outputs of the inverse contiguous pass, CNT adjacent elements at
// off + q stride of every q < Q: the refinement epilogue, the solution P
// (complex-interleaved, zero imaginary part), or a real array
template <int Q, int CNT, typename Real>
PP_D void put_runs(const PPLinePassArgs& a, long off, int stride, int plane, const Real (*x)[CNT], Real sc)
{
    using C = typename V2<Real>::type;
    if (a.acc) {
        // u = u_prev + scale * correction + zero-mode constant, in FP64
        const double zc = a.zplane ? a.zscale * a.zplane[plane] : 0.0;
        double* u = a.acc + off;
#pragma unroll
        for (int q = 0; q < Q; ++q) {
            double r[CNT];
#pragma unroll
            for (int c = 0; c < CNT; ++c)
                r[c] = (a.acc_read ? u[q * stride + c] : 0.0) + a.out_scale * (double)x[q][c] + zc;
            if (a.dst) {
                double2* d = reinterpret_cast<double2*>(a.dst) + off + q * stride;
#pragma unroll
                for (int c = 0; c < CNT; ++c) d[c] = make_double2(r[c], 0.0);
            } else {
#pragma unroll
                for (int c = 0; c < CNT; ++c) u[q * stride + c] = r[c];
            }
        }
        return;
    }
    if (a.out_cplx) {
        C* d = reinterpret_cast<C*>(a.dst) + off;
        if constexpr (sizeof(Real) == 8 && CNT % 2 == 0) {  // (vec_out: pairs of points start on 32 bytes)
            if (a.vec_out) {
#pragma unroll
                for (int q = 0; q < Q; ++q)
#pragma unroll
                    for (int c = 0; c < CNT; c += 2)
                        st4(reinterpret_cast<double*>(d + q * stride + c), sc * x[q][c], 0.0, sc * x[q][c + 1], 0.0);
                return;
            }
        }
#pragma unroll
        for (int q = 0; q < Q; ++q)
#pragma unroll
            for (int c = 0; c < CNT; ++c) d[q * stride + c] = mkc<C>(sc * x[q][c], (Real)0);
        return;
    }
    Real* d = reinterpret_cast<Real*>(a.dst) + off;
#pragma unroll
    for (int q = 0; q < Q; ++q)
#pragma unroll
        for (int c = 0; c < CNT; ++c) d[q * stride + c] = sc * x[q][c];
}

template <typename Real, int N, int E, int L, int FAM, bool INV, bool STR>
PP_D void rh_body(const PPLinePassArgs& a)
{
    using C = typename V2<Real>::type;
    using G = Geo<N, E, L, STR>;
    constexpr int M = G::M, T = G::T;
    constexpr bool Q4 = FAM == F_Q4;
    extern __shared__ __align__(16) unsigned char rh_smem[];
    C* sb = reinterpret_cast<C*>(rh_smem);

    const int tid = threadIdx.x;
    const int tile = blockIdx.x;
    const int plane = tile / a.tiles_per_plane;
    const int l0 = (tile - plane * a.tiles_per_plane) * L;
    const int nl = min(L, a.nlines - l0);
    // thread -> (line l, t).  Contiguous: t fastest.  Strided: the line
    // fastest, and t in the order 0, T/2, 1, T-1, 2, T-2, ..
    int l, t, mirror, swap;  // lanes of thread T - t and T - 1 - t of this line
    const int lane = tid & 31;
    if constexpr (STR) {
        l = tid & (L - 1);
        const int s = tid / L;
        t = (s & 1) ? (s == 1 ? T / 2 : T - (s >> 1)) : (s >> 1);
        if (T == 1) t = 0;
        mirror = s < 2 ? lane : (lane ^ L);
        swap = 0;
    } else {
        l = tid / T;
        t = tid - l * T;
        mirror = (lane & ~(T - 1)) | ((T - t) & (T - 1));
        swap = lane ^ (T - 1);
    }
    const bool live = l < nl;
    const long base = (long)plane * a.plane_stride + (long)l0 * (a.tile_stride ? a.tile_stride : a.line_stride) +
                      (long)l * a.line_stride;
    const C* tw = reinterpret_cast<const C*>(a.tw);
    const C* cs = reinterpret_cast<const C*>(a.cs2);
    const Real* src = reinterpret_cast<const Real*>(a.src);
    const long es = a.elem_stride;
    // real value of element e of the line
    const int mul = a.in_cplx ? 2 : 1;
    auto X = [&](int e) -> Real { return src[(base + (long)e * es) * mul]; };

    C v[E];
    // ---- 1. registers of the first pass: point t + T q in v[q] ------------------------
    if constexpr (FAM == F_R2C || (!INV && !STR && !Q4)) {
        // contiguous, real input: quads (DCT-II, DST-II) or pairs (R2C)
        constexpr int W = FAM == F_R2C ? 2 : 4;  // adjacent elements a load
        Real x[E / (W / 2)][W];
#pragma unroll
        for (int q = 0; q < E / (W / 2); ++q) {
            const int e = W * (t + T * q);
#pragma unroll
            for (int c = 0; c < W; ++c) x[q][c] = (Real)0;
            if (live) {
                if (a.vec16) {
                    if constexpr (W == 4) {
                        ld4(src + base + e, x[q]);
                    } else {
                        const C p = *reinterpret_cast<const C*>(src + base + e);
                        x[q][0] = p.x;
                        x[q][1] = p.y;
                    }
                } else {
#pragma unroll
                    for (int c = 0; c < W; ++c) x[q][c] = X(e + c);
                }
            }
        }
        // the Dirichlet lift of the plain solve's forward x pass: b = f dz^2 - lift,
        // the dz^2 factor applied to the outputs
        if (a.rhs_scale && a.lift.any && live) {
            const double inv = 1.0 / (a.dz * a.dz);
            const PPLift& F = a.lift;
            const int j = l0 + l;
            const double* zr = (F.z0 && plane == 0) ? F.z0 + (long)a.nx * j
                               : (F.z1 && plane == a.nz - 1) ? F.z1 + (long)a.nx * j : nullptr;
            const double* yr = (F.y0 && j == 0) ? F.y0 + (long)a.nx * plane
                               : (F.y1 && j == a.ny - 1) ? F.y1 + (long)a.nx * plane : nullptr;
            if (zr || yr) {
#pragma unroll
                for (int q = 0; q < E / (W / 2); ++q)
#pragma unroll
                    for (int c = 0; c < W; ++c) {
                        const int e = W * (t + T * q) + c;
                        const double s = (zr ? zr[e] : 0.0) + (yr ? yr[e] : 0.0);
                        x[q][c] = (Real)((double)x[q][c] - s * inv);
                    }
            }
            if (F.x0 && t == 0) x[0][0] = (Real)((double)x[0][0] - F.x0[j + (long)a.ny * plane] * inv);
            if (F.x1 && t == T - 1)
                x[E / (W / 2) - 1][W - 1] =
                    (Real)((double)x[E / (W / 2) - 1][W - 1] - F.x1[j + (long)a.ny * plane] * inv);
        }
        if constexpr (FAM == F_R2C) {
#pragma unroll
            for (int q = 0; q < E; ++q) v[q] = mkc<C>(x[q][0], x[q][1]);
        } else {
            constexpr int H = E / 2;
#pragma unroll
            for (int q = 0; q < H; ++q) {
                if (FAM == F_DCT2) {
                    // z_s = x_{4s} + i x_{4s+2} here, z_{M-1-s} = x_{4s+3} + i x_{4s+1} at T-1-t
                    v[q] = mkc<C>(x[q][0], x[q][2]);
                    v[E - 1 - q] = shfc(mkc<C>(x[q][3], x[q][1]), swap);
                } else {
                    // x'_j = (-1)^j x_{N-1-j}: z_{M/2+s} = -(x_{4s} + i x_{4s+2}) here,
                    // z_{M/2-1-s} = x_{4s+3} + i x_{4s+1} at T-1-t
                    v[q + H] = mkc<C>(-x[q][0], -x[q][2]);
                    v[H - 1 - q] = shfc(mkc<C>(x[q][3], x[q][1]), swap);
                }
            }
        }
    } else if constexpr (!INV && !Q4) {
        // strided: the rows of z_m directly, from both ends of the line:
        // lower half (m < M/2) x_{4m} + i x_{4m+2}, upper half the odd rows from the
        // end; DST-II: x'_j = (-1)^j x_{N-1-j} swaps the two and negates the upper one
        constexpr int H = E / 2;
        const long st = es * mul, step = 4 * T * st;
        const Real* lo = src + base * mul + 4 * t * st;             // rows 4 t + 4 T q (+ 2)
        const Real* hi = src + base * mul + (N - 1 - 4 * t) * st;   // rows N-1 - 4 t - 4 T q (- 2)
        Real x[H][4];
        if (live) {
#pragma unroll
            for (int q = 0; q < H; ++q) {
                x[q][0] = lo[q * step];
                x[q][1] = lo[q * step + 2 * st];
                x[q][2] = hi[-q * step];
                x[q][3] = hi[-q * step - 2 * st];
            }
        } else {
#pragma unroll
            for (int q = 0; q < H; ++q) x[q][0] = x[q][1] = x[q][2] = x[q][3] = (Real)0;
        }
#pragma unroll
        for (int q = 0; q < H; ++q) {
            if (FAM == F_DCT2) {
                v[q] = mkc<C>(x[q][0], x[q][1]);
                v[q + H] = mkc<C>(x[q][2], x[q][3]);
            } else {
                v[q] = mkc<C>(x[q][2], x[q][3]);
                v[q + H] = mkc<C>(-x[q][0], -x[q][1]);
            }
        }
    } else if constexpr (Q4) {
        // z_m = (x_{2m} + i x_{N-1-2m}) e^{-i pi m / N}; DST-IV reverses its input
        const bool rev = a.kind == PP_KIND_DST4;
        if constexpr (STR) {
#pragma unroll
            for (int q = 0; q < E; ++q) v[q] = mkc<C>(0, 0);
            if (live) {
                const long st = es * mul, step = 2 * T * st;
                const Real* lo = src + base * mul + 2 * t * st;            // rows 2 m
                const Real* hi = src + base * mul + (N - 1 - 2 * t) * st;  // rows N-1 - 2 m
#pragma unroll
                for (int q = 0; q < E; ++q) v[q] = mkc<C>(lo[q * step], hi[-q * step]);
            }
            if (rev) {
#pragma unroll
                for (int q = 0; q < E; ++q) v[q] = mkc<C>(v[q].y, v[q].x);
            }
        } else {
            Real x[E][2];
#pragma unroll
            for (int q = 0; q < E; ++q) {
                const int e = 2 * (t + T * q);
                x[q][0] = x[q][1] = (Real)0;
                if (live) {
                    if (a.vec16) {
                        const C p = *reinterpret_cast<const C*>(src + base + e);
                        x[q][0] = p.x;
                        x[q][1] = p.y;
                    } else {
                        x[q][0] = X(e);
                        x[q][1] = X(e + 1);
                    }
                }
            }
            if (a.rhs_scale && a.lift.any && live) {
                const double inv = 1.0 / (a.dz * a.dz);
                const PPLift& F = a.lift;
                const int j = l0 + l;
                const double* zr = (F.z0 && plane == 0) ? F.z0 + (long)a.nx * j
                                   : (F.z1 && plane == a.nz - 1) ? F.z1 + (long)a.nx * j : nullptr;
                const double* yr = (F.y0 && j == 0) ? F.y0 + (long)a.nx * plane
                                   : (F.y1 && j == a.ny - 1) ? F.y1 + (long)a.nx * plane : nullptr;
                if (zr || yr) {
#pragma unroll
                    for (int q = 0; q < E; ++q)
#pragma unroll
                        for (int c = 0; c < 2; ++c) {
                            const int e = 2 * (t + T * q) + c;
                            const double s = (zr ? zr[e] : 0.0) + (yr ? yr[e] : 0.0);
                            x[q][c] = (Real)((double)x[q][c] - s * inv);
                        }
                }
                if (F.x0 && t == 0) x[0][0] = (Real)((double)x[0][0] - F.x0[j + (long)a.ny * plane] * inv);
                if (F.x1 && t == T - 1)
                    x[E - 1][1] = (Real)((double)x[E - 1][1] - F.x1[j + (long)a.ny * plane] * inv);
            }
            // x_{2p+1} belongs to z_{M-1-p}, at T-1-t
#pragma unroll
            for (int q = 0; q < E; ++q) {
                const Real o = shf(x[q][1], swap);
                v[E - 1 - q].y = o;
                v[q].x = x[q][0];
            }
            if (rev) {
#pragma unroll
                for (int q = 0; q < E; ++q) v[q] = mkc<C>(v[q].y, v[q].x);
            }
        }
#pragma unroll
        for (int q = 0; q < E; ++q) v[q] = c_mul(v[q], __ldg(&cs[t + T * q]));
    } else {
        // inverse: thread t forms Z_k and Z_{M-k}, k = t + T j, j < E / 2, from
        // V_k and V_{M-k}: A = V_k + conj V_{M-k}, B = e^{2 pi i k / N} (V_k - conj V_{M-k}),
        // Z_k = A + i B, Z_{M-k} = conj(A - i B); k = 0 with k = M / 2
        constexpr int H = E / 2;
        const Real h = (Real)0.70710678118654752440084436210484904;
        C zk[H], zm[H];  // V_k, V_{M-k}, then Z_k, Z_{M-k}
        C vh = mkc<C>(0, 0);  // V_{M/2} (thread 0)
        if constexpr (FAM == F_C2R) {
            const C* lo = reinterpret_cast<const C*>(src) + base + t;
            const C* hi = reinterpret_cast<const C*>(src) + base + (M - t);
#pragma unroll
            for (int j = 0; j < H; ++j) zk[j] = zm[j] = mkc<C>(0, 0);
            if (live && !a.in_cplx) {
                // the spectrum of a non-periodic y is real: the y transform drops the
                // imaginary part (src/signalProc.cpp:160-195)
                const Real* rl = src + base + t;
                const Real* rh = src + base + (M - t);
#pragma unroll
                for (int j = 0; j < H; ++j) {
                    zk[j].x = rl[T * j];
                    zm[j].x = rh[-T * j];
                }
                if (t == 0) vh.x = rl[M / 2];
            } else if (live) {
#pragma unroll
                for (int j = 0; j < H; ++j) {
                    zk[j] = lo[T * j];
                    zm[j] = hi[-T * j];
                }
                if (t == 0) vh = lo[M / 2];
            }
        } else {
            // X'_k, X'_{N-k}, X'_{M-k}, X'_{M+k}; in the place of k = 0's second and
            // fourth, k = M/2's X'_{M/2}, X'_{N-M/2}.  X'_k = X_k, or (-1)^k X_{N-1-k}
            // for DST-III (N, M even: the four have one sign, applied to V below)
            const long st = (FAM == F_DST2 ? -es : es) * mul, step = T * st;
            const Real* p = src + base * mul + (FAM == F_DST2 ? (N - 1) * es * mul : 0);
            const Real* pa = p + t * st;
            const Real* pb = p + (N - t) * st;
            const Real* pc = p + (M - t) * st;
            const Real* pd = p + (M + t) * st;
            Real x[H][4];
            if (live) {
#pragma unroll
                for (int j = 0; j < H; ++j) {
                    x[j][0] = pa[j * step];
                    x[j][1] = j == 0 ? *(t == 0 ? p + (M / 2) * st : pb) : pb[-j * step];
                    x[j][2] = pc[-j * step];
                    x[j][3] = j == 0 ? *(t == 0 ? p + (N - M / 2) * st : pd) : pd[j * step];
                }
            } else {
#pragma unroll
                for (int j = 0; j < H; ++j) x[j][0] = x[j][1] = x[j][2] = x[j][3] = (Real)0;
            }
            auto pre = [&](Real xk, Real xn, C w) -> C {  // (1/2) e^{i t_k} (X_k - i X_{N-k})
                return mkc<C>((Real)0.5 * (w.x * xk + w.y * xn), (Real)0.5 * (w.y * xk - w.x * xn));
            };
#pragma unroll
            for (int j = 0; j < H; ++j) {
                const bool z = j == 0 && t == 0;
                const C w = __ldg(&cs[z ? M / 2 : t + T * j]);
                // e^{i t_{M-k}} = e^{i pi / 4} e^{-i t_k}
                const C wm = mkc<C>(h * (w.x + w.y), h * (w.x - w.y));
                if (z) {
                    // V_0 and V_M are real
                    vh = pre(x[0][1], x[0][3], w);
                    if (FAM == F_DST2 && ((M / 2) & 1)) vh = mkc<C>(-vh.x, -vh.y);
                    zk[0] = mkc<C>((Real)0.5 * x[0][0], 0);
                    zm[0] = mkc<C>(h * x[0][2], 0);
                } else {
                    zk[j] = pre(x[j][0], x[j][1], w);
                    zm[j] = pre(x[j][2], x[j][3], wm);
                    if (FAM == F_DST2 && ((t + T * j) & 1)) {
                        zk[j] = mkc<C>(-zk[j].x, -zk[j].y);
                        zm[j] = mkc<C>(-zm[j].x, -zm[j].y);
                    }
                }
            }
        }
#pragma unroll
        for (int j = 0; j < H; ++j) {
            C w = __ldg(&tw[t + T * j]);  // e^{-2 pi i k / N}
            w.y = -w.y;
            const C Vk = zk[j], Vm = zm[j];
            if (j == 0 && t == 0) {
                // Z_0 = (V_0 + V_M) + i (V_0 - V_M), Z_{M/2} = 2 conj V_{M/2}
                zk[0] = mkc<C>(Vk.x + Vm.x, Vk.x - Vm.x);
                zm[0] = mkc<C>((Real)2 * vh.x, -(Real)2 * vh.y);
            } else {
                const C A = mkc<C>(Vk.x + Vm.x, Vk.y - Vm.y);
                const C B = c_mul(mkc<C>(Vk.x - Vm.x, Vk.y + Vm.y), w);
                zk[j] = mkc<C>(A.x - B.y, A.y + B.x);
                zm[j] = mkc<C>(A.x + B.y, B.x - A.y);
            }
        }
        // Z_{M-k} to thread T - t (register E-1-j; thread 0 keeps its own at E-j,
        // and k = M/2 at E/2)
#pragma unroll
        for (int j = 0; j < H; ++j) v[j] = zk[j];
        C r[H];
#pragma unroll
        for (int j = 0; j < H; ++j) r[j] = shfc(zm[j], mirror);
#pragma unroll
        for (int j = 0; j < H; ++j) {
            // register H + j: E-1-(H-1-j) from the mirror; thread 0: E-(H-j) for j > 0, k = M/2 at j = 0
            const C own = j == 0 ? zm[0] : zm[H - j];
            const C oth = r[H - 1 - j];
            v[H + j] = t == 0 ? own : oth;
        }
    }

    // ---- 2. the FFT of M points ------------------------------------------------------------
    constexpr int S = (INV && !Q4) ? +1 : -1;
    constexpr int TWS = Q4 ? 1 : 2;  // the table holds W_N (W_M for DCT-IV / DST-IV)
    dft<S, E>(v);
    passes<S, M, E, L, STR, 1, G>(v, sb, l, t, tw, TWS);

    // ---- 3. post-processing and stores --------------------------------------------------
    const Real sc = (Real)(a.out_scale * (a.rhs_scale ? a.dz * a.dz : 1.0));
    const bool ownst = a.o_elem_stride != 0;
    const long oes = ownst ? a.o_elem_stride : a.elem_stride;
    const long ols = ownst ? a.o_line_stride : a.line_stride;
    const long ops = ownst ? a.o_plane_stride : a.plane_stride;
    const long ots = ownst ? a.o_tile_stride : a.tile_stride;
    const long ob = (long)plane * ops + (long)l0 * (ots ? ots : ols) + (long)l * ols;
    Real* dst = reinterpret_cast<Real*>(a.dst);
    auto put = [&](int e, Real x) {
        if (live) dst[ob + (long)e * oes] = sc * x;
    };
    if constexpr (Q4) {
        // w_p = e^{-i pi (4p+1)/(4N)} Z_p: X_{2p} = c Re w_p, X_{N-1-2p} = -c Im w_p
        // (c = 2 forward, 1 inverse); DST-IV flips the sign of the odd outputs
        const Real c = INV ? (Real)1 : (Real)2;
        const Real so = a.kind == PP_KIND_DST4 ? c : -c;
#pragma unroll
        for (int j = 0; j < E; ++j) {
            const C w = c_mul(v[j], __ldg(&cs[M + t + T * j]));
            v[j] = mkc<C>(c * w.x, so * w.y);
        }
        if constexpr (STR) {
#pragma unroll
            for (int j = 0; j < E; ++j) {
                const int p = t + T * j;
                put(2 * p, v[j].x);
                put(N - 1 - 2 * p, v[j].y);
            }
        } else {
            Real x[E][2];
#pragma unroll
            for (int j = 0; j < E; ++j) {
                // X_{2p+1} from z_{M-1-p}, at T-1-t
                x[j][0] = v[j].x;
                x[j][1] = shf(v[E - 1 - j].y, swap);
            }
            if (live) {
                if constexpr (INV) {
                    put_runs<E>(a, ob + 2 * t, 2 * T, plane, x, sc);
                } else if (a.vec_out) {
                    C* d = reinterpret_cast<C*>(dst + ob + 2 * t);
#pragma unroll
                    for (int j = 0; j < E; ++j) d[j * T] = mkc<C>(sc * x[j][0], sc * x[j][1]);
                } else {
#pragma unroll
                    for (int j = 0; j < E; ++j) {
                        dst[ob + 2 * (t + j * T)] = sc * x[j][0];
                        dst[ob + 2 * (t + j * T) + 1] = sc * x[j][1];
                    }
                }
            }
        }
    } else if constexpr (!INV) {
        constexpr int H = E / 2;
        const Real h = (Real)0.70710678118654752440084436210484904;
#pragma unroll
        for (int j = 0; j < H; ++j) {
            const int k = t + T * j;
            const C snd = t == 0 ? v[(E - j) % E] : v[E - 1 - j];
            const C Zp = shfc(snd, mirror);
            const C Zk = v[j];
            auto emit = [&](int kk, C U) {  // X_kk = 2 Re U, X_{N-kk} = -2 Im U
                const Real xa = (Real)2 * U.x, xb = (Real)-2 * U.y;
                if (FAM == F_DST2) {
                    // output e = N-1-k with sign (-1)^e
                    const bool odd = ((N - 1 - kk) & 1) != 0;
                    put(N - 1 - kk, odd ? -xa : xa);
                    if (kk > 0) put(kk - 1, odd ? -xb : xb);
                } else {
                    put(kk, xa);
                    if (kk > 0) put(N - kk, xb);
                }
            };
            auto emit_c = [&](int kk, C V) {
                if (live) reinterpret_cast<C*>(dst)[ob + kk] = mkc<C>(sc * V.x, sc * V.y);
            };
            if (j == 0 && t == 0) {
                // k = 0 and M (real), and k = M/2 (V = conj Z)
                const Real v0 = Zk.x + Zk.y, vM = Zk.x - Zk.y;
                const C Vh = mkc<C>(v[H].x, -v[H].y);
                if constexpr (FAM == F_R2C) {
                    emit_c(0, mkc<C>(v0, 0));
                    emit_c(M, mkc<C>(vM, 0));
                    emit_c(M / 2, Vh);
                } else {
                    emit(0, mkc<C>(v0, 0));
                    const Real xM = (Real)2 * h * vM;
                    if (FAM == F_DST2) put(N - 1 - M, ((N - 1 - M) & 1) ? -xM : xM);
                    else put(M, xM);
                    const C w = __ldg(&cs[M / 2]);
                    emit(M / 2, mkc<C>(Vh.x * w.x + Vh.y * w.y, Vh.y * w.x - Vh.x * w.y));
                }
            } else {
            const C Ek = mkc<C>((Real)0.5 * (Zk.x + Zp.x), (Real)0.5 * (Zk.y - Zp.y));
            const C Ok = mkc<C>((Real)0.5 * (Zk.y + Zp.y), (Real)-0.5 * (Zk.x - Zp.x));
            const C WO = c_mul(Ok, __ldg(&tw[k]));
            const C Vk = c_add(Ek, WO);
            const C Vm = mkc<C>(Ek.x - WO.x, WO.y - Ek.y);
            if constexpr (FAM == F_R2C) {
                emit_c(k, Vk);
                emit_c(M - k, Vm);
            } else {
                const C w = __ldg(&cs[k]);  // (cos t_k, sin t_k)
                const C wm = mkc<C>(h * (w.x + w.y), h * (w.x - w.y));
                emit(k, mkc<C>(Vk.x * w.x + Vk.y * w.y, Vk.y * w.x - Vk.x * w.y));
                emit(M - k, mkc<C>(Vm.x * wm.x + Vm.y * wm.y, Vm.y * wm.x - Vm.x * wm.y));
            }
            }
        }
        if constexpr (FAM == F_R2C) {
            // the rows of the half spectra are padded to the y pass's tile width:
            // the padding columns are zeroed, since the y pass's row segments
            // carry them along
            for (int e = M + 1 + t; e < (int)ols; e += T)
                if (live) reinterpret_cast<C*>(dst)[ob + e] = mkc<C>(0, 0);
        }
    } else if constexpr (FAM == F_C2R) {
        Real x[E][2];
#pragma unroll
        for (int j = 0; j < E; ++j) {
            x[j][0] = v[j].x;
            x[j][1] = v[j].y;
        }
        if (live) put_runs<E>(a, ob + 2 * t, 2 * T, plane, x, sc);
    } else if constexpr (STR) {
        // DCT-III output order x_{2i} = v_i, x_{2i+1} = v_{N-1-i}; DST-III reverses
        // with sign (-1)^e
        constexpr int H = E / 2;
        if (live) {
            Real* lo = dst + ob + 4 * t * oes;
            Real* hi = dst + ob + (N - 1 - 4 * t) * oes;
            const long step = 4 * T * oes;
#pragma unroll
            for (int q = 0; q < H; ++q) {
                const C a_ = FAM == F_DCT2 ? v[q] : v[q + H];
                const C b_ = FAM == F_DCT2 ? v[q + H] : mkc<C>(-v[q].x, -v[q].y);
                lo[q * step] = sc * a_.x;
                lo[q * step + 2 * oes] = sc * a_.y;
                hi[-q * step] = sc * b_.x;
                hi[-q * step - 2 * oes] = sc * b_.y;
            }
        }
    } else {
        constexpr int H = E / 2;
        Real x[H][4];
#pragma unroll
        for (int q = 0; q < H; ++q) {
            const C o = shfc(v[(FAM == F_DCT2 ? E : H) - 1 - q], swap);
            if (FAM == F_DCT2) {
                x[q][0] = v[q].x;
                x[q][1] = o.y;
                x[q][2] = v[q].y;
                x[q][3] = o.x;
            } else {
                x[q][0] = v[q + H].x;
                x[q][1] = -o.y;
                x[q][2] = v[q + H].y;
                x[q][3] = -o.x;
            }
        }
        if (live) put_runs<H>(a, ob + 4 * t, 4 * T, plane, x, sc);
    }
}

// 16 points a thread: 128 registers, four CTAs of 128 threads per SM (no spills
// but a few bytes of DCT-IV); 8 points a thread: 80 registers, 768 threads per SM
template <typename Real, int N, int E, int L, int FAM, bool INV, bool STR>
__global__ void __launch_bounds__(Geo<N, E, L, STR>::NT, (E == 16 ? 512 : 768) / Geo<N, E, L, STR>::NT) rh_kernel(PPLinePassArgs a)
{
    rh_body<Real, N, E, L, FAM, INV, STR>(a);
}

// points a thread and lines a CTA of a length (contiguous / strided)
constexpr int points(int n) { return n <= 128 ? 8 : 16; }
constexpr int lines_c(int n) { return n >= 1024 ? 4 : n >= 512 ? 8 : 16; }
constexpr int lines_s(int n) { return n <= 128 ? 16 : 8; }

template <typename Real, int N, int FAM, bool INV, bool STR>
cudaError_t launch_one(const PPLinePassArgs& a, cudaStream_t st)
{
    constexpr int E = points(N), L = STR ? lines_s(N) : lines_c(N);
    using G = Geo<N, E, L, STR>;
    using C = typename V2<Real>::type;
    constexpr size_t smem = G::slots * sizeof(C);
    auto kfn = rh_kernel<Real, N, E, L, FAM, INV, STR>;
    if (smem > 48 * 1024) {
        const cudaError_t e = cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
    }
    kfn<<<a.nplanes * a.tiles_per_plane, G::NT, smem, st>>>(a);
    return cudaGetLastError();
}

template <typename Real, int N>
cudaError_t launch_n(const PPLinePassArgs& a, bool inverse, bool strided, cudaStream_t st)
{
    if (a.kind == PP_KIND_FFT) {
        if (strided || !a.half) return cudaErrorInvalidValue;
        return inverse ? launch_one<Real, N, F_C2R, true, false>(a, st) : launch_one<Real, N, F_R2C, false, false>(a, st);
    }
#define PP_RH(F)                                                                                                   \
    (strided ? (inverse ? launch_one<Real, N, F, true, true>(a, st) : launch_one<Real, N, F, false, true>(a, st)) \
             : (inverse ? launch_one<Real, N, F, true, false>(a, st) : launch_one<Real, N, F, false, false>(a, st)))
    switch (a.kind) {
    case PP_KIND_DST2: return PP_RH(F_DST2);
    case PP_KIND_DCT2: return PP_RH(F_DCT2);
    default: return PP_RH(F_Q4);
    }
#undef PP_RH
}

// lines a CTA (0: the length has no such kernel)
inline int lines(int n, bool strided)
{
    switch (n) {
    case 32: case 64: case 128: case 256: case 512: case 1024: return strided ? lines_s(n) : lines_c(n);
    default: return 0;
    }
}

template <typename Real>
cudaError_t launch(const PPLinePassArgs& a, bool inverse, bool strided, cudaStream_t st)
{
    switch (a.n) {
    case 32: return launch_n<Real, 32>(a, inverse, strided, st);
    case 64: return launch_n<Real, 64>(a, inverse, strided, st);
    case 128: return launch_n<Real, 128>(a, inverse, strided, st);
    case 256: return launch_n<Real, 256>(a, inverse, strided, st);
    case 512: return launch_n<Real, 512>(a, inverse, strided, st);
    case 1024: return launch_n<Real, 1024>(a, inverse, strided, st);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace pp_rh
