// Transform pass for line lengths other than powers of two whose FFT factors into
// 2, 3, 5, 7, 11 and 13, by a plan of radices: up to 4096 FFT points, less 46
// counts from 2860 on (2970, 3240, 3456, ..) that would need more butterflies a
// thread than its registers take and stay with the generic kernel.
//
// The same per-family pre/post-processing as pp_linepass.cu (see the reference
// citations there), on the fewest complex points:
//   even N: DCT-II/III, DST-II/III, DCT-IV / DST-IV and the periodic half
//     spectra run one real line as a complex FFT of M = N / 2 (pp_rhalf.cuh
//     has the algebra);
//   odd N: DCT-II/III and DST-II/III run two real lines as one complex FFT of
//     M = N (pp_lp2.cuh);
//   the full complex family: M = N.
// A CTA holds L FFT lines in shared memory, point i of line l at i LP + l, so
// that a phase of 8 lanes on 8 lines, or (LP odd) on 8 consecutive points of
// one line, reads 8 distinct banks.  Phases: (1) global memory -> FFT input,
// the pre-processing folded in (a thread forms the pair k, M - k of the
// inverse transforms); (2) Stockham passes in place, of radix up to 20: every
// thread reads its butterflies into registers, the CTA meets, and writes them
// back: two passes where M is a product of two such radices (107 of the 125
// counts up to 320, and 324, 360, 400), else three (125, 147, 243, 250, 500, ..),
// four for 40 counts from 625 on; (3) FFT output -> global memory with the
// post-processing.
//
// The lengths that people choose (pp_mr_ct_*.cu: the decimal edges 50, 60, 100,
// 200, 300, 500, 1000, the multiples 48, 96, 144, 192, 288, 384, 576, 768 and
// their like, even and of factors 2, 3 and 5) are instances with the plan known at
// compile time; the others take one kernel that reads it at run time, its passes
// functions of their own, where that beats the generic kernel (pays, pp_mr.cu).  Long
// contiguous lines m 2^k run the register kernel instead (pp_lpm_takes).
//
// What bounds it is the shared-memory pipe (about 8 + 8 + 16 passes + 8 + 8 bytes
// a point, 50 - 68 % busy), then the latency of the phases at 14 to 20 warps
// per SM; each phase issues all its loads, twiddles too, before it uses one (with
// loads and uses in turn 200^3 took 0.297 ms, at run time 0.42).  FP64, ms per
// solve, before (pp_linepass.cu; * a register kernel for m 2^k) -> run-time plan
// -> compile-time plan:
//   200^3 N-N            0.888 -> 0.34 -> 0.188    384^3 N-N *  1.25 -> 1.08
//   500 x 400 x 300 D-D  6.48      ->     1.33     192^3 P-P *  0.184 -> 0.146
//   1000 x 800 x 100     9.06  -> 4.2  -> 1.78     960^2 x 128 * 5.05 -> 3.02 (x by the
//                                                  register kernel; 3.52 all planned)
// The generic kernel of before (one complex FFT of N per real line, radix <= 8 in
// two ping-pong buffers, half a dozen passes over them) stays for larger prime
// factors, for odd lengths of DCT-IV / DST-IV and for small grids (pays).
#pragma once

#include "pp_rhalf.cuh"

namespace pp_mr {

using pp_rh::V2;

// ---- DFTs of R points in registers ------------------------------------------------------
// cos and sin of 2 pi m / P, m = 1 .. (P - 1) / 2 (folded at compile time)
template <int P>
PP_HD constexpr double prime_cos(int m)
{
    constexpr double c7[3] = {0.623489801858733530525004884004239810, -0.222520933956314404288902564496794760,
                              -0.900968867902419126236102319507445052};
    constexpr double c11[5] = {0.841253532831181168861811648919367717, 0.415415013001886425529274149229623203,
                               -0.142314838273285140443792668616369669, -0.654860733945285064056925072466293554,
                               -0.959492973614497389890368057066327700};
    constexpr double c13[6] = {0.885456025653209895900375522015098878, 0.568064746731155802511807559127516624,
                               0.120536680255323053349067687452543582, -0.354604887042535625969637892600018475,
                               -0.748510748171101098634630599701351384, -0.970941817426052027156982276293789228};
    return P == 7 ? c7[m - 1] : P == 11 ? c11[m - 1] : c13[m - 1];
}
template <int P>
PP_HD constexpr double prime_sin(int m)
{
    constexpr double s7[3] = {0.781831482468029808708444526674057750, 0.974927912181823607018131682993931217,
                              0.433883739117558120475768332848358754};
    constexpr double s11[5] = {0.540640817455597582107635954318691695, 0.909631995354518371411715383079028460,
                               0.989821441880932732376092037776718787, 0.755749574354258283774035843972344420,
                               0.281732556841429697711417915346616899};
    constexpr double s13[6] = {0.464723172043768545656015335133104777, 0.822983865893656394579617423439381990,
                               0.992708874098053992800751649492520179, 0.935016242685414823439784599837830729,
                               0.663122658240795202376785492666766279, 0.239315664287557767148753726260211895};
    return P == 7 ? s7[m - 1] : P == 11 ? s11[m - 1] : s13[m - 1];
}

// a prime P: sums and differences of the points j, P - j
template <int SIGN, int P, typename C>
PP_D void dft_prime(C* v)
{
    using R = typename CReal<C>::type;
    constexpr int H = (P - 1) / 2;
    C s[H], d[H];
#pragma unroll
    for (int j = 0; j < H; ++j) {
        s[j] = c_add(v[j + 1], v[P - 1 - j]);
        d[j] = c_sub(v[j + 1], v[P - 1 - j]);
    }
    const C v0 = v[0];
#pragma unroll
    for (int j = 0; j < H; ++j) v[0] = c_add(v[0], s[j]);
#pragma unroll
    for (int k = 1; k <= H; ++k) {
        C a = v0, b = mkc<C>(0, 0);
#pragma unroll
        for (int j = 1; j <= H; ++j) {
            const int m = (j * k) % P;
            const R c = (R)prime_cos<P>(m <= H ? m : P - m);
            const R sn = (R)(m <= H ? prime_sin<P>(m) : -prime_sin<P>(P - m));
            a = mkc<C>(a.x + c * s[j - 1].x, a.y + c * s[j - 1].y);
            b = mkc<C>(b.x + sn * d[j - 1].x, b.y + sn * d[j - 1].y);
        }
        b = c_mul_si<SIGN>(b);
        v[k] = c_add(a, b);
        v[P - k] = c_sub(a, b);
    }
}

template <int SIGN, int R, typename C>
PP_D void dft(C* v);

// R = A B, A and B coprime: n = (B n1 + A n2) mod R, and k the index with
// k = k1 mod A, k = k2 mod B, so that no twiddles come between (Good 1958)
template <int SIGN, int A, int B, typename C>
PP_D void dft_coprime(C* v)
{
    C y[B][A];
#pragma unroll
    for (int n2 = 0; n2 < B; ++n2) {
#pragma unroll
        for (int n1 = 0; n1 < A; ++n1) y[n2][n1] = v[(B * n1 + A * n2) % (A * B)];
        dft<SIGN, A>(y[n2]);
    }
    // multiples of B that are 1 mod A, of A that are 1 mod B
    constexpr auto unit = [](int step, int mod) constexpr {
        int x = step;
        while (x % mod != 1 % mod) x += step;
        return x;
    };
    constexpr int ua = unit(B, A), ub = unit(A, B);
#pragma unroll
    for (int k1 = 0; k1 < A; ++k1) {
        C z[B];
#pragma unroll
        for (int n2 = 0; n2 < B; ++n2) z[n2] = y[n2][k1];
        dft<SIGN, B>(z);
#pragma unroll
        for (int k2 = 0; k2 < B; ++k2) v[(ua * k1 + ub * k2) % (A * B)] = z[k2];
    }
}

template <int SIGN, typename C>
PP_D void dft9(C* v)
{
    using R = typename CReal<C>::type;
    const R c1 = (R)0.766044443118978035202392650555416673, s1 = (R)0.642787609686539326322643409907263432;
    const R c2 = (R)0.173648177666930348851716626769314796, s2 = (R)0.984807753012208059366743024589523013;
    const R c4 = (R)-0.939692620785908384054109277324731470, s4 = (R)0.342020143325668733044099614682259580;
    C y[3][3];
#pragma unroll
    for (int n2 = 0; n2 < 3; ++n2) {
#pragma unroll
        for (int n1 = 0; n1 < 3; ++n1) y[n2][n1] = v[3 * n1 + n2];
        dft3<SIGN>(y[n2]);
    }
    y[1][1] = pp_rh::cmulc<SIGN>(y[1][1], c1, s1);
    y[1][2] = pp_rh::cmulc<SIGN>(y[1][2], c2, s2);
    y[2][1] = pp_rh::cmulc<SIGN>(y[2][1], c2, s2);
    y[2][2] = pp_rh::cmulc<SIGN>(y[2][2], c4, s4);
#pragma unroll
    for (int k1 = 0; k1 < 3; ++k1) {
        C z[3] = {y[0][k1], y[1][k1], y[2][k1]};
        dft3<SIGN>(z);
#pragma unroll
        for (int k2 = 0; k2 < 3; ++k2) v[k1 + 3 * k2] = z[k2];
    }
}

template <int SIGN, int R, typename C>
PP_D void dft(C* v)
{
    if constexpr (R == 3) dft3<SIGN>(v);
    else if constexpr (R == 5) dft5<SIGN>(v);
    else if constexpr (R == 2 || R == 4 || R == 8 || R == 16) pp_rh::dft<SIGN, R>(v);
    else if constexpr (R == 7 || R == 11 || R == 13) dft_prime<SIGN, R>(v);
    else if constexpr (R == 9) dft9<SIGN>(v);
    else if constexpr (R == 6) dft_coprime<SIGN, 2, 3>(v);
    else if constexpr (R == 10) dft_coprime<SIGN, 2, 5>(v);
    else if constexpr (R == 12) dft_coprime<SIGN, 4, 3>(v);
    else if constexpr (R == 14) dft_coprime<SIGN, 2, 7>(v);
    else if constexpr (R == 15) dft_coprime<SIGN, 3, 5>(v);
    else if constexpr (R == 18) dft_coprime<SIGN, 2, 9>(v);
    else dft_coprime<SIGN, 4, 5>(v);  // 20
}

// butterflies of radix r that a thread holds at once, at most
PP_HD constexpr int held(int r) { return r <= 2 ? 8 : r == 3 ? 5 : r <= 5 ? 4 : r <= 10 ? 2 : 1; }

// ---- the plan of m points -----------------------------------------------------------------
// the radices: the fewest passes, then the largest smallest radix (balanced
// passes keep the same threads busy)
struct Radices {
    int npass = PP_MR_MAXPASS + 1, low = 0, r[PP_MR_MAXPASS] = {};
};
constexpr void search(int m, int from, int depth, int* cur, Radices& best)
{
    constexpr int radix[17] = {20, 18, 16, 15, 14, 13, 12, 11, 10, 9, 8, 7, 6, 5, 4, 3, 2};
    if (m == 1) {
        const int low = depth ? cur[depth - 1] : 0;
        if (depth < best.npass || (depth == best.npass && low > best.low)) {
            best.npass = depth;
            best.low = low;
            for (int i = 0; i < depth; ++i) best.r[i] = cur[i];
        }
        return;
    }
    if (depth >= PP_MR_MAXPASS || depth >= best.npass) return;
    for (int i = from; i < 17; ++i)
        if (m % radix[i] == 0) {
            cur[depth] = radix[i];
            search(m / radix[i], i, depth + 1, cur, best);  // not increasing
        }
}
constexpr unsigned magic_of(int d) { return d == 1 ? 0u : (unsigned)((1ull << 32) / d) + 1u; }

// Lines and threads: at most 4096 points (a 64 KB tile) and 256 threads; 8 or
// 16 lines where they fit (64 / 128-byte row segments of the strided pass), and
// the thread count (whole warps) that leaves the fewest idle in the passes'
// rounds, then about 12 points a thread.  m = 0 in the result: no plan.
constexpr PPMrPlan make_plan(int m)
{
    PPMrPlan p{};
    if (m < 4 || m > 4096) return p;
    Radices b;
    int cur[PP_MR_MAXPASS] = {};
    search(m, 0, 0, cur, b);
    if (b.npass > PP_MR_MAXPASS) return p;
    double top = -1.0;
    for (int o = 0; o < 5; ++o) {
        const int L = o == 0 ? 8 : o == 1 ? 16 : 4 >> (o - 2);
        if (m * L > 4096 || (o >= 2 && p.L)) continue;
        for (int t = 32; t <= 256; t += 32) {
            double util = 0.0;
            bool fits = true;
            for (int q = 0; q < b.npass; ++q) {
                const int total = m / b.r[q] * L, rounds = (total + t - 1) / t;
                fits = fits && rounds <= held(b.r[q]);
                util += (double)total / ((double)rounds * t) / b.npass;
            }
            const double off = (double)m * L / t - 12.0;
            const double score = util - 0.02 * (off < 0 ? -off : off) - (L == 16 ? 0.25 : 0.0);
            if (fits && score > top) {
                top = score;
                p.L = L;
                p.threads = t;
            }
        }
    }
    if (p.L == 0) return p;
    p.m = m;
    while ((1 << p.lgl) < p.L) ++p.lgl;
    p.npass = b.npass;
    int ns = 1;
    for (int q = 0; q < b.npass; ++q) {
        p.radix[q] = b.r[q];
        p.magic[q] = magic_of(ns);
        ns *= b.r[q];
    }
    return p;
}

// x / d for x < 2^17, d < 2^13, magic = floor(2^32 / d) + 1 (0: d = 1)
PP_D int fdiv(int x, unsigned magic) { return magic ? (int)__umulhi((unsigned)x, magic) : x; }

// One Stockham pass of radix R and span ns, in place: butterfly j of line l.
// B: butterflies a thread may hold; tg = threads >> lgl, threads a point index apart
template <int SIGN, int R, int B, typename C>
PP_D void pass_body(C* sb, int m, int L, int lgl, int LP, int ns, unsigned magic, int tg, const C* __restrict__ tw,
                    int tws, const C* __restrict__ pre)
{
    const int nb = m / R;
    const int l = threadIdx.x & (L - 1), j0 = threadIdx.x >> lgl;
    C* col = sb + l;
    C u[B][R];
    int out[B];
#pragma unroll
    for (int b = 0; b < B; ++b) {
        const int j = j0 + b * tg;
        if (j < nb) {
#pragma unroll
            for (int q = 0; q < R; ++q) u[b][q] = col[(j + q * nb) * LP];
            if (ns > 1) {
                const int hi = fdiv(j, magic), k = j - hi * ns;
                out[b] = hi * ns * R + k;
                const int ks = k * (nb / ns) * tws;  // W^{q k m / (ns R)}
#pragma unroll
                for (int q = 1; q < R; ++q) {
                    C f = __ldg(&tw[q * ks]);
                    if (SIGN > 0) f.y = -f.y;
                    u[b][q] = c_mul(u[b][q], f);
                }
            } else {
                out[b] = j * R;
                if (pre) {
#pragma unroll
                    for (int q = 0; q < R; ++q) u[b][q] = c_mul(u[b][q], __ldg(&pre[j + q * nb]));
                }
            }
            dft<SIGN, R>(u[b]);
        }
    }
    __syncthreads();
#pragma unroll
    for (int b = 0; b < B; ++b) {
        if (j0 + b * tg < nb) {
#pragma unroll
            for (int q = 0; q < R; ++q) col[(out[b] + q * ns) * LP] = u[b][q];
        }
    }
    __syncthreads();
}
// of a plan known at run time: a function of its own (inlined into the switch
// over the radices, the kernel spills 4 KB a thread)
template <int SIGN, int R, typename C>
__device__ __noinline__ void pass_rt(C* sb, int m, int L, int lgl, int LP, int ns, unsigned magic, int tg,
                                     const C* __restrict__ tw, int tws, const C* __restrict__ pre)
{
    pass_body<SIGN, R, held(R)>(sb, m, L, lgl, LP, ns, magic, tg, tw, tws, pre);
}

// A plan known at compile time (MT points a line), or at run time (MT = 0)
template <int MT>
struct Plan {
    static constexpr PPMrPlan P = make_plan(MT);
    PP_D explicit Plan(const PPMrPlan&) {}
    static constexpr int Pm = P.m, PL = P.L, Plgl = P.lgl, Pthreads = P.threads;
    static PP_D constexpr int m() { return Pm; }
    static PP_D constexpr int L() { return PL; }
    static PP_D constexpr int lgl() { return Plgl; }
    static PP_D constexpr int threads() { return Pthreads; }
    // items of a thread among n of every line
    static constexpr int items(int n) { return (n + P.threads / P.L - 1) / (P.threads / P.L); }
    static constexpr int points()  // held by a thread, at most
    {
        int e = 0;
        for (int q = 0; q < P.npass; ++q) {
            const int total = P.m / P.radix[q] * P.L, rounds = (total + P.threads - 1) / P.threads;
            if (rounds * P.radix[q] > e) e = rounds * P.radix[q];
        }
        return e;
    }
    template <int S, int Q, int NS, bool Q4, typename C>
    PP_D void passes(C* sb, int LP, const C* tw, int tws, const C* cs) const
    {
        if constexpr (Q < P.npass) {
            constexpr int R = P.radix[Q], total = P.m / R * P.L, B = (total + P.threads - 1) / P.threads;
            constexpr unsigned magic = P.magic[Q];
            pass_body<S, R, B>(sb, m(), L(), lgl(), LP, NS, magic, threads() >> lgl(), tw, tws,
                               Q4 && Q == 0 ? cs : nullptr);
            passes<S, Q + 1, NS * R, Q4>(sb, LP, tw, tws, cs);
        }
    }
};
template <>
struct Plan<0> {
    const PPMrPlan& p;
    PP_D explicit Plan(const PPMrPlan& q) : p(q) {}
    static constexpr int items(int) { return 0; }
    PP_D int m() const { return p.m; }
    PP_D int L() const { return p.L; }
    PP_D int lgl() const { return p.lgl; }
    PP_D int threads() const { return p.threads; }
    template <int S, int Q, int NS, bool Q4, typename C>
    PP_D void passes(C* sb, int LP, const C* tw, int tws, const C* cs) const
    {
        int ns = 1;
        const int tg = p.threads >> p.lgl;
        for (int q = 0; q < p.npass; ++q) {
            const int r = p.radix[q];
            const C* pt = Q4 && q == 0 ? cs : nullptr;
#define PP_MR_PASS(R) \
    case R: pass_rt<S, R>(sb, p.m, p.L, p.lgl, LP, ns, p.magic[q], tg, tw, tws, pt); break;
            switch (r) {
                PP_MR_PASS(2) PP_MR_PASS(3) PP_MR_PASS(4) PP_MR_PASS(5) PP_MR_PASS(6) PP_MR_PASS(7) PP_MR_PASS(8)
                PP_MR_PASS(9) PP_MR_PASS(10) PP_MR_PASS(11) PP_MR_PASS(12) PP_MR_PASS(13) PP_MR_PASS(14)
                PP_MR_PASS(15) PP_MR_PASS(16) PP_MR_PASS(18) PP_MR_PASS(20)
            }
#undef PP_MR_PASS
            ns *= r;
        }
    }
};

// real lines by even N (DCT-II/III, DST-II/III), DCT-IV / DST-IV (even N),
// half spectra (even N, contiguous), complex lines, real lines of odd N in pairs
enum Kind : int { K_REAL = 0, K_Q4 = 1, K_HALF = 2, K_CPLX = 3, K_PACK = 4 };

// Items i0, i0 + G, .. < n: U loads are issued together, then used
template <int U, typename LD, typename ST>
PP_D void staged(int i0, int n, int G, LD ld, ST st)
{
    for (int i = i0; i < n; i += U * G) {
        decltype(ld(0)) x[U];
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (i + u * G < n) x[u] = ld(i + u * G);
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (i + u * G < n) st(i + u * G, x[u]);
    }
}
template <typename R, typename C>
struct Quad {  // four values and the pair's twiddles
    R a, b, c, d;
    C w, v;
};

template <typename Real, int K, bool INV, bool STR, int MT>
PP_D void mr_body(const PPLinePassArgs& a, const PPMrPlan& pl)
{
    using C = typename V2<Real>::type;
    extern __shared__ __align__(16) unsigned char mr_smem[];
    C* sb = reinterpret_cast<C*>(mr_smem);
    const Plan<MT> p(pl);
    const int tid = threadIdx.x, nth = p.threads();
    const int M = p.m(), L = p.L(), lgl = p.lgl();
    // (N by the plan, so that it is a constant where the plan is)
    const int N = (K == K_CPLX || K == K_PACK) ? M : 2 * M;
    const int LP = STR || L == 1 ? L : L + 1;
    constexpr int ND = K == K_PACK ? 2 : 1;  // data lines of an FFT line
    const int tile = blockIdx.x;
    const int plane = tile / a.tiles_per_plane;
    const int l0 = (tile - plane * a.tiles_per_plane) * (L * ND);
    const int nl = min(L * ND, a.nlines - l0);
    // a thread keeps its line and steps through its points / pairs by G: the line
    // fastest in the strided pass, the points in the contiguous one
    const int G = nth >> lgl;
    const int l = STR ? tid & (L - 1) : tid / G;
    const int i0 = STR ? tid >> lgl : tid - l * G;
    const bool live = l * ND < nl, live2 = ND == 2 && 2 * l + 1 < nl;
    // unit strides: the elements of a line in the contiguous pass, the lines in
    // the strided one
    const long ls = STR ? 1 : a.line_stride, es = STR ? a.elem_stride : 1;
    const long at = (long)plane * a.plane_stride + (long)l0 * (a.tile_stride ? a.tile_stride : ls) + l * ND * ls;
    const int mul = a.in_cplx ? 2 : 1;
    const Real* src = reinterpret_cast<const Real*>(a.src) + at * mul;
    const C* srcc = reinterpret_cast<const C*>(a.src) + at;
    const long em = es * mul, lm = ls * mul;
    const C* tw = reinterpret_cast<const C*>(a.tw);
    const C* cs = reinterpret_cast<const C*>(a.cs2);
    const bool dst2 = a.kind == PP_KIND_DST2, rev = a.kind == PP_KIND_DST4;
    const Real h = (Real)0.70710678118654752440084436210484904;
    C* col = sb + l;  // point i at col[i LP]
    Real* rcol = reinterpret_cast<Real*>(col);
    auto half_at = [&](int j) -> Real& { return rcol[2 * ((j >> 1) * LP) + (j & 1)]; };  // real j of the line

    // the forward x pass of the plain solve subtracts the Dirichlet lift (b = f dz^2 -
    // lift, the dz^2 factor applied to the outputs) from the few elements on a face:
    // where they lie in the FFT input (1b), or as the odd lengths load them
    const PPLift& F = a.lift;
    const bool face = K == K_PACK && !INV && !STR && sizeof(Real) == 8 && a.rhs_scale && F.any &&
                      (F.x0 || F.x1 || (F.z0 && plane == 0) || (F.z1 && plane == a.nz - 1) || (F.y0 && l0 == 0) ||
                       (F.y1 && l0 + nl >= a.ny));
    auto lift = [&](int d, int e) -> Real {
        const int j = l0 + l * ND + d;
        double s = 0.0;
        if (F.z0 && plane == 0) s += F.z0[e + (long)a.nx * j];
        if (F.z1 && plane == a.nz - 1) s += F.z1[e + (long)a.nx * j];
        if (F.x0 && e == 0) s += F.x0[j + (long)a.ny * plane];
        if (F.x1 && e == a.nx - 1) s += F.x1[j + (long)a.ny * plane];
        if (F.y0 && j == 0) s += F.y0[e + (long)a.nx * plane];
        if (F.y1 && j == a.ny - 1) s += F.y1[e + (long)a.nx * plane];
        return (Real)(s / (a.dz * a.dz));
    };
    auto X = [&](int e) -> Real {  // real element e of the (first) line
        Real x = src[e * em];
        if (face) x -= lift(0, e);
        return x;
    };
    auto Y = [&](int e) -> Real {  // of the second line (K_PACK)
        if (!live2) return (Real)0;
        Real x = src[e * em + lm];
        if (face) x -= lift(1, e);
        return x;
    };
    auto pre = [&](Real xk, Real xn, C w) -> C {  // (1/2) e^{i t_k} (X_k - i X_{N-k})
        return mkc<C>((Real)0.5 * (w.x * xk + w.y * xn), (Real)0.5 * (w.y * xk - w.x * xn));
    };
    const int H = M / 2 + 1;  // pairs (k, M - k) of a line

    // loads in flight: every item of a thread where the plan is known at compile
    // time (about ten points), four otherwise; half as many of pairs
    constexpr int U = MT > 0 ? Plan<MT>::items(MT) : 4, UH = MT > 0 ? (Plan<MT>::items(MT / 2 + 1) + 1) / 2 : 2;
    static_assert(U <= 20 && UH <= 10, "registers for the loads in flight");

    // ---- 1. FFT input ------------------------------------------------------------------
    if (!live) {
        for (int i = i0; i < M; i += G) col[i * LP] = mkc<C>(0, 0);
    } else if constexpr (K == K_CPLX) {
        auto st = [&](int i, C v) { col[i * LP] = v; };
        if (a.in_cplx) staged<U>(i0, M, G, [&](int i) { return srcc[i * es]; }, st);
        else staged<U>(i0, M, G, [&](int i) { return mkc<C>(X(i), (Real)0); }, st);
    } else if constexpr (!STR && (K == K_HALF || K == K_Q4 || K == K_REAL) && (K == K_Q4 || !INV)) {
        // contiguous reals, in pairs x_{2i}, x_{2i+1}
        auto st = [&](int i, C v) {
            if constexpr (K == K_HALF) {
                col[i * LP] = v;
            } else if constexpr (K == K_Q4) {
                // raw z_m = x_{2m} + i x_{N-1-2m} (DST-IV: of the reversed line), its
                // factor e^{-i pi m / N} goes into the first pass: x_{2i} belongs to
                // z_i, x_{2i+1} to z_{M-1-i}
                rcol[2 * (i * LP) + (rev ? 1 : 0)] = v.x;
                rcol[2 * ((M - 1 - i) * LP) + (rev ? 0 : 1)] = v.y;
            } else {
                // Makhoul's order v_j = x'_{2j}, v_{N-1-j} = x'_{2j+1}; x' = x, or
                // x'_j = (-1)^j x_{N-1-j} for DST-II: x_{2i} is v_i, or -v_{M+i},
                // x_{2i+1} is v_{N-1-i}, or v_{M-1-i}
                half_at(dst2 ? M + i : i) = dst2 ? -v.x : v.x;
                half_at(dst2 ? M - 1 - i : N - 1 - i) = v.y;
            }
        };
        if (a.vec16) staged<U>(i0, M, G, [&](int i) { return reinterpret_cast<const C*>(src)[i]; }, st);
        else staged<2>(i0, M, G, [&](int i) { return mkc<C>(X(2 * i), X(2 * i + 1)); }, st);
    } else if constexpr (K == K_Q4) {
        staged<U>(i0, M, G, [&](int i) { return mkc<C>(X(2 * i), X(N - 1 - 2 * i)); },
                  [&](int i, C v) { col[i * LP] = rev ? mkc<C>(v.y, v.x) : v; });
    } else if constexpr (K == K_REAL && !INV) {
        // strided: the two rows of z_i = v_{2i} + i v_{2i+1}
        staged<U>(i0, M, G, [&](int i) {
            Real v[2];
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const int j = 2 * i + c;
                const bool lo = j < M;
                const int e = lo ? 2 * j : 2 * N - 1 - 2 * j;
                v[c] = X(dst2 ? N - 1 - e : e);
            }
            return mkc<C>(v[0], v[1]);
        }, [&](int i, C v) {
            if (dst2) {  // x'_j of the upper half carries the minus sign
                if (2 * i >= M) v.x = -v.x;
                if (2 * i + 1 >= M) v.y = -v.y;
            }
            col[i * LP] = v;
        });
    } else if constexpr (K == K_PACK && !INV) {
        // two lines a complex line, Makhoul's order
        staged<4>(i0, M, G, [&](int e) { return mkc<C>(X(e), Y(e)); },
                  [&](int e, C v) {
                      const int j = dst2 ? N - 1 - e : e;
                      if (dst2 && (j & 1)) v = mkc<C>(-v.x, -v.y);
                      col[((j & 1) ? N - 1 - (j >> 1) : (j >> 1)) * LP] = v;
                  });
    } else if constexpr (K == K_PACK) {
        // Z_k = V1_k + i V2_k and Z_{N-k} = conj V1_k + i conj V2_k, k <= (N - 1) / 2;
        // X'_k = X_k, or (-1)^k X_{N-1-k} for DST-III (N odd: k and N - k differ in sign)
        staged<2>(i0, H, G, [&](int k) {
            const int ea = dst2 ? N - 1 - k : k, eb = k == 0 ? ea : dst2 ? k - 1 : N - k;
            return Quad<Real, C>{X(ea), X(eb), Y(ea), Y(eb), __ldg(&cs[k]), C{}};
        }, [&](int k, const Quad<Real, C>& x) {
            C V1, V2;
            if (k == 0) {
                V1 = mkc<C>((Real)0.5 * x.a, 0);
                V2 = mkc<C>((Real)0.5 * x.c, 0);
            } else {
                const C w = x.w;
                const Real sa = (dst2 && (k & 1)) ? (Real)-1 : (Real)1, sn = dst2 ? -sa : sa;
                V1 = pre(sa * x.a, sn * x.b, w);
                V2 = pre(sa * x.c, sn * x.d, w);
            }
            col[k * LP] = mkc<C>(V1.x - V2.y, V1.y + V2.x);
            if (k > 0) col[(N - k) * LP] = mkc<C>(V1.x + V2.y, V2.x - V1.y);
        });
    } else {
        // inverse, even N: Z_k = A + i B, Z_{M-k} = conj(A - i B),
        // A = V_k + conj V_{M-k}, B = e^{2 pi i k / N} (V_k - conj V_{M-k})
        auto use = [&](int k, Quad<Real, C> x) {
            C Vk, Vm;
            if constexpr (K == K_HALF) {
                Vk = mkc<C>(x.a, k ? x.b : (Real)0);
                Vm = mkc<C>(x.c, k ? x.d : (Real)0);
            } else {
                if (dst2) {
                    if (k & 1) {
                        x.a = -x.a;
                        x.b = -x.b;
                    }
                    if ((M - k) & 1) {
                        x.c = -x.c;
                        x.d = -x.d;
                    }
                }
                if (k == 0) {
                    Vk = mkc<C>((Real)0.5 * x.a, 0);
                    Vm = mkc<C>(h * x.c, 0);
                } else {
                    const C w = x.w;
                    const C wm = mkc<C>(h * (w.x + w.y), h * (w.x - w.y));  // e^{i pi / 4} e^{-i t_k}
                    Vk = pre(x.a, x.b, w);
                    Vm = pre(x.c, x.d, wm);
                }
            }
            const C w = mkc<C>(x.v.x, -x.v.y);
            const C A = mkc<C>(Vk.x + Vm.x, Vk.y - Vm.y);
            const C B = c_mul(mkc<C>(Vk.x - Vm.x, Vk.y + Vm.y), w);
            col[k * LP] = mkc<C>(A.x - B.y, A.y + B.x);
            if (k > 0 && 2 * k != M) col[(M - k) * LP] = mkc<C>(A.x + B.y, B.x - A.y);
        };
        if constexpr (K == K_HALF) {
            if (a.in_cplx)
                staged<UH>(i0, H, G, [&](int k) {
                    const C p_ = srcc[k], q_ = srcc[M - k];
                    return Quad<Real, C>{p_.x, p_.y, q_.x, q_.y, C{}, __ldg(&tw[k])};
                }, use);
            else  // the spectrum of a non-periodic y is real: the y transform drops the
                  // imaginary part (src/signalProc.cpp:160-195)
                staged<UH>(i0, H, G, [&](int k) {
                    return Quad<Real, C>{src[k], (Real)0, src[M - k], (Real)0, C{}, __ldg(&tw[k])};
                }, use);
        } else {
            staged<UH>(i0, H, G, [&](int k) {
                // X'_k, X'_{N-k}, X'_{M-k}, X'_{M+k}; X'_k = X_k, or (-1)^k X_{N-1-k} for DST-III
                const int ea = dst2 ? N - 1 - k : k, eb = k == 0 ? ea : dst2 ? k - 1 : N - k;
                const int ec = dst2 ? N - 1 - M + k : M - k, ed = dst2 ? N - 1 - M - k : M + k;
                return Quad<Real, C>{X(ea), X(eb), X(ec), X(ed < 0 ? 0 : ed), __ldg(&cs[k]), __ldg(&tw[k])};
            }, use);
        }
    }
    // ---- 1b. the lift, where the face's elements lie: tests between the loads or in
    //      their use cost every grid with boundary data on x (320^3 D-D, forward x
    //      0.298 ms, 0.152 now, 0.112 without data) and registers every other one ----------
    if constexpr (!INV && !STR && K != K_PACK && sizeof(Real) == 8) {
        if (a.rhs_scale && F.any &&
            (F.x0 || F.x1 || (F.z0 && plane == 0) || (F.z1 && plane == a.nz - 1) || (F.y0 && l0 == 0) ||
             (F.y1 && l0 + nl >= a.ny))) {
            __syncthreads();
            const int j = l0 + l;  // y row of the line
            const double* zr = (F.z0 && plane == 0) ? F.z0 + (long)a.nx * j
                               : (F.z1 && plane == a.nz - 1) ? F.z1 + (long)a.nx * j : nullptr;
            const double* yr = (F.y0 && j == 0) ? F.y0 + (long)a.nx * plane
                               : (F.y1 && j == a.ny - 1) ? F.y1 + (long)a.nx * plane : nullptr;
            auto take = [&](int e) {
                double s = zr ? zr[e] : 0.0;
                if (F.x0 && e == 0) s += F.x0[j + (long)a.ny * plane];
                if (F.x1 && e == N - 1) s += F.x1[j + (long)a.ny * plane];
                if (yr) s += yr[e];
                const double v = s / (a.dz * a.dz);
                const int i = e >> 1;
                if constexpr (K == K_CPLX) {
                    rcol[2 * e * LP] -= v;
                } else if constexpr (K == K_HALF) {
                    half_at(e) -= v;
                } else if constexpr (K == K_Q4) {
                    rcol[(e & 1) ? 2 * ((M - 1 - i) * LP) + (rev ? 0 : 1) : 2 * (i * LP) + (rev ? 1 : 0)] -= v;
                } else {
                    Real& x = half_at((e & 1) ? (dst2 ? M - 1 - i : N - 1 - i) : dst2 ? M + i : i);
                    x = dst2 && !(e & 1) ? x + v : x - v;
                }
            };
            if (live && (zr || yr)) {
                for (int e = i0; e < N; e += G) take(e);
            } else if (live && i0 == 0) {
                if (F.x0) take(0);
                if (F.x1) take(N - 1);
            }
        }
    }
    __syncthreads();

    // ---- 2. the FFT ----------------------------------------------------------------------
    constexpr int S = (INV && K != K_Q4) ? +1 : -1;
    constexpr int TWS = (K == K_REAL || K == K_HALF) ? 2 : 1;  // the table holds W_N (W_M otherwise)
    p.template passes<S, 0, 1, K == K_Q4>(sb, LP, tw, TWS, cs);

    // ---- 3. outputs ------------------------------------------------------------------------
    if (!live) return;
    const Real sc = (Real)(a.out_scale * (a.rhs_scale ? a.dz * a.dz : 1.0));
    const bool own = a.o_elem_stride != 0;
    const long oes = STR ? (own ? a.o_elem_stride : a.elem_stride) : 1;
    const long ols = STR ? 1 : (own ? a.o_line_stride : a.line_stride);
    const long ops = own ? a.o_plane_stride : a.plane_stride;
    const long ots = own ? a.o_tile_stride : a.tile_stride;
    const long ob = (long)plane * ops + (long)l0 * (ots ? ots : ols) + l * ND * ols;
    Real* dst = reinterpret_cast<Real*>(a.dst) + ob;
    C* dstc = reinterpret_cast<C*>(a.dst) + ob;
    // one output of line d of the FFT line (inverse contiguous: the solution or the epilogue)
    auto put = [&](int d, int e, Real x) {
        if constexpr (INV && !STR) {
            const Real v[1][1] = {{x}};
            pp_rh::put_runs<1>(a, ob + d * ols + e, 0, plane, v, sc);
        } else {
            dst[d * ols + e * oes] = sc * x;
        }
    };
    // pairs of adjacent outputs 2i, 2i + 1 of the contiguous passes: val(i) gives both
    auto put_pairs = [&](auto val) {
        if constexpr (!INV) {
            if (a.vec_out) {
#pragma unroll 4
                for (int i = i0; i < M; i += G) {
                    const C v = val(i);
                    reinterpret_cast<C*>(dst)[i] = mkc<C>(sc * v.x, sc * v.y);
                }
                return;
            }
        } else if constexpr (sizeof(Real) == 8) {
            if (!a.acc && a.out_cplx && a.vec_out) {
#pragma unroll 4
                for (int i = i0; i < M; i += G) {
                    const C v = val(i);
                    pp_rh::st4(reinterpret_cast<double*>(dstc + 2 * i), sc * v.x, 0.0, sc * v.y, 0.0);
                }
                return;
            }
        } else if (a.acc && a.dst) {
            // the refined solve's last sweep: u + scale * correction + zero-mode constant
            const double zc = a.zplane ? a.zscale * a.zplane[plane] : 0.0;
            double2* P = reinterpret_cast<double2*>(a.dst) + ob;
            staged<U>(i0, M, G, [&](int i) {
                return a.acc_read ? make_double2(a.acc[ob + 2 * i], a.acc[ob + 2 * i + 1]) : make_double2(0.0, 0.0);
            }, [&](int i, double2 u) {
                const C v = val(i);
                P[2 * i] = make_double2(u.x + a.out_scale * (double)v.x + zc, 0.0);
                P[2 * i + 1] = make_double2(u.y + a.out_scale * (double)v.y + zc, 0.0);
            });
            return;
        }
        for (int i = i0; i < M; i += G) {
            const C v = val(i);
            put(0, 2 * i, v.x);
            put(0, 2 * i + 1, v.y);
        }
    };
    // the padding columns of the spectrum's rows stay zero
    if constexpr (!INV && !STR && K != K_HALF) {
        for (int e = N + i0; e < (int)ols; e += G)
#pragma unroll
            for (int d = 0; d < ND; ++d) {
                if (d == 1 && !live2) continue;
                if (a.out_cplx) dstc[d * ols + e] = mkc<C>(0, 0);
                else dst[d * ols + e] = (Real)0;
            }
    }
    // DCT-II value pair of U = e^{-i t_k} V_k: X_k = 2 Re U, X_{N-k} = -2 Im U;
    // DST-II: output e = N-1-k with sign (-1)^e
    auto emit = [&](int d, int k, C V, C w, bool second) {
        const C U = mkc<C>(V.x * w.x + V.y * w.y, V.y * w.x - V.x * w.y);
        Real xa = (Real)2 * U.x, xb = (Real)-2 * U.y;
        const int ea = dst2 ? N - 1 - k : k, eb = dst2 ? k - 1 : N - k;
        if (dst2 && (ea & 1)) xa = -xa;
        if (dst2 && (eb & 1)) xb = -xb;
        put(d, ea, xa);
        if (second) put(d, eb, xb);
    };
    if constexpr (K == K_CPLX) {
#pragma unroll 4
        for (int i = i0; i < M; i += G) {
            const C z = col[i * LP];
            if (a.acc) {
                const Real v[1][1] = {{z.x}};
                pp_rh::put_runs<1>(a, ob + i * oes, 0, plane, v, sc);
            } else if (a.out_cplx) {
                dstc[i * oes] = mkc<C>(sc * z.x, sc * z.y);
            } else {
                dst[i * oes] = sc * z.x;
            }
        }
    } else if constexpr (K == K_Q4) {
        // w_p = e^{-i pi (4p+1)/(4N)} Z_p: X_{2p} = c Re w_p, X_{N-1-2p} = -c Im w_p
        // (c = 2 forward, 1 inverse); DST-IV flips the sign of the odd outputs
        const Real c = INV ? (Real)1 : (Real)2;
        const Real so = rev ? c : -c;
        if constexpr (STR)
            staged<(U + 1) / 2>(i0, M, G, [&](int i) {
                const C z = col[i * LP], w = __ldg(&cs[M + i]);
                return Quad<Real, C>{z.x, z.y, w.x, w.y, C{}, C{}};
            }, [&](int i, const Quad<Real, C>& z) {
                put(0, 2 * i, c * (z.a * z.c - z.b * z.d));
                put(0, N - 1 - 2 * i, so * (z.a * z.d + z.b * z.c));
            });
        else put_pairs([&](int i) {
            const C z = col[i * LP], w = __ldg(&cs[M + i]);
            const C zn = col[(M - 1 - i) * LP], wn = __ldg(&cs[N - 1 - i]);
            return mkc<C>(c * (z.x * w.x - z.y * w.y), so * (zn.x * wn.y + zn.y * wn.x));
        });
    } else if constexpr (K == K_HALF && INV) {
        put_pairs([&](int i) { return col[i * LP]; });
    } else if constexpr ((K == K_REAL || K == K_HALF) && !INV) {
        // E = (Z_k + conj Z_{M-k}) / 2, O = (Z_k - conj Z_{M-k}) / (2 i):
        // V_k = E + W_N^k O, V_{M-k} = conj(E - W_N^k O); k = 0 with M, both real
        staged<UH>(i0, H, G, [&](int k) {
            const C Zk = col[k * LP], Zp = col[(k ? M - k : 0) * LP];
            return Quad<Real, C>{Zk.x, Zk.y, Zp.x, Zp.y, K == K_HALF ? C{} : __ldg(&cs[k]), __ldg(&tw[k])};
        }, [&](int k, const Quad<Real, C>& z) {
            const C Ek = mkc<C>((Real)0.5 * (z.a + z.c), (Real)0.5 * (z.b - z.d));
            const C Ok = mkc<C>((Real)0.5 * (z.b + z.d), (Real)-0.5 * (z.a - z.c));
            const C WO = c_mul(Ok, z.v);
            const C Vk = c_add(Ek, WO), Vm = mkc<C>(Ek.x - WO.x, WO.y - Ek.y);
            if constexpr (K == K_HALF) {
                dstc[k] = mkc<C>(sc * Vk.x, sc * Vk.y);
                if (2 * k != M) dstc[M - k] = mkc<C>(sc * Vm.x, sc * Vm.y);
            } else {
                const C w = z.w;
                const C wm = mkc<C>(h * (w.x + w.y), h * (w.x - w.y));
                emit(0, k, Vk, w, k > 0);
                if (2 * k != M) emit(0, M - k, Vm, wm, k > 0);  // (M = N - M)
            }
        });
        if constexpr (K == K_HALF) {
            // the padding columns of the rows are zeroed: the y pass's row
            // segments carry them along
            for (int e = M + 1 + i0; e < (int)ols; e += G) dstc[e] = mkc<C>(0, 0);
        }
    } else if constexpr (K == K_PACK && !INV) {
        // X_k and X_{N-k} of both lines from Z_k and Z_{N-k}
#pragma unroll 2
        for (int k = i0; k < H; k += G) {
            const C Zk = col[k * LP], Zn = col[(k ? N - k : 0) * LP];
            const C w = __ldg(&cs[k]);
            emit(0, k, mkc<C>((Real)0.5 * (Zk.x + Zn.x), (Real)0.5 * (Zk.y - Zn.y)), w, k > 0);
            if (live2) emit(1, k, mkc<C>((Real)0.5 * (Zk.y + Zn.y), (Real)-0.5 * (Zk.x - Zn.x)), w, k > 0);
        }
    } else if constexpr (K == K_PACK) {
#pragma unroll 4
        for (int e = i0; e < M; e += G) {
            const int j = dst2 ? N - 1 - e : e;
            C z = col[((j & 1) ? N - 1 - (j >> 1) : (j >> 1)) * LP];
            if (dst2 && (e & 1)) z = mkc<C>(-z.x, -z.y);
            put(0, e, z.x);
            if (live2) put(1, e, z.y);
        }
    } else {
        // DCT-III / DST-III: x_e = v_{pos(e)}, or (-1)^e v_{pos(N-1-e)}
        if constexpr (STR) {
#pragma unroll 4
            for (int i = i0; i < M; i += G) {
                const C z = col[i * LP];
                const Real v[2] = {z.x, z.y};
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    const int j = 2 * i + c;
                    const int e = j < M ? 2 * j : 2 * N - 1 - 2 * j;
                    const int o = dst2 ? N - 1 - e : e;
                    put(0, o, dst2 && (o & 1) ? -v[c] : v[c]);
                }
            }
        } else {
            put_pairs([&](int i) {
                const Real xa = half_at(dst2 ? M + i : i);
                const Real xb = half_at(dst2 ? M - 1 - i : N - 1 - i);
                return mkc<C>(xa, dst2 ? -xb : xb);
            });
        }
    }
}

// the run-time planned kernel
template <typename Real, int K, bool INV, bool STR>
__global__ void __launch_bounds__(256, 2) mr_kernel(PPLinePassArgs a, PPMrPlan p)
{
    mr_body<Real, K, INV, STR, 0>(a, p);
}
// planned at compile time: M points
constexpr int ct_blocks(int points, int threads, bool f32_forward)
{
    return (points <= 10 ? 768 : points <= 12 || f32_forward ? 640 : 512) / threads;
}
template <typename Real, int K, bool INV, bool STR, int M>
__global__ void __launch_bounds__(Plan<M>::P.threads, ct_blocks(Plan<M>::points(), Plan<M>::P.threads, sizeof(Real) == 4 && !INV && !STR))
mrc_kernel(PPLinePassArgs a)
{
    mr_body<Real, K, INV, STR, M>(a, PPMrPlan{});
}

template <typename Real, int K, int M>
cudaError_t launch_kind(const PPLinePassArgs& a, const PPMrPlan& p, bool inverse, bool strided, cudaStream_t st)
{
    using C = typename V2<Real>::type;
    const size_t smem = (size_t)p.m * (strided || p.L == 1 ? p.L : p.L + 1) * sizeof(C);
    auto go = [&](auto kfn, auto... more) -> cudaError_t {
        if (smem > 48 * 1024) {
            const cudaError_t e = cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
            if (e != cudaSuccess) return e;
        }
        kfn<<<a.nplanes * a.tiles_per_plane, p.threads, smem, st>>>(a, more...);
        return cudaGetLastError();
    };
    // (contiguous FP64 passes that run the register kernel of pp_lp2.cuh have no instance here)
    constexpr auto elsewhere = [](bool inv, bool str) constexpr {
        const int n = K == K_CPLX ? M : 2 * M;
        const int kind = K == K_REAL ? (int)PP_KIND_DCT2 : K == K_Q4 ? (int)PP_KIND_DCT4 : (int)PP_KIND_FFT;
        return M > 0 && sizeof(Real) == 8 && !str && pp_lpm_takes(n, kind, K == K_HALF, inv);
    };
#define PP_MR(INV, STR)                                                                    \
    do {                                                                                   \
        if constexpr (elsewhere(INV, STR)) return cudaErrorInvalidValue;                   \
        else if constexpr (M > 0) return go(mrc_kernel<Real, K, INV, STR, M>);             \
        else return go(mr_kernel<Real, K, INV, STR>, p);                                   \
    } while (0)
    if constexpr (K == K_HALF) {
        if (strided) return cudaErrorInvalidValue;
        if (inverse) PP_MR(true, false);
        PP_MR(false, false);
    } else {
        if (inverse && strided) PP_MR(true, true);
        if (inverse) PP_MR(true, false);
        if (strided) PP_MR(false, true);
        PP_MR(false, false);
    }
#undef PP_MR
}

template <typename Real>
cudaError_t launch_real(const PPLinePassArgs& a, const PPMrPlan& p, bool inverse, bool strided, cudaStream_t st)
{
    if (a.kind == PP_KIND_DST2 || a.kind == PP_KIND_DCT2)
        return a.n % 2 ? launch_kind<Real, K_PACK, 0>(a, p, inverse, strided, st)
                       : launch_kind<Real, K_REAL, 0>(a, p, inverse, strided, st);
    return launch_kind<Real, K_Q4, 0>(a, p, inverse, strided, st);
}
template <typename Real>
cudaError_t launch_periodic(const PPLinePassArgs& a, const PPMrPlan& p, bool inverse, bool strided, cudaStream_t st)
{
    return a.half ? launch_kind<Real, K_HALF, 0>(a, p, inverse, strided, st)
                  : launch_kind<Real, K_CPLX, 0>(a, p, inverse, strided, st);
}
// the length N planned at compile time
template <typename Real, int N>
cudaError_t launch_ct(const PPLinePassArgs& a, const PPMrPlan& p, bool inverse, bool strided, cudaStream_t st)
{
    if (a.kind == PP_KIND_FFT)
        return a.half ? launch_kind<Real, K_HALF, N / 2>(a, p, inverse, strided, st)
                      : launch_kind<Real, K_CPLX, N>(a, p, inverse, strided, st);
    if (a.kind == PP_KIND_DST2 || a.kind == PP_KIND_DCT2)
        return launch_kind<Real, K_REAL, N / 2>(a, p, inverse, strided, st);
    return launch_kind<Real, K_Q4, N / 2>(a, p, inverse, strided, st);
}

}  // namespace pp_mr
