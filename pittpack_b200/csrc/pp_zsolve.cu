// Batched z-direction tridiagonal solve.
//
// The reference gathers each strided z-line into a buffer and runs a serial
// Thomas sweep per line (solveThmBatch, src/pencilDcmp.cpp:5066-5105 ->
// TriDiag::thomasLowMem, src/triDiag.cpp:1693-1822; periodic z through
// TriDiag::shermanMorrisonThomas, src/triDiag.cpp:1961-2108).  The system of
// mode (kx, ky) is
//     x_{k-1} + lambda x_k + x_{k+1} = r_k,   lambda = getEigenVal(ky, kx)
//     (src/pencilDcmp.cpp:4393-4417), computed here on the fly per system,
// with the ends modified by the z boundary: Dirichlet b = lambda - 1, Neumann
// b = lambda + 1 (src/triDiag.cpp:1733-1751), periodic: cyclic corners 1.
// Zero mode (|lambda + 2| < 1e-10): the reference replaces row 0 by x_0 = r_0
// (src/triDiag.cpp:1753-1776); for periodic z it solves the cyclic system
// with row 0 replaced by x_0 + x_{N-1} = (r_0 + r_{N-1}) / 2
// (shermanMorrisonThomasV1, src/triDiag.cpp:2112-2255).
//
// B200 layout and algorithm:
//   * a CTA owns TS adjacent kx columns of one ky row; it reads the TS x nz
//     tile into shared memory, solves, and writes the tile back: in the
//     z-tiled layout (the tile one contiguous block) with one bulk copy per
//     lane's block of rows where the rows live in registers, else with
//     coalesced row segments (rows skewed by one slot every 16 to spread
//     banks);
//   * a group of P lanes (P = 32 / systems per warp) solves one system by the
//     partition method: lane L owns a contiguous block of M ~ nz/P rows and
//     eliminates it so that every interior unknown is expressed through the
//     block's first and last unknown (a forward sweep, a backward sweep for
//     the first row, a recovery sweep), leaving two equations per lane; the
//     rows stay in registers where the counts allow.  Interior rows have the
//     same coefficients in every block, so the pivots and spikes of a block
//     depend only on lambda; the CTA builds them into a shared table (one
//     reciprocal per entry) that every lane reads, and the sweeps do not
//     divide: the system's first and last rows scale their blocks' ends;
//   * eliminating each lane's first unknown leaves a P-row tridiagonal system
//     in the lanes' last unknowns, solved by parallel cyclic reduction over
//     warp shuffles (on the ring of lanes for periodic systems); each lane
//     then recovers its interior rows;
//   * every elimination carries a row by its off-diagonals and its sum, and
//     forms the diagonal from them (Grassmann, Taksar and Heyman 1985; Alfa,
//     Xue and Ye 2002): with lambda = -(2 + e) the matrix is a diagonally
//     dominant M-matrix whose row sums (e inside) all steps only add up, so
//     that nothing cancels where the lowest modes are nearly singular.  Error
//     against the exact solution of a lowest mode's system, 2-norm, diagonals
//     formed directly -> from the sums: 200 rows 5e-14 -> 3e-16, 300 rows
//     1.3e-13 -> 3e-16, 512 rows 2.4e-13 -> 3e-16, whatever the number of lanes;
//   * where a lane keeps 9 .. 34 rows (complex 9 .. 19) in registers, they form
//     two blocks whose sweeps run side by side (two independent FP64
//     recurrences per lane: the sweeps are bound by the latency of their
//     dependent operations), and one more elimination step on the lane reduces
//     the two blocks' rows to one before the shuffles.  Row counts that do not
//     divide by the lanes, or are odd, shorten the second block by one or two
//     rows (before, they kept one block of up to 32 rows on grids of 256^2
//     systems and their rows in shared memory on smaller ones: 192^3 z solve
//     0.064 -> 0.028 ms, 200^3 0.089 -> 0.056, 96^3 0.019 -> 0.011).
#include <type_traits>

#include "pp_common.cuh"
#include "pp_kernels.h"

namespace {

PP_D double zmul(double s, double x) { return s * x; }
PP_D double2 zmul(double s, double2 x) { return make_double2(s * x.x, s * x.y); }
PP_D double zsub(double a, double b) { return a - b; }
PP_D double2 zsub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
PP_D double zadd(double a, double b) { return a + b; }
PP_D double2 zadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
template <typename T>
PP_D T zzero();
template <>
PP_D double zzero<double>() { return 0.0; }
template <>
PP_D double2 zzero<double2>() { return make_double2(0.0, 0.0); }

// warp shuffles within segments of w lanes (one lane group)
PP_D double zshfl(double v, int src, int w) { return __shfl_sync(0xffffffffu, v, src, w); }
PP_D double2 zshfl(double2 v, int src, int w)
{
    return make_double2(__shfl_sync(0xffffffffu, v.x, src, w), __shfl_sync(0xffffffffu, v.y, src, w));
}

// asynchronous global -> shared copies (LDGSTS): no register staging, every
// copy of a tile in flight at once
PP_D void cp_async8(void* smem, const void* gmem)
{
    const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(sa), "l"(gmem) : "memory");
}
PP_D void cp_async16(void* smem, const void* gmem)
{
    const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(gmem) : "memory");
}
PP_D void cp_async4(void* smem, const void* gmem)
{
    const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(sa), "l"(gmem) : "memory");
}
PP_D void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// skewed position of row k inside a system's column of the tile
PP_HD int zpos(int k) { return k + (k >> 4); }
PP_HD int zpitch(int nz) { return (zpos(nz - 1) + 1) | 1; }

// Thread order of the tile's load and store (element e of the TS x nz tile ->
// system s, row k).  Shared memory serves a warp's 8-byte accesses in two
// phases of 16 threads (16-byte ones in four of 8), so a phase of W threads
// takes the W / TS rows k0 + r TS (r < W / TS) of its TS systems: with an odd
// column pitch p the slots s p + k0 + r TS are W distinct banks.  The rows of
// a phase pair then lie in two 128-byte segments of global memory.
PP_D void zt_elem(int e, int TS, int lts, int esz, int* s, int* k)
{
    const int lw = esz == 16 ? 3 : 4;
    const int W = 1 << lw;
    if (TS > W) {
        *k = e >> lts;
        *s = e & (TS - 1);
        return;
    }
    const int blk = e >> (lw + lts);        // W rows of the tile
    const int f = e & ((W << lts) - 1);
    const int ph = f >> lw;                 // phase: rows ph + r TS
    const int jj = f & (W - 1);
    *s = jj & (TS - 1);
    *k = (blk << lw) + ph + ((jj >> lts) << lts);
}
// f(s, k) for every element of the tile (s < ts, k < nz) in that order.  A
// thread keeps its system and steps its row: by blockDim.x / TS when the CTA
// covers whole periods of the order (W TS elements, TS where TS > W); else
// by blockDim.x / W within a period (R = period / blockDim.x steps) and on
// to the next period's W rows.  blockDim.x is a power of two >= 32.
template <typename T, typename F>
PP_D void zt_each(int TS, int lts, int nz, int ts, F f)
{
    const int esz = (int)sizeof(T);
    const int W = esz == 16 ? 8 : 16;
    const int period = TS > W ? TS : W * TS;
    int s, k;
    zt_elem(threadIdx.x, TS, lts, esz, &s, &k);
    if (s >= ts) return;
    if ((int)blockDim.x >= period) {
        const int kst = blockDim.x >> lts;
        for (; k < nz; k += kst) f(s, k);
    } else {
        const int R = period / blockDim.x, dk = blockDim.x / W;
        for (int r = 0; k < nz;) {
            f(s, k);
            if (++r == R) {
                r = 0;
                k += W - (R - 1) * dk;
            } else {
                k += dk;
            }
        }
    }
}

// The reduced system of a lane group, one row per lane L in the lanes' last
// unknowns l:  ra l_{L-1} + rb l_L + rc l_{L+1} = rd,  lane indices wrapping
// (periodic z; otherwise ra = 0 on the first lane and rc = 0 on the last),
// given by its off-diagonals and its sum rs = ra + rb + rc.  Solved by parallel
// cyclic reduction over warp shuffles on the ring of lanes: after log2 P steps
// a row's neighbours on both sides are itself, and its sum is what is left (in
// a chain the off-diagonals have become zero).  Returns l_L.
template <typename T>
PP_D T zsolve_reduced(double ra, double rs, double rc, T rd, int lane, int P)
{
    const double inv0 = 1.0 / (P == 1 ? rs : rs - ra - rc);
    rd = zmul(inv0, rd);
    ra *= inv0;
    rc *= inv0;
    rs *= inv0;
    for (int st = 1; st < P; st <<= 1) {
        const int prv = (lane - st) & (P - 1), nxt = (lane + st) & (P - 1);
        const double ap = zshfl(ra, prv, P), sp = zshfl(rs, prv, P);
        const T dp = zshfl(rd, prv, P);
        const double cn = zshfl(rc, nxt, P), sn = zshfl(rs, nxt, P);
        const T dn = zshfl(rd, nxt, P);
        // (the row's diagonal is 1; minus its off-diagonals times the neighbours' rows)
        rs = rs - ra * sp - rc * sn;
        rd = zsub(zsub(rd, zmul(ra, dp)), zmul(rc, dn));
        ra = -ra * ap;
        rc = -rc * cn;
        const double inv = 1.0 / (2 * st == P ? rs : rs - ra - rc);
        rd = zmul(inv, rd);
        ra *= inv;
        rc *= inv;
        rs *= inv;
    }
    return rd;
}

// The end rows of a block.  Every block has the same interior rows, so its two
// end equations (zsolve_split) come from the pivot table at its last row k:
//   E0: f + e0a l_prev + e0c l = ..   gamma_k, alpha_k, sum psi_k = 1 + gamma_k + alpha_k,
//   E1: e1a f + l + e1c f_next = ..   alpha_k, gamma_k, the same sum.
// A block that ends the system has no neighbour there, and its row is scaled:
// by 1 / (psi_k - alpha_k) at a Neumann end (diagonal lambda + 1), by
// 1 / (1 - gamma_k) at a Dirichlet one (lambda - 1).  Selects, not branches: the
// divisions of a lane's two ends overlap.
struct ZRow {
    double a, c, sum, scale;  // coefficients towards the neighbour and across the block, sum, scale
};
PP_D ZRow zend(bool end, bool neumann, double g, double al, double psi)
{
    ZRow r;
    r.scale = 1.0 / (end ? (neumann ? psi - al : 1.0 - g) : 1.0);
    r.a = end ? 0.0 : g;
    r.c = al * r.scale;
    r.sum = end && !neumann ? 1.0 + r.c : psi * r.scale;
    return r;
}
// E0, scale the factor of its right-hand side d_0 - (row 1's); pin: row 0 of the
// system is x_0 = d_0, or x_0 + x_{nz-1} = d_0 for periodic z
PP_D ZRow zfirst(bool first, bool pin, bool periodic, bool neumann, double g, double al, double psi)
{
    ZRow r = zend(first && !periodic, neumann, g, al, psi);
    r.scale *= g;
    if (first && pin) {
        r.a = periodic ? 1.0 : 0.0;
        r.c = 0.0;
        r.sum = 1.0 + r.a;
        r.scale = 1.0;
    }
    return r;
}

// The partition solve of one system by its lane group with each lane's MT
// rows (registers xr, MT = nz / P) split into two blocks of H = MT / 2 rows,
// A = xr[0, H) and B = xr[H, MT), whose sweeps run side by side (two
// independent recurrences per lane instead of one of twice the length).
// Every block is eliminated as in the one-block solve: forward sweep, spike
// row of the block's first unknown f, its last row E1 -- leaving
//   E0: f + e0a l_prev + e0c l = e0d,   E1: e1a f + l + e1c f_next = e1d
// per block, l the block's last unknown and prev / next the adjacent blocks
// (B of the previous lane, B of this lane for A; A of this lane, A of the
// next lane for B).  Eliminating every f leaves one row per block in the l's;
// eliminating l_A (its neighbours l_B of the previous lane and of this one)
// leaves one row per lane in the l_B's, solved by zsolve_reduced; l_A, both
// f's and the blocks' interior rows follow.  tab holds the interior pivots of
// a block of H rows (gamma_i, alpha_i, i < H), psiA and psiB the sums of the
// blocks' end rows; d0 is row 0's right-hand side (after the periodic
// zero-mode averaging); row 0 of the system is the first row of A on lane 0
// and row nz - 1 the last row of B on lane P - 1.
// UNEV: a lane has M = MT, MT - 1 or MT - 2 rows; block B is the shorter one
// (HB = M - H rows), the branches on it are confined to its last three rows.
template <int MT, bool UNEV, typename T>
PP_D void zsolve_split(T (&xr)[MT], const double2* tab, double psiA, double psiB, T d0, int M, bool live, bool clear,
                       int lane, int P, bool periodic, bool pin, bool nlo, bool nhi)
{
    constexpr int H = MT / 2;
    static_assert(H >= (UNEV ? 5 : 4), "blocks of at least four rows, three in the shorter one");
    const int HB = UNEV ? M - H : H;
    const double* tg = reinterpret_cast<const double*>(tab);  // gamma_i = tg[2i], alpha_i = tg[2i+1]
    // ---- forward sweeps of A and B ----------------------------------------------------
    T dA = zzero<T>(), dB = zzero<T>();
    if (live) {
#pragma unroll
        for (int i = 1; i < H; ++i) {
            const double ga = tg[2 * i];
            dA = (i == 1) ? zmul(ga, xr[i]) : zmul(ga, zsub(xr[i], dA));
            xr[i] = dA;
            if (UNEV && i > H - 3 && i > HB - 1) continue;  // past B's last row
            dB = (i == 1) ? zmul(ga, xr[H + i]) : zmul(ga, zsub(xr[H + i], dB));
            xr[H + i] = dB;
        }
    }
    // ---- backward sweeps: row 1 of a block in terms of its first and last unknowns
    T rA = zzero<T>(), rB = zzero<T>();
    if (live) {
        rA = xr[H - 2];
        rB = xr[MT - 2];
#pragma unroll
        for (int i = H - 3; i >= 1; --i) {
            const double g = tg[2 * i];
            rA = zsub(xr[i], zmul(g, rA));
            // (UNEV: B's sweep starts at its row HB - 2)
            if (UNEV && i > H - 5 && i >= HB - 2) rB = xr[H + i];
            else rB = zsub(xr[H + i], zmul(g, rB));
        }
    }
    // ---- E0 and E1 of both blocks -------------------------------------------------------
    const double2 tA = tab[H - 1], tB = UNEV ? tab[HB - 1] : tA;
    const ZRow fa = zfirst(lane == 0, pin, periodic, nlo, tA.x, tA.y, psiA);
    const ZRow lb = zend(lane == P - 1 && !periodic, nhi, tB.x, tB.y, psiB);
    const T e0dA = zmul(fa.scale, zsub(d0, lane == 0 && pin ? zzero<T>() : rA));
    const T e0dB = zmul(tB.x, zsub(live ? xr[H] : zzero<T>(), rB));
    dB = zmul(lb.scale, dB);
    // ---- rows of the blocks' last unknowns (off-diagonals and sums) ---------------------
    // l_A:  raA l_B(prev lane) + rbA l_A + rcA l_B = rdA
    const double raA = -tA.y * fa.a, rcA = -tA.x * tB.y, rsA = psiA - tA.y * fa.sum - tA.x * psiB;
    const T rdA = zsub(zsub(dA, zmul(tA.y, e0dA)), zmul(tA.x, e0dB));
    // l_B:  raB l_A + rbB l_B + rcB l_A(next lane) = rdB
    const int nxt = (lane + 1) & (P - 1);
    const double nc0 = zshfl(fa.c, nxt, P), ns0 = zshfl(fa.sum, nxt, P);
    const T nd0 = zshfl(e0dA, nxt, P);
    const double raB = -lb.c * tB.x, rcB = -lb.a * nc0, rsB = lb.sum - lb.c * psiB - lb.a * ns0;
    const T rdB = zsub(zsub(dB, zmul(lb.c, e0dB)), zmul(lb.a, nd0));
    // l_A = pd - pa l_B(prev lane) - pc l_B, substituted into the l_B rows
    const double iA = 1.0 / (rsA - raA - rcA);
    const double pa = raA * iA, pc = rcA * iA, ps = rsA * iA;
    const T pd = zmul(iA, rdA);
    const double npc = zshfl(pc, nxt, P), nps = zshfl(ps, nxt, P);
    const T npd = zshfl(pd, nxt, P);
    const T lB = zsolve_reduced(-raB * pa, rsB - raB * ps - rcB * nps, -rcB * npc,
                                zsub(zsub(rdB, zmul(raB, pd)), zmul(rcB, npd)), lane, P);
    const T lBp = zshfl(lB, (lane + P - 1) & (P - 1), P);
    const T lA = zsub(zsub(pd, zmul(pa, lBp)), zmul(pc, lB));
    const T fA = zsub(zsub(e0dA, zmul(fa.a, lBp)), zmul(fa.c, lA));
    const T fB = zsub(zsub(e0dB, zmul(tB.x, lA)), zmul(tB.y, lB));
    // ---- recover both blocks' rows ------------------------------------------------------
    if (!live) return;
    if (clear) {
#pragma unroll
        for (int i = 0; i < MT; ++i) xr[i] = zzero<T>();
        return;
    }
    T xa = lA, xb = lB;
    xr[H - 1] = lA;
    if (UNEV) {
#pragma unroll
        for (int i = H - 3; i < H; ++i)
            if (i == HB - 1) xr[H + i] = lB;
    } else {
        xr[MT - 1] = lB;
    }
#pragma unroll
    for (int i = H - 2; i >= 1; --i) {
        const double2 ti = tab[i];
        xa = zsub(zsub(xr[i], zmul(ti.y, fA)), zmul(ti.x, xa));
        xr[i] = xa;
        if (UNEV && i > H - 4 && i > HB - 2) continue;
        xb = zsub(zsub(xr[H + i], zmul(ti.y, fB)), zmul(ti.x, xb));
        xr[H + i] = xb;
    }
    xr[0] = fA;
    xr[H] = fB;
}

// shared-memory layout of one CTA
struct ZLayout {
    int pitch;       // tile column pitch (elements)
    int mmax;        // table rows per group
    int groups;      // groups (systems in flight) per CTA
    int P;           // lanes per system
    size_t tile_off, tab_off, red_off, stg_off, bytes;
};

// g32: the FP32 spectrum is first copied into a staging area [k][s] of
// TS x nz FP32 elements behind the rest
PP_HD ZLayout zlayout(int TS, int nz, int P, bool cplx, int nthreads, bool g32 = false)
{
    ZLayout L;
    const size_t e = cplx ? 16 : 8;
    L.P = P;
    L.pitch = zpitch(nz);
    L.mmax = (nz + P - 1) / P + 1;
    L.groups = nthreads / P;
    L.tile_off = 0;
    L.tab_off = (size_t)TS * L.pitch * e;
    // (the bulk-copied tile: a chunk of the lane's rows and 16 bytes per lane)
    const size_t chunks = (size_t)P * (((size_t)(nz + P - 1) / P) * TS * e + 16);
    if (chunks > L.tab_off) L.tab_off = chunks;
    L.tab_off = (L.tab_off + 15) & ~(size_t)15;
    // scratch of the pivot-table build: the u_i recurrence of every system
    L.red_off = L.tab_off + (size_t)TS * L.mmax * 16;
    L.bytes = L.red_off + (size_t)TS * L.mmax * 8;
    L.stg_off = (L.bytes + 15) & ~(size_t)15;
    if (g32) L.bytes = L.stg_off + (size_t)TS * nz * (cplx ? 8 : 4);
    return L;
}

template <typename T>
struct ZTo32;
template <>
struct ZTo32<double> {
    using type = float;
    static PP_D double up(float v) { return (double)v; }
    static PP_D float down(double v) { return (float)v; }
};
template <>
struct ZTo32<double2> {
    using type = float2;
    static PP_D double2 up(float2 v) { return make_double2(v.x, v.y); }
    static PP_D float2 down(double2 v) { return make_float2((float)v.x, (float)v.y); }
};
// a stored element (FP64, or FP32 for the refined solve's spectra) to and from
// the FP64 arithmetic type T
template <typename T>
PP_D T zup(T v) { return v; }
template <typename T>
PP_D T zup(typename ZTo32<T>::type v) { return ZTo32<T>::up(v); }
template <typename TG, typename T>
PP_D TG zdown(T v)
{
    if constexpr (std::is_same<TG, T>::value) return v;
    else return ZTo32<T>::down(v);
}

// G32: the spectrum in global memory is FP32 (refined mixed-precision solve);
// all arithmetic stays FP64 (the shared tile too, except in the bulk-copied
// chunks, which hold the stored elements).  MT > 0: every lane keeps its rows
// in registers through the three sweeps, reading and writing its rows of the
// tile once -- exactly MT rows each (CAP = false, nz = P MT), or M = nz / P or
// one more under static i < M guards (CAP = true: at most 8 in one block, MT - 2
// to MT in the split solve); MT = 0: any nz, the sweeps work on the tile in
// shared memory.  SPLIT: two half blocks (zsolve_split).
template <bool CPLX, bool G32, int MT, bool CAP, bool SPLIT>
PP_D void zsolve_body(PPZArgs a)
{
    using T = typename std::conditional<CPLX, double2, double>::type;
    using T32 = typename ZTo32<T>::type;
    extern __shared__ __align__(16) unsigned char zsm_raw[];
    const int nx = a.nx, ny = a.ny, nz = a.nz;
    const int P = a.P;
    const ZLayout Lz = zlayout(a.TS, nz, P, CPLX, blockDim.x, G32);
    T* tile = reinterpret_cast<T*>(zsm_raw + Lz.tile_off);

    const int group = threadIdx.x / P;
    const int lane = threadIdx.x - group * P;

    const int ky = blockIdx.x / a.tiles_x;
    const int kx0 = (blockIdx.x - ky * a.tiles_x) * a.TS;
    const int ts = min(a.TS, nx - kx0);
    T* g = reinterpret_cast<T*>(a.data);
    T32* g32 = reinterpret_cast<T32*>(a.data);
    // row k of system s at k * plane + col0 + s: the usual [k][ky][kx] layout,
    // or the z-tiled one, where this CTA's tile is one contiguous block
    const long plane = a.tiled ? (long)a.TS : (long)nx * ny;
    const long col0 = a.tiled ? (long)blockIdx.x * nz * a.TS : (long)ky * nx + kx0;
    // Bulk-copied tiles: z-tiled, and the split kernels or complex spectra with
    // uneven rows in registers.  Each lane block of the tile (the lane's rows x TS systems, contiguous in global
    // memory) moves as one bulk copy (the copy engine, not the LSU pipe) into a
    // chunk of shared memory,
    // the chunks 16 bytes past the longest block so that the lanes of a phase
    // read distinct banks (or two-way shared ones at one system per half
    // warp); the tile goes back the same way.  FP32 spectra (G32) stay FP32 in
    // the chunks: the lanes convert their rows on the way into and out of
    // registers.  Lane L's block is rows L brows + min(L, brem) on, brows + 1
    // of them for the first brem lanes, brows for the rest.
    using TG = typename std::conditional<G32, T32, T>::type;  // element in global memory
    const int brows = SPLIT && !CAP ? MT : nz / P, brem = SPLIT && !CAP ? 0 : nz - brows * P;
    const int crow = a.TS * (int)sizeof(TG);                  // bytes of one tile row
    const int cpitch = (brows + (brem ? 1 : 0)) * crow + 16;
    const bool bulk = (SPLIT || (CAP && CPLX)) && a.tiled && ts == a.TS && crow % 16 == 0 &&
                      (size_t)P * cpitch <= Lz.tab_off && (reinterpret_cast<uintptr_t>(a.data) & 15) == 0;
    __shared__ __align__(8) unsigned long long zbar;
    const unsigned bar = smem_u32(&zbar);
    unsigned char* gtile = G32 ? reinterpret_cast<unsigned char*>(g32 + col0) : reinterpret_cast<unsigned char*>(g + col0);

    // ---- load the tile asynchronously (thread -> (system, row) without division:
    //      TS is a power of two) and build the pivot tables while it lands ------------
    const int lts = __ffs(a.TS) - 1;
    {
        const int s = threadIdx.x & (a.TS - 1);
        const int kstep = blockDim.x >> lts;
        if (s < ts && !bulk) {
            if (G32) {
                // FP32 elements copied asynchronously into the staging area;
                // converted to the FP64 tile once they have landed
                T32* stg = reinterpret_cast<T32*>(zsm_raw + Lz.stg_off);
                for (int k = threadIdx.x >> lts; k < nz; k += kstep) {
                    if (sizeof(T32) == 8) cp_async8(&stg[k * a.TS + s], &g32[k * plane + col0 + s]);
                    else cp_async4(&stg[k * a.TS + s], &g32[k * plane + col0 + s]);
                }
            }
        }
        if (bulk) {
            if (threadIdx.x == 0) {
                mbar_init(bar);
                mbar_expect(bar, (unsigned)(nz * crow));
                for (int c = 0; c < P; ++c)
                    bulk_g2s(zsm_raw + (size_t)c * cpitch, gtile + (size_t)(c * brows + min(c, brem)) * crow,
                             (unsigned)((brows + (c < brem ? 1 : 0)) * crow), bar);
            }
        } else if (!G32)
            zt_each<T>(a.TS, lts, nz, ts, [&](int s2, int k) {
                if (sizeof(T) == 16) cp_async16(&tile[s2 * Lz.pitch + zpos(k)], &g[k * plane + col0 + s2]);
                else cp_async8(&tile[s2 * Lz.pitch + zpos(k)], &g[k * plane + col0 + s2]);
            });
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    }
    // interior pivots of a block, depending only on lambda = -(2 + e): with
    // u_0 = 1, u_1 = 2 + e, u_i = (2 + e) u_{i-1} - u_{i-2} (Chebyshev U_i(1 + e/2)),
    //   gamma_i = -u_{i-1} / u_i,  alpha_i = -1 / u_i,
    // the same numbers as the Thomas recurrence gamma_i = 1 / (lambda - gamma_{i-1}),
    // and the sums psi_i = 1 + gamma_i + alpha_i = w_i / u_i, w_i = e (u_0 + .. + u_{i-1}),
    // of the end rows.  By the differences v_i = u_i - u_{i-1} = v_{i-1} + e u_{i-1} = 1 + w_i
    // all are sums of positive terms: full relative accuracy for any e >= 0.
    // One thread per system; the divisions are independent.  u_i grows like
    // |lambda|^i, so where mm log2|lambda| could leave the double range the
    // division recurrence is used instead.
    // Phase 1, one thread per system: u_i by the recurrence (FMAs only) into
    // the scratch bytes, or -- where u_i could overflow -- the division
    // recurrence straight into the table, marked by u_0 = 0.
    double* bsc = reinterpret_cast<double*>(zsm_raw + Lz.red_off);
    const int mm = Lz.mmax;
    const int mcount = SPLIT ? MT / 2 : mm - 1;  // rows of the longest block: entries 1 .. mcount - 1
    // block lengths of a launch: one where every lane has MT rows, else two (the
    // split solve's second blocks and its first: three)
    constexpr int NPSI = MT > 0 && !CAP ? 1 : SPLIT ? 3 : 2;
    // psi of the last row of the longest block, of one a row shorter (both in the
    // table's unused entry 0) and of one two rows shorter (past the scratch's u_i)
    auto psi_of = [&](int s, int j) -> double& {
        double* t0 = reinterpret_cast<double*>(zsm_raw + Lz.tab_off) + 2 * (size_t)s * mm;
        return j < 2 ? t0[j] : bsc[(size_t)s * mm + mm - 1];
    };
    for (int s = threadIdx.x; s < ts; s += blockDim.x) {
        const double lam = (-2.0 + a.ax[kx0 + s] * a.Cx) + a.ay[ky] * a.Cy;
        const double e = -(lam + 2.0);
        double* u = bsc + (size_t)s * mm;
        if ((double)mcount * log2(fabs(lam) + 1.0) < 900.0) {
            double uc = 1.0, v = 1.0, w = 0.0;
            u[0] = 1.0;
            for (int i = 1; i < mcount; ++i) {
                w += e * uc;
                v += e * uc;
                uc += v;
                u[i] = uc;
                if (i >= mcount - NPSI) psi_of(s, mcount - 1 - i) = w;  // (divided by u_i in phase 2)
            }
        } else {
            // q_i = 1 + t_i = 2 + e - 1 / q_{i-1}, t_i = e + t_{i-1} / q_{i-1};
            // gamma_i = -1 / q_i, alpha_i = alpha_{i-1} / q_i, psi_i = (e + psi_{i-1}) / q_i
            double2* tb = reinterpret_cast<double2*>(zsm_raw + Lz.tab_off) + (size_t)s * mm;
            double t = 1.0 + e, al = -1.0, psi = 0.0;
            for (int i = 1; i < mcount; ++i) {
                const double p = 1.0 / (1.0 + t);
                al *= p;
                psi = (e + psi) * p;
                tb[i] = make_double2(-p, al);
                if (i >= mcount - NPSI) psi_of(s, mcount - 1 - i) = psi;
                t = e + t * p;
            }
            u[0] = 0.0;
        }
    }
    __syncthreads();
    // Phase 2, every thread: gamma_i = -u_{i-1} / u_i, alpha_i = -1 / u_i, one
    // reciprocal per entry, the entries of all systems spread over the CTA
    {
        // blockDim.x / TS threads per system (both powers of two)
        const int ltp = __ffs(blockDim.x) - 1 - lts;
        const int s = threadIdx.x >> ltp;
        const double* u = bsc + (size_t)s * mm;
        if (s < ts && u[0] != 0.0)
            for (int i = (threadIdx.x & ((1 << ltp) - 1)) + 1; i < mcount; i += 1 << ltp) {
                const double inv = -1.0 / u[i];
                reinterpret_cast<double2*>(zsm_raw + Lz.tab_off)[(size_t)s * mm + i] = make_double2(u[i - 1] * inv, inv);
                if (i >= mcount - NPSI) psi_of(s, mcount - 1 - i) *= -inv;
            }
    }
    cp_async_wait_all();
    if (bulk) {
        // a bounded wait (about a second of polls): a CTA whose copies never
        // land counts itself and leaves without output, with every thread
        const bool landed = mbar_wait0(bar, 1L << 22);
        if (__syncthreads_or(!landed)) {
            if (threadIdx.x == 0 && a.err) atomicAdd(a.err, 1);
            return;
        }
    } else {
        __syncthreads();
    }
    if (G32 && !bulk) {
        const T32* stg = reinterpret_cast<const T32*>(zsm_raw + Lz.stg_off);
        const int s = threadIdx.x & (a.TS - 1);
        const int kstep = blockDim.x >> lts;
        if (s < ts)
            for (int k = threadIdx.x >> lts; k < nz; k += kstep)
                tile[s * Lz.pitch + zpos(k)] = ZTo32<T>::up(stg[k * a.TS + s]);
        __syncthreads();
    }

    const int bsz = nz / P;
    const int rem = nz - bsz * P;
    constexpr bool EXACT = MT > 0 && !CAP;
    const int M = EXACT ? MT : bsz + (lane < rem ? 1 : 0);
    const int s0 = lane * bsz + min(lane, rem);
    const bool periodic = a.zlo == PP_Z_PERIODIC;
    const bool has_d = a.zlo == PP_Z_DIRICHLET || a.zhi == PP_Z_DIRICHLET;
    const unsigned full = 0xffffffffu;

    // all groups of a warp run the same number of iterations (warp-synchronous steps)
    const int ngroups = Lz.groups;
    const int iters = (a.TS + ngroups - 1) / ngroups;
    for (int it = 0; it < iters; ++it) {
        const int s = group + it * ngroups;
        const bool live = s < ts;
        const int kx = kx0 + (live ? s : 0);
        const double lam = (-2.0 + a.ax[kx] * a.Cx) + a.ay[ky] * a.Cy;
        const bool zero = fabs(lam + 2.) < 1.e-10;
        const bool pin = zero && (periodic || a.pin_always || !has_d);
        T* col = tile + (live ? s : 0) * Lz.pitch;
        const double2* tab = reinterpret_cast<const double2*>(zsm_raw + Lz.tab_off) + (size_t)(live ? s : 0) * Lz.mmax;
        // the lane's rows: registers (MT > 0) or the tile column
        // with MT a power of two >= 8 and s0 = lane MT, zpos(s0 + i) = zpos(s0) + zpos(i)
        // (s0 + i never crosses a multiple of 16 that s0 does not); 10, 12, 20
        // and 24 rows index the skewed column directly
        constexpr bool ZP2 = (MT & (MT - 1)) == 0;
        T xr[MT > 0 ? MT : 1];
        T* xcol = col + zpos(s0);
        // (bulk) the lane's rows of system s in its chunk, TS apart
        TG* lrow = reinterpret_cast<TG*>(zsm_raw + (size_t)lane * cpitch) + (live ? s : 0);
        if constexpr (EXACT) {
            if (bulk) {
#pragma unroll
                for (int i = 0; i < MT; ++i) xr[i] = live ? zup<T>(lrow[i * a.TS]) : zzero<T>();
            } else if constexpr (ZP2) {
#pragma unroll
                for (int i = 0; i < MT; ++i) xr[i] = live ? xcol[zpos(i)] : zzero<T>();
            } else {
#pragma unroll
                for (int i = 0; i < MT; ++i) xr[i] = live ? col[zpos(s0 + i)] : zzero<T>();
            }
        } else if constexpr (MT > 0) {
#pragma unroll
            for (int i = 0; i < MT; ++i)
                xr[i] = (live && i < M) ? (bulk ? zup<T>(lrow[i * a.TS]) : col[zpos(s0 + i)]) : zzero<T>();
        }
        auto X = [&](int i) -> T& {
            if constexpr (MT > 0) return xr[i];
            else return col[zpos(s0 + i)];
        };

        // a Neumann first / last row, else a Dirichlet one
        const bool nlo = a.zlo == PP_Z_NEUMANN, nhi = a.zhi == PP_Z_NEUMANN;

        if constexpr (SPLIT) {
            T d0 = zzero<T>();
            if (live) {
                d0 = xr[0];
                if (lane == 0 && periodic && pin) {
                    const T last = bulk ? zup<T>(reinterpret_cast<const TG*>(zsm_raw + (size_t)(P - 1) * cpitch)[(brows - 1) * a.TS + s])
                                        : col[zpos(nz - 1)];
                    d0 = zmul(0.5, zadd(d0, last));
                }
            }
            zsolve_split<MT, CAP>(xr, tab, psi_of(live ? s : 0, 0), psi_of(live ? s : 0, CAP ? MT - M : 0), d0, M, live,
                                  zero && a.skip_zero, lane, P, periodic, pin, nlo, nhi);
        } else {
            // ---- forward sweep of the lane's block -------------------------------------
            // row i (i >= 1) becomes alpha_i x_0 + x_i + gamma_i x_{i+1} = delta_i; delta
            // overwrites the RHS in the tile (only this lane touches these rows)
            T rD0 = zzero<T>(), dprev = zzero<T>();
            const double* tg = reinterpret_cast<const double*>(tab);  // gamma_i = tg[2i], alpha_i = tg[2i+1]
            if (live) {
                rD0 = X(0);
                // the tile still holds every lane's input here (registers are
                // written back at the end)
                if (s0 == 0 && periodic && pin) {
                    // row nz - 1: the last of lane P - 1's brows rows
                    const T last = bulk ? zup<T>(reinterpret_cast<const TG*>(zsm_raw + (size_t)(P - 1) * cpitch)[(brows - 1) * a.TS + s])
                                        : col[zpos(nz - 1)];
                    rD0 = zmul(0.5, zadd(rD0, last));
                }
#pragma unroll
                for (int i = 1; i < (MT > 0 ? MT : M); ++i) {
                    if (CAP && i >= M) break;
                    const T D = X(i);
                    dprev = (i == 1) ? zmul(tg[2 * i], D) : zmul(tg[2 * i], zsub(D, dprev));
                    X(i) = dprev;
                }
            }
            __syncwarp(full);

            // ---- backward sweep: row 1 in terms of x_0 and x_{M-1} ------------------------
            // x_1 = dr - gamma_{M-2} x_0 - alpha_{M-2} x_{M-1} (the spikes are entries of
            // the inverse of the block's interior matrix); only dr is swept.
            T dr = zzero<T>();
            if (live && M >= 3) {
                if constexpr (CAP) {
                    // registers indexed statically: rows above M - 2 are skipped
#pragma unroll
                    for (int i = MT - 2; i >= 1; --i) {
                        if (i > M - 2) continue;
                        dr = (i == M - 2) ? X(i) : zsub(X(i), zmul(tg[2 * i], dr));
                    }
                } else {
                    dr = X(M - 2);
#pragma unroll
                    for (int i = M - 3; i >= 1; --i) dr = zsub(X(i), zmul(tg[2 * i], dr));
                }
            }
            // ---- E0 and E1 ----------------------------------------------------------------
            // E0: f_L + e0a l_{L-1} + e0c l_L = e0d,  E1: e1a f_L + l_L + e1c f_{L+1} = e1d
            // in the lane's first (f) and last (l) unknowns
            const double2 tk = tab[M - 1];
            const double psi = psi_of(live ? s : 0, EXACT ? 0 : mcount - M);
            const ZRow fa = zfirst(lane == 0, pin, periodic, nlo, tk.x, tk.y, psi);
            const ZRow lb = zend(lane == P - 1 && !periodic, nhi, tk.x, tk.y, psi);
            const double e0a = fa.a, e0c = fa.c, e1a = lb.c, e1c = lb.a;
            const T e0d = zmul(fa.scale, zsub(rD0, lane == 0 && pin ? zzero<T>() : dr));
            const T e1d = zmul(lb.scale, dprev);

            // ---- reduced system ---------------------------------------------------------------
            // Eliminating every f_L with E0 leaves a tridiagonal system in l alone, one
            // row per lane (the Schur complement, an M-matrix with the original):
            //   -e1a e0a l_{L-1} + .. l_L - e1c e0c' l_{L+1} = e1d - e1a e0d - e1c e0d'
            // of the sum of E1's - e1a E0's - e1c E0's'   (' : lane L+1)
            // The lane indices wrap (periodic z); without it e0a = 0 on the first lane
            // and e1c = 0 on the last, so the wrapped values carry no weight.  It is
            // solved by parallel cyclic reduction over warp shuffles, and f_L follows
            // from E0.
            const int nxt = (lane + 1) & (P - 1);
            const double nc0 = zshfl(e0c, nxt, P), ns0 = zshfl(fa.sum, nxt, P);
            const T nd0 = zshfl(e0d, nxt, P);
            const double ra = -e1a * e0a, rc = -e1c * nc0, rs = lb.sum - e1a * fa.sum - e1c * ns0;
            const T rd = zsub(zsub(e1d, zmul(e1a, e0d)), zmul(e1c, nd0));
            const T xl = zsolve_reduced(ra, rs, rc, rd, lane, P);
            const T xlp = zshfl(xl, (lane + P - 1) & (P - 1), P);
            const T xf = zsub(zsub(e0d, zmul(e0a, xlp)), zmul(e0c, xl));
            // ---- recover the block's rows ---------------------------------------------------
            if (live && zero && a.skip_zero) {
                // the kx = ky = 0 column is solved separately (in FP64 from plane sums)
#pragma unroll
                for (int i = 0; i < (MT > 0 ? MT : M); ++i) X(i) = zzero<T>();
            } else if (live && CAP) {
                T xn = xl;
#pragma unroll
                for (int i = MT - 1; i >= 1; --i) {
                    if (i > M - 1) continue;
                    if (i == M - 1) {
                        X(i) = xl;
                    } else {
                        const double2 ti = tab[i];
                        xn = zsub(zsub(X(i), zmul(ti.y, xf)), zmul(ti.x, xn));
                        X(i) = xn;
                    }
                }
                X(0) = xf;
            } else if (live) {
                T xn = xl;
                X(M - 1) = xl;
#pragma unroll
                for (int i = M - 2; i >= 1; --i) {
                    const double2 ti = tab[i];
                    xn = zsub(zsub(X(i), zmul(ti.y, xf)), zmul(ti.x, xn));
                    X(i) = xn;
                }
                X(0) = xf;
            }
        }
        if constexpr (EXACT) {
            if (live && bulk) {
#pragma unroll
                for (int i = 0; i < MT; ++i) lrow[i * a.TS] = zdown<TG>(xr[i]);
            } else if (live) {
                if constexpr (ZP2) {
#pragma unroll
                    for (int i = 0; i < MT; ++i) xcol[zpos(i)] = xr[i];
                } else {
#pragma unroll
                    for (int i = 0; i < MT; ++i) col[zpos(s0 + i)] = xr[i];
                }
            }
        } else if constexpr (MT > 0) {
            if (live) {
#pragma unroll
                for (int i = 0; i < MT; ++i) {
                    if (i >= M) continue;
                    if (bulk) lrow[i * a.TS] = zdown<TG>(xr[i]);
                    else col[zpos(s0 + i)] = xr[i];
                }
            }
        }
        __syncwarp(full);
    }
    if (bulk) fence_proxy_async_smem();  // the rows written above, read by the bulk copies
    __syncthreads();

    if (bulk) {
        if (threadIdx.x == 0) {
            for (int c = 0; c < P; ++c)
                bulk_s2g(gtile + (size_t)(c * brows + min(c, brem)) * crow, zsm_raw + (size_t)c * cpitch,
                         (unsigned)((brows + (c < brem ? 1 : 0)) * crow));
            bulk_commit_wait_read();
        }
    } else if (G32) {
        const int s = threadIdx.x & (a.TS - 1);
        const int kstep = blockDim.x >> lts;
        if (s < ts)
            for (int k = threadIdx.x >> lts; k < nz; k += kstep)
                g32[k * plane + col0 + s] = ZTo32<T>::down(tile[s * Lz.pitch + zpos(k)]);
    } else
        zt_each<T>(a.TS, lts, nz, ts, [&](int s2, int k) { g[k * plane + col0 + s2] = tile[s2 * Lz.pitch + zpos(k)]; });
}


template <bool CPLX, bool G32, int MT, bool CAP, bool SPLIT>
__global__ void __launch_bounds__(PP_Z_THREADS) zsolve_kernel(PPZArgs a)
{
    zsolve_body<CPLX, G32, MT, CAP, SPLIT>(a);
}
// The split kernels held to 128 registers (two CTAs of 256 threads, or four
// of 128, per SM): their sweeps are bound by the latency of dependent FP64
// operations, and the extra resident warps outweigh a few spilled values
// (512^3: real 32 rows per lane 0.436 -> 0.380 ms, complex 16 rows 0.446 ->
// 0.381 ms, 40 to 50 bytes spilled each; FP32 complex spectra 0.37 -> 0.33 ms).
// Not for FP32 real spectra of exact row counts, whose conversions make the cap
// cost more than it gains (0.33 -> 0.36 ms); their uneven counts from 25 on take
// it (512 x 512 planes, 27 rows 230 -> 187 us, 29 238 -> 191, 33 246 -> 201; FP64
// 33 rows 133 -> 109).  A separate kernel: naming a minimum of one CTA per SM in
// the other kernels' launch bounds lets the compiler spend more registers on them
// than the one-argument form does.
template <bool CPLX, bool G32, int MT, bool CAP>
__global__ void __launch_bounds__(PP_Z_THREADS, 2) zsolve_split_r128_kernel(PPZArgs a)
{
    zsolve_body<CPLX, G32, MT, CAP, true>(a);
}
// the split kernel a launch takes (only that one is compiled)
template <bool CPLX, bool G32, int MT, bool CAP>
void (*split_kernel())(PPZArgs)
{
    if constexpr (CPLX ? MT <= 16 : (!G32 || (CAP && MT >= 26))) return zsolve_split_r128_kernel<CPLX, G32, MT, CAP>;
    else return zsolve_kernel<CPLX, G32, MT, CAP, true>;
}
}  // namespace

int pp_zsolve_lanes(int nz, bool cplx, long systems)
{
    // (the error does not depend on the lanes: rows are carried by their sums)
    // the fewest lanes that keep every lane's rows in registers: fewer lanes mean
    // fewer steps of the reduced system's PCR per row (384 x 384 x 272, real: 8
    // lanes of 34 rows 0.164 ms, 16 of 17 0.209; 192 x 160 x 144, complex: 8 of 18
    // rows 0.041 ms, 16 of 9 0.052), up to the counts whose registers leave too
    // few warps (384 x 384 x 288: 8 of 36 rows 0.246 ms, 16 of 18 0.211; 192 x
    // 192 x 160, complex: 8 of 20 0.058 ms, 16 of 10 0.048)
    const int rows = cplx ? 19 : 34;
    int P = 1;
    while (P < 32 && (nz + P - 1) / P > rows) P *= 2;
    // few systems: more lanes with shorter sweeps, while the GPU has room for
    // them and a lane keeps at least nine rows (64^3: 4 lanes of 16 rows take 2 us
    // less than 2 of 32; 192 x 192 planes are past this)
    while (P < 32 && systems * P < 32768 && nz / (2 * P) >= 9) P *= 2;
    while (P > 1 && P > nz / 2) P /= 2;
    return P;
}

// launch shape: systems per CTA (one lane group each) and threads per CTA,
// keeping the CTA within ~56 KB of shared memory so about four fit on an SM
void pp_zsolve_config(int nz, bool cplx, int nx, int* TS, int* threads)
{
    const int P = pp_zsolve_lanes(nz, cplx, 1);
    int ts = PP_Z_THREADS / P;
    auto bytes = [&](int t) {
        const int th = t * P < 32 ? 32 : t * P;
        return zlayout(t, nz, P, cplx, th).bytes;
    };
    while (ts > 1 && bytes(ts) > 56 * 1024) ts >>= 1;
    while (ts > 1 && ts > nx) ts >>= 1;
    *TS = ts;
    *threads = ts * P < 32 ? 32 : ts * P;
}

// a lane count the kernel accepts: a power of two <= 32 leaving every lane at
// least two rows
int pp_zsolve_valid_lanes(int nz, int P)
{
    return P >= 1 && P <= 32 && (P & (P - 1)) == 0 && (P == 1 || P <= nz / 2);
}

size_t pp_zsolve_smem_p(int TS, int nz, bool cplx, int P)
{
    const int th = TS * P < 32 ? 32 : TS * P;
    return zlayout(TS, nz, P, cplx, th).bytes;
}

// the launch shape for a chosen lane count (0 or invalid: the default) and
// systems per CTA (0: as many as fit ~56 KB of shared memory)
void pp_zsolve_config_p(int nz, bool cplx, int nx, int lanes, int* TS, int* threads, int systems, int ny)
{
    const int P = pp_zsolve_valid_lanes(nz, lanes) ? lanes : pp_zsolve_lanes(nz, cplx, (long)nx * ny);
    int ts = PP_Z_THREADS / P;
    if (systems >= 1 && (systems & (systems - 1)) == 0 && systems <= ts) {
        ts = systems;
        while (ts > 1 && pp_zsolve_smem_p(ts, nz, cplx, P) > 200 * 1024) ts >>= 1;
    }
    while (ts > 1 && systems == 0 && pp_zsolve_smem_p(ts, nz, cplx, P) > 56 * 1024) ts >>= 1;
    while (ts > 1 && ts > nx) ts >>= 1;
    // small grids: CTAs for every SM, in row segments of at least eight columns
    while (ts > 8 && systems == 0 && ts * P > 32 && (long)ny * ((nx + ts - 1) / ts) < 296) ts >>= 1;
    *TS = ts;
    *threads = ts * P < 32 ? 32 : ts * P;
}

int pp_zsolve_max_nz(bool cplx, bool g32)
{
    int lo = 3, hi = 1 << 16;  // lo fits, hi does not
    while (hi - lo > 1) {
        const int mid = (lo + hi) / 2;
        if (zlayout(1, mid, 32, cplx, 32, g32).bytes <= (size_t)227 * 1024) lo = mid;
        else hi = mid;
    }
    return lo;
}

cudaError_t pp_launch_zsolve(const PPZArgs& a0, bool cplx, cudaStream_t st)
{
    if (a0.nz < 3 || a0.nz > pp_zsolve_max_nz(cplx, a0.data_fp32 != 0)) return cudaErrorInvalidValue;
    PPZArgs a = a0;
    if (!pp_zsolve_valid_lanes(a.nz, a.P)) a.P = pp_zsolve_lanes(a.nz, cplx, (long)a.nx * a.ny);
    const int threads = a.TS * a.P < 32 ? 32 : a.TS * a.P;
    if (threads > PP_Z_THREADS) return cudaErrorInvalidValue;
    const size_t smem = zlayout(a.TS, a.nz, a.P, cplx, threads, a.data_fp32 != 0).bytes;
    if (smem > 227 * 1024) return cudaErrorInvalidValue;
    dim3 grid(a.ny * a.tiles_x), block(threads);
    cudaError_t e;
    // rows per lane fixed at compile time where every lane has the same count;
    // else the smallest register capacity that holds every lane's rows
    const int rows = a.nz / a.P, rmax = (a.nz + a.P - 1) / a.P;
    const int mt = (a.nz % a.P == 0 && (rows == 8 || rows == 16 || ((rows == 10 || rows == 12) && cplx) ||
                                        ((rows == 20 || rows == 24 || rows == 32) && !cplx))) ? rows : 0;
    // (uneven counts: the next even capacity of the split path, or up to 8 rows)
    const int most = cplx ? 19 : 34;
    const int cap = mt || rmax > most ? 0 : rmax <= 8 ? 8 : (rmax + 1) / 2 * 2;
#define PP_ZL(C, G, M, K) PP_ZLF((zsolve_kernel<C, G, M, K, false>))
#define PP_ZLK(C, G, M, K)                                                                                      \
    do {                                                                                                        \
        PP_ZLF((split_kernel<C, G, M, K>()));                                                                  \
    } while (0)
#define PP_ZLF(KFN)                                                                                             \
    do {                                                                                                        \
        auto kfn = KFN;                                                                                         \
        if ((e = cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)) != cudaSuccess) \
            return e;                                                                                           \
        kfn<<<grid, block, smem, st>>>(a);                                                                      \
    } while (0)
// (the row counts a complex or real launch never takes are replaced by ones
// it does, so that no dead instance is compiled)
#define PP_ZLM(C, G)                                  \
    do {                                              \
        if (mt == 8) PP_ZL(C, G, 8, false);           \
        else if (mt == 16) PP_ZLK(C, G, 16, false);   \
        else if (mt == 32 && !C) PP_ZLK(C, G, (C ? 16 : 32), false); \
        else if (mt == 24 && !C) PP_ZLK(C, G, (C ? 16 : 24), false); \
        else if (mt == 12 && C) PP_ZLK(C, G, (C ? 12 : 16), false); \
        else if (mt == 20 && !C) PP_ZLK(C, G, (C ? 16 : 20), false); \
        else if (mt == 10 && C) PP_ZLK(C, G, (C ? 10 : 16), false); \
        else if (cap == 8) PP_ZL(C, G, 8, true);      \
        else if (cap == 10) PP_ZLK(C, G, 10, true);   \
        else if (cap == 12) PP_ZLK(C, G, 12, true);   \
        else if (cap == 14) PP_ZLK(C, G, 14, true);   \
        else if (cap == 16) PP_ZLK(C, G, 16, true);   \
        else if (cap == 18) PP_ZLK(C, G, 18, true);   \
        else if (cap == 20) PP_ZLK(C, G, 20, true);   \
        else if (cap == 22) PP_ZLK(C, G, (C ? 16 : 22), true); \
        else if (cap == 24) PP_ZLK(C, G, (C ? 16 : 24), true); \
        else if (cap == 26) PP_ZLK(C, G, (C ? 16 : 26), true); \
        else if (cap == 28) PP_ZLK(C, G, (C ? 16 : 28), true); \
        else if (cap == 30) PP_ZLK(C, G, (C ? 16 : 30), true); \
        else if (cap == 32) PP_ZLK(C, G, (C ? 16 : 32), true); \
        else if (cap == 34) PP_ZLK(C, G, (C ? 16 : 34), true); \
        else PP_ZL(C, G, 0, false);                   \
    } while (0)
    if (cplx && a.data_fp32) PP_ZLM(true, true);
    else if (cplx) PP_ZLM(true, false);
    else if (a.data_fp32) PP_ZLM(false, true);
    else PP_ZLM(false, false);
#undef PP_ZLM
#undef PP_ZL
#undef PP_ZLK
#undef PP_ZLF
    return cudaGetLastError();
}
