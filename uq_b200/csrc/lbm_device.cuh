// Device-side building blocks of the D2Q13 thermal LBM step (sm_100a).
//
// Every function restates a piece of the reference FP64 CPU solver
// CODE/C++/VS2010/simLB/simLB/cpuLBM.cpp (cited per function) for the GPU's
// layout: per sample, 13 planes, one per direction, each ny rows of `pitch`
// nodes, x fastest; a node of plane i is the pair (f_i, h_i), so that f and h,
// which every stage treats alike, move in one 8- (FP32) or 16-byte (FP64)
// access and are the two lanes of the packed FP32 arithmetic.  Templates take
// the storage type S (double or float) and the compute type C; moment sums
// are always accumulated in double.
#pragma once

#include <cstdint>

namespace uqlbm {

constexpr int NQ = 13;
constexpr int NPL = 26;  // f and h values of a node

// element of direction i (f: fh = 0, h: fh = 1) at node offset o (in the
// plane), relative to the sample's plane 0
__host__ __device__ constexpr long long el(int i, int fh, long long plane, long long o)
{
    return 2 * (i * plane + o) + fh;
}

// node-flag byte: cell type in bits 0-1 (0 fluid, 1 permanent, 2 solid);
// bits 2-5 say whether the 5-point x / y stencil of the node meets a solid
// node or the domain edge (then the exact boundary-aware stencil runs).
constexpr uint8_t NF_TYPE = 3;
constexpr uint8_t NF_SOLX = 4;
constexpr uint8_t NF_SOLY = 8;
constexpr uint8_t NF_EDGX = 16;   // near a clamped/mirrored x edge
constexpr uint8_t NF_EDGY = 32;
constexpr uint8_t NF_WRPX = 64;   // x stencil wraps across a periodic edge
constexpr uint8_t NF_WRPY = 128;

// sample flag bits
constexpr int SF_PERX = 1, SF_PERY = 2, SF_MIRN = 4, SF_MIRS = 8, SF_MIRE = 16, SF_MIRW = 32;

struct SampleParams {
    int nx, ny, pitch, flags;
    int rk, fm;          // RKMETHOD, FMETHOD
    int ntile;           // tiles of this sample in the full tile list
    int first_tile;
    long long state_off; // element offset of plane 0 in every state buffer (even)
    long long plane;     // nodes per plane
    long long node_off;  // offset into per-node arrays
    long long lat_off;   // nodes (nx ny each) of the samples before, in a batch
    int xoff, yoff;      // offsets into the per-column / per-row spacing tables
    double R, bR, K, Tc, inv_sRTc, RTc, mu, Pr, dt, c;
    // Reference rest state of the stored deviations (mixed path): the state
    // holds f - f_ref, h - h_ref with f_ref, h_ref the equilibria at
    // (rho0, 0, 0, T0); rho0 = shref = 0 (full storage) on the FP64 path.
    double rho0, T0n, shref;  // T0n = T0 / Tc
    double inv_mu, inv_Tc, two_over_bR;
    int wide;  // FP32 WENO5 weights in the range-safe form (see weno_face)
    double eps1;  // FP64: WENO5's epsilon for values not scaled by |e|, 1e-6 / c^2
    // ghost columns of the stage buffers (0 or GHOST_X): x-periodic samples
    // keep, left and right of every row of buffers 2 and 3, the periodic
    // images of the gx columns at the other edge, so the staged halo boxes
    // of tiles at those edges load them as they load any interior node.
    // Rows stay aligned (pitch >= nx + 2 gx, a multiple of 32): the right
    // ghosts follow the row, the left ones are the last gx nodes of the
    // row before (the sample's region starts GHOST_SLACK elements before
    // plane 0 for the first row's).  The per-node arrays have no ghosts.
    int gx;
    // viscosity law (codeCL.py:986-990): 0 constant mu, 1 VHS, 2 Sutherland;
    // mu(T) = mu (T/visc_T)^visc_exp [(visc_T + visc_S)/(T + visc_S)]
    int visc;
    double visc_exp, visc_S, visc_T;
};

constexpr int GHOST_X = 4;       // = the staged box's x halo
constexpr int GHOST_SLACK = 32;  // state elements before plane 0 of a sample with ghosts (keeps it aligned)

// What a block needs before it can ask for its boxes and sweep them (the
// sample's parameters arrive meanwhile).
struct Tile {
    int sample;
    int x0, y0;
    int gid;      // index of the tile in the batch's full tile list
    int kind;     // TILE_* bits
    float c;      // (float)SampleParams::c
    double eps1;  // SampleParams::eps1
};

// Kinds of tiles in the stencil phases.  A sweep tile's fluxes all come from
// its staged box, line by line (see k_flux): every node of the tile and its
// 3-node halo is plain fluid, or the exceptions are of the forms that are
// filled into the box first (TILE_FIX): a clamped or periodic domain edge,
// permanent nodes, a straight wall (row 0 or row ny - 1 solid in all the
// columns the tile sees; TILE_WALLS, TILE_WALLN).  The other tiles (solids
// elsewhere, mirror edges) are general: node flags choose per flux.
constexpr int TILE_SWEEP = 1, TILE_FIX = 2, TILE_WALLS = 4, TILE_WALLN = 8;
constexpr int TILE_FM_SHIFT = 4;  // 2 bits: 0 NND, 1 WENO5, 2 WENO5 with the range-safe weights
constexpr int TILE_GHOST = 64;    // the sample has ghost columns
constexpr int TILE_WRAP = 128;    // a TILE_FIX tile that only wraps (no clamped edge, fixed node or wall)
__host__ __device__ inline bool tile_sweep(const Tile &t) { return (t.kind & TILE_SWEEP) != 0; }
// order of the tiles in a stencil run: tiles to complete (the longer ones)
// first, then those that only wrap, then plain ones; general tiles last
__host__ __device__ inline int tile_rank(const Tile &t)
{
    return !(t.kind & TILE_SWEEP) ? 3 : (t.kind & TILE_WRAP) ? 1 : (t.kind & TILE_FIX) ? 0 : 2;
}
__host__ __device__ inline int tile_fm(int kind) { return (kind >> TILE_FM_SHIFT) & 3; }

// lattice (setupVars, cpuLBM.cpp:376-388) in units of c, its signs, and the
// reflection maps of mirIndex (cpuLBM.cpp:1147-1169)
__constant__ int c_EX[NQ] = {0, 1, 0, -1, 0, 1, -1, -1, 1, 2, 0, -2, 0};
__constant__ int c_EY[NQ] = {0, 0, 1, 0, -1, 1, 1, -1, -1, 0, 2, 0, -2};
__constant__ int c_MIR_NS[NQ] = {0, 1, 4, 3, 2, 8, 7, 6, 5, 9, 12, 11, 10};
__constant__ int c_MIR_EW[NQ] = {0, 3, 2, 1, 4, 6, 5, 8, 7, 11, 10, 9, 12};

// the same lattice as compile-time constants (for unrolled direction loops)
constexpr int kEX[NQ] = {0, 1, 0, -1, 0, 1, -1, -1, 1, 2, 0, -2, 0};
constexpr int kEY[NQ] = {0, 0, 1, 0, -1, 1, 1, -1, -1, 0, 2, 0, -2};

// the same as functions: compile-time values in unrolled loops, no table
__host__ __device__ constexpr int lat_ex(int i)
{
    return (i == 1 || i == 5 || i == 8) ? 1 : (i == 3 || i == 6 || i == 7) ? -1 : i == 9 ? 2 : i == 11 ? -2 : 0;
}
__host__ __device__ constexpr int lat_ey(int i)
{
    return (i == 2 || i == 5 || i == 6) ? 1 : (i == 4 || i == 7 || i == 8) ? -1 : i == 10 ? 2 : i == 12 ? -2 : 0;
}
constexpr bool lat_fn_match()
{
    for (int i = 0; i < NQ; ++i)
        if (lat_ex(i) != kEX[i] || lat_ey(i) != kEY[i]) return false;
    return true;
}
static_assert(lat_fn_match(), "lattice functions differ from the table");

__device__ __forceinline__ int isgn(int a) { return (a > 0) - (a < 0); }

// Round-to-nearest operations the compiler may neither fuse nor split:
// NND, WENO5, the flux divergence, the wall fluxes and, on the FP32 path,
// the equilibria and the RK3 stage updates are written with them so that
// every compiled instance (the
// simple-tile paths per scheme, the boundary-aware
// paths, the wall factors, the tile-shape instances) rounds a node the same
// way, and results do not depend on which path a node took (tile shape,
// batch packing).
__device__ __forceinline__ float xmul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double xmul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float xadd(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double xadd(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float xsub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ double xsub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ float xfma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double xfma(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ float xneg(float a) { return -a; }
__device__ __forceinline__ double xneg(double a) { return -a; }
__device__ __forceinline__ float xmin(float a, float b) { return fminf(a, b); }
__device__ __forceinline__ double xmin(double a, double b) { return fmin(a, b); }
// The same operations on a packed pair of FP32 values (the f and h planes
// of one face), one sm_100 f32x2 instruction each: every lane is rounded
// exactly as the scalar operation rounds it, so a face reconstructed in
// pairs equals the scalar reconstruction bit for bit.  a - b is formed as
// fma(b, -1, a), which is a - b correctly rounded.
__device__ __forceinline__ float2 xmul(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 xadd(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 xsub(float2 a, float2 b) { return __ffma2_rn(b, make_float2(-1.f, -1.f), a); }
__device__ __forceinline__ float2 xfma(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 xneg(float2 a) { return make_float2(-a.x, -a.y); }
__device__ __forceinline__ float2 xmin(float2 a, float2 b) { return make_float2(fminf(a.x, b.x), fminf(a.y, b.y)); }

// and on a pair of FP64 values, lane by lane
__device__ __forceinline__ double2 xmul(double2 a, double2 b) { return make_double2(xmul(a.x, b.x), xmul(a.y, b.y)); }
__device__ __forceinline__ double2 xadd(double2 a, double2 b) { return make_double2(xadd(a.x, b.x), xadd(a.y, b.y)); }
__device__ __forceinline__ double2 xsub(double2 a, double2 b) { return make_double2(xsub(a.x, b.x), xsub(a.y, b.y)); }
__device__ __forceinline__ double2 xfma(double2 a, double2 b, double2 c)
{
    return make_double2(xfma(a.x, b.x, c.x), xfma(a.y, b.y, c.y));
}

// the (f, h) pair of a storage or compute type
template <class C>
struct PairOf;
template <>
struct PairOf<float> { using type = float2; };
template <>
struct PairOf<double> { using type = double2; };
template <class C>
using Pair = typename PairOf<C>::type;
__device__ __forceinline__ float2 make_pair2(float a, float b) { return make_float2(a, b); }
__device__ __forceinline__ double2 make_pair2(double a, double b) { return make_double2(a, b); }

// a constant in the arithmetic type (both lanes of a pair)
template <class C>
__device__ __forceinline__ C kc(double v) { return C(v); }
template <>
__device__ __forceinline__ float2 kc<float2>(double v) { return make_float2((float)v, (float)v); }
template <>
__device__ __forceinline__ double2 kc<double2>(double v) { return make_double2(v, v); }

// FP64 reciprocal of a normal number whose reciprocal is normal (zero and
// infinity give NaN): PTX's approximate reciprocal, whose operand and result
// have 20 fraction bits, and one cubic Newton (Chebyshev) step, y (1 + e + e^2)
// with e = 1 - d y; |e| < 2^-18 leaves e^3 < 2^-54, so the result is the
// correctly rounded one or its neighbour.  It takes a third of the operations
// of a division and no branch for special operands (a division per face was a
// fifth of the FP64 sweeps).
__device__ __forceinline__ double rcp64(double d)
{
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
    const double e = __fma_rn(-d, y, 1.0);
    return __fma_rn(y, __fma_rn(e, e, e), y);
}

// ------------------------------------------------------------ equilibria
// equilibrium2D (cpuLBM.cpp:785-844) with the polynomials of
// inlineFunctions.cpp:10-61, evaluated per symmetry family.  Normalised
// u, v, T are u/sqrt(R Tc), v/sqrt(R Tc), T/Tc; with a = u^2, c = v^2:
//   f0      = 1 + 5/2 T^2 + 5/2 T (a + c - 1) + (a^2 + c^2)/4 + a c - 5/4 (a + c)
//   f1, f3  = E1(u, v) +- O1(u, v);   f2, f4 = E1(v, u) +- O1(v, u)
//   f5..f8  = (T + a +- u)(T + c +- v) / 4
//   f9, f11 = E9(u) +- O9(u);         f10, f12 = E9(v) +- O9(v)
// times rho, and the h families times rho R Tc.
template <class C>
struct EqState {
    C rho, u, v, T, K, rRTc;  // normalised velocity/temperature
};

template <class C>
__device__ __forceinline__ EqState<C> eq_state(double rho, double ux, double uy, double Tn, const SampleParams &sp)
{
    EqState<C> e;
    e.rho = (C)rho;
    e.u = (C)(ux * sp.inv_sRTc);
    e.v = (C)(uy * sp.inv_sRTc);
    e.T = (C)Tn;
    e.K = (C)sp.K;
    e.rRTc = (C)(rho * sp.RTc);
    return e;
}

// family 0: direction 0
template <class C>
__device__ __forceinline__ void eq_fam0(const EqState<C> &q, C &f0, C &h0)
{
    const C a = q.u * q.u, c = q.v * q.v, s2 = a + c, pc = a * c, T = q.T, T2 = T * T, T3 = T2 * T, K = q.K;
    f0 = q.rho * (C(1) + C(2.5) * T2 + C(2.5) * T * (s2 - C(1)) + C(0.25) * (a * a + c * c) + pc - C(1.25) * s2);
    h0 = q.rRTc * (T3 * (C(1.25) * K + C(20.0 / 3.0)) + T2 * ((C(1.25) * K + C(11.25)) * s2 - C(1.25) * K - C(5))
                   + T * (C(0.125) * K * (s2 * s2 + C(2) * pc) - C(0.625) * K * s2 + C(0.5) * K + C(2.5) * s2 * s2
                          + C(2.5) * pc - C(5) * s2 + C(1))
                   + s2 * s2 * s2 * C(0.125) + C(0.25) * pc * s2 - C(0.625) * s2 * s2 + C(0.5) * s2);
}

// family 1: directions 1..4 (out[0..3] = f1..f4, h1..h4)
template <class C>
__device__ __forceinline__ void eq_fam1(const EqState<C> &q, C *f, C *h)
{
    const C T = q.T, T2 = T * T, T3 = T2 * T, K = q.K;
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const C U = k == 0 ? q.u : q.v;
        const C W = k == 0 ? q.v : q.u;
        const C A = U * U, Cc = W * W;
        C E = -T2 + T * (C(2.0 / 3.0) - C(1.5) * A - C(0.5) * Cc) + C(2.0 / 3.0) * A - A * A * C(1.0 / 6.0) - C(0.5) * A * Cc;
        C O = U * (C(2.0 / 3.0) - T - A * C(1.0 / 6.0) - C(0.5) * Cc);
        f[k] = q.rho * (E + O);
        f[k + 2] = q.rho * (E - O);
        E = T3 * (C(-0.5) * K - C(8.0 / 3.0))
            + T2 * (-(C(0.75) * K + C(6.5)) * A - (C(0.25) * K + C(2.5)) * Cc + K * C(1.0 / 3.0) + C(4.0 / 3.0))
            + T * (-(K * C(1.0 / 12.0) + C(19.0 / 12.0)) * A * A - (C(0.25) * K + C(3.5)) * A * Cc
                   + (K * C(1.0 / 3.0) + C(7.0 / 3.0)) * A - C(0.25) * Cc * Cc + Cc * C(1.0 / 3.0))
            - A * A * A * C(1.0 / 12.0) - A * A * Cc * C(1.0 / 3.0) + A * A * C(1.0 / 3.0) - C(0.25) * A * Cc * Cc
            + A * Cc * C(1.0 / 3.0);
        O = U * (T2 * (C(-0.5) * K - C(3))
                 + T * (-(K * C(1.0 / 12.0) + C(7.0 / 6.0)) * A - (C(0.25) * K + C(2.5)) * Cc + K * C(1.0 / 3.0) + C(4.0 / 3.0))
                 - A * A * C(1.0 / 12.0) - A * Cc * C(1.0 / 3.0) + A * C(1.0 / 3.0) - C(0.25) * Cc * Cc + Cc * C(1.0 / 3.0));
        h[k] = q.rRTc * (E + O);
        h[k + 2] = q.rRTc * (E - O);
    }
}

// family 5: directions 5..8
template <class C>
__device__ __forceinline__ void eq_fam5(const EqState<C> &q, C *f, C *h)
{
    const C u = q.u, v = q.v, a = u * u, c = v * v, s2 = a + c, pc = a * c, T = q.T, T2 = T * T, T3 = T2 * T, K = q.K;
    const C Ap = T + a + u, Am = T + a - u, Bp = T + c + v, Bm = T + c - v, r4 = C(0.25) * q.rho;
    f[0] = r4 * (Ap * Bp);
    f[1] = r4 * (Am * Bp);
    f[2] = r4 * (Am * Bm);
    f[3] = r4 * (Ap * Bm);
    const C k8 = C(0.125) * K;
    const C EE = T3 * (k8 + C(2.0 / 3.0)) + T2 * (k8 + C(1.125)) * s2 + T * ((k8 + C(1.5)) * pc + C(0.125) * (a * a + c * c))
                 + C(0.125) * pc * s2;
    const C OE = u * (T2 * (k8 + C(0.75)) + T * ((k8 + C(1.125)) * c + C(0.125) * a) + C(0.125) * c * s2);
    const C EO = v * (T2 * (k8 + C(0.75)) + T * ((k8 + C(1.125)) * a + C(0.125) * c) + C(0.125) * a * s2);
    const C OO = u * v * (T * (k8 + C(0.75)) + C(0.125) * s2);
    h[0] = q.rRTc * (EE + OE + EO + OO);
    h[1] = q.rRTc * (EE - OE + EO - OO);
    h[2] = q.rRTc * (EE - OE - EO + OO);
    h[3] = q.rRTc * (EE + OE - EO - OO);
}

// family 9: directions 9..12
template <class C>
__device__ __forceinline__ void eq_fam9(const EqState<C> &q, C *f, C *h)
{
    const C T = q.T, T2 = T * T, T3 = T2 * T, K = q.K;
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const C U = k == 0 ? q.u : q.v;
        const C W = k == 0 ? q.v : q.u;
        const C A = U * U, Cc = W * W;
        C E = C(0.125) * T2 + T * (C(0.25) * A - C(1.0 / 24.0)) + (A * A - A) * C(1.0 / 24.0);
        C O = U * (C(0.25) * T + (A - C(1)) * C(1.0 / 12.0));
        f[k] = q.rho * (E + O);
        f[k + 2] = q.rho * (E - O);
        E = T3 * (K * C(1.0 / 16.0) + C(1.0 / 3.0))
            + T2 * ((C(0.125) * K + C(17.0 / 16.0)) * A + Cc * C(1.0 / 16.0) - K * C(1.0 / 48.0) - C(1.0 / 12.0))
            + T * ((K * C(1.0 / 48.0) + C(1.0 / 3.0)) * A * A - (K * C(1.0 / 48.0) + C(7.0 / 48.0)) * A + C(0.125) * A * Cc
                   - Cc * C(1.0 / 48.0))
            + (A * A * A + A * A * Cc - A * A - A * Cc) * C(1.0 / 48.0);
        O = U * (T2 * (C(0.125) * K + C(0.75)) + T * ((K * C(1.0 / 24.0) + C(11.0 / 24.0)) * A - K * C(1.0 / 24.0) - C(1.0 / 6.0) + C(0.125) * Cc)
                 + (A * A + A * Cc - A - Cc) * C(1.0 / 24.0));
        h[k] = q.rRTc * (E + O);
        h[k + 2] = q.rRTc * (E - O);
    }
}

// ------------------------------------------------ equilibria as deviations
// The same polynomials as deviations from the rest state (rho0, 0, 0, T0)
// of the sample, for the FP32 path: f_eq - f_ref = rho dP + (rho - rho0) P0
// where dP = P(u, v, T) - P(0, 0, T0) keeps only terms that vanish at rest:
// the T-only part g(T) - g(T0) is factored as (T - T0) G(T, T0), so no
// O(1) terms cancel in FP32.  Likewise for h with the factor R Tc.
template <class C>
struct EqDev {
    C rho, drho, u, v, T, tau, T0, K, RTc;
};

template <class C>
__device__ __forceinline__ EqDev<C> eq_dev(double rho, double ux, double uy, double T, const SampleParams &sp)
{
    EqDev<C> e;
    e.rho = (C)rho;
    e.drho = (C)(rho - sp.rho0);
    e.u = (C)(ux * sp.inv_sRTc);
    e.v = (C)(uy * sp.inv_sRTc);
    const double Tn = T / sp.Tc;
    e.T = (C)Tn;
    e.tau = (C)(Tn - sp.T0n);
    e.T0 = (C)sp.T0n;
    e.K = (C)sp.K;
    e.RTc = (C)sp.RTc;
    return e;
}

// ------------------------- FP32 deviations: explicitly rounded, lanes paired
// Every operation is explicitly rounded (no compiler contraction), so every
// kernel that computes a node's equilibria gives it the same bits.  The terms
// are those of eq_fam0 .. eq_fam9 less their values at rest, regrouped (common
// factors, Horner form).  In
// families 1 and 9 the two axis pairs (k = 0: U = u, W = v; k = 1: U = v,
// W = u) are the two lanes of packed f32x2 operations; in family 5 the
// lanes are the sign of u in f (for v + and -) and (OE, EO) in h.
__device__ __forceinline__ float2 bc2(float s) { return make_float2(s, s); }

__device__ __forceinline__ void eqd_fam0(const EqDev<float> &q, float &f0, float &h0)
{
    const float u = q.u, v = q.v, T = q.T, K = q.K, T0 = q.T0, tau = q.tau;
    const float a = xmul(u, u), c = xmul(v, v), s2 = xadd(a, c), pc = xmul(a, c), T2 = xmul(T, T);
    const float S2 = xadd(T, T0), S3 = xfma(T, S2, xmul(T0, T0));
    // dP = s2 (5/2 T - 5/4 + s2/4) + pc/2 + 5/2 tau (S2 - 1), P0 = 1 + 5/2 T0 (T0 - 1)
    const float dP = xfma(s2, xfma(0.25f, s2, xfma(2.5f, T, -1.25f)),
                          xfma(0.5f, pc, xmul(xmul(2.5f, tau), xadd(S2, -1.0f))));
    const float P0 = xfma(xmul(2.5f, T0), xadd(T0, -1.0f), 1.0f);
    f0 = xfma(q.rho, dP, xmul(q.drho, P0));
    // dQ = T2 (5/4 K + 45/4) s2 + T (s2 ((K/8 + 5/2) s2 - 5/8 K - 5) + (K/4 + 5/2) pc)
    //      + s2 (s2 (s2/8 - 5/8) + pc/4 + 1/2) + tau (k3 S3 + k2 S2 + k1),
    // Q0 = T0 (T0 (T0 k3 + k2) + k1)
    const float k3 = xfma(1.25f, K, 20.0f / 3.0f), k2 = xfma(-1.25f, K, -5.0f), k1 = xfma(0.5f, K, 1.0f);
    const float tT = xfma(s2, xfma(xfma(0.125f, K, 2.5f), s2, xfma(-0.625f, K, -5.0f)), xmul(xfma(0.25f, K, 2.5f), pc));
    const float rest = xmul(s2, xfma(s2, xfma(0.125f, s2, -0.625f), xfma(0.25f, pc, 0.5f)));
    const float tG = xmul(tau, xfma(k3, S3, xfma(k2, S2, k1)));
    const float dQ = xfma(T2, xmul(xfma(1.25f, K, 11.25f), s2), xfma(T, tT, xadd(rest, tG)));
    const float Q0 = xmul(T0, xfma(T0, xfma(T0, k3, k2), k1));
    h0 = xmul(q.RTc, xfma(q.rho, dQ, xmul(q.drho, Q0)));
}

__device__ __forceinline__ void eqd_fam1(const EqDev<float> &q, float *f, float *h)
{
    const float T = q.T, K = q.K, T0 = q.T0, tau = q.tau, T2 = xmul(T, T);
    const float S2 = xadd(T, T0), S3 = xfma(T, S2, xmul(T0, T0));
    const float kh3 = xfma(-0.5f, K, -8.0f / 3.0f), kh2 = xfma(K, 1.0f / 3.0f, 4.0f / 3.0f);
    const float P0 = xmul(T0, xsub(2.0f / 3.0f, T0));
    const float Q0 = xmul(xmul(T0, T0), xfma(T0, kh3, kh2));
    const float tGf = xmul(tau, xsub(2.0f / 3.0f, S2));
    const float tGh = xmul(tau, xfma(kh3, S3, xmul(kh2, S2)));
    const float2 U = make_float2(q.u, q.v), W = make_float2(q.v, q.u);
    const float2 A = xmul(U, U), Cc = xmul(W, W), vT = bc2(T), vT2 = bc2(T2), vr = bc2(q.rho);
    // f: E = T (-3/2 A - Cc/2) + A (m - A/6) + tau Gf, O = U (m - T - A/6), m = 2/3 - Cc/2
    const float2 m = xfma(kc<float2>(-0.5), Cc, kc<float2>(2.0 / 3.0));
    const float2 Ef = xfma(vT, xfma(kc<float2>(-1.5), A, xmul(kc<float2>(-0.5), Cc)),
                           xfma(A, xfma(kc<float2>(-1.0 / 6.0), A, m), bc2(tGf)));
    const float2 Of = xmul(U, xfma(kc<float2>(-1.0 / 6.0), A, xsub(m, vT)));
    const float2 dP0 = bc2(xmul(q.drho, P0));
    const float2 fp = xfma(vr, xadd(Ef, Of), dP0), fm = xfma(vr, xsub(Ef, Of), dP0);
    f[0] = fp.x; f[1] = fp.y; f[2] = fm.x; f[3] = fm.y;
    // h: with CB = Cc (1/3 - Cc/4) and R = A (1/3 - A/12 - Cc/3) + CB,
    // E = T2 (c1 A + c2 Cc) + T (A (c3 A + c4 Cc + c5) + CB) + A R + tau Gh,
    // O = U (T2 c8 + T (c6 A + c2 Cc + kh2) + R)
    const float c1 = xfma(-0.75f, K, -6.5f), c2 = xfma(-0.25f, K, -2.5f), c3 = xfma(K, -1.0f / 12.0f, -19.0f / 12.0f);
    const float c4 = xfma(-0.25f, K, -3.5f), c5 = xfma(K, 1.0f / 3.0f, 7.0f / 3.0f), c6 = xfma(K, -1.0f / 12.0f, -7.0f / 6.0f);
    const float c8 = xfma(-0.5f, K, -3.0f);
    const float2 CB = xmul(Cc, xfma(kc<float2>(-0.25), Cc, kc<float2>(1.0 / 3.0)));
    const float2 R = xfma(A, xfma(kc<float2>(-1.0 / 12.0), A, xfma(kc<float2>(-1.0 / 3.0), Cc, kc<float2>(1.0 / 3.0))), CB);
    const float2 Eh = xfma(vT2, xfma(bc2(c1), A, xmul(bc2(c2), Cc)),
                           xfma(vT, xfma(A, xfma(bc2(c3), A, xfma(bc2(c4), Cc, bc2(c5))), CB), xfma(A, R, bc2(tGh))));
    const float2 Oh = xmul(U, xfma(vT2, bc2(c8), xfma(vT, xfma(bc2(c6), A, xfma(bc2(c2), Cc, bc2(kh2))), R)));
    const float2 dQ0 = bc2(xmul(q.drho, Q0)), vR = bc2(q.RTc);
    const float2 hp = xmul(vR, xfma(vr, xadd(Eh, Oh), dQ0)), hm = xmul(vR, xfma(vr, xsub(Eh, Oh), dQ0));
    h[0] = hp.x; h[1] = hp.y; h[2] = hm.x; h[3] = hm.y;
}

__device__ __forceinline__ void eqd_fam5(const EqDev<float> &q, float *f, float *h)
{
    const float u = q.u, v = q.v, T = q.T, K = q.K, T0 = q.T0, tau = q.tau;
    const float a = xmul(u, u), c = xmul(v, v), s2 = xadd(a, c), pc = xmul(a, c), T2 = xmul(T, T);
    const float S2 = xadd(T, T0), S3 = xfma(T, S2, xmul(T0, T0));
    // f = rho (base + (T (X + Y) + X Y)/4) + drho P0, X = a +- u, Y = c +- v
    const float P0 = xmul(0.25f, xmul(T0, T0)), base = xmul(xmul(0.25f, tau), S2);
    const float2 X = make_float2(xadd(a, u), xsub(a, u));
    const float2 vT = bc2(T), vr = bc2(q.rho), vb = bc2(base), dP0 = bc2(xmul(q.drho, P0));
    const float2 Yp = bc2(xadd(c, v)), Ym = bc2(xsub(c, v));
    const float2 fp = xfma(vr, xfma(kc<float2>(0.25), xfma(X, Yp, xmul(vT, xadd(X, Yp))), vb), dP0);
    const float2 fm = xfma(vr, xfma(kc<float2>(0.25), xfma(X, Ym, xmul(vT, xadd(X, Ym))), vb), dP0);
    f[0] = fp.x; f[1] = fp.y; f[2] = fm.y; f[3] = fm.x;
    // h = RTc (rho (EE +- OE +- EO +- OO) + drho Q0) with
    // EE = T2 (k8 + 9/8) s2 + T ((k8 + 5/4) pc + s2^2/8) + pc s2/8 + tau (k8 + 2/3) S3,
    // (OE, EO) = (u, v) (T2 (k8 + 3/4) + T ((k8 + 9/8) (c, a) + (a, c)/8) + (c, a) s2/8),
    // OO = u v (T (k8 + 3/4) + s2/8)
    const float k8 = xmul(0.125f, K), e1 = xadd(k8, 0.75f), e2 = xadd(k8, 1.125f), e3 = xadd(k8, 2.0f / 3.0f);
    const float Q0 = xmul(xmul(xmul(T0, T0), T0), e3);
    const float EE = xfma(T2, xmul(e2, s2),
                          xfma(T, xfma(xadd(k8, 1.25f), pc, xmul(0.125f, xmul(s2, s2))),
                               xfma(xmul(0.125f, pc), s2, xmul(xmul(tau, e3), S3))));
    const float2 P = make_float2(a, c), Q = make_float2(c, a);
    const float2 OEO = xmul(make_float2(u, v),
                            xfma(bc2(T2), bc2(e1), xfma(vT, xfma(bc2(e2), Q, xmul(kc<float2>(0.125), P)),
                                                         xmul(kc<float2>(0.125), xmul(Q, bc2(s2))))));
    const float OO = xmul(xmul(u, v), xfma(T, e1, xmul(0.125f, s2)));
    const float p = xadd(EE, OO), mm = xsub(EE, OO), so = xadd(OEO.x, OEO.y), dd = xsub(OEO.x, OEO.y);
    const float2 vR = bc2(q.RTc), dQ0 = bc2(xmul(q.drho, Q0));
    const float2 h01 = xmul(vR, xfma(vr, make_float2(xadd(p, so), xsub(mm, dd)), dQ0));
    const float2 h23 = xmul(vR, xfma(vr, make_float2(xsub(p, so), xadd(mm, dd)), dQ0));
    h[0] = h01.x; h[1] = h01.y; h[2] = h23.x; h[3] = h23.y;
}

__device__ __forceinline__ void eqd_fam9(const EqDev<float> &q, float *f, float *h)
{
    const float T = q.T, K = q.K, T0 = q.T0, tau = q.tau, T2 = xmul(T, T);
    const float S2 = xadd(T, T0), S3 = xfma(T, S2, xmul(T0, T0));
    const float kh3 = xfma(K, 1.0f / 16.0f, 1.0f / 3.0f), kh2 = xfma(K, -1.0f / 48.0f, -1.0f / 12.0f);
    const float P0 = xmul(T0, xfma(0.125f, T0, -1.0f / 24.0f));
    const float Q0 = xmul(xmul(T0, T0), xfma(T0, kh3, kh2));
    const float tGf = xmul(tau, xfma(0.125f, S2, -1.0f / 24.0f));
    const float tGh = xmul(tau, xfma(kh3, S3, xmul(kh2, S2)));
    const float2 U = make_float2(q.u, q.v), W = make_float2(q.v, q.u);
    const float2 A = xmul(U, U), Cc = xmul(W, W), vT = bc2(T), vT2 = bc2(T2), vr = bc2(q.rho);
    const float2 qT = bc2(xmul(0.25f, T)), Am1 = xadd(A, kc<float2>(-1.0));
    // f: E = A (T/4 + (A - 1)/24) + tau Gf, O = U (T/4 + (A - 1)/12)
    const float2 Ef = xfma(A, xfma(kc<float2>(1.0 / 24.0), Am1, qT), bc2(tGf));
    const float2 Of = xmul(U, xfma(kc<float2>(1.0 / 12.0), Am1, qT));
    const float2 dP0 = bc2(xmul(q.drho, P0));
    const float2 fp = xfma(vr, xadd(Ef, Of), dP0), fm = xfma(vr, xsub(Ef, Of), dP0);
    f[0] = fp.x; f[1] = fp.y; f[2] = fm.x; f[3] = fm.y;
    // h: with M = (A + Cc)(A - 1),
    // E = T2 (d1 A + Cc/16) + T (A (d2 A + Cc/8 - d3) - Cc/48) + A M/48 + tau Gh,
    // O = U (T2 d4 + T (d5 A + Cc/8 + d6) + M/24)
    const float d1 = xfma(0.125f, K, 17.0f / 16.0f), d2 = xfma(K, 1.0f / 48.0f, 1.0f / 3.0f);
    const float d3 = xfma(K, 1.0f / 48.0f, 7.0f / 48.0f), d4 = xfma(0.125f, K, 0.75f);
    const float d5 = xfma(K, 1.0f / 24.0f, 11.0f / 24.0f), d6 = xfma(K, -1.0f / 24.0f, -1.0f / 6.0f);
    const float2 M = xmul(xadd(A, Cc), Am1);
    const float2 Eh = xfma(vT2, xfma(bc2(d1), A, xmul(kc<float2>(1.0 / 16.0), Cc)),
                           xfma(vT, xfma(A, xfma(bc2(d2), A, xfma(kc<float2>(0.125), Cc, bc2(xneg(d3)))),
                                         xmul(kc<float2>(-1.0 / 48.0), Cc)),
                                xfma(kc<float2>(1.0 / 48.0), xmul(A, M), bc2(tGh))));
    const float2 Oh = xmul(U, xfma(vT2, bc2(d4), xfma(vT, xfma(bc2(d5), A, xfma(kc<float2>(0.125), Cc, bc2(d6))),
                                                      xmul(kc<float2>(1.0 / 24.0), M))));
    const float2 dQ0 = bc2(xmul(q.drho, Q0)), vR = bc2(q.RTc);
    const float2 hp = xmul(vR, xfma(vr, xadd(Eh, Oh), dQ0)), hm = xmul(vR, xfma(vr, xsub(Eh, Oh), dQ0));
    h[0] = hp.x; h[1] = hp.y; h[2] = hm.x; h[3] = hm.y;
}

// Equilibria of one family in the stored representation: full values on the
// FP64 path, deviations from the rest state on the FP32 path.
template <class C, bool DEV>
struct EqArgs;
template <class C>
struct EqArgs<C, false> {
    EqState<C> q;
    __device__ __forceinline__ EqArgs(double rho, double ux, double uy, double T, const SampleParams &sp)
        : q(eq_state<C>(rho, ux, uy, xmul(T, sp.inv_Tc), sp)) {}
    // Ends the sharing of subexpressions between the families before and
    // after it: kept for four families they are more registers than the few
    // products that form them again are worth (RK3 stage 3 spilled 850 bytes
    // a thread, 224 so).
    __device__ __forceinline__ void part() { asm volatile("" : "+d"(q.u), "+d"(q.v), "+d"(q.T), "+d"(q.K)); }
    __device__ __forceinline__ void fam(int f, C *fe, C *he) const
    {
        if (f == 0) eq_fam0(q, fe[0], he[0]);
        else if (f == 1) eq_fam1(q, fe, he);
        else if (f == 2) eq_fam5(q, fe, he);
        else eq_fam9(q, fe, he);
    }
};
template <class C>
struct EqArgs<C, true> {
    EqDev<C> q;
    __device__ __forceinline__ EqArgs(double rho, double ux, double uy, double T, const SampleParams &sp)
        : q(eq_dev<C>(rho, ux, uy, T, sp)) {}
    __device__ __forceinline__ void part() {}
    __device__ __forceinline__ void fam(int f, C *fe, C *he) const
    {
        if (f == 0) eqd_fam0(q, fe[0], he[0]);
        else if (f == 1) eqd_fam1(q, fe, he);
        else if (f == 2) eqd_fam5(q, fe, he);
        else eqd_fam9(q, fe, he);
    }
};

// all 26 values (init, pointwise stages)
template <class C>
__device__ __forceinline__ void eq_all(const EqState<C> &q, C *f, C *h)
{
    eq_fam0(q, f[0], h[0]);
    eq_fam1(q, f + 1, h + 1);
    eq_fam5(q, f + 5, h + 5);
    eq_fam9(q, f + 9, h + 9);
}

// ---------------------------------------------------------------- moments
// macroProp/macroPropShort (cpuLBM.cpp:877-970): FP64 sums over the node's
// 13 f and 13 h values.  The relaxation times tau_f = mu/p, tau_h =
// tau_f/Pr, tau_hf = tau_h tau_f / (tau_f - tau_h) (cpuLBM.cpp:952-955)
// enter every formula as their inverses, which are all linear in
// q = p / mu: 1/tau_f = q, 1/tau_h = Pr q, 1/tau_hf = (Pr - 1) q (so
// Pr = 1 gives 1/tau_hf = 0, the reference's x / inf).
struct Macro {
    double rho, ux, uy, T, p, q;
};

// LAW false: the samples have constant viscosity (no pow, whose call the
// registers live across it would have to be saved for)
template <bool LAW = true>
__device__ __forceinline__ Macro macro_from_sums(double r, double rux, double ruy, double sh, const SampleParams &sp)
{
    // stored deviations: add the rest state's rho0 and sum of h (0 when the
    // state is stored in full)
    // every operation explicitly rounded: each kernel gives a node the same
    // moments
    r = __dadd_rn(sp.rho0, r);
    sh = __dadd_rn(sp.shref, sh);
    Macro m;
    const double ir = __drcp_rn(r);
    m.rho = r;
    m.ux = __dmul_rn(rux, ir);
    m.uy = __dmul_rn(ruy, ir);
    const double usq = __fma_rn(m.uy, m.uy, __dmul_rn(m.ux, m.ux));
    m.T = __dmul_rn(__fma_rn(sh, ir, __dmul_rn(-0.5, usq)), sp.two_over_bR);
    m.p = __dmul_rn(__dmul_rn(r, sp.R), m.T);
    if (!LAW || sp.visc == 0) {
        m.q = m.p * sp.inv_mu;  // 1/tau_f = p/mu
    } else {
        double mu = sp.mu * pow(m.T / sp.visc_T, sp.visc_exp);
        if (sp.visc == 2) mu *= (sp.visc_T + sp.visc_S) / (m.T + sp.visc_S);
        m.q = m.p / mu;
    }
    return m;
}

// ---------------------------------------------------------- index and BCs
// index (cpuLBM.cpp:1033-1113): periodic wrap, mirror (-i-1 / 2N-i-1 with a
// reflection flag) or zeroth-order extrapolation (clamp).
__device__ __forceinline__ int bc_index(const SampleParams &sp, int i, int pm, int axis, int &mir)
{
    i += pm;
    mir = 0;
    const int N = axis == 0 ? sp.nx : sp.ny;
    if (i < 0) {
        if (sp.flags & (axis == 0 ? SF_PERX : SF_PERY)) i = N + i;
        else if (sp.flags & (axis == 0 ? SF_MIRW : SF_MIRS)) { i = -i - 1; mir = 1; }
        else i = 0;
    } else if (i > N - 1) {
        if (sp.flags & (axis == 0 ? SF_PERX : SF_PERY)) i = i - N;
        else if (sp.flags & (axis == 0 ? SF_MIRE : SF_MIRN)) { i = 2 * N - i - 1; mir = 1; }
        else i = N - 1;
    }
    return i;
}

// -------------------------------------------------------------- NND, WENO5
// Reconstructions of one face, f and h together as the lanes of a pair, from
// upwind-ordered values s0..s4 (NND: the middle three).  Everything that
// depends on one or three neighbouring values only is a function of its own,
// so that the faces of a line form it once (line_diffs); a single face
// (face5) takes the same operations, so the same bits.
//
// FP32 works on the values times |e|, as the reference does.  These flows
// amplify rounding by orders of magnitude over tens of steps, so the
// operations and their order are fixed: results do not change with the
// kernel's structure.  FP64 has room for a cheaper form on the differences
// of the unscaled values (below).

// what a direction's component along the axis gives a face: |e| (FP32), or
// epsilon / |e|^2 (FP64, whose flux differences are multiplied by |e| later)
template <class C>
struct FaceArg;
template <>
struct FaceArg<float> {
    float2 ae, aeh;  // |e|, |e| / 2
};
template <>
struct FaceArg<double> {
    double2 eps;
};
template <class C>
__device__ __forceinline__ FaceArg<C> face_arg(float c, double eps1, int comp)
{
    const bool two = comp == 2 || comp == -2;
    if constexpr (sizeof(C) == 4) {
        const float ae = two ? 2.f * c : c;
        return FaceArg<C>{make_float2(ae, ae), make_float2(0.5f * ae, 0.5f * ae)};
    } else {
        const double e = two ? 0.25 * eps1 : eps1;
        return FaceArg<C>{make_double2(e, e)};
    }
}
template <class C>
__device__ __forceinline__ FaceArg<C> face_arg(const SampleParams &sp, int comp)
{
    return face_arg<C>((float)sp.c, sp.eps1, comp);
}

// minmod with the reference's case order (cpuLBM.cpp:1130-1145): same
// signs -> the smaller magnitude (equal magnitudes mean a == b), else 0
template <class C>
__device__ __forceinline__ C minmod(C a, C b)
{
    return a * b > C(0) ? (fabs(a) < fabs(b) ? a : b) : C(0);
}

// FP32 reciprocal: PTX rcp.approx, inline, so that no compiled instance may
// lower a division another way: a face then rounds the same in every kernel
// that reconstructs it.  d is a positive normal number (a sum of weights, or
// eps + b_k).
__device__ __forceinline__ float rcp_approx(float d)
{
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
    return r;
}
// the quotients of both lanes, a reciprocal each.  (FP64: one reciprocal of
// the product of the denominators, multiplied back, takes as many operations
// but for a reciprocal's start, rounds twice more, and its product of 16th
// powers leaves the FP64 range at densities of 1e24 that vary by 1e-2.  A
// 1024^2 step 0.450 ms that way, 0.448 this way; an ensemble of 16 0.992 and
// 0.994.)
__device__ __forceinline__ float2 face_div(float2 n, float2 d)
{
    return __fmul2_rn(n, make_float2(rcp_approx(d.x), rcp_approx(d.y)));
}
__device__ __forceinline__ double2 face_div(double2 n, double2 d)
{
    return make_double2(xmul(n.x, rcp64(d.x)), xmul(n.y, rcp64(d.y)));
}

// WENO5 (cpuLBM.cpp:1358-1403): Jiang-Shu indicators b_k, linear weights
// 1/10, 6/10, 3/10, epsilon 1e-6.  The nonlinear weights d_k/(eps+b_k)^2
// normalised by their sum are formed as d_k prod_{j!=k} (eps+b_j)^2 over the
// same sum (one division per face).  That fourth power leaves the FP32 range
// on dimensional data; for samples whose scales allow that
// (SampleParams::wide, set on the host) the FP32 weights are formed as
// d_k (m/(eps+b_k))^2 instead, m the smallest eps+b_j, each ratio in (0, 1].

// ---- FP32.  w = |e| s / 2: half the scaled value, so that the smoothness
// terms need no factors (a quarter of a slope's square is the square of its
// half).  Factors of two round nothing, so they are moved to where they cost
// no operation.
struct WenoCurv32 {
    float2 d, k;  // half the second difference, 13/3 of it
};
__device__ __forceinline__ WenoCurv32 weno_curv(float2 w0, float2 w1, float2 w2)
{
    const float2 d = xfma(kc<float2>(-2), w1, xadd(w0, w2));
    return WenoCurv32{d, xmul(make_float2(4.f * (float)(13.0 / 12.0), 4.f * (float)(13.0 / 12.0)), d)};
}
// the face from its five points and the curvatures at the middle three
template <bool WIDE>
__device__ __forceinline__ float2 weno_face(float2 p0, float2 p1, float2 p2, float2 p3, float2 p4, const WenoCurv32 &c0,
                                            const WenoCurv32 &c1, const WenoCurv32 &c2)
{
    using V = float2;
    // half the one-sided slopes of the three stencils
    const V l0 = xfma(kc<V>(3), p2, xfma(kc<V>(-4), p1, p0));
    const V l1 = xsub(p1, p3);
    const V l2 = xfma(kc<V>(-4), p3, xfma(kc<V>(3), p2, p4));
    // eps + b_k
    const V a0 = xfma(c0.k, c0.d, xfma(l0, l0, kc<V>(1e-6)));
    const V a1 = xfma(c1.k, c1.d, xfma(l1, l1, kc<V>(1e-6)));
    const V a2 = xfma(c2.k, c2.d, xfma(l2, l2, kc<V>(1e-6)));
    V w0, w1, w2;  // weights; of the middle one minus a half
    constexpr float k1 = -0.5f * (float)0.6;
    if constexpr (WIDE) {
        const V m = xmin(a0, xmin(a1, a2));
        const V s0 = face_div(m, a0), s1 = face_div(m, a1), s2 = face_div(m, a2);
        w0 = xmul(kc<V>(0.1), xmul(s0, s0));
        w1 = xmul(make_float2(k1, k1), xmul(s1, s1));
        w2 = xmul(kc<V>(0.3), xmul(s2, s2));
    } else {
        const V b0 = xmul(a0, a0), b1 = xmul(a1, a1), b2 = xmul(a2, a2);
        w0 = xmul(kc<V>(0.1), xmul(b1, b2));
        w1 = xmul(make_float2(k1, k1), xmul(b0, b2));
        w2 = xmul(kc<V>(0.3), xmul(b0, b1));
    }
    // candidate reconstructions, times 3/2 (the middle one: times -3)
    const V r0 = xfma(kc<V>(5.5), p2, xfma(kc<V>(-3.5), p1, p0));
    const V r1 = xfma(kc<V>(-2), p3, xfma(kc<V>(-5), p2, p1));
    const V r2 = xfma(kc<V>(-0.5), p4, xfma(kc<V>(2.5), p3, p2));
    return face_div(xfma(w2, r2, xfma(w1, r1, xmul(w0, r0))), xmul(kc<V>(1.5), xadd(xfma(kc<V>(-2), w1, w0), w2)));
}
// NND (cpuLBM.cpp:1328-1356): c = |e| s1, the differences to |e| s2, |e| s0
__device__ __forceinline__ float2 nnd_face(float2 s0, float2 s1, float2 s2, float2 c, const FaceArg<float> &g)
{
    const float2 nae = make_float2(-g.ae.x, -g.ae.y);
    const float2 nf = xfma(nae, s2, c), b = xfma(nae, s0, c);  // minus the forward difference, the backward one
    return xfma(kc<float2>(0.5), make_float2(minmod(-nf.x, b.x), minmod(-nf.y, b.y)), c);
}

// ---- FP64, on first differences e_j = s_{j+1} - s_j and second differences
// d_k of the unscaled values: both schemes are homogeneous, so |e| can
// multiply the flux difference once.  With the one-sided slopes m_k,
//   eps + b_k = t_k + m_k^2,  t_k = 13/12 d_k^2 + eps,
//   m0 = e1 + d0/2, m1 = e1 + d1/2, m2 = e2 - d2/2,
// and the candidates are s + c_k/2, c0 = e1 + 2/3 d0, c1 = e1 + 2/3 d1,
// c2 = e2 - d2/3 (weights 1, 6, 3): 29 operations a face in a line against
// 39 for the form above, and the correction to the centre value is small
// where the flow is smooth.
__device__ __forceinline__ double2 weno_t(double2 d, double2 eps)
{
    return xfma(xmul(kc<double2>(13.0 / 12.0), d), d, eps);
}
__device__ __forceinline__ double2 weno_face(double2 s, double2 e1, double2 e2, double2 d0, double2 d1, double2 d2,
                                             double2 t0, double2 t1, double2 t2)
{
    using V = double2;
    const V m0 = xfma(kc<V>(0.5), d0, e1), m1 = xfma(kc<V>(0.5), d1, e1), m2 = xfma(kc<V>(-0.5), d2, e2);
    const V a0 = xfma(m0, m0, t0), a1 = xfma(m1, m1, t1), a2 = xfma(m2, m2, t2);
    const V p0 = xmul(a0, a0), p1 = xmul(a1, a1), p2 = xmul(a2, a2), g = xmul(kc<V>(3.0), p0);
    const V w0 = xmul(p1, p2), y = xmul(g, p2), w2 = xmul(g, p1);  // weights 1, 6 / 2, 3
    const V c0 = xfma(kc<V>(2.0 / 3.0), d0, e1), c2 = xfma(kc<V>(-1.0 / 3.0), d2, e2);
    const V c1 = xfma(kc<V>(4.0 / 3.0), d1, xadd(e1, e1));  // twice c1
    const V num = xfma(y, c1, xfma(w2, c2, xmul(w0, c0)));
    const V den = xfma(kc<V>(2.0), y, xadd(w0, w2));
    return xfma(kc<V>(0.5), face_div(num, den), s);
}
__device__ __forceinline__ double2 nnd_face(double2 s1, double2 e0, double2 e1)
{
    return xfma(kc<double2>(0.5), make_double2(minmod(e1.x, e0.x), minmod(e1.y, e0.y)), s1);
}

// one face; FM: 0 NND, 1 WENO5, 2 WENO5 with the range-safe weights (FP32)
template <int FM>
__device__ __forceinline__ float2 face5(float2 s0, float2 s1, float2 s2, float2 s3, float2 s4, const FaceArg<float> &g)
{
    if constexpr (FM == 0) return nnd_face(s1, s2, s3, xmul(g.ae, s2), g);
    else {
        const float2 p0 = xmul(g.aeh, s0), p1 = xmul(g.aeh, s1), p2 = xmul(g.aeh, s2), p3 = xmul(g.aeh, s3),
                     p4 = xmul(g.aeh, s4);
        return weno_face<FM == 2>(p0, p1, p2, p3, p4, weno_curv(p0, p1, p2), weno_curv(p1, p2, p3),
                                  weno_curv(p2, p3, p4));
    }
}
template <int FM>
__device__ __forceinline__ double2 face5(double2 s0, double2 s1, double2 s2, double2 s3, double2 s4,
                                         const FaceArg<double> &g)
{
    const double2 e1 = xsub(s2, s1), e2 = xsub(s3, s2);
    if constexpr (FM == 0) return nnd_face(s2, e1, e2);
    else {
        const double2 d0 = xsub(e1, xsub(s1, s0)), d1 = xsub(e2, e1), d2 = xsub(xsub(s4, s3), e2);
        return weno_face(s2, e1, e2, d0, d1, d2, weno_t(d0, g.eps), weno_t(d1, g.eps), weno_t(d2, g.eps));
    }
}

// the scheme read at run time (general tiles, wall factors); one compiled
// copy of each scheme, out of line
template <class C>
__device__ __noinline__ Pair<C> face5_rt(int fm, Pair<C> s0, Pair<C> s1, Pair<C> s2, Pair<C> s3, Pair<C> s4,
                                         FaceArg<C> g)
{
    if (fm == 0) return face5<0>(s0, s1, s2, s3, s4, g);
    if constexpr (sizeof(C) == 4)
        if (fm == 2) return face5<2>(s0, s1, s2, s3, s4, g);
    return face5<1>(s0, s1, s2, s3, s4, g);
}

// flux differences along a line of LEN nodes: v[k] are the values at nodes
// k - 3 in upwind order (k = 0 .. LEN + 4), out[n] = F(n) - F(n - 1) for the
// nodes n = 0 .. LEN - 1, F(n) the face downwind of node n.  hook(n, F) may
// replace the face (n = -1 .. LEN - 1; walls).
template <int FM, int LEN, class HOOK>
__device__ __forceinline__ void line_diffs(const float2 (&v)[LEN + 5], const FaceArg<float> &g, float2 (&out)[LEN],
                                           HOOK hook)
{
    float2 prev;
    if constexpr (FM == 0) {
#pragma unroll
        for (int n = -1; n < LEN; ++n) {
            const float2 F = hook(n, nnd_face(v[n + 2], v[n + 3], v[n + 4], xmul(g.ae, v[n + 3]), g));
            if (n >= 0) out[n] = xsub(F, prev);
            prev = F;
        }
    } else {
        float2 p0 = xmul(g.aeh, v[0]), p1 = xmul(g.aeh, v[1]), p2 = xmul(g.aeh, v[2]), p3 = xmul(g.aeh, v[3]);
        WenoCurv32 c0 = weno_curv(p0, p1, p2), c1 = weno_curv(p1, p2, p3);
#pragma unroll
        for (int n = -1; n < LEN; ++n) {
            const float2 p4 = xmul(g.aeh, v[n + 5]);
            const WenoCurv32 c2 = weno_curv(p2, p3, p4);
            const float2 F = hook(n, weno_face<FM == 2>(p0, p1, p2, p3, p4, c0, c1, c2));
            if (n >= 0) out[n] = xsub(F, prev);
            prev = F;
            p0 = p1;
            p1 = p2;
            p2 = p3;
            p3 = p4;
            c0 = c1;
            c1 = c2;
        }
    }
}
template <int FM, int LEN, class HOOK>
__device__ __forceinline__ void line_diffs(const double2 (&v)[LEN + 5], const FaceArg<double> &g, double2 (&out)[LEN],
                                           HOOK hook)
{
    using V = double2;
    V prev;
    if constexpr (FM == 0) {
        V e0 = xsub(v[2], v[1]);
#pragma unroll
        for (int n = -1; n < LEN; ++n) {
            const V e1 = xsub(v[n + 4], v[n + 3]);
            const V F = hook(n, nnd_face(v[n + 3], e0, e1));
            if (n >= 0) out[n] = xsub(F, prev);
            prev = F;
            e0 = e1;
        }
    } else {
        V e1 = xsub(v[2], v[1]), e2 = xsub(v[3], v[2]);
        V d0 = xsub(e1, xsub(v[1], v[0])), d1 = xsub(e2, e1);
        V t0 = weno_t(d0, g.eps), t1 = weno_t(d1, g.eps);
#pragma unroll
        for (int n = -1; n < LEN; ++n) {
            const V e3 = xsub(v[n + 5], v[n + 4]);
            const V d2 = xsub(e3, e2);
            const V t2 = weno_t(d2, g.eps);
            const V F = hook(n, weno_face(v[n + 3], e1, e2, d0, d1, d2, t0, t1, t2));
            if (n >= 0) out[n] = xsub(F, prev);
            prev = F;
            e1 = e2;
            e2 = e3;
            d0 = d1;
            d1 = d2;
            t0 = t1;
            t1 = t2;
        }
    }
}
__device__ __forceinline__ int scheme_of(const SampleParams &sp) { return sp.fm ? (sp.wide ? 2 : 1) : 0; }

// extrapolation over a solid edge (stencil): 2 f(m1) - f(m2)
template <class V>
__device__ __forceinline__ V extrapolate(V f1, V f2)
{
    return xsub(xadd(f1, f1), f2);
}

// One sample's stage buffer and node flags; offsets inside a sample fit in
// 32 bits (26 values of up to 2^26 nodes).
template <class S>
struct StageView {
    const S *__restrict__ st;        // plane 0 of the sample in the stage buffer
    const uint8_t *__restrict__ nf;  // node flags of the sample
    int plane;
    int pitch;
};

// the (f, h) pair of direction i at (x, y)
template <class S>
__device__ __forceinline__ Pair<S> ldv(const StageView<S> &v, int i, int x, int y)
{
    return __ldg(reinterpret_cast<const Pair<S> *>(v.st) + (i * v.plane + y * v.pitch + x));
}

// Exact stencil + reconstruction (stencil, cpuLBM.cpp:1171-1326, then NND/
// WENO5) for the flux (FP64: divided by |e|) of direction i along `axis` at
// (x, y): boundary-aware indices with reflections, and the linear
// extrapolation 2 f(m1) - f(m2) over the first solid/fluid edge met by the
// stencil.
template <class S, class C>
__device__ __noinline__ Pair<C> flux_exact(const SampleParams &sp, const StageView<S> &v, int x, int y, int i, int axis)
{
    const int ev = axis == 0 ? c_EX[i] : c_EY[i];
    const int e = isgn(ev);
    const int L = sp.fm ? 5 : 3, low = (L - 1) / 2, j0 = 2 - low;  // NND: the middle three of five
    const int pos = axis == 0 ? x : y;
    const int j1 = pos - e * low;
    Pair<C> S5[5];
    int sld[5];
    int any = 0;
#pragma unroll
    for (int j = 0; j < 5; ++j) {
        if (j < L) {
            int m;
            const int r = bc_index(sp, j1, e * j, axis, m);
            const int ii = m ? (axis == 0 ? c_MIR_EW[i] : c_MIR_NS[i]) : i;
            const int xr = axis == 0 ? r : x, yr = axis == 0 ? y : r;
            S5[j] = ldv(v, ii, xr, yr);
            sld[j] = (v.nf[yr * v.pitch + xr] & NF_TYPE) == 2;
            any |= sld[j];
        }
    }
    if (any) {
        int diff = 0, jj = 0, pe = 0, m;
        for (int j = 0; j < L - 1; ++j) {
            diff = sld[j] - sld[j + 1];
            if (diff > 0) { jj = j; pe = bc_index(sp, j1, e * j, axis, m); break; }
            if (diff < 0) { jj = j + 1; pe = bc_index(sp, j1, e * (j + 1), axis, m); break; }
        }
        const int r1 = bc_index(sp, pe, e * diff, axis, m);
        const int r2 = bc_index(sp, pe, e * 2 * diff, axis, m);
        const Pair<C> v1 = axis == 0 ? ldv(v, i, r1, y) : ldv(v, i, x, r1);
        const Pair<C> v2 = axis == 0 ? ldv(v, i, r2, y) : ldv(v, i, x, r2);
        const Pair<C> ext = extrapolate(v1, v2);
        // S5[jj] = ext; S5[jj - diff] = ext when inside the stencil
#pragma unroll
        for (int j = 0; j < 5; ++j)
            if (j < L && (j == jj || (j == jj - diff))) S5[j] = ext;
    }
    const FaceArg<C> g = face_arg<C>(sp, ev);
    if (j0) return face5_rt<C>(0, S5[0], S5[0], S5[1], S5[2], S5[2], g);
    return face5_rt<C>(scheme_of(sp), S5[0], S5[1], S5[2], S5[3], S5[4], g);
}

// Outgoing face flux (FP64: divided by |e|) of direction i along `axis` at a
// non-solid node; nodes with no solid and no clamped or mirrored edge within
// the stencil read the five neighbours directly (with single periodic wrap
// across a periodic edge).
template <class S, class C>
__device__ __forceinline__ Pair<C> flux_axis(const SampleParams &sp, const StageView<S> &v, int x, int y, int i,
                                             int axis, uint8_t nflag)
{
    const int ev = axis == 0 ? c_EX[i] : c_EY[i];
    const uint8_t slow = axis == 0 ? (NF_SOLX | NF_EDGX) : (NF_SOLY | NF_EDGY);
    if (nflag & slow) return flux_exact<S, C>(sp, v, x, y, i, axis);
    const int e = ev > 0 ? 1 : -1;
    const bool wrap = (nflag & (axis == 0 ? NF_WRPX : NF_WRPY)) != 0;
    const int N = axis == 0 ? sp.nx : sp.ny, pos = axis == 0 ? x : y;
    Pair<C> q[5];
#pragma unroll
    for (int j = 0; j < 5; ++j) {
        int r = pos + e * (j - 2);
        if (wrap) {
            r += r < 0 ? N : 0;
            r -= r >= N ? N : 0;
        }
        q[j] = axis == 0 ? ldv(v, i, r, y) : ldv(v, i, x, r);
    }
    return face5_rt<C>(scheme_of(sp), q[0], q[1], q[2], q[3], q[4], face_arg<C>(sp, ev));
}

// wallFluxes (cpuLBM.cpp:1502-1590): for a solid node next to fluid,
// alpha = (f flux of the fluid 4-neighbours into it) / (|e| f out of it),
// weighted by the solid cell's 1/dx, 1/dy; one alpha for f and h.  Works on
// full values (stored values + fr, the rest state of stored deviations) and
// gives alpha - 1.  Sums in FP64, every operation explicitly rounded: the
// stencil kernels form the factor of a straight wall themselves, with the
// same bits.
__constant__ int c_WXX[4] = {-1, 1, 0, 0};
__constant__ int c_WYY[4] = {0, 0, -1, 1};
__constant__ int c_WII[4][4] = {{1, 5, 8, 9}, {3, 6, 7, 11}, {2, 5, 6, 10}, {4, 7, 8, 12}};
__constant__ int c_WINV[4][4] = {{3, 6, 7, 11}, {1, 5, 8, 9}, {4, 8, 7, 12}, {2, 6, 5, 10}};

// sums of the fluxes in (F: a face flux, FP64's divided by |e|) and out
// (v: a stored value), fr the rest value, ce = |e|, dd the cell width
__device__ __forceinline__ double wall_in(double acc, float F, double fr, double ce, double dd)
{
    return __dadd_rn(acc, __ddiv_rn(__fma_rn(ce, fr, (double)F), dd));
}
__device__ __forceinline__ double wall_in(double acc, double F, double fr, double ce, double dd)
{
    return __dadd_rn(acc, __ddiv_rn(__dmul_rn(ce, __dadd_rn(F, fr)), dd));
}
__device__ __forceinline__ double wall_out(double acc, double v, double fr, double ce, double dd)
{
    return __dadd_rn(acc, __ddiv_rn(__dmul_rn(__dadd_rn(v, fr), ce), dd));
}
__device__ __forceinline__ double wall_ratio_m1(double fin, double fout) { return __dsub_rn(__ddiv_rn(fin, fout), 1.0); }

// wallFluxes' alpha |e| f on full values, written for stored ones: |e| times
// f_s + (alpha - 1)(f_s + f_ref), f and h (FP64: divided by |e|)
template <class C>
__device__ __forceinline__ Pair<C> wall_flux(C am1, Pair<C> fs, const double *fr, int i, const FaceArg<C> &g)
{
    const Pair<C> v = make_pair2(xfma(am1, xadd(fs.x, (C)fr[i]), fs.x), xfma(am1, xadd(fs.y, (C)fr[NQ + i]), fs.y));
    if constexpr (sizeof(C) == 4) return xmul(g.ae, v);
    else return v;
}

template <class S, class C>
__device__ double wall_alpha_m1(const SampleParams &sp, const StageView<S> &v, int x, int y, double dxm, double dym,
                                const double *fr)
{
    double fin = 0, fout = 0;
    for (int j = 0; j < 4; ++j) {
        int m;
        const int xm = bc_index(sp, x, c_WXX[j], 0, m);
        const int ym = bc_index(sp, y, c_WYY[j], 1, m);
        const uint8_t fl = v.nf[ym * v.pitch + xm];
        if ((fl & NF_TYPE) >= 2) continue;
        const int axis = j < 2 ? 0 : 1;
        const double dd = axis == 0 ? dxm : dym;
        for (int q = 0; q < 4; ++q) {
            const int i = c_WII[j][q], io = c_WINV[j][q];
            const double ci = sp.c * abs(axis == 0 ? c_EX[i] : c_EY[i]);
            const double co = sp.c * abs(axis == 0 ? c_EX[io] : c_EY[io]);
            fin = wall_in(fin, flux_axis<S, C>(sp, v, xm, ym, i, axis, fl).x, fr[i], ci, dd);
            fout = wall_out(fout, (double)ldv(v, io, x, y).x, fr[io], co, dd);
        }
    }
    return wall_ratio_m1(fin, fout);
}

}  // namespace uqlbm
