// Per-node pieces shared by the pointwise and the stencil kernels: moment
// sums, e_i . u, ghost-column images.
#pragma once

#include "lbm_device.cuh"
#include "lbm_kernels.h"

namespace uqlbm {

// the sample's plane 0 of a buffer as (f, h) pairs
template <class S>
__device__ __forceinline__ Pair<S> *pair_base(S *base, const SampleParams &sp)
{
    return reinterpret_cast<Pair<S> *>(base + sp.state_off);
}
template <class S>
__device__ __forceinline__ const Pair<S> *pair_base(const S *base, const SampleParams &sp)
{
    return reinterpret_cast<const Pair<S> *>(base + sp.state_off);
}

// a second load of a value that was loaded before, not its register kept
__device__ __forceinline__ float2 load_again(const float2 *p)
{
    float2 v;
    asm volatile("ld.global.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(p));
    return v;
}

// Ghost columns (SampleParams::gx): a node within gx of an x edge also
// stores its stage-buffer values at its periodic image beyond the other
// edge.  The offset of that image (0: none) for the node at x; a stage value
// stored at o is, when this is nonzero, stored at o + offset too.
__device__ __forceinline__ int ghost_offset(const SampleParams &sp, int x)
{
    return sp.gx ? (x < sp.gx ? sp.nx : (x >= sp.nx - sp.gx ? -sp.nx : 0)) : 0;
}

// macroPropShort of one node from its 13 pairs, read through rd(i).
// The momentum sums are formed as sums of the values times the directions'
// integer components (0, +-1, +-2: exact, and no operation for 0 in the
// unrolled loops), scaled by c once.
__device__ __forceinline__ void mom_add(double &acc, int e, double v)
{
    if (e == 1) acc = __dadd_rn(acc, v);
    else if (e == -1) acc = __dsub_rn(acc, v);
    else if (e != 0) acc = __fma_rn((double)e, v, acc);
}

struct MomentSums {
    double r = 0, rx = 0, ry = 0, sh = 0;
    // i is a compile-time value in the unrolled loops
    __device__ __forceinline__ void add(int i, double f, double h)
    {
        r = __dadd_rn(r, f);
        mom_add(rx, lat_ex(i), f);
        mom_add(ry, lat_ey(i), f);
        sh = __dadd_rn(sh, h);
    }
    // the sums of v - d from those of v and of d: the small d are added up
    // among themselves, and the large sums rounded once (taking each d from
    // the sums of v rounds them 12 times: RK3's error of one step, f and h
    // together, 1.17e-15 of the values so, 0.94e-15 this way; Couette 40 x 45)
    __device__ __forceinline__ MomentSums less(const MomentSums &d) const
    {
        MomentSums m;
        m.r = __dsub_rn(r, d.r);
        m.rx = __dsub_rn(rx, d.rx);
        m.ry = __dsub_rn(ry, d.ry);
        m.sh = __dsub_rn(sh, d.sh);
        return m;
    }
    template <bool LAW = true>
    __device__ __forceinline__ Macro macro(const SampleParams &sp) const
    {
        return macro_from_sums<LAW>(r, __dmul_rn(sp.c, rx), __dmul_rn(sp.c, ry), sh, sp);
    }
};

template <bool LAW = true, class RD>
__device__ __forceinline__ Macro node_macro_rd(RD rd, const SampleParams &sp)
{
    MomentSums m;
#pragma unroll
    for (int i = 0; i < NQ; ++i) {
        const auto v = rd(i);
        m.add(i, (double)v.x, (double)v.y);
    }
    return m.macro<LAW>(sp);
}

// the same with st the sample's plane 0 and o the node's offset
template <class S>
__device__ __forceinline__ Macro node_macro(const Pair<S> *__restrict__ st, const SampleParams &sp, long long o)
{
    return node_macro_rd([&](int i) { return st[(long long)i * sp.plane + o]; }, sp);
}

// e_i . (cu, cv) for direction i, with cu = c u and cv = c v: the
// components are 0, +-1 or +-2, so each term is exact and only a diagonal
// direction adds (i a compile-time value in the unrolled loops)
template <class C>
__device__ __forceinline__ C e_dot(int i, C cu, C cv)
{
    const int ex = lat_ex(i), ey = lat_ey(i);
    const C x = ex == 1 ? cu : ex == -1 ? -cu : C(ex) * cu;
    const C y = ey == 1 ? cv : ey == -1 ? -cv : C(ey) * cv;
    return ex == 0 ? y : ey == 0 ? x : xadd(x, y);
}

// ------------------------------------------------- relaxations and updates
// Implicit BGK relaxation of one node at the moments m, FP64: over w dt,
// c = w dt (1/tau_f, 1/tau_h), g = w dt/tau_hf.  The stages are formed as
// distances from the equilibrium, which contract, and never as differences
// of two nearby stage values times c: with c = dt/tau up to 100, those
// differences would carry c times the rounding of the values.
struct Relax64 {
    double2 c, ic;  // c, 1/(1 + c)
    double g, cu, cv;
    __device__ __forceinline__ Relax64(const Macro &m, const SampleParams &sp, double w)
    {
        const double dt = xmul(w, sp.dt);  // m.q = 1/tau_f
        c = make_double2(xmul(dt, m.q), xmul(dt, xmul(sp.Pr, m.q)));
        ic = make_double2(rcp64(xadd(1.0, c.x)), rcp64(xadd(1.0, c.y)));
        g = xmul(dt, xmul(xsub(sp.Pr, 1.0), m.q));
        cu = xmul(sp.c, m.ux);
        cv = xmul(sp.c, m.uy);
    }
    // g e_i.u: h relaxes by ch (he - h) - g e.u (fe - f)
    __device__ __forceinline__ double coupling(int i) const { return xmul(g, e_dot<double>(i, cu, cv)); }
    // e - f1 from d0 = e - f: f1 = (f + c e)/(1 + c), h1 = (h + ch he - g eu (fe - f1))/(1 + ch)
    // (cpuLBM.cpp:1619-1663, 1819-1865)
    __device__ __forceinline__ double2 stage1(int i, double2 d0) const
    {
        const double f = xmul(d0.x, ic.x);
        return make_double2(f, xmul(xfma(coupling(i), f, d0.y), ic.y));
    }
    // e - f2 from d0 = e - f: f2 = (f + c f1)/(1 + c),
    // h2 = (h + ch h1 - g eu (f1 - f2))/(1 + ch) (cpuLBM.cpp:1869-1924, the
    // reference's -c (e - f1) + c e = c f1, its two coupling terms combined)
    __device__ __forceinline__ double2 stage2(int i, double2 d0) const
    {
        const double2 d1 = stage1(i, d0), r = xfma(c, d1, d0);
        const double f = xmul(r.x, ic.x);
        return make_double2(f, xmul(xfma(coupling(i), xsub(f, d1.x), r.y), ic.y));
    }
};

// Pointwise stages: RK1 stage 1 (RK = 0) or RK3 stages 1 and 2 (RK = 1).
// FP32: every operation explicitly rounded, in a fixed order.
template <class C, int RK>
struct PointStage;
template <int RK>
struct PointStage<float, RK> {
    float cf, ch, icf, ich, hg, g, dt, cu, cv;
    __device__ __forceinline__ PointStage(const Macro &m, const SampleParams &sp)
    {
        const float rq = (float)m.q, Pr = (float)sp.Pr;  // 1/tau_f
        dt = (float)sp.dt;
        const float w = RK == 1 ? xmul(0.5f, dt) : dt;
        cf = xmul(w, rq);
        ch = xmul(xmul(w, Pr), rq);
        g = xmul(xsub(Pr, 1.f), rq);
        hg = xmul(w, g);
        icf = __fdiv_rn(1.f, xadd(1.f, cf));
        ich = __fdiv_rn(1.f, xadd(1.f, ch));
        cu = xmul((float)sp.c, (float)m.ux);
        cv = xmul((float)sp.c, (float)m.uy);
    }
    __device__ __forceinline__ float2 value(int i, float2 v, float2 e) const
    {
        const float eu = e_dot<float>(i, cu, cv);
        if constexpr (RK == 1) {
            // (cpuLBM.cpp:1819-1924) with the stage-2 forms reduced:
            // -cf (fe - f1) + cf fe = cf f1, -ch (he - h1) + ch he = ch h1,
            // and the two coupling terms combine to hg eu (f1 - f2)
            const float hge = xmul(hg, eu);
            const float2 cc = make_float2(cf, ch);
            const float2 X = xfma(cc, e, v);
            const float f1 = xmul(X.x, icf);
            const float h1 = xmul(xsub(X.y, xmul(hge, xsub(e.x, f1))), ich);
            const float f2 = xmul(xfma(cf, f1, v.x), icf);
            const float h2 = xmul(xfma(ch, h1, xsub(v.y, xmul(hge, xsub(f1, f2)))), ich);
            return make_float2(f2, h2);
        } else {
            // cpuLBM.cpp:1619-1663
            const float f1 = xmul(xfma(cf, e.x, v.x), icf);
            const float h1 = xmul(xfma(ch, e.y, xfma(-xmul(dt, eu), xmul(xsub(e.x, f1), g), v.y)), ich);
            return make_float2(f1, h1);
        }
    }
};
template <int RK>
struct PointStage<double, RK> {
    Relax64 r;
    __device__ __forceinline__ PointStage(const Macro &m, const SampleParams &sp) : r(m, sp, RK == 1 ? 0.5 : 1.0) {}
    __device__ __forceinline__ double2 value(int i, double2 v, double2 e) const
    {
        const double2 d0 = xsub(e, v);
        return xsub(e, RK == 1 ? r.stage2(i, d0) : r.stage1(i, d0));
    }
};

// The pointwise stage that a step begins with, of a node with state v and
// moments m: RK3's stages 1 and 2 (RK 1) or RK1's stage 1 (RK 0), each value
// given to store(i, value).  Whether the equilibrium's mass check
// (sum f_eq = rho, in the stored values rho - rho0) fails.
template <class C, int RK, class STORE>
__device__ __forceinline__ bool first_stage(const Pair<C> (&v)[NQ], const Macro &m, const SampleParams &sp, double eq_tol,
                                            STORE store)
{
    EqArgs<C, sizeof(C) == 4> q(m.rho, m.ux, m.uy, m.T, sp);
    const PointStage<C, RK> p(m, sp);
    double sf = 0;
#pragma unroll
    for (int fam = 0; fam < 4; ++fam) {
        C fe[4], he[4];
        q.part();
        q.fam(fam, fe, he);
#pragma unroll
        for (int k = 0; k < (fam ? 4 : 1); ++k) {
            const int i = fam ? 4 * fam - 3 + k : 0;
            sf += (double)fe[k];
            store(i, p.value(i, v[i], make_pair2(fe[k], he[k])));
        }
    }
    return fabs(sf - (m.rho - sp.rho0)) > eq_tol * (sizeof(C) == 8 ? 1.0 : fmax(1.0, fabs(m.rho)));
}

// RK3 stage 3 (cpuLBM.cpp:1928-1993) and the part of the update
// (cpuLBM.cpp:1999-2042) that does not need the stage-3 fluxes, of direction
// i: from the state v, the divergence D of stage 2's fluxes, and the
// equilibria at stage 1's (= 2's) and stage 3's moments, the stage value n3
// and the partial update acc.  FP32: in the order that its results are
// compared in, D first.
struct Stage3 {
    float2 A2, A3;
    float hdt, cu1, cv1, cu3, cv3, g2, g3, ia3, ib3;
    __device__ __forceinline__ Stage3(const Macro &m1, const Macro &m3, const SampleParams &sp)
    {
        cu1 = xmul((float)sp.c, (float)m1.ux);
        cv1 = xmul((float)sp.c, (float)m1.uy);
        const float rq1 = (float)m1.q, rq3 = (float)m3.q, Pr = (float)sp.Pr;
        hdt = xmul((float)sp.dt, 0.5f);
        cu3 = xmul((float)sp.c, (float)m3.ux);
        cv3 = xmul((float)sp.c, (float)m3.uy);
        // hdt (1/tau_f, 1/tau_h) of stages 2 and 3, 1/tau_hf
        A2 = make_float2(xmul(hdt, rq1), xmul(hdt, xmul(Pr, rq1)));
        A3 = make_float2(xmul(hdt, rq3), xmul(hdt, xmul(Pr, rq3)));
        g2 = xmul(xsub(Pr, 1.f), rq1);
        g3 = xmul(xsub(Pr, 1.f), rq3);
        ia3 = __fdiv_rn(1.f, xadd(1.f, A3.x));
        ib3 = __fdiv_rn(1.f, xadd(1.f, A3.y));
    }
    // D1: the distance of stage 2's value from its equilibrium
    __device__ __forceinline__ void update(int i, float2 v, float2 D, float2 D1, float2 e3, float2 &n3, float2 &acc) const
    {
        const float eu2 = e_dot<float>(i, cu1, cv1), eu3 = e_dot<float>(i, cu3, cv3);
        const float2 X = xfma(A2, D1, xfma(A3, e3, i ? xsub(v, D) : v));
        const float f3 = xmul(X.x, ia3);
        // hdt times the coupling term
        const float hc = xmul(hdt, xfma(xmul(eu2, g2), D1.x, xmul(xmul(eu3, g3), xsub(e3.x, f3))));
        n3 = make_float2(f3, xmul(xsub(X.y, hc), ib3));
        acc = xfma(A3, xsub(e3, n3), xfma(A2, D1, i ? xfma(kc<float2>(-0.5), D, v) : v));
        acc.y = xsub(acc.y, hc);
    }
};

// The same on the FP64 path, in two halves: what the state alone gives, formed
// while the sweeps of the block's other warps still run, and the rest once the
// fluxes are there.  A third fewer operations than stage by stage, and the
// state is loaded once (a 1024^2 step 0.471 -> 0.449 ms).
struct Stage3Base {  // from stage 1's (= 2's) moments
    Relax64 r;
    __device__ __forceinline__ Stage3Base(const Macro &m1, const SampleParams &sp) : r(m1, sp, 0.5) {}
    // v + dt/2 (e - f2)/tau (h with its coupling term)
    __device__ __forceinline__ double2 base(int i, double2 v, double2 e1) const
    {
        const double2 d2 = r.stage2(i, xsub(e1, v));
        double2 b = xfma(r.c, d2, v);
        b.y = xfma(-r.coupling(i), d2.x, b.y);
        return b;
    }
};
struct Stage3Rest {  // from stage 3's moments
    Relax64 r;
    __device__ __forceinline__ Stage3Rest(const Macro &m3, const SampleParams &sp) : r(m3, sp, 0.5) {}
    __device__ __forceinline__ void update(int i, double2 b, double2 D, double2 e3, double2 &n3, double2 &acc) const
    {
        // f3 relaxes from b - D
        const double2 d3 = r.stage1(i, xsub(e3, i ? xsub(b, D) : b));
        n3 = xsub(e3, d3);
        acc = xfma(r.c, d3, i ? xfma(kc<double2>(-0.5), D, b) : b);
        acc.y = xfma(-r.coupling(i), d3.x, acc.y);
    }
};

// RK1 (MODE 3, cpuLBM.cpp:1674-1710), EULER (4, :2130-2168) and EULER_EQ (5,
// :2220-2258) updates of direction i from the state v, the divergence D and
// the equilibrium e at the state's moments; RK1's stage value is formed again
template <class C, int MODE>
struct Update;
template <int MODE>
struct Update<float, MODE> {
    PointStage<float, 0> p;
    __device__ __forceinline__ Update(const Macro &m, const SampleParams &sp) : p(m, sp) {}
    __device__ __forceinline__ float2 value(int i, float2 v, float2 D, float2 e) const
    {
        if constexpr (MODE == 5) return i ? xsub(e, D) : e;
        const float2 d = xsub(e, MODE == 3 ? p.value(i, v, e) : v);
        float2 n = xfma(make_float2(p.cf, p.ch), d, i ? xsub(v, D) : v);
        n.y = xfma(-xmul(xmul(p.dt, e_dot<float>(i, p.cu, p.cv)), p.g), d.x, n.y);
        return n;
    }
};
template <int MODE>
struct Update<double, MODE> {
    Relax64 r;
    __device__ __forceinline__ Update(const Macro &m, const SampleParams &sp) : r(m, sp, 1.0) {}
    // the update without its flux term, - D
    __device__ __forceinline__ double2 base(int i, double2 v, double2 e) const
    {
        if constexpr (MODE == 5) return e;
        const double2 d0 = xsub(e, v), d = MODE == 3 ? r.stage1(i, d0) : d0;
        double2 n = xfma(r.c, d, v);
        n.y = xfma(-r.coupling(i), d.x, n.y);
        return n;
    }
};

}  // namespace uqlbm
