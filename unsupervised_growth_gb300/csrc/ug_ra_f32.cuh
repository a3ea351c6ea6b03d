// Single-precision HVC(RA) Debrabant step, one or two neurons per thread.
//
// Same equations as the reference's HH2_test (c++/src/HH2_test.cpp:613-754,
// RHS :866-890, gating c++/include/HH2_test.h:265-276), written once over a lane
// type V: `float` (one neuron per thread) or `f2` (two, every add/mul/fma one packed
// f32x2 instruction).  Each operation rounds alike in both, so a neuron's trajectory is
// the same bits either way.
//  * exponentials are MUFU ex2 with log2(e) folded into the affine argument;
//  * the seven reciprocals of a stage (mInf, nInf/tauN, lInf, hInf/tauH, rInf,
//    cInf and ca/(ca+6)) come from two MUFU rcp: 1/a = b/(ab) etc.;
//  * (x - c) k products are single multiply-adds with the constants folded in, and a
//    negated factor is built negated (1 + e as -1 - e) instead of negated afterwards.
// Per neuron and step: 32 ex2 + 8 rcp on the SFU.
//
// What bounds it, measured on one warp and on four warps per SM scheduler: a packed step is
// about 720 instructions, 470 of them on the FMA pipe at two cycles each (the wide multiplies
// of Philox four), and takes 1450 cycles of a scheduler with four warps resident.  A lone warp
// is bound by the dependency chain of the four stages: 1310 cycles per packed step and 765 per
// scalar one.  Before the noise values and the spike detection were branch-free (below) the
// step held 29 branches and a lone warp took 2080 cycles.
#pragma once
#include "ug_neuron.cuh"

namespace ug {

__device__ __forceinline__ float mufu_ex2(float x)
{
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float mufu_rcp(float x)
{
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

typedef float2 f2;
__device__ __forceinline__ f2 S(float s) { return make_float2(s, s); }
__device__ __forceinline__ f2 operator+(f2 a, f2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ f2 operator-(f2 a, f2 b) { return __ffma2_rn(b, S(-1.0f), a); }
__device__ __forceinline__ f2 operator*(f2 a, f2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) { return __ffma2_rn(a, b, c); }

// Lane operations.  The scalar ones are the rounding intrinsics, which the compiler does
// not contract, so they round as the packed instructions do.
__device__ __forceinline__ float v_add(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float v_sub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float v_mul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float v_fma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ float v_ex2(float a) { return mufu_ex2(a); }
__device__ __forceinline__ float v_rcp(float a) { return mufu_rcp(a); }
__device__ __forceinline__ f2 v_add(f2 a, f2 b) { return a + b; }
__device__ __forceinline__ f2 v_sub(f2 a, f2 b) { return a - b; }
__device__ __forceinline__ f2 v_mul(f2 a, f2 b) { return a * b; }
__device__ __forceinline__ f2 v_fma(f2 a, f2 b, f2 c) { return fma2(a, b, c); }
__device__ __forceinline__ f2 v_ex2(f2 a) { return make_float2(mufu_ex2(a.x), mufu_ex2(a.y)); }
__device__ __forceinline__ f2 v_rcp(f2 a) { return make_float2(mufu_rcp(a.x), mufu_rcp(a.y)); }

template <class V>
struct Lanes;   // neurons per thread, a value in every lane, one lane's value
template <>
struct Lanes<float> {
    static constexpr int n = 1;
    static __device__ __forceinline__ float all(float s) { return s; }
    static __device__ __forceinline__ float get(float v, int) { return v; }
    static __device__ __forceinline__ float make(const float* x) { return x[0]; }
};
template <>
struct Lanes<f2> {
    static constexpr int n = 2;
    static __device__ __forceinline__ f2 all(float s) { return S(s); }
    static __device__ __forceinline__ float get(f2 v, int k) { return k ? v.y : v.x; }
    static __device__ __forceinline__ f2 make(const float* x) { return make_float2(x[0], x[1]); }
};

template <class V>
struct RAVec { V Vs, Vd, n, h, l, r, c, Ca; };

// log2(e)-scaled affine arguments: exp(k (v + b)) = ex2(K v + K b), K = k log2 e
#define UG_L2E 1.4426950408889634
#define UG_EXA(k) ((float)((k) * UG_L2E))
#define UG_EXB(k, b) ((float)((k) * (b) * UG_L2E))

template <class V>
struct RACell {
    V GdCa;            // the neuron's calcium conductance
    V cs, cd;          // GsL EL + mus and GdL EL + mud: the constant parts of the leak terms
};

// The per-neuron constants; mus, mud = 100000 mu / A.
template <class V>
__device__ __forceinline__ RACell<V> ra_cell(V EL, V GdCa, float mus, float mud)
{
    typedef RAConst K;
    typedef Lanes<V> L;
    RACell<V> P;
    P.GdCa = GdCa;
    P.cs = v_fma(EL, L::all((float)K::GsL), L::all(mus));
    P.cd = v_fma(EL, L::all((float)K::GdL), L::all(mud));
    return P;
}

// G: Gexc_d + Ginh_d, Gi: Ginh_d, at the stage's time.
template <class V>
__device__ __forceinline__ RAVec<V> ra_rhs(const RAVec<V>& y, V G, V Gi, const RACell<V>& P)
{
    typedef RAConst K;
#define C(x) Lanes<V>::all(x)
    const V vs = y.Vs, vd = y.Vd;
    // gating exponentials (HH2_test.h:265-276)
    const V Em = v_ex2(v_fma(vs, C(UG_EXA(-1.0 / 9.5)), C(UG_EXB(-1.0 / 9.5, 30.0))));
    const V En = v_ex2(v_fma(vs, C(UG_EXA(-0.1)), C(UG_EXB(-0.1, 35.0))));
    const V Et = v_ex2(v_fma(vs, C(UG_EXA(1.0 / 15.0)), C(UG_EXB(1.0 / 15.0, 27.0))));
    const V El = v_ex2(v_fma(vs, C(UG_EXA(-0.2)), C(UG_EXB(-0.2, 40.0))));
    const V Eh = v_ex2(v_fma(vs, C(UG_EXA(1.0 / 7.0)), C(UG_EXB(1.0 / 7.0, 45.0))));
    const V Eth = v_ex2(v_fma(vs, C(UG_EXA(1.0 / 6.0)), C(UG_EXB(1.0 / 6.0, 40.5))));
    const V Er = v_ex2(v_fma(vd, C(UG_EXA(-0.1)), C(UG_EXB(-0.1, 5.0))));
    const V Ec = v_ex2(v_fma(vd, C(UG_EXA(-1.0 / 7.0)), C(UG_EXB(-1.0 / 7.0, -10.0))));
    // denominators; the two of n and h are built from -(1 + En) and -(1 + Eh), which the
    // gating derivatives below take as well
    const V Dm = v_add(Em, C(1.0f));
    const V an = v_sub(C(-1.0f), En), bn = v_add(Et, C(1.0f));
    const V Dn = v_mul(an, v_fma(bn, C(-0.1f), C(-0.5f)));            // (1+En)(0.1(1+Et) + 0.5)
    const V Dl = v_add(El, C(1.0f));
    const V ah = v_sub(C(-1.0f), Eh), bh = v_add(Eth, C(1.0f));
    const V Dh = v_mul(ah, v_fma(bh, C(-0.1f), C(-0.75f)));
    const V Dr = v_add(Er, C(1.0f));
    const V Dc = v_add(Ec, C(1.0f));
    const V Dca = v_add(y.Ca, C(6.0f));
    // group A: 1/Dm, 1/Dn, 1/Dl from one reciprocal
    const V pmn = v_mul(Dm, Dn);
    const V rA = v_rcp(v_mul(pmn, Dl));
    const V iDl = v_mul(pmn, rA);
    const V rmn = v_mul(Dl, rA);
    const V iDm = v_mul(Dn, rmn), iDn = v_mul(Dm, rmn);
    // group B: 1/Dh, 1/Dr, 1/Dc, 1/Dca from one reciprocal
    const V phr = v_mul(Dh, Dr), pcc = v_mul(Dc, Dca);
    const V rB = v_rcp(v_mul(phr, pcc));
    const V rhr = v_mul(pcc, rB), rcc = v_mul(phr, rB);
    const V iDh = v_mul(Dr, rhr), iDr = v_mul(Dh, rhr), iDc = v_mul(Dca, rcc), iDca = v_mul(Dc, rcc);

    RAVec<V> k;
    const V m = iDm;
    const V m3 = v_mul(v_mul(m, m), m);
    const V n2 = v_mul(y.n, y.n);
    const V n4 = v_mul(n2, n2);
    // kVs = GsL (EL - vs) + GsNa m^3 h (EsNa - vs) + (GsK n^4 + GsKLT l)(EsK - vs) + mus
    //       + (vd - vs) 100000 / (Rc As); every (x - c) k is one multiply-add
    const V dv = v_sub(vd, vs);
    V t = v_fma(vs, C(-(float)K::GsL), P.cs);
    t = v_fma(v_mul(m3, y.h), v_fma(vs, C(-(float)K::GsNa), C((float)(K::GsNa * K::EsNa))), t);
    t = v_fma(v_fma(n4, C((float)K::GsK), v_mul(y.l, C((float)K::GsKLT))), v_sub(C((float)K::EsK), vs), t);
    k.Vs = v_fma(dv, C((float)(100000.0 / (K::Rc * K::As))), t);
    // kVd = GdL (EL - vd) + GdCa r^2 (EdCa - vd) - GdCaK (vd - EdK) c ca / (ca + 6)
    //       - Ge vd + Gi (Egaba - vd) + mud + (vs - vd) 100000 / (Rc Ad)
    const V gr2 = v_mul(v_mul(P.GdCa, y.r), y.r);
    const V eca = v_sub(C((float)K::EdCa), vd);
    V u = v_fma(vd, C(-(float)K::GdL), P.cd);
    u = v_fma(gr2, eca, u);
    u = v_fma(v_mul(v_sub(vd, C((float)K::EdK)), y.c), v_mul(v_mul(y.Ca, iDca), C(-(float)K::GdCaK)), u);
    u = v_fma(G, v_sub(C(0.0f), vd), v_fma(Gi, C((float)K::Egaba), u));
    k.Vd = v_fma(dv, C(-(float)(100000.0 / (K::Rc * K::Ad))), u);
    // kn = (nInf - n)/tauN = (1 - n (1 + En)) bn / Dn ; kh likewise
    k.n = v_mul(v_mul(v_fma(y.n, an, C(1.0f)), bn), iDn);
    k.h = v_mul(v_mul(v_fma(y.h, ah, C(1.0f)), bh), iDh);
    k.l = v_mul(v_sub(iDl, y.l), C(0.1f));
    k.r = v_sub(iDr, y.r);
    k.c = v_mul(v_sub(iDc, y.c), C(1.0f / 15.0f));
    k.Ca = v_fma(gr2, v_mul(eca, C(0.1f)), v_mul(y.Ca, C(-0.02f)));
    return k;
}

#define UG_RA_FOR(M) M(Vs) M(Vd) M(n) M(h) M(l) M(r) M(c) M(Ca)

// The step's noise: amplitude times point value, for the two draws of each compartment.
template <class V>
struct RANoise { V a1s, a2s, a1d, a2d; };

// One Debrabant step.
template <class V>
__device__ __forceinline__ void ra_debrabant_v(RAVec<V>& s, V& Ge, V& Gi, const RACell<V>& P, const RAStep<float>& p,
                                               const RANoise<V>& z)
{
    const V dt = C(p.dt);
    const V Ge1 = v_mul(Ge, C(p.e1)), Gi1 = v_mul(Gi, C(p.e1)), Gi2 = v_mul(Gi, C(p.e2));
    // Gexc + Ginh at the stages' times (the half step's has one rounding, as the compiler
    // contracts the packed form; written out, so that the scalar form has it too)
    const V G0 = v_add(Ge, Gi), G1 = v_add(Ge1, Gi1), G2 = v_fma(Ge, C(p.e2), Gi2);

    RAVec<V> y = s;
    y.Vs = v_fma(z.a1s, C(-0.01844540496323970f), v_fma(z.a2s, C(-0.1866426386543421f), s.Vs));
    y.Vd = v_fma(z.a1d, C(-0.01844540496323970f), v_fma(z.a2d, C(-0.1866426386543421f), s.Vd));
    const RAVec<V> a1 = ra_rhs(y, G0, Gi, P);

    RAVec<V> h4, up;   // running sums of stage 4's increment and of the update
#define M(f) h4.f = v_mul(a1.f, C(-0.4526683126055039f)); up.f = v_mul(a1.f, C(1.0f / 6.0f)); y.f = v_fma(dt, a1.f, s.f);
    UG_RA_FOR(M)
#undef M
    y.Vs = v_fma(z.a1s, C(0.8017012756521233f), v_fma(z.a2s, C(-0.8575745885712401f), y.Vs));
    y.Vd = v_fma(z.a1d, C(0.8017012756521233f), v_fma(z.a2d, C(-0.8575745885712401f), y.Vd));
    const RAVec<V> a2 = ra_rhs(y, G1, Gi1, P);

    const V d8 = C(p.dt * 0.125f);
#define M(f) h4.f = v_fma(a2.f, C(-0.4842227708685013f), h4.f); up.f = v_fma(a2.f, C(-0.005430430675258792f), up.f); \
             y.f = v_fma(d8, v_fma(a1.f, C(3.0f), a2.f), s.f);
    UG_RA_FOR(M)
#undef M
    y.Vs = v_fma(z.a1s, C(0.5092227024816198f), v_fma(z.a2s, C(-0.4723392695015512f), y.Vs));
    y.Vd = v_fma(z.a1d, C(0.5092227024816198f), v_fma(z.a2d, C(-0.4723392695015512f), y.Vd));
    const RAVec<V> a3 = ra_rhs(y, G2, Gi2, P);

#define M(f) h4.f = v_fma(a3.f, C(1.9368910834740051f), h4.f); up.f = v_fma(a3.f, C(2.0f / 3.0f), up.f); \
             y.f = v_fma(dt, h4.f, s.f);
    UG_RA_FOR(M)
#undef M
    y.Vs = v_fma(z.a1s, C(0.9758794209767762f), v_fma(z.a2s, C(0.3060354860326548f), y.Vs));
    y.Vd = v_fma(z.a1d, C(0.9758794209767762f), v_fma(z.a2d, C(0.3060354860326548f), y.Vd));
    const RAVec<V> a4 = ra_rhs(y, G1, Gi1, P);

#define M(f) s.f = v_fma(dt, v_fma(a4.f, C(0.1720970973419255f), up.f), s.f);
    UG_RA_FOR(M)
#undef M
    s.Vs = v_fma(z.a1s, C(100000.0f), s.Vs);
    s.Vd = v_fma(z.a1d, C(100000.0f), s.Vd);
    Ge = Ge1;
    Gi = Gi1;
}
#undef C

// The noise value of a word: the 30-point distribution index is (u * 30) >> 32, and
// index >= k exactly when u >= ceil(k 2^32 / 30), so unsigned comparisons against those
// bounds pick the value: 2.4494897f (sqrt(6)), its negative, 1, -1, 0.  Written as selects, because the
// compiler makes branches of the nested conditional expression: a lone warp's packed step
// took 2040 cycles with those, 1600 with the selects.  (A 30-entry table in shared memory
// indexed by the high product measured the same, within 1 %, with four warps per scheduler.)
__device__ __forceinline__ float ra_point_f(uint32_t u)
{
    float r;
    asm("{\n\t.reg .pred p, q, s, t;\n\t.reg .f32 a, b, c;\n\t"
        "setp.lt.u32 p, %1, 143165577;\n\t"
        "setp.lt.u32 q, %1, 286331154;\n\t"
        "setp.lt.u32 s, %1, 1574821342;\n\t"
        "setp.lt.u32 t, %1, 2863311531;\n\t"
        "selp.f32 a, 0fBF800000, 0f00000000, t;\n\t"
        "selp.f32 b, 0f3F800000, a, s;\n\t"
        "selp.f32 c, 0fC01CC470, b, q;\n\t"
        "selp.f32 %0, 0f401CC470, c, p;\n\t}"
        : "=f"(r)
        : "r"(u));
    return r;
}

// White noise of one or two neurons of a trial: block step - 1 of each neuron's stream
// (Philox4x32-10 with the key schedule of RAStep::ks).  The first two rounds split into a
// part of the neuron and trial, kept here, and a part of the step (and trial), shared by the
// thread's neurons, so a step runs eight rounds per neuron and two products for the rest.
template <class V>
struct RANoiseStream {
    uint32_t hi[Lanes<V>::n], lo[Lanes<V>::n];   // M0 times the neuron's word after round 1
    uint32_t tlo;                                // low half of M1 times the trial
    uint32_t tag;

    __device__ __forceinline__ void init(const uint32_t* entity, uint32_t trial, uint32_t tag_,
                                         const uint32_t* ks)
    {
        const uint64_t p1 = (uint64_t)0xCD9E8D57u * trial;
        tlo = (uint32_t)p1;
        tag = tag_;
#pragma unroll
        for (int k = 0; k < Lanes<V>::n; ++k) {
            const uint64_t p0 = (uint64_t)0xD2511F53u * ((uint32_t)(p1 >> 32) ^ entity[k] ^ ks[0]);
            hi[k] = (uint32_t)(p0 >> 32) ^ ks[3];
            lo[k] = (uint32_t)p0;
        }
    }
    // The scaled noise of step `step`; ns, nd are the compartments' amplitudes.
    __device__ __forceinline__ RANoise<V> draw(uint32_t step, float ns, float nd, const uint32_t* ks) const
    {
        const uint64_t q0 = (uint64_t)0xD2511F53u * (step - 1u);
        const uint64_t q1 = (uint64_t)0xCD9E8D57u * ((uint32_t)(q0 >> 32) ^ tag ^ ks[1]);
        const uint32_t b0 = (uint32_t)(q1 >> 32) ^ tlo ^ ks[2], b1 = (uint32_t)q1;
        float w[4][Lanes<V>::n];
#pragma unroll
        for (int k = 0; k < Lanes<V>::n; ++k) {
            uint32_t c0 = b0, c1 = b1, c2 = hi[k] ^ (uint32_t)q0, c3 = lo[k];
#pragma unroll
            for (int r = 2; r < 10; ++r) {
                const uint64_t p0 = (uint64_t)0xD2511F53u * c0, p1 = (uint64_t)0xCD9E8D57u * c2;
                const uint32_t n0 = (uint32_t)(p1 >> 32) ^ c1 ^ ks[2 * r];
                const uint32_t n2 = (uint32_t)(p0 >> 32) ^ c3 ^ ks[2 * r + 1];
                c1 = (uint32_t)p1;
                c3 = (uint32_t)p0;
                c0 = n0;
                c2 = n2;
            }
            w[0][k] = ra_point_f(c0);
            w[1][k] = ra_point_f(c1);
            w[2][k] = ra_point_f(c2);
            w[3][k] = ra_point_f(c3);
        }
        typedef Lanes<V> L;
        return RANoise<V>{v_mul(L::all(ns), L::make(w[0])), v_mul(L::all(ns), L::make(w[1])),
                          v_mul(L::all(nd), L::make(w[2])), v_mul(L::all(nd), L::make(w[3]))};
    }
};

// Spike detection on the state before the step, without branches (HH2_test::state_check,
// HH2_test.cpp:561-594): flags fs, fd are 0 / 1; bit `shift` of soma / dend is set on a spike.
__device__ __forceinline__ void ra_check_f(float Vs, float Vd, int& fs, int& fd, uint32_t& soma, uint32_t& dend,
                                           int shift)
{
    const int below_s = Vs < -35.0f, above_s = Vs > -30.0f;
    soma |= (uint32_t)(fs & below_s) << shift;
    fs = fs ? 1 - below_s : above_s;
    const int below_d = Vd < -35.0f, above_d = Vd >= -30.0f;
    dend |= (uint32_t)((1 - fd) & above_d) << shift;
    fd = fd ? 1 - below_d : above_d;
}

}  // namespace ug
