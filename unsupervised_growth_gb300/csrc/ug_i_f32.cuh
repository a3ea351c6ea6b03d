// Single-precision HVC(I) DP8 step and the interneuron noise pre-pass.
//
// Equations of HHI_buffer (c++/src/HHI_buffer.cpp:426-690, rates
// c++/include/HHI_buffer.h:173-180), arranged for the SFU and issue budget:
//  * the three rates with slope -1/10 in v share one exponential:
//      E1 = exp(-(v+15)/10), exp(-(v+22)/10) = E1 e^-0.7, exp(-(v+4)/10) = E1 e^1.1,
//      and exp(-v/5) = (E1 e^1.5)^2;
//  * the four reciprocals of a stage (an, am, bh, wInf) come from one MUFU rcp;
//  * (n, m) and (V, h) travel as f32x2 pairs through the tableau sums: n and m obey the
//    same equation, so their pair goes through it without being taken apart;
//  * the removable singularities of the two rates x / (1 - exp(-x/10)) need their series
//    only within |x| < 1e-3.  The step runs without it, keeping the smallest |x| of its
//    stages, and a step that came that close (a few in a thousand spikes' steps) is taken
//    again with the series.  The selects and series of every stage were a fifth of the step:
//    1215 -> 937 instructions, a lone warp 1560 -> 1400 cycles, four warps per scheduler
//    7.20 -> 6.40 ms for the same work.
// Per neuron and stage: 4 ex2 + 1 rcp (60 SFU operations per step).
// All scalar operations are rounding intrinsics, so that no compiler contraction decides a
// result: the two forms of the step, and every kernel that takes it, give the same bits.
//
// The Poisson noise of an interneuron does not depend on its state
// (HHI_buffer::noise_check, HHI_buffer.cpp:278-294 only compares the neuron's
// clock with the next noise time), so the single build draws every noise event
// of the trial before integrating: k_noise_events stores (step, conductance
// kick) pairs per channel, consuming the neuron's stream in the reference's
// order (exc before inh within a step).  The integrator then applies kicks at
// their steps with no double-precision work in its loop.
#pragma once
#include "ug_ra_f32.cuh"

namespace ug {

struct IK2 { f2 nm, Vh; float w; };

// x / (1 - exp(-x/10)) near x = 0: the series 10 + x/2 + x^2/120
constexpr float kINear = 1e-3f;
__device__ __forceinline__ float i_vtrap_series(float x)
{
    return __fmaf_rn(x, __fmaf_rn(x, 1.0f / 120.0f, 0.5f), 10.0f);
}

// kSeries: with the series where |x| < kINear; without it, `near_x` collects the smallest |x|.
template <bool kSeries>
__device__ __forceinline__ IK2 i_rhs_x(f2 nm, f2 Vh, float w, float Ge, float Gi, float& near_x)
{
    typedef IConst K;
    const float v = Vh.x, h = Vh.y, n = nm.x, m = nm.y;
    const float E1 = mufu_ex2(__fmaf_rn(v, UG_EXA(-0.1), UG_EXB(-0.1, 15.0)));   // exp(-(v+15)/10)
    const float Ebn = mufu_ex2(__fmaf_rn(v, UG_EXA(-1.0 / 80.0), UG_EXB(-1.0 / 80.0, 25.0)));
    const float Ebm = mufu_ex2(__fmaf_rn(v, UG_EXA(-1.0 / 18.0), UG_EXB(-1.0 / 18.0, 47.0)));
    const float Eah = mufu_ex2(__fmaf_rn(v, UG_EXA(-0.05), UG_EXB(-0.05, 34.0)));
    const float x1 = __fadd_rn(v, 15.0f), x2 = __fadd_rn(v, 22.0f);
    float D1 = __fsub_rn(1.0f, E1);
    float D2 = __fmaf_rn(E1, -0.49658530379140947f, 1.0f);                       // 1 - exp(-(v+22)/10)
    if constexpr (kSeries) {
        if (fabsf(x1) < kINear) D1 = 1.0f;
        if (fabsf(x2) < kINear) D2 = 1.0f;
    } else {
        near_x = fminf(near_x, fminf(fabsf(x1), fabsf(x2)));
    }
    const float Ew0 = __fmul_rn(E1, 4.4816890703380645f);                        // exp(-v/10)
    const float D3 = __fmaf_rn(E1, 3.0041660239464334f, 1.0f);                   // 1 + exp(-(v+4)/10)
    const float D4 = __fmaf_rn(Ew0, Ew0, 1.0f);                                  // 1 + exp(-v/5)
    // four reciprocals from one
    const float p12 = __fmul_rn(D1, D2), p34 = __fmul_rn(D3, D4);
    const float r = mufu_rcp(__fmul_rn(p12, p34));
    const float r12 = __fmul_rn(p34, r), r34 = __fmul_rn(p12, r);
    float f1 = __fmul_rn(x1, __fmul_rn(D2, r12)), f2_ = __fmul_rn(x2, __fmul_rn(D1, r12));
    if constexpr (kSeries) {
        if (fabsf(x1) < kINear) f1 = i_vtrap_series(x1);
        if (fabsf(x2) < kINear) f2_ = i_vtrap_series(x2);
    }
    const float an = __fmul_rn(0.15f, f1), am = f2_;
    const float bh = __fmul_rn(10.0f, __fmul_rn(D4, r34));
    const float bn = __fmul_rn(0.2f, Ebn), bm = __fmul_rn(40.0f, Ebm), ah = __fmul_rn(0.7f, Eah);
    const float n2 = __fmul_rn(n, n);
    const float m3 = __fmul_rn(__fmul_rn(m, m), m);
    float kv = __fmul_rn(-(float)K::gL, __fsub_rn(v, (float)K::El));
    kv = __fmaf_rn(__fmul_rn(__fmul_rn(-(float)K::gNa, h), m3), __fsub_rn(v, (float)K::Ena), kv);
    const float gk = __fmaf_rn((float)K::gKHT, w, __fmul_rn(__fmul_rn((float)K::gKdr, n2), n2));
    kv = __fmaf_rn(-gk, __fsub_rn(v, (float)K::Ek), kv);
    kv = __fmaf_rn(-Ge, v, kv);
    kv = __fmaf_rn(-Gi, __fsub_rn(v, (float)K::Ei), kv);
    IK2 k;
    // (kn, km) = (an, am)(1 - (n, m)) - (bn, bm)(n, m)
    k.nm = fma2(make_float2(an, am), S(1.0f) - nm, make_float2(-bn, -bm) * nm);
    k.Vh = make_float2(kv, __fmaf_rn(ah, __fsub_rn(1.0f, h), __fmul_rn(-bh, h)));
    k.w = __fmaf_rn(D3, r34, -w);                                                // wInf - w
    return k;
}

// One DP8 step; returns the smallest |x| of its stages (kSeries false), see i_dp8_x.
// p.ge, p.gi: conductance decay factors of the 12 stages (float build: constants).
template <bool kSeries>
__device__ __forceinline__ float i_dp8_form(IStateR<float>& s, const IStep<float>& p)
{
    const DPT B7[] = {UG_DP_B7}, B8[] = {UG_DP_B8}, B9[] = {UG_DP_B9}, B10[] = {UG_DP_B10}, B11[] = {UG_DP_B11},
              B12[] = {UG_DP_B12}, BO[] = {UG_DP_OUT};
    const DPT* tb[6] = {B7, B8, B9, B10, B11, B12};
    const int cnt[6] = {4, 5, 6, 7, 8, 9};
    const int acount[5] = {1, 2, 2, 3, 3};
    const int astage[5][3] = {{0, 0, 0}, {0, 1, 0}, {0, 2, 0}, {0, 2, 3}, {0, 3, 4}};
    const double acoef[5][3] = {{1, 0, 0}, {1, 3, 0}, {1, 3, 0}, {20, -75, 75}, {3, 15, 12}};
    const double aden[5] = {18, 48, 32, 64, 80};
    const f2 dt2 = S(p.dt);
    const f2 nm0 = make_float2(s.n, s.m), Vh0 = make_float2(s.V, s.h);
    f2 knm[12] = {}, kVh[12] = {};
    float kw[12] = {};
    float near_x = 1e30f;
    // sum (+)= coefficient x stage derivative
    f2 anm, aVh;
    float aw;
    auto term = [&](bool first, int q, float c) {
        const f2 dnm = knm[q], dVh = kVh[q];
        const float dw = kw[q];
        anm = first ? dnm * S(c) : fma2(dnm, S(c), anm);
        aVh = first ? dVh * S(c) : fma2(dVh, S(c), aVh);
        aw = first ? __fmul_rn(dw, c) : __fmaf_rn(dw, c, aw);
    };
#pragma unroll
    for (int st = 0; st < 12; ++st) {
        f2 nm = nm0, Vh = Vh0;
        float w = s.w;
        if (st > 0) {
            if (st <= 5) {
                const int a = st - 1;
#pragma unroll
                for (int j = 0; j < 3; ++j)
                    if (j < acount[a]) term(j == 0, astage[a][j], (float)(acoef[a][j] / aden[a]));
            } else {
                const DPT* t = tb[st - 6];
#pragma unroll
                for (int j = 0; j < 9; ++j)
                    if (j < cnt[st - 6]) term(j == 0, t[j].s, (float)(t[j].num / t[j].den));
            }
            nm = fma2(dt2, anm, nm0);
            Vh = fma2(dt2, aVh, Vh0);
            w = __fmaf_rn(p.dt, aw, s.w);
        }
        const IK2 k = i_rhs_x<kSeries>(nm, Vh, w, __fmul_rn(s.Ge, p.ge[st]), __fmul_rn(s.Gi, p.gi[st]), near_x);
        knm[st] = k.nm;
        kVh[st] = k.Vh;
        kw[st] = k.w;
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) term(j == 0, BO[j].s, (float)(BO[j].num / BO[j].den));
    const f2 nm = fma2(dt2, anm, nm0), Vh = fma2(dt2, aVh, Vh0);
    s.V = Vh.x;
    s.h = Vh.y;
    s.n = nm.x;
    s.m = nm.y;
    s.w = __fmaf_rn(p.dt, aw, s.w);
    s.Ge = __fmul_rn(s.Ge, p.ge[11]);
    s.Gi = __fmul_rn(s.Gi, p.gi[11]);
    return near_x;
}

// Interneuron spike detection without branches (HHI_buffer::state_check,
// HHI_buffer.cpp:260-276): bit `shift` of fired is set on a spike.
__device__ __forceinline__ void i_check_f(float V, int& flag, uint32_t& fired, int shift)
{
    const int below = V < -25.0f, above = V > -20.0f;
    fired |= (uint32_t)(flag & below) << shift;
    flag = flag ? 1 - below : above;
}

// The step with the series, out of line: it runs a few times in a thousand spikes, and inlined
// it cost a lone warp's step 90 cycles of 1540.  (p stays where it is, in the kernel's
// parameters or in shared memory: the parameter is a __grid_constant__.)
static __device__ __noinline__ IStateR<float> i_dp8_series(IStateR<float> s, const IStep<float>& p)
{
    i_dp8_form<true>(s, p);
    return s;
}

// One DP8 step, with the series of the vtrap rates where a stage needs it.
__device__ __forceinline__ void i_dp8_x(IStateR<float>& s, const IStep<float>& p)
{
    IStateR<float> y = s;
    if (i_dp8_form<false>(y, p) < kINear) y = i_dp8_series(s, p);
    s = y;
}

}  // namespace ug
