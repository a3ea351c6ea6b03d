// Double-precision integrators of one interval with eight lanes per neuron.
//
// What bounds the double build is the FP64 pipe of an SM sub-partition: an operation takes it
// 64 cycles whatever number of the warp's lanes take part.  With one neuron per thread
// (interval_ra_body, interval_i_body) a step is one long chain of such operations: about 2080
// of them for HVC(RA), 5750 for HVC(I), mostly the divisions of the Butcher tableau and one
// exponential after the other, and a batch of a few hundred neurons keeps a few warps busy.
// Here lane c of a group of eight holds component c of a neuron: each component's stage sums,
// each exponential and each rate's quotient is the same instruction on another lane, and the
// terms of the membrane equations meet in shuffles.  Divisions by a fixed divisor take three
// operations (div_known, ug_hd.h).  About 410 and 900 operations a step are left: 602 HVC(RA) and 150
// HVC(I) neurons, both kernels of one interval, 2.40 -> 0.41 ms.
//
// Every value is rounded as in the general bodies, operation by operation (this unit is
// compiled without contraction), so both give the same bits.
#pragma once
#include "ug_trial.cuh"

namespace ug {

constexpr int kLanes = 8;           // lanes of a neuron
constexpr int kLaneNeurons = 32 / kLanes;

__device__ __forceinline__ double pick8(int c, double a0, double a1, double a2, double a3, double a4, double a5,
                                        double a6, double a7)
{
    return c < 4 ? (c < 2 ? (c == 0 ? a0 : a1) : (c == 2 ? a2 : a3)) : (c < 6 ? (c == 4 ? a4 : a5) : (c == 6 ? a6 : a7));
}

// The value of lane `from` of the own group of eight.
__device__ __forceinline__ double grp(double x, int from) { return __shfl_sync(0xffffffffu, x, from, kLanes); }

// x, negated where neg
__device__ __forceinline__ double flip(double x, bool neg)
{
    return __hiloint2double(__double2hiint(x) ^ (neg ? 0x80000000 : 0), __double2loint(x));
}

// ---------------------------------------------------------------- HVC(RA)
// Lanes: 0 Vs, 1 n, 2 Vd, 3 l, 4 h, 5 Ca, 6 r, 7 c.  Exponential of each lane: 0 m, 1 n, 2 tau of
// n, 3 l, 4 h, 5 tau of h, 6 r, 7 c.  G: the inhibitory conductance on lane 5, else the excitatory.
struct RALanes {
    int c;
    bool soma_side;                     // the lane's exponential and current term see Vs, not Vd
    double xa, xd, xz; bool xneg;       // exponential of (+-)(v + xa) / xd
    double num1;                        // over 1 + exp
    double W;                           // divisor of the second quotient, where it is fixed
    double cz, Ec;                      // current term: cz (power) (v - Ec)
    double ncg;                         // -0.1 GdCa
    double EL, mu, sqsig, As, Asz;
};

__device__ __forceinline__ RALanes ra_lanes(int c, double EL, double GdCa, const RAStep<double>& p)
{
    typedef RAConst K;
    RALanes k;
    k.c = c;
    k.soma_side = c <= 5;               // of the exponentials; the current terms: 0, 1, 3, 4
    k.xa = pick8(c, 30, 35, 27, 40, 45, 40.5, 5, -10);
    k.xd = pick8(c, 9.5, 10, 15, 5, 7, 6, 10, 7);
    k.xz = pick8(c, 1 / 9.5, 1 / 10.0, 1 / 15.0, 1 / 5.0, 1 / 7.0, 1 / 6.0, 1 / 10.0, 1 / 7.0);
    k.xneg = !(c == 2 || c == 4 || c == 5);
    k.num1 = c == 2 ? 0.5 : c == 5 ? 0.75 : 1.0;
    k.W = pick8(c, K::Rc * K::As, 0.1, 1.0, 10.0, 0.1, K::Rc * K::Ad, 1.0, 15.0);
    k.cz = pick8(c, -K::GsL, K::GsK, -K::GdL, K::GsKLT, K::GsNa, 0.0, GdCa, 0.0);
    k.Ec = pick8(c, EL, K::EsK, EL, K::EsK, K::EsNa, K::Egaba, K::EdCa, 0.0);
    k.ncg = -0.1 * GdCa;
    k.EL = EL;
    k.As = (c == 2 ? K::Ad : K::As) * K::cm;
    k.Asz = c == 2 ? 1.0 / (K::Ad * K::cm) : 1.0 / (K::As * K::cm);
    k.mu = 100000 * (0.0 + (c == 2 ? p.mu_d : p.mu_s)) / (c == 2 ? K::Ad : K::As);
    k.sqsig = p.sq * (c == 2 ? p.sig_d : p.sig_s);
    return k;
}

// The derivative of the lane's component at the stage values y (ra_rhs_d).
__device__ __forceinline__ double ra_rhs_lane(const RALanes& k, double y, double G)
{
    typedef RAConst K;
    const int c = k.c;
    const double vs = grp(y, 0), vd = grp(y, 2), cc = grp(y, 7);
    const double x = flip((k.soma_side ? vs : vd) + k.xa, k.xneg);
    const double D1 = k.num1 / (1 + exp(div_known(x, k.xd, k.xz)));
    // lane 0: m, its square and cube; other lanes: of their own value
    const double u = c == 0 ? D1 : y;
    const double u2 = u * u, u3 = u2 * u, u4 = u3 * u;
    const double m3 = grp(u3, 0);
    const double six = grp(6 / (c == 5 ? y : 1.0), 5);             // 6 / ca
    const double tau = __shfl_down_sync(0xffffffffu, D1, 1, kLanes);
    const double W1 = (c == 2 ? 1.0 : 0.1) + (c == 2 ? six : tau);
    const double W = c == 1 || c == 2 || c == 4 ? W1 : k.W;
    // second quotient: the gates' rates, the coupling of the compartments (0: onto the soma,
    // 5: onto the dendrite) and the calcium-dependent potassium current (2)
    const bool coup = c == 0 || c == 5;
    const double from = c == 0 || c == 2 ? vd : c == 5 ? vs : D1;
    const double to = c == 0 ? vs : c == 2 ? K::EdK : c == 5 ? vd : y;
    double num2 = from - to;
    num2 = (coup ? 100000.0 : c == 2 ? K::GdCaK : 1.0) * num2;
    num2 = num2 * (c == 2 ? cc : 1.0);
    const double D2 = num2 / W;
    // currents
    const double vE = ((c == 0 || c == 1 || c == 3 || c == 4) ? vs : vd) - k.Ec;
    double z = k.cz * (c == 1 ? u4 : c == 4 ? m3 : c == 6 ? u2 : y);
    const double zh = z * y;
    z = c == 0 || c == 2 ? k.cz : c == 4 ? zh : c == 5 || c == 7 ? G : z;
    const double T = z * vE;
    const double kCa = grp(k.ncg * y * y * vE, 6) - 0.02 * y;
    // lane 0: T0 - T4 - T1 - T3 + mu + coupling; lane 2: T2 - T6 - D2 - T7 - T5 + mu + coupling
    const double t1 = grp(T, c == 0 ? 4 : 6), t2 = grp(T, 1), t3 = grp(T, c == 0 ? 3 : 7), t4 = grp(T, 5);
    double kV = T - t1;
    kV = kV - (c == 0 ? t2 : D2);
    kV = kV - t3;
    kV = kV - (c == 0 ? 0.0 : t4);
    kV = kV + k.mu;
    kV = kV + grp(D2, c == 0 ? 0 : 5);
    return c == 0 || c == 2 ? kV : c == 5 ? kCa : D2;
}

// One Debrabant step of the lane's component (ra_debrabant); J1, J2: the noise points of the
// lane's compartment.
__device__ __forceinline__ void ra_debrabant_lane(const RALanes& k, double& s, double& G, double dt, double e1, double e2,
                                                  double J1, double J2)
{
    const bool isV = k.c == 0 || k.c == 2;
    auto noise = [&](double sum) {      // sq sig (sum) / A; the gates have none
        const double v = div_known(k.sqsig * sum, k.As, k.Asz);
        return isV ? v : 0.0;
    };
    const double a1 = ra_rhs_lane(k, s + noise(-0.01844540496323970 * J1 - 0.1866426386543421 * J2), G);
    const double G1 = G * e1, G2 = G * e2;
    const double a2 = ra_rhs_lane(k, s + dt * a1 + noise(0.8017012756521233 * J1 - 0.8575745885712401 * J2), G1);
    const double a3 = ra_rhs_lane(k, s + dt * (3 * a1 + a2) * 0.125 + noise(0.5092227024816198 * J1 - 0.4723392695015512 * J2), G2);
    const double b1 = -0.4526683126055039, b2 = -0.4842227708685013, b3 = 1.9368910834740051;
    const double a4 = ra_rhs_lane(k, s + dt * (b1 * a1 + b2 * a2 + b3 * a3) +
                                     noise(0.9758794209767762 * J1 + 0.3060354860326548 * J2), G1);
    const double q2 = 0.005430430675258792, q4 = 0.1720970973419255;
    const double last = div_known(k.sqsig * J1 * 100000, k.As, k.Asz);
    s = s + dt * (div_known(a1, 6.0, 1 / 6.0) - q2 * a2 + div_known(2 * a3, 3.0, 1 / 3.0) + q4 * a4) + (isV ? last : 0.0);
    G = G1;
}

// HVC(RA) part of one interval, of neurons x = 0..B n_ra - 1, four to a warp (interval_ra_body).
__global__ void __launch_bounds__(kBlock, 1) k_interval_ra_lanes(NetDev<double> n, BatchDev<double> bt, int q, int s0,
                                                                 int s1, RAStep<double> rc)
{
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long all = (long long)bt.B * n.n_ra;
    const int c = (int)(t % kLanes);
    const bool valid = t / kLanes < all;
    const size_t x = (size_t)min(t / kLanes, all - 1);      // lanes past the end follow the last neuron
    const int b = (int)(x / n.n_ra), i = (int)(x - (size_t)b * n.n_ra);
    const int at = (int)pick8(c, 0, 2, 1, 4, 3, 7, 5, 6);   // the lane's array of bt.ra
    double s = bt.ra[at][x], G = bt.ra[c == 5 ? 9 : 8][x];
    const int flags = bt.ra_flags[x];
    int fl = c == 2 ? (flags >> 1) & 1 : flags & 1;
    if (q > 0) {
        const size_t slot = (size_t)((q - 1) % n.ring) * bt.B * n.n_ra + x;
        const long long ai = bt.ring_ra_inh[slot], ae = bt.ring_ra_exc[slot];
        __syncwarp();
        if (ai | ae) {
            if (valid && c == 0) {
                bt.ring_ra_inh[slot] = 0;
                bt.ring_ra_exc[slot] = 0;
            }
            G = G + (c == 5 ? (double)ai * kFixInv : ((double)ae * kFixInv) / RAConst::Ad);
        }
    }
    const int kick = bt.kick_step[x];
    const StreamId sid = make_stream(n.seed, kNoiseRAWhite, n.net_id, (uint32_t)i, bt.trial[b]);
    const RALanes k = ra_lanes(c, n.Erest[i], n.GCa[i], rc);
    uint32_t spikes = 0;                                    // lane 0: somatic, lane 2: dendritic
    for (int st = s0; st <= s1; ++st) {
        if (st == kick && c != 5) G = G + 3.0;
        const double e1 = n.ra_decay[2 * st], e2 = n.ra_decay[2 * st + 1];
        const bool low = s < -35.0, high = c == 2 ? s >= -30.0 : s > -30.0;
        spikes |= (uint32_t)(c == 2 ? !fl && high : fl && low) << (st - s0);
        fl = fl ? !low : high;
        const Philox4 w = stream_block(sid, (uint32_t)st - 1);
        ra_debrabant_lane(k, s, G, rc.dt, e1, e2, ra_point(point_index(c == 2 ? w.z : w.x)),
                          ra_point(point_index(c == 2 ? w.w : w.y)));
    }
    const uint32_t dend = __shfl_sync(0xffffffffu, spikes, 2, kLanes);
    const int fd = __shfl_sync(0xffffffffu, fl, 2, kLanes);
    if (valid) {
        bt.ra[at][x] = s;
        if (c == 5 || c == 7) bt.ra[c == 5 ? 9 : 8][x] = G;
    }
    const uint32_t soma = valid && c == 0 ? spikes : 0u;
    if (valid && c == 0) {
        bt.ra_flags[x] = (flags & ~3) | fl | (fd << 1);
        if (soma) {
            bt.ra_nsoma[x] += __popc(soma);
            if (bt.ra_first_soma[x] < 0) bt.ra_first_soma[x] = s0 + __ffs(soma) - 1;
            record_spikes(bt.spk_count, bt.spk_buf, bt.spk_cap, bt.error, b, i, kSpikeSoma, soma, s0);
        }
        if (dend) {
            bt.ra_ndend[x] += __popc(dend);
            if (bt.ra_first_dend[x] < 0) bt.ra_first_dend[x] = s0 + __ffs(dend) - 1;
            record_spikes(bt.spk_count, bt.spk_buf, bt.spk_cap, bt.error, b, i, kSpikeDend, dend, s0);
        }
        if (bt.soma_bits) bt.soma_bits[(size_t)(q & 1) * bt.B * n.n_ra + x] = (int)soma;
        if (bt.act_rows) queue_row(bt, q, (int)x, soma);
    }
    ra_scatter(n, bt, soma, i, b, s0);
}

// ----------------------------------------------------------------- HVC(I)
// Lanes: 0 V, 1 n, 2 m, 3 h, 4 w.  Exponential of each lane: 1 and 5 of n, 2 and 6 of m, 3 and 7
// of h, 4 of w.  G: the inhibitory conductance on lane 6, else the excitatory.
struct ILanes {
    int c;
    double xa, xd, xz;      // exponential of -(v + xa) / xd
    double mul;             // numerator of the quotient: mul (v + xa) on lanes 1 and 2, else mul
    double fc;              // factor of the exponential of lanes 5..7
    double cz, Ec;          // current term: cz (power) (v - Ec)
};

__device__ __forceinline__ ILanes i_lanes(int c)
{
    typedef IConst K;
    ILanes k;
    k.c = c;
    k.xa = pick8(c, 0, 15, 22, 4, 0, 25, 47, 34);
    k.xd = pick8(c, 5, 10, 10, 10, 5, 80, 18, 20);
    k.xz = pick8(c, 1 / 5.0, 1 / 10.0, 1 / 10.0, 1 / 10.0, 1 / 5.0, 1 / 80.0, 1 / 18.0, 1 / 20.0);
    k.mul = pick8(c, 1, 0.15, 1, 10, 1, 1, 1, 1);
    k.fc = pick8(c, 1, 1, 1, 1, 1, 0.2, 40, 0.7);
    k.cz = pick8(c, -K::gL, K::gKdr, 1, K::gNa, K::gKHT, 1, 1, 1);
    k.Ec = pick8(c, K::El, K::Ek, 0, K::Ena, K::Ek, 0, K::Ei, 0);
    return k;
}

// The derivative of the lane's component at the stage values y (i_rhs_d); Gs: G at the stage.
// Lanes without a component answer 1, so that their sums stay away from zero.
__device__ __forceinline__ double i_rhs_lane(const ILanes& k, double y, double Gs)
{
    const int c = k.c;
    const double v = grp(y, 0);
    const double x = v + k.xa;
    const double E = exp(div_known(-x, k.xd, k.xz));
    const bool trap = c == 1 || c == 2;
    const double xm = k.mul * x;
    const double Q = (trap ? xm : k.mul) / (1 + flip(E, trap));
    const double F = __shfl_down_sync(0xffffffffu, k.fc * E, 4, kLanes);   // lanes 1..3: of 5..7
    const double A = c == 3 ? F : Q, Bq = c == 3 ? Q : F;
    const double kk = A * (1 - y) - Bq * y;
    const double kw = Q - y;
    const double y2 = y * y, y3 = y2 * y, y4 = y3 * y;
    const double m3 = grp(y3, 2);
    double z = k.cz * (c == 1 ? y4 : y);
    const double zm = z * m3;
    z = c == 0 ? k.cz : c == 3 ? zm : c >= 5 ? Gs : z;
    const double T = z * (v - k.Ec);
    double kV = grp(T, 0) - grp(T, 3);
    kV = kV - grp(T, 1);
    kV = kV - grp(T, 4);
    kV = kV - grp(T, 5);
    kV = kV - grp(T, 6);
    kV = kV + 0.0;
    return c == 0 ? kV : c <= 3 ? kk : c == 4 ? kw : 1.0;
}

// One DP8 step of the lane's component (i_dp8); d: the decay factors of the lane's G.
__device__ __forceinline__ void i_dp8_lane(const ILanes& ln, double& s, double& G, double dt, const double* d)
{
    const DPT B7[] = {UG_DP_B7}, B8[] = {UG_DP_B8}, B9[] = {UG_DP_B9}, B10[] = {UG_DP_B10}, B11[] = {UG_DP_B11},
              B12[] = {UG_DP_B12}, BO[] = {UG_DP_OUT};
    const DPT* tb[6] = {B7, B8, B9, B10, B11, B12};
    const int cnt[6] = {4, 5, 6, 7, 8, 9};
    const int acount[5] = {1, 2, 2, 3, 3};
    const int astage[5][3] = {{0, 0, 0}, {0, 1, 0}, {0, 2, 0}, {0, 2, 3}, {0, 3, 4}};
    const double acoef[5][3] = {{1, 0, 0}, {1, 3, 0}, {1, 3, 0}, {20, -75, 75}, {3, 15, 12}};
    const double aden[5] = {18, 48, 32, 64, 80};
    double k[12];
#pragma unroll
    for (int st = 0; st < 12; ++st) {
        double y = s;
        if (st > 0 && st <= 5) {
            const int a = st - 1;
            double sum = acoef[a][0] * k[astage[a][0]];
#pragma unroll
            for (int j = 1; j < 3; ++j)
                if (j < acount[a]) sum = sum + acoef[a][j] * k[astage[a][j]];
            y = s + div_known(dt * sum, aden[a], 1.0 / aden[a]);
        } else if (st > 5) {
            const DPT* t = tb[st - 6];
            double sum = div_known(t[0].num * k[t[0].s], t[0].den, 1.0 / t[0].den);
#pragma unroll
            for (int j = 1; j < 9; ++j)
                if (j < cnt[st - 6]) sum = sum + div_known(t[j].num * k[t[j].s], t[j].den, 1.0 / t[j].den);
            y = s + dt * sum;
        }
        k[st] = i_rhs_lane(ln, y, G * d[st]);
    }
    double out = div_known(BO[0].num * k[BO[0].s], BO[0].den, 1.0 / BO[0].den);
#pragma unroll
    for (int j = 1; j < 8; ++j) out = out + div_known(BO[j].num * k[BO[j].s], BO[j].den, 1.0 / BO[j].den);
    s = s + dt * out;
    G = G * d[11];
}

// HVC(I) part of one interval, of interneurons x = 0..B n_i - 1, four to a warp (interval_i_body).
__global__ void __launch_bounds__(kBlock, 1) k_interval_i_lanes(NetDev<double> n, BatchDev<double> bt, int q, int s0,
                                                                int s1, IStep<double> ic)
{
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long all = (long long)bt.B * n.n_i;
    const int c = (int)(t % kLanes);
    const bool valid = t / kLanes < all;
    const size_t x = (size_t)min(t / kLanes, all - 1);
    const int b = (int)(x / n.n_i), i = (int)(x - (size_t)b * n.n_i);
    const bool inh = c == 6;
    const int at = min(c, 4);
    double s = c <= 4 ? bt.iv[at][x] : 1.0, G = bt.iv[inh ? 6 : 5][x];
    if (q > 0) {
        const size_t slot = (size_t)((q - 1) % n.ring) * bt.B * n.n_i + x;
        const long long ae = bt.ring_i_exc[slot];
        __syncwarp();
        if (ae) {
            if (valid && c == 0) bt.ring_i_exc[slot] = 0;
            if (!inh) G = G + (double)ae * kFixInv;
        }
    }
    double ne = bt.i_noise[2 * x], ni = bt.i_noise[2 * x + 1];
    int se = bt.i_noise_step[2 * x], si = bt.i_noise_step[2 * x + 1];
    uint32_t word = bt.i_word[x];
    int flag = bt.i_flag[x];
    const StreamId sid = make_stream(n.seed, kNoiseIPoisson, n.net_id, (uint32_t)i, bt.trial[b]);
    const ILanes k = i_lanes(c);
    uint32_t fired = 0;
    for (int st = s0; st <= s1; ++st) {
        const int below = s < -25.0, above = s > -20.0;     // lane 0: V
        fired |= (uint32_t)(flag & below) << (st - s0);
        flag = flag ? 1 - below : above;
        // the events move every lane's place in the stream, and the conductance of their own
        if (st == se) {
            double g = G;
            se = i_noise_event(n.T, n.num_steps, st, ne, g, sid, word);
            if (!inh) G = g;
        }
        if (st == si) {
            double g = G;
            si = i_noise_event(n.T, n.num_steps, st, ni, g, sid, word);
            if (inh) G = g;
        }
        double d[12];
        const double* dec = n.i_decay + (size_t)24 * st + (inh ? 12 : 0);
#pragma unroll
        for (int j = 0; j < 12; ++j) d[j] = dec[j];
        i_dp8_lane(k, s, G, ic.dt, d);
    }
    __syncwarp();
    if (valid) {
        if (c <= 4) bt.iv[at][x] = s;
        if (c == 5 || inh) bt.iv[inh ? 6 : 5][x] = G;
    }
    fired = valid && c == 0 ? fired : 0u;
    if (valid && c == 0) {
        bt.i_noise[2 * x] = ne;
        bt.i_noise[2 * x + 1] = ni;
        bt.i_noise_step[2 * x] = se;
        bt.i_noise_step[2 * x + 1] = si;
        bt.i_word[x] = word;
        bt.i_flag[x] = flag;
        if (fired) {
            bt.i_nspk[x] += __popc(fired);
            if (bt.i_first[x] < 0) bt.i_first[x] = s0 + __ffs(fired) - 1;
            record_spikes(bt.spk_count, bt.spk_buf, bt.spk_cap, bt.error, b, i, kSpikeInter, fired, s0);
        }
    }
    i_scatter(n, bt, fired, i, b, s0);
}

}  // namespace ug
