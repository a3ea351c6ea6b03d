// Test trials of a small batch in one cooperative launch: every sync interval of
// trial_no_stdp_fixedSpread (NetworkGrowthSimulator.cpp:12747-13117) of every instance runs
// inside k_test_trial, a warp keeping its neurons in registers from the first interval to the
// last.
//
// A batch that does not fill the GPU is bound by the step chain of its neurons and, with a
// launch or two per interval, by what surrounds it: the launch, the graph's fork and join, the
// state's way through L2 and the refilling of the instruction caches cost as much as the
// steps (2000 HVC(RA) + 550 HVC(I), one trial: 13 of 20 us per interval).  Here an interval
// ends with an arrival on a counter of the instance, and begins with a wait for the arrivals
// it depends on: instances never wait for each other, an interneuron interval only for the
// HVC(RA) neurons' previous one, an HVC(RA) interval for both kinds'.  The interneurons' step
// is the longer one, so they run on without a pause and the HVC(RA) neurons' waits are hidden
// beside them.
//
// Every wait is bounded (ug_async.cuh): one that gives up sets kErrTimeout, every warp leaves
// at its next wait, and the host reports UG_ETIMEOUT.
#pragma once
#include "ug_async.cuh"
#include "ug_trial.cuh"

namespace ug {

constexpr int kUnitWarps = 4;    // warps (units) per block, one per SM scheduler
// Arrival counters of an instance, a 128-byte line each: HVC(RA), and HVC(I) apart for even and
// odd intervals.  An HVC(RA) warp waits for both kinds, so none is a whole interval ahead of
// another; an interneuron warp waits for the HVC(RA) warps only and can finish an interval
// before a slower one has finished the last, which one common count would take for it.
constexpr int kCtlWords = 96, kCtlInter = 32;

// The launch's part of the trial: intervals q0 .. q1 - 1 (Q: the steps after the last sync).
struct TestLoop {
    const int* sync_end;   // [Q] last step of each sync interval
    int Q, q0, q1;
    int ra_units, i_units; // warps per instance of the two kinds
    int ra_pad;            // HVC(RA) warps of all instances, rounded up to whole blocks
    unsigned* ctl;         // [B][kCtlWords] arrivals, zero at the trial's start
};

__device__ __forceinline__ unsigned* unit_ctl(const TestLoop& L, int b) { return L.ctl + (size_t)b * kCtlWords; }

// The interneurons' counter of interval q; it reaches (q / 2 + 1) times their warps.
__device__ __forceinline__ unsigned* inter_ctl(unsigned* ctl, int q) { return ctl + kCtlInter * (1 + (q & 1)); }

__device__ __forceinline__ unsigned load_acquire(const unsigned* p)
{
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// The warp's memory operations so far, then one arrival (a release, not a full fence: one
// 2000/550 trial 26.3 -> 25.3 ms).
__device__ __forceinline__ void unit_arrive(unsigned* count)
{
    __syncwarp();
    if ((threadIdx.x & 31) == 0)
        asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(count), "r"(1u) : "memory");
}

// Waits until *count >= want0 and *inter >= want1 (each lane of two polls one of them); false
// if the wait, or another warp's, gave up.
__device__ __forceinline__ bool unit_wait(const unsigned* count, unsigned want0, const unsigned* inter, unsigned want1,
                                          int* error)
{
    const int lane = threadIdx.x & 31;
    const unsigned want = lane == 0 ? want0 : lane == 1 ? want1 : 0u;
    const unsigned* p = lane == 1 ? inter : count;
    const bool ok = poll_bounded<false>(0xffffffffu, error, kErrTimeout, nullptr,
                                 [&] { return want == 0u || load_acquire(p) >= want; });
    __syncwarp();
    return ok;
}

// V: the lane type of the HVC(RA) warps (ug_ra_f32.cuh).
template <class V>
__global__ void __launch_bounds__(32 * kUnitWarps, Lanes<V>::n == 1 ? 1 : 4)
    k_test_trial(NetDev<float> n, BatchDev<float> bt, RAStep<float> rc, const __grid_constant__ IStep<float> ic,
                 TestLoop L)
{
    const int unit = (int)blockIdx.x * kUnitWarps + (int)(threadIdx.x >> 5), lane = (int)(threadIdx.x & 31);
    if (unit < L.ra_pad) {
        constexpr int N = Lanes<V>::n;
        const int b = unit / L.ra_units, t = (unit % L.ra_units) * 32 + lane;
        if (b >= bt.B) return;
        unsigned* ctl = unit_ctl(L, b);
        const int i0 = N * t;
        const bool any = i0 < n.n_ra;
        RAUnit<V, true> u;
        const int first = L.q0 == 0 ? 1 : L.sync_end[L.q0 - 1] + 1;
        u.load(n, bt, rc, any ? t : 0, b, first);   // a thread without a neuron steps neuron 0 and stores nothing
        if (!any)
#pragma unroll
            for (int k = 0; k < N; ++k) u.valid[k] = false;
        int s0 = first;
        for (int q = L.q0; q < L.q1; ++q) {
            if (q > L.q0 && !unit_wait(ctl, (unsigned)q * L.ra_units, inter_ctl(ctl, q - 1),
                                       (unsigned)((q - 1) / 2 + 1) * L.i_units, bt.error))
                return;
            if (q > 0) u.sync_kicks(n, bt, q - 1);
            if (q == L.Q) break;
            const int s1 = L.sync_end[q];
            uint32_t soma[N] = {}, dend[N] = {};
            u.template steps<false>(n, bt, rc, s0, s1, soma, dend);
#pragma unroll
            for (int k = 0; k < N; ++k) ra_scatter(n, bt, soma[k], i0 + k, b, s0);
            unit_arrive(ctl);
#pragma unroll
            for (int k = 0; k < N; ++k)
                if (soma[k] | dend[k]) ra_spike_stats(bt, u.at(n, k), i0 + k, b, s0, soma[k], dend[k]);
            s0 = s1 + 1;
        }
        u.store(n, bt);
    } else {
        const int w = unit - L.ra_pad;
        const int b = w / max(L.i_units, 1), i = (w % max(L.i_units, 1)) * 32 + lane;
        if (L.i_units == 0 || b >= bt.B) return;
        unsigned* ctl = unit_ctl(L, b);
        const bool any = i < n.n_i;
        IUnit u(n, bt, any ? i : 0, b, L.q0 > 0);
        int s0 = L.q0 == 0 ? 1 : L.sync_end[L.q0 - 1] + 1;
        for (int q = L.q0; q < L.q1; ++q) {
            if (q > L.q0 && !unit_wait(ctl, (unsigned)q * L.ra_units, ctl, 0u, bt.error)) return;
            if (q > 0 && any) u.sync_kicks(n, bt, q - 1);
            if (q == L.Q) break;
            const int s1 = L.sync_end[q];
            uint32_t fired = 0;
            u.template steps<false>(n, bt, ic, s0, s1, i, b, fired);
            if (!any) fired = 0;
            i_scatter(n, bt, fired, i, b, s0);
            unit_arrive(inter_ctl(ctl, q));
            u.spike_stats(bt, i, b, s0, fired);
            s0 = s1 + 1;
        }
        if (any) u.store(bt);
    }
}

}  // namespace ug
