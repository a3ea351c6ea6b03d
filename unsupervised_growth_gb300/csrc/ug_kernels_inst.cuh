// Shared body of the per-precision launcher translation units.
#pragma once
#include "ug_launch.h"
#ifdef UG_DOUBLE_UNIT
#include "ug_f64_lanes.cuh"
#endif

namespace ug {

#define UG_TIMED(lc, name, launch)                                      \
    do {                                                                \
        if ((lc).timer) {                                               \
            cudaError_t e_ = (lc).timer->begin(name, (lc).main);        \
            if (e_ != cudaSuccess) return e_;                           \
        }                                                               \
        launch;                                                         \
        if ((lc).timer) {                                               \
            cudaError_t e_ = (lc).timer->end((lc).main);                \
            if (e_ != cudaSuccess) return e_;                           \
        }                                                               \
    } while (0)

// Single build only: pre-draw the interneurons' noise events of the trial.
inline void launch_noise_events(const NetDev<double>&, const BatchDev<double>&, const LaunchCtx&) {}
inline void launch_noise_events(const NetDev<float>& n, const BatchDev<float>& b, const LaunchCtx& lc)
{
    if (n.n_i == 0) return;
    if (lc.timer) lc.timer->begin("k_noise_events", lc.main);
    constexpr int kPer = kNoiseThreads / 32;
    k_noise_gaps<float><<<dim3((n.n_i + kPer - 1) / kPer, b.B), kNoiseThreads, 0, lc.main>>>(n, b, 0, b.ev_cap);
    k_noise_events<float><<<dim3((n.n_i + kNoiseWalk - 1) / kNoiseWalk, b.B), kNoiseWalk, 0, lc.main>>>(
        n, b, n.num_steps - 1, b.ev_cap, false);
    if (lc.timer) lc.timer->end(lc.main);
}

#ifdef UG_DOUBLE_UNIT
// Threads per block of the double-precision integrators: one warp per block for small
// batches, so that a single trial spreads over as many SMs as it has warps (GB300's FP64
// pipe is narrow, and a trial of 2000 neurons is only 63 + 18 warps).
inline int dp_block(int B) { return B < 16 ? 32 : kBlock; }

// Batches up to these many neurons go to the kernels with eight lanes per neuron.  They make
// eight times the warps with a fifth of the operations each, so they are the faster ones until
// the FP64 pipes of all sub-partitions are busy.  Measured, one interval of both kernels:
// 602 HVC(RA) / 150 HVC(I) 2.40 -> 0.41 ms, 4800 / 1200 2.41 -> 0.72, 9600 / 2400 3.57 -> 1.29
// (general HVC(RA) beside lanes for HVC(I): 0.88, 0.88, 1.40); 16 000 / 4000: lanes for both
// 2.19, general HVC(RA) 1.67; 40 000 / 10 000 6.21 -> 5.65 with lanes for HVC(I); 16 000 / 16 000
// 3.62 general, 4.10 with lanes for HVC(I).  Blocks of one warp spread over the SMs: 4 warps of
// one SM take 76 cycles an operation instead of 64 (602 / 150: blocks of 128 threads 0.44 ms).
// Recorded neurons (traces, inhibition tracking) stay with the general kernels.
constexpr int kLanesMaxRA = 10000, kLanesMaxI = 12000, kLanesBlock = 32;
inline bool dp_lanes(long long neurons, int most) { return neurons <= most; }
inline unsigned dp_lanes_grid(long long neurons) { return (unsigned)((neurons * kLanes + kLanesBlock - 1) / kLanesBlock); }

inline void launch_i(const NetDev<double>& n, const BatchDev<double>& b, int q, int s0, int s1,
                     const IStep<double>& ic, cudaStream_t st, const LaunchCtx& lc)
{
    if (lc.timer) lc.timer->begin("k_interval_i", lc.main);
    if (!b.trace_i && dp_lanes((long long)b.B * n.n_i, kLanesMaxI)) {
        k_interval_i_lanes<<<dp_lanes_grid((long long)b.B * n.n_i), kLanesBlock, 0, st>>>(n, b, q, s0, s1, ic);
        if (lc.timer) lc.timer->end(lc.main);
        return;
    }
    const int t = dp_block(b.B);
    const dim3 g((n.n_i + t - 1) / t, b.B);
    if (b.trace_i)
        k_interval_i<double, true><<<g, t, 0, st>>>(n, b, q, s0, s1, ic);
    else
        k_interval_i<double><<<g, t, 0, st>>>(n, b, q, s0, s1, ic);
    if (lc.timer) lc.timer->end(lc.main);
}
#endif

inline void launch_i(const NetDev<float>& n, const BatchDev<float>& b, int q, int s0, int s1, const IStep<float>& ic,
                     cudaStream_t st, const LaunchCtx& lc)
{
    if (lc.timer) lc.timer->begin("k_interval_i", lc.main);
    const dim3 g((unsigned)(((long long)b.B * n.n_i + kBlock - 1) / kBlock));   // flat over (instance, interneuron)
    if (b.trace_i)
        k_interval_i_x<float, true><<<g, kBlock, 0, st>>>(n, b, q, s0, s1, ic);
    else
        k_interval_i_x<float><<<g, kBlock, 0, st>>>(n, b, q, s0, s1, ic);
    if (lc.timer) lc.timer->end(lc.main);
}

template <class R>
cudaError_t launch_trial_init(const NetDev<R>& n, const BatchDev<R>& b, const LaunchCtx& lc)
{
    const dim3 grid((n.n_ra + kBlock - 1) / kBlock + (n.n_i + kBlock - 1) / kBlock, b.B);
    UG_TIMED(lc, "k_trial_init", (k_trial_init<R><<<grid, kBlock, 0, lc.main>>>(n, b)));
    launch_noise_events(n, b, lc);
    return cudaGetLastError();
}

template <class R>
cudaError_t launch_state_init(const NetDev<R>& n, const BatchDev<R>& b, cudaStream_t st)
{
    const dim3 grid((n.n_ra + kBlock - 1) / kBlock + (n.n_i + kBlock - 1) / kBlock, b.B);
    k_trial_init<R><<<grid, kBlock, 0, st>>>(n, b);
    return cudaGetLastError();
}

template <class R>
cudaError_t launch_noise_segment(const NetDev<R>& n, const BatchDev<R>& b, int end, int k0, int k1, cudaStream_t st)
{
    if constexpr (sizeof(R) == 4) {
        if (n.n_i == 0) return cudaSuccess;
        constexpr int kPer = kNoiseThreads / 32;
        k_noise_gaps<float><<<dim3((n.n_i + kPer - 1) / kPer, b.B), kNoiseThreads, 0, st>>>(n, b, k0, k1);
        k_noise_events<float><<<dim3((n.n_i + kNoiseWalk - 1) / kNoiseWalk, b.B), kNoiseWalk, 0, st>>>(n, b, end, k1,
                                                                                                     k0 > 0);
        return cudaGetLastError();
    }
    return cudaErrorNotSupported;
}

// Form of a batch of test trials: one launch when all its warps can be resident at once and
// they make no more rounds of the GPU's schedulers (a warp each) than the per-interval
// launches, which pack the neurons of all trials without a partly empty last warp per trial.
// Measured, ms a batch, one launch against per-interval launches: 2000/550, 12 trials (600
// warps) 33.2 / 36.2, 24 (1200) 46.5 / 52.4, 48 (2400) 75.9 / 82.4; 777/194, 24 (480 warps,
// one round each) 27.7 / 32.7, 48 (960, two each) 41.0 / 46.7, but 32 (640 warps, two rounds
// against one) 42.8 / 32.9.  One HVC(RA) neuron per thread while each warp has a scheduler to
// itself (the step chain bounds it: 765 cycles a step against 1310 with two; 8 trials of
// 777/194 24.5 ms against 27.7 for 24 with two), two from there on.
constexpr int kTestMaxRounds = 4;   // 4 blocks of 4 warps per SM are resident
template <class R>
cudaError_t test_trial_plan(int n_ra, int n_i, int B, TestPlan* plan)
{
    *plan = TestPlan();
    if constexpr (sizeof(R) == 4) {
        int dev = 0, sms = 0, coop = 0;
        cudaError_t e = cudaGetDevice(&dev);
        if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (e == cudaSuccess) e = cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
        if (e != cudaSuccess || !coop) return e;
        for (int lanes = 1; lanes <= 2; ++lanes) {
            TestPlan p;
            p.ra_units = (n_ra + 32 * lanes - 1) / (32 * lanes);
            p.i_units = (n_i + 31) / 32;
            const long long ra = (long long)B * p.ra_units, in = (long long)B * p.i_units;
            const long long pad = (ra + kUnitWarps - 1) / kUnitWarps * kUnitWarps;
            const long long blocks = (pad + in + kUnitWarps - 1) / kUnitWarps;
            const long long flat = ((long long)B * ((n_ra + 1) / 2) + kBlock - 1) / kBlock +
                                   ((long long)B * n_i + kBlock - 1) / kBlock;
            const long long rounds = (blocks + sms - 1) / sms;   // a block has a warp per scheduler
            if (rounds > (lanes == 1 ? 1 : std::min<long long>(kTestMaxRounds, (flat + sms - 1) / sms))) continue;
            int per_sm = 0;
            e = lanes == 1
                    ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_test_trial<float>, 32 * kUnitWarps, 0)
                    : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_test_trial<f2>, 32 * kUnitWarps, 0);
            if (e != cudaSuccess) return e;
            if (blocks > (long long)per_sm * sms) continue;
            p.lanes = lanes;
            p.blocks = (int)blocks;
            p.ra_pad = (int)pad;
            *plan = p;
            return cudaSuccess;
        }
    }
    return cudaSuccess;
}

template <class R>
cudaError_t launch_test_trial(const NetDev<R>& n, const BatchDev<R>& b, const RAStep<R>& rc, const IStep<R>& ic,
                              const TestPlan& plan, const int* sync_end, int Q, int q0, int q1, unsigned* ctl,
                              cudaStream_t st)
{
    if constexpr (sizeof(R) == 4) {
        TestLoop L;
        L.sync_end = sync_end;
        L.Q = Q; L.q0 = q0; L.q1 = q1;
        L.ra_units = plan.ra_units; L.i_units = plan.i_units; L.ra_pad = plan.ra_pad;
        L.ctl = ctl;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)plan.blocks);
        cfg.blockDim = dim3(32 * kUnitWarps);
        cfg.stream = st;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeCooperative;   // every block resident at once, or the launch fails
        at[0].val.cooperative = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        return plan.lanes == 1 ? cudaLaunchKernelEx(&cfg, k_test_trial<float>, n, b, rc, ic, L)
                               : cudaLaunchKernelEx(&cfg, k_test_trial<f2>, n, b, rc, ic, L);
    }
    return cudaErrorNotSupported;
}

// HVC(RA) interval kernel: the double build steps one neuron per thread, the
// single build two neurons per thread with packed f32x2 arithmetic.
#ifdef UG_DOUBLE_UNIT
inline void launch_ra(const NetDev<double>& n, const BatchDev<double>& b, int q, int s0, int s1,
                      const RAStep<double>& rc, const LaunchCtx& lc)
{
    const int t = dp_block(b.B);
    const dim3 g((n.n_ra + t - 1) / t, b.B);
    if (lc.timer) lc.timer->begin("k_interval_ra", lc.main);
    if (!b.ginh_slot && !b.trace_ra && dp_lanes((long long)b.B * n.n_ra, kLanesMaxRA))
        k_interval_ra_lanes<<<dp_lanes_grid((long long)b.B * n.n_ra), kLanesBlock, 0, lc.main>>>(n, b, q, s0, s1, rc);
    else if (b.ginh_slot || b.trace_ra)
        k_interval_ra<double, true><<<g, t, 0, lc.main>>>(n, b, q, s0, s1, rc);
    else
        k_interval_ra<double><<<g, t, 0, lc.main>>>(n, b, q, s0, s1, rc);
    if (lc.timer) lc.timer->end(lc.main);
}
#endif

inline void launch_ra(const NetDev<float>& n, const BatchDev<float>& b, int q, int s0, int s1, const RAStep<float>& rc,
                      const LaunchCtx& lc)
{
    const dim3 g((unsigned)(((long long)b.B * ((n.n_ra + 1) / 2) + kBlock - 1) / kBlock));   // flat over (instance, pair)
    if (lc.timer) lc.timer->begin("k_interval_ra", lc.main);
    if (b.ginh_slot || b.trace_ra)
        k_interval_ra_x2<float, true><<<g, kBlock, 0, lc.main>>>(n, b, q, s0, s1, rc);
    else
        k_interval_ra_x2<float><<<g, kBlock, 0, lc.main>>>(n, b, q, s0, s1, rc);
    if (lc.timer) lc.timer->end(lc.main);
}

// Both single-build integrators of one interval in one launch (fused_interval).
inline void launch_fused(const NetDev<double>&, const BatchDev<double>&, int, int, int, const RAStep<double>&,
                         const IStep<double>&, const LaunchCtx&)
{
}
inline void launch_fused(const NetDev<float>& n, const BatchDev<float>& b, int q, int s0, int s1,
                         const RAStep<float>& rc, const IStep<float>& ic, const LaunchCtx& lc)
{
    const unsigned nb_ra = (unsigned)(((long long)b.B * ((n.n_ra + 1) / 2) + kBlock - 1) / kBlock);
    const unsigned nb_i = (unsigned)(((long long)b.B * n.n_i + kBlock - 1) / kBlock);
    if (lc.timer) lc.timer->begin("k_interval_x", lc.main);
    k_interval_x<float><<<nb_ra + nb_i, kBlock, 0, lc.main>>>(n, b, q, s0, s1, rc, ic, nb_ra);
    if (lc.timer) lc.timer->end(lc.main);
}

template <class R>
cudaError_t launch_interval(const NetDev<R>& n, const BatchDev<R>& b, int q, int s0, int s1, const RAStep<R>& rc,
                            const IStep<R>& ic, const LaunchCtx& lc)
{
    if (fused_interval<R>(n, b, lc)) {
        launch_fused(n, b, q, s0, s1, rc, ic, lc);
        return cudaGetLastError();
    }
    // Overlap the two kernels only when a batch is too small to fill the GPU on
    // its own; large batches run them back to back so each SM executes one
    // kernel's code at a time (the integrators do not fit the instruction cache together).
    const bool fork = !lc.timer && lc.side && lc.side != lc.main && n.n_i > 0 && b.B < 16;
    cudaStream_t si = fork ? lc.side : lc.main;
    if (fork) {
        cudaError_t e = cudaEventRecord(lc.fork, lc.main);
        if (e == cudaSuccess) e = cudaStreamWaitEvent(lc.side, lc.fork, 0);
        if (e != cudaSuccess) return e;
    }
    launch_ra(n, b, q, s0, s1, rc, lc);
    if (n.n_i > 0) launch_i(n, b, q, s0, s1, ic, si, lc);
    if (fork) {
        cudaError_t e = cudaEventRecord(lc.join, lc.side);
        if (e == cudaSuccess) e = cudaStreamWaitEvent(lc.main, lc.join, 0);
        if (e != cudaSuccess) return e;
    }
    return cudaGetLastError();
}

template <class R>
cudaError_t launch_growth_reset(const GrowthDev& g, const LaunchCtx& lc)
{
    UG_TIMED(lc, "k_growth_reset", (k_growth_reset<R><<<1024, 256, 0, lc.main>>>(g)));
    return cudaGetLastError();
}

// The tail of an interval goes on lc.tail when there is one (and no timer).
inline cudaError_t tail_fork(const LaunchCtx& lc, cudaStream_t* ts)
{
    *ts = lc.main;
    if (lc.timer || !lc.tail || lc.tail == lc.main) return cudaSuccess;
    cudaError_t e = cudaEventRecord(lc.tail_fork, lc.main);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(lc.tail, lc.tail_fork, 0);
    *ts = lc.tail;
    return e;
}

// Deliveries of the interval's RA spikes to RA targets (after the previous
// interval's tail), then the sync's post events, LTP and axon remodeling as
// this interval's tail.
template <class R>
cudaError_t launch_growth_sync(const GrowthDev& g, const NetDev<R>& n, const BatchDev<R>& b, int q, int s0, int s1,
                               const LaunchCtx& lc, bool& tail_open)
{
    cudaError_t e = launch_tail_join(lc, tail_open);
    if (e != cudaSuccess) return e;
    const dim3 rows((g.n + kBlock - 1) / kBlock, g.B);
    const dim3 wrows((g.n + kRowWarps - 1) / kRowWarps, g.B);
    UG_TIMED(lc, "k_growth_rows", (k_growth_rows<R><<<wrows, 32 * kRowWarps, kRowWarps * sizeof(RowShared), lc.main>>>(g, n, b, q, s0, s1)));
    cudaStream_t ts;
    e = tail_fork(lc, &ts);
    if (e != cudaSuccess) return e;
    UG_TIMED(lc, "k_growth_newpost", (k_growth_newpost<R><<<g.B, 1024, 0, ts>>>(g, n, b, q, s0, s1)));
    UG_TIMED(lc, "k_growth_ltp", (k_growth_ltp<R><<<rows, kBlock, 0, ts>>>(g, n, s1)));
    if (ts != lc.main) {
        e = cudaEventRecord(lc.tail_join, ts);
        tail_open = true;
    }
    return e == cudaSuccess ? cudaGetLastError() : e;
}

template <class R>
cudaError_t launch_growth_epilogue(const GrowthDev& g, const LaunchCtx& lc)
{
    if (g.epi_blocks > 0) {   // rows staged by the bulk copy engine
        UG_TIMED(lc, "k_growth_epilogue", (k_growth_epilogue_bulk<R><<<g.epi_blocks, kEpiWarps * 32, kEpiSmem, lc.main>>>(g)));
        return cudaGetLastError();
    }
    const dim3 rows((g.n + kBlock / 32 - 1) / (kBlock / 32), g.B);   // a warp per row
    UG_TIMED(lc, "k_growth_epilogue", (k_growth_epilogue<R><<<rows, kBlock, 0, lc.main>>>(g)));
    return cudaGetLastError();
}

// Dynamic shared memory of k_growth_trial: one row buffer per warp.
constexpr size_t kTrialSmem = (size_t)kTrialWarps * sizeof(RowShared);

inline cudaError_t units_attributes(const void* kernel)
{
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTrialSmem);
}

// Whether an SM takes a block of `kernel`, a form of k_growth_units (its shared memory is most
// of an SM's); a device that refuses the size is no error, the per-interval launches run.
template <class K>
bool units_resident(K kernel)
{
    int per_sm = 0;
    cudaError_t e = units_attributes((const void*)kernel);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kTrialThreads, kTrialSmem);
    if (e != cudaSuccess) cudaGetLastError();
    return e == cudaSuccess && per_sm > 0;
}

template <class R>
cudaError_t growth_trial_plan(int n_ra, int n_i, int req_ra, int req_i, GrowthPlan* plan)
{
    *plan = GrowthPlan();
    int dev = 0, sms = 0, per_sm = 0, coop = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
    int ra_w = 0, i_w = 0;
    if (e != cudaSuccess || !coop || !trial_widths(req_ra, req_i, &ra_w, &i_w)) return e;
    if constexpr (sizeof(R) == 4) {
        const bool resident[2] = {units_resident(k_growth_units<float, false>) && units_resident(k_growth_units<float, true>),
                                  units_resident(k_growth_units<f2, false>) && units_resident(k_growth_units<f2, true>)};
        plan->units = units_shape(n_ra, n_i, req_ra, req_i, sms, resident);
        plan->blocks = plan->units.blocks();
        return cudaSuccess;
    } else {
        e = units_attributes((const void*)k_growth_trial<R>);
        if (e == cudaSuccess)
            e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_growth_trial<R>, kTrialThreads, kTrialSmem);
        if (e != cudaSuccess) return e;
        int nb_sync = 0;
        plan->trial.ra_w = ra_w;
        plan->trial.i_w = i_w;
        trial_roles(n_ra, n_i, ra_w, i_w, &plan->trial.nb_ra, &plan->trial.nb_i, &nb_sync);
        const long long total = (long long)plan->trial.nb_ra + plan->trial.nb_i + nb_sync;
        if (per_sm > 0 && total <= (long long)per_sm * sms) plan->blocks = (int)total;
        return cudaSuccess;
    }
}

template <class R>
cudaError_t launch_growth_trial(const GrowthDev& g, const NetDev<R>& n, BatchDev<R> b, const RAStep<R>& rc,
                                const IStep<R>& ic, const GrowthPlan& plan, const int* sync_end, int Q,
                                unsigned long long* ctl, int2* act_rows, cudaStream_t st)
{
    cudaError_t e = cudaMemsetAsync(ctl, 0, growth_ctl_words(Q) * sizeof(unsigned long long), st);
    if (e != cudaSuccess) return e;
    b.member = 0;
    b.live_streams = g.st_num;
    b.heavy = 0;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)plan.blocks);
    cfg.blockDim = dim3(kTrialThreads);
    cfg.dynamicSmemBytes = kTrialSmem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;   // every block resident at once, or the launch fails
    at[0].val.cooperative = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    if constexpr (sizeof(R) == 4) {
        UnitsLoop L;
        static_cast<UnitsShape&>(L) = plan.units;
        L.sync_end = sync_end;
        L.Q = Q;
        L.ctl = ctl;
        L.rows = act_rows;
        L.rows_cap = 2 * n.n_ra;
        b.soma_bits = nullptr;   // the spike bits travel with the queued rows
        GrowthDev gb = g;
        gb.beat = ctl + kCtlBeat;
        if (b.trace_ra || b.trace_i || b.ginh_slot)
            return L.lanes == 1 ? cudaLaunchKernelEx(&cfg, k_growth_units<float, true>, gb, n, b, rc, ic, L)
                                   : cudaLaunchKernelEx(&cfg, k_growth_units<f2, true>, gb, n, b, rc, ic, L);
        return L.lanes == 1 ? cudaLaunchKernelEx(&cfg, k_growth_units<float, false>, gb, n, b, rc, ic, L)
                               : cudaLaunchKernelEx(&cfg, k_growth_units<f2, false>, gb, n, b, rc, ic, L);
    } else {
        TrialLoop L = plan.trial;
        L.sync_end = sync_end;
        L.Q = Q;
        L.bar = reinterpret_cast<unsigned*>(ctl);
        L.posted = L.bar + 1;
        b.act_rows = act_rows;
        b.act_cnt = reinterpret_cast<int*>(ctl) + 4;
        b.act_cap = n.n_ra;
        return cudaLaunchKernelEx(&cfg, k_growth_trial<R>, g, n, b, rc, ic, L);
    }
}

// Grid of the bulk-copy epilogue for B networks of n neurons (0: rows not 16-byte aligned
// in every array, so the warp epilogue runs), after allowing its shared memory.
template <class R>
cudaError_t epilogue_bulk_grid(int n, int B, int* blocks)
{
    *blocks = 0;
    if (n % 16 != 0 || n <= 0) return cudaSuccess;
    cudaError_t e = cudaFuncSetAttribute(k_growth_epilogue_bulk<R>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)kEpiSmem);
    if (e != cudaSuccess) return e;
    int dev = 0, sms = 0, per_sm = 0;
    e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess)
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_growth_epilogue_bulk<R>, kEpiWarps * 32, kEpiSmem);
    if (e != cudaSuccess) return e;
    const long long rows = (long long)n * B;
    const long long want = (rows + kEpiWarps - 1) / kEpiWarps;
    *blocks = (int)std::min<long long>(want, (long long)std::max(per_sm, 1) * sms);
    return cudaSuccess;
}

template <class R>
cudaError_t launch_growth_remove(const GrowthDev& g, const int* rep, int nrep, cudaStream_t st)
{
    const dim3 rows((g.n + kBlock - 1) / kBlock, g.B);
    k_growth_remove<R><<<rows, kBlock, 0, st>>>(g, rep, nrep);
    return cudaGetLastError();
}

template <class R>
cudaError_t launch_check_bad(const NetDev<R>& n, const BatchDev<R>& b, int* bad, cudaStream_t st)
{
    const size_t total = (size_t)b.B * n.n_ra;
    k_check_bad<R><<<(unsigned)((total + 255) / 256), 256, 0, st>>>(n, b, bad);
    return cudaGetLastError();
}

template <class R>
cudaError_t launch_growth_head(const TailDev<R>& t, int* bad, cudaStream_t st)
{
    k_growth_head<R><<<1, 1, 0, st>>>(t, bad);
    return cudaGetLastError();
}

template <class R>
cudaError_t launch_growth_tail(const TailDev<R>& t, cudaStream_t st)
{
    k_growth_tail<R><<<1, kTailThreads, 0, st>>>(t);
    return cudaGetLastError();
}

template <class K>
static int occupancy(K kernel, int threads, size_t smem)
{
    int nb = 0, dev = 0, sms = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kernel, threads, smem) != cudaSuccess) return 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
    return nb * sms;
}

template <class R>
cudaError_t group_grids(GroupDev& d, int ra_blocks_per_sm, int i_blocks_per_sm)
{
    int dev = 0, sms = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    d.grid[kListInit] = occupancy(kl_trial_init<R>, kBlock, 0);
    d.grid[kListGaps] = occupancy(kl_noise_gaps<R>, kNoiseThreads, 0);
    d.grid[kListNoise] = occupancy(kl_noise_events<R>, kNoiseWalk, 0);
    d.grid[kListRA] = occupancy(kl_interval_ra<R>, kBlock, 0);
    d.grid[kListI] = occupancy(kl_interval_i<R>, kBlock, 0);
    if (ra_blocks_per_sm > 0) d.grid[kListRA] = std::min(d.grid[kListRA], ra_blocks_per_sm * sms);
    if (i_blocks_per_sm > 0) d.grid[kListI] = std::min(d.grid[kListI], i_blocks_per_sm * sms);
    d.grid[kListReset] = occupancy(kl_growth_reset<R>, 256, 0);
    d.grid[kListNewpost] = occupancy(kl_growth_newpost<R>, 1024, 0);
    d.grid[kListLtp] = occupancy(kl_growth_ltp<R>, kBlock, 0);
    d.grid[kListCheck] = occupancy(kl_check_bad<R>, 256, 0);
    d.grid[kNumLists] = occupancy(kl_growth_rows<R>, 32 * kRowWarps, kRowWarps * sizeof(RowShared));
    // the heavy-row kernel's buffers exceed the default 48 KB of dynamic shared memory
    e = cudaFuncSetAttribute(kl_growth_rows_heavy<R>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)(sizeof(RowShared) + sizeof(HeavyShared)));
    if (e != cudaSuccess) return e;
    d.grid[kNumLists + 1] = occupancy(kl_growth_rows_heavy<R>, 32 * kHeavyWarps, sizeof(RowShared) + sizeof(HeavyShared));
    for (int k = 0; k <= kNumLists + 1; ++k)
        if (d.grid[k] <= 0) return cudaErrorInvalidConfiguration;
    return cudaSuccess;
}

template <class R>
cudaError_t launch_group_trial(const GroupDev& d, const std::vector<int>& sync_steps, int num_steps, bool growth,
                               const LaunchCtx& lc, int64_t* launches)
{
    typedef GroupMember<R> M;
    const M* mem = static_cast<const M*>(d.members);
    const int* c = d.count;
    int64_t cnt = 0;
    cudaError_t e = cudaSuccess;
    if (growth) {
        e = cudaMemsetAsync(d.act_cnt, 0, 4 * sizeof(int), lc.main);
        if (e != cudaSuccess) return e;
    }
    UG_TIMED(lc, "k_trial_init", (kl_trial_init<R><<<d.grid[kListInit], kBlock, 0, lc.main>>>(mem, d.items[kListInit], c + kListInit)));
    ++cnt;
    if constexpr (sizeof(R) == 4) {
        UG_TIMED(lc, "k_noise_events", (kl_noise_gaps<R><<<d.grid[kListGaps], kNoiseThreads, 0, lc.main>>>(mem, d.items[kListGaps], c + kListGaps)));
        UG_TIMED(lc, "k_noise_events", (kl_noise_events<R><<<d.grid[kListNoise], kNoiseWalk, 0, lc.main>>>(mem, d.items[kListNoise], c + kListNoise)));
        cnt += 2;
    }
    if (growth) {
        UG_TIMED(lc, "k_growth_reset", (kl_growth_reset<R><<<d.grid[kListReset], 256, 0, lc.main>>>(mem, d.items[kListReset], c + kListReset)));
        ++cnt;
    }
    const bool fork = d.fork && !lc.timer && lc.side && lc.side != lc.main;
    bool tail_open = false;
    const int Q = (int)sync_steps.size();
    for (int q = 0; q <= Q; ++q) {
        const int s0 = q == 0 ? 1 : (q < Q ? sync_steps[q - 1] + 1 : num_steps);
        const int s1 = q < Q ? sync_steps[q] : num_steps - 1;
        if (fork) {
            e = cudaEventRecord(lc.fork, lc.main);
            if (e == cudaSuccess) e = cudaStreamWaitEvent(lc.side, lc.fork, 0);
            if (e != cudaSuccess) return e;
        }
        if (d.track)
            UG_TIMED(lc, "k_interval_ra", (kl_interval_ra<R, true><<<d.grid[kListRA], kBlock, 0, lc.main>>>(mem, d.items[kListRA], c + kListRA, growth ? d.act_cnt : nullptr, q, s0, s1)));
        else
            UG_TIMED(lc, "k_interval_ra", (kl_interval_ra<R><<<d.grid[kListRA], kBlock, 0, lc.main>>>(mem, d.items[kListRA], c + kListRA, growth ? d.act_cnt : nullptr, q, s0, s1)));
        if (lc.timer) lc.timer->begin("k_interval_i", lc.main);
        kl_interval_i<R><<<d.grid[kListI], kBlock, 0, fork ? lc.side : lc.main>>>(mem, d.items[kListI], c + kListI, q, s0, s1);
        if (lc.timer) lc.timer->end(lc.main);
        cnt += 2;
        if (fork) {
            e = cudaEventRecord(lc.join, lc.side);
            if (e == cudaSuccess) e = cudaStreamWaitEvent(lc.main, lc.join, 0);
            if (e != cudaSuccess) return e;
        }
        if (growth && q < Q) {
            e = launch_tail_join(lc, tail_open);
            if (e != cudaSuccess) return e;
            // heavy rows (a block each) beside the warp-path rows: different rows, disjoint state
            const bool rfork = !lc.timer && lc.side && lc.side != lc.main;
            if (rfork) {
                e = cudaEventRecord(lc.fork, lc.main);
                if (e == cudaSuccess) e = cudaStreamWaitEvent(lc.side, lc.fork, 0);
                if (e != cudaSuccess) return e;
            }
            UG_TIMED(lc, "k_growth_rows_heavy", (kl_growth_rows_heavy<R><<<d.grid[kNumLists + 1], 32 * kHeavyWarps, sizeof(RowShared) + sizeof(HeavyShared), rfork ? lc.side : lc.main>>>(mem, d.act_rows, d.act_cnt, d.act_cap, d.T, q, s0, s1)));
            UG_TIMED(lc, "k_growth_rows", (kl_growth_rows<R><<<d.grid[kNumLists], 32 * kRowWarps, kRowWarps * sizeof(RowShared), lc.main>>>(mem, d.act_rows, d.act_cnt, d.act_cap, d.T, q, s0, s1)));
            if (rfork) {
                e = cudaEventRecord(lc.join, lc.side);
                if (e == cudaSuccess) e = cudaStreamWaitEvent(lc.main, lc.join, 0);
                if (e != cudaSuccess) return e;
            }
            cudaStream_t ts;
            e = tail_fork(lc, &ts);
            if (e != cudaSuccess) return e;
            UG_TIMED(lc, "k_growth_newpost", (kl_growth_newpost<R><<<d.grid[kListNewpost], 1024, 0, ts>>>(mem, d.items[kListNewpost], c + kListNewpost, q, s0, s1)));
            UG_TIMED(lc, "k_growth_ltp", (kl_growth_ltp<R><<<d.grid[kListLtp], kBlock, 0, ts>>>(mem, d.items[kListLtp], c + kListLtp, s1)));
            if (ts != lc.main) {
                e = cudaEventRecord(lc.tail_join, ts);
                if (e != cudaSuccess) return e;
                tail_open = true;
            }
            cnt += 4;
        }
    }
    e = launch_tail_join(lc, tail_open);
    if (e != cudaSuccess) return e;
    if (growth) {
        UG_TIMED(lc, "k_growth_epilogue", (kl_growth_epilogue<R><<<d.grid[kListLtp], kBlock, 0, lc.main>>>(mem, d.items[kListLtp], c + kListLtp)));
        ++cnt;
    }
    UG_TIMED(lc, "k_check_bad", (kl_check_bad<R><<<d.grid[kListCheck], 256, 0, lc.main>>>(mem, d.items[kListCheck], c + kListCheck, d.bad)));
    ++cnt;
    if (launches) *launches += cnt;
    return cudaGetLastError();
}

}  // namespace ug
