// One growth trial of one network in one cooperative launch, single build: every sync
// interval of trial_1stSoma_pre_1stSoma_post_delays_fixedSpread
// (NetworkGrowthSimulator.cpp:8923-9564) runs inside k_growth_units.  Blocks take one of four
// roles, and a role waits for exactly what it reads, on arrival counters, instead of for the
// whole grid:
//   HVC(RA) warps  integrate interval q with their neurons in registers, scatter the RA->I
//                  kicks and queue the rows that spiked or have streams open;
//                  before: sync q - 1's kicks, i.e. every warp's interval q - 1 and the
//                  deliveries of its rows;
//   HVC(I) warps   integrate interval q and scatter the I->RA kicks;
//                  before: the HVC(RA) warps' interval q - 1;
//   row blocks     replay the deliveries of q's queued rows (g_row, a warp per row);
//                  before: the HVC(RA) warps' interval q, and the closing of sync q - 1;
//   sync blocks    close sync q: its new post-synaptic events (the first sync block, from the
//                  queued rows that spiked), then LTP / LTD and axon remodeling of every row;
//                  before: the deliveries of q.
// An interval is the HVC(RA) steps and then the slowest of the deliveries (2000 / 550: 40 900
// cycles, of which an HVC(RA) warp steps 9700 and waits 28 300), with the interneurons' steps
// (19 400) and the sync beside it; in small networks (300 / 100: 24 300) the interneurons' steps.
// Rows have blocks of their own, each on an SM of its own, because a row is a chain of
// latencies (11 200 cycles on average): on the integrators' SMs its double-precision
// operations queue up with theirs, and the instruction caches are refilled between integration
// and delivery.  The order of every operation on a row, a pair or a neuron is the per-interval
// path's, so both give the same bits.
//
// Every wait is bounded (ug_async.cuh): one that gives up sets kErrTimeout, every block leaves
// at its next wait, and the host reports UG_ETIMEOUT.  An interval's deliveries can take a
// second and more (18 000 HVC(RA), 200 training neurons, fast synapses), so a wait gives up
// when the interval's work has not advanced for a second: a warp that takes up a further row
// or has delivered an event that changed its row, and a sync block that takes up further rows,
// say so.
#pragma once
#include "ug_growth_trial.cuh"
#include "ug_test_trial.cuh"

namespace ug {

// Counters of the launch, zero at the launch: words of the launch, each in a 128-byte line of
// its own, and words of every interval, in an array per kind.  A role that no other waits for
// may be any number of intervals behind the HVC(RA) warps: the first sync block, while they
// integrate intervals without rows; a row block that has had no row for some time.  An
// interval's words never change once it is complete, so such a role reads in them what the
// others read, and takes no later interval's arrivals or rows for those of its own.
enum GrowthCtl {
    kCtlPos = 0,        // queue positions handed out
    kCtlPosted = 16,    // intervals whose post events are in place << 32 | those that had any;
                        // the word after it: the last of those that had any
    kCtlLtp = 32,       // sync block arrivals, one each per interval that had post events
    kCtlBeat = 48,      // advances while an interval's rows or LTP take long (poll_bounded)
    kCtlIntervals = 64  // the intervals' words: kCtlKinds arrays of ctl_stride(Q)
};
enum GrowthCtlKind {
    kCtlRA,             // HVC(RA) arrivals << 32 | rows queued
    kCtlI,              // HVC(I) arrivals
    kCtlDone,           // rows delivered
    kCtlKinds
};
// An array's words: 16 columns of whole 128-byte lines, consecutive intervals in different
// columns, so that one interval's arrivals do not meet the polls of the one before.
__host__ __device__ constexpr int ctl_column(int Q) { return (Q + 255) / 256 * 16; }
__host__ __device__ constexpr int ctl_stride(int Q) { return 16 * ctl_column(Q); }
// Words of a trial of Q sync intervals.
__host__ __device__ constexpr size_t growth_ctl_words(int Q) { return kCtlIntervals + (size_t)kCtlKinds * ctl_stride(Q); }
struct UnitsLoop : UnitsShape {
    const int* sync_end;   // [Q] last step of each sync interval
    int Q;                 // sync intervals before the trailing one
    unsigned long long* ctl;
    // Ring of queued rows (row, somatic spike bits).  An interval's rows lie behind those of all
    // earlier ones, as many as their words say; those of the last interval with rows may still
    // be read (by the first sync block) while the next one's are queued, but no third one's:
    // rows are delivered once every earlier sync is closed, and the HVC(RA) warps wait for that.
    int2* rows;
    int rows_cap;          // at least two intervals' rows
    __device__ __forceinline__ unsigned long long* at(GrowthCtlKind kind, int q) const
    {
        return ctl + kCtlIntervals + kind * ctl_stride(Q) + (q & 15) * ctl_column(Q) + (q >> 4);
    }
    __device__ __forceinline__ int2& row(unsigned pos) const { return rows[pos % (unsigned)rows_cap]; }
};

__device__ __forceinline__ unsigned long long load_acquire64(const unsigned long long* p)
{
    unsigned long long v;
    asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void add_release64(unsigned long long* p, unsigned long long v)
{
    asm volatile("red.release.gpu.global.add.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ void store_release64(unsigned long long* p, unsigned long long v)
{
    asm volatile("st.release.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// An HVC(RA) warp after interval q: all warps' interval q, and the deliveries of its rows.
__device__ __forceinline__ bool ra_wait(const UnitsLoop& L, int q, int* error)
{
    const int lane = threadIdx.x & 31;
    const unsigned long long* p = L.at(lane == 0 ? kCtlRA : lane == 1 ? kCtlI : kCtlDone, q);
    const unsigned want = (unsigned)(lane == 0 ? L.ra_units : L.i_units);
    const bool ok = poll_bounded<true>(0xffffffffu, error, kErrTimeout, L.ctl + kCtlBeat, [&] {
        const unsigned long long v = lane < 3 ? load_acquire64(p) : 0ull;
        const unsigned queued = (unsigned)__shfl_sync(0xffffffffu, v, 0);
        return lane == 0 ? (unsigned)(v >> 32) >= want : lane == 1 ? (unsigned)v >= want
                                                         : lane == 2 ? (unsigned)v >= queued : true;
    });
    __syncwarp();
    return ok;
}

template <class V, bool kTrack>
__device__ __forceinline__ void units_ra(const NetDev<float>& n, const BatchDev<float>& bt, const RAStep<float>& rc,
                                         const UnitsLoop& L, int unit)
{
    constexpr int N = Lanes<V>::n;
    const int lane = threadIdx.x & 31, t = unit * 32 + lane, i0 = N * t;
    const bool any = i0 < n.n_ra;
    RAUnit<V, true> u;
    u.load(n, bt, rc, any ? t : 0, 0, 1);   // a thread without a neuron steps neuron 0 and stores nothing
    if (!any)
#pragma unroll
        for (int k = 0; k < N; ++k) u.valid[k] = false;
    int s0 = 1;
    for (int q = 0; q <= L.Q; ++q) {
        if (q > 0) {
            if (!ra_wait(L, q - 1, bt.error)) return;
            u.sync_kicks(n, bt, q - 1);
        }
        if (q == L.Q) break;   // the steps after the last sync: none, its kicks only
        int live[N];
#pragma unroll
        for (int k = 0; k < N; ++k) live[k] = u.valid[k] ? __ldcg(&bt.live_streams[u.ent[k]]) : 0;
        const int s1 = L.sync_end[q];
        uint32_t soma[N] = {}, dend[N] = {};
        u.template steps<kTrack>(n, bt, rc, s0, s1, soma, dend);
        unsigned queued = 0;
#pragma unroll
        for (int k = 0; k < N; ++k) {
            scatter_warp(soma[k], i0 + k, s0, n.T, n.num_steps, n.syncidx, n.ring, n.ra2i_off, n.ra2i_tgt, n.ra2i_wq,
                         n.ra2i_d, bt.ring_i_exc, (size_t)n.n_i, 0);
            const bool row = u.valid[k] && (soma[k] != 0 || live[k] != 0);
            const unsigned m = __ballot_sync(0xffffffffu, row);
            if (m) {
                unsigned pos = 0;
                if (lane == 0) pos = (unsigned)atomicAdd(L.ctl + kCtlPos, (unsigned long long)__popc(m));
                pos = __shfl_sync(0xffffffffu, pos, 0) + __popc(m & ((1u << lane) - 1u));
                if (row) L.row(pos) = make_int2(i0 + k, (int)soma[k]);
                queued += __popc(m);
            }
        }
        __syncwarp();
        if (lane == 0) add_release64(L.at(kCtlRA, q), (1ull << 32) + queued);
#pragma unroll
        for (int k = 0; k < N; ++k)
            if (soma[k] | dend[k]) ra_spike_stats(bt, u.at(n, k), i0 + k, 0, s0, soma[k], dend[k]);
        s0 = s1 + 1;
    }
    u.store(n, bt);
}

template <bool kTrack>
__device__ __forceinline__ void units_i(const NetDev<float>& n, const BatchDev<float>& bt, const IStep<float>& ic,
                                        const UnitsLoop& L, int unit)
{
    const int lane = threadIdx.x & 31, i = unit * 32 + lane;
    const bool any = i < n.n_i;
    IUnit u(n, bt, any ? i : 0, 0, false);
    int s0 = 1;
    for (int q = 0; q <= L.Q; ++q) {
        if (q > 0) {
            const unsigned want = (unsigned)L.ra_units;
            const bool ok = poll_bounded<true>(0xffffffffu, bt.error, kErrTimeout, L.ctl + kCtlBeat, [&] {
                return lane != 0 || (unsigned)(load_acquire64(L.at(kCtlRA, q - 1)) >> 32) >= want;
            });
            if (!ok) return;
            __syncwarp();
            if (any) u.sync_kicks(n, bt, q - 1);
        }
        if (q == L.Q) break;
        const int s1 = L.sync_end[q];
        uint32_t fired = 0;
        u.template steps<kTrack>(n, bt, ic, s0, s1, i, any ? 0 : 1, fired);   // traces are of instance 0
        if (!any) fired = 0;
        i_scatter(n, bt, fired, i, 0, s0);
        __syncwarp();
        if (lane == 0) add_release64(L.at(kCtlI, q), 1ull);
        u.spike_stats(bt, i, 0, s0, fired);
        s0 = s1 + 1;
    }
    if (any) u.store(bt);
}

// Thread 0 waits (ready returns whether it is done, and may leave values in sh), then the block.
template <class F>
__device__ __forceinline__ bool block_wait(const UnitsLoop& L, int* error, F&& ready)
{
    __shared__ int s_ok;
    __syncthreads();
    if (threadIdx.x == 0) s_ok = poll_bounded<true>(1u, error, kErrTimeout, L.ctl + kCtlBeat, ready) ? 1 : 0;
    __syncthreads();
    return s_ok != 0;
}

__device__ __forceinline__ void units_rows(const GrowthDev& g, const NetDev<float>& n, const BatchDev<float>& bt,
                                           const UnitsLoop& L, int k, RowShared* row_smem)
{
    __shared__ double sh_T[2][2 * kSegSteps];
    __shared__ unsigned s_queued;
    __shared__ int s_ok;
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    unsigned before = 0;   // rows queued in the intervals before q
    for (int q = 0; q < L.Q; ++q) {
        const int s0 = q == 0 ? 1 : L.sync_end[q - 1] + 1, s1 = L.sync_end[q];
        double* T = sh_T[q & 1];
        g_stage_times(T, n.T, s0, s1);
        // The interval's rows are known once the HVC(RA) warps are through with it; if this block
        // has any, sync q - 1 must be closed: its post events, and where it had any, every
        // row's LTP.  One lane of the first warp polls each.
        if (w == 0) {
            const unsigned want = (unsigned)L.ra_units;
            const unsigned long long* p = lane == 0 ? L.at(kCtlRA, q) : L.ctl + (lane == 1 ? kCtlPosted : kCtlLtp);
            unsigned queued = 0;
            const bool ok = poll_bounded<true>(0xffffffffu, g.error, kErrTimeout, L.ctl + kCtlBeat, [&] {
                const unsigned long long v = lane < 3 ? load_acquire64(p) : 0ull;
                queued = (unsigned)__shfl_sync(0xffffffffu, v, 0);
                const unsigned posts = (unsigned)__shfl_sync(0xffffffffu, v, 1);
                const bool here = (unsigned)k < queued;
                return lane == 0   ? (unsigned)(v >> 32) >= want
                       : lane == 1 ? !here || (unsigned)(v >> 32) >= (unsigned)q
                       : lane == 2 ? !here || v >= (unsigned long long)posts * L.nb_sync
                                   : true;
            });
            if (lane == 0) {
                s_ok = ok ? 1 : 0;
                s_queued = queued;
            }
        }
        __syncthreads();
        if (!s_ok) return;
        const unsigned count = s_queued;
        __syncthreads();   // the next interval's wait may write s_queued
        if ((unsigned)k < count) {
            // row e of the interval: block e % nb_row, so that rows spread over the SMs first
            RowStreams st;
            int head = 0, num = 0, row = -1;
            for (unsigned e = (unsigned)(k + w * L.nb_row); e < count; e += (unsigned)(L.nb_row * kTrialWarps)) {
                if (row >= 0 && lane == 0) advance_beat(L.ctl + kCtlBeat);   // the warp's last row is done
                const int2 r = L.row(before + e);
                row = r.x;
                g_row(g, n, bt, (uint32_t)r.y, 0, row, s0, s1, T, row_smem[w], lane, head, num, st);
                __syncwarp();
            }
            __syncthreads();
            if (threadIdx.x == 0) {
                const unsigned mine = (count - (unsigned)k + (unsigned)L.nb_row - 1u) / (unsigned)L.nb_row;
                add_release64(L.at(kCtlDone, q), mine);
            }
            if (row >= 0) g_row_prefetch(g, 0, row, head, num, st, lane);
        }
        before += count;
    }
}

// LTP, LTD and remodeling of this sync block's share of the rows, at the sync of step s1.
__device__ __forceinline__ void units_ltp(const GrowthDev& g, const NetDev<float>& n, const UnitsLoop& L, int k, int s1)
{
    for (int bx = k; bx * kTrialThreads < g.n; bx += L.nb_sync) {
        if (bx != k && threadIdx.x == 0) advance_beat(L.ctl + kCtlBeat);
        g_ltp_body(g, n, s1, 2 * bx, 0);   // rows 256 bx ..
    }
    __syncthreads();
    if (threadIdx.x == 0) add_release64(L.ctl + kCtlLtp, 1ull);
}

// The first sync block: the post events of every interval, and its share of the LTP.
__device__ __forceinline__ void units_newpost(const GrowthDev& g, const NetDev<float>& n, const UnitsLoop& L)
{
    __shared__ unsigned s_queued;
    unsigned before = 0, posts = 0;   // rows queued in the intervals before q; those that had post events
    for (int q = 0; q < L.Q; ++q) {
        const int s0 = q == 0 ? 1 : L.sync_end[q - 1] + 1, s1 = L.sync_end[q];
        const unsigned want = (unsigned)L.ra_units;
        if (!block_wait(L, g.error, [&] {
                const unsigned long long v = load_acquire64(L.at(kCtlRA, q));
                s_queued = (unsigned)v;
                return (unsigned)(v >> 32) >= want && (unsigned)load_acquire64(L.at(kCtlDone, q)) >= (unsigned)v;
            }))
            return;
        const unsigned count = s_queued;
        int K = 0;
        if (count) {
            K = g_newpost_rows(g, n, count, [&](unsigned e) { return L.row(before + e); }, s0, s1);
            __syncthreads();
        }
        if (K > 0) ++posts;
        if (threadIdx.x == 0) {
            if (K > 0) L.ctl[kCtlPosted + 1] = (unsigned long long)q;
            store_release64(L.ctl + kCtlPosted, ((unsigned long long)(q + 1) << 32) + posts);
        }
        if (K > 0) units_ltp(g, n, L, 0, s1);
        before += count;
    }
}

// The other sync blocks: their share of the LTP of the intervals that had post events.  The
// next such interval's deliveries wait for these arrivals and its post events for the
// deliveries, so at most one is outstanding.
__device__ __forceinline__ void units_sync(const GrowthDev& g, const NetDev<float>& n, const UnitsLoop& L, int k)
{
    __shared__ unsigned long long s_posted;
    __shared__ int s_q;
    unsigned closed = 0, posts = 0;
    while (closed < (unsigned)L.Q) {
        if (!block_wait(L, g.error, [&] {
                s_posted = load_acquire64(L.ctl + kCtlPosted);
                s_q = (int)*(volatile unsigned long long*)(L.ctl + kCtlPosted + 1);
                return (unsigned)(s_posted >> 32) > closed;
            }))
            return;
        closed = (unsigned)(s_posted >> 32);
        if ((unsigned)s_posted != posts) {
            posts = (unsigned)s_posted;
            units_ltp(g, n, L, k, L.sync_end[s_q]);
        }
    }
}

// V: the lane type of the HVC(RA) warps.  kTrack: traces of the listed neurons and inhibition
// tracking (a kernel of its own, as for the interval kernels: 450 / 113 with every neuron's
// inhibition at 1 ms, a trial with its weights read back 116 -> 31.6 ms against five
// launches per interval).
template <class V, bool kTrack>
__global__ void __launch_bounds__(kTrialThreads, 1)
    k_growth_units(GrowthDev g, NetDev<float> n, BatchDev<float> bt, RAStep<float> rc,
                   const __grid_constant__ IStep<float> ic, UnitsLoop L)
{
    extern __shared__ __align__(16) unsigned char units_smem[];
    int blk = (int)blockIdx.x;
    const int w = (int)(threadIdx.x >> 5);
    if (blk < L.nb_ra) {
        const int unit = blk * L.ra_per + w;
        if (w < L.ra_per && unit < L.ra_units) units_ra<V, kTrack>(n, bt, rc, L, unit);
        return;
    }
    blk -= L.nb_ra;
    if (blk < L.nb_i) {
        const int unit = blk * L.i_per + w;
        if (w < L.i_per && unit < L.i_units) units_i<kTrack>(n, bt, ic, L, unit);
        return;
    }
    blk -= L.nb_i;
    if (blk == 0) units_newpost(g, n, L);
    else if (blk < L.nb_sync) units_sync(g, n, L, blk);
    else units_rows(g, n, bt, L, blk - L.nb_sync, reinterpret_cast<RowShared*>(units_smem));
}

}  // namespace ug
