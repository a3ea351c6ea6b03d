// Shapes of the one-launch growth trials: which networks take one, and how its blocks share
// the roles.  Host arithmetic alone, so that tests compile it without a GPU.
#pragma once
#include <algorithm>

namespace ug {

constexpr int kTrialThreads = 256;
constexpr int kTrialWarps = kTrialThreads / 32;

// Threads per block of the integrating roles (whole warps, at most kTrialThreads): by default
// one integrating warp per block, so that a trial spreads over as many SMs as it has
// integrating warps; wider roles put several integrating warps on one SM scheduler.
constexpr int kRoleThreads = 32;

// The role widths of a request (0: the default); false unless each is a multiple of 32
// in [32, kTrialThreads].
inline bool trial_widths(int req_ra, int req_i, int* ra_w, int* i_w)
{
    *ra_w = req_ra ? req_ra : kRoleThreads;
    *i_w = req_i ? req_i : kRoleThreads;
    for (int w : {*ra_w, *i_w})
        if (w < 32 || w > kTrialThreads || w % 32) return false;
    return true;
}

// Blocks of k_growth_units (single build) per role.
struct UnitsShape {
    int lanes = 0;             // HVC(RA) neurons per thread; 0: no shape, per-interval launches
    int ra_units, i_units;     // warps of the two integrating roles
    int ra_per, i_per;         // of them per block
    int nb_ra, nb_i, nb_sync, nb_row;
    int blocks() const { return lanes ? nb_ra + nb_i + nb_sync + nb_row : 0; }
};
constexpr int kSyncBlocks = 16, kRowBlocks = 64;              // at most
constexpr int kEnoughRowBlocks = 32, kMinRowBlocks = 8;       // rather than wider roles; at least
// Above this many HVC(RA) neurons the per-interval launches are the faster ones: they give the
// rows and the LTP every SM, and of a large network's interval those are the most part.
// Measured, ms a trial, one launch / per interval, networks with 10 training neurons:
// 2000 HVC(RA) 40.2 / 56.7, 5000 77.9 / 92.8, 7500 118 / 130, 10 000 161 / 165, 12 000
// 204 / 200, 18 000 342 / 305; with several hundred and synapses that grow fast: 3000 131 / 148,
// 5000 456 / 469 (1000 training neurons: 765 / 759), 7500 1668 / 1660, 8000 1473 / 1467 (1000:
// 4334 / 4196), 10 000 16 960 / 11 530.
constexpr int kUnitsMaxRA = 8000;

// One HVC(RA) neuron per thread where the roles fit the SMs, a block each, else two.  The rows
// take what the other roles leave, up to kRowBlocks blocks.  req_ra, req_i as trial_widths;
// resident: whether an SM takes a block of the kernel with one, with two neurons per thread.
inline UnitsShape units_shape(int n_ra, int n_i, int req_ra, int req_i, int sms, const bool (&resident)[2])
{
    UnitsShape none;
    int ra_w = 0, i_w = 0;
    if (n_ra > kUnitsMaxRA || !trial_widths(req_ra, req_i, &ra_w, &i_w)) return none;
    for (int lanes = 1; lanes <= 2; ++lanes) {
        if (!resident[lanes - 1]) continue;
        // by default as few warps to a block as leave the rows enough blocks
        for (int per = 1; per <= kTrialWarps; per *= 2) {
            UnitsShape u;
            u.ra_units = (n_ra + 32 * lanes - 1) / (32 * lanes);
            u.i_units = (n_i + 31) / 32;
            u.ra_per = req_ra ? ra_w / 32 : per;
            u.i_per = req_i ? i_w / 32 : per;
            u.nb_ra = (u.ra_units + u.ra_per - 1) / u.ra_per;
            u.nb_i = (u.i_units + u.i_per - 1) / u.i_per;
            u.nb_sync = std::min(kSyncBlocks, (n_ra + kTrialThreads - 1) / kTrialThreads);
            u.nb_row = std::min(kRowBlocks, sms - u.nb_ra - u.nb_i - u.nb_sync);
            if (u.nb_row < (per < kTrialWarps ? kEnoughRowBlocks : kMinRowBlocks)) continue;
            u.lanes = lanes;
            return u;
        }
    }
    return none;
}

}  // namespace ug
