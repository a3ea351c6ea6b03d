"""Test batches in one cooperative launch (k_test_trial) against the per-interval launches:
the same bits, over the sizes where its warps, lanes and segments have edges.

The trial is trial_no_stdp_fixedSpread (NetworkGrowthSimulator.cpp:12747-13117).  Both forms
make the same operations in the same order per neuron, and kicks add in fixed point, so the
tolerance is exact equality."""
import numpy as np
import pytest

from tests.helpers import small_chain, sorted_spikes

pytestmark = pytest.mark.gpu

# n_ra, n_i, trials, steps: warps of 32 (one HVC(RA) neuron per thread) and 64 (two), a last
# warp with one neuron, none left over, two interneurons, a trial too short for two segments,
# batches with one and with two neurons per thread, and one of more warps than fit
CASES = [(32, 32, 1, 9000), (33, 31, 2, 9000), (65, 2, 3, 9000), (64, 33, 15, 5600), (60, 20, 16, 9000),
         (60, 20, 3, 700), (33, 20, 250, 5600), (129, 65, 130, 5600), (40, 33, 900, 1400)]


def _results(rn, trials):
    stats = [rn.trial_stats(w) for w in (0, 1, 2)]
    out = [a for pair in stats for a in pair]
    for k in sorted({0, trials // 2, trials - 1}):
        out += [sorted_spikes(*rn.spikes(k, w)) for w in (0, 1, 2)]
        out += [rn.neuron_state(k, w) for w in (0, 1)]
    return out


@pytest.mark.parametrize("n_ra,n_i,trials,steps", CASES)
@pytest.mark.parametrize("delay", [None, 0.0])
def test_one_launch_matches_interval_launches(engine32, n_ra, n_i, trials, steps, delay):
    net = small_chain(seed=11 + n_ra, n_ra=n_ra, n_i=n_i, groups=4, group=n_ra // 4, num_steps=steps)
    net.training_spread = np.linspace(-98.0, -90.0, len(net.training))   # the chain starts within the trial
    if delay is not None:
        for a in (net.ra2i_d, net.i2ra_d, net.d_rara):
            a[:] = delay
    rn = engine32.load_network(net)
    try:
        rn.run_test_trials(5, trials)
        one = _results(rn, trials)
        rn.run_test_trials(5, trials)   # again: the arrival counters and lists start over
        again = _results(rn, trials)
        engine32.set_interval_fusion(False)
        rn.run_test_trials(5, trials)
        apart = _results(rn, trials)
    finally:
        engine32.set_interval_fusion(True)
        rn.free()
    assert steps < 1000 or one[0].sum() > 0
    for a, b, c in zip(one, again, apart):
        assert np.array_equal(a, c) and np.array_equal(b, c)
