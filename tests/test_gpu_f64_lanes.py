"""The double-precision integrators with eight lanes per neuron against the general ones, which
take the batches with recorded neurons: the same bits, over the sizes where groups of four
neurons have remainders and on both sides of the rule that chooses.

Step and kicks are HH2_test.cpp:613-754 and HHI_buffer.cpp:426-690.  Both forms round the same
operations in the same order, so the tolerance is exact equality."""
import numpy as np
import pytest

from tests.helpers import small_chain, sorted_spikes

pytestmark = pytest.mark.gpu

# n_ra, n_i, trials: last warps with one, two, three and four neurons, one warp alone, and
# batches of more HVC(RA) neurons, and of more of both, than the lanes take
CASES = [(16, 2, 1), (33, 31, 3), (301, 75, 2), (34, 7, 15), (64, 20, 157), (40, 50, 251)]


def _results(rn, trials):
    out = [a for w in (0, 1, 2) for a in rn.trial_stats(w)]
    for k in sorted({0, trials // 2, trials - 1}):
        out += [sorted_spikes(*rn.spikes(k, w)) for w in (0, 1, 2)]
        out += [rn.neuron_state(k, w) for w in (0, 1)]
    return out


@pytest.mark.parametrize("n_ra,n_i,trials", CASES)
def test_lanes_match_general_kernels(engine64, n_ra, n_i, trials):
    net = small_chain(seed=17 + n_ra, n_ra=n_ra, n_i=n_i, groups=4, group=n_ra // 4, num_steps=2500)
    net.training_spread = np.linspace(-98.0, -90.0, len(net.training))   # the chain starts within the trial
    rn = engine64.load_network(net)
    try:
        rn.run_test_trials(3, trials)
        lanes = _results(rn, trials)
        rn.set_recording([0], [0])
        rn.run_test_trials(3, trials)
        general = _results(rn, trials)
    finally:
        rn.free()
    assert lanes[0].sum() > 0
    for a, b in zip(lanes, general):
        assert np.array_equal(a, b)
