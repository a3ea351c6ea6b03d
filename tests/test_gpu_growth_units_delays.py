"""The single build's one-launch growth trial (k_growth_units) with delays that end within a
sync interval: no delivery stream stays open, so intervals without a queued row follow the
spikes at once, and the HVC(RA) warps run on while the first sync block still takes up an
interval's post events (some hundred of them here, each with a pass over every row's
presynaptic events).  The next spikes come three to eight intervals later.  Every role must
read its own interval's arrivals and rows however far the others are ahead.

The per-interval launches make the same operations in the same order
(NetworkGrowthSimulator.cpp:8923-9564), so the tolerance is exact equality."""
import numpy as np
import pytest

from tests.helpers import FAST_MAT, FAST_SYN, small_growth, sorted_spikes

pytestmark = pytest.mark.gpu

INTERVAL_MS = 0.25

# n_ra, n_i, training neurons, delays 0..width ms, synapses that saturate (Nss 2) or not
CASES = [(600, 150, 200, 0.0, True), (600, 150, 200, 0.1, False), (600, 150, 200, 0.25, True),
         (1300, 40, 500, 0.0, False), (300, 75, 300, 0.0, True)]


@pytest.mark.parametrize("n_ra,n_i,n_tr,width,fast", CASES)
def test_short_delays_match_interval_launches(engine32, n_ra, n_i, n_tr, width, fast):
    net = small_growth(seed=31 + n_ra, n_ra=n_ra, n_i=n_i, n_tr=n_tr, syn=FAST_SYN if fast else dict(FAST_SYN, Nss=10),
                       mat=FAST_MAT, delays="uniform", delay_width=width)
    # half of the training set at once, the others three to eight intervals later
    late = np.arange(len(net.training)) % 12
    net.training_spread = np.where(late < 6, 0.0, (late - 3) * INTERVAL_MS)
    out = []
    try:
        for one in (True, False):
            engine32.set_growth_launch(one)
            rn = engine32.load_network(net)
            l0 = engine32.launch_count()
            rn.run_growth_trials(0, 3, True)
            out.append((engine32.launch_count() - l0, rn.weights(), rn.synapse_list(0), rn.synapse_list(1),
                        [sorted_spikes(*rn.spikes(0, w)) for w in (0, 1, 2)],
                        [rn.neuron_state(0, w) for w in (0, 1)]))
            rn.free()
    finally:
        engine32.set_growth_launch(True)
    one, per = out
    assert one[0] <= 30 < per[0]
    assert len(one[4][0]) > n_tr // 2 and one[1].max() > 0.0   # spikes, and potentiation
    assert np.array_equal(one[1], per[1]) and one[2] == per[2] and one[3] == per[3]
    for a, b in zip(one[4] + one[5], per[4] + per[5]):
        assert np.array_equal(a, b)
