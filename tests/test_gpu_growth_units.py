"""The single build's one-launch growth trial (k_growth_units) where its roles have edges: one
and two HVC(RA) neurons per thread, warps with one neuron, few and many rows in an interval,
few interneurons.  The per-interval launches make the same operations in the same order
(NetworkGrowthSimulator.cpp:8923-9564), so the tolerance is exact equality."""
import numpy as np
import pytest

from tests.helpers import FAST_MAT, FAST_SYN, small_growth, sorted_spikes

pytestmark = pytest.mark.gpu

# n_ra, n_i, steps, role widths: 33 and 65 leave a warp one neuron; 3600 in blocks of one warp
# exceeds the SMs with one neuron per thread, so two are stepped
CASES = [(33, 14, 25000, (0, 0)), (65, 33, 25000, (64, 32)), (300, 2, 25000, (0, 0)), (3600, 40, 9000, (32, 32))]


@pytest.mark.parametrize("n_ra,n_i,steps,shape", CASES)
def test_units_match_interval_launches(engine32, n_ra, n_i, steps, shape):
    net = small_growth(seed=21 + n_ra, n_ra=n_ra, n_i=n_i, n_tr=8, syn=FAST_SYN, mat=FAST_MAT, delays="uniform",
                       delay_width=1.0, num_steps=steps)
    # every training neuron fires at once (many rows in one interval), before a short trial ends
    net.training_spread = np.full(len(net.training), -95.0 if steps < 25000 else 0.0)
    out = []
    try:
        engine32.set_growth_trial_shape(*shape)
        for one in (True, False):
            engine32.set_growth_launch(one)
            rn = engine32.load_network(net)
            l0 = engine32.launch_count()
            rn.run_growth_trials(0, 2, True)
            out.append((engine32.launch_count() - l0, rn.weights(), rn.synapse_list(0), rn.synapse_list(1),
                        [sorted_spikes(*rn.spikes(0, w)) for w in (0, 1, 2)],
                        [rn.neuron_state(0, w) for w in (0, 1)]))
            rn.free()
    finally:
        engine32.set_growth_launch(True)
        engine32.set_growth_trial_shape(0, 0)
    one, per = out
    assert one[0] <= 20 < per[0]
    assert len(one[4][0]) > 0
    assert np.array_equal(one[1], per[1]) and one[2] == per[2] and one[3] == per[3]
    for a, b in zip(one[4] + one[5], per[4] + per[5]):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("n_ra,n_i,steps,shape", [(33, 14, 25000, (0, 0)), (3600, 40, 9000, (32, 32))])
@pytest.mark.parametrize("what", ["inhibition", "traces"])
def test_units_record_what_interval_launches_record(engine32, n_ra, n_i, steps, shape, what):
    net = small_growth(seed=5 + n_ra, n_ra=n_ra, n_i=n_i, n_tr=8, syn=FAST_SYN, mat=FAST_MAT, delays="uniform",
                       delay_width=1.0, num_steps=steps)
    net.training_spread = np.full(len(net.training), -95.0 if steps < 25000 else 0.0)
    out = []
    try:
        engine32.set_growth_trial_shape(*shape)
        for one in (True, False):
            engine32.set_growth_launch(one)
            rn = engine32.load_network(net)
            if what == "inhibition":
                rn.set_inhibition_tracking(0.7)
            else:
                rn.set_recording([0, n_ra - 1], [0, n_i - 1])
            l0 = engine32.launch_count()
            rn.run_growth_trials(0, 2, True)
            rec = [rn.inhibitory_conductance()[0]] if what == "inhibition" else [rn.trace(w, k) for w in (0, 1) for k in (0, 1)]
            out.append([engine32.launch_count() - l0, rn.weights(), *rec, *[rn.neuron_state(0, w) for w in (0, 1)]])
            rn.free()
    finally:
        engine32.set_growth_launch(True)
        engine32.set_growth_trial_shape(0, 0)
    one, per = out
    assert one[0] <= 20 < per[0]
    for a, b in zip(one[1:], per[1:]):
        assert np.array_equal(a, b)
