"""The form of the single build's one-launch growth trial with two HVC(RA) neurons per thread
(k_growth_units<f2>): taken when blocks of one neuron per thread leave the rows too few SMs,
here 4201 neurons in blocks of one warp (an odd count: the last thread has one neuron).  The
per-interval launches make the same operations in the same order
(NetworkGrowthSimulator.cpp:8923-9564), so the tolerance is exact equality."""
import numpy as np
import pytest

from tests.helpers import FAST_MAT, FAST_SYN, small_growth, sorted_spikes
from tests.test_plans import plans, units_shape  # noqa: F401  (a fixture)

pytestmark = pytest.mark.gpu

N_RA, N_I, SHAPE = 4201, 40, (32, 32)


@pytest.mark.parametrize("record", [None, "inhibition", "traces"])
def test_two_lanes_match_interval_launches(engine32, plans, record):  # noqa: F811
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert units_shape(plans, N_RA, N_I, SHAPE, sms)[1]["lanes"] == 2
    net = small_growth(seed=17, n_ra=N_RA, n_i=N_I, n_tr=12, syn=FAST_SYN, mat=FAST_MAT, delays="uniform",
                       delay_width=1.0)
    net.training_spread = np.linspace(0.0, 6.0, len(net.training))
    out = []
    try:
        engine32.set_growth_trial_shape(*SHAPE)
        for one in (True, False):
            engine32.set_growth_launch(one)
            rn = engine32.load_network(net)
            if record == "inhibition":
                rn.set_inhibition_tracking(5.0)
            elif record == "traces":
                rn.set_recording([0, 1, N_RA - 1], [0, N_I - 1])
            l0 = engine32.launch_count()
            rn.run_growth_trials(0, 2, True)
            got = [rn.weights()] + [sorted_spikes(*rn.spikes(0, w)) for w in (0, 1, 2)]
            got += [rn.neuron_state(0, w) for w in (0, 1)]
            if record == "inhibition":
                got.append(rn.inhibitory_conductance()[0])
            elif record == "traces":
                got += [rn.trace(0, 0), rn.trace(0, 1), rn.trace(0, 2), rn.trace(1, 0), rn.trace(1, 1)]
            out.append((engine32.launch_count() - l0, rn.synapse_list(0), rn.synapse_list(1), got))
            rn.free()
    finally:
        engine32.set_growth_launch(True)
        engine32.set_growth_trial_shape(0, 0)
    one, per = out
    assert one[0] <= 20 < per[0]
    assert len(one[3][1]) > 0 and one[3][0].max() > 0.0   # spikes, and potentiation
    assert one[1] == per[1] and one[2] == per[2]
    for a, b in zip(one[3], per[3]):
        assert np.array_equal(a, b)
