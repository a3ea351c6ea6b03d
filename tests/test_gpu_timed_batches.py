"""A test batch with per-kernel timing on runs per-interval launches of its own and leaves the
captured graph of the network's batch, and the launch form it was captured with, as they were:
the same bits throughout, and the untimed batches' launch count before and after."""
import numpy as np
import pytest

from tests.helpers import small_chain

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("trials", [1, 20])
def test_timed_batch_leaves_the_captured_one(engine32, trials):
    rn = engine32.load_network(small_chain(seed=6, num_steps=6000))
    counts, results = [], []
    try:
        for timed in (False, True, False, False):
            engine32.set_kernel_timing(timed)
            before = engine32.launch_count()
            rn.run_test_trials(3, trials)
            counts.append(engine32.launch_count() - before)
            results.append([a for w in (0, 1, 2) for a in rn.trial_stats(w)] + [rn.neuron_state(0, w) for w in (0, 1)])
    finally:
        engine32.set_kernel_timing(False)
        rn.free()
    assert counts[0] == counts[2] == counts[3] < counts[1]
    for r in results[1:]:
        for a, b in zip(results[0], r):
            assert np.array_equal(a, b)
