"""Failure detection without a GPU fault, for the waits of the one-launch trials' roles
(poll_bounded): an arrival that nothing makes ends the wait after a second; a wait for work
that goes on advancing holds out until it is done; one for work that has stopped advancing
ends a second after that.  The device stays usable each time."""
import time

import pytest

from tests.helpers import small_chain

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("which,status,least,most", [(3, "UG_ETIMEOUT", 0.9, 10.0), (4, "UG_OK", 1.5, 10.0),
                                                     (5, "UG_ETIMEOUT", 1.2, 10.0)])
def test_waits_end_a_second_after_the_last_progress(which, status, least, most, engine32):
    from unsupervised_growth_gb300.engine import probe_bounded_wait
    t0 = time.perf_counter()
    assert probe_bounded_wait(0, which) == status
    waited = time.perf_counter() - t0
    assert least < waited < most, waited
    rn = engine32.load_network(small_chain(seed=5, num_steps=6000))
    rn.run_test_trials(0, 1)
    rn.trial_stats(0)
    rn.free()
