"""The connection kernels of the topology generator where their distance filter, tiles and
length pass have edges, against the topology oracle on the same streams
(sample_connections, NetworkGrowthSimulator.cpp:620-705): amplitudes above 1 and near 0, Gaussians
wider than the sphere and narrower than the spacing, targets one past a tile.

Decisions are compared exactly; lengths to 1e-13 relative and 1e-10 microns, as CUDA's acos may
round differently from the host's in the last bit."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

CASES = [("sphere", 1025, 300, 3.0, 60.0), ("sphere", 1100, 129, 1e-4, 900.0), ("sphere", 33, 14, 0.5, 1e6),
         ("sphere", 500, 130, 1.0, 3.0), ("square", 1025, 257, 0.5, 60.0), ("square", 300, 81, 0.02, 5000.0)]


@pytest.mark.parametrize("arrangement,n_ra,n_i,A,sigma", CASES)
def test_connections_match_oracle(engine64, arrangement, n_ra, n_i, A, sigma):
    p = dict(A_RA2I=A, SIGMA_RA2I=sigma, B_I2RA=A / 2, SIGMA_I2RA=2 * sigma)
    t = engine64.generate_topology(p, n_ra, n_i, 5, seed=31, arrangement=arrangement)
    r = O.generate_topology(p, n_ra, n_i, 5, seed=31, arrangement=arrangement)
    try:
        for which, key in ((0, "ri"), (1, "ir")):
            off, tgt, ln = t.connections(which)
            assert np.array_equal(off, r[key][0]) and np.array_equal(tgt, r[key][1])
            np.testing.assert_allclose(ln, r[key][2], rtol=1e-13, atol=1e-10)
    finally:
        t.free()
