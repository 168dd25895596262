"""Correlation ranges far below the distance between tiles: most off-diagonal tiles are many orders of magnitude
below the nugget, have rank 0, and their sketches' squared norms leave the range of a double.

Against the NumPy oracle: identical ranks, log-likelihood within 1e-9 relative (the bound of the other
sizes: FP64 rounding times the conditioning, with a margin of ten)."""
import numpy as np
import pytest

from oracle import tlr_oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def tlr():
    import adaptive_tlr_pilots_b200 as m
    yield m
    m.release_plans()


@pytest.mark.parametrize("n,b,rng_", [(2000, 100, 0.02), (2000, 100, 0.01), (2000, 100, 0.007), (2000, 100, 0.005),
                                      (4000, 100, 0.01), (2010, 201, 0.007), (2400, 600, 0.006)])
def test_short_ranges_match_oracle(tlr, n, b, rng_):
    rng = np.random.default_rng(n + b)
    S = rng.random((n, 2))
    S = S[O.morton_order(S)]
    y = rng.standard_normal(n)
    bounds = O.tile_bounds(n, b)
    theta = (1.0, rng_, 0.05)
    ll_o, _, info_o = O.tlr_loglik(S, y, theta, bounds, "adaptive", 0.9)
    ll, _, info = tlr.tlr_loglik(S, y, theta, bounds, "adaptive", 0.9)
    assert info["completed"] and info_o["completed"]
    assert info["stored_sigma"] == info_o["stored_sigma"]
    assert info["stored_factor"] == info_o["stored_factor"]
    assert abs(ll - ll_o) <= 1e-9 * abs(ll_o)
