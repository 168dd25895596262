"""The recompression kernel at the sizes where its work split changes: tile sizes around the row
capacities of its shapes (128, 256, 512, 1024 rows), a last tile of a few sites, ranks on both sides of
a panel block (8 columns) and of the cores held in shared memory, and the Matern 5/2 kernel.

Against the NumPy oracle: identical initial and factor ranks.  The log-likelihood bound is 1e-9
relative: the ranks agree, every factor entry carries FP64 rounding times the conditioning that the
parity fixtures show (1e-10), and tiles at the sketch's margin another 1e-9 / few."""
import numpy as np
import pytest

from oracle import tlr_oracle as O

pytestmark = pytest.mark.gpu
CASES = [  # (n, b, theta, rule, value)
    (53, 7, (1.0, 0.3, 0.05), "adaptive", 0.9),
    (700, 127, (1.0, 0.3, 0.05), "adaptive", 0.9),
    (641, 128, (1.3, 0.2, 0.02), "fixed", 1e-6),
    (660, 129, (1.0, 0.1, 0.01), "adaptive", 0.5),
    (1290, 256, (1.0, 0.3, 0.05), "fixed", 1e-9),   # ranks past 8: several panel blocks, large cores
    (1031, 257, (0.7, 0.15, 0.005), "adaptive", 0.3),
    (2051, 512, (1.0, 0.3, 0.05), "adaptive", 0.9),
    (2055, 513, (1.0, 0.2, 0.05), "fixed", 1e-5),
]


@pytest.fixture(scope="module")
def tlr():
    import adaptive_tlr_pilots_b200 as m
    yield m
    m.release_plans()


@pytest.mark.parametrize("n,b,theta,rule,value", CASES)
def test_recompression_shapes_match_oracle(tlr, n, b, theta, rule, value):
    rng = np.random.default_rng(n)
    S = rng.random((n, 2))
    S = S[O.morton_order(S)]
    y = np.sin(5 * S[:, 0]) + 0.3 * rng.standard_normal(n)
    bounds = O.tile_bounds(n, b)
    log = {}
    ll_o, fac, info_o = O.tlr_loglik(S, y, theta, bounds, rule, value, rank_log=log)
    ll, f, info = tlr.tlr_loglik(S, y, theta, bounds, rule, value)
    assert info["completed"] == info_o["completed"]
    assert info["stored_sigma"] == info_o["stored_sigma"]
    assert info["stored_factor"] == info_o["stored_factor"]
    assert info["max_rank_factor"] == info_o["max_rank_factor"]
    assert abs(ll - ll_o) <= 1e-9 * abs(ll_o)
