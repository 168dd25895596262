"""Nuggets far below those of the parity fixtures.  The panel solve and the solves with the factor multiply by the
inverses of the 32 x 32 diagonal blocks, whose condition grows as the nugget falls.

Log-likelihood against the NumPy oracle, which substitutes: the entries of L^-1 V carry about 10 eps / sqrt(eta) here
(eta = 1e-5: 1e-14 either way), the log determinant and the quadratic form their sum over a spectrum of
condition 1000 / eta: 1e-10 relative at eta = 1e-3, 1e-8 at 1e-5.  Solves against a dense triangular solve with
the same factor: n eps cond(L), cond(L) about sqrt(1000 / eta) = 1e4."""
import numpy as np
import pytest

from oracle import tlr_oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def tlr():
    import adaptive_tlr_pilots_b200 as m
    yield m
    m.set_kernel(1.5)
    m.release_plans()


def _data(n):
    rng = np.random.default_rng(n)
    S = rng.random((n, 2))
    S = S[O.morton_order(S)]
    return S, np.sin(5 * S[:, 0]) + 0.3 * rng.standard_normal(n)


@pytest.mark.parametrize("eta,bound", [(1e-3, 1e-10), (1e-5, 1e-8)])
@pytest.mark.parametrize("n,b", [(1000, 250), (1501, 301)])
def test_loglik_matches_oracle(tlr, n, b, eta, bound):
    S, y = _data(n)
    bounds = O.tile_bounds(n, b)
    theta = (1.0, 0.1, eta)
    ll_o, _, info_o = O.tlr_loglik(S, y, theta, bounds, "adaptive", 0.9)
    ll, _, info = tlr.tlr_loglik(S, y, theta, bounds, "adaptive", 0.9)
    assert info["completed"] and info_o["completed"]
    assert info["stored_sigma"] == info_o["stored_sigma"]
    assert abs(ll - ll_o) <= bound * abs(ll_o)


def test_solves_match_dense_triangular(tlr):
    from scipy.linalg import solve_triangular
    n, b = 1501, 301
    S, y = _data(n)
    plan = tlr.Plan(n, b)
    plan.set_data(S, y)
    plan.evaluate((1.0, 0.1, 1e-5), "adaptive", 0.9)
    edges = [a for a, _ in O.tile_bounds(n, b)] + [n]
    L = np.zeros((n, n))
    for k in range(plan.nB):
        L[edges[k]:edges[k + 1], edges[k]:edges[k + 1]] = plan.diag_tile(k)
        for i in range(k + 1, plan.nB):
            u, v = plan.offdiag_tile(i, k)
            L[edges[i]:edges[i + 1], edges[k]:edges[k + 1]] = u @ v.T
    B = np.random.default_rng(3).standard_normal((n, 5))
    for trans in (False, True):
        X = plan.solve(B, trans=trans).cpu().numpy()
        R = solve_triangular(L, B, lower=True, trans=int(trans))
        assert np.abs(X - R).max() <= n * 2.3e-16 * 1e4 * np.abs(R).max()
    plan.close()
