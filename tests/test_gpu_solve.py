"""Solves with the factor (tlr_factor_solve) at the edges of their work split: panels of 32 rows, row
blocks of 8, chunks of 8 and 32 columns, odd tile sizes and a last tile of a few rows, both directions.

Against a dense triangular solve with the same factor.  Bound: c n eps cond(L) with cond(L) about
sqrt(n / eta) < 300 at these sizes gives below 1e-10 of the largest entry."""
import numpy as np
import pytest

from oracle import tlr_oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def tlr():
    import adaptive_tlr_pilots_b200 as m
    yield m


@pytest.mark.parametrize("n,b", [(40, 50), (513, 64), (700, 33), (901, 127), (1501, 250), (2055, 513), (3000, 1000)])
def test_solves_match_dense_triangular(tlr, n, b):
    from scipy.linalg import solve_triangular
    rng = np.random.default_rng(n)
    S = rng.random((n, 2))
    S = S[O.morton_order(S)]
    plan = tlr.Plan(n, b)
    plan.set_data(S, rng.standard_normal(n))
    plan.evaluate((1.0, 0.3, 0.05), "adaptive", 0.9)
    edges = [a for a, _ in O.tile_bounds(n, b)] + [n]
    L = np.zeros((n, n))
    for k in range(plan.nB):
        L[edges[k]:edges[k + 1], edges[k]:edges[k + 1]] = plan.diag_tile(k)
        for i in range(k + 1, plan.nB):
            u, v = plan.offdiag_tile(i, k)
            L[edges[i]:edges[i + 1], edges[k]:edges[k + 1]] = u @ v.T
    for m in (1, 8, 9, 33, 70):
        B = rng.standard_normal((n, m))
        for trans in (False, True):
            X = plan.solve(B, trans=trans).cpu().numpy()
            R = solve_triangular(L, B, lower=True, trans=int(trans))
            assert np.abs(X - R).max() <= 1e-10 * np.abs(R).max(), (m, trans)
    plan.close()
