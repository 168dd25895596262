"""Kernels whose work split depends on the tile size, at the sizes where it changes: panels of 32 columns
in the diagonal factorization and the panel solve (31, 32, 33), the cluster sizes of the diagonal
factorization (256, 257), the column budget of the panel solve (512 and above), the sketch's row tiles
(319, 320, 321), odd tile sizes (unpaired loads), ranks past 32 in the panel solve and past 64 in the
recompression (the plan's columns grow), steps with more and with fewer pairs than SMs, and a last tile of a
few sites.

Against the NumPy oracle: identical ranks; log-likelihood within 1e-9 relative (FP64 rounding times the
conditioning that the parity fixtures show, 1e-10, and a margin of ten).  The GEMM at its larger tile
shape, which one product takes from 2,500 x 2,500 on, has the bound of its product: 1e-13 of
sum_k |a_ik| |b_kj|."""
import numpy as np
import pytest

from oracle import tlr_oracle as O

pytestmark = pytest.mark.gpu
CASES = [  # (n, b, theta, rule, value)
    (95, 31, (1.0, 0.3, 0.05), "fixed", 1e-6),
    (101, 32, (1.0, 0.3, 0.05), "fixed", 1e-6),
    (100, 33, (1.0, 0.3, 0.05), "fixed", 1e-6),
    (960, 319, (1.0, 0.2, 0.05), "adaptive", 0.9),
    (963, 320, (1.0, 0.2, 0.05), "adaptive", 0.9),
    (1300, 321, (1.0, 0.2, 0.05), "adaptive", 0.9),
    (1540, 512, (1.0, 0.1, 0.01), "adaptive", 0.3),
    (3001, 1000, (1.0, 0.2, 0.05), "adaptive", 0.9),
    (770, 256, (1.0, 0.1, 0.005), "fixed", 1e-6),
    (775, 257, (1.0, 0.1, 0.005), "fixed", 1e-6),
    (2400, 600, (1.0, 0.05, 0.002), "fixed", 1e-6),
    (2080, 100, (1.0, 0.3, 0.05), "adaptive", 0.9),   # 190, 171, ... pairs: both sides of one per SM
    (3990, 200, (1.0, 0.2, 0.05), "adaptive", 0.9),
]


@pytest.fixture(scope="module")
def tlr():
    import adaptive_tlr_pilots_b200 as m
    yield m
    m.release_plans()


def _data(n):
    rng = np.random.default_rng(n)
    S = rng.random((n, 2))
    S = S[O.morton_order(S)]
    return S, np.sin(5 * S[:, 0]) + 0.3 * rng.standard_normal(n)


@pytest.mark.parametrize("n,b,theta,rule,value", CASES)
def test_tile_sizes_match_oracle(tlr, n, b, theta, rule, value):
    S, y = _data(n)
    bounds = O.tile_bounds(n, b)
    ll_o, _, info_o = O.tlr_loglik(S, y, theta, bounds, rule, value)
    ll, _, info = tlr.tlr_loglik(S, y, theta, bounds, rule, value)
    assert info["completed"] == info_o["completed"]
    assert info["stored_sigma"] == info_o["stored_sigma"]
    assert info["max_rank_factor"] == info_o["max_rank_factor"]
    assert abs(ll - ll_o) <= 1e-9 * abs(ll_o)


@pytest.mark.parametrize("transA,transB,pad,shift", [(0, 0, 0, 0), (1, 0, 1, 0), (0, 1, 0, 1), (1, 1, 1, 1)])
def test_gemm_large_tiles(tlr, transA, transB, pad, shift):
    import torch
    from adaptive_tlr_pilots_b200 import _lib
    from test_gpu_gemm import _run
    assert _run((torch, _lib, _lib.load()), "fp64", transA, transB, 2501, 2563, 33, -1.0, 1.0, pad, shift) <= 1e-13
