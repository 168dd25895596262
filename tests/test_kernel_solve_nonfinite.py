"""k_tri_solve on the host (emu/cuda_emu.h) with an infinity or NaN in the right-hand side: it reaches the rows that
depend on it and no others, as in a substitution; the other columns of the chunk keep their values."""
import numpy as np
import pytest

import host_cuda

MAIN = r"""
#include "tlr_solve.cu"
using namespace tlr;
// usage: main b trans row value columns -> L (lower, by columns), the right-hand sides, the solutions
int main(int argc, char** argv) {
  const int b = atoi(argv[1]), trans = atoi(argv[2]), row = atoi(argv[3]), m = atoi(argv[5]), np = (b + 31) / 32;
  const double value = atof(argv[4]);
  std::mt19937 rng(5);
  std::uniform_real_distribution<double> u(-1.0, 1.0);
  std::vector<double> D((size_t)b * b), inv((size_t)np * 1024), X((size_t)b * m);
  for (int c = 0; c < b; ++c)
    for (int r = 0; r < b; ++r) D[(size_t)c * b + r] = r < c ? NAN : r == c ? 2.0 + u(rng) : 0.1 * u(rng);
  for (auto& x : X) x = u(rng);
  if (row >= 0) X[(size_t)b + row] = value;  // the second column
  for (double v : D) printf("%a\n", v);
  for (double v : X) printf("%a\n", v);
  emu::Config cfg;
  emu::run(dim3((np + 1) / 2), dim3(64), 1, 0, cfg, [&] { k_diag_inv(D.data(), b, b, 0, np, inv.data()); });
  const std::string err = emu::run(dim3((m + kSC - 1) / kSC), dim3(kSW * 32), 1, (size_t)kSC * (np * 32 + 8) * 8, cfg, [&] {
    if (trans) k_tri_solve<true>(D.data(), inv.data(), b, b, np, 0, X.data(), b, m);
    else k_tri_solve<false>(D.data(), inv.data(), b, b, np, 0, X.data(), b, m);
  });
  if (!err.empty()) return 1;
  for (double v : X) printf("%a\n", v);
}
"""


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    return host_cuda.build(tmp_path_factory.mktemp("solve"), MAIN)


@pytest.mark.parametrize("b,row,value", [(40, -1, 0), (33, 7, "nan"), (70, 40, "inf"), (70, 69, "-inf"), (70, 0, "nan")])
@pytest.mark.parametrize("trans", [0, 1])
def test_nonfinite_right_hand_sides(exe, b, row, value, trans):
    m = 3
    v = np.array([float(x) if x in ("nan", "-nan", "inf", "-inf") else float.fromhex(x)
                  for x in host_cuda.run(exe, b, trans, row, value, m).split()])
    L = np.tril(v[:b * b].reshape(b, b).T)
    B = v[b * b:b * b + b * m].reshape(m, b).T
    X = v[b * b + b * m:].reshape(m, b).T
    want = B.copy()
    for s in range(b):
        r = b - 1 - s if trans else s
        done = range(r + 1, b) if trans else range(r)
        for q in done:
            with np.errstate(invalid="ignore"):
                want[r] -= (L[q, r] if trans else L[r, q]) * want[q]
        want[r] /= L[r, r]
    assert np.array_equal(np.isfinite(X), np.isfinite(want))
    ok = np.isfinite(want)
    assert np.abs(X[ok] - want[ok]).max() <= 1e-12
