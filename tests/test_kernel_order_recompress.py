"""k_recompress and k_recompress_general on the host (emu/cuda_emu.h) under every order of their threads: one
factorization step of three trailing pairs, with panels of one block of columns and of several, and cores past order 32.  The bits do
not depend on the order; the updated tile is U V^T - U_ik V_ik^T V_jk U_jk^T up to the rule's threshold; and a
status word that another kernel sets while a CTA's threads read it ends the CTA as a whole."""
import pytest

import host_cuda

MAIN = r"""
#include "tlr_recompress.cu"
#define tidx tidx_factor  // both files have their own
#include "tlr_factor.cu"
#undef tidx
using namespace tlr;
// usage: main general b rank cap seed cta_order thread_order flip_after [fall scale]
int main(int argc, char** argv) {
  const int general = atoi(argv[1]), b = atoi(argv[2]), r = atoi(argv[3]), cap = atoi(argv[4]);
  emu::Config cfg;
  cfg.seed = (unsigned)atoi(argv[5]);
  cfg.cta = (emu::Order)atoi(argv[6]);
  cfg.thread = (emu::Order)atoi(argv[7]);
  cfg.flip_after = atoi(argv[8]);
  cfg.flip_value = 3;
  const double fall = argc > 9 ? atof(argv[9]) : 0.6, scale = argc > 10 ? atof(argv[10]) : 1.0;
  const int nB = 4, n = 3 * b + b / 2, ntiles = 6;  // the last tile is ragged
  std::vector<char> ctl(kControlBytes, 0);
  int* status = reinterpret_cast<int*>(ctl.data());
  cfg.flip_word = status;
  auto* prm = const_cast<EvalParams*>(eval_params(status));
  prm->rule_fixed = 1;
  prm->thr_rel = 1e-7;
  prm->round_store = 0;
  std::mt19937 rng(11);
  std::uniform_real_distribution<double> u(-1.0, 1.0);
  std::vector<double> U((size_t)ntiles * b * cap, 0.0), V(U);
  std::vector<int> rank(ntiles);
  // orthogonal columns of falling norm in U, orthonormal ones in V
  auto columns = [&](double* X, int rows, int cols, double s, double fall) {
    for (int c = 0; c < cols; ++c) {
      double* x = X + (size_t)c * b;
      for (int a = 0; a < rows; ++a) x[a] = u(rng);
      for (int pass = 0; pass < 3; ++pass) {
        for (int d = 0; d < c && pass < 2; ++d) {
          const double* y = X + (size_t)d * b;
          double dot = 0.0;
          for (int a = 0; a < rows; ++a) dot += x[a] * y[a];
          for (int a = 0; a < rows; ++a) x[a] -= dot * y[a];
        }
        double nn = 0.0;
        for (int a = 0; a < rows; ++a) nn += x[a] * x[a];
        for (int a = 0; a < rows; ++a) x[a] /= sqrt(nn);
      }
    }
    for (int c = 0; c < cols; ++c, s *= fall)
      for (int a = 0; a < rows; ++a) X[(size_t)c * b + a] *= s;
  };
  auto id = [](int i, int j) { return i * (i - 1) / 2 + j; };
  for (int i = 1; i < nB; ++i)
    for (int j = 0; j < i; ++j) {
      const int t = id(i, j), rt = std::min(r - (i + j) % 3, i == 3 ? b / 2 : b);
      rank[t] = rt;
      // scaled: the updated tiles and the factor of their update that is not U_ik's side
      columns(&U[(size_t)t * b * cap], i == 3 ? b / 2 : b, rt, j > 0 || i == 1 ? scale : 1.0, j > 0 || i == 1 ? fall : 0.6);
      columns(&V[(size_t)t * b * cap], b, rt, 1.0, 1.0);
    }
  auto tile = [&](const std::vector<double>& A, const std::vector<double>& B, int t, int rt) {
    std::vector<double> M((size_t)b * b, 0.0);
    for (int q = 0; q < rt; ++q)
      for (int c = 0; c < b; ++c)
        for (int a = 0; a < b; ++a) M[(size_t)c * b + a] += A[((size_t)t * cap + q) * b + a] * B[((size_t)t * cap + q) * b + c];
    return M;
  };
  std::map<int, std::vector<double>> want;
  for (int i = 2; i < nB; ++i)
    for (int j = 1; j < i; ++j) {
      auto M = tile(U, V, id(i, j), rank[id(i, j)]);
      const auto Li = tile(U, V, id(i, 0), rank[id(i, 0)]), Lj = tile(U, V, id(j, 0), rank[id(j, 0)]);
      for (int c = 0; c < b; ++c)
        for (int a = 0; a < b; ++a)
          for (int q = 0; q < b; ++q) M[(size_t)c * b + a] -= Li[(size_t)q * b + a] * Lj[(size_t)q * b + c];
      want[id(i, j)] = M;
    }
  int next = 0;
  const int grid = 2;
  const size_t slot = std::max(rc_slot_doubles(b, cap), rc_general_slot_doubles(b, cap));
  std::vector<double> scratch(grid * slot, NAN);
  std::vector<int> rlog(8), blog(8);
  std::string err;
  if (general)
    err = emu::run(dim3(grid), dim3(kGcT), 1, 0, cfg, [&] {
      k_recompress_general(n, b, 0, nB, U.data(), V.data(), rank.data(), cap, scratch.data(), slot, &next, rlog.data(),
                           blog.data(), status);
    });
  else
    err = emu::run(dim3(grid), dim3(256), 1, sizeof(RcShared<4, 4, 0>), cfg, [&] {
      k_recompress<4, 4, 1, 0>(n, b, 0, nB, U.data(), V.data(), rank.data(), cap, scratch.data(), slot, &next, rlog.data(), 0,
                               1, 3, status);
    });
  if (!err.empty()) {
    printf("error %s\n", err.c_str());
    return 0;
  }
  if (*status) {
    printf("status %d\n", *status);
    return 0;
  }
  double worst = 0.0;
  for (auto& [t, M] : want) {
    if (scale != 1.0 && t != id(2, 1) && t != id(3, 1)) continue;  // U_jk of j = 2 is of ordinary size
    const auto G = tile(U, V, t, rank[t]);
    double e = 0.0, f = 0.0;
    for (size_t q = 0; q < M.size(); ++q) {
      e += (G[q] - M[q]) / scale * ((G[q] - M[q]) / scale);
      f += M[q] / scale * (M[q] / scale);
    }
    worst = std::max(worst, e >= 0.0 ? sqrt(e / f) : 9.0);
  }
  printf("error %.17g\n", worst);
  for (int t = 0; t < ntiles; ++t) {
    printf("%d\n", rank[t]);
    for (int q = 0; q < rank[t]; ++q)
      for (int a = 0; a < b; ++a) printf("%a %a\n", U[((size_t)t * cap + q) * b + a], V[((size_t)t * cap + q) * b + a]);
  }
}
"""


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    return host_cuda.build(tmp_path_factory.mktemp("recompress"), MAIN)


# (kernel, b, rank, cap): narrow panels; ragged odd tiles; two panel blocks; cores past order 32
@pytest.mark.parametrize("general,b,rank,cap", [(0, 24, 5, 64), (0, 33, 8, 64), (0, 40, 13, 64), (0, 48, 22, 64), (1, 24, 5, 64)])
def test_thread_order_leaves_the_bits(exe, general, b, rank, cap):
    first = host_cuda.run(exe, general, b, rank, cap, 1, 0, 0, -1)
    assert first.startswith("error ") and float(first.split()[1]) <= 1e-7, first[:200]
    for seed, cta, thread in [(1, 1, 1), (2, 2, 2)]:
        assert host_cuda.run(exe, general, b, rank, cap, seed, cta, thread, -1) == first, (seed, cta, thread)


@pytest.mark.parametrize("general", [0, 1])
@pytest.mark.parametrize("thread", [0, 1])
@pytest.mark.parametrize("after", [64, 128, 224])
def test_status_set_while_a_cta_reads_it(exe, general, thread, after):
    assert host_cuda.run(exe, general, 24, 5, 64, 1, 0, thread, after, timeout=60) == "status 3\n"


@pytest.mark.parametrize("b,rank,fall,scale", [(24, 6, 1e-20, 1e-75), (40, 14, 1e-8, 1e-60), (48, 23, 3e-5, 1e-60)])
def test_columns_far_below_the_first(exe, b, rank, fall, scale):
    """Columns down to 1e-155, whose squared norms are below the smallest double that has a reciprocal."""
    out = host_cuda.run(exe, 0, b, rank, 64, 1, 0, 0, -1, fall, scale)
    assert out.startswith("error ") and float(out.split()[1]) <= 1e-7, out[:200]
