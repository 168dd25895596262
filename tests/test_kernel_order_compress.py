"""k_orth and k_finalize on the host (emu/cuda_emu.h) under every order of their threads: two covariance tiles (one
ragged) at sketch widths with the reflectors in shared memory and in global scratch, and with cores
of one warp and of the whole CTA.  The bits do not depend on the order; the basis is orthonormal and the pair
meets the rule; and a status word that another CTA sets while a CTA's threads read it ends the CTA as a whole."""
import pytest

import host_cuda

MAIN = r"""
#include "tlr_compress.cu"
using namespace tlr;
// usage: main b k in_smem scale seed cta_order thread_order flip_orth flip_finalize [threshold]
int main(int argc, char** argv) {
  const int b = atoi(argv[1]), k = atoi(argv[2]), in_smem = atoi(argv[3]);
  const double scale = atof(argv[4]);
  emu::Config cfg;
  cfg.seed = (unsigned)atoi(argv[5]);
  cfg.cta = (emu::Order)atoi(argv[6]);
  cfg.thread = (emu::Order)atoi(argv[7]);
  cfg.flip_value = 3;
  const int n = 2 * b + b / 2, nc = 2, ldp = kMaxSketch, cap = 64;
  std::vector<char> ctl(kControlBytes, 0);
  int* status = reinterpret_cast<int*>(ctl.data());
  cfg.flip_word = status;
  auto* prm = const_cast<EvalParams*>(eval_params(status));
  prm->rule_fixed = 1;
  prm->thr_rel = argc > 10 ? atof(argv[10]) : 1e-7;
  const int ti[] = {2, 2}, tj[] = {0, 1};  // storage tiles 0 and 1; tile row 2 is ragged
  int need[] = {1, 1}, rank[] = {-1, -1};
  auto T = [&](int c, int a, int q) { return scale / (1.0 + 0.04 * (ti[c] * b + a - tj[c] * b - q)); };
  std::vector<double> Z((size_t)nc * b * ldp, 0.0), C(Z), U((size_t)nc * b * cap, 0.0), V(U);
  const size_t slot = orth_slot_doubles(b, kMaxSketch);
  std::vector<double> g(nc * slot, NAN), gsv((size_t)nc * 2 * ldp * ldp, NAN), parts(nc), fparts(nc), tail(2), fro(2);
  int rlog[2] = {0, 0}, blog[2] = {0, 0};
  auto bi = [&](int c) { return std::min(b, n - ti[c] * b); };
  for (int c = 0; c < nc; ++c)
    for (int q = 0; q < k; ++q) {
      std::vector<double> y(b, 0.0);
      for (int a = 0; a < bi(c); ++a)
        for (int w = 0; w < b; ++w) y[a] += T(c, a, w) * omega_entry(c, w, q);
      for (int w = 0; w < b; ++w) {
        double s = 0.0;
        for (int a = 0; a < bi(c); ++a) s += T(c, a, w) * y[a];
        Z[((size_t)c * ldp + q) * b + w] = s;
      }
    }
  using S = Side<4, 4>;
  constexpr int kLdx = S::kLdx;
  const size_t core = ((size_t)k * (k + 1) + 1) / 2 * 2, pan = std::max<size_t>((size_t)kLdx * (in_smem ? k : 8), k * k);
  cfg.flip_after = atoi(argv[8]);
  std::string err = emu::run(dim3(nc), dim3(128), 1, sizeof(PanelShared<4, 4>) + pan * 8, cfg, [&] {
    k_orth<4, 4>(Z.data(), n, b, k, ldp, 0, tj, need, g.data(), slot, in_smem, status);
  });
  double orth = 0.0;
  if (err.empty() && !*status) {
    for (int c = 0; c < nc; ++c)
      for (int p = 0; p < std::min(k, b); ++p)
        for (int q = 0; q <= p; ++q) {
          double s = p == q ? -1.0 : 0.0;
          for (int w = 0; w < b; ++w) s += Z[((size_t)c * ldp + p) * b + w] * Z[((size_t)c * ldp + q) * b + w];
          orth = std::max(orth, s == s ? fabs(s) : 9.0);
        }
    for (int c = 0; c < nc; ++c) {
      for (int q = 0; q < k; ++q)
        for (int a = 0; a < bi(c); ++a) {
          double s = 0.0;
          for (int w = 0; w < b; ++w) s += T(c, a, w) * Z[((size_t)c * ldp + q) * b + w];
          C[((size_t)c * ldp + q) * b + a] = s;
        }
      for (int a = 0; a < bi(c); ++a)
        for (int w = 0; w < b; ++w) {
          double e = T(c, a, w);
          fparts[c] += e * e;
          for (int q = 0; q < k; ++q) e -= C[((size_t)c * ldp + q) * b + a] * Z[((size_t)c * ldp + q) * b + w];
          parts[c] += e * e;
        }
    }
    cfg.flip_after = atoi(argv[9]);
    err = emu::run(dim3(nc), dim3(128), 1, sizeof(PanelShared<4, 4>) + (core + pan) * 8, cfg, [&] {
      k_finalize<4, 4>(n, b, k, ldp, cap, 4, 0, ti, tj, need, Z.data(), C.data(), parts.data(), fparts.data(), 1, g.data(), slot,
                       gsv.data(), U.data(), V.data(), rank, 1, in_smem, rlog, tail.data(), fro.data(), blog, status);
    });
  }
  if (!err.empty()) {
    printf("error %s\n", err.c_str());
    return 0;
  }
  if (*status) {
    printf("status %d\n", *status);
    return 0;
  }
  double worst = 0.0;
  for (int c = 0; c < nc; ++c) {
    double e2 = 0.0;
    for (int a = 0; a < bi(c); ++a)
      for (int w = 0; w < b; ++w) {
        double e = T(c, a, w) / scale;
        for (int q = 0; q < rank[c]; ++q) e -= U[((size_t)c * cap + q) * b + a] / scale * V[((size_t)c * cap + q) * b + w];
        e2 += e * e;
      }
    worst = std::max(worst, sqrt(e2) * (scale / fro[c]));
    if (!(e2 >= 0.0)) worst = 9.0;
  }
  double vorth = 0.0;
  for (int c = 0; c < nc; ++c)
    for (int p = 0; p < rank[c]; ++p)
      for (int q = 0; q <= p; ++q) {
        double s = p == q ? -1.0 : 0.0;
        for (int w = 0; w < b; ++w) s += V[((size_t)c * cap + p) * b + w] * V[((size_t)c * cap + q) * b + w];
        vorth = std::max(vorth, s == s ? fabs(s) : 9.0);
      }
  printf("error %.17g orth %.17g ranks %d %d V %.17g\n", worst, orth, rank[0], rank[1], vorth);
  for (int c = 0; c < nc; ++c)
    for (int q = 0; q < rank[c]; ++q)
      for (int w = 0; w < b; ++w) printf("%a %a\n", U[((size_t)c * cap + q) * b + w], V[((size_t)c * cap + q) * b + w]);
}
"""


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    return host_cuda.build(tmp_path_factory.mktemp("compress"), MAIN)


def _check(out):
    w = out.split()
    assert w[0] == "error" and w[2] == "orth", out[:200]
    assert float(w[1]) <= 1e-7          # the rule's threshold
    assert float(w[3]) <= 1e-13         # k eps with a margin
    assert 0 < int(w[5]) <= int(w[6]) < 16


@pytest.mark.parametrize("b,k,in_smem", [(24, 16, 1), (33, 32, 1), (70, 32, 0), (40, 64, 0), (70, 64, 0)])
def test_thread_order_leaves_the_bits(exe, b, k, in_smem):
    first = host_cuda.run(exe, b, k, in_smem, 1, 1, 0, 0, -1, -1)
    _check(first)
    for seed, cta, thread in [(1, 1, 1), (2, 2, 2)]:
        assert host_cuda.run(exe, b, k, in_smem, 1, seed, cta, thread, -1, -1) == first, (seed, cta, thread)


@pytest.mark.parametrize("thread", [0, 1])
@pytest.mark.parametrize("orth,finalize", [(32, -1), (96, -1), (-1, 32), (-1, 96), (-1, 160)])
def test_status_set_while_a_cta_reads_it(exe, thread, orth, finalize):
    assert host_cuda.run(exe, 24, 16, 1, 1, 1, 0, thread, orth, finalize, timeout=60) == "status 3\n"


@pytest.mark.parametrize("k,in_smem", [(16, 1), (32, 1), (64, 0)])
@pytest.mark.parametrize("scale", [1e-62, 1e-68, 1e-72, 1e70])
def test_tiles_of_any_size(exe, k, in_smem, scale):
    """The columns of T^T T P are squares of the tile's entries, and their norms are squared once more: the basis
    and the pair are those of a tile of ordinary size."""
    _check(host_cuda.run(exe, 48, k, in_smem, scale, 1, 0, 0, -1, -1))


@pytest.mark.parametrize("k", [24, 32, 64])
def test_right_vectors_at_rounding_level(exe, k):
    """A threshold below 1e-14 of the tile keeps singular values at rounding level: their right vectors are
    orthonormal too (the recompression relies on it).  Bound: k eps with a margin."""
    w = host_cuda.run(exe, 24, k, int(k <= 32), 1, 1, 0, 0, -1, -1, 1e-15).split()
    assert w[0] == "error" and float(w[8]) <= 1e-13, w[:10]
