"""k_potrf_cluster under every order of its CTAs: the factor, z, the block inverses and the other outputs have the
same bits whichever CTA of the cluster runs ahead (on the host, see emu/cuda_emu.h), and the factor is
NumPy's within FP64 rounding times the condition of these tiles."""
import numpy as np
import pytest

import host_cuda

MAIN = r"""
#include "tlr_potrf.cu"
#include "tlr_device.cuh"
// usage: main G b seed cta_order thread_order -> the outputs as text
int main(int argc, char** argv) {
  const int G = atoi(argv[1]), b = atoi(argv[2]);
  emu::Config cfg;
  cfg.seed = (unsigned)atoi(argv[3]);
  cfg.cta = (emu::Order)atoi(argv[4]);
  cfg.thread = (emu::Order)atoi(argv[5]);
  const int np = (b + 31) / 32;
  std::vector<double> D((size_t)b * b), Linv((size_t)np * 1024, 7.0), rhs(b), z(b), ld(1), qp(1);
  for (int c = 0; c < b; ++c)
    for (int r = 0; r < b; ++r) {
      const double h = abs(r - c) / 20.0;
      D[(size_t)c * b + r] = r < c ? NAN : (1.0 + h) * exp(-h) + (r == c ? 0.05 : 0.0);
    }
  for (int r = 0; r < b; ++r) rhs[r] = sin(0.3 * r);
  std::vector<char> ctl(tlr::kControlBytes, 0);
  int* status = reinterpret_cast<int*>(ctl.data());
  auto body = [&] {
    if (G == 4) tlr::k_potrf_cluster<4>(D.data(), Linv.data(), b, b, 0, rhs.data(), z.data(), ld.data(), qp.data(), status);
    else tlr::k_potrf_cluster<8>(D.data(), Linv.data(), b, b, 0, rhs.data(), z.data(), ld.data(), qp.data(), status);
  };
  const std::string err = emu::run(dim3(G), dim3(256), G, 0, cfg, body);
  if (!err.empty()) {
    printf("error %s\n", err.c_str());
    return 0;
  }
  printf("%d %a %a\n", *status, ld[0], qp[0]);
  for (int c = 0; c < b; ++c)
    for (int r = c; r < b; ++r) printf("%a\n", D[(size_t)c * b + r]);
  for (double v : z) printf("%a\n", v);
  for (double v : Linv) printf("%a\n", v);
}
"""


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    return host_cuda.build(tmp_path_factory.mktemp("potrf"), MAIN)


@pytest.mark.parametrize("G,b", [(4, 30), (8, 32), (4, 70), (4, 129), (8, 161)])
def test_cluster_order_leaves_the_bits(exe, G, b):
    first = host_cuda.run(exe, G, b, 1, 0, 0)
    assert first.startswith("0 "), first[:200]
    i = np.arange(b)
    h = np.abs(i[:, None] - i[None, :]) / 20.0
    A = (1 + h) * np.exp(-h) + 0.05 * np.eye(b)
    L = np.linalg.cholesky(A)
    got = [float.fromhex(v) for v in first.split("\n")[1:1 + b * (b + 1) // 2]]
    # backward error b eps ||A||, condition about ||A|| / 0.05 < 2000
    assert np.abs(np.array(got) - L.T[np.triu_indices(b)]).max() <= 2000 * b * 2.3e-16 * 2
    # CTA 0 first, last, and CTAs and warps in random order
    for seed, cta, thread in [(1, 1, 0), (1, 0, 1), (2, 2, 2), (3, 2, 2)]:
        assert host_cuda.run(exe, G, b, seed, cta, thread) == first, (seed, cta, thread)
