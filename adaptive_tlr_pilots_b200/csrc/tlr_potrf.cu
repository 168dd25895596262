// Cholesky of one diagonal tile per thread-block cluster, then the tile's forward-solve block.
//
// Reference: codes/17_tlr_cholesky_pilot.py:171-177 (scipy.linalg.cholesky of A_kk; a pivot that
// is not positive stops the factorization, failed_at = k) and 230-240 (z_k = L_kk^{-1} rhs_k).
//
// A cluster of G CTAs works on the column-major lower triangle of A_kk (L2-resident),
// right-looking in panels of 32 columns.  The tile is far too small to be bound by FP64 rate or bytes
// (b = 500: 42 MFLOP, 2 MB): what counts is the chain through the 32 x 32 diagonal blocks, one
// reciprocal square root, two multiply-adds and a shuffle per column (about 150 cycles), so everything
// else is kept off it:
//   * every CTA keeps the chain to itself: warp 1 solves the 32 rows below the diagonal block, warp 0
//     updates the next diagonal block with them and factors it (redundantly: identical inputs give
//     identical results, so no broadcast, and a non-positive pivot stops every CTA at the same panel).
//     The inputs are identical because CTA 0 writes what every CTA has read (the first diagonal block,
//     those 32 rows) only past a cluster barrier that follows the reads; within the panel the solved
//     rows come from each CTA's own copy in shared memory;
//   * the other rows are dealt out to the cluster and solved by substitution in registers, a thread
//     per row, with the tile's right-hand side as one more row (z_p); then rhs_rows -= X z_p (the fused
//     forward solve);
//   * the trailing matrix advances in 32 x 16 pieces on the FP64 tensor cores, one piece per warp, while
//     warp 0 factors; its fragments are read from L2 through L1 (a panel's lines enter L1 only after
//     the panel is final, because every other access to the tile bypasses L1);
//   * two cluster barriers per panel, split into arrive and wait: warp 0 runs past the first.
// Measured (one tile alone): b = 100: 109 -> 35 us, b = 250: 300 -> 72 us, b = 500: 820 -> 162 us,
// b = 1000: 8400 -> 623 us against the form that inverted each diagonal block and updated with
// CUDA-core products from a staged panel.
#include <cooperative_groups.h>

#include "tlr_device.cuh"
#include "tlr_kernels.h"

namespace cg = cooperative_groups;

namespace tlr {

namespace {

constexpr int kPB = 32;        // panel width
constexpr int kPL = kPB + 2;   // column pitch of a 32 x 32 block in shared memory (16-byte columns)

// Substitution with L11 (columns of lc, pitch kPL; dinv = 1 / diagonal): a <- a L11^{-T} for one row
// held in registers.  A column's entries are loaded while the column before is applied.
__device__ __forceinline__ void solve_row(double (&a)[kPB], const double* lc, const double* dinv) {
  double l[2][kPB], di[2];
  auto fetch = [&](int c, double (&v)[kPB], double& d) {
    d = dinv[c];
#pragma unroll
    for (int j = (c + 1) & ~1; j < kPB; j += 2) {
      const double2 x = *reinterpret_cast<const double2*>(lc + c * kPL + j);
      v[j] = x.x;
      v[j + 1] = x.y;
    }
  };
  fetch(0, l[0], di[0]);
#pragma unroll
  for (int c = 0; c < kPB; ++c) {
    if (c + 1 < kPB) fetch(c + 1, l[(c + 1) & 1], di[(c + 1) & 1]);
    a[c] *= di[c & 1];
#pragma unroll
    for (int j = c + 1; j < kPB; ++j) a[j] = fma(-a[c], l[c & 1][j], a[j]);
  }
}

// Cholesky of a 32 x 32 block by one warp, lane = row, the row in registers (the lower part; a block
// narrower than 32 is padded with the identity).  Column c of L goes to lc + c kPL, the reciprocal of
// its diagonal entry to dinv[c].  Returns 1 when a pivot is not positive.
__device__ __forceinline__ int factor_block(double (&row)[kPB], double* lc, double* dinv) {
  const int lane = threadIdx.x & 31;
  int bad = 0;
  double d = __shfl_sync(0xffffffffu, row[0], 0);
#pragma unroll
  for (int c = 0; c < kPB; ++c) {
    bad |= !(d > 0.0);
    const double rs = rsqrt(d);
    const double l = row[c] * rs;  // at lane c: sqrt(d) to two roundings
    row[c] = l;
    if (c + 1 < kPB) {
      // the next pivot from its own lane, ahead of the other updates
      d = __shfl_sync(0xffffffffu, fma(-l, l, row[c + 1]), c + 1);
      row[c + 1] = fma(-l, __shfl_sync(0xffffffffu, l, c + 1), row[c + 1]);
    }
    lc[c * kPL + lane] = l;
    if (lane == c) dinv[c] = rs;
    __syncwarp();
    if (c + 2 < kPB) {
      if (c & 1) row[c + 2] = fma(-l, lc[c * kPL + c + 2], row[c + 2]);
#pragma unroll
      for (int j = (c + 3) & ~1; j < kPB; j += 2) {
        const double2 v = *reinterpret_cast<const double2*>(lc + c * kPL + j);
        row[j] = fma(-l, v.x, row[j]);
        row[j + 1] = fma(-l, v.y, row[j + 1]);
      }
    }
  }
  return bad;
}

// Fragments of all eight k steps (the 32 panel columns) for NR 8-row tiles from row r0 of the panel rows
// P (column pitch ld, m rows below the diagonal block).
template <int NR>
__device__ __forceinline__ void panel_frag(double (&f)[8][NR], const double* P, int ld, int m, int r0) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int kk = 0; kk < 8; ++kk) {
    const double* col = P + (size_t)(4 * kk + t) * ld;
#pragma unroll
    for (int i = 0; i < NR; ++i) {
      const int r = r0 + 8 * i + g;
      f[kk][i] = r < m ? col[r] : 0.0;
    }
  }
}

// G CTAs per tile, 8 warps each: 0 the diagonal chain, 1 the 32 rows below it, 2 to 6 the other rows, 7
// the right-hand side; 1 to 7 the trailing pieces
template <int G>
__global__ void __cluster_dims__(G, 1, 1) __launch_bounds__(256)
    k_potrf_cluster(double* TLR_RESTRICT D, double* TLR_RESTRICT Linv, int n, int b, int k, double* TLR_RESTRICT rhs, double* TLR_RESTRICT z,
                    double* TLR_RESTRICT ldpart, double* TLR_RESTRICT qpart, int* TLR_RESTRICT status) {
  constexpr int NW = 8;
  cg::cluster_group cluster = cg::this_cluster();
  const int g = (int)cluster.block_rank();
  __shared__ __align__(16) double Lc[2][kPB * kPL];
  __shared__ __align__(16) double X0[kPB * kPL];  // the 32 solved rows below the diagonal block
  __shared__ __align__(16) double Cs[kPB * kPL];  // the next diagonal block
  __shared__ double dinv[2][kPB], dinv2[kPB];
  __shared__ double zp[kPB];
  __shared__ int go, fail[2];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, fg = lane >> 2, ft = lane & 3;
  // the status word is read once by rank 0 and shared through distributed shared memory, so every CTA
  // takes the same branch even when another stream writes the status meanwhile
  if (tid == 0) go = (g == 0) ? (*status == 0) : 0;
  cluster.sync();
  const int ok = *cluster.map_shared_rank(&go, 0);
  const int bk = min(b, n - k * b);
  double* A = D + (size_t)k * b * b;
  double row[kPB];  // warp 0: the current diagonal block; row warps: a row below it
  if (warp == 0) {  // every CTA reads the first diagonal block: CTA 0 writes L_11 over it past the barrier
    const int pw = min(kPB, bk);
#pragma unroll
    for (int j = 0; j < kPB; ++j)
      row[j] = (lane < pw && j <= lane) ? __ldcg(A + (size_t)j * b + lane) : (j == lane ? 1.0 : 0.0);
  }
  cluster.sync();  // and rank 0's shared memory stays valid until every CTA has read it
  if (!ok) return;
  double* rk = rhs + (size_t)k * b;
  const bool al = (b & 1) == 0;
  if (g == 0 && tid == 0) add_work(status, 8, (double)bk * bk * bk / 3.0 + (double)bk * bk, 8.0 * bk * bk);
  double ldacc = 0.0, qacc = 0.0;
  if (warp == 0) {
    const int bad = factor_block(row, Lc[0], dinv[0]);
    if (lane == 0) fail[0] = bad;
  }
  __syncthreads();
  int cur = 0;
  for (int p0 = 0; p0 < bk; p0 += kPB, cur ^= 1) {
    if (fail[cur]) {
      if (g == 0 && tid == 0) atomicCAS(status, 0, k + 1);
      return;  // every CTA of the cluster leaves at the same panel
    }
    const int pw = min(kPB, bk - p0), m = bk - p0 - pw;
    double* P = A + (size_t)p0 * b + p0 + pw;         // the panel's rows below the diagonal block
    double* T = A + (size_t)(p0 + pw) * b + p0 + pw;  // the trailing matrix
    const double* lc = Lc[cur];
    // ---- rows below: block 0 in every CTA, the others dealt out to the cluster; the right-hand side
    const int nrb = (m + 31) / 32;
    static_assert(4 * G + 1 + (G - 1) >= (G == 4 ? 8 : 32), "a row warp takes at most one block, the last none");
    const bool rhs_warp = warp == NW - 1;
    const int rb = warp == 1 ? 0 : 1 + g + G * (warp - 2), r = rb * 32 + lane;
    const bool rows = warp > 0 && !rhs_warp && rb < nrb;
    const bool act = rhs_warp ? lane == 0 : r < m;
    if (rhs_warp || rows) {
#pragma unroll
      for (int q = 0; q < kPB; ++q)
        row[q] = (act && q < pw) ? __ldcg(rhs_warp ? rk + p0 + q : P + (size_t)q * b + r) : 0.0;
      solve_row(row, lc, dinv[cur]);
      if (rhs_warp) {
        if (lane == 0) {
#pragma unroll
          for (int q = 0; q < kPB; ++q) zp[q] = row[q];
        }
      } else {
        if (warp == 1) {
#pragma unroll
          for (int q = 0; q < kPB; ++q) X0[q * kPL + lane] = row[q];  // to the tile past the barrier
        } else if (act) {
#pragma unroll
          for (int q = 0; q < kPB; ++q)
            if (q < pw) __stcg(P + (size_t)q * b + r, row[q]);
        }
      }
    } else if (warp == 6 && g == G - 1) {
      // a warp without rows: the inverse of the diagonal block for the panel solves, column `lane` of it as
      // the solution for e_lane (with the quotients 1 / L_cc, as k_diag_inv)
      dinv2[lane] = 1.0 / lc[lane * kPL + lane];
      __syncwarp();
#pragma unroll
      for (int q = 0; q < kPB; ++q) row[q] = q == lane ? 1.0 : 0.0;
      solve_row(row, lc, dinv2);
      double* o = Linv + ((size_t)k * ((b + 31) / 32) + p0 / kPB) * 1024 + lane * 32;
#pragma unroll
      for (int q = 0; q < kPB; q += 2) *reinterpret_cast<double2*>(o + q) = make_double2(row[q], row[q + 1]);
    } else if (warp == 0 && g == 0) {
#pragma unroll
      for (int j = 0; j < kPB; ++j)
        if (lane < pw && j <= lane) __stcg(A + (size_t)(p0 + j) * b + p0 + lane, row[j]);
      if (lane < pw) ldacc += log(lc[lane * kPL + lane]);
    }
    __syncthreads();
    if (rows && r < m && (warp > 1 || g == 0)) {  // rhs -= X z_p
      double s[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
      for (int q = 0; q < kPB; ++q) s[q & 3] = fma(row[q], zp[q], s[q & 3]);
      __stcg(rk + p0 + pw + r, __ldcg(rk + p0 + pw + r) - ((s[0] + s[1]) + (s[2] + s[3])));
    }
    if (rhs_warp && lane == 0) {
#pragma unroll
      for (int q = 0; q < kPB; ++q) {
        qacc = fma(row[q], row[q], qacc);
        if (g == 0 && q < pw) z[(size_t)k * b + p0 + q] = row[q];
      }
    }
    if (m == 0) break;
    cluster.barrier_arrive();  // this CTA's part of the panel is final
    if (warp == 0) {
      // ---- the next diagonal block: C - X X^T on its lower 8 x 8 tiles, then its factor
      const int pn = min(kPB, m);
      double acc[4][4][2];  // tile (columns 8 nj, rows 8 mi): lane holds column fg, rows 2 ft, 2 ft + 1
#pragma unroll
      for (int nj = 0; nj < 4; ++nj)
#pragma unroll
        for (int mi = nj; mi < 4; ++mi)
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int c = 8 * nj + fg, q = 8 * mi + 2 * ft + h;
            acc[nj][mi][h] = (q < pn && c <= q) ? __ldcg(T + (size_t)c * b + q) : 0.0;
          }
      double f[8][4];
      panel_frag<4>(f, X0, kPL, kPB, 0);
#pragma unroll
      for (int kk = 0; kk < 8; ++kk)
#pragma unroll
        for (int nj = 0; nj < 4; ++nj) {
          const double a = -f[kk][nj];
#pragma unroll
          for (int mi = nj; mi < 4; ++mi) dmma884(acc[nj][mi][0], acc[nj][mi][1], a, f[kk][mi]);
        }
      __syncwarp();
#pragma unroll
      for (int nj = 0; nj < 4; ++nj)
#pragma unroll
        for (int mi = nj; mi < 4; ++mi)
          *reinterpret_cast<double2*>(Cs + (8 * nj + fg) * kPL + 8 * mi + 2 * ft) =
              make_double2(acc[nj][mi][0], acc[nj][mi][1]);
      __syncwarp();
#pragma unroll
      for (int j = 0; j < kPB; ++j)
        row[j] = (lane < pn && j <= lane) ? Cs[j * kPL + lane] : (j == lane ? 1.0 : 0.0);
      __syncwarp();
      const int bad = factor_block(row, Lc[cur ^ 1], dinv[cur ^ 1]);
      if (lane == 0) fail[cur ^ 1] = bad;
      cluster.barrier_wait();
    } else {
      // ---- the rest of the trailing lower triangle in pieces of 32 rows x 16 columns.  Warp 4, which
      // shares warp 0's scheduler, takes pieces only where the update outweighs the diagonal chain
      const bool helper = nrb > 12;
      const int nwork = helper ? NW - 1 : NW - 2, wid = warp - 1 - (!helper && warp > 4 ? 1 : 0);
      const int npiece = warp == 4 && !helper ? 0 : nrb * (nrb + 1);
      bool waited = false;
      for (int pc = 2 + g + G * wid; pc < npiece; pc += G * nwork) {
        const int blk = pc >> 1;
        int rbk = (int)((sqrtf(8.0f * blk + 1.0f) - 1.0f) * 0.5f);
        while (rbk * (rbk + 1) / 2 > blk) --rbk;
        while ((rbk + 1) * (rbk + 2) / 2 <= blk) ++rbk;
        const int cb = blk - rbk * (rbk + 1) / 2;
        const int r0 = rbk * 32, c0 = cb * 32 + (pc & 1) * 16;
        double acc[2][4][2];
#pragma unroll
        for (int nj = 0; nj < 2; ++nj)
#pragma unroll
          for (int mi = 0; mi < 4; ++mi) {
            const int c = c0 + 8 * nj + fg, q = r0 + 8 * mi + 2 * ft;
            const double* cp = T + (size_t)c * b + q;
            if (al && c < m && q + 1 < m) {
              const double2 v = __ldcg(reinterpret_cast<const double2*>(cp));
              acc[nj][mi][0] = v.x;
              acc[nj][mi][1] = v.y;
            } else {
              acc[nj][mi][0] = c < m && q < m ? __ldcg(cp) : 0.0;
              acc[nj][mi][1] = c < m && q + 1 < m ? __ldcg(cp + 1) : 0.0;
            }
          }
        if (!waited) cluster.barrier_wait();  // the panel is final
        waited = true;
        double fa[8][2], fb[8][4];
        if (cb == 0) panel_frag<2>(fa, X0, kPL, kPB, c0);
        else panel_frag<2>(fa, P, b, m, c0);
        panel_frag<4>(fb, P, b, m, r0);
#pragma unroll
        for (int kk = 0; kk < 8; ++kk)
#pragma unroll
          for (int nj = 0; nj < 2; ++nj) {
            const double a = -fa[kk][nj];
#pragma unroll
            for (int mi = 0; mi < 4; ++mi) dmma884(acc[nj][mi][0], acc[nj][mi][1], a, fb[kk][mi]);
          }
#pragma unroll
        for (int nj = 0; nj < 2; ++nj)
#pragma unroll
          for (int mi = 0; mi < 4; ++mi) {
            const int c = c0 + 8 * nj + fg, q = r0 + 8 * mi + 2 * ft;
            double* cp = T + (size_t)c * b + q;
            if (c >= m) continue;
            if (al && q + 1 < m && q >= c)
              __stcg(reinterpret_cast<double2*>(cp), make_double2(acc[nj][mi][0], acc[nj][mi][1]));
            else {
              if (q < m && q >= c) __stcg(cp, acc[nj][mi][0]);
              if (q + 1 < m && q + 1 >= c) __stcg(cp + 1, acc[nj][mi][1]);
            }
          }
      }
      if (!waited) cluster.barrier_wait();
      if (rhs_warp && g == 0 && lane < m) {  // every CTA has read these rows
#pragma unroll
        for (int q = 0; q < kPB; ++q)
          if (q < pw) __stcg(P + (size_t)q * b + lane, X0[q * kPL + lane]);
      }
    }
    cluster.sync();  // the trailing matrix and the next diagonal block's factor are in place
  }
  if (g == 0) {
    if (warp == 0) {
      ldacc = warp_sum(ldacc);
      if (lane == 0) ldpart[k] = 2.0 * ldacc;
    } else if (warp == NW - 1 && lane == 0) {
      qpart[k] = qacc;
    }
  }
}

}  // namespace

int launch_potrf(double* D, double* Linv, int n, int b, int k, double* rhs, double* z, double* ldpart, double* qpart,
                 int* status, cudaStream_t s) {
  // four CTAs share the rows and the trailing pieces of the smaller tiles (one CTA takes 41 us at
  // b = 100 against 35: its chain and its update meet on one SM), eight those past 256 rows
  if (b <= 256) k_potrf_cluster<4><<<4, 256, 0, s>>>(D, Linv, n, b, k, rhs, z, ldpart, qpart, status);
  else k_potrf_cluster<8><<<8, 256, 0, s>>>(D, Linv, n, b, k, rhs, z, ldpart, qpart, status);
  return (int)cudaGetLastError();
}

}  // namespace tlr
