// Backward pass: gradient of the TLR log-likelihood in (sigma2, range, eta).
//
// No counterpart in the reference (it has no gradient code; its only derivatives are finite
// differences, codes/15_pilot_standard_errors.py:21-31).  With Sigma_t = L L^T the TLR factor of
// the forward pass (ranks frozen), the gradient is
//     dl/dtheta = 1/2 alpha^T dSigma alpha - 1/2 tr(Z dSigma),  alpha = Sigma_t^{-1} y,  Z = Sigma_t^{-1}
// with Z's tiles from the selected-inversion (Takahashi) recurrence on the tile factor, i.e. the
// blocked Cholesky adjoint with the truncations passed through unchanged (oracle:
// oracle/tlr_oracle.py:tlr_loglik_grad).  Reverse step m, with Vp = L_mm^{-T} [V_jm]_{j>m}:
//     Z_im = -sum_{j>m} (Z_ij U_jm) Vp_j^T                       (i > m; Z_ij = Z_ji^T for j > i)
//     Z_mm = L_mm^{-T} L_mm^{-1} - sum_{j>m} (Z_jm^T U_jm) Vp_j^T
// The products Z_ij U_jm are formed once, when Z_ij is, for every m < j, so each dense Z tile is
// read from HBM a fixed number of times.  dSigma tiles are regenerated from the sites inside the
// contraction kernel, never stored.
//
// With C_im = [Z_ij U_jm]_{j>m} (b_i x R_m, contiguous) these are single GEMMs of inner dimension
// R_m = sum_j r_jm; the C blocks are written when Z_ij is formed (column-scattered GEMM output).
// Kernels: a batched FP64 GEMM with optional column scatter, a batched lower-triangular
// inverse (L^{-1} of every diagonal tile), the TLR backward solve for alpha, and the fused dSigma
// generation + contraction.
#include <cooperative_groups.h>

#include "tlr_device.cuh"
#include "tlr_kernels.h"

namespace cg = cooperative_groups;

namespace tlr {

// ----------------------------------------------------------------------------------------
// Batched FP64 GEMM  C = alpha op(A) op(B) + beta C on the FP64 tensor cores (mma m8n8k4, exact
// FP64 fused multiply-adds).  WM x WN warps of 32 x 8 NJ outputs each (NJ = 4: a k step of four reads eight
// fragments for sixteen products), K in slices of 16 through three stages of shared memory filled by
// cp.async (16 bytes where the operand's rows allow, else 8).  A slice keeps the operand's own order:
// [k][m] when the m index is contiguous in memory, [m][k] when k is; both pitches put a fragment's lanes
// in distinct banks.  A job may scatter its output columns: column n then goes to ccol[n] (leading rows
// contiguous) instead of C + n ldc.
// 128 x 64 tiles (two CTAs an SM) where the launch has two waves of them, 64 x 32 (four warps) where it
// has not: one 500 x 500 x 500 product is 32 of the large tiles.  Bound by the FP64 tensor pipe (17 cycles
// a step and scheduler); the backward pass's products at N = 50,000, b = 500: 104 -> 71 ms against 64 x 64
// tiles staged through registers.
constexpr int kDgK = 16, kDgStages = 3, kDgPk = kDgK + 4;
template <int WM, int WN, int NJ>
struct DgShape {
  static constexpr int kM = 32 * WM, kN = 8 * NJ * WN, kT = 32 * WM * WN;
  static constexpr int kPm = kM + 4, kPn = kN + 4;                  // pitches of [k][m], [k][n]; kDgPk of [.][k]
  static constexpr int kA = kM * kDgPk, kB = kN * kDgPk;            // doubles per stage (the larger layout)
  static constexpr size_t kSmem = (size_t)kDgStages * (kA + kB) * sizeof(double);
  static_assert(kA >= kDgK * kPm && kB >= kDgK * kPn, "stage sizes");
};
using DgLarge = DgShape<4, 2, 4>;
using DgSmall = DgShape<2, 2, 2>;

__device__ __forceinline__ void cp_async8(void* smem, const void* gmem, int src_bytes) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(s), "l"(gmem), "r"(src_bytes) : "memory");
}

// One operand's slice to shared memory: `rows` x 16 (rows: the m or n index, r0 + row below nr), element
// (row, k) at src[row ld + k] when kcont, else src[k ld + row].
template <int ROWS, int THREADS>
__device__ __forceinline__ void dg_slice(double* dst, const double* src, int ld, bool kcont, bool vec, int r0, int nr,
                                         int k0, int nk) {
  constexpr int P = ROWS + 4;
#pragma unroll
  for (int e = threadIdx.x; e < ROWS * kDgK / 2; e += THREADS) {
    const int row = kcont ? e / (kDgK / 2) : 2 * (e % (ROWS / 2)), k = kcont ? 2 * (e % (kDgK / 2)) : e / (ROWS / 2);
    const int gr = r0 + row, gk = k0 + k;
    double* d = dst + (kcont ? row * kDgPk + k : k * P + row);
    const double* g = src + (kcont ? (size_t)gr * ld + gk : (size_t)gk * ld + gr);
    const int have = gr >= nr || gk >= nk ? 0 : min(2, kcont ? nk - gk : nr - gr);  // elements inside
    if (vec) {
      cp_async16(d, have ? g : src, 8 * have);
    } else {
      cp_async8(d, have > 0 ? g : src, have > 0 ? 8 : 0);
      cp_async8(d + 1, have > 1 ? g + 1 : src, have > 1 ? 8 : 0);
    }
  }
}

template <int WM, int WN, int NJ, bool TA, bool TB>
__device__ __forceinline__ void dgemm_tile(const GemmJob& jb, int m0, int n0, double* sm) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  using S = DgShape<WM, WN, NJ>;
  const int wm0 = (warp % WM) * 32, wn0 = (warp / WM) * 8 * NJ;
  const bool va = ((reinterpret_cast<size_t>(jb.A) | ((size_t)jb.lda * 8)) & 15) == 0;
  const bool vb = ((reinterpret_cast<size_t>(jb.B) | ((size_t)jb.ldb * 8)) & 15) == 0;
  double acc[4][NJ][2];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < NJ; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
  const int nk = (jb.K + kDgK - 1) / kDgK;
  auto issue = [&](int s) {
    if (s < nk) {
      double* st = sm + (size_t)(s % kDgStages) * (S::kA + S::kB);
      dg_slice<S::kM, S::kT>(st, jb.A, jb.lda, TA, va, m0, jb.M, s * kDgK, jb.K);
      dg_slice<S::kN, S::kT>(st + S::kA, jb.B, jb.ldb, !TB, vb, n0, jb.N, s * kDgK, jb.K);
    }
    cp_async_commit();  // one group per slice, empty past the end
  };
  for (int s = 0; s < kDgStages - 1; ++s) issue(s);
  for (int s = 0; s < nk; ++s) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(kDgStages - 2) : "memory");
    __syncthreads();  // slice s is here, and every warp is done with the stage that the next copy fills
    issue(s + kDgStages - 1);
    const double* As = sm + (size_t)(s % kDgStages) * (S::kA + S::kB);
    const double* Bs = As + S::kA;
#pragma unroll
    for (int kq = 0; kq < kDgK / 4; ++kq) {
      double a[4], b[NJ];
#pragma unroll
      for (int i = 0; i < 4; ++i)
        a[i] = TA ? As[(wm0 + 8 * i + g) * kDgPk + 4 * kq + t] : As[(4 * kq + t) * S::kPm + wm0 + 8 * i + g];
#pragma unroll
      for (int j = 0; j < NJ; ++j)
        b[j] = TB ? Bs[(4 * kq + t) * S::kPn + wn0 + 8 * j + g] : Bs[(wn0 + 8 * j + g) * kDgPk + 4 * kq + t];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < NJ; ++j) dmma884(acc[i][j][0], acc[i][j][1], a[i], b[j]);
    }
  }
#pragma unroll
  for (int j = 0; j < NJ; ++j)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int gn = n0 + wn0 + 8 * j + 2 * t + h;
      if (gn >= jb.N) continue;
      double* cc = jb.ccol ? jb.ccol[gn] : jb.C + (size_t)gn * jb.ldc;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int gm = m0 + wm0 + 8 * i + g;
        if (gm >= jb.M) continue;
        const double v = jb.alpha * acc[i][j][h];
        cc[gm] = (jb.beta == 0.0) ? v : fma(jb.beta, cc[gm], v);
      }
    }
}

template <int WM, int WN, int NJ>
__global__ void __launch_bounds__(32 * WM * WN, 16 / (WM * WN)) k_dgemm_batched(const GemmJob* TLR_RESTRICT jobs,
                                                                                 const int* TLR_RESTRICT status,
                                                                                 int kind) {
  if (*status != 0) return;
  using S = DgShape<WM, WN, NJ>;
  const GemmJob jb = jobs[blockIdx.z];
  const int m0 = blockIdx.y * S::kM, n0 = blockIdx.x * S::kN;
  if (m0 >= jb.M || n0 >= jb.N) return;
  extern __shared__ __align__(16) double dg_smem[];
  if (jb.transA) {
    if (jb.transB) dgemm_tile<WM, WN, NJ, true, true>(jb, m0, n0, dg_smem);
    else dgemm_tile<WM, WN, NJ, true, false>(jb, m0, n0, dg_smem);
  } else {
    if (jb.transB) dgemm_tile<WM, WN, NJ, false, true>(jb, m0, n0, dg_smem);
    else dgemm_tile<WM, WN, NJ, false, false>(jb, m0, n0, dg_smem);
  }
  if (threadIdx.x == 0) {
    const int mt = min(S::kM, jb.M - m0), nt = min(S::kN, jb.N - n0);
    add_work(status, kind, 2.0 * jb.K * mt * nt, 8.0 * ((double)mt * nt + (double)(mt + nt) * jb.K));
  }
}

int launch_dgemm_batched(const GemmJob* jobs, int njobs, int max_m, int max_n, const int* status, int kind,
                         cudaStream_t s) {
  if (njobs <= 0) return 0;
  auto blocks = [](int n, int per) { return (unsigned)((n + per - 1) / per); };
  const long large = (long)blocks(max_n, DgLarge::kN) * blocks(max_m, DgLarge::kM) * njobs;
  if (large >= 4 * kSms) {  // two waves of two CTAs an SM
    cudaFuncSetAttribute(k_dgemm_batched<4, 2, 4>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)DgLarge::kSmem);
    k_dgemm_batched<4, 2, 4><<<dim3(blocks(max_n, DgLarge::kN), blocks(max_m, DgLarge::kM), (unsigned)njobs), DgLarge::kT,
                               DgLarge::kSmem, s>>>(jobs, status, kind);
  } else {
    cudaFuncSetAttribute(k_dgemm_batched<2, 2, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)DgSmall::kSmem);
    k_dgemm_batched<2, 2, 2><<<dim3(blocks(max_n, DgSmall::kN), blocks(max_m, DgSmall::kM), (unsigned)njobs), DgSmall::kT,
                               DgSmall::kSmem, s>>>(jobs, status, kind);
  }
  return (int)cudaGetLastError();
}

// ----------------------------------------------------------------------------------------
// Li_k = L_kk^{-1} for every diagonal tile: blocked forward substitution on the identity, one
// CTA per (tile, 32-column block); columns are independent.
__global__ void __launch_bounds__(256) k_tri_inv(const double* TLR_RESTRICT D, double* TLR_RESTRICT Li, int n,
                                                int b, const int* TLR_RESTRICT status) {
  if (*status != 0) return;
  const int k = blockIdx.y, cb = blockIdx.x;
  const int bk = min(b, n - k * b);
  const int c0 = cb * 32;
  if (c0 >= bk) return;
  const int cw = min(32, bk - c0);
  const double* L = D + (size_t)k * b * b;
  double* X = Li + (size_t)k * b * b;
  __shared__ double L11[32][33];
  __shared__ double Xp[32][33];
  const int tid = threadIdx.x;
  if (tid == 0 && cb == 0) add_work(status, 13, (double)bk * bk * bk / 3.0, 16.0 * bk * bk);
  // X[:, c0:c0+cw] = identity columns
  for (int c = 0; c < cw; ++c)
    for (int a = tid; a < bk; a += 256) X[(size_t)(c0 + c) * b + a] = (a == c0 + c) ? 1.0 : 0.0;
  __syncthreads();
  for (int p0 = (c0 / 32) * 32; p0 < bk; p0 += 32) {
    const int pw = min(32, bk - p0);
    for (int e = tid; e < 32 * 32; e += 256) {
      const int a = e & 31, c = e >> 5;
      L11[a][c] = (a < pw && c < pw && a >= c) ? L[(size_t)(p0 + c) * b + p0 + a] : 0.0;
    }
    __syncthreads();
    if (tid < cw) {
      double* xc = X + (size_t)(c0 + tid) * b + p0;
      double x[32];
#pragma unroll
      for (int a = 0; a < 32; ++a) x[a] = (a < pw) ? xc[a] : 0.0;
#pragma unroll
      for (int a = 0; a < 32; ++a) {
        if (a < pw) {
          double s = x[a];
#pragma unroll
          for (int c = 0; c < a; ++c) s -= L11[a][c] * x[c];
          x[a] = s / L11[a][a];
        }
      }
#pragma unroll
      for (int a = 0; a < 32; ++a)
        if (a < pw) { xc[a] = x[a]; Xp[a][tid] = x[a]; }
    }
    __syncthreads();
    for (int row = p0 + pw + tid; row < bk; row += 256) {
      double l[32];
#pragma unroll
      for (int c = 0; c < 32; ++c) l[c] = (c < pw) ? L[(size_t)(p0 + c) * b + row] : 0.0;
      for (int q = 0; q < cw; ++q) {
        double s = 0.0;
#pragma unroll
        for (int c = 0; c < 32; ++c) s = fma(l[c], Xp[c][q], s);
        X[(size_t)(c0 + q) * b + row] -= s;
      }
    }
    __syncthreads();
  }
}

int launch_tri_inv(const double* D, double* Li, int n, int b, int nB, const int* status, cudaStream_t s) {
  dim3 grid((unsigned)((b + 31) / 32), (unsigned)nB);
  k_tri_inv<<<grid, 256, 0, s>>>(D, Li, n, b, status);
  return (int)cudaGetLastError();
}

// ----------------------------------------------------------------------------------------
// Column-block copies (gathers of U / V factors into contiguous panels).
__global__ void k_copy_cols(const CopyJob* TLR_RESTRICT jobs, const int* TLR_RESTRICT status) {
  if (*status != 0) return;
  const CopyJob jb = jobs[blockIdx.y];
  const size_t total = (size_t)jb.rows * jb.cols;
  for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (size_t)gridDim.x * blockDim.x) {
    const int r = (int)(e % jb.rows), c = (int)(e / jb.rows);
    jb.dst[(size_t)c * jb.ldd + r] = jb.src[(size_t)c * jb.lds + r];
  }
}

int launch_copy_cols(const CopyJob* jobs, int njobs, const int* status, cudaStream_t s) {
  if (njobs <= 0) return 0;
  dim3 grid(32u, (unsigned)njobs);
  k_copy_cols<<<grid, 256, 0, s>>>(jobs, status);
  return (int)cudaGetLastError();
}

// ----------------------------------------------------------------------------------------
// alpha_m = L_mm^{-T} (z_m - sum_{i>m} V_im (U_im^T alpha_i))   (codes/17_tlr_cholesky_pilot.py:243-256
// restated for one block row).  One cluster of kAC CTAs, three phases separated by the cluster
// barrier: t = [U_im^T alpha_i]_{i>m} (one warp per entry, lanes over rows); rhs = z_m - sum_i
// V_im t_i (rows split across the cluster, four threads per row); alpha_m = L_mm^{-T} rhs (one
// warp per output, lanes over the column of L_mm^{-1}).  t and rhs live in `work` (L2).
constexpr int kAC = 8;

__global__ void __cluster_dims__(kAC, 1, 1) __launch_bounds__(256)
    k_alpha_step(int n, int b, int m, int nB, const double* TLR_RESTRICT U, const double* TLR_RESTRICT V,
                 const int* TLR_RESTRICT rank, int cap, const double* TLR_RESTRICT Li, const double* TLR_RESTRICT z,
                 double* TLR_RESTRICT alpha, double* TLR_RESTRICT work, const int* TLR_RESTRICT status) {
  cg::cluster_group cluster = cg::this_cluster();
  const int g = (int)cluster.block_rank();
  __shared__ int go;
  __shared__ int off[1025];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) go = (g == 0) ? (*status == 0) : 0;
  cluster.sync();
  const int ok = *cluster.map_shared_rank(&go, 0);
  cluster.sync();  // rank 0's shared memory stays valid until every CTA has read it
  if (!ok) return;
  const int bm = min(b, n - m * b);
  double* rhs = work;      // b
  double* tq = work + b;   // sum_{i>m} r_im
  const int R = block_offsets(off, nB - m - 1, [&](int q) { return rank[(m + 1 + q) * (m + q) / 2 + m]; });
  const int nw = kAC * 8, gw = g * 8 + warp;
  for (int e = gw; e < R; e += nw) {
    int lo = 0, hi = nB - m - 1;  // off[lo] <= e < off[lo + 1]
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (off[mid] <= e) lo = mid; else hi = mid;
    }
    const int i = m + 1 + lo, q = e - off[lo];
    const int bi = min(b, n - i * b);
    const double* u = U + ((size_t)i * (i - 1) / 2 + m) * b * cap + (size_t)q * b;
    const double* ai = alpha + (size_t)i * b;
    double sacc = 0.0;
    for (int a = lane; a < bi; a += 32) sacc = fma(u[a], ai[a], sacc);
    sacc = warp_sum(sacc);
    if (lane == 0) tq[e] = sacc;
  }
  cluster.sync();
  {
    const int per = (bm + kAC - 1) / kAC;
    const int r0 = g * per, r1 = min(bm, r0 + per);
    const int quarter = tid & 3;
    for (int base = r0; base < r1; base += 64) {  // the same trip count in every thread (shuffles)
      const int a = base + (tid >> 2);
      const bool act = a < r1;
      double sacc = 0.0;
      if (act)
        for (int lo = 0; lo < nB - m - 1; ++lo) {
          const int i = m + 1 + lo, r = off[lo + 1] - off[lo];
          const double* v = V + ((size_t)i * (i - 1) / 2 + m) * b * cap;
          for (int q = quarter; q < r; q += 4) sacc = fma(v[(size_t)q * b + a], tq[off[lo] + q], sacc);
        }
      sacc += __shfl_xor_sync(0xffffffffu, sacc, 1);
      sacc += __shfl_xor_sync(0xffffffffu, sacc, 2);
      if (act && quarter == 0) rhs[a] = z[(size_t)m * b + a] - sacc;
    }
  }
  cluster.sync();
  // alpha_m = L_mm^{-T} rhs: (Li^T rhs)_a = sum_{c >= a} Li[c][a] rhs[c]
  const double* L = Li + (size_t)m * b * b;
  for (int a = gw; a < bm; a += nw) {
    const double* col = L + (size_t)a * b;
    double sacc = 0.0;
    for (int c = a + lane; c < bm; c += 32) sacc = fma(col[c], rhs[c], sacc);
    sacc = warp_sum(sacc);
    if (lane == 0) alpha[(size_t)m * b + a] = sacc;
  }
}

int launch_alpha_step(int n, int b, int m, int nB, const double* U, const double* V, const int* rank, int cap,
                      const double* Li, const double* z, double* alpha, double* work, const int* status,
                      cudaStream_t s) {
  k_alpha_step<<<kAC, 256, 0, s>>>(n, b, m, nB, U, V, rank, cap, Li, z, alpha, work, status);
  return (int)cudaGetLastError();
}

// ----------------------------------------------------------------------------------------
// Contraction of dSigma (regenerated) with Sbar = 1/2 (alpha_i alpha_m^T - Z_im) over the tiles
// (i, m), i >= m, of block column m; weight 2 for off-diagonal tiles.  One CTA per 128 x 32 block, sixteen
// entries a thread (a column's rows, so Z is read along its columns), then one reduction of the three sums;
// partial sums [3] per CTA into part (fixed slots: deterministic final reduction).  Bound by the FP64
// square root and exponential of every entry; N = 50,000: 11.9 -> 9.5 ms per evaluation against four
// entries a thread and three block sums.
constexpr int kDtRows = 128, kDtCols = 32;

int dtrace_parts(int b) { return ((b + kDtRows - 1) / kDtRows) * ((b + kDtCols - 1) / kDtCols); }

__global__ void __launch_bounds__(256) k_dtrace_step(const double* TLR_RESTRICT xy, int n, int b, int m, int nB,
                                                    double sigma2, double inv_range, int nu5, double eta,
                                                    const double* TLR_RESTRICT Zbuf,
                                                    const double* TLR_RESTRICT alpha, double* TLR_RESTRICT part,
                                                    const int* TLR_RESTRICT status) {
  if (*status != 0) return;
  const int ncb = (b + kDtCols - 1) / kDtCols, per_tile = ((b + kDtRows - 1) / kDtRows) * ncb;
  const int i = m + blockIdx.x / per_tile;
  const int blk = blockIdx.x % per_tile;
  const int r0 = (blk / ncb) * kDtRows, c0 = (blk % ncb) * kDtCols;
  double* out = part + (size_t)blockIdx.x * 3;
  const int bi = min(b, n - i * b), bm = min(b, n - m * b);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  double g0 = 0.0, g1 = 0.0, g2 = 0.0;
  const double* Z = Zbuf + (size_t)(i - m) * b * b;  // Z_im, column-major, ld b
  const double2* p2 = reinterpret_cast<const double2*>(xy);
  // thread: rows r0 + lane + 32 u (u < 4), columns c0 + warp + 8 q (q < 4)
  double2 pa[4];
  double aa[4];
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const int a = min(r0 + lane + 32 * u, bi - 1);
    pa[u] = p2[(size_t)i * b + a];
    aa[u] = alpha[(size_t)i * b + a];
  }
  const double cx = nu5 ? kSqrt5 : kSqrt3;
#pragma unroll
  for (int q = 0; q < kDtCols / 8; ++q) {
    const int c = c0 + warp + 8 * q;
    if (c >= bm) continue;
    const double2 pc = p2[(size_t)m * b + c];
    const double amc = alpha[(size_t)m * b + c];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int a = r0 + lane + 32 * u;
      if (a >= bi) continue;
      const double dx = pa[u].x - pc.x, dy = pa[u].y - pc.y;
      // dk/d sigma2 = k; dk/d range = sigma2 x^2 e^{-x} / range (nu 3/2) or
      // sigma2 x^2 (1 + x) e^{-x} / (3 range) (nu 5/2)
      const double h = sqrt(fmax(dx * dx + dy * dy, 0.0));
      const double x = cx * h * inv_range;
      const double e = exp(-x);
      const double sbar = 0.5 * (aa[u] * amc - Z[(size_t)c * b + a]);
      double ds = (nu5 ? 1.0 + x + x * x / 3.0 : 1.0 + x) * e;
      const double dr = nu5 ? sigma2 * x * x * (1.0 + x) / 3.0 * e * inv_range : sigma2 * x * x * e * inv_range;
      if (i == m && a == c) {
        ds += eta;
        g2 = fma(sigma2, sbar, g2);
      }
      g0 = fma(ds, sbar, g0);
      g1 = fma(dr, sbar, g1);
    }
  }
  __shared__ double red[3][8];
  g0 = warp_sum(g0);
  g1 = warp_sum(g1);
  g2 = warp_sum(g2);
  if (lane == 0) {
    red[0][warp] = g0;
    red[1][warp] = g1;
    red[2][warp] = g2;
  }
  __syncthreads();
  if (tid < 3) {
    double s = 0.0;
#pragma unroll
    for (int w = 0; w < 8; ++w) s += red[tid][w];
    out[tid] = (i == m ? 1.0 : 2.0) * s;
  }
}

int launch_dtrace_step(const double* xy, int n, int b, int m, int nB, double sigma2, double inv_range, int nu5,
                       double eta, const double* Zbuf, const double* alpha, double* part, const int* status,
                       cudaStream_t s) {
  k_dtrace_step<<<(nB - m) * dtrace_parts(b), 256, 0, s>>>(xy, n, b, m, nB, sigma2, inv_range, nu5, eta, Zbuf, alpha,
                                                           part, status);
  return (int)cudaGetLastError();
}

// final deterministic reduction of the gradient partials: fixed per-thread strides, then a
// fixed-order block reduction
__global__ void __launch_bounds__(1024) k_grad_finish(const double* part, long nparts, double* grad,
                                                     const int* status) {
  __shared__ double red[40];
  if (*status != 0) {
    if (threadIdx.x == 0) grad[0] = grad[1] = grad[2] = 0.0;
    return;
  }
  double g[3] = {0.0, 0.0, 0.0};
  for (long q = threadIdx.x; q < nparts; q += blockDim.x)
    for (int a = 0; a < 3; ++a) g[a] += part[3 * q + a];
  for (int a = 0; a < 3; ++a) {
    const double t = block_sum(g[a], red);
    if (threadIdx.x == 0) grad[a] = t;
  }
}

int launch_grad_finish(const double* part, long nparts, double* grad, const int* status, cudaStream_t s) {
  k_grad_finish<<<1, 1024, 0, s>>>(part, nparts, grad, status);
  return (int)cudaGetLastError();
}

}  // namespace tlr
