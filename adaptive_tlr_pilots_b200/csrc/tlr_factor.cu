// Right-looking TLR Cholesky, forward solve and log-likelihood (FP64 parity path).
//
// Reference: codes/17_tlr_cholesky_pilot.py:168-205 (factorization), 230-240 (forward solve)
// and 259-266 (log-likelihood).  Per step k, in stream order:
//   k_diag_build(k)   A_kk = Sigma_kk - sum_{m<k} U_km (V_km^T V_km) U_km^T   (deferred updates,
//                     subtracted in the order m = 0, 1, ... of the reference's step-by-step updates)
//   k_potrf(k)        blocked Cholesky of A_kk (status k+1 when a pivot is not positive, as LAPACK
//                     potrf), log det partial, z_k = L_kk^{-1} rhs_k
//   k_trsm(k)         V_ik <- L_kk^{-1} V_ik for i > k; W_ik = V_ik^T V_ik; Y_ik = U_ik W_ik;
//                     rhs_i -= U_ik (V_ik^T z_k)
//   k_recompress(k)   A_ij <- truncate([U_ij, -U_ik W], [V_ij, U_jk]) for k < j < i, W = V_ik^T V_jk,
//                     skipped when r_ik = 0 or r_jk = 0 (17:189-194): tlr_recompress.cu, and
//                     k_recompress_general below under the storage rule 'mixed'
// Layout in HBM: diagonal tiles column-major (ld b); off-diagonal factors U, V column-major
// (ld b, cap columns per tile); tile (i, j), i > j, has index i (i - 1) / 2 + j.
#include "tlr_kernels.h"
#include "tlr_panel.cuh"

namespace tlr {

__device__ __forceinline__ int tidx(int i, int j) { return i * (i - 1) / 2 + j; }

// ----------------------------------------------------------------------------------------
// A_kk = Sigma_kk - sum_{m<k} Y_km U_km^T, Y_km = U_km W_km (written by the panel solve of step m):
// the deferred diagonal updates as one product of inner dimension R_k = sum_m r_km on the FP64 tensor
// cores.  One CTA per lower-triangular 32 x 32 block.  The kernel is on the factorization's serial chain
// and has few CTAs, so its time is the latency of the loads: the eight warps take every eighth group of four
// inner indices each, with the operands read straight from L2 (64-byte pieces of four columns) one group
// ahead and no barrier in between, and their sums are added at the end.  N = 10,007, b = 250: 0.83 -> 0.58 ms per
// evaluation, N = 50,000, b = 500: 3.6 -> 1.9 ms, against blocks staged through shared memory.
constexpr int kDgTab = 1024;   // inner columns whose addresses are tabulated at a time
constexpr int kDgPitch = 34;

__global__ void __launch_bounds__(256, 2) k_diag_build(const double* TLR_RESTRICT xy, int n, int b, int k,
                                                      const double* TLR_RESTRICT U, const double* TLR_RESTRICT Y,
                                                      const int* TLR_RESTRICT rank, int cap, double* TLR_RESTRICT D,
                                                      const int* TLR_RESTRICT status) {
  if (*status != 0) return;
  const EvalParams& prm = *eval_params(status);
  const double sigma2 = prm.sigma2, inv_range = prm.inv_range, nugget = prm.nugget;
  const int nu5 = prm.nu5;
  int blk = blockIdx.x, rb = 0;
  while (blk > rb) { blk -= rb + 1; ++rb; }
  const int cb = blk;
  const int bk = min(b, n - k * b);
  const int r0 = rb * 32, c0 = cb * 32;
  __shared__ int off[1025];
  __shared__ int tab[kDgTab];  // column m cap + q of block row k, -1 past the last
  __shared__ __align__(16) double red[4][32 * kDgPitch];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  const int R = block_offsets(off, k, [&](int m) { return rank[tidx(k, m)]; });
  if (tid == 0 && rb == 0 && cb == 0) add_work(status, 7, 0.5 * 2.0 * bk * bk * R, 4.0 * bk * bk);
  const size_t row_base = (size_t)tidx(k, 0) * b * cap;  // tiles (k, 0), (k, 1), ... follow one another
  const double* Yk = Y + row_base;
  const double* Uk = U + row_base;
  double acc[4][4][2];  // [column block][row block]: row 8 p + 2 t (+ 1) of column 8 q + g
#pragma unroll
  for (int q = 0; q < 4; ++q)
#pragma unroll
    for (int p = 0; p < 4; ++p) acc[q][p][0] = acc[q][p][1] = 0.0;
  auto load = [&](double (&u)[4], double (&y)[4], int i, int cnt) {
    const int c = i < cnt ? tab[i + t] : -1;
    const double* up = Uk + (size_t)max(c, 0) * b + g;
    const double* yp = Yk + (size_t)max(c, 0) * b + g;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      u[q] = c >= 0 && c0 + 8 * q + g < bk ? -up[c0 + 8 * q] : 0.0;
      y[q] = c >= 0 && r0 + 8 * q + g < bk ? yp[r0 + 8 * q] : 0.0;
    }
  };
#pragma unroll 1
  for (int base = 0; base < R; base += kDgTab) {
    const int cnt = min(kDgTab, (R - base + 3) & ~3);
    for (int m = tid; m < k; m += 256) {
      const int o = off[m] - base, r = off[m + 1] - off[m];
      for (int q = max(0, -o); q < min(r, kDgTab - o); ++q) tab[o + q] = m * cap + q;
    }
    for (int e = R - base + tid; e < cnt; e += 256) tab[e] = -1;
    __syncthreads();
    double u[4], y[4];
    load(u, y, 4 * warp, cnt);
#pragma unroll 1
    for (int i = 4 * warp; i < cnt; i += 32) {
      double un[4], yn[4];
      load(un, yn, i + 32, cnt);
#pragma unroll
      for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int p = 0; p < 4; ++p) dmma884(acc[q][p][0], acc[q][p][1], u[q], y[p]);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        u[q] = un[q];
        y[q] = yn[q];
      }
    }
    __syncthreads();
  }
#pragma unroll 1
  for (int half = 1; half >= 0; --half) {  // the upper warps' sums, then the lower warps' onto them
    if ((warp >> 2) == half) {
      double* rd = red[warp & 3] + g * kDgPitch + 2 * t;
#pragma unroll
      for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int p = 0; p < 4; ++p) {
          double2* d = reinterpret_cast<double2*>(rd + 8 * q * kDgPitch + 8 * p);
          double2 v = make_double2(acc[q][p][0], acc[q][p][1]);
          if (half == 0) {
            const double2 w = *d;
            v = make_double2(v.x + w.x, v.y + w.y);
          }
          *d = v;
        }
    }
    __syncthreads();
  }
  double* A = D + (size_t)k * b * b;
  const double2* p2 = reinterpret_cast<const double2*>(xy);
  const int ag = r0 + lane;
  const double2 pa = p2[k * b + min(ag, bk - 1)];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int cl = warp + 8 * q, cg = c0 + cl;
    const double2 pc = p2[k * b + min(cg, bk - 1)];
    const double cov = matern_cov(pa.x, pa.y, pc.x, pc.y, sigma2, inv_range, nu5) + (ag == cg ? nugget : 0.0);
    const int e = cl * kDgPitch + lane;
    const double sum = (red[0][e] + red[1][e]) + (red[2][e] + red[3][e]);
    if (ag < bk && cg <= ag) A[(size_t)cg * b + ag] = cov + sum;
  }
}

// ----------------------------------------------------------------------------------------
// Panel solve for column k: one CTA per row tile i > k.  V_ik <- L_kk^{-1} V_ik runs through the tile in
// panels of 32 rows: X_p <- inv_p X_p with the inverse of the panel's diagonal block (formed beside POTRF),
// then the rows below lose L[., p] X_p, both on the FP64 tensor cores with a column of X as a row of the
// tiles (lane (g, t): column g, rows 2t and 2t + 1), the factor's operands loaded ahead of the barrier.
// A product with the inverse has the block's condition in its error where a substitution has the right-hand
// side's.  Against 80-bit arithmetic (N = 1,000, b = 500, 40 right singular vectors, ranges 0.1 to 1, both kernels)
// the two are equal at the nuggets of use: 3e-16 to 8e-16 at eta = 0.05, 1e-15 to 2e-15 at 0.002; below that the
// products lose up to a factor of three (9e-15 against 3e-15 at 1e-5, range 0.1, nu = 5/2).
// Then W' = V^T [V, z_k] and [Y, -rhs update] = U W'.  Bound by the chain of panels (two barriers and two
// short products each) and, per SM, by reading L from L2.  Sixteen warps, so that the products with U,
// whose loads wait on L2, have twice the warps in flight.  Per launch at N = 50,000, b = 500: 184 us with a
// 32-step substitution per panel and column in one thread, 110 with the inverses and eight warps,
// 90 now; ranks up to 65 at N = 20,000: 15.5 -> 10.7 ms per evaluation against eight warps.
constexpr int kTsW = 16;    // warps
constexpr int kTsPitch = 36; // of the solved panel
constexpr int kTsCols = 32; // columns of V per pass (16 for tiles past 512 rows)

// One pass: NCB blocks of 8 columns in xs (pitch ld, npk panels of 32 rows, zero past bk).  L is read in
// blocks of 16 rows, whole 128-byte lines of a column: the lane's two rows 2 g and 2 g + 1 are row g of two
// products, so that its results are rows 4 t .. 4 t + 3.
template <int NCB>
__device__ __forceinline__ void trsm_pass(const double* TLR_RESTRICT L, const double* TLR_RESTRICT inv, int b, int bk,
                                          double* xs, int ld, double* xp) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  const int npk = (bk + 31) / 32;
  const bool al = (b & 1) == 0;
  auto frag = [&](double2 (&f)[8], int p, int q) {  // rows 32 p + 32 + 16 q + 2 g (+ 1), columns 32 p + 4 kk + t
    const int r = 32 * p + 32 + 16 * q + 2 * g;
    const bool in = q < 2 * (npk - 1 - p) && r < bk;
    const double* src = L + (size_t)(32 * p + t) * b + r;
#pragma unroll
    for (int kk = 0; kk < 8; ++kk, src += 4 * (size_t)b) {
      f[kk] = make_double2(0.0, 0.0);
      if (in) {
        if (al) f[kk] = *reinterpret_cast<const double2*>(src);
        else f[kk] = make_double2(src[0], r + 1 < bk ? src[1] : 0.0);
      }
    }
  };
  auto invfrag = [&](double (&w)[8], int p) {
    if ((warp >> 2) >= NCB) return;
    const double* ip = inv + (size_t)p * 1024 + 8 * (warp & 3) + g;
#pragma unroll
    for (int kk = 0; kk < 8; ++kk) w[kk] = ip[(4 * kk + t) * 32];
  };
  double2 f[8];
  double w[8];
  invfrag(w, 0);
  frag(f, 0, warp);
#pragma unroll 1
  for (int p = 0; p < npk; ++p) {
    const int p0 = p * 32, nrest = 2 * (npk - 1 - p);  // blocks of 16 rows below
    if ((warp >> 2) < NCB) {  // rows 8 (warp % 4) .. of X_p, column block warp / 4
      const int cb = warp >> 2;
      const double* xc = xs + (size_t)(8 * cb + g) * ld + p0 + t;
      double a0[2] = {0.0, 0.0}, a1[2] = {0.0, 0.0};
#pragma unroll
      for (int kk = 0; kk < 8; kk += 2) {
        dmma884(a0[0], a0[1], xc[4 * kk], w[kk]);
        dmma884(a1[0], a1[1], xc[4 * kk + 4], w[kk + 1]);
      }
      *reinterpret_cast<double2*>(xp + (8 * cb + g) * kTsPitch + 8 * (warp & 3) + 2 * t) =
          make_double2(a0[0] + a1[0], a0[1] + a1[1]);
    }
    __syncthreads();
    if (p + 1 < npk) invfrag(w, p + 1);  // comes while this panel updates
    for (int e = tid; e < NCB * 128; e += kTsW * 32) {  // the solved panel back to xs (not read again here)
      const int c = e >> 4, r = 2 * (e & 15);
      *reinterpret_cast<double2*>(xs + (size_t)c * ld + p0 + r) =
          *reinterpret_cast<const double2*>(xp + c * kTsPitch + r);
    }
#pragma unroll 1
    for (int q = warp; p + 1 < npk; q += kTsW) {
      const bool more = q + kTsW < nrest;
      double2 fn[8];  // the block after this one, or the next panel's first
      frag(fn, more ? p : p + 1, more ? q + kTsW : warp);
      if (q < nrest) {
#pragma unroll 1  // the blocks at once would spill (11.1 against 10.7 ms)
        for (int cb = 0; cb < NCB; ++cb) {
          double2* xr = reinterpret_cast<double2*>(xs + (size_t)(8 * cb + g) * ld + p0 + 32 + 16 * q + 4 * t);
          const double* xc = xp + (8 * cb + g) * kTsPitch + t;
          double2 v0 = xr[0], v1 = xr[1];
#pragma unroll
          for (int kk = 0; kk < 8; ++kk) {
            const double a = -xc[4 * kk];
            dmma884(v0.x, v1.x, a, f[kk].x);
            dmma884(v0.y, v1.y, a, f[kk].y);
          }
          xr[0] = v0;
          xr[1] = v1;
        }
      }
#pragma unroll
      for (int kk = 0; kk < 8; ++kk) f[kk] = fn[kk];
      if (!more) break;
    }
    __syncthreads();
  }
}

__global__ void __launch_bounds__(kTsW * 32)
    k_trsm(const double* TLR_RESTRICT D, const double* TLR_RESTRICT Linv, int n, int b, int k, int nB, int cols,
           double* TLR_RESTRICT U, double* TLR_RESTRICT V, double* TLR_RESTRICT Wd, double* TLR_RESTRICT Y,
           const int* TLR_RESTRICT rank, int cap, const double* TLR_RESTRICT z, double* TLR_RESTRICT rhs,
           int* TLR_RESTRICT prec, int* TLR_RESTRICT blog_trsm, int prank, int pworld, const int* TLR_RESTRICT status) {
  if (*status != 0) return;
  const EvalParams& prm = *eval_params(status);
  const int round_store = prm.round_store, rmode = prm.rmode;
  const double thr_abs = prm.thr_abs;
  const int i = k + 1 + blockIdx.x;
  if (i >= nB || i % pworld != prank) return;  // block-row partition: this rank's rows only
  const int t0 = tidx(i, k);
  const int r = rank[t0];
  if (r == 0) return;
  const int bk = min(b, n - k * b), bi = min(b, n - i * b);
  const double* L = D + (size_t)k * b * b;
  const double* inv = Linv + (size_t)k * ((b + 31) / 32) * 1024;
  double* Vt = V + (size_t)t0 * b * cap;
  double* Ut = U + (size_t)t0 * b * cap;
  if (threadIdx.x == 0) add_work(status, 9, (double)bk * bk * r + 2.0 * bk * r * r + 4.0 * bk * r,
                                 8.0 * ((double)bk * bk * 0.5 + 2.0 * bk * r + bi * r));
  extern __shared__ __align__(16) double xs[];
  __shared__ __align__(16) double xp[kTsCols * kTsPitch];
  __shared__ double red[kTsW][64];
  __shared__ double Ws[32 * 33];
  __shared__ double zt[128];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  const int rows = (bk + 31) / 32 * 32, ld = rows + 4;
  const bool al = (b & 1) == 0;
  for (int q0 = 0; q0 < r; q0 += cols) {
    const int rq = min(cols, r - q0), ncb = (rq + 7) >> 3, ncx = ncb <= 2 ? ncb : 4;
    for (int e = tid; e < rows * 8 * ncx; e += kTsW * 32) {
      const int a = e % rows, c = e / rows;
      xs[(size_t)c * ld + a] = (c < rq && a < bk) ? Vt[(size_t)(q0 + c) * b + a] : 0.0;
    }
    __syncthreads();
    if (ncb == 1) trsm_pass<1>(L, inv, b, bk, xs, ld, xp);
    else if (ncb == 2) trsm_pass<2>(L, inv, b, bk, xs, ld, xp);
    else trsm_pass<4>(L, inv, b, bk, xs, ld, xp);
    for (int e = tid; e < rows * rq; e += kTsW * 32) {
      const int a = e % rows, c = e / rows;
      if (a < bk) Vt[(size_t)(q0 + c) * b + a] = xs[(size_t)c * ld + a];
    }
    __syncthreads();
  }
  if (round_store) {  // storage rule 'mixed': the factor tile rounded under the full budget (17:183-184)
    __shared__ double rred[40];
    const int bits = cta_round_pair(Ut, Vt, bi, bk, r, b, thr_abs, rred, rmode == kRankReplay ? blog_trsm[t0] : 0);
    if (tid == 0) {
      prec[t0] = bits;
      if (rmode == kRankRecord) blog_trsm[t0] = bits;
    }
    __syncthreads();
  }
  // W' = V^T [V, z_k] (r x (r + 1)), V from shared memory when it is there whole and unrounded
  const bool held = r <= cols && !round_store;
  const double* Vs = held ? xs : Vt;
  const int ldv = held ? ld : b, mv = held ? rows : bk;
  const double* zk = z + (size_t)k * b;
  double* W = r <= 32 ? Ws : Wd + (size_t)t0 * cap * cap;
  const int ldw = r <= 32 ? 33 : cap;
  for (int vb = 0; 8 * vb <= r; ++vb)
    for (int ub = 0; ub <= vb && 8 * ub < r; ++ub) {
      const double* pu = Vs + (size_t)min(8 * ub + g, r - 1) * ldv;
      const int v = 8 * vb + g;
      const bool isz = v >= r;
      const double* pv = isz ? zk : Vs + (size_t)v * ldv;
      const int mz = isz ? bk : mv;
      const bool alu = held || al, alz = isz ? al : alu;  // z_k starts on 16 bytes for even b
      double a0 = 0.0, a1 = 0.0, b0 = 0.0, b1 = 0.0;
#pragma unroll 4
      for (int row = 8 * warp; row < bk; row += 8 * kTsW) {
        const double2 x = load2(pu, row + 2 * t, mv, alu), y = load2(pv, row + 2 * t, mz, alz);
        dmma884(a0, a1, x.x, y.x);
        dmma884(b0, b1, x.y, y.y);
      }
      red[warp][g * 8 + 2 * t] = a0 + b0;
      red[warp][g * 8 + 2 * t + 1] = a1 + b1;
      __syncthreads();
      if (tid < 64) {
        double s = 0.0;
#pragma unroll
        for (int w = 0; w < kTsW; ++w) s += red[w][tid];
        const int u = 8 * ub + (tid >> 3), c = 8 * vb + (tid & 7);
        if (u < r && c < r) {
          W[u * ldw + c] = s;
          if (ub != vb) W[c * ldw + u] = s;
        } else if (u < r && c == r) {
          zt[u] = s;
        }
      }
      __syncthreads();
    }
  // [Y_ik, x] = U_ik W': the factor of the deferred diagonal update of tile i, and rhs_i -= x
  double* Yt = Y + (size_t)t0 * b * cap;
  double* ri = rhs + (size_t)i * b;
  const int nob = r / 8 + 1;
  for (int blk = warp; 8 * blk < bi; blk += kTsW)
    for (int o0 = 0; o0 < nob; o0 += 4) {
      double acc[4][2];
#pragma unroll
      for (int o = 0; o < 4; ++o) acc[o][0] = acc[o][1] = 0.0;
      const int row = 8 * blk + g;
#pragma unroll 2
      for (int u0 = 0; u0 < r; u0 += 4) {
        const int u = u0 + t;
        const double x = (u < r && row < bi) ? Ut[(size_t)u * b + row] : 0.0;
#pragma unroll
        for (int o = 0; o < 4; ++o)
          if (o0 + o < nob) {
            const int c = 8 * (o0 + o) + g;
            dmma884(acc[o][0], acc[o][1], u < r ? (c < r ? W[u * ldw + c] : (c == r ? zt[u] : 0.0)) : 0.0, x);
          }
      }
#pragma unroll
      for (int o = 0; o < 4; ++o) {
        const int c = 8 * (o0 + o) + g;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int a = 8 * blk + 2 * t + h;
          if (a < bi && c < r) Yt[(size_t)c * b + a] = acc[o][h];
          else if (a < bi && c == r) ri[a] -= acc[o][h];
        }
      }
    }
}

// ----------------------------------------------------------------------------------------
// Recompression under the storage rule 'mixed' (the other rules: tlr_recompress.cu).  Persistent grid;
// each CTA owns one slot of global scratch (L2-resident working arrays).
struct GenScratch {
  double *W, *Ru, *Rv, *M, *Vs, *A, *B;
};

static __host__ __device__ inline size_t gen_slot(double* base, int b, int cap, GenScratch* out) {
  const size_t c2 = (size_t)cap * cap, bc = (size_t)b * cap;
  size_t o = 0;
  auto take = [&](size_t n) {
    double* p = base + o;
    o += n;
    return p;
  };
  GenScratch s;
  s.W = take(c2);
  s.Ru = take(4 * c2);
  s.Rv = take(4 * c2);
  s.M = take(4 * c2);
  s.Vs = take(4 * c2);
  s.A = take(2 * bc);
  s.B = take(2 * bc);
  if (out) *out = s;
  return (o + 1) & ~(size_t)1;
}

size_t rc_general_slot_doubles(int b, int cap) { return gen_slot(nullptr, b, cap, nullptr); }

// C = A^T B (p x q, column v of C at C + v ldc), task e of p * ceil(q / 4) by one warp: row u of C, four
// consecutive columns, so a column of A is read once for four dots.
__device__ __forceinline__ void atb4_task(const double* A, int lda, const double* B, int ldb, int m, int p, int q,
                                          double* C, int ldc, int e) {
  const int lane = threadIdx.x & 31;
  {
    const int u = e % p, v0 = (e / p) * 4;
    const double* a = A + (size_t)u * lda;
    const double* b0 = B + (size_t)v0 * ldb;
    const double* b1 = B + (size_t)min(v0 + 1, q - 1) * ldb;
    const double* b2 = B + (size_t)min(v0 + 2, q - 1) * ldb;
    const double* b3 = B + (size_t)min(v0 + 3, q - 1) * ldb;
    double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
    for (int t = lane; t < m; t += 32) {
      const double x = a[t];
      s0 += x * b0[t];
      s1 += x * b1[t];
      s2 += x * b2[t];
      s3 += x * b3[t];
    }
    s0 = warp_sum(s0);
    s1 = warp_sum(s1);
    s2 = warp_sum(s2);
    s3 = warp_sum(s3);
    if (lane == 0) {
      C[(size_t)v0 * ldc + u] = s0;
      if (v0 + 1 < q) C[(size_t)(v0 + 1) * ldc + u] = s1;
      if (v0 + 2 < q) C[(size_t)(v0 + 2) * ldc + u] = s2;
      if (v0 + 3 < q) C[(size_t)(v0 + 3) * ldc + u] = s3;
    }
  }
}

// General recompression of one trailing pair, the reference's recompress as written
// (codes/17_tlr_cholesky_pilot.py:119-133): Householder QR of A = [U_ij, -U_ik W] and
// B = [V_ij, U_jk] (no orthogonality assumed), SVD of the core R_u R_v^T by one-sided Jacobi on
// its transpose, the rule's rank, U' = Q_u U_w s, V' = Q_v V_w.  The storage rule 'mixed' uses it:
// its rounded factors are no longer orthogonal, which the structured projection needs.  The new
// pair overwrites the tile (i, j); with round_store it is then rounded under the budget left after
// truncation (17:203-204).  Returns the new rank, or -1 after setting an error status.
__device__ int rc_general_pair(int bi, int bj, int b, int cap, int r1, int ri, int rj, const double* Uik,
                               const double* Ujk, const double* W, double* Uw, double* Vw, GenScratch& S,
                               double* sig, int* perm, int* iflag, double* red, int* rsel, int rule_fixed,
                               double thr_rel, double thr_abs, int round_store, int* rlog_pp, int* blog_pp,
                               int rmode, int* status) {
  const int tid = threadIdx.x, nt = blockDim.x;
  const int s = r1 + rj, ls = 2 * cap;
  const int ku = min(bi, s), kv = min(bj, s);
  double* A = S.A;  // b x 2 cap
  double* B = S.B;  // b x 2 cap
  for (int q = 0; q < r1; ++q) {
    for (int a = tid; a < bi; a += nt) A[(size_t)q * b + a] = Uw[(size_t)q * b + a];
    for (int a = tid; a < bj; a += nt) B[(size_t)q * b + a] = Vw[(size_t)q * b + a];
  }
  for (int q = 0; q < rj; ++q) {
    for (int a = tid; a < bi; a += nt) {
      double acc = 0.0;
      for (int p = 0; p < ri; ++p) acc = fma(Uik[(size_t)p * b + a], W[(size_t)q * cap + p], acc);
      A[(size_t)(r1 + q) * b + a] = -acc;
    }
    for (int a = tid; a < bj; a += nt) B[(size_t)(r1 + q) * b + a] = Ujk[(size_t)q * b + a];
  }
  __syncthreads();
  // A = Q_u R_u, B = Q_v R_v (R upper trapezoidal ku x s / kv x s, Q explicit bi x ku / bj x kv)
  cta_geqr2(A, b, bi, s, sig, red);
  cta_copy_r(A, b, ku, s, S.Ru, ls);
  cta_org2r(A, b, bi, ku, sig);
  cta_geqr2(B, b, bj, s, sig, red);
  cta_copy_r(B, b, kv, s, S.Rv, ls);
  cta_org2r(B, b, bj, kv, sig);
  // Z = (R_u R_v^T)^T (kv x ku): Z[c][a] = sum_t R_u[a][t] R_v[c][t], t >= max(a, c)
  for (int e = tid; e < ku * kv; e += nt) {
    const int c = e % kv, a = e / kv;
    double acc = 0.0;
    for (int t = max(a, c); t < s; ++t) acc = fma(S.Ru[(size_t)t * ls + a], S.Rv[(size_t)t * ls + c], acc);
    S.M[(size_t)a * ls + c] = acc;
  }
  __syncthreads();
  // Z J = Z' (orthogonal columns): core = J Z'^T, left singular vectors J, right Z' / sigma
  cta_jacobi_svd(S.M, ls, kv, ku, S.Vs, ls, sig, perm, iflag, 40, 1e-28);
  if (tid == 0) {
    double srt[256];
    double fro2 = 0.0;
    for (int q = 0; q < ku; ++q) srt[q] = sig[perm[q]];
    for (int q = ku - 1; q >= 0; --q) fro2 += srt[q] * srt[q];
    const double thr = rule_fixed ? thr_rel * sqrt(fro2) : thr_abs;
    int r = select_rank(srt, ku, 0.0, thr, nullptr);
    if (r < 0) r = ku;
    if (rmode == kRankReplay) r = min(*rlog_pp, ku);
    else if (rmode == kRankRecord) *rlog_pp = r;
    double tail2 = 0.0;
    for (int q = ku - 1; q >= r; --q) tail2 += srt[q] * srt[q];
    if (r > cap) {
      atomicCAS(status, 0, -2);
      r = -1;
    }
    rsel[0] = r;
    reinterpret_cast<double*>(rsel + 2)[0] = sqrt(tail2);
  }
  __syncthreads();
  const int rn = rsel[0];
  const double tail = reinterpret_cast<double*>(rsel + 2)[0];
  if (rn < 0) return -1;
  // U' = Q_u (J[:, perm c] sigma), V' = Q_v (Z'[:, perm c] / sigma): over the tile's own slot
  for (int c = 0; c < rn; ++c) {
    const int pc = perm[c];
    const double sg = sig[pc], inv = sg > 0.0 ? 1.0 / sg : 0.0;
    const double* jc = S.Vs + (size_t)pc * ls;
    const double* zc = S.M + (size_t)pc * ls;
    for (int a = tid; a < bi; a += nt) {
      double acc = 0.0;
      for (int q = 0; q < ku; ++q) acc = fma(A[(size_t)q * b + a], jc[q], acc);
      Uw[(size_t)c * b + a] = acc * sg;
    }
    for (int a = tid; a < bj; a += nt) {
      double acc = 0.0;
      for (int q = 0; q < kv; ++q) acc = fma(B[(size_t)q * b + a], zc[q], acc);
      Vw[(size_t)c * b + a] = acc * inv;
    }
  }
  __syncthreads();
  if (round_store) {
    const int bits = cta_round_pair(Uw, Vw, bi, bj, rn, b, thr_abs - tail, red, rmode == kRankReplay ? *blog_pp : 0);
    if (tid == 0 && rmode == kRankRecord) *blog_pp = bits;
  }
  return rn;
}

constexpr int kGcT = 256;       // threads per pair
constexpr int kGcBlocks = 3;    // resident CTAs per SM

int rc_general_blocks_per_sm() { return kGcBlocks; }

__global__ void __launch_bounds__(kGcT, kGcBlocks)
    k_recompress_general(int n, int b, int k, int nB, double* TLR_RESTRICT U, double* TLR_RESTRICT V,
                         int* TLR_RESTRICT rank, int cap, double* TLR_RESTRICT scratch, size_t slot_doubles,
                         int* TLR_RESTRICT next_pair, int* TLR_RESTRICT rlog, int* TLR_RESTRICT blog,
                         int* TLR_RESTRICT status) {
  if (cta_failed(status)) return;
  const EvalParams& prm = *eval_params(status);
  const int rule_fixed = prm.rule_fixed, rmode = prm.rmode;
  const double thr_rel = prm.thr_rel, thr_abs = prm.thr_abs;
  const long mB = nB - k - 1, npairs = mB * (mB - 1) / 2;  // trailing tiles, their pairs (i, j), k < j < i
  GenScratch S;
  gen_slot(scratch + (size_t)blockIdx.x * slot_doubles, b, cap, &S);
  __shared__ double red[40];
  __shared__ double sig[256];
  __shared__ int perm[256];
  __shared__ int iflag[2];
  __shared__ __align__(8) int gsel[4];
  const int tid = threadIdx.x, warp = tid >> 5;
  if (blockIdx.x == 0 && tid < 32) {  // the panel column k is read once per step
    int sum = 0;
    for (int i = k + 1 + tid; i < nB; i += 32) sum += rank[tidx(i, k)];
    sum = __reduce_add_sync(0xffffffffu, sum);
    if (tid == 0) add_work(status, 10, 0.0, 16.0 * b * sum);
  }
  // each CTA starts on pair blockIdx.x and then takes the next unclaimed one (*next_pair counts the
  // claims past the grid; zero at launch)
  __shared__ long q_next;
  auto claim = [&]() -> long {
    __syncthreads();
    if (threadIdx.x == 0) q_next = (long)gridDim.x + atomicAdd(next_pair, 1);
    __syncthreads();
    return q_next;
  };
  for (long pp = blockIdx.x; pp < npairs; pp = claim()) {
    long ii = (long)((1.0 + sqrt(1.0 + 8.0 * (double)pp)) * 0.5);
    while (ii * (ii - 1) / 2 > pp) --ii;
    while ((ii + 1) * ii / 2 <= pp) ++ii;
    const int i = k + 1 + (int)ii, j = k + 1 + (int)(pp - ii * (ii - 1) / 2);
    const int tij = tidx(i, j), tik = tidx(i, k), tjk = tidx(j, k);
    const int r1 = rank[tij], ri = rank[tik], rj = rank[tjk];
    if (ri == 0 || rj == 0) continue;
    const int bi = min(b, n - i * b), bj = min(b, n - j * b), bk = min(b, n - k * b);
    const double* Vik = V + (size_t)tik * b * cap;
    const double* Vjk = V + (size_t)tjk * b * cap;
    const int s = r1 + rj;
    __syncthreads();
    const int nW = ri * ((rj + 3) >> 2);  // W = V_ik^T V_jk (ri x rj)
    for (int e = warp; e < nW; e += kGcT / 32) atb4_task(Vik, b, Vjk, b, bk, ri, rj, S.W, cap, e);
    __syncthreads();
    const int rn = rc_general_pair(bi, bj, b, cap, r1, ri, rj, U + (size_t)tik * b * cap, U + (size_t)tjk * b * cap, S.W,
                                   U + (size_t)tij * b * cap, V + (size_t)tij * b * cap, S, sig, perm, iflag, red, gsel,
                                   rule_fixed, thr_rel, thr_abs, 1, rlog + pp, blog + pp, rmode, status);
    if (rn < 0) return;
    if (tid == 0) {
      rank[tij] = rn;
      add_work(status, 10, 4.0 * b * ri * rj + 16.0 * b * s * s + 4.0 * b * s * rn,
               8.0 * ((double)(bi + bj) * r1 + (double)(bi + bj) * rn));
    }
    __syncthreads();
  }
}

int launch_recompress_general(int n, int b, int k, int nB, double* U, double* V, int* rank, int cap, double* scratch,
                              size_t slot_doubles, int nslots, int* next_pair, int* rlog_step, int* blog_step,
                              int* status, cudaStream_t s) {
  const long mB = nB - k - 1, npairs = mB * (mB - 1) / 2;
  if (npairs <= 0) return 0;
  const int grid = (int)std::min<long>(npairs, nslots);
  k_recompress_general<<<grid, kGcT, 0, s>>>(n, b, k, nB, U, V, rank, cap, scratch, slot_doubles, next_pair, rlog_step,
                                             blog_step, status);
  return (int)cudaGetLastError();
}

// ----------------------------------------------------------------------------------------
__global__ void k_finish(int nB, int n, const double* ldpart, const double* qpart, double* out,
                         const int* status) {
  if (threadIdx.x != 0) return;
  if (*status != 0) { out[0] = 0.0; out[1] = 0.0; out[2] = 0.0; return; }
  double ld = 0.0, q = 0.0;
  for (int k = 0; k < nB; ++k) { ld += ldpart[k]; q += qpart[k]; }
  const double log2pi = 1.8378770664093454836;
  out[0] = -0.5 * (q + ld + (double)n * log2pi);
  out[1] = ld;
  out[2] = q;
}

// ----------------------------------------------------------------------------------------
int launch_diag_build(const double* xy, int n, int b, int k, const double* U, const double* Y, const int* rank,
                      int cap, double* D, const int* status, cudaStream_t s) {
  const int bk = std::min(b, n - k * b);
  const int nb = (bk + 31) / 32;
  k_diag_build<<<nb * (nb + 1) / 2, 256, 0, s>>>(xy, n, b, k, U, Y, rank, cap, D, status);
  return (int)cudaGetLastError();
}

int launch_trsm(const double* D, const double* Linv, int n, int b, int k, int nB, double* U, double* V, double* Wd,
                double* Y, const int* rank, int cap, const double* z, double* rhs, int* prec, int* blog_trsm, int prank,
                int pworld, const int* status, cudaStream_t s) {
  if (nB - k - 1 <= 0) return 0;
  const int cols = b <= 512 ? kTsCols : kTsCols / 2;
  const size_t sm = (size_t)cols * ((b + 31) / 32 * 32 + 4) * sizeof(double);
  cudaFuncSetAttribute(k_trsm, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  k_trsm<<<nB - k - 1, kTsW * 32, sm, s>>>(D, Linv, n, b, k, nB, cols, U, V, Wd, Y, rank, cap, z, rhs, prec, blog_trsm,
                                           prank, pworld, status);
  return (int)cudaGetLastError();
}

int launch_finish(int nB, int n, const double* ldpart, const double* qpart, double* out, const int* status,
                  cudaStream_t s) {
  k_finish<<<1, 32, 0, s>>>(nB, n, ldpart, qpart, out, status);
  return (int)cudaGetLastError();
}

}  // namespace tlr
