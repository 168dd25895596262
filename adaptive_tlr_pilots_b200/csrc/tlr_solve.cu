// Solves and products with the TLR factor left in a plan by an evaluation (kriging prediction,
// simulation of fields without a dense factor).
//
// Reference: codes/17_tlr_cholesky_pilot.py:218-227 (tlr_matvec_L, Y = L Z), 230-240
// (tlr_forward, L X = B) and 243-256 (tlr_backward, L^T X = Z), each for m right-hand sides.
// Right-looking block order: after the diagonal block X_k is solved, its contribution leaves
// every other block row at once (one CTA per block row and 32-column chunk), so a solve is 2 nB
// launches whatever m.  Column-major N x m operands (ld = N), in place.
//
// A solve is one chain through the N rows, so its time is the chain's latency (the products are
// m N b flops, microseconds).  The inverses of the 32 x 32 diagonal blocks of every L_kk are kept from
// the factorization, so a panel step is a 32 x 32 by 32 x 8 product and an update of the other rows,
// both on the FP64 tensor cores.  What is left is the wait for L: the registers of a row block are
// loaded with the next panel's as soon as they are used (16-byte loads, whole lines of a column), and the
// coupling kernel keeps eight row blocks of a column (four with several column blocks) in flight per warp.
// Per launch at b = 500, one column: diagonal solve 49 -> 33 us (L) and 43 -> 37 us (L^T), coupling
// 26 -> 8.4 us against loads next to their use.  Kriging at N = 20,000, b = 500 with 300 sites (two solves
// of one column, one of 300): 174 ms with one thread per column by substitution, 6.7 ms now.
#include <float.h>

#include "tlr_device.cuh"
#include "tlr_kernels.h"

namespace tlr {

namespace {

__device__ __forceinline__ int stidx(int i, int j) { return i * (i - 1) / 2 + j; }

constexpr int kSC = 8;       // columns per CTA in the diagonal solves
constexpr int kSW = 8;       // warps per CTA
constexpr int kSPitch = 34;  // column pitch of a 32 x 32 block in shared memory

__device__ __forceinline__ double2 pair_at(const double* s, int row, int m, bool al) {
  if (al && row + 1 < m) return *reinterpret_cast<const double2*>(s + row);
  return make_double2(row < m ? s[row] : 0.0, row + 1 < m ? s[row + 1] : 0.0);
}

// The inverses of the 32 x 32 diagonal blocks of L_kk (column-major, zero above the diagonal, padded with
// the identity): one warp per block, lane j solves L x = e_j in registers.
__global__ void __launch_bounds__(64) k_diag_inv(const double* TLR_RESTRICT D, int n, int b, int k, int np,
                                                double* TLR_RESTRICT inv) {
  __shared__ __align__(16) double lc[2][32 * kSPitch];
  __shared__ double dinv[2][32];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int q = blockIdx.x * 2 + w;
  if (q >= np) return;
  const int p0 = q * 32;
  const int pw = max(0, min(32, min(b, n - k * b) - p0));
  const double* L = D + (size_t)k * b * b + (size_t)p0 * b + p0;
#pragma unroll 8
  for (int c = 0; c < 32; ++c) {
    const double v = (lane < pw && c < pw && lane >= c) ? L[(size_t)c * b + lane] : (lane == c ? 1.0 : 0.0);
    lc[w][c * kSPitch + lane] = v;
    if (lane == c) dinv[w][c] = 1.0 / v;
  }
  __syncwarp();
  double x[32];
#pragma unroll
  for (int r = 0; r < 32; ++r) x[r] = r == lane ? 1.0 : 0.0;
#pragma unroll
  for (int c = 0; c < 32; ++c) {
    x[c] *= dinv[w][c];
#pragma unroll
    for (int j = c + 1; j < 32; ++j) x[j] = fma(-x[c], lc[w][c * kSPitch + j], x[j]);
  }
  double* o = inv + ((size_t)k * np + q) * 1024 + lane * 32;
#pragma unroll
  for (int r = 0; r < 32; r += 2) *reinterpret_cast<double2*>(o + r) = make_double2(x[r], x[r + 1]);
}

// One column by one warp, row by row.
template <bool TRANS>
__device__ __noinline__ void substitute(const double* L, int b, int bk, double* x) {
  const int lane = threadIdx.x & 31;
  for (int s = 0; s < bk; ++s) {
    const int r = TRANS ? bk - 1 - s : s;
    double acc = 0.0;
    for (int q = lane; q < s; q += 32) {
      const int o = TRANS ? bk - 1 - q : q;  // solved before row r
      acc = fma(TRANS ? L[(size_t)r * b + o] : L[(size_t)o * b + r], x[o], acc);
    }
    acc = warp_sum(acc);
    if (lane == 0) x[r] = (x[r] - acc) / L[(size_t)r * b + r];
    __syncwarp();
  }
}

// X_k <- L_kk^{-1} X_k (TRANS false) or L_kk^{-T} X_k (true), kSC columns per CTA in shared memory, panels
// of 32 rows: X_p <- inv_p X_p, then the other rows lose L[., p] X_p.  Tiles of the products have a column
// of X as their row (lane (g, t) holds column g, rows 2t and 2t + 1).  A right-hand side with an infinity or NaN
// is substituted row by row: the products multiply it by the zeros of the inverses and would carry it to rows
// that do not depend on it.
template <bool TRANS>
__global__ void __launch_bounds__(kSW * 32) k_tri_solve(const double* TLR_RESTRICT D, const double* TLR_RESTRICT inv,
                                                       int n, int b, int np, int k, double* TLR_RESTRICT X, int ldx,
                                                       int m) {
  const int bk = min(b, n - k * b), npk = (bk + 31) / 32;
  const int c0 = blockIdx.x * kSC, nc = min(kSC, m - c0);
  const double* L = D + (size_t)k * b * b;
  inv += (size_t)k * np * 1024;
  extern __shared__ __align__(16) double xs[];  // kSC columns, pitch ld: disjoint banks for the fragments
  constexpr int kXpPitch = TRANS ? 40 : 36;  // likewise
  __shared__ __align__(16) double xp[kSC * kXpPitch];
  const int ld = npk * 32 + (TRANS ? 8 : 4);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  auto store = [&]() {
    for (int e = tid; e < npk * 32 * nc; e += kSW * 32) {
      const int r = e % (npk * 32), c = e / (npk * 32);
      if (r < bk) X[(size_t)(c0 + c) * ldx + (size_t)k * b + r] = xs[c * ld + r];
    }
  };
  bool finite = true;
  for (int e = tid; e < npk * 32 * kSC; e += kSW * 32) {
    const int r = e % (npk * 32), c = e / (npk * 32);
    const double v = (c < nc && r < bk) ? X[(size_t)(c0 + c) * ldx + (size_t)k * b + r] : 0.0;
    finite = finite && fabs(v) <= DBL_MAX;
    xs[c * ld + r] = v;
  }
  if (__syncthreads_or(!finite)) {
    if (warp < nc) substitute<TRANS>(L, b, bk, xs + warp * ld);
    __syncthreads();
    store();
    return;
  }
  const bool al = (b & 1) == 0;
  // row blocks of 16 that panel pi leaves to be solved, the next panel's first
  auto rest = [&](int pi) { return (npk - 1 - pi) * 2; };
  auto row0 = [&](int p0, int q) { return TRANS ? p0 - 16 - 16 * q : p0 + 32 + 16 * q; };
  // Block q of panel pi, zero past the tile's last row.  L: rows r0 + 2 g (+ 1) of column p0 + 4 kk + t, row g of
  // two products.  L^T: columns r0 + g and r0 + 8 + g, rows p0 + 8 kk + 2 t (+ 1), the t of two steps.
  auto frag = [&](double2 (&f)[8], int pi, int q) {
    const int p0 = (TRANS ? npk - 1 - pi : pi) * 32, r0 = row0(p0, q);
    if (q >= rest(pi)) return;
    const double* src = L + (size_t)(TRANS ? r0 + g : p0 + t) * b + (TRANS ? p0 : r0 + 2 * g) + (TRANS ? 2 * t : 0);
    const size_t sb = b;
    if (al && (TRANS ? p0 + 32 : r0 + 16) <= bk) {  // no branch or predicate per load
#pragma unroll
      for (int kk = 0; kk < 8; ++kk)
        f[kk] = *reinterpret_cast<const double2*>(src + (TRANS ? 8 * sb * (kk >> 2) + 8 * (kk & 3) : 4 * sb * kk));
    } else {
#pragma unroll
      for (int kk = 0; kk < 8; ++kk) {
        const int row = TRANS ? p0 + 8 * (kk & 3) + 2 * t : r0 + 2 * g;
        const double* e = src + (TRANS ? 8 * sb * (kk >> 2) + 8 * (kk & 3) : 4 * sb * kk);
        f[kk].x = row < bk ? e[0] : 0.0;
        f[kk].y = row + 1 < bk ? e[1] : 0.0;
      }
    }
  };
  // inv[row 8 (warp % 4) + g][col 4 kk + t] of panel pi, or inv^T
  auto invfrag = [&](double (&w)[8], int pi) {
    if (warp >= 4) return;
    const double* ip = inv + (size_t)(TRANS ? npk - 1 - pi : pi) * 1024;
    const int i = 8 * (warp & 3) + g;
#pragma unroll
    for (int kk = 0; kk < 8; ++kk) w[kk] = TRANS ? ip[i * 32 + 4 * kk + t] : ip[(4 * kk + t) * 32 + i];
  };
  auto update = [&](const double2 (&f)[8], int pi, int q) {
    const int r0 = row0((TRANS ? npk - 1 - pi : pi) * 32, q);
    const double* xc = xp + g * kXpPitch;
    if (TRANS) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        double2* xr = reinterpret_cast<double2*>(xs + g * ld + r0 + 8 * h + 2 * t);
        double2 x = *xr;
        double s0 = 0.0, s1 = 0.0;
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) {
          const double2 a = *reinterpret_cast<const double2*>(xc + 8 * kk + 2 * t);
          dmma884(x.x, x.y, -a.x, f[4 * h + kk].x);
          dmma884(s0, s1, -a.y, f[4 * h + kk].y);
        }
        *xr = make_double2(x.x + s0, x.y + s1);
      }
    } else {
      double2* xr = reinterpret_cast<double2*>(xs + g * ld + r0 + 4 * t);
      double2 v0 = xr[0], v1 = xr[1];
#pragma unroll
      for (int kk = 0; kk < 8; ++kk) {
        const double a = -xc[4 * kk + t];
        dmma884(v0.x, v1.x, a, f[kk].x);
        dmma884(v0.y, v1.y, a, f[kk].y);
      }
      xr[0] = v0;
      xr[1] = v1;
    }
  };
  // The registers of a block are loaded with the next panel's as soon as they are used: a load has the
  // rest of the panel and the next panel's solve to come in.
  constexpr int kHeld = 4;  // blocks per warp: tiles of 512 rows
  double2 f[kHeld][8];
  double w[8];
  invfrag(w, 0);
#pragma unroll
  for (int u = 0; u < kHeld; ++u) frag(f[u], 0, warp + u * kSW);
#pragma unroll 1
  for (int pi = 0; pi < npk; ++pi) {
    const int p0 = (TRANS ? npk - 1 - pi : pi) * 32, nrest = rest(pi);
    if (warp < 4) {  // rows 8 warp .. of X_p
      double a0[2] = {0.0, 0.0}, a1[2] = {0.0, 0.0};
#pragma unroll
      for (int kk = 0; kk < 8; kk += 2) {
        dmma884(a0[0], a0[1], xs[g * ld + p0 + 4 * kk + t], w[kk]);
        dmma884(a1[0], a1[1], xs[g * ld + p0 + 4 * kk + 4 + t], w[kk + 1]);
      }
      *reinterpret_cast<double2*>(xp + g * kXpPitch + 8 * warp + 2 * t) = make_double2(a0[0] + a1[0], a0[1] + a1[1]);
    }
    if (pi + 1 < npk) invfrag(w, pi + 1);
    __syncthreads();
    if (tid < 128) {  // the solved panel back to xs (read again at the end only)
      const int c = tid >> 4, r = 2 * (tid & 15);
      *reinterpret_cast<double2*>(xs + c * ld + p0 + r) = *reinterpret_cast<const double2*>(xp + c * kXpPitch + r);
    }
#pragma unroll
    for (int u = 0; u < kHeld; ++u) {
      const int q = warp + u * kSW;
      if (q < nrest) update(f[u], pi, q);
      if (u == 0) {
#pragma unroll 1
        for (int e = warp + kHeld * kSW; e < nrest; e += kSW) {  // tiles past 512 rows
          frag(f[0], pi, e);
          update(f[0], pi, e);
        }
      }
      frag(f[u], pi + 1, q);  // nothing past the last panel
    }
    __syncthreads();
  }
  store();
}

// trans 0: X_i -= U_ik (V_ik^T X_k) for i > k;  trans 1: X_j -= V_kj (U_kj^T X_k) for j < k.
// One CTA per (block row, chunk of 8 NC columns): T = P^T X_k with the rows split over the warps in blocks
// of 8, then X_o -= E T, both on the FP64 tensor cores.
template <int NC>
__global__ void __launch_bounds__(kSW * 32) k_solve_update(const double* TLR_RESTRICT U, const double* TLR_RESTRICT V,
                                                          const int* TLR_RESTRICT rank, int cap, int n, int b, int k,
                                                          double* TLR_RESTRICT X, int ldx, int m, int trans) {
  const int o = trans ? (int)blockIdx.x : k + 1 + (int)blockIdx.x;  // the block row updated
  const int t0 = trans ? stidx(k, o) : stidx(o, k);
  const int r = rank[t0];
  if (r == 0) return;
  const int c0 = blockIdx.y * 8 * NC;
  const int bk = min(b, n - k * b), bo = min(b, n - o * b);
  // project with the factor on the k side, expand with the one on the other side
  const double* P = (trans ? U : V) + (size_t)t0 * b * cap;
  const double* E = (trans ? V : U) + (size_t)t0 * b * cap;
  __shared__ double red[kSW / 2][NC * 64];
  __shared__ double T[128][8 * NC + 1];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  // 16-byte row pairs of the factor and of X (whose base comes from the caller)
  const bool alp = (b & 1) == 0, alx = alp && (ldx & 1) == 0 && (reinterpret_cast<size_t>(X) & 15) == 0;
  const double* xk = X + (size_t)k * b;
  constexpr int kRb = NC == 1 ? 8 : 4;  // row blocks whose loads are in flight together
  for (int u0 = 0; u0 < r; u0 += 8) {
    const double* pc = P + (size_t)min(u0 + g, r - 1) * b;
    double acc[NC][2];
#pragma unroll
    for (int c = 0; c < NC; ++c) acc[c][0] = acc[c][1] = 0.0;
#pragma unroll 1
    for (int row = 8 * warp; row < bk; row += 8 * kSW * kRb) {
      double2 a[kRb], x[kRb][NC];
#pragma unroll
      for (int p = 0; p < kRb; ++p) {
        const int rr = row + 8 * kSW * p + 2 * t;
        a[p] = pair_at(pc, rr, bk, alp);
#pragma unroll
        for (int c = 0; c < NC; ++c) x[p][c] = pair_at(xk + (size_t)min(c0 + 8 * c + g, m - 1) * ldx, rr, bk, alx);
      }
#pragma unroll
      for (int p = 0; p < kRb; ++p)
#pragma unroll
        for (int c = 0; c < NC; ++c) {
          dmma884(acc[c][0], acc[c][1], a[p].x, x[p][c].x);
          dmma884(acc[c][0], acc[c][1], a[p].y, x[p][c].y);
        }
    }
    // the upper warps hand their parts to the lower ones, whose sums are added below
    for (int half = 1; half >= 0; --half) {
      if (warp / (kSW / 2) == half) {
        double* rd = red[warp % (kSW / 2)] + g * 8 + 2 * t;
#pragma unroll
        for (int c = 0; c < NC; ++c)
#pragma unroll
          for (int h = 0; h < 2; ++h) rd[c * 64 + h] = half ? acc[c][h] : acc[c][h] + rd[c * 64 + h];
      }
      __syncthreads();
    }
    for (int e = tid; e < NC * 64; e += kSW * 32) {
      const int c = e >> 6, u = (e >> 3) & 7, v = e & 7;
      double s = 0.0;
#pragma unroll
      for (int w = 0; w < kSW / 2; ++w) s += red[w][e];
      if (u0 + u < r) T[u0 + u][8 * c + v] = s;
    }
    __syncthreads();
  }
  double* xo = X + (size_t)o * b;
#pragma unroll 1
  for (int row = 8 * warp; row < bo; row += 8 * kSW * kRb) {
    double acc[kRb][NC][2];
#pragma unroll
    for (int p = 0; p < kRb; ++p)
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        const double2 v =
            pair_at(xo + (size_t)min(c0 + 8 * c + g, m - 1) * ldx, row + 8 * kSW * p + 2 * t, bo, alx);
        acc[p][c][0] = v.x;
        acc[p][c][1] = v.y;
      }
#pragma unroll 2
    for (int q0 = 0; q0 < r; q0 += 4) {
      const int u = q0 + t;
      const double* ec = E + (size_t)min(u, r - 1) * b + g;
      double e[kRb];
#pragma unroll
      for (int p = 0; p < kRb; ++p) e[p] = row + 8 * kSW * p + g < bo ? ec[row + 8 * kSW * p] : 0.0;
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        const double a = u < r ? -T[u][8 * c + g] : 0.0;
#pragma unroll
        for (int p = 0; p < kRb; ++p) dmma884(acc[p][c][0], acc[p][c][1], a, e[p]);
      }
    }
#pragma unroll
    for (int p = 0; p < kRb; ++p)
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        if (c0 + 8 * c + g >= m) continue;
        const int rr = row + 8 * kSW * p + 2 * t;
        double* d = xo + (size_t)(c0 + 8 * c + g) * ldx + rr;
        if (alx && rr + 1 < bo) *reinterpret_cast<double2*>(d) = make_double2(acc[p][c][0], acc[p][c][1]);
        else {
          if (rr < bo) d[0] = acc[p][c][0];
          if (rr + 1 < bo) d[1] = acc[p][c][1];
        }
      }
  }
}

// Y_k = L_kk Z_k + sum_{j<k} U_kj (V_kj^T Z_j); one CTA per (block row, 32-column chunk).
__global__ void __launch_bounds__(256) k_matvec_L(const double* TLR_RESTRICT D, const double* TLR_RESTRICT U,
                                                 const double* TLR_RESTRICT V, const int* TLR_RESTRICT rank,
                                                 int cap, int n, int b, const double* TLR_RESTRICT Z, int ldz,
                                                 double* TLR_RESTRICT Y, int ldy, int m) {
  const int k = blockIdx.x;
  const int c0 = blockIdx.y * 32, nc = min(32, m - c0);
  const int bk = min(b, n - k * b);
  const double* L = D + (size_t)k * b * b;
  __shared__ double T[64][33];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int e = tid; e < bk * nc; e += 256) {
    const int a = e % bk, c = e / bk;
    const double* zc = Z + (size_t)(c0 + c) * ldz + (size_t)k * b;
    double acc = 0.0;
    for (int q = 0; q <= a; ++q) acc = fma(L[(size_t)q * b + a], zc[q], acc);
    Y[(size_t)(c0 + c) * ldy + (size_t)k * b + a] = acc;
  }
  for (int j = 0; j < k; ++j) {
    const int t = stidx(k, j);
    const int r = rank[t];
    if (r == 0) continue;
    const int bj = min(b, n - j * b);
    const double* Ut = U + (size_t)t * b * cap;
    const double* Vt = V + (size_t)t * b * cap;
    for (int q0 = 0; q0 < r; q0 += 64) {
      const int rq = min(64, r - q0);
      __syncthreads();
      for (int e = warp; e < rq * nc; e += 8) {
        const int q = e % rq, c = e / rq;
        const double* vc = Vt + (size_t)(q0 + q) * b;
        const double* zc = Z + (size_t)(c0 + c) * ldz + (size_t)j * b;
        double acc = 0.0;
        for (int a = lane; a < bj; a += 32) acc = fma(vc[a], zc[a], acc);
        acc = warp_sum(acc);
        if (lane == 0) T[q][c] = acc;
      }
      __syncthreads();
      for (int e = tid; e < bk * nc; e += 256) {
        const int a = e % bk, c = e / bk;
        double acc = 0.0;
        for (int q = 0; q < rq; ++q) acc = fma(Ut[(size_t)(q0 + q) * b + a], T[q][c], acc);
        Y[(size_t)(c0 + c) * ldy + (size_t)k * b + a] += acc;
      }
    }
  }
}

}  // namespace

size_t diag_inv_doubles(int b, int nB) { return (size_t)nB * ((b + 31) / 32) * 1024; }

int launch_diag_inv(const double* D, int n, int b, int k, double* Linv, cudaStream_t s) {
  const int np = (b + 31) / 32;
  k_diag_inv<<<(np + 1) / 2, 64, 0, s>>>(D, n, b, k, np, Linv);
  return (int)cudaGetLastError();
}

int launch_factor_solve(const double* D, const double* Linv, const double* U, const double* V, const int* rank, int cap,
                        int n, int b, int nB, double* X, int m, int trans, cudaStream_t s) {
  const int np = (b + 31) / 32;
  const size_t sm = (size_t)kSC * (np * 32 + 8) * sizeof(double);
  const auto tri = trans ? k_tri_solve<true> : k_tri_solve<false>;
  cudaFuncSetAttribute(tri, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  for (int q = 0; q < nB; ++q) {
    const int k = trans ? nB - 1 - q : q;
    tri<<<(m + kSC - 1) / kSC, kSW * 32, sm, s>>>(D, Linv, n, b, np, k, X, n, m);
    const int rows = trans ? k : nB - k - 1;
    if (rows > 0) {
      if (m <= 8) k_solve_update<1><<<dim3(rows, 1), kSW * 32, 0, s>>>(U, V, rank, cap, n, b, k, X, n, m, trans);
      else k_solve_update<4><<<dim3(rows, (m + 31) / 32), kSW * 32, 0, s>>>(U, V, rank, cap, n, b, k, X, n, m, trans);
    }
  }
  return (int)cudaGetLastError();
}

int launch_factor_matvec(const double* D, const double* U, const double* V, const int* rank, int cap, int n, int b,
                         int nB, const double* Z, double* Y, int m, cudaStream_t s) {
  const dim3 g(nB, (m + 31) / 32);
  k_matvec_L<<<g, 256, 0, s>>>(D, U, V, rank, cap, n, b, Z, n, Y, n, m);
  return (int)cudaGetLastError();
}

}  // namespace tlr
