// Recompression of the trailing tiles at one factorization step (fixed and adaptive rules).
//
// Reference: codes/17_tlr_cholesky_pilot.py:186-205 (the Schur update of tile (i, j)) and 119-133
// (recompress: QR of the stacked factors, SVD of the core, the rank rule).
//   A_ij <- truncate(U_ij V_ij^T - U_ik W U_jk^T), W = V_ik^T V_jk, for k < j < i.
//
// The stored pairs have structure that the reference's dense QR cannot use: U_ij has orthogonal
// columns and V_ij orthonormal ones.  With q = min(r_ik, r_jk) the update is written as X Y^T with q
// columns, X = -U_ik W, Y = U_jk (r_jk <= r_ik) or X = U_ik, Y = -U_jk W^T (r_ik < r_jk), and per side
//   C = Q1^T X, X <- X - Q1 C, twice (block Gram-Schmidt, Q1 = the normalised U_ij or V_ij);
//   Householder QR X = Q2 R2 (the V side also forms Q3 = its Q, re-orthogonalised against V_ij);
// then M = [[diag, 0], [0, 0]] + [C; R2] [D; R3]^T of order s = r_ij + q, Householder R of M, one-sided
// Jacobi on the rows of R (right singular vectors and values of M), the rank rule, and
//   U' = U_ij G_top + X G_bot,  V' = [V_ij, Q3] Vs_r.
//
// One CTA per pair: two groups of GW warps work on the U and the V side at the same time (named
// barriers inside a group).  The kernel is bound by chains of dependent small steps, not by bytes or
// FP64 operations (about 0.3 M fused multiply-adds and 0.2 MB per pair at b = 500, rank 5), so the
// design shortens the chains:
//   * a b x 8 panel block lives in registers in the FP64 tensor cores' fragment layout through both
//     Gram-Schmidt passes: inner products and updates are mma m8n8k4 steps over the warp's own rows,
//     with one cross-warp sum per product;
//   * the panel QR keeps the panel in registers by rows and takes all inner products of a column step
//     in one reduction: one barrier per column;
//   * the core SVD runs on eight lanes per column pair in shared memory, its rotation from reciprocal
//     and square-root approximations (see jacobi_rows), while the V group forms Q3;
//   * the next pair is claimed and its ranks are read while the current one is worked on.
// Panels wider than 8 columns go through the same steps block by block (blocked Householder: the
// reflector blocks are applied as I - V T V^T), with the arrays that do not fit in shared memory in
// the CTA's slot of global scratch (L2).
#include "tlr_device.cuh"
#include "tlr_kernels.h"

namespace tlr {

namespace {

constexpr int kFs = 32;      // largest core order kept in shared memory whole (M, G, H and C)
constexpr int kFlong = 24;   // largest long side of W kept in shared memory
constexpr int kRu = 3;       // blocks of 8 columns per reduction of a product
constexpr int kLdq = 9;      // row pitch of the shared [C; R] arrays
constexpr int kLdg = 32;     // row pitch of the shared G arrays
constexpr int kSmall = kFs * (kFs + 1) + (kFs + kFlong) * kLdg + kFs * kLdg + 8 * kLdg;  // M, GU, GV, Gb

__device__ __forceinline__ int tidx(int i, int j) { return i * (i - 1) / 2 + j; }
__host__ __device__ constexpr int round8(int v) { return (v + 7) & ~7; }

// Approximate reciprocal and reciprocal square root (about 20 bits; rcp.approx / rsqrt.approx).
__device__ __forceinline__ double rcp_approx(double x) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
  return r;
}
__device__ __forceinline__ double rsqrt_approx(double x) {
  double r;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
  return r;
}

template <int N>
__device__ __forceinline__ void bar_sync(int id) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "n"(N) : "memory");
}
__device__ __forceinline__ void bar_sync_n(int id, int n) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory"); }
template <int N>
__device__ __forceinline__ void bar_arrive(int id) {
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "n"(N) : "memory");
}

// rows row, row + 1 of a column (zero past m); al: row pairs are 16-byte aligned
__device__ __forceinline__ double2 load2(const double* s, int row, int m, bool al) {
  if (al && row + 1 < m) return *reinterpret_cast<const double2*>(s + row);
  double2 v;
  v.x = row < m ? s[row] : 0.0;
  v.y = row + 1 < m ? s[row + 1] : 0.0;
  return v;
}

// One side's warps.  Rows are dealt out in blocks of 8, block gw + GW p to warp gw; lane (g, t) holds
// of an 8-column panel block column g, rows 8 blk + 2t and 2t + 1: the layout of the B operand and of
// the accumulator of mma m8n8k4, with the two rows as the k index of two steps.
template <int GW, int NBLK>
struct Side {
  static constexpr int GT = GW * 32;
  static constexpr int kRows = 8 * NBLK * GW;
  static constexpr int kLdx = kRows + 8;  // column pitch of a panel: double2 columns fall in disjoint banks
  static constexpr int kRpt = NBLK / 4;   // rows per thread in the row layout of the panel QR
  int gw, lane, g, t, tg, bar, m;
  bool al;

  __device__ __forceinline__ void sync() const { bar_sync<GT>(bar); }

  // columns c0 .. c0 + nc of a panel
  __device__ __forceinline__ void load(double (&x)[NBLK][2], const double* src, int ld, int c0, int nc) const {
    const double* s = src + (size_t)(c0 + min(g, nc - 1)) * ld;
#pragma unroll
    for (int p = 0; p < NBLK; ++p) {
      const double2 v = load2(s, 8 * (gw + GW * p) + 2 * t, m, al);
      x[p][0] = g < nc ? v.x : 0.0;
      x[p][1] = g < nc ? v.y : 0.0;
    }
  }

  // x += sign * src coef: src nu columns (rows past mrow read as zero), coef[u ldc + v]
  __device__ __forceinline__ void update(double (&x)[NBLK][2], const double* src, int ld, int nu, int mrow,
                                         const double* coef, int ldc, int nv, double sign) const {
    for (int k0 = 0; k0 < nu; k0 += 4) {
      const int u = k0 + t;
      const double a = (u < nu && g < nv) ? sign * coef[u * ldc + g] : 0.0;
      const double* s = src + (size_t)min(u, nu - 1) * ld;
      double b[NBLK];
#pragma unroll
      for (int p = 0; p < NBLK; ++p) {
        const int row = 8 * (gw + GW * p) + g;
        b[p] = row < mrow ? s[row] : 0.0;
      }
#pragma unroll
      for (int p = 0; p < NBLK; ++p) dmma884(x[p][0], x[p][1], a, b[p]);
    }
  }

  // The products src^T x (nu x 8): red takes the warps' parts of kRu blocks at a time; entry (u, v) of
  // the sum goes through `put(u, v, sum, norm2)`.  With NORM the squared column norms of src come along.
  template <bool NORM, class Put>
  __device__ __forceinline__ void dot(const double (&x)[NBLK][2], const double* src, int ld, int nu, int mrow,
                                      bool aligned, double* red, double* redn, Put put) const {
    for (int u0 = 0; u0 < nu; u0 += 8 * kRu) {
      const int nub = min(kRu, (nu - u0 + 7) >> 3);
      for (int ub = 0; ub < nub; ++ub) {
        const double* s = src + (size_t)min(u0 + 8 * ub + g, nu - 1) * ld;
        double a0 = 0.0, a1 = 0.0, b0 = 0.0, b1 = 0.0, nn = 0.0;
        constexpr int kCh = NBLK < 8 ? NBLK : 8;
#pragma unroll
        for (int pc = 0; pc < NBLK; pc += kCh) {
          double2 v[kCh];
#pragma unroll
          for (int p = 0; p < kCh; ++p) v[p] = load2(s, 8 * (gw + GW * (pc + p)) + 2 * t, mrow, aligned);
#pragma unroll
          for (int p = 0; p < kCh; ++p) {
            dmma884(a0, a1, v[p].x, x[pc + p][0]);
            dmma884(b0, b1, v[p].y, x[pc + p][1]);
            if (NORM) nn = fma(v[p].x, v[p].x, fma(v[p].y, v[p].y, nn));
          }
        }
        double* rd = red + (ub * GW + gw) * 64 + g * 8 + 2 * t;
        rd[0] = a0 + b0;
        rd[1] = a1 + b1;
        if (NORM) {
          nn += __shfl_xor_sync(0xffffffffu, nn, 1);
          nn += __shfl_xor_sync(0xffffffffu, nn, 2);
          if (t == 0) redn[(ub * GW + gw) * 8 + g] = nn;
        }
      }
      sync();
      for (int e = tg; e < nub * 64; e += GT) {
        const int ub = e >> 6, uu = (e >> 3) & 7, v = e & 7, u = u0 + 8 * ub + uu;
        if (u < nu) {
          double sum = 0.0, n2 = 0.0;
#pragma unroll
          for (int w = 0; w < GW; ++w) {
            sum += red[(ub * GW + w) * 64 + uu * 8 + v];
            if (NORM) n2 += redn[(ub * GW + w) * 8 + uu];
          }
          put(u, v, sum, n2);
        }
      }
      sync();
    }
  }

  // Householder QR of a block of nc columns whose pivots are rows r0 .. r0 + nc - 1 (dlarfg convention);
  // the rows above r0 are final.  The panel passes through xs (kLdx x 8) into registers by rows.  Row r
  // of the block (r <= pivot) goes to R[r ldq + j]; the reflectors (unit at the pivot, zero above) to
  // panel when it is given, with their T factor (8 x 8) to tf.  qred: 2 (8 GW + 8) doubles.
  __device__ __forceinline__ void qr(const double (&x)[NBLK][2], double* xs, int r0, int nc, int nrow, double* qred,
                                     double* R, int ldq, double* zt, double* tau, double* tf, double* panel) const {
#pragma unroll
    for (int p = 0; p < NBLK; ++p)
      *reinterpret_cast<double2*>(xs + g * kLdx + 8 * (gw + GW * p) + 2 * t) = make_double2(x[p][0], x[p][1]);
    sync();
    double y[kRpt][8];
#pragma unroll
    for (int i = 0; i < kRpt; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j) y[i][j] = xs[j * kLdx + tg + GT * i];
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      if (c < nc) {
        const int piv = r0 + c;
        double p[8], xc[kRpt];
#pragma unroll
        for (int i = 0; i < kRpt; ++i) xc[i] = tg + GT * i > piv ? y[i][c] : 0.0;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          p[j] = xc[0] * y[0][j];
#pragma unroll
          for (int i = 1; i < kRpt; ++i) p[j] = fma(xc[i], y[i][j], p[j]);
        }
        // eight sums over the warp at once: each exchange halves the values a lane carries
        const bool h4 = lane & 16, h2 = lane & 8, h1 = lane & 4;
        double q4[4], q2[2], q1;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const double snd = h4 ? p[j] : p[j + 4];
          q4[j] = (h4 ? p[j + 4] : p[j]) + __shfl_xor_sync(0xffffffffu, snd, 16);
        }
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const double snd = h2 ? q4[j] : q4[j + 2];
          q2[j] = (h2 ? q4[j + 2] : q4[j]) + __shfl_xor_sync(0xffffffffu, snd, 8);
        }
        {
          const double snd = h1 ? q2[0] : q2[1];
          q1 = (h1 ? q2[1] : q2[0]) + __shfl_xor_sync(0xffffffffu, snd, 4);
        }
        q1 += __shfl_xor_sync(0xffffffffu, q1, 2);
        q1 += __shfl_xor_sync(0xffffffffu, q1, 1);
        double* rb = qred + (c & 1) * (8 * GW + 8);
        if ((lane & 3) == 0) rb[gw * 8 + (lane >> 4) * 4 + ((lane >> 3) & 1) * 2 + ((lane >> 2) & 1)] = q1;
        if (tg == piv) {
#pragma unroll
          for (int j = 0; j < 8; ++j) rb[8 * GW + j] = y[0][j];
        }
        sync();
        double s[8], pv[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          s[j] = rb[j];
          pv[j] = rb[8 * GW + j];
        }
#pragma unroll
        for (int w = 1; w < GW; ++w)
#pragma unroll
          for (int j = 0; j < 8; ++j) s[j] += rb[w * 8 + j];
        const double alpha = pv[c], sig2 = s[c];
        double beta = alpha, tc = 0.0, scale = 1.0;
        if (sig2 != 0.0) {
          beta = -copysign(sqrt(alpha * alpha + sig2), alpha);
          tc = (beta - alpha) / beta;
          scale = 1.0 / (alpha - beta);
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const double z = fma(scale, s[j], pv[j]);
          if (j > c) {
            const double w = tc * z, f = w * scale;
#pragma unroll
            for (int i = 0; i < kRpt; ++i) y[i][j] = fma(-f, xc[i], y[i][j]);
            if (tg == piv) y[0][j] -= w;
          } else if (j < c) {
            if (tg == 0) zt[j * 8 + c] = z;  // v_j^T v_c
          }
        }
#pragma unroll
        for (int i = 0; i < kRpt; ++i)
          if (tg + GT * i > piv) y[i][c] = xc[i] * scale;
        if (tg == piv) y[0][c] = beta;
        if (tg == 0) tau[c] = tc;
      }
    }
    if (tg < nrow) {
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (j < nc) R[tg * ldq + j] = tg <= r0 + j ? y[0][j] : 0.0;
    }
    if (panel) {
#pragma unroll
      for (int i = 0; i < kRpt; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const int row = tg + GT * i;
          panel[j * kLdx + row] = (j >= nc || row < r0 + j) ? 0.0 : (row == r0 + j ? 1.0 : y[i][j]);
        }
      sync();
      if (tg < 8) {  // row tg of T: T_cc = tau_c, T_jc = -tau_c sum_m T_jm (v_m^T v_c)
        double tr[8];
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          double acc = 0.0;
#pragma unroll
          for (int k = 0; k < c; ++k)
            if (c < nc && k >= tg) acc = fma(tr[k], zt[k * 8 + c], acc);
          const double tc = c < nc ? tau[c] : 0.0;
          tr[c] = c < tg ? 0.0 : (c == tg ? tc : -tc * acc);
          tf[tg * 8 + c] = tr[c];
        }
      }
    }
    sync();
  }

  // x <- (I - V T^T V^T) x (trans) or (I - V T V^T) x for one reflector block
  __device__ __forceinline__ void apply_block(double (&x)[NBLK][2], const double* panel, const double* tf, bool trans,
                                              double* red, double* tmp, double* coef) const {
    dot<false>(x, panel, kLdx, 8, kRows, true, red, nullptr,
               [&](int u, int v, double sum, double) { tmp[u * 8 + v] = sum; });
    for (int e = tg; e < 64; e += GT) {
      const int u = e >> 3, v = e & 7;
      double acc = 0.0;
#pragma unroll
      for (int k = 0; k < 8; ++k) acc = fma(trans ? tf[k * 8 + u] : tf[u * 8 + k], tmp[k * 8 + v], acc);
      coef[e] = acc;
    }
    sync();
    update(x, panel, kLdx, 8, kRows, coef, 8, 8, -1.0);
  }
};

// R of the Householder QR of the s x s row-major M by one warp (s <= 32): lanes hold columns, nsp
// lanes per column share its rows.  The entries below the diagonal are set to zero.
__device__ void warp_core_r(double* M, int ldm, int s) {
  const int lane = threadIdx.x & 31;
  const int w = s <= 8 ? 8 : s <= 16 ? 16 : 32, nsp = 32 / w;
  const int j = lane & (w - 1), sp = lane / w;
  const int jc = min(j, s - 1);
  for (int c = 0; c < s - 1; ++c) {
    double s0 = 0.0, s1 = 0.0, d0 = 0.0, d1 = 0.0;
    int r = c + 1 + sp;
    for (; r + nsp < s; r += 2 * nsp) {
      const double a = M[r * ldm + c], b = M[(r + nsp) * ldm + c];
      s0 = fma(a, a, s0);
      d0 = fma(a, M[r * ldm + jc], d0);
      s1 = fma(b, b, s1);
      d1 = fma(b, M[(r + nsp) * ldm + jc], d1);
    }
    if (r < s) {
      const double a = M[r * ldm + c];
      s0 = fma(a, a, s0);
      d0 = fma(a, M[r * ldm + jc], d0);
    }
    double sig2 = s0 + s1, dt = d0 + d1;
    for (int o = w; o < 32; o <<= 1) {
      sig2 += __shfl_xor_sync(0xffffffffu, sig2, o);
      dt += __shfl_xor_sync(0xffffffffu, dt, o);
    }
    const double alpha = M[c * ldm + c], mj = M[c * ldm + jc];
    double beta = alpha, tc = 0.0, scale = 1.0;
    if (sig2 != 0.0) {
      beta = -copysign(sqrt(alpha * alpha + sig2), alpha);
      tc = (beta - alpha) / beta;
      scale = 1.0 / (alpha - beta);
    }
    const double wj = tc * fma(scale, dt, mj), f = wj * scale;
    __syncwarp();
    if (j > c && j < s) {
      for (int q = c + 1 + sp; q < s; q += nsp) M[q * ldm + j] = fma(-f, M[q * ldm + c], M[q * ldm + j]);
      if (sp == 0) M[c * ldm + j] = mj - wj;
    }
    if (lane == c) M[c * ldm + c] = beta;
    __syncwarp();
  }
  for (int e = lane; e < s * s; e += 32) {
    const int a = e / s, c = e - a * s;
    if (a > c) M[a * ldm + c] = 0.0;
  }
  __syncwarp();
}

// The same by a whole group (s > 32): a thread per column.
template <int GT>
__device__ void group_core_r(double* M, int ldm, int s, int tg, int bar) {
  for (int c = 0; c < s - 1; ++c) {
    double sig2 = 0.0;
    for (int r = c + 1; r < s; ++r) sig2 = fma(M[r * ldm + c], M[r * ldm + c], sig2);
    const double alpha = M[c * ldm + c];
    double beta = alpha, tc = 0.0, scale = 1.0;
    if (sig2 != 0.0) {
      beta = -copysign(sqrt(alpha * alpha + sig2), alpha);
      tc = (beta - alpha) / beta;
      scale = 1.0 / (alpha - beta);
    }
    for (int j = c + 1 + tg; j < s; j += GT) {
      double d0 = 0.0, d1 = 0.0;
      int r = c + 1;
      for (; r + 1 < s; r += 2) {
        d0 = fma(M[r * ldm + c], M[r * ldm + j], d0);
        d1 = fma(M[(r + 1) * ldm + c], M[(r + 1) * ldm + j], d1);
      }
      if (r < s) d0 = fma(M[r * ldm + c], M[r * ldm + j], d0);
      const double w = tc * fma(scale, d0 + d1, M[c * ldm + j]), f = w * scale;
      for (int q = c + 1; q < s; ++q) M[q * ldm + j] = fma(-f, M[q * ldm + c], M[q * ldm + j]);
      M[c * ldm + j] -= w;
    }
    bar_sync<GT>(bar);
    if (tg == 0) M[c * ldm + c] = beta;
  }
  bar_sync<GT>(bar);
  for (int e = tg; e < s * s; e += GT) {
    const int a = e / s, c = e - a * s;
    if (a > c) M[a * ldm + c] = 0.0;
  }
  bar_sync<GT>(bar);
}

// One-sided Jacobi on the rows of the s x s row-major M by the first nact warps of a group (all call
// it): on return the rows are mutually orthogonal.  Round-robin ordering, eight lanes per pair of rows,
// nn[c] = the squared row norms, fresh at the start of a sweep and updated by the rotation formulas.
// A pair is rotated unless |cos| <= s eps, or a row lies below 1e-14 of the largest norm (the rounding
// noise of the projections).  The angle comes from approximate reciprocals and square roots (a
// relative error of 1e-6 in tan leaves 1e-6 of the pair's cos, which later sweeps remove); the cosine
// is brought to full precision by two steps of Newton's iteration for 1 / sqrt, so each rotation is
// orthogonal to rounding.  A sweep in which every cos and every tan stayed below 3e-9 is the last:
// what it leaves is of the order of their squares.
template <int RL>
__device__ void jacobi_rows(double* M, int ldm, int s, double* nn, unsigned long long* mx, int* flag, int warp,
                            int lane, int nact, int bar) {
  const int h = lane & 7, sub = warp * 4 + (lane >> 3), nsub = 4 * nact;
  const int np = (s + 1) & ~1, npairs = np / 2, iters = (npairs + nsub - 1) / nsub;
  const double tol = (double)(s > 4 ? s : 4) * 2.220446049250313e-16, tol2 = tol * tol;
  auto sync = [&]() {
    if (nact == 1) __syncwarp();
    else bar_sync_n(bar, nact * 32);
  };
  if (warp == 0 && lane == 0) {
    flag[0] = 0;
    mx[0] = 0ull;
  }
  sync();
  for (int sweep = 0; sweep < 40; ++sweep) {
    for (int c0 = 0; c0 < s; c0 += nsub) {
      const int c = c0 + sub;
      double a = 0.0;
      if (c < s)
        for (int e = h; e < s; e += 8) a = fma(M[c * ldm + e], M[c * ldm + e], a);
      a += __shfl_xor_sync(0xffffffffu, a, 4);
      a += __shfl_xor_sync(0xffffffffu, a, 2);
      a += __shfl_xor_sync(0xffffffffu, a, 1);
      if (c < s && h == 0) {
        nn[c] = a;
        atomicMax(&mx[sweep & 1], (unsigned long long)__double_as_longlong(a));
      }
    }
    sync();
    if (warp == 0 && lane == 0) {
      flag[(sweep + 1) & 1] = 0;
      mx[(sweep + 1) & 1] = 0ull;
    }
    const double floor2 = 1e-28 * __longlong_as_double((long long)mx[sweep & 1]);
    for (int round = 0; round < np - 1; ++round) {
      for (int it = 0; it < iters; ++it) {
        const int pr = it * nsub + sub;
        int a = pr - 1 + round, b = np - 2 - pr + round;
        if (a >= np - 1) a -= np - 1;
        if (b >= np - 1) b -= np - 1;
        a = pr == 0 ? 0 : 1 + a;
        b = 1 + b;
        const bool act = pr < npairs && a < s && b < s;
        const int p = act ? min(a, b) : 0, q = act ? max(a, b) : 0;
        double* mp = M + p * ldm;
        double* mq = M + q * ldm;
        constexpr int kL = RL > 0 ? RL : 1;
        double vx[kL], vy[kL], apq = 0.0;
        if (RL > 0) {
#pragma unroll
          for (int i = 0; i < kL; ++i) {
            const int e = h + 8 * i;
            vx[i] = e < s ? mp[e] : 0.0;
            vy[i] = e < s ? mq[e] : 0.0;
            apq = fma(vx[i], vy[i], apq);
          }
        } else {
          for (int e = h; e < s; e += 8) apq = fma(mp[e], mq[e], apq);
        }
        apq += __shfl_xor_sync(0xffffffffu, apq, 4);
        apq += __shfl_xor_sync(0xffffffffu, apq, 2);
        apq += __shfl_xor_sync(0xffffffffu, apq, 1);
        const double app = nn[p], aqq = nn[q], a2 = apq * apq, pq = app * aqq;
        if (act && apq != 0.0 && a2 > tol2 * pq && fmin(app, aqq) > floor2) {
          // tan of the angle: the smaller root of t^2 + 2 zeta t - 1 = 0, zeta = (a_qq - a_pp) / (2 a_pq)
          const double d = aqq - app;
          double tn;
          if (fabs(d) > 2.0e7 * fabs(apq)) tn = apq * rcp_approx(d);
          else {
            const double zeta = 0.5 * d * rcp_approx(apq), w = fma(zeta, zeta, 1.0);
            tn = copysign(rcp_approx(fma(w, rsqrt_approx(w), fabs(zeta))), zeta);
          }
          const double u = fma(tn, tn, 1.0);
          double cs = rsqrt_approx(u);
          cs = fma(0.5 * cs, fma(-u * cs, cs, 1.0), cs);
          cs = fma(0.5 * cs, fma(-u * cs, cs, 1.0), cs);
          const double sn = cs * tn;
          if (RL > 0) {
#pragma unroll
            for (int i = 0; i < kL; ++i) {
              const int e = h + 8 * i;
              if (e < s) {
                mp[e] = cs * vx[i] - sn * vy[i];
                mq[e] = sn * vx[i] + cs * vy[i];
              }
            }
          } else {
            for (int e = h; e < s; e += 8) {
              const double x = mp[e], y = mq[e];
              mp[e] = cs * x - sn * y;
              mq[e] = sn * x + cs * y;
            }
          }
          if (h == 0) {
            nn[p] = app - tn * apq;
            nn[q] = aqq + tn * apq;
            if (a2 > 1e-17 * pq || fabs(tn) > 3e-9) flag[sweep & 1] = 1;
          }
        }
      }
      sync();
    }
    if (!flag[sweep & 1]) break;
  }
}

}  // namespace

// Trailing pairs held by the first m of a rank's rows ii0, ii0 + w, ... (row ii holds ii pairs).
__host__ __device__ inline long rc_pairs_before(long m, long ii0, long w) { return m * ii0 + w * m * (m - 1) / 2; }

long rc_npairs(int k, int nB, int prank, int pworld) {
  const long mB = nB - k - 1;
  const long ii0 = ((prank - (k + 1)) % pworld + pworld) % pworld;
  return rc_pairs_before(ii0 < mB ? (mB - 1 - ii0) / pworld + 1 : 0, ii0, pworld);
}

// Pair qq of the rank's trailing pairs: rows ii (i = k + 1 + ii, i % pworld == prank) hold ii pairs each
// (rows 0..m-1 of the rank C(m) = m ii0 + pworld m (m - 1) / 2); pp = its index among all trailing pairs.
__device__ __forceinline__ void rc_decode(long qq, long ii0, int pworld, int k, int& i, int& j, long& pp) {
  const double hb = (double)ii0 - 0.5 * pworld;
  long m = (long)((-hb + sqrt(hb * hb + 2.0 * pworld * (double)qq)) / pworld);
  while (m > 0 && rc_pairs_before(m, ii0, pworld) > qq) --m;
  while (rc_pairs_before(m + 1, ii0, pworld) <= qq) ++m;
  const int ii = (int)(ii0 + m * pworld), jj = (int)(qq - rc_pairs_before(m, ii0, pworld));
  pp = (long)ii * (ii - 1) / 2 + jj;
  i = k + 1 + ii;
  j = k + 1 + jj;
}

namespace {

// Global scratch of one CTA, for what does not fit in shared memory (wide panels, large cores).
struct WideScratch {
  double *pu, *pv, *cru, *crv, *w, *coefu, *coefv, *m, *gu, *gv, *gb, *tu, *tv;
};

template <int LDX>
__host__ __device__ inline size_t wide_slot(double* base, int cap, WideScratch* out) {
  const size_t c8 = round8(cap), c2 = 2 * (size_t)cap;
  size_t o = 0;
  auto take = [&](size_t n) {
    double* p = base + o;
    o += (n + 1) & ~(size_t)1;
    return p;
  };
  WideScratch s;
  s.pu = take(LDX * c8);
  s.pv = take(LDX * c8);
  s.cru = take(c2 * (c8 + 1));
  s.crv = take(c2 * (c8 + 1));
  s.w = take(c8 * cap);
  s.coefu = take(8 * (size_t)cap);
  s.coefv = take(8 * (size_t)cap);
  s.m = take(c2 * (c2 + 1));
  s.gu = take(c2 * c8);
  s.gv = take(c2 * c8);
  s.gb = take(cap * c8);
  s.tu = take(8 * c8);
  s.tv = take(8 * c8);
  if (out) *out = s;
  return o;
}

struct RcPair {
  long pp;
  int i, j, r1, ri, rj;
};

template <int GW, int NBLK>
struct RcShared {
  static constexpr int kLdx = Side<GW, NBLK>::kLdx;
  static constexpr int kXu = 8 * kLdx > kSmall ? 8 * kLdx : kSmall;
  double xu[kXu];                      // U panel for its QR, product parts; then M, GU, GV, Gb
  double xv[8 * kLdx];                 // V panel: reflectors, then Q3
  double redv[kRu * GW * 64];          // product parts of the V side
  double redn[2][kRu * GW * 8];        // column norm parts
  double coef[2][kFs * 8];             // coefficients of a side's update
  double cr[2][kFs * kLdq];            // [C; R2], [D; R3]
  double w[8 * kFlong];                // W, long side x 8
  double tf[2][64], zt[2][64], tau[2][8], tmp[2][64];
  double qred[2][2 * (8 * GW + 8)];
  double n1[128], ninv[128], nvv[128], nvinv[128];
  double sig[256], srt[256];
  unsigned long long mx[2];
  RcPair pair[2];
  int perm[256];
  int flag[2], rsel;
};

}  // namespace

template <int GW, int NBLK, int MINB>
__global__ void __launch_bounds__(GW * 64, MINB)
    k_recompress(int n, int b, int k, int nB, double* TLR_RESTRICT U, double* TLR_RESTRICT V, int* TLR_RESTRICT rank,
                 int cap, double* TLR_RESTRICT scratch, size_t slot_doubles, int* TLR_RESTRICT next_pair,
                 int* TLR_RESTRICT rlog, int prank, int pworld, long npairs, int* TLR_RESTRICT status) {
  if (*status != 0) return;
  using S = Side<GW, NBLK>;
  constexpr int GT = S::GT, LDX = S::kLdx;
  extern __shared__ __align__(16) unsigned char rc_raw[];
  auto& sm = *reinterpret_cast<RcShared<GW, NBLK>*>(rc_raw);
  const EvalParams& prm = *eval_params(status);
  const int rule_fixed = prm.rule_fixed, rmode = prm.rmode;
  const double thr_rel = prm.thr_rel, thr_abs = prm.thr_abs;
  const long ii0 = ((prank - (k + 1)) % pworld + pworld) % pworld;
  const int tid = threadIdx.x, warp = tid >> 5;
  const int side = warp / GW;  // 0: U, 1: V
  S sd;
  sd.gw = warp - side * GW;
  sd.lane = tid & 31;
  sd.g = sd.lane >> 2;
  sd.t = sd.lane & 3;
  sd.tg = tid - side * GT;
  sd.bar = 1 + side;
  sd.al = (b & 1) == 0;
  WideScratch ws;
  wide_slot<LDX>(scratch + (size_t)blockIdx.x * slot_doubles, cap, &ws);
  const size_t slot = (size_t)b * cap;

  // pairs are handed out dynamically: a CTA starts on pair blockIdx.x and claims the next one while it
  // works (*next_pair counts the claims past the grid; zero at launch); pairs with a zero panel rank
  // are skipped (17:189-194)
  auto fetch = [&](long qq, RcPair& out) {
    for (; qq < npairs; qq = (long)gridDim.x + atomicAdd(next_pair, 1)) {
      RcPair p;
      rc_decode(qq, ii0, pworld, k, p.i, p.j, p.pp);
      p.ri = rank[tidx(p.i, k)];
      p.rj = rank[tidx(p.j, k)];
      if (p.ri == 0 || p.rj == 0) continue;
      p.r1 = rank[tidx(p.i, p.j)];
      out = p;
      return;
    }
    out.i = -1;
  };
  if (blockIdx.x == 0 && tid == 0) {  // the panel column k is read once per step
    double by = 0.0;
    for (int i = k + 1; i < nB; ++i) by += 8.0 * 2.0 * b * rank[tidx(i, k)];
    add_work(status, 10, 0.0, by);
  }
  if (tid == GT) fetch(blockIdx.x, sm.pair[0]);
  __syncthreads();
  for (int turn = 0;; turn ^= 1) {
    const RcPair pr = sm.pair[turn];
    if (pr.i < 0) return;
    const int i = pr.i, j = pr.j, r1 = pr.r1, ri = pr.ri, rj = pr.rj;
    const int bi = min(b, n - i * b), bj = min(b, n - j * b), bk = min(b, n - k * b);
    const int tij = tidx(i, j);
    const size_t oij = (size_t)tij * slot, oik = (size_t)tidx(i, k) * slot, ojk = (size_t)tidx(j, k) * slot;
    const bool short_v = rj <= ri;  // Y = U_jk and X = -U_ik W; else X = U_ik and Y = -U_jk W^T
    const int q = short_v ? rj : ri, lng = short_v ? ri : rj, s = r1 + q;
    const int nblk = (q + 7) >> 3;
    const bool fast = q <= 8 && s <= kFs && lng <= kFlong;
    sd.m = side ? bj : bi;
    const double* Q1 = (side ? V : U) + oij;
    const double* Pk = side ? U + ojk : U + oik;
    double* panel = fast ? (side ? sm.xv : sm.xu) : (side ? ws.pv : ws.pu);
    double* cr = fast ? sm.cr[side] : (side ? ws.crv : ws.cru);
    double* coef = fast ? sm.coef[side] : (side ? ws.coefv : ws.coefu);
    double* tfb = fast ? sm.tf[side] : (side ? ws.tv : ws.tu);
    double* Wq = fast ? sm.w : ws.w;
    const int ldq = fast ? kLdq : round8(cap) + 1;
    double* red = side ? sm.redv : sm.xu;
    double* nrm = side ? sm.nvv : sm.n1;
    double* nrminv = side ? sm.nvinv : sm.ninv;

    // ---- W (long x short) = V_long^T V_short, both groups: parts of kRu x 1 blocks per warp in xu
    {
      const double* vl = V + (short_v ? oik : ojk);
      const double* vs = V + (short_v ? ojk : oik);
      for (int vb = 0; vb < nblk; ++vb) {
        const int nv = min(8, q - 8 * vb);
        const double* sv = vs + (size_t)(8 * vb + min(sd.g, nv - 1)) * b;
        for (int u0 = 0; u0 < lng; u0 += 8 * kRu) {
          const int nub = min(kRu, (lng - u0 + 7) >> 3);
          constexpr int kH = NBLK / 2;
          double2 y[kH];
#pragma unroll
          for (int p = 0; p < kH; ++p) y[p] = load2(sv, 8 * (warp + 2 * GW * p) + 2 * sd.t, bk, sd.al);
          for (int ub = 0; ub < nub; ++ub) {
            const double* su = vl + (size_t)min(u0 + 8 * ub + sd.g, lng - 1) * b;
            double2 x[kH];
#pragma unroll
            for (int p = 0; p < kH; ++p) x[p] = load2(su, 8 * (warp + 2 * GW * p) + 2 * sd.t, bk, sd.al);
            double a0 = 0.0, a1 = 0.0, b0 = 0.0, b1 = 0.0;
#pragma unroll
            for (int p = 0; p < kH; ++p) {
              dmma884(a0, a1, x[p].x, y[p].x);
              dmma884(b0, b1, x[p].y, y[p].y);
            }
            double* rd = sm.xu + (ub * 2 * GW + warp) * 64 + sd.g * 8 + 2 * sd.t;
            rd[0] = a0 + b0;
            rd[1] = a1 + b1;
          }
          __syncthreads();
          for (int e = tid; e < nub * 64; e += 2 * GT) {
            const int ub = e >> 6, uu = (e >> 3) & 7, v = e & 7, u = u0 + 8 * ub + uu;
            if (u < lng) {
              double sum = 0.0;
#pragma unroll
              for (int w = 0; w < 2 * GW; ++w) sum += sm.xu[(ub * 2 * GW + w) * 64 + uu * 8 + v];
              Wq[((size_t)vb * lng + u) * 8 + v] = v < nv ? sum : 0.0;
            }
          }
          __syncthreads();
        }
      }
    }

    // ---- the side's panel, block by block: projection, earlier reflector blocks, QR
    double x[NBLK][2];
    const bool prod = side == 0 ? short_v : !short_v;  // this side's panel is -P W
    for (int vb = 0; vb < nblk; ++vb) {
      const int nv = min(8, q - 8 * vb);
      if (prod) {
#pragma unroll
        for (int p = 0; p < NBLK; ++p) x[p][0] = x[p][1] = 0.0;
        sd.update(x, Pk, b, lng, sd.m, Wq + (size_t)vb * lng * 8, 8, 8, -1.0);
      } else {
        sd.load(x, Pk, b, 8 * vb, nv);
      }
      if (r1 > 0) {
        double* crb = cr + 8 * vb;
        if (vb == 0)
          sd.template dot<true>(x, Q1, b, r1, sd.m, sd.al, red, sm.redn[side], [&](int u, int v, double sum, double n2) {
            const double nr = sqrt(n2), inv = n2 > 0.0 ? 1.0 / nr : 0.0;
            if (v == 0) {
              nrm[u] = nr;
              nrminv[u] = inv;
            }
            const double inc = inv * sum;
            if (v < nv) crb[u * ldq + v] = inc;
            coef[u * 8 + v] = inv * inc;
          });
        else
          sd.template dot<false>(x, Q1, b, r1, sd.m, sd.al, red, nullptr, [&](int u, int v, double sum, double) {
            const double inv = nrminv[u], inc = inv * sum;
            if (v < nv) crb[u * ldq + v] = inc;
            coef[u * 8 + v] = inv * inc;
          });
        sd.update(x, Q1, b, r1, sd.m, coef, 8, 8, -1.0);
        sd.template dot<false>(x, Q1, b, r1, sd.m, sd.al, red, nullptr, [&](int u, int v, double sum, double) {
          const double inv = nrminv[u], inc = inv * sum;
          if (v < nv) crb[u * ldq + v] += inc;
          coef[u * 8 + v] = inv * inc;
        });
        sd.update(x, Q1, b, r1, sd.m, coef, 8, 8, -1.0);
      }
      for (int pb = 0; pb < vb; ++pb)
        sd.apply_block(x, panel + (size_t)pb * 8 * LDX, tfb + pb * 64, true, red, sm.tmp[side], coef);
      double* xs = side ? sm.xv : sm.xu;
      const bool keep = side == 1 || vb + 1 < nblk;
      sd.qr(x, xs, 8 * vb, nv, q, sm.qred[side], cr + (size_t)r1 * ldq + 8 * vb, ldq, sm.zt[side], sm.tau[side],
            tfb + vb * 64, keep ? panel + (size_t)vb * 8 * LDX : nullptr);
    }

    const int ldm = s | 1;
    double* M = s * ldm <= RcShared<GW, NBLK>::kXu && (!fast || s <= kFs) ? sm.xu : ws.m;
    double* GU = fast ? sm.xu + kFs * (kFs + 1) : ws.gu;
    double* GV = fast ? GU + (kFs + kFlong) * kLdg : ws.gv;
    double* Gb = fast ? GV + kFs * kLdg : ws.gb;
    const int ldg = fast ? kLdg : round8(cap);
    if (side == 1) {
      bar_arrive<2 * GT>(3);  // D, R3 and the V norms are in place
      if (sd.tg == 0) fetch((long)gridDim.x + atomicAdd(next_pair, 1), sm.pair[turn ^ 1]);
      // ---- Q3 = the QR's Q, one block of columns at a time from the last, then once more against V_ij
      for (int vb = nblk - 1; vb >= 0; --vb) {
        const int nv = min(8, q - 8 * vb);
#pragma unroll
        for (int p = 0; p < NBLK; ++p) {
          const int row = 8 * (sd.gw + GW * p) + 2 * sd.t;
          x[p][0] = (sd.g < nv && row == 8 * vb + sd.g) ? 1.0 : 0.0;
          x[p][1] = (sd.g < nv && row + 1 == 8 * vb + sd.g) ? 1.0 : 0.0;
        }
        for (int pb = vb; pb >= 0; --pb)
          sd.apply_block(x, panel + (size_t)pb * 8 * LDX, tfb + pb * 64, false, red, sm.tmp[1], coef);
        if (r1 > 0) {
          sd.template dot<false>(x, Q1, b, r1, sd.m, sd.al, red, nullptr, [&](int u, int v, double sum, double) {
            const double inv = nrminv[u];
            coef[u * 8 + v] = inv * inv * sum;
          });
          sd.update(x, Q1, b, r1, sd.m, coef, 8, 8, -1.0);
        }
        __syncwarp();  // a warp reads and writes its own rows of the panel
#pragma unroll
        for (int p = 0; p < NBLK; ++p)
          *reinterpret_cast<double2*>(panel + (size_t)(8 * vb + sd.g) * LDX + 8 * (sd.gw + GW * p) + 2 * sd.t) =
              make_double2(x[p][0], x[p][1]);
        sd.sync();
      }
      bar_sync<2 * GT>(4);  // the rank and the coefficients are in place
    } else {
      bar_sync<2 * GT>(3);
      // ---- core M = diag + [C; R2] [D; R3]^T, its R, the SVD and the rank
      const double* cv = fast ? sm.cr[1] : ws.crv;
      for (int a = sd.gw; a < s; a += GW)
        for (int c = sd.lane; c < s; c += 32) {
          double acc = (a == c && a < r1) ? sm.n1[a] * sm.nvv[a] : 0.0;
          for (int v = 0; v < q; ++v) acc = fma(cr[(size_t)a * ldq + v], cv[(size_t)c * ldq + v], acc);
          M[a * ldm + c] = acc;
        }
      sd.sync();
      if (s <= 32) {
        if (sd.gw == 0) warp_core_r(M, ldm, s);
      } else {
        group_core_r<GT>(M, ldm, s, sd.tg, sd.bar);
      }
      sd.sync();
      const int nact = min(GW, (s + 7) / 8);
      if (s > 1 && sd.gw < nact) {
        if (s <= 16) jacobi_rows<2>(M, ldm, s, sm.sig, sm.mx, sm.flag, sd.gw, sd.lane, nact, 5);
        else if (s <= 32) jacobi_rows<4>(M, ldm, s, sm.sig, sm.mx, sm.flag, sd.gw, sd.lane, nact, 5);
        else jacobi_rows<0>(M, ldm, s, sm.sig, sm.mx, sm.flag, sd.gw, sd.lane, nact, 5);
      }
      sd.sync();
      for (int c0 = 0; c0 < s; c0 += 4 * GW) {  // singular values: the row norms
        const int c = c0 + (sd.tg >> 3), h = sd.lane & 7;
        double a = 0.0;
        if (c < s)
          for (int e = h; e < s; e += 8) a = fma(M[c * ldm + e], M[c * ldm + e], a);
        a += __shfl_xor_sync(0xffffffffu, a, 4);
        a += __shfl_xor_sync(0xffffffffu, a, 2);
        a += __shfl_xor_sync(0xffffffffu, a, 1);
        if (c < s && h == 0) {
          sm.sig[c] = sqrt(a);
          sm.perm[c] = c;
        }
      }
      sd.sync();
      for (int c = sd.tg; c < s; c += GT) {  // descending order, ties by index
        const double sc = sm.sig[c];
        int pos = 0;
        for (int d = 0; d < s; ++d) {
          const double v = sm.sig[d];
          pos += (v > sc) || (v == sc && d < c);
        }
        sm.perm[pos] = c;
        sm.srt[pos] = sc;
      }
      sd.sync();
      if (sd.gw == 0) {
        // tail2[t] = sum_{u >= t} sigma_u^2 from the smallest up (17:113), the smallest rank that meets
        // the threshold
        if (sd.lane == 0) {
          double acc = 0.0;
          for (int c = s - 1; c >= 0; --c) {
            acc += sm.srt[c] * sm.srt[c];
            sm.srt[c] = acc;
          }
        }
        __syncwarp();
        const double thr = rule_fixed ? thr_rel * sqrt(sm.srt[0]) : thr_abs;
        int r = s;
        for (int c0 = 0; c0 < s && r == s; c0 += 32) {
          const int c = c0 + sd.lane;
          const unsigned hit = __ballot_sync(0xffffffffu, c < s && sqrt(sm.srt[c]) <= thr);
          if (hit) r = c0 + __ffs(hit) - 1;
        }
        if (sd.lane == 0) {
          if (rmode == kRankReplay) r = min(rlog[pr.pp], s);  // frozen: the rank recorded at another theta
          else if (rmode == kRankRecord) rlog[pr.pp] = r;
          if (r > cap) {
            atomicCAS(status, 0, -2);
            r = -1;
          }
          sm.rsel = r;
          if (r >= 0)  // 4 b r_ik r_jk + 8 b s^2 + 4 b s r' flops; old and new pair read / written
            add_work(status, 10, 4.0 * b * ri * rj + 8.0 * b * s * s + 4.0 * b * s * r,
                     8.0 * ((double)(bi + bj) * r1 + (double)(bi + bj) * r));
        }
      }
      sd.sync();
      const int rn = sm.rsel;
      if (rn > 0) {
        // right singular vector c of M: row perm[c] over its norm.  GV: coefficients of V_ij and Q3;
        // GU: coefficients of U_ij and U_ik, (R_v^T v_c) with its lower part times -W when X = -U_ik W
        for (int kk = sd.gw; kk < s; kk += GW)
          for (int c = sd.lane; c < rn; c += 32) {
            const int pc = sm.perm[c];
            const double sg = sm.sig[pc], inv = sg > 0.0 ? 1.0 / sg : 0.0;
            const double* vc = M + pc * ldm;
            const double v = vc[kk] * inv;
            GV[kk * ldg + c] = kk < r1 ? v * sm.nvinv[kk] : v;
            if (kk < r1) GU[kk * ldg + c] = v * sm.nvv[kk];
            else {
              double acc = 0.0;
              for (int a = 0; a < s; ++a) acc = fma(cv[(size_t)a * ldq + kk - r1], vc[a], acc);
              (short_v ? Gb + (kk - r1) * ldg : GU + kk * ldg)[c] = acc * inv;
            }
          }
        if (short_v) {
          sd.sync();
          for (int u = sd.gw; u < ri; u += GW)
            for (int c = sd.lane; c < rn; c += 32) {
              double acc = 0.0;
              for (int v = 0; v < q; ++v)
                acc = fma(-Wq[((size_t)(v >> 3) * lng + u) * 8 + (v & 7)], Gb[v * ldg + c], acc);
              GU[(r1 + u) * ldg + c] = acc;
            }
        }
      }
      bar_sync<2 * GT>(4);
    }

    // ---- U' = U_ij G_top + U_ik G_bot, V' = V_ij G_top + Q3 G_bot, over the old pair: a warp reads and
    // writes its own rows, and every product of a row block is formed before its store
    const int rn = sm.rsel;
    if (rn < 0) return;
    double* out = (side ? V : U) + oij;
    const double* co = side ? GV : GU;
    const double* src2 = side ? panel : Pk;
    const int ld2 = side ? LDX : b, n2 = side ? q : ri, m2 = side ? (int)S::kRows : sd.m;
    if (rn > 0 && rn <= 8) {
#pragma unroll
      for (int p = 0; p < NBLK; ++p) x[p][0] = x[p][1] = 0.0;
      if (r1 > 0) sd.update(x, Q1, b, r1, sd.m, co, ldg, rn, 1.0);
      sd.update(x, src2, ld2, n2, m2, co + r1 * ldg, ldg, rn, 1.0);
      __syncwarp();
      if (sd.g < rn) {
        double* o = out + (size_t)sd.g * b;
#pragma unroll
        for (int p = 0; p < NBLK; ++p) {
          const int row = 8 * (sd.gw + GW * p) + 2 * sd.t;
          if (sd.al && row + 1 < sd.m) *reinterpret_cast<double2*>(o + row) = make_double2(x[p][0], x[p][1]);
          else {
            if (row < sd.m) o[row] = x[p][0];
            if (row + 1 < sd.m) o[row + 1] = x[p][1];
          }
        }
      }
    } else if (rn > 8) {
      const int ncb = (rn + 7) >> 3;
      for (int p = 0; p < NBLK; ++p) {
        const int blk = 8 * (sd.gw + GW * p);
        if (blk >= sd.m) break;
        double acc[16][2];
#pragma unroll
        for (int cb = 0; cb < 16; ++cb) acc[cb][0] = acc[cb][1] = 0.0;
        auto part = [&](const double* src, int ld, int nu, int mrow, const double* cf) {
          const int row = blk + sd.g;
          for (int k0 = 0; k0 < nu; k0 += 4) {
            const int u = k0 + sd.t;
            const double bb = (u < nu && row < mrow) ? src[(size_t)u * ld + row] : 0.0;
#pragma unroll
            for (int cb = 0; cb < 16; ++cb)
              if (cb < ncb) {
                const double a = (u < nu && 8 * cb + sd.g < rn) ? cf[u * ldg + 8 * cb + sd.g] : 0.0;
                dmma884(acc[cb][0], acc[cb][1], a, bb);
              }
          }
        };
        if (r1 > 0) part(Q1, b, r1, sd.m, co);
        part(src2, ld2, n2, m2, co + r1 * ldg);
        __syncwarp();
#pragma unroll
        for (int cb = 0; cb < 16; ++cb)
          if (8 * cb + sd.g < rn) {
            double* o = out + (size_t)(8 * cb + sd.g) * b;
            const int row = blk + 2 * sd.t;
            if (row < sd.m) o[row] = acc[cb][0];
            if (row + 1 < sd.m) o[row + 1] = acc[cb][1];
          }
      }
    }
    if (tid == 0) rank[tij] = rn;
    __syncthreads();
  }
}

namespace {

template <int GW, int NBLK, int MINB>
struct RcShape {
  static constexpr int kPerSm = MINB;
  static size_t slot(int cap) { return wide_slot<Side<GW, NBLK>::kLdx>(nullptr, cap, nullptr); }
  static int launch(int grid, int n, int b, int k, int nB, double* U, double* V, int* rank, int cap, double* scratch,
                    size_t slot_doubles, int* next_pair, int* rlog, int prank, int pworld, long npairs, int* status,
                    cudaStream_t s) {
    const size_t sm = sizeof(RcShared<GW, NBLK>);
    cudaFuncSetAttribute(k_recompress<GW, NBLK, MINB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    k_recompress<GW, NBLK, MINB><<<grid, GW * 64, sm, s>>>(n, b, k, nB, U, V, rank, cap, scratch, slot_doubles, next_pair,
                                                           rlog, prank, pworld, npairs, status);
    return (int)cudaGetLastError();
  }
};
using Rc128 = RcShape<4, 4, 3>;
using Rc256 = RcShape<4, 8, 3>;
using Rc512 = RcShape<4, 16, 2>;
using Rc1024 = RcShape<8, 16, 1>;

}  // namespace

int rc_blocks_per_sm(int b) {
  return b <= 128 ? Rc128::kPerSm : b <= 256 ? Rc256::kPerSm : b <= 512 ? Rc512::kPerSm : Rc1024::kPerSm;
}
size_t rc_slot_doubles(int b, int cap) {
  return b <= 128 ? Rc128::slot(cap) : b <= 256 ? Rc256::slot(cap) : b <= 512 ? Rc512::slot(cap) : Rc1024::slot(cap);
}

int launch_recompress(int n, int b, int k, int nB, double* U, double* V, int* rank, int cap, double* scratch,
                      size_t slot_doubles, int nslots, int* next_pair, int* rlog_step, int prank, int pworld,
                      int* status, cudaStream_t s) {
  const long npairs = rc_npairs(k, nB, prank, pworld);
  if (npairs <= 0) return 0;
  const int grid = (int)std::min<long>(npairs, nslots);
  auto run = [&](auto shape) {
    return shape.launch(grid, n, b, k, nB, U, V, rank, cap, scratch, slot_doubles, next_pair, rlog_step, prank, pworld,
                        npairs, status, s);
  };
  if (b <= 128) return run(Rc128{});
  if (b <= 256) return run(Rc256{});
  if (b <= 512) return run(Rc512{});
  return run(Rc1024{});
}

}  // namespace tlr
