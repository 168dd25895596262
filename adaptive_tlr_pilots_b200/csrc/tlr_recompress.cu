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
//   * the core's QR and SVD run in one warp's registers (jacobi_warp), while the V group forms Q3;
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

// Householder reflector of a column with pivot entry alpha and sig2 = the squared norm below it:
// H = I - kappa v v^T, v = (d; the entries below), H maps the column to beta at the pivot (the dlarfg
// sign).  v is left unscaled, kappa = 1 / (nrm (nrm + |alpha|)), so one division follows the square
// root (an FP64 step costs about 23 cycles of latency here, a square root 120, a division 77).
struct Reflector {
  double beta, d, kappa;
};
__device__ __forceinline__ Reflector reflector(double alpha, double sig2) {
  Reflector r{alpha, 0.0, 0.0};
  if (sig2 != 0.0) {
    const double h = fma(alpha, alpha, sig2), nrm = sqrt(h);
    r.beta = -copysign(nrm, alpha);
    r.d = alpha - r.beta;
    r.kappa = 1.0 / fma(fabs(alpha), nrm, h);
  }
  return r;
}

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
                                         const double* coef, int ldc, double sign) const {
    constexpr int kU = NBLK >= 16 ? 1 : 16 / NBLK;  // k steps whose loads are in flight together
#pragma unroll 1
    for (int k0 = 0; k0 < nu; k0 += 4 * kU) {
      double a[kU], b[kU][NBLK];
#pragma unroll
      for (int q = 0; q < kU; ++q) {
        const int u = k0 + 4 * q + t;
        a[q] = u < nu ? sign * coef[u * ldc + g] : 0.0;
        const double* s = src + (size_t)min(u, nu - 1) * ld;
#pragma unroll
        for (int p = 0; p < NBLK; ++p) {
          const int row = 8 * (gw + GW * p) + g;
          b[q][p] = row < mrow ? s[row] : 0.0;
        }
      }
#pragma unroll
      for (int q = 0; q < kU; ++q)
#pragma unroll
        for (int p = 0; p < NBLK; ++p) dmma884(x[p][0], x[p][1], a[q], b[q][p]);
    }
  }

  // The products src^T x (nu x 8): red takes the warps' parts of kRu blocks at a time; entry (u, v) of
  // the sum goes through `put(u, v, sum, norm2)` with the squared norm of column u of src.
  template <class Put>
  __device__ __forceinline__ void dot(const double (&x)[NBLK][2], const double* src, int ld, int nu, int mrow,
                                      bool aligned, double* red, double* redn, Put put) const {
#pragma unroll 1
    for (int u0 = 0; u0 < nu; u0 += 8 * kRu) {
      const int nub = min(kRu, (nu - u0 + 7) >> 3);
#pragma unroll 1
      for (int ub = 0; ub < nub; ++ub) {
        const double* s = src + (size_t)min(u0 + 8 * ub + g, nu - 1) * ld;
        double a0 = 0.0, a1 = 0.0, b0 = 0.0, b1 = 0.0, nn = 0.0;
        constexpr int kCh = NBLK < 8 ? NBLK : 8;
#pragma unroll
        for (int pc = 0; pc < NBLK; pc += kCh) {
          double2 v[kCh];
          if (aligned && 8 * (gw + GW * (pc + kCh - 1)) + 8 <= mrow) {
#pragma unroll
            for (int p = 0; p < kCh; ++p)
              v[p] = *reinterpret_cast<const double2*>(s + 8 * (gw + GW * (pc + p)) + 2 * t);
          } else {
#pragma unroll
            for (int p = 0; p < kCh; ++p) v[p] = load2(s, 8 * (gw + GW * (pc + p)) + 2 * t, mrow, aligned);
          }
#pragma unroll
          for (int p = 0; p < kCh; ++p) {
            dmma884(a0, a1, v[p].x, x[pc + p][0]);
            dmma884(b0, b1, v[p].y, x[pc + p][1]);
            nn = fma(v[p].x, v[p].x, fma(v[p].y, v[p].y, nn));
          }
        }
        double* rd = red + (ub * GW + gw) * 64 + g * 8 + 2 * t;
        rd[0] = a0 + b0;
        rd[1] = a1 + b1;
        nn += __shfl_xor_sync(0xffffffffu, nn, 1);
        nn += __shfl_xor_sync(0xffffffffu, nn, 2);
        if (t == 0) redn[(ub * GW + gw) * 8 + g] = nn;
      }
      sync();
#pragma unroll 1
      for (int e = tg; e < nub * 64; e += GT) {
        const int ub = e >> 6, uu = (e >> 3) & 7, v = e & 7, u = u0 + 8 * ub + uu;
        if (u < nu) {
          double sum = 0.0, n2 = 0.0;
#pragma unroll
          for (int w = 0; w < GW; ++w) {
            sum += red[(ub * GW + w) * 64 + uu * 8 + v];
            n2 += redn[(ub * GW + w) * 8 + uu];
          }
          put(u, v, sum, n2);
        }
      }
      sync();
    }
  }

  // out (ld b, rn columns) = src1 c1 + src2 c2 over the warp's rows, PC row blocks x CB column blocks at
  // a time: every product of a row block is formed before its store, so out may be src1
  template <int CB>
  __device__ __forceinline__ void output(double* out, int b, int rn, const double* src1, int n1, const double* c1,
                                         const double* src2, int ld2, int n2, int m2, const double* c2, int ldc) const {
    constexpr int PC = CB >= NBLK ? 1 : NBLK / CB;
#pragma unroll 1
    for (int p0 = 0; p0 < NBLK; p0 += PC) {
      if (8 * (gw + GW * p0) >= m) break;
      double acc[PC][CB][2];
#pragma unroll
      for (int p = 0; p < PC; ++p)
#pragma unroll
        for (int cb = 0; cb < CB; ++cb) acc[p][cb][0] = acc[p][cb][1] = 0.0;
#pragma unroll 1
      for (int k0 = 0, part = n1 > 0 ? 0 : 1; part < 2;) {
        const int nu = part ? n2 : n1, ld = part ? ld2 : b, mrow = part ? m2 : m;
        const double* cf = part ? c2 : c1;
        const int u = k0 + t;
        const double* s = (part ? src2 : src1) + (size_t)min(u, nu - 1) * ld;
        double bb[PC], a[CB];
#pragma unroll
        for (int p = 0; p < PC; ++p) {
          const int row = 8 * (gw + GW * (p0 + p)) + g;
          bb[p] = row < mrow ? s[row] : 0.0;
        }
#pragma unroll
        for (int cb = 0; cb < CB; ++cb) a[cb] = (u < nu && 8 * cb + g < rn) ? cf[u * ldc + 8 * cb + g] : 0.0;
#pragma unroll
        for (int cb = 0; cb < CB; ++cb)
#pragma unroll
          for (int p = 0; p < PC; ++p) dmma884(acc[p][cb][0], acc[p][cb][1], a[cb], bb[p]);
        k0 += 4;
        if (k0 >= nu) {
          k0 = 0;
          ++part;
        }
      }
      __syncwarp();
#pragma unroll
      for (int cb = 0; cb < CB; ++cb)
        if (8 * cb + g < rn) {
          double* o = out + (size_t)(8 * cb + g) * b;
#pragma unroll
          for (int p = 0; p < PC; ++p) {
            const int row = 8 * (gw + GW * (p0 + p)) + 2 * t;
            if (al && row + 1 < m) *reinterpret_cast<double2*>(o + row) = make_double2(acc[p][cb][0], acc[p][cb][1]);
            else {
              if (row < m) o[row] = acc[p][cb][0];
              if (row + 1 < m) o[row + 1] = acc[p][cb][1];
            }
          }
        }
    }
  }

  // Householder QR of a block of nc columns whose pivots are rows r0 .. r0 + nc - 1 (dlarfg convention);
  // the rows above r0 are final.  The panel passes through xs (kLdx x 8) into registers by rows.  Row r
  // of the block (r <= pivot) goes to R[r ldq + j]; the reflectors (zero above the pivot) to panel when
  // it is given, with their T factor (8 x 8) to tf.  qred: 2 (8 GW + 8) doubles.
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
    // one body for every column (the code of a pair runs once per pair, so its size is instruction
    // fetches): the current column is y[.][0], the panel rotates by one column a step, and position j
    // holds column (j + c) mod 8
#pragma unroll 1
    for (int c = 0; c < nc; ++c) {
      const int piv = r0 + c, live = 8 - c;  // positions from `live` on: finished reflectors
      double p[8], xc[kRpt];
#pragma unroll
      for (int i = 0; i < kRpt; ++i) xc[i] = tg + GT * i > piv ? y[i][0] : 0.0;
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
      const Reflector rf = reflector(pv[0], s[0]);
#pragma unroll
      for (int j = 1; j < 8; ++j) {
        const double z = fma(rf.d, pv[j], s[j]);
        const double w = j < live ? rf.kappa * z : 0.0;
#pragma unroll
        for (int i = 0; i < kRpt; ++i) y[i][j] = fma(-w, xc[i], y[i][j]);
        if (tg == piv) y[0][j] = fma(-w, rf.d, y[0][j]);
        if (tg == 0 && j >= live) zt[(j - live) * 8 + c] = z;  // v_j^T v_c
      }
      if (tg == 0) {
        tau[c] = rf.kappa;
        tau[8 + c] = rf.d;
      }
#pragma unroll
      for (int i = 0; i < kRpt; ++i) {
        double y0 = y[i][0];
        if (i == 0 && tg == piv) y0 = rf.beta;
#pragma unroll
        for (int j = 0; j < 7; ++j) y[i][j] = y[i][j + 1];
        y[i][7] = y0;
      }
    }
    if (tg < nrow) {
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int col = (j + nc) & 7;
        if (col < nc) R[tg * ldq + col] = tg <= r0 + col ? y[0][j] : 0.0;
      }
    }
    if (panel) {
      sync();
#pragma unroll
      for (int i = 0; i < kRpt; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const int row = tg + GT * i, col = (j + nc) & 7;
          panel[col * kLdx + row] = (col >= nc || row < r0 + col) ? 0.0 : (row == r0 + col ? tau[8 + col] : y[i][j]);
        }
      if (tg < 8) {  // row tg of T: T_cc = kappa_c, T_jc = -kappa_c sum_m T_jm (v_m^T v_c)
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

};

// R of the Householder QR of the s x s row-major M by one warp (s <= NR <= 32): lane j holds column j,
// the pivot column is broadcast through buf (2 x 32 doubles), and the rows move up by one a step, so a
// step has no row offset.  The entries below the diagonal are set to zero.
template <int NR>
__device__ __noinline__ void warp_core_r(double* M, int ldm, int s, double* buf) {
  const int j = threadIdx.x & 31;
  double m[NR];
#pragma unroll
  for (int i = 0; i < NR; ++i) m[i] = (i < s && j < s) ? M[i * ldm + j] : 0.0;
#pragma unroll 1
  for (int c = 0; c < s; ++c) {
    double* xb = buf + (c & 1) * 32;
    if (j == c) {
#pragma unroll
      for (int i = 0; i < NR; i += 2) *reinterpret_cast<double2*>(xb + i) = make_double2(m[i], m[i + 1]);
    }
    __syncwarp();
    double x[NR], sa[4] = {0.0, 0.0, 0.0, 0.0}, da[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
    for (int i = 0; i < NR; i += 2) {
      const double2 v = *reinterpret_cast<const double2*>(xb + i);
      x[i] = v.x;
      x[i + 1] = v.y;
    }
#pragma unroll
    for (int i = 1; i < NR; ++i) {
      sa[i & 3] = fma(x[i], x[i], sa[i & 3]);
      da[i & 3] = fma(x[i], m[i], da[i & 3]);
    }
    const Reflector rf = reflector(x[0], (sa[0] + sa[1]) + (sa[2] + sa[3]));
    const double w = rf.kappa * fma(rf.d, m[0], (da[0] + da[1]) + (da[2] + da[3]));
    if (j < s) M[c * ldm + j] = j < c ? 0.0 : (j == c ? rf.beta : fma(-w, rf.d, m[0]));
#pragma unroll
    for (int i = 1; i < NR; ++i) m[i - 1] = fma(-w, x[i], m[i]);
    m[NR - 1] = 0.0;
  }
  __syncwarp();
}

// The same by a whole group (s > 32): a thread per column.
template <int GT>
__device__ void group_core_r(double* M, int ldm, int s, int tg, int bar) {
  for (int c = 0; c < s - 1; ++c) {
    double sg[4] = {0.0, 0.0, 0.0, 0.0};
    for (int r0 = c + 1; r0 < s; r0 += 4)
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const double x = r0 + u < s ? M[(r0 + u) * ldm + c] : 0.0;
        sg[u] = fma(x, x, sg[u]);
      }
    const double sig2 = (sg[0] + sg[1]) + (sg[2] + sg[3]);
    const Reflector rf = reflector(M[c * ldm + c], sig2);
    for (int j = c + 1 + tg; j < s; j += GT) {
      double d0 = 0.0, d1 = 0.0;
      int r = c + 1;
      for (; r + 1 < s; r += 2) {
        d0 = fma(M[r * ldm + c], M[r * ldm + j], d0);
        d1 = fma(M[(r + 1) * ldm + c], M[(r + 1) * ldm + j], d1);
      }
      if (r < s) d0 = fma(M[r * ldm + c], M[r * ldm + j], d0);
      const double w = rf.kappa * fma(rf.d, M[c * ldm + j], d0 + d1);
      for (int q = c + 1; q < s; ++q) M[q * ldm + j] = fma(-w, M[q * ldm + c], M[q * ldm + j]);
      M[c * ldm + j] = fma(-w, rf.d, M[c * ldm + j]);
    }
    bar_sync<GT>(bar);
    if (tg == 0) M[c * ldm + c] = rf.beta;
  }
  bar_sync<GT>(bar);
  for (int e = tg; e < s * s; e += GT) {
    const int a = e / s, c = e - a * s;
    if (a > c) M[a * ldm + c] = 0.0;
  }
  bar_sync<GT>(bar);
}

// One-sided Jacobi on the rows of the s x s row-major M: on return the rows are mutually orthogonal.
// Round-robin ordering.  A pair (p, q) is rotated unless |cos| <= s eps, or a row lies below 1e-14 of the
// largest norm (the rounding noise of the projections).  The squared row norms are fresh at the start
// of a sweep and updated by the rotation formulas.  A sweep in which every cos and every tan stayed
// below 3e-9 is the last: what it leaves is of the order of their squares.
//
// tan of the angle is the smaller root of t^2 + 2 zeta t - 1 = 0, zeta = (a_qq - a_pp) / (2 a_pq), from
// approximate reciprocals and square roots: a relative error of 1e-6 in tan leaves 1e-6 of the pair's
// cos, which later sweeps remove.  The cosine is brought to full precision by the series of
// (1 - e)^(-1/2), so each rotation is orthogonal to rounding.
struct Rotation {
  double tn, cs;
  bool rot, big;
};
__device__ __forceinline__ Rotation rotation(double app, double aqq, double apq, double tol2, double floor2) {
  Rotation r;
  const double a2 = apq * apq, pq = app * aqq;
  r.rot = a2 > tol2 * pq && fmin(app, aqq) > floor2;
  const double zeta = 0.5 * (aqq - app) * rcp_approx(apq), w = fma(zeta, zeta, 1.0);
  r.tn = copysign(rcp_approx(fma(w, rsqrt_approx(w), fabs(zeta))), zeta);
  const double u = fma(r.tn, r.tn, 1.0), c0 = rsqrt_approx(u), e = fma(-u, c0 * c0, 1.0);
  r.cs = fma(c0 * e, fma(0.375, e, 0.5), c0);
  if (!r.rot) {
    r.tn = 0.0;
    r.cs = 1.0;
  }
  r.big = r.rot && (a2 > 1e-17 * pq || fabs(r.tn) > 3e-9);
  return r;
}

// One warp, s <= 64 / LP: LP lanes hold a pair of rows in registers (RL elements of each a lane), and
// the rows move between the lane groups by shuffles after every round (the circle method), so a round
// is one chain without shared memory or barriers: 450 cycles at LP = 4, RL = 4, 710 at LP = 2, RL = 16.
template <int LP, int RL>
__device__ __noinline__ void jacobi_warp(double* M, int ldm, int s) {
  const int lane = threadIdx.x & 31, grp = lane / LP, h = lane % LP;
  const int np = (s + 1) & ~1, m = np / 2, ry = np - 1 - grp;
  const bool first = grp == 0, last = grp == m - 1;
  double x[RL], y[RL];
#pragma unroll
  for (int i = 0; i < RL; ++i) {
    const int e = h + LP * i;
    x[i] = (grp < m && e < s) ? M[grp * ldm + e] : 0.0;
    y[i] = (grp < m && ry < s && e < s) ? M[ry * ldm + e] : 0.0;
  }
  const double tol = (double)(s > 4 ? s : 4) * 2.220446049250313e-16, tol2 = tol * tol;
  auto sum = [&](double a) {
#pragma unroll
    for (int o = LP / 2; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
    return a;
  };
  double floor2 = 0.0;
  for (int sweep = 0; sweep < 40; ++sweep) {
    double nx = 0.0, ny = 0.0;
#pragma unroll
    for (int i = 0; i < RL; ++i) {
      nx = fma(x[i], x[i], nx);
      ny = fma(y[i], y[i], ny);
    }
    nx = sum(nx);
    ny = sum(ny);
    if (sweep == 0) floor2 = 1e-28 * warp_max(fmax(nx, ny));
    bool big = false;
#pragma unroll 1
    for (int round = 0; round < np - 1; ++round) {
      double a[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
      for (int i = 0; i < RL; ++i) a[i & 3] = fma(x[i], y[i], a[i & 3]);
      const double apq = sum(RL > 2 ? (a[0] + a[1]) + (a[2] + a[3]) : a[0] + a[1]);
      const Rotation r = rotation(nx, ny, apq, tol2, floor2);
      big = big || r.big;
      nx = fma(-r.tn, apq, nx);
      ny = fma(r.tn, apq, ny);
      auto move = [&](double& up, double& dn) {  // the upper rows move down a group, the lower ones up
        const double d = __shfl_down_sync(0xffffffffu, up, LP), u = __shfl_up_sync(0xffffffffu, dn, LP);
        up = first ? up : (last ? dn : d);
        dn = first ? d : u;
      };
#pragma unroll
      for (int i = 0; i < RL; ++i) {
        const double xi = x[i];
        x[i] = r.cs * fma(-r.tn, y[i], xi);
        y[i] = r.cs * fma(r.tn, xi, y[i]);
        if (m > 1) move(x[i], y[i]);
      }
      if (m > 1) move(nx, ny);
    }
    if (!__any_sync(0xffffffffu, big)) break;
  }
  // np - 1 rounds bring every row back to its place
#pragma unroll
  for (int i = 0; i < RL; ++i) {
    const int e = h + LP * i;
    if (grp < m && e < s) M[grp * ldm + e] = x[i];
    if (grp < m && ry < s && e < s) M[ry * ldm + e] = y[i];
  }
}

// Larger orders by a whole group of GT threads: eight lanes per pair, the rows in M (shared or global).
template <int GT>
__device__ void jacobi_group(double* M, int ldm, int s, double* nn, unsigned long long* mx, int* flag, int tg, int bar) {
  const int h = tg & 7, sub = tg >> 3;
  constexpr int nsub = GT / 8;
  const int np = (s + 1) & ~1, npairs = np / 2, iters = (npairs + nsub - 1) / nsub;
  const double tol = (double)s * 2.220446049250313e-16, tol2 = tol * tol;
  if (tg == 0) {
    flag[0] = 0;
    mx[0] = 0ull;
  }
  bar_sync<GT>(bar);
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
    bar_sync<GT>(bar);
    if (tg == 0) {  // every read of the last sweep's flag lies before that barrier
      flag[(sweep + 1) & 1] = 0;
      mx[(sweep + 1) & 1] = 0ull;
    }
    const double floor2 = 1e-28 * __longlong_as_double((long long)mx[sweep & 1]);
#pragma unroll 1
    for (int round = 0; round < np - 1; ++round) {
#pragma unroll 1
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
        double apq = 0.0;
#pragma unroll 8
        for (int e = h; e < s; e += 8) apq = fma(mp[e], mq[e], apq);
        apq += __shfl_xor_sync(0xffffffffu, apq, 4);
        apq += __shfl_xor_sync(0xffffffffu, apq, 2);
        apq += __shfl_xor_sync(0xffffffffu, apq, 1);
        const double app = nn[p], aqq = nn[q];
        const Rotation r = rotation(app, aqq, apq, tol2, floor2);
        if (act && r.rot) {
#pragma unroll 4
          for (int e = h; e < s; e += 8) {
            const double x = mp[e], y = mq[e];
            mp[e] = r.cs * fma(-r.tn, y, x);
            mq[e] = r.cs * fma(r.tn, x, y);
          }
          if (h == 0) {
            nn[p] = fma(-r.tn, apq, app);
            nn[q] = fma(r.tn, apq, aqq);
            if (r.big) flag[sweep & 1] = 1;
          }
        }
      }
      bar_sync<GT>(bar);
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
  double xv[8 * kLdx];                 // V panel: reflectors, then Q3 (directly after xu)
  double redv[kRu * GW * 64];          // product parts of the V side
  double redn[2][kRu * GW * 8];        // column norm parts
  double coef[2][kFs * 8];             // coefficients of a side's update
  double cr[2][kFs * kLdq];            // [C; R2], [D; R3]
  double w[8 * kFlong];                // W, long side x 8
  double tf[2][64], zt[2][64], tau[2][16], tmp[2][64];
  double qred[2][2 * (8 * GW + 8)];
  double n1[128], ninv[128], nvv[128], nvinv[128];
  double sig[256], val[256], srt[256];
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

    const int ldm = s | 1;
    // the core lies over xu (wide pairs: over xu and xv, whose panel is in the scratch slot)
    double* M = s * ldm <= RcShared<GW, NBLK>::kXu + 8 * LDX ? sm.xu : ws.m;
    double* GU = fast ? sm.xu + kFs * (kFs + 1) : ws.gu;
    double* GV = fast ? GU + (kFs + kFlong) * kLdg : ws.gv;
    double* Gb = fast ? GV + kFs * kLdg : ws.gb;
    const int ldg = fast ? kLdg : round8(cap);

    // ---- stage 0: the side's panel, block by block: projection, earlier reflector blocks, QR.
    // Stage 1 (V side): Q3 = the QR's Q, a block of columns at a time from the last, then once more
    // against V_ij.  Both are a list of steps x <- x - src coef with coef from the products src^T x, and
    // share one copy of the code.
    const bool prod = side == 0 ? short_v : !short_v;  // this side's panel is -P W
#pragma unroll 1
    for (int stage = 0; stage <= side; ++stage) {
#pragma unroll 1
      for (int bb = 0; bb < nblk; ++bb) {
        const int vb = stage == 0 ? bb : nblk - 1 - bb, nv = min(8, q - 8 * vb);
        double x[NBLK][2];
        if (stage == 0 && !prod) {
          sd.load(x, Pk, b, 8 * vb, nv);
        } else {
#pragma unroll
          for (int p = 0; p < NBLK; ++p) {
            const int row = 8 * (sd.gw + GW * p) + 2 * sd.t - 8 * vb;
            const bool unit = stage == 1 && sd.g < nv;
            x[p][0] = (unit && row == sd.g) ? 1.0 : 0.0;
            x[p][1] = (unit && row + 1 == sd.g) ? 1.0 : 0.0;
          }
        }
        // steps of stage 0: [-P W], Q1, Q1, blocks 0 .. vb - 1; of stage 1: blocks vb .. 0, Q1
        const int pre = stage == 0 && prod ? 1 : 0, nq = r1 > 0 ? (stage == 0 ? 2 : 1) : 0;
        const int nsteps = pre + nq + (stage == 0 ? vb : vb + 1);
#pragma unroll 1
        for (int st = 0; st < nsteps; ++st) {
          const int at = st - pre;  // < 0: the product -P W
          const bool onq = at >= 0 && (stage == 0 ? at < nq : at > vb);
          const double *src = Pk, *cf = Wq + (size_t)vb * lng * 8;
          int ld = b, nu = lng, mrow = sd.m;
          if (at >= 0) {
            const int pb = stage == 0 ? at - nq : vb - at;
            src = onq ? Q1 : panel + (size_t)pb * 8 * LDX;
            ld = onq ? b : LDX;
            nu = onq ? r1 : 8;
            mrow = onq ? sd.m : (int)S::kRows;
            cf = coef;
            const bool norms = onq && stage == 0 && vb == 0 && at == 0;
            double* crb = onq && stage == 0 ? cr + 8 * vb : nullptr;
            double* tmp = sm.tmp[side];
            sd.dot(x, src, ld, nu, mrow, onq ? sd.al : true, red, sm.redn[side], [&](int u, int v, double sum, double n2) {
              if (!onq) {
                tmp[u * 8 + v] = sum;
                return;
              }
              double inv;
              if (norms) {
                const double nr = sqrt(n2);
                inv = n2 > 0.0 ? 1.0 / nr : 0.0;
                if (v == 0) {
                  nrm[u] = nr;
                  nrminv[u] = inv;
                }
              } else {
                inv = nrminv[u];
              }
              const double inc = inv * sum;
              if (crb && v < nv) crb[u * ldq + v] = at == 0 ? inc : crb[u * ldq + v] + inc;
              coef[u * 8 + v] = inv * inc;
            });
            if (!onq) {  // (I - V T^T V^T) x in stage 0, (I - V T V^T) x in stage 1
              const double* tf = tfb + pb * 64;
              for (int e = sd.tg; e < 64; e += GT) {
                const int u = e >> 3, v = e & 7;
                double acc = 0.0;
#pragma unroll
                for (int kk = 0; kk < 8; ++kk) acc = fma(stage == 0 ? tf[kk * 8 + u] : tf[u * 8 + kk], tmp[kk * 8 + v], acc);
                coef[e] = acc;
              }
              sd.sync();
            }
          }
          sd.update(x, src, ld, nu, mrow, cf, 8, -1.0);
        }
        if (stage == 0) {
          double* xs = side ? sm.xv : sm.xu;
          const bool keep = side == 1 || vb + 1 < nblk;
          sd.qr(x, xs, 8 * vb, nv, q, sm.qred[side], cr + (size_t)r1 * ldq + 8 * vb, ldq, sm.zt[side], sm.tau[side],
                tfb + vb * 64, keep ? panel + (size_t)vb * 8 * LDX : nullptr);
        } else {
          __syncwarp();  // a warp reads and writes its own rows of the panel
#pragma unroll
          for (int p = 0; p < NBLK; ++p)
            *reinterpret_cast<double2*>(panel + (size_t)(8 * vb + sd.g) * LDX + 8 * (sd.gw + GW * p) + 2 * sd.t) =
                make_double2(x[p][0], x[p][1]);
          sd.sync();
        }
      }
      if (side == 1 && stage == 0) {
        bar_arrive<2 * GT>(3);  // D, R3 and the V norms are in place
        if (sd.tg == 0) fetch((long)gridDim.x + atomicAdd(next_pair, 1), sm.pair[turn ^ 1]);
      }
    }

    if (side == 1) {
      bar_sync<2 * GT>(4);  // the rank and the coefficients are in place
    } else {
      bar_sync<2 * GT>(3);
      // ---- core M = diag + [C; R2] [D; R3]^T, its R, the SVD and the rank
      const double* cv = fast ? sm.cr[1] : ws.crv;
      for (int e = sd.tg; e < s * s; e += GT) {
        const int a = e / s, c = e - a * s;
        const double *ca = cr + (size_t)a * ldq, *cc = cv + (size_t)c * ldq;
        double a0 = (a == c && a < r1) ? sm.n1[a] * sm.nvv[a] : 0.0, a1 = 0.0;
        for (int v = 0; v < q; v += 2) {
          a0 = fma(ca[v], cc[v], a0);
          if (v + 1 < q) a1 = fma(ca[v + 1], cc[v + 1], a1);
        }
        M[a * ldm + c] = a0 + a1;
      }
      sd.sync();
      if (s <= 32) {
        if (sd.gw == 0) {
          if (s <= 8) warp_core_r<8>(M, ldm, s, sm.srt);
          else if (s <= 16) warp_core_r<16>(M, ldm, s, sm.srt);
          else if (s <= 24) warp_core_r<24>(M, ldm, s, sm.srt);
          else warp_core_r<32>(M, ldm, s, sm.srt);
        }
      } else {
        group_core_r<GT>(M, ldm, s, sd.tg, sd.bar);
      }
      sd.sync();
      if (s <= 32) {
        if (sd.gw == 0) {
          if (s <= 8) jacobi_warp<4, 2>(M, ldm, s);
          else if (s <= 16) jacobi_warp<4, 4>(M, ldm, s);
          else jacobi_warp<2, 16>(M, ldm, s);
        }
      } else {
        jacobi_group<GT>(M, ldm, s, sm.sig, sm.mx, sm.flag, sd.tg, sd.bar);
      }
      sd.sync();
      for (int c0 = 0; c0 < s; c0 += 8 * GW) {  // singular values: the row norms; sig = their reciprocals
        const int c = c0 + (sd.tg >> 2), h = sd.lane & 3;
        double a0 = 0.0, a1 = 0.0;
        if (c < s)
          for (int e = h; e < s; e += 8) {
            a0 = fma(M[c * ldm + e], M[c * ldm + e], a0);
            if (e + 4 < s) a1 = fma(M[c * ldm + e + 4], M[c * ldm + e + 4], a1);
          }
        double a = a0 + a1;
        a += __shfl_xor_sync(0xffffffffu, a, 2);
        a += __shfl_xor_sync(0xffffffffu, a, 1);
        if (c < s && h == 0) {
          const double nr = sqrt(a);
          sm.sig[c] = nr > 0.0 ? 1.0 / nr : 0.0;
          sm.val[c] = nr;
          sm.perm[c] = c;
        }
      }
      sd.sync();
      for (int c = sd.tg; c < s; c += GT) {  // descending order, ties by index
        const double sc = sm.val[c];
        int pos = 0;
#pragma unroll 4
        for (int d = 0; d < s; ++d) {
          const double v = sm.val[d];
          pos += (v > sc) || (v == sc && d < c);
        }
        sm.perm[pos] = c;
        sm.srt[pos] = sc * sc;
      }
      sd.sync();
      if (sd.gw == 0) {
        // tail2[t] = sum_{u >= t} sigma_u^2 from the smallest up (17:113), the smallest rank that meets
        // the threshold
        if (s <= 32) {
          double a = sd.lane < s ? sm.srt[sd.lane] : 0.0;
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            const double up = __shfl_down_sync(0xffffffffu, a, o);
            if (sd.lane + o < 32) a += up;
          }
          if (sd.lane < s) sm.srt[sd.lane] = a;
        } else if (sd.lane == 0) {
          double acc = 0.0;
          for (int c = s - 1; c >= 0; --c) {
            acc += sm.srt[c];
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
      bar_sync<2 * GT>(4);
    }

    // ---- coefficients of the new pair; right singular vector c of M is row perm[c] over its norm.
    // V side, GV: of V_ij and Q3.  U side, GU: of U_ij and U_ik, R_v^T v_c with its lower part times -W
    // when X = -U_ik W
    const int rn = sm.rsel;
    if (rn < 0) return;
    for (int e = sd.tg; e < s * rn; e += GT) {
      const int kk = e / rn, c = e - kk * rn;
      const int pc = sm.perm[c];
      const double inv = sm.sig[pc];
      const double* vc = M + pc * ldm;
      if (side == 1) {
        GV[kk * ldg + c] = vc[kk] * inv * (kk < r1 ? sm.nvinv[kk] : 1.0);
      } else if (kk < r1) {
        GU[kk * ldg + c] = vc[kk] * inv * sm.nvv[kk];
      } else {
        const double* dv = (fast ? sm.cr[1] : ws.crv) + (kk - r1);
        double a0 = 0.0, a1 = 0.0;
        for (int a = 0; a < s; a += 2) {
          a0 = fma(dv[(size_t)a * ldq], vc[a], a0);
          if (a + 1 < s) a1 = fma(dv[(size_t)(a + 1) * ldq], vc[a + 1], a1);
        }
        (short_v ? Gb + (kk - r1) * ldg : GU + kk * ldg)[c] = (a0 + a1) * inv;
      }
    }
    sd.sync();
    if (side == 0 && short_v) {
      for (int e = sd.tg; e < ri * rn; e += GT) {
        const int u = e / rn, c = e - u * rn;
        double a0 = 0.0, a1 = 0.0;
        for (int v = 0; v < q; v += 2) {
          const double* w = Wq + ((size_t)(v >> 3) * lng + u) * 8 + (v & 7);
          a0 = fma(-w[0], Gb[v * ldg + c], a0);
          if (v + 1 < q) a1 = fma(-w[1], Gb[(v + 1) * ldg + c], a1);
        }
        GU[(r1 + u) * ldg + c] = a0 + a1;
      }
      sd.sync();
    }

    // ---- U' = U_ij G_top + U_ik G_bot, V' = V_ij G_top + Q3 G_bot, over the old pair: a warp reads and
    // writes its own rows
    if (rn > 0) {
      double* out = (side ? V : U) + oij;
      const double* co = side ? GV : GU;
      const double* src2 = side ? panel : Pk;
      const int ld2 = side ? LDX : b, n2 = side ? q : ri, m2 = side ? (int)S::kRows : sd.m;
      if (rn <= 8) sd.template output<1>(out, b, rn, Q1, r1, co, src2, ld2, n2, m2, co + r1 * ldg, ldg);
      else if (rn <= 16) sd.template output<2>(out, b, rn, Q1, r1, co, src2, ld2, n2, m2, co + r1 * ldg, ldg);
      else if (rn <= 32) sd.template output<4>(out, b, rn, Q1, r1, co, src2, ld2, n2, m2, co + r1 * ldg, ldg);
      else sd.template output<16>(out, b, rn, Q1, r1, co, src2, ld2, n2, m2, co + r1 * ldg, ldg);
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
using Rc128 = RcShape<4, 4, 2>;
using Rc256 = RcShape<4, 8, 2>;
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
