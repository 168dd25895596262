// Panel building blocks shared by the recompression and the initial compression: tall panels of 8
// columns in the FP64 tensor cores' fragment layout, their products, Householder QR and blocked
// reflectors, and one-sided Jacobi on small cores.
#pragma once
#include "tlr_device.cuh"

namespace tlr {

constexpr int kRu = 3;  // blocks of 8 columns per reduction of a product

// Householder reflector of a column with pivot entry alpha and sig2 = the squared norm below it:
// H = I - kappa v v^T, v = (d; the entries below), H maps the column to beta at the pivot (the dlarfg
// sign).  v is left unscaled, kappa = 1 / (nrm (nrm + |alpha|)), so one division follows the square
// root (an FP64 step costs about 23 cycles of latency here, a square root 120, a division 77).
// The squared norm alpha^2 + sig2 has to lie within 2^-500 .. 2^500: past that kappa and the products with v
// would leave the range of a double (kappa is infinite for norms below 7e-155, and the columns of T^T T P
// are squares of a tile's entries).  A column outside is first multiplied by 2^(500 column_lift), which changes
// no bit of the reflector; beta is divided by it.  Integers, so that an ordinary column pays a few cycles.
__device__ __forceinline__ int column_lift(double norm2) {
  constexpr int kLow = (1023 - 500) << 20, kHigh = (1023 + 500) << 20;  // high words of 2^-500, 2^500
  if ((unsigned)(__double2hiint(norm2) - kLow) <= (unsigned)(kHigh - kLow) || norm2 == 0.0) return 0;
  return norm2 < 1.0 ? 1 : -1;
}
__device__ __forceinline__ double lifted(int lift, double v) {
  return lift == 0 ? v : v * (lift > 0 ? 0x1p500 : 0x1p-500);
}
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
    int lift = 0;
#pragma unroll 1
    for (int c = 0, step = 0; c < nc; ++step) {
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
      double* rb = qred + (step & 1) * (8 * GW + 8);
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
      if (lift == 0) {
        lift = column_lift(fma(pv[0], pv[0], s[0]));
        if (lift != 0) {  // the same in every thread: the rows from the pivot on, and the sums once more
#pragma unroll
          for (int i = 0; i < kRpt; ++i)
            if (tg + GT * i >= piv) y[i][0] = lifted(lift, y[i][0]);
          continue;
        }
      }
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
        if (i == 0 && tg == piv) y0 = lifted(-lift, rf.beta);
#pragma unroll
        for (int j = 0; j < 7; ++j) y[i][j] = y[i][j + 1];
        y[i][7] = y0;
      }
      lift = 0;
      ++c;
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
    double x[NR], sig2, dt;
    int lift = 0;
#pragma unroll
    for (int i = 0; i < NR; i += 2) {
      const double2 v = *reinterpret_cast<const double2*>(xb + i);
      x[i] = v.x;
      x[i + 1] = v.y;
    }
#pragma unroll 1
    for (;;) {
      double sa[4] = {0.0, 0.0, 0.0, 0.0}, da[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
      for (int i = 1; i < NR; ++i) {
        sa[i & 3] = fma(x[i], x[i], sa[i & 3]);
        da[i & 3] = fma(x[i], m[i], da[i & 3]);
      }
      sig2 = (sa[0] + sa[1]) + (sa[2] + sa[3]);
      dt = (da[0] + da[1]) + (da[2] + da[3]);
      if (lift != 0) break;
      lift = column_lift(fma(x[0], x[0], sig2));
      if (lift == 0) break;
#pragma unroll
      for (int i = 0; i < NR; ++i) x[i] = lifted(lift, x[i]);
    }
    const Reflector rf = reflector(x[0], sig2);
    const double w = rf.kappa * fma(rf.d, m[0], dt);
    if (j < s) M[c * ldm + j] = j < c ? 0.0 : (j == c ? lifted(-lift, rf.beta) : fma(-w, rf.d, m[0]));
#pragma unroll
    for (int i = 1; i < NR; ++i) m[i - 1] = fma(-w, x[i], m[i]);
    m[NR - 1] = 0.0;
  }
  __syncwarp();
}

// The same by a whole group (s > 32): the rows of a column split over up to four adjacent lanes.
template <int GT, bool SHARED>
__device__ __noinline__ void group_core_r(double* M, int ldm, int s, int tg, int bar) {
  if (SHARED) __builtin_assume(__isShared(M));
  const int nsp = s <= GT / 4 ? 4 : s <= GT / 2 ? 2 : 1, sp = tg % nsp;
  for (int c = 0; c < s - 1; ++c) {
    double sig2, alpha = M[c * ldm + c];
    int lift = 0;
#pragma unroll 1
    for (;;) {
      double sg[4] = {0.0, 0.0, 0.0, 0.0};
      for (int r0 = c + 1 + sp; r0 < s; r0 += 8 * nsp) {
        double x[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) x[u] = r0 + u * nsp < s ? M[(r0 + u * nsp) * ldm + c] : 0.0;
#pragma unroll
        for (int u = 0; u < 8; ++u) sg[u & 3] = fma(x[u], x[u], sg[u & 3]);
      }
      sig2 = (sg[0] + sg[1]) + (sg[2] + sg[3]);
      for (int o = 1; o < nsp; o <<= 1) sig2 += __shfl_xor_sync(0xffffffffu, sig2, o);
      if (lift != 0) break;
      lift = column_lift(fma(alpha, alpha, sig2));
      if (lift == 0) break;
      bar_sync<GT>(bar);  // the same in every thread: the column below the pivot is the reflector's alone
      for (int r = c + 1 + tg; r < s; r += GT) M[r * ldm + c] = lifted(lift, M[r * ldm + c]);
      alpha = lifted(lift, alpha);
      bar_sync<GT>(bar);
    }
    const Reflector rf = reflector(alpha, sig2);
    const int step = GT / nsp;
    for (int j0 = c + 1; j0 < s; j0 += step) {  // the same trip count in every thread (shuffles)
      const int j = j0 + tg / nsp, jc = min(j, s - 1);
      double d[4] = {0.0, 0.0, 0.0, 0.0};
      for (int r0 = c + 1 + sp; r0 < s; r0 += 8 * nsp) {
        double x[8], y[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const bool in = r0 + u * nsp < s;
          x[u] = in ? M[(r0 + u * nsp) * ldm + c] : 0.0;
          y[u] = in ? M[(r0 + u * nsp) * ldm + jc] : 0.0;
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) d[u & 3] = fma(x[u], y[u], d[u & 3]);
      }
      double dt = (d[0] + d[1]) + (d[2] + d[3]);
      for (int o = 1; o < nsp; o <<= 1) dt += __shfl_xor_sync(0xffffffffu, dt, o);
      const double mj = M[c * ldm + jc], w = rf.kappa * fma(rf.d, mj, dt);
      __syncwarp();
      if (j < s) {
        // eight rows at a time: their loads come ahead of the stores, which the compiler could not reorder
        for (int q0 = c + 1 + sp; q0 < s; q0 += 8 * nsp) {
          double xc[8], xj[8];
#pragma unroll
          for (int u = 0; u < 8; ++u) {
            const int q = min(q0 + u * nsp, s - 1);
            xc[u] = M[q * ldm + c];
            xj[u] = M[q * ldm + j];
          }
#pragma unroll
          for (int u = 0; u < 8; ++u)
            if (q0 + u * nsp < s) M[(q0 + u * nsp) * ldm + j] = fma(-w, xc[u], xj[u]);
        }
        if (sp == 0) M[c * ldm + j] = fma(-w, rf.d, mj);
      }
    }
    bar_sync<GT>(bar);
    if (tg == 0) M[c * ldm + c] = lifted(-lift, rf.beta);
  }
  bar_sync<GT>(bar);
  for (int e = tg; e < s * s; e += GT) {
    const int a = e / s, c = e - a * s;
    if (a > c) M[a * ldm + c] = 0.0;
  }
  bar_sync<GT>(bar);
}

// One-sided Jacobi on the rows of the s x s row-major M: on return the rows are mutually orthogonal.
// Round-robin ordering.  A pair (p, q) is rotated unless |cos| <= s eps, or a row's squared norm lies below
// floor_rel times the largest: 1e-28 in the recompression (the rounding noise of the projections), 1e-200 in the
// initial compression, whose small rows carry right vectors that have to be orthonormal as well (what is
// left out there only keeps the angle's quotients within the range of a double).  The squared row norms are fresh at the start
// of a sweep and updated by the rotation formulas.  A sweep in which every cos and every tan stayed
// below 3e-9 is the last: what it leaves is of the order of their squares.
//
// tan of the angle is the smaller root of a_pq t^2 + (a_qq - a_pp) t - a_pq = 0: from approximate reciprocals
// and square roots (about 1e-6), then one step of Newton's method on that equation (about 1e-12).  Without
// the step each rotation leaves 1e-6 of the pair's cos, so the last sweep ends at 3e-15 instead of
// rounding level, and columns of U 1e-8 below the first lose their orthogonality (the structured
// projection relies on it: the log-likelihood under the fixed rule 1e-8 at N = 20,000 moved by 5e-8).
// The cosine is brought to full precision by the series of (1 - e)^(-1/2), so each rotation is
// orthogonal to rounding.
struct Rotation {
  double tn, cs;
  bool rot, big;
};
__device__ __forceinline__ Rotation rotation(double app, double aqq, double apq, double tol2, double floor2) {
  Rotation r;
  const double a2 = apq * apq, pq = app * aqq;
  r.rot = a2 > tol2 * pq && fmin(app, aqq) > floor2;
  const double d = aqq - app, zeta = 0.5 * d * rcp_approx(apq), w = fma(zeta, zeta, 1.0);
  const double t0 = copysign(rcp_approx(fma(w, rsqrt_approx(w), fabs(zeta))), zeta);
  r.tn = fma(-fma(fma(apq, t0, d), t0, -apq), rcp_approx(fma(2.0 * apq, t0, d)), t0);
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
__device__ __noinline__ void jacobi_warp(double* M, int ldm, int s, double floor_rel) {
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
    if (sweep == 0) floor2 = floor_rel * warp_max(fmax(nx, ny));
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

// Larger orders by a whole group of GT threads, the rows in M (shared or global): LP lanes per pair, RL
// elements a lane in registers (s <= LP RL where they are to hold it all: lanes past s still take FP64 slots,
// so the caller picks RL by s).
template <int GT, int LP, int RL, bool SHARED>
__device__ __noinline__ void jacobi_group(double* M, int ldm, int s, double floor_rel, double* nn, unsigned long long* mx,
                                          int* flag, int tg, int bar) {
  if (SHARED) __builtin_assume(__isShared(M));
  __builtin_assume(__isShared(nn));
  const int h = tg % LP, sub = tg / LP;
  constexpr int nsub = GT / LP;
  auto sum = [&](double a) {
#pragma unroll
    for (int o = LP / 2; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
    return a;
  };
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
        for (int e = h; e < s; e += LP) a = fma(M[c * ldm + e], M[c * ldm + e], a);
      a = sum(a);
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
    const double floor2 = floor_rel * __longlong_as_double((long long)mx[sweep & 1]);
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
        // the pair's elements in registers between the product and the rotation (RL a lane; past that only
        // the first RL stay, the others are read again)
        double vx[RL], vy[RL], d[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
        for (int u = 0; u < RL; ++u) {
          const int e = h + u * LP;
          vx[u] = e < s ? mp[e] : 0.0;
          vy[u] = e < s ? mq[e] : 0.0;
        }
#pragma unroll
        for (int u = 0; u < RL; ++u) d[u & 3] = fma(vx[u], vy[u], d[u & 3]);
        for (int e = h + RL * LP; e < s; e += LP) d[0] = fma(mp[e], mq[e], d[0]);
        const double apq = sum((d[0] + d[1]) + (d[2] + d[3]));
        const double app = nn[p], aqq = nn[q];
        __syncwarp();  // every lane of the pair has the norms that lane h = 0 replaces below
        const Rotation r = rotation(app, aqq, apq, tol2, floor2);
        if (act && r.rot) {
#pragma unroll
          for (int u = 0; u < RL; ++u) {
            const int e = h + u * LP;
            if (e < s) {
              mp[e] = r.cs * fma(-r.tn, vy[u], vx[u]);
              mq[e] = r.cs * fma(r.tn, vx[u], vy[u]);
            }
          }
          for (int e = h + RL * LP; e < s; e += LP) {
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

}  // namespace tlr
