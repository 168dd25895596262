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
//
// Recompression per FP64 evaluation, against one group of 256 threads per pair with a column at a time in
// shared memory: N = 1,030, b = 100 3.7 -> 0.78 ms; N = 10,007, b = 250 17.9 -> 4.8; N = 50,000, b = 500
// 138 -> 45.6; N = 20,000, b = 500, range 0.1 (ranks to 65) 382 -> 52.  The range test of the reflectors
// (tlr_panel.cuh) is 1 to 4 % of that (43.9 without it at N = 50,000).
#include "tlr_kernels.h"
#include "tlr_panel.cuh"

namespace tlr {

namespace {

constexpr int kFs = 32;      // largest core order kept in shared memory whole (M, G, H and C)
constexpr int kFlong = 24;   // largest long side of W kept in shared memory
constexpr int kLdq = 9;      // row pitch of the shared [C; R] arrays
constexpr int kLdg = 32;     // row pitch of the shared G arrays
constexpr double kFloor = 1e-28;  // rows of a core below 1e-14 of its largest are rounding noise
constexpr int kSmall = kFs * (kFs + 1) + (kFs + kFlong) * kLdg + kFs * kLdg + 8 * kLdg;  // M, GU, GV, Gb

__device__ __forceinline__ int tidx(int i, int j) { return i * (i - 1) / 2 + j; }
__host__ __device__ constexpr int round8(int v) { return (v + 7) & ~7; }

}  // namespace

// Trailing pairs held by the first m of a rank's rows ii0, ii0 + w, ... (row ii holds ii pairs).
__host__ __device__ inline long rc_pairs_before(long m, long ii0, long w) { return m * ii0 + w * m * (m - 1) / 2; }

long rc_npairs(int k, int nB, int prank, int pworld) {
  const long mB = nB - k - 1;
  const long ii0 = ((prank - (k + 1)) % pworld + pworld) % pworld;
  return rc_pairs_before(ii0 < mB ? (mB - 1 - ii0) / pworld + 1 : 0, ii0, pworld);
}

// Pair qq of the rank's trailing pairs (i, j); pp = its index among all trailing pairs in the order of the
// rank map (row ii, then jj).  On one rank the pairs come by distance from the diagonal, i - j = 1 first: the
// ranks fall with it, so the longest pairs start first.  On a block-row partition rows ii (i = k + 1 + ii,
// i % pworld == prank) hold ii pairs each (rows 0..m-1 of the rank C(m) = m ii0 + pworld m (m - 1) / 2).
__device__ __forceinline__ void rc_decode(long qq, long npairs, long ii0, int pworld, int k, int mB, int& i, int& j,
                                          long& pp) {
  if (pworld == 1) qq = npairs - 1 - qq;
  const double hb = (double)ii0 - 0.5 * pworld;
  long m = (long)((-hb + sqrt(hb * hb + 2.0 * pworld * (double)qq)) / pworld);
  while (m > 0 && rc_pairs_before(m, ii0, pworld) > qq) --m;
  while (rc_pairs_before(m + 1, ii0, pworld) <= qq) ++m;
  int ii = (int)(ii0 + m * pworld), jj = (int)(qq - rc_pairs_before(m, ii0, pworld));
  if (pworld == 1) ii = mB - ii + jj;  // group ii holds the ii pairs at distance mB - ii
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

template <int GW, int NBLK, int XU>
struct RcShared {
  static constexpr int kLdx = Side<GW, NBLK>::kLdx;
  static constexpr int kXu0 = 8 * kLdx > kSmall ? 8 * kLdx : kSmall;
  static constexpr int kXu = XU > kXu0 ? XU : kXu0;
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

template <int GW, int NBLK, int MINB, int XU>
__global__ void __launch_bounds__(GW * 64, MINB)
    k_recompress(int n, int b, int k, int nB, double* TLR_RESTRICT U, double* TLR_RESTRICT V, int* TLR_RESTRICT rank,
                 int cap, double* TLR_RESTRICT scratch, size_t slot_doubles, int* TLR_RESTRICT next_pair,
                 int* TLR_RESTRICT rlog, int prank, int pworld, long npairs, int* TLR_RESTRICT status) {
  if (cta_failed(status)) return;
  using S = Side<GW, NBLK>;
  constexpr int GT = S::GT, LDX = S::kLdx;
  extern __shared__ __align__(16) unsigned char rc_raw[];
  auto& sm = *reinterpret_cast<RcShared<GW, NBLK, XU>*>(rc_raw);
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
      rc_decode(qq, npairs, ii0, pworld, k, nB - k - 1, p.i, p.j, p.pp);
      p.ri = rank[tidx(p.i, k)];
      p.rj = rank[tidx(p.j, k)];
      if (p.ri == 0 || p.rj == 0) continue;
      p.r1 = rank[tidx(p.i, p.j)];
      out = p;
      return;
    }
    out.i = -1;
  };
  if (blockIdx.x == 0 && tid < 32) {  // the panel column k is read once per step
    int sum = 0;
    for (int i = k + 1 + tid; i < nB; i += 32) sum += rank[tidx(i, k)];
    sum = __reduce_add_sync(0xffffffffu, sum);
    if (tid == 0) add_work(status, 10, 0.0, 16.0 * b * sum);
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
    double* M = s * ldm <= RcShared<GW, NBLK, XU>::kXu + 8 * LDX ? sm.xu : ws.m;

    // ---- stage 0: the side's panel, block by block: projection, earlier reflector blocks, QR.
    // Stage 1 (V side): Q3 = the QR's Q, a block of columns at a time from the last, then once more
    // against V_ij.  Both are a list of steps x <- x - src coef with coef from the products src^T x, and
    // share one copy of the code.
    // core M = diag + [C; R2] [D; R3]^T
    const double *cu = fast ? sm.cr[0] : ws.cru, *cv = fast ? sm.cr[1] : ws.crv;
    auto form_core = [&](int first, int step) {
      for (int e = first; e < s * s; e += step) {
        const int a = e / s, c = e - a * s;
        const double *ca = cu + (size_t)a * ldq, *cc = cv + (size_t)c * ldq;
        double a0 = (a == c && a < r1) ? sm.n1[a] * sm.nvv[a] : 0.0, a1 = 0.0;
        for (int v = 0; v < q; v += 2) {
          a0 = fma(ca[v], cc[v], a0);
          if (v + 1 < q) a1 = fma(ca[v + 1], cc[v + 1], a1);
        }
        M[a * ldm + c] = a0 + a1;
      }
    };
    // orders past 32: the U group forms the core and its R while the V group forms Q3, then both rotate
    auto large_core = [&]() {
      const bool near = M == sm.xu;
      if (side == 0) {
        form_core(sd.tg, GT);
        sd.sync();
        if (near) group_core_r<GT, true>(M, ldm, s, sd.tg, sd.bar);
        else group_core_r<GT, false>(M, ldm, s, sd.tg, sd.bar);
      }
      bar_sync<2 * GT>(5);
      constexpr int kLp = MINB == 1 ? 4 : 8;  // one turn per round while the registers hold the rows
      if (!near) jacobi_group<2 * GT, 8, 16, false>(M, ldm, s, kFloor, sm.sig, sm.mx, sm.flag, tid, 6);
      else if (s <= 64) jacobi_group<2 * GT, 8, 8, true>(M, ldm, s, kFloor, sm.sig, sm.mx, sm.flag, tid, 6);
      else if (s <= 96) jacobi_group<2 * GT, kLp, 96 / kLp, true>(M, ldm, s, kFloor, sm.sig, sm.mx, sm.flag, tid, 6);
      else jacobi_group<2 * GT, kLp, 128 / kLp, true>(M, ldm, s, kFloor, sm.sig, sm.mx, sm.flag, tid, 6);
    };
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
      if (s > 32) large_core();
      bar_sync<2 * GT>(4);  // the rank and the coefficients are in place
    } else {
      bar_sync<2 * GT>(3);
      // ---- the core, its R, the SVD and the rank
      if (s > 32) {
        large_core();
      } else {
        form_core(sd.tg, GT);
        sd.sync();
        if (sd.gw == 0) {
          if (s <= 8) {
            warp_core_r<8>(M, ldm, s, sm.srt);
            jacobi_warp<4, 2>(M, ldm, s, kFloor);
          } else if (s <= 16) {
            warp_core_r<16>(M, ldm, s, sm.srt);
            jacobi_warp<4, 4>(M, ldm, s, kFloor);
          } else if (s <= 24) {
            warp_core_r<24>(M, ldm, s, sm.srt);
            jacobi_warp<2, 16>(M, ldm, s, kFloor);
          } else {
            warp_core_r<32>(M, ldm, s, sm.srt);
            jacobi_warp<2, 16>(M, ldm, s, kFloor);
          }
        }
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
    // their arrays: behind the core in shared memory where they fit, else in the scratch slot
    const int ldg = fast ? kLdg : round8(rn), core = fast ? kFs * (kFs + 1) : (s * ldm + 1) & ~1;
    const bool near = fast || (M == sm.xu && core + (r1 + ri + s + q) * ldg <= RcShared<GW, NBLK, XU>::kXu + 8 * LDX);
    double* GU = near ? sm.xu + core : ws.gu;
    double* GV = near ? GU + (fast ? kFs + kFlong : r1 + ri) * ldg : ws.gv;
    double* Gb = near ? GV + (fast ? kFs : s) * ldg : ws.gb;
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
        const double* dv = cv + (kk - r1);
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
      else if (rn <= 64) sd.template output<8>(out, b, rn, Q1, r1, co, src2, ld2, n2, m2, co + r1 * ldg, ldg);
      else sd.template output<16>(out, b, rn, Q1, r1, co, src2, ld2, n2, m2, co + r1 * ldg, ldg);
    }
    if (tid == 0) rank[tij] = rn;
    __syncthreads();
  }
}

namespace {

template <int GW, int NBLK, int MINB, int XU = 0>
struct RcShape {
  static constexpr int kPerSm = MINB;
  static size_t slot(int cap) { return wide_slot<Side<GW, NBLK>::kLdx>(nullptr, cap, nullptr); }
  static int launch(int grid, int n, int b, int k, int nB, double* U, double* V, int* rank, int cap, double* scratch,
                    size_t slot_doubles, int* next_pair, int* rlog, int prank, int pworld, long npairs, int* status,
                    cudaStream_t s) {
    const size_t sm = sizeof(RcShared<GW, NBLK, XU>);
    cudaFuncSetAttribute(k_recompress<GW, NBLK, MINB, XU>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    k_recompress<GW, NBLK, MINB, XU><<<grid, GW * 64, sm, s>>>(n, b, k, nB, U, V, rank, cap, scratch, slot_doubles, next_pair,
                                                           rlog, prank, pworld, npairs, status);
    return (int)cudaGetLastError();
  }
};
constexpr int kTallXu = 18496;  // doubles of xu that hold, with xv, a core of order 150
constexpr int kFewPairs = kSms;  // one per SM
// calls f with the shape for a tile size, a rank capacity and whether the step has at most kFewPairs pairs
// (all shapes of a tile size have the same rows, so the same scratch slots)
template <class F>
auto rc_shape(int b, int cap, bool few, F f) {
  // A capacity past 64 (asked for, or a plan that grew at a rank above it) allows cores that do not fit beside a
  // second CTA's shared memory; a step waits for them (1.8 ms each through L2), so one CTA keeps the SM:
  // recompression at N = 20,000, range 0.1, ranks to 65, 62 -> 53 ms.  The host queues a step before its ranks
  // are known, so the capacity decides and low ranks pay for it: capacity 128 against 64 at mean ranks of 5
  // to 7, N = 1,030, b = 100 0.79 -> 0.81 ms, N = 4,000, b = 250 1.74 -> 1.83, N = 10,007, b = 250 4.8 -> 5.2,
  // N = 50,000, b = 500 45.9 -> 49.2 (the forward pass 129.5 -> 133.0), N = 20,000, range 0.2 12.3 -> 11.9.
  if (cap > 64) {
    if (b <= 128) return f(RcShape<4, 4, 1, kTallXu>{});
    if (b <= 256) return f(RcShape<4, 8, 1, kTallXu>{});
    if (b <= 512) return f(RcShape<4, 16, 1, kTallXu>{});
    return f(RcShape<8, 16, 1>{});
  }
  // No second CTA to share the SM with: all its registers to one (255 a thread; b > 256 spills nothing then, the
  // smaller shapes 80 bytes against 150).  Recompression per evaluation: N = 1,030, b = 100 0.83 -> 0.77 ms,
  // N = 4,000, b = 250 1.93 -> 1.68, N = 4,000, b = 203 2.94 -> 2.56; sixteen warps in its place 0.83, 1.84, 2.78
  // (all without the reflectors' range test).
  if (few) {
    if (b <= 128) return f(RcShape<4, 4, 1>{});
    if (b <= 256) return f(RcShape<4, 8, 1>{});
    if (b <= 512) return f(RcShape<4, 16, 1>{});
  }
  if (b <= 128) return f(RcShape<4, 4, 2>{});
  if (b <= 256) return f(RcShape<4, 8, 2>{});
  if (b <= 512) return f(RcShape<4, 16, 2>{});
  return f(RcShape<8, 16, 1>{});
}

}  // namespace

int rc_blocks_per_sm(int b, int cap) {
  return rc_shape(b, cap, false, [](auto shape) { return decltype(shape)::kPerSm; });
}
size_t rc_slot_doubles(int b, int cap) {
  return rc_shape(b, cap, false, [&](auto shape) { return shape.slot(cap); });
}

int launch_recompress(int n, int b, int k, int nB, double* U, double* V, int* rank, int cap, double* scratch,
                      size_t slot_doubles, int nslots, int* next_pair, int* rlog_step, int prank, int pworld,
                      int* status, cudaStream_t s) {
  const long npairs = rc_npairs(k, nB, prank, pworld);
  if (npairs <= 0) return 0;
  const int grid = (int)std::min<long>(npairs, nslots);
  const long m = nB - k - 1;  // all ranks' pairs, so that a partitioned step takes the same shape
  return rc_shape(b, cap, m * (m - 1) / 2 <= kFewPairs, [&](auto shape) {
    return shape.launch(grid, n, b, k, nB, U, V, rank, cap, scratch, slot_doubles, next_pair, rlog_step, prank, pworld,
                        npairs, status, s);
  });
}

}  // namespace tlr
