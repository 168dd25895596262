// Initial compression of the off-diagonal covariance tiles (FP64 parity path).
//
// Reference: codes/17_tlr_cholesky_pilot.py:151-166 (tile generation) and 107-116
// (truncate_svd: full SVD of every b x b tile, rank = smallest r with tail[r] <= threshold).
//
// B200 design.  A full b x b SVD per tile is O(b^3) and is where the reference spends
// 54-66% of its time.  Here each tile goes through a batched randomized range finder
// whose rank decision is exact to rounding:
//   T        generated once per chunk from the Morton-ordered coordinates (row-major, HBM);
//   Z = T^T (T P) four times, each followed by a Householder orthonormalisation (P <- Q(Z));
//   C = T P, rho^2 = ||T - C P^T||_F^2 computed element by element (no cancellation);
//   R_C from a Householder QR of C, one-sided Jacobi SVD of R_C -> sigma, W;
//   tail[r]^2 = rho^2 + sum_{t>=r} sigma_t^2 (same accumulation order as the reference);
//   the rank is accepted when r <= k - margin, so the unresolved directions lie far below
//   the threshold; otherwise the tile is redone with k doubled (16, 32, 64, 128).
// The truncated pair is U = C W_r (= Q_C U_w Sigma_r), V = P W_r, so U has orthogonal
// columns and V orthonormal columns, exactly the structure of the reference's U*s, Vt^T.
#include <type_traits>

#include "tlr_kernels.h"
#include "tlr_panel.cuh"

namespace tlr {

constexpr int kMaxSketch = 128;  // widest sketch level
constexpr double kCoreFloor = 1e-200;  // of the squared row norms in the Jacobi SVD
__host__ __device__ inline int tile_pitch(int b) { return (b + 1) & ~1; }  // 16-byte rows of the generated tiles

__device__ __forceinline__ double omega_entry(uint32_t tile, uint32_t row, uint32_t col) {
  // splitmix64 (Steele, Lea, Flood 2014) on (tile, row, col): a fixed, reproducible test matrix
  uint64_t x = ((uint64_t)tile << 42) ^ ((uint64_t)row << 21) ^ (uint64_t)col;
  x += 0x9E3779B97F4A7C15ull;
  x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
  x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
  x ^= x >> 31;
  return (double)(x >> 11) * (2.0 / 9007199254740992.0) - 1.0;
}

// ----------------------------------------------------------------------------------------
// T[c] = sigma2 * matern32(dist(S_i, S_j)), row-major with leading dimension tile_pitch(b).
__global__ void k_gen_offdiag(const double* TLR_RESTRICT xy, int n, int b, int tile_base,
                              const int* TLR_RESTRICT ti, const int* TLR_RESTRICT tj, double* TLR_RESTRICT T,
                              const int* TLR_RESTRICT status) {
  if (*status != 0) return;
  const EvalParams& prm = *eval_params(status);
  const double sigma2 = prm.sigma2, inv_range = prm.inv_range;
  const int nu5 = prm.nu5;
  const int c = blockIdx.y;
  const int t = tile_at(status, tile_base + c);
  const int i = ti[t], j = tj[t];
  const int i0 = i * b, j0 = j * b;
  const int bi = min(b, n - i0), bj = min(b, n - j0);
  const int ldt = tile_pitch(b);
  double* Tc = T + (size_t)c * b * ldt;
  const int total = bi * bj;
  if (blockIdx.x == 0 && threadIdx.x == 0) add_work(status, 1, 0.0, 8.0 * total);
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < total; e += gridDim.x * blockDim.x) {
    const int a = e / bj, q = e - a * bj;
    const double2 pa = reinterpret_cast<const double2*>(xy)[i0 + a];
    const double2 pq = reinterpret_cast<const double2*>(xy)[j0 + q];
    Tc[(size_t)a * ldt + q] = matern_cov(pa.x, pa.y, pq.x, pq.y, sigma2, inv_range, nu5);
  }
}

// ----------------------------------------------------------------------------------------
// The range finder's products on the FP64 tensor cores.  One CTA of W warps per (tile, group of 8 NT
// columns of P); warp w owns columns [CW w, CW w + CW) of T, so a CTA covers tiles up to W CW wide.
//   T streams through shared memory in slabs of H rows, double-buffered with cp.async (the next slab's
//   copy runs under this slab's products).  Per slab R:
//     phase A  Y_R = T_R P: each warp multiplies its column strip by its rows of P (held in registers
//              for the whole kernel) -> an H x 8 NT partial; the W partials are summed in a fixed order
//              (mode 1 writes that sum: the rows R of C = T P);
//     phase B  Z[strip] += T_R[:, strip]^T Y_R, accumulated in registers across slabs.
//   Every T element is read from HBM once per launch and group and used by both phases from shared
//   memory.
//   MODE 0: the sketch Z = T^T T P.  MODE 1: the projection C = T P.  MODE 2 (one 16-column group,
//   k = 16): the projection and, in place of phase B, the residual of the slab on the tensor cores,
//   E_R = T_R - C_R P^T (accumulator started at T_R, operand -C_R), with rho^2 = sum E^2 and
//   ||T||^2 summed per lane in a fixed order and over the CTA in warp order into parts[c],
//   fparts[c] (one block per tile): T leaves HBM once for both.
// Bound by the FP64 tensor pipe (17 cycles per m8n8k4 step and scheduler).  The shape follows the tile so
// that no warp multiplies padding: 4, 8 or 16 warps of 32 columns up to b = 128, 256, 512; up to 1024
// sixteen warps of 64 columns with 8 columns of P (the registers of 16 would spill), at the price of
// reading T twice as often.  T's rows are padded to an even pitch, so odd tile sizes take it too.
// Sketch passes of one FP64 evaluation: N = 12,000, b = 1000 24.3 -> 3.2 ms, N = 10,007, b = 250
// 3.6 -> 1.7 ms, N = 4,000, b = 203 1.64 -> 0.68 ms, N = 1,030, b = 100 0.29 -> 0.16 ms against one
// 512-wide shape for even b <= 512 and CUDA-core products for the others.
template <int W, int CW, int NT, int H>
struct SketchShape {
  static constexpr int kCols = W * CW;
  static constexpr int kPitch = kCols + 4;  // conflict-free fragments
  static constexpr int kYp = 8 * NT + 2;    // pitch of the per-warp partials
  static constexpr int kYs = 8 * NT + 1;    // pitch of the summed Y_R
  static constexpr size_t kSmem = ((size_t)2 * H * kPitch + (size_t)W * H * kYp + (size_t)H * kYs) * sizeof(double);
};

template <int MODE, int W, int CW, int NT, int H>
__global__ void __launch_bounds__(W * 32, 16 / W)
    k_sketch_mma(const double* TLR_RESTRICT T, int n, int b, int tile_base, const int* TLR_RESTRICT ti,
                 const int* TLR_RESTRICT tj, const int* TLR_RESTRICT need, const double* TLR_RESTRICT P,
                 double* TLR_RESTRICT out, int ldp, int omega, double* TLR_RESTRICT parts,
                 double* TLR_RESTRICT fparts, const int* TLR_RESTRICT status) {
  using Sh = SketchShape<W, CW, NT, H>;
  constexpr int kPitch = Sh::kPitch, kYp = Sh::kYp, kYs = Sh::kYs, kMt = H / 8;
  static_assert(MODE != 2 || NT == 2, "the fused residual needs the whole k = 16 panel");
  if (*status != 0) return;
  const int c = blockIdx.x, grp = blockIdx.y;
  if (!need[c]) return;
  const int t = tile_at(status, tile_base + c);
  const int bi = min(b, n - ti[t] * b), bj = min(b, n - tj[t] * b);
  if (threadIdx.x == 0) {
    add_work(status, MODE == 0 ? 2 : 4, (MODE == 0 ? 4.0 : 2.0) * bi * bj * 8 * NT,
             8.0 * ((double)bi * bj + (omega ? 0.0 : bj * 8.0 * NT) + (MODE == 0 ? bj : bi) * 8.0 * NT));
    if (MODE == 2) add_work(status, 5, 2.0 * bi * bj * 17, 0.0);
  }
  extern __shared__ __align__(16) double sk_smem[];
  double* Ts = sk_smem;                          // [2][H][kPitch]
  double* Yp = Ts + (size_t)2 * H * kPitch;      // [W][H][kYp]
  double* Ys = Yp + (size_t)W * H * kYp;         // [H][kYs]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, tg = lane & 3;
  const int ldt = tile_pitch(b);
  const double* Tc = T + (size_t)c * b * ldt;
  const size_t pbase = (size_t)c * b * ldp;
  const int col0 = warp * CW;
  const int nslab = (bi + H - 1) / H;

  // slab s -> stage s & 1: H rows x kCols columns in 16-byte pieces, zero past bi / bj
  auto issue = [&](int s) {
    double* dst = Ts + (size_t)(s & 1) * H * kPitch;
    const int a0 = s * H;
#pragma unroll
    for (int e = tid; e < H * (Sh::kCols / 2); e += W * 32) {
      const int r = e / (Sh::kCols / 2), col = 2 * (e % (Sh::kCols / 2));
      const int row = a0 + r;
      const int bytes = row < bi ? (col + 1 < bj ? 16 : (col < bj ? 8 : 0)) : 0;
      cp_async16(dst + (size_t)r * kPitch + col, bytes ? Tc + (size_t)row * ldt + col : Tc, bytes);
    }
    cp_async_commit();
  };
  issue(0);

  // B fragments of P for phase A: rows col0 + 4 kk + tg, columns 8 nt + g of the group
  double pf[CW / 4][NT];
#pragma unroll
  for (int kk = 0; kk < CW / 4; ++kk)
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
      const int row = col0 + 4 * kk + tg, q = (grp * NT + nt) * 8 + g;
      pf[kk][nt] = row < bj ? (omega ? omega_entry((uint32_t)t, (uint32_t)row, (uint32_t)q)
                                     : P[pbase + (size_t)q * b + row])
                            : 0.0;
    }
  double za[CW / 8][NT][2];
#pragma unroll
  for (int m = 0; m < CW / 8; ++m)
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) za[m][nt][0] = za[m][nt][1] = 0.0;
  // MODE 2: B fragments of P^T for the residual, P rows col0 + 8 j + g, columns 4 kq + tg
  double pt[4][CW / 8];
  double rho = 0.0, fro = 0.0;
  if (MODE == 2) {
#pragma unroll
    for (int kq = 0; kq < 4; ++kq)
#pragma unroll
      for (int j = 0; j < CW / 8; ++j) {
        const int row = col0 + 8 * j + g;
        pt[kq][j] = row < bj ? P[pbase + (size_t)(4 * kq + tg) * b + row] : 0.0;
      }
  }

  for (int s = 0; s < nslab; ++s) {
    cp_async_wait_all();
    __syncthreads();  // slab s visible to all; every warp is done with slab s - 1
    if (s + 1 < nslab) issue(s + 1);
    const double* Tsl = Ts + (size_t)(s & 1) * H * kPitch;
    double ya[kMt][NT][2];
#pragma unroll
    for (int m = 0; m < kMt; ++m)
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) ya[m][nt][0] = ya[m][nt][1] = 0.0;
#pragma unroll
    for (int kk = 0; kk < CW / 4; ++kk)
#pragma unroll
      for (int m = 0; m < kMt; ++m) {
        const double a = Tsl[(size_t)(8 * m + g) * kPitch + col0 + 4 * kk + tg];
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) dmma884(ya[m][nt][0], ya[m][nt][1], a, pf[kk][nt]);
      }
    double* yp = Yp + (size_t)warp * H * kYp;
#pragma unroll
    for (int m = 0; m < kMt; ++m)
#pragma unroll
      for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int h = 0; h < 2; ++h) yp[(8 * m + g) * kYp + 8 * nt + 2 * tg + h] = ya[m][nt][h];
    __syncthreads();
#pragma unroll
    for (int e = tid; e < H * 8 * NT; e += W * 32) {
      const int r = e / (8 * NT), q = e % (8 * NT);
      double sum = 0.0;
#pragma unroll
      for (int w = 0; w < W; ++w) sum += Yp[(size_t)w * H * kYp + r * kYp + q];
      if (MODE != 0) {
        const int row = s * H + r;
        if (row < bi) out[pbase + (size_t)(grp * 8 * NT + q) * b + row] = sum;
      }
      if (MODE != 1) Ys[r * kYs + q] = sum;
    }
    if (MODE == 1) continue;
    __syncthreads();
    if (MODE == 2) {
      // E_R[:, strip] = T_R[:, strip] - C_R P[strip, :]^T
      double e[kMt][CW / 8][2];
#pragma unroll
      for (int m = 0; m < kMt; ++m)
#pragma unroll
        for (int j = 0; j < CW / 8; ++j)
#pragma unroll
          for (int h = 0; h < 2; ++h) e[m][j][h] = Tsl[(size_t)(8 * m + g) * kPitch + col0 + 8 * j + 2 * tg + h];
#pragma unroll
      for (int kq = 0; kq < 4; ++kq)
#pragma unroll
        for (int m = 0; m < kMt; ++m) {
          const double a = -Ys[(8 * m + g) * kYs + 4 * kq + tg];
#pragma unroll
          for (int j = 0; j < CW / 8; ++j) dmma884(e[m][j][0], e[m][j][1], a, pt[kq][j]);
        }
#pragma unroll
      for (int m = 0; m < kMt; ++m) {
        const bool rin = s * H + 8 * m + g < bi;
#pragma unroll
        for (int j = 0; j < CW / 8; ++j)
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            if (rin && col0 + 8 * j + 2 * tg + h < bj) {
              const double tv = Tsl[(size_t)(8 * m + g) * kPitch + col0 + 8 * j + 2 * tg + h];
              rho = fma(e[m][j][h], e[m][j][h], rho);
              fro = fma(tv, tv, fro);
            }
          }
      }
      continue;
    }
    if constexpr (MODE == 0) {  // the sketch's second product; the other modes left above
#pragma unroll
      for (int kq = 0; kq < H / 4; ++kq) {
        double bf[NT];
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) bf[nt] = Ys[(4 * kq + tg) * kYs + 8 * nt + g];
#pragma unroll
        for (int m = 0; m < CW / 8; ++m) {
          const double a = Tsl[(size_t)(4 * kq + tg) * kPitch + col0 + 8 * m + g];
#pragma unroll
          for (int nt = 0; nt < NT; ++nt) dmma884(za[m][nt][0], za[m][nt][1], a, bf[nt]);
        }
      }
    }
  }
  if (MODE == 2) {
    rho = warp_sum(rho);
    fro = warp_sum(fro);
    __syncthreads();
    if (lane == 0) {
      Yp[warp] = rho;
      Yp[W + warp] = fro;
    }
    __syncthreads();
    if (tid == 0) {
      double a = 0.0, f = 0.0;
      for (int w = 0; w < W; ++w) {
        a += Yp[w];
        f += Yp[W + w];
      }
      parts[c] = a;
      fparts[c] = f;
    }
  }
  if (MODE == 0) {
#pragma unroll
    for (int m = 0; m < CW / 8; ++m) {
      const int col = col0 + 8 * m + g;
      if (col < bj)
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
          for (int h = 0; h < 2; ++h)
            out[pbase + (size_t)((grp * NT + nt) * 8 + 2 * tg + h) * b + col] = za[m][nt][h];
    }
  }
}

// ----------------------------------------------------------------------------------------
// Blocked Householder QR of a bt x k panel by one CTA (a tlr::Side of GW warps): blocks of 8 columns go
// through the earlier reflector blocks and their own QR in registers, products and updates on the FP64
// tensor cores.  Bound by its chain of k column steps (about 800 cycles each, one barrier) and, for k > 8,
// the block applications between them; per FP64 evaluation at N = 50,000, b = 500: k_orth 25.8 -> 12.6 ms,
// k_finalize 15.9 -> 5.5 ms against a column-by-column QR with the core's SVD in shared memory; at
// N = 1,030, b = 100: 0.54 -> 0.30 and 0.68 -> 0.16 ms.
template <int GW, int NBLK>
struct PanelShared {
  static constexpr int kLdx = Side<GW, NBLK>::kLdx;
  double red[kRu * GW * 64], redn[kRu * GW * 8];
  double coef[64], tmp[64], zt[64], tau[16];
  double qred[2 * (8 * GW + 8)];
  double tf[16 * 64];  // T of every reflector block (k <= 128)
};

template <int GW, int NBLK>
__device__ __forceinline__ Side<GW, NBLK> panel_side(int m, bool al) {
  Side<GW, NBLK> sd;
  sd.tg = threadIdx.x;
  sd.gw = threadIdx.x >> 5;
  sd.lane = threadIdx.x & 31;
  sd.g = sd.lane >> 2;
  sd.t = sd.lane & 3;
  sd.bar = 1;
  sd.m = m;
  sd.al = al;
  return sd;
}

// x <- (I - V T^T V^T) x (trans) or (I - V T V^T) x for one reflector block
template <int GW, int NBLK>
__device__ __forceinline__ void apply_block(const Side<GW, NBLK>& sd, double (&x)[NBLK][2], const double* panel,
                                            const double* tf, bool trans, PanelShared<GW, NBLK>& sh) {
  using S = Side<GW, NBLK>;
  sd.dot(x, panel, S::kLdx, 8, S::kRows, true, sh.red, sh.redn,
         [&](int u, int v, double sum, double) { sh.tmp[u * 8 + v] = sum; });
  for (int e = sd.tg; e < 64; e += S::GT) {
    const int u = e >> 3, v = e & 7;
    double acc = 0.0;
#pragma unroll
    for (int k = 0; k < 8; ++k) acc = fma(trans ? tf[k * 8 + u] : tf[u * 8 + k], sh.tmp[k * 8 + v], acc);
    sh.coef[e] = acc;
  }
  sd.sync();
  sd.update(x, panel, S::kLdx, 8, S::kRows, sh.coef, 8, -1.0);
}

// QR of the panel src (leading dimension ld, ke columns): reflector blocks in panel (shared memory when
// in_smem, block vb at panel + 8 vb kLdx) with their T factors in sh.tf; xs is the transpose buffer (one
// block; the block itself when the panel is in shared memory).  R (row-major, pitch ldr, nrow rows) when
// given.  The last block's reflectors are kept only when keep_last.
template <int GW, int NBLK>
__device__ __forceinline__ void panel_qr(const Side<GW, NBLK>& sd, const double* src, int ld, int ke, double* panel,
                                         double* xs, bool in_smem, double* R, int ldr, int nrow, bool keep_last,
                                         PanelShared<GW, NBLK>& sh) {
  constexpr int kLdx = Side<GW, NBLK>::kLdx;
  const int nb = (ke + 7) >> 3;
#pragma unroll 1
  for (int vb = 0; vb < nb; ++vb) {
    const int nv = min(8, ke - 8 * vb);
    double x[NBLK][2];
    sd.load(x, src, ld, 8 * vb, nv);
#pragma unroll 1
    for (int pb = 0; pb < vb; ++pb) apply_block(sd, x, panel + (size_t)pb * 8 * kLdx, sh.tf + pb * 64, true, sh);
    double* blk = panel + (size_t)vb * 8 * kLdx;
    sd.qr(x, in_smem ? blk : xs, 8 * vb, nv, nrow, sh.qred, R + 8 * vb, ldr, sh.zt, sh.tau, sh.tf + vb * 64,
          (keep_last || vb + 1 < nb) ? blk : nullptr);
  }
}

// Z <- Q of the Householder QR of Z (bj x k).  One CTA per tile.
template <int GW, int NBLK>
__global__ void __launch_bounds__(GW * 32, 16 / GW) k_orth(double* TLR_RESTRICT Z, int n, int b, int k, int ldp,
                                                          int tile_base, const int* TLR_RESTRICT tj,
                                                          const int* TLR_RESTRICT need, double* TLR_RESTRICT gscratch,
                                                          size_t slot, int in_smem, const int* TLR_RESTRICT status) {
  if (cta_failed(status)) return;
  const int c = blockIdx.x;
  if (!need[c]) return;
  constexpr int kLdx = Side<GW, NBLK>::kLdx;
  const int bj = min(b, n - tj[tile_at(status, tile_base + c)] * b);
  const int ke = min(k, bj);  // a tile narrower than k gets a full basis and zero columns
  if (threadIdx.x == 0) add_work(status, 3, 4.0 * bj * ke * ke, 16.0 * bj * k);
  extern __shared__ __align__(16) double smem[];
  auto& sh = *reinterpret_cast<PanelShared<GW, NBLK>*>(smem);
  double* xs = smem + sizeof(PanelShared<GW, NBLK>) / sizeof(double);
  double* panel = in_smem ? xs : gscratch + (size_t)c * slot;
  double* Zc = Z + (size_t)c * b * ldp;
  const auto sd = panel_side<GW, NBLK>(bj, (b & 1) == 0);
  panel_qr(sd, Zc, b, ke, panel, xs, in_smem != 0, Zc, 0, 0, true, sh);
  const int nb = (ke + 7) >> 3;
#pragma unroll 1
  for (int vb = (k >> 3) - 1; vb >= 0; --vb) {  // Q from the last block of columns on
    double x[NBLK][2];
#pragma unroll
    for (int p = 0; p < NBLK; ++p)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int row = 8 * (sd.gw + GW * p) + 2 * sd.t + h, col = 8 * vb + sd.g;
        x[p][h] = (row == col && col < ke) ? 1.0 : 0.0;
      }
#pragma unroll 1
    for (int pb = min(vb, nb - 1); pb >= 0 && vb < nb; --pb)
      apply_block(sd, x, panel + (size_t)pb * 8 * kLdx, sh.tf + pb * 64, false, sh);
    double* z = Zc + (size_t)(8 * vb + sd.g) * b;
#pragma unroll
    for (int p = 0; p < NBLK; ++p) {
      const int row = 8 * (sd.gw + GW * p) + 2 * sd.t;
      if (sd.al && row + 1 < bj) *reinterpret_cast<double2*>(z + row) = make_double2(x[p][0], x[p][1]);
      else {
        if (row < bj) z[row] = x[p][0];
        if (row + 1 < bj) z[row + 1] = x[p][1];
      }
    }
  }
}

// ----------------------------------------------------------------------------------------
// Residual of the projection, per column block of 64: parts[c][blk] = sum (T - C P^T)^2 over
// the block, fparts[c][blk] = sum T^2 over the block.  Element-wise, no cancellation.
__global__ void __launch_bounds__(256) k_resid(const double* TLR_RESTRICT T, int n, int b, int k, int ldp,
                                              int tile_base, const int* TLR_RESTRICT ti,
                                              const int* TLR_RESTRICT tj, const int* TLR_RESTRICT need,
                                              const double* TLR_RESTRICT P, const double* TLR_RESTRICT C,
                                              double* TLR_RESTRICT parts, double* TLR_RESTRICT fparts,
                                              int nblk, const int* TLR_RESTRICT status) {
  if (*status != 0) return;
  const int c = blockIdx.x, blk = blockIdx.y;
  if (!need[c]) return;
  const int t = tile_at(status, tile_base + c);
  const int bi = min(b, n - ti[t] * b), bj = min(b, n - tj[t] * b);
  const int q0 = blk * 64;
  if (q0 >= bj) {
    if (threadIdx.x == 0) { parts[c * nblk + blk] = 0.0; fparts[c * nblk + blk] = 0.0; }
    return;
  }
  const int qn = min(64, bj - q0);
  if (threadIdx.x == 0) add_work(status, 5, 2.0 * bi * qn * (k + 1), 8.0 * ((double)bi * qn + (bi + qn) * k));
  extern __shared__ double smem[];
  double* Pb = smem;              // [64][k+1]  P rows q0..q0+63
  double* Cs = Pb + 64 * (k + 1); // [16][k+1]  C rows of the strip
  double* red = Cs + 16 * (k + 1);
  const size_t pbase = (size_t)c * b * ldp;
  for (int e = threadIdx.x; e < 64 * k; e += 256) {
    const int r = e % 64, q = e / 64;
    Pb[r * (k + 1) + q] = (r < qn) ? P[pbase + (size_t)q * b + q0 + r] : 0.0;
  }
  const int ldt = tile_pitch(b);
  const double* Tc = T + (size_t)c * b * ldt;
  double acc = 0.0, facc = 0.0;
  const int col = threadIdx.x & 63, rsub = threadIdx.x >> 6;  // 4 row lanes x 64 columns
  for (int a0 = 0; a0 < bi; a0 += 16) {
    const int hrows = min(16, bi - a0);
    __syncthreads();
    for (int e = threadIdx.x; e < 16 * k; e += 256) {
      const int r = e % 16, q = e / 16;
      Cs[r * (k + 1) + q] = (r < hrows) ? C[pbase + (size_t)q * b + a0 + r] : 0.0;
    }
    __syncthreads();
    if (col < qn) {
      // rows rsub, rsub + 4, rsub + 8, rsub + 12 of the strip as four independent chains (each
      // element is still T - sum_q C P in q order; rows past the strip contribute nothing)
      double tv[4], sv[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int r = rsub + 4 * u;
        tv[u] = r < hrows ? Tc[(size_t)(a0 + r) * ldt + q0 + col] : 0.0;
        sv[u] = tv[u];
      }
      const double* pr = Pb + col * (k + 1);
#pragma unroll 4
      for (int q = 0; q < k; ++q) {
        const double pq = pr[q];
#pragma unroll
        for (int u = 0; u < 4; ++u) sv[u] = fma(-Cs[(rsub + 4 * u) * (k + 1) + q], pq, sv[u]);
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        if (rsub + 4 * u < hrows) {
          acc = fma(sv[u], sv[u], acc);
          facc = fma(tv[u], tv[u], facc);
        }
      }
    }
  }
  const double tot = block_sum(acc, red);
  const double ftot = block_sum(facc, red);
  if (threadIdx.x == 0) { parts[c * nblk + blk] = tot; fparts[c * nblk + blk] = ftot; }
}

// ----------------------------------------------------------------------------------------
// Rank decision and output of the truncated pair for every tile still in need: R of the Householder QR
// of C, one-sided Jacobi on the rows of R (right singular vectors and values of C), the rank rule with the
// residual's rho^2, U = C W_r, V = P W_r.  One CTA per tile.
template <int GW, int NBLK>
__global__ void __launch_bounds__(GW * 32, 16 / GW)
    k_finalize(int n, int b, int k, int ldp, int cap, int margin, int tile_base, const int* TLR_RESTRICT ti,
               const int* TLR_RESTRICT tj, int* TLR_RESTRICT need, const double* TLR_RESTRICT P,
               const double* TLR_RESTRICT C, const double* TLR_RESTRICT parts, const double* TLR_RESTRICT fparts,
               int nblk, double* TLR_RESTRICT gscratch, size_t slot, double* TLR_RESTRICT gsv, double* TLR_RESTRICT Uo,
               double* TLR_RESTRICT Vo, int* TLR_RESTRICT rank, int last_level, int in_smem, int* TLR_RESTRICT rlog,
               double* TLR_RESTRICT tail0, double* TLR_RESTRICT fro0, int* TLR_RESTRICT blog, int* TLR_RESTRICT status) {
  if (cta_failed(status)) return;
  const EvalParams& prm = *eval_params(status);
  const int rule_fixed = prm.rule_fixed, rmode = prm.rmode, round_store = prm.round_store;
  const double thr_rel = prm.thr_rel, thr_abs = prm.thr_abs;
  const int c = blockIdx.x;
  if (!need[c]) return;
  constexpr int GT = GW * 32;
  const int t = tile_at(status, tile_base + c);
  const int bi = min(b, n - ti[t] * b), bj = min(b, n - tj[t] * b);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) add_work(status, 6, 4.0 * bi * k * k + 6.0 * 8.0 * k * k * k, 8.0 * (bi + bj) * k);
  __shared__ double red[40], nn[128], val[128], inv[128], srt[129];
  __shared__ unsigned long long mx[2];
  __shared__ int perm[128], flag[2], rsel;
  extern __shared__ __align__(16) double smem[];
  auto& sh = *reinterpret_cast<PanelShared<GW, NBLK>*>(smem);
  const int ldm = k + 1;
  double* M = smem + sizeof(PanelShared<GW, NBLK>) / sizeof(double);  // k x (k + 1)
  double* xs = M + ((k * ldm + 1) & ~1);
  double* panel = in_smem ? xs : gscratch + (size_t)c * slot;
  const size_t pbase = (size_t)c * b * ldp;
  auto sd = panel_side<GW, NBLK>(bi, (b & 1) == 0);
  // every column runs, past the tile's rows too (zero rows and no reflector there)
  panel_qr(sd, C + pbase, b, k, panel, xs, in_smem != 0, M, ldm, k, false, sh);
  sd.sync();
  if (k <= 32) {
    if (warp == 0) {
      if (k <= 16) jacobi_warp<4, 4>(M, ldm, k, kCoreFloor);
      else jacobi_warp<2, 16>(M, ldm, k, kCoreFloor);
    }
  } else {
    if (k <= 64) jacobi_group<GT, 8, 8, true>(M, ldm, k, kCoreFloor, nn, mx, flag, tid, 1);
    else jacobi_group<GT, 8, 16, true>(M, ldm, k, kCoreFloor, nn, mx, flag, tid, 1);
  }
  sd.sync();
  for (int q0 = 0; q0 < k; q0 += GT / 4) {  // singular values: the row norms
    const int q = q0 + (tid >> 2), h = tid & 3;
    double a0 = 0.0, a1 = 0.0;
    if (q < k)
      for (int e = h; e < k; e += 8) {
        a0 = fma(M[q * ldm + e], M[q * ldm + e], a0);
        if (e + 4 < k) a1 = fma(M[q * ldm + e + 4], M[q * ldm + e + 4], a1);
      }
    double a = a0 + a1;
    a += __shfl_xor_sync(0xffffffffu, a, 2);
    a += __shfl_xor_sync(0xffffffffu, a, 1);
    if (q < k && h == 0) {
      const double nr = sqrt(a);
      val[q] = nr;
      inv[q] = nr > 0.0 ? 1.0 / nr : 0.0;
      perm[q] = q;
    }
  }
  sd.sync();
  for (int q = tid; q < k; q += GT) {  // descending order, ties by index
    const double vq = val[q];
    int pos = 0;
#pragma unroll 4
    for (int d = 0; d < k; ++d) {
      const double v = val[d];
      pos += (v > vq) || (v == vq && d < q);
    }
    perm[pos] = q;
    srt[pos] = vq * vq;
  }
  sd.sync();
  if (tid == 0) {
    double rho2 = 0.0, fro2 = 0.0;
    for (int q = 0; q < nblk; ++q) {
      rho2 += parts[c * nblk + q];
      fro2 += fparts[c * nblk + q];
    }
    double acc = rho2;  // srt[q] <- rho^2 + sum_{u >= q} sigma_u^2, from the smallest up (17:113)
    srt[k] = acc;
    for (int q = k - 1; q >= 0; --q) {
      acc += srt[q];
      srt[q] = acc;
    }
    red[0] = rho2;
    red[1] = fro2;
  }
  sd.sync();
  if (warp == 0) {
    const double fro2 = red[1], thr = rule_fixed ? thr_rel * sqrt(fro2) : thr_abs;
    int r = -1;
    for (int q0 = 0; q0 <= k && r < 0; q0 += 32) {
      const unsigned hit = __ballot_sync(0xffffffffu, q0 + lane <= k && sqrt(srt[min(q0 + lane, k)]) <= thr);
      if (hit) r = q0 + __ffs(hit) - 1;
    }
    if (lane == 0) {
      if (rmode == kRankReplay) r = rlog[t];  // frozen: the rank recorded at another theta
      const bool exact = (k >= bj) || (k >= bi);
      int out;
      if (r >= 0 && (r <= k - margin || exact)) out = r;
      else if (last_level) out = -2;  // compression limit reached
      else out = -1;                  // redo with a larger k
      if (out >= 0 && out > cap) out = -3;
      if (out >= 0) {  // truncation error ||T - T_r||_F and ||T||_F of the accepted tile
        tail0[t] = sqrt(srt[min(out, k)]);
        fro0[t] = sqrt(fro2);
      }
      rsel = out;
    }
  }
  sd.sync();
  const int r = rsel;
  if (r == -1) return;
  if (r < 0) {
    if (tid == 0) atomicCAS(status, 0, r == -2 ? -5 : -2);
    return;
  }
  // U = C W_r, V = P W_r: column q of W is row perm[q] of M over its norm
  double* Ut = Uo + (size_t)t * b * cap;
  double* Vt = Vo + (size_t)t * b * cap;
  if (r > 0) {
    double* cf = k <= 32 ? xs : gsv + (size_t)c * 2 * k * k;  // the reflector panel is done
    const int ldc = k;
    for (int e = tid; e < k * r; e += GT) {
      const int q = e / k, u = e - q * k;
      cf[u * ldc + q] = M[perm[q] * ldm + u] * inv[perm[q]];
    }
    sd.sync();
    for (int s = 0; s < 2; ++s) {
      sd.m = s ? bj : bi;
      const double* src = (s ? P : C) + pbase;
      double* out = s ? Vt : Ut;
      if (r <= 8) sd.template output<1>(out, b, r, src, 0, cf, src, b, k, sd.m, cf, ldc);
      else if (r <= 16) sd.template output<2>(out, b, r, src, 0, cf, src, b, k, sd.m, cf, ldc);
      else if (r <= 32) sd.template output<4>(out, b, r, src, 0, cf, src, b, k, sd.m, cf, ldc);
      else sd.template output<16>(out, b, r, src, 0, cf, src, b, k, sd.m, cf, ldc);
    }
  }
  if (round_store) {  // storage rule 'mixed': rounded under the budget left after truncation (17:163-164)
    __syncthreads();
    const int bits = cta_round_pair(Ut, Vt, bi, bj, r, b, thr_abs - tail0[t], red, rmode == kRankReplay ? blog[t] : 0);
    if (tid == 0 && rmode == kRankRecord) blog[t] = bits;
  }
  if (tid == 0) {
    rank[t] = r;
    need[c] = 0;
    if (rmode == kRankRecord) rlog[t] = r;
  }
}

// ----------------------------------------------------------------------------------------
// launchers
int launch_gen_offdiag(const double* xy, int n, int b, int tile_base, const int* ti, const int* tj,
                       double* T, int nchunk, const int* status, cudaStream_t s) {
  dim3 grid((unsigned)((b * b + 1023) / 1024), (unsigned)nchunk);
  k_gen_offdiag<<<grid, 256, 0, s>>>(xy, n, b, tile_base, ti, tj, T, status);
  return (int)cudaGetLastError();
}

template <int MODE, int W, int CW, int NT, int H>
static int run_sketch(int nchunk, int k, const double* T, int n, int b, int tile_base, const int* ti, const int* tj,
                      const int* need, const double* P, double* out, int ldp, int omega, double* parts, double* fparts,
                      const int* status, cudaStream_t s) {
  constexpr size_t sm = SketchShape<W, CW, NT, H>::kSmem;
  cudaFuncSetAttribute(k_sketch_mma<MODE, W, CW, NT, H>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  k_sketch_mma<MODE, W, CW, NT, H><<<dim3((unsigned)nchunk, (unsigned)(k / (8 * NT))), W * 32, sm, s>>>(
      T, n, b, tile_base, ti, tj, need, P, out, ldp, omega, parts, fparts, status);
  return (int)cudaGetLastError();
}

int launch_sketch(const double* T, int n, int b, int k, int tile_base, const int* ti, const int* tj,
                  const int* need, const double* P, double* out, int ldp, int omega, int mode, int nchunk,
                  const int* status, cudaStream_t s) {
  auto run = [&](auto m) {
    constexpr int M = decltype(m)::value;
    if (b <= 128)
      return run_sketch<M, 4, 32, 2, 16>(nchunk, k, T, n, b, tile_base, ti, tj, need, P, out, ldp, omega, nullptr, nullptr,
                                         status, s);
    if (b <= 256)
      return run_sketch<M, 8, 32, 2, 16>(nchunk, k, T, n, b, tile_base, ti, tj, need, P, out, ldp, omega, nullptr, nullptr,
                                         status, s);
    if (b <= 512)
      return run_sketch<M, 16, 32, 2, 16>(nchunk, k, T, n, b, tile_base, ti, tj, need, P, out, ldp, omega, nullptr,
                                          nullptr, status, s);
    return run_sketch<M, 16, 64, 1, 8>(nchunk, k, T, n, b, tile_base, ti, tj, need, P, out, ldp, omega, nullptr, nullptr,
                                       status, s);
  };
  return mode == 0 ? run(std::integral_constant<int, 0>{}) : run(std::integral_constant<int, 1>{});
}

bool project_resid_fused(int b, int k) { return k == 16 && b <= 512; }

int launch_project_resid(const double* T, int n, int b, int tile_base, const int* ti, const int* tj,
                         const int* need, const double* P, double* C, int ldp, double* parts, double* fparts,
                         int nchunk, const int* status, cudaStream_t s) {
  if (!project_resid_fused(b, 16)) return (int)cudaErrorInvalidValue;
  if (b <= 128)
    return run_sketch<2, 4, 32, 2, 16>(nchunk, 16, T, n, b, tile_base, ti, tj, need, P, C, ldp, 0, parts, fparts, status, s);
  if (b <= 256)
    return run_sketch<2, 8, 32, 2, 16>(nchunk, 16, T, n, b, tile_base, ti, tj, need, P, C, ldp, 0, parts, fparts, status, s);
  return run_sketch<2, 16, 32, 2, 16>(nchunk, 16, T, n, b, tile_base, ti, tj, need, P, C, ldp, 0, parts, fparts, status, s);
}

size_t tile_doubles(int b) { return (size_t)b * tile_pitch(b); }

// The CTA shape of the panel kernels for a tile size: calls f with (warps, row blocks per warp)
template <class F>
static int panel_shape(int b, F f) {
  if (b <= 128) return f(std::integral_constant<int, 4>{}, std::integral_constant<int, 4>{});
  if (b <= 256) return f(std::integral_constant<int, 4>{}, std::integral_constant<int, 8>{});
  if (b <= 512) return f(std::integral_constant<int, 8>{}, std::integral_constant<int, 8>{});
  return f(std::integral_constant<int, 8>{}, std::integral_constant<int, 16>{});
}

// doubles of the global panel scratch per tile (the reflectors of the widest level)
size_t orth_slot_doubles(int b, int kmax) {
  size_t n = 0;
  panel_shape(b, [&](auto gw, auto nblk) {
    n = (size_t)Side<decltype(gw)::value, decltype(nblk)::value>::kLdx * kmax;
    return 0;
  });
  return n;
}

// Reflector panels up to this size (with the core) stay in shared memory: at k = 16 that leaves two or
// three CTAs an SM, at k = 32 and b = 500 it would leave one (13.9 against 11.9 ms of k_orth per FP64
// evaluation at N = 50,000), so the wider panels go to the tile's global scratch, which L2 holds.
constexpr size_t kPanelSmem = 70 * 1024;

int launch_orth(double* Z, int n, int b, int k, int ldp, int tile_base, const int* tj, const int* need,
                double* gscratch, int nchunk, const int* status, cudaStream_t s) {
  return panel_shape(b, [&](auto gw, auto nblk) {
    constexpr int GW = decltype(gw)::value, NBLK = decltype(nblk)::value;
    constexpr int kLdx = Side<GW, NBLK>::kLdx;
    const int in_smem = (size_t)kLdx * k * 8 <= kPanelSmem;
    const size_t sm = sizeof(PanelShared<GW, NBLK>) + (size_t)kLdx * (in_smem ? k : 8) * 8;
    cudaFuncSetAttribute(k_orth<GW, NBLK>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    k_orth<GW, NBLK><<<nchunk, GW * 32, sm, s>>>(Z, n, b, k, ldp, tile_base, tj, need, gscratch,
                                                 orth_slot_doubles(b, kMaxSketch), in_smem, status);
    return (int)cudaGetLastError();
  });
}

int launch_resid(const double* T, int n, int b, int k, int ldp, int tile_base, const int* ti, const int* tj,
                 const int* need, const double* P, const double* C, double* parts, double* fparts, int nblk,
                 int nchunk, const int* status, cudaStream_t s) {
  const size_t sm = ((size_t)64 * (k + 1) + 16 * (k + 1) + 40) * 8;
  cudaFuncSetAttribute(k_resid, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  dim3 grid((unsigned)nchunk, (unsigned)nblk);
  k_resid<<<grid, 256, sm, s>>>(T, n, b, k, ldp, tile_base, ti, tj, need, P, C, parts, fparts, nblk, status);
  return (int)cudaGetLastError();
}

int launch_finalize(int n, int b, int k, int ldp, int cap, int margin, int tile_base, const int* ti, const int* tj,
                    int* need, const double* P, const double* C, const double* parts, const double* fparts,
                    int nblk, double* gscratch, double* gsv, double* U, double* V, int* rank, int last_level,
                    int nchunk, int* rlog, double* tail0, double* fro0, int* blog, int* status, cudaStream_t s) {
  return panel_shape(b, [&](auto gw, auto nb) {
    constexpr int GW = decltype(gw)::value, NBLK = decltype(nb)::value;
    constexpr int kLdx = Side<GW, NBLK>::kLdx;
    const size_t core = ((size_t)k * (k + 1) + 1) / 2 * 2;
    const int in_smem = (core + (size_t)kLdx * k) * 8 <= kPanelSmem;
    // the panel's place also holds the k x r coefficients (k <= 32)
    const size_t pan = std::max<size_t>((size_t)kLdx * (in_smem ? k : 8), k <= 32 ? (size_t)k * k : 0);
    const size_t sm = sizeof(PanelShared<GW, NBLK>) + (core + pan) * 8;
    cudaFuncSetAttribute(k_finalize<GW, NBLK>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    k_finalize<GW, NBLK><<<nchunk, GW * 32, sm, s>>>(n, b, k, ldp, cap, margin, tile_base, ti, tj, need, P, C, parts,
                                                     fparts, nblk, gscratch, orth_slot_doubles(b, kMaxSketch), gsv, U, V,
                                                     rank, last_level, in_smem, rlog, tail0, fro0, blog, status);
    return (int)cudaGetLastError();
  });
}

}  // namespace tlr
