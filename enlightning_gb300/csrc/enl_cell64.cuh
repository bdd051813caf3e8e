// FP64 cell routine of the batched engine, reading per-tile planes.
//
// Same right-hand side as fortran/rhs_hybrid_high_llf.m4:121-358 (and the
// eight sibling variants), in FP64, for a cell of a staged halo tile whose
// velocities u = rho u / rho, v = rho v / rho (every halo position) and
// fluxes F_k = u w_k (+ p for k = 1), G_k = v w_k (+ p for k = 2) (interior
// rows / columns) the block computed once into shared memory.  On this GPU
// the FP64 pipe does two fused multiply-adds per clock per SM while FP32 and
// integer work is ~60x cheaper, so the routine spends FP64 operations only
// where the value needs them:
//   * reciprocals are an FP32 hardware seed refined in FP64 (rcp64: three
//     fused multiply-adds, within a couple of units in the last place) and
//     constant divisors are multiplications;
//   * velocities and fluxes come from the planes (a cell used to divide 23
//     times);
//   * the hybrid switch decides bit for bit as the reference's division
//     would (enl_ratio.cuh), in single precision unless a ratio lies close to
//     the threshold.
// Results stay within rounding of the reference's (the engine is held to the
// oracle at 1e-12 relative L2 per field).
#pragma once
#include "enl_eos.cuh"
#include "enl_fast.cuh"
#include "enl_ratio.cuh"
#include "enl_triple.cuh"

namespace enl {

// FP64 planes of a 38 x (TH + 6) halo tile (rows of kBW64 doubles; TH = 8 in
// the batched engine): u and v at every position, the half fluxes F_0..4 / 2
// on the TH interior rows and G_0..4 / 2 on the 32 interior columns (rows of
// 32).
constexpr int kBW64 = 38;
template <int TH>
struct Geo64 {
  static constexpr int BH = TH + 6;
  static constexpr int Pos = kBW64 * BH;
  static constexpr int PF = TH * kBW64, PG = BH * 32;
  static constexpr int OffV = Pos, OffF = 2 * Pos, OffG = OffF + 5 * PF;
  static constexpr int Elems = OffG + 5 * PG;
};

// Accessor of one cell: the staged tile (7 fields, planes of Pos) and the
// planes, centred on the cell.
template <int TH>
struct SAcc64P {
  using G = Geo64<TH>;
  const double* t;
  const double* pl;
  int c;       // (cy + 3) * kBW64 + cx + 3
  int cf, cg;  // cy * kBW64 + cx + 3 in the F planes, (cy + 3) * 32 + cx in the G planes
  __device__ double w(int k, int di, int dj) const { return t[k * G::Pos + c + dj * kBW64 + di]; }
  __device__ double p(int di, int dj) const { return t[5 * G::Pos + c + dj * kBW64 + di]; }
  __device__ double t_(int di, int dj) const { return t[6 * G::Pos + c + dj * kBW64 + di]; }
  __device__ double u(int di, int dj) const { return pl[c + dj * kBW64 + di]; }
  __device__ double v(int di, int dj) const { return pl[G::OffV + c + dj * kBW64 + di]; }
  __device__ double fx(int k, int di) const { return pl[G::OffF + k * G::PF + cf + di]; }
  __device__ double gy(int k, int dj) const { return pl[G::OffG + k * G::PG + cg + dj * 32]; }
};
template <int TH>
__device__ __forceinline__ SAcc64P<TH> acc64p(const double* t, const double* pl, int cx, int cy) {
  return SAcc64P<TH>{t, pl, (cy + 3) * kBW64 + cx + 3, cy * kBW64 + cx + 3, (cy + 3) * 32 + cx};
}

// x / 2 by the exponent, on the integer pipe (zeros and normal results; the
// others by the multiplication).
__device__ __forceinline__ double half64(double x) {
  const int hi = __double2hiint(x);
  const unsigned e = (unsigned)hi & 0x7ff00000u;
  if (e - 0x00200000u < 0x7fd00000u) return __hiloint2double(hi - 0x00100000, __double2loint(x));
  if ((((unsigned)hi << 1) | (unsigned)__double2loint(x)) == 0u) return x;
  return 0.5 * x;
}

// The planes of a tile of w x h cells from its staged box, by the whole block
// of 256 threads (no barrier inside).  One seeded reciprocal of rho per halo
// position; the flux planes hold half fluxes (halving is exact).  F_0 = rho u
// and G_0 = rho v are state fields, F_2 = G_1 = rho u v.  The positions past a
// multiple of 256 fall on the last warp, not on warp 0, which also stages the
// engine's next tile.
template <int TH>
__device__ __forceinline__ void build_planes64(const double* tile, double* pl, int w, int h) {
  using G = Geo64<TH>;
  for (int e = 255 - (int)threadIdx.x; e < G::Pos; e += 256) {
    const int row = e / kBW64, col = e - row * kBW64;
    if (row >= h + 6 || col >= w + 6) continue;  // beyond a ragged tile
    const double w1 = tile[G::Pos + e], w2 = tile[2 * G::Pos + e];
    const double ir = rcp64(tile[e]);
    const double u = w1 * ir, v = w2 * ir, hu = half64(u), hv = half64(v);
    const double hp = half64(tile[5 * G::Pos + e]);
    pl[e] = u;
    pl[G::OffV + e] = v;
    const double huv = hu * w2;  // F_2 / 2 = G_1 / 2
    if (row >= 3 && row < 3 + TH) {
      double* f = pl + G::OffF + (row - 3) * kBW64 + col;
      f[0] = half64(w1);
      f[G::PF] = fma(hu, w1, hp);
      f[2 * G::PF] = huv;
      f[3 * G::PF] = hu * tile[3 * G::Pos + e];
      f[4 * G::PF] = hu * tile[4 * G::Pos + e];
    }
    if (col >= 3 && col < 3 + 32) {
      double* g = pl + G::OffG + row * 32 + (col - 3);
      g[0] = half64(w2);
      g[G::PG] = huv;
      g[2 * G::PG] = fma(hv, w2, hp);
      g[3 * G::PG] = hv * tile[3 * G::Pos + e];
      g[4 * G::PG] = hv * tile[4 * G::Pos + e];
    }
  }
}

// Switch of one cell (SCHEME as in enl_physics.cuh).
template <int SCHEME, int TH>
__device__ __forceinline__ int switch64(const SAcc64P<TH>& A, const RhsConst& P) {
  if (SCHEME == kWeno) return 1;
  if (SCHEME == kDrp) return 0;
  if (P.level != 0) return 1;
  double r[5];
#pragma unroll
  for (int q = 0; q < 5; ++q) r[q] = A.w(0, q - 2, 0);
  int tag = sensor_line(r, P.sensor_eps, P.sensor_eps32);
#pragma unroll
  for (int q = 0; q < 5; ++q) r[q] = A.w(0, 0, q - 2);
  return tag || sensor_line(r, P.sensor_eps, P.sensor_eps32);
}

// Viscous, entropy-production and relaxation sources H1..H4
// (rhs_hybrid_high_llf.m4:161-237) from the planes, 72 FP64 operations.
//
// The reference's H3 = sigma - rho / T_n c_vn M_n + cond holds three pairs
// that cancel: kappa |grad T|^2 / T^2 enters sigma with a plus and the
// conduction with a minus, and with A_n = (T / T_n - 1) c_vn
//   rho / T A_n M_n - rho / T_n c_vn M_n = -rho c_vn M_n / T.
// What remains is (viscous heating + kappa lap T - c_vn H4) / T with H4 = rho
// M_n.  The differences stay unscaled and the viscosities, the grid spacings
// and the literals 4/3 and 2/3 are in the launch constants (make_rhs_const); the
// heating muB (u_x + v_y)^2 + mu/2 (phi_xx^2 + 2 phi_xy^2 + phi_yy^2) is the
// quadratic form qa (u_x^2 + v_y^2) + qb u_x v_y + mu phi_xy^2.  As the
// reference writes it the sources took 122 operations.
template <int TH>
__device__ __forceinline__ void sources64(const SAcc64P<TH>& A, const RhsConst& P, double H[5]) {
  const double u0 = A.u(0, 0), v0 = A.v(0, 0);
  const double ue = A.u(1, 0), uw = A.u(-1, 0), un = A.u(0, 1), us = A.u(0, -1);
  const double ve = A.v(1, 0), vw = A.v(-1, 0), vn = A.v(0, 1), vs = A.v(0, -1);
  {
    const double uxx = fma(-2.0, u0, uw + ue), uyy = fma(-2.0, u0, us + un);
    const double vxy = (A.v(1, 1) - A.v(1, -1)) - (A.v(-1, 1) - A.v(-1, -1));
    H[1] = fma(P.h_long0, uxx, fma(P.h_mixed, vxy, P.h_trans1 * uyy));
    const double vxx = fma(-2.0, v0, vw + ve), vyy = fma(-2.0, v0, vs + vn);
    const double uxy = (A.u(1, 1) - A.u(1, -1)) - (A.u(-1, 1) - A.u(-1, -1));
    H[2] = fma(P.h_long1, vyy, fma(P.h_mixed, uxy, P.h_trans0 * vxx));
  }
  const double Tc = A.t_(0, 0);
  const double rho = A.w(0, 0, 0);
  const double T_n = A.w(4, 0, 0) * rcp64(rho);
  H[4] = (rho * P.inv_tau_n) * (Tc - T_n);
  const double tmp1 = P.T_star_n * rcp64(T_n);
  const double c_vn = (P.R078 * (tmp1 * tmp1)) * (fabs(tmp1) < 700.0 ? exp64(-tmp1) : exp(-tmp1));
  const double ux = (ue - uw) * P.inv_2dx0, vy = (vn - vs) * P.inv_2dx1;
  const double phi = fma(un - us, P.inv_2dx1, (ve - vw) * P.inv_2dx0);
  const double heat = fma(ux, fma(P.q_b, vy, P.q_a * ux), fma(P.q_a * vy, vy, (P.mu * phi) * phi));
  const double txx = fma(-2.0, Tc, A.t_(-1, 0) + A.t_(1, 0)), tyy = fma(-2.0, Tc, A.t_(0, -1) + A.t_(0, 1));
  H[3] = rcp64(Tc) * fma(-c_vn, H[4], fma(P.k_0, txx, fma(P.k_1, tyy, heat)));
}

// K = H - dF/dx - dG/dy of the five fields of a DRP cell (Tam-Webb,
// rhs_hybrid_high_llf.m4:258-268), H overwritten.  The coefficients are divided
// by the first one, which the launch constants drp_0 and drp_1 hold with the
// grid spacing and a factor 2 for the planes' half fluxes.
template <int TH>
__device__ __forceinline__ void drp_flux64(const SAcc64P<TH>& A, const RhsConst& P, double H[5]) {
  constexpr double b2 = Lit::a2 / Lit::a1, b3 = Lit::a3 / Lit::a1;
#pragma unroll
  for (int k = 0; k < 5; ++k) {
    const double fx =
        fma(b3, A.fx(k, 3) - A.fx(k, -3), fma(b2, A.fx(k, 2) - A.fx(k, -2), A.fx(k, 1) - A.fx(k, -1)));
    const double gy =
        fma(b3, A.gy(k, 3) - A.gy(k, -3), fma(b2, A.gy(k, 2) - A.gy(k, -2), A.gy(k, 1) - A.gy(k, -1)));
    H[k] = fma(-fx, P.drp_0, fma(-gy, P.drp_1, H[k]));
  }
}

// Maximum of the magnitudes of n doubles of stride s around p (n odd), as
// fmax gives it for numbers (magnitudes order as their bit patterns), on the
// integer pipe.
template <int QR>
__device__ __forceinline__ double max_abs64(const double* p, int s) {
  long long m = 0;
#pragma unroll
  for (int q = -QR; q <= QR; ++q) m = max(m, __double_as_longlong(p[q * s]) & 0x7fffffffffffffffll);
  return __longlong_as_double(m);
}

// Half split speeds of a cell along x and y, rhs_hybrid_high_llf.m4:270-284.
template <int ORDER, bool LLF, int TH>
__device__ __forceinline__ void split_speeds64(const SAcc64P<TH>& A, const RhsConst& P, int cj, double& ha,
                                               double& hb) {
  if (!LLF) {
    ha = hb = 0.5 * P.alpha;
    return;
  }
  constexpr int qr = ORDER == 5 ? 3 : 2;
  const double mx = max_abs64<qr>(A.pl + A.c, 1);
  if (P.c_lr == 0.0) {
    // (x + c) + 0 h is x + c, and x + c rounds monotonically in x: the
    // maximum of the sums is the sum with the maximum (same doubles)
    ha = 0.5 * (mx + P.c);
    hb = 0.5 * (max_abs64<qr>(A.pl + SAcc64P<TH>::G::OffV + A.c, kBW64) + P.c);
  } else {
    const double hrow = P.ylo + P.dy * ((double)cj + 0.5);
    ha = 0.5 * ((mx + P.c) + P.c_lr * hrow);
    double ag = 0.0;
#pragma unroll
    for (int q = -qr; q <= qr; ++q) {
      const double h = P.ylo + P.dy * ((double)(cj + q) + 0.5);
      ag = fmax(ag, (fabs(A.v(0, q)) + P.c) + P.c_lr * h);
    }
    hb = 0.5 * ag;
  }
}

// The WENO cells of a tile, by the whole block of 256 threads: a task is one
// field of up to 32 cells (one per lane), and the warps take the tasks in
// turn, so a tile with few WENO cells still occupies every warp (a warp that
// computed all five fields of its cells kept the other seven waiting at the
// next barrier).  Tiles of one or two rows have fewer such tasks than warps:
// there a task is one field along one direction.  `list` (cell indices cy * 32
// + cx) holds the nw WENO cells of a mixed tile; without it every cell of the
// w x h tile is one.  j0 is the index of the tile's first row for the height
// of the split speeds.  D[p * 32 TH + cell] receives the flux part -(dF/dx +
// dG/dy) of field p or, with one or two rows, the unscaled differences along x
// of field p < 5 and along y of field p - 5, which weno_join64 scales and adds
// with the same operations: a cell's result does not depend on the size of its
// patch.
template <int TH>
constexpr int kFluxParts64 = TH <= 2 ? 10 : 5;
// -(dF/dx + dG/dy) from weno_flux64's differences (rounded as written: the
// compiler must not fuse the last product into the caller's sum).
template <int ORDER>
__device__ __forceinline__ double weno_scaled64(const RhsConst& P, double dfx, double dgy) {
  return __dmul_rn(ORDER == 5 ? Lit::c1_6 : 0.5, fma(dfx, P.inv_dx0, __dmul_rn(dgy, P.inv_dx1)));
}
template <int ORDER, bool LLF, int TH>
__device__ __forceinline__ void weno_tasks64(const double* tile, const double* pl, const RhsConst& P, int j0, int w,
                                             int h, const int* list, int nw, double* D) {
  using G = Geo64<TH>;
  constexpr int kParts = kFluxParts64<TH>;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nchunk = list ? (nw + 31) >> 5 : h;
  for (int t = warp; t < kParts * nchunk; t += 8) {
    const int part = t / nchunk, q = t - part * nchunk;
    int cell;
    if (list) {
      if (q * 32 + lane >= nw) continue;
      cell = list[q * 32 + lane];
    } else {
      if (lane >= w) continue;
      cell = q * 32 + lane;
    }
    const int cx = cell & 31, cy = cell >> 5;
    const int k = kParts == 5 || part < 5 ? part : part - 5;
    const SAcc64P<TH> A = acc64p<TH>(tile, pl, cx, cy);
    double ha, hb;
    split_speeds64<ORDER, LLF, TH>(A, P, j0 + cy, ha, hb);
    const double* wk = tile + k * G::Pos + A.c;
    const double* fk = pl + G::OffF + k * G::PF + A.cf;
    const double* gk = pl + G::OffG + k * G::PG + A.cg;
    double d;
    if constexpr (kParts == 5) {
      const double dfx = weno_flux64<ORDER>(wk, 1, fk, 1, ha);
      const double dgy = weno_flux64<ORDER>(wk, kBW64, gk, 32, hb);
      d = weno_scaled64<ORDER>(P, dfx, dgy);
    } else {
      const bool y = part >= 5;
      d = weno_flux64<ORDER>(wk, y ? kBW64 : 1, y ? gk : fk, y ? 32 : 1, y ? hb : ha);
    }
    D[part * (32 * TH) + cell] = d;
  }
}
// After weno_tasks64 and a barrier: leaves the flux part of field k of a cell
// in D[k * 32 TH + cell], by the whole block of 256 threads, with a barrier
// where there is something to join.  (Joined by the cells' own threads, one or
// two warps of the eight, 24 x 16 cells took 18.6 us, so 16.8.  What it makes
// of cells that are not WENO cells is not read.)
template <int ORDER, int TH>
__device__ __forceinline__ void weno_join64(double* D, const RhsConst& P) {
  if constexpr (kFluxParts64<TH> == 10) {
    constexpr int n = 5 * 32 * TH;
    for (int e = threadIdx.x; e < n; e += 256) D[e] = weno_scaled64<ORDER>(P, D[e], D[e + n]);
    __syncthreads();
  }
}

// Accessor of the learned switch's features on an FP64 tile: density and
// pressure as single-precision perturbations (the features use differences
// and ratios of differences only).
struct SAcc64Feat {
  const double* t;
  int c;
  double rho0, p0;
  static constexpr int kPos = Geo64<8>::Pos;
  __device__ float w(int k, int di, int dj) const {
    return (float)(t[k * kPos + c + dj * kBW64 + di] - (k == 0 ? rho0 : 0.0));
  }
  __device__ float p(int di, int dj) const { return (float)(t[5 * kPos + c + dj * kBW64 + di] - p0); }
};

}  // namespace enl
