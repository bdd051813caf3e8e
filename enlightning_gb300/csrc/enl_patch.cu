// Per-patch FP64 kernels behind the drop-in F77 entry points.
//
//   rhs_           fortran/rhs_*.m4           (rhs_tile_kernel)
//   runge_kutta_   fortran/runge_kutta.m4     (runge_kutta_kernel)
//   update_state_  fortran/update_state.m4    (update_state_kernel)
//   tag_cells_     fortran/tag_cells.m4       (tag_cells_kernel)
//   enl_phys_bc    enlightning.C:790-1013     (phys_bc_kernel)
//   enl_absorb     enlightning.C:634-786      (absorb_kernel)
//   enl_patch_stage  one RK stage: bc, rhs, then the rest in update_kernel
//
// Every kernel addresses its patch through a pitched view (first stored cell,
// row pitch, field stride) so that the same code serves SAMRAI's contiguous
// CellData arrays and patches embedded in a larger level array.
#include <algorithm>
#include <climits>
#include <cmath>
#include <cstdio>

#include "enl_cell64.cuh"

namespace enl {

int rhs_variant();

// The right-hand side of one patch, by tiles of 32 x TH cells, one block of
// 256 threads each: the block copies the halo box of the 7 fields into shared
// memory (8-byte asynchronous copies: a patch's rows start anywhere, so
// neither wider copies nor TMA boxes fit them), forms velocities and half
// fluxes once per position, computes the flux parts of its WENO cells field by
// field (weno_tasks64), and every thread finishes one cell.  The arithmetic is
// the batched engine's (enl_cell64.cuh).  Bound by the FP64 and FP32 pipes.
// One thread per cell reading the patch through L1, with 23 FP64 divisions and
// 40 FP64 reconstructions a WENO cell, took 444 us on 512x512 (hybrid, level
// 0), 111 us on 131x93 (fine level) and 118 us on 24x16 (level 0); this takes
// 113, 33 and 21 us.
//
// TH: 8 rows for large patches (the least work for the halo: 14 rows of
// planes for 8 of cells); fewer rows when the patch has too few tiles for the
// SMs (rhs_rows).
template <int SCHEME, int ORDER, bool LLF, int TH>
__global__ void __launch_bounds__(256, 2)
    rhs_tile_kernel(const double* __restrict__ w, const double* __restrict__ pres, const double* __restrict__ temp,
                    long pitch, long fstride, int g0, int g1, const double* __restrict__ H0, double* __restrict__ KK,
                    long opitch, long ofstride, int nx, int ny, const __grid_constant__ RhsConst P,
                    int* __restrict__ flags) {
  using G = Geo64<TH>;
  extern __shared__ __align__(16) double sm[];
  double* tile = sm;
  double* pl = tile + 7 * G::Pos;
  double* flux = pl + G::Elems;
  __shared__ int s_list[32 * TH];
  __shared__ int s_cnt[8];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int i0 = blockIdx.x * 32, j0 = blockIdx.y * TH;
  const int tw = min(32, nx - i0), th = min(TH, ny - j0);
  const long o0 = (long)(j0 + g1 - 3) * pitch + (i0 + g0 - 3);
  for (int e = tid; e < 7 * G::Pos; e += 256) {
    const int k = e / G::Pos, r = e - k * G::Pos, row = r / kBW64, col = r - row * kBW64;
    if (row < th + 6 && col < tw + 6) {
      const double* src = (k < 5 ? w + k * fstride : (k == 5 ? pres : temp)) + o0 + row * pitch + col;
      asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned)__cvta_generic_to_shared(tile + e)),
                   "l"(src));
    }
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  const bool valid = warp < th && lane < tw;
  int flag = 0;
  if (valid) flag = switch64<SCHEME, TH>(acc64p<TH>(tile, pl, lane, warp), P);
  build_planes64<TH>(tile, pl, tw, th);
  const unsigned bw = __ballot_sync(0xffffffffu, valid && flag);
  if (lane == 0) s_cnt[warp] = __popc(bw);
  __syncthreads();
  int nw = 0, ow = 0;
#pragma unroll
  for (int q = 0; q < (TH < 8 ? TH : 8); ++q) {
    if (q < warp) ow += s_cnt[q];
    nw += s_cnt[q];
  }
  if (SCHEME != kDrp && nw > 0) {
    const bool all = nw == tw * th;
    if (!all) {
      if (valid && flag) s_list[ow + __popc(bw & ((1u << lane) - 1u))] = tid;
      __syncthreads();
    }
    weno_tasks64<ORDER, LLF, TH>(tile, pl, P, j0, tw, th, all ? nullptr : s_list, nw, flux);
    __syncthreads();
    weno_join64<ORDER, TH>(flux, P);
  }
  if (!valid) return;
  const SAcc64P<TH> A = acc64p<TH>(tile, pl, lane, warp);
  const long o = (long)(j0 + warp) * opitch + (i0 + lane);
  double H[5];
  H[0] = H0[o];
  sources64(A, P, H);
  if (flag) {
#pragma unroll
    for (int k = 0; k < 5; ++k) H[k] += flux[k * (32 * TH) + tid];
  } else {
    drp_flux64(A, P, H);
  }
#pragma unroll
  for (int k = 0; k < 5; ++k) KK[k * ofstride + o] = H[k];
  if (flags) flags[o] = flag;
}

// runge_kutta.m4:60-63, association kept: (a1*ww + a2*w_n) + (beta*dt)*KK.
// A thread takes a cell of all fields: bound by launching on a small patch and
// by memory on a large one.  (A thread with four cells of one field in flight
// did the same on 512 x 512, 16.6 us, and less well where its blocks are many
// for their cells: 16 x 5000 12.4 and 26.8 us, 300 x 217 7.0 and 8.0.)
__global__ void runge_kutta_kernel(double* __restrict__ wn, long pitch, long fstride, int g0, int g1,
                                   const double* __restrict__ ww, const double* __restrict__ KK, long ipitch,
                                   long ifstride, int nx, int ny, int nequ, double a1, double a2, double bdt) {
  const int ci = blockIdx.x * blockDim.x + threadIdx.x, cj = blockIdx.y * blockDim.y + threadIdx.y;
  if (ci >= nx || cj >= ny) return;
  const long g = (long)(cj + g1) * pitch + (ci + g0), c = (long)cj * ipitch + ci;
  for (int k = 0; k < nequ; ++k)
    wn[k * fstride + g] = __dadd_rn(__dadd_rn(__dmul_rn(a1, ww[k * ifstride + c]), __dmul_rn(a2, wn[k * fstride + g])),
                                    __dmul_rn(bdt, KK[k * ifstride + c]));
}

// update_state.m4:87-107 (eos64).
__global__ void update_state_kernel(const double* __restrict__ w, double* __restrict__ pres,
                                    double* __restrict__ temp, long pitch, long fstride, int g0, int g1,
                                    int nx, int ny, double ylo, double dy, const __grid_constant__ EosConst64 E) {
  int ci = blockIdx.x * blockDim.x + threadIdx.x;
  int cj = blockIdx.y * blockDim.y + threadIdx.y;
  if (ci >= nx || cj >= ny) return;
  long g = (long)(cj + g1) * pitch + (ci + g0);
  double p, T;
  eos64(E, w[g], w[3 * fstride + g], row_height64(ylo, dy, cj), p, T);
  pres[g] = p;
  temp[g] = T;
}

// tag_cells.m4:58-108, bit-exact (enl_ratio.cuh).
__global__ void tag_cells_kernel(int* __restrict__ tags, long tpitch, const double* __restrict__ w,
                                 const double* __restrict__ H0, long pitch, int g0, int g1, int nx, int ny,
                                 int tag_val, double ep0, float ep0f, double ep1, float ep1f) {
  int ci = blockIdx.x * blockDim.x + threadIdx.x;
  int cj = blockIdx.y * blockDim.y + threadIdx.y;
  if (ci >= nx || cj >= ny) return;
  long g = (long)(cj + g1) * pitch + (ci + g0);
  tags[(long)cj * tpitch + ci] = tag_cell64(H0 + g, w + g, pitch, ep0, ep0f, ep1, ep1f) ? tag_val : 0;
}

// Physical-boundary fill, enlightning.C:830-1008.  Each ghost cell of an edge
// box receives the first interior cell of its row or column (the reference's
// cascading copy), the normal momentum negated on REFLECT sides.  The nodes
// (corners) then copy along x from the cell next to the corner box, an edge
// ghost or a neighbour-filled one, x-momentum negated when the adjacent x side
// is REFLECT.  An edge ghost is itself a copy of an interior cell, so a node
// takes that cell's value and no ghost is read that this kernel writes: edges
// and nodes go in one launch (they were up to eight: 3 us each on the GPU and
// as much on the host for a 24x16 patch's 12 us of arithmetic).  The fields
// are w_n (5), pressure, temperature, source; blockIdx.y picks one.
struct PatchFields8 {
  double* f[8];
};

struct BandArgs {
  PatchFields8 F;
  long pitch;
  int nx, ny, g0, g1, fill0, fill1;
  int touches, reflect;  // bit per side L, R, B, T
  int cells;             // band cells of the sides touched and of their nodes
};

__global__ void phys_bc_kernel(const __grid_constant__ BandArgs A) {
  const int k = blockIdx.y;
  double* f = A.F.f[k];
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < A.cells; t += gridDim.x * blockDim.x) {
    int r = t, i = -1, j = -1, si = 0, sj = 0;
    bool neg = false;
    const int nsx = A.ny * A.fill0, nsy = A.nx * A.fill1, nn = A.fill0 * A.fill1;
#pragma unroll
    for (int side = 0; side < 4; ++side) {
      if (!(A.touches & (1 << side)) || i >= 0) continue;
      const int n = side < 2 ? nsx : nsy;
      if (r >= n) {
        r -= n;
        continue;
      }
      if (side < 2) {
        const int d = r % A.fill0;
        sj = j = r / A.fill0 + A.g1;
        si = side == 0 ? A.g0 : A.g0 + A.nx - 1;
        i = side == 0 ? A.g0 - 1 - d : A.g0 + A.nx + d;
        neg = k == 1 && (A.reflect & (1 << side));
      } else {
        const int d = r / A.nx;
        si = i = r - d * A.nx + A.g0;
        sj = side == 2 ? A.g1 : A.g1 + A.ny - 1;
        j = side == 2 ? A.g1 - 1 - d : A.g1 + A.ny + d;
        neg = k == 2 && (A.reflect & (1 << side));
      }
    }
    if (i < 0) {
#pragma unroll
      for (int loc = 0; loc < 4; ++loc) {
        const int xs = loc & 1, ys = 2 + (loc >> 1);
        if (!((A.touches >> xs | A.touches >> ys) & 1) || i >= 0) continue;
        if (r >= nn) {
          r -= nn;
          continue;
        }
        const int dx = r % A.fill0, dy = r / A.fill0;
        j = ys == 3 ? A.g1 + A.ny + dy : A.g1 - 1 - dy;
        i = xs ? A.g0 + A.nx + dx : A.g0 - 1 - dx;
        si = xs ? A.g0 + A.nx - 1 : A.g0;
        // the row's ghost beside the node: filled from the interior when the
        // patch touches that side, a neighbour's cell otherwise
        const bool filled = (A.touches >> ys) & 1;
        sj = filled ? (ys == 3 ? A.g1 + A.ny - 1 : A.g1) : j;
        neg = (k == 1 && ((A.reflect >> xs) & 1)) != (k == 2 && filled && ((A.reflect >> ys) & 1));
      }
    }
    const double v = f[(long)sj * A.pitch + si];
    f[(long)j * A.pitch + i] = neg ? -v : v;
  }
}

// Absorbing envelope, enlightning.C:671-783, including the loop-exit rules:
// along x each row runs from the boundary side while the previous envelope
// value differs from 1 by more than 1e-8 (the first row starts from the
// envelope of the first cell, later rows from tmp = 0); along y the same rule
// runs over rows.  dir: 0 = L, 1 = R, 2 = B, 3 = T.
//
// The distance from the side grows along the walk, and the envelope with it,
// so whether the walk reaches a cell follows from the cell before it alone:
// one thread per cell applies the sides that reach it in the reference's
// order.  A block covers 32 x 8 cells and computes the factors of its columns
// and rows once; blocks that no side reaches leave without touching the
// patch.  Walking the rows and columns serially (a thread per row, an FP64
// exponential per cell) took 4.2 ms of a 131x93 patch's 4.3 ms step.
struct AbsorbConst {
  double xlo0, xlo1, dx0, dx1, gxlo0, gxlo1, gxhi0, gxhi1, w2, p0, T0, rho0;
};

// -exp(-log(2.0) / SQUARE(W) * SQUARE(d)) + 1 (enlightning.C:676).
__device__ __forceinline__ double envelope(double d, double w2) {
  return __dadd_rn(-exp(__dmul_rn(__ddiv_rn(-log(2.0), w2), __dmul_rn(d, d))), 1.0);
}

// (q - q_amb) * tmp + q_amb, rounded as written (no contraction).
__device__ __forceinline__ double relax_to(double q, double amb, double tmp) {
  return __dadd_rn(__dmul_rn(__dsub_rn(q, amb), tmp), amb);
}

__device__ __forceinline__ void absorb_apply(PatchFields8 F, long g, double tmp, const AbsorbConst& A) {
  F.f[5][g] = relax_to(F.f[5][g], A.p0, tmp);
  F.f[6][g] = relax_to(F.f[6][g], A.T0, tmp);
  F.f[0][g] = relax_to(F.f[0][g], A.rho0, tmp);
  F.f[1][g] = __dmul_rn(F.f[1][g], tmp);
  F.f[2][g] = __dmul_rn(F.f[2][g], tmp);
  F.f[3][g] = __dmul_rn(F.f[3][g], tmp);
  F.f[4][g] = relax_to(F.f[4][g], __dmul_rn(A.T0, A.rho0), tmp);
}

// Factors of a block's columns (L, R) and rows (B, T), and whether the walk from
// the side reaches them (2: not in the first row), by the block's first 128
// threads; true when any is reached.
struct AbsorbShared {
  double f[4][32];
  unsigned char r[4][32];
};
__device__ __forceinline__ bool absorb_factors(AbsorbShared& S, int tid, int i0, int j0, int nx, int ny, int dirs,
                                               const AbsorbConst& A) {
  if (tid >= 128) return false;
  const int dir = tid >> 5, q = tid & 31;
  const int n = dir < 2 ? nx : ny, c = (dir < 2 ? i0 : j0) + q;
  int r = 0;
  if ((dirs & (1 << dir)) && c < n && (dir < 2 || q < 8)) {
    auto dist = [&](int m) {
      if (dir < 2) {
        const double xc = A.xlo0 + A.dx0 * ((double)m + 0.5);
        return dir == 0 ? (xc - A.gxlo0) : (A.gxhi0 - xc);
      }
      const double yc = A.xlo1 + A.dx1 * ((double)m + 0.5);
      return dir == 2 ? (yc - A.gxlo1) : (A.gxhi1 - yc);
    };
    auto go_on = [](double tmp) { return fabs(1.0 - tmp) > 1.0e-8; };
    const bool first = c == ((dir & 1) ? n - 1 : 0);
    if (first) {
      // the edge cell itself is walked without a test in x, except on the
      // first row, and with its own factor's test there and in y
      const double f = envelope(dist(c), A.w2);
      r = go_on(f) ? 1 : (dir < 2 ? 2 : 0);
      S.f[dir][q] = f;
    } else {
      // beyond 6 widths the factor is within 2e-11 of 1: the walk has ended
      const double d = dist((dir & 1) ? c + 1 : c - 1);
      if (d * d < 36.0 * A.w2 && go_on(envelope(d, A.w2))) {
        r = 1;
        S.f[dir][q] = envelope(dist(c), A.w2);
      }
    }
  }
  S.r[dir][q] = (unsigned char)r;
  return r != 0;
}
__device__ __forceinline__ int absorb_reached(const AbsorbShared& S, int lx, int ly, int cj) {
  int reach = 0;
#pragma unroll
  for (int dir = 0; dir < 4; ++dir) {
    const int r = S.r[dir][dir < 2 ? lx : ly];
    if (r == 1 || (r == 2 && cj != 0)) reach |= 1 << dir;
  }
  return reach;
}
// v: w_n (5), pressure, temperature of a cell, relaxed by the sides that reach
// it in the reference's order.
__device__ __forceinline__ void absorb_cell(const AbsorbShared& S, int reach, int lx, int ly, const AbsorbConst& A,
                                            double v[7]) {
  const double rT = __dmul_rn(A.T0, A.rho0);
#pragma unroll
  for (int dir = 0; dir < 4; ++dir) {
    if (!(reach & (1 << dir))) continue;
    const double tmp = S.f[dir][dir < 2 ? lx : ly];
    v[5] = relax_to(v[5], A.p0, tmp);
    v[6] = relax_to(v[6], A.T0, tmp);
    v[0] = relax_to(v[0], A.rho0, tmp);
    v[1] = __dmul_rn(v[1], tmp);
    v[2] = __dmul_rn(v[2], tmp);
    v[3] = __dmul_rn(v[3], tmp);
    v[4] = relax_to(v[4], rT, tmp);
  }
}

__global__ void __launch_bounds__(256) absorb_kernel(PatchFields8 F, long pitch, int nx, int ny, int g0, int g1,
                                                     int dirs, AbsorbConst A) {
  __shared__ AbsorbShared S;
  const int tid = threadIdx.x, i0 = blockIdx.x * 32, j0 = blockIdx.y * 8;
  if (!__syncthreads_or(absorb_factors(S, tid, i0, j0, nx, ny, dirs, A))) return;
  const int lx = tid & 31, ly = tid >> 5, ci = i0 + lx, cj = j0 + ly;
  if (ci >= nx || cj >= ny) return;
  const int reach = absorb_reached(S, lx, ly, cj);
  if (!reach) return;
  const long g = (long)(cj + g1) * pitch + (ci + g0);
  double v[7];
#pragma unroll
  for (int k = 0; k < 7; ++k) v[k] = F.f[k][g];
  absorb_cell(S, reach, lx, ly, A, v);
#pragma unroll
  for (int k = 0; k < 7; ++k) F.f[k][g] = v[k];
}

// runge_kutta, update_state and the absorbing envelope of a stage in one pass
// (enl_patch_stage): the same operations on the same values as the three
// kernels, without the passes over w_n, p and T between them and two launches
// less.  Bound by its 22 doubles a cell on a large patch, by launches on a small
// one: an advance of a 512 x 512 patch took 547 us before and 526 after, of a
// 24 x 16 one 195 and 128 (most of that from one library call for a stage's four).
struct UpdateArgs {
  PatchFields8 F;  // w_n, pressure, temperature
  const double *ww, *KK;
  long pitch;
  int nx, ny, g0, g1, dirs;
  double a1, a2, bdt, ylo, dy;
  EosConst64 E;
  AbsorbConst A;
};
__global__ void __launch_bounds__(256) update_kernel(const __grid_constant__ UpdateArgs U) {
  __shared__ AbsorbShared S;
  const int tid = threadIdx.x, i0 = blockIdx.x * 32, j0 = blockIdx.y * 8;
  const int lx = tid & 31, ly = tid >> 5, ci = i0 + lx, cj = j0 + ly;
  const bool valid = ci < U.nx && cj < U.ny;
  const long g = (long)(cj + U.g1) * U.pitch + (ci + U.g0), c = (long)cj * U.nx + ci, fs = (long)U.nx * U.ny;
  double v[7], u[5], k[5];
  if (valid) {
#pragma unroll
    for (int q = 0; q < 5; ++q) {
      u[q] = U.ww[q * fs + c];
      v[q] = U.F.f[q][g];
      k[q] = U.KK[q * fs + c];
    }
#pragma unroll
    for (int q = 0; q < 5; ++q)
      v[q] = __dadd_rn(__dadd_rn(__dmul_rn(U.a1, u[q]), __dmul_rn(U.a2, v[q])), __dmul_rn(U.bdt, k[q]));
    eos64(U.E, v[0], v[3], row_height64(U.ylo, U.dy, cj), v[5], v[6]);
  }
  if (U.dirs && __syncthreads_or(absorb_factors(S, tid, i0, j0, U.nx, U.ny, U.dirs, U.A)) && valid) {
    const int reach = absorb_reached(S, lx, ly, cj);
    if (reach) absorb_cell(S, reach, lx, ly, U.A, v);
  }
  if (valid) {
#pragma unroll
    for (int q = 0; q < 7; ++q) U.F.f[q][g] = v[q];
  }
}

// The same walks serially, for a patch that lies partly outside the domain
// (its distance from a side is not positive at the walk's first cell, so the
// factors need not grow along the walk): one thread per row or column, and one
// kernel per side, since what depends on the side lies on the walk's chain (64 x
// 64 cells, four sides: 873 us with the side as an argument, 728 so).
template <int DIR>
__global__ void absorb_walk_kernel(PatchFields8 F, long pitch, int nx, int ny, int g0, int g1, AbsorbConst A) {
  const double ep = 1.0e-8;
  constexpr bool x = DIR < 2, upper = DIR & 1;
  const int t = blockIdx.x * blockDim.x + threadIdx.x, len = x ? nx : ny;
  if (t >= (x ? ny : nx)) return;
  auto dist = [&](int c) {
    const double q = x ? A.xlo0 + A.dx0 * ((double)c + 0.5) : A.xlo1 + A.dx1 * ((double)c + 0.5);
    return upper ? ((x ? A.gxhi0 : A.gxhi1) - q) : (q - (x ? A.gxlo0 : A.gxlo1));
  };
  double tmp = (!x || t == 0) ? envelope(dist(upper ? len - 1 : 0), A.w2) : 0.0;
  for (int n = 0; (fabs(1.0 - tmp) > ep) && n < len; ++n) {
    const int c = upper ? len - 1 - n : n;
    tmp = envelope(dist(c), A.w2);
    absorb_apply(F, x ? (long)(t + g1) * pitch + (c + g0) : (long)(c + g1) * pitch + (t + g0), tmp, A);
  }
}

// ---------------------------------------------------------------------------
// host helpers
// ---------------------------------------------------------------------------

RhsConst make_rhs_const(const double* xlo, const double* dx, double alpha, double kappa, double mu,
                        double muB, double R, double T_star_n, double tau_n, const double* tol, int level,
                        double c, double c_lr) {
  RhsConst P;
  P.inv_dx0 = 1.0 / dx[0];
  P.inv_dx1 = 1.0 / dx[1];
  P.inv_dx0sq = 1.0 / (dx[0] * dx[0]);
  P.inv_dx1sq = 1.0 / (dx[1] * dx[1]);
  P.inv_2dx0 = 1.0 / (2.0 * dx[0]);
  P.inv_2dx1 = 1.0 / (2.0 * dx[1]);
  P.inv_4dxdy = 1.0 / ((4.0 * dx[0]) * dx[1]);
  P.kappa = kappa;
  P.mu = mu;
  P.muB = muB;
  P.R = R;
  P.T_star_n = T_star_n;
  P.inv_tau_n = 1.0 / tau_n;
  P.alpha = alpha;
  P.c = c;
  P.c_lr = c_lr;
  P.ylo = xlo[1];
  P.dy = dx[1];
  // ep = 0.9*tolerance(2)*(xi**2)/(1-0.9*(tolerance(2)**2)), xi = 1
  // (rhs_hybrid_high_llf.m4:114-115); this file is built without FMA
  // contraction of host code so the value is the reference's.
  const double xi = 1.0;
  P.sensor_eps = ((Lit::c0_9 * tol[2]) * (xi * xi)) / (1.0 - Lit::c0_9 * (tol[2] * tol[2]));
  P.sensor_eps32 = ratio_eps32(P.sensor_eps);
  P.level = level;
  const double lon = muB + Lit::c4_3 * mu, mix = muB + (1.0 - Lit::c2_3) * mu;
  P.h_long0 = lon * P.inv_dx0sq;
  P.h_long1 = lon * P.inv_dx1sq;
  P.h_trans0 = mu * P.inv_dx0sq;
  P.h_trans1 = mu * P.inv_dx1sq;
  P.h_mixed = mix * P.inv_4dxdy;
  P.q_a = muB + 0.5 * mu * (Lit::c4_3 * Lit::c4_3 + Lit::c2_3 * Lit::c2_3);
  P.q_b = 2.0 * muB - 2.0 * mu * (Lit::c4_3 * Lit::c2_3);
  P.k_0 = kappa * P.inv_dx0sq;
  P.k_1 = kappa * P.inv_dx1sq;
  P.R078 = Lit::c0_78 * R;
  P.drp_0 = 2.0 * Lit::a1 * P.inv_dx0;
  P.drp_1 = 2.0 * Lit::a1 * P.inv_dx1;
  return P;
}

// Rows per tile.  With fewer rows more blocks share a patch, and each does more
// work for its halo (TH + 6 rows of planes for TH of cells).  Two blocks run on
// an SM.  Measured, hybrid scheme on level 0 / on a fine level (WENO in every
// cell), us for 8, 4, 2, 1 rows:
//   32x32    62 38 25 21    / 58 35 23 17
//   131x93   66 40 39 46    / 59 35 33 42
//   256x256  69 59 59 85    / 93 99 101 132
//   384x384  97 78 89 154   / 175 184 211 278
//   512x512  129 113 144 257 / 289 300 349 477
//   700x700  181 202 247 462 / 506 535 629 883
// the lower-order hybrid scheme and DRP alone:
//   32x32    42 27 20 17    / 19 12 11 11
//   131x93   47 29 29 35    / 19 12 13 15
//   256x256  52 48 51 77    / 31 31 37 48
//   512x512  115 113 143 251 / 97 97 113 155
//   700x700  179 203 257 461 / 171 175 207 284
// so 8 rows from four waves of blocks on, 4 from one wave, 2 from half a wave.
static int rhs_rows(int nx, int ny) {
  const long cols = (nx + 31) / 32;
  int dev = 0, nsm = 1;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  if (cols * ((ny + 7) / 8) >= 8l * nsm) return 8;
  if (cols * ((ny + 3) / 4) >= 2l * nsm) return 4;
  return cols * ((ny + 1) / 2) >= nsm ? 2 : 1;
}

// Sides with an envelope, and whether every walk from them starts inside the
// domain (so that the factors grow along it).
static bool absorb_dirs(const AbsorbConst& A, int nx, int ny, const int* bc, int& dirs) {
  const double first[4] = {(A.xlo0 + A.dx0 * 0.5) - A.gxlo0, A.gxhi0 - (A.xlo0 + A.dx0 * (nx - 0.5)),
                           (A.xlo1 + A.dx1 * 0.5) - A.gxlo1, A.gxhi1 - (A.xlo1 + A.dx1 * (ny - 0.5))};
  dirs = 0;
  bool inside = A.dx0 > 0.0 && A.dx1 > 0.0 && A.w2 > 0.0;
  for (int dir = 0; dir < 4; ++dir)
    if (bc[dir] == kAbsorb) {
      dirs |= 1 << dir;
      inside = inside && first[dir] > 0.0;
    }
  return inside;
}

struct RhsCall {
  const double *w, *pres, *temp;
  long pitch, fstride;
  int g0, g1;
  const double* H0;
  double* KK;
  long opitch, ofstride;
  int nx, ny;
  int* flags;
};

template <int SCHEME, int ORDER, bool LLF, int TH>
static void launch_rhs_rows(const RhsCall& c, const RhsConst& P) {
  constexpr size_t bytes = (7 * Geo64<TH>::Pos + Geo64<TH>::Elems + kFluxParts64<TH> * 32 * TH) * sizeof(double);
  auto fn = rhs_tile_kernel<SCHEME, ORDER, LLF, TH>;
  if (bytes > 48 * 1024) cudaFuncSetAttribute((const void*)fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  const dim3 grid((c.nx + 31) / 32, (c.ny + TH - 1) / TH);
  fn<<<grid, 256, bytes, stream()>>>(c.w, c.pres, c.temp, c.pitch, c.fstride, c.g0, c.g1, c.H0, c.KK, c.opitch,
                                     c.ofstride, c.nx, c.ny, P, c.flags);
}

template <int SCHEME, int ORDER, bool LLF>
static void launch_rhs_scheme(const RhsCall& c, const RhsConst& P) {
  switch (rhs_rows(c.nx, c.ny)) {
    case 8: return launch_rhs_rows<SCHEME, ORDER, LLF, 8>(c, P);
    case 4: return launch_rhs_rows<SCHEME, ORDER, LLF, 4>(c, P);
    case 2: return launch_rhs_rows<SCHEME, ORDER, LLF, 2>(c, P);
    default: return launch_rhs_rows<SCHEME, ORDER, LLF, 1>(c, P);
  }
}

static int launch_rhs(int variant, const RhsCall& c, const RhsConst& P) {
  switch (variant) {
    case 0: launch_rhs_scheme<kHybrid, 5, true>(c, P); break;
    case 1: launch_rhs_scheme<kHybrid, 5, false>(c, P); break;
    case 2: launch_rhs_scheme<kHybrid, 3, true>(c, P); break;
    case 3: launch_rhs_scheme<kHybrid, 3, false>(c, P); break;
    case 4: launch_rhs_scheme<kWeno, 5, true>(c, P); break;
    case 5: launch_rhs_scheme<kWeno, 5, false>(c, P); break;
    case 6: launch_rhs_scheme<kWeno, 3, true>(c, P); break;
    case 7: launch_rhs_scheme<kWeno, 3, false>(c, P); break;
    case 8: launch_rhs_scheme<kDrp, 5, false>(c, P); break;
    default:
      set_error(ENL_ERR_ARG);
      return ENL_ERR_ARG;
  }
  return check_launch("rhs");
}

// Pitched launch used by the engine's plain path: w points at the first stored
// cell (ghost width 3 on both sides of the patch).
int launch_rhs_pitched(int variant, const double* w, const double* pres, const double* temp, long pitch,
                       long fstride, const double* H0, double* KK, long opitch, long ofstride, int nx, int ny,
                       const RhsConst& P) {
  return launch_rhs(variant, RhsCall{w, pres, temp, pitch, fstride, 3, 3, H0, KK, opitch, ofstride, nx, ny, nullptr},
                    P);
}

}  // namespace enl

using namespace enl;

static inline dim3 grid2d(int nx, int ny, dim3 b) { return dim3((nx + b.x - 1) / b.x, (ny + b.y - 1) / b.y); }

extern "C" {

int enl_rhs(int variant, int ifirst0, int ilast0, int ifirst1, int ilast1, int gcw0, int gcw1,
            const double* xlo, const double* dx, const double* w_n, long w_pitch, long w_fstride,
            const double* source, double* rhs, long out_pitch, long out_fstride, const double* pressure,
            const double* temperature, double weno_alpha, double kappa, double mu, double muB, double R,
            double T_star_n, double tau_n, const double* tag_tolerance, int level, double c, double c_lr,
            int* flags) {
  int nx = ilast0 - ifirst0 + 1, ny = ilast1 - ifirst1 + 1;
  if (nx <= 0 || ny <= 0 || gcw0 < 3 || gcw1 < 3 || !w_n || !rhs || !source || !pressure || !temperature ||
      !xlo || !dx || !tag_tolerance || w_pitch < nx + 2 * gcw0 || out_pitch < nx) {
    set_error(ENL_ERR_ARG);
    return ENL_ERR_ARG;
  }
  RhsConst P = make_rhs_const(xlo, dx, weno_alpha, kappa, mu, muB, R, T_star_n, tau_n, tag_tolerance, level,
                              c, c_lr);
  return launch_rhs(variant, RhsCall{w_n, pressure, temperature, w_pitch, w_fstride, gcw0, gcw1, source, rhs,
                                     out_pitch, out_fstride, nx, ny, flags},
                    P);
}

void rhs_(const int& ifirst0, const int& ilast0, const int& ifirst1, const int& ilast1, const int& gcw0,
          const int& gcw1, const double* xlo, const double* dx, const double* w_n, const double* source,
          double* rhs, const double* pressure, const double* temperature, const double& weno_alpha,
          const double& kappa, const double& mu, const double& muB, const double& R, const double& T_star_n,
          const double& T_star_o, const double& tau_n, const double& tau_o, const double* tag_tolerance,
          const int& level, const double& c, const double& c_lr, const int& nequ) {
  (void)T_star_o;
  (void)tau_o;
  if (nequ != kNequ) {
    set_error(ENL_ERR_ARG);
    return;
  }
  int nx = ilast0 - ifirst0 + 1, ny = ilast1 - ifirst1 + 1;
  long pitch = nx + 2 * gcw0, fstride = pitch * (ny + 2 * gcw1);
  enl_rhs(rhs_variant(), ifirst0, ilast0, ifirst1, ilast1, gcw0, gcw1, xlo, dx, w_n, pitch, fstride, source,
          rhs, nx, (long)nx * ny, pressure, temperature, weno_alpha, kappa, mu, muB, R, T_star_n, tau_n,
          tag_tolerance, level, c, c_lr, nullptr);
}

void runge_kutta_(const int& ifirst0, const int& ilast0, const int& ifirst1, const int& ilast1,
                  const int& gcw0, const int& gcw1, const double& dt, const double& alpha_1,
                  const double& alpha_2, const double& beta, double* w_n, const double* w, const double* rhs,
                  const int& nequ) {
  int nx = ilast0 - ifirst0 + 1, ny = ilast1 - ifirst1 + 1;
  if (nx <= 0 || ny <= 0 || nequ < 1 || !w_n || !w || !rhs) {
    set_error(ENL_ERR_ARG);
    return;
  }
  long pitch = nx + 2 * gcw0, fstride = pitch * (ny + 2 * gcw1);
  const dim3 block(32, 4);
  runge_kutta_kernel<<<grid2d(nx, ny, block), block, 0, stream()>>>(w_n, pitch, fstride, gcw0, gcw1, w, rhs, nx,
                                                                    (long)nx * ny, nx, ny, nequ, alpha_1, alpha_2,
                                                                    beta * dt);
  check_launch("runge_kutta");
}

void update_state_(const double* dx, const double* xlo, const int& ifirst0, const int& ilast0,
                   const int& ifirst1, const int& ilast1, const int& gcw0, const int& gcw1, const double* w_n,
                   double* pressure, double* temperature, const double& rho0, const double& c,
                   const double& gamma1, const double& c_p, const double& p0, const double& T0,
                   const double& c_lr, const double& c_v, const double& R_tilde, const double& M,
                   const double& R, const int& nequ) {
  (void)R_tilde;
  (void)M;
  (void)nequ;
  int nx = ilast0 - ifirst0 + 1, ny = ilast1 - ifirst1 + 1;
  if (nx <= 0 || ny <= 0 || !w_n || !pressure || !temperature || !dx || !xlo) {
    set_error(ENL_ERR_ARG);
    return;
  }
  long pitch = nx + 2 * gcw0, fstride = pitch * (ny + 2 * gcw1);
  const EosConst64 E = make_eos_const64(rho0, c, c_lr, gamma1, c_p, p0, T0, c_v, R);
  dim3 block(32, 4);
  update_state_kernel<<<grid2d(nx, ny, block), block, 0, stream()>>>(w_n, pressure, temperature, pitch,
                                                                       fstride, gcw0, gcw1, nx, ny, xlo[1], dx[1], E);
  check_launch("update_state");
}

void tag_cells_(const int& ifirst0, const int& ilast0, const int& ifirst1, const int& ilast1, const int& gcw0,
                const int& gcw1, int* tags, const double* w_n, const double* source, const int& refine_tag_val,
                const double* tag_tolerance, const int& nequ) {
  (void)nequ;
  int nx = ilast0 - ifirst0 + 1, ny = ilast1 - ifirst1 + 1;
  if (nx <= 0 || ny <= 0 || gcw0 < 1 || gcw1 < 1 || !tags || !w_n || !source || !tag_tolerance) {
    set_error(ENL_ERR_ARG);
    return;
  }
  long pitch = nx + 2 * gcw0;
  const double xi = 1.0;
  double ep0 = ((Lit::c0_9 * tag_tolerance[0]) * (xi * xi)) / (1.0 - Lit::c0_9 * (tag_tolerance[0] * tag_tolerance[0]));
  double ep1 = ((Lit::c0_9 * tag_tolerance[1]) * (xi * xi)) / (1.0 - Lit::c0_9 * (tag_tolerance[1] * tag_tolerance[1]));
  dim3 block(32, 4);
  tag_cells_kernel<<<grid2d(nx, ny, block), block, 0, stream()>>>(tags, nx, w_n, source, pitch, gcw0, gcw1, nx,
                                                                  ny, refine_tag_val, ep0, ratio_eps32(ep0), ep1,
                                                                  ratio_eps32(ep1));
  check_launch("tag_cells");
}

int enl_phys_bc(int ifirst0, int ilast0, int ifirst1, int ilast1, int gcw0, int gcw1, const int* touches,
                const int* bc, int fill0, int fill1, double* w_n, double* pressure, double* temperature,
                double* source) {
  int nx = ilast0 - ifirst0 + 1, ny = ilast1 - ifirst1 + 1;
  if (nx <= 0 || ny <= 0 || !touches || !bc || fill0 < 0 || fill1 < 0 || fill0 > gcw0 || fill1 > gcw1 || !w_n ||
      !pressure || !temperature || !source) {
    set_error(ENL_ERR_ARG);
    return ENL_ERR_ARG;
  }
  long pitch = nx + 2 * gcw0, fstride = pitch * (ny + 2 * gcw1);
  BandArgs A;
  for (int k = 0; k < 5; ++k) A.F.f[k] = w_n + k * fstride;
  A.F.f[5] = pressure;
  A.F.f[6] = temperature;
  A.F.f[7] = source;
  A.pitch = pitch;
  A.nx = nx;
  A.ny = ny;
  A.g0 = gcw0;
  A.g1 = gcw1;
  A.fill0 = fill0;
  A.fill1 = fill1;
  A.touches = A.reflect = 0;
  long cells = 0;
  for (int side = 0; side < 4; ++side) {
    if (touches[side]) {
      A.touches |= 1 << side;
      cells += side < 2 ? (long)ny * fill0 : (long)nx * fill1;
    }
    if (bc[side] == kReflect) A.reflect |= 1 << side;
  }
  for (int loc = 0; loc < 4; ++loc)
    if (touches[loc & 1] || touches[2 + (loc >> 1)]) cells += (long)fill0 * fill1;
  if (cells == 0) return ENL_OK;
  if (cells > INT_MAX / 2) {
    set_error(ENL_ERR_ARG);
    return ENL_ERR_ARG;
  }
  A.cells = (int)cells;
  phys_bc_kernel<<<dim3((unsigned)std::min<long>((cells + 127) / 128, 4096), 8), 128, 0, stream()>>>(A);
  return check_launch("phys_bc");
}

int enl_absorb(int ifirst0, int ilast0, int ifirst1, int ilast1, int gcw0, int gcw1, const double* patch_xlo,
               const double* dx, const double* grid_xlo, const double* grid_xhi, const int* bc,
               double absorb_width, double p0, double T0, double rho0, double* w_n, double* pressure,
               double* temperature) {
  int nx = ilast0 - ifirst0 + 1, ny = ilast1 - ifirst1 + 1;
  if (nx <= 0 || ny <= 0 || !patch_xlo || !dx || !grid_xlo || !grid_xhi || !bc || !w_n || !pressure ||
      !temperature) {
    set_error(ENL_ERR_ARG);
    return ENL_ERR_ARG;
  }
  if (!(bc[0] == kAbsorb || bc[1] == kAbsorb || bc[2] == kAbsorb || bc[3] == kAbsorb)) return ENL_OK;
  long pitch = nx + 2 * gcw0, fstride = pitch * (ny + 2 * gcw1);
  PatchFields8 F;
  for (int k = 0; k < 5; ++k) F.f[k] = w_n + k * fstride;
  F.f[5] = pressure;
  F.f[6] = temperature;
  F.f[7] = nullptr;
  AbsorbConst A{patch_xlo[0], patch_xlo[1], dx[0], dx[1], grid_xlo[0], grid_xlo[1], grid_xhi[0], grid_xhi[1],
                absorb_width * absorb_width, p0, T0, rho0};
  int dirs = 0;
  const bool inside = absorb_dirs(A, nx, ny, bc, dirs);
  if (inside) {
    absorb_kernel<<<dim3((nx + 31) / 32, (ny + 7) / 8), 256, 0, stream()>>>(F, pitch, nx, ny, gcw0, gcw1, dirs, A);
  } else {
    auto walk = [&](auto kernel, int dir) {
      if (dirs & (1 << dir))
        kernel<<<((dir < 2 ? ny : nx) + 127) / 128, 128, 0, stream()>>>(F, pitch, nx, ny, gcw0, gcw1, A);
    };
    walk(absorb_walk_kernel<0>, 0);
    walk(absorb_walk_kernel<1>, 1);
    walk(absorb_walk_kernel<2>, 2);
    walk(absorb_walk_kernel<3>, 3);
  }
  return check_launch("absorb");
}

int enl_patch_stage(const enl_patch* P, double dt, double alpha_1, double alpha_2, double beta, int fill_ghosts) {
  if (!P) {
    set_error(ENL_ERR_ARG);
    return ENL_ERR_ARG;
  }
  const int *b = P->box, g0 = P->gcw[0], g1 = P->gcw[1];
  const int nx = b[1] - b[0] + 1, ny = b[3] - b[2] + 1;
  if (nx <= 0 || ny <= 0 || !P->w_n || !P->w || !P->rhs || !P->source || !P->pressure || !P->temperature) {
    set_error(ENL_ERR_ARG);
    return ENL_ERR_ARG;
  }
  int st = ENL_OK;
  if (fill_ghosts)
    st = enl_phys_bc(b[0], b[1], b[2], b[3], g0, g1, P->touches, P->bc, P->fill[0], P->fill[1], P->w_n, P->pressure,
                     P->temperature, P->source_g);
  const long pitch = nx + 2 * g0, fstride = pitch * (ny + 2 * g1);
  if (st == ENL_OK)
    st = enl_rhs(rhs_variant(), b[0], b[1], b[2], b[3], g0, g1, P->xlo, P->dx, P->w_n, pitch, fstride, P->source, P->rhs,
                 nx, (long)nx * ny, P->pressure, P->temperature, P->weno_alpha, P->kappa, P->mu, P->muB, P->R,
                 P->T_star_n, P->tau_n, P->tol, P->level, P->c, P->c_lr, nullptr);
  if (st != ENL_OK) return st;
  UpdateArgs U;
  for (int k = 0; k < 5; ++k) U.F.f[k] = P->w_n + k * fstride;
  U.F.f[5] = P->pressure;
  U.F.f[6] = P->temperature;
  U.F.f[7] = nullptr;
  U.ww = P->w;
  U.KK = P->rhs;
  U.pitch = pitch;
  U.nx = nx;
  U.ny = ny;
  U.g0 = g0;
  U.g1 = g1;
  U.a1 = alpha_1;
  U.a2 = alpha_2;
  U.bdt = beta * dt;
  U.ylo = P->xlo[1];
  U.dy = P->dx[1];
  U.E = make_eos_const64(P->rho0, P->c, P->c_lr, P->gamma1, P->c_p, P->p0, P->T0, P->c_v, P->R);
  U.A = AbsorbConst{P->xlo[0],     P->xlo[1],     P->dx[0],       P->dx[1],
                    P->grid_xlo[0], P->grid_xlo[1], P->grid_xhi[0], P->grid_xhi[1],
                    P->absorb_width * P->absorb_width, P->p0, P->T0, P->rho0};
  const bool inside = absorb_dirs(U.A, nx, ny, P->bc, U.dirs);
  const bool apart = U.dirs && !inside;  // the serial walks follow in their own launches
  if (apart) U.dirs = 0;
  update_kernel<<<dim3((nx + 31) / 32, (ny + 7) / 8), 256, 0, stream()>>>(U);
  st = check_launch("patch stage");
  if (st == ENL_OK && apart)
    st = enl_absorb(b[0], b[1], b[2], b[3], g0, g1, P->xlo, P->dx, P->grid_xlo, P->grid_xhi, P->bc, P->absorb_width,
                    P->p0, P->T0, P->rho0, P->w_n, P->pressure, P->temperature);
  return st;
}

}  // extern "C"
