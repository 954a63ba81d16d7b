// The vertical implicit correction (VIC) of the hydro stage, FP64, the full
// 5x5 block-tridiagonal scheme (integration/implicit-scheme 9) on Cartesian
// blocks without solids or species.  Included by sg_stage.cu inside its
// anonymous namespace, once per storage type `real`; the solve always
// computes in FP64.
//
// Reference (paths inside the snapy project):
//   src/implicit/implicit_hydro.cpp:301-560   forward_masked
//   src/implicit/vic_assemble_impl.h:45-214   the blocks a, b, c of a cell
//   src/implicit/flux_decomposition_impl.h    Roe average, |A|, Jacobians
//   src/implicit/vic_gravity_work_impl.h      the energy row's face work
//   src/hydro/gravity_work.hpp:300-366        the corrected-PE rows K
//   src/implicit/forward_sweep_impl.h:30-131  block-Thomas forward sweep
//   src/math/ludcmp.h, src/math/lubksb.h      scaled partial-pivot LU
//   src/implicit/vic_kernels.h:100-160        back substitution, Woodbury
//   src/implicit/vic_redistribute_impl.h      constituent column, cell map
//   src/implicit/implicit_hydro.cpp:713-792   the gravity-work remainder
// Per stage, as the work's parallelism dictates: the blocks of every cell
// (vic_assemble_kernel, a thread per cell, the cells' and faces' common values
// through its CTA's shared memory), the block-Thomas sweep of each column
// (vic_solve_kernel, four columns a warp or a warp a column; sg_psolve.cuh and
// sg_rsolve.cuh hold the partitioned and the refined forms), and the column's
// redistribution, remainder and RK combine (vic_finish_kernel, a CTA per few
// columns).  In the FP64 forms but the partitioned one every product is summed
// in index order, so the results are bit for bit the CPU oracle's.
#pragma once

// Divisions of column and layer counts run in 32 bits: a block's interior
// cells take 800 bytes of scratch each, so there are fewer than 2^32 of them,
// and a 64-bit division costs a hundred instructions a thread
__device__ __forceinline__ unsigned udiv(size_t a, int b) {
  return (unsigned)a / (unsigned)b;
}

struct VicScratch {
  double *du, *du0, *A, *B, *C, *D, *Z0, *Z1;
  size_t cells;
};

__device__ __forceinline__ VicScratch vic_scratch(const BlockDev& B) {
  VicScratch s;
  const int ng = B.ng;
  const size_t nx1 = B.nc1 - 2 * ng;
  const size_t nx2 = B.nc2 > 1 ? B.nc2 - 2 * ng : 1;
  const size_t nx3 = B.nc3 > 1 ? B.nc3 - 2 * ng : 1;
  s.cells = nx1 * nx2 * nx3;
  s.du = B.vic;
  s.du0 = s.du + 5 * s.cells;
  s.A = s.du0 + 5 * s.cells;
  s.B = s.A + 25 * s.cells;
  s.C = s.B + 25 * s.cells;
  s.D = s.C + 25 * s.cells;
  s.Z0 = s.D + 5 * s.cells;
  s.Z1 = s.Z0 + 5 * s.cells;
  return s;
}

// the arrays of the refined solve (sg_rsolve.cuh) keep columns 32 at a time:
// an array of E values per cell holds, for tile t of w = min(32, ncol - 32 t)
// columns and each layer, E rows of w values (row e of column c at e w + c),
// padded to a multiple of 4, so a layer's span starts and ends on 16 bytes
struct VicTile {
  static __host__ __device__ __forceinline__ int chunk(int E, int w) {
    return (E * w + 3) & ~3;
  }
  // the first value of a tile (those before it are full)
  static __host__ __device__ __forceinline__ size_t base(int E, size_t tile, int n) {
    return tile * (size_t)n * (32 * E);
  }
  static __host__ __device__ __forceinline__ int width(size_t ncol, size_t tile) {
    const size_t left = ncol - 32 * tile;
    return left < 32 ? (int)left : 32;
  }
  // the values of the whole array
  static __host__ __device__ __forceinline__ size_t total(int E, size_t ncol, int n) {
    const size_t full = ncol / 32;
    const int rem = (int)(ncol % 32);
    return base(E, full, n) + (rem ? (size_t)n * chunk(E, rem) : 0);
  }
};

// the refined-solve part of an implicit-precision float32 block's scratch
// (after the FP64 part, 16-byte aligned), in tiles: the blocks A, B, C, the
// pivot blocks' inverses PI, C' (25 values a cell each), the residuals, then
// the sweep's y (R, 5) and the first solution X0 (5), at most 156 of the 160
// floats a cell; then, per column, each pass's largest |d| (stat, 6) and the
// direct-solve mask.  The corrections and the wall rows' third-point vectors
// (DK, at most 3 x 8 floats a cell, and E, 10 a column) take
// the FP64 part's C slots and the FP64 residual (r64, 5 doubles a cell, w to
// a row, no padding) its B slots, which a refined block uses only for the
// columns it leaves to the FP64 solve, afterwards
struct VicScratch32 {
  float *A, *B, *C, *PI, *CP, *R, *X0, *DK, *E, *stat;
  size_t dk;  // the values of one correction's array: correction k at DK + k dk
  double* r64;
  int* mask;
  size_t ncol;
};

__device__ __forceinline__ VicScratch32 vic_scratch32(const BlockDev& B,
                                                      const VicScratch& S,
                                                      int n) {
  VicScratch32 t;
  const size_t c = S.cells;
  float* f = reinterpret_cast<float*>(B.vic + (size_t)kVicDoublesPerCell * c);
  t.ncol = udiv(c, n);
  const size_t t25 = VicTile::total(25, t.ncol, n);
  const size_t t5 = VicTile::total(5, t.ncol, n);
  t.A = f;
  t.B = f + t25;
  t.C = f + 2 * t25;
  t.PI = f + 3 * t25;
  t.CP = f + 4 * t25;
  t.R = f + 5 * t25;
  t.X0 = t.R + t5;
  float* d = reinterpret_cast<float*>(S.C);
  t.DK = d;
  t.dk = t5;
  t.E = d + 3 * t5;
  t.r64 = S.B;
  t.stat = f + kVicFloatsPerCell * c;
  t.mask = reinterpret_cast<int*>(t.stat + 6 * t.ncol);
  return t;
}

// a column's FP32 block: entry k of layer i at p[i layer + k w]
struct VicCol32 {
  const float* p;
  size_t layer;
  int w;
  __device__ __forceinline__ VicCol32(const float* a, size_t ncol, size_t col, int n) {
    const size_t tile = col >> 5;
    w = VicTile::width(ncol, tile);
    layer = VicTile::chunk(25, w);
    p = a + VicTile::base(25, tile, n) + (col & 31);
  }
  __device__ __forceinline__ double operator()(int i, int k) const {
    return widen_exact(p[i * layer + (size_t)k * w]);
  }
};

// the padded (x3, x2) row of interior column `col` (x2 fastest)
__device__ __forceinline__ size_t vic_row(const BlockDev& B, size_t col) {
  const int ng = B.ng;
  if (B.nc3 == 1) return B.nc2 > 1 ? col + ng : 0;
  const int nx2 = B.nc2 > 1 ? B.nc2 - 2 * ng : 1;
  const unsigned k = udiv(col, nx2), j = (unsigned)col - k * nx2;
  return (size_t)(k + ng) * B.nc2 + (B.nc2 > 1 ? j + ng : 0);
}

// bit of the per-block status word: a column's solve failed this step
constexpr int kVicFailed = 32;

// a column left to the FP64 solve: the running count and the step's
// monitor count (implicit.fp64_columns)
__device__ __forceinline__ void count_fp64_column(const StageParams& p, int b) {
  atomicAdd(&p.fallbacks[b], 1ull);
  if (p.counts) atomicAdd(&p.counts[b * kCountSlots + kCountFp64Columns], 1ull);
}

// the flux Jacobian's entries that are not 0, 1, a velocity or gamma - 1:
// (1,0) (1,1) (1,2) (1,3) (2,0) (3,0) (4,0) .. (4,4); gq = (gm1 + 1) / gm1
constexpr int kJac = 11;
template <typename T>
__device__ __forceinline__ void vflux_jacobian(T (&J)[kJac], T gm1, T gq,
                                               const T* w) {
  T v1 = w[1], v2 = w[2], v3 = w[3], rho = w[0], pres = w[4];
  T s2 = v1 * v1 + v2 * v2 + v3 * v3;
  const T e = gq * pres / rho;
  J[0] = gm1 * s2 / 2 - v1 * v1;
  J[1] = (T(2.) - gm1) * v1;
  J[2] = -gm1 * v2;
  J[3] = -gm1 * v3;
  J[4] = -v1 * v2;
  J[5] = -v1 * v3;
  J[6] = ((gm1 - 1) * s2 / 2 - e) * v1;
  J[7] = e + s2 / 2 - gm1 * v1 * v1;
  J[8] = -gm1 * v2 * v1;
  J[9] = -gm1 * v3 * v1;
  J[10] = (gm1 + 1) * v1;
}

// |A| = R |Lambda| R^-1 at the face between wl and wr (Roe average)
template <typename T>
__device__ __forceinline__ void vabs_jacobian(T (&A)[25], T gm1, T rgm1,
                                              T rgp1, const T* wl,
                                              const T* wr) {
  // every quotient as written below; those sharing a divisor divide by
  // its reciprocal (vdiv: the same bits; rgm1 = 1 / gm1, rgp1 = 1 / (gm1 +
  // 1)), and 1 / (2 hp), -1 / hp are the reciprocals themselves
  const T gp1 = gm1 + T(1.);
  T sqrtdl = sqrt(wl[0]), sqrtdr = sqrt(wr[0]);
  T isdlpdr = T(1.0) / (sqrtdl + sqrtdr);
  T pr[5];
  pr[0] = sqrtdl * sqrtdr;
  pr[1] = (sqrtdl * wl[1] + sqrtdr * wr[1]) * isdlpdr;
  pr[2] = (sqrtdl * wl[2] + sqrtdr * wr[2]) * isdlpdr;
  pr[3] = (sqrtdl * wl[3] + sqrtdr * wr[3]) * isdlpdr;
  T el = vdiv(wl[4], gm1, rgm1) +
              T(0.5) * wl[0] * (wl[1] * wl[1] + wl[2] * wl[2] + wl[3] * wl[3]);
  T er = vdiv(wr[4], gm1, rgm1) +
              T(0.5) * wr[0] * (wr[1] * wr[1] + wr[2] * wr[2] + wr[3] * wr[3]);
  T hbar = ((el + wl[4]) / sqrtdl + (er + wr[4]) / sqrtdr) * isdlpdr;
  pr[4] = vdiv((hbar - T(0.5) * (pr[1] * pr[1] + pr[2] * pr[2] + pr[3] * pr[3])) *
                   gm1, gp1, rgp1) * pr[0];
  const T rr = T(1.) / pr[0];
  T cs = sqrt(vdiv(pr[4] * gp1, pr[0], rr));
  T r = pr[0], u = pr[1], v = pr[2], w = pr[3], p = pr[4];
  T lam[5] = {fabs(u - cs), fabs(u), fabs(u + cs), fabs(u), fabs(u)};
  T ke = T(0.5) * (u * u + v * v + w * w);
  T hp = vdiv(vdiv(gp1, gm1, rgm1) * p, r, rr);
  T h = hp + ke;
  const T d1 = T(2.) * cs * hp, d2 = T(2.) * hp;
  const T r1 = T(1.) / d1, r2 = T(1.) / d2, rh = T(1.) / hp;
  // A = (R Lambda) R^-1 with the products of R's and R^-1's zeros left out
  // (each sum's other terms in their order: R's first three columns are full,
  // its fourth holds 1 and v in the last three rows, its fifth 1 and w; the
  // last two rows of R^-1 are (-v, 0, 1, 0, 0) and (-w, 0, 0, 1, 0))
  const T Ri[3][5] = {
      {vdiv(cs * ke + u * hp, d1, r1), vdiv(-hp - cs * u, d1, r1),
       vdiv(-v, d2, r2), vdiv(-w, d2, r2), r2},
      {vdiv(hp - ke, hp, rh), vdiv(u, hp, rh), vdiv(v, hp, rh),
       vdiv(w, hp, rh), -rh},
      {vdiv(cs * ke - u * hp, d1, r1), vdiv(hp - cs * u, d1, r1),
       vdiv(-v, d2, r2), vdiv(-w, d2, r2), r2}};
  const T R[5][3] = {{lam[0], lam[1], lam[2]},
                     {(u - cs) * lam[0], u * lam[1], (u + cs) * lam[2]},
                     {v * lam[0], v * lam[1], v * lam[2]},
                     {w * lam[0], w * lam[1], w * lam[2]},
                     {(h - u * cs) * lam[0], ke * lam[1], (h + u * cs) * lam[2]}};
#pragma unroll
  for (int i = 0; i < 5; ++i)
#pragma unroll
    for (int c = 0; c < 5; ++c) {
      T s = R[i][0] * Ri[0][c];
      s += R[i][1] * Ri[1][c];
      s += R[i][2] * Ri[2][c];
      A[i * 5 + c] = s;
    }
  const T l3 = lam[3], vl = v * lam[3], wl4 = w * lam[4];
  A[10] += l3 * -v;
  A[12] += l3;
  A[15] += lam[4] * -w;
  A[18] += lam[4];
  A[20] += vl * -v;
  A[20] += wl4 * -w;
  A[22] += vl;
  A[23] += wl4;
}

// the primitives of a cell (u of the storage type -> FP64 W); an FP32
// block under gravity stores anomalies, to which the base's FP64 totals
// are added first (base null: u holds totals)
__device__ __forceinline__ void vic_prim(const real* u, size_t plane,
                                         size_t cell, double gammad,
                                         double* w, const double* base = nullptr,
                                         int nc1 = 0) {
  double uc[NHYDRO];
#pragma unroll
  for (int v = 0; v < NHYDRO; ++v) uc[v] = as_f64(u[v * plane + cell]);
  if (base) {
    const int i = (int)(cell % nc1);
    uc[IDN] = base_rho(base, nc1)[i] + uc[IDN];
    uc[IPR] = base_e(base, nc1)[i] + uc[IPR];
  }
  cons2prim<double>(uc, w, gammad);
}

// the same primitives in FP32 (FP32 assembly): the state in FP32, the base
// rounded to FP32 and added to the anomaly in FP32
__device__ __forceinline__ void vic_prim32(const real* u, size_t plane,
                                           size_t cell, float gammad,
                                           float* w, const double* base,
                                           int nc1) {
  float uc[NHYDRO];
#pragma unroll
  for (int v = 0; v < NHYDRO; ++v) uc[v] = (float)u[v * plane + cell];
  if (base) {
    const int i = (int)(cell % nc1);
    uc[IDN] = narrow_exact(base_rho(base, nc1)[i]) + uc[IDN];
    uc[IPR] = narrow_exact(base_e(base, nc1)[i]) + uc[IPR];
  }
  cons2prim<float>(uc, w, gammad);
}

// the corrected-PE slope weights of layer k of n, from the block's x1 geometry
// table, and the first of their three layers
__device__ __forceinline__ void vic_slope_tab(const BlockDev& B, int n, int k,
                                              double* wt, int* i0) {
  const double* t = B.x1tab + 6 * k;
  wt[0] = t[0];
  wt[1] = t[1];
  wt[2] = t[2];
  int kc = k < 1 ? 1 : (k > n - 2 ? n - 2 : k);
  *i0 = kc - 1;
}


// the K rows of layer k: mid, lo, hi bands and the wall third points
struct VicK {
  double mid, lo, hi, t0, t1, gv;
};

__device__ __forceinline__ VicK vic_krows(const BlockDev& B, int n, int k) {
  VicK K;
  double wt[3];
  int i0;
  vic_slope_tab(B, n, k, wt, &i0);
  double gv = B.x1tab[6 * k + 3];  // grav1 h^2 / 12
  double bm = k == 0 ? wt[0] : (k == n - 1 ? wt[2] : wt[1]);
  double bl = k == 0 ? 0. : (k == n - 1 ? wt[1] : wt[0]);
  double bh = k == n - 1 ? 0. : (k == 0 ? wt[1] : wt[2]);
  K.gv = gv;
  K.mid = gv * bm;
  K.lo = k >= 1 ? bl * gv : 0.;
  K.hi = k <= n - 2 ? bh * gv : 0.;
  K.t0 = K.t1 = 0.;
  if (k == 0) K.t0 = gv * wt[2];
  if (k == n - 1) K.t1 = gv * wt[0];
  return K;
}

// (1) the blocks of every interior cell, the K coupling in their (IPR, IDN)
// entries and du[IPR] -= K du[IDN] (its explicit row kept in du0), in the
// compute type T: double, or float under implicit-precision float32.  The FP64
// instantiation performs the reference's operations in its order.
#ifndef SG_ASM32_CTAS
#define SG_ASM32_CTAS 3
#endif
#ifndef SG_ASM64_CTAS
#define SG_ASM64_CTAS 3
#endif
// the assembly's CTA: columns side by side, threads, CTAs an SM (the register
// budget it is held to), and its shared arrays
template <typename T>
struct AsmShape {
  static constexpr bool f32 = sizeof(T) == sizeof(float);
  static constexpr int cw = f32 ? kAsmCols32 : 1;
  static constexpr int threads = f32 ? kAsmThreads32 : kAsmThreads64;
  static constexpr int ctas = f32 ? SG_ASM32_CTAS : SG_ASM64_CTAS;
};
template <typename T>
struct AsmSmem {
  T W[5][AsmShape<T>::threads], J[kJac][AsmShape<T>::threads],
      A[25][AsmShape<T>::threads];
};

// a block's constants of the assembly in the compute type (in FP64 those
// without dt come from the table, BlockDev::asmc)
template <typename T>
struct AsmConst {
  T grav, gm1, gm1r, area, vol, half_inv_vol, rvol, rdt, dtc, gq, rgm1, rgp1;
  __device__ AsmConst(const BlockDev& B, double dtc_, double rdtc) {
    grav = T(B.grav1);
    gm1 = T(B.gammad - 1.);
    gm1r = T(0.5 * (B.gammad + B.gammad) - 1.);
    area = T(B.dx3 * B.dx2);
    vol = T(B.asmc[0]);
    dtc = T(dtc_);
    if constexpr (sizeof(T) == sizeof(float)) {
      half_inv_vol = T(0.5) / vol;
      rvol = T(1.) / vol;
      rdt = T(1.) / dtc;
      gq = (gm1 + T(1.)) / gm1;
      rgm1 = T(1.) / gm1r;
      rgp1 = T(1.) / (gm1r + T(1.));
    } else {
      half_inv_vol = B.asmc[1];
      rvol = B.asmc[2];
      rdt = rdtc;
      gq = B.asmc[3];
      rgm1 = B.asmc[4];
      rgp1 = B.asmc[5];
    }
  }
};

template <typename T>
__device__ __forceinline__ void vic_assemble_cell(
    const BlockDev& B, const VicScratch& S, double dtc, double rdtc, size_t col,
    int i, bool f32copy, const AsmConst<T>& kc, const AsmSmem<T>& sm, int t,
    const double (&du0)[5]) {
  constexpr int cw = AsmShape<T>::cw;
  const int ng = B.ng, n = B.nc1 - 2 * ng;
  const T grav = kc.grav, gm1 = kc.gm1;
  const T area = kc.area, vol = kc.vol;
  const double* x1v = B.x1v + ng;
  const double* x1f = B.x1f + ng;
  const bool wood = n >= 3;
  const T half_inv_vol = kc.half_inv_vol;
  const T rvol = kc.rvol;
  const T lower = vdiv(T(0.5) * area * as_real<T>(x1v[i] - x1f[i]), vol, rvol);
  const T upper = vdiv(T(0.5) * area * as_real<T>(x1f[i + 1] - x1v[i]), vol, rvol);
  const int tl = t - cw, th = t + cw;
  const T rdt = kc.rdt, gl = grav * lower, gu = grav * upper;
  const bool partial = B.implicit == 1;
  // the K rows over dt_corr (the partial matrix adds its own below)
  T kmid = T(0.), klo = T(0.), khi = T(0.);
  const VicK K = wood ? vic_krows(B, n, i) : VicK{};
  if (wood && !partial) {
    kmid = vdiv(as_real<T>(K.mid), kc.dtc, rdt);
    klo = vdiv(as_real<T>(K.lo), kc.dtc, rdt);
    khi = vdiv(as_real<T>(K.hi), kc.dtc, rdt);
  }
  // entry k (a compile-time constant where these are called): the |A| of the
  // faces below and above, and what the flux Jacobian of the cell at x adds
  // (its zeros left out)
  auto am = [&](int k) -> T { return sm.A[k][tl]; };
  auto ap = [&](int k) -> T { return sm.A[k][t]; };
  auto jac = [&](int k, int x, T v, T sign) -> T {
    if (k == 1) return v + sign;
    if (k >= 5 && k <= 8) return v + sign * sm.J[k - 5][x];
    if (k == 9) return v + sign * gm1;
    if (k == 10) return v + sign * sm.J[4][x];
    if (k == 11) return v + sign * sm.W[2][x];
    if (k == 12 || k == 18) return v + sign * sm.W[1][x];
    if (k == 15) return v + sign * sm.J[5][x];
    if (k == 16) return v + sign * sm.W[3][x];
    if (k >= 20) return v + sign * sm.J[k - 14][x];
    return v;
  };
  // b = -(|A-| + J-) A / 2V, c = -(|A+| - J+) A / 2V, and a = (|A-| + |A+|)
  // A / 2V - Phi + 1 / dt, with the energy row's face work, the walls' mirror
  // (m1 flips) and the K rows
  auto bval = [&](int k) -> T {
    T v = -jac(k, tl, am(k), T(1.)) * area * half_inv_vol;
    if (k >= 20) v -= gl * am(k - 20);
    if (k == 21) v -= gl;
    if (k == 20) v -= klo;
    return v;
  };
  auto cval = [&](int k) -> T {
    T v = -jac(k, th, ap(k), T(-1.)) * area * half_inv_vol;
    if (k >= 20) v += gu * ap(k - 20);
    if (k == 21) v -= gu;
    if (k == 20) v -= khi;
    return v;
  };
  auto aval = [&](int k, T bw, T cw_) -> T {  // bw, cw_: b and c
    T v = (am(k) * area + ap(k) * area) * half_inv_vol;
    if (k == 5 || k == 21) v -= grav;
    if (k % 6 == 0) v += rdt;
    if (k >= 20) v -= grav * (upper * ap(k - 20) - lower * am(k - 20));
    if (k == 21) v += grav * (T(1.) - lower - upper);
    const T flip = k % 5 == 1 ? T(-1.) : T(1.);
    if (i == 0) v += bw * flip;
    if (i == n - 1) v += cw_ * flip;
    if (k == 20) v -= kmid;
    return v;
  };
  const size_t cell = col * n + i;
  // (the finish reads the explicit energy row only of a column that failed;
  // the other rows stay in du)
  S.du0[4 * S.cells + cell] = du0[4];
  double du4 = du0[4];
  // the partial matrix (implicit-scheme 1, assembled in FP64 or FP32 and
  // solved in FP64 by vic_solve3_kernel): its 3x3
  // blocks are the {rho, m1, E} rows and columns of the same entries, and
  // the m_t columns of those rows (the same terms, energy-row face work and
  // wall mirror included) fold into the density column at the cell's v_t
  // and into the right-hand side at the frozen remainder
  // q_t = du[m_t] - v_t du[rho] (src/implicit/vic_assemble_impl.h:152-214);
  // the neighbours' folds are skipped at the merged walls
  if (wood) {
    // du[IPR] -= (K du0[IDN])_i : the IDN row is read only (FP64 always)
    const double* dn = S.du + col * n;
    double s = K.mid * dn[i];
    if (i >= 1) s += K.lo * dn[i - 1];
    if (i <= n - 2) s += K.hi * dn[i + 1];
    if (i == 0) s += K.t0 * dn[2];
    if (i == n - 1) s += K.t1 * dn[n - 3];
    du4 = du0[4] - s;
    S.du[4 * S.cells + cell] = du4;
  }
  if (partial) {
    const int rows[3] = {0, 1, 4};
    T a3[9], b3[9], c3[9], rc[3] = {T(0.), T(0.), T(0.)}, aT[6], bT[6], cT[6];
#pragma unroll
    for (int r = 0; r < 3; ++r) {
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        const int k = rows[r] * 5 + rows[q];
        b3[r * 3 + q] = bval(k);
        c3[r * 3 + q] = cval(k);
        a3[r * 3 + q] = aval(k, b3[r * 3 + q], c3[r * 3 + q]);
      }
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const int e = rows[r] * 5 + 2 + k;
        bT[r * 2 + k] = bval(e);
        cT[r * 2 + k] = cval(e);
        aT[r * 2 + k] = aval(e, bT[r * 2 + k], cT[r * 2 + k]);
      }
    }
    auto fold = [&](T* blk, const T* tb, int j, int x) {
      const double* dj = S.du + col * n + j;  // row v at dj[v * cells]
      const T drho = T(dj[0]);
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const T v = sm.W[2 + k][x];
        const T qt = T(dj[(size_t)(2 + k) * S.cells]) - v * drho;
        if (v != T(0.))
#pragma unroll
          for (int r = 0; r < 3; ++r) blk[r * 3] = blk[r * 3] + tb[r * 2 + k] * v;
        if (qt != T(0.))
#pragma unroll
          for (int r = 0; r < 3; ++r) rc[r] = rc[r] + tb[r * 2 + k] * qt;
      }
    };
    fold(a3, aT, i, t);
    if (i > 0) fold(b3, bT, i - 1, tl);
    if (i < n - 1) fold(c3, cT, i + 1, th);
    if (wood) {
      a3[6] -= vdiv(as_real<T>(K.mid), kc.dtc, rdt);
      b3[6] -= vdiv(as_real<T>(K.lo), kc.dtc, rdt);
      c3[6] -= vdiv(as_real<T>(K.hi), kc.dtc, rdt);
    }
    // a cell's row of 25: the 3x3 block, row-major, then (A only) the
    // right-hand-side term of the fold
#pragma unroll
    for (int k = 0; k < 9; ++k) {
      S.A[cell * 25 + k] = (double)a3[k];
      S.B[cell * 25 + k] = (double)b3[k];
      S.C[cell * 25 + k] = (double)c3[k];
    }
#pragma unroll
    for (int r = 0; r < 3; ++r) S.A[cell * 25 + 9 + r] = (double)rc[r];
    return;
  }
  T a[25], b[25], c_[25];
#pragma unroll
  for (int k = 0; k < 25; ++k) {
    b[k] = bval(k);
    c_[k] = cval(k);
    a[k] = aval(k, b[k], c_[k]);
  }
  if (sizeof(T) == sizeof(float) && f32copy) {
    // the refined solve's tiles: the blocks in FP32 (exact: its residuals and
    // the masked columns' direct solve widen them), and the right-hand side du
    // / dt_corr in FP64 (its residuals') and in FP32 (its first sweep's)
    const VicScratch32 F = vic_scratch32(B, S, n);
    const size_t tile = col >> 5, c = col & 31;
    const int w = VicTile::width(F.ncol, tile);
    const size_t o = VicTile::base(25, tile, n) + (size_t)i * VicTile::chunk(25, w) + c;
    float *pa = F.A + o, *pb = F.B + o, *pc = F.C + o;
#pragma unroll
    for (int k = 0; k < 25; ++k) {
      pa[(size_t)k * w] = (float)a[k];
      pb[(size_t)k * w] = (float)b[k];
      pc[(size_t)k * w] = (float)c_[k];
    }
    float* pr = F.R + VicTile::base(5, tile, n) + (size_t)i * VicTile::chunk(5, w) + c;
    double* pd = F.r64 + VicTile::base(5, tile, n) + (size_t)i * 5 * w + c;
#pragma unroll
    for (int v = 0; v < 5; ++v) {
      const double q = vdiv(v == 4 ? du4 : du0[v], dtc, rdtc);
      pd[(size_t)v * w] = q;
      pr[(size_t)v * w] = narrow_exact(q);
    }
    return;
  }
#pragma unroll
  for (int k = 0; k < 25; ++k) {
    S.A[cell * 25 + k] = (double)a[k];
    S.B[cell * 25 + k] = (double)b[k];
    S.C[cell * 25 + k] = (double)c_[k];
  }
}

// The assembly, a CTA per run of padded layers of the columns taken one
// after the other (each with the ghost below it and the one above), a thread
// per padded cell: its primitives and Jacobian once, then the |A| of its upper
// face once, then the blocks of its cell from its own and its neighbours'
// values in shared memory.  A CTA's first and last layers are the next ones'
// too (they lend their values), so no column length leaves threads idle.  FP64
// runs take one column, 128 cells; FP32 runs take eight columns by 32 layers,
// so a warp's stores to the refined solve's tiles fill 32-byte sectors.
//
// Bound by the FP64 pipe in FP64 (about 700 instructions a cell; a thread
// that assembled its cell alone took 1280: three cells' primitives, two
// Jacobians, both faces' |A|, the zeros' products), by its loads and stores
// in FP32, which at three CTAs an SM spills 156 B a thread (80 registers; two
// CTAs an SM do not, and take 1.3 times as long).  Measured per launch (us),
// before and now: 512 x 128 FP64 212 / 125, 45 x 37 x 48 319 / 151, 301 x 75
// 108 / 64, nine members 330 / 210; FP32 64 members 418 / 258, four served
// requests 738 / 579.
template <typename T>
__global__ void __launch_bounds__(AsmShape<T>::threads, AsmShape<T>::ctas)
    vic_assemble_kernel(const BlockDev* __restrict__ tab, StageParams p) {
  constexpr int cw = AsmShape<T>::cw, rows = AsmShape<T>::threads / cw;
  __shared__ AsmSmem<T> sm;
  const BlockDev& B = tab[blockIdx.y];
  if (!B.implicit || (B.implicit_f32 != 0) != (sizeof(T) == sizeof(float)))
    return;
  const int nc1 = B.nc1, n = nc1 - 2 * B.ng;
  const VicScratch S = vic_scratch(B);
  const size_t ncol = udiv(S.cells, n), run = ((ncol + cw - 1) / cw) * (n + 2);
  const size_t first = (size_t)blockIdx.x * (rows - 2);
  if (first + 2 >= run) return;
  const int t = threadIdx.x, row = t / cw;
  const size_t at = first + row, g = udiv(at, n + 2);
  const int i = (int)(at - g * (n + 2)) - 1;  // -1: the ghost below, n: above
  const size_t col = g * cw + t % cw;
  const bool on = at < run && col < ncol;
  const double dtc = p.w2 * p.dt[blockIdx.y];
  const double rdtc = 1. / dtc;
  const AsmConst<T> kc(B, dtc, rdtc);
  const bool inner = on && i >= 0 && i < n && row > 0 && row < rows - 1;
  // the tendency arrives while the primitives and the |A| are formed
  double du0[5] = {0., 0., 0., 0., 0.};
  if (inner) {
#pragma unroll
    for (int v = 0; v < 5; ++v) du0[v] = S.du[v * S.cells + col * n + i];
  }
  T w[5];
  if (on) {
    const real* uin = static_cast<const real*>(B.buf[p.in]);
    const size_t plane = (size_t)nc1 * B.nc2 * B.nc3;
    const size_t cell = vic_row(B, col) * nc1 + B.ng + i;
    if constexpr (sizeof(T) == sizeof(float)) {
      // FP32 assembly: the primitives in FP32 from the FP32 state and the
      // base rounded to FP32 (the blocks are FP32 either way)
      vic_prim32(uin, plane, cell, (float)B.gammad, w, B.base, nc1);
    } else {
      vic_prim(uin, plane, cell, B.gammad, w, B.base, nc1);
    }
    T J[kJac];
    vflux_jacobian(J, kc.gm1, kc.gq, w);
#pragma unroll
    for (int k = 0; k < 5; ++k) sm.W[k][t] = w[k];
#pragma unroll
    for (int k = 0; k < kJac; ++k) sm.J[k][t] = J[k];
  }
  __syncthreads();
  if (on && i < n && row < rows - 1) {
    T A[25], wn[5];
#pragma unroll
    for (int k = 0; k < 5; ++k) wn[k] = sm.W[k][t + cw];
    vabs_jacobian(A, kc.gm1r, kc.rgm1, kc.rgp1, w, wn);
#pragma unroll
    for (int k = 0; k < 25; ++k) sm.A[k][t] = A[k];
  }
  __syncthreads();
  if (inner)
    vic_assemble_cell<T>(B, S, dtc, rdtc, col, i,
                         sizeof(T) == sizeof(float) && p.refine != 0 && B.implicit == 9,
                         kc, sm, t, du0);
}

// ---------------------------------------------------------------------------
// (2) the block-Thomas sweep, back substitution and Woodbury update.
//
// GB300 issues one FP64 warp instruction per SM every 16 cycles however many
// lanes it carries, so the solve packs kVicCols columns into each warp with
// kVicLanes lanes per column, and gives every lane work in every FP64
// instruction: lane q of a column owns right-hand-side column q of the
// layer's system  lu [a' | d' | z0' | z1'] = [c | rhs | e0 | e1]  (q < 5: the
// columns of c and a'; 5: d; 6, 7: the Woodbury vectors), and during the
// factorisation column q of the block (q < 5).
//
// The LU is the reference's scaled partial-pivot Crout factorisation
// (src/math/ludcmp.h) run column-per-lane in right-looking order: at step j
// the pivot column's lane picks the pivot, every lane swaps its own column's
// rows, and the later columns subtract L[i][j] U[j][c].  Each entry receives
// exactly the Crout subtractions, k ascending, so the factors are bit for
// bit the sequential ones; the failure screens of ludcmp (non-finite sums,
// zero rows, the pivot tolerance) are evaluated on the same values and any
// failure fails the column, as in the reference.  The back-solve is lubksb
// (src/math/lubksb.h) per lane: its row exchanges touch only rows not yet
// reduced, so they are applied first.
constexpr int kVicCols = 4;   // columns per warp (one warp per CTA)
constexpr int kVicLanes = 8;  // lanes per column

// a group-wide AND over the kVicLanes lanes of this lane's column
__device__ __forceinline__ bool vgroup_all(bool v, int g) {
  unsigned bad = __ballot_sync(0xffffffffu, !v);
  return ((bad >> (kVicLanes * g)) & 0xffu) == 0u;
}

__device__ __forceinline__ double vshfl(double v, int src) {
  return __shfl_sync(0xffffffffu, v, src, kVicLanes);
}

// non-negative finite doubles order like their bit patterns
__device__ __forceinline__ unsigned long long vbits(double x) {
  return static_cast<unsigned long long>(__double_as_longlong(x));
}

// finite, tested on the exponent bits (integer pipes, not the FP64 one)
__device__ __forceinline__ bool vfinite(double x) {
  return ((__double_as_longlong(x) >> 52) & 0x7ff) != 0x7ff;
}

__device__ __forceinline__ double div_rcp(double a, double b, double r) {
  return vdiv<double>(a, b, r);
}

template <typename T>
__device__ __forceinline__ T vpick5(int k, T a0, T a1, T a2, T a3, T a4) {
  return k == 0 ? a0 : k == 1 ? a1 : k == 2 ? a2 : k == 3 ? a3 : a4;
}

// step J of the factorisation on this lane's column x (lanes q < 5 hold the
// block's columns; vv, scale and indx are per-lane copies of the row data)
template <int J>
__device__ __forceinline__ void vlu_step(double (&x)[5], double (&vv)[5],
                                         double (&scale)[5], double (&rsc)[5],
                                         int (&indx)[5], bool& good, int q,
                                         bool colane) {
  // pivot search on column J: the last row of the largest vv |a|
  unsigned long long best = 0ull;
  int imax = J;
#pragma unroll
  for (int i2 = J; i2 < 5; ++i2) {
    double dum = vv[i2] * fabs(x[i2]);
    if (q == J) good = good && vfinite(dum);
    if (vbits(dum) >= best) {
      best = vbits(dum);
      imax = i2;
    }
  }
  imax = __shfl_sync(0xffffffffu, imax, J, kVicLanes);
  indx[J] = imax;
#pragma unroll
  for (int i2 = J + 1; i2 < 5; ++i2)
    if (imax == i2) {
      if (colane) {
        double t = x[J];
        x[J] = x[i2];
        x[i2] = t;
      }
      vv[i2] = vv[J];
      double t = scale[J];
      scale[J] = scale[i2];
      scale[i2] = t;
      t = rsc[J];
      rsc[J] = rsc[i2];
      rsc[i2] = t;
    }
  if (J < 4) {
    double dinv = 1.0 / vshfl(x[J], J);
    double l[5];
#pragma unroll
    for (int i2 = J + 1; i2 < 5; ++i2) {
      l[i2] = vshfl(x[i2], J) * dinv;
      if (q == J) x[i2] = l[i2];
    }
    if (colane && q > J) {
#pragma unroll
      for (int i2 = J + 1; i2 < 5; ++i2) x[i2] = x[i2] - l[i2] * x[J];
    }
  }
}

struct VicSolveSmem {
  double lu[kVicCols][25];         // the factorised block of each column
  double vec[kVicCols][2][15];     // back substitution: d, z0, z1 of a layer
  double rd[kVicCols][5];          // 1 / the diagonal of each factorisation
};

// The same sweep with a warp for one column (a block's wsolve), for batches
// whose columns leave sub-partitions idle: the elimination and the
// factorisation a lane per entry (lane 5 c + r: row r of column c, the
// right-hand side the sixth column), the back-solve four lanes per
// right-hand-side column (lane 4 q + h: row h + 1; row 0 rides on the lane
// of row 4 once that row is solved).  A layer is then about 130 FP64
// instructions in sequence where four columns share a warp in 210, with an
// eighth of the other instructions (a lane holds an entry, not a column), and
// its row exchanges are real branches.  Every value takes the operations of
// the four-column form in its order (each entry its subtractions k ascending,
// the same quotients), so the solution is the same bit for bit.  512 columns
// of 128 layers: 1360 us per launch with four columns a warp, 783 with one.
struct VicWarpSmem {
  double b[25], c[25], lu[25];  // the layer's b, c and factors, row-major
  double s[40];     // the previous solution: column q's row k at 5 q + k
  double dv[5], z[5], rd[5];    // rhs rows, the diagonal's reciprocals
  double v[2][15];  // back substitution: d, z0, z1 of a layer
  int perm[5];      // the factorisation's row of each row
};

__device__ __forceinline__ void vic_column_warp(const BlockDev& Bk,
                                                const VicScratch& S, size_t col,
                                                int n, double dtc,
                                                VicWarpSmem& w, int* status) {
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x;
  const int c = lane / 5, r = lane - 5 * c;
  const bool in25 = lane < 25, ind = lane >= 25 && lane < 30;
  const double rdtc = 1.0 / dtc;
  const bool wood = n >= 3;
  double* A = S.A + col * n * 25;
  const double* Bm = S.B + col * n * 25;
  const double* C = S.C + col * n * 25;
  double* D = S.D + col * n * 5;
  double* Z0 = S.Z0 + col * n * 5;
  double* Z1 = S.Z1 + col * n * 5;
  const double* du = S.du + col * n;  // row v at du[v * cells + i]
  auto from = [&](double v, int src) { return __shfl_sync(full, v, src); };

  // the input screen: du of every layer finite
  bool fin = true;
  for (int e = lane; e < 5 * n; e += 32)
    fin = fin && vfinite(du[(size_t)(e / n) * S.cells + (e % n)]);
  bool ok = __all_sync(full, fin);

  // a layer's entries arrive one layer ahead
  const int at = r * 5 + c;
  double na = 0., nb = 0., nc = 0., nd = 0.;
  auto fetch = [&](int i) {
    if (in25) {
      na = A[i * 25 + at];
      nb = Bm[i * 25 + at];
      nc = C[i * 25 + at];
    } else if (ind) {
      nd = du[(size_t)r * S.cells + i];
    }
  };
  fetch(0);
  const int q = lane >> 2, h = lane & 3, row = h + 1, g0 = lane & ~3;
  for (int i = 0; i < n && ok; ++i) {
    double x = na;
    const double bv = nb, cv = nc;
    const double dq = div_rcp(nd, dtc, rdtc);
    if (ind) x = dq;
    if (i + 1 < n) fetch(i + 1);
    if (in25) {
      w.b[at] = bv;
      w.c[at] = cv;
    }
    __syncwarp();
    // x -= b s'  (a[i] - b[i] a'[i-1] and rhs - b[i] d'[i-1]), k in order;
    // z0's five rows from the products of 25 lanes
    double z = i == 0 && lane == 4 ? 1. : 0.;
    if (i > 0) {
      if (lane < 30) {
        double t = w.b[r * 5] * w.s[c * 5];
#pragma unroll
        for (int k = 1; k < 5; ++k) t = t + w.b[r * 5 + k] * w.s[c * 5 + k];
        x = x - t;
      }
      const double pz = in25 ? bv * w.s[30 + c] : 0.;
      double t = from(pz, r);
#pragma unroll
      for (int k = 1; k < 5; ++k) t = t + from(pz, 5 * k + r);
      z = z - t;
    }

    // ---- the factorisation, the right-hand side's forward sweep with it ----
    bool good = !in25 || vfinite(x);
    unsigned long long ab = in25 ? vbits(fabs(x)) : 0ull, mx = 0ull;
#pragma unroll
    for (int k = 0; k < 5; ++k) {
      const unsigned long long o = __shfl_sync(full, ab, 5 * k + r);
      mx = o > mx ? o : mx;
    }
    double big = __longlong_as_double(static_cast<long long>(mx));
    double vv = 1.0 / big;
    good = good && mx != 0ull && vfinite(vv);
    int perm = r;
    double rd = 0.;
#pragma unroll
    for (int J = 0; J < 5; ++J) {
      const double dum = vv * fabs(x);
      if (c == J && r >= J) good = good && vfinite(dum);
      unsigned long long best = 0ull;
      int imax = J;
#pragma unroll
      for (int k = J; k < 5; ++k) {
        const unsigned long long o = __shfl_sync(full, vbits(dum), 5 * J + k);
        if (o >= best) {
          best = o;
          imax = k;
        }
      }
      if (imax != J) {  // the whole warp
        const int src = r == J ? imax : (r == imax ? J : r);
        const int sl = lane < 30 ? 5 * c + src : lane;
        x = from(x, sl);
        vv = from(vv, sl);
        big = from(big, sl);
        perm = __shfl_sync(full, perm, sl);
      }
      const double dinv = 1.0 / from(x, 6 * J);
      if (c == J && r == J) rd = dinv;
      if (J < 4) {
        if (in25 && c == J && r > J) x = x * dinv;
        const double l = from(x, 5 * J + r);
        const double u = from(x, lane < 30 ? 5 * c + J : lane);
        if (lane < 30 && c > J && r > J) x = x - l * u;
      }
    }
    if (in25) {
      good = good && vfinite(x);
      // the pivot tolerance on the final diagonal and scale
      if (c == r)
        good = good && !(div_rcp(fabs(x), big, vv) <= 8. * 5 * 2.220446049250313e-16);
    }
    ok = __all_sync(full, good);
    if (in25) {
      w.lu[at] = x;
      if (c == r) w.rd[r] = rd;
    } else if (ind) {
      w.dv[r] = x;
    }
    if (lane < 5) {
      w.z[lane] = z;
      w.perm[lane] = perm;
    }
    __syncwarp();

    // ---- lubksb: columns 0-4 of c, d (forward done), z0, z1 ----
    const int p0 = w.perm[0], pr = w.perm[row];
    double y0, y;
    if (q < 5) {
      y0 = w.c[p0 * 5 + q];
      y = w.c[pr * 5 + q];
    } else if (q == 5) {
      y0 = w.dv[0];
      y = w.dv[row];
    } else if (q == 6) {
      y0 = w.z[p0];
      y = w.z[pr];
    } else {
      y0 = i == n - 1 && p0 == 4 ? 1. : 0.;
      y = i == n - 1 && pr == 4 ? 1. : 0.;
    }
    const double* lr = w.lu + row * 5;
    if (q != 5) y = y - lr[0] * y0;
#pragma unroll
    for (int jj = 1; jj < 4; ++jj) {
      const double v = from(y, g0 + jj - 1);
      if (q != 5 && row > jj) y = y - lr[jj] * v;
    }
    const double* ur = h == 3 ? w.lu : lr;  // the products of row 0 or its own
    const double x4 = from(div_rcp(y, w.lu[24], w.rd[4]), g0 + 3);
    const double m4 = ur[4] * x4;
    const double x3 = from(div_rcp(y - m4, w.lu[18], w.rd[3]), g0 + 2);
    const double m3 = ur[3] * x3;
    const double x2 = from(div_rcp((y - m3) - m4, w.lu[12], w.rd[2]), g0 + 1);
    const double m2 = ur[2] * x2;
    const double x1 = from(div_rcp(((y - m2) - m3) - m4, w.lu[6], w.rd[1]), g0);
    const double m1 = ur[1] * x1;
    const double x0 =
        from(div_rcp((((y0 - m1) - m2) - m3) - m4, w.lu[0], w.rd[0]), g0 + 3);
    const double xs = h == 0 ? x1 : (h == 1 ? x2 : (h == 2 ? x3 : x4));
    ok = __all_sync(full, (q >= 6 && !wood) || (vfinite(xs) && vfinite(x0))) && ok;
    if (q < 5) {
      double* a = A + i * 25 + q;
      a[row * 5] = xs;
      if (h == 0) a[0] = x0;
    } else {
      double* o = (q == 5 ? D : (q == 6 ? Z0 : Z1)) + i * 5;
      o[row] = xs;
      if (h == 0) o[0] = x0;
    }
    w.s[5 * q + row] = xs;
    if (h == 0) w.s[5 * q] = x0;
    __syncwarp();
  }

  // ---- back substitution: x[i] -= a'[i] x[i+1] for d, z0, z1 ----
  if (ok) {
    const int v = lane / 5;
    const bool on = lane < 15;
    double* vec = v == 0 ? D : (v == 1 ? Z0 : Z1);
    if (on) w.v[0][lane] = w.s[25 + lane];
    double ar[5] = {0., 0., 0., 0., 0.}, cur = 0.;
    auto load = [&](int i) {
      if (!on) return;
#pragma unroll
      for (int k = 0; k < 5; ++k) ar[k] = A[i * 25 + r * 5 + k];
      cur = vec[i * 5 + r];
    };
    load(n - 2);
    __syncwarp();
    int at2 = 0;
    for (int i = n - 2; i >= 0; --i) {
      const double a0 = ar[0], a1 = ar[1], a2 = ar[2], a3 = ar[3], a4 = ar[4];
      const double now = cur;
      if (i > 0) load(i - 1);
      if (on) {
        const double* xn = w.v[at2] + v * 5;
        double t = a0 * xn[0];
        t = t + a1 * xn[1];
        t = t + a2 * xn[2];
        t = t + a3 * xn[3];
        t = t + a4 * xn[4];
        const double val = now - t;
        vec[i * 5 + r] = val;
        w.v[at2 ^ 1][lane] = val;
      }
      __syncwarp();
      at2 ^= 1;
    }
    if (wood) {
      VicK K0 = vic_krows(Bk, n, 0), K1 = vic_krows(Bk, n, n - 1);
      const double k0 = -K0.t0 / dtc, k1 = -K1.t1 / dtc;
      const int a0 = 2, a1 = n - 3;
      double m00 = 1. + k0 * Z0[a0 * 5], m01 = k0 * Z1[a0 * 5];
      double m10 = k1 * Z0[a1 * 5], m11 = 1. + k1 * Z1[a1 * 5];
      double r0 = k0 * D[a0 * 5], r1 = k1 * D[a1 * 5];
      double det = m00 * m11 - m01 * m10;
      double al0 = (m11 * r0 - m01 * r1) / det;
      double al1 = (m00 * r1 - m10 * r0) / det;
      __syncwarp();  // read before any lane updates D
      for (int e = lane; e < 5 * n; e += 32) {
        double d = D[e];
        d -= Z0[e] * al0;
        d -= Z1[e] * al1;
        D[e] = d;
        ok = ok && vfinite(d);
      }
    } else {
      for (int e = lane; e < 5 * n; e += 32) ok = ok && vfinite(D[e]);
    }
    ok = __all_sync(full, ok);
  }
  // a failed column is marked in its solution: the finish keeps du0
  if (!ok && lane == 0) {
    D[0] = __longlong_as_double(0x7ff8000000000000ll);
    atomicOr(&status[blockIdx.y], kVicFailed);
  }
}

// BLK32: the refined solve's masked columns, whose blocks are the FP32 ones
// (a separate instantiation, so the direct solve's block loads carry no
// select)
template <bool BLK32>
__global__ void __launch_bounds__(32)
    vic_solve_kernel(const BlockDev* __restrict__ tab, StageParams p,
                     int* status) {
  __shared__ union {
    VicSolveSmem four;
    VicWarpSmem one;
  } smem;
  VicSolveSmem& sm = smem.four;
  const BlockDev& Bk = tab[blockIdx.y];
  if (!Bk.implicit || Bk.implicit == 1) return;  // scheme 1: vic_solve3
  const VicScratch S = vic_scratch(Bk);
  const int n = Bk.nc1 - 2 * Bk.ng;
  const size_t ncol = udiv(S.cells, n);
  if (!BLK32 && Bk.wsolve && !Bk.psw) {
    if (blockIdx.x < ncol)
      vic_column_warp(Bk, S, blockIdx.x, n, p.w2 * p.dt[blockIdx.y], smem.one, status);
    return;
  }
  if ((size_t)blockIdx.x * kVicCols >= ncol) return;  // the whole warp
  const int lane = threadIdx.x, g = lane / kVicLanes, q = lane % kVicLanes;
  const size_t col = (size_t)blockIdx.x * kVicCols + g;
  bool valid = col < ncol;
  // an implicit-precision float32 block solves here only the columns its
  // refined solve left to FP64 (the mask); a warp with none leaves at once
  if (BLK32 && Bk.implicit_f32) {
    const VicScratch32 F = vic_scratch32(Bk, S, n);
    const int mk = valid ? F.mask[col] : 0;
    valid = valid && (mk == 1 || mk == 2);
    if (!__any_sync(0xffffffffu, valid)) return;
    // mask 2: the partitioned FP64 solve took the column first and
    // counted it
    if (valid && mk == 1 && q == 0) count_fp64_column(p, blockIdx.y);
  }
  // an FP64-assembled block with the partitioned form (vic_psolve_kernel,
  // which ran first): only the columns it marked
  if (Bk.psw && !Bk.implicit_f32) {
    const int* mask =
        reinterpret_cast<const int*>(Bk.psw + kPswDoublesPerCell * S.cells);
    valid = valid && mask[col < ncol ? col : ncol - 1] != 0;
    if (!__any_sync(0xffffffffu, valid)) return;
  }
  // a group past the last column (or unmasked) shadows a column and never
  // stores
  const size_t cc = col < ncol ? col : ncol - 1;
  const double dtc = p.w2 * p.dt[blockIdx.y];
  const double rdtc = 1.0 / dtc;  // every du / dt_corr divides by it
  const bool wood = n >= 3;
  const int m = wood ? 8 : 6;  // right-hand sides in use
  double* A = S.A + cc * n * 25;
  const double* Bm = S.B + cc * n * 25;
  const double* C = S.C + cc * n * 25;
  // the refined solve's masked columns: the blocks are the FP32 ones
  // (assembled in FP32, exact), widened; a' still goes to the FP64 A
  const bool blk32 = BLK32 && Bk.implicit_f32;
  const VicScratch32 F32 = blk32 ? vic_scratch32(Bk, S, n) : VicScratch32{};
  const VicCol32 A32(F32.A, ncol, cc, n), B32(F32.B, ncol, cc, n),
      C32(F32.C, ncol, cc, n);
  // entry k of layer i
  auto blkA = [&](int i, int k) -> double { return blk32 ? A32(i, k) : A[i * 25 + k]; };
  auto blkB = [&](int i, int k) -> double { return blk32 ? B32(i, k) : Bm[i * 25 + k]; };
  auto blkC = [&](int i, int k) -> double { return blk32 ? C32(i, k) : C[i * 25 + k]; };
  double* D = S.D + cc * n * 5;
  double* Z0 = S.Z0 + cc * n * 5;
  double* Z1 = S.Z1 + cc * n * 5;
  const double* du = S.du + cc * n;  // row v at du[v * cells + i]
  double* vout = q == 5 ? D : (q == 6 ? Z0 : Z1);
  const unsigned full = 0xffffffffu;

  // the input screen: du of every layer finite
  bool fin = true;
  for (int e = q; e < 5 * n; e += kVicLanes)
    fin = fin && vfinite(du[(size_t)(e / n) * S.cells + (e % n)]);
  // every ballot runs on all 32 lanes: evaluate before combining
  const bool fin_all = vgroup_all(fin, g);
  bool ok = valid && fin_all;

  double s[5];   // this lane's solution column of the previous layer
  double b[25];  // the b block of the layer (loaded one layer ahead)
#pragma unroll
  for (int k = 0; k < 5; ++k) s[k] = 0.;
#pragma unroll
  for (int e = 0; e < 25; ++e) b[e] = blkB(0, e);
  for (int i = 0; i < n; ++i) {
    if (!__any_sync(full, ok)) break;
    // this lane's column of a (q < 5), of c, and the right-hand sides
    double x[5], c5[5];
    if (q < 5) {
#pragma unroll
      for (int r = 0; r < 5; ++r) {
        x[r] = blkA(i, r * 5 + q);
        c5[r] = blkC(i, r * 5 + q);
      }
    } else {
#pragma unroll
      for (int r = 0; r < 5; ++r) {
        x[r] = (r == 4 && ((q == 6 && i == 0) || (q == 7 && i == n - 1))) ? 1.
                                                                         : 0.;
        c5[r] = 0.;
      }
    }
    // du / dt_corr, one row per lane, gathered on lane 5
    double dq = q < 5 ? div_rcp(du[(size_t)q * S.cells + i], dtc, rdtc) : 0.;
#pragma unroll
    for (int r = 0; r < 5; ++r) {
      double v = vshfl(dq, r);
      if (q == 5) x[r] = v;
    }
    // x -= b s'  (a[i] - b[i] a'[i-1] and rhs - b[i] d'[i-1]), k in order
    if (i > 0) {
#pragma unroll
      for (int r = 0; r < 5; ++r) {
        double t = b[r * 5] * s[0];
#pragma unroll
        for (int k = 1; k < 5; ++k) t = t + b[r * 5 + k] * s[k];
        x[r] = x[r] - t;
      }
    }
    if (i + 1 < n) {
#pragma unroll
      for (int e = 0; e < 25; ++e) b[e] = blkB(i + 1, e);
    }

    // ---- the factorisation (lanes q < 5 hold the columns) ----
    bool good = true;
    const bool colane = q < 5;
    unsigned long long mx[5];
#pragma unroll
    for (int r = 0; r < 5; ++r) {
      if (colane) good = good && vfinite(x[r]);
      mx[r] = colane ? vbits(fabs(x[r])) : 0ull;
    }
#pragma unroll
    for (int off = 4; off >= 1; off >>= 1)
#pragma unroll
      for (int r = 0; r < 5; ++r) {
        unsigned long long o = __shfl_xor_sync(full, mx[r], off, kVicLanes);
        mx[r] = o > mx[r] ? o : mx[r];
      }
    double scale[5], vv[5], rsc[5];
#pragma unroll
    for (int r = 0; r < 5; ++r) {
      scale[r] = __longlong_as_double(static_cast<long long>(mx[r]));
      good = good && mx[r] != 0ull;
    }
    {
      double big = vpick5(q < 5 ? q : 0, scale[0], scale[1], scale[2],
                          scale[3], scale[4]);
      double inv = 1.0 / big;
#pragma unroll
      for (int r = 0; r < 5; ++r) vv[r] = rsc[r] = vshfl(inv, r);
    }
#pragma unroll
    for (int r = 0; r < 5; ++r) good = good && vfinite(vv[r]);
    int indx[5];
    vlu_step<0>(x, vv, scale, rsc, indx, good, q, colane);
    vlu_step<1>(x, vv, scale, rsc, indx, good, q, colane);
    vlu_step<2>(x, vv, scale, rsc, indx, good, q, colane);
    vlu_step<3>(x, vv, scale, rsc, indx, good, q, colane);
    vlu_step<4>(x, vv, scale, rsc, indx, good, q, colane);
    if (colane) {
#pragma unroll
      for (int r = 0; r < 5; ++r) good = good && vfinite(x[r]);
      // the pivot tolerance of every step, on the final diagonal and scale
      // (|d| / scale, from the scale's reciprocal carried through the swaps)
      double dg = vpick5(q, x[0], x[1], x[2], x[3], x[4]);
      double sc = vpick5(q, scale[0], scale[1], scale[2], scale[3], scale[4]);
      double rs = vpick5(q, rsc[0], rsc[1], rsc[2], rsc[3], rsc[4]);
      good = good && !(div_rcp(fabs(dg), sc, rs) <= 8. * 5 * 2.220446049250313e-16);
      // stage the factors, and the diagonal's reciprocals, for every lane's
      // back-solve
#pragma unroll
      for (int r = 0; r < 5; ++r) sm.lu[g][r * 5 + q] = x[r];
      sm.rd[g][q] = 1.0 / dg;
    }
    const bool good_all = vgroup_all(good, g);
    ok = ok && good_all;
    __syncwarp();

    // ---- lubksb on this lane's right-hand side ----
    double sol[5];
#pragma unroll
    for (int r = 0; r < 5; ++r) sol[r] = colane ? c5[r] : x[r];
#pragma unroll
    for (int rr = 0; rr < 5; ++rr) {
      const int ip = indx[rr];
#pragma unroll
      for (int k = rr + 1; k < 5; ++k)
        if (ip == k) {
          double t = sol[k];
          sol[k] = sol[rr];
          sol[rr] = t;
        }
    }
    const double* lu = sm.lu[g];
#pragma unroll
    for (int rr = 1; rr < 5; ++rr)
#pragma unroll
      for (int jj = 0; jj < rr; ++jj) sol[rr] = sol[rr] - lu[rr * 5 + jj] * sol[jj];
#pragma unroll
    for (int rr = 4; rr >= 0; --rr) {
#pragma unroll
      for (int jj = rr + 1; jj < 5; ++jj)
        sol[rr] = sol[rr] - lu[rr * 5 + jj] * sol[jj];
      sol[rr] = div_rcp(sol[rr], lu[rr * 5 + rr], sm.rd[g][rr]);
    }
    bool f = true;
    if (q < m) {
#pragma unroll
      for (int r = 0; r < 5; ++r) f = f && vfinite(sol[r]);
    }
    const bool f_all = vgroup_all(f, g);
    ok = ok && f_all;
    if (valid) {
      if (colane) {
#pragma unroll
        for (int r = 0; r < 5; ++r) A[i * 25 + r * 5 + q] = sol[r];
      } else if (q < m) {
#pragma unroll
        for (int r = 0; r < 5; ++r) vout[i * 5 + r] = sol[r];
      }
    }
#pragma unroll
    for (int r = 0; r < 5; ++r) s[r] = sol[r];
    __syncwarp();
  }

  // ---- back substitution: x[i] -= a'[i] x[i+1] for d, z0, z1 ----
  // lane q handles the (vector, row) pairs q and q + 8 of the 15
  if (__any_sync(full, ok)) {
    if (q >= 5) {
#pragma unroll
      for (int r = 0; r < 5; ++r) sm.vec[g][0][(q - 5) * 5 + r] = s[r];
    }
    __syncwarp();
    int cur = 0;
    for (int i = n - 2; i >= 0; --i) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int pr = q + kVicLanes * h;
        if (pr < 15) {
          const int v = pr / 5, r = pr % 5;
          const double* xn = sm.vec[g][cur] + v * 5;
          const double* ar = A + i * 25 + r * 5;
          double t = ar[0] * xn[0];
#pragma unroll
          for (int k = 1; k < 5; ++k) t = t + ar[k] * xn[k];
          double* vec = v == 0 ? D : (v == 1 ? Z0 : Z1);
          double val = vec[i * 5 + r] - t;
          if (ok) vec[i * 5 + r] = val;
          sm.vec[g][cur ^ 1][pr] = val;
        }
      }
      __syncwarp();
      cur ^= 1;
    }
    if (wood && ok) {
      VicK K0 = vic_krows(Bk, n, 0), K1 = vic_krows(Bk, n, n - 1);
      double k0 = -K0.t0 / dtc, k1 = -K1.t1 / dtc;
      k0 = k0 * 1.;
      k1 = k1 * 1.;
      const int a0 = 2, a1 = n - 3;
      double m00 = 1. + k0 * Z0[a0 * 5], m01 = k0 * Z1[a0 * 5];
      double m10 = k1 * Z0[a1 * 5], m11 = 1. + k1 * Z1[a1 * 5];
      double r0 = k0 * D[a0 * 5], r1 = k1 * D[a1 * 5];
      double det = m00 * m11 - m01 * m10;
      double al0 = (m11 * r0 - m01 * r1) / det;
      double al1 = (m00 * r1 - m10 * r0) / det;
      // this column's lanes (ok and wood are uniform over them) finish
      // reading D and Z before any of them updates D
      __syncwarp(0xffu << (kVicLanes * g));
      for (int e = q; e < 5 * n; e += kVicLanes) {
        double d = D[e];
        d -= Z0[e] * al0;
        d -= Z1[e] * al1;
        D[e] = d;
      }
    }
    __syncwarp();
    bool f = true;
    if (ok)
      for (int e = q; e < 5 * n; e += kVicLanes) f = f && vfinite(D[e]);
    const bool d_all = vgroup_all(f, g);
    ok = ok && d_all;
  }
  // a failed column is marked in its solution: the finish keeps du0
  if (valid && !ok && q == 0) {
    D[0] = __longlong_as_double(0x7ff8000000000000ll);
    atomicOr(&status[blockIdx.y], kVicFailed);
  }
}

// ---------------------------------------------------------------------------
// (2p) the partial matrix (implicit-scheme 1): the 3x3 block-Thomas sweep of
// ForwardSweep with N = 3 (src/implicit/forward_sweep_impl.h:30-131), one
// thread per column: the right-hand side less the assembly's fold term, the
// block screened by ludcmp<3> and inverted explicitly (adjugate over the
// determinant), d = inv (rhs - b d_prev), a' = inv c, the two Woodbury unit
// vectors of the energy row, then vic_backward_substitute (each vector only
// if its first layer is finite) and the Woodbury update on the 3-vectors.
// The solution leaves in D rows 0, 1 and 4 (the tangential rows keep the
// explicit du; the finish moves them with the face mass).  Its chain is
// short (about 200 FP64 operations per layer), so a thread per column keeps
// every lane of an FP64 instruction on its own column.
__device__ __forceinline__ bool vic_ludcmp3_ok(const double* m) {
  double a[9];
#pragma unroll
  for (int k = 0; k < 9; ++k) {
    a[k] = m[k];
    if (!vfinite(a[k])) return false;
  }
  double vv[3], scale[3];
  const double tol = 8. * 3 * 2.220446049250313e-16;
  for (int i = 0; i < 3; ++i) {
    double big = 0.;
    for (int j = 0; j < 3; ++j) {
      const double t = fabs(a[i * 3 + j]);
      if (t > big) big = t;
    }
    if (big == 0.) return false;
    scale[i] = big;
    vv[i] = 1.0 / big;
    if (!vfinite(vv[i])) return false;
  }
  for (int j = 0; j < 3; ++j) {
    for (int i = 0; i < j; ++i) {
      double sum = a[i * 3 + j];
      for (int k = 0; k < i; ++k) sum -= a[i * 3 + k] * a[k * 3 + j];
      if (!vfinite(sum)) return false;
      a[i * 3 + j] = sum;
    }
    double big = 0.;
    int imax = 0;
    for (int i = j; i < 3; ++i) {
      double sum = a[i * 3 + j];
      for (int k = 0; k < j; ++k) sum -= a[i * 3 + k] * a[k * 3 + j];
      if (!vfinite(sum)) return false;
      a[i * 3 + j] = sum;
      const double dum = vv[i] * fabs(sum);
      if (!vfinite(dum)) return false;
      if (dum >= big) {
        big = dum;
        imax = i;
      }
    }
    if (j != imax) {
      for (int k = 0; k < 3; ++k) {
        const double t = a[imax * 3 + k];
        a[imax * 3 + k] = a[j * 3 + k];
        a[j * 3 + k] = t;
      }
      vv[imax] = vv[j];
      const double t = scale[imax];
      scale[imax] = scale[j];
      scale[j] = t;
    }
    if (fabs(a[j * 3 + j]) / scale[j] <= tol) return false;
    if (j != 2) {
      const double dum = 1.0 / a[j * 3 + j];
      for (int i = j + 1; i < 3; ++i) a[i * 3 + j] *= dum;
    }
  }
#pragma unroll
  for (int k = 0; k < 9; ++k)
    if (!vfinite(a[k])) return false;
  return true;
}

__device__ __forceinline__ void vmat3_mul(double* out, const double* a,
                                          const double* b) {
#pragma unroll
  for (int r = 0; r < 3; ++r)
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      double s = a[r * 3] * b[c];
      s += a[r * 3 + 1] * b[3 + c];
      s += a[r * 3 + 2] * b[6 + c];
      out[r * 3 + c] = s;
    }
}

__device__ __forceinline__ void vmat3_vec(double* out, const double* a,
                                          const double* v) {
#pragma unroll
  for (int r = 0; r < 3; ++r) {
    double s = a[r * 3] * v[0];
    s += a[r * 3 + 1] * v[1];
    s += a[r * 3 + 2] * v[2];
    out[r] = s;
  }
}

__global__ void __launch_bounds__(kThreads)
    vic_solve3_kernel(const BlockDev* __restrict__ tab, StageParams p,
                      int* status) {
  const BlockDev& Bk = tab[blockIdx.y];
  if (Bk.implicit != 1) return;
  const VicScratch S = vic_scratch(Bk);
  const int n = Bk.nc1 - 2 * Bk.ng;
  const size_t ncol = udiv(S.cells, n);
  const size_t col = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (col >= ncol) return;
  const double dtc = p.w2 * p.dt[blockIdx.y];
  const double rdtc = 1. / dtc;  // du / dt_corr divides by it (vdiv)
  const bool wood = n >= 3;
  double* A = S.A + col * n * 25;
  const double* Bm = S.B + col * n * 25;
  const double* C = S.C + col * n * 25;
  double* D = S.D + col * n * 5;
  double* Z0 = S.Z0 + col * n * 5;
  double* Z1 = S.Z1 + col * n * 5;
  const double* du = S.du + col * n;  // row v at du[v * cells + i]
  const size_t cs = S.cells;
  bool ok = true;
  for (int e = 0; e < 5 * n; ++e)
    ok = ok && vfinite(du[(size_t)(e / n) * cs + (e % n)]);
  double ap[9], dp[3], y0[3] = {0., 0., 0.}, y1[3] = {0., 0., 0.};
  for (int i = 0; i < n && ok; ++i) {
    double m[9], bb[9], cc[9], rc[3];
#pragma unroll
    for (int k = 0; k < 9; ++k) {
      m[k] = A[i * 25 + k];
      bb[k] = Bm[i * 25 + k];
      cc[k] = C[i * 25 + k];
    }
#pragma unroll
    for (int r = 0; r < 3; ++r) rc[r] = A[i * 25 + 9 + r];
    double rhs[3] = {vdiv(du[i], dtc, rdtc), vdiv(du[cs + i], dtc, rdtc),
                     vdiv(du[4 * cs + i], dtc, rdtc)};
#pragma unroll
    for (int r = 0; r < 3; ++r)
      if (rc[r] != 0.) rhs[r] -= rc[r];
    if (i > 0) {
      double t[9];
      vmat3_mul(t, bb, ap);
#pragma unroll
      for (int k = 0; k < 9; ++k) m[k] -= t[k];
    }
    if (!vic_ludcmp3_ok(m)) {
      ok = false;
      break;
    }
    // the adjugate over the determinant, expanded along column 0
    const double c00 = m[4] * m[8] - m[5] * m[7];
    const double c10 = m[2] * m[7] - m[1] * m[8];
    const double c20 = m[1] * m[5] - m[2] * m[4];
    const double det = m[0] * c00 + m[3] * c10 + m[6] * c20;
    const double rd = 1. / det;
    const double inv[9] = {c00 * rd,
                           c10 * rd,
                           c20 * rd,
                           (m[5] * m[6] - m[3] * m[8]) * rd,
                           (m[0] * m[8] - m[2] * m[6]) * rd,
                           (m[2] * m[3] - m[0] * m[5]) * rd,
                           (m[3] * m[7] - m[4] * m[6]) * rd,
                           (m[1] * m[6] - m[0] * m[7]) * rd,
                           (m[0] * m[4] - m[1] * m[3]) * rd};
    double t[3], u[3];
    if (i > 0) {
      vmat3_vec(u, bb, dp);
#pragma unroll
      for (int r = 0; r < 3; ++r) t[r] = rhs[r] - u[r];
    } else {
#pragma unroll
      for (int r = 0; r < 3; ++r) t[r] = rhs[r];
    }
    vmat3_vec(dp, inv, t);
    if (wood) {
      if (i > 0) {
        vmat3_vec(u, bb, y0);
#pragma unroll
        for (int r = 0; r < 3; ++r) t[r] = (r == 2 && i == 0 ? 1. : 0.) - u[r];
      } else {
        t[0] = 0.;
        t[1] = 0.;
        t[2] = 1.;
      }
      vmat3_vec(y0, inv, t);
      if (i > 0) {
        vmat3_vec(u, bb, y1);
#pragma unroll
        for (int r = 0; r < 3; ++r) t[r] = (r == 2 && i == n - 1 ? 1. : 0.) - u[r];
      } else {
        t[0] = 0.;
        t[1] = 0.;
        t[2] = i == n - 1 ? 1. : 0.;
      }
      vmat3_vec(y1, inv, t);
    }
    vmat3_mul(ap, inv, cc);
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      ok = ok && vfinite(dp[r]);
#pragma unroll
      for (int q = 0; q < 3; ++q) ok = ok && vfinite(ap[r * 3 + q]);
    }
#pragma unroll
    for (int k = 0; k < 9; ++k) A[i * 25 + k] = ap[k];
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      D[i * 5 + r] = dp[r];
      Z0[i * 5 + r] = y0[r];
      Z1[i * 5 + r] = y1[r];
    }
  }
  if (ok) {
    bool f0 = wood, f1 = wood;
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      f0 = f0 && vfinite(Z0[r]);
      f1 = f1 && vfinite(Z1[r]);
    }
    for (int i = n - 2; i >= 0; --i) {
      double a[9], t[3];
#pragma unroll
      for (int k = 0; k < 9; ++k) a[k] = A[i * 25 + k];
      vmat3_vec(t, a, dp);
#pragma unroll
      for (int r = 0; r < 3; ++r) {
        dp[r] = D[i * 5 + r] - t[r];
        D[i * 5 + r] = dp[r];
      }
      if (f0) {
        vmat3_vec(t, a, y0);
#pragma unroll
        for (int r = 0; r < 3; ++r) {
          y0[r] = Z0[i * 5 + r] - t[r];
          Z0[i * 5 + r] = y0[r];
        }
      }
      if (f1) {
        vmat3_vec(t, a, y1);
#pragma unroll
        for (int r = 0; r < 3; ++r) {
          y1[r] = Z1[i * 5 + r] - t[r];
          Z1[i * 5 + r] = y1[r];
        }
      }
    }
    double al0 = 0., al1 = 0.;
    if (wood) {
      VicK K0 = vic_krows(Bk, n, 0), K1 = vic_krows(Bk, n, n - 1);
      double k0 = -K0.t0 / dtc, k1 = -K1.t1 / dtc;
      k0 = k0 * 1.;
      k1 = k1 * 1.;
      const int a0 = 2, a1 = n - 3;
      double m00 = 1. + k0 * Z0[a0 * 5], m01 = k0 * Z1[a0 * 5];
      double m10 = k1 * Z0[a1 * 5], m11 = 1. + k1 * Z1[a1 * 5];
      double r0 = k0 * D[a0 * 5], r1 = k1 * D[a1 * 5];
      double det = m00 * m11 - m01 * m10;
      al0 = (m11 * r0 - m01 * r1) / det;
      al1 = (m00 * r1 - m10 * r0) / det;
    }
    for (int i = 0; i < n; ++i) {
      double d[3];
#pragma unroll
      for (int r = 0; r < 3; ++r) {
        d[r] = D[i * 5 + r];
        if (wood) {
          d[r] -= Z0[i * 5 + r] * al0;
          d[r] -= Z1[i * 5 + r] * al1;
        }
        ok = ok && vfinite(d[r]);
      }
      D[i * 5] = d[0];
      D[i * 5 + 1] = d[1];
      D[i * 5 + 2] = 0.;
      D[i * 5 + 3] = 0.;
      D[i * 5 + 4] = d[2];
    }
  }
  // a failed column is marked in its solution: the finish keeps du0
  if (!ok) {
    D[0] = __longlong_as_double(0x7ff8000000000000ll);
    atomicOr(&status[blockIdx.y], kVicFailed);
  }
}

// (3) redistribution, the gravity-work remainder and the RK combine, a CTA
// per fin_cols columns with the columns' work in shared memory.  What a cell
// needs of its own runs a thread per cell; the constituent column's serial
// passes (the sums R and S, the face-mass prefix M with the availability
// clamp) run a lane per column and keep only their chain: three additions
// and two comparisons a layer, the comparisons on the bit patterns, so the
// FP64 pipe (a warp instruction per 64 cycles) sees the additions alone.
//
// Bound by the FP64 pipe: about 55 instructions a cell, and 4 a layer for
// the passes of a CTA's columns.  Measured per launch (us), before (a warp
// per column, its passes on lane 0; wide batches three launches, a thread per
// column for the passes) and now: 512 columns of 128 FP64 138 and 45, 301 of
// 75 85 and 25, 384 of 100 FP32 106 and 35, 4,096 of 64 113 and 65, nine FP64
// members 153 and 58, 64 members 477 and 286, four served requests 829 and
// 612.
constexpr int kFinThreads = 256;

// a > b and a < 0 from the bit patterns: the order of the doubles, without
// the FP64 pipe (no NaN comes here: a column with one has failed)
__device__ __forceinline__ bool dgt(double a, double b) {
  long long x = __double_as_longlong(a), y = __double_as_longlong(b);
  x ^= (x >> 63) & 0x7fffffffffffffffll;
  y ^= (y >> 63) & 0x7fffffffffffffffll;
  return x > y;
}
__device__ __forceinline__ bool dneg(double a) {
  const long long x = __double_as_longlong(a);
  return x < 0 && (x << 1) != 0;
}

__global__ void __launch_bounds__(kFinThreads, 4)
    vic_finish_kernel(const BlockDev* __restrict__ tab, StageParams p) {
  extern __shared__ __align__(16) unsigned char fin_smem[];
  __shared__ double sR[32], sS[32], sRS[32];
  __shared__ int sok[32];
  const BlockDev& B = tab[blockIdx.y];
  if (!B.implicit) return;
  const VicScratch S = vic_scratch(B);
  const int ng = B.ng, nc1 = B.nc1, n = nc1 - 2 * ng;
  const int cols = fin_cols(n, p.fin_len);
  const size_t ncol = udiv(S.cells, n), col0 = (size_t)blockIdx.x * cols;
  if (col0 >= ncol) return;
  const int nc = ncol - col0 < (size_t)cols ? (int)(ncol - col0) : cols;
  const int tid = threadIdx.x, lane = tid & 31, wq = tid >> 5;
  const size_t plane = (size_t)nc1 * B.nc2 * B.nc3;
  const real* uin = static_cast<const real*>(B.buf[p.in]);
  const real* u0 = static_cast<const real*>(B.buf[p.u0]);
  real* uout = static_cast<real*>(B.buf[p.out]);
  const double vol = B.dx3 * (B.dx2 * B.dx1);
  const double rvol = 1. / vol;  // the quotients by vol divide by it (vdiv)
  const size_t cs = S.cells;
  const bool wood = n >= 3;
  const bool partial = B.implicit == 1;
  const int pitch = fin_pitch(n);
  const int len = p.fin_len;
  double* aM = reinterpret_cast<double*>(fin_smem);  // phi, X, then M
  double* aR = aM + len;  // the density, the available mass, the IDN row
  double* aQ = aR + len;  // rho V, then the moved mass q
  double* aV = aQ + len;  // q / V
  double* aW = aV + len;  // D_rho - du_rho
  double* aT2 = aW + len;  // partial: the tangential velocities, 0 .. n
  double* aT3 = aT2 + len;
  if (tid < nc) sok[tid] = vfinite(S.D[(col0 + tid) * n * 5]);
  __syncthreads();

  // per cell: the density, phi = (D_rho - du_rho) V
  const int cells = nc * n;
  for (int e = tid; e < cells; e += kFinThreads) {
    const int c = e / n, i = e - c * n;
    if (!sok[c]) continue;
    const size_t col = col0 + c, g = col * n + i;
    const size_t base = vic_row(B, col) * nc1 + ng;
    const int o = c * pitch + i;
    double w[5];
    vic_prim(uin, plane, base + i, B.gammad, w, B.base, nc1);
    aR[o] = w[0];
    aQ[o] = w[0] * vol;
    const double rest = S.D[g * 5] - S.du[g];
    aM[o] = rest * vol;
    aW[o] = rest;
    if (partial) {
      aT2[o] = w[2];
      aT3[o] = w[3];
      if (i == n - 1) {  // the ghost above, the donor of the top face
        vic_prim(uin, plane, base + n, B.gammad, w, B.base, nc1);
        aT2[o + 1] = w[2];
        aT3[o + 1] = w[3];
      }
    }
  }
  __syncthreads();
  // per column: R = sum phi on one warp, S = sum rho V on another
  if (wq < 2 && lane < nc && sok[lane]) {
    const double* a = (wq ? aQ : aM) + lane * pitch;
    double s = 0;
#pragma unroll 4
    for (int i = 0; i < n; ++i) s += a[i];
    if (wq) {
      sS[lane] = s;
      sRS[lane] = 1. / s;
    } else {
      sR[lane] = s;
    }
  }
  __syncthreads();
  // per cell: what M loses over the layer, and the mass it can give
  for (int e = tid; e < cells; e += kFinThreads) {
    const int c = e / n, i = e - c * n;
    if (!sok[c]) continue;
    const int o = c * pitch + i;
    aM[o] = aM[o] - sR[c] * vdiv(aQ[o], sS[c], sRS[c]);
    double avail = (aR[o] * 1. + S.du[(col0 + c) * n + i]) * vol;
    if (dneg(avail)) avail = 0;
    aR[o] = avail;
  }
  __syncthreads();
  // per column: the face-mass prefix and the availability clamp
  if (wq == 0 && lane < nc && sok[lane]) {
    double* m = aM + lane * pitch;
    double* q = aQ + lane * pitch;
    const double* av = aR + lane * pitch;
    double M = 0, avail = av[0];
    q[0] = 0.;
#pragma unroll 4
    for (int i = 0; i + 1 < n; ++i) {
      const double x = m[i], up = av[i + 1];
      m[i] = M;
      M -= x;
      double f = M;
      if (dgt(f, avail)) f = avail;
      if (dgt(-up, f)) f = -up;
      q[i + 1] = f;
      avail = up + f;
    }
    m[n - 1] = M;
    m[n] = 0.;
    q[n] = 0.;
  }
  __syncthreads();
  // per face: q / V
  for (int e = tid; e < cells; e += kFinThreads) {
    const int c = e / n, i = e - c * n, o = c * pitch + i;
    if (sok[c]) aV[o] = vdiv(aQ[o], vol, rvol);
  }
  __syncthreads();
  // per cell: the IDN row with its dry increment (the faces in order, the
  // lower one's first)
  for (int e = tid; e < cells; e += kFinThreads) {
    const int c = e / n, i = e - c * n, o = c * pitch + i;
    if (!sok[c]) continue;
    double dn = i > 0 ? 0. + aV[o] : 0.;
    if (i + 1 < n) dn = dn - aV[o + 1];
    aR[o] = S.du[(col0 + c) * n + i] + dn;
  }
  __syncthreads();

  // passive scalars: the clamped dry transfer of each x1 face (zero for a
  // failed column), for their share of it
  if (B.nscalar > 0)
    for (int e = tid; e < nc * (n + 1); e += kFinThreads) {
      const int c = e / (n + 1), f = e - c * (n + 1);
      B.vicq[vic_row(B, col0 + c) * nc1 + ng + f] = sok[c] ? aQ[c * pitch + f] : 0.;
    }
  // the x1 step field of an implicit block (FluxRegister::end_stage after
  // ImplicitHydroImpl::post_, src/implicit/implicit_hydro.cpp:625-673): the
  // stage's T_1 plus the solve's face transfers per unit area and time,
  // "vic.mass_dry" q / (dt A) on row IDN and "vic.momentum_t"
  // -sum_{k < f} (du - du0)_k V / (dt A) on rows IVY and IVZ (the prefix from
  // the bottom wall, top face included; the partial matrix posts the donor
  // transfer q w_t of each face, :520-530,662-666), then the prescribed wall
  // faces.  A failed column posts nothing.  Each face's adds run in the
  // reference's order, +0 posts included (a -0 total becomes +0)
  if (double* S1 = B.step[0]) {
    const double dt = p.dt[blockIdx.y];
    const double kdt = dt * (B.dx3 * B.dx2), rkdt = 1. / kdt;
    const double w1s = p.w1, w2dt = p.w2 * dt;
    const bool first = p.first != 0;
    const int nf = n + 1;
    const double* T = B.t1;
    const bool wlo = B.bc[0] == kBcReflecting, whi = B.bc[1] == kBcReflecting;
    auto tot = [&](size_t col, int v, int f) {
      return T[((size_t)v * ncol + col) * nf + f];
    };
    auto at = [&](size_t col, int v, int f) {
      return S1 + v * plane + vic_row(B, col) * nc1 + ng + f;
    };
    for (int e = tid; e < nc * nf; e += kFinThreads) {
      const int c = e / nf, f = e - c * nf;
      const size_t col = col0 + c;
      double t0 = tot(col, IDN, f), t1 = tot(col, IVX, f), t4 = tot(col, IPR, f);
      if (sok[c]) t0 = t0 + vdiv(aQ[c * pitch + f], kdt, rkdt);
      if ((f == 0 && wlo) || (f == n && whi)) t0 = t4 = 0.;
      step_set(at(col, IDN, f), t0, w1s, w2dt, first);
      step_set(at(col, IVX, f), t1, w1s, w2dt, first);
      step_set(at(col, IPR, f), t4, w1s, w2dt, first);
    }
    if (tid < nc) {
      const size_t col = col0 + tid;
      const bool ok = sok[tid] != 0;
      const double *D = S.D + col * n * 5, *du = S.du + col * n;
      const int o = tid * pitch;
      double sy = 0., sz = 0.;
      for (int f = 0; f < nf; ++f) {
        double ty = tot(col, IVY, f), tz = tot(col, IVZ, f);
        if (ok && partial) {
          const double q = aQ[o + f];
          const int donor = q > 0. ? f - 1 : f;
          ty = ty + vdiv(q * aT2[o + donor], kdt, rkdt);
          tz = tz + vdiv(q * aT3[o + donor], kdt, rkdt);
        } else if (ok) {
          double py = 0., pz = 0.;
          if (f > 0) {
            sy = sy + (D[(f - 1) * 5 + 2] - du[2 * cs + f - 1]) * vol;
            sz = sz + (D[(f - 1) * 5 + 3] - du[3 * cs + f - 1]) * vol;
            py = -sy;
            pz = -sz;
          }
          ty = ty + vdiv(py, kdt, rkdt);
          tz = tz + vdiv(pz, kdt, rkdt);
        }
        step_set(at(col, IVY, f), ty, w1s, w2dt, first);
        step_set(at(col, IVZ, f), tz, w1s, w2dt, first);
      }
    }
  }

  // per cell: the map of the solution, the partial matrix's tangential
  // transfers, the gravity-work remainder and the RK combine (a failed
  // column keeps the explicit du)
  const real w0 = real(p.w0), w1 = real(p.w1), w2 = real(p.w2);
  for (int e = tid; e < cells; e += kFinThreads) {
    const int c = e / n, i = e - c * n, o = c * pitch + i;
    const size_t col = col0 + c, g = col * n + i;
    const double* du = S.du + g;
    double d[5];
    if (sok[c]) {
      const double* D = S.D + g * 5;
      d[0] = aR[o];
      d[1] = D[1];
      if (!partial) {
        d[2] = D[2];
        d[3] = D[3];
      } else {
        // vic_tangential_momentum_column (src/implicit/
        // vic_redistribute_impl.h:178-200): each face's moved total mass
        // carries the donor (upwind) cell's tangential velocity, the face
        // below first; a zero transfer leaves du as it is
        const double* vt[2] = {aT2 + o, aT3 + o};
#pragma unroll
        for (int t = 0; t < 2; ++t) {
          double a = S.du[(2 + t) * cs + g];
          if (i > 0) {
            const double q = aQ[o];
            const double pm = q * vt[t][q > 0 ? -1 : 0];
            if (pm != 0) a += vdiv(pm, vol, rvol);
          }
          if (i + 1 < n) {
            const double q = aQ[o + 1];
            const double pm = q * vt[t][q > 0 ? 0 : 1];
            if (pm != 0) a -= vdiv(pm, vol, rvol);
          }
          d[2 + t] = a;
        }
      }
      const double* gt = B.x1tab + 6 * i;  // [4], [5]: g dz above, below
      const double projected = vdiv(aM[o] - aM[o + 1], vol, rvol);
      const double ph = -B.grav1 * B.x1v[ng + i];
      const double pw = ph * (aW[o] - projected);
      const double mv_lo = aQ[o] - aM[o], mv_hi = aQ[o + 1] - aM[o + 1];
      const double cw = vdiv(-(-gt[4] * mv_hi - -gt[5] * mv_lo), vol, rvol);
      double e4 = D[4] + (pw + cw);
      if (wood) {
        // the remainder g1 sigma^2 s[du - du0] - K (raw - du0)
        double wt[3];
        int i0;
        vic_slope_tab(B, n, i, wt, &i0);
        const VicK K = vic_krows(B, n, i);
        const int s0 = i0 - i;
        double sl = wt[0] * (aR[o + s0] - du[s0]);
        sl += wt[1] * (aR[o + s0 + 1] - du[s0 + 1]);
        sl += wt[2] * (aR[o + s0 + 2] - du[s0 + 2]);
        double wk = K.gv * sl;
        double s = K.mid * aW[o];
        if (i >= 1) s += K.lo * aW[o - 1];
        if (i <= n - 2) s += K.hi * aW[o + 1];
        if (i == 0) s += K.t0 * aW[o + 2];
        if (i == n - 1) s += K.t1 * aW[o - 2];
        wk -= s;
        e4 += wk;
      }
      d[4] = e4;
    } else {
#pragma unroll
      for (int v = 0; v < 4; ++v) d[v] = du[v * cs];
      d[4] = S.du0[4 * cs + g];
    }
    const size_t cell = vic_row(B, col) * nc1 + ng + i;
#pragma unroll
    for (int v = 0; v < NHYDRO; ++v) {
      const size_t q = v * plane + cell;
      uout[q] = w0 * u0[q] + w1 * uin[q] + w2 * as_real<real>(d[v]);
    }
  }
}
