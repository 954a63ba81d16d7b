// The refined solve of implicit-precision float32 blocks of implicit-scheme
// 9.  Included by sg_stage.cu after sg_vic.cuh, inside its anonymous
// namespace.
//
// The system of a column is T x = b, T the block-tridiagonal matrix of the
// FP32-assembled 5x5 blocks (B_i, A_i, C_i) plus the two third-point entries
// of the corrected-PE wall rows (layer 0's energy row reads the density of
// layer 2, layer n - 1's that of layer n - 3), and b = du / dt_corr.  It is
// solved by mixed-precision iterative refinement (the scheme of LAPACK's
// dsgesv): an FP32 solve M^-1, then p.refine corrections d = M^-1 r with
// r = b - T x formed beyond FP64 accuracy and x summed in FP64.
//
//   vic_factor32_kernel    M^-1's factors and the first solution
//   vic_residual_kernel    r = b - T x (or the previous r less T d)
//   vic_correct32_kernel   d = M^-1 r
//   vic_accept_kernel      the sum of the passes into D, the acceptance
//
// M^-1 is the FP32 block-Thomas sweep with the Woodbury step of the two wall
// entries, so T's own wall entries are refined with the rest and only one
// right-hand side needs corrections (the two Woodbury vectors stay FP32, as
// part of M^-1).  The pivot blocks are inverted in place without pivoting:
// the blocks are 1/dt_corr plus the |A| of both faces, and the elimination
// order changes the rounding of M^-1 alone, never the solution (one
// correction gains 2e-7 either way, measured on Straka and convection
// columns, at rest and moving).  A pivot that cancels to below 40 eps of its
// diagonal, a value that is not finite, or an estimated error above 2^-44 of
// the solution after the last correction masks the column, and it takes the
// FP64 solve (vic_psolve_kernel, vic_solve_kernel), as the reference retries
// a failed FP32 column in FP64 (src/hydro/hydro.cpp:436-466).
//
// Layout.  Columns are taken 32 at a time: an array of E values per cell
// keeps, for each tile of w <= 32 columns and each layer, E rows of w
// values, padded to 16 bytes (VicTile).  A warp owns a tile in the sweeps, a
// lane a column: every load, copy and store of a layer is one contiguous
// span, and the 5x5 algebra has no shuffles, no pivot search and no
// synchronisation between lanes.  A layer's span arrives in a ring in shared
// memory by 16-byte asynchronous copies a few layers ahead of the sweep.
//
// What bounds it: the bytes a cell moves (about 0.8 KB in the factor sweep,
// 0.4 KB in a residual, 0.5 KB in a correction), and, with few columns, the
// chain of a column's layers.  The form before it (eight lanes a column,
// pivoted LU factors kept per layer, three right-hand sides corrected, a
// cell's blocks in a padded row of its own) used a part of each 32-byte
// sector it read and was bound by its chains and those loads.  The 64-member
// ensemble (21,120 columns, 1.44 M cells), per launch, before and after: the
// first sweep 815 and 286 us, a residual 634 and 225, a correction 613 and
// 130, the acceptance 95 (in the correction before), the columns left to FP64
// 278 and 36 (7 of 21,120 and none); a step 14.95 and 7.57 ms.  Convection
// 64^3 (4,096 columns): a step 3.59 and 2.02 ms.
#pragma once

constexpr int kFacRing = 4;  // layers in the factor's forward ring
constexpr int kFacSlot = 3 * 800 + 160;
constexpr int kFacBack = 8;  // and in its back substitution's
constexpr int kFacBackSlot = kFacSlot * kFacRing / kFacBack;
constexpr int kCorRing = 6;  // the correction's forward ring
constexpr int kCorSlot = 2 * 800 + 160;
constexpr int kCorBack = 11;  // and its back substitution's
constexpr int kCorBackSlot = 800 + 160;
static_assert(kFacBackSlot >= 800 + 2 * 160, "ring");
static_assert(kCorBack * kCorBackSlot <= kCorRing * kCorSlot, "ring");

__device__ __forceinline__ bool vfinite32(float x) {
  return ((__float_as_uint(x) >> 23) & 0xffu) != 0xffu;
}

__device__ __forceinline__ void cpa16(void* s, const void* g) {
  const unsigned a = static_cast<unsigned>(__cvta_generic_to_shared(s));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(a), "l"(g)
               : "memory");
}
__device__ __forceinline__ void cpa_commit() {
  asm volatile("cp.async.commit_group;\n" ::: "memory");
}
// this thread's copies of all but the newest N groups are complete
template <int N>
__device__ __forceinline__ void cpa_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// the warp's copy of nf floats (a multiple of 4, both ends on 16 bytes)
__device__ __forceinline__ void tile_fill(float* s, const float* g, int nf,
                                          int lane) {
  for (int e = 4 * lane; e < nf; e += 128) cpa16(s + e, g + e);
}

// 1 / p to about half an ulp without a branch: the approximate reciprocal and
// one Newton step (a subnormal p gives infinity, and masks the column)
__device__ __forceinline__ float rcp_near(float p) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(p));
  return fmaf(r, fmaf(-p, r, 1.f), r);
}

// the inverse of a 5x5 block in place (Gauss-Jordan, no pivoting: see above);
// false where a pivot cancels or is not finite
__device__ __forceinline__ bool invert5(float (&a)[25]) {
  float dg[5];
#pragma unroll
  for (int k = 0; k < 5; ++k) dg[k] = fabsf(a[6 * k]);
  bool good = true;
#pragma unroll
  for (int k = 0; k < 5; ++k) {
    const float p = a[6 * k];
    good = good && fabsf(p) > 8.f * 5.f * 1.1920929e-7f * dg[k] && vfinite32(p);
    const float ip = rcp_near(p);
#pragma unroll
    for (int j = 0; j < 5; ++j)
      if (j != k) a[5 * k + j] *= ip;
#pragma unroll
    for (int i = 0; i < 5; ++i) {
      if (i == k) continue;
      const float f = a[5 * i + k];
#pragma unroll
      for (int j = 0; j < 5; ++j)
        if (j != k) a[5 * i + j] = fmaf(-f, a[5 * k + j], a[5 * i + j]);
      a[5 * i + k] = -f * ip;
    }
    a[6 * k] = ip;
  }
  return good;
}

// the rows of N values a lane's column has in a slot (or an array's layer)
template <int N>
__device__ __forceinline__ void tile_get(float (&v)[N], const float* s, int w) {
#pragma unroll
  for (int e = 0; e < N; ++e) v[e] = s[e * w];
}

// y -= M x and y = M x of a 5x5 block
__device__ __forceinline__ void msub5(const float (&m)[25], const float (&x)[5],
                                      float (&y)[5]) {
#pragma unroll
  for (int k = 0; k < 5; ++k)
#pragma unroll
    for (int r = 0; r < 5; ++r) y[r] = fmaf(-m[5 * r + k], x[k], y[r]);
}
__device__ __forceinline__ void mul5(const float (&m)[25], const float (&x)[5],
                                     float (&y)[5]) {
#pragma unroll
  for (int r = 0; r < 5; ++r) y[r] = m[5 * r] * x[0];
#pragma unroll
  for (int k = 1; k < 5; ++k)
#pragma unroll
    for (int r = 0; r < 5; ++r) y[r] = fmaf(m[5 * r + k], x[k], y[r]);
}

// a pass's solution of one value from the sweep's and the Woodbury vectors,
// one rounding order for every kernel that forms it
__device__ __forceinline__ float wood32(float x, float z0, float z1, float al0,
                                        float al1) {
  return fmaf(-z1, al1, fmaf(-z0, al0, x));
}

// the Woodbury weights of the two wall entries k0, k1 from the densities of
// x, z0, z1 at layers 2 and n - 3
template <typename T>
__device__ __forceinline__ void wood_weights(T k0, T k1, T x2, T x3, T z02, T z03,
                                             T z12, T z13, T& al0, T& al1) {
  const T m00 = T(1.) + k0 * z02, m01 = k0 * z12;
  const T m10 = k1 * z03, m11 = T(1.) + k1 * z13;
  const T r0 = k0 * x2, r1 = k1 * x3;
  const T det = m00 * m11 - m01 * m10;
  al0 = (m11 * r0 - m01 * r1) / det;
  al1 = (m00 * r1 - m10 * r0) / det;
}

// The factors (the pivot blocks' inverses and C') and the first solution of
// a tile: the forward sweep for b and, of the Woodbury unit vectors, the
// lower one alone (the upper one's is zero below its own layer), the back
// substitution of all three, the Woodbury weights.  A layer's A, B and b are
// read into registers while the layer before it is eliminated, its C while
// its own pivot is inverted: with a warp or two per scheduler nothing else
// hides those loads.  W: the tile's width at compile time (32), or 0 to take
// it from wr
template <int W>
__device__ __forceinline__ void factor_tile(const BlockDev& Bk,
                                            const StageParams& p,
                                            const VicScratch32& F, int n,
                                            size_t tile, int wr, double dtc,
                                            float* ring) {
  const int w = W ? W : wr;
  const int lane = threadIdx.x;
  const bool on = lane < w;
  const int c25 = VicTile::chunk(25, w), c5 = VicTile::chunk(5, w);
  const size_t o25 = VicTile::base(25, tile, n), o5 = VicTile::base(5, tile, n);
  const float *A = F.A + o25, *B = F.B + o25, *C = F.C + o25;
  float *PI = F.PI + o25, *CP = F.CP + o25, *R = F.R + o5, *X0 = F.X0 + o5;
  float *Z0 = F.Z0 + o5, *Z1 = F.Z1 + o5;

  auto fissue = [&](int i) {
    if (i < n) {
      float* s = ring + (i & (kFacRing - 1)) * kFacSlot;
      tile_fill(s, A + (size_t)i * c25, c25, lane);
      tile_fill(s + 800, B + (size_t)i * c25, c25, lane);
      tile_fill(s + 1600, C + (size_t)i * c25, c25, lane);
      tile_fill(s + 2400, R + (size_t)i * c5, c5, lane);
    }
    cpa_commit();
  };
  bool ok = true;
  float cp[25], y[5], z0[5], z1[5];
#pragma unroll
  for (int k = 0; k < 25; ++k) cp[k] = 0.f;
#pragma unroll
  for (int k = 0; k < 5; ++k) y[k] = z0[k] = z1[k] = 0.f;
  // one layer: a, b, t are the layer's, read by the step before; na, nb, nt
  // the next one's
  auto step = [&](int i, float (&a)[25], float (&b)[25], float (&t)[5],
                  float (&na)[25], float (&nb)[25], float (&nt)[5]) {
    cpa_wait<kFacRing - 3>();  // layer i + 1 is here
    __syncwarp();              // and layer i - 1's slot is read
    fissue(i + kFacRing - 1);
    const float* s = ring + ((i + 1) & (kFacRing - 1)) * kFacSlot + lane;
    tile_get(nb, s + 800, w);
    tile_get(na, s, w);
    tile_get(nt, s + 2400, w);
    float tz[5] = {0.f, 0.f, 0.f, 0.f, i == 0 ? 1.f : 0.f};
#pragma unroll
    for (int k = 0; k < 5; ++k)
#pragma unroll
      for (int r = 0; r < 5; ++r)
#pragma unroll
        for (int c = 0; c < 5; ++c)
          a[5 * r + c] = fmaf(-b[5 * r + k], cp[5 * k + c], a[5 * r + c]);
    msub5(b, y, t);
    msub5(b, z0, tz);
    float cc[25];
    tile_get(cc, ring + (i & (kFacRing - 1)) * kFacSlot + 1600 + lane, w);
    ok = invert5(a) && ok;
    mul5(a, t, y);
    mul5(a, tz, z0);
#pragma unroll
    for (int r = 0; r < 5; ++r)
#pragma unroll
      for (int c = 0; c < 5; ++c) {
        float q = a[5 * r] * cc[c];
#pragma unroll
        for (int k = 1; k < 5; ++k) q = fmaf(a[5 * r + k], cc[5 * k + c], q);
        cp[5 * r + c] = q;
      }
    if (on) {
      float* pi = PI + (size_t)i * c25 + lane;
      float* co = CP + (size_t)i * c25 + lane;
#pragma unroll
      for (int e = 0; e < 25; ++e) pi[e * w] = a[e];
#pragma unroll
      for (int e = 0; e < 25; ++e) co[e * w] = cp[e];
#pragma unroll
      for (int r = 0; r < 5; ++r) {
        R[(size_t)i * c5 + r * w + lane] = y[r];
        Z0[(size_t)i * c5 + r * w + lane] = z0[r];
      }
    }
    if (i == n - 1) {
#pragma unroll
      for (int r = 0; r < 5; ++r) z1[r] = a[5 * r + 4];
    }
  };
#pragma unroll
  for (int j = 0; j < kFacRing - 1; ++j) fissue(j);
  float a0[25], b0[25], t0[5], a1[25], b1[25], t1[5];
  cpa_wait<kFacRing - 2>();
  __syncwarp();
  tile_get(a0, ring + lane, w);
  tile_get(b0, ring + 800 + lane, w);
  tile_get(t0, ring + 2400 + lane, w);
  for (int i = 0; i < n; i += 2) {
    step(i, a0, b0, t0, a1, b1, t1);
    if (i + 1 < n) step(i + 1, a1, b1, t1, a0, b0, t0);
  }
  cpa_wait<0>();
  __syncwarp();  // y, z0 and C' are stored before other lanes copy them

  // ---- back: x_i = y_i - C'_i x_(i+1) of the three vectors ----
  float x2 = 0.f, x3 = 0.f, z02 = 0.f, z03 = 0.f, z12 = 0.f, z13 = 0.f;
  auto put = [&](int i) {
    if (on) {
#pragma unroll
      for (int r = 0; r < 5; ++r) {
        X0[(size_t)i * c5 + r * w + lane] = y[r];
        Z0[(size_t)i * c5 + r * w + lane] = z0[r];
        Z1[(size_t)i * c5 + r * w + lane] = z1[r];
      }
    }
    if (i == 2) x2 = y[0], z02 = z0[0], z12 = z1[0];
    if (i == n - 3) x3 = y[0], z03 = z0[0], z13 = z1[0];
  };
  auto bissue = [&](int j) {  // step j is layer n - 2 - j
    if (j < n - 1) {
      const int i = n - 2 - j;
      float* s = ring + (j & (kFacBack - 1)) * kFacBackSlot;
      tile_fill(s, CP + (size_t)i * c25, c25, lane);
      tile_fill(s + 800, R + (size_t)i * c5, c5, lane);
      tile_fill(s + 960, Z0 + (size_t)i * c5, c5, lane);
    }
    cpa_commit();
  };
  auto bget = [&](int j, float (&c)[25], float (&u)[5], float (&v)[5]) {
    const float* s = ring + (j & (kFacBack - 1)) * kFacBackSlot + lane;
    tile_get(c, s, w);
    tile_get(u, s + 800, w);
    tile_get(v, s + 960, w);
  };
  auto bstep = [&](int j, float (&c)[25], float (&u)[5], float (&v)[5],
                   float (&nc)[25], float (&nu)[5], float (&nv)[5]) {
    cpa_wait<kFacBack - 2>();  // step j + 1's layer is here
    __syncwarp();              // and step j's slot is read
    bissue(j + kFacBack);
    bget(j + 1, nc, nu, nv);
    float v1[5] = {0.f, 0.f, 0.f, 0.f, 0.f};
    msub5(c, y, u);
    msub5(c, z0, v);
    msub5(c, z1, v1);
#pragma unroll
    for (int r = 0; r < 5; ++r) y[r] = u[r], z0[r] = v[r], z1[r] = v1[r];
    put(n - 2 - j);
  };
  float u0[5], v0[5], u1[5], v1[5];
#pragma unroll
  for (int j = 0; j < kFacBack; ++j) bissue(j);
  put(n - 1);
  cpa_wait<kFacBack - 1>();
  __syncwarp();
  bget(0, a0, u0, v0);
  for (int j = 0; j < n - 1; j += 2) {
    bstep(j, a0, u0, v0, a1, u1, v1);
    if (j + 1 < n - 1) bstep(j + 1, a1, u1, v1, a0, u0, v0);
  }
  cpa_wait<0>();

  if (!on) return;
  const size_t col = tile * 32 + lane;
  float al0 = 0.f, al1 = 0.f;
  if (n >= 3)
    wood_weights<float>(narrow_exact(-vic_krows(Bk, n, 0).t0 / dtc),
                        narrow_exact(-vic_krows(Bk, n, n - 1).t1 / dtc), x2, x3,
                        z02, z03, z12, z13, al0, al1);
  F.AL[col] = al0;
  F.AL[F.ncol + col] = al1;
  F.mask[col] = ok ? 0 : 1;
}

__global__ void __launch_bounds__(32)
    vic_factor32_kernel(const BlockDev* __restrict__ tab, StageParams p) {
  __shared__ __align__(16) float ring[kFacRing * kFacSlot];
  const BlockDev& Bk = tab[blockIdx.y];
  // (scheme-9 blocks only: a scheme-1 block assembled in FP32 is solved
  // in FP64 by vic_solve3_kernel)
  if (Bk.implicit != 9 || !Bk.implicit_f32) return;
  const VicScratch S = vic_scratch(Bk);
  const int n = Bk.nc1 - 2 * Bk.ng;
  const VicScratch32 F = vic_scratch32(Bk, S, n);
  const size_t tile = blockIdx.x;
  if (tile * 32 >= F.ncol) return;
  const int w = VicTile::width(F.ncol, tile);
  const double dtc = p.w2 * p.dt[blockIdx.y];
  if (w == 32)
    factor_tile<32>(Bk, p, F, n, tile, w, dtc, ring);
  else
    factor_tile<0>(Bk, p, F, n, tile, w, dtc, ring);
}

// s_h + s_l += t d in float-float arithmetic, t and d floats: the product
// split exactly by an FMA (the two-product of Dekker's method), the sum by
// Knuth's two-sum; the low parts gather in s_l.  Every step is a single
// rounding (__fmul_rn / __fadd_rn are never contracted)
__device__ __forceinline__ void ff_madd(float& sh, float& sl, float t, float d) {
  const float p = __fmul_rn(t, d);
  const float e = __fmaf_rn(t, d, -p);
  const float s2 = __fadd_rn(sh, p);
  const float bp = __fadd_rn(s2, -sh);
  const float err =
      __fadd_rn(__fadd_rn(sh, -__fadd_rn(s2, -bp)), __fadd_rn(p, -bp));
  sl = __fadd_rn(sl, __fadd_rn(err, e));
  sh = s2;
}

// s_h + (m_h + m_l) += t d, t and d floats, to well beyond FP64 accuracy:
// the product split exactly (Dekker's two-product by an FMA), its high part
// added to s_h by Knuth's two-sum, and the two exact remainders (the sum's
// rounding error and the product's low part) gathered in the float-float
// pair m_h + m_l.  The pair holds terms of 2^-24 of the products, so its
// own error is about 2^-48 of that: 2^-72 of the sum of |t d|
__device__ __forceinline__ void ff_acc(float& mh, float& ml, float v) {
  const float s2 = __fadd_rn(mh, v);
  const float bp = __fadd_rn(s2, -mh);
  ml = __fadd_rn(ml, __fadd_rn(__fadd_rn(mh, -__fadd_rn(s2, -bp)),
                               __fadd_rn(v, -bp)));
  mh = s2;
}

__device__ __forceinline__ void tf_madd(float& sh, float& mh, float& ml, float t,
                                        float d) {
  const float p = __fmul_rn(t, d);
  const float e = __fmaf_rn(t, d, -p);
  const float s2 = __fadd_rn(sh, p);
  const float bp = __fadd_rn(s2, -sh);
  const float err =
      __fadd_rn(__fadd_rn(sh, -__fadd_rn(s2, -bp)), __fadd_rn(p, -bp));
  sh = s2;
  ff_acc(mh, ml, err);
  ff_acc(mh, ml, e);
}

// The residual of every cell, a warp per tile and layer, a lane per column,
// rounded to FP32 into R for the correction's sweeps.
// * The first correction's (corr 1) is b - T x, x the first solution
//   (the factor sweep's with its Woodbury step): T x as a sum of exact float products (tf_madd, on the FP32
//   pipe, to about 2^-72 of the sum of |t x|), then b minus that sum in
//   FP64 (three subtractions, the first exact).
// * A later one is the previous r less T d, d the FP32 correction x grew by:
//   T d in float-float on the FP32 pipe (its error, 2^-48 of the sum of
//   |t d| with |d| about 2^-22 |x|, is far below the FP64 rounding of r).
// Every load is a tile's row of 32 consecutive values.
template <int W>
__device__ __forceinline__ void residual_row(const BlockDev& Bk,
                                             const VicScratch32& F, int n,
                                             size_t tile, int i, int wr, int corr,
                                             bool keep, double dtc) {
  const int w = W ? W : wr;
  const int lane = threadIdx.x & 31;
  if (lane >= w) return;
  const int c25 = VicTile::chunk(25, w), c5 = VicTile::chunk(5, w);
  const size_t o25 = VicTile::base(25, tile, n) + (size_t)i * c25 + lane;
  const size_t o5 = VicTile::base(5, tile, n) + lane;
  const float* X = (corr == 1 ? F.X0 : F.DK + (size_t)(corr - 2) * F.dk) + o5;
  const float *Z0 = F.Z0 + o5, *Z1 = F.Z1 + o5;
  const size_t col = tile * 32 + lane;
  const float al0 = F.AL[(size_t)(2 * corr - 2) * F.ncol + col];
  const float al1 = F.AL[(size_t)(2 * corr - 1) * F.ncol + col];
  double* r64 = F.r64 + VicTile::base(5, tile, n) + (size_t)i * 5 * w + lane;
  double t[5];
#pragma unroll
  for (int r = 0; r < 5; ++r) t[r] = r64[r * w];
  float sh[5] = {0.f, 0.f, 0.f, 0.f, 0.f}, mh[5] = {0.f, 0.f, 0.f, 0.f, 0.f},
        ml[5] = {0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int m = 0; m < 3; ++m) {  // the cell, below, above
    if ((m == 1 && i == 0) || (m == 2 && i == n - 1)) continue;
    const float* M = (m == 0 ? F.A : (m == 1 ? F.B : F.C)) + o25;
    const size_t e = (size_t)(m == 0 ? i : (m == 1 ? i - 1 : i + 1)) * c5;
    float x[5];
#pragma unroll
    for (int k = 0; k < 5; ++k)
      x[k] = wood32(X[e + k * w], Z0[e + k * w], Z1[e + k * w], al0, al1);
    if (corr == 1) {
#pragma unroll
      for (int r = 0; r < 5; ++r)
#pragma unroll
        for (int k = 0; k < 5; ++k)
          tf_madd(sh[r], mh[r], ml[r], M[(5 * r + k) * w], x[k]);
    } else {
#pragma unroll
      for (int r = 0; r < 5; ++r)
#pragma unroll
        for (int k = 0; k < 5; ++k) ff_madd(sh[r], mh[r], M[(5 * r + k) * w], x[k]);
    }
  }
#pragma unroll
  for (int r = 0; r < 5; ++r)
    t[r] = ((t[r] - widen_exact(sh[r])) - widen_exact(mh[r])) - widen_exact(ml[r]);
  if (n >= 3) {  // the wall rows' third points
    if (i == 0) {
      const size_t e = (size_t)2 * c5;
      t[4] -= (-vic_krows(Bk, n, 0).t0 / dtc) *
              widen_exact(wood32(X[e], Z0[e], Z1[e], al0, al1));
    }
    if (i == n - 1) {
      const size_t e = (size_t)(n - 3) * c5;
      t[4] -= (-vic_krows(Bk, n, n - 1).t1 / dtc) *
              widen_exact(wood32(X[e], Z0[e], Z1[e], al0, al1));
    }
  }
#pragma unroll
  for (int r = 0; r < 5; ++r) {
    if (keep) r64[r * w] = t[r];
    F.R[o5 + (size_t)i * c5 + r * w] = narrow_exact(t[r]);
  }
}

__global__ void __launch_bounds__(kThreads)
    vic_residual_kernel(const BlockDev* __restrict__ tab, StageParams p,
                        int corr) {
  const BlockDev& Bk = tab[blockIdx.y];
  if (Bk.implicit != 9 || !Bk.implicit_f32) return;
  const VicScratch S = vic_scratch(Bk);
  const int n = Bk.nc1 - 2 * Bk.ng;
  const VicScratch32 F = vic_scratch32(Bk, S, n);
  const size_t rows = ((F.ncol + 31) / 32) * n;  // (tile, layer) rows
  const bool keep = corr < p.refine;             // a later correction reads r
  const double dtc = p.w2 * p.dt[blockIdx.y];
  for (size_t q = (size_t)blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5);
       q < rows; q += (size_t)gridDim.x * (kThreads / 32)) {
    const size_t tile = q / n;
    const int i = (int)(q - tile * n);
    const int w = VicTile::width(F.ncol, tile);
    if (w == 32)
      residual_row<32>(Bk, F, n, tile, i, w, corr, keep, dtc);
    else
      residual_row<0>(Bk, F, n, tile, i, w, corr, keep, dtc);
  }
}

// A correction's sweeps of a tile: y_i = P_i^-1 (r_i - B_i y_(i-1)) going up,
// d_i = y_i - C'_i d_(i+1) coming down, and the Woodbury weights (the kernels
// that read d apply them).  The layer after the one in hand is in registers
// before it is needed, as in the factor's sweeps
template <int W>
__device__ __forceinline__ void correct_tile(const BlockDev& Bk,
                                             const VicScratch32& F, int n,
                                             size_t tile, int wr, int corr,
                                             double dtc, float* ring) {
  const int w = W ? W : wr;
  const int lane = threadIdx.x;
  const bool on = lane < w;
  const int c25 = VicTile::chunk(25, w), c5 = VicTile::chunk(5, w);
  const size_t o25 = VicTile::base(25, tile, n), o5 = VicTile::base(5, tile, n);
  const float *PI = F.PI + o25, *B = F.B + o25, *CP = F.CP + o25;
  float* R = F.R + o5;
  float* X = F.DK + (size_t)(corr - 1) * F.dk + o5;

  int islot = 0, gslot = 0;
  auto fissue = [&](int i) {
    if (i < n) {
      float* s = ring + islot * kCorSlot;
      tile_fill(s, PI + (size_t)i * c25, c25, lane);
      tile_fill(s + 800, B + (size_t)i * c25, c25, lane);
      tile_fill(s + 1600, R + (size_t)i * c5, c5, lane);
    }
    islot = islot + 1 == kCorRing ? 0 : islot + 1;
    cpa_commit();
  };
  auto fget = [&](float (&pi)[25], float (&b)[25], float (&t)[5]) {
    const float* s = ring + gslot * kCorSlot + lane;
    gslot = gslot + 1 == kCorRing ? 0 : gslot + 1;
    tile_get(b, s + 800, w);
    tile_get(t, s + 1600, w);
    tile_get(pi, s, w);
  };
  float y[5] = {0.f, 0.f, 0.f, 0.f, 0.f};
  auto fstep = [&](int i, float (&pi)[25], float (&b)[25], float (&t)[5],
                   float (&npi)[25], float (&nb)[25], float (&nt)[5]) {
    cpa_wait<kCorRing - 2>();  // layer i + 1 is here
    __syncwarp();              // and layer i's slot is read
    fissue(i + kCorRing);
    fget(npi, nb, nt);
    msub5(b, y, t);
    mul5(pi, t, y);
    if (on) {
#pragma unroll
      for (int r = 0; r < 5; ++r) R[(size_t)i * c5 + r * w + lane] = y[r];
    }
  };
#pragma unroll
  for (int j = 0; j < kCorRing; ++j) fissue(j);
  float p0[25], b0[25], t0[5], p1[25], b1[25], t1[5];
  cpa_wait<kCorRing - 1>();
  __syncwarp();
  fget(p0, b0, t0);
  for (int i = 0; i < n; i += 2) {
    fstep(i, p0, b0, t0, p1, b1, t1);
    if (i + 1 < n) fstep(i + 1, p1, b1, t1, p0, b0, t0);
  }
  cpa_wait<0>();
  __syncwarp();

  float x2 = 0.f, x3 = 0.f;
  auto put = [&](int i) {
    if (on) {
#pragma unroll
      for (int r = 0; r < 5; ++r) X[(size_t)i * c5 + r * w + lane] = y[r];
    }
    if (i == 2) x2 = y[0];
    if (i == n - 3) x3 = y[0];
  };
  islot = gslot = 0;
  auto bissue = [&](int j) {  // step j is layer n - 2 - j
    if (j < n - 1) {
      const int i = n - 2 - j;
      float* s = ring + islot * kCorBackSlot;
      tile_fill(s, CP + (size_t)i * c25, c25, lane);
      tile_fill(s + 800, R + (size_t)i * c5, c5, lane);
    }
    islot = islot + 1 == kCorBack ? 0 : islot + 1;
    cpa_commit();
  };
  auto bget = [&](float (&c)[25], float (&u)[5]) {
    const float* s = ring + gslot * kCorBackSlot + lane;
    gslot = gslot + 1 == kCorBack ? 0 : gslot + 1;
    tile_get(c, s, w);
    tile_get(u, s + 800, w);
  };
  auto bstep = [&](int j, float (&c)[25], float (&u)[5], float (&nc)[25],
                   float (&nu)[5]) {
    cpa_wait<kCorBack - 2>();
    __syncwarp();
    bissue(j + kCorBack);
    bget(nc, nu);
    msub5(c, y, u);
#pragma unroll
    for (int r = 0; r < 5; ++r) y[r] = u[r];
    put(n - 2 - j);
  };
#pragma unroll
  for (int j = 0; j < kCorBack; ++j) bissue(j);
  put(n - 1);
  cpa_wait<kCorBack - 1>();
  __syncwarp();
  bget(p0, t0);
  for (int j = 0; j < n - 1; j += 2) {
    bstep(j, p0, t0, p1, t1);
    if (j + 1 < n - 1) bstep(j + 1, p1, t1, p0, t0);
  }
  cpa_wait<0>();

  if (!on) return;
  const size_t col = tile * 32 + lane;
  float al0 = 0.f, al1 = 0.f;
  if (n >= 3) {
    const float *Z0 = F.Z0 + o5 + lane, *Z1 = F.Z1 + o5 + lane;
    const size_t e2 = (size_t)2 * c5, e3 = (size_t)(n - 3) * c5;
    wood_weights<float>(narrow_exact(-vic_krows(Bk, n, 0).t0 / dtc),
                        narrow_exact(-vic_krows(Bk, n, n - 1).t1 / dtc), x2, x3,
                        Z0[e2], Z0[e3], Z1[e2], Z1[e3], al0, al1);
  }
  F.AL[(size_t)(2 * corr) * F.ncol + col] = al0;
  F.AL[(size_t)(2 * corr + 1) * F.ncol + col] = al1;
}

__global__ void __launch_bounds__(32)
    vic_correct32_kernel(const BlockDev* __restrict__ tab, StageParams p,
                         int corr) {
  __shared__ __align__(16) float ring[kCorRing * kCorSlot];
  const BlockDev& Bk = tab[blockIdx.y];
  if (Bk.implicit != 9 || !Bk.implicit_f32) return;
  const VicScratch S = vic_scratch(Bk);
  const int n = Bk.nc1 - 2 * Bk.ng;
  const VicScratch32 F = vic_scratch32(Bk, S, n);
  const size_t tile = blockIdx.x;
  if (tile * 32 >= F.ncol) return;
  const int w = VicTile::width(F.ncol, tile);
  const double dtc = p.w2 * p.dt[blockIdx.y];
  if (w == 32)
    correct_tile<32>(Bk, F, n, tile, w, corr, dtc, ring);
  else
    correct_tile<0>(Bk, F, n, tile, w, corr, dtc, ring);
}

// The end of the refined solve, a CTA per tile, its warps over the layers:
// D = x0 + d_1 + ... in FP64 (each pass's solution with its Woodbury step),
// and each column's convergence: the error the last correction leaves is
// about |d| rho, rho = |d| / |d_prev| the observed contraction, accepted at
// or below 2^-44 of the largest |x|.  The FP32 solve (p.refine < 0) has no
// corrections: D is the sweep's solution with the Woodbury step in FP64 on
// the widened FP32 vectors, accepted where it is finite
__global__ void __launch_bounds__(kThreads)
    vic_accept_kernel(const BlockDev* __restrict__ tab, StageParams p) {
  __shared__ float smax[3][kThreads / 32][32];
  __shared__ int sfin[kThreads / 32][32];
  const BlockDev& Bk = tab[blockIdx.y];
  if (Bk.implicit != 9 || !Bk.implicit_f32) return;
  const VicScratch S = vic_scratch(Bk);
  const int n = Bk.nc1 - 2 * Bk.ng;
  const VicScratch32 F = vic_scratch32(Bk, S, n);
  const size_t tile = blockIdx.x;
  if (tile * 32 >= F.ncol) return;
  const int w = VicTile::width(F.ncol, tile);
  const int lane = threadIdx.x & 31, wq = threadIdx.x >> 5;
  const int c5 = VicTile::chunk(5, w);
  const size_t o5 = VicTile::base(5, tile, n) + lane;
  const size_t col = tile * 32 + lane;
  const int nk = p.refine > 0 ? p.refine : 0;
  float mx = 0.f, dp = 0.f, dl = 0.f;  // |x0|, the last two updates
  bool fin = true;
  if (lane < w) {
    double* D = S.D + col * n * 5;
    if (p.refine < 0) {
      double ad0 = 0., ad1 = 0.;
      if (n >= 3) {
        const double dtc = p.w2 * p.dt[blockIdx.y];
        const size_t e2 = o5 + (size_t)2 * c5, e3 = o5 + (size_t)(n - 3) * c5;
        wood_weights<double>(
            -vic_krows(Bk, n, 0).t0 / dtc, -vic_krows(Bk, n, n - 1).t1 / dtc,
            widen_exact(F.X0[e2]), widen_exact(F.X0[e3]), widen_exact(F.Z0[e2]),
            widen_exact(F.Z0[e3]), widen_exact(F.Z1[e2]), widen_exact(F.Z1[e3]),
            ad0, ad1);
      }
      for (int i = wq; i < n; i += kThreads / 32)
#pragma unroll
        for (int r = 0; r < 5; ++r) {
          const size_t e = o5 + (size_t)i * c5 + r * w;
          double d = widen_exact(F.X0[e]);
          d -= widen_exact(F.Z0[e]) * ad0;
          d -= widen_exact(F.Z1[e]) * ad1;
          fin = fin && vfinite(d);
          D[i * 5 + r] = d;
        }
    } else {
      float al0[4], al1[4];
      for (int q = 0; q <= nk; ++q) {
        al0[q] = F.AL[(size_t)(2 * q) * F.ncol + col];
        al1[q] = F.AL[(size_t)(2 * q + 1) * F.ncol + col];
      }
      for (int i = wq; i < n; i += kThreads / 32) {
        float x[4][5], z0[5], z1[5];
#pragma unroll
        for (int r = 0; r < 5; ++r) {
          const size_t e = o5 + (size_t)i * c5 + r * w;
          z0[r] = F.Z0[e];
          z1[r] = F.Z1[e];
          x[0][r] = F.X0[e];
#pragma unroll
          for (int q = 1; q < 4; ++q)
            x[q][r] = q <= nk ? F.DK[(size_t)(q - 1) * F.dk + e] : 0.f;
        }
#pragma unroll
        for (int r = 0; r < 5; ++r) {
          double sum = 0.;
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            if (q > nk) break;
            const float d = wood32(x[q][r], z0[r], z1[r], al0[q], al1[q]);
            const float m = fabsf(d);
            fin = fin && vfinite32(d);
            if (q == 0) mx = fmaxf(mx, m);
            if (q == nk - 1) dp = fmaxf(dp, m);
            if (q == nk) dl = fmaxf(dl, m);
            sum = q == 0 ? widen_exact(d) : sum + widen_exact(d);
          }
          D[i * 5 + r] = sum;
        }
      }
    }
  }
  smax[0][wq][lane] = mx;
  smax[1][wq][lane] = dp;
  smax[2][wq][lane] = dl;
  sfin[wq][lane] = fin;
  __syncthreads();
  if (wq || lane >= w) return;
  for (int q = 1; q < kThreads / 32; ++q) {
    mx = fmaxf(mx, smax[0][q][lane]);
    dp = fmaxf(dp, smax[1][q][lane]);
    dl = fmaxf(dl, smax[2][q][lane]);
    fin = fin && sfin[q][lane];
  }
  if (p.refine > 0) {
    const float rho = dp > 0.f ? fminf(dl / dp, 1.f) : 0.f;
    fin = fin && dl * rho <= 0x1p-44f * mx;
  }
  // the last update and the scale, kept for inspection (nothing reads them)
  F.stat[col * 6] = dl;
  F.stat[col * 6 + 3] = mx;
  if (!fin) F.mask[col] = 1;
}
