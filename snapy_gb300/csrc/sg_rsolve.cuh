// The refined solve of implicit-precision float32 blocks of implicit-scheme
// 9.  Included by sg_stage.cu after sg_vic.cuh, inside its anonymous
// namespace.
//
// The system of a column is T x = b, T the block-tridiagonal matrix of the
// FP32-assembled 5x5 blocks (B_i, A_i, C_i) plus the two third-point entries of the
// corrected-PE wall rows (layer 0's energy row reads the density of layer 2,
// layer n - 1's that of layer n - 3), and b = du / dt_corr.  It is solved by
// mixed-precision iterative refinement (the scheme of LAPACK's dsgesv): an
// FP32 solve M^-1, then p.refine corrections d = M^-1 r with r = b - T x
// formed beyond FP64 accuracy and x summed in FP64.  The last correction's
// size and its gain estimate the error it leaves; p.accept bounds it.  The
// FP32 form (sg_set_solve -1) makes one correction and accepts FP32's
// rounding, 2^-24 of the solution: M^-1 alone can lose digits in a strong
// wind, which nothing would show.
//
//   vic_factor32_kernel    M^-1's factors and the first solution
//   vic_residual_kernel    r = b - T x (or the previous r less T d)
//   vic_correct32_kernel   d = M^-1 r; after the last, the acceptance
//   vic_sum_kernel         x0 + d1 + ... into D
//
// M^-1 eliminates a column from both walls at once towards a middle layer m:
// x_i = y_i - C'_i x_(i+1) below it, x_i = y_i - B'_i x_(i-1) above it, the
// middle layer solved from both neighbours, then back out to the walls.  No
// fill, the operations of the one-way sweep, half its chain.  A wall row's
// third point is eliminated with its layer: x_0 = y_0 - C'_0 x_1 - e x_2[0]
// with e = k0 P_0^-1 e_4, which takes k0-fold B_1 e from C_1's density
// column, so there are no Woodbury vectors to solve or apply.  (This needs
// two layers either side of the middle: columns of fewer than five layers
// take the FP64 solve.)  The pivot blocks are inverted in place without row
// exchanges, the tangential momenta last: the diagonal of such a row is 1 /
// dt_corr less a share of |A| that grows with the square of the wind across
// the column, so it passes through zero in a strong wind, and eliminating the
// energy row first takes that share away.  The order changes the rounding of
// M^-1 alone, never the solution.  A correction's gain in a model of 32 layers
// of 50 m, winds to 350 m/s, steps of 1 to 100 sound crossings of a layer,
// mean and worst: 1e-7 to 3e-6 and 9e-5 (with scaled partial pivoting 1e-7 to
// 1e-6 and 6e-5; tangential momenta before the energy 1e-7 to 3e-5 and 3e-3,
// which left one column in eleven to FP64).  A pivot that cancels to below 40 eps
// of its diagonal, a value that is not finite, or an estimated error above
// p.accept (2^-44) of the solution masks the column,
// and it takes the FP64 solve (vic_psolve_kernel, vic_solve_kernel), as the
// reference retries a failed FP32 column in FP64 (src/hydro/hydro.cpp:436-466).
//
// Layout.  Columns are taken 32 at a time: an array of E values per cell
// keeps, for each tile of w <= 32 columns and each layer, E rows of w
// values, padded to 16 bytes (VicTile).  Two warps own a tile in the sweeps
// (one from each wall), a lane a column: every load, copy and store of a
// layer is one contiguous span, and the 5x5 algebra has no shuffles, no pivot
// search and no synchronisation between lanes.
//
// What bounds it: the bytes a cell moves (about 0.7 KB in the factor sweep,
// 0.4 KB in a residual, 0.4 KB in a correction), and, with few columns, the
// instructions of a column's layers one after the other: a layer's copies are
// at constant offsets from pointers that step by a layer, and |x| and its
// finiteness are one integer maximum.  Measured per launch (us), before (a
// column on eight lanes, one way, LU factors and three right-hand sides) and
// now, 64-member ensemble (21,120 columns, 1.44 M cells): first sweep 815 and
// 225, a residual 634 and 166 (the first) or 126, a correction 613 and
// 95; the sum, apart now, 56.  384 columns of 100: first sweep 56,
// correction 24 (this layout swept one way 154 and 83, from both walls with
// the Woodbury vectors 65 and 42); 4,096 of 64: 60 and 25.
#pragma once

__device__ __forceinline__ bool vfinite32(float x) {
  return ((__float_as_uint(x) >> 23) & 0xffu) != 0xffu;
}

__device__ __forceinline__ void cpa16(unsigned s, const void* g) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(g)
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

// a lane's share of the warp's copy of nf floats (a multiple of 4, both ends
// on 16 bytes), to its own shared address s from its own source g (each 16
// bytes a lane past the span's first): with nf known, copies at constant
// offsets and one predicate
__device__ __forceinline__ void tile_fill(unsigned s, const float* g, int nf,
                                          int lane) {
#pragma unroll
  for (int e = 0; e < 800; e += 128)
    if (e + 4 * lane < nf) cpa16(s + 4 * e, g + e);
}

// 1 / p to about half an ulp without a branch: the approximate reciprocal and
// one Newton step (a subnormal p gives infinity, and masks the column)
__device__ __forceinline__ float rcp_near(float p) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(p));
  return fmaf(r, fmaf(-p, r, 1.f), r);
}

// the inverse of a 5x5 block in place (Gauss-Jordan, the diagonal in the order
// given above); false where a pivot cancels or is not finite
__device__ __forceinline__ bool invert5(float (&a)[25]) {
  float dg[5];
#pragma unroll
  for (int k = 0; k < 5; ++k) dg[k] = fabsf(a[6 * k]);
  bool good = true;
  constexpr int order[5] = {IDN, IVX, IPR, IVY, IVZ};
#pragma unroll
  for (int q = 0; q < 5; ++q) {
    const int k = order[q];
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


// the arrays of one tile, each at the tile's first value
struct RTile {
  float *A, *B, *C, *PI, *CP, *R, *X0, *DK;
  size_t dk;       // the values of one correction's array
  double* r64;     // the FP64 residual, rows of w, no padding
  float* E;        // the walls' e, rows of w: the lower's 0-4, the upper's 5-9
  float* stat;     // per column 6: the largest |x0|, |d1|, |d2|, ...
  int* mask;       // per column
  const BlockDev* blk;
  int n, w, m;  // the block's layers, the tile's columns, the middle layer
  size_t tile;
};

// tile x of block blockIdx.y; false where there is none to solve
__device__ __forceinline__ bool rtile_at(const BlockDev* __restrict__ tab,
                                         size_t x, RTile& t) {
  t.blk = tab + blockIdx.y;
  // (scheme-9 blocks only: a scheme-1 block assembled in FP32 is solved
  // in FP64 by vic_solve3_kernel)
  if (t.blk->implicit != 9 || !t.blk->implicit_f32) return false;
  const VicScratch S = vic_scratch(*t.blk);
  t.n = t.blk->nc1 - 2 * t.blk->ng;
  t.m = (t.n - 1) / 2;
  const VicScratch32 F = vic_scratch32(*t.blk, S, t.n);
  t.tile = x;
  if (x * 32 >= F.ncol) return false;
  t.w = VicTile::width(F.ncol, x);
  const size_t o25 = VicTile::base(25, x, t.n), o5 = VicTile::base(5, x, t.n);
  t.A = F.A + o25;
  t.B = F.B + o25;
  t.C = F.C + o25;
  t.PI = F.PI + o25;
  t.CP = F.CP + o25;
  t.R = F.R + o5;
  t.X0 = F.X0 + o5;
  t.DK = F.DK + o5;
  t.dk = F.dk;
  t.r64 = F.r64 + o5;
  t.E = F.E + x * 320;
  t.stat = F.stat + x * 192;
  t.mask = F.mask + x * 32;
  return true;
}

// the tile and the first of the eight layers that CTA blockIdx.x takes
__device__ __forceinline__ bool rtile_layers(const BlockDev* __restrict__ tab,
                                             RTile& t, int& i0) {
  const BlockDev& B = tab[blockIdx.y];
  const unsigned lg = (unsigned)(B.nc1 - 2 * B.ng + 7) / 8, x = blockIdx.x / lg;
  i0 = 8 * (int)(blockIdx.x - x * lg);
  return rtile_at(tab, x, t) && t.n >= 5;
}

// what the two warps of a tile trade: the upper side's relation at the
// middle, the middle's solution, each side's column flags and largest |x|
struct MeetSmem {
  float c[25][32], y[5][32], x[5][32];
  unsigned mx[2][32];
  int ok[2][32];
};

constexpr unsigned kInfBits = 0x7f800000u;
__device__ __forceinline__ unsigned largest(const float (&x)[5]) {
  unsigned m = 0;
#pragma unroll
  for (int r = 0; r < 5; ++r) m = max(m, __float_as_uint(x[r]) & 0x7fffffffu);
  return m;
}

// The rings' depth costs a big batch warps per SM and gains a small one
// nothing: the sweeps are bound by their instructions (64 members, us per
// launch when the depths were set: the correction 118 with 6 layers, two CTAs
// an SM, and 103 with 3, five; the first sweep 259 with 8 and 235 with 5; 384
// columns the same with 3 to 6)
constexpr int kFacBack = 5;  // layers in a warp's ring, the factor's way out
constexpr int kBackSlot = 800 + 160;
constexpr int kFacFloats = 2 * kFacBack * kBackSlot;  // both warps' rings
constexpr int kCorRing = 3;  // the correction's way in
constexpr int kCorSlot = 2 * 800 + 160;
constexpr int kCorBack = 5;  // and its way out
constexpr int kCorFloats = 2 * kCorRing * kCorSlot;
static_assert(kCorBack * kBackSlot <= kCorRing * kCorSlot, "ring");
// (within the 48 KB a CTA has without asking)
static_assert(4 * (kFacFloats > kCorFloats ? kFacFloats : kCorFloats) +
                      sizeof(MeetSmem) <= 48 * 1024, "shared memory");

// rows of N values of a lane's column straight from an array's layer
template <int N>
__device__ __forceinline__ void row_get(float (&v)[N], const float* g, int w) {
#pragma unroll
  for (int e = 0; e < N; ++e) v[e] = __ldcg(g + e * w);
}

// the way out from the middle of one side: x_i = y_i - C' x_prev for its cnt
// layers from the middle's neighbour to the wall, into X; the wall layer
// takes off e x[its third point].  y and C' arrive through a ring of RING
// layers.  Returns the bits of the largest |x| (at or above infinity's where
// one is not finite)
template <int RING>
__device__ __forceinline__ unsigned sweep_out(const float* CP, const float* Y,
                                              float* X, int c25, int c5, int w,
                                              int n, int cnt, bool up,
                                              const float (&e)[5], float (&x)[5],
                                              float* ring) {
  const int lane = threadIdx.x & 31;
  const bool on = lane < w;
  unsigned mx = 0;  // the bits order like the magnitudes, NaN above infinity
  const size_t first = up ? n - cnt : cnt - 1;  // the middle's neighbour
  const ptrdiff_t s25 = up ? c25 : -c25, s5 = up ? c5 : -c5;
  const float *gc = CP + first * c25 + 4 * lane, *gy = Y + first * c5 + 4 * lane;
  float* px = X + first * c5 + lane;
  const unsigned rb = smem_u32(ring) + 16 * lane;
  int islot = 0, gslot = 0, left = cnt;
  auto issue = [&]() {
    if (left > 0) {
      const unsigned q = rb + islot * (4 * kBackSlot);
      tile_fill(q, gc, c25, lane);
      tile_fill(q + 3200, gy, c5, lane);
      gc += s25;
      gy += s5;
      --left;
    }
    islot = islot + 1 == RING ? 0 : islot + 1;
    cpa_commit();
  };
  auto get = [&](float (&c)[25], float (&u)[5]) {
    const float* q = ring + gslot * kBackSlot + lane;
    gslot = gslot + 1 == RING ? 0 : gslot + 1;
    tile_get(c, q, w);
    tile_get(u, q + 800, w);
  };
  float p1 = x[0], p2 = x[0];  // the densities of the last two layers
  auto step = [&](int s, float (&c)[25], float (&u)[5], float (&nc)[25],
                  float (&nu)[5]) {
    cpa_wait<RING - 2>();  // the next layer is here
    __syncwarp();          // and this one's slot is read
    issue();
    get(nc, nu);
    msub5(c, x, u);
    if (s == 0) {
#pragma unroll
      for (int r = 0; r < 5; ++r) u[r] = fmaf(-e[r], p2, u[r]);
    }
    p2 = p1;
    p1 = u[0];
#pragma unroll
    for (int r = 0; r < 5; ++r) {
      x[r] = u[r];
      mx = max(mx, __float_as_uint(x[r]) & 0x7fffffffu);
    }
    if (on) {
#pragma unroll
      for (int r = 0; r < 5; ++r) px[r * w] = x[r];
    }
    px += s5;
  };
  float c0[25], u0[5], c1[25], u1[5];
#pragma unroll
  for (int j = 0; j < RING; ++j) issue();
  cpa_wait<RING - 1>();
  __syncwarp();
  get(c0, u0);
  for (int s = cnt - 1; s >= 0; s -= 2) {
    step(s, c0, u0, c1, u1);
    if (s > 0) step(s - 1, c1, u1, c0, u0);
  }
  cpa_wait<0>();
  return mx;
}

// The factors (the pivot blocks' inverses and C' or B') and the first
// solution of a tile, from both walls to the middle and back out.  A layer's
// A, near coupling and b are read into registers while the layer before it
// is eliminated, its far coupling while its own pivot is inverted: with a
// warp or two per scheduler nothing else hides those loads.  W: the tile's
// width at compile time (32), or 0 to take it from the tile
template <int W>
__device__ __forceinline__ void factor_tile(const RTile& T, const StageParams& p,
                                            MeetSmem& sm, float* ring) {
  const int w = W ? W : T.w, n = T.n, m = T.m;
  const int lane = threadIdx.x & 31;
  const bool up = threadIdx.x >= 32;
  const bool on = lane < w;
  const int at = on ? lane : 0;  // lanes past the tile shadow its first column
  const int c25 = VicTile::chunk(25, w), c5 = VicTile::chunk(5, w);
  const int cnt = up ? n - 1 - m : m;  // layers before the middle
  const float* near = up ? T.C : T.B;
  const float* far = up ? T.B : T.C;
  const double dtc = p.w2 * p.dt[blockIdx.y];
  const VicK K = vic_krows(*T.blk, n, up ? n - 1 : 0);
  const float k3 = narrow_exact(-(up ? K.t1 : K.t0) / dtc);
  auto layer = [&](int s) { return (size_t)(up ? n - 1 - s : s); };
  bool ok = true;
  float cp[25], y[5], e[5];
#pragma unroll
  for (int k = 0; k < 25; ++k) cp[k] = 0.f;
#pragma unroll
  for (int k = 0; k < 5; ++k) y[k] = e[k] = 0.f;
  auto get = [&](int s, float (&a)[25], float (&b)[25], float (&t)[5]) {
    row_get(b, near + layer(s) * c25 + at, w);
    row_get(a, T.A + layer(s) * c25 + at, w);
    row_get(t, T.R + layer(s) * c5 + at, w);
  };
  // one layer: a, b, t are the layer's, read by the step before; na, nb, nt
  // the next one's (the middle's after the last)
  auto step = [&](int s, float (&a)[25], float (&b)[25], float (&t)[5],
                  float (&na)[25], float (&nb)[25], float (&nt)[5]) {
    float cc[25];
    row_get(cc, far + layer(s) * c25 + at, w);
    get(s + 1, na, nb, nt);
#pragma unroll
    for (int k = 0; k < 5; ++k)
#pragma unroll
      for (int r = 0; r < 5; ++r)
#pragma unroll
        for (int c = 0; c < 5; ++c)
          a[5 * r + c] = fmaf(-b[5 * r + k], cp[5 * k + c], a[5 * r + c]);
    msub5(b, y, t);
    ok = invert5(a) && ok;
    mul5(a, t, y);
    if (s == 1) {  // the wall's third point is this layer's far neighbour
#pragma unroll
      for (int r = 0; r < 5; ++r)
#pragma unroll
        for (int k = 0; k < 5; ++k) cc[5 * r] = fmaf(-b[5 * r + k], e[k], cc[5 * r]);
    }
#pragma unroll
    for (int r = 0; r < 5; ++r)
#pragma unroll
      for (int c = 0; c < 5; ++c) {
        float q = a[5 * r] * cc[c];
#pragma unroll
        for (int k = 1; k < 5; ++k) q = fmaf(a[5 * r + k], cc[5 * k + c], q);
        cp[5 * r + c] = q;
      }
    if (s == 0) {
#pragma unroll
      for (int r = 0; r < 5; ++r) e[r] = k3 * a[5 * r + 4];
    }
    if (on) {
      float* pi = T.PI + layer(s) * c25 + lane;
      float* co = T.CP + layer(s) * c25 + lane;
#pragma unroll
      for (int k = 0; k < 25; ++k) pi[k * w] = a[k];
#pragma unroll
      for (int k = 0; k < 25; ++k) co[k * w] = cp[k];
#pragma unroll
      for (int r = 0; r < 5; ++r) T.R[layer(s) * c5 + r * w + lane] = y[r];
    }
  };
  float a0[25], b0[25], t0[5], a1[25], b1[25], t1[5];
  get(0, a0, b0, t0);
  for (int s = 0; s < cnt; s += 2) {
    step(s, a0, b0, t0, a1, b1, t1);
    if (s + 1 < cnt) {
      step(s + 1, a1, b1, t1, a0, b0, t0);
    } else {
#pragma unroll
      for (int k = 0; k < 25; ++k) a0[k] = a1[k], b0[k] = b1[k];
#pragma unroll
      for (int k = 0; k < 5; ++k) t0[k] = t1[k];
    }
  }
  if (on) {
#pragma unroll
    for (int r = 0; r < 5; ++r) T.E[(up ? 5 + r : r) * w + lane] = e[r];
  }
  // the middle, on the lower warp (its a, b, t are in hand)
  float x[5];
  if (up) {
#pragma unroll
    for (int k = 0; k < 25; ++k) sm.c[k][lane] = cp[k];
#pragma unroll
    for (int r = 0; r < 5; ++r) sm.y[r][lane] = y[r];
  }
  __syncthreads();
  if (!up) {
    float cc[25];
    row_get(cc, T.C + (size_t)m * c25 + at, w);
    msub5(b0, y, t0);
#pragma unroll
    for (int r = 0; r < 5; ++r) y[r] = sm.y[r][lane];
    msub5(cc, y, t0);
#pragma unroll
    for (int k = 0; k < 5; ++k)
#pragma unroll
      for (int c = 0; c < 5; ++c) {
        const float cu = sm.c[5 * k + c][lane];
#pragma unroll
        for (int r = 0; r < 5; ++r)
          a0[5 * r + c] = fmaf(-cc[5 * r + k], cu,
                               fmaf(-b0[5 * r + k], cp[5 * k + c], a0[5 * r + c]));
      }
    ok = invert5(a0) && ok;
    mul5(a0, t0, x);
    if (on) {
#pragma unroll
      for (int k = 0; k < 25; ++k) T.PI[(size_t)m * c25 + k * w + lane] = a0[k];
#pragma unroll
      for (int r = 0; r < 5; ++r) T.X0[(size_t)m * c5 + r * w + lane] = x[r];
    }
#pragma unroll
    for (int r = 0; r < 5; ++r) sm.x[r][lane] = x[r];
  }
  __syncthreads();
  if (up) {
#pragma unroll
    for (int r = 0; r < 5; ++r) x[r] = sm.x[r][lane];
  }
  unsigned mx = largest(x);
  mx = max(mx, sweep_out<kFacBack>(T.CP, T.R, T.X0, c25, c5, w, n, cnt, up, e, x,
                                   ring + (up ? kFacBack * kBackSlot : 0)));
  sm.mx[up][lane] = mx;
  sm.ok[up][lane] = ok;
  __syncthreads();
  if (up || !on) return;
  mx = max(mx, sm.mx[1][lane]);
  T.stat[lane * 6] = __uint_as_float(mx);
  T.mask[lane] = sm.ok[0][lane] && sm.ok[1][lane] ? 0 : 1;
}

__global__ void __launch_bounds__(64)
    vic_factor32_kernel(const BlockDev* __restrict__ tab, StageParams p) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ MeetSmem sm;
  RTile T;
  if (!rtile_at(tab, blockIdx.x, T)) return;
  if (T.n < 5) {  // too few layers (see above): the FP64 solve, not counted
    if (threadIdx.x < T.w) T.mask[threadIdx.x] = 2;
    return;
  }
  float* ring = reinterpret_cast<float*>(smem_raw);
  if (T.w == 32)
    factor_tile<32>(T, p, sm, ring);
  else
    factor_tile<0>(T, p, sm, ring);
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
// * The first correction's (corr 1) is b - T x, x the first solution: T x
//   as a sum of exact float products (tf_madd, on the FP32 pipe, to about
//   2^-72 of the sum of |t x|), then b minus that sum in FP64 (three
//   subtractions, the first exact).
// * A later one is the previous r less T d, d the FP32 correction x grew by:
//   T d in float-float on the FP32 pipe (its error, 2^-48 of the sum of
//   |t d| with |d| about 2^-22 |x|, is far below the FP64 rounding of r).
// Every load is a tile's row of 32 consecutive values.
template <bool FIRST, int W>
__device__ __forceinline__ void residual_row(const RTile& T, int i, int corr,
                                             bool keep, double dtc) {
  const int w = W ? W : T.w, n = T.n;
  const int lane = threadIdx.x & 31;
  if (lane >= w) return;
  const int c25 = VicTile::chunk(25, w), c5 = VicTile::chunk(5, w);
  const float* X = (FIRST ? T.X0 : T.DK + (size_t)(corr - 2) * T.dk) + lane;
  double* r64 = T.r64 + (size_t)i * 5 * w + lane;
  double t[5];
#pragma unroll
  for (int r = 0; r < 5; ++r) t[r] = r64[r * w];
  float sh[5] = {0.f, 0.f, 0.f, 0.f, 0.f}, mh[5] = {0.f, 0.f, 0.f, 0.f, 0.f},
        ml[5] = {0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int m = 0; m < 3; ++m) {  // the cell, below, above
    if ((m == 1 && i == 0) || (m == 2 && i == n - 1)) continue;
    const size_t e = (size_t)(m == 0 ? i : (m == 1 ? i - 1 : i + 1)) * c5;
    float x[5];
#pragma unroll
    for (int k = 0; k < 5; ++k) x[k] = X[e + k * w];
    const float* M = (m == 0 ? T.A : (m == 1 ? T.B : T.C)) + (size_t)i * c25 + lane;
    if (FIRST) {
#pragma unroll
      for (int r = 0; r < 5; ++r)
#pragma unroll
        for (int k = 0; k < 5; ++k)
          tf_madd(sh[r], mh[r], ml[r], M[(5 * r + k) * w], x[k]);
    } else {
#pragma unroll
      for (int r = 0; r < 5; ++r)
#pragma unroll
        for (int k = 0; k < 5; ++k)
          ff_madd(sh[r], mh[r], M[(5 * r + k) * w], x[k]);
    }
  }
#pragma unroll
  for (int r = 0; r < 5; ++r) t[r] = (t[r] - widen_exact(sh[r])) - widen_exact(mh[r]);
  if (FIRST) {  // (a later one leaves ml at zero)
#pragma unroll
    for (int r = 0; r < 5; ++r) t[r] = t[r] - widen_exact(ml[r]);
  }
  // the wall rows' third points
  if (i == 0)
    t[4] -= (-vic_krows(*T.blk, n, 0).t0 / dtc) * widen_exact(X[(size_t)2 * c5]);
  if (i == n - 1)
    t[4] -= (-vic_krows(*T.blk, n, n - 1).t1 / dtc) *
            widen_exact(X[(size_t)(n - 3) * c5]);
#pragma unroll
  for (int r = 0; r < 5; ++r) {
    if (keep) r64[r * w] = t[r];
    T.R[(size_t)i * c5 + lane + r * w] = narrow_exact(t[r]);
  }
}

// eight layers of a tile per CTA
template <bool FIRST>
__global__ void __launch_bounds__(kThreads, 3)
    vic_residual_kernel(const BlockDev* __restrict__ tab, StageParams p,
                        int corr) {
  RTile T;
  int i0;
  if (!rtile_layers(tab, T, i0)) return;
  const int i = i0 + (threadIdx.x >> 5);
  if (i >= T.n) return;
  const bool keep = corr < p.refine;  // a later correction reads r
  const double dtc = p.w2 * p.dt[blockIdx.y];
  if (T.w == 32)
    residual_row<FIRST, 32>(T, i, corr, keep, dtc);
  else
    residual_row<FIRST, 0>(T, i, corr, keep, dtc);
}

// A correction's sweeps of a tile, the factor's on r with its factors, and
// after the last one the column's acceptance: the error it leaves is about
// |d| rho, rho = |d| / |d_prev| the observed contraction, accepted at or
// below p.accept of the largest |x|
template <int W>
__device__ __forceinline__ void correct_tile(const RTile& T, const StageParams& p,
                                             int corr, MeetSmem& sm, float* ring) {
  const int w = W ? W : T.w, n = T.n, m = T.m;
  const int lane = threadIdx.x & 31;
  const bool up = threadIdx.x >= 32;
  const bool on = lane < w;
  const int at = on ? lane : 0;
  const int c25 = VicTile::chunk(25, w), c5 = VicTile::chunk(5, w);
  const int cnt = up ? n - 1 - m : m;
  const int steps = up ? cnt : cnt + 1;  // the lower warp's last: the middle
  const float* near = up ? T.C : T.B;
  float* X = T.DK + (size_t)(corr - 1) * T.dk;
  ring += up ? kCorRing * kCorSlot : 0;
  float e[5];
#pragma unroll
  for (int r = 0; r < 5; ++r) e[r] = T.E[(up ? 5 + r : r) * w + at];

  const ptrdiff_t s25 = up ? -c25 : c25, s5 = up ? -c5 : c5;
  const size_t first = up ? n - 1 : 0;
  const float *gp = T.PI + first * c25 + 4 * lane, *gn = near + first * c25 + 4 * lane;
  const float* gr = T.R + first * c5 + 4 * lane;
  float* py = T.R + first * c5 + lane;
  const unsigned rb = smem_u32(ring) + 16 * lane;
  int islot = 0, gslot = 0, left = steps;
  auto issue = [&]() {
    if (left > 0) {
      const unsigned q = rb + islot * (4 * kCorSlot);
      tile_fill(q, gp, c25, lane);
      tile_fill(q + 3200, gn, c25, lane);
      tile_fill(q + 6400, gr, c5, lane);
      gp += s25;
      gn += s25;
      gr += s5;
      --left;
    }
    islot = islot + 1 == kCorRing ? 0 : islot + 1;
    cpa_commit();
  };
  auto get = [&](float (&pi)[25], float (&b)[25], float (&t)[5]) {
    const float* q = ring + gslot * kCorSlot + lane;
    gslot = gslot + 1 == kCorRing ? 0 : gslot + 1;
    tile_get(b, q + 800, w);
    tile_get(t, q + 1600, w);
    tile_get(pi, q, w);
  };
  float y[5] = {0.f, 0.f, 0.f, 0.f, 0.f};
  auto step = [&](float (&pi)[25], float (&b)[25], float (&t)[5],
                  float (&npi)[25], float (&nb)[25], float (&nt)[5]) {
    cpa_wait<kCorRing - 2>();  // the next layer is here
    __syncwarp();              // and this one's slot is read
    issue();
    get(npi, nb, nt);
    msub5(b, y, t);
    mul5(pi, t, y);
    if (on) {
#pragma unroll
      for (int r = 0; r < 5; ++r) py[r * w] = y[r];
    }
    py += s5;
  };
#pragma unroll
  for (int j = 0; j < kCorRing; ++j) issue();
  float p0[25], b0[25], t0[5], p1[25], b1[25], t1[5];
  cpa_wait<kCorRing - 1>();
  __syncwarp();
  get(p0, b0, t0);
  for (int s = 0; s < cnt; s += 2) {
    step(p0, b0, t0, p1, b1, t1);
    if (s + 1 < cnt) {
      step(p1, b1, t1, p0, b0, t0);
    } else {
#pragma unroll
      for (int k = 0; k < 25; ++k) p0[k] = p1[k], b0[k] = b1[k];
#pragma unroll
      for (int k = 0; k < 5; ++k) t0[k] = t1[k];
    }
  }
  cpa_wait<0>();
  if (up) {
#pragma unroll
    for (int r = 0; r < 5; ++r) sm.y[r][lane] = y[r];
  } else {
    row_get(b1, T.C + (size_t)m * c25 + at, w);
  }
  __syncthreads();
  float x[5];
  if (!up) {
    msub5(b0, y, t0);
#pragma unroll
    for (int r = 0; r < 5; ++r) y[r] = sm.y[r][lane];
    msub5(b1, y, t0);
    mul5(p0, t0, x);
    if (on) {
#pragma unroll
      for (int r = 0; r < 5; ++r) X[(size_t)m * c5 + r * w + lane] = x[r];
    }
#pragma unroll
    for (int r = 0; r < 5; ++r) sm.x[r][lane] = x[r];
  }
  __syncthreads();
  if (up) {
#pragma unroll
    for (int r = 0; r < 5; ++r) x[r] = sm.x[r][lane];
  }
  unsigned mx = largest(x);
  mx = max(mx, sweep_out<kCorBack>(T.CP, T.R, X, c25, c5, w, n, cnt, up, e, x, ring));
  sm.mx[up][lane] = mx;
  __syncthreads();
  if (up || !on) return;
  mx = max(mx, sm.mx[1][lane]);
  float* st = T.stat + lane * 6;
  const float dl = __uint_as_float(mx), dp = st[corr - 1];
  st[corr] = dl;
  bool fin = mx < kInfBits;
  if (corr == p.refine) {
    const float rho = dp > 0.f ? fminf(dl / dp, 1.f) : 0.f;
    fin = fin && dl * rho <= p.accept * st[0];
  }
  if (!fin) T.mask[lane] = 1;
}

__global__ void __launch_bounds__(64)
    vic_correct32_kernel(const BlockDev* __restrict__ tab, StageParams p,
                         int corr) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ MeetSmem sm;
  RTile T;
  if (!rtile_at(tab, blockIdx.x, T) || T.n < 5) return;
  float* ring = reinterpret_cast<float*>(smem_raw);
  if (T.w == 32)
    correct_tile<32>(T, p, corr, sm, ring);
  else
    correct_tile<0>(T, p, corr, sm, ring);
}

// D = x0 + d1 + ... in FP64, eight layers of a tile per CTA: read by rows of
// columns, written by columns (40 consecutive values) through shared memory
__global__ void __launch_bounds__(kThreads)
    vic_sum_kernel(const BlockDev* __restrict__ tab, StageParams p) {
  __shared__ double s[32][41];
  RTile T;
  int i0;
  if (!rtile_layers(tab, T, i0)) return;
  const int lane = threadIdx.x & 31, q = threadIdx.x >> 5, w = T.w;
  const int nk = p.refine;
  if (i0 + q < T.n && lane < w) {
    const size_t o = (size_t)(i0 + q) * VicTile::chunk(5, w) + lane;
    float x[4][5];
#pragma unroll
    for (int r = 0; r < 5; ++r) {
      x[0][r] = T.X0[o + r * w];
#pragma unroll
      for (int k = 1; k < 4; ++k)
        x[k][r] = k <= nk ? T.DK[(size_t)(k - 1) * T.dk + o + r * w] : 0.f;
    }
#pragma unroll
    for (int r = 0; r < 5; ++r) {
      double sum = widen_exact(x[0][r]);
#pragma unroll
      for (int k = 1; k < 4; ++k)
        if (k <= nk) sum += widen_exact(x[k][r]);
      s[lane][5 * q + r] = sum;
    }
  }
  __syncthreads();
  const VicScratch S = vic_scratch(*T.blk);
  const int len = 5 * min(8, T.n - i0);
  double* D = S.D + (T.tile * 32 * T.n + i0) * 5;
  for (int e = threadIdx.x; e < w * len; e += kThreads) {
    const int c = e / len, k = e - c * len;
    D[(size_t)c * T.n * 5 + k] = s[c][k];
  }
}
