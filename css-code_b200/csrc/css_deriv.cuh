// css_deriv.cuh -- whole-field compact derivatives (css_deriv, the terms of
// the explicit viscosity and the radiative diffusion, torch.ops.css.deriv)
// and their adjoints.
//
// Every kernel gives a line to a lane and 32 lines to a warp.  Along r and phi
// the 32 lines are consecutive theta, so a lane reads its line straight from
// global memory (256 bytes a warp load) into registers, solves it and stores
// it: nothing is staged.  Along theta a warp transposes its 32 lines through a
// tile.  The floor of a pass is HBM (a field in, a field out: 268 MB, 41 us at
// 6550 GB/s on 128x256x512).  Measured there, r / theta / phi: 53 / 81 / 41 us
// forward and 55 / 78 / 65 us adjoint, against 297 / 235 / 253 us with 16-line
// tiles staged in shared memory (16 of 128 threads solving) and 1410 us for an
// adjoint that gathered a dense 32 x 40 block column per point.  What keeps
// the others off the floor is the latency of their loads at 7 to 14 warps an
// SM (146 to 254 registers, or the theta tiles' shared memory): 3.8 to 6.4 of
// the cycles between two issues.
#pragma once
#include "css_kernels.cuh"

namespace css {

// one derivative of a launch: out = d^order x with the closures of bdry and
// the face data lo / hi (NULL: zero)
struct DerivItem {
  const double *x;
  double *out;
  const double *lo, *hi;
  int bdry, order;
};
constexpr int DERIV_MAX = 8;  // derivatives of one launch (grid z)
struct DerivBatch {
  DerivItem it[DERIV_MAX];
};

constexpr int DV_NT = 128;

// index maps of a line read from global memory, j 1-based from the block's
// first point; along phi the halo of the first and last block wraps
struct GlobR {
  long long s;
  __device__ __forceinline__ long long operator()(int j) const { return (j - 1) * s; }
};
template <int M>
struct GlobP {
  int s, m, lo, hi;  // lo / hi: what a halo point below / above adds
  __device__ __forceinline__ int operator()(int j) const {
    const int mm = M > 0 ? M : m;
    return (j - 1) * s + (j < 1 ? lo : (j > mm ? hi : 0));
  }
};
struct GlobOut {
  long long s;
  __device__ __forceinline__ long long operator()(int j) const { return j * s; }
};

// 8 bytes from global to shared memory without a register between
__device__ __forceinline__ void cp_async8(double *dst, const double *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }
// k / d of 0 <= k < 32 * 264 by a multiplication (inv = inv_of(d), d <= 264)
__device__ __forceinline__ unsigned inv_of(int d) { return 0xFFFFFFFFu / (unsigned)d + 1u; }
__device__ __forceinline__ int div_by(int k, unsigned inv) { return (int)__umulhi((unsigned)k, inv); }

// A line of run-time length m >= 10: line_solve_a's arithmetic with the
// forward values in a column of shared memory (t[j * ts], which may be the
// output column itself, or the input line where that is as dense: point j is
// read before row j is written) and the interior points read once, four ahead
// of the row that needs them.
template <int ORDER, class P, class X, class O>
__device__ __forceinline__ void line_solve_g(P xb, const X &xi, int m, int dtype, int bdry,
                                             double bclo, double bchi, const double *__restrict__ G, int gs,
                                             double dnum, double scale, int phi, double *t, int ts, double *ob,
                                             const O &oi) {
  const double *g1 = G, *g2 = G + gs, *g3 = G + 2 * gs;
  const double a1 = (ORDER == 1) ? -1.0 / 3.0 : -2.0 / 11.0;
  double r1, r2, rm1, rm;
  if (ORDER == 1) {
    r2 = d1_row_lo2(xb, xi, dtype);
    r1 = d1_row_lo1(xb, xi, dtype, bdry, bclo, dnum, r2);
    rm1 = d1_row_hi1(xb, xi, m, dtype);
    rm = d1_row_hi2(xb, xi, m, dtype, bdry, bchi, dnum, rm1);
  } else {
    r1 = d2_row_lo1(xb, xi, dtype, bdry, bclo, dnum);
    r2 = d2_row_lo2(xb, xi, dtype);
    rm1 = d2_row_hi1(xb, xi, m, dtype);
    rm = d2_row_hi2(xb, xi, m, dtype, bdry, bchi, dnum);
  }
  double w[8];  // x(j-2) .. x(j+1) of the next row, then the four points after them
#pragma unroll
  for (int k = 0; k < 8; k++) w[k] = xb[xi(k + 1)];
  double v = __ldg(g2 + 1) * r1;
  t[0] = v;
  v = phi ? __ldg(g2 + 2) * (r2 + a1 * v) : __ldg(g2 + 2) * r2 + __ldg(g3 + 2) * v;
  t[ts] = v;
  for (int j = 3; j <= m - 2; j += 4) {
    double nx[4], c[4];  // c: the rows' coefficients (a table holds m + 2)
#pragma unroll
    for (int k = 0; k < 4; k++) nx[k] = j + 6 + k <= m ? xb[xi(j + 6 + k)] : 0.0;
#pragma unroll
    for (int k = 0; k < 4; k++) c[k] = __ldg(g2 + j + k);
#pragma unroll
    for (int k = 0; k < 4; k++) {
      if (j + k <= m - 2) {
        const double d =
            ORDER == 1 ? (7.0 / 9.0) * (w[k + 3] - w[k + 1]) + (1.0 / 36.0) * (w[k + 4] - w[k])
                       : HaloD2::c1 * (w[k + 3] - 2.0 * w[k + 2] + w[k + 1]) +
                             HaloD2::c2 * (w[k] - 2.0 * w[k + 2] + w[k + 4]);
        v = c[k] * (d + a1 * v);
        t[(j + k - 1) * ts] = v;
      }
    }
#pragma unroll
    for (int k = 0; k < 4; k++) {
      w[k] = w[k + 4];
      w[k + 4] = nx[k];
    }
  }
  if (phi) {
    v = __ldg(g2 + m - 1) * (rm1 + a1 * v);
    t[(m - 2) * ts] = v;
    v = __ldg(g2 + m) * (rm + a1 * v);
  } else {
    v = __ldg(g2 + m - 1) * rm1 + __ldg(g3 + m - 1) * v;
    t[(m - 2) * ts] = v;
    v = __ldg(g2 + m) * rm + __ldg(g3 + m) * v;
  }
  ob[oi(m - 1)] = scale * v;
  for (int j0 = m - 1; j0 >= 1; j0 -= 4) {  // four rows' values in hand before the chain
    double q[4], c[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const int j = max(j0 - k, 1);
      q[k] = t[(j - 1) * ts];
      c[k] = __ldg(g1 + j + 1);
    }
#pragma unroll
    for (int k = 0; k < 4; k++)
      if (j0 - k >= 1) {
        v = q[k] + c[k] * v;
        ob[oi(j0 - k - 1)] = scale * v;
      }
  }
}

// Derivatives along r (DIR 0) or phi (DIR 2).  grid: x = lines / DV_NT, y =
// block, z = derivative.  M: block length when all are 16 or 32 points long
// (the line in registers), 0: run-time lengths (forward values in shared
// memory, maxm doubles a thread; the block size is chosen so that they fit).
template <int DIR, int M>
__global__ void __launch_bounds__(DV_NT, M == 32 ? 3 : 4) k_deriv_s(CssGeo g, const __grid_constant__ DerivBatch B) {
  extern __shared__ double sm[];
  const DerivItem &I = B.it[blockIdx.z];
  const CssDir &D = g.d[DIR];
  const int b = blockIdx.y, m = M > 0 ? M : D.size[b], a0 = D.start[b];
  const int nlines = DIR == 0 ? g.nth * g.nphi : g.nth * g.nr;
  const int line = blockIdx.x * blockDim.x + threadIdx.x;
  if (line >= nlines) return;
  const long long s = DIR == 0 ? (long long)g.nth * g.nphi : g.nth;
  const long long base = (DIR == 0 ? line : line % g.nth + (long long)(line / g.nth) * g.nth * g.nphi) + a0 * s;
  const int dtype = DIR == 0 ? dtype_of(D, b) : 3, bdry = DIR == 0 ? I.bdry : 0;
  double lo = 0.0, hi = 0.0;
  if (DIR == 0) {
    if (D.lphys[b] && I.lo) lo = __ldg(I.lo + line);
    if (D.rphys[b] && I.hi) hi = __ldg(I.hi + line);
  }
  const double dn = D.dnum[b], sc = I.order == 1 ? dn : dn * dn;
  const double *G = tabp(g, DIR, b, I.order, bdry);
  const int wrap = g.nth * g.nphi;
  const GlobR xr{s};
  const GlobP<M> xp{g.nth, m, a0 == 0 ? wrap : 0, a0 + m == g.nphi ? -wrap : 0};
  auto go = [&](auto ord, const auto &xi) {
    constexpr int ORD = decltype(ord)::value;
    if constexpr (M > 0)
      line_solve_c<ORD, M>(I.x + base, xi, dtype, bdry, lo, hi, G, g.tstride, dn, sc, DIR == 2, I.out + base,
                           GlobOut{s});
    else
      line_solve_g<ORD>(I.x + base, xi, m, dtype, bdry, lo, hi, G, g.tstride, dn, sc, DIR == 2, sm + threadIdx.x,
                        blockDim.x, I.out + base, GlobOut{s});
  };
  auto both = [&](const auto &xi) {
    if (I.order == 1) go(std::integral_constant<int, 1>{}, xi);
    else go(std::integral_constant<int, 2>{}, xi);
  };
  if constexpr (DIR == 0) both(xr);
  else both(xp);
}

// doubles of shared memory a warp's theta tile takes: 32 lines with their
// halos, then 32 solved lines; both strides odd, so the 32 lanes of a solve
// touch distinct banks.  Lines of run-time length are solved in place.
__host__ __device__ constexpr int dv_theta_in(int m) { return (m + 8) | 1; }
__host__ __device__ constexpr int dv_theta_out(int m) { return m | 1; }
__host__ __device__ constexpr int dv_theta_warp(int m, bool fixed) {
  return 32 * (dv_theta_in(m) + (fixed ? dv_theta_out(m) : 0));
}

// Derivatives along theta.  grid: x = groups of 32 lines / tiles a CTA, y =
// block, z = derivative.  A line is a (phi, r) row; consecutive rows are
// contiguous in memory.  M > 0: a warp has its own tile, two a CTA.  M = 0: a
// CTA of 128 threads brings one tile by asynchronous copies and stores it, its
// first warp solves it in place: 21 us on 64x500x96 in theta blocks of 100
// points and 16.5 us on 20x200x30, where a warp that loaded, solved into a
// second tile and stored alone took 86 and 45 us.
template <int M>
__global__ void __launch_bounds__(M > 0 ? 64 : 128) k_deriv_t(CssGeo g, const __grid_constant__ DerivBatch B) {
  extern __shared__ double sm[];
  const DerivItem &I = B.it[blockIdx.z];
  const CssDir &D = g.d[1];
  const int b = blockIdx.y, m = M > 0 ? M : D.size[b], t0 = D.start[b];
  const int lane = threadIdx.x & 31, nlines = g.nphi * g.nr, nth = g.nth;
  const int row0 = (M > 0 ? blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5) : blockIdx.x) * 32;
  if (row0 >= nlines) return;
  const int SI = dv_theta_in(m), SO = dv_theta_out(m), w = m + 8;
  double *X = sm + (M > 0 ? (size_t)(threadIdx.x >> 5) * dv_theta_warp(M, true) : 0), *O = X + 32 * SI;
  const double *src = I.x + (size_t)row0 * nth + t0 - 4;
  const int nrow = min(32, nlines - row0);
  if constexpr (M > 0) {
    // every load of the tile is issued before the first store to it
    constexpr int W = M + 8, H = W / 2;
#pragma unroll
    for (int h = 0; h < 2; h++) {
      double v[H];
#pragma unroll
      for (int k = 0; k < H; k++) {
        const int idx = lane + 32 * (k + h * H), l = idx / W, c = idx - l * W, t = t0 - 4 + c;
        v[k] = l < nrow && t >= 0 && t < nth ? __ldg(src + (size_t)l * nth + c) : 0.0;
      }
#pragma unroll
      for (int k = 0; k < H; k++) {
        const int idx = lane + 32 * (k + h * H), l = idx / W, c = idx - l * W;
        X[l * SI + c] = v[k];
      }
    }
  } else {
    const unsigned inv = inv_of(w);
    for (int k = threadIdx.x; k < nrow * w; k += blockDim.x) {
      const int l = div_by(k, inv), c = k - l * w, t = t0 - 4 + c;
      if (t >= 0 && t < nth) cp_async8(X + l * SI + c, src + (size_t)l * nth + c);
      else X[l * SI + c] = 0.0;
    }
    cp_async_wait();
    __syncthreads();
  }
  __syncwarp();
  const int row = row0 + lane;
  if (row < nlines && (M > 0 || threadIdx.x < 32)) {
    const double lo = (D.lphys[b] && I.lo) ? __ldg(I.lo + row) : 0.0;
    const double hi = (D.rphys[b] && I.hi) ? __ldg(I.hi + row) : 0.0;
    const int dtype = dtype_of(D, b), ir = row / g.nphi;
    double *const x = X + lane * SI + 4;
    const double *G = tabp(g, 1, b, I.order, I.bdry);
    const double dn = D.dnum[b];
    // D2bydt2's Neumann datum takes the radial spacing
    if (I.order == 1) {
      if constexpr (M > 0)
        line_solve_c<1, M>(x, StridedIn{1}, dtype, I.bdry, lo, hi, G, g.tstride, dn, dn, 0, O + lane * SO,
                           StridedOut{1});
      else
        line_solve_g<1>((const double *)x, StridedIn{1}, m, dtype, I.bdry, lo, hi, G, g.tstride, dn, dn, 0, x, 1, x,
                        StridedOut{1});
    } else {
      const double d2 = dnum_d2_theta(g, ir);
      if constexpr (M > 0)
        line_solve_c<2, M>(x, StridedIn{1}, dtype, I.bdry, lo, hi, G, g.tstride, d2, dn * dn, 0, O + lane * SO,
                           StridedOut{1});
      else
        line_solve_g<2>((const double *)x, StridedIn{1}, m, dtype, I.bdry, lo, hi, G, g.tstride, d2, dn * dn, 0, x, 1,
                        x, StridedOut{1});
    }
  }
  if (M > 0) __syncwarp();
  else __syncthreads();
  double *dst = I.out + (size_t)row0 * nth + t0;
  if constexpr (M == 32) {
#pragma unroll 8
    for (int l = 0; l < nrow; l++) dst[(size_t)l * nth + lane] = O[l * SO + lane];
  } else {
    const double *const o = M > 0 ? O : X + 4;
    const int so = M > 0 ? SO : SI;
    const unsigned inv = inv_of(m);
    for (int k = M > 0 ? lane : threadIdx.x; k < nrow * m; k += M > 0 ? 32 : blockDim.x) {
      const int l = div_by(k, inv), c = k - l * m;
      dst[(size_t)l * nth + c] = o[l * so + c];
    }
  }
}

// ---------------------------------------------------------------------------
// Adjoint (the backward of torch.ops.css.deriv): gx = D^T g with zero
// boundary data.  A block's derivative is scale * U^-1 L^-1 R x: rows R over
// its m points and the four halo points on either side, then the two Thomas
// sweeps.  So gx = R^T L^-T U^-T (scale g): the sweeps transposed, O(1) a
// point, then the rows transposed.  R's interior rows are the five-point
// stencils; its first two and last two rows (halo or physical closures) come
// as tables E of 4 x 12 coefficients, rows 1 and 2 over columns -3..8 and
// rows m-1 and m over columns m-7..m+4, which the host reads off the same
// row functions with unit inputs.
//
// A lane walks a whole line block by block, because a block also feeds the
// last four points of the block before it and the first four of the one
// after it: what it adds above is carried to the next block, and its own
// last four points wait for the next block's addition below.  Along phi the
// walk closes on itself: the first block's first four points wait for the
// last block.  The order of every sum is fixed.
// ---------------------------------------------------------------------------
constexpr int ADJ_W = 12;
constexpr int ADJ_TAB = 4 * ADJ_W;  // doubles of a block's edge table
// doubles of a theta row: four waiting points, then the block; odd
__host__ __device__ constexpr int adj_theta_stride(int m) { return (m + 4) | 1; }

// One block: incoming gradients in t[k * ts] (k = 0 .. m-1).  On return t
// holds this block's part of gx at its own points, lo[4] what it adds to the
// four points below (nearest last) and hi[4] to the four above.  M > 0: the
// block length at compile time, t a register array (ts 1); M = 0: t in
// shared memory, four points read ahead of the chain that uses them.
template <int ORDER, int M>
__device__ __forceinline__ void adj_block(double *t, int ts, int m_, const double *__restrict__ G, int gs,
                                          const double *__restrict__ E, double scale, double lo[4], double hi[4]) {
  // run-time lengths: four rows' points and coefficients in hand before the chain
  constexpr int CH = M > 0 ? M : 4;
  const int m = M > 0 ? M : m_;
  const double *g1 = G, *g2 = G + gs, *g3 = G + 2 * gs;
  double v = 0.0;
  for (int j0 = 1; j0 <= m; j0 += CH) {  // U^-T, ascending
    double q[CH], c[4];
#pragma unroll
    for (int k = 0; k < CH; k++) q[k] = j0 + k <= m ? t[(j0 + k - 1) * ts] : 0.0;
    if constexpr (M == 0) {
#pragma unroll
      for (int k = 0; k < 4; k++) c[k] = __ldg(g1 + min(j0 + k, m));
    }
#pragma unroll
    for (int k = 0; k < CH; k++)
      if (j0 + k <= m) {
        v = j0 + k > 1 ? q[k] + (M > 0 ? __ldg(g1 + j0 + k) : c[k & 3]) * v : q[k];
        t[(j0 + k - 1) * ts] = v;
      }
  }
  v = 0.0;
  for (int j0 = m; j0 >= 1; j0 -= CH) {  // L^-T, descending
    double q[CH], c[4], d[4];
#pragma unroll
    for (int k = 0; k < CH; k++) q[k] = j0 - k >= 1 ? t[(j0 - k - 1) * ts] : 0.0;
    if constexpr (M == 0) {
#pragma unroll
      for (int k = 0; k < 4; k++) {
        const int j = max(j0 - k, 1);
        c[k] = __ldg(g3 + j + 1);
        d[k] = __ldg(g2 + j);
      }
    }
#pragma unroll
    for (int k = 0; k < CH; k++)
      if (j0 - k >= 1) {
        v = j0 - k < m ? q[k] + (M > 0 ? __ldg(g3 + j0 - k + 1) : c[k & 3]) * v : q[k];
        t[(j0 - k - 1) * ts] = (scale * (M > 0 ? __ldg(g2 + j0 - k) : d[k & 3])) * v;
      }
  }
  const double y1 = t[0], y2 = t[ts], ym1 = t[(m - 2) * ts], ym = t[(m - 1) * ts];
#pragma unroll
  for (int k = 0; k < 4; k++) {
    lo[k] = __ldg(E + k) * y1 + __ldg(E + ADJ_W + k) * y2;
    hi[k] = __ldg(E + 2 * ADJ_W + 8 + k) * ym1 + __ldg(E + 3 * ADJ_W + 8 + k) * ym;
  }
  // R^T: the interior rows 3 .. m-2, then the edge rows' columns; a .. d are
  // y(k-2) .. y(k+1) of the interior rows
  double a = 0.0, b = 0.0, c = 0.0, d = 0.0;
  for (int j0 = 1; j0 <= m; j0 += CH) {
    double q[CH];
#pragma unroll
    for (int k = 0; k < CH; k++) q[k] = j0 + k <= m - 4 ? t[(j0 + k + 1) * ts] : 0.0;  // y(j + 2)
#pragma unroll
    for (int k = 0; k < CH; k++) {
      const int j = j0 + k;
      if (j <= m) {
        const double e = q[k];
        double z = ORDER == 1 ? (7.0 / 9.0) * (b - d) + (1.0 / 36.0) * (a - e)
                              : HaloD2::c1 * (b - 2.0 * c + d) + HaloD2::c2 * (a - 2.0 * c + e);
        if (j <= 8) z += __ldg(E + 3 + j) * y1 + __ldg(E + ADJ_W + 3 + j) * y2;
        if (j >= m - 7) z += __ldg(E + 2 * ADJ_W + j - m + 7) * ym1 + __ldg(E + 3 * ADJ_W + j - m + 7) * ym;
        t[(j - 1) * ts] = z;
        a = b; b = c; c = d; d = e;
      }
    }
  }
}

// Adjoint along r (DIR 0) or phi (DIR 2): 32 consecutive theta a warp.  M:
// every block 16 or 32 points long (the block in registers); 0: run-time
// lengths (a column of shared memory, maxm doubles a thread).
template <int DIR, int ORDER, int M>
__global__ void __launch_bounds__(DV_NT) k_adj_s(CssGeo g, const double *__restrict__ E,
                                                 const double *__restrict__ gin, double *__restrict__ gout, int bdry) {
  extern __shared__ double sm[];
  const CssDir &D = g.d[DIR];
  const int nlines = DIR == 0 ? g.nth * g.nphi : g.nth * g.nr;
  const int line = blockIdx.x * blockDim.x + threadIdx.x;
  if (line >= nlines) return;
  const size_t s = DIR == 0 ? (size_t)g.nth * g.nphi : g.nth;
  const size_t base = DIR == 0 ? line : line % g.nth + (size_t)(line / g.nth) * g.nth * g.nphi;
  const double *x = gin + base;
  double *o = gout + base;
  double reg[M > 0 ? M : 1];
  double *t = M > 0 ? reg : sm + threadIdx.x;
  const int ts = M > 0 ? 1 : (int)blockDim.x;
  double lo[4], hi[4], up[4] = {0.0, 0.0, 0.0, 0.0}, wait[4], first[4], below[4];
  for (int b = 0; b < D.nb; b++) {
    const int m = M > 0 ? M : D.size[b], a0 = M > 0 ? b * M : D.start[b];
#pragma unroll(M > 0 ? M : 8)
    for (int k = 0; k < m; k++) t[k * ts] = __ldg(x + (size_t)(a0 + k) * s);
    const double dn = D.dnum[b];
    adj_block<ORDER, M>(t, ts, m, tabp(g, DIR, b, ORDER, bdry), g.tstride, E + (size_t)b * ADJ_TAB,
                        ORDER == 1 ? dn : dn * dn, lo, hi);
    if (b > 0) {
#pragma unroll
      for (int k = 0; k < 4; k++) o[(size_t)(a0 - 4 + k) * s] = wait[k] + lo[k];
    } else {
#pragma unroll
      for (int k = 0; k < 4; k++) below[k] = lo[k];
    }
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const double v = t[k * ts] + up[k];
      if (DIR == 2 && b == 0) first[k] = v;
      else o[(size_t)(a0 + k) * s] = v;
      wait[k] = t[(m - 4 + k) * ts];
      up[k] = hi[k];
    }
#pragma unroll(M > 0 ? M : 8)
    for (int k = 4; k < m - 4; k++) o[(size_t)(a0 + k) * s] = t[k * ts];
  }
  const int n = DIR == 0 ? g.nr : g.nphi;
#pragma unroll
  for (int k = 0; k < 4; k++) {
    o[(size_t)(n - 4 + k) * s] = DIR == 2 ? wait[k] + below[k] : wait[k];
    if (DIR == 2) o[(size_t)k * s] = first[k] + up[k];
  }
}

// Adjoint along theta: the warp's 32 rows pass through its own tile block by
// block.
template <int ORDER, int M>
__global__ void __launch_bounds__(64) k_adj_t(CssGeo g, const double *__restrict__ E, const double *__restrict__ gin,
                                              double *__restrict__ gout, int bdry) {
  extern __shared__ double sm[];
  const CssDir &D = g.d[1];
  const int lane = threadIdx.x & 31, nlines = g.nphi * g.nr, nth = g.nth;
  const int row0 = (blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * 32;
  if (row0 >= nlines) return;
  const int nrow = min(32, nlines - row0);
  const int SR = adj_theta_stride(M > 0 ? M : D.maxm);
  double *T = sm + (size_t)(threadIdx.x >> 5) * 32 * SR, *t = T + lane * SR + 4;
  const double *src = gin + (size_t)row0 * nth;
  double *dst = gout + (size_t)row0 * nth;
  double lo[4], hi[4], up[4] = {0.0, 0.0, 0.0, 0.0};
  for (int b = 0; b < D.nb; b++) {
    const int m = M > 0 ? M : D.size[b], t0 = M > 0 ? b * M : D.start[b];
#pragma unroll(M > 0 ? M : 4)
    for (int k0 = 0; k0 < 32 * m; k0 += 32) {
      const int k = k0 + lane, l = k / m, c = k - l * m;
      if (l < nrow) T[l * SR + 4 + c] = __ldg(src + (size_t)l * nth + t0 + c);
    }
    __syncwarp();
    if (lane < nrow) {
      const double dn = D.dnum[b], sc = ORDER == 1 ? dn : dn * dn;
      const double *G = tabp(g, 1, b, ORDER, bdry), *Eb = E + (size_t)b * ADJ_TAB;
      if constexpr (M > 0) {
        double reg[M];
#pragma unroll
        for (int k = 0; k < M; k++) reg[k] = t[k];
        adj_block<ORDER, M>(reg, 1, M, G, g.tstride, Eb, sc, lo, hi);
#pragma unroll
        for (int k = 0; k < M; k++) t[k] = k < 4 ? reg[k] + up[k] : reg[k];
      } else {
        adj_block<ORDER, 0>(t, 1, m, G, g.tstride, Eb, sc, lo, hi);
#pragma unroll
        for (int k = 0; k < 4; k++) t[k] += up[k];
      }
#pragma unroll
      for (int k = 0; k < 4; k++) {
        up[k] = hi[k];
        if (b > 0) t[k - 4] += lo[k];
      }
    }
    __syncwarp();
    // points t0-4 .. t0+m-5, and the last four once no block follows
    const int c0 = b > 0 ? -4 : 0, n = (b + 1 < D.nb ? m - 4 : m) - c0;
    if (n == 32) {
#pragma unroll 8
      for (int l = 0; l < nrow; l++) dst[(size_t)l * nth + t0 + c0 + lane] = T[l * SR + 4 + c0 + lane];
    } else {
      for (int k = lane; k < nrow * n; k += 32) {
        const int l = k / n, c = c0 + k - l * n;
        dst[(size_t)l * nth + t0 + c] = T[l * SR + 4 + c];
      }
    }
    __syncwarp();
    if (lane < nrow) {
#pragma unroll
      for (int k = 0; k < 4; k++) t[k - 4] = t[m - 4 + k];
    }
    __syncwarp();
  }
}

// Adjoint on few lines: W warps a CTA take W blocks in a row of the same 32
// lines, so that the sweeps of a line's blocks run side by side where the
// lines alone leave the chip idle (adj_warps has the line and both sides).
// What a block adds to its neighbours passes through shared memory (two
// buffers in turn, one barrier a group of blocks); the last four points of a
// group wait for the next group's first block.  Block lengths at run time; the
// same sums in the same order as above.  tile: 32 lines of a block, theta rows
// at an odd stride.
__host__ __device__ constexpr int adj_w_tile(int dir, int m) { return 32 * (dir == 1 ? m | 1 : m); }
__host__ __device__ constexpr int adj_w_smem(int dir, int m, int w) {  // doubles
  return w * (adj_w_tile(dir, m) + 2 * 8 * 32) + 2 * 8 * 32 + 8 * 32;
}
template <int DIR, int ORDER>
__global__ void __launch_bounds__(256) k_adj_w(CssGeo g, const double *__restrict__ E, const double *__restrict__ gin,
                                               double *__restrict__ gout, int bdry) {
  extern __shared__ double sm[];
  const CssDir &D = g.d[DIR];
  const int W = blockDim.y, wy = threadIdx.y, lane = threadIdx.x, nb = D.nb;
  const int nlines = DIR == 0 ? g.nth * g.nphi : (DIR == 1 ? g.nphi * g.nr : g.nth * g.nr);
  const int line0 = blockIdx.x * 32, line = line0 + lane, nrow = min(32, nlines - line0);
  const bool live = lane < nrow;
  const size_t s = DIR == 0 ? (size_t)g.nth * g.nphi : (DIR == 1 ? 1 : g.nth);
  const size_t base = DIR == 0 ? line : (DIR == 1 ? (size_t)line * g.nth
                                                  : line % g.nth + (size_t)(line / g.nth) * g.nth * g.nphi);
  const int SR = DIR == 1 ? D.maxm | 1 : 1, ts = DIR == 1 ? 1 : 32;
  double *const T = sm + (size_t)wy * adj_w_tile(DIR, D.maxm), *const t = T + lane * SR;
  double *const ex = sm + (size_t)W * adj_w_tile(DIR, D.maxm);  // [2][W][8][32]: lo, hi of the blocks of a group
  double *const carry = ex + 2 * W * 8 * 32;                    // [2][8][32]: a group's waiting points, its last hi
  double *const wrap = carry + 2 * 8 * 32;                      // [8][32]: phi's first four points, first lo
  double lo[4], hi[4];
  int last = 0;  // the last point of this warp's last block
  for (int c0 = 0, par = 0; c0 < nb; c0 += W, par ^= 1) {
    const int b = c0 + wy, m = b < nb ? D.size[b] : 0, a0 = b < nb ? D.start[b] : 0;
    double *const e = ex + (size_t)par * W * 8 * 32 + lane;
    if (b < nb) {
      if (DIR == 1) {
        const double *src = gin + (size_t)line0 * g.nth + a0;
        const unsigned inv = inv_of(m);
        for (int k = lane; k < nrow * m; k += 32) {
          const int l = div_by(k, inv), c = k - l * m;
          cp_async8(T + l * SR + c, src + (size_t)l * g.nth + c);
        }
      } else if (live) {
        const double *src = gin + base + (size_t)a0 * s;
        for (int k = 0; k < m; k++) cp_async8(t + k * 32, src + (size_t)k * s);
      }
      cp_async_wait();
      __syncwarp();
      if (live) {
        const double dn = D.dnum[b];
        adj_block<ORDER, 0>(t, ts, m, tabp(g, DIR, b, ORDER, bdry), g.tstride, E + (size_t)b * ADJ_TAB,
                            ORDER == 1 ? dn : dn * dn, lo, hi);
#pragma unroll
        for (int k = 0; k < 4; k++) {
          e[(wy * 8 + k) * 32] = lo[k];
          e[(wy * 8 + 4 + k) * 32] = hi[k];
        }
      }
      last = m - 1;
    }
    __syncthreads();
    if (b >= nb) continue;
    const double *const cin = carry + (par ^ 1) * 8 * 32 + lane;
    double *const cout = carry + par * 8 * 32 + lane, *const wr = wrap + lane;
    const bool next = b + 1 < nb, held = next && wy + 1 == W;
    if (live) {
#pragma unroll
      for (int k = 0; k < 4; k++) {
        if (DIR == 2 && b == 0) {  // waits for the last block
          wr[k * 32] = t[k * ts];
          wr[(4 + k) * 32] = lo[k];
        } else {
          t[k * ts] += wy > 0 ? e[((wy - 1) * 8 + 4 + k) * 32] : (c0 > 0 ? cin[(4 + k) * 32] : 0.0);
        }
        if (wy == 0 && c0 > 0) gout[base + (size_t)(a0 - 4 + k) * s] = cin[k * 32] + lo[k];
        if (held) {
          cout[k * 32] = t[(m - 4 + k) * ts];
          cout[(4 + k) * 32] = hi[k];
        } else if (next) {
          t[(m - 4 + k) * ts] += e[((wy + 1) * 8 + k) * 32];
        }
      }
    }
    const int k0 = DIR == 2 && b == 0 ? 4 : 0, k1 = held || (DIR == 2 && !next) ? m - 4 : m;
    if (DIR == 1) {
      __syncwarp();
      double *dst = gout + (size_t)line0 * g.nth + a0;
      const unsigned inv = inv_of(k1);
      for (int k = lane; k < nrow * k1; k += 32) {
        const int l = div_by(k, inv), c = k - l * k1;
        dst[(size_t)l * g.nth + c] = T[l * SR + c];
      }
      __syncwarp();
    } else if (live) {
#pragma unroll 8
      for (int k = k0; k < k1; k++) gout[base + (size_t)(a0 + k) * s] = t[k * 32];
    }
  }
  if (DIR == 2) {
    __syncthreads();
    if ((nb - 1) % W == wy && live) {
      const double *const wr = wrap + lane;
#pragma unroll
      for (int k = 0; k < 4; k++) {
        gout[base + (size_t)(g.nphi - 4 + k) * s] = t[(last - 3 + k) * 32] + wr[(4 + k) * 32];
        gout[base + (size_t)k * s] = wr[k * 32] + hi[k];
      }
    }
  }
}

// ---------------------------------------------------------------------------
// The radial parts of B = curl A for radial blocks of run-time length: a lane
// takes a (theta, phi) column, z 0 r A_theta for B_phi, z 1 r A_phi for
// B_theta, read straight from global memory (the arithmetic of k_curl_r).
// In tiles of 8 to 16 lines, as k_curl_r takes the 16- and 32-point blocks, a
// CTA had few lanes solving: 199 us a launch against 81 (FP32), 198 against
// 86 (FP64) on the ensemble's ragged shells.
// ---------------------------------------------------------------------------
template <typename TS>
struct CurlLine {  // r A along r, from the block's first radius
  const TS *p;
  const double *r;
  size_t ps;
  __device__ __forceinline__ double operator[](int k) const {
    return (double)__ldg(p + (long long)k * (long long)ps) * __ldg(r + k);
  }
};
template <typename TS>
__global__ void __launch_bounds__(DV_NT) k_curl_rg(CssGeo g, const TS *__restrict__ a, double *__restrict__ out,
                                                   int apply_bc) {
  extern __shared__ double sm[];
  const CssDir &D = g.d[0];
  const int b = blockIdx.y, z = blockIdx.z, m = D.size[b], r0 = D.start[b], ts = blockDim.x;
  const int line = blockIdx.x * blockDim.x + threadIdx.x;
  if (line >= g.nth * g.nphi) return;
  const size_t n = (size_t)g.ncell, ps = (size_t)g.nth * g.nphi, base = (size_t)r0 * ps + line;
  double *t = sm + threadIdx.x;
  const int bdry = g.ibcr[z == 0 ? 10 : 11];
  line_solve_g<1>(CurlLine<TS>{a + z * n + base, g.r_ind + r0, ps}, StridedIn{1}, m, dtype_of(D, b), bdry, 0.0, 0.0,
                  tabp(g, 0, b, 1, bdry), g.tstride, D.dnum[b], D.dnum[b], 0, t, ts, t, StridedOut{ts});
  const int it = line % g.nth;
  double *o = out + (z == 0 ? n : 0) + base;  // B_phi, B_theta
  for (int j0 = 0; j0 < m; j0 += 4) {
    double in[4];
#pragma unroll
    for (int k = 0; k < 4; k++) in[k] = j0 + k < m ? o[(size_t)(j0 + k) * ps] : 0.0;
#pragma unroll
    for (int k = 0; k < 4; k++) {
      if (j0 + k >= m) continue;
      const int ir = r0 + j0 + k;
      double d = t[(j0 + k) * ts];
      if (g.non_uniform) d = d * g.dxdr[ir];
      double v = z == 0 ? in[k] + d * g.r_inv[ir] : in[k] - d * g.r_inv[ir];
      if (apply_bc) {  // this half's component; the B_phi half zeroes B_r
        double other = 0.0;
        const bool br0 = z == 0 ? curl_faces(g, it, ir, other, v) : curl_faces(g, it, ir, v, other);
        if (z == 0 && br0) out[2 * n + base + (size_t)(j0 + k) * ps] = 0.0;
      }
      o[(size_t)(j0 + k) * ps] = v;
    }
  }
}

}  // namespace css
