// css_stage.cuh -- the second half of an RK stage for any radial block
// length and either storage of the stage states: Radial_Terms (+ Lorentz)
// with Density_Terms_Radial, the open radial faces, Density_Terms_Theta on the
// theta-wall blocks, the stage combination (Step_RK4 or the TVD schemes) and
// Bound, in one pass.  It follows the plane pass (k_thph), which has written
// the tendency of the theta and phi sweeps, with Density_Terms_Theta off the
// theta walls, the temperature, and d(rho)/dtheta with a zero wall datum on
// the wall blocks (rtw).
//
// Against the four-kernel stage these runs took before, the tendency is
// written once and read once instead of passing through the phi, radial and
// update kernels, and no tile is loaded twice.  Bound by the latency of its
// global reads (238 bytes a cell hydro, 376 MHD in FP64): on 100x176x304 4.5
// of the cycles between two issues wait on global loads, 2.4 on fixed
// latencies, 1.2 on barriers, HBM at 42 %, the FP64 pipe at 15 %.  Per stage,
// measured against the radial and update kernels: 100x176x304 in blocks of
// 20 radii 696 -> 379 us, open faces on 64x128x256 209 -> 162 us, FP32 stage
// states of MHD 128x128x256 650 -> 540 us (434 in k_rstage, which takes
// 32-point blocks).  Reading the lines from global
// memory instead of a TMA slab took 436 us on the first of them.
#pragma once
#include "css_deriv.cuh"
#include "css_fused.cuh"

namespace css {

constexpr int SG_NT = 256;

// one theta column of a field's slab in shared memory (rows of 32 theta), from
// the block's first radius: FP64 as stored, FP32 about its background (bg
// NULL: none)
template <typename TS>
struct SLine {
  const TS *p;
  const double *bg;
  int nth;
  __device__ __forceinline__ double operator[](int k) const {
    double x = (double)p[k * 32];
    if constexpr (sizeof(TS) == 4) {
      if (bg) x += __ldg(bg + (long long)k * nth);
    }
    return x;
  }
};

// slab (state fields of storage size ts, then B_theta and B_phi), derivative
// tiles, a face datum a line, an mbarrier
__host__ __device__ constexpr size_t stage_smem(int mag, int m, int ts) {
  return (size_t)32 * (m + 8) * (5 * ts + (mag ? 16 : 0)) + 8 * ((size_t)(mag ? 8 : 6) * m * 32 + 32 + 1);
}
constexpr size_t SG_SMEM = 227 * 1024;  // a stage whose slab and tiles are larger takes the four kernels

// rows of 32 theta a warp takes at a time, and CTAs an SM (registers):
// closed hydro slabs of short blocks leave room for three CTAs, the others
// for two or one
template <int KIND>
struct StageCfg {
  static constexpr int R = KIND == 0 ? 1 : 2, CTAS = KIND == 0 ? 3 : 2;
};

// One (radial block, 32 theta, phi) slab a CTA.  The block's m radii with
// 4-point halos arrive by TMA; a warp solves one derivative of the 32 lines
// from it, the forward values in the derivative's own tile; then each warp
// takes whole rows of 32 theta.  A theta-wall block lies inside one chunk of
// 32 (blocks of 16 or 32 points), so its wall datum comes from the wall's
// lane.  KIND: 0 closed hydro, 1 hydro with open radial faces, 2 MHD.  STG:
// the RK4 stage 1..4 (as k_rstage), or -1: a TVD stage, stage_rt 5 or 6 (as
// k_rhot_update).
template <typename TS, typename TO, int KIND, int STG>
__global__ void __launch_bounds__(SG_NT, StageCfg<KIND>::CTAS) k_rstage_g(CssGeo g, const TS *__restrict__ cur,
                                                       const double *__restrict__ bf, const double *dv,
                                                       const double *v0, double *vs, TO *nx,
                                                       const double *__restrict__ tbuf,
                                                       const double *__restrict__ rtw, int wallm, int stage_rt,
                                                       double dtcur, double ca, double cb, double dsld, int *flag,
                                                       const __grid_constant__ SlabMaps sc,
                                                       const __grid_constant__ SlabMaps sb) {
  constexpr int mag = KIND == 2, nv = mag ? 8 : 5, ND = mag ? 8 : 6, R = StageCfg<KIND>::R;
  extern __shared__ __align__(128) double sm[];
  const CssDir &D = g.d[0];
  const int lane = threadIdx.x & 31, wrp = threadIdx.x >> 5;
  const int nchunk = (g.nth + 31) / 32, br = blockIdx.x / nchunk, t0 = (blockIdx.x - br * nchunk) * 32, ip = blockIdx.y;
  const int m = D.size[br], r0 = D.start[br], nth = g.nth, nr = g.nr;
  const size_t n = (size_t)g.ncell, ps = (size_t)nth * g.nphi;
  const int it = t0 + lane, itc = min(it, nth - 1);
  const bool live = it < nth;
  const size_t base = (size_t)r0 * ps + (size_t)ip * nth + itc;  // (theta, phi) of the block's first radius
  const size_t bgo = (size_t)r0 * nth + itc;
  const int FB = m * 32, FH = (m + 8) * 32;
  TS *const H = reinterpret_cast<TS *>(sm);                // rho w v u s
  double *const HB = reinterpret_cast<double *>(H + 5 * FH);  // B_theta B_phi
  double *const O = HB + (mag ? 2 * FH : 0), *const datum = O + ND * FB;
  uint64_t *const bar = reinterpret_cast<uint64_t *>(datum + 32);
  if (threadIdx.x == 0) {
    mbar_init(bar, 1);
    mbar_fence_init();
    mbar_expect_tx(bar, (unsigned)(FH * (5 * sizeof(TS) + (mag ? 16 : 0))));
    for (int f = 0; f < 5; f++) tma_load_4d(H + f * FH, &sc.slab, t0, ip, r0 - 4, f, bar);
    if (mag)
      for (int f = 0; f < 2; f++) tma_load_4d(HB + f * FH, &sb.slab, t0, ip, r0 - 4, f, bar);
  }
  const int dtype = dtype_of(D, br);
  const bool top_open = KIND == 1 && D.rphys[br] && g.top_inout, bot_open = KIND == 1 && D.lphys[br] && g.bot_inout;
  const bool need_s = STG >= 0 ? !(STG == 1 && !g.sldiffusion) : (stage_rt == 6 && dsld != 0.0);
  const bool need_c = STG < 0 && cb != 0.0;
  // the lines the pointwise phase reads, toward L2 (two 128-byte halves a row)
  {
    const int ns = 6 + (mag ? 1 : 0) + nv + (need_s ? nv : 0);
    for (int k = threadIdx.x; k < ns * m * 2; k += SG_NT) {
      const int f = k / (m * 2), rr = (k >> 1) % m, t = t0 + (k & 1) * 16;
      if (t >= nth) continue;
      const double *b;
      if (f < 5) b = dv + (size_t)f * n;
      else if (f == 5) b = tbuf;
      else if (mag && f == 6) b = bf + 2 * n;
      else {
        const int q = f - 6 - (mag ? 1 : 0);
        b = q < nv ? v0 + (size_t)q * n : vs + (size_t)(q - nv) * n;
      }
      prefetch_l2(b + (size_t)(r0 + rr) * ps + (size_t)ip * nth + t);
    }
  }
  __syncthreads();  // the barrier is initialised before anyone waits on it
  if (__syncthreads_or(!mbar_wait_bounded(bar, 0u, kWaitCycles))) {
    if (threadIdx.x == 0) {
      atomicOr(flag, kFlagTimeout);
      mbar_wait_bounded(bar, 0u, kWaitCycles);
    }
    return;
  }
  // ---- radial solves: derivative wrp (dw dv du ds d2s drho0 [dbt dbp]), line = lane ----
  if (wrp < ND && !(wrp == 4 && !g.slaplacian)) {
    const int k = wrp;
    const int var = (0x87155432u >> (4 * k)) & 15;  // field whose closure derivative k takes: 2 3 4 5 5 1 7 8
    const int bdry = (k == 5 && top_open) ? 2 : g.ibcr[var];
    double *o = O + k * FB + lane;
    const double dn = D.dnum[br];
    auto go = [&](auto x) {
      double lo = 0.0, hi = 0.0;
      if (k == 0 || k == 1) {  // stress-free datum w/r/dxdr (rhs_mpi.f90:578-614)
        if (D.lphys[br] && g.bottom_stress_free) lo = x[0] / g.r1 / g.dxdr[0];
        if (D.rphys[br]) {
          if (g.top_stress_free) hi = x[m - 1] / g.r2 / g.dxdr[nr - 1];
          else hi = x[m - 1];
        }
      }
      if (k == 3 || k == 4) {  // constant-flux datum (rhs_mpi.f90:584-592, :616-624)
        lo = g.s_flux_lo;
        hi = g.s_flux_hi;
      }
      if (bot_open) lo = 0.0;  // open faces: data of w, v, u, s zero (rhs_mpi.f90:594-596, :626-628)
      if (top_open) hi = 0.0;
      if (k == 4)
        line_solve_g<2>(x, StridedIn{1}, m, dtype, bdry, lo, hi, tabp(g, 0, br, 2, bdry), g.tstride, dn, dn * dn, 0, o, 32, o,
                        StridedOut{32});
      else
        line_solve_g<1>(x, StridedIn{1}, m, dtype, bdry, lo, hi, tabp(g, 0, br, 1, bdry), g.tstride, dn, dn, 0, o, 32, o,
                        StridedOut{32});
    };
    if (!mag || k < 6) {
      const int f = k <= 3 ? k + 1 : (k == 4 ? 4 : 0);  // w v u s s rho
      go(SLine<TS>{H + f * FH + 4 * 32 + lane,
                   sizeof(TS) == 4 && f == 0 ? bg_rho(g) + bgo : (sizeof(TS) == 4 && f == 4 ? bg_s(g) + bgo : nullptr),
                   nth});
    } else {
      go(SLine<double>{HB + (k - 6) * FH + 4 * 32 + lane, nullptr, nth});
    }
  }
  __syncthreads();

  // field f of the state at row j of this column
  auto st = [&](int f, int j) {
    double x = (double)H[f * FH + (j + 4) * 32 + lane];
    if constexpr (sizeof(TS) == 4) {
      if (f == 0) x += __ldg(bg_rho(g) + bgo + (size_t)j * nth);
      if (f == 4) x += __ldg(bg_s(g) + bgo + (size_t)j * nth);
    }
    return x;
  };
  auto gather = [&](int j, RadIn &q) {
    const size_t id = base + (size_t)j * ps;
    const double *ol = O + j * 32 + lane;
    q.u = st(3, j);
    q.rho = st(0, j);
    q.t = __ldg(tbuf + id);
    q.dw_r = ol[0]; q.dv_r = ol[FB]; q.du_r = ol[2 * FB]; q.ds_r = ol[3 * FB]; q.d2s_r = ol[4 * FB];
    if (mag) {
      q.bt = HB[(j + 4) * 32 + lane]; q.bp = HB[FH + (j + 4) * 32 + lane]; q.br = __ldg(bf + 2 * n + id);
      q.dbt_r = ol[6 * FB]; q.dbp_r = ol[7 * FB];
    }
  };
  // hydrostatic datum of d(rho)/dr on a physical face (rhs_mpi.f90:1750-1768)
  const int phys = D.lphys[br] ? 1 : (D.rphys[br] && !top_open ? 2 : 0);
  if (phys) {
    if (wrp == 0) {
      const int j = phys == 1 ? 0 : m - 1;
      const size_t id = base + (size_t)j * ps;
      RadIn q;
      gather(j, q);
      double drho = __ldg(dv + id), dw = __ldg(dv + n + id), dvv = __ldg(dv + 2 * n + id), du = __ldg(dv + 3 * n + id),
             ds = __ldg(dv + 4 * n + id);
      radial_point<mag>(g, r0 + j, q, drho, dw, dvv, du, ds);
      double d;
      if (bot_open) {
        d = g.invpconst * q.rho * du / q.t;  // rhs_mpi.f90:1894
      } else {
        if (g.lbcr_rho == 4 || g.lbcr_rho == (phys == 1 ? 2 : 3)) d = du * q.rho * g.invpconst / q.t;
        else d = q.rho;
        if (g.non_uniform) d = d / g.dxdr[phys == 1 ? 0 : nr - 1];
      }
      datum[lane] = d;
    }
    __syncthreads();
  }
  const double *resp = g.resp_r + (size_t)(2 * br + (phys == 2 ? 1 : 0)) * g.tstride;
  // the theta walls: this lane's cell in a wall block, and the wall's lane
  const int lo_wall = t0 == 0 ? wallm : 0, hi_wall = t0 + 32 >= nth ? nth - wallm : nth;
  const bool in_lo = it < lo_wall, in_hi = live && it >= hi_wall;
  const int btw = in_hi ? g.d[1].nb - 1 : 0;
  const double rl = in_lo ? __ldg(g.resp_t + it + 1)
                          : (in_hi ? __ldg(g.resp_t + (size_t)(2 * btw + 1) * g.tstride + it - hi_wall + 1) : 0.0);
  const bool chunk_wall = lo_wall > 0 || hi_wall < nth;
  const bool twall = it == 0 || it == nth - 1;
  int bad = 0;
  // whole rows of 32 theta, R at a time: every load of a field's values is
  // issued before the first store
  for (int j0 = wrp; j0 < m; j0 += 8 * R) {
    double d[R][5];
    bool ok[R];
#pragma unroll
    for (int h = 0; h < R; h++) {
      const int j = min(j0 + 8 * h, m - 1), ir = r0 + j;
      ok[h] = j0 + 8 * h < m && live;
      const size_t id = base + (size_t)j * ps;
      RadIn q;
      gather(j, q);
      double drho = __ldg(dv + id), dw = __ldg(dv + n + id), dvv = __ldg(dv + 2 * n + id), du = __ldg(dv + 3 * n + id),
             ds = __ldg(dv + 4 * n + id);
      const double w = st(1, j);
      const double rz = in_lo || in_hi ? __ldg(rtw + (((size_t)ir * g.nphi + ip) * 2 + (in_hi ? 1 : 0)) * 32 +
                                               (in_hi ? it - hi_wall : it))
                                       : 0.0;
      radial_point<mag>(g, ir, q, drho, dw, dvv, du, ds);
      double w1 = O[5 * FB + j * 32 + lane];  // Density_Terms_Radial
      if (phys) w1 = w1 + datum[lane] * resp[j + 1];
      const double orho = 1.0 / q.rho;
      if (top_open || bot_open) {
        // Top_/Bottom_Inflow_Outflow: no dxdr, their own product orders
        // (rhs_mpi.f90:2032-2033, :1906-1907), then the face plane's
        // relaxation (:2042-2066, :1913-1952)
        drho = drho - q.u * w1;
        if (top_open) du = du - g.pconst * q.t * orho * w1;
        else du = du - g.pconst * q.t * w1 * orho;
        inout_face(g, j, m, top_open, [&](int f, int dd) { return st(f + 1, j + dd); }, (size_t)ip * nth + itc, drho,
                   dvv, du, ds);
      } else {
        if (g.non_uniform) w1 = w1 * g.dxdr[ir];
        drho = drho - q.u * w1;
        w1 = w1 * orho;
        du = du - g.pconst * q.t * w1;
      }
      if (phys == 2 && j == m - 1 && !g.set_stop) {  // rhs_mpi.f90:1807-1818
        drho = drho + q.rho * (g.t0 - q.t) / (g.damping_time * (g.gamma - 2.0) * q.t);
        ds = ds - g.cv * (g.t0 - q.t) / (g.damping_time * (g.gamma - 2.0) * q.t);
      }
      // Density_Terms_Theta on a theta-wall block (rhs_mpi.f90:1522-1605):
      // the zero-datum derivative plus the wall's datum times the block's
      // unit response
      if (chunk_wall) {
        const double dat = g.r_ind[ir] * g.invpconst * dw * q.rho / q.t;
        const double dlo = __shfl_sync(0xffffffffu, dat, 0), dhi = __shfl_sync(0xffffffffu, dat, (nth - 1 - t0) & 31);
        if (in_lo || in_hi) {
          double x1 = g.r_inv[ir] * (rz + (in_hi ? dhi : dlo) * rl);
          drho = drho - w * x1;
          x1 = x1 * orho;
          dw = dw - g.pconst * x1 * q.t;
        }
      }
      if (KIND == 1 && ir == 0 && g.bottom_specified)  // prescribed bottom, u_theta (rhs_mpi.f90:1932)
        dw = dw + g.inout[IO_BOT_TAU] * (g.inout[IO_BOT_TCONST] * g.ashv[ps + (size_t)ip * nth + itc] - w);
      if (g.xi_cs < 1.0) drho = (g.xi_cs * g.xi_cs) * drho;
      d[h][0] = drho; d[h][1] = dw; d[h][2] = dvv; d[h][3] = du; d[h][4] = ds;
    }
    // ---- stage combination and Bound (rhs_mpi.f90:2395-2491).  Every value
    // is read once, before the same thread writes that address (nx may be
    // vars0), so the reads take the non-coherent path. ----
#pragma unroll
    for (int iv = 0; iv < nv; iv++) {
      double dd[R], aa[R], ss[R], cc[R];
#pragma unroll
      for (int h = 0; h < R; h++) {
        const int j = min(j0 + 8 * h, m - 1);
        const size_t qi = (size_t)iv * n + base + (size_t)j * ps;
        dd[h] = iv < 5 ? d[h][iv < 5 ? iv : 0] : __ldg(dv + qi);
        aa[h] = __ldg(v0 + qi);
        ss[h] = need_s ? __ldg(vs + qi) : 0.0;
        cc[h] = need_c ? (iv < 5 ? st(iv < 5 ? iv : 0, j) : (double)__ldg(cur + qi)) : 0.0;
      }
#pragma unroll
      for (int h = 0; h < R; h++) {
        if (!ok[h]) continue;
        const int j = j0 + 8 * h, ir = r0 + j;
        const size_t id = base + (size_t)j * ps, qi = (size_t)iv * n + id;
        const double dd_ = dd[h], a = aa[h];
        double o;
        if (STG == 1) {
          vs[qi] = g.sldiffusion ? ss[h] + dd_ / 6.0 : dd_;
          o = a + dtcur * dd_;
        } else if (STG == 4) {
          o = a + dtcur * (ss[h] + dd_ / 6.0);
        } else if (STG > 0) {
          vs[qi] = ss[h] + dd_ / 3.0;
          o = a + dtcur * dd_;
        } else {
          o = ca * a + cb * cc[h] + dtcur * dd_;
          if (need_s) o = o + dsld * ss[h];
        }
        const bool rlo = ir == 0, rhi = ir == nr - 1;
        if (twall || rlo || rhi) {
          if (iv == 1 && twall) o = 0.0;
          if (iv == 3 && !g.theta_stress_free && twall) o = 0.0;
          if (rlo) {
            if ((iv == 1 || iv == 2) && !g.bottom_stress_free) o = 0.0;
            if (iv == 3 && !(KIND == 1 && g.bot_inout)) o = 0.0;
          }
          if (rhi && !(KIND == 1 && g.top_inout)) {  // an open top keeps every field (rhs_mpi.f90:2420-2432)
            if ((iv == 1 || iv == 2) && !g.top_stress_free) o = 0.0;
            if (iv == 3) o = 0.0;
          }
          if (iv >= 5) {
            if (g.theta_perf_conductor) {
              if ((iv == 6 || iv == 7) && twall) o = 0.0;
            } else if (iv == 5 && twall) {
              o = 0.0;
            }
            if (rlo) {
              if (g.bottom_radial_field) { if (iv == 7) o = 0.0; }
              else if (g.bottom_perfect_cond) { if (iv == 5 || iv == 6) o = 0.0; }
            }
            if (rhi) {
              if (g.top_radial_field) { if (iv == 7) o = 0.0; }
              else if (g.top_perfect_cond) { if (iv == 5 || iv == 6) o = 0.0; }
            }
          }
        }
        if (!isfinite(o)) bad = 1;
        double bgv = 0.0;
        if constexpr (sizeof(TO) == 4) {
          if (iv == 0) bgv = bg_rho(g)[bgo + (size_t)j * nth];
          else if (iv == 4) bgv = bg_s(g)[bgo + (size_t)j * nth];
        }
        nx[qi] = st_store<TO>(o, bgv);
      }
    }
  }
  if (bad && flag) atomicOr(flag, 1);
}

}  // namespace css
