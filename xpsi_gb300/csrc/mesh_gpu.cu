// mesh_gpu.cu -- K0: the hot-region cell meshes of a batch, built on the GPU
// from the steps of mesh_math.h (xpsi/cellmesh/mesh.pyx:23-417,
// polar_mesh.pyx:23-430, mesh_tools.pyx:18-890) and written straight into
// the packed per-row and per-cell arrays the rays and integrator kernels read
// (the packing of xpsi/HotRegion.py:774-1017 / Likelihood.py:297-432 that
// the host path does in numpy).
//
// Seven launches over all meshes of the batch, eight where it may queue many
// cells:
//   1. the 1000-point table of area(colat..lims[1]) per mesh, one thread (few
//      meshes: one warp) per entry (1000 independent adaptive quadratures);
//   2. per mesh: the cell area, the S - 1 parallels and the columns' edges (the
//      reference's running sums), and the trigonometry the cells share;
//   3. one warp per parallel: its centre colatitude, radius, gravity, tilt and
//      the packed row values;
//   4. one thread per cell: the corner / centre membership tests; cells
//      wholly inside or outside get their area at once, cells cut by a
//      region boundary (~1 %) are queued;
//   5. from 5000 queued cells on, their area quadratures four cells to a warp,
//      eight lanes a cell (those whose integral vanishes are left to 6);
//   6. one CTA of two warps per queued cell, or per cell left, taken from a
//      shared counter: its area quadrature, a panel to each warp (21
//      Gauss-Kronrod nodes over the lanes, the interval list in shared memory)
//      -- the same adaptive scheme the host builder runs serially;
//   7. a CTA for each dyadic piece of the cells touched at a corner, and one
//      for each of those cells' sums (two launches).
// The serial quadratures of steps 1 and 3 keep their interval list (128
// intervals) in local memory; the host builder's limit of 4000 gives bitwise
// the same meshes (these integrals converge in far fewer intervals).
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <vector>

#include "../../include/xpsi_gb300.h"
#include "mesh_math.h"

namespace xg {
namespace {

using namespace xgm;
using DWork = WorkT<128>;
constexpr double kC = 2.99792458e8;

struct MeshJob {
  MeshPlan pl;
  Star s;
  int64_t row_off, cell_off;
  double r_s, R_over_rs, lag_scale, omit_azimuth, logT;
  int antiphased;
};

// The area integral of mesh_math.h (integrateArea) by a warp: the first
// panel's 21 nodes, one per lane, summed in the serial rule's order (the same
// bits); the integrand is smooth, so a panel that does not converge, which
// takes the serial bisection, is the exception.
__device__ double warp_area(double lo, double hi, const Star &s, int av, DWork &w) {
  const int lane = threadIdx.x & 31;
  const int NH = XG_K21_HALF - 1;  // 10
  if (!(hi > lo)) return integrateArea(lo, hi, s, av, w);
  const double c = 0.5 * (lo + hi), h = 0.5 * (hi - lo), ah = fabs(h);
  double v = 0.0;
  if (lane < 21) {
    const int jn = lane < 10 ? lane : lane - 10;  // 0-9: c - dx_j, 10-19: c + dx_j, 20: c
    double theta = c;
    if (lane < 20) {
      const double dx = h * XG_K21_X[jn];
      theta = lane < 10 ? c - dx : c + dx;
    }
    if (!are_equal(theta, 0.0)) {
      const double mu = cos(theta);
      const double radius = radiusNormalised(mu, s.epsilon, s.zeta, s.shape);
      const double ft = f_theta(mu, radius, s.epsilon, s.zeta, s.shape);
      v = radius * radius * sqrt(1.0 + ft * ft) * sin(theta);
      if (av != 0) v = theta * v;
    }
  }
  const double fc = __shfl_sync(0xffffffffu, v, 20);
  double rk = XG_K21_WK[NH] * fc, rg = XG_K21_WG[NH] * fc, ra = fabs(rk);
#pragma unroll 1
  for (int q = 0; q < NH; q++) {
    const double f1 = __shfl_sync(0xffffffffu, v, q), f2 = __shfl_sync(0xffffffffu, v, q + 10);
    rk += XG_K21_WK[q] * (f1 + f2);
    rg += XG_K21_WG[q] * (f1 + f2);
    ra += XG_K21_WK[q] * (fabs(f1) + fabs(f2));
  }
  const double mean = 0.5 * rk;
  double rc = XG_K21_WK[NH] * fabs(fc - mean);
#pragma unroll 1
  for (int q = 0; q < NH; q++) {
    const double f1 = __shfl_sync(0xffffffffu, v, q), f2 = __shfl_sync(0xffffffffu, v, q + 10);
    rc += XG_K21_WK[q] * (fabs(f1 - mean) + fabs(f2 - mean));
  }
  const double r0 = rk * h;
  ra *= ah;
  rc *= ah;
  double e = fabs((rk - rg) * h);
  if (rc != 0.0 && e != 0.0) {
    const double x = 200.0 * e / rc, sc = x * sqrt(x);
    e = sc < 1.0 ? rc * sc : rc;
  }
  const double eps = 2.220446049250313e-16, dmin = 2.2250738585072014e-308;
  if (ra > dmin / (50.0 * eps)) e = (e < 50.0 * eps * ra) ? 50.0 * eps * ra : e;
  const double er = 1.0e-13, tol = er * fabs(r0);
  const bool done = (e <= 50.0 * eps * ra && e > tol) || (e <= tol && e != rc) || e == 0.0;
  if (!done || r0 == 0.0) return integrateArea(lo, hi, s, av, w);
  return s.R_eq * s.R_eq * r0;
}

// one entry per thread (many meshes), or per warp (kWarp: up to kWarpTables
// meshes, where the batch leaves the chip idle and a thread's chain of 21
// nodes is what it waits for: one mesh 87 us by threads)
constexpr int kWarpTables = 8;
template <bool kWarp>
__global__ void __launch_bounds__(128) mesh_table_kernel(const MeshJob *jobs, double *tab) {
  const int m = blockIdx.y;
  const int i = kWarp ? blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)
                      : blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= kAreaTab) return;
  const MeshJob &J = jobs[m];
  DWork w;
  const double lo = mesh_table_colat(J.pl, i), hi = J.pl.lims[1];
  if (kWarp) {
    const double A = warp_area(lo, hi, J.s, 0, w);
    if ((threadIdx.x & 31) == 0) tab[(size_t)m * kAreaTab + i] = A;
  } else {
    tab[(size_t)m * kAreaTab + i] = integrateArea(lo, hi, J.s, 0, w);
  }
}

// what the cells of a mesh share, formed once: the region with its angles'
// cosines and sines, and per column the azimuth of its left edge (the
// reference's running sum of cell widths) and the cosines its membership tests
// need
struct MeshTrig {
  Region g;
  double cos_cr;  // cos of the ceding radius
};
struct ColTrig {
  double left, c_left, s_left, c_mid, s_mid;  // cos of the azimuth from each region's meridian
};
struct RowTmp {
  double lower, upper, colat, effGrav;
  double cl, sl, cu, su, cc, sc;  // cos and sin of lower, upper, colat
};

// per mesh: the cell area, the parallels, the columns' edges.  The running
// sums (parallels' areas, edges) are single threads' chains of additions; the
// rest is a thread per parallel or column.
__global__ void __launch_bounds__(128) mesh_parallels_kernel(const MeshJob *jobs,
                                                             const double *tab, double *par_out,
                                                             double *mesh_tmp, MeshTrig *trig,
                                                             ColTrig *cols, int S_max) {
  extern __shared__ double sm[];
  double *colat = sm, *eta_i = sm + kAreaTab, *edge = eta_i + S_max;
  const int m = blockIdx.x;
  const MeshJob &J = jobs[m];
  const int S = (int)J.pl.S;
  const double *T = tab + (size_t)m * kAreaTab;
  double cellArea, eta;
  mesh_cell_area(J.pl, T[kAreaTab - 1], cellArea, eta);
  for (int i = threadIdx.x; i < kAreaTab; i += blockDim.x) colat[i] = mesh_table_colat(J.pl, i);
  if (threadIdx.x == 0) {
    double i_eta = (double)J.pl.S * eta;
    for (int i = 0; i + 1 < S; i++) {
      i_eta -= eta;
      eta_i[i] = i_eta;
    }
    mesh_tmp[2 * m] = cellArea;
    mesh_tmp[2 * m + 1] = eta;
  }
  if (threadIdx.x == 32) {
    double e = J.pl.polar ? -PI : -J.pl.boundary_phi;
    for (int j = 0; j <= S; j++) {
      edge[j] = e;
      e = e + J.pl.delta_phi;
    }
    MeshTrig t;
    t.g = mesh_region(J.pl);
    t.cos_cr = t.g.cos_cede;
    trig[m] = t;
  }
  __syncthreads();
  for (int i = threadIdx.x; i + 1 < S; i += blockDim.x)
    par_out[(size_t)m * S_max + i] = steffen_at(T, colat, kAreaTab, eta_i[i]);
  for (int j = threadIdx.x; j <= S; j += blockDim.x) {
    ColTrig c;
    const double l = edge[j], mid = l + 0.5 * J.pl.delta_phi;
    c.left = l;
    c.c_left = cos(l);
    c.s_left = cos(l - J.pl.superAzi);
    c.c_mid = cos(mid);
    c.s_mid = cos(mid - J.pl.superAzi);
    cols[(size_t)m * (S_max + 1) + j] = c;
  }
}

// a warp per parallel: its centre colatitude, radius, gravity and tilt, the
// packed row values (as the host packing forms them), and what its cells need
__global__ void __launch_bounds__(128) mesh_rows_kernel(const MeshJob *jobs, int n_mesh,
                                                        int64_t n_rows, const double *par,
                                                        int S_max, const double *mesh_tmp,
                                                        xgpu_mesh_batch_out o, RowTmp *row_tmp) {
  const int64_t row = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (row >= n_rows) return;
  int lo = 0, hi = n_mesh - 1;
  while (lo < hi) {  // last mesh whose row_off <= row
    const int mid = (lo + hi + 1) >> 1;
    if (jobs[mid].row_off <= row) lo = mid; else hi = mid - 1;
  }
  const int m = lo;
  const MeshJob &J = jobs[m];
  const size_t i = (size_t)(row - J.row_off);
  double lower, upper;
  mesh_row_bounds(J.pl, par + (size_t)m * S_max, i, lower, upper);
  const double eta = mesh_tmp[2 * m + 1];
  DWork w;
  RowOut r;
  r.colat = warp_area(lower, upper, J.s, 1, w) / eta;
  mesh_row_at(J.s, r);
  const double u = J.r_s / r.r;
  double C = (1.0 / u - J.R_over_rs);
  C += log((1.0 / u - 1.0) / (J.R_over_rs - 1.0));
  C *= J.r_s / kC;
  // one sine and cosine instruction stream for the three colatitudes
  const int lane = threadIdx.x & 31;
  const double th = lane == 0 ? lower : lane == 1 ? upper : r.colat;
  const double ct = cos(th), st = sin(th);
  RowTmp t;
  t.lower = lower; t.upper = upper; t.colat = r.colat; t.effGrav = r.effGrav;
  t.cl = __shfl_sync(0xffffffffu, ct, 0); t.sl = __shfl_sync(0xffffffffu, st, 0);
  t.cu = __shfl_sync(0xffffffffu, ct, 1); t.su = __shfl_sync(0xffffffffu, st, 1);
  t.cc = __shfl_sync(0xffffffffu, ct, 2); t.sc = __shfl_sync(0xffffffffu, st, 2);
  if (lane == 0) {
    row_tmp[row] = t;
    o.u[row] = u;
    o.r_s[row] = J.r_s;
    o.maxAlpha[row] = r.maxAlpha;
    o.radius[row] = r.r;
    o.cos_gamma[row] = r.cos_gamma;
    o.theta0[row] = J.pl.invert ? PI - r.colat : r.colat;
    o.lag_C[row] = C;
    o.lag_scale[row] = J.lag_scale;
    o.row_mesh[row] = m;
  }
}

// mesh_cell_kind from the shared trigonometry: each test "angular distance
// to a region's centre <= its radius" is decided on cosines, with the bit
// patterns; one closer than 1e-12 to its edge (the rounding of either side is
// 1e-15), or with a cosine at 1 to rounding, whose arccosine may be NaN, takes
// eval_psi's arccosine (a mesh has a few: the edge cells' corners touch the
// region's boundary).  p1-p5 as there.
__device__ int cell_kind(const MeshPlan &pl, const MeshTrig &t, const RowTmp &r, const ColTrig &a,
                         const ColTrig &b, size_t i) {
  const Region &g = t.g;
  auto near = [](double x, double cR) {
    return negative(fabs(x - cR) - 1.0e-12) || !negative(fabs(x) - (1.0 - 1.0e-12));
  };
  auto corner = [&](double ct, double st, const double cphi, const double sphi) {
    const double x = g.cos_colat * ct + g.sin_colat * st * cphi;
    const bool in = near(x, t.cos_cr) ? acos(x) <= pl.cedeRadius : negative(t.cos_cr - x);
    if (!in) return 2;
    const double y = g.cos_sc * ct + g.sin_sc * st * sphi;
    return (near(y, g.cos_sr) ? pl.superRadius <= acos(y) : negative(y - g.cos_sr)) ? 1 : 0;
  };
  int p1, p3;
  const bool pole = pl.polar && i == 0;
  if (pole) {
    p1 = p3 = pl.cedeColat <= pl.cedeRadius ? (pl.superRadius <= pl.superColat ? 1 : 0) : 2;
  } else {
    p1 = corner(r.cl, r.sl, a.c_left, a.s_left);
    p3 = corner(r.cl, r.sl, b.c_left, b.s_left);
  }
  const int p2 = corner(r.cu, r.su, a.c_left, a.s_left);
  const int p4 = corner(r.cu, r.su, b.c_left, b.s_left);
  const int p5 = corner(r.cc, r.sc, a.c_mid, a.s_mid);
  if (!(p1 == p2 && p2 == p3 && p3 == p4 && p4 == p5)) return 2;
  if (pl.superRadius > 0.0) {
    auto in = [&](const double *q) {
      return r.lower <= q[0] && q[0] <= r.upper && a.left <= q[1] && q[1] <= b.left;
    };
    if (in(pl.sp1) || in(pl.sp2) || in(pl.sp3) || in(pl.sp4)) return 2;
  }
  return p5 == 1 ? 1 : 0;
}

// ---------------------------------------------------------------------------
// The quadrature of mesh_math.h (qag21, dyadic, integrate) by a CTA of two
// warps: a bisection step's two 21-point panels go one to each warp, a node
// to a lane, and the first warp finishes both (the rule's error formula of
// the two panels side by side on its even and odd lanes), keeps the list and
// picks the next interval while the second waits.  The bound is the FP64
// pipe: a warp's FP64 instruction takes it 64 cycles (76 with all four
// partitions busy) however many lanes it has, so what counts is FP64
// instructions per warp; and a cell's bisections are a serial chain (10-50
// steps, up to the list's 128 where an arc ends inside the cell), which is
// what a small batch waits for.  The sums pack two of the rule's four sums
// into a warp's two halves.  Every thread takes the same branches.  Measured
// against 16 lanes of a warp per cell: one blackbody spot (148 cut cells)
// 2.07 -> 0.38 ms, 100 of them 6.4 -> 6.2 ms (345 FP64 instructions per cell
// and step, the pipe 84 % busy).
// ---------------------------------------------------------------------------
constexpr int kCutThreads = 64;
constexpr int kCutList = 128;
struct CutList {
  double al[kCutList], bl[kCutList], rl[kCutList], el[kCutList];
  double panel[2][4];  // Kronrod, Gauss, |f| and |f - mean| sums of the step's panels
  double next[2], out;  // the next interval; the integral
  int go;               // another step follows
};

__device__ __forceinline__ int k21_slot(int n) { return n < 10 ? n : (n == 10 ? 10 : n - 11); }

// one panel by the calling warp, the four sums into `out`.  Lanes 0-15 carry
// a node each and lanes 16-20 the other five, which fold onto five of the
// first 16.  The pairing and the order of the sums are those of 16 lanes
// taking the 42 nodes of a step in turn (first panel: nodes l and l + 16;
// second: nodes l - 5 and l + 11), the order in which the meshes were always
// summed.
template <typename F>
__device__ __forceinline__ void warp_panel(const F &f, bool second, double a, double b,
                                           double *out) {
  const int lane = threadIdx.x & 31;
  const double c = 0.5 * (a + b), h = 0.5 * (b - a);
  double v = 0.0;
  if (lane < 21) {
    const int m = lane >= 16 ? lane : (second ? (lane < 5 ? lane + 11 : lane - 5) : lane);
    const double x = m == 10 ? 0.0 : XG_K21_X[k21_slot(m)];
    // c - h x, c, c + h x
    v = f(fma(h, m < 10 ? -x : x, c));
  }
  // the first half of the warp sums with the Kronrod weights, the second
  // with the Gauss weights; then the first |f - mean|, the second |f|
  const int fold = second ? 5 : 0, lo = lane & 15;
  const int m1 = second ? (lo < 5 ? lo + 11 : lo - 5) : lo;
  const bool two = lo >= fold && lo < fold + 5;
  const int m2 = lo - fold + 16;
  const double v1 = __shfl_sync(0xffffffffu, v, lo);
  const double v2 = __shfl_sync(0xffffffffu, v, two ? m2 : lo);
  const double wk1 = XG_K21_WK[k21_slot(m1)], wk2 = two ? XG_K21_WK[k21_slot(m2)] : 0.0;
  double w1 = wk1, w2 = wk2;
  if (lane >= 16) {
    w1 = XG_K21_WG[k21_slot(m1)];
    w2 = two ? XG_K21_WG[k21_slot(m2)] : 0.0;
  }
  double s = fma(w2, v2, w1 * v1);
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  const double mean = lane < 16 ? 0.5 * s : 0.0;
  double t = fma(wk2, fabs(v2 - mean), wk1 * fabs(v1 - mean));
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  if (lo == 0) {
    out[lane >> 4] = s;
    out[2 + (lane >> 4)] = t;
  }
}

struct WPanel {
  double res, err, rabs, rasc;
};
__device__ __forceinline__ bool below(double a, double b) {
  return ordered_bits(a) < ordered_bits(b);
}
// result and error estimate of a panel from its sums (QUADPACK's formulas;
// the tests on non-negative finite values by their bit patterns)
__device__ __forceinline__ WPanel k21_finish(const double *p, double a, double b) {
  const double h = 0.5 * (b - a), ah = fabs(h);
  const double rk = p[0], rg = p[1];
  WPanel P;
  P.res = rk * h;
  const double rc = p[2] * ah, ra = p[3] * ah;
  double e = fabs((rk - rg) * h);
  if (ordered_bits(rc) != 0 && ordered_bits(e) != 0) {
    const double x = 200.0 * e / rc, sc = x * sqrt(x);  // x^1.5 without pow
    e = below(sc, 1.0) ? rc * sc : rc;
  }
  const double eps = 2.220446049250313e-16, dmin = 2.2250738585072014e-308;
  if (below(dmin / (50.0 * eps), ra)) {
    const double fl = 50.0 * eps * ra;
    if (below(e, fl)) e = fl;
  }
  P.err = e;
  P.rabs = ra;
  P.rasc = rc;
  return P;
}

// the first interval of largest error, compared as signed 64-bit patterns
// (the errors are non-negative): identical in every lane
__device__ __forceinline__ int worst_interval(const double *el, int size, int lane) {
  long long e = LLONG_MIN;
  int k = 0;
  for (int i = lane; i < size; i += 32) {
    const long long v = __double_as_longlong(el[i]);
    if (v > e) { e = v; k = i; }
  }
  const int hi = (int)(e >> 32);
  const int mh = __reduce_max_sync(0xffffffffu, hi);
  const unsigned lo = hi == mh ? (unsigned)e : 0u;
  const unsigned ml = __reduce_max_sync(0xffffffffu, lo);
  return (int)__reduce_min_sync(0xffffffffu,
                                (hi == mh && (unsigned)e == ml) ? (unsigned)k : 0x7fffffffu);
}

template <typename F>
__device__ double cta_qag21(const F &f, double a, double b, double epsabs, double er,
                            CutList &L) {
  const double eps = 2.220446049250313e-16, dmin = 2.2250738585072014e-308;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  // the first panel
  if (w == 0) {
    warp_panel(f, false, a, b, L.panel[0]);
    __syncwarp();
    const WPanel P = k21_finish(L.panel[0], a, b);
    const double r0 = P.res, e0 = P.err;
    const double tol = (epsabs < er * fabs(r0)) ? er * fabs(r0) : epsabs;
    const bool done = (e0 <= 50.0 * eps * P.rabs && e0 > tol) || (e0 <= tol && e0 != P.rasc) ||
                      e0 == 0.0;
    if (lane == 0) {
      L.al[0] = a; L.bl[0] = b; L.rl[0] = r0; L.el[0] = e0;
      L.next[0] = a; L.next[1] = b;
      L.out = r0;
      L.go = !done;
    }
  }
  __syncthreads();
  double area = L.rl[0], errsum = L.el[0];
  int size = 1, iter = 1, k = 0, rnd1 = 0, rnd2 = 0;
  while (L.go) {
    const double ai = L.next[0], bi = L.next[1];
    const double mid = 0.5 * (ai + bi);
    warp_panel(f, w == 1, w ? mid : ai, w ? bi : mid, L.panel[w]);
    __syncthreads();
    if (w == 0) {
      const double ri = L.rl[k], ei = L.el[k];
      // even lanes finish the first panel, odd lanes the second
      const bool odd = lane & 1;
      const WPanel P = k21_finish(L.panel[odd], odd ? mid : ai, odd ? bi : mid);
      const double r1 = __shfl_sync(0xffffffffu, P.res, 0), r2 = __shfl_sync(0xffffffffu, P.res, 1);
      const double e1 = __shfl_sync(0xffffffffu, P.err, 0), e2 = __shfl_sync(0xffffffffu, P.err, 1);
      const bool flat = __any_sync(0xffffffffu, ordered_bits(P.rasc) == ordered_bits(P.err));
      const double r12 = r1 + r2, e12 = e1 + e2;
      errsum += e12 - ei;
      area += r12 - ri;
      if (!flat) {
        if (!below(1.0e-5 * fabs(r12), fabs(ri - r12)) && !below(e12, 0.99 * ei)) rnd1++;
        if (iter >= 10 && below(ei, e12)) rnd2++;
      }
      const double rt = er * fabs(area);
      const double tol = below(epsabs, rt) ? rt : epsabs;
      const bool above = below(tol, errsum);
      int fail = 0;
      if (above) {
        if (rnd1 >= 6 || rnd2 >= 20) fail = 2;
        const double edge = (1.0 + 100.0 * eps) * (fabs(mid) + 1000.0 * dmin);
        if (!below(edge, fabs(ai)) && !below(edge, fabs(bi))) fail = 3;
      }
      const int nw = size++;
      const bool swap = below(e1, e2);  // the half of larger error stays in place
      if (lane == 0) {
        L.al[k] = swap ? mid : ai; L.bl[k] = swap ? bi : mid;
        L.rl[k] = swap ? r2 : r1; L.el[k] = swap ? e2 : e1;
        L.al[nw] = swap ? ai : mid; L.bl[nw] = swap ? mid : bi;
        L.rl[nw] = swap ? r1 : r2; L.el[nw] = swap ? e1 : e2;
      }
      __syncwarp();
      iter++;
      const bool go = iter < kCutList && !fail && above;
      if (go) {
        k = worst_interval(L.el, size, lane);
        if (lane == 0) {
          L.next[0] = L.al[k];
          L.next[1] = L.bl[k];
        }
      } else {
        double sum = 0.0;
        for (int i = 0; i < size; i++) sum += L.rl[i];
        if (lane == 0) {
          L.out = sum;
          L.go = 0;
        }
      }
    }
    __syncthreads();
  }
  const double r = L.out;
  __syncthreads();  // the next integral's first panel rewrites the list
  return r;
}

// piece k of the dyadic cut of [lo, hi] toward an endpoint; false past the
// last one (the cut has reached the endpoint's rounding)
__device__ __forceinline__ bool dyadic_piece(double lo, double hi, bool toward_lo, int k,
                                             double &p0, double &p1) {
  const double Lw = hi - lo;
  const double s1 = ldexp(Lw, -(k + 1)), s0 = ldexp(Lw, -k);
  p0 = toward_lo ? lo + s1 : hi - s0;
  p1 = toward_lo ? lo + s0 : hi - s1;
  return p0 < p1 && !(toward_lo ? p0 <= lo : p1 >= hi);
}
// the sum over the pieces in turn, until four are negligible; the first
// n_done pieces' integrals are given
template <typename F>
__device__ double cta_dyadic(const F &f, double lo, double hi, bool toward_lo, double er,
                             CutList &L, const double *done, int n_done) {
  double sum = 0.0;
  int seen = 0, quiet = 0;
  for (int k = 0; k < 2100; k++) {
    double p0, p1;
    if (!dyadic_piece(lo, hi, toward_lo, k, p0, p1)) break;
    const double r = k < n_done ? done[k] : cta_qag21(f, p0, p1, 0.0, er, L);
    sum += r;
    if (r != 0.0) seen = 1;
    if (seen && fabs(r) <= 1.0e-17 * fabs(sum)) {
      if (++quiet >= 4) break;
    } else {
      quiet = 0;
    }
  }
  return sum;
}

// the relative tolerance integrate() (mesh_math.h) runs at for CQUAD's 1e-8
constexpr double kCutTol = 1.0e-13;

// an integral whose interior nodes all see zero but an endpoint does not, cut
// in two halves: dyadic pieces toward such an endpoint, else plainly
struct DyadicSplit {
  double a, b;
  bool at_a, at_b;
};
template <typename F>
__device__ double cta_halves(const F &f, const DyadicSplit &d, CutList &L, const double *done,
                             int n_done) {
  const double m = 0.5 * (d.a + d.b);
  const double rl = d.at_a ? cta_dyadic(f, d.a, m, true, kCutTol, L, done, n_done)
                    : n_done ? done[0] : cta_qag21(f, d.a, m, 0.0, kCutTol, L);
  const double rr = d.at_b ? cta_dyadic(f, m, d.b, false, kCutTol, L, done + n_done, n_done)
                    : n_done ? done[n_done] : cta_qag21(f, m, d.b, 0.0, kCutTol, L);
  return rl + rr;
}
// integrate() of mesh_math.h over [a, b], a < b; true in `split` (when asked
// for): the halves of d are left to the caller
template <typename F>
__device__ double cta_integrate(const F &f, double a, double b, CutList &L, DyadicSplit *d,
                                bool &split) {
  split = false;
  double sign = 1.0;
  if (b < a) { const double t = a; a = b; b = t; sign = -1.0; }
  if (a == b) return 0.0;
  double r = cta_qag21(f, a, b, 0.0, kCutTol, L);
  if (r == 0.0) {
    const double fa = f(a), fb = f(b);
    if (fa != 0.0 || fb != 0.0) {
      const DyadicSplit h{a, b, fa != 0.0, fb != 0.0};
      if (d != nullptr && sign > 0.0) {
        *d = h;
        split = true;
        return 0.0;
      }
      r = cta_halves(f, h, L, nullptr, 0);
    }
  }
  return sign * r;
}

__device__ __forceinline__ int mesh_of_cell(const MeshJob *jobs, int n_mesh, int64_t c) {
  int lo = 0, hi = n_mesh - 1;
  while (lo < hi) {  // last mesh whose cell_off <= c
    const int mid = (lo + hi + 1) >> 1;
    if (jobs[mid].cell_off <= c) lo = mid; else hi = mid - 1;
  }
  return lo;
}

__device__ __forceinline__ void put_area(const MeshJob &J, xgpu_mesh_batch_out &o, int64_t c,
                                         size_t i, size_t j, double A) {
  const size_t S = J.pl.S;
  o.cellArea[c] = A;
  o.radiates[c] = A > 0.0 ? 1 : 0;
  if (J.pl.sym) {
    const int64_t cm = J.cell_off + (int64_t)(i * S + (S - 1 - j));
    o.cellArea[cm] = A;
    o.radiates[cm] = A > 0.0 ? 1 : 0;
  }
}

// one thread per cell of the batch (cells of mesh m at [cell_off, cell_off + S^2))
__global__ void __launch_bounds__(128) mesh_cells_kernel(const MeshJob *jobs, int n_mesh,
                                                         int64_t n_cells, xgpu_mesh_batch_out o,
                                                         const RowTmp *row_tmp,
                                                         const double *mesh_tmp,
                                                         const MeshTrig *trig,
                                                         const ColTrig *cols, int S_max,
                                                         int64_t *queue, unsigned *n_queue) {
  const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= n_cells) return;
  const int m = mesh_of_cell(jobs, n_mesh, c);
  const MeshJob &J = jobs[m];
  const size_t S = J.pl.S;
  const int64_t k = c - J.cell_off;
  const size_t i = (size_t)(k / (int64_t)S), j = (size_t)(k - (int64_t)i * (int64_t)S);
  const RowTmp &r = row_tmp[J.row_off + (int64_t)i];
  // azimuth (shifted by the omitted region's azimuth, half a turn when
  // antiphased) and the atmosphere parameters of the cell
  double ph = mesh_phi(J.pl, j) - J.omit_azimuth;
  if (J.antiphased) ph = ph + PI;
  o.phi[c] = ph;
  o.params[2 * c] = J.logT;
  o.params[2 * c + 1] = r.effGrav;
  const size_t j_max = J.pl.j_max;
  if (j < j_max) {
    const ColTrig *ct = cols + (size_t)m * (S_max + 1) + j;
    const int kind = cell_kind(J.pl, trig[m], r, ct[0], ct[1], i);
    if (kind == 2) queue[atomicAdd(n_queue, 1u)] = c;
    else put_area(J, o, c, i, j, kind == 1 ? mesh_tmp[2 * m] : 0.0);
  } else if (!J.pl.sym || j < S - j_max) {
    // columns no mirror reaches keep area 0
    o.cellArea[c] = 0.0;
    o.radiates[c] = 0;
  }
}

// A cell that a region's arc touches at a corner only has an integral that the
// first panel's nodes miss and its dyadic pieces resolve, some 60 quadratures
// of about 7 bisections each: in turn 400 steps, ten times any other cell, so
// its pieces are set aside (room for `cap` cells; one that finds none runs
// them in turn), integrated a CTA each, and summed in order at the end.
constexpr int kPieces = 64;  // of a half; what lies beyond is integrated in turn
struct SplitCell {
  int64_t cell;
  DyadicSplit d;
  bool last;  // the integral between the boundary's crossings: nothing follows
};
struct SplitList {
  SplitCell *cells;
  double *piece;    // [cap][2][kPieces]
  unsigned *count;  // cells set aside; the piece items' counter
  unsigned cap;
};

// a queued cell's integrand
__device__ __forceinline__ void cut_cell(const MeshJob *jobs, int n_mesh, const RowTmp *row_tmp,
                                         const MeshTrig *trig, const ColTrig *cols, int S_max,
                                         int64_t c, int &m, size_t &i, size_t &j, double &lower,
                                         double &upper, CutCell &f) {
  m = mesh_of_cell(jobs, n_mesh, c);
  const MeshJob &J = jobs[m];
  const size_t S = J.pl.S;
  const int64_t k = c - J.cell_off;
  i = (size_t)(k / (int64_t)S);
  j = (size_t)(k - (int64_t)i * (int64_t)S);
  const RowTmp &r = row_tmp[J.row_off + (int64_t)i];
  lower = r.lower;
  upper = r.upper;
  const ColTrig *ct = cols + (size_t)m * (S_max + 1) + j;
  f.init(CellIntegrand{J.s, trig[m].g, ct[0].left, ct[1].left}, lower, upper);
}
// the area from the first integral: the reference integrates again between
// the boundary's crossings where it vanishes
__device__ __forceinline__ void finish_cell(const MeshJob &J, xgpu_mesh_batch_out &o, int64_t c,
                                            size_t i, size_t j, double lower, double upper,
                                            const CutCell &f, double integral, CutList &L) {
  if (are_equal(integral, 0.0)) {
    double tmin, tmax;
    bool split;
    if (cell_fallback_interval(lower, upper, f.f.pa, f.f.pb, f.f.g, tmin, tmax))
      integral = cta_integrate(f, tmin, tmax, L, nullptr, split);
  }
  if (threadIdx.x == 0) put_area(J, o, c, i, j, J.s.R_eq * J.s.R_eq * integral);
}

// ---------------------------------------------------------------------------
// Many queued cells: eight lanes per cell, four cells per warp.  With the
// chip full what counts is the FP64 pipe, so the warp's instructions are
// filled: a bisection step's 42 nodes are six instruction streams for four
// cells (a CTA of two warps takes two for one), and the sums, the panels'
// error formulas and the list's bookkeeping run for the four at once.  The
// groups step together; one whose cell is done takes the next.  A first panel
// is a step whose second panel is idle.  The sums have the order of
// warp_panel (lane l holds its slots l and l + 8), so the areas are the same
// bits.  A cell whose integral vanishes (the reference looks at it again) is
// left to the boundary kernel.
// Measured, CTA per cell against this: 100 blackbody spots 6.35, 5.33 ms; 256
// prior vectors of two regions 80.8, 66.5 ms (fewer cells do not fill the
// groups: the rule kPackedMin).  With the nodes queued
// between the integrand's stages (PackQueue) and four sums to a reduction the
// two large batches take 4.23 and 49.4 ms (5.32 and 60.3 without).  Two CTAs per SM keep the
// pipe full (82-85 % busy) and leave each group several cells; four leave
// lone cells in their warps at the end (6.33 ms for the 100 spots).
// ---------------------------------------------------------------------------
constexpr int kPackThreads = 128, kPackCells = kPackThreads / 8, kPackList = kCutList;
constexpr int kPackCtasPerSm = 2;
struct PackLists {
  double al[kPackList], bl[kPackList], rl[kPackList], el[kPackList];
  double v[2][21];
  CutCell f;
};
// The nodes of a warp's step: cosine and sine of the colatitude, and the
// queues of those that need a boundary's azimuth and of those whose value is
// wanted (group 42 + panel 21 + node, and the node's place above 8 bits).  An
// FP64 instruction costs the same for one lane as for 32, and only 43 % and 63
// % of the nodes get there: queued, they take 3 and 4 turns in place of 6.
constexpr int kPackNodes = 4 * 42;
struct PackQueue {
  double mu[kPackNodes], st[kPackNodes];
  unsigned short edge[kPackNodes], value[kPackNodes];
};
struct PackSmem {
  PackLists lists[kPackCells];
  PackQueue queues[kPackThreads / 32];
};
// about 130 cells a spot and 460 a vector of two regions; CTA per cell against
// packed: 20 spots 1.55, 1.90 ms, 40 2.70, 2.12, 60 3.96, 2.96; 7 vectors 2.49,
// 2.57, 11 3.33, 3.28, 13 4.05, 3.60; 9 prior vectors 2.78, 3.18
constexpr unsigned kPackedMin = 5000;
struct CellQueue {
  int64_t *cells, *left;  // queued; left to the boundary kernel
  unsigned *count;        // queued, next of the boundary kernel, left, next of the packed one
  unsigned packed_min;    // queued cells from which the packed kernel takes them
};
// sums of four values over the lanes of a group, to every lane, with four
// additions (the bits of four butterflies of three): a lane carries one of them
// once the others' share is handed over
__device__ __forceinline__ double hand_over(double low, double high, int lane, int o) {
  const bool up = lane & o;
  return (up ? high : low) + __shfl_xor_sync(0xffffffffu, up ? low : high, o);
}
__device__ __forceinline__ void group_sum4(double &a, double &b, double &c, double &d, int lane) {
  double v = hand_over(hand_over(a, b, lane, 4), hand_over(c, d, lane, 4), lane, 2);
  v += __shfl_xor_sync(0xffffffffu, v, 1);
  const int g0 = lane & 24;
  a = __shfl_sync(0xffffffffu, v, g0);
  b = __shfl_sync(0xffffffffu, v, g0 + 4);
  c = __shfl_sync(0xffffffffu, v, g0 + 2);
  d = __shfl_sync(0xffffffffu, v, g0 + 6);
}
__global__ void __launch_bounds__(kPackThreads, kPackCtasPerSm) mesh_packed_kernel(
    const MeshJob *jobs, int n_mesh, xgpu_mesh_batch_out o, const RowTmp *row_tmp,
    const MeshTrig *trig, const ColTrig *cols, int S_max, CellQueue Q) {
  extern __shared__ double pack_smem[];
  PackSmem &S = *reinterpret_cast<PackSmem *>(pack_smem);
  const unsigned n = Q.count[0];
  if (n < Q.packed_min) return;
  const double eps = 2.220446049250313e-16, dmin = 2.2250738585072014e-308;
  const int lane = threadIdx.x & 31, l = lane & 7, g0 = lane & 24;
  PackLists &L = S.lists[threadIdx.x >> 3];
  PackLists *LW = S.lists + (threadIdx.x >> 5) * 4;  // the warp's four
  PackQueue &N = S.queues[threadIdx.x >> 5];
  int64_t c = 0;
  int m = 0;
  size_t i = 0, j = 0;
  bool have = false, more = true, first = false;
  double ai = 0.0, bi = 0.0, area = 0.0, errsum = 0.0;
  int size = 0, iter = 0, k = 0, rnd1 = 0, rnd2 = 0;
  for (;;) {
    if (!have && more) {
      unsigned q = 0;
      if (l == 0) q = atomicAdd(&Q.count[3], 1u);
      q = __shfl_sync(0xffu << g0, q, g0);
      more = q < n;
      if (more) {
        c = Q.cells[q];
        CutCell f;
        cut_cell(jobs, n_mesh, row_tmp, trig, cols, S_max, c, m, i, j, ai, bi, f);
        if (l == 0) L.f = f;
        have = first = true;
      }
    }
    __syncwarp();
    if (!__any_sync(0xffffffffu, have)) return;
    // the step's nodes: their places
    const double mid = first ? bi : 0.5 * (ai + bi);
    int n_edge = 0, n_value = 0;
    const unsigned below_me = (1u << lane) - 1u;
    auto push = [&](unsigned short *queue, int &count, bool on, int item) {
      const unsigned mask = __ballot_sync(0xffffffffu, on);
      if (on) queue[count + __popc(mask & below_me)] = (unsigned short)item;
      count += __popc(mask);
    };
#pragma unroll 1
    for (int p = 0; p < 6; p++) {
      const int z = p >= 3, nd = l + 8 * (p - 3 * z);
      const double a = z ? mid : ai, b = z ? bi : mid;
      const double ctr = 0.5 * (a + b), h = 0.5 * (b - a);
      const int id = (g0 >> 3) * 42 + z * 21 + nd;
      int where = -1;
      if (have && nd < 21 && !(first && z)) {
        const double x = nd == 10 ? 0.0 : XG_K21_X[k21_slot(nd)];
        const double theta = fma(h, nd < 10 ? -x : x, ctr);
        double mu, st, keep = 0.0;
        where = L.f.place(theta, mu, st);
        if (where >= 0) {
          N.mu[id] = mu;
          N.st[id] = st;
          keep = where & CutCell::kEdge ? theta : L.f.f.pb - L.f.f.pa;
        }
        L.v[z][nd] = keep;  // the colatitude, the width, then the value
      }
      push(N.edge, n_edge, where >= 0 && (where & CutCell::kEdge), id | where << 8);
      push(N.value, n_value, where >= 0 && !(where & CutCell::kEdge), id);
    }
    // the widths of those at a boundary
#pragma unroll 1
    for (int t = lane; t - lane < n_edge; t += 32) {
      __syncwarp();
      int id = 0;
      bool some = false;
      if (t < n_edge) {
        const int item = N.edge[t];
        id = item & 255;
        PackLists &G = LW[id / 42];
        double &v = G.v[0][id % 42];
        const double w = G.f.width(v, item >> 8, N.mu[id], N.st[id]);
        some = ordered_bits(w) != 0;
        v = some ? w : 0.0;
      }
      push(N.value, n_value, some, id);
    }
    // the values
    __syncwarp();
#pragma unroll 1
    for (int t = lane; t < n_value; t += 32) {
      const int id = N.value[t];
      PackLists &G = LW[id / 42];
      double &v = G.v[0][id % 42];
      v = G.f.value(v, N.mu[id], N.st[id]);
    }
    __syncwarp();
    // the four sums of either panel; even lanes keep the first's
    double ps[4], v1[2][2], v2[2][2], k1[2][2], k2[2][2], sk[2], sg[2], sm[2], sa[2];
#pragma unroll
    for (int z = 0; z < 2; z++) {
#pragma unroll
      for (int t = 0; t < 2; t++) {
        const int lo = l + 8 * t;
        const int m1 = z ? (lo < 5 ? lo + 11 : lo - 5) : lo;
        const bool two = z ? (lo >= 5 && lo < 10) : lo < 5;
        const int m2 = z ? lo + 11 : lo + 16;
        v1[z][t] = L.v[z][m1];
        v2[z][t] = two ? L.v[z][m2] : v1[z][t];
        k1[z][t] = XG_K21_WK[k21_slot(m1)];
        k2[z][t] = two ? XG_K21_WK[k21_slot(m2)] : 0.0;
        const double g1 = XG_K21_WG[k21_slot(m1)], g2 = two ? XG_K21_WG[k21_slot(m2)] : 0.0;
        const double a = fma(k2[z][t], v2[z][t], k1[z][t] * v1[z][t]);
        const double b = fma(g2, v2[z][t], g1 * v1[z][t]);
        sk[z] = t ? sk[z] + a : a;
        sg[z] = t ? sg[z] + b : b;
      }
    }
    group_sum4(sk[0], sg[0], sk[1], sg[1], lane);
#pragma unroll
    for (int z = 0; z < 2; z++) {
      const double mean = 0.5 * sk[z];
      sm[z] = fma(k2[z][0], fabs(v2[z][0] - mean), k1[z][0] * fabs(v1[z][0] - mean));
      sm[z] += fma(k2[z][1], fabs(v2[z][1] - mean), k1[z][1] * fabs(v1[z][1] - mean));
      sa[z] = fma(k2[z][0], fabs(v2[z][0]), k1[z][0] * fabs(v1[z][0]));
      sa[z] += fma(k2[z][1], fabs(v2[z][1]), k1[z][1] * fabs(v1[z][1]));
    }
    group_sum4(sm[0], sa[0], sm[1], sa[1], lane);
    const bool odd = lane & 1;
    ps[0] = odd ? sk[1] : sk[0];
    ps[1] = odd ? sg[1] : sg[0];
    ps[2] = odd ? sm[1] : sm[0];
    ps[3] = odd ? sa[1] : sa[0];
    const WPanel P = k21_finish(ps, odd ? mid : ai, odd ? bi : mid);
    const double r1 = __shfl_sync(0xffffffffu, P.res, g0);
    const double r2 = __shfl_sync(0xffffffffu, P.res, g0 + 1);
    const double e1 = __shfl_sync(0xffffffffu, P.err, g0);
    const double e2 = __shfl_sync(0xffffffffu, P.err, g0 + 1);
    const double ra = __shfl_sync(0xffffffffu, P.rabs, g0);
    const double rc = __shfl_sync(0xffffffffu, P.rasc, g0);
    const bool flat = (__ballot_sync(0xffffffffu, ordered_bits(P.rasc) == ordered_bits(P.err)) &
                       (0xffu << g0)) != 0u;
    bool go = false, leave = false;
    double out = 0.0;
    if (have && first) {
      const double tol = below(0.0, kCutTol * fabs(r1)) ? kCutTol * fabs(r1) : 0.0;
      const bool done = (e1 <= 50.0 * eps * ra && e1 > tol) || (e1 <= tol && e1 != rc) ||
                        e1 == 0.0;
      if (l == 0) {
        L.al[0] = ai; L.bl[0] = bi; L.rl[0] = r1; L.el[0] = e1;
      }
      area = r1;
      errsum = e1;
      size = iter = 1;
      k = rnd1 = rnd2 = 0;
      first = false;
      go = !done;
      out = r1;
      leave = !(ai < bi);
    } else if (have) {
      const double ri = L.rl[k], ei = L.el[k];
      const double r12 = r1 + r2, e12 = e1 + e2;
      errsum += e12 - ei;
      area += r12 - ri;
      if (!flat) {
        if (!below(1.0e-5 * fabs(r12), fabs(ri - r12)) && !below(e12, 0.99 * ei)) rnd1++;
        if (iter >= 10 && below(ei, e12)) rnd2++;
      }
      const double rt = kCutTol * fabs(area);
      const double tol = below(0.0, rt) ? rt : 0.0;
      const bool above = below(tol, errsum);
      int fail = 0;
      if (above) {
        if (rnd1 >= 6 || rnd2 >= 20) fail = 2;
        const double edge = (1.0 + 100.0 * eps) * (fabs(mid) + 1000.0 * dmin);
        if (!below(edge, fabs(ai)) && !below(edge, fabs(bi))) fail = 3;
      }
      const int nw = size++;
      const bool swap = below(e1, e2);  // the half of larger error stays in place
      __syncwarp(0xffu << g0);  // its lanes have read the list
      if (l == 0) {
        L.al[k] = swap ? mid : ai; L.bl[k] = swap ? bi : mid;
        L.rl[k] = swap ? r2 : r1; L.el[k] = swap ? e2 : e1;
        L.al[nw] = swap ? ai : mid; L.bl[nw] = swap ? mid : bi;
        L.rl[nw] = swap ? r1 : r2; L.el[nw] = swap ? e1 : e2;
      }
      iter++;
      go = iter < kCutList && !fail && above;
    }
    __syncwarp();
    // the first interval of largest error, as worst_interval
    long long we = LLONG_MIN;
    int wk = 0;
    if (have && go)
      for (int q = l; q < size; q += 8) {
        const long long e = __double_as_longlong(L.el[q]);
        if (e > we) { we = e; wk = q; }
      }
#pragma unroll
    for (int s = 4; s > 0; s >>= 1) {
      const long long e = __shfl_xor_sync(0xffffffffu, we, s);
      const int q = __shfl_xor_sync(0xffffffffu, wk, s);
      if (e > we || (e == we && q < wk)) { we = e; wk = q; }
    }
    if (have && go && !leave) {
      k = wk;
      ai = L.al[k];
      bi = L.bl[k];
    } else if (have) {
      if (!leave) {
        if (iter > 1) {
          out = 0.0;
          for (int q = 0; q < size; q++) out += L.rl[q];
        }
        leave = are_equal(out, 0.0);
      }
      if (l == 0) {
        const MeshJob &J = jobs[m];
        if (leave) Q.left[atomicAdd(&Q.count[2], 1u)] = c;
        else put_area(J, o, c, i, j, J.s.R_eq * J.s.R_eq * out);
      }
      have = false;
    }
    __syncwarp();
  }
}

// one CTA per queued cell: the area quadrature of a cell cut by a boundary.
// A CTA starts with the cell of its own index (a small batch's cells spread
// over the SMs) and takes the next from a shared counter (n_queue[1]) when it
// finishes one, as the cells' costs differ by 5x or more (10-50 bisection
// steps); each cell's result is independent of which CTA integrates it.
constexpr int kCutCtasPerSm = 8;
__global__ void __launch_bounds__(kCutThreads, kCutCtasPerSm) mesh_boundary_kernel(
    const MeshJob *jobs, int n_mesh, xgpu_mesh_batch_out o, const RowTmp *row_tmp,
    const MeshTrig *trig, const ColTrig *cols, int S_max, CellQueue Q, SplitList sl) {
  __shared__ CutList L;
  __shared__ unsigned s_q;
  const bool packed = Q.count[0] >= Q.packed_min;
  const unsigned n = packed ? Q.count[2] : Q.count[0];
  const int64_t *queue = packed ? Q.left : Q.cells;
  for (unsigned q = blockIdx.x; q < n; q = s_q) {
    const int64_t c = queue[q];
    int m;
    size_t i, j;
    double lower, upper;
    CutCell f;
    cut_cell(jobs, n_mesh, row_tmp, trig, cols, S_max, c, m, i, j, lower, upper, f);
    DyadicSplit d;
    bool split, last = false;
    double integral = cta_integrate(f, lower, upper, L, &d, split);
    if (!split && are_equal(integral, 0.0)) {
      // (finish_cell's second integral, whose pieces may be set aside as well:
      // in turn they held 256 prior vectors' kernel up, 6.3 ms, now 4.1)
      double tmin, tmax;
      last = cell_fallback_interval(lower, upper, f.f.pa, f.f.pb, f.f.g, tmin, tmax);
      if (last) integral = cta_integrate(f, tmin, tmax, L, &d, split);
    }
    __syncthreads();  // every thread has read the last s_q
    const MeshJob &J = jobs[m];
    if (split) {
      if (threadIdx.x == 0) {
        const unsigned at = atomicAdd(&sl.count[0], 1u);
        if (at < sl.cap) sl.cells[at] = SplitCell{c, d, last};
        s_q = at;
      }
      __syncthreads();
      const bool room = s_q < sl.cap;
      __syncthreads();
      if (!room) {
        integral = cta_halves(f, d, L, nullptr, 0);
        if (!last) finish_cell(J, o, c, i, j, lower, upper, f, integral, L);
      }
      split = room || !last;
    }
    if (!split && threadIdx.x == 0) put_area(J, o, c, i, j, J.s.R_eq * J.s.R_eq * integral);
    if (threadIdx.x == 0) s_q = gridDim.x + atomicAdd(&Q.count[1], 1u);
    __syncthreads();
  }
}

// the dyadic pieces of the cells set aside, one CTA per piece
__global__ void __launch_bounds__(kCutThreads, kCutCtasPerSm) mesh_pieces_kernel(
    const MeshJob *jobs, int n_mesh, const RowTmp *row_tmp, const MeshTrig *trig,
    const ColTrig *cols, int S_max, SplitList sl) {
  __shared__ CutList L;
  __shared__ unsigned s_q;
  const unsigned n = min(sl.count[0], sl.cap) * (2u * kPieces);
  for (unsigned q = blockIdx.x; q < n; q = s_q) {
    const SplitCell sc = sl.cells[q / (2u * kPieces)];
    const unsigned h = (q / kPieces) & 1u, k = q % kPieces;
    const DyadicSplit &d = sc.d;
    const double mid = 0.5 * (d.a + d.b), lo = h ? mid : d.a, hi = h ? d.b : mid;
    double p0 = lo, p1 = hi;
    const bool any = (h ? d.at_b : d.at_a) ? dyadic_piece(lo, hi, h == 0, (int)k, p0, p1) : k == 0;
    if (any) {
      int m;
      size_t i, j;
      double lower, upper;
      CutCell f;
      cut_cell(jobs, n_mesh, row_tmp, trig, cols, S_max, sc.cell, m, i, j, lower, upper, f);
      const double r = cta_qag21(f, p0, p1, 0.0, kCutTol, L);
      if (threadIdx.x == 0) sl.piece[q] = r;
    }
    __syncthreads();
    if (threadIdx.x == 0) s_q = gridDim.x + atomicAdd(&sl.count[1], 1u);
    __syncthreads();
  }
}

// ... and their areas, one CTA per cell
__global__ void __launch_bounds__(kCutThreads) mesh_split_kernel(
    const MeshJob *jobs, int n_mesh, xgpu_mesh_batch_out o, const RowTmp *row_tmp,
    const MeshTrig *trig, const ColTrig *cols, int S_max, SplitList sl) {
  __shared__ CutList L;
  const unsigned n = min(sl.count[0], sl.cap);
  for (unsigned q = blockIdx.x; q < n; q += gridDim.x) {
    const SplitCell sc = sl.cells[q];
    int m;
    size_t i, j;
    double lower, upper;
    CutCell f;
    cut_cell(jobs, n_mesh, row_tmp, trig, cols, S_max, sc.cell, m, i, j, lower, upper, f);
    const double integral =
        cta_halves(f, sc.d, L, sl.piece + (size_t)q * 2 * kPieces, kPieces);
    const MeshJob &J = jobs[m];
    if (!sc.last) finish_cell(J, o, sc.cell, i, j, lower, upper, f, integral, L);
    else if (threadIdx.x == 0) put_area(J, o, sc.cell, i, j, J.s.R_eq * J.s.R_eq * integral);
    __syncthreads();
  }
}

// a call's device scratch: one allocation, parts at 256-byte boundaries
struct MeshScratch {
  size_t jobs, tab, row, mesh, par, trig, cols, queue, left, count, split, piece, total;
  unsigned cap;  // of the split list
  bool pack;     // the packed kernel is launched
};
MeshScratch mesh_scratch(size_t n, size_t n_rows, size_t n_cells, size_t S_max) {
  MeshScratch o{};
  auto part = [&](size_t bytes) {
    const size_t at = o.total;
    o.total += (bytes + 255) & ~size_t(255);
    return at;
  };
  o.jobs = part(sizeof(MeshJob) * n);
  o.tab = part(sizeof(double) * n * kAreaTab);
  o.row = part(sizeof(RowTmp) * n_rows);
  o.mesh = part(sizeof(double) * 2 * n);
  o.par = part(sizeof(double) * n * S_max);
  o.trig = part(sizeof(MeshTrig) * n);
  o.cols = part(sizeof(ColTrig) * n * (S_max + 1));
  o.queue = part(sizeof(int64_t) * n_cells);
  // the packed kernel is launched where the batch may queue enough cells (a
  // region's edge cuts some two cells of each parallel, up to about six)
  o.pack = n_rows >= kPackedMin / 6;
  o.left = part(o.pack ? sizeof(int64_t) * n_cells : 0);
  o.count = part(6 * sizeof(unsigned));
  o.cap = (unsigned)(4 * n + 64);
  o.split = part(sizeof(SplitCell) * o.cap);
  o.piece = part(sizeof(double) * 2 * kPieces * o.cap);
  return o;
}

}  // namespace
}  // namespace xg

extern "C" int64_t xgpu_mesh_scratch_bytes(int n, int64_t n_rows, int64_t n_cells, size_t S_max) {
  if (n <= 0) return 0;
  return (int64_t)xg::mesh_scratch((size_t)n, (size_t)n_rows, (size_t)n_cells, S_max).total;
}

extern "C" int xgpu_mesh_batch(int n, const xgpu_mesh_member *members, int64_t n_rows,
                               int64_t n_cells, const xgpu_mesh_batch_out *out, void *stream) {
  using namespace xg;
  if (n <= 0) return 0;
  if (members == nullptr || out == nullptr) return -2;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  std::vector<MeshJob> jobs((size_t)n);
  size_t S_max = 2;
  int64_t rows = 0, cells = 0;
  for (int m = 0; m < n; m++) {
    const xgpu_mesh_member &q = members[m];
    if (q.S < 2) return -2;
    MeshJob &J = jobs[(size_t)m];
    mesh_plan(q.polar != 0, q.num_cells, q.S, q.cede_radius, q.cede_colatitude, q.super_radius,
              q.super_colatitude, q.super_azimuth, J.pl);
    J.s = Star{q.R_eq, q.epsilon, q.zeta, 0.0, q.star_shape_ind};
    J.row_off = q.row_off;
    J.cell_off = q.cell_off;
    J.r_s = q.r_s;
    J.R_over_rs = q.R_eq / q.r_s;
    J.lag_scale = q.lag_scale;
    J.omit_azimuth = q.omit_azimuth;
    J.antiphased = q.antiphased;
    J.logT = q.logT;
    if (q.row_off != rows || q.cell_off != cells) return -2;  // packed in member order
    rows += (int64_t)q.S;
    cells += (int64_t)(q.S * q.S);
    S_max = std::max(S_max, q.S);
  }
  if (rows != n_rows || cells != n_cells) return -2;
  // (the parallels' shared memory: up to 14,000 of them a mesh)
  const size_t smem = sizeof(double) * (kAreaTab + 2 * S_max + 1);
  if (smem > 48 * 1024 &&
      (smem > 227 * 1024 ||
       cudaFuncSetAttribute(mesh_parallels_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                            (int)smem) != cudaSuccess)) {
    cudaGetLastError();
    return -5;
  }
  const MeshScratch o = mesh_scratch((size_t)n, (size_t)n_rows, (size_t)n_cells, S_max);
  const int S_m = (int)S_max;
  unsigned char *base = nullptr;
  if (cudaMallocAsync(reinterpret_cast<void **>(&base), o.total, st) != cudaSuccess) return -5;
  MeshJob *d_jobs = reinterpret_cast<MeshJob *>(base + o.jobs);
  double *tab = reinterpret_cast<double *>(base + o.tab);
  RowTmp *row_tmp = reinterpret_cast<RowTmp *>(base + o.row);
  double *mesh_tmp = reinterpret_cast<double *>(base + o.mesh);
  double *par = reinterpret_cast<double *>(base + o.par);
  MeshTrig *trig = reinterpret_cast<MeshTrig *>(base + o.trig);
  ColTrig *cols = reinterpret_cast<ColTrig *>(base + o.cols);
  int64_t *queue = reinterpret_cast<int64_t *>(base + o.queue);
  unsigned *n_queue = reinterpret_cast<unsigned *>(base + o.count);
  SplitList sl{};
  sl.cap = o.cap;
  sl.cells = reinterpret_cast<SplitCell *>(base + o.split);
  sl.piece = reinterpret_cast<double *>(base + o.piece);
  sl.count = n_queue + 4;
  const CellQueue Q{queue, reinterpret_cast<int64_t *>(base + o.left), n_queue,
                    o.pack ? kPackedMin : UINT_MAX};
  // (a copy from pageable memory has been staged when cudaMemcpyAsync
  // returns, so the host jobs may go out of scope)
  cudaMemcpyAsync(d_jobs, jobs.data(), sizeof(MeshJob) * (size_t)n, cudaMemcpyHostToDevice, st);
  // queue length, next cell, cells left, next packed; cells set aside, next piece
  cudaMemsetAsync(n_queue, 0, 6 * sizeof(unsigned), st);
  if (n <= kWarpTables)
    mesh_table_kernel<true><<<dim3((kAreaTab + 3) / 4, (unsigned)n), 128, 0, st>>>(d_jobs, tab);
  else
    mesh_table_kernel<false><<<dim3((kAreaTab + 127) / 128, (unsigned)n), 128, 0, st>>>(d_jobs,
                                                                                       tab);
  mesh_parallels_kernel<<<(unsigned)n, 128, smem, st>>>(d_jobs, tab, par, mesh_tmp, trig, cols,
                                                        S_m);
  mesh_rows_kernel<<<(unsigned)((n_rows + 3) / 4), 128, 0, st>>>(d_jobs, n, n_rows, par, S_m,
                                                                 mesh_tmp, *out, row_tmp);
  mesh_cells_kernel<<<(unsigned)((n_cells + 127) / 128), 128, 0, st>>>(
      d_jobs, n, n_cells, *out, row_tmp, mesh_tmp, trig, cols, S_m, queue, n_queue);
  if (o.pack) {
    const size_t lists = sizeof(PackSmem);
    cudaFuncSetAttribute(mesh_packed_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)lists);
    mesh_packed_kernel<<<152 * kPackCtasPerSm, kPackThreads, lists, st>>>(
        d_jobs, n, *out, row_tmp, trig, cols, S_m, Q);
  }
  mesh_boundary_kernel<<<152 * kCutCtasPerSm, kCutThreads, 0, st>>>(
      d_jobs, n, *out, row_tmp, trig, cols, S_m, Q, sl);
  mesh_pieces_kernel<<<152 * kCutCtasPerSm, kCutThreads, 0, st>>>(d_jobs, n, row_tmp, trig, cols,
                                                                 S_m, sl);
  mesh_split_kernel<<<(unsigned)std::min<size_t>(sl.cap, 152), kCutThreads, 0, st>>>(
      d_jobs, n, *out, row_tmp, trig, cols, S_m, sl);
  const cudaError_t e = cudaGetLastError();
  cudaFreeAsync(base, st);
  return e == cudaSuccess ? 0 : -5;
}
