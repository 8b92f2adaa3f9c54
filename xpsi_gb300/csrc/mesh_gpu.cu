// mesh_gpu.cu -- K0: the hot-region cell meshes of a batch, built on the GPU
// from the steps of mesh_math.h (xpsi/cellmesh/mesh.pyx:23-417,
// polar_mesh.pyx:23-430, mesh_tools.pyx:18-890) and written straight into
// the packed per-row and per-cell arrays the rays and integrator kernels read
// (the packing of xpsi/HotRegion.py:774-1017 / Likelihood.py:297-432 that
// the host path does in numpy).
//
// Four launches over all meshes of the batch:
//   1. the 1000-point table of area(colat..lims[1]) per mesh, one thread per
//      entry (1000 independent adaptive quadratures);
//   2. per mesh: the cell area and the S - 1 parallels (one thread, the
//      reference's running sum), then one thread per parallel for its
//      centre colatitude, radius, gravity, tilt and the packed row values;
//   3. one thread per cell: the corner / centre membership tests; cells
//      wholly inside or outside get their area at once, cells cut by a
//      region boundary (~1 %) are queued;
//   4. one CTA of two warps per queued cell, taken from a shared counter: its
//      area quadrature, a panel to each warp (21 Gauss-Kronrod nodes over the
//      lanes, the interval list in shared memory) -- the same adaptive scheme
//      the host builder runs serially.
// The per-thread quadratures of steps 1-2 keep their interval list (128
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

__global__ void __launch_bounds__(128) mesh_table_kernel(const MeshJob *jobs, double *tab) {
  const int m = blockIdx.y;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= kAreaTab) return;
  const MeshJob &J = jobs[m];
  DWork w;
  tab[(size_t)m * kAreaTab + i] =
      integrateArea(mesh_table_colat(J.pl, i), J.pl.lims[1], J.s, 0, w);
}

// per mesh: parallels, then the rows.  row_tmp[row] = (lower, upper, colatC,
// effective gravity); mesh_tmp[m] = (cellArea, eta)
__global__ void __launch_bounds__(128) mesh_rows_kernel(const MeshJob *jobs, const double *tab,
                                                        xgpu_mesh_batch_out o, double *row_tmp,
                                                        double *mesh_tmp) {
  extern __shared__ double sm[];
  double *colat = sm, *par = sm + kAreaTab;
  const int m = blockIdx.x;
  const MeshJob &J = jobs[m];
  const size_t S = J.pl.S;
  const double *T = tab + (size_t)m * kAreaTab;
  for (int i = threadIdx.x; i < kAreaTab; i += blockDim.x) colat[i] = mesh_table_colat(J.pl, i);
  __syncthreads();
  __shared__ double s_eta;
  if (threadIdx.x == 0) {
    double cellArea, eta;
    mesh_cell_area(J.pl, T[kAreaTab - 1], cellArea, eta);
    mesh_parallels(J.pl, colat, T, eta, par);
    s_eta = eta;
    mesh_tmp[2 * m] = cellArea;
    mesh_tmp[2 * m + 1] = eta;
  }
  __syncthreads();
  const double eta = s_eta;
  for (size_t i = threadIdx.x; i < S; i += blockDim.x) {
    double lower, upper;
    mesh_row_bounds(J.pl, par, i, lower, upper);
    DWork w;
    const RowOut r = mesh_row(J.s, lower, upper, eta, w);
    const int64_t row = J.row_off + (int64_t)i;
    row_tmp[4 * row] = lower;
    row_tmp[4 * row + 1] = upper;
    row_tmp[4 * row + 2] = r.colat;
    row_tmp[4 * row + 3] = r.effGrav;
    // packed row values, as the host packing forms them
    const double u = J.r_s / r.r;
    o.u[row] = u;
    o.r_s[row] = J.r_s;
    o.maxAlpha[row] = r.maxAlpha;
    o.radius[row] = r.r;
    o.cos_gamma[row] = r.cos_gamma;
    o.theta0[row] = J.pl.invert ? PI - r.colat : r.colat;
    double C = (1.0 / u - J.R_over_rs);
    C += log((1.0 / u - 1.0) / (J.R_over_rs - 1.0));
    C *= J.r_s / kC;
    o.lag_C[row] = C;
    o.lag_scale[row] = J.lag_scale;
    o.row_mesh[row] = m;
  }
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

template <typename F>
__device__ double cta_dyadic(const F &f, double lo, double hi, bool toward_lo, double er,
                             CutList &L) {
  const double Lw = hi - lo;
  double sum = 0.0;
  int seen = 0, quiet = 0;
  for (int k = 0; k < 2100; k++) {
    const double s1 = ldexp(Lw, -(k + 1)), s0 = ldexp(Lw, -k);
    const double p0 = toward_lo ? lo + s1 : hi - s0;
    const double p1 = toward_lo ? lo + s0 : hi - s1;
    if (!(p0 < p1) || (toward_lo ? p0 <= lo : p1 >= hi)) break;
    const double r = cta_qag21(f, p0, p1, 0.0, er, L);
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

template <typename F>
__device__ double cta_integrate(const F &f, double a, double b, double epsabs, double epsrel,
                                CutList &L) {
  double sign = 1.0;
  if (b < a) { const double t = a; a = b; b = t; sign = -1.0; }
  if (a == b) return 0.0;
  double er = (1.0e-13 < epsrel) ? 1.0e-13 : epsrel;
  if (epsabs <= 0.0 && er < 50.0 * 2.220446049250313e-16) er = 50.0 * 2.220446049250313e-16;
  double r = cta_qag21(f, a, b, epsabs, er, L);
  if (r == 0.0) {
    const double fa = f(a), fb = f(b);
    if (fa != 0.0 || fb != 0.0) {
      const double m = 0.5 * (a + b);
      const double rl = fa != 0.0 ? cta_dyadic(f, a, m, true, er, L)
                                  : cta_qag21(f, a, m, 0.0, er, L);
      const double rr = fb != 0.0 ? cta_dyadic(f, m, b, false, er, L)
                                  : cta_qag21(f, m, b, 0.0, er, L);
      r = rl + rr;
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
                                                         const double *row_tmp,
                                                         const double *mesh_tmp,
                                                         int64_t *queue, unsigned *n_queue) {
  const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= n_cells) return;
  const int m = mesh_of_cell(jobs, n_mesh, c);
  const MeshJob &J = jobs[m];
  const size_t S = J.pl.S;
  const int64_t k = c - J.cell_off;
  const size_t i = (size_t)(k / (int64_t)S), j = (size_t)(k - (int64_t)i * (int64_t)S);
  const int64_t row = J.row_off + (int64_t)i;
  // azimuth (shifted by the omitted region's azimuth, half a turn when
  // antiphased) and the atmosphere parameters of the cell
  double ph = mesh_phi(J.pl, j) - J.omit_azimuth;
  if (J.antiphased) ph = ph + PI;
  o.phi[c] = ph;
  o.params[2 * c] = J.logT;
  o.params[2 * c + 1] = row_tmp[4 * row + 3];
  const size_t j_max = J.pl.j_max;
  if (j < j_max) {
    double leftmost, rightmost;
    const int kind = mesh_cell_kind(J.pl, i, j, row_tmp[4 * row], row_tmp[4 * row + 1],
                                    row_tmp[4 * row + 2], leftmost, rightmost);
    if (kind == 2) queue[atomicAdd(n_queue, 1u)] = c;
    else put_area(J, o, c, i, j, kind == 1 ? mesh_tmp[2 * m] : 0.0);
  } else if (!J.pl.sym || j < S - j_max) {
    // columns no mirror reaches keep area 0
    o.cellArea[c] = 0.0;
    o.radiates[c] = 0;
  }
}

// one CTA per queued cell: the area quadrature of a cell cut by a boundary.
// A CTA starts with the cell of its own index (a small batch's cells spread
// over the SMs) and takes the next from a shared counter (n_queue[1]) when it
// finishes one, as the cells' costs differ by 5x or more (10-50 bisection
// steps); each cell's result is independent of which CTA integrates it.
constexpr int kCutCtasPerSm = 8;
__global__ void __launch_bounds__(kCutThreads, kCutCtasPerSm) mesh_boundary_kernel(
    const MeshJob *jobs, int n_mesh, xgpu_mesh_batch_out o, const double *row_tmp,
    const int64_t *queue, unsigned *n_queue) {
  __shared__ CutList L;
  __shared__ unsigned s_q;
  const unsigned n = n_queue[0];
  for (unsigned q = blockIdx.x; q < n; q = s_q) {
    const int64_t c = queue[q];
    const int m = mesh_of_cell(jobs, n_mesh, c);
    const MeshJob &J = jobs[m];
    const size_t S = J.pl.S;
    const int64_t k = c - J.cell_off;
    const size_t i = (size_t)(k / (int64_t)S), j = (size_t)(k - (int64_t)i * (int64_t)S);
    const int64_t row = J.row_off + (int64_t)i;
    const double lower = row_tmp[4 * row], upper = row_tmp[4 * row + 1];
    double pa, pb;
    mesh_cell_kind(J.pl, i, j, lower, upper, row_tmp[4 * row + 2], pa, pb);
    const Region g = mesh_region(J.pl);
    CutCell f;
    f.init(CellIntegrand{J.s, g, pa, pb}, lower, upper);
    double integral = cta_integrate(f, lower, upper, 0.0, 1.0e-8, L);
    if (are_equal(integral, 0.0)) {
      double tmin, tmax;
      if (cell_fallback_interval(lower, upper, pa, pb, g, tmin, tmax))
        integral = cta_integrate(f, tmin, tmax, 0.0, 1.0e-8, L);
    }
    __syncthreads();  // every thread has read the last s_q
    if (threadIdx.x == 0) {
      put_area(J, o, c, i, j, J.s.R_eq * J.s.R_eq * integral);
      s_q = gridDim.x + atomicAdd(&n_queue[1], 1u);
    }
    __syncthreads();
  }
}

}  // namespace
}  // namespace xg

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
  MeshJob *d_jobs = nullptr;
  double *tab = nullptr, *row_tmp = nullptr, *mesh_tmp = nullptr;
  int64_t *queue = nullptr;
  unsigned *n_queue = nullptr;
  if (cudaMallocAsync(&d_jobs, sizeof(MeshJob) * (size_t)n, st) != cudaSuccess) return -5;
  if (cudaMallocAsync(&tab, sizeof(double) * (size_t)n * kAreaTab, st) != cudaSuccess ||
      cudaMallocAsync(&row_tmp, sizeof(double) * 4 * (size_t)n_rows, st) != cudaSuccess ||
      cudaMallocAsync(&mesh_tmp, sizeof(double) * 2 * (size_t)n, st) != cudaSuccess ||
      cudaMallocAsync(&queue, sizeof(int64_t) * (size_t)n_cells, st) != cudaSuccess ||
      cudaMallocAsync(&n_queue, 2 * sizeof(unsigned), st) != cudaSuccess) {
    cudaFreeAsync(d_jobs, st);
    return -5;
  }
  // (a copy from pageable memory has been staged when cudaMemcpyAsync
  // returns, so the host jobs may go out of scope)
  cudaMemcpyAsync(d_jobs, jobs.data(), sizeof(MeshJob) * (size_t)n, cudaMemcpyHostToDevice, st);
  cudaMemsetAsync(n_queue, 0, 2 * sizeof(unsigned), st);  // queue length, next cell
  mesh_table_kernel<<<dim3((kAreaTab + 127) / 128, (unsigned)n), 128, 0, st>>>(d_jobs, tab);
  const size_t smem = sizeof(double) * (kAreaTab + S_max);
  mesh_rows_kernel<<<(unsigned)n, 128, smem, st>>>(d_jobs, tab, *out, row_tmp, mesh_tmp);
  mesh_cells_kernel<<<(unsigned)((n_cells + 127) / 128), 128, 0, st>>>(
      d_jobs, n, n_cells, *out, row_tmp, mesh_tmp, queue, n_queue);
  mesh_boundary_kernel<<<152 * kCutCtasPerSm, kCutThreads, 0, st>>>(d_jobs, n, *out, row_tmp,
                                                                     queue, n_queue);
  const cudaError_t e = cudaGetLastError();
  cudaFreeAsync(d_jobs, st);
  cudaFreeAsync(tab, st);
  cudaFreeAsync(row_tmp, st);
  cudaFreeAsync(mesh_tmp, st);
  cudaFreeAsync(queue, st);
  cudaFreeAsync(n_queue, st);
  return e == cudaSuccess ? 0 : -5;
}
