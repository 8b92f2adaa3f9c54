// likelihood.cu -- K6: expected counts per phase bin and the background-
// marginalised Poisson log-likelihood, replacing
//   xpsi/tools/compute_expected_counts.pyx:66-197 and
//   xpsi/likelihoods/default_background_marginalisation.pyx:38-734.
//
// One warp per (likelihood evaluation, channel).  Lanes integrate the
// Akima-periodic phase interpolant of each component over their phase bins
// and hold one phase bin each for the channel sums (Newton steps, Gaussian
// width, the normalisation A), which are reduced with xor-butterfly shuffles
// so every lane holds the same bits and control flow stays warp-uniform;
// the marginal integral is one 61-point Gauss-Kronrod panel on each side of
// the peak, two nodes to a lane, where those meet relative 1e-13 by their own
// error estimate, else a QUADPACK-style adaptive Gauss-Kronrod-21 quadrature run
// to it, whose 21 node evaluations per panel are spread over the lanes.  The
// reference's CQUAD call (:416-419) asks for relative 1e-8 on
// this smooth integrand, so both converge to the same integral.  The channel
// terms are summed per evaluation in channel order by a second kernel, which
// also applies the reference's early exits (slim cut :677-684, vanished
// integral :423-429).
#include <climits>

#include "common.cuh"
#include "kernels.h"
#include "log_table.h"

namespace xg {
namespace {

// Natural logarithm of a positive, normal double-float m with a table:
// m = 2^e f, f in [0.75, 1.5) (as df_log), then f = c (f / c) with c the
// nearest node 0.75 + i / 128 (|f / c - 1| <= 1 / 192) and
//   ln f = ln c + 2 atanh(s),  s = (f - c) / (f + c),  |s| <= 1 / 385,
// the series 2 s (1 + s^2 / 3 + s^4 / 5) truncated below 1e-17 relative
// (the s^4 / 5 term in float, its rounding ~1e-19); ln c from the table
// (gen_log_table.py, float pairs).  About half the work of df_log's
// 11-term series.  tab: the table in shared memory.
__device__ __forceinline__ DF df_log_t(DF m, const DF *tab) {
  const DF ln2{0.6931471824645996f, -1.9046542121259336e-09f};
  const DF third{0.3333333432674408f, -9.934107758624577e-09f};
  const int bits = __float_as_int(m.h);
  int e = ((bits >> 23) & 0xff) - 127;
  if ((bits & 0x7fffff) >= 0x400000) e += 1;
  const float sc = __int_as_float((127 - e) << 23);
  const DF f{__fmul_rn(m.h, sc), __fmul_rn(m.l, sc)};
  int i = __float2int_rn((f.h - 0.75f) * 128.0f);
  i = min(max(i, 0), XG_LOGT_N - 1);
  const float c = 0.75f + (float)i * 0.0078125f;
  const DF s = df_div(df_add(f, DF{-c, 0.0f}), df_add(f, DF{c, 0.0f}));
  const DF s2 = df_mul(s, s);
  const float s4_5 = __fmul_rn(__fmul_rn(s2.h, s2.h), 0.2f);
  const DF p = df_add(DF{1.0f, 0.0f}, df_add(df_mul(s2, third), DF{s4_5, 0.0f}));
  return df_add(df_fma(DF{(float)e, 0.0f}, ln2, tab[i]), df_mul(df_add(s, s), p));
}

__device__ __noinline__ double exp_large(double x) { return exp(x); }
// exp(x) of a double-float x, returned as a double: x = k ln 2 + r with
// |r| <= ln 2 / 2 (ln 2 in parts, gen_log_table.py: k times the first two
// exact for |k| < 2^11), exp(r) by its Taylor series through r^13 / 13! in
// double-float (truncation below 4e-18 relative), joined with 2^k by bits; 0 below
// the double range, the FP64 exp beyond ln 2^1000.
__device__ __forceinline__ double df_exp_d(DF x) {
  if (x.h != x.h) return (double)x.h;
  if (x.h < -760.0f) return 0.0;
  if (x.h > 690.0f) return exp_large((double)x.h + (double)x.l);
  const float kf = rintf(x.h * 1.44269504088896341f);
  const int k = (int)kf;
  DF r = df_add(x, DF{-kf * XG_LN2_1, 0.0f});
  r = df_add(r, DF{-kf * XG_LN2_2, 0.0f});
  r = df_fma(DF{-kf, 0.0f}, DF{XG_LN2_3, XG_LN2_4}, r);
  DF p{XG_EXPT[XG_EXPT_N - 1][0], XG_EXPT[XG_EXPT_N - 1][1]};
#pragma unroll
  for (int n = XG_EXPT_N - 2; n >= 0; n--) p = df_fma(p, r, DF{XG_EXPT[n][0], XG_EXPT[n][1]});
  return df_join_bits(p, k);
}

constexpr int kWarps = 4;
constexpr int kMaxB = 64;      // phase bins per channel held in shared memory
constexpr int kQagLimit = 256; // interval list of the marginal quadrature
constexpr int kMaxPiecesPerLane = 8;  // pulse knots per lane in the warp's Akima build

struct WarpSmem {
  double star[kMaxB];
  double data[kMaxB];
  DF q[kMaxB];        // SCALE / c_j(Bi): the relative form of the integrand
  float dataf[kMaxB];  // counts (exact in float below 2^24)
  double al[kQagLimit], bl[kQagLimit], rl[kQagLimit], el[kQagLimit];
};

struct Marg {
  int n;
  double SCALE, T, A;
  const double *data, *star;
  // relative form (set when every c_j(Bi) > 0, or 0 without counts: A = x(Bi))
  int rel;
  double Bi;
  const DF *q;
  const float *dataf;
  const DF *logt;  // df_log_t's table (shared memory)
  DF nS;           // n SCALE as a pair (relative form)
};

// :84-138, as the reference writes it
__device__ __noinline__ double marginal_integrand_direct(const Marg &m, double B) {
  double x = 0.0;
  for (int j = 0; j < m.n; j++) {
    double c = m.SCALE * (m.star[j] + B);
    if (c > 0.0) x += m.data[j] * log(c) - c;
    else if (are_equal(c, 0.0) && are_equal(m.data[j], 0.0)) {}
    else return 0.0;
  }
  return exp(x - m.A);
}

// The same integrand in relative form.  With c_j(B) = SCALE (s_j + B) and
// A = x(Bi),
//   x(B) - A = sum_j d_j log(c_j(B) / c_j(Bi)) - n SCALE (B - Bi),
// whose terms are O(d_j |B - Bi| / c_j) instead of O(d_j log c_j): no
// cancellation against A.  The ratio 1 + (B - Bi) SCALE / c_j(Bi), its
// logarithm, the sum and its exponential are taken in double-float
// arithmetic (FP32 pipes); a node where
// some ratio is not positive (c_j(B) <= 0) takes the direct form, which
// holds the reference's tests for that case.
__device__ __forceinline__ double marginal_integrand(const Marg &m, double B) {
  if (!m.rel) {
    const Marg mc = m;
    return marginal_integrand_direct(mc, B);
  }
  const DF dB = df_split_bits(B - m.Bi, 0);
  const DF one{1.0f, 0.0f};
  DF acc{0.0f, 0.0f};
  for (int j = 0; j < m.n; j++) {
    const DF r = df_fma(dB, m.q[j], one);
    if (!(r.h > 0.0f)) {
      const Marg mc = m;
      return marginal_integrand_direct(mc, B);
    }
    if (m.dataf[j] != 0.0f) acc = df_fma(DF{m.dataf[j], 0.0f}, df_log_t(r, m.logt), acc);
  }
  return df_exp_d(df_sub(acc, df_mul(m.nS, dB)));
}

// sum over the warp; the butterfly adds the same pairs in every lane, so all
// lanes return identical bits
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
// warp_sum of two and of four values, each half (quarter) of the warp carrying
// one of them once the others' share is handed over: five and six additions
// in place of ten and twenty, the same bits (the FP64 pipe takes 64 cycles
// for one, a shuffle two)
__device__ __forceinline__ double hand_over(double low, double high, int lane, int o) {
  const bool up = lane & o;
  return (up ? high : low) + __shfl_xor_sync(0xffffffffu, up ? low : high, o);
}
__device__ __forceinline__ void warp_sum2(double &a, double &b, int lane) {
  double v = hand_over(a, b, lane, 16);
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  a = __shfl_sync(0xffffffffu, v, 0);
  b = __shfl_sync(0xffffffffu, v, 16);
}
__device__ __forceinline__ void warp_sum4(double (&a)[4], int lane) {
  const double u = hand_over(a[0], a[1], lane, 16), w = hand_over(a[2], a[3], lane, 16);
  double v = hand_over(u, w, lane, 8);
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
#pragma unroll
  for (int i = 0; i < 4; i++)
    a[i] = __shfl_sync(0xffffffffu, v, (i & 1 ? 16 : 0) + (i & 2 ? 8 : 0));
}

// The Akima-periodic pieces of one component's pulse through (x[i], y[i]),
// i < n, built once per warp in double-float arithmetic: the pulse scaled
// by 2^-e (e the binary exponent of its largest value, exact) into yd[],
// the chord slopes into ch[], each interval's (k1, k2, k3) into k1[], k2[],
// k3[] (akima_piece_df, with the grid's 1/h and 1/h^2 from ih[], ih2[]), then
// yd[] over ch[] -- the
// pieces akima_periodic_integral forms again for every bin that reaches
// them, here once, on the FP32 pipes (~2^-48 relative).  Returns e; ends
// with __syncwarp.
__device__ __forceinline__ int akima_pieces_warp_df(const double *x, const double *y, int n,
                                                    const DF *ih, const DF *ih2, DF *ch, DF *k1,
                                                    DF *k2, DF *k3, int lane) {
  int e = INT_MIN;
  bool inf = false;
  for (int q = lane; q < n; q += 32) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(y[q]);
    const int f = (int)((b >> 52) & 0x7ff);
    if (f == 0x7ff) inf = true;
    else if (f != 0) e = max(e, f - 1022);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    e = max(e, __shfl_xor_sync(0xffffffffu, e, o));
    inf = __shfl_xor_sync(0xffffffffu, (int)inf, o) != 0 || inf;
  }
  if (inf || e == INT_MIN) e = 0;
  // yd (in k3[] for now) and the chords
  for (int q = lane; q < n; q += 32) k3[q] = df_split_bits(y[q], -e);
  __syncwarp();
  for (int q = lane; q < n - 1; q += 32)
    ch[q] = df_mul(df_sub(k3[q + 1], k3[q]), ih[q]);
  __syncwarp();
  DF yq[kMaxPiecesPerLane];
  int c = 0;
  for (int q = lane; q < n; q += 32) yq[c++] = k3[q];
  __syncwarp();
  for (int i = lane; i < n - 1; i += 32) {
    DF a1, a2, a3;
    akima_piece_df(ch[periodic_chord(i - 2, n)], ch[periodic_chord(i - 1, n)], ch[i],
                   ch[periodic_chord(i + 1, n)], ch[periodic_chord(i + 2, n)], ih[i], ih2[i],
                   a1, a2, a3);
    k1[i] = a1;
    k2[i] = a2;
    k3[i] = a3;
  }
  __syncwarp();
  c = 0;
  for (int q = lane; q < n; q += 32) ch[q] = yq[c++];
  __syncwarp();
  return e;
}
// akima_periodic_integral over [lo, hi] from the pieces of
// akima_pieces_warp_df (yd in yd[]), in units of 2^e
// (hd: the intervals' lengths; only the two ends' offsets are formed in FP64,
// and the lower end's value in the first interval alone, which the lanes take
// together)
__device__ __forceinline__ DF akima_integral_df(const double *x, const DF *hd, const DF *yd,
                                                int n, const DF *k1, const DF *k2, const DF *k3,
                                                double lo, double hi) {
  const DF third{0.3333333432674408f, -9.934107758624577e-09f};
  const int ia = locate_bits(x, n, lo), ib = locate_bits(x, n, hi);
  const DF u = df_split_bits(lo - x[ia], 0), w = df_split_bits(hi - x[ib], 0);
  DF acc{0.0f, 0.0f};
#pragma unroll 1
  for (int i = ia; i <= ib; i++) {
    // F(t) = t (y + t (k1 / 2 + t (k2 / 3 + t k3 / 4)))
    const DF c1{0.5f * k1[i].h, 0.5f * k1[i].l}, c3{0.25f * k3[i].h, 0.25f * k3[i].l};
    const DF c2 = df_mul(k2[i], third), y = yd[i];
    auto F = [&](DF t) { return df_mul(t, df_fma(t, df_fma(t, df_fma(t, c3, c2), c1), y)); };
    DF v = F(i == ib ? w : hd[i]);
    if (i == ia) v = df_sub(v, F(u));
    acc = df_add(acc, v);
  }
  return acc;
}

// :140-173: y and x of the Newton step -y / x at B, whose Gaussian width is
// sqrt(2 / x); lane-parallel over the phase bins.  pow(s, 2.0) of the
// reference is s * s, as its C compiler emits it.
__device__ __forceinline__ void newton_sums(const Marg &m, double B, int lane, double &y,
                                            double &x) {
  x = y = 0.0;
  for (int j = lane; j < m.n; j += 32) {
    // d / s and d / s^2 from one reciprocal (an ulp from the two divisions)
    const double is = 1.0 / (m.star[j] + B);
    const double t = m.data[j] * is;
    y += t;
    x += t * is;
  }
  warp_sum2(y, x, lane);
  y = 2.0 * m.T - 2.0 * y;
  x *= 2.0;
}
// |step| > epsilon width (:336), as y^2 > 2 epsilon^2 x where that says the
// same: no root and no division
__device__ __forceinline__ bool newton_far(double y, double x, double epsilon) {
  if (epsilon > 0.0 && x > 0.0 && x < 1.0e300) return y * y > 2.0 * epsilon * epsilon * x;
  return fabs(y / x) > epsilon * sqrt(2.0 / x);
}

// The 21-point Gauss-Kronrod panels of the marginal quadrature, evaluated by
// the warp: lane l holds node l and node l + 32 of up to two panels (nodes
// 0..20 the first, 21..41 the second; within a panel, nodes 0..9 at
// c - h X[j], 10 at c, 11..20 at c + h X[j]).  The weighted sums of the
// rule are lane-parallel xor-butterfly reductions (identical bits in every
// lane); the error estimate follows QUADPACK (the (200 e / rc)^1.5 scaling,
// the 50 eps round-off floor).
struct Panel {
  double res, err, rabs, rasc;
};

__device__ __forceinline__ int gk21_slot(int n) { return n < 10 ? n : (n == 10 ? 10 : n - 11); }

__device__ __forceinline__ double gk21_node(double a, double b, int n) {
  const int NH = XG_K21_HALF - 1;
  double c = 0.5 * (a + b), h = 0.5 * (b - a);
  if (n < NH) return c - h * XG_K21_X[n];
  if (n == NH) return c;
  return c + h * XG_K21_X[n - NH - 1];
}

__device__ __forceinline__ Panel gk21_finish(double rk, double rg, double ra, double rc, double a,
                                             double b) {
  const double h = 0.5 * (b - a), ah = fabs(h);
  Panel P;
  P.res = rk * h;
  ra *= ah;
  rc *= ah;
  double e = fabs((rk - rg) * h);
  if (rc != 0.0 && e != 0.0) {
    const double x = 200.0 * e / rc, sc = x * sqrt(x);  // x^1.5
    e = sc < 1.0 ? rc * sc : rc;
  }
  const double eps = 2.220446049250313e-16, dmin = 2.2250738585072014e-308;
  if (ra > dmin / (50.0 * eps)) {
    const double fl = 50.0 * eps * ra;
    if (fl > e) e = fl;
  }
  P.err = e;
  P.rabs = ra;
  P.rasc = rc;
  return P;
}

// one panel [a1, b1] (two: also [a2, b2]); returns the panels' sums
__device__ void warp_panels(const Marg &m, int lane, double a1, double b1, double a2, double b2,
                            bool two, Panel &P1, Panel &P2) {
  const int total = two ? 42 : 21;
  double f0 = 0.0, f1 = 0.0;
  if (lane < total) f0 = marginal_integrand(m, lane < 21 ? gk21_node(a1, b1, lane)
                                                         : gk21_node(a2, b2, lane - 21));
  if (lane + 32 < total) f1 = marginal_integrand(m, gk21_node(a2, b2, lane + 32 - 21));
  double rk1 = 0.0, rg1 = 0.0, ra1 = 0.0, rk2 = 0.0, rg2 = 0.0, ra2 = 0.0;
  if (lane < total) {
    if (lane < 21) {
      const int s = gk21_slot(lane);
      rk1 = XG_K21_WK[s] * f0; rg1 = XG_K21_WG[s] * f0; ra1 = XG_K21_WK[s] * fabs(f0);
    } else {
      const int s = gk21_slot(lane - 21);
      rk2 = XG_K21_WK[s] * f0; rg2 = XG_K21_WG[s] * f0; ra2 = XG_K21_WK[s] * fabs(f0);
    }
  }
  if (lane + 32 < total) {
    const int s = gk21_slot(lane + 32 - 21);
    rk2 += XG_K21_WK[s] * f1; rg2 += XG_K21_WG[s] * f1; ra2 += XG_K21_WK[s] * fabs(f1);
  }
  rk1 = warp_sum(rk1); rg1 = warp_sum(rg1); ra1 = warp_sum(ra1);
  if (two) { rk2 = warp_sum(rk2); rg2 = warp_sum(rg2); ra2 = warp_sum(ra2); }
  const double mean1 = 0.5 * rk1, mean2 = 0.5 * rk2;
  double rc1 = 0.0, rc2 = 0.0;
  if (lane < total) {
    if (lane < 21) rc1 = XG_K21_WK[gk21_slot(lane)] * fabs(f0 - mean1);
    else rc2 = XG_K21_WK[gk21_slot(lane - 21)] * fabs(f0 - mean2);
  }
  if (lane + 32 < total) rc2 += XG_K21_WK[gk21_slot(lane + 32 - 21)] * fabs(f1 - mean2);
  rc1 = warp_sum(rc1);
  P1 = gk21_finish(rk1, rg1, ra1, rc1, a1, b1);
  if (two) {
    rc2 = warp_sum(rc2);
    P2 = gk21_finish(rk2, rg2, ra2, rc2, a2, b2);
  }
}

// index of the first largest error among el[0..size) (QUADPACK's choice of
// the interval to bisect), by a warp arg-max with ties to the lower index;
// identical in every lane (a NaN error counts as -inf)
__device__ __forceinline__ int warp_worst(const double *el, int size, int lane) {
  double v = -INFINITY;
  int k = 0x7fffffff;
  for (int i = lane; i < size; i += 32) {
    const double e = isnan(el[i]) ? -INFINITY : el[i];
    if (k == 0x7fffffff || e > v) {
      v = e;
      k = i;
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const double v2 = __shfl_xor_sync(0xffffffffu, v, o);
    const int k2 = __shfl_xor_sync(0xffffffffu, k, o);
    if (v2 > v || (v2 == v && k2 < k)) {
      v = v2;
      k = k2;
    }
  }
  return k;
}

// adaptive GK21 (same scheme as the rays' QAG), warp-cooperative; a < b
__device__ __noinline__ double warp_qag21_core(const Marg &m, WarpSmem &w, int lane, double a, double b,
                                  double epsabs, double er) {
  const double eps = 2.220446049250313e-16, dmin = 2.2250738585072014e-308;
  Panel P0, Pu;
  warp_panels(m, lane, a, b, 0.0, 0.0, false, P0, Pu);
  const double r0 = P0.res, e0 = P0.err, ra0 = P0.rabs, rc0 = P0.rasc;
  double tol = fmax(epsabs, er * fabs(r0));
  double rfloor = 50.0 * eps * ra0;
  if ((e0 <= rfloor && e0 > tol) || (e0 <= tol && e0 != rc0) || e0 == 0.0) return r0;
  if (lane == 0) { w.al[0] = a; w.bl[0] = b; w.rl[0] = r0; w.el[0] = e0; }
  __syncwarp();
  int size = 1, iter = 1, k = 0, rnd1 = 0, rnd2 = 0, fail = 0;
  double area = r0, errsum = e0;
  do {
    double ai = w.al[k], bi = w.bl[k], ri = w.rl[k], ei = w.el[k];
    double a1 = ai, b1 = 0.5 * (ai + bi), a2 = b1, b2 = bi;
    Panel P1, P2;
    warp_panels(m, lane, a1, b1, a2, b2, true, P1, P2);
    const double r1 = P1.res, e1 = P1.err, rc1 = P1.rasc;
    const double r2 = P2.res, e2 = P2.err, rc2 = P2.rasc;
    double r12 = r1 + r2, e12 = e1 + e2;
    errsum += e12 - ei;
    area += r12 - ri;
    if (rc1 != e1 && rc2 != e2) {
      double delta = ri - r12;
      if (fabs(delta) <= 1.0e-5 * fabs(r12) && e12 >= 0.99 * ei) rnd1++;
      if (iter >= 10 && e12 > ei) rnd2++;
    }
    tol = fmax(epsabs, er * fabs(area));
    if (errsum > tol) {
      if (rnd1 >= 6 || rnd2 >= 20) fail = 2;
      double edge = (1.0 + 100.0 * eps) * (fabs(a2) + 1000.0 * dmin);
      if (fabs(a1) <= edge && fabs(b2) <= edge) fail = 3;
    }
    int nw = size++;
    __syncwarp();
    if (lane == 0) {
      if (e2 > e1) {
        w.al[k] = a2; w.bl[k] = b2; w.rl[k] = r2; w.el[k] = e2;
        w.al[nw] = a1; w.bl[nw] = b1; w.rl[nw] = r1; w.el[nw] = e1;
      } else {
        w.al[k] = a1; w.bl[k] = b1; w.rl[k] = r1; w.el[k] = e1;
        w.al[nw] = a2; w.bl[nw] = b2; w.rl[nw] = r2; w.el[nw] = e2;
      }
    }
    __syncwarp();
    k = warp_worst(w.el, size, lane);
    iter++;
  } while (iter < kQagLimit && !fail && errsum > tol);
  double sum = 0.0;
  for (int i = lane; i < size; i += 32) sum += w.rl[i];
  sum = warp_sum(sum);
  __syncwarp();
  return sum;
}

// dyadic pieces toward an endpoint holding all the mass (see warp_marginal)
__device__ double warp_dyadic(const Marg &m, WarpSmem &w, int lane, double lo, double hi,
                              bool toward_lo, double er) {
  const double L = hi - lo;
  double sum = 0.0;
  int seen = 0, quiet_after = 0;
  for (int k = 0; k < 2100; k++) {
    double s1 = ldexp(L, -(k + 1)), s0 = ldexp(L, -k);
    double p0 = toward_lo ? lo + s1 : hi - s0;
    double p1 = toward_lo ? lo + s0 : hi - s1;
    if (!(p0 < p1) || (toward_lo ? p0 <= lo : p1 >= hi)) break;
    double r = warp_qag21_core(m, w, lane, p0, p1, 0.0, er);
    sum += r;
    if (r != 0.0) seen = 1;
    if (seen && fabs(r) <= 1.0e-17 * fabs(sum)) {
      if (++quiet_after >= 4) break;
    } else {
      quiet_after = 0;
    }
  }
  return sum;
}

// The marginal integral over [a, b] from one 61-point Gauss-Kronrod panel on
// each side of the integrand's peak (one in all where the peak lies on an
// end), two nodes to a lane (61 of its 64 slots): a window of ten standard
// deviations either way is smooth enough that they meet the adaptive rule's
// tolerance, at two node evaluations per lane and panel against two for each
// of the eight or so bisections, whose sums and error estimates (FP64, one per
// warp) were the kernel's larger half.  The integrand is an exponential, so
// its own sum is the rule's |f| sum; the error estimate is QUADPACK's, its
// ratio in float.  Returns false where they do not meet it.  One copy of the
// integrand's code serves the four nodes.
__device__ __forceinline__ bool warp_peak61(const Marg &m, int lane, double a, double b,
                                            double er, double &out) {
  const int NH = XG_K61_HALF - 1;  // 30
  const bool inside = a < m.Bi && m.Bi < b;
  const double mid = inside ? m.Bi : b;
  double c[2], h[2];
  c[0] = 0.5 * (a + mid), h[0] = 0.5 * (mid - a);
  c[1] = 0.5 * (mid + b), h[1] = 0.5 * (b - mid);
  // the four values, shifted through registers: panel 0 in f3, f2
  double f3 = 0.0, f2 = 0.0, f1 = 0.0, f0 = 0.0;
#pragma unroll 1
  for (int z = 0; z < 4; z++) {
    const int n = lane + 32 * (z & 1);
    double v = 0.0;
    if (n <= 2 * NH && (z < 2 || inside)) {
      const int s = n <= NH ? n : n - NH - 1;
      const double x = n < NH ? -XG_K61_X[s] : (n == NH ? 0.0 : XG_K61_X[s]);
      v = marginal_integrand(m, fma(z < 2 ? h[0] : h[1], x, z < 2 ? c[0] : c[1]));
    }
    f3 = f2; f2 = f1; f1 = f0; f0 = v;
  }
  const int n1 = lane + 32;
  const int s0 = lane <= NH ? lane : lane - NH - 1;
  const bool two = n1 <= 2 * NH;
  const double k0 = XG_K61_WK[s0], g0 = XG_K61_WG[s0];
  const double k1 = two ? XG_K61_WK[n1 - NH - 1] : 0.0, g1 = two ? XG_K61_WG[n1 - NH - 1] : 0.0;
  double sum[4] = {fma(k1, f2, k0 * f3), fma(g1, f2, g0 * f3), fma(k1, f0, k0 * f1),
                   fma(g1, f0, g0 * f1)};
  warp_sum4(sum, lane);
  const double ma = 0.5 * sum[0], mb = 0.5 * sum[2];
  double rc[2] = {fma(k1, fabs(f2 - ma), k0 * fabs(f3 - ma)),
                  fma(k1, fabs(f0 - mb), k0 * fabs(f1 - mb))};
  warp_sum2(rc[0], rc[1], lane);
  double r = 0.0, e = 0.0;
#pragma unroll
  for (int p = 0; p < 2; p++) {
    if (p == 1 && !inside) break;
    const double res = sum[2 * p] * h[p];
    // err = rasc min(1, (200 |K - G| / rasc)^1.5): the half-width cancels from
    // the ratio
    const float dk = fabsf((float)(sum[2 * p] - sum[2 * p + 1])), rcf = (float)rc[p];
    float q = dk;
    if (rcf != 0.0f && dk != 0.0f) {
      const float x = 200.0f * dk / rcf, sc = x * sqrtf(x);
      q = sc < 1.0f ? rcf * sc : rcf;
    }
    r += res;
    e += fmax((double)q * h[p], 50.0 * 2.220446049250313e-16 * res);
  }
  out = r;
  return r > 0.0 && e <= er * r;
}

// adaptive GK21 over [a, b]; when every interior node sees zero but an endpoint
// does not (a channel without counts has a window ~1e91 wide whose integrand
// decays on the scale 1 / exposure), the window is cut into dyadic pieces
// toward that endpoint, as a Clenshaw-Curtis rule with endpoint nodes would
// resolve it.
__device__ __noinline__ double warp_adaptive(const Marg &m, WarpSmem &w, int lane, double a,
                                            double b, double epsabs, double er) {
  double r = warp_qag21_core(m, w, lane, a, b, epsabs, er);
  if (r == 0.0) {
    double fa = marginal_integrand(m, a);
    double fb = marginal_integrand(m, b);
    if (fa != 0.0 || fb != 0.0) {
      double mid = 0.5 * (a + b);
      double rl = (fa != 0.0) ? warp_dyadic(m, w, lane, a, mid, true, er)
                              : warp_qag21_core(m, w, lane, a, mid, 0.0, er);
      double rr = (fb != 0.0) ? warp_dyadic(m, w, lane, mid, b, false, er)
                              : warp_qag21_core(m, w, lane, mid, b, 0.0, er);
      r = rl + rr;
    }
  }
  return r;
}
// The upper end of the window without the tail where the relative form's
// integrand underflows to zero: its logarithm is at most
//   D log(1 + t q) - n SCALE t,  t = B - Bi, D the counts, q the largest
// SCALE / c_j(Bi) of a bin with counts,
// which is concave in t, so it stays below where it has fallen to -760.  The
// windows this is for are ten times 1e90 wide (no width could be formed, the
// star vanishing in a bin): the dyadic cut then took some 400 pieces, a
// channel of 384,000 23 of the kernel's 34 ms.
__device__ __noinline__ double warp_tail(const DF *q, const float *dataf, int n, double nS,
                                         double Bi, double counts, double b, int lane) {
  float most = 0.0f;
  for (int j = lane; j < n; j += 32)
    if (dataf[j] != 0.0f) most = fmaxf(most, q[j].h);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) most = fmaxf(most, __shfl_xor_sync(0xffffffffu, most, o));
  const double qm = 1.000001 * (double)most;
  double t = 760.0 / nS;
  for (int k = 0; k < 64 && t < b - Bi; k++, t *= 2.0)
    if (counts * log1p(t * qm) - nS * t < -760.0) return Bi + t;
  return b;
}

// the marginal integral over [a, b] at relative min(epsrel, 1e-13)
__device__ __forceinline__ double warp_marginal(const Marg &m, WarpSmem &w, int lane, double a, double b,
                                double epsabs, double epsrel) {
  const double eps = 2.220446049250313e-16;
  double sign = 1.0;
  if (b < a) { double t = a; a = b; b = t; sign = -1.0; }
  if (a == b) return 0.0;
  double er = epsrel < 1.0e-13 ? epsrel : 1.0e-13;
  if (epsabs <= 0.0 && er < 50.0 * eps) er = 50.0 * eps;
  double peak;
  if (m.rel && warp_peak61(m, lane, a, b, er, peak)) return sign * peak;
  const Marg mc = m;  // (what the calls below see stays out of the hot path's registers)
  return sign * warp_adaptive(mc, w, lane, a, b, epsabs, er);
}

// one channel of one evaluation, by a warp
__device__ __forceinline__ void like_channel(const LikeArgs &a, WarpSmem &w, const DF *s_logt,
                                             const DF *s_h, const DF *s_ih, const DF *s_ih2,
                                             int lane, int v, int ch) {
  __syncwarp();  // the last channel's readers of w are done
  const int B = a.B, N_P = a.N_P;
  const double n = (double)B;
  const double SCALE = a.exposure / n;
  const double T = a.exposure;
  // expected star count rate per phase bin (compute_expected_counts.pyx:66-197).
  // Each component's Akima pieces are built once by the warp (in the
  // quadrature's interval lists, free until the marginal integral) and
  // integrated over every bin; pulses longer than those lists take the
  // per-bin form.
  const bool warp_pieces = N_P > 1 && N_P <= kQagLimit && N_P <= 32 * kMaxPiecesPerLane;
  for (int j = lane; j < B; j += 32) w.star[j] = 0.0;
  if (warp_pieces) {
    DF *yd = reinterpret_cast<DF *>(w.el), *k1 = reinterpret_cast<DF *>(w.al);
    DF *k2 = reinterpret_cast<DF *>(w.bl), *k3 = reinterpret_cast<DF *>(w.rl);
    const double *xs = a.comp_phases;
    const long long x_lo = ordered(xs[0]), x_hi = ordered(xs[N_P - 1]);
    for (int h = 0; h < a.H; h++) {
      const double *pulse = a.signals + (((size_t)v * a.H + h) * a.K + ch) * N_P;
      const double sh = a.shifts[(size_t)v * a.H + h];
      const bool neg = a.allow_negative[h] == 1;
      const int ex = akima_pieces_warp_df(xs, pulse, N_P, s_ih, s_ih2, yd, k1, k2, k3, lane);
      for (int j = lane; j < B; j += 32) {
        double st = w.star[j];
        double pa = a.phase_edges[j] + sh, pb = a.phase_edges[j + 1] + sh;
        if (are_equal(pb - pa, 1.0)) { pa = 0.0; pb = 1.0; }
        else { pa -= floor(pa); pb -= floor(pb); }
        // the reference's argument checks (akima_periodic_integral)
        // (comparisons by bits; a NaN gives a NaN as before)
        auto piece = [&](double lo, double hi) -> double {
          const long long lb = ordered(lo), hb = ordered(hi);
          if (lb > hb || lb < x_lo || hb > x_hi) return nan("");
          if (lb == hb) return 0.0;
          return df_join_bits(akima_integral_df(xs, s_h, yd, N_P, k1, k2, k3, lo, hi), ex);
        };
        const bool whole = ordered(pa) < ordered(pb);  // else the bin wraps: two parts
#pragma unroll 1
        for (int part = 0; part < (whole ? 1 : 2); part++) {
          const double val = piece(part ? 0.0 : pa, whole || part ? pb : 1.0);
          if (val > 0.0 || neg) st += val;
        }
        w.star[j] = st;
      }
      __syncwarp();
    }
  }
  for (int j = lane; j < B; j += 32) {
    double st = w.star[j];
    for (int h = 0; h < a.H && !warp_pieces; h++) {
      const double *pulse = a.signals + (((size_t)v * a.H + h) * a.K + ch) * N_P;
      const double sh = a.shifts[(size_t)v * a.H + h];
      const bool neg = a.allow_negative[h] == 1;
      if (N_P > 1) {
        double pa = a.phase_edges[j] + sh, pb = a.phase_edges[j + 1] + sh;
        if (are_equal(pb - pa, 1.0)) { pa = 0.0; pb = 1.0; }
        else { pa -= floor(pa); pb -= floor(pb); }
        double val;
        if (pa < pb) {
          val = akima_periodic_integral(a.comp_phases, pulse, N_P, pa, pb);
          if (val > 0.0 || neg) st += val;
        } else {
          val = akima_periodic_integral(a.comp_phases, pulse, N_P, pa, 1.0);
          if (val > 0.0 || neg) st += val;
          val = akima_periodic_integral(a.comp_phases, pulse, N_P, 0.0, pb);
          if (val > 0.0 || neg) st += val;
        }
      } else if (j == 0) {
        st = pulse[0];
      }
    }
    if (st < 0.0) st = 0.0;
    if (a.background) st += a.background[(size_t)ch * B + j];
    st *= n;
    w.star[j] = st;
    w.data[j] = a.counts[(size_t)ch * B + j];
  }
  __syncwarp();
  double av_STAR = 0.0, av_DATA = 0.0;
  for (int j = lane; j < B; j += 32) {
    av_STAR += w.star[j];
    av_DATA += w.data[j];
  }
  warp_sum2(av_STAR, av_DATA, lane);
  const double dsum = av_DATA;
  const size_t o = (size_t)v * a.K + ch;
  int flag = 0;
  double term = 0.0, Bout = 0.0;
  if (a.slim >= 0.0) {
    double limit = av_STAR * SCALE - a.slim * sqrt(av_STAR * SCALE) - av_DATA;
    if (limit > 0.0) flag = 1;
  }
  const double *support = a.support + 2 * (size_t)ch;
  Marg m{B, SCALE, T, 0.0, w.data, w.star, 0, 0.0, w.q, w.dataf, s_logt};
  double Bfinal = 0.0;
  if (!flag) {
    av_STAR /= n;
    av_DATA /= T;
    double Bv;
    if (are_equal(av_DATA, 0.0) && are_equal(av_STAR, 0.0)) {
      double lower = 0.0;
      if (lower < support[0]) lower = support[0];
      double upper = 10.0 / T;
      if (upper > support[1] && support[1] > 0.0) upper = support[1];
      Bv = 0.0;
      term = log((exp(-1.0 * lower * T) - exp(-1.0 * upper * T)) / T);
    } else {
      double B_min = 0.0;
      Bv = av_DATA - av_STAR;
      if (Bv <= B_min) {
        // where some bin's star rate is zero (within 1e-12), the smallest
        // positive count (by bits, a lane per bin)
        bool dark = false;
        long long least = LLONG_MAX;
        for (int j = lane; j < B; j += 32) {
          const long long sb = __double_as_longlong(w.star[j]) & LLONG_MAX;
          const long long db = __double_as_longlong(w.data[j]);
          dark |= sb < __double_as_longlong(1.0e-12);
          if (db > 0 && db <= __double_as_longlong(INFINITY)) least = min(least, db);
        }
        Bv = B_min;
        if (__any_sync(0xffffffffu, dark)) {
#pragma unroll
          for (int o = 16; o > 0; o >>= 1)
            least = min(least, __shfl_xor_sync(0xffffffffu, least, o));
          if (least != LLONG_MAX) {
            Bv = 0.01 * __longlong_as_double(least) / SCALE;
            B_min = 0.1 * Bv;
          }
        }
      }
      int counter = 0;
      // the reference's Newton loop (:336-352) has no step limit; 10000 steps
      // bound it here (convergence takes a handful)
#pragma unroll 1
      for (int steps = 0;; steps++) {
        double y, x;
        newton_sums(m, Bv, lane, y, x);
        if (counter >= 2 || steps >= 10000 || !newton_far(y, x, a.epsilon)) break;
        Bv += -1.0 * y / x;
        if (Bv < B_min) {
          if (B_min > 0.0) counter += 1;
          else counter = 2;
          Bv = B_min;
        }
      }
      double std_est = 0.0;
      for (int j = lane; j < B; j += 32) {
        const double sb = w.star[j] + Bv;
        std_est += w.data[j] / (sb * sb);
      }
      std_est = warp_sum(std_est);
      if (std_est > 0.0) std_est = sqrt(1.0 / std_est);
      else std_est = 1e90;
      double lower = Bv - a.sigmas * std_est, upper = Bv + a.sigmas * std_est;
      if (lower < B_min) lower = B_min;
      double Bi = Bv;
      if (lower < support[0]) {
        lower = support[0];
        if (upper < support[0] && support[1] > 0.0) { upper = support[1]; Bi = support[0]; }
        else if (upper < support[0]) { upper = support[0] + a.sigmas * std_est; Bi = support[0]; }
      }
      if (upper > support[1] && support[1] > 0.0) {
        upper = support[1];
        if (lower > support[1]) { lower = support[0]; Bi = support[1]; }
      }
      if (Bi < lower) Bi = lower;
      else if (Bi > upper) Bi = upper;
      double A = 0.0;
      for (int j = lane; j < B; j += 32) {
        double c = SCALE * (w.star[j] + Bi);
        if (c > 0.0) A += w.data[j] * log(c) - c;
        else if (are_equal(c, 0.0) && are_equal(w.data[j], 0.0)) {}
        else A += a.llzero;
      }
      A = warp_sum(A);
      m.A = A;
      // relative form of the integrand when every c_j(Bi) > 0, or 0 in a bin
      // without counts (its ratio is not asked for,
      // and no B of the window lies below)
      const double nS = (double)m.n * SCALE;
      bool pos = nS > 1.0e-10;
      for (int j = lane; j < B; j += 32) {
        const double c = SCALE * (w.star[j] + Bi);
        pos = pos && (c > 0.0 || (c == 0.0 && w.data[j] == 0.0 && lower >= Bi));
        w.q[j] = c > 0.0 ? df_split(SCALE / c) : DF{0.0f, 0.0f};
        w.dataf[j] = (float)w.data[j];
      }
      __syncwarp();
      if (__all_sync(0xffffffffu, pos)) {
        m.rel = 1;
        m.Bi = Bi;
        m.nS = df_split(nS);
      }
      double result;
      if (dsum == 0.0) {
        // no counts in the channel: every term is -c_j, so the integrand is
        // exp(-T (B - Bi)) exactly and its integral over the window is closed
        // form (the reference's quadrature converges to this value)
        result = exp(-T * (lower - Bi)) * (-expm1(-T * (upper - lower))) / T;
      } else {
        // (a window of ten standard deviations reaches 4000 from 160,000
        // counts on)
        if (m.rel && nS * (upper - Bi) > 4000.0)
          upper = warp_tail(w.q, w.dataf, B, nS, Bi, dsum, upper, lane);
        result = warp_marginal(m, w, lane, lower, upper, a.epsabs, a.epsrel);
      }
      if (result > 0.0) term = log(result) + A + a.precomp[ch];
      else flag = 2;
    }
    Bfinal = Bv;
    Bout = Bv;
  }
  if (lane == 0) {
    a.chan_ll[o] = term;
    a.chan_flag[o] = flag;
    if (a.mcl_bg && flag == 0) {
      a.mcl_bg[o] = Bout * T;
      double Bs = Bout;
      if (Bs < support[0]) Bs = support[0];
      else if (Bs > support[1] && support[1] > 0.0) Bs = support[1];
      a.mcl_bg_s[o] = Bs * T;
    }
  }
  if (a.star) {
    for (int j = lane; j < B; j += 32) {
      double s = w.star[j];
      if (flag == 0) s = SCALE * (s + Bfinal);
      a.star[o * B + j] = s;
    }
  }
}

// What bounds it: the FP64 pipe (Newton's reciprocals, the sums over the bins,
// the normalisation's logarithm: some 300 instructions of 16 cycles per SM),
// then FP32 issue (the integrand's logarithms) and instruction fetch, so the
// integrand, the bins' integrals and Newton's sums are one copy of code each
// and the adaptive rule a call.  Persistent CTAs form the phase grid's
// reciprocals once.  With some 600 FP64 instructions per channel and inlined
// copies (FP64 pipe 66 % busy, a third of the stalls for instructions): 1500
// channels 134 us, 100 vectors of 300 channels 1188 us, 24 vectors of 1500
// 1779 us; now 110, 910 and 1417 us.
__global__ void __launch_bounds__(32 * kWarps) like_channel_kernel(LikeArgs a) {
  __shared__ WarpSmem ws[kWarps];
  __shared__ DF s_logt[XG_LOGT_N];
  // the phase grid's h, 1 / h and 1 / h^2 as pairs, shared by the warps' Akima builds
  __shared__ DF s_h[kQagLimit], s_ih[kQagLimit], s_ih2[kQagLimit];
  for (int t = threadIdx.x; t < XG_LOGT_N; t += blockDim.x) s_logt[t] = DF{XG_LOGT[t][0], XG_LOGT[t][1]};
  for (int t = threadIdx.x; t < a.N_P - 1 && t < kQagLimit; t += blockDim.x) {
    const double h = a.comp_phases[t + 1] - a.comp_phases[t];
    s_h[t] = df_split_bits(h, 0);
    s_ih[t] = df_split(1.0 / h);
    s_ih2[t] = df_split(1.0 / (h * h));
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  WarpSmem &w = ws[wid];
  const long total = (long)a.n_vec * a.K;
  for (long gw = (long)blockIdx.x * kWarps + wid; gw < total; gw += (long)gridDim.x * kWarps)
    like_channel(a, w, s_logt, s_h, s_ih, s_ih2, lane, (int)(gw / a.K), (int)(gw % a.K));
}

// (s, c) += x with Neumaier's compensation: s + c carries the sum to about
// twice the working precision whatever the order of magnitudes
__device__ __forceinline__ void comp_add(double &s, double &c, double x) {
  const double t = s + x;
  // (|s| >= |x| by the bit patterns)
  const bool larger = (__double_as_longlong(s) & LLONG_MAX) >=
                      (__double_as_longlong(x) & LLONG_MAX);
  c += larger ? (s - t) + x : (x - t) + s;
  s = t;
}

// per-evaluation sum over channels and the reference's early exits: one CTA
// per evaluation; the first flagged channel (lowest index) decides the
// early exit (:677-684, :423-429), otherwise the channel terms are summed
// with compensation (each thread over its channels, then the lanes' sums and
// corrections by a fixed butterfly and the warps' in order: bitwise
// reproducible)
constexpr int kFinalWarps = 4;
__global__ void __launch_bounds__(32 * kFinalWarps) like_finalize_kernel(LikeArgs a) {
  __shared__ double s_s[kFinalWarps], s_c[kFinalWarps];
  __shared__ int s_first[kFinalWarps];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int v = blockIdx.x;
  double LL = 0.0, LLc = 0.0;
  int first = 0x7fffffff;
  // (eight channels' loads in flight: one by one they took half of 18 us)
  constexpr int kAhead = 8;
  for (int base = threadIdx.x; base < a.K; base += kAhead * blockDim.x) {
    double term[kAhead];
    int flag[kAhead];
#pragma unroll
    for (int z = 0; z < kAhead; z++) {
      const int ch = base + z * blockDim.x;
      const size_t o = (size_t)v * a.K + ch;
      flag[z] = ch < a.K ? a.chan_flag[o] : 0;
      term[z] = ch < a.K ? a.chan_ll[o] : 0.0;
    }
#pragma unroll
    for (int z = 0; z < kAhead; z++) {
      const int ch = base + z * blockDim.x;
      if (ch >= a.K) break;
      if (flag[z] != 0) first = min(first, ch);
      else comp_add(LL, LLc, term[z]);
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    first = min(first, __shfl_xor_sync(0xffffffffu, first, o));
    const double s2 = __shfl_xor_sync(0xffffffffu, LL, o);
    const double c2 = __shfl_xor_sync(0xffffffffu, LLc, o);
    // both lanes of a pair form the same (s, c): add the lower lane's pair
    // to the higher's in a fixed order
    double s = (lane & o) ? s2 : LL, c = (lane & o) ? c2 : LLc;
    comp_add(s, c, (lane & o) ? LL : s2);
    c += (lane & o) ? LLc : c2;
    LL = s;
    LLc = c;
  }
  if (lane == 0) {
    s_s[wid] = LL;
    s_c[wid] = LLc;
    s_first[wid] = first;
  }
  __syncthreads();
  if (threadIdx.x != 0) return;
  for (int w = 1; w < kFinalWarps; w++) {
    comp_add(LL, LLc, s_s[w]);
    LLc += s_c[w];
    first = min(first, s_first[w]);
  }
  LL = LL + LLc;
  int st = kOk;
  if (first != 0x7fffffff) {
    const int f = a.chan_flag[(size_t)v * a.K + first];
    // llzero * (0.1 + 0.9 U): U from a hash of (evaluation, channel)
    uint32_t hsh = (uint32_t)v * 2654435761u ^ (uint32_t)first * 40503u ^ 0x9e3779b9u;
    hsh ^= hsh >> 16; hsh *= 0x7feb352du; hsh ^= hsh >> 15; hsh *= 0x846ca68bu; hsh ^= hsh >> 16;
    const double U = (double)(hsh >> 8) / 16777215.0;
    LL = a.llzero * (0.1 + 0.9 * U);
    st = (f == 1) ? kSlimCut : kQuadFail;
  }
  a.loglike[v] = LL;
  a.status[v] = st;
}

}  // namespace

void launch_likelihood(const LikeArgs &a, cudaStream_t st) {
  long warps = (long)a.n_vec * a.K;
  if (warps <= 0) return;
  unsigned blocks = (unsigned)((warps + kWarps - 1) / kWarps);
  // (at most 16 CTAs per SM, four of them resident: each takes several channels,
  // and the phase grid's reciprocals are formed 16 times per SM at most)
  like_channel_kernel<<<blocks < 152u * 16u ? blocks : 152u * 16u, 32 * kWarps, 0, st>>>(a);
  like_finalize_kernel<<<a.n_vec, 32 * kFinalWarps, 0, st>>>(a);
}

}  // namespace xg

namespace xg {
namespace {
// default_background_marginalisation.pyx:38-68: -sum_j ln(d_ij!)
__global__ void precomp_kernel(int K, int B, const int32_t *counts, double *out) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= K) return;
  double s = 0.0;
  for (int j = 0; j < B; j++) s += lgamma((double)(uint32_t)counts[(size_t)i * B + j] + 1.0);
  out[i] = -s;
}
}  // namespace

void launch_precomputation(int K, int B, const int32_t *counts, double *out, cudaStream_t st) {
  if (K <= 0) return;
  precomp_kernel<<<(K + 127) / 128, 128, 0, st>>>(K, B, counts, out);
}
}  // namespace xg

// ---------------------------------------------------------------------------
// Allocation-free variant of the batched likelihood entry point.
//
// Some callers cannot allocate device memory when they call the likelihood:
// a sampler or serving host whose framework owns all device memory through
// its own pool (allocations from outside the pool fail or fragment it), and
// code that must run in a fixed memory budget known in advance.  For them
// xgpu_likelihood_batch_static takes device inputs and outputs from the
// caller, as xgpu_likelihood_batch does, and keeps the per-(evaluation,
// channel) scratch -- the channel's log-likelihood term and its early-exit
// flag -- in the fixed array below, which every GPU that loads this library
// holds until the process exits.
// ---------------------------------------------------------------------------
#include <mutex>

#include "../../include/xpsi_gb300.h"

namespace {

// 4 MiB: 12 bytes per (evaluation, channel) -> at most 349525 of them
constexpr size_t kLikeScratchBytes = size_t(4) << 20;
constexpr size_t kLikeScratchPerChannel = sizeof(double) + sizeof(int32_t);
static __device__ __align__(256) unsigned char g_like_scratch[kLikeScratchBytes];

// device address of g_like_scratch per device, looked up with that device
// current (the host-side name of the array is not a device address) and
// kept with the unique id of the context it belongs to: a context created
// anew (after cudaDeviceReset) has a new id, and the address is looked up
// again instead of reusing one from the destroyed context
std::mutex g_like_scratch_mu;
void *g_like_scratch_addr[64] = {};
unsigned long long g_like_scratch_ctx[64] = {};

using CtxGetCurrent = int (*)(void **);
using CtxGetId = int (*)(void *, unsigned long long *);

// the current context's unique id, through the driver entry points the
// runtime hands out (no link-time dependency on the driver library); 0 if
// they are unavailable
unsigned long long current_context_id() {
  static CtxGetCurrent get_cur = nullptr;
  static CtxGetId get_id = nullptr;
  static bool looked = false;
  if (!looked) {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &p, 12000, cudaEnableDefault, &q) ==
            cudaSuccess && q == cudaDriverEntryPointSuccess)
      get_cur = reinterpret_cast<CtxGetCurrent>(p);
    p = nullptr;
    if (cudaGetDriverEntryPointByVersion("cuCtxGetId", &p, 12000, cudaEnableDefault, &q) ==
            cudaSuccess && q == cudaDriverEntryPointSuccess)
      get_id = reinterpret_cast<CtxGetId>(p);
    looked = true;
  }
  void *ctx = nullptr;
  unsigned long long id = 0;
  if (get_cur && get_id && get_cur(&ctx) == 0 && ctx && get_id(ctx, &id) == 0) return id;
  return 0;
}

int like_scratch_address(void **out) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return -4;
  std::lock_guard<std::mutex> lk(g_like_scratch_mu);
  const unsigned long long ctx = current_context_id();
  if (!g_like_scratch_addr[dev] || ctx == 0 || ctx != g_like_scratch_ctx[dev]) {
    void *p = nullptr;
    if (cudaGetSymbolAddress(&p, g_like_scratch) != cudaSuccess || p == nullptr) return -4;
    g_like_scratch_addr[dev] = p;
    g_like_scratch_ctx[dev] = ctx;
  }
  *out = g_like_scratch_addr[dev];
  return 0;
}

}  // namespace

extern "C" int xgpu_likelihood_batch_static(const xgpu_likelihood_batch_data *d,
                                            void *stream) {
  if (d == nullptr || d->n_vec < 0 || d->K <= 0) return -2;
  if (d->B > 64 || d->N_P < 5) return -2;
  const size_t n = (size_t)d->n_vec * (size_t)d->K;
  if (n > kLikeScratchBytes / kLikeScratchPerChannel) return -3;
  void *base = nullptr;
  int rc = like_scratch_address(&base);
  if (rc) return rc;
  if (n == 0) return 0;
  xg::LikeArgs a{};
  a.n_vec = d->n_vec; a.K = d->K; a.B = d->B; a.H = d->H; a.N_P = d->N_P;
  a.exposure = d->exposure; a.epsabs = d->epsabs; a.epsrel = d->epsrel;
  a.epsilon = d->epsilon; a.sigmas = d->sigmas; a.llzero = d->llzero; a.slim = d->slim;
  a.phase_edges = d->phase_edges; a.comp_phases = d->comp_phases; a.counts = d->counts;
  a.precomp = d->precomp; a.support = d->support; a.background = d->background;
  a.signals = d->signals; a.shifts = d->shifts; a.allow_negative = d->allow_negative;
  // every (evaluation, channel) term and flag is written by the channel
  // kernel before the finalize kernel reads it, so nothing needs clearing
  a.chan_ll = static_cast<double *>(base);
  a.chan_flag = reinterpret_cast<int32_t *>(static_cast<unsigned char *>(base) + n * sizeof(double));
  a.star = d->star; a.mcl_bg = d->mcl_bg; a.mcl_bg_s = d->mcl_bg_support;
  a.loglike = d->loglike; a.status = d->status;
  xg::launch_likelihood(a, static_cast<cudaStream_t>(stream));
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}
