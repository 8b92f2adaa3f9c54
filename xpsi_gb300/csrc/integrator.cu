// integrator.cu -- K2+K3: the cell-mesh integrator for azimuthally invariant
// hot regions, replacing
// xpsi/cellmesh/integrator_for_azimuthal_invariance.pyx:70-665 with the
// blackbody (hot_BB.pyx:54-98) and numerical 4-D (hot_Num4D.pyx:248-461)
// atmospheres.
//
// Work decomposition (CTAs that take items in turn: a chunk of consecutive
// parallels of one mesh, and all or a share of its energies):
//   1. leaf geometry, in a pre-pass with a CTA per parallel, one thread per leaf
//      pair (k, N_L-1-k): image deflection,
//      cos alpha / lag / d cos alpha from the Steffen ray tables, Doppler and
//      aberration factors (:342-441);
//   2. one thread runs the sequential visibility state machine that fills the
//      phase knots through invisible intervals (:480-549) and records, per
//      profile column, which leaf's radiation it carries (or zero);
//   3. per chunk of energies: the specific intensities of every column
//      (:445-478) -> Akima-periodic piece coefficients in shared memory
//      (:566-569) -> the sums of A_ij max(S, 0) over cells x phases
//      (:571-598), from power sums over runs of cells in one knot interval;
//   4. per-chunk partial sums are reduced in a fixed order and divided by
//      E keV (:605-612), so results are bitwise reproducible run to run.
//
// Num4D call history.  The reference evaluator keeps its stencil base node
// between calls and clamps an out-of-table cos(emission angle) only on the
// call that moves the node (hot_Num4D.pyx:300-351).  mu * eta exceeds the
// table's mu range on the approaching limb, so for such leaves the first
// energy is evaluated at the clamped mu = mu_max when the previously
// evaluated leaf sat below the table's third-to-last mu node, and every
// other energy extrapolates the last stencil.  The kernels reproduce the
// reference's single-thread call order exactly: a geometry pre-pass and a
// per-mesh scan hand each parallel the state its first evaluation sees.
#include <climits>
#include <type_traits>

#include "common.cuh"
#include "kernels.h"

namespace xg {

namespace {

constexpr int kThreads = 256;
constexpr int kEPT = 8;  // energies per accumulation task
constexpr int kMaxCellsF = 256;  // cells per parallel held as FP32 pairs in shared memory
constexpr int kMaxPhases = 1024;  // signal phases held as FP32 pairs in shared memory
constexpr int kStrip = 8;  // Akima pieces per thread, built from a sliding window of chords

// Akima piece of one energy row: value at the left knot and the three
// polynomial coefficients (FP64: 32 bytes, two 16-byte shared loads; FP32:
// one 16-byte load).
template <typename WT>
struct __align__(16) PieceT {
  WT y, k1, k2, k3;
};
using Piece = PieceT<double>;

struct RowCtx {
  int S1, N_R, J, IO;
  const double *D, *CA, *LG;  // ray tables of the row
  int jalt;                   // first ray with deflection > pi/2
  double alt_xmin;            // cos(D[jalt])
  double radius, Grav_z, cos_gamma, sin_gamma, cos_th, sin_th, th_over_pi, beta, Lorentz;
  double maxDefl, cos_i, sin_i, inclination;
  double vec0, vec1;
};

struct GeoSmem {
  double *phase, *leafphase, *Z, *ABB, *GEOM;
  double *rD;  // the parallel's deflection table, staged for the binary searches
  int *src, *calc, *term, *clamp0;
  int *flags;  // [0] terminate, [1] invisible image, [2] any evaluation, [3] last_top
  // the rest is the Stokes kernel's:
  double *lgE;  // [EC] log10 of the chunk's energies, or the energies (2-D tables)
  double *lzs;  // [N_L] log10(Z), or Z, per leaf (2-D tables)
  int *sc_exp;  // [EC] binary exponent of the largest |profile value| per energy row
  DF *ih, *ih2;  // [N_L] 1/h and 1/h^2 of the phase intervals
  double *c2chi = nullptr, *s2chi = nullptr;  // [N_L] cos, sin of twice the polarisation
                                              // angle
};


// knot spacings around interval i of an n-knot table, for steffen_piece's
// slopes: one table's spacings serve several value tables
struct SteffenH {
  double h, hl, hr;
  bool first, last;
};
// steffen_piece() with the spacings given and the values at i - 1 .. i + 2
// (the same operations)
__device__ __forceinline__ Cubic steffen_from(const SteffenH &g, double x0, double ym, double y0,
                                              double y1, double y2) {
  const double s = (y1 - y0) / g.h;
  auto slope = [](double sl, double sr, double hl, double hr) {
    const double p = (sl * hr + sr * hl) / (hl + hr);
    const double mag = fmin(fabs(sl), fmin(fabs(sr), 0.5 * fabs(p)));
    return (copysign(1.0, sl) + copysign(1.0, sr)) * mag;
  };
  const double d0 = g.first ? s : slope((y0 - ym) / g.hl, s, g.hl, g.h);
  const double d1 = g.last ? s : slope(s, (y2 - y1) / g.hr, g.h, g.hr);
  Cubic c;
  c.x0 = x0;
  c.y0 = y0;
  c.k1 = d0;
  c.k2 = (3.0 * s - 2.0 * d0 - d1) / g.h;
  c.k3 = (d0 + d1 - 2.0 * s) / (g.h * g.h);
  return c;
}

// per-leaf geometry, integrator_for_azimuthal_invariance.pyx:342-441.  The
// interval of the main table is found once for cos alpha and lag, each
// table's piece formed once for value and derivative, and the interval of the
// reversed table on cos(deflection) found from the main one's (its knots are
// the cosines of the same deflections), so four cosines replace a bisection's
// ten.
__device__ void leaf_geometry(const RowCtx &c, int I, int k, int N_L, int leaf_lim,
                              const double *leaves, GeoSmem &g) {
  double cos_psi = c.cos_i * c.cos_th + c.sin_i * c.sin_th * cos(leaves[k]);
  double psi = image_deflection(I, acos(cos_psi));
  double sin_psi = sin(psi);
  if (!are_equal(psi, 0.0) && are_equal(sin_psi, 0.0)) {
    double _i = (c.cos_i >= 0.0) ? c.inclination + c.inclination * 1.0e-6
                                 : c.inclination - c.inclination * 1.0e-6;
    cos_psi = cos(_i) * c.cos_th + sin(_i) * c.sin_th * cos(leaves[k]);
    psi = image_deflection(I, acos(cos_psi));
    sin_psi = sin(psi);
  }
  const int N_R = c.N_R;
  int calc = 0, term = 0;
  double sin_alpha = 0.0, mu = 0.0, cos_a = 0.0, dca = 0.0;
  int iv = 0;
  SteffenH hm{};
  bool alt = false;
  if (psi <= c.maxDefl) {
    if (psi < c.D[0] || psi > c.D[N_R - 1]) {
      term = 1;
    } else {
      alt = psi <= kHalfPi && cos_psi >= c.alt_xmin;
      iv = locate_bits<true>(c.D, N_R, psi);
      hm.h = c.D[iv + 1] - c.D[iv];
      hm.first = iv == 0;
      hm.last = iv + 1 == N_R - 1;
      if (!hm.first) hm.hl = c.D[iv] - c.D[iv - 1];
      if (!hm.last) hm.hr = c.D[iv + 2] - c.D[iv + 1];
      Cubic q;
      double at;
      if (alt) {
        // knots x(t) = cos(D[jalt - t]), t = 0 .. jalt, ascending; x(t) <= cos psi
        AltX ax{c.D, c.jalt};
        const int n = c.jalt + 1;
        const long long v = ordered(cos_psi);
        int t = min(max(c.jalt - iv - 1, 0), n - 2);
        double x0 = ax(t), x1 = ax(t + 1);
        while (t < n - 2 && ordered(x1) <= v) {
          t++;
          x0 = x1;
          x1 = ax(t + 1);
        }
        while (t > 0 && ordered(x0) > v) {
          t--;
          x1 = x0;
          x0 = ax(t);
        }
        SteffenH ha;
        ha.h = x1 - x0;
        ha.first = t == 0;
        ha.last = t + 1 == n - 1;
        ha.hl = ha.first ? 1.0 : x0 - ax(t - 1);
        ha.hr = ha.last ? 1.0 : ax(t + 2) - x1;
        const int d = c.jalt - t;  // the value table's index of knot t
        q = steffen_from(ha, x0, ha.first ? 0.0 : c.CA[d + 1], c.CA[d], c.CA[d - 1],
                         ha.last ? 0.0 : c.CA[d - 2]);
        at = cos_psi;
      } else {
        q = steffen_from(hm, c.D[iv], hm.first ? 0.0 : c.CA[iv - 1], c.CA[iv], c.CA[iv + 1],
                         hm.last ? 0.0 : c.CA[iv + 2]);
        at = psi;
      }
      cos_a = cubic_eval(q, at);
      dca = cubic_deriv(q, at);
      sin_alpha = sqrt(1.0 - cos_a * cos_a);
      mu = cos_a * c.cos_gamma;
      if (!are_equal(psi, 0.0)) {
        double cos_delta = (c.cos_i - c.cos_th * cos_psi) / (c.sin_th * sin_psi);
        if (c.th_over_pi < 0.5) mu = mu + sin_alpha * c.sin_gamma * cos_delta;
        else mu = mu - sin_alpha * c.sin_gamma * cos_delta;
      }
      calc = (mu > 0.0) ? 1 : 0;
    }
  }
  if (calc && !term) {
    double deriv = dca;
    // the reference's exp(log|deriv| - log|sin psi|), as the quotient
    // (the same zero, infinite and NaN cases; an ulp apart)
    if (!alt) deriv = fabs(deriv) / fabs(sin_psi);
    const Cubic ql = steffen_from(hm, c.D[iv], hm.first ? 0.0 : c.LG[iv - 1], c.LG[iv],
                                  c.LG[iv + 1], hm.last ? 0.0 : c.LG[iv + 2]);
    const double plag = cubic_eval(ql, psi);
    for (int ks = 0; ks < 2; ks++) {
      if ((0 < k && k < leaf_lim - 1) || (k == 0 && ks == 0) ||
          (k == leaf_lim - 1 && N_L % 2 == 1 && ks == 0) ||
          (k == leaf_lim - 1 && N_L % 2 == 0)) {
        int kdx = (ks == 0) ? k : N_L - 1 - k;
        double superlum, eta, cos_xi = 0.0;
        if (!are_equal(psi, 0.0)) {
          cos_xi = sin_alpha * c.sin_i * sin(leaves[kdx]) / sin_psi;
          superlum = 1.0 + c.beta * cos_xi;
          eta = c.Lorentz / superlum;
        } else {
          superlum = 1.0;
          eta = c.Lorentz;
        }
        g.Z[kdx] = eta * c.Grav_z;
        g.ABB[kdx] = mu * eta;
        g.GEOM[kdx] = mu * fabs(deriv) * c.Grav_z * eta * eta * eta / superlum;
        g.leafphase[kdx] = leaves[kdx] + plag;
        if (g.c2chi) {  // integratorIQU_for_azimuthal_invariance.pyx:463-466
          const double chi = pol_angle(leaves[kdx], sin_psi, cos_psi, sin_alpha, cos_a, c.sin_th,
                                       c.cos_th, c.sin_i, c.cos_i, c.sin_gamma, c.cos_gamma,
                                       c.Grav_z, mu, eta, c.beta, c.Lorentz, cos_xi);
          g.c2chi[kdx] = cos(2 * chi);
          g.s2chi[kdx] = sin(2 * chi);
        }
      }
    }
  }
  g.calc[k] = calc;
  g.term[k] = term;
}

// sequential visibility state machine, :480-563.  Runs on one thread.
// Returns through g.flags: [0] terminate, [1] no visibility in this image.
// Tracks the Num4D call-history flag `top` (last evaluated mu*eta above the
// table's third-to-last mu node) and marks columns whose first energy sees a
// clamped mu; *first receives the first evaluated leaf.
__device__ void state_machine(int N_L, int leaf_lim, const double *leaves, GeoSmem &g,
                              bool num4d, double mu_top3, double mu_max, int &top,
                              int &any_eval, int *first = nullptr) {
  int InvisFlag = 2, InvisPhase = 0;
  double step;
  int term = 0;
  for (int m = 0; m < N_L; m++) g.src[m] = -1;
  for (int k = 0; k < leaf_lim; k++) {
    if (g.term[k]) { term = 1; break; }
    if (g.calc[k]) {
      for (int ks = 0; ks < 2; ks++) {
        if ((0 < k && k < leaf_lim - 1) || (k == 0 && ks == 0) ||
            (k == leaf_lim - 1 && N_L % 2 == 1 && ks == 0) ||
            (k == leaf_lim - 1 && N_L % 2 == 0)) {
          int kdx = (ks == 0) ? k : N_L - 1 - k;
          // the reference writes the knot when it reaches this leaf (:441);
          // earlier gap fills may have passed over this position
          g.phase[kdx] = g.leafphase[kdx];
          g.src[kdx] = kdx;
          if (num4d) {
            double a = g.ABB[kdx];
            g.clamp0[kdx] = (a > mu_max && !top) ? 1 : 0;
            top = (a > mu_top3) ? 1 : 0;
          }
          if (!any_eval && first) *first = kdx;
          any_eval = 1;
        }
      }
      if (k == 0) {
        g.phase[N_L - 1] = g.phase[0] + kTwoPi;
        g.src[N_L - 1] = g.src[0];
      } else if (k > 0 && InvisFlag == 2) {
        step = leaves[k] / (double)k;
        for (int m = N_L - k; m < N_L; m++) g.phase[m] = g.phase[m - 1] + step;
        for (int m = N_L - k; m < N_L; m++) g.src[m] = -1;
        g.phase[0] = g.phase[N_L - 1] - kTwoPi;
        for (int m = 1; m < k; m++) g.phase[m] = g.phase[m - 1] + step;
        g.src[0] = -1;
        for (int m = 1; m < k; m++) g.src[m] = -1;
      } else if (InvisFlag == 1) {
        step = g.phase[k] - g.phase[InvisPhase - 1];
        step = step / (double)(k - InvisPhase + 1);
        for (int m = InvisPhase; m < k; m++) g.phase[m] = g.phase[m - 1] + step;
        step = g.phase[N_L - InvisPhase] - g.phase[N_L - 1 - k];
        step = step / (double)(k - InvisPhase + 1);
        for (int m = N_L - k; m < N_L - InvisPhase; m++) g.phase[m] = g.phase[m - 1] + step;
      }
      InvisFlag = 0;
    } else {
      if (InvisFlag == 0) {
        step = g.phase[N_L - k] - g.phase[k - 1];
        step = step / (double)(N_L - 2 * k + 1);
        for (int m = k; m < N_L - k; m++) g.phase[m] = g.phase[m - 1] + step;
        for (int m = k; m < N_L - k; m++) g.src[m] = -1;
        InvisFlag = 1;
        InvisPhase = k;
      }
    }
  }
  int invis = 0;
  if (!term) {
    if (InvisFlag == 2) {
      invis = 1;
    } else {
      for (int m = 1; m < N_L; m++)
        // (rising by their bits, as nearly all do, says it in fewer instructions)
        if (!(ordered(g.phase[m]) > ordered(g.phase[m - 1])) &&
            at_most(g.phase[m], g.phase[m - 1])) {
          term = 1;
          break;
        }
    }
  }
  g.flags[0] = term;
  g.flags[1] = invis;
}

// the parallel's context, formed by the first warp (the FP64 pipe takes an
// instruction of every warp in turn, so one warp's worth serves the CTA) into
// `sc`; false when no cell of it radiates.  Ends with a block barrier.
__device__ bool load_row(const IntegrateArgs &a, const MemberDesc &M, int64_t row, int i,
                         RowCtx &c, RowCtx *sc) {
  // first radiating cell of the parallel (:286-296)
  if (threadIdx.x < 32) {
    const int32_t *rad = a.radiates + M.cell_off + (int64_t)i * M.S1;
    int best = M.S1;
    for (int j = threadIdx.x; j < M.S1; j += 32)
      if (rad[j] == 1) { best = min(best, j); break; }
    for (int o = 16; o > 0; o >>= 1) best = min(best, __shfl_xor_sync(0xffffffffu, best, o));
    RowCtx r{};
    r.J = best;
    r.S1 = M.S1;
    if (best < M.S1) {
      r.N_R = a.N_R;
      r.D = a.deflection + row * a.N_R;
      r.CA = a.cos_alpha + row * a.N_R;
      r.LG = a.lag + row * a.N_R;
      r.jalt = a.N_R - 1;  // set by stage_deflection()
      r.radius = a.radius[row];
      r.Grav_z = sqrt(1.0 - a.u[row]);
      r.cos_gamma = a.cos_gamma[row];
      r.sin_gamma = sqrt(1.0 - r.cos_gamma * r.cos_gamma);
      double th = a.theta0[row];
      r.cos_th = cos(th);
      r.sin_th = sin(th);
      r.th_over_pi = th / kPi;
      r.beta = r.radius * M.omega * r.sin_th / (kC * r.Grav_z);
      r.Lorentz = sqrt(1.0 - r.beta * r.beta);
      r.maxDefl = a.maxDeflection[row];
      r.inclination = M.inclination;
      r.cos_i = cos(M.inclination);
      r.sin_i = sin(M.inclination);
      // (a failed row's deflection, NaN or below zero, has no images)
      r.IO = M.image_order_limit > 0 ? M.image_order_limit
                                     : (r.maxDefl > 0.0 ? (int)ceil(r.maxDefl / kPi) : 0);
      const double *vec = a.params + (M.cell_off + (int64_t)i * M.S1 + best) * a.n_params;
      r.vec0 = vec[0];
      r.vec1 = vec[1];
    }
    if (threadIdx.x == 0) *sc = r;
  }
  __syncthreads();
  c = *sc;
  __syncthreads();
  return c.J < M.S1;
}

// Copy the parallel's deflection table to shared memory (the leaf searches
// probe it ~10 times per lookup) and find the first ray deflected beyond
// pi/2 (:301-303; the reference's scan is unbounded, here it stops at the
// last ray; a NaN ends it, as there, and its cosine rules the second table
// out).  All threads of the CTA call it.
__device__ void stage_deflection(RowCtx &c, GeoSmem &g, int *s_jalt) {
  const int N_R = c.N_R;
  for (int t = threadIdx.x; t < N_R; t += blockDim.x) g.rD[t] = c.D[t];
  if (threadIdx.x == 0) *s_jalt = N_R - 1;
  __syncthreads();
  for (int t = threadIdx.x; t < N_R - 1; t += blockDim.x)
    if (!at_most(g.rD[t], kHalfPi)) atomicMin(s_jalt, t);
  __syncthreads();
  c.jalt = *s_jalt;
  c.D = g.rD;
  c.alt_xmin = cos(c.D[c.jalt]);
  __syncthreads();
}



struct AtmSmem {
  double *gmu, *gE;      // grids of mu and log10(E/kT)
  double *smu, *sE;      // inverse Lagrange denominators per stencil base, 4 each
  float *fgmu, *fgE;     // FP32 copies of the grids, for the guided searches
  float *fphase;         // FP32 copy of the phase knots
  float *fphase_lo;      // phase knot minus its FP32 copy
  float *fcphi, *fcphi_lo;  // cell azimuths of the parallel as float pairs (<= kMaxCellsF)
  float *fcarea, *fcarea_lo;  // cell areas of the parallel as float pairs (<= kMaxCellsF)
};

// inverse denominators of the 4-point Lagrange basis on grid[b..b+3]
// (hot_Num4D.pyx:177-188, computed in the reference's order)
__device__ __forceinline__ void lagrange_space(const double *P, int b, double s[4]) {
  double s0 = 1.0 / (P[b] - P[b + 1]); s0 /= P[b] - P[b + 2]; s0 /= P[b] - P[b + 3];
  double s1 = 1.0 / (P[b + 1] - P[b]); s1 /= P[b + 1] - P[b + 2]; s1 /= P[b + 1] - P[b + 3];
  double s2 = 1.0 / (P[b + 2] - P[b]); s2 /= P[b + 2] - P[b + 1]; s2 /= P[b + 2] - P[b + 3];
  double s3 = 1.0 / (P[b + 3] - P[b]); s3 /= P[b + 3] - P[b + 1]; s3 /= P[b + 3] - P[b + 2];
  s[0] = s0; s[1] = s1; s[2] = s2; s[3] = s3;
}

__device__ __forceinline__ void lagrange_w(const double *P, const double *S, int b, double x,
                                           double w[4]) {
  double d0 = (x - P[b + 1]) * (x - P[b + 2]) * (x - P[b + 3]);
  double d1 = (x - P[b]) * (x - P[b + 2]) * (x - P[b + 3]);
  double d2 = (x - P[b]) * (x - P[b + 1]) * (x - P[b + 3]);
  double d3 = (x - P[b]) * (x - P[b + 1]) * (x - P[b + 2]);
  w[0] = d0 * S[4 * b]; w[1] = d1 * S[4 * b + 1]; w[2] = d2 * S[4 * b + 2];
  w[3] = d3 * S[4 * b + 3];
}

// the table grids of a numerical atmosphere in shared memory: mu and E
// nodes, the inverse Lagrange denominators of every stencil base, and the
// FP32 copies the guided stencil searches use; ends with a block barrier
__device__ __forceinline__ void stage_table_grids(const Atmos4D &A, AtmSmem &as, int nmu,
                                                  int nEt) {
  for (int t = threadIdx.x; t < nmu; t += blockDim.x) as.gmu[t] = A.mu[t];
  for (int t = threadIdx.x; t < nEt; t += blockDim.x) as.gE[t] = A.logE[t];
  __syncthreads();
  for (int b = threadIdx.x; b <= nmu - 4; b += blockDim.x) lagrange_space(as.gmu, b, as.smu + 4 * b);
  for (int b = threadIdx.x; b <= nEt - 4; b += blockDim.x) lagrange_space(as.gE, b, as.sE + 4 * b);
  for (int t = threadIdx.x; t < nmu; t += blockDim.x) as.fgmu[t] = (float)as.gmu[t];
  for (int t = threadIdx.x; t < nEt; t += blockDim.x) as.fgE[t] = (float)as.gE[t];
  __syncthreads();
}

// stencil_base with the bisection run on the grid's FP32 copy (FP32 pipe)
// and finished with FP64 comparisons.  Rounding to float is monotone, so the
// float search never stops below the FP64 answer, and stepping down while
// g[lo] > v lands on it exactly: the result equals stencil_base(g, n, v).
__device__ __forceinline__ int stencil_base_guided(const double *g, const float *fg, int n,
                                                   double v) {
  const float vf = (float)v;
  int lo = 0, hi = n - 1;
  while (hi > lo + 1) {
    const int mid = (lo + hi) >> 1;
    if (fg[mid] > vf) hi = mid; else lo = mid;
  }
  while (lo > 0 && g[lo] > v) lo--;
  int b = lo - 1;
  if (b < 0) b = 0;
  if (b > n - 4) b = n - 4;
  return b;
}

// Num4D intensity for a parallel whose (log T, log g) stencil has been
// contracted into `slab` [nmu][nE]: the remaining 4 x 4 (mu, energy) stencil
// (hot_Num4D.pyx:248-439; the stencil bases are those the reference's cached
// walk lands on, see the file header for the mu > 1 case).  It is split in
// two: the mu stencil depends only on the profile column (its cos emission
// angle), so a thread evaluating one column at several energies forms it
// once.  The caller passes v3 = log10(E / E_eff) as log10 E - log10 Z -
// log10 E_eff from per-energy and per-leaf logarithms.
struct MuStencil {
  int b2;
  double w2[4];
};
__device__ __forceinline__ MuStencil mu_stencil(const Atmos4D &A, const AtmSmem &as, double mu,
                                                bool clamp_mu) {
  double v2 = mu;
  const double mu_hi = as.gmu[A.nmu - 1];
  if (v2 > mu_hi && clamp_mu) v2 = mu_hi;
  if (v2 < as.gmu[0]) v2 = as.gmu[0];
  MuStencil m;
  m.b2 = stencil_base_guided(as.gmu, as.fgmu, A.nmu, v2);
  lagrange_w(as.gmu, as.smu, m.b2, v2, m.w2);
  return m;
}
// the stencil sum itself (a Stokes Q table: no positive part, no factor)
__device__ __forceinline__ double eval_table_raw(const Atmos4D &A, const AtmSmem &as,
                                                 const double *slab, const MuStencil &m,
                                                 double v3) {
  if (v3 < as.gE[0]) v3 = as.gE[0];
  if (v3 > as.gE[A.nE - 1]) v3 = as.gE[A.nE - 1];
  const int b3 = stencil_base_guided(as.gE, as.fgE, A.nE, v3);
  double w3[4];
  lagrange_w(as.gE, as.sE, b3, v3, w3);
  double I = 0.0;
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const double *r = slab + (size_t)(m.b2 + k) * A.nE + b3;
    const double t = w3[0] * r[0] + w3[1] * r[1] + w3[2] * r[2] + w3[3] * r[3];
    I += m.w2[k] * t;
  }
  return I;
}
__device__ __forceinline__ double eval_num4d_e(const Atmos4D &A, const AtmSmem &as,
                                               const double *slab, const MuStencil &m,
                                               double v3, double p3) {
  if (v3 < as.gE[0]) v3 = as.gE[0];
  if (v3 > as.gE[A.nE - 1]) v3 = as.gE[A.nE - 1];
  const int b3 = stencil_base_guided(as.gE, as.fgE, A.nE, v3);
  double w3[4];
  lagrange_w(as.gE, as.sE, b3, v3, w3);
  double I = 0.0;
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const double *r = slab + (size_t)(m.b2 + k) * A.nE + b3;
    const double t = w3[0] * r[0] + w3[1] * r[1] + w3[2] * r[2] + w3[3] * r[3];
    I += m.w2[k] * t;
  }
  if (I < 0.0) return 0.0;
  return I * p3;
}

// a double-float pair times 2^d, d <= 0 (exact down to the float range)
__device__ __forceinline__ DF df_scale(DF a, int d) {
  if (d < -125) return DF{0.0f, 0.0f};
  const float f = __int_as_float((127 + d) << 23);
  return DF{a.h * f, a.l * f};
}

// binary exponent x of |f| = m 2^x, m in [0.5, 1), of a nonzero finite float
// from its bit pattern
__device__ __forceinline__ int float_exponent(float f) {
  const int b = (__float_as_int(f) >> 23) & 0xff;
  return b != 0 ? b - 126 : -149 + (32 - __clz(__float_as_int(f) & 0x7fffff));
}
// a double-float times 2^d (0 where 2^d leaves the float range)
__device__ __forceinline__ DF df_times_pow2(DF a, int d) {
  if (d < -126 || d > 127) return DF{0.0f, 0.0f};
  const float f = __int_as_float((127 + d) << 23);
  return DF{a.h * f, a.l * f};
}

// FP32 forms for the mixed-precision integrator

// an Akima piece in double-float form, scaled by a power of two per energy
// row (same 32 bytes as the FP64 piece it replaces in shared memory)
struct __align__(16) PieceDF {
  DF y, k1, k2, k3;
};
__device__ __forceinline__ int stencil_base_f(const float *g, int n, float v) {
  int lo = 0, hi = n - 1;
  while (hi > lo + 1) {
    int mid = (lo + hi) >> 1;
    if (g[mid] > v) hi = mid; else lo = mid;
  }
  int b = lo - 1;
  if (b < 0) b = 0;
  if (b > n - 4) b = n - 4;
  return b;
}

__device__ __forceinline__ void lagrange_wf(const float *P, const float *S, int b, float x,
                                            float w[4]) {
  float d0 = (x - P[b + 1]) * (x - P[b + 2]) * (x - P[b + 3]);
  float d1 = (x - P[b]) * (x - P[b + 2]) * (x - P[b + 3]);
  float d2 = (x - P[b]) * (x - P[b + 1]) * (x - P[b + 3]);
  float d3 = (x - P[b]) * (x - P[b + 1]) * (x - P[b + 2]);
  w[0] = d0 * S[4 * b]; w[1] = d1 * S[4 * b + 1]; w[2] = d2 * S[4 * b + 2];
  w[3] = d3 * S[4 * b + 3];
}

// Num4D intensity in the mixed form: the slab and the Lagrange weights in
// FP32, the mu stencil (b2, w2) formed once per profile column; the energy
// coordinate's offset u from the stencil base b3 is the rounding of an FP64
// one, so the weights see the FP32 rounding of an offset of a few grid
// spacings (~1e-9 absolute) rather than that of the coordinate (~3e-8, the
// same on every evaluation of a parallel: a systematic shift).
__device__ __forceinline__ float eval_num4d_f(const float *offs, const float *space, int nE,
                                              const float *slab, int b2, float4 w2, int b3,
                                              float u, float p3) {
  const float *o = offs + 3 * b3;  // node offsets gE[b3 + i] - gE[b3], i = 1..3
  const float d0 = u, d1 = u - o[0], d2 = u - o[1], d3 = u - o[2];
  const float *S = space + 4 * b3;
  const float w3[4] = {d1 * d2 * d3 * S[0], d0 * d2 * d3 * S[1], d0 * d1 * d3 * S[2],
                       d0 * d1 * d2 * S[3]};
  const float w[4] = {w2.x, w2.y, w2.z, w2.w};
  float I = 0.0f;
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const float *r = slab + (size_t)(b2 + k) * nE + b3;
    const float t = w3[0] * r[0] + w3[1] * r[1] + w3[2] * r[2] + w3[3] * r[3];
    I += w[k] * t;
  }
  if (I < 0.0f) return 0.0f;
  return I * p3;
}

__device__ __forceinline__ float eval_bb_f(float E, float kT) {
  return E * E * E / expm1f(E / kT);
}

// energies per chunk: as many as keep every thread in the per-cell sums and the
// coefficients within 96 KB
__host__ __device__ inline int energy_chunk(int N_L, int N_P, int N_E, int piece_bytes) {
  int ec = 8;
  while (ec < 32 && (long)N_P * (ec * 2 / kEPT) <= kThreads && ec * 2 <= N_E + kEPT) ec *= 2;
  while (ec > 8 && (size_t)ec * N_L * piece_bytes > 96 * 1024) ec /= 2;
  return ec;
}

struct Layout {
  int N_L, EC, nmu, nE;
  size_t bytes;
};

// nmu, nE: Num4D grid sizes (0 when no mesh uses the numerical atmosphere)
__host__ __device__ inline Layout make_layout(int N_L, int N_P, int N_E, int nmu = 0,
                                              int nE = 0, int piece_bytes = 32, int N_R = 0) {
  Layout L;
  L.N_L = N_L;
  L.nmu = nmu;
  L.nE = nE;
  const int ec = energy_chunk(N_L, N_P, N_E, piece_bytes);
  L.EC = ec;
  L.bytes = (size_t)5 * N_L * sizeof(double)      // phase, leafphase, Z, ABB, GEOM
            + (size_t)ec * N_L * piece_bytes       // coefficients
            + (size_t)(nmu + nE) * 5 * sizeof(double)  // Num4D grids + inverse denominators
            + (size_t)(nmu + nE) * sizeof(float)       // the grids' FP32 copies
            + (size_t)(2 * N_L + 4 * kMaxCellsF) * sizeof(float)  // knots, cells as pairs
            + (size_t)N_R * sizeof(double)  // staged deflection table
            + (size_t)(ec + N_L) * sizeof(double)  // lgE, lzs
            + (size_t)2 * N_L * sizeof(DF)         // ih, ih2
            + (size_t)(4 * N_L + 8 + ec) * sizeof(int) + 64;
  return L;
}

// bytes carve() takes with no coefficients and no atmosphere arrays (the
// geometry pre-pass)
inline size_t geometry_bytes(int N_L, int N_R) {
  return (size_t)N_R * sizeof(double) + (size_t)8 * N_L * sizeof(double) + 16 /* alignment */ +
         (size_t)(4 * N_L + 8) * sizeof(int) + 16;
}

__device__ GeoSmem carve(char *base, int N_L, int EC, double **coef, int nmu = 0, int nE = 0,
                         AtmSmem *atm = nullptr, int piece_bytes = 32, int N_R = 0) {
  GeoSmem g;
  double *d = reinterpret_cast<double *>(base);
  g.rD = d; d += N_R;
  g.phase = d; d += N_L;
  g.leafphase = d; d += N_L;
  g.Z = d; d += N_L;
  g.ABB = d; d += N_L;
  g.GEOM = d; d += N_L;
  g.lzs = d; d += N_L;
  g.lgE = d; d += EC;
  g.ih = reinterpret_cast<DF *>(d); d += N_L;
  g.ih2 = reinterpret_cast<DF *>(d); d += N_L;
  d = reinterpret_cast<double *>((reinterpret_cast<uintptr_t>(d) + 15) & ~uintptr_t(15));
  *coef = d; d += (size_t)EC * N_L * piece_bytes / 8;
  if (atm) {
    atm->gmu = d; d += nmu;
    atm->gE = d; d += nE;
    atm->smu = d; d += (size_t)4 * nmu;
    atm->sE = d; d += (size_t)4 * nE;
    float *f = reinterpret_cast<float *>(d);
    atm->fgmu = f; f += nmu;
    atm->fgE = f; f += nE;
    atm->fphase = f; f += N_L;
    atm->fphase_lo = f; f += N_L;
    atm->fcphi = f; f += kMaxCellsF;
    atm->fcphi_lo = f; f += kMaxCellsF;
    atm->fcarea = f; f += kMaxCellsF;
    atm->fcarea_lo = f; f += kMaxCellsF;
    d = reinterpret_cast<double *>((reinterpret_cast<uintptr_t>(f) + 15) & ~uintptr_t(15));
  }
  int *ip = reinterpret_cast<int *>(d);
  g.src = ip; ip += N_L;
  g.calc = ip; ip += N_L;
  g.term = ip; ip += N_L;
  g.clamp0 = ip; ip += N_L;
  g.flags = ip; ip += 8;
  g.sc_exp = ip;
  return g;
}

// ---------------------------------------------------------------------------
// Geometry pre-pass, one CTA per parallel: its images' leaf geometry and
// visibility, once, into a record per image that the integrator's CTAs read
// (however many share the parallel's energies), and for the table
// atmospheres whether the parallel evaluates the atmosphere and whether its
// last evaluation leaves the mu stencil at the top of the table.  The work is
// FP64 (trigonometry, the Steffen pieces, a serial walk over the leaves):
// here many parallels' CTAs share an SM and keep the pipe busy, in the
// integrator two of a CTA's warps ran it and the rest waited.
//
// Record of an image, per profile column: the knot's phase, 1 / redshift
// factor Z, cosine mu eta, geometric factor (doubles, [N_L] each), then a
// byte: kColLit the column carries a leaf's radiation (else it is dark and
// the three values are undefined), kColClamp its first energy sees the mu
// clamp, kColFirst it is the parallel's first evaluation.
// ---------------------------------------------------------------------------
constexpr unsigned kColLit = 1, kColClamp = 2, kColFirst = 4;
constexpr int kImgTerm = 1 << 30;  // the image after the parallel's records is the terminate

__host__ __device__ inline int64_t image_doubles(int N_L) { return 4 * (int64_t)N_L + (N_L + 7) / 8; }

// one image of the parallel by the whole CTA: leaf geometry, state machine
// and, when it is visible, the record (rec, or none when null).  s[0], s[1], s[2]: the mu stencil's top
// state, any evaluation so far, the parallel's first evaluated leaf.  Returns
// 0 visible, 1 not visible, 2 terminate.  Ends with a block barrier.
__device__ int image_record(const RowCtx &c, int I, int N_L, const double *leaves, GeoSmem &g,
                            bool table, double mu_top3, double mu_max, int *s, int *s_z,
                            double *rec) {
  const int leaf_lim = (N_L % 2 == 0) ? N_L / 2 : (N_L + 1) / 2;
  for (int k = threadIdx.x; k < leaf_lim; k += blockDim.x)
    leaf_geometry(c, I, k, N_L, leaf_lim, leaves, g);
  __syncthreads();
  const bool before = s[1] != 0;
  __syncthreads();
  if (threadIdx.x == 0) {
    int top = s[0], any = s[1], first = s[2];
    state_machine(N_L, leaf_lim, leaves, g, table, mu_top3, mu_max, top, any, &first);
    s[0] = top;
    s[1] = any;
    s[2] = first;
  }
  __syncthreads();
  const int out = g.flags[0] ? 2 : (g.flags[1] ? 1 : 0);
  if (out == 0) {
    uint8_t *fl = reinterpret_cast<uint8_t *>(rec + 4 * (size_t)N_L);
    float zlo = INFINITY, zhi = 0.0f;
    for (int t = threadIdx.x; t < N_L; t += blockDim.x) {
      const int q = g.src[t];
      if (rec) rec[t] = g.phase[t];
      unsigned f = 0;
      if (q >= 0) {
        if (rec) {
          rec[N_L + t] = g.Z[q];
          rec[2 * N_L + t] = g.ABB[q];
          rec[3 * N_L + t] = g.GEOM[q];
        }
        zlo = fminf(zlo, (float)g.Z[q]);
        zhi = fmaxf(zhi, (float)g.Z[q]);
        f = kColLit | ((table && g.clamp0[q]) ? kColClamp : 0u) |
            ((!before && q == s[2]) ? kColFirst : 0u);
      }
      if (rec) fl[t] = (uint8_t)f;
    }
    if (s_z) {  // the lit columns' smallest and largest Z (positive floats order as ints)
      atomicMin(&s_z[0], __float_as_int(zlo));
      atomicMax(&s_z[1], __float_as_int(zhi));
    }
  }
  __syncthreads();
  return out;
}

constexpr int kPlanThreads = 128;  // the geometry pre-pass's CTA

// chunks of mesh m for a target cost: count (write == false) or write them
// from index c0; returns the count.  Costs are whole numbers, so that nothing
// here waits for the FP64 pipe.
__device__ int plan_mesh(const IntegrateArgs &a, int m, long long target, bool write, int c0) {
  const MemberDesc M = a.members[m];
  int n = 0;
  long long acc = 0;
  int64_t start = M.row_off;
  for (int64_t s = 0; s < M.S0; s++) {
    const int64_t row = M.row_off + s;
    const long long c = (long long)a.row_cost[row];
    if (acc > 0 && acc + c > target) {
      if (write) {
        a.chunk_r0[c0 + n] = start;
        a.chunk_r1[c0 + n] = row;
        a.chunk_cost[c0 + n] = (float)acc;
      }
      n++;
      acc = 0;
      start = row;
    }
    acc += c;
  }
  if (M.S0 > 0) {
    if (write) {
      a.chunk_r0[c0 + n] = start;
      a.chunk_r1[c0 + n] = M.row_off + M.S0;
      a.chunk_cost[c0 + n] = (float)acc;
    }
    n++;
  }
  return n;
}

// exclusive scan of per-thread values over the block; returns the total
__device__ int block_exclusive_scan(int v, int *s_buf, int &excl) {
  const int t = threadIdx.x;
  s_buf[t] = v;
  __syncthreads();
  for (int o = 1; o < kPlanThreads; o <<= 1) {
    const int x = t >= o ? s_buf[t - o] : 0;
    __syncthreads();
    s_buf[t] += x;
    __syncthreads();
  }
  excl = s_buf[t] - v;
  const int total = s_buf[kPlanThreads - 1];
  __syncthreads();
  return total;
}

// The chunks of the call, by the first CTA of the geometry pre-pass, which
// neither needs them nor leaves the chip before it (also log10 of the
// energies).  As a launch of its own between the costs and the pre-pass it took
// 40 us of a 64-parallel call's 690, 29 of one spot's 1205.
__device__ __noinline__ void plan_chunks(const IntegrateArgs &a) {
  __shared__ long long s_sum[kPlanThreads];
  __shared__ int s_scan[kPlanThreads];
  __shared__ int s_hist[64], s_cur[64];
  const int t = threadIdx.x;
  for (int p = t; p < a.N_E; p += kPlanThreads) a.lgE[p] = log10(a.energies[p]);
  // total cost
  long long sum = 0;
  for (int64_t r = t; r < a.n_rows; r += kPlanThreads) sum += (long long)a.row_cost[r];
  s_sum[t] = sum;
  __syncthreads();
  for (int o = kPlanThreads / 2; o > 0; o >>= 1) {
    if (t < o) s_sum[t] += s_sum[t + o];
    __syncthreads();
  }
  // (whole costs exceed the quotient where they exceed its whole part)
  long long target = max(1ll, s_sum[0] / max(1, a.target_chunks));
  // meshes [m0, m1) of this thread
  const int per = (a.n_members + kPlanThreads - 1) / kPlanThreads;
  const int m0 = min(a.n_members, t * per), m1 = min(a.n_members, m0 + per);
  int excl = 0, total = 0;
  for (int pass = 0; pass < 2; pass++) {
    int cnt = 0;
    for (int m = m0; m < m1; m++) cnt += plan_mesh(a, m, target, false, 0);
    total = block_exclusive_scan(cnt, s_scan, excl);
    if (total <= a.max_chunks) break;
    // the bound cannot be exceeded in exact arithmetic; should rounding ever
    // do it, one chunk per mesh fits
    target = LLONG_MAX / 2;
  }
  int c = excl;
  for (int m = m0; m < m1; m++) {
    a.chunk_first[m] = c;
    c += plan_mesh(a, m, target, true, c);
  }
  if (t == 0) {
    a.chunk_first[a.n_members] = total;
    *a.chunk_count = total;
  }
  // heaviest first: counting sort on floor(log2 cost), descending
  if (t < 64) s_hist[t] = 0;
  __syncthreads();
  for (int k = t; k < total; k += kPlanThreads) {
    int e = 0;
    frexpf(a.chunk_cost[k], &e);
    atomicAdd(&s_hist[min(63, max(0, e))], 1);
  }
  __syncthreads();
  if (t == 0) {
    int run = 0;
    for (int b = 63; b >= 0; b--) {
      s_cur[b] = run;
      run += s_hist[b];
    }
  }
  __syncthreads();
  for (int k = t; k < total; k += kPlanThreads) {
    int e = 0;
    frexpf(a.chunk_cost[k], &e);
    a.chunk_order[atomicAdd(&s_cur[min(63, max(0, e))], 1)] = k;
  }
}

// a CTA per parallel; kPlan: after one that plans the call's chunks
template <bool kPlan>
__global__ void __launch_bounds__(kPlanThreads) geometry_kernel(IntegrateArgs a) {
  extern __shared__ __align__(16) char smem[];
  if (kPlan && blockIdx.x == 0) {
    plan_chunks(a);
    return;
  }
  const int64_t row = (int64_t)blockIdx.x - (kPlan ? 1 : 0);
  const int m = a.row_member[row];
  const MemberDesc M = a.members[m];
  const int i = (int)(row - M.row_off);
  const int N_L = a.N_L;
  double *coef;
  GeoSmem g = carve(smem, N_L, 0, &coef, 0, 0, nullptr, 32, a.N_R);
  __shared__ RowCtx s_row;
  __shared__ int s_jalt, s_state[3], s_z[2];
  __shared__ long long s_base;
  RowCtx c;
  if (threadIdx.x == 0) {
    s_state[0] = s_state[1] = s_state[2] = 0;
    s_z[0] = __float_as_int(INFINITY);
    s_z[1] = 0;
    s_base = -1;
  }
  const bool lit = load_row(a, M, row, i, c, &s_row);
  int n = 0;
  if (lit) {
    // records for the images the parallel's deflection reaches (image I lies
    // beyond I pi); none for one beyond what a ray table keeps (100 pi), NaN or
    // infinite, so that no row can take or move the others' room
    const int need =
        c.maxDefl >= 0.0 && c.maxDefl <= 101.0 * kPi ? min(c.IO, (int)(c.maxDefl / kPi) + 1) : 0;
    if (threadIdx.x == 0 && a.geo && need > 0) {
      const long long b = (long long)atomicAdd(a.geo_count, (unsigned long long)need);
      s_base = b + need <= a.geo_cap ? b : -1;
    }
    stage_deflection(c, g, &s_jalt);
    const bool table = a.atmos.I != nullptr;
    const double mu_max = table ? a.atmos.mu[a.atmos.nmu - 1] : 0.0;
    const double mu_top3 = table ? a.atmos.mu[a.atmos.nmu - 3] : 0.0;
    for (int I = 0; I < c.IO; I++) {
      // (without room for the parallel's images the integrator forms them again)
      double *rec = s_base >= 0 && I < need ? a.geo + (s_base + I) * image_doubles(N_L) : nullptr;
      const int got = image_record(c, I, N_L, a.leaves, g, table, mu_top3, mu_max, s_state, s_z,
                                   rec);
      if (got == 0) { n++; continue; }
      if (got == 2) n |= kImgTerm;
      break;
    }
    if ((n & ~kImgTerm) > need && threadIdx.x == 0) s_base = -1;
  }
  if (threadIdx.x == 0) {
    if (a.row_has_eval) {
      a.row_has_eval[row] = (uint8_t)s_state[1];
      a.row_last_top[row] = (uint8_t)s_state[0];
    }
    if (a.row_info) {
      RowInfo r;
      r.geo = s_base;
      if (a.rows_again && s_base < 0 && (n & ~kImgTerm) > 0)
        atomicAdd(reinterpret_cast<unsigned long long *>(a.rows_again), 1ull);
      r.images = n;
      r.cell = c.J;
      r.z_lo = __int_as_float(s_z[0]);
      r.z_hi = __int_as_float(s_z[1]);
      a.row_info[row] = r;
    }
  }
}

// serial over the parallels of each mesh, in the reference's call order
__global__ void num4d_scan_kernel(IntegrateArgs a) {
  int m = blockIdx.x * blockDim.x + threadIdx.x;
  if (m >= a.n_members) return;
  const MemberDesc M = a.members[m];
  if (M.atm != 2 && M.atm != 4 && M.atm != 6) return;
  uint8_t carry = 0;
  for (int i = 0; i < M.S0; i++) {
    int64_t row = M.row_off + i;
    a.row_entry_top[row] = carry;
    if (a.row_has_eval[row]) carry = a.row_last_top[row];
  }
}

// ---------------------------------------------------------------------------
// Cell x phase sums (:571-598).  A task is one signal phase and kEPT energies
// of the current chunk; it walks the radiating cells of the parallel in
// azimuth order, so a cell's interval is found by stepping forward from the
// previous cell's (one or two knot comparisons) rather than by bisection, and
// each (cell, energy) costs the piece's Horner form plus one FMA.
// ---------------------------------------------------------------------------
constexpr int kWrapLimit = 1024;  // 2 pi shifts of a cell phase (a few suffice)

// the phase of cell j at a signal phase, wrapped into the knot range
// (:575-586), with phases as unevaluated float pairs (hi + lo) and error-free
// sums, so the offset t keeps ~1e-14 rad absolute accuracy instead of one
// FP32 ulp of the phase (~5e-7 rad)
template <bool kCached>
struct CellPhaseF {
  const float *knot, *knot_lo;
  int N_L;
  float x_lo, x_hi, ph, ph_lo, tp, tp_lo;
  const float *cphi, *cphi_lo;  // the parallel's cell azimuths as pairs (kCached)
  const double *cphi_d;
  // interval and offset th + tl of cell j's phase
  __device__ __forceinline__ int offset(int j, int hint, float &th, float &tl) const {
    float cp, cp_lo;
    if (kCached) {
      cp = cphi[j];
      cp_lo = cphi_lo[j];
    } else {
      const double c = cphi_d[j];
      cp = (float)c;
      cp_lo = (float)(c - (double)cp);
    }
    float x, lo;
    two_sum(ph, cp, x, lo);
    lo += ph_lo + cp_lo;
    if (x > x_hi) {
      for (int w = 0; x > x_hi && w < kWrapLimit; w++) {
        float e;
        two_sum(x, -tp, x, e);
        lo += e - tp_lo;
      }
    } else if (x < x_lo) {
      for (int w = 0; x < x_lo && w < kWrapLimit; w++) {
        float e;
        two_sum(x, tp, x, e);
        lo += e + tp_lo;
      }
    }
    if (!(x >= x_lo && x <= x_hi)) return -1;
    int iv = hint;
    if (iv < 0 || knot[iv] > x) iv = locate(knot, N_L, x);
    else
      while (iv < N_L - 2 && knot[iv + 1] <= x) iv++;
    float e3;
    two_sum(x, -knot[iv], th, e3);
    tl = e3 + lo - knot_lo[iv];
    return iv;
  }
  __device__ __forceinline__ int operator()(int j, int hint, float &t) const {
    float th, tl;
    const int iv = offset(j, hint, th, tl);
    t = th + tl;
    return iv;
  }
  __device__ __forceinline__ int operator()(int j, int hint, DF &t) const {
    float th, tl;
    const int iv = offset(j, hint, th, tl);
    t = fast_two_sum(th, tl);
    return iv;
  }
};

template <bool kCached>
struct AreaF {
  const float *Af;  // the parallel's cell areas (kCached)
  const double *A;
  __device__ __forceinline__ float operator()(int j) const {
    return kCached ? Af[j] : (float)A[j];
  }
};
template <bool kCached>
struct AreaDF {
  const float *Ah, *Al;  // the parallel's cell areas as pairs (kCached)
  const double *A;
  __device__ __forceinline__ DF operator()(int j) const {
    return kCached ? DF{Ah[j], Al[j]} : df_split(A[j]);
  }
};

// the reference adds an interpolant value when it is > 0 (:593-594)
__device__ __forceinline__ bool positive(float v) { return v > 0.0f; }

// Mixed form: the sums over the radiating cells of one parallel at one signal
// phase for the lane's Z energies; eight lanes share a phase, energies e + 8 z
// of the chunk to lane e.  The lanes place a batch of eight cells (interval
// and offset) in shared memory, then walk it in the cells' order; a piece is
// read where the interval changes, about every third cell.  FP32 issue bounds
// it: five instructions per cell and energy (three FMAs, the reference's test,
// an FMA) and eight per cell that the Z energies share.  With lanes over the
// phases each cell read eight pieces, every (phase, eight energies) placed
// the cells again, and branches kept the eight chains from overlapping (issue
// slots 42 % busy); with one energy per lane the shared part weighed most.
// 64 vectors of two Num4D regions at sqrt_num_cells 96: 28.4 ms lanes over
// phases, 19.6 one energy per lane, 14.7 now.
// True in `bad`: a cell phase cannot be wrapped into the knot range (the
// reference's terminate).
constexpr int kCellLanes = 8;
struct CellStage {
  float2 ta[kThreads];  // offset and area
  int iv[kThreads];
};
template <int Z, typename CP, typename AR>
__device__ __forceinline__ void cell_phase_sums_f(const CP &cp, const AR &area, int S1,
                                                  const int32_t *rad, const float4 *piece, int es,
                                                  CellStage &cs, bool &bad, float (&acc)[Z]) {
  const int lane = threadIdx.x & 31, e = lane % kCellLanes, shift = lane - e;
  float2 *ta = cs.ta + (threadIdx.x - e);
  int *ivs = cs.iv + (threadIdx.x - e);
  int cur = -1;
  bool lost = false;
  float4 q[Z];
#pragma unroll
  for (int z = 0; z < Z; z++) {
    acc[z] = 0.0f;
    q[z] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  for (int b = 0; b < S1; b += kCellLanes) {
    const int j = b + e;
    const bool on = j < S1 && rad[j] == 1;
    const uint32_t lit = __ballot_sync(0xffffffffu, on) & 0xffu;  // the same in every group
    const int n = __popc(lit);
    if (n == 0) continue;
    __syncwarp();  // the last batch's readers are done
    if (on) {
      float t;
      const int iv = cp(j, -1, t);
      lost |= iv < 0;
      const int at = __popc(lit & ((1u << e) - 1u));
      ta[at] = make_float2(t, area(j));
      ivs[at] = max(iv, 0);
    }
    __syncwarp();
    const bool change = e < n && ivs[e] != (e > 0 ? ivs[e - 1] : cur);
    uint32_t read = __ballot_sync(0xffffffffu, change) >> shift;
    cur = ivs[n - 1];
    for (int i = 0; i < n; i++) {
      if (read & 1u) {
        const float4 *p = piece + ivs[i] * es + e;
#pragma unroll
        for (int z = 0; z < Z; z++) q[z] = p[kCellLanes * z];
      }
      read >>= 1;
      const float2 c = ta[i];
#pragma unroll
      for (int z = 0; z < Z; z++) {
        const float sv =
            __fmaf_rn(c.x, __fmaf_rn(c.x, __fmaf_rn(c.x, q[z].w, q[z].z), q[z].y), q[z].x);
        if (positive(sv)) acc[z] = __fmaf_rn(c.y, sv, acc[z]);
      }
    }
  }
  bad = ((__ballot_sync(0xffffffffu, lost) >> shift) & 0xffu) != 0u;
}

// ---------------------------------------------------------------------------
// The FP64 form's Akima pieces of a chunk of energies in shared memory:
// piece (iv, e) is two float4, (y, k1) and (k2, k3) as float pairs, at
// iv * es + e of two arrays.  Energies are adjacent, so the lanes of a group
// that take the energies of one knot interval read consecutive float4; the
// row stride es = EC + 1 (odd) keeps accesses along iv (column intensities,
// the per-cell form) off a single bank group.
// ---------------------------------------------------------------------------
struct PieceRows {
  float4 *a, *b;
  int es;
  __device__ __forceinline__ PieceDF at(int iv, int e) const {
    const float4 p = a[iv * es + e], q = b[iv * es + e];
    return PieceDF{{p.x, p.y}, {p.z, p.w}, {q.x, q.y}, {q.z, q.w}};
  }
  __device__ __forceinline__ DF &y(int iv, int e) const {
    return *reinterpret_cast<DF *>(&a[iv * es + e]);
  }
  __device__ __forceinline__ double &yd(int iv, int e) const {
    return *reinterpret_cast<double *>(&a[iv * es + e]);
  }
  __device__ __forceinline__ int &ex(int iv, int e) const {
    return reinterpret_cast<int *>(&a[iv * es + e])[2];
  }
  __device__ __forceinline__ void put_k(int iv, int e, DF k1, DF k2, DF k3) const {
    float4 &p = a[iv * es + e];
    p.z = k1.h;
    p.w = k1.l;
    b[iv * es + e] = make_float4(k2.h, k2.l, k3.h, k3.l);
  }
};

// the same sums cell by cell in double-float arithmetic, kEPT energies per thread, on
// scaled pieces (the sign test is on the high part: h + l has the sign of h;
// with the elsewhere correction every value is added, :593-594)
template <typename CP, typename AR>
__device__ __forceinline__ bool cell_phase_sums_df(const CP &cp, const AR &area, int S1,
                                                   const int32_t *rad, const PieceRows &pc,
                                                   int pb, bool add_all, DF (&acc)[kEPT]) {
  int hint = -1;
  for (int j = 0; j < S1; j++) {
    if (rad[j] != 1) continue;
    DF t;
    const int iv = cp(j, hint, t);
    if (iv < 0) return false;
    hint = iv;
    const DF A = area(j);
    // every energy slot of the task is evaluated (slots past the chunk's
    // energies read pieces of the coefficient area that the caller ignores)
    // and the positive part is a select: no branch inside the cell, so the
    // kEPT independent double-float chains interleave
#pragma unroll
    for (int e = 0; e < kEPT; e++) {
      const PieceDF q = pc.at(iv, pb + e);
      const DF sv = df_fma(t, df_fma(t, df_fma(t, q.k3, q.k2), q.k1), q.y);
      const DF nx = df_fma(A, sv, acc[e]);
      const bool take = add_all || sv.h > 0.0f;
      acc[e].h = take ? nx.h : acc[e].h;
      acc[e].l = take ? nx.l : acc[e].l;
    }
  }
  return true;
}

// ---------------------------------------------------------------------------
// Power-sum form of the FP64 path's cell x phase sums (the form that runs).
// At a signal phase k the cells of a parallel fall, in azimuth order, into
// runs of consecutive radiating cells whose wrapped phase lies in the same
// knot interval iv (a run ends where the interval changes).  Over a run every
// energy row evaluates the same cubic piece, so
//     sum_j A_j S_E(t_j) = y W0 + k1 W1 + k2 W2 + k3 W3,  Wp = sum_j A_j t_j^p,
// and the power sums Wp depend on the geometry only: they are formed once
// per (parallel, image) and reused by all N_E energies.  This holds where
// the reference adds every value (the elsewhere correction) or where the
// piece is positive on its whole interval; a piece that is <= 0 on its whole
// interval adds nothing.  A piece whose sign changes inside its interval is
// evaluated cell by cell over the run, with the reference's test (:593-594).
// The sign of a piece on [0, h] is bounded by its Bernstein coefficients
// (the curve lies in their convex hull), with a margin of 1e-5 of the
// piece's scale so that rounding cannot flip the classification.
//
// What bounds the sums is FP32 issue: 41 instructions per run and energy
// (four products of pairs into a running pair, below) where the
// per-cell form spends 62 per cell and energy, and a parallel has about
// three cells per run.  The lanes of a group of EC take the chunk's energies
// of one signal phase: they share the run list, the knot interval and the
// records, so nothing diverges and the pieces are read as consecutive
// float4; with lanes over the phases (each its own runs and intervals) the
// same sums ran no faster than the per-cell form.
//
// Run records live in global scratch (L2), per CTA: run r of cell half c (the
// two halves of the parallel's cells are walked by different threads) of
// phase k is record (2 k + c) w_cap + r: two float4 with the float pairs of
// W0, W1 and W2, W3, and an int with the interval (bits 0-9), the first cell
// (bits 10-19) and the cell span (bits 20-29).  A group stages kStage records
// at a time in shared memory (one load per lane, a block ahead): read one by
// one from L2 they cost 600 cycles a run against the 100 of its arithmetic.
// ---------------------------------------------------------------------------
__host__ __device__ inline size_t integrate_wsum_bytes_dev(int N_P, int cap) {
  const size_t n = (size_t)2 * cap * N_P;
  return (n * (2 * sizeof(float4) + sizeof(int)) + 255) & ~size_t(255);
}
constexpr int kStage = 8;
// The last record is empty: no area, in an interval of zeros that follows the
// pieces (of an actual piece, whose coefficients need not be finite where knots
// nearly coincide, it would add 0 times infinity).
struct RunStage {
  float4 w[2 * kStage + 2];
  uint4 meta[kStage + 1];  // interval and cells, class masks of the interval
};

struct WRuns {
  float4 *w;
  int *meta;
  int cap;
  __device__ __forceinline__ size_t first(int k, int half) const {
    return (size_t)(2 * k + half) * cap;
  }
};

__device__ __forceinline__ WRuns wruns_of(unsigned char *base, int cap, int N_P) {
  const size_t n = (size_t)2 * cap * N_P;
  WRuns w;
  w.w = reinterpret_cast<float4 *>(base);
  w.meta = reinterpret_cast<int *>(w.w + 2 * n);
  w.cap = cap;
  return w;
}

// |y| + |k1| h + |k2| h^2 + |k3| h^3 up to which a piece takes the power sums
// (a row's largest value is in [0.5, 1)): beyond it, at a knot interval much
// wider than its neighbours, the four terms cancel
constexpr float kPieceScale = 4.0f;
// knot intervals shorter than this are walked cell by cell: a cell's offset
// may leave [0, h] by the rounding of its phase there
constexpr float kShortKnot = 1.0e-4f;

// piece classes: 0 adds nothing, 1 power sums, 2 cell by cell; yn and tr are
// the value and the tangent at the right knot.  The Bernstein coefficients
// are the end values and the ends' tangent points y + k1 h / 3 and yn - tr h
// / 3.  One that is zero because the knot is dark and its tangent flat (what
// Akima's weights give next to a dark stretch, to rounding) bounds the curve
// at zero to rounding, so it does not make the piece a sign-changing one: most
// pieces at the edges of dark stretches are of that kind.
__device__ __forceinline__ int piece_class(const PieceDF &q, float yn, float tr, float h,
                                           bool add_all) {
  const float y = q.y.h, a1 = q.k1.h * h, a2 = q.k2.h * h * h, a3 = q.k3.h * h * h * h;
  const float scale = fabsf(y) + fabsf(a1) + fabsf(a2) + fabsf(a3);
  if (scale == 0.0f) return 0;
  if (!(scale <= kPieceScale) || h < kShortKnot) return 2;
  if (add_all) return 1;
  const float margin = 1.0e-5f * scale, flat = 1.0e-11f * scale, ar = tr * h;
  // -1, 0 or 1: a coefficient's sign; 2: too close to zero to tell
  auto sign = [&](float b, bool zero) {
    return zero ? 0 : (b > margin ? 1 : (b < -margin ? -1 : 2));
  };
  const int s0 = sign(y, y == 0.0f), s3 = sign(yn, yn == 0.0f);
  const int s1 = sign(y + a1 * (1.0f / 3.0f), y == 0.0f && fabsf(a1) <= flat);
  const int s2 = sign(yn - ar * (1.0f / 3.0f), yn == 0.0f && fabsf(ar) <= flat);
  const int lo = min(min(s0, s1), min(s2, s3)), hi = max(max(s0, s1), max(s2, s3));
  if (hi == 2) return 2;
  return lo >= 0 ? 1 : (hi <= 0 ? 0 : 2);
}

// the runs of signal phase k over cells [jb, je) of the parallel; returns
// the number of runs written, or -1 when a cell phase cannot be wrapped
// into the knot range (the reference's terminate)
template <typename CP, typename AR>
__device__ __forceinline__ int build_runs(const CP &cp, const AR &area, int jb, int je,
                                          const int32_t *rad, const WRuns &w, int half, int k) {
  int n = 0, cur = -1, j0 = 0, span = 0, hint = -1;
  const DF zero{0.0f, 0.0f};
  DF w0 = zero, w1 = zero, w2 = zero, w3 = zero;
  auto flush = [&]() {
    const size_t r = w.first(k, half) + n;
    w.w[2 * r] = make_float4(w0.h, w0.l, w1.h, w1.l);
    w.w[2 * r + 1] = make_float4(w2.h, w2.l, w3.h, w3.l);
    w.meta[r] = cur | (j0 << 10) | (span << 20);
    n++;
  };
  for (int j = jb; j < je; j++) {
    if (rad[j] != 1) continue;
    DF t;
    const int iv = cp(j, hint, t);
    if (iv < 0) return -1;
    hint = iv;
    if (iv != cur) {
      if (cur >= 0) flush();
      cur = iv;
      j0 = j;
      w0 = w1 = w2 = w3 = zero;
    }
    const DF A = area(j);
    const DF At = df_mul(A, t), At2 = df_mul(At, t), At3 = df_mul(At2, t);
    w0 = df_add(w0, A);
    w1 = df_add(w1, At);
    w2 = df_add(w2, At2);
    w3 = df_add(w3, At3);
    span = j - j0 + 1;
  }
  if (cur >= 0) flush();
  return n;
}

// the run's cells one by one (a piece whose sign changes on its interval)
template <typename CP, typename AR>
__device__ __forceinline__ DF run_cells(const CP &cp, const AR &area, const int32_t *rad, int iv,
                                        int j0, int span, const PieceDF &q, bool add_all, DF acc) {
  for (int j = j0; j < j0 + span; j++) {
    if (rad[j] != 1) continue;
    DF t;
    if (cp(j, iv, t) != iv) continue;
    const DF sv = df_fma(t, df_fma(t, df_fma(t, q.k3, q.k2), q.k1), q.y);
    if (add_all || sv.h > 0.0f) acc = df_fma(area(j), sv, acc);
  }
  return acc;
}

// the power of two above v >= 0 (the smallest normal number for v = 0), or
// twice it
__device__ __forceinline__ float lead_of(float v, bool twice) {
  return __int_as_float((__float_as_int(v) & 0x7f800000) + ((twice ? 2 : 1) << 23));
}

// s += a b, the rounding going to x: |s| exceeds the product, so d = t - s is
// exact and fma(a, b, -d) is what t lost
__device__ __forceinline__ void lead_acc(float a, float b, float &s, float &x) {
  const float t = __fmaf_rn(a, b, s);
  const float d = __fsub_rn(t, s);
  x = __fadd_rn(x, __fmaf_rn(a, b, -d));
  s = t;
}

// sum at signal phase k for energy slot e of the chunk, from the power sums
// of the parallel's runs; a group of EC lanes (a divisor of the warp) calls it
// with its own k, all groups of the warp together.  A run's four products are
// added to a lead, the power of two above the sum of their magnitudes (what
// some of them take away leaves it above the rest), so that each is added by
// one FMA whose error two more instructions recover exactly -- against the six
// of an error-free sum of unordered terms; their cross products and errors
// gather in x at the run's own magnitude, and the run's value joins the pair
// (s, c) by one error-free sum; taking the lead off is exact where the run's
// value is positive or, with values of either sign (add_all), the lead twice
// as large.  (A lead common to all runs saves nine
// instructions and loses two bits.)  flags[2 iv]: energies of interval iv that are
// not of class 1; flags[2 iv + 1]: those of them that add nothing; a run none
// of whose energies adds anything is dropped when it is staged.
// (n0, n1: the run counts of phase k's two halves; k2, m0, m1: the same of
// the group's next phase, whose first block is fetched while the last one of
// this phase is used)
struct RunFetch {
  float4 v[2];
  int mt = 0;
  // records b .. b + kStage - 1 of phase k: lane e of the group loads half a
  // record (EC = 8: two halves) and, the first kStage lanes, its int
  __device__ __forceinline__ void fetch(const WRuns &w, int k, int n0, int n1, int b, int e,
                                        int EC) {
    const int n = n0 + n1;
    const size_t f0 = w.first(k, 0), f1 = w.first(k, 1) - n0;
#pragma unroll
    for (int z = 0; z < 2; z++) {
      const int h = e + z * EC, i = b + (h >> 1);
      if (h < 2 * kStage && i < n && (z == 0 || EC < 2 * kStage))
        v[z] = w.w[2 * ((i < n0 ? f0 : f1) + i) + (h & 1)];
    }
    const int i = b + e;
    if (e < kStage && i < n) mt = w.meta[(i < n0 ? f0 : f1) + i];
  }
};
template <typename CP, typename AR>
__device__ __forceinline__ DF run_sum(const CP &cp, const AR &area, const int32_t *rad,
                                      const WRuns &w, int k, int n0, int n1, int k2, int m0,
                                      int m1, int EC, int ne, const PieceRows &pc,
                                      const uint32_t *flags, RunStage *stages, bool add_all,
                                      RunFetch &rf) {
  const int lane = threadIdx.x & 31, e = threadIdx.x % EC, sub = lane / EC;
  RunStage &st = stages[threadIdx.x / EC];
  const uint32_t lit = ne == 32 ? 0xffffffffu : ((1u << ne) - 1u);
  float s = 0.0f, c = 0.0f;
  DF walked{0.0f, 0.0f};
  const int n = n0 + n1;
  const int n_max = __reduce_max_sync(0xffffffffu, n);
  if (n_max == 0) rf.fetch(w, k2, m0, m1, 0, e, EC);
  for (int b = 0; b < n_max; b += kStage) {
    __syncwarp();  // the last block's readers are done
    bool alive = false;
    if (e < 2 * kStage) st.w[e] = rf.v[0];
    if (EC < 2 * kStage) st.w[e + EC] = rf.v[1];
    if (e < kStage && b + e < n) {
      const int iv = rf.mt & 1023;
      const uint2 fl = *reinterpret_cast<const uint2 *>(flags + 2 * iv);
      st.meta[e] = make_uint4((uint32_t)rf.mt, fl.x, fl.y, 0u);
      alive = (fl.x & fl.y & lit) != lit;
    }
    uint32_t todo = __ballot_sync(0xffffffffu, alive) >> (sub * EC);
    todo &= (1u << kStage) - 1u;
    __syncwarp();
    if (b + kStage < n_max) rf.fetch(w, k, n0, n1, b + kStage, e, EC);
    else rf.fetch(w, k2, m0, m1, 0, e, EC);
    // two runs at a time (the last may be the empty record): their chains are
    // independent, and the groups of the warp stay together
    while (__any_sync(0xffffffffu, todo != 0u)) {
      float h[2], x[2];
      uint32_t at[2];
      bool odd[2];
#pragma unroll
      for (int z = 0; z < 2; z++) {
        const int r = todo ? __ffs(todo) - 1 : kStage;
        todo &= todo - 1;
        const uint4 m = st.meta[r];
        const int iv = (int)(m.x & 1023u);
        const float4 p = pc.a[iv * pc.es + e], q = pc.b[iv * pc.es + e];
        const float4 A = st.w[2 * r], B = st.w[2 * r + 1];
        x[z] = __fmul_rn(p.x, A.y);
        x[z] = __fmaf_rn(p.y, A.x, x[z]);
        x[z] = __fmaf_rn(p.z, A.w, x[z]);
        x[z] = __fmaf_rn(p.w, A.z, x[z]);
        x[z] = __fmaf_rn(q.x, B.y, x[z]);
        x[z] = __fmaf_rn(q.y, B.x, x[z]);
        x[z] = __fmaf_rn(q.z, B.w, x[z]);
        x[z] = __fmaf_rn(q.w, B.z, x[z]);
        // (a power sum is negative where rounding put a cell's offset below
        // its knot)
        const float mag = __fmaf_rn(
            fabsf(q.z), fabsf(B.z),
            __fmaf_rn(fabsf(q.x), fabsf(B.x), __fmaf_rn(fabsf(p.z), fabsf(A.z),
                                                        __fmul_rn(fabsf(p.x), fabsf(A.x)))));
        const float lead = lead_of(mag, add_all);
        float v = lead;
        lead_acc(p.x, A.x, v, x[z]);
        lead_acc(p.z, A.z, v, x[z]);
        lead_acc(q.x, B.x, v, x[z]);
        lead_acc(q.z, B.z, v, x[z]);
        h[z] = __fsub_rn(v, lead);
        // (the empty record has no flag set)
        odd[z] = (m.y >> e) & 1u;
        at[z] = (m.z >> e) & 1u ? 0u : m.x;
      }
      // (after both, so that no branch parts their chains)
      if (__any_sync(0xffffffffu, odd[0] || odd[1])) {
#pragma unroll
        for (int z = 0; z < 2; z++) {
          if (!odd[z]) continue;
          h[z] = x[z] = 0.0f;
          if (at[z] == 0u) continue;  // adds nothing
          const int iv = (int)(at[z] & 1023u);
          walked = run_cells(cp, area, rad, iv, (int)((at[z] >> 10) & 1023u),
                             (int)((at[z] >> 20) & 1023u), pc.at(iv, e), add_all, walked);
        }
        __syncwarp();
      }
#pragma unroll
      for (int z = 0; z < 2; z++) {
        float t, err;
        two_sum(s, h[z], t, err);
        const DF sc = fast_two_sum(t, __fadd_rn(c, __fadd_rn(err, x[z])));
        s = sc.h;
        c = sc.l;
      }
    }
  }
  return df_add(df_norm(s, c), walked);
}

// ---------------------------------------------------------------------------
// beaming modification of the hot intensity I at energy E (the comoving
// energy the atmosphere sees) and emission cosine mu, hot_wrapper.pyx:153-199:
// 1: I (1 + abb E^cbb mu + bbb E^dbb mu^2); 2: the same with the analytical
// normalisation 0.5 / (0.5 + abb E^cbb / 3 + bbb E^dbb / 4); 3: normalised by
// the trapezoidal mu-integrals of I and of the modified I over nimu nodes
// mu = 1/nimu, 2/nimu, ... (the reference's accumulated sums), eval_mu(mu)
// giving the unmodified intensity there.  Negative results are 0.
// ---------------------------------------------------------------------------
template <typename EvalMu>
__device__ double beamed_intensity(int opt, const double *b, double E, double mu, double I_hot,
                                   const EvalMu &eval_mu) {
  const double fa = b[0] * pow(E, b[2]), fb = b[1] * pow(E, b[3]);
  double I = 0.0;
  if (opt == 1) {
    I = (1.0 + fa * mu + fb * (mu * mu)) * I_hot;
  } else if (opt == 2) {
    const double anorm = 0.5 / (0.5 + (1.0 / 3.0) * b[0] * pow(E, b[2]) +
                                (1.0 / 4.0) * b[1] * pow(E, b[3]));
    I = anorm * (1.0 + fa * mu + fb * (mu * mu)) * I_hot;
  } else if (opt == 3) {
    const double nimu = b[4];
    const long n = nimu > 0.0 ? (long)nimu : 0;
    double m = 0.0, nom = 0.0, den = 0.0;
    for (long k = 0; k < n; k++) {
      m = m + (1.0 / nimu);
      const double dmu = (k == 0 || (double)k == nimu - 1.0) ? (0.5 / nimu) : (1.0 / nimu);
      const double Ik = eval_mu(m);
      const double fk = 1.0 + fa * m + fb * (m * m);
      den = den + m * fk * Ik * dmu;
      nom = nom + m * Ik * dmu;
    }
    if (are_equal(den, 0.0)) I = 0.0;
    else I = (nom / den) * (1.0 + fa * mu + fb * (mu * mu)) * I_hot;
  } else {
    return I_hot;
  }
  return I < 0.0 ? 0.0 : I;
}

// Energy coordinates log10 E as 64-bit integers in units of 2^-54: the
// differences log10 E - log10 Z - log10 E_eff - node are exact, on the integer
// pipe (in FP64 each rounds at 2^-52 and takes the FP64 pipe seven
// instructions per column value, comparisons and conversions included).
constexpr double kFix = 18014398509481984.0;  // 2^54
__device__ __forceinline__ long long fix_of(double v) { return __double2ll_rn(v * kFix); }
// u / 2^54 as a float pair
__device__ __forceinline__ DF fix_df(long long u) {
  const int uh = (int)(u >> 32);
  if (uh >= (1 << 24) || uh < -(1 << 24)) return df_split((double)u * (1.0 / kFix));
  const unsigned ul = (unsigned)u;
  constexpr float s32 = 0x1p-22f, s16 = 0x1p-38f, s0 = 0x1p-54f;
  // three exact pieces; fast_two_sum's condition holds for the first two (the
  // high one is 0 or at least 2^-22)
  const DF a = fast_two_sum((float)uh * s32, (float)(ul >> 16) * s16);
  return fast_two_sum(a.h, __fadd_rn(a.l, (float)(ul & 0xffffu) * s0));
}
// the base node of the 4-point stencil around v on an ascending grid of n
// nodes, and lo the largest node index <= n - 2 at or below v (0 below the
// grid); lo < 0 on entry: unknown, else a walk from it
__device__ __forceinline__ int stencil_base_fix(const long long *g, int n, long long v, int &lo) {
  if (lo < 0) {
    lo = 0;
    int hi = n - 1;
    while (hi > lo + 1) {
      const int mid = (lo + hi) >> 1;
      if (g[mid] > v) hi = mid; else lo = mid;
    }
  } else {
    while (lo < n - 2 && g[lo + 1] <= v) lo++;
    while (lo > 0 && g[lo] > v) lo--;
  }
  return min(max(lo - 1, 0), n - 4);
}

// Num4D intensity of the FP64 form from a slab held as double-float pairs
// whose energy-node columns are scaled by 2^-xe: the reference's stencils,
// with the energy coordinate's offset u from the stencil's base node b3 exact
// and the Lagrange products and the 4 x 4 contraction in double-float
// arithmetic (~2^-48 relative, on the FP32 pipes).  Returns the stencil sum
// before the positive part (the caller clamps it at 0) as a double-float
// times 2^xr (xr the largest column exponent of the energy stencil).
struct EGrid {
  const DF *o, *s;  // offsets g[b + i] - g[b] (i = 1..3) and inverse Lagrange denominators
  const int *xe;
  int nE;
};
// the energy stencil's weights (scaled to the largest column exponent xr)
__device__ __forceinline__ void energy_weights(const EGrid &E, int b3, DF u0, DF (&w3)[4],
                                               int &xr) {
  const DF *o = E.o + 3 * b3;
  const DF u1 = df_sub(u0, o[0]), u2 = df_sub(u0, o[1]), u3 = df_sub(u0, o[2]);
  const DF u01 = df_mul(u0, u1), u23 = df_mul(u2, u3);
  const DF *S = E.s + 4 * b3;
  // the nodes' column scales relative to the largest of the four (<= 1)
  const int x0 = E.xe[b3], x1 = E.xe[b3 + 1], x2 = E.xe[b3 + 2], x3 = E.xe[b3 + 3];
  xr = max(max(x0, x1), max(x2, x3));
  w3[0] = df_scale(df_mul(df_mul(u1, u23), S[0]), x0 - xr);
  w3[1] = df_scale(df_mul(df_mul(u0, u23), S[1]), x1 - xr);
  w3[2] = df_scale(df_mul(df_mul(u01, u3), S[2]), x2 - xr);
  w3[3] = df_scale(df_mul(df_mul(u01, u2), S[3]), x3 - xr);
}
__device__ __forceinline__ DF eval_num4d_dfx(const EGrid &E, const DF *slab, int b2, const DF *w2,
                                             int b3, DF u0, int &xr) {
  DF w3[4];
  energy_weights(E, b3, u0, w3, xr);
  float sh = 0.0f, sl = 0.0f;
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const DF *r = slab + (size_t)(b2 + k) * E.nE + b3;
    float th = 0.0f, tl = 0.0f;
#pragma unroll
    for (int i = 0; i < 4; i++) df_acc_mul(w3[i], r[i], th, tl);
    df_acc_mul(w2[k], df_norm(th, tl), sh, sl);
  }
  return df_norm(sh, sl);
}

// The same along one profile column, whose mu stencil every energy shares: the
// four energy nodes of the stencil with the mu contraction done, kept from one
// energy to the next (the nodes move by one or none between neighbouring
// energies of a fine grid), so that an energy costs four products and four
// per new node instead of twenty.
struct NodeWindow {
  DF T[4];
  int at = -1;  // the base node T holds
  __device__ __forceinline__ static DF node(const EGrid &E, const DF *slab, const DF *w2, int n) {
    float h = 0.0f, l = 0.0f;
#pragma unroll
    for (int k = 0; k < 4; k++) df_acc_mul(w2[k], slab[(size_t)k * E.nE + n], h, l);
    return df_norm(h, l);
  }
  // slab: at the mu stencil's base row
  __device__ __forceinline__ DF eval(const EGrid &E, const DF *slab, const DF *w2, int b3, DF u0,
                                     int &xr) {
    if (at < 0 || b3 > at + 4 || b3 < at - 4) {
      at = b3;
#pragma unroll 1
      for (int i = 0; i < 4; i++) {
        T[0] = T[1]; T[1] = T[2]; T[2] = T[3];
        T[3] = node(E, slab, w2, b3 + i);
      }
    }
#pragma unroll 1
    while (at < b3) {
      at++;
      T[0] = T[1]; T[1] = T[2]; T[2] = T[3];
      T[3] = node(E, slab, w2, at + 3);
    }
#pragma unroll 1
    while (at > b3) {
      at--;
      T[3] = T[2]; T[2] = T[1]; T[1] = T[0];
      T[0] = node(E, slab, w2, at);
    }
    DF w3[4];
    energy_weights(E, b3, u0, w3, xr);
    float h = 0.0f, l = 0.0f;
#pragma unroll
    for (int i = 0; i < 4; i++) df_acc_mul(w3[i], T[i], h, l);
    return df_norm(h, l);
  }
};

// ---------------------------------------------------------------------------
// main integrator kernel
// ---------------------------------------------------------------------------
// shared memory of the integrator, in order (offsets for the launch, pointers
// in the kernel)
struct IntSmem {
  char *piece;  // the chunk's pieces; the leaf geometry's arrays where a CTA forms it itself
  double *Z, *abb, *geom;          // per profile column
  long long *lz;                   // log10 Z + log10 E_eff in units of 2^-54
  // the same in FP64: 2-D tables (log10 Z, or Z with E in electron rest
  // energies) and the mixed form
  double *lzd;
  DF *ih, *ih2;                    // 1 / h and 1 / h^2 of the phase intervals (FP64 form)
  DF *mw;                          // [4] mu stencil weights per column (FP64 form, 4-D table)
  float4 *mwf;                     // the same (mixed form)
  DF *cfm;                         // norm 10^(3 log T) GEOM as mantissa and exponent
  int *cfx, *mb, *flag;            // exponent; mu stencil base; kCol* bits
  float *fphase, *fphase_lo, *fh, *finvZ, *fgeom;
  double *gmu, *smu, *gE, *sE;     // grids and inverse Lagrange denominators
  long long *gEi;                  // energy grid in units of 2^-54
  DF *dgEo, *dsE;
  float *fgmu, *fgE, *fsmu, *fsE, *fgEo;
  int *xe;
  float *fcphi, *fcphi_lo, *fcarea, *fcarea_lo;
  long long *lgE;                  // the chunk's log10 E in units of 2^-54
  double *lgEd;                    // the same in FP64 (2-D tables: log10 E, or E)
  int *sc_exp;
  uint32_t *flags;
  int *nruns;
  float2 *phase;
  RunStage *stages;
  CellStage *cells;                // mixed form
  size_t bytes;
};
// the integrator's dynamic shared memory at most (with the statically
// allocated part, 227 KB): the form without runs takes every size that 200 KB
// held with the pieces in rows of EC and the ray table staged per CTA
constexpr size_t kIntSmemMax = 225 * 1024;
// float4 of either array of the FP64 form's pieces.  With runs an interval of
// zeros follows the last, and the arrays end on 128 bytes: with the second one
// and what follows 16 bytes off its banks, 24 vectors' kernel took 17.35 ms
// against 17.12.
__host__ __device__ inline size_t piece_array(int N_L, int EC, bool runs) {
  const size_t n = (size_t)(EC + 1) * N_L;
  return runs ? (n + (EC + 1) + 7) & ~size_t(7) : n;
}
template <bool kMixed>
__host__ __device__ inline IntSmem int_smem(char *base, int N_L, int N_P, int EC, int nmu, int nE,
                                            bool tab2, bool runs) {
  IntSmem o{};
  size_t at = 0;
  auto take = [&](auto *&p, size_t n) {
    using T = std::remove_reference_t<decltype(*p)>;
    at = (at + 15) & ~size_t(15);
    p = reinterpret_cast<T *>(base + at);
    at += n * sizeof(T);
  };
  const size_t pieces = kMixed ? (size_t)(EC + 1) * N_L * sizeof(PieceT<float>)
                               : 2 * piece_array(N_L, EC, runs) * sizeof(float4);
  const size_t geo = (size_t)N_L * 8 * sizeof(double) + (size_t)(4 * N_L + 8) * sizeof(int) + 64;
  take(o.piece, pieces > geo ? pieces : geo);
  take(o.Z, N_L); take(o.abb, N_L); take(o.geom, N_L);
  const bool tab4 = nE > 0 && !tab2;
  if (tab4) take(o.lz, N_L);
  if (tab2 || (tab4 && kMixed)) take(o.lzd, N_L);
  if (!kMixed) { take(o.ih, N_L); take(o.ih2, N_L); }
  if (tab4 && !kMixed) { take(o.mw, 4 * N_L); take(o.cfm, N_L); take(o.cfx, N_L); }
  if (tab4 && kMixed) take(o.mwf, N_L);
  if (tab4) take(o.mb, N_L);
  take(o.flag, N_L);
  take(o.fphase, N_L); take(o.fphase_lo, N_L);
  if (kMixed) { take(o.fh, N_L); take(o.finvZ, N_L); take(o.fgeom, N_L); }
  if (nE > 0) { take(o.gmu, nmu); take(o.smu, 4 * nmu); take(o.fgmu, nmu); }
  if (tab2) { take(o.gE, nE); take(o.sE, 4 * nE); take(o.fgE, nE); }
  if (tab4) take(o.gEi, nE);
  if (tab4 && !kMixed) { take(o.dgEo, 3 * nE); take(o.dsE, 4 * nE); take(o.xe, nE); }
  if (tab4 && kMixed) {
    take(o.fsmu, 4 * nmu); take(o.fsE, 4 * nE); take(o.fgEo, 3 * nE); take(o.gE, nE);
  }
  take(o.fcphi, kMaxCellsF); take(o.fcphi_lo, kMaxCellsF);
  take(o.fcarea, kMaxCellsF); take(o.fcarea_lo, kMaxCellsF);
  if (tab4) take(o.lgE, EC);
  if (tab2 || (tab4 && kMixed)) take(o.lgEd, EC);
  take(o.sc_exp, EC);
  if (N_P <= kMaxPhases) take(o.phase, N_P);
  if (!kMixed) take(o.flags, 2 * N_L);
  if (kMixed) take(o.cells, 1);
  if (runs) { take(o.nruns, 2 * N_P); take(o.stages, kThreads / EC); }
  o.bytes = (at + 15) & ~size_t(15);
  return o;
}

// a parallel's atmosphere constants, formed by one warp
struct RowAtm {
  double vec0, vec1, kT, kT_c, p3, lgE_eff, wT[4], wg[4];
  int bT, bg;
};

// One CTA takes items (a chunk of consecutive parallels of one mesh, and one
// of n_eg groups of its energy chunks) from a shared counter.  Bound: FP32
// issue and the FP64 pipe about equally, two CTAs of 8 warps per SM (pieces and
// grids fill half an SM's shared memory).  What FP64 is left per parallel is
// the table contraction over the reachable energy nodes and, per image, the mu
// stencils and 1 / h of the knots; energy coordinates are integers, and values
// change between double and float pair on the integer pipe.  24 vectors at
// sqrt_num_cells 96 (two Num4D regions, 128 leaves, 128 energies): 30 ms with
// those in FP64 and the geometry formed here, 16.0 ms now; 100 blackbody spots
// (64 leaves, 64 energies): 4.7 ms, 1.9 ms now.
// WT = double: the plain FP64 drop-in.  WT = float: the mixed-precision form
// (geometry, visibility and knots in FP64; atmosphere, Akima pieces and the
// cell x phase sums in FP32; per-chunk partials in FP64).
template <typename WT>
__global__ void __launch_bounds__(kThreads, 2) integrate_kernel(IntegrateArgs a) {
  constexpr bool kMixed = std::is_same<WT, float>::value;
  extern __shared__ __align__(16) char smem[];
  const int N_L = a.N_L, N_E = a.N_E, N_P = a.N_P, EC = a.EC;
  const int nmu = a.atmos.I ? a.atmos.nmu : 0, nEt = a.atmos.I ? a.atmos.nE : 0;
  // 2-D tables (atmos.I is [nmu][nE], no 10^(3 log T)): atm 4, Pol_Num2D's
  // I on (mu, log10 E') (hot_Num2D.pyx:187-400); atm 6, a split atmosphere
  // reduced once per call to (mu, E) with E' in electron rest energies
  // (integrator_for_azimuthal_invariance_split.pyx:270-275,457-476)
  const bool tab2 = a.table2d && !kMixed;
  // power-sum form (FP64 path with scratch)
  const bool use_w = !kMixed && a.wsum != nullptr;
  const IntSmem sm = int_smem<kMixed>(smem, N_L, N_P, EC, nmu, nEt, a.table2d != 0, use_w);
  PieceT<WT> *co4 = reinterpret_cast<PieceT<WT> *>(sm.piece);  // mixed form
  const PieceRows pr{reinterpret_cast<float4 *>(sm.piece),
                     reinterpret_cast<float4 *>(sm.piece) + piece_array(N_L, EC, use_w),
                     EC + 1};
  __shared__ RowAtm s_ra;
  __shared__ RowCtx s_row;
  __shared__ int s_item, s_jalt, s_state[3], s_win[2];
  __shared__ float s_erange[2];
  // a beaming modification's (abb, bbb, cbb, dbb, nimu) for the parallel
  __shared__ double s_beam[5];
  const WRuns wr = use_w ? wruns_of(a.wsum + (size_t)blockIdx.x *
                                                 integrate_wsum_bytes_dev(N_P, a.w_cap),
                                    a.w_cap, N_P)
                         : WRuns{};
  double *slab = a.slab ? a.slab + (size_t)blockIdx.x * nmu * nEt : nullptr;
  float *slabf = reinterpret_cast<float *>(slab);
  const DF *slabd = reinterpret_cast<const DF *>(slab);
  AtmSmem as{};  // the FP64 stencil functions' view of the grids
  if (nEt > 0) {
    as.gmu = sm.gmu; as.smu = sm.smu; as.fgmu = sm.fgmu;
    as.gE = sm.gE; as.sE = sm.sE; as.fgE = sm.fgE;
    const double *mu = a.atmos.mu, *lE = a.atmos.logE;
    for (int t = threadIdx.x; t < nmu; t += blockDim.x) {
      sm.gmu[t] = mu[t];
      sm.fgmu[t] = (float)mu[t];
      if (t <= nmu - 4) {
        double s4[4];
        lagrange_space(mu, t, s4);
        for (int q = 0; q < 4; q++) {
          sm.smu[4 * t + q] = s4[q];
          if (kMixed) sm.fsmu[4 * t + q] = (float)s4[q];
        }
      }
    }
    for (int t = threadIdx.x; t < nEt; t += blockDim.x) {
      double s4[4] = {0.0, 0.0, 0.0, 0.0};
      if (t <= nEt - 4) lagrange_space(lE, t, s4);
      if (a.table2d) {
        sm.gE[t] = lE[t];
        sm.fgE[t] = (float)lE[t];
        for (int q = 0; q < 4; q++) sm.sE[4 * t + q] = s4[q];
      } else {
        sm.gEi[t] = fix_of(lE[t]);
        if (kMixed) sm.gE[t] = lE[t];
        for (int q = 0; q < 4; q++) {
          if (kMixed) sm.fsE[4 * t + q] = (float)s4[q];
          else sm.dsE[4 * t + q] = df_split(s4[q]);
        }
        for (int q = 0; q < 3; q++) {
          const double o = t + q + 1 < nEt ? lE[t + q + 1] - lE[t] : 0.0;
          if (kMixed) sm.fgEo[3 * t + q] = (float)o;
          else sm.dgEo[3 * t + q] = df_split(o);
        }
      }
    }
  }
  const EGrid eg4{sm.dgEo, sm.dsE, sm.xe, nEt};
  if (sm.phase)
    for (int t = threadIdx.x; t < N_P; t += blockDim.x) {
      const DF v = df_split(a.phases[t]);
      sm.phase[t] = make_float2(v.h, v.l);
    }
  if (use_w) {
    // (the geometry formed in the pieces' place ends before interval N_L of
    // either array: 80 N_L + 48 bytes against 144 N_L or more)
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int t = threadIdx.x; t <= EC; t += blockDim.x)
      pr.a[N_L * (EC + 1) + t] = pr.b[N_L * (EC + 1) + t] = zero;
    for (int t = threadIdx.x; t < kThreads / EC; t += blockDim.x) {
      sm.stages[t].w[2 * kStage] = sm.stages[t].w[2 * kStage + 1] = zero;
      sm.stages[t].meta[kStage] = make_uint4((uint32_t)N_L, 0u, 0u, 0u);
    }
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int n_iv = N_L - 1, strips = (n_iv + kStrip - 1) / kStrip;
  // energy chunks of equal size, at most EC energies each
  const int nec = (N_E + EC - 1) / EC, ec = (N_E + nec - 1) / nec;
  // a thread's profile columns and its share of their energies: with N_L
  // columns or fewer than threads a column belongs to `parts` threads
  const int parts = max(1, kThreads / N_L);
  const int part0 = N_L <= kThreads ? threadIdx.x / N_L : 0;
  const int col0 = N_L <= kThreads ? (part0 < parts ? (int)threadIdx.x - part0 * N_L : N_L)
                                   : threadIdx.x;
  const double mu_max = nEt ? a.atmos.mu[nmu - 1] : 0.0;
  const double mu_top3 = nEt ? a.atmos.mu[nmu - 3] : 0.0;
  const bool corr = !kMixed && a.correction != nullptr;
  constexpr float tp = (float)kTwoPi;
  const int n_items = *a.chunk_count * a.n_eg;

  for (;;) {
    __syncthreads();
    if (threadIdx.x == 0) s_item = atomicAdd(a.item_next, 1);
    __syncthreads();
    const int item = s_item;
    if (item >= n_items) break;
    const int chunk = a.chunk_order[item / a.n_eg], eg = item % a.n_eg;
    const int ec_lo = (int)((long long)nec * eg / a.n_eg);
    const int ec_hi = (int)((long long)nec * (eg + 1) / a.n_eg);
    const int e_lo = ec_lo * ec, e_hi = min(N_E, ec_hi * ec);
    const int64_t r0 = a.chunk_r0[chunk], r1 = a.chunk_r1[chunk];
    const int m = a.row_member[r0];
    const MemberDesc M = a.members[m];
    const bool erest = (M.atm == 6);
    const bool num4d = (M.atm == 2) || tab2;
    const bool t4 = num4d && !tab2;
    const double norm = num4d ? kErg / kHKeV : kErg * kPlanck;
    // the plain Num4D columns without beaming or correction keep their
    // intensities as double-float mantissas with exponents up to the row
    // scaling (uniform over the CTA: a chunk is one mesh's rows)
    const bool dfy = !kMixed && t4 && M.beam_opt == 0 && !corr;
    double *part = a.partial + (size_t)chunk * N_E * N_P;
    // partials [N_P][N_E] in either form: the sums' lanes are energies
    for (int t = threadIdx.x; t < N_P * (e_hi - e_lo); t += blockDim.x) {
      const int k = t / (e_hi - e_lo), e = e_lo + t - k * (e_hi - e_lo);
      part[(size_t)k * N_E + e] = 0.0;
    }
    if (t4 && warp == 0) {  // the item's range of log10 E
      float lo = INFINITY, hi = -INFINITY;
      for (int p = e_lo + lane; p < e_hi; p += 32) {
        lo = fminf(lo, (float)a.lgE[p]);
        hi = fmaxf(hi, (float)a.lgE[p]);
      }
      for (int o = 16; o > 0; o >>= 1) {
        lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
        hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
      }
      if (lane == 0) { s_erange[0] = lo; s_erange[1] = hi; }
    }
    // algorithmic FLOPs per (parallel, image), the cost model of the
    // likelihood path: leaf work N_L (60 + N_E f_atm) and spline work
    // N_E (30 N_L + C N_P 14), f_atm 12 (blackbody) or 1350 (4-D table)
    double flops = 0.0;
    const double f_atm = num4d ? 1350.0 : 12.0;

    for (int64_t row = r0; row < r1; row++) {
      const RowInfo ri = a.row_info[row];
      const int images = ri.images & ~kImgTerm;
      const int i = (int)(row - M.row_off);
      const double *cellA = a.cellArea + M.cell_off + (int64_t)i * M.S1;
      const double *cellPhi = a.phi + M.cell_off + (int64_t)i * M.S1;
      const int32_t *rad = a.radiates + M.cell_off + (int64_t)i * M.S1;
      if (images > 0) {
        __syncthreads();  // the last parallel's readers are done
        if (warp == 0) {
          const int64_t cell = M.cell_off + (int64_t)i * M.S1 + ri.cell;
          const double *vec = a.params + cell * a.n_params;
          const double v0 = vec[0], v1 = vec[1];
          double vT = v0, vg = v1;
          if (t4) {
            if (vT < a.atmos.logT[0]) vT = a.atmos.logT[0];
            if (vT > a.atmos.logT[a.atmos.nT - 1]) vT = a.atmos.logT[a.atmos.nT - 1];
            if (vg < a.atmos.logg[0]) vg = a.atmos.logg[0];
            if (vg > a.atmos.logg[a.atmos.ng - 1]) vg = a.atmos.logg[a.atmos.ng - 1];
          }
          // lane by lane the same instructions: the powers 10^(log T), 10^(3
          // log T), the elsewhere's; the T and g stencils
          const double pw = pow(10.0, lane == 0 ? v0
                                      : lane == 1 ? 3.0 * vT
                                      : (corr ? a.correction[cell * a.n_correction] : 0.0));
          const double kT = (kKB / kKeV) * __shfl_sync(0xffffffffu, pw, 0);
          const double p3 = __shfl_sync(0xffffffffu, pw, 1);
          const double kT_c = (kKB / kKeV) * __shfl_sync(0xffffffffu, pw, 2);
          if (t4 && lane < 2) {
            const double *P = lane ? a.atmos.logg : a.atmos.logT;
            const int n = lane ? a.atmos.ng : a.atmos.nT;
            const double x = lane ? vg : vT;
            const int b = stencil_base(P, n, x);
            double w[4];
            lagrange4(P, b, x, w);
            for (int q = 0; q < 4; q++) (lane ? s_ra.wg : s_ra.wT)[q] = w[q];
            if (lane) s_ra.bg = b; else s_ra.bT = b;
          }
          if (lane == 0) {
            s_ra.vec0 = v0;
            s_ra.vec1 = v1;
            s_ra.kT = kT;
            s_ra.kT_c = corr ? kT_c : 0.0;
            s_ra.p3 = t4 ? p3 : 1.0;
            s_ra.lgE_eff = t4 ? log10(kT) : 0.0;
            s_state[0] = num4d ? (int)a.row_entry_top[row] : 0;
            s_state[1] = s_state[2] = 0;
            // parameters 2-6 of the parallel's first radiating cell
            if (M.beam_opt > 0)
              for (int b = 0; b < 5; b++) s_beam[b] = vec[2 + b];
            if (t4) {
              // the energy nodes any of the item's columns can reach: from the
              // range of log10 E and of the lit columns' Z, with slack well
              // above the floats' rounding
              const float l = (float)s_ra.lgE_eff;
              const float vlo = s_erange[0] - log10f(ri.z_hi) - l - 1.0e-3f;
              const float vhi = s_erange[1] - log10f(ri.z_lo) - l + 1.0e-3f;
              int lo0 = -1, lo1 = -1;
              const int b0 = stencil_base_fix(sm.gEi, nEt, fix_of((double)vlo), lo0);
              const int b1 = stencil_base_fix(sm.gEi, nEt, fix_of((double)vhi), lo1);
              s_win[0] = b0;
              s_win[1] = b1 + 4;
            }
          }
        } else if (M.S1 <= kMaxCellsF) {
          // cell azimuths and areas as float pairs
          for (int t = threadIdx.x - 32; t < M.S1; t += blockDim.x - 32) {
            const DF p = df_split_bits(cellPhi[t], 0), ar = df_split_bits(cellA[t], 0);
            sm.fcphi[t] = p.h;
            sm.fcphi_lo[t] = p.l;
            sm.fcarea[t] = ar.h;
            sm.fcarea_lo[t] = ar.l;
          }
        }
        __syncthreads();
      }
      const double p3 = s_ra.p3, kT = s_ra.kT, kT_c = s_ra.kT_c;
      const float kT_f = (float)kT, p3f = (float)p3;
      // mixed form: the FP32 roundings of the constant factors norm and
      // 10^(3 log T) are undone exactly on the parallel's FP64 partials
      const double fix = !kMixed ? 1.0
                         : num4d ? (norm * p3) / ((double)(float)norm * (double)p3f)
                                 : norm / (double)(float)norm;
      if (images > 0 && t4) {
        // contract the (log T, log g) stencil of this parallel once over the
        // reachable energy nodes:
        // slab[mu][logE] = sum_ij w_T[i] w_g[j] table[bT+i][bg+j][mu][logE]
        const int n0 = s_win[0], wn = s_win[1] - n0, nw = nmu * wn;
        double wT[4], wg[4];
#pragma unroll
        for (int q = 0; q < 4; q++) { wT[q] = s_ra.wT[q]; wg[q] = s_ra.wg[q]; }
        const size_t S1t = (size_t)nmu * nEt, S0t = (size_t)a.atmos.ng * S1t;
        const size_t base = s_ra.bT * S0t + s_ra.bg * S1t;
        if (kMixed && a.atmos.I32 != nullptr) {
          // FP32 contraction from the FP32 copy of the table
          float wTf[4], wgf[4];
#pragma unroll
          for (int q = 0; q < 4; q++) { wTf[q] = (float)wT[q]; wgf[q] = (float)wg[q]; }
          for (int w = threadIdx.x; w < nw; w += blockDim.x) {
            const int mu_i = w / wn, t = mu_i * nEt + n0 + (w - mu_i * wn);
            float r = 0.0f;
#pragma unroll
            for (int ii = 0; ii < 4; ii++) {
              const float *q = a.atmos.I32 + base + ii * S0t + t;
              float u = wgf[0] * __ldg(q) + wgf[1] * __ldg(q + S1t) + wgf[2] * __ldg(q + 2 * S1t) +
                        wgf[3] * __ldg(q + 3 * S1t);
              r += wTf[ii] * u;
            }
            slabf[t] = r;
          }
        } else {
          if (!kMixed) {
            for (int e = threadIdx.x; e < wn; e += blockDim.x) sm.xe[n0 + e] = kZeroExp;
            __syncthreads();
          }
          for (int w = threadIdx.x; w < nw; w += blockDim.x) {
            const int mu_i = w / wn, e = n0 + (w - mu_i * wn), t = mu_i * nEt + e;
            double r = 0.0;
#pragma unroll
            for (int ii = 0; ii < 4; ii++) {
              const double *q = a.atmos.I + base + ii * S0t + t;
              double u = wg[0] * __ldg(q) + wg[1] * __ldg(q + S1t) + wg[2] * __ldg(q + 2 * S1t) +
                         wg[3] * __ldg(q + 3 * S1t);
              r += wT[ii] * u;
            }
            if (kMixed) {
              slabf[t] = (float)r;
            } else {
              slab[t] = r;
              atomicMax(&sm.xe[e], binary_exponent(r));
            }
          }
          if (!kMixed) {
            // the FP64 form keeps the slab as double-float pairs, each energy
            // node's column (all mu) scaled by 2^-xe[e] (exact), xe the binary
            // exponent of its largest value, so that the pairs keep full
            // relative precision across the table's exponential tail
            __syncthreads();
            DF *o = reinterpret_cast<DF *>(slab);
            for (int w = threadIdx.x; w < nw; w += blockDim.x) {
              const int mu_i = w / wn, e = n0 + (w - mu_i * wn), t = mu_i * nEt + e;
              o[t] = df_split_bits(slab[t], -sm.xe[e]);
            }
          }
        }
        __syncthreads();
      }
      for (int I = 0; I < images; I++) {
        const double *rec;
        if (ri.geo >= 0) {
          rec = a.geo + (ri.geo + I) * image_doubles(N_L);
        } else {
          // no room was left for the parallel's records: form the image here
          double *own = a.geo + (a.geo_cap + blockIdx.x) * image_doubles(N_L);
          double *coef;
          GeoSmem g = carve(sm.piece, N_L, 0, &coef, 0, 0, nullptr, 32, 0);
          RowCtx c;
          load_row(a, M, row, i, c, &s_row);
          if (threadIdx.x == 0) s_jalt = c.N_R - 1;
          __syncthreads();
          for (int t = threadIdx.x; t < c.N_R - 1; t += blockDim.x)
            if (!at_most(c.D[t], kHalfPi)) atomicMin(&s_jalt, t);
          __syncthreads();
          c.jalt = s_jalt;
          c.alt_xmin = cos(c.D[c.jalt]);
          image_record(c, I, N_L, a.leaves, g, num4d, mu_top3, mu_max, s_state, nullptr, own);
          rec = own;
        }
        const uint8_t *rfl = reinterpret_cast<const uint8_t *>(rec + 4 * (size_t)N_L);
        // (the parallel's entry state was not known to the pre-pass; a record
        // formed here has it)
        const bool entry_top = num4d && ri.geo >= 0 && a.row_entry_top[row] != 0;
        for (int t = threadIdx.x; t < N_L; t += blockDim.x) {
          unsigned f = rfl[t];
          if (entry_top && (f & kColFirst)) f &= ~kColClamp;
          sm.flag[t] = (int)f;
          const double ph = rec[t];
          const DF pd = df_split_bits(ph, 0);
          sm.fphase[t] = pd.h;
          sm.fphase_lo[t] = pd.l;
          if (t < N_L - 1) {
            const double h = rec[t + 1] - ph;
            if (kMixed) {
              sm.fh[t] = (float)h;
            } else {
              const double r = 1.0 / h;
              sm.ih[t] = df_split_bits(r, 0);
              sm.ih2[t] = df_split_bits(1.0 / (h * h), 0);
            }
          }
          if (f & kColLit) {
            const double Z = rec[N_L + t], abb = rec[2 * N_L + t], geom = rec[3 * N_L + t];
            sm.Z[t] = Z;
            sm.abb[t] = abb;
            sm.geom[t] = geom;
            if (kMixed) {
              sm.finvZ[t] = (float)(1.0 / Z);
              sm.fgeom[t] = (float)geom;
            }
            if (tab2) sm.lzd[t] = erest ? Z : log10(Z);
            if (t4) {
              const double lz = log10(Z) + s_ra.lgE_eff;
              sm.lz[t] = fix_of(lz);
              if constexpr (kMixed) {
                sm.lzd[t] = lz;
                const float v = fmaxf((float)abb, sm.fgmu[0]);
                const int b = stencil_base_f(sm.fgmu, nmu, v);
                float w[4];
                lagrange_wf(sm.fgmu, sm.fsmu, b, v, w);
                sm.mb[t] = b;
                sm.mwf[t] = make_float4(w[0], w[1], w[2], w[3]);
              } else {
                const MuStencil ms = mu_stencil(a.atmos, as, abb, false);
                sm.mb[t] = ms.b2;
#pragma unroll
                for (int q = 0; q < 4; q++) sm.mw[4 * t + q] = df_split_bits(ms.w2[q], 0);
                const double cf = norm * p3 * geom;
                MaxExponent mx;
                mx.fold(cf);
                const int x = mx.exponent();
                sm.cfx[t] = x;
                sm.cfm[t] = df_split_bits(cf, -x);
              }
            }
          }
        }
        __syncthreads();
        auto cell_phase = [&](auto cached, int k) {
          float2 ph;
          if (sm.phase) {
            ph = sm.phase[k];
          } else {
            // (on the integer pipe: the compiler evaluates both sides)
            const DF v = df_split_bits(a.phases[k], 0);
            ph = make_float2(v.h, v.l);
          }
          return CellPhaseF<decltype(cached)::value>{
              sm.fphase, sm.fphase_lo, N_L, sm.fphase[0], sm.fphase[N_L - 1], ph.x, ph.y, tp,
              (float)(kTwoPi - (double)tp), sm.fcphi, sm.fcphi_lo, cellPhi};
        };
        if (use_w) {
          // the runs of every signal phase, each half of the cells by its own
          // thread (energy independent: formed once per parallel and image)
          const int hc = (M.S1 + 1) / 2;
          const AreaDF<true> ar{sm.fcarea, sm.fcarea_lo, cellA};
          for (int t = threadIdx.x; t < 2 * N_P; t += blockDim.x) {
            const int k = t % N_P, half = t / N_P;
            const CellPhaseF<true> cp = cell_phase(std::true_type{}, k);
            const int n =
                build_runs(cp, ar, half * hc, min(M.S1, (half + 1) * hc), rad, wr, half, k);
            // no cell of the parallel is added at this phase where one cannot
            // be wrapped (either half's failure voids both, as in the per-cell
            // form)
            if (n < 0) atomicExch(&a.member_status[m], (int)kPulseFail);
            sm.nruns[half * N_P + k] = n;
          }
        }
        if (threadIdx.x == 0 && a.flop_counter && eg == 0) {
          int Cr = 0;
          for (int j = 0; j < M.S1; j++) Cr += (rad[j] == 1);
          flops += (double)N_L * (60.0 + N_E * f_atm) +
                   (double)N_E * (30.0 * N_L + (double)Cr * N_P * 14.0);
        }

        for (int e0 = e_lo; e0 < e_hi; e0 += ec) {
          const int ne = min(ec, e_hi - e0);
          if (num4d) {
            for (int t = threadIdx.x; t < ne; t += blockDim.x) {
              if (tab2) sm.lgEd[t] = erest ? a.energies[e0 + t] : a.lgE[e0 + t];
              else sm.lgE[t] = fix_of(a.lgE[e0 + t]);
              if (kMixed) sm.lgEd[t] = a.lgE[e0 + t];
            }
          }
          __syncthreads();
          // specific intensities of every profile column (:445-478): a thread
          // takes one column and its part of the chunk's energies, so the
          // energy stencil moves by a node or two from one to the next
          const int per = (ne + parts - 1) / parts, pl0 = part0 * per, pl1 = min(ne, pl0 + per);
          for (int col = col0; col < N_L; col += kThreads) {
            const int f = sm.flag[col];
            int lo = -1;
            MuStencil ms{};
            NodeWindow nodes;
            if (tab2 && (f & kColLit)) ms = mu_stencil(a.atmos, as, sm.abb[col], false);
            for (int pl = pl0; pl < pl1; pl++) {
              const int p = e0 + pl;
              if (!(f & kColLit)) {
                if constexpr (kMixed) co4[col * (EC + 1) + pl].y = 0.0f;
                else if (dfy) pr.y(col, pl) = DF{0.0f, 0.0f};
                else pr.yd(col, pl) = 0.0;
                continue;
              }
              // a leaf's first energy may see the clamped mu; with beaming
              // option 3 every call is followed by calls up to mu = 1, so no
              // out-of-table mu is ever clamped
              const bool clamp = p == 0 && (f & kColClamp) && M.beam_opt != 3;
              int b3 = 0;
              DF u{0.0f, 0.0f};
              if (t4) {
                const long long v0 = sm.lgE[pl] - sm.lz[col];
                long long v = max(v0, sm.gEi[0]);
                v = min(v, sm.gEi[nEt - 1]);
                b3 = stencil_base_fix(sm.gEi, nEt, v, lo);
                if (kMixed) {
                  // (the FP32 rounding of the offset sees its FP64 value)
                  const double vd = v == v0 ? sm.lgEd[pl] - sm.lzd[col]
                                            : sm.gE[v0 < v ? 0 : nEt - 1];
                  u.h = (float)(vd - sm.gE[b3]);
                } else {
                  u = fix_df(v - sm.gEi[b3]);
                }
              }
              if constexpr (kMixed) {
                float I_E;
                if (t4) {
                  int b2 = sm.mb[col];
                  float4 w2 = sm.mwf[col];
                  if (clamp) {
                    const float v = fminf((float)sm.abb[col], sm.fgmu[nmu - 1]);
                    b2 = stencil_base_f(sm.fgmu, nmu, v);
                    float w[4];
                    lagrange_wf(sm.fgmu, sm.fsmu, b2, v, w);
                    w2 = make_float4(w[0], w[1], w[2], w[3]);
                  }
                  I_E = eval_num4d_f(sm.fgEo, sm.fsE, nEt, slabf, b2, w2, b3, u.h, p3f);
                } else {
                  I_E = eval_bb_f((float)a.energies[p] * sm.finvZ[col], kT_f);
                }
                co4[col * (EC + 1) + pl].y = (float)norm * I_E * sm.fgeom[col];
              } else {
                double I_E;
                if (t4) {
                  int xr;
                  DF I;
                  if (clamp) {
                    const MuStencil mc = mu_stencil(a.atmos, as, sm.abb[col], true);
                    DF w2[4];
#pragma unroll
                    for (int q = 0; q < 4; q++) w2[q] = df_split(mc.w2[q]);
                    I = eval_num4d_dfx(eg4, slabd, mc.b2, w2, b3, u, xr);
                  } else {
                    I = nodes.eval(eg4, slabd + (size_t)sm.mb[col] * nEt, sm.mw + 4 * col, b3, u,
                                   xr);
                  }
                  if (I.h < 0.0f) I = DF{0.0f, 0.0f};
                  if (dfy) {
                    // y = I 2^xr col_factor kept as a double-float mantissa
                    // and an exponent (no round trip through FP64)
                    pr.y(col, pl) = df_mul(I, sm.cfm[col]);
                    pr.ex(col, pl) = xr + sm.cfx[col];
                    continue;
                  }
                  I_E = df_value(I) * pow2_double(xr) * p3;
                } else if (num4d) {
                  // atm 6: E' = E / Z in electron rest energies (:457-458)
                  const double v3 = erest ? (sm.lgEd[pl] / sm.lzd[col]) * 0.001956951
                                          : sm.lgEd[pl] - sm.lzd[col];
                  I_E = eval_num4d_e(a.atmos, as, a.atmos.I,
                                     clamp ? mu_stencil(a.atmos, as, sm.abb[col], true) : ms, v3,
                                     p3);
                } else {
                  I_E = eval_bb(a.energies[p] / sm.Z[col], kT);
                  // the burst blackbody's limb darkening (hot_BB_burst.pyx)
                  if (M.atm == 3) I_E = I_E * (0.421 + 0.868 * sm.abb[col]);
                }
                const double I_c =
                    corr ? eval_bb(a.energies[p] / sm.Z[col], kT_c) * (kErg * kPlanck) : 0.0;
                // with a beaming modification the raw intensity is kept
                // here and modified in the pass below
                pr.yd(col, pl) = M.beam_opt > 0 ? I_E : (I_E * norm - I_c) * sm.geom[col];
              }
            }
            if (!kMixed && M.beam_opt > 0 && (f & kColLit)) {
              // the beaming modification (hot_wrapper.pyx:153-199) of the
              // column's intensities
              int lb = -1;
              for (int pl = pl0; pl < pl1; pl++) {
                const int p = e0 + pl;
                const double I_raw = pr.yd(col, pl);
                double I_E;
                if (num4d) {
                  int b3 = 0;
                  DF u{0.0f, 0.0f};
                  double v3 = 0.0;
                  if (t4) {
                    long long v = sm.lgE[pl] - sm.lz[col];
                    v = max(v, sm.gEi[0]);
                    v = min(v, sm.gEi[nEt - 1]);
                    b3 = stencil_base_fix(sm.gEi, nEt, v, lb);
                    u = fix_df(v - sm.gEi[b3]);
                  } else {
                    v3 = erest ? (sm.lgEd[pl] / sm.lzd[col]) * 0.001956951
                               : sm.lgEd[pl] - sm.lzd[col];
                  }
                  const double Ep = erest ? v3 : a.energies[p] / sm.Z[col];
                  I_E = beamed_intensity(M.beam_opt, s_beam, Ep, sm.abb[col], I_raw,
                                         [&](double mu_k) {
                    const MuStencil mk = mu_stencil(a.atmos, as, mu_k, false);
                    if (tab2) return eval_num4d_e(a.atmos, as, a.atmos.I, mk, v3, p3);
                    DF w2[4];
#pragma unroll
                    for (int q = 0; q < 4; q++) w2[q] = df_split(mk.w2[q]);
                    int xr;
                    const DF I = eval_num4d_dfx(eg4, slabd, mk.b2, w2, b3, u, xr);
                    return I.h < 0.0f ? 0.0 : df_value(I) * pow2_double(xr) * p3;
                  });
                } else {
                  const double Ep = a.energies[p] / sm.Z[col];
                  const double I0 = eval_bb(Ep, kT);  // the blackbody has no mu dependence
                  I_E = beamed_intensity(M.beam_opt, s_beam, Ep, sm.abb[col], I_raw,
                                         [&](double) { return I0; });
                }
                const double I_c =
                    corr ? eval_bb(a.energies[p] / sm.Z[col], kT_c) * (kErg * kPlanck) : 0.0;
                pr.yd(col, pl) = (I_E * norm - I_c) * sm.geom[col];
              }
            }
          }
          __syncthreads();
          // Akima-periodic piece coefficients (:566-569): a thread builds kStrip
          // consecutive pieces of one energy row from a sliding window of the
          // five chords each piece needs, so each chord is formed once per
          // strip instead of five times
          if constexpr (kMixed) {
            for (int t = threadIdx.x; t < EC * strips; t += blockDim.x) {
              const int pl = t % EC, i0 = (t / EC) * kStrip;
              const int i1 = min(i0 + kStrip, n_iv);
              if (pl >= ne) continue;
              PieceT<WT> *yr = co4 + pl;
              const int es = EC + 1;
              auto chord = [&](int j) -> WT {
                const int q = periodic_chord(j, N_L);
                // knot spacings from the FP64 knots: adjacent knots closer
                // than an FP32 ulp stay distinct
                return (yr[(q + 1) * es].y - yr[q * es].y) / sm.fh[q];
              };
              WT m0 = chord(i0 - 2), m1 = chord(i0 - 1), m2 = chord(i0), m3 = chord(i0 + 1),
                 m4 = chord(i0 + 2);
              for (int iv = i0; iv < i1; iv++) {
                if (iv > i0) {
                  m0 = m1; m1 = m2; m2 = m3; m3 = m4;
                  m4 = chord(iv + 2);
                }
                WT k1, k2, k3;
                akima_piece(m0, m1, m2, m3, m4, (WT)sm.fh[iv], k1, k2, k3);
                PieceT<WT> *o = yr + iv * es;
                o->k1 = k1;
                o->k2 = k2;
                o->k3 = k3;
              }
            }
            __syncthreads();
          } else {
            // scale each energy row by a power of two (exact) so that its
            // largest profile value lies in [0.5, 1): double-float values then
            // keep the row's full relative precision whatever its magnitude
            for (int pl = warp; pl < ne; pl += kThreads / 32) {
              MaxExponent mx;
              for (int col = lane; col < N_L; col += 32) {
                if (dfy) {
                  // values m 2^x: the exponent from the bits
                  const float h = pr.y(col, pl).h;
                  if (h != 0.0f && h == h) {
                    if (isinf(h)) mx.inf = true;
                    else mx.e = max(mx.e, pr.ex(col, pl) + float_exponent(h));
                  }
                } else {
                  mx.fold(pr.yd(col, pl));
                }
              }
              mx.merge_warp();
              if (lane == 0) sm.sc_exp[pl] = mx.exponent();
            }
            __syncthreads();
            for (int t = threadIdx.x; t < EC * N_L; t += blockDim.x) {
              const int col = t / EC, pl = t - col * EC;
              if (pl >= ne) continue;
              if (dfy) {  // the value times 2^(x - the row's) in float arithmetic (exact)
                const DF mv = pr.y(col, pl);
                pr.y(col, pl) = mv.h == 0.0f
                                    ? DF{0.0f, 0.0f}
                                    : df_times_pow2(mv, pr.ex(col, pl) - sm.sc_exp[pl]);
              } else {
                pr.y(col, pl) = df_split_bits(pr.yd(col, pl), -sm.sc_exp[pl]);
              }
            }
            __syncthreads();
            // a group of EC lanes takes a strip, a lane an energy; the classes
            // of a piece's energies are gathered by ballot
            const int sub = lane / EC;
            for (int t = threadIdx.x; t < ((EC * strips + 31) & ~31); t += blockDim.x) {
              const int pl = t % EC, i0 = (t / EC) * kStrip;
              const int i1 = min(i0 + kStrip, n_iv);
              const bool on = pl < ne;
              auto chord = [&](int j) -> DF {
                const int q = periodic_chord(j, N_L);
                return df_mul(df_sub(pr.y(q + 1, pl), pr.y(q, pl)), sm.ih[q]);
              };
              DF m0{}, m1{}, m2{}, m3{}, m4{};
              if (on && i0 < i1) {
                m0 = chord(i0 - 2); m1 = chord(i0 - 1); m2 = chord(i0); m3 = chord(i0 + 1);
                m4 = chord(i0 + 2);
              }
              for (int z = 0; z < kStrip; z++) {
                const int iv = i0 + z;
                const bool here = on && iv < i1;
                int cls = 1;
                if (here) {
                  if (z > 0) {
                    m0 = m1; m1 = m2; m2 = m3; m3 = m4;
                    m4 = chord(iv + 2);
                  }
                  DF k1, k2, k3, tr;
                  akima_piece_df(m0, m1, m2, m3, m4, sm.ih[iv], sm.ih2[iv], k1, k2, k3, tr);
                  pr.put_k(iv, pl, k1, k2, k3);
                  const float h = (sm.fphase[iv + 1] - sm.fphase[iv]) +
                                  (sm.fphase_lo[iv + 1] - sm.fphase_lo[iv]);
                  cls = piece_class(PieceDF{pr.y(iv, pl), k1, k2, k3}, pr.y(iv + 1, pl).h, tr.h,
                                    h, corr);
                }
                const uint32_t odd = __ballot_sync(0xffffffffu, cls != 1);
                const uint32_t none = __ballot_sync(0xffffffffu, cls == 0);
                if (pl == 0 && iv < i1) {
                  const uint32_t mask = EC == 32 ? 0xffffffffu : ((1u << EC) - 1u);
                  sm.flags[2 * iv] = (odd >> (sub * EC)) & mask;
                  sm.flags[2 * iv + 1] = (none >> (sub * EC)) & mask;
                }
              }
            }
            __syncthreads();
          }
          // cell x phase accumulation (:571-598).  Power sums: a group of EC
          // lanes takes a signal phase, a lane an energy.  Per-cell form: a
          // thread takes a signal phase and kEPT energies.
          if (use_w) {
            const int e = threadIdx.x % EC, grp = threadIdx.x / EC, step = kThreads / EC;
            const AreaDF<true> ar{sm.fcarea, sm.fcarea_lo, cellA};
            RunFetch rf;
            auto counts = [&](int k, int &n0, int &n1) {
              n0 = n1 = 0;
              if (k < N_P) {
                n0 = sm.nruns[k];
                n1 = sm.nruns[N_P + k];
                if (n0 < 0 || n1 < 0) n0 = n1 = 0;
              }
            };
            int n0, n1;
            counts(grp, n0, n1);
            rf.fetch(wr, grp, n0, n1, 0, e, EC);
            for (int k0 = 0; k0 < N_P; k0 += step) {
              const int k = k0 + grp, kc = min(k, N_P - 1);
              const bool mine = e < ne && k < N_P;
              // partials [N_P][N_E]: the lanes' energies are adjacent
              double *dst = part + (size_t)kc * N_E + e0 + e;
              const double before = mine ? *dst : 0.0;
              int m0, m1;
              counts(k + step, m0, m1);
              const DF v = run_sum(cell_phase(std::true_type{}, kc), ar, rad, wr, kc, n0, n1,
                                   k + step, m0, m1, EC, ne, pr, sm.flags, sm.stages, corr, rf);
              if (mine) *dst = before + df_join_bits(v, sm.sc_exp[e]);
              n0 = m0;
              n1 = m1;
            }
          } else if constexpr (kMixed) {
            const int e = threadIdx.x % kCellLanes, grp = threadIdx.x / kCellLanes;
            auto sums = [&](auto cached, auto per_lane) {
              constexpr int Z = decltype(per_lane)::value;
              const AreaF<decltype(cached)::value> ar{sm.fcarea, cellA};
              for (int k0 = 0; k0 < N_P; k0 += kThreads / kCellLanes) {
                const int k = k0 + grp, kc = min(k, N_P - 1);
                double *dst = part + (size_t)kc * N_E + e0 + e;
                bool bad;
                float v[Z];
                cell_phase_sums_f<Z>(cell_phase(cached, kc), ar, M.S1, rad,
                                     reinterpret_cast<const float4 *>(co4), EC + 1, *sm.cells,
                                     bad, v);
                if (bad) {
                  atomicExch(&a.member_status[m], (int)kPulseFail);
                } else if (k < N_P) {
#pragma unroll
                  for (int z = 0; z < Z; z++)
                    if (e + kCellLanes * z < ne) dst[kCellLanes * z] += (double)v[z] * fix;
                }
              }
            };
            auto by_cells = [&](auto per_lane) {
              if (M.S1 <= kMaxCellsF) sums(std::true_type{}, per_lane);
              else sums(std::false_type{}, per_lane);
            };
            if (EC == 32) by_cells(std::integral_constant<int, 4>{});
            else if (EC == 16) by_cells(std::integral_constant<int, 2>{});
            else by_cells(std::integral_constant<int, 1>{});
          } else {
            const int ntasks = N_P * (EC / kEPT);
            auto sums = [&](auto cached) {
              constexpr bool kCached = decltype(cached)::value;
              for (int task = threadIdx.x; task < ntasks; task += blockDim.x) {
                const int k = task % N_P, grp = task / N_P;
                const int pb = grp * kEPT;
                if (pb >= ne) continue;
                const CellPhaseF<kCached> cp = cell_phase(cached, k);
                DF acc[kEPT];
#pragma unroll
                for (int e = 0; e < kEPT; e++) acc[e] = DF{0.0f, 0.0f};
                const AreaDF<kCached> ar{sm.fcarea, sm.fcarea_lo, cellA};
                if (!cell_phase_sums_df(cp, ar, M.S1, rad, pr, pb, corr, acc)) {
                  atomicExch(&a.member_status[m], (int)kPulseFail);
                  continue;
                }
#pragma unroll
                for (int e = 0; e < kEPT; e++)
                  if (pb + e < ne)
                    part[(size_t)k * N_E + e0 + pb + e] +=
                        scale_pow2(df_value(acc[e]), sm.sc_exp[pb + e]);
              }
            };
            if (M.S1 <= kMaxCellsF) sums(std::true_type{});
            else sums(std::false_type{});
          }
          __syncthreads();
        }
      }
      if (ri.images & kImgTerm) {
        // the reference terminates here: nothing after it in the chunk is added
        if (threadIdx.x == 0) atomicExch(&a.member_status[m], (int)kPulseFail);
        break;
      }
    }
    if (threadIdx.x == 0 && a.flop_counter && flops > 0.0) atomicAdd(a.flop_counter, flops);
  }
}

// ---------------------------------------------------------------------------
// Stokes I, Q, U (integratorIQU_for_azimuthal_invariance.pyx:68-743) for the
// blackbody (Q = 0) and burst blackbody (hot_BB_burst.pyx) atmospheres: one
// CTA per parallel and group of its energy chunks (gridDim.y of them).  Per chunk of energies the I, Q and U profiles of the
// leaves are scaled, splined (Akima periodic) and summed over cells x phases
// in double-float exactly as the FP64 integrator does for I; Q and U are
// added wherever I is (:646-650).
// ---------------------------------------------------------------------------
constexpr int kStokesPiece = 3 * (int)sizeof(PieceDF);

template <typename CP, typename AR>
__device__ __forceinline__ bool cell_phase_sums_stokes(const CP &cp, const AR &area, int S1,
                                                       const int32_t *rad, const PieceDF *pI,
                                                       const PieceDF *pQ, const PieceDF *pU,
                                                       int N_L, int pb, int ne, bool add_all,
                                                       DF (&aI)[kEPT], DF (&aQ)[kEPT],
                                                       DF (&aU)[kEPT]) {
  int hint = -1;
  for (int j = 0; j < S1; j++) {
    if (rad[j] != 1) continue;
    DF t;
    const int iv = cp(j, hint, t);
    if (iv < 0) return false;
    hint = iv;
    const DF A = area(j);
#pragma unroll
    for (int e = 0; e < kEPT; e++) {
      if (pb + e < ne) {
        const int o = (pb + e) * N_L + iv;
        const PieceDF q = pI[o];
        const DF sv = df_fma(t, df_fma(t, df_fma(t, q.k3, q.k2), q.k1), q.y);
        if (sv.h > 0.0f || add_all) {
          aI[e] = df_fma(A, sv, aI[e]);
          const PieceDF qq = pQ[o], qu = pU[o];
          aQ[e] = df_fma(A, df_fma(t, df_fma(t, df_fma(t, qq.k3, qq.k2), qq.k1), qq.y), aQ[e]);
          aU[e] = df_fma(A, df_fma(t, df_fma(t, df_fma(t, qu.k3, qu.k2), qu.k1), qu.y), aU[e]);
        }
      }
    }
  }
  return true;
}

size_t stokes_smem(int N_L, int N_P, int N_E, int N_R, int nmu, int nE) {
  const Layout L = make_layout(N_L, N_P, N_E, nmu, nE, kStokesPiece, N_R);
  return L.bytes + (size_t)2 * N_L * sizeof(double) + (size_t)2 * L.EC * sizeof(int) + 64;
}

__global__ void __launch_bounds__(kThreads, 1) stokes_kernel(IntegrateArgs a) {
  extern __shared__ __align__(16) char smem[];
  const int64_t row = blockIdx.x;
  const int m = a.row_member[row];
  const MemberDesc M = a.members[m];
  const int i = (int)(row - M.row_off);
  const int N_L = a.N_L, N_E = a.N_E, N_P = a.N_P;
  const int leaf_lim = (N_L % 2 == 0) ? N_L / 2 : (N_L + 1) / 2;
  // 2-D table atmospheres: atm 4 (Pol_Num2D, I and Q on (mu, log10 E'),
  // hot_Num2D.pyx:187-400) and atm 6 (split I and Q reduced to (mu, E), E'
  // in electron rest energies,
  // integratorIQU_for_azimuthal_invariance_split.pyx:310-322,515-530)
  const bool tab2 = (M.atm == 4 || M.atm == 6);
  const bool erest = (M.atm == 6);
  const int nmu = a.atmos.I ? a.atmos.nmu : 0, nEt = a.atmos.I ? a.atmos.nE : 0;
  const Layout L = make_layout(N_L, N_P, N_E, nmu, nEt, kStokesPiece, a.N_R);
  const int EC = L.EC;
  double *coef;
  AtmSmem as{};
  GeoSmem g = carve(smem, N_L, EC, &coef, nmu, nEt, &as, kStokesPiece, a.N_R);
  double *xd = reinterpret_cast<double *>(
      (reinterpret_cast<uintptr_t>(g.sc_exp + EC) + 15) & ~uintptr_t(15));
  g.c2chi = xd;
  g.s2chi = xd + N_L;
  int *scQ = reinterpret_cast<int *>(xd + 2 * N_L), *scU = scQ + EC;
  Piece *coI = reinterpret_cast<Piece *>(coef);
  Piece *coQ = coI + (size_t)EC * N_L, *coU = coQ + (size_t)EC * N_L;
  __shared__ int s_jalt, s_top, s_any;
  __shared__ RowCtx s_row;
  double *part = a.partial + (size_t)row * 3 * N_E * N_P;
  RowCtx c;
  if (!load_row(a, M, row, i, c, &s_row)) return;
  stage_deflection(c, g, &s_jalt);
  if (tab2) stage_table_grids(a.atmos, as, nmu, nEt);
  if (threadIdx.x == 0) {
    s_top = tab2 ? (int)a.row_entry_top[row] : 0;
    s_any = 0;
  }
  __syncthreads();
  const double mu_max = tab2 ? a.atmos.mu[nmu - 1] : 0.0;
  const double mu_top3 = tab2 ? a.atmos.mu[nmu - 3] : 0.0;
  const bool burst = (M.atm == 3);
  // hot_BB_burst.pyx, hot_Num2D.pyx:359-367, hot_Num5D_split.pyx:538-563
  const double norm = tab2 ? kErg / kHKeV : kErg * kPlanck;
  const double kT = (kKB / kKeV) * pow(10.0, c.vec0);
  const bool corr = a.correction != nullptr;
  const double kT_c =
      corr ? (kKB / kKeV) *
                 pow(10.0, a.correction[(M.cell_off + (int64_t)i * M.S1 + c.J) * a.n_correction])
           : 0.0;
  const double *cellA = a.cellArea + M.cell_off + (int64_t)i * M.S1;
  const double *cellPhi = a.phi + M.cell_off + (int64_t)i * M.S1;
  const int32_t *rad = a.radiates + M.cell_off + (int64_t)i * M.S1;
  const int n_iv = N_L - 1, strips = (n_iv + kStrip - 1) / kStrip;
  for (int I = 0; I < c.IO; I++) {
    for (int k = threadIdx.x; k < leaf_lim; k += blockDim.x)
      leaf_geometry(c, I, k, N_L, leaf_lim, a.leaves, g);
    __syncthreads();
    if (threadIdx.x == 0) {
      int top = s_top, any = s_any;
      state_machine(N_L, leaf_lim, a.leaves, g, tab2, mu_top3, mu_max, top, any);
      s_top = top;
      s_any = any;
    }
    __syncthreads();
    if (g.flags[0]) {
      if (threadIdx.x == 0) atomicExch(&a.member_status[m], (int)kPulseFail);
      return;
    }
    if (g.flags[1]) break;
    for (int t = threadIdx.x; t < N_L; t += blockDim.x) {
      const float hi = (float)g.phase[t];
      as.fphase[t] = hi;
      as.fphase_lo[t] = (float)(g.phase[t] - (double)hi);
    }
    if (M.S1 <= kMaxCellsF) {
      for (int t = threadIdx.x; t < M.S1; t += blockDim.x) {
        const float hi = (float)cellPhi[t];
        as.fcphi[t] = hi;
        as.fcphi_lo[t] = (float)(cellPhi[t] - (double)hi);
        const float ah = (float)cellA[t];
        as.fcarea[t] = ah;
        as.fcarea_lo[t] = (float)(cellA[t] - (double)ah);
      }
    }
    for (int t = threadIdx.x; t < N_L - 1; t += blockDim.x) {
      const double h = g.phase[t + 1] - g.phase[t];
      g.ih[t] = df_split(1.0 / h);
      g.ih2[t] = df_split(1.0 / (h * h));
    }
    if (tab2) {
      for (int t = threadIdx.x; t < N_L; t += blockDim.x) {
        const int sidx = g.src[t];
        if (sidx >= 0) g.lzs[sidx] = erest ? g.Z[sidx] : log10(g.Z[sidx]);
      }
    }
    __syncthreads();
    const int nec = (N_E + EC - 1) / EC;
    const int e_lo = EC * (int)(nec * blockIdx.y / gridDim.y);
    const int e_hi = min(N_E, EC * (int)(nec * (blockIdx.y + 1) / gridDim.y));
    for (int e0 = e_lo; e0 < e_hi; e0 += EC) {
      const int ne = min(EC, e_hi - e0);
      if (tab2) {
        for (int t = threadIdx.x; t < ne; t += blockDim.x)
          g.lgE[t] = erest ? a.energies[e0 + t] : log10(a.energies[e0 + t]);
        __syncthreads();
      }
      // I, Q cos 2chi and Q sin 2chi of every profile column (:468-497)
      int mu_col = -1;
      MuStencil ms{};
      for (int t = threadIdx.x; t < ne * N_L; t += blockDim.x) {
        const int pl = t / N_L, col = t - pl * N_L;
        const int p = e0 + pl;
        const int s = g.src[col];
        double yI = 0.0, yQ = 0.0, yU = 0.0;
        if (s >= 0) {
          const double Ep = a.energies[p] / g.Z[s];
          const double abb = g.ABB[s];
          double I_E, Q_E = 0.0;
          if (tab2) {
            // the walk's mu clamp applies to a leaf's first energy only
            const double v3 = erest ? (g.lgE[pl] / g.lzs[s]) * 0.001956951
                                    : g.lgE[pl] - g.lzs[s];
            MuStencil m1;
            if (p == 0 && g.clamp0[s]) {
              m1 = mu_stencil(a.atmos, as, abb, true);
            } else {
              if (s != mu_col) {
                ms = mu_stencil(a.atmos, as, abb, false);
                mu_col = s;
              }
              m1 = ms;
            }
            I_E = eval_num4d_e(a.atmos, as, a.atmos.I, m1, v3, 1.0);
            if (a.table_q) Q_E = eval_table_raw(a.atmos, as, a.table_q, m1, v3);
          } else {
            I_E = eval_bb(Ep, kT);
            if (burst) {
              I_E = I_E * (0.421 + 0.868 * abb);
              Q_E = (0.1171 * (abb - 1.) / (1. + 3.582 * abb)) * I_E;
            }
          }
          const double I_c = corr ? eval_bb(Ep, kT_c) * (kErg * kPlanck) : 0.0;
          yI = (I_E * norm - I_c) * g.GEOM[s];
          yQ = ((Q_E * g.c2chi[s]) * norm) * g.GEOM[s];
          yU = ((Q_E * g.s2chi[s]) * norm) * g.GEOM[s];
        }
        coI[pl * N_L + col].y = yI;
        coQ[pl * N_L + col].y = yQ;
        coU[pl * N_L + col].y = yU;
      }
      __syncthreads();
      // an exact power-of-two scale per (component, energy row)
      const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
      for (int r = warp; r < 3 * ne; r += kThreads / 32) {
        const int comp = r / ne, pl = r - comp * ne;
        const Piece *co = comp == 0 ? coI : (comp == 1 ? coQ : coU);
        double mx = 0.0;
        for (int col = lane; col < N_L; col += 32) mx = fmax(mx, fabs(co[pl * N_L + col].y));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        int ex = 0;
        if (mx > 0.0 && mx <= 1.7976931348623157e308) frexp(mx, &ex);
        if (lane == 0) (comp == 0 ? g.sc_exp : (comp == 1 ? scQ : scU))[pl] = ex;
      }
      __syncthreads();
      for (int t = threadIdx.x; t < 3 * ne * N_L; t += blockDim.x) {
        const int comp = t / (ne * N_L), u = t - comp * ne * N_L;
        Piece *co = comp == 0 ? coI : (comp == 1 ? coQ : coU);
        const int *sc = comp == 0 ? g.sc_exp : (comp == 1 ? scQ : scU);
        const double v = co[u].y;
        reinterpret_cast<PieceDF *>(co)[u].y = df_split(ldexp(v, -sc[u / N_L]));
      }
      __syncthreads();
      for (int t = threadIdx.x; t < 3 * ne * strips; t += blockDim.x) {
        const int comp = t / (ne * strips), u = t - comp * ne * strips;
        const int pl = u / strips, i0 = (u - pl * strips) * kStrip;
        const int i1 = min(i0 + kStrip, n_iv);
        PieceDF *yr = reinterpret_cast<PieceDF *>(comp == 0 ? coI : (comp == 1 ? coQ : coU)) +
                      pl * N_L;
        auto chord = [&](int j) -> DF {
          const int q = periodic_chord(j, N_L);
          return df_mul(df_sub(yr[q + 1].y, yr[q].y), g.ih[q]);
        };
        DF m0 = chord(i0 - 2), m1 = chord(i0 - 1), m2 = chord(i0), m3 = chord(i0 + 1),
           m4 = chord(i0 + 2);
        for (int iv = i0; iv < i1; iv++) {
          if (iv > i0) {
            m0 = m1; m1 = m2; m2 = m3; m3 = m4;
            m4 = chord(iv + 2);
          }
          DF k1, k2, k3;
          akima_piece_df(m0, m1, m2, m3, m4, g.ih[iv], g.ih2[iv], k1, k2, k3);
          yr[iv].k1 = k1;
          yr[iv].k2 = k2;
          yr[iv].k3 = k3;
        }
      }
      __syncthreads();
      // cell x phase accumulation (:612-650)
      const int ntasks = N_P * ((ne + kEPT - 1) / kEPT);
      for (int task = threadIdx.x; task < ntasks; task += blockDim.x) {
        const int k = task % N_P, pb = (task / N_P) * kEPT;
        const double phd = a.phases[k];
        const float ph = (float)phd;
        const float tp = (float)kTwoPi;
        DF aI[kEPT], aQ[kEPT], aU[kEPT];
#pragma unroll
        for (int e = 0; e < kEPT; e++) aI[e] = aQ[e] = aU[e] = DF{0.0f, 0.0f};
        auto sums = [&](auto cached) {
          constexpr bool kCached = decltype(cached)::value;
          const CellPhaseF<kCached> cp{as.fphase, as.fphase_lo, N_L, as.fphase[0],
                                       as.fphase[N_L - 1], ph, (float)(phd - (double)ph), tp,
                                       (float)(kTwoPi - (double)tp), as.fcphi, as.fcphi_lo,
                                       cellPhi};
          const AreaDF<kCached> ar{as.fcarea, as.fcarea_lo, cellA};
          return cell_phase_sums_stokes(cp, ar, M.S1, rad, reinterpret_cast<const PieceDF *>(coI),
                                        reinterpret_cast<const PieceDF *>(coQ),
                                        reinterpret_cast<const PieceDF *>(coU), N_L, pb, ne, corr,
                                        aI, aQ, aU);
        };
        if (!(M.S1 <= kMaxCellsF ? sums(std::true_type{}) : sums(std::false_type{}))) {
          atomicExch(&a.member_status[m], (int)kPulseFail);
          continue;
        }
#pragma unroll
        for (int e = 0; e < kEPT; e++) {
          if (pb + e < ne) {
            const int p = e0 + pb + e;
            part[(size_t)p * N_P + k] += ldexp(df_value(aI[e]), g.sc_exp[pb + e]);
            part[(size_t)(N_E + p) * N_P + k] += ldexp(df_value(aQ[e]), scQ[pb + e]);
            part[(size_t)(2 * N_E + p) * N_P + k] += ldexp(df_value(aU[e]), scU[pb + e]);
          }
        }
      }
      __syncthreads();
    }
  }
}

// the parallels' Stokes partials of each member in order, / (E keV) (:715-725)
__global__ void reduce_stokes_kernel(IntegrateArgs a) {
  const int m = blockIdx.y, comp = blockIdx.z;
  const MemberDesc M = a.members[m];
  const int n = a.N_E * a.N_P;
  double *out = comp == 0 ? a.flux : (comp == 1 ? a.flux_q : a.flux_u);
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
    double s = 0.0;
    for (int r = 0; r < M.S0; r++)
      s += a.partial[((size_t)(M.row_off + r) * 3 + comp) * n + t];
    const int p = t / a.N_P;
    out[M.flux_off + t] = s / (a.energies[p] * kKeV);
  }
}

// ---------------------------------------------------------------------------
// The split atmosphere's (mu, E) table at the first cell's (t_e, t_bb, tau)
// (integrator_for_azimuthal_invariance_split.pyx:270-275 calls
// hot_Num5D_split.pyx:267-481 once per (mu, E) node, mu outer, from a fresh
// evaluator).  The cached walk's state at each call is known in closed form:
// on t_e, t_bb, tau the first call moves the base node from 0 (clamping a
// query beyond the top of the grid on that call only) and later calls leave
// it; a query on the node mu_k or E_k has base node min(max(k - 2, 0), n - 4).
// On those two dimensions only the weight of the node itself is nonzero, so
// the 64 remaining terms are summed in the reference's order with its
// products (numerators, then inverse denominators, multiplied dimension by
// dimension) and without contraction, which reproduces its rounding.  One
// thread per (mu, E) node.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void walk_factors(const double *P, int b, double x, double D[4],
                                             double S[4]) {
  D[0] = x - P[b + 1]; D[0] *= x - P[b + 2]; D[0] *= x - P[b + 3];
  D[1] = x - P[b];     D[1] *= x - P[b + 2]; D[1] *= x - P[b + 3];
  D[2] = x - P[b];     D[2] *= x - P[b + 1]; D[2] *= x - P[b + 3];
  D[3] = x - P[b];     D[3] *= x - P[b + 1]; D[3] *= x - P[b + 2];
  S[0] = 1.0 / (P[b] - P[b + 1]);     S[0] /= P[b] - P[b + 2];     S[0] /= P[b] - P[b + 3];
  S[1] = 1.0 / (P[b + 1] - P[b]);     S[1] /= P[b + 1] - P[b + 2]; S[1] /= P[b + 1] - P[b + 3];
  S[2] = 1.0 / (P[b + 2] - P[b]);     S[2] /= P[b + 2] - P[b + 1]; S[2] /= P[b + 2] - P[b + 3];
  S[3] = 1.0 / (P[b + 3] - P[b]);     S[3] /= P[b + 3] - P[b + 1]; S[3] /= P[b + 3] - P[b + 2];
}

__global__ void split_reduce_kernel(SplitArgs a) {
  const int n3 = a.n[3], n4 = a.n[4];
  // the first call's walk on t_e, t_bb, tau from base node 0
  __shared__ int b[3];
  __shared__ double vfirst[3];
  if (threadIdx.x < 3) {
    const int d = threadIdx.x, n = a.n[d];
    const double *P = a.grid[d];
    double v = a.vec[d];
    int bn = 0;
    if (v > P[2] && n != 4) {
      for (int it = 0; it < n && v > P[bn + 2]; it++) {
        if (bn < n - 4) {
          bn++;
        } else {
          if (v >= P[n - 1]) v = P[n - 1];
          break;
        }
      }
    }
    b[d] = bn;
    vfirst[d] = v;
  }
  __syncthreads();
  const size_t s3 = (size_t)n4, s2 = (size_t)n3 * n4, s1 = (size_t)a.n[2] * s2,
               s0 = (size_t)a.n[1] * s1;
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n3 * n4; t += gridDim.x * blockDim.x) {
    const int i = t / n4, j = t - i * n4;
    double D[3][4], S[3][4];
#pragma unroll
    for (int d = 0; d < 3; d++) walk_factors(a.grid[d], b[d], t == 0 ? vfirst[d] : a.vec[d], D[d], S[d]);
    const int b3 = min(max(i - 2, 0), n3 - 4), b4 = min(max(j - 2, 0), n4 - 4);
    double D3[4], S3[4], D4[4], S4[4];
    walk_factors(a.grid[3], b3, a.grid[3][i], D3, S3);
    walk_factors(a.grid[4], b4, a.grid[4][j], D4, S4);
    const double d3 = D3[i - b3], sp3 = S3[i - b3], d4 = D4[j - b4], sp4 = S4[j - b4];
    const double *T = a.I + (size_t)i * s3 + j;
    double I = 0.0;
    for (int k0 = 0; k0 < 4; k0++)
      for (int k1 = 0; k1 < 4; k1++)
        for (int k2 = 0; k2 < 4; k2++) {
          double dp = D[0][k0];
          dp = __dmul_rn(dp, D[1][k1]); dp = __dmul_rn(dp, D[2][k2]);
          dp = __dmul_rn(dp, d3); dp = __dmul_rn(dp, d4);
          double sp = S[0][k0];
          sp = __dmul_rn(sp, S[1][k1]); sp = __dmul_rn(sp, S[2][k2]);
          sp = __dmul_rn(sp, sp3); sp = __dmul_rn(sp, sp4);
          const double v = T[(size_t)(b[0] + k0) * s0 + (size_t)(b[1] + k1) * s1 +
                             (size_t)(b[2] + k2) * s2];
          I = __dadd_rn(I, __dmul_rn(__dmul_rn(dp, sp), v));
        }
    a.out[t] = I;
  }
}

// ---------------------------------------------------------------------------
// Work plan.  A parallel's cost is dominated by its images: each image
// repeats the profile columns, the splines and the cell x phase sums, and a
// star near the photon sphere (R -> 1.5 r_s) has rays deflected by several
// pi, so its parallels carry up to ~8 images against the usual 1-2.  The
// image count per parallel, ceil(max deflection / pi) (or the mesh's image
// order limit), is known only after the ray tables are built on the device,
// so the chunks are planned there:
//   cost(parallel) = images x (kCostImage + radiating cells) + kCostRow
// in units of one radiating cell's sums over one image (the fixed per-image
// work -- columns, splines, leaf geometry -- measured at about 28 cells, the
// per-parallel slab contraction at about 6), or 1 for a parallel with no
// radiating cell.  The consecutive parallels of each mesh are cut greedily
// into chunks of about total / target_chunks (a chunk closes before the
// parallel that would take it past the target), which bounds the count by
// 2 target_chunks + members.  The CTAs take the chunks heaviest first
// (a counting sort on floor(log2 cost)), so the few heavy chunks start in
// the first wave instead of forming the tail.  Chunk boundaries depend only
// on the costs, so every result is independent of the order in which the
// CTAs run.
// ---------------------------------------------------------------------------
constexpr float kCostImage = 28.0f;
constexpr float kCostRow = 6.0f;

__global__ void row_cost_kernel(IntegrateArgs a) {
  const int lane = threadIdx.x & 31;
  const int64_t row = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (blockIdx.x == 0 && threadIdx.x == 0) {  // the call's counters
    *a.item_next = 0;
    *a.geo_count = 0;
  }
  if (row >= a.n_rows) return;
  const MemberDesc M = a.members[a.row_member[row]];
  const int64_t i = row - M.row_off;
  const int32_t *rad = a.radiates + M.cell_off + i * M.S1;
  int cr = 0;
  for (int j = lane; j < M.S1; j += 32) cr += (rad[j] == 1);
  for (int o = 16; o > 0; o >>= 1) cr += __shfl_xor_sync(0xffffffffu, cr, o);
  if (lane == 0) {
    float c = 1.0f;
    if (cr > 0) {
      const double md = a.maxDeflection[row];
      int io = M.image_order_limit > 0 ? M.image_order_limit
                                       : (md > 0.0 ? (int)ceil(md / kPi) : 1);
      io = max(1, min(io, 64));
      c = (float)io * (kCostImage + (float)cr) + kCostRow;
    }
    a.row_cost[row] = c;
  }
}

// ordered reduction of the chunk partials and the 1/(E keV) factor (:605-612)
__global__ void reduce_flux_kernel(IntegrateArgs a) {
  const int m = blockIdx.y;
  const MemberDesc M = a.members[m];
  const int n = a.N_E * a.N_P;
  const int c0 = a.chunk_first[m], c1 = a.chunk_first[m + 1];
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
    double s = 0.0;
    for (int c = c0; c < c1; c++) s += a.partial[(size_t)c * n + t];
    const int p = t % a.N_E, k = t / a.N_E;  // partials are [N_P][N_E]
    a.flux[M.flux_off + (int64_t)p * a.N_P + k] = s / (a.energies[p] * kKeV);
  }
}

}  // namespace

// the geometry pre-pass and, for a table atmosphere, each parallel's entry
// state of the mu walk: a scan of the parallels in call order
template <bool kPlan>
static void launch_geometry(const IntegrateArgs &a, cudaStream_t st) {
  const size_t smem = geometry_bytes(a.N_L, a.N_R);
  // (the attribute is per device: set on every launch, which is cheap)
  cudaFuncSetAttribute(geometry_kernel<kPlan>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       200 * 1024);
  const unsigned grid = (unsigned)(a.n_rows + (kPlan ? 1 : 0));
  geometry_kernel<kPlan><<<grid, kPlanThreads, smem, st>>>(a);
  if (a.atmos.I != nullptr) num4d_scan_kernel<<<(a.n_members + 127) / 128, 128, 0, st>>>(a);
}

size_t integrate_wsum_bytes(int N_P, int max_cells, int *w_cap) {
  const int cap = (max_cells + 1) / 2;
  if (w_cap) *w_cap = cap;
  return integrate_wsum_bytes_dev(N_P, cap);
}

bool integrate_runs_fit(int N_L, int N_P, int EC, int nmu, int nE, int table2d) {
  return N_P <= kMaxPhases &&
         int_smem<false>(nullptr, N_L, N_P, EC, nmu, nE, table2d, true).bytes <= kIntSmemMax;
}

int64_t integrate_image_doubles(int N_L) { return image_doubles(N_L); }

int integrate_energy_chunk(int N_L, int N_P, int N_E, int mixed) {
  if (!mixed) return energy_chunk(N_L, N_P, N_E, (int)sizeof(PieceDF));
  // mixed form: lanes are energies, so the chunk that leaves the fewest lanes
  // idle, the larger of two (a cell is placed once per chunk), in 96 KB
  int best = 8;
  for (int ec = 16; ec <= 32; ec *= 2)
    if ((size_t)ec * N_L * sizeof(PieceT<float>) <= 96 * 1024 &&
        (N_E + ec - 1) / ec * ec <= (N_E + best - 1) / best * best)
      best = ec;
  return best;
}

void launch_integrate(const IntegrateArgs &a, cudaStream_t st) {
  if (a.n_members <= 0) return;
  const int nmu = a.atmos.I ? a.atmos.nmu : 0, nE = a.atmos.I ? a.atmos.nE : 0;
  // the work plan from the parallels' costs (needs the ray tables), beside the
  // geometry pre-pass
  row_cost_kernel<<<(unsigned)((a.n_rows * 32 + 256) / 256), 256, 0, st>>>(a);
  launch_geometry<true>(a, st);
  const long items = (long)a.max_chunks * a.n_eg;
  const unsigned ctas = (unsigned)(items < a.ctas ? items : a.ctas);
  if (a.mixed) {
    const size_t bytes = int_smem<true>(nullptr, a.N_L, a.N_P, a.EC, nmu, nE, a.table2d,
                                              false).bytes;
    cudaFuncSetAttribute(integrate_kernel<float>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         kIntSmemMax);
    integrate_kernel<float><<<ctas, kThreads, bytes, st>>>(a);
  } else {
    const size_t bytes = int_smem<false>(nullptr, a.N_L, a.N_P, a.EC, nmu, nE, a.table2d,
                                               a.wsum != nullptr).bytes;
    cudaFuncSetAttribute(integrate_kernel<double>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         kIntSmemMax);
    integrate_kernel<double><<<ctas, kThreads, bytes, st>>>(a);
  }
  dim3 grid((a.N_E * a.N_P + 255) / 256, a.n_members);
  reduce_flux_kernel<<<grid, 256, 0, st>>>(a);
}


void launch_split_reduce(const SplitArgs &a, cudaStream_t st) {
  const int n = a.n[3] * a.n[4];
  split_reduce_kernel<<<(n + 255) / 256, 256, 0, st>>>(a);
}

size_t stokes_smem_bytes(int N_L, int N_P, int N_E, int N_R, int nmu, int nE) {
  return stokes_smem(N_L, N_P, N_E, N_R, nmu, nE);
}

size_t stokes_partial_doubles(const IntegrateArgs &a) {
  return (size_t)a.n_rows * 3 * a.N_E * a.N_P;
}

int launch_stokes(const IntegrateArgs &a, cudaStream_t st) {
  if (a.n_members <= 0) return 0;
  const int nmu = a.atmos.I ? a.atmos.nmu : 0, nE = a.atmos.I ? a.atmos.nE : 0;
  const size_t smem = stokes_smem(a.N_L, a.N_P, a.N_E, a.N_R, nmu, nE);
  if (smem > 227 * 1024) return -2;
  if (a.atmos.I != nullptr) launch_geometry<false>(a, st);
  if (cudaFuncSetAttribute(stokes_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)smem) != cudaSuccess)
    return -5;
  // Groups of a parallel's energy chunks: the count that takes the fewest
  // turns of the chip (one CTA per SM by registers), a CTA's geometry counted
  // as a chunk and a half: a call of 40 parallels of 7 chunks 1092 us with one
  // group, 556 us with this rule's.
  const int EC = energy_chunk(a.N_L, a.N_P, a.N_E, kStokesPiece);
  const int nec = (a.N_E + EC - 1) / EC;
  int n_eg = 1;
  double best = 1.0e300;
  for (int n = 1; n <= nec; n++) {
    const double turns = (double)((a.n_rows * n + 151) / 152);
    const double cost = turns * (1.5 + (nec + n - 1) / n);
    if (cost < best) {
      best = cost;
      n_eg = n;
    }
  }
  stokes_kernel<<<dim3((unsigned)a.n_rows, (unsigned)n_eg), kThreads, smem, st>>>(a);
  const int n = a.N_E * a.N_P;
  dim3 grid((n + 255) / 256, a.n_members, 3);
  reduce_stokes_kernel<<<grid, 256, 0, st>>>(a);
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}

}  // namespace xg
