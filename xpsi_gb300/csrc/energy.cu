// energy.cu -- K4: integration of the specific-flux signal over instrument
// input-energy intervals, replacing xpsi/tools/energy_integrator.pyx:27-114.
//
// One CTA per (signal, block of `cols` phase columns).  The integrand
// E S(E) ln 10 of the block's columns, its chords in log10 E and the Akima
// pieces on them (periodic ends, as the reference uses, :54) are formed in
// shared memory once; then one thread per (interval, column) output
// integrates the pieces it covers exactly, clipped at the highest energy
// (:91-103).  FP64 throughout, whose pipe bounds it: a piece's four divisions
// are formed once for the one to three outputs that cover it, and outputs find
// their pieces by bit patterns.
#include "common.cuh"
#include "kernels.h"

namespace xg {
namespace {

constexpr int kEThreads = 256;

__global__ void __launch_bounds__(kEThreads) energy_kernel(EnergyArgs a, int cols) {
  extern __shared__ double sm[];
  const int N_E = a.N_E, N_P = a.N_P, ne = a.n_edges;
  double *logE = sm;                   // [N_E]
  double *wE = logE + N_E;             // [N_E] 10^logE
  double *edges = wE + N_E;            // [ne]
  double *Y = edges + ne;              // [N_E][cols] integrand
  double *CH = Y + (size_t)N_E * cols;  // [N_E - 1][cols] chords
  double *P1 = CH + (size_t)(N_E - 1) * cols;  // [N_E - 1][cols] the pieces' coefficients
  double *P2 = P1 + (size_t)(N_E - 1) * cols, *P3 = P2 + (size_t)(N_E - 1) * cols;
  __shared__ int s_stop;
  const int s = blockIdx.y;
  const int k0 = blockIdx.x * cols;
  const double *sig = a.signal + a.in_off[s];
  double *out = a.out + a.out_off[s];
  const double div = a.scale_per ? a.scale_per[s] : 1.0;
  const double ln10 = log(10.0);
  for (int t = threadIdx.x; t < N_E; t += blockDim.x) {
    logE[t] = a.logE[t];
    wE[t] = pow(10.0, a.logE[t]);
  }
  for (int t = threadIdx.x; t < ne; t += blockDim.x) edges[t] = a.logEdges[t];
  if (threadIdx.x == 0) s_stop = ne - 1;
  __syncthreads();
  const double maxE = logE[N_E - 1];
  // the reference stops after the first interval that reaches past the
  // highest energy (:103); later intervals keep their initial zero
  for (int j = threadIdx.x; j + 1 < ne; j += blockDim.x)
    if (edges[j + 1] > maxE) atomicMin(&s_stop, j + 1);
  // y_j = 10^logE_j * (signal_j / d^2) * ln 10, evaluated in the reference's order
  for (int t = threadIdx.x; t < N_E * cols; t += blockDim.x) {
    const int j = t / cols, c = t - j * cols, k = k0 + c;
    double v = 0.0;
    if (k < N_P) {
      v = sig[(size_t)j * N_P + k];
      if (a.scale_per) v = v / div;
    }
    Y[t] = wE[j] * v * ln10;
  }
  __syncthreads();
  for (int t = threadIdx.x; t < (N_E - 1) * cols; t += blockDim.x) {
    const int q = t / cols;
    CH[t] = (Y[t + cols] - Y[t]) / (logE[q + 1] - logE[q]);
  }
  __syncthreads();
  for (int t = threadIdx.x; t < (N_E - 1) * cols; t += blockDim.x) {
    const int i = t / cols, c = t - i * cols;
    auto chord = [&](int q) -> double { return CH[periodic_chord(q, N_E) * cols + c]; };
    akima_piece(chord(i - 2), chord(i - 1), chord(i), chord(i + 1), chord(i + 2),
                logE[i + 1] - logE[i], P1[t], P2[t], P3[t]);
  }
  __syncthreads();
  const int stop = s_stop;
  // largest i in [0, N_E - 2] with logE[i] <= v, by the bit patterns
  auto find = [&](double v) {
    const long long vb = ordered(v);
    int lo = 0, hi = N_E - 1;
    while (hi > lo + 1) {
      const int mid = (lo + hi) >> 1;
      if (ordered(logE[mid]) > vb) hi = mid; else lo = mid;
    }
    return lo;
  };
  for (int t = threadIdx.x; t < (ne - 1) * cols; t += blockDim.x) {
    const int j = t / cols, c = t - j * cols, k = k0 + c;
    if (k >= N_P) continue;
    double val;
    if (j >= stop) {
      val = 0.0;
    } else {
      const double lo = edges[j];
      const double hi = edges[j + 1] > maxE ? maxE : edges[j + 1];
      if (lo > hi || lo < logE[0] || hi > maxE) {
        val = nan("");
      } else if (lo == hi) {
        val = 0.0;
      } else {
        const int ia = find(lo), ib = find(hi);
        double acc = 0.0;
        for (int i = ia; i <= ib; i++) {
          const int q = i * cols + c;
          const double u = (i == ia) ? lo - logE[i] : 0.0;
          const double w = (i == ib) ? hi - logE[i] : logE[i + 1] - logE[i];
          acc += piece_integral(Y[q], P1[q], P2[q], P3[q], u, w);
        }
        val = acc;
      }
    }
    if (a.accumulate) {
      if (j < stop) out[(size_t)j * N_P + k] += val;
    } else {
      out[(size_t)j * N_P + k] = val;
    }
  }
}

}  // namespace

void launch_energy(const EnergyArgs &a, cudaStream_t st) {
  if (a.n_signals <= 0) return;
  // Phase columns per CTA: 16, fewer while that leaves SMs without a CTA (one
  // signal of 128 phases and energies: 8 CTAs of 16 columns, 118 us with a
  // piece formed per output; 64 of two, 19 us; below two the CTA's own powers
  // and edges outweigh its columns) or its shared memory does not fit.  48
  // signals: 396 us, 304 us now.
  auto bytes = [&](int cols) {
    return (size_t)(2 * a.N_E + a.n_edges + (size_t)(5 * a.N_E - 4) * cols) * sizeof(double);
  };
  int cols = 16;
  while (cols > 2 && (int64_t)((a.N_P + cols - 1) / cols) * a.n_signals < 152) cols /= 2;
  while (cols > 1 && bytes(cols) > 200 * 1024) cols /= 2;
  cudaFuncSetAttribute(energy_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
  dim3 grid((a.N_P + cols - 1) / cols, a.n_signals);
  energy_kernel<<<grid, kEThreads, bytes(cols), st>>>(a, cols);
}

}  // namespace xg
