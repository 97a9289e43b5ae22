// The fitted amplitude at arbitrary points for kernels made of harmonics (pball groups, dirichlet columns), the
// binned fit's sqrt_density / predict / predict_grid (rahuljhu/band-limited-ml blml_binned.py:451-500). Such a kernel
// is exactly a weighted sum of plane waves, so
//     g(x) = sum_b e_b K(x - z_b) = sum_q C_q exp(2 pi i nu_q . u),   C = W (v^H e),  u = (x - origin) / h,
// with the spectrum C from the mat-vec plan's forward stages (blml_spectrum). A warp takes kPwPts query points: the
// lanes split the axis-1 frequencies (their phases computed once per chunk), every coefficient loaded serves all the
// points, the axis-0 phases are computed 32 frequencies at a time, one per lane and point, and read back as broadcasts;
// a fixed-order warp reduction ends the points. Phases are reduced to [-1/2, 1/2] cycles before sincospi, so the large
// products nu u of wide lattices keep their accuracy.
// Bound: float64 arithmetic, 8 flops per point and harmonic. (One point per warp with the axis-0 phase formed by every
// lane spent most of it on sincospi: 800 us for 50,000 points of an 85 x 85 band, now 208.)
#include "common.cuh"

namespace blml {

constexpr int kPwWarps = 8;              // warps per CTA
constexpr int kPwPts = 4;                // query points per warp

__device__ __forceinline__ cpx<double> phase(double nu, double u) {
  double c = nu * u;
  c -= rint(c);
  double sn, cs;
  sincospi(2.0 * c, &sn, &cs);
  return {cs, sn};
}

// spec (H1 x H2 complex, row-major), f1 (H1), f2 (H2) cycles per lattice index, U (m x 2) lattice coordinates; C
// axis-1 frequencies per lane and chunk; V: spec's coefficients in one 16-byte load (16-byte aligned), else in two
template <int C, bool V>
__global__ void __launch_bounds__(32 * kPwWarps, 2) k_planewave_points(int H1, int H2, const double* __restrict__ f1,
                                                                        const double* __restrict__ f2,
                                                                        const cpx<double>* __restrict__ spec, int64_t m,
                                                                        const double* __restrict__ U,
                                                                        cpx<double>* __restrict__ g) {
  __shared__ double2 ph1[kPwWarps][32][kPwPts];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t i0 = ((int64_t)blockIdx.x * kPwWarps + warp) * kPwPts;
  if (i0 >= m) return;                                  // whole warps leave together
  double u1[kPwPts], u2[kPwPts];
#pragma unroll
  for (int p = 0; p < kPwPts; p++) {
    const int64_t i = min(i0 + p, m - 1);               // points past the end repeat the last one, not stored
    u1[p] = U[2 * i]; u2[p] = U[2 * i + 1];
  }
  cpx<double> acc[kPwPts];
#pragma unroll
  for (int p = 0; p < kPwPts; p++) acc[p] = {0.0, 0.0};
  for (int c0 = 0; c0 < H2; c0 += 32 * C) {
    cpx<double> ph2[C][kPwPts];
    int q2[C];
#pragma unroll
    for (int c = 0; c < C; c++) {
      q2[c] = c0 + lane + 32 * c;
      const bool in = q2[c] < H2;
      if (!in) q2[c] = 0;
#pragma unroll
      for (int p = 0; p < kPwPts; p++) {
        ph2[c][p] = phase(f2[q2[c]], u2[p]);
        if (!in) ph2[c][p] = {0.0, 0.0};
      }
    }
    for (int b = 0; b < H1; b += 32) {
      __syncwarp();
#pragma unroll
      for (int p = 0; p < kPwPts; p++) {
        const cpx<double> v = phase(f1[min(b + lane, H1 - 1)], u1[p]);
        ph1[warp][lane][p] = make_double2(v.re, v.im);
      }
      __syncwarp();
      const int nq = min(32, H1 - b);
      for (int q = 0; q < nq; q++) {
        const cpx<double>* row = spec + (int64_t)(b + q) * H2;
        cpx<double> part[kPwPts];
#pragma unroll
        for (int p = 0; p < kPwPts; p++) part[p] = {0.0, 0.0};
#pragma unroll
        for (int c = 0; c < C; c++) {
          cpx<double> s;
          if (V) { const double2 v = __ldg(reinterpret_cast<const double2*>(row + q2[c])); s = {v.x, v.y}; }
          else s = row[q2[c]];
#pragma unroll
          for (int p = 0; p < kPwPts; p++) part[p] = cfma(s, ph2[c][p], part[p]);
        }
#pragma unroll
        for (int p = 0; p < kPwPts; p++) {
          const double2 v = ph1[warp][q][p];
          acc[p] = cfma(part[p], cpx<double>{v.x, v.y}, acc[p]);
        }
      }
    }
  }
#pragma unroll
  for (int p = 0; p < kPwPts; p++) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      acc[p].re += __shfl_down_sync(0xffffffffu, acc[p].re, o);
      acc[p].im += __shfl_down_sync(0xffffffffu, acc[p].im, o);
    }
    if (lane == 0 && i0 + p < m) g[i0 + p] = acc[p];
  }
}

}  // namespace blml

using namespace blml;

extern "C" {

int blml_planewave_points(int H1, int H2, const double* f1, const double* f2, const double* spec, int64_t m,
                          const double* U, double* g, void* stream) {
  if (H1 < 1 || H2 < 1 || m < 0) { set_error("blml_planewave_points: H1, H2 >= 1, m >= 0"); return BLML_ERR_ARG; }
  if (m == 0) return BLML_OK;
  if (!f1 || !f2 || !spec || !U || !g) { set_error("blml_planewave_points: null pointer"); return BLML_ERR_ARG; }
  const int64_t per = kPwWarps * kPwPts;
  const unsigned blocks = (unsigned)((m + per - 1) / per);
  const int chunks = (H2 + 127) / 128, c = (H2 + 32 * chunks - 1) / (32 * chunks);     // up to 4 frequencies per lane
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  auto run = [&](auto kern) {
    kern<<<blocks, 32 * kPwWarps, 0, st>>>(H1, H2, f1, f2, reinterpret_cast<const cpx<double>*>(spec), m, U,
                                           reinterpret_cast<cpx<double>*>(g));
  };
  const bool v = (reinterpret_cast<uintptr_t>(spec) & 15) == 0;
  if (c <= 1) v ? run(k_planewave_points<1, true>) : run(k_planewave_points<1, false>);
  else if (c == 2) v ? run(k_planewave_points<2, true>) : run(k_planewave_points<2, false>);
  else if (c == 3) v ? run(k_planewave_points<3, true>) : run(k_planewave_points<3, false>);
  else v ? run(k_planewave_points<4, true>) : run(k_planewave_points<4, false>);
  BLML_CHECK_LAUNCH("blml_planewave_points");
  return BLML_OK;
}

}  // extern "C"
