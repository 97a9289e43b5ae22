// The fitted amplitude at arbitrary points (BLMLQuick.sqrt_density / predict, rahuljhu/band-limited-ml
// blml_trivial.py:3288-3320 with the continuous product kernel of :2573): g(x_i) = sum_b e_b prod_c K_c(x_ic - z_bc)
// over the fit's B bin centres z_b, the kernel evaluated exactly (not from a lattice table: the query points are off
// the lattice). A warp holds 32 query points; the 8 warps of a block share them and take every eighth bin of a staged
// tile, the blocks of a cluster take slices of the bins, and the sums are joined in a fixed order (shared memory, then
// distributed shared memory), so a few hundred points still fill the GPU. A ball unit over a group of D columns
// (blml_trivial.py:580-591, 135-143) is one radial value per pair: prod fc p(s), s = ||fc (x - z)|| over the group,
// p(s) = (1/2)^(D/2) J_(D/2)(pi s) / s^(D/2) -- CUDA's jn for whole orders; for half orders the power series below
// nu + 12 and, above, upward recurrence from the closed forms of J_1/2 and J_3/2 (the standard methods).
// Bound: float64 arithmetic, about 90 instructions per pair of a sinc and a dirichlet column. sin(pi y) is the odd
// near-minimax polynomial below on the reduced argument, and a pair's factors share one division (numerators and
// denominators multiplied apart). 20,000 points by 17,000 bins of a sinc and a dirichlet column: 23.0 -> 2.64 ms (the old
// grid, one thread per point over every bin, was 79 blocks; its sinpi, fmod and three divisions the rest).
#include <cooperative_groups.h>
#include "common.cuh"

namespace blml {

constexpr int kPtThreads = 256;
constexpr int kPtTile = 256;
constexpr int kPtMaxD = 8;

__device__ __forceinline__ double sinc_unit(double f, double t) {
  // f sinc(f t) = sin(pi f t) / (pi t), f at t = 0
  return t == 0.0 ? f : sinpi(f * t) / (M_PI * t);
}

__device__ __forceinline__ double point_unit(const blml_point_col& c, double t) {
  if (c.kind == BLML_PT_SINC) return sinc_unit(c.f, t);
  if (c.kind == BLML_PT_SLITS) return sinc_unit(c.f, t) - (c.fi > 0 ? sinc_unit(c.fi, t) : 0.0);
  // dirichlet: (sin(pi M u / P) - sin(pi Mi u / P)) / sin(pi u / P) / P, u = |t| folded into [0, P / 2]
  const double P = c.P;
  double u = fmod(fabs(t), P);
  u = fmin(u, P - u);
  if (u < 1e-10) return (c.M - c.Mi) / P;
  return (sinpi(c.M * u / P) - sinpi(c.Mi * u / P)) / sinpi(u / P) / P;
}

// J_(twice_nu / 2)(x), x >= 0, twice_nu odd: the power series sum_k (-1)^k (x/2)^(2k+nu) / (k! Gamma(k+nu+1)) below
// x = nu + 12 (upward recurrence loses accuracy below the order), above it J_{m+1} = (2m / x) J_m - J_{m-1} from
// J_1/2 = c sin x and J_3/2 = c (sin x / x - cos x), c = sqrt(2 / (pi x))
__device__ __noinline__ double bessel_half_order(int twice_nu, double x) {
  const double nu = 0.5 * twice_nu;
  if (x < nu + 12.0) {
    const double xs = 0.5 * x;
    double term = pow(xs, nu) / tgamma(nu + 1.0), acc = term;
    for (int k = 1; k < 80; k++) {
      term = -term * xs * xs / (k * (k + nu));
      acc += term;
    }
    return acc;
  }
  const double c = sqrt(2.0 / (M_PI * x));
  double jm = c * sin(x), jc = c * (sin(x) / x - cos(x)), m = 0.5;
  if (twice_nu == 1) return jm;
  while (m + 1.0 < nu - 1e-9) {
    const double jn1 = (2.0 * (m + 1.0) / x) * jc - jm;
    jm = jc; jc = jn1; m += 1.0;
  }
  return jc;
}

// the ball profile p(s) in D dims; p0 = p(0) = pi^(D/2) (1/2)^D / Gamma(D/2 + 1), the ball's volume
__device__ __noinline__ double ball_profile(double s, int D, double p0) {
  if (s == 0.0) return p0;
  const double x = M_PI * s;
  const double J = (D % 2 == 0) ? jn(D / 2, x) : bessel_half_order(D, x);
  return pow(0.5, 0.5 * D) * J / pow(s, 0.5 * D);
}

// sin(pi r), |r| <= 1/2: r P(r^2), P the degree-8 polynomial of least relative error for sin(pi sqrt s) / sqrt s on
// [0, 1/4] (Remez exchange in 50-digit arithmetic, coefficients rounded to float64: 4e-17 relative)
__device__ __forceinline__ double sinpi_core(double r) {
  const double s = r * r;
  double p = 7.6947271574417395e-07;
  p = fma(p, s, -2.1903185407119565e-05);
  p = fma(p, s, 0.00046629968877016405);
  p = fma(p, s, -0.0073704304787627463);
  p = fma(p, s, 0.082145886569892815);
  p = fma(p, s, -0.59926452931873819);
  p = fma(p, s, 2.550164039877294);
  p = fma(p, s, -5.1677127800499694);
  p = fma(p, s, 3.1415926535897931);
  return r * p;
}
// nearest integer by adding 1.5 2^52 (|y| < 2^51): its parity in the sum's low bit
constexpr double kRound = 6755399441055744.0, kRoundMax = 2251799813685248.0;
__device__ __forceinline__ double sinpi_fast(double y) {
  if (!(fabs(y) < kRoundMax)) return sinpi(y);                    // (also NaN)
  const double n = y + kRound;
  const double v = sinpi_core(y - (n - kRound));
  return __hiloint2double(__double2hiint(v) ^ (__double2loint(n) << 31), __double2loint(v));
}

// one column's factor as num / den, multiplied into the pair's
__device__ __forceinline__ void point_factor(const blml_point_col& c, double inv_p, double t, double& num, double& den) {
  if (c.kind == BLML_PT_DIRICHLET) {
    const double k = t * inv_p;
    if (!(fabs(k) < kRoundMax)) { num *= point_unit(c, t); return; }
    const double u = fma(-((k + kRound) - kRound), c.P, t);       // t folded into [-P / 2, P / 2]
    if (fabs(u) < 1e-10) { num *= (c.M - c.Mi) / c.P; return; }
    const double r = u * inv_p;
    double v = sinpi_fast(c.M * r);
    if (c.Mi) v -= sinpi_fast(c.Mi * r);
    num *= v; den *= sinpi_core(r) * c.P;
    return;
  }
  // sinc and slits: sin(pi f t) / (pi t) to rounding f (1 - (pi f t)^2 / 6), so f, below |f t| = 1e-9
  const double y = c.f * t;
  const bool slits = c.kind == BLML_PT_SLITS && c.fi > 0;
  if (fabs(y) < 1e-9) { num *= slits ? c.f - c.fi : c.f; return; }
  double v = sinpi_fast(y);
  if (slits) v -= sinpi_fast(c.fi * t);
  num *= v; den *= M_PI * t;
}

constexpr int kPtWarps = kPtThreads / 32;
template <int D>
__global__ void __launch_bounds__(kPtThreads) k_point_rows(int64_t m, const double* __restrict__ X, int64_t B,
                                                          int64_t slice, const double* __restrict__ Z,
                                                          const double* __restrict__ e,
                                                          const __grid_constant__ blml_point_cols cols,
                                                          double* __restrict__ g) {
  __shared__ double zs[kPtTile * D];
  __shared__ double es[kPtTile];
  __shared__ double sums[kPtWarps][32];
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, splits = (int)cl.num_blocks(), rank = (int)cl.block_rank();
  const int64_t i = (int64_t)(blockIdx.x / splits) * 32 + lane;
  double x[D], inv_p[D];
#pragma unroll
  for (int c = 0; c < D; c++) {
    x[c] = i < m ? X[i * D + c] : 0.0;
    inv_p[c] = cols.c[c].kind == BLML_PT_DIRICHLET ? 1.0 / cols.c[c].P : 0.0;
  }
  double acc = 0.0;
  const int64_t b_end = min(B, (int64_t)(rank + 1) * slice);
  for (int64_t b0 = (int64_t)rank * slice; b0 < b_end; b0 += kPtTile) {
    const int nt = (int)(b_end - b0 < kPtTile ? b_end - b0 : kPtTile);
    __syncthreads();
    for (int j = threadIdx.x; j < nt * D; j += kPtThreads) zs[j] = Z[b0 * D + j];
    for (int j = threadIdx.x; j < nt; j += kPtThreads) es[j] = e[b0 + j];
    __syncthreads();
    for (int j = warp; j < nt; j += kPtWarps) {
      double num = es[j], den = 1.0;
#pragma unroll
      for (int c = 0; c < D; c++) {
        const blml_point_col& cc = cols.c[c];
        if (cc.kind == BLML_PT_BALL) {
          if (cc.fi == 0.0) continue;                             // a ball group's value sits on its first column
          double s2 = 0.0;
#pragma unroll
          for (int c2 = 0; c2 < D; c2++)
            if ((cc.M >> c2) & 1) {
              const double t = cols.c[c2].f * (x[c2] - zs[j * D + c2]);
              s2 += t * t;
            }
          num *= cc.fi * ball_profile(sqrt(s2), cc.Mi, cc.P);
        } else {
          point_factor(cc, inv_p[c], x[c] - zs[j * D + c], num, den);
        }
      }
      acc += num / den;
    }
  }
  sums[warp][lane] = acc;
  __syncthreads();
  if (warp == 0) {
    double v = 0.0;
#pragma unroll
    for (int w = 0; w < kPtWarps; w++) v += sums[w][lane];
    sums[0][lane] = v;
  }
  cl.sync();
  if (rank == 0 && warp == 0 && i < m) {
    double v = 0.0;
    for (int b = 0; b < splits; b++) v += cl.map_shared_rank(&sums[0][0], b)[lane];
    g[i] = v;
  }
  cl.sync();                                                      // the other blocks' sums stay until they are read
}

// Point sums of several densities (blml_local.py:555-560, point_rows_multi: FusedFit's joint and marginals at
// points): g[i][m] = sum_b W[b][m] prod_u (bit u of masks[m] ? K_u(x_i - z_b) : 1), every unit's value computed once
// per (point, bin) pair; unit_of[c] is the unit of column c (a ball group's value sits on its first column).
constexpr int kPtMaxM = 8;
struct PtMulti { int unit_of[kPtMaxD]; unsigned masks[kPtMaxM]; };

__global__ void __launch_bounds__(kPtThreads) k_point_rows_multi(int64_t m, int d, int U, const double* __restrict__ X,
                                                                int64_t B, const double* __restrict__ Z,
                                                                const double* __restrict__ W, int Mm,
                                                                blml_point_cols cols, PtMulti pm,
                                                                double* __restrict__ g) {
  __shared__ double zs[kPtTile * kPtMaxD];
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  double x[kPtMaxD];
  for (int c = 0; c < d; c++) x[c] = i < m ? X[i * d + c] : 0.0;
  double acc[kPtMaxM];
  for (int q = 0; q < kPtMaxM; q++) acc[q] = 0.0;
  for (int64_t b0 = 0; b0 < B; b0 += kPtTile) {
    const int nt = (int)(B - b0 < kPtTile ? B - b0 : kPtTile);
    __syncthreads();
    for (int j = threadIdx.x; j < nt * d; j += blockDim.x) zs[j] = Z[b0 * d + j];
    __syncthreads();
    if (i < m) {
      for (int j = 0; j < nt; j++) {
        double fac[kPtMaxD];
        for (int u = 0; u < U; u++) fac[u] = 1.0;
        for (int c = 0; c < d; c++) {
          const blml_point_col& cc = cols.c[c];
          if (cc.kind == BLML_PT_BALL) {
            if (cc.fi == 0.0) continue;
            double s2 = 0.0;
            for (int c2 = 0; c2 < d; c2++)
              if ((cc.M >> c2) & 1) {
                const double t = cols.c[c2].f * (x[c2] - zs[j * d + c2]);
                s2 += t * t;
              }
            fac[pm.unit_of[c]] = cc.fi * ball_profile(sqrt(s2), cc.Mi, cc.P);
          } else {
            fac[pm.unit_of[c]] = point_unit(cc, x[c] - zs[j * d + c]);
          }
        }
        const int64_t b = b0 + j;
        for (int q = 0; q < Mm; q++) {
          double p = W[b * Mm + q];
          for (int u = 0; u < U; u++)
            if ((pm.masks[q] >> u) & 1u) p *= fac[u];
          acc[q] += p;
        }
      }
    }
  }
  if (i < m)
    for (int q = 0; q < Mm; q++) g[i * Mm + q] = acc[q];
}

}  // namespace blml

using namespace blml;

// the columns' kinds and ball groups checked, copied into cc; nonzero (with the error set) when they are not valid
static int check_point_cols(int d, const blml_point_col* cols, blml_point_cols& cc, const char* who) {
  for (int c = 0; c < d; c++) {
    cc.c[c] = cols[c];
    const int k = cols[c].kind;
    if (k != BLML_PT_SINC && k != BLML_PT_SLITS && k != BLML_PT_DIRICHLET && k != BLML_PT_BALL) {
      set_error("%s: column %d: kind %d (sinc, slits, dirichlet or ball)", who, c, k);
      return 1;
    }
    if (k == BLML_PT_DIRICHLET && !(cols[c].P > 0)) {
      set_error("%s: column %d: dirichlet period must be positive", who, c);
      return 1;
    }
    if (k == BLML_PT_BALL) {
      // the group mask holds this column and only ball columns; the first column of the group carries prod fc (fi),
      // the group size (Mi) and p(0) (P), the others fi = 0
      const int mask = cols[c].M;
      int lead = -1, size = 0;
      for (int c2 = 0; c2 < d; c2++)
        if ((mask >> c2) & 1) { size++; if (lead < 0) lead = c2; }
      bool ok = mask > 0 && mask < (1 << d) && ((mask >> c) & 1) && cols[c].f > 0;
      for (int c2 = 0; c2 < d && ok; c2++)
        if ((mask >> c2) & 1) ok = cols[c2].kind == BLML_PT_BALL && cols[c2].M == mask;
      if (ok && c == lead) ok = cols[c].Mi == size && cols[c].fi > 0 && cols[c].P > 0;
      if (ok && c != lead) ok = cols[c].fi == 0.0;
      if (!ok) {
        set_error("%s: column %d: inconsistent ball group (mask %d)", who, c, mask);
        return 1;
      }
    }
  }
  return 0;
}

extern "C" {

int blml_point_rows(int64_t m, int d, const double* X, int64_t B, const double* Z, const double* e,
                    const blml_point_col* cols, double* g, void* stream) {
  if (m < 0 || B < 0 || d < 1 || d > kPtMaxD || !cols) {
    set_error("blml_point_rows: 1 <= d <= %d columns, m, B >= 0", kPtMaxD);
    return BLML_ERR_ARG;
  }
  if (m == 0) return BLML_OK;
  if (!X || !g || (B > 0 && (!Z || !e))) { set_error("blml_point_rows: null pointer"); return BLML_ERR_ARG; }
  blml_point_cols cc;
  if (check_point_cols(d, cols, cc, "blml_point_rows")) return BLML_ERR_ARG;
  // clusters of up to 8 blocks share 32 points' bins until 8 blocks per SM are reached, at least 256 bins each
  const int64_t groups = (m + 31) / 32;
  int splits = 1;
  while (splits < 8 && groups * splits < 8 * 148 && B / (2 * splits) >= kPtTile) splits *= 2;
  const int64_t slice = (B + splits - 1) / splits;
  if (groups * splits > 0x7fffffffLL) { set_error("blml_point_rows: too many points"); return BLML_ERR_ARG; }
  cudaLaunchConfig_t lc{};
  lc.gridDim = dim3((unsigned)(groups * splits)); lc.blockDim = dim3(kPtThreads);
  lc.stream = reinterpret_cast<cudaStream_t>(stream);
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = (unsigned)splits; at.val.clusterDim.y = 1; at.val.clusterDim.z = 1;
  lc.attrs = &at; lc.numAttrs = 1;
#define PT_ROWS(DD) case DD: cudaLaunchKernelEx(&lc, k_point_rows<DD>, m, X, B, slice, Z, e, cc, g); break;
  switch (d) { PT_ROWS(1) PT_ROWS(2) PT_ROWS(3) PT_ROWS(4) PT_ROWS(5) PT_ROWS(6) PT_ROWS(7) PT_ROWS(8) }
#undef PT_ROWS
  BLML_CHECK_LAUNCH("blml_point_rows");
  return BLML_OK;
}

int blml_point_rows_multi(int64_t m, int d, const double* X, int64_t B, const double* Z, const double* W, int Mm,
                          const blml_point_col* cols, const int* unit_of, int U, const unsigned* masks, double* g,
                          void* stream) {
  if (m < 0 || B < 0 || d < 1 || d > kPtMaxD || !cols || !unit_of || !masks || Mm < 1 || Mm > kPtMaxM || U < 1 ||
      U > d) {
    set_error("blml_point_rows_multi: 1 <= d <= %d columns, 1 <= U <= d units, 1 <= Mm <= %d densities", kPtMaxD,
              kPtMaxM);
    return BLML_ERR_ARG;
  }
  if (m == 0) return BLML_OK;
  if (!X || !g || (B > 0 && (!Z || !W))) { set_error("blml_point_rows_multi: null pointer"); return BLML_ERR_ARG; }
  blml_point_cols cc;
  if (check_point_cols(d, cols, cc, "blml_point_rows_multi")) return BLML_ERR_ARG;
  PtMulti pm;
  for (int c = 0; c < kPtMaxD; c++) pm.unit_of[c] = 0;
  for (int c = 0; c < d; c++) {
    if (unit_of[c] < 0 || unit_of[c] >= U) { set_error("blml_point_rows_multi: column %d: unit %d of %d", c, unit_of[c], U); return BLML_ERR_ARG; }
    pm.unit_of[c] = unit_of[c];
  }
  for (int q = 0; q < kPtMaxM; q++) pm.masks[q] = q < Mm ? masks[q] : 0u;
  for (int q = 0; q < Mm; q++)
    if (pm.masks[q] >> U) { set_error("blml_point_rows_multi: density %d masks a unit beyond %d", q, U); return BLML_ERR_ARG; }
  const int64_t blocks = (m + kPtThreads - 1) / kPtThreads;
  k_point_rows_multi<<<(unsigned)blocks, kPtThreads, 0, reinterpret_cast<cudaStream_t>(stream)>>>(m, d, U, X, B, Z, W,
                                                                                                 Mm, cc, pm, g);
  BLML_CHECK_LAUNCH("blml_point_rows_multi");
  return BLML_OK;
}

}  // extern "C"
