// Pair accumulation over occupied lattice bins from the product kernel's value tables:
//     rows:  s_r = sum_j w_j prod_u T_u[idx_u(ZA_r, ZB_j)]   (+ d/dtheta rows with grad)
//     cols:  out[r, j] = prod_u T_u[idx_u(ZA_r, ZB_j)]
// Every CTA keeps the value tables in shared memory and streams the columns j in chunks (coordinates and weights
// staged in shared memory, read as warp broadcasts). Each thread owns rows; products are in REAL (float or
// double, the reference's f32 flag), sums in float64. Column slices of one row block are reduced in a fixed order
// by a second kernel, so results are deterministic (the reference combines slices with float64 atomics).
// Before any launch the coordinates are checked against the tables' extents on the device, so a stale table is an
// error, never an out-of-range read.
#include <limits.h>
#include <mutex>
#include <cuda.h>
#include "common.cuh"

namespace blml {

constexpr int RQ = 4;               // radial rows: grid points per lattice step (linear interpolation)
constexpr int PR_THREADS = 128;     // rows per CTA (one per thread)
constexpr int PR_CHUNK = 256;       // columns staged per shared-memory chunk
constexpr int MAXD = 8, MAXU = 8, MAXG = 4, MAXW = 8;

struct ColMeta {
  int d, U, G, nW, LR;
  int code[MAXD], grp[MAXD], dim_unit[MAXD];
  int64_t base[MAXD], J[MAXD], mk[MAXD], nb[MAXD];
  int grp_unit[MAXG];
  int wunit[MAXW], wcol[MAXW], wgrp[MAXW];
  int64_t dbase[MAXW];
  int64_t Tn, dTn;
};

template <typename REAL>
__device__ __forceinline__ REAL col_value(const ColMeta& cm, const REAL* T, int k, int64_t za, int64_t zb) {
  const int code = cm.code[k];
  int64_t idx;
  if (code == 0) idx = cm.base[k] + za - zb + cm.J[k];
  else if (code == 3) idx = cm.base[k] + za * cm.mk[k] + zb;
  else {                                     // circular distance, |za - zb| < nb
    const int64_t nb = cm.nb[k];
    int64_t m = za - zb;
    if (m < 0) m += nb; else if (m >= nb) m -= nb;
    if (m > nb - m) m = nb - m;
    idx = cm.base[k] + m;
  }
  return T[idx];
}

// One pair's unit factors (fac[u]) and the group indices (r2 / torus index per group).
template <typename REAL>
__device__ __forceinline__ void pair_factors(const ColMeta& cm, const REAL* T, const REAL* RT, const int64_t* za,
                                             const int64_t* zb, REAL* fac, int64_t* r2, bool* tor) {
  for (int g = 0; g < cm.G; g++) { r2[g] = 0; tor[g] = false; }
  for (int k = 0; k < cm.d; k++) {
    const int code = cm.code[k];
    const int64_t off = za[k] - zb[k];
    if (code == 2) { r2[cm.grp[k]] += off * off; continue; }
    if (code == 4) {
      const int g = cm.grp[k]; const int64_t nb = cm.nb[k];
      const int64_t m = off < 0 ? off + nb : off;
      r2[g] = r2[g] * nb + m; tor[g] = true; continue;
    }
    fac[cm.dim_unit[k]] = col_value(cm, T, k, za[k], zb[k]);
  }
  for (int g = 0; g < cm.G; g++) {
    const REAL* row = RT + (int64_t)g * cm.LR;
    if (tor[g]) { fac[cm.grp_unit[g]] = row[r2[g]]; continue; }
    const double t = sqrt((double)r2[g]) * RQ; const int i0 = (int)t; const REAL f = (REAL)(t - i0);
    fac[cm.grp_unit[g]] = row[i0] * (REAL(1) - f) + row[i0 + 1] * f;
  }
}

// derivative entry q of a pair (the reference's dval): a column's derivative row (raw offsets, rank tables), a
// group's torus row, or a radial row on the r grid times the offset of column wcol[q] for a shift entry
template <typename REAL>
__device__ __forceinline__ REAL dval(const ColMeta& cm, const REAL* dT, const REAL* dR, int q, const int64_t* za,
                                     const int64_t* zb, const int64_t* r2, const bool* tor) {
  const int g = cm.wgrp[q], k = cm.wcol[q];
  if (g >= 0 && tor[g]) return dR[(int64_t)q * cm.LR + r2[g]];
  if (g < 0) {
    const int64_t idx = cm.code[k] == 3 ? za[k] * cm.mk[k] + zb[k] : za[k] - zb[k] + cm.J[k];
    return dT[cm.dbase[q] + idx];
  }
  const double t = sqrt((double)r2[g]) * RQ; const int i0 = (int)t; const REAL f = (REAL)(t - i0);
  REAL v = dR[(int64_t)q * cm.LR + i0] * (REAL(1) - f) + dR[(int64_t)q * cm.LR + i0 + 1] * f;
  if (k >= 0) v *= (REAL)(za[k] - zb[k]);
  return v;
}

// General rows kernel: any column codes, groups and derivative entries. grid (row blocks, column slices).
// part[slice][r] (and dpart[slice][r][q]) are the slice sums.
template <typename REAL, bool GRAD>
__global__ void __launch_bounds__(PR_THREADS) k_rows_general(ColMeta cm, const REAL* Tg, const REAL* RTg,
                                                             const REAL* dTg, const REAL* dRg, const int64_t* ZA,
                                                             int64_t R, const int64_t* ZB, const double* w,
                                                             int64_t j0s, int64_t slice, int64_t M, double* part,
                                                             double* dpart) {
  extern __shared__ unsigned char smem_raw[];
  REAL* Ts = reinterpret_cast<REAL*>(smem_raw);
  REAL* RTs = Ts + cm.Tn;
  const int64_t nRT = (int64_t)cm.G * cm.LR;
  for (int64_t i = threadIdx.x; i < cm.Tn; i += blockDim.x) Ts[i] = Tg[i];
  for (int64_t i = threadIdx.x; i < nRT; i += blockDim.x) RTs[i] = RTg[i];
  __syncthreads();
  const int64_t r = (int64_t)blockIdx.x * PR_THREADS + threadIdx.x;
  const int64_t j0 = j0s + (int64_t)blockIdx.y * slice, j1 = min(M, j0 + slice);
  int64_t za[MAXD];
  const bool live = r < R;
  for (int k = 0; k < cm.d; k++) za[k] = live ? ZA[r * cm.d + k] : 0;
  double acc = 0.0, dacc[MAXW];
  for (int q = 0; q < MAXW; q++) dacc[q] = 0.0;
  REAL fac[MAXU + 1];
  for (int u = 0; u < MAXU; u++) fac[u] = REAL(1);
  int64_t r2[MAXG]; bool tor[MAXG];
  for (int64_t j = j0; j < j1 && live; j++) {
    const double wj = w[j];
    if (wj == 0.0) continue;
    int64_t zb[MAXD];
    for (int k = 0; k < cm.d; k++) zb[k] = ZB[j * cm.d + k];
    pair_factors<REAL>(cm, Ts, RTs, za, zb, fac, r2, tor);
    REAL pre[MAXU + 1];
    pre[0] = REAL(1);
    for (int u = 0; u < cm.U; u++) pre[u + 1] = pre[u] * fac[u];
    acc += (double)pre[cm.U] * wj;
    if (GRAD) {
      REAL suf[MAXU + 1];
      suf[cm.U] = REAL(1);
      for (int u = cm.U - 1; u >= 0; u--) suf[u] = suf[u + 1] * fac[u];
      for (int q = 0; q < cm.nW; q++) {
        const int u = cm.wunit[q];
        const REAL dv = dval<REAL>(cm, dTg, dRg, q, za, zb, r2, tor);
        dacc[q] += (double)(dv * pre[u] * suf[u + 1]) * wj;
      }
    }
  }
  if (!live) return;
  part[(int64_t)blockIdx.y * R + r] = acc;
  if (GRAD)
    for (int q = 0; q < cm.nW; q++) dpart[((int64_t)blockIdx.y * R + r) * cm.nW + q] = dacc[q];
}

// Fused rows of several densities over the same pairs (blml_local.py:213-286, rows_multi): s[r][m] = sum_j W[j][m]
// prod_u (bit u of umask[m] ? fac_u : 1), the unit factors computed once per pair and each density multiplying the
// units its mask keeps, in unit order (the joint: every unit; a marginal: the units of its columns). part[slice][r][m].
constexpr int MAXM = 8;
struct DensMasks { unsigned bits[MAXM]; };

template <typename REAL>
__global__ void __launch_bounds__(PR_THREADS) k_rows_multi(ColMeta cm, const REAL* Tg, const REAL* RTg,
                                                           const int64_t* ZA, int64_t R, const int64_t* ZB,
                                                           const double* W, int Mm, DensMasks dm, int64_t slice,
                                                           int64_t M, double* part) {
  extern __shared__ unsigned char smem_raw[];
  REAL* Ts = reinterpret_cast<REAL*>(smem_raw);
  REAL* RTs = Ts + cm.Tn;
  const int64_t nRT = (int64_t)cm.G * cm.LR;
  for (int64_t i = threadIdx.x; i < cm.Tn; i += blockDim.x) Ts[i] = Tg[i];
  for (int64_t i = threadIdx.x; i < nRT; i += blockDim.x) RTs[i] = RTg[i];
  __syncthreads();
  const int64_t r = (int64_t)blockIdx.x * PR_THREADS + threadIdx.x;
  const int64_t j0 = (int64_t)blockIdx.y * slice, j1 = min(M, j0 + slice);
  int64_t za[MAXD];
  const bool live = r < R;
  for (int k = 0; k < cm.d; k++) za[k] = live ? ZA[r * cm.d + k] : 0;
  double acc[MAXM];
  for (int m = 0; m < MAXM; m++) acc[m] = 0.0;
  REAL fac[MAXU + 1];
  for (int u = 0; u < MAXU; u++) fac[u] = REAL(1);
  int64_t r2[MAXG]; bool tor[MAXG];
  for (int64_t j = j0; j < j1 && live; j++) {
    int64_t zb[MAXD];
    for (int k = 0; k < cm.d; k++) zb[k] = ZB[j * cm.d + k];
    pair_factors<REAL>(cm, Ts, RTs, za, zb, fac, r2, tor);
    for (int m = 0; m < Mm; m++) {
      const double wj = W[j * Mm + m];
      if (wj == 0.0) continue;
      REAL p = REAL(1);
      for (int u = 0; u < cm.U; u++) p = p * (((dm.bits[m] >> u) & 1u) ? fac[u] : REAL(1));
      acc[m] += (double)p * wj;
    }
  }
  if (!live) return;
  for (int m = 0; m < Mm; m++) part[((int64_t)blockIdx.y * R + r) * Mm + m] = acc[m];
}

__host__ __device__ constexpr size_t align16(size_t b) { return (b + 15) & ~(size_t)15; }

// Fast rows kernel for product kernels without groups (every unit one column: offset, rank and circular tables).
// Each table lies in shared memory as one that a linear index reads -- circular columns unfolded to 2 nb - 1 offsets --,
// so a column's lookup is one add (the row's byte address plus the column's byte offset) and one shared-memory load.
// Columns are taken in unit order. A thread holds RPT rows; a chunk's columns are staged as packed byte offsets (read as
// 16-byte broadcasts that the RPT rows share) with the first position at which a column differs from the one before it:
// the products over the leading positions are kept and only those from there on are formed again, so columns in
// lexicographic order (unique bins) cost their last positions only. Products in REAL in unit order, sums in float64 over
// the slice's columns in order.
// GRAD: with ND >= nW derivative entries, d . prefix . suffix as the general kernel forms them.
constexpr int kRfMax = MAXD;
struct RowsFast {
  int col[kRfMax];                       // the column at each position
  int kind[kRfMax];                      // 0 offset, 1 circular, 3 rank
  int base[kRfMax], len[kRfMax], org[kRfMax], mul[kRfMax], nb[kRfMax];   // table; row address org + za mul; unfolded period
  int64_t zmin[kRfMax];                  // subtracted from both coordinates (offset and circular tables)
  int so[kRfMax];                        // the table in shared memory (elements)
  int nW, dpos[MAXW], dbase[MAXW], dlen[MAXW], dso[MAXW];                // derivative entries: position, table
  int total;                             // shared-memory elements of all tables
};
// shared memory: the tables, then per staged column its packed offsets, then its weight
__host__ __device__ constexpr int rf_words(int D) { return (D + 1 + 3) / 4 * 4; }
template <typename REAL> __host__ __device__ constexpr size_t rf_smem(int total, int D) {
  return align16((size_t)total * sizeof(REAL)) + (size_t)PR_CHUNK * (rf_words(D) * sizeof(int) + sizeof(double));
}

template <typename REAL, int D, int RPT, int ND>
__global__ void __launch_bounds__(PR_THREADS) k_rows_fast(const __grid_constant__ RowsFast rf, const REAL* Tg,
                                                          const REAL* dTg, const int64_t* ZA, int64_t R,
                                                          const int64_t* ZB, const double* w, int64_t slice, int64_t M,
                                                          double* part, double* dpart) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int W = rf_words(D), ES = sizeof(REAL);
  REAL* Ts = reinterpret_cast<REAL*>(smem_raw);
  int* zs = reinterpret_cast<int*>(smem_raw + align16((size_t)rf.total * sizeof(REAL)));
  double* ws = reinterpret_cast<double*>(zs + PR_CHUNK * W);
#pragma unroll
  for (int k = 0; k < D; k++)
    for (int i = threadIdx.x; i < rf.len[k]; i += PR_THREADS) {
      int s = i;
      if (rf.kind[k] == 1) { s = i - (rf.nb[k] - 1); s = s < 0 ? s + rf.nb[k] : s; s = min(s, rf.nb[k] - s); }
      Ts[rf.so[k] + i] = Tg[rf.base[k] + s];
    }
#pragma unroll
  for (int q = 0; q < ND; q++)
    if (q < rf.nW)
      for (int i = threadIdx.x; i < rf.dlen[q]; i += PR_THREADS) Ts[rf.dso[q] + i] = dTg[rf.dbase[q] + i];
  const int64_t r0 = (int64_t)blockIdx.x * (PR_THREADS * RPT) + threadIdx.x;
  int pb[RPT][D], db[ND ? ND : 1];       // byte addresses of the rows' tables (a derivative entry's: its column's, moved)
#pragma unroll
  for (int m = 0; m < RPT; m++) {
    // rows past the end repeat the thread's first one (a thread past it: row R - 1) and are not stored
    const int64_t r = min(r0 + (int64_t)m * PR_THREADS < R ? r0 + (int64_t)m * PR_THREADS : r0, R - 1);
#pragma unroll
    for (int k = 0; k < D; k++) {
      const int za = (int)(ZA[r * D + rf.col[k]] - rf.zmin[k]);
      pb[m][k] = (rf.so[k] + rf.org[k] + za * rf.mul[k]) * ES;
    }
  }
#pragma unroll
  for (int q = 0; q < ND; q++) {
    db[q] = 0;
#pragma unroll
    for (int k = 0; k < D; k++)
      if (q < rf.nW && rf.dpos[q] == k) db[q] = pb[0][k] + (rf.dso[q] - rf.so[k]) * ES;
  }
  double acc[RPT], dacc[ND ? ND : 1];
#pragma unroll
  for (int m = 0; m < RPT; m++) acc[m] = 0.0;
#pragma unroll
  for (int q = 0; q < ND; q++) dacc[q] = 0.0;
  const int64_t j0 = (int64_t)blockIdx.y * slice, j1 = min(M, j0 + slice);
  for (int64_t c0 = j0; c0 < j1; c0 += PR_CHUNK) {
    const int n = (int)(j1 - c0 < PR_CHUNK ? j1 - c0 : PR_CHUNK);
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += PR_THREADS) {
      const int64_t* z = ZB + (c0 + i) * D;
      const int64_t* zp = z - D;
      int lvl = i == 0 ? 0 : D;
#pragma unroll
      for (int k = D - 1; k >= 0; k--) {
        const int64_t v = z[rf.col[k]] - rf.zmin[k];
        zs[i * W + 1 + k] = (rf.kind[k] == 3 ? (int)v : -(int)v) * ES;
        if (i > 0 && v != zp[rf.col[k]] - rf.zmin[k]) lvl = k;
      }
      zs[i * W] = lvl;
      ws[i] = w[c0 + i];
    }
    __syncthreads();
    REAL pre[RPT][D];
    for (int jj = 0; jj < n; jj++) {
      int z[W];
#pragma unroll
      for (int q = 0; q < W / 4; q++) {
        const int4 v = reinterpret_cast<const int4*>(zs + jj * W)[q];
        z[4 * q] = v.x; z[4 * q + 1] = v.y; z[4 * q + 2] = v.z; z[4 * q + 3] = v.w;
      }
      const double wj = ws[jj];
      const int lvl = z[0];
      if constexpr (ND == 0) {
        // positions below lvl keep their products; the last is always formed
        auto from = [&](int k) {
#pragma unroll
          for (int m = 0; m < RPT; m++) {
            const REAL t = *reinterpret_cast<const REAL*>(smem_raw + (pb[m][k] + z[1 + k]));
            pre[m][k] = k ? pre[m][k ? k - 1 : 0] * t : t;
          }
        };
        if (D >= 2 && lvl < D - 1) {
          if (D >= 3 && lvl < D - 2) {
#pragma unroll
            for (int k = 0; k < D - 2; k++) from(k);
          }
          if (D >= 2) from(D >= 2 ? D - 2 : 0);
        }
        from(D - 1);
#pragma unroll
        for (int m = 0; m < RPT; m++) acc[m] = fma((double)pre[m][D - 1], wj, acc[m]);
      } else {
        REAL t[D], p[D + 1], sf[D + 1];
#pragma unroll
        for (int k = 0; k < D; k++) t[k] = *reinterpret_cast<const REAL*>(smem_raw + (pb[0][k] + z[1 + k]));
        p[0] = REAL(1); sf[D] = REAL(1);
#pragma unroll
        for (int k = 0; k < D; k++) p[k + 1] = p[k] * t[k];
#pragma unroll
        for (int k = D - 1; k >= 0; k--) sf[k] = sf[k + 1] * t[k];
        acc[0] += (double)p[D] * wj;
#pragma unroll
        for (int q = 0; q < ND; q++)
          if (q < rf.nW) {
            const int k = rf.dpos[q];
            REAL a = p[0], b = sf[1];
            int zo = z[1];
#pragma unroll
            for (int i = 1; i < D; i++)
              if (k == i) { a = p[i]; b = sf[i + 1]; zo = z[1 + i]; }
            const REAL dv = *reinterpret_cast<const REAL*>(smem_raw + (db[q] + zo));
            dacc[q] += (double)(dv * a * b) * wj;
          }
      }
    }
  }
#pragma unroll
  for (int m = 0; m < RPT; m++)
    if (r0 + (int64_t)m * PR_THREADS < R) part[(int64_t)blockIdx.y * R + r0 + (int64_t)m * PR_THREADS] = acc[m];
  if (ND && r0 < R)
#pragma unroll
    for (int q = 0; q < ND; q++)
      if (q < rf.nW) dpart[((int64_t)blockIdx.y * R + r0) * rf.nW + q] = dacc[q];
}

__global__ void k_sum_slices(const double* part, int nsl, int64_t n, double* out) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    double s = 0.0;
    for (int y = 0; y < nsl; y++) s += part[(int64_t)y * n + i];
    out[i] = s;
  }
}

// out[r, j] = S(ZA_r, ZB_j); with out_m, also the product over the units whose bit in dep_units is clear (the
// marginal of the columns outside the dep mask, from the same lookups)
template <typename REAL, typename OUT>
__global__ void k_cols(ColMeta cm, const REAL* T, const REAL* RT, const int64_t* ZA, int64_t R, const int64_t* ZB,
                       int64_t M, OUT* out, OUT* out_m, unsigned dep_units) {
  for (int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < R * M;
       idx += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = idx / M, j = idx % M;
    int64_t za[MAXD], zb[MAXD], r2[MAXG]; bool tor[MAXG];
    REAL fac[MAXU];
    for (int u = 0; u < MAXU; u++) fac[u] = REAL(1);
    for (int k = 0; k < cm.d; k++) { za[k] = ZA[r * cm.d + k]; zb[k] = ZB[j * cm.d + k]; }
    pair_factors<REAL>(cm, T, RT, za, zb, fac, r2, tor);
    REAL v = REAL(1), vdep = REAL(1);
    for (int u = 0; u < cm.U; u++) {
      if ((dep_units >> u) & 1u) vdep *= fac[u];
      else v *= fac[u];
    }
    out[idx] = (OUT)(v * vdep);
    if (out_m) out_m[idx] = (OUT)v;
  }
}

// lattice coordinates of bin centres: round(Z / h) in float64, ties to even (np.round's rule, so bit-exact with it)
__global__ void k_lattice_coords(const double* Z, int64_t n, int d, const double* h, int64_t* out) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n * d; i += (int64_t)gridDim.x * blockDim.x)
    out[i] = (int64_t)rint(Z[i] / h[i % d]);
}

// per column: min and max of ZA and ZB (for the extent check); out[4 * k + {0,1,2,3}] = minA, maxA, minB, maxB
__global__ void k_coord_range(const int64_t* ZA, int64_t R, const int64_t* ZB, int64_t M, int d, long long* out) {
  const int k = blockIdx.x;
  long long mnA = LLONG_MAX, mxA = LLONG_MIN, mnB = LLONG_MAX, mxB = LLONG_MIN;
  for (int64_t i = threadIdx.x; i < R; i += blockDim.x) { long long v = ZA[i * d + k]; mnA = min(mnA, v); mxA = max(mxA, v); }
  for (int64_t i = threadIdx.x; i < M; i += blockDim.x) { long long v = ZB[i * d + k]; mnB = min(mnB, v); mxB = max(mxB, v); }
  __shared__ long long sh[4][256];
  sh[0][threadIdx.x] = mnA; sh[1][threadIdx.x] = mxA; sh[2][threadIdx.x] = mnB; sh[3][threadIdx.x] = mxB;
  __syncthreads();
  for (int s = blockDim.x / 2; s > 0; s >>= 1) {
    if ((int)threadIdx.x < s) {
      sh[0][threadIdx.x] = min(sh[0][threadIdx.x], sh[0][threadIdx.x + s]);
      sh[1][threadIdx.x] = max(sh[1][threadIdx.x], sh[1][threadIdx.x + s]);
      sh[2][threadIdx.x] = min(sh[2][threadIdx.x], sh[2][threadIdx.x + s]);
      sh[3][threadIdx.x] = max(sh[3][threadIdx.x], sh[3][threadIdx.x + s]);
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) for (int q = 0; q < 4; q++) out[4 * k + q] = sh[q][0];
}

// The same ranges with the table metadata, for one read-back: blocks take strided elements with a fixed column per
// thread (coalesced rows), their ranges go to part[block][4 d], and k_rows_meta joins them behind a copy of the metadata
// arrays (MetaList's, in order).
constexpr int kRangeBlocks = 64;
__global__ void __launch_bounds__(256) k_rows_ranges(const int64_t* ZA, int64_t R, const int64_t* ZB, int64_t M, int d,
                                                     long long* part) {
  __shared__ long long sh[4][256];
  const int T = 256 / d * d, tid = threadIdx.x;
  long long v[4] = {LLONG_MAX, LLONG_MIN, LLONG_MAX, LLONG_MIN};
  if (tid < T) {
    for (int64_t e = (int64_t)blockIdx.x * T + tid; e < R * d; e += (int64_t)gridDim.x * T) {
      const long long z = ZA[e]; v[0] = min(v[0], z); v[1] = max(v[1], z);
    }
    if (ZB == ZA && M == R) { v[2] = v[0]; v[3] = v[1]; }
    else
      for (int64_t e = (int64_t)blockIdx.x * T + tid; e < M * d; e += (int64_t)gridDim.x * T) {
        const long long z = ZB[e]; v[2] = min(v[2], z); v[3] = max(v[3], z);
      }
  }
  for (int q = 0; q < 4; q++) sh[q][tid] = v[q];
  __syncthreads();
  if (tid < 4 * d) {
    const int k = tid / 4, q = tid - 4 * k;
    long long x = sh[q][k];
    for (int i = k + d; i < T; i += d) x = (q & 1) ? max(x, sh[q][i]) : min(x, sh[q][i]);
    part[(int64_t)blockIdx.x * 4 * d + tid] = x;
  }
}

struct MetaList { const int64_t* src[12]; int n[12]; };
__global__ void __launch_bounds__(256) k_rows_meta(MetaList ml, const long long* part, int d, long long* out) {
  const int tid = threadIdx.x;
  if (tid < 4 * d) {                     // out[0 .. 4 d): min / max of ZA, min / max of ZB per column
    long long x = part[tid];
    for (int b = 1; b < kRangeBlocks; b++) {
      const long long y = part[b * 4 * d + tid];
      x = (tid & 1) ? max(x, y) : min(x, y);
    }
    out[tid] = x;
  }
  int at = 4 * d;
  for (int q = 0; q < 12; q++) {
    if (tid < ml.n[q]) out[at + tid] = ml.src[q][tid];
    at += ml.n[q];
  }
}

}  // namespace blml

using namespace blml;

// the metadata arrays of a table set, in the order both read-backs use
static int meta_list(const blml_tables* tb, MetaList& ml) {
  if (!tb || tb->d < 1 || tb->d > MAXD || tb->U < 1 || tb->U > MAXU || tb->G < 0 || tb->G > MAXG || tb->nW < 0 ||
      tb->nW > MAXW) {
    set_error("pair tables: d <= %d, units <= %d, groups <= %d, derivative entries <= %d", MAXD, MAXU, MAXG, MAXW);
    return BLML_ERR_ARG;
  }
  const int d = tb->d;
  const int64_t* src[12] = {tb->kinds, tb->base, tb->Jk, tb->mk, tb->nbins, tb->grp, tb->dim_unit, tb->grp_unit,
                            tb->wunit, tb->wcol, tb->wgrp, tb->dbase};
  const int n[12] = {d, d, d, d, d, d, d, tb->G, tb->nW, tb->nW, tb->nW, tb->nW};
  for (int q = 0; q < 12; q++) {
    if (n[q] && !src[q]) { set_error("pair tables: a metadata array is missing"); return BLML_ERR_ARG; }
    ml.src[q] = src[q]; ml.n[q] = n[q];
  }
  return BLML_OK;
}

// the metadata (meta_list's arrays one after another) checked into cm
static int parse_meta(const blml_tables* tb, const int64_t* v, ColMeta& cm) {
  const int d = tb->d;
  cm.d = d; cm.U = tb->U; cm.G = tb->G; cm.nW = tb->nW; cm.LR = tb->LR;
  cm.Tn = tb->nT; cm.dTn = tb->ndT;
  const int64_t *codes = v, *base = v + d, *J = v + 2 * d, *mk = v + 3 * d, *nb = v + 4 * d, *grp = v + 5 * d,
                *du = v + 6 * d, *gu = v + 7 * d, *wu = gu + tb->G, *wc = wu + tb->nW, *wg = wc + tb->nW, *db = wg + tb->nW;
  for (int k = 0; k < d; k++) {
    cm.code[k] = (int)codes[k]; cm.base[k] = base[k]; cm.J[k] = J[k]; cm.mk[k] = mk[k]; cm.nb[k] = nb[k];
    cm.grp[k] = (int)grp[k]; cm.dim_unit[k] = (int)du[k];
    if (codes[k] < 0 || codes[k] > 4) { set_error("pair tables: column %d has kind code %lld", k, (long long)codes[k]); return BLML_ERR_ARG; }
    if ((codes[k] == 2 || codes[k] == 4) && (grp[k] < 0 || grp[k] >= tb->G)) { set_error("pair tables: column %d group", k); return BLML_ERR_ARG; }
    if (!(codes[k] == 2 || codes[k] == 4) && (du[k] < 0 || du[k] >= tb->U)) { set_error("pair tables: column %d unit", k); return BLML_ERR_ARG; }
  }
  for (int k = 0; k < d; k++) {              // every column block lies inside the flat value array
    int64_t len = 0;
    if (cm.code[k] == 0) len = 2 * cm.J[k] + 1;
    else if (cm.code[k] == 3) len = cm.mk[k] * cm.mk[k];
    else if (cm.code[k] == 1) len = cm.nb[k] / 2 + 1;
    if (cm.base[k] < 0 || cm.base[k] + len > cm.Tn || cm.J[k] < 0 || cm.mk[k] < 0 || cm.nb[k] < 0) {
      set_error("pair tables: column %d block outside the value array of %lld", k, (long long)cm.Tn);
      return BLML_ERR_ARG;
    }
  }
  for (int g = 0; g < tb->G; g++) {
    cm.grp_unit[g] = (int)gu[g];
    if (gu[g] < 0 || gu[g] >= tb->U) { set_error("pair tables: group %d unit", g); return BLML_ERR_ARG; }
  }
  for (int q = 0; q < tb->nW; q++) {
    cm.wunit[q] = (int)wu[q]; cm.wcol[q] = (int)wc[q]; cm.wgrp[q] = (int)wg[q]; cm.dbase[q] = db[q];
    bool ok = wu[q] >= 0 && wu[q] < tb->U && wg[q] < tb->G && wc[q] < d;
    if (ok && wg[q] < 0) {                   // a column's derivative row: inside dT, with the column's block length
      const int k = (int)wc[q];
      ok = k >= 0 && (cm.code[k] == 0 || cm.code[k] == 3) && db[q] >= 0 &&
           db[q] + (cm.code[k] == 3 ? cm.mk[k] * cm.mk[k] : 2 * cm.J[k] + 1) <= cm.dTn;
    }
    if (!ok) { set_error("pair tables: derivative entry %d outside its tables", q); return BLML_ERR_ARG; }
  }
  return BLML_OK;
}

constexpr int kMetaMax = 7 * MAXD + MAXG + 4 * MAXW;

static int read_meta(const blml_tables* tb, ColMeta& cm, cudaStream_t st) {
  MetaList ml;
  int e = meta_list(tb, ml);
  if (e) return e;
  int64_t v[kMetaMax];
  int at = 0;
  for (int q = 0; q < 12; q++) {
    if (ml.n[q]) e = cuda_status(cudaMemcpyAsync(v + at, ml.src[q], ml.n[q] * sizeof(int64_t), cudaMemcpyDeviceToHost, st), "pair tables");
    if (e) return e;
    at += ml.n[q];
  }
  e = cuda_status(cudaStreamSynchronize(st), "pair tables");
  return e ? e : parse_meta(tb, v, cm);
}

// the per-column coordinate ranges hr[4 k + (0..3)] = min / max of ZA, min / max of ZB against the tables' extents:
// offsets within +-J (offset rows), ranks within the rank table, folded coordinates within the period (circular /
// torus), radii within the radial row
static int extents_ok(const ColMeta& cm, const long long* hr) {
  double rad[MAXG] = {0, 0, 0, 0};
  for (int k = 0; k < cm.d; k++) {
    const long long mnA = hr[4 * k], mxA = hr[4 * k + 1], mnB = hr[4 * k + 2], mxB = hr[4 * k + 3];
    const long long span = std::max(mxA - mnB, mxB - mnA);
    bool ok = true;
    switch (cm.code[k]) {
      case 0: ok = span <= cm.J[k]; break;
      case 3: ok = mnA >= 0 && mnB >= 0 && mxA < cm.mk[k] && mxB < cm.mk[k]; break;
      case 1: case 4: ok = mnA >= 0 && mnB >= 0 && mxA < cm.nb[k] && mxB < cm.nb[k]; break;
      case 2: rad[cm.grp[k]] += (double)span * (double)span; break;
    }
    if (!ok) {
      set_error("pair tables: column %d coordinates outside the tables' span (stale tables)", k);
      return BLML_ERR_ARG;
    }
  }
  for (int k = 0; k < cm.d; k++)
    if (cm.code[k] == 2 && sqrt(rad[cm.grp[k]]) * RQ + 1 >= cm.LR) {
      set_error("pair tables: radial group %d radius outside its row (stale tables)", cm.grp[k]);
      return BLML_ERR_ARG;
    }
  return BLML_OK;
}

// the coordinates must lie in the tables' extents: offsets within +-J (offset rows), ranks within the rank table,
// folded coordinates within the period (circular / torus), radii within the radial row
static int check_extents(const ColMeta& cm, const int64_t* ZA, int64_t R, const int64_t* ZB, int64_t M,
                         cudaStream_t st, long long* ranges = nullptr) {
  if (R == 0 || M == 0) return BLML_OK;
  long long* dr = nullptr;
  long long hr[4 * MAXD];
  int e = cuda_status(cudaMallocAsync((void**)&dr, 4 * cm.d * sizeof(long long), st), "pair extents");
  if (e) return e;
  k_coord_range<<<cm.d, 256, 0, st>>>(ZA, R, ZB, M, cm.d, dr);
  count_launches(1);
  e = cuda_status(cudaMemcpyAsync(hr, dr, 4 * cm.d * sizeof(long long), cudaMemcpyDeviceToHost, st), "pair extents");
  cudaFreeAsync(dr, st);
  if (!e) e = cuda_status(cudaStreamSynchronize(st), "pair extents");
  if (e) return e;
  if (ranges)
    for (int i = 0; i < 4 * cm.d; i++) ranges[i] = hr[i];
  return extents_ok(cm, hr);
}

// column slices of a rows launch (R, M >= 1): about 16 blocks of 128 rows per SM, at least 256 columns each, whichever kernel
// runs. 4 blocks per SM and 1,024 columns were slower for each, though a block of the general and multi-density kernels copies
// all tables for its slice (us, float64, three-column bins by themselves; 600, 3,000, 12,000 bins): a ball of three columns
// 694, 1,194, 2,385 -> 236, 314, 1,955, with tables of 133 KB 705, 1,199, 4,399 -> 239, 379, 4,182; pball x sinc 726, 1,260,
// 2,752 -> 247, 329, 2,380; three densities of ball x sinc 1,094, 1,875, 4,105 -> 372, 485, 2,660. The partials: at most
// 16 x 148 x 128 + R sums a density or derivative entry.
static void rows_slices(int64_t R, int64_t M, int64_t& nsl, int64_t& slice, int64_t most = 65535) {
  const int64_t rblocks = (R + PR_THREADS - 1) / PR_THREADS;
  nsl = std::max<int64_t>(1, std::min<int64_t>((16 * 148 + rblocks - 1) / rblocks, (M + 255) / 256));
  nsl = std::min<int64_t>(nsl, most);
  slice = (M + nsl - 1) / nsl;
  nsl = (M + slice - 1) / slice;
}

// the fast kernel's tables; false when a column or derivative entry needs the general kernel (groups, units that are not
// one column each, tables past shared memory)
static bool rows_fast(const ColMeta& cm, const long long* hr, int grad, size_t es, RowsFast& rf) {
  if (cm.G || cm.U != cm.d) return false;
  int pos_of[MAXD], seen = 0;
  for (int k = 0; k < cm.d; k++) {
    if (cm.dim_unit[k] >= cm.d || ((seen >> cm.dim_unit[k]) & 1)) return false;
    seen |= 1 << cm.dim_unit[k]; pos_of[k] = cm.dim_unit[k];
  }
  rf = RowsFast{};
  int64_t total = 0;
  for (int k = 0; k < cm.d; k++) {
    const int p = pos_of[k], code = cm.code[k];
    if (code != 0 && code != 1 && code != 3) return false;
    if (code == 1 && cm.nb[k] < 1) return false;
    const int64_t len = code == 0 ? 2 * cm.J[k] + 1 : code == 1 ? 2 * cm.nb[k] - 1 : cm.mk[k] * cm.mk[k];
    rf.col[p] = k; rf.kind[p] = code; rf.base[p] = (int)cm.base[k]; rf.nb[p] = (int)cm.nb[k];
    rf.so[p] = (int)total; rf.len[p] = (int)len;
    rf.org[p] = code == 0 ? (int)cm.J[k] : code == 1 ? (int)cm.nb[k] - 1 : 0;
    rf.mul[p] = code == 3 ? (int)cm.mk[k] : 1;
    rf.zmin[p] = code == 3 ? 0 : hr[4 * k + 2];
    total += len;
    if (total * (int64_t)es > 220 * 1024) return false;
  }
  if (grad) {
    rf.nW = cm.nW;
    for (int q = 0; q < cm.nW; q++) {
      const int k = cm.wcol[q];
      if (cm.wgrp[q] >= 0 || k < 0 || cm.wunit[q] != cm.dim_unit[k] || cm.code[k] == 1) return false;
      rf.dpos[q] = pos_of[k]; rf.dbase[q] = (int)cm.dbase[q]; rf.dso[q] = (int)total; rf.dlen[q] = rf.len[pos_of[k]];
      total += rf.dlen[q];
      if (total * (int64_t)es > 220 * 1024) return false;
    }
  }
  rf.total = (int)total;
  return true;
}

// the launch of the rows kernel that serves cm: values and, with grad, derivative partials per slice
template <typename REAL>
static int rows_launch(const ColMeta& cm, const long long* hr, const REAL* T, const REAL* RT, const REAL* dT,
                       const REAL* dR, const int64_t* ZA, int64_t R, const int64_t* ZB, int64_t M, const double* w,
                       int grad, int64_t nsl, int64_t slice, double* part, double* dpart, cudaStream_t st,
                       const char* who) {
  bool offset_only = cm.G == 0 && !grad;
  for (int k = 0; k < cm.d; k++) offset_only = offset_only && cm.code[k] == 0;
  const size_t tsz = (size_t)cm.Tn * sizeof(REAL);
  if (offset_only && align16(tsz) + align16((size_t)PR_CHUNK * cm.d * sizeof(int)) + PR_CHUNK * sizeof(double) > 200 * 1024) {
    set_error("%s: tables too large for shared memory", who); return BLML_ERR_UNSUPPORTED;
  }
  if (tsz + (size_t)cm.G * cm.LR * sizeof(REAL) > 200 * 1024) {
    set_error("%s: tables too large for shared memory", who); return BLML_ERR_UNSUPPORTED;
  }
  RowsFast rf;
  if (rows_fast(cm, hr, grad, sizeof(REAL), rf) && rf_smem<REAL>(rf.total, cm.d) <= 224 * 1024) {
    const size_t sm = rf_smem<REAL>(rf.total, cm.d);
    // two rows per thread share a column's offsets and weight while that still leaves 4 blocks per SM
    const bool two = !grad && (R + 2 * PR_THREADS - 1) / (2 * PR_THREADS) * nsl >= 4 * 148;
    auto run = [&](auto kern, int rpt) -> int {
      if (sm > 48 * 1024) {
        const int e = cuda_status(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm), who);
        if (e) return e;
      }
      const dim3 grid((unsigned)((R + PR_THREADS * rpt - 1) / (PR_THREADS * rpt)), (unsigned)nsl);
      kern<<<grid, PR_THREADS, sm, st>>>(rf, T, dT, ZA, R, ZB, w, slice, M, part, dpart);
      return BLML_OK;
    };
#define ROWS_FAST(DD) case DD: \
      return !grad ? (two ? run(k_rows_fast<REAL, DD, 2, 0>, 2) : run(k_rows_fast<REAL, DD, 1, 0>, 1)) \
                   : cm.nW <= 4 ? run(k_rows_fast<REAL, DD, 1, 4>, 1) : run(k_rows_fast<REAL, DD, 1, 8>, 1);
    switch (cm.d) { ROWS_FAST(1) ROWS_FAST(2) ROWS_FAST(3) ROWS_FAST(4) ROWS_FAST(5) ROWS_FAST(6) ROWS_FAST(7) ROWS_FAST(8) }
#undef ROWS_FAST
  }
  const size_t sm = tsz + (size_t)cm.G * cm.LR * sizeof(REAL);
  const dim3 grid((unsigned)((R + PR_THREADS - 1) / PR_THREADS), (unsigned)nsl);
  if (grad) {
    cudaFuncSetAttribute(k_rows_general<REAL, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    k_rows_general<REAL, true><<<grid, PR_THREADS, sm, st>>>(cm, T, RT, dT, dR, ZA, R, ZB, w, 0, slice, M, part, dpart);
  } else {
    cudaFuncSetAttribute(k_rows_general<REAL, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    k_rows_general<REAL, false><<<grid, PR_THREADS, sm, st>>>(cm, T, RT, dT, dR, ZA, R, ZB, w, 0, slice, M, part, dpart);
  }
  return BLML_OK;
}

// ws: the slice partials (nsl R (1 + nW) doubles)
template <typename REAL>
static int rows_impl(const ColMeta& cm, const long long* hr, const REAL* T, const REAL* RT, const REAL* dT,
                     const REAL* dR, const int64_t* ZA, int64_t R, const int64_t* ZB, int64_t M, const double* w,
                     int grad, double* s, double* ds, cudaStream_t st, double* part) {
  int64_t nsl, slice;
  rows_slices(R, M, nsl, slice);
  const int nW = grad ? cm.nW : 0;
  double* dpart = part + (size_t)nsl * R;
  int e = rows_launch<REAL>(cm, hr, T, RT, dT, dR, ZA, R, ZB, M, w, grad, nsl, slice, part, dpart, st, "blml_rows");
  if (!e) e = cuda_status(cudaGetLastError(), "blml_rows");
  if (e) return e;
  count_launches(2);                         // the rows kernel and the slice sum
  k_sum_slices<<<std::min<int64_t>((R + 255) / 256, 4096), 256, 0, st>>>(part, (int)nsl, R, s);
  if (nW) {
    k_sum_slices<<<std::min<int64_t>((R * nW + 255) / 256, 4096), 256, 0, st>>>(dpart, (int)nsl, R * nW, ds);
    count_launches(1);
  }
  return cuda_status(cudaGetLastError(), "blml_rows finish");
}

// device scratch of a rows call: the read-back block, then the slice partials
constexpr int64_t kPrepBytes = ((kRangeBlocks + 1) * 4 * MAXD + kMetaMax) * (int64_t)sizeof(long long);

static int64_t rows_bytes(int64_t R, int64_t M, int nW) {
  int64_t nsl, slice;
  rows_slices(R, M, nsl, slice);
  return (kPrepBytes + 255) / 256 * 256 + nsl * R * (1 + nW) * (int64_t)sizeof(double);
}

// metadata and coordinate ranges in one read-back (prep: kPrepBytes of device scratch), both checked
static int rows_prepare(const blml_tables* tb, const int64_t* ZA, int64_t R, const int64_t* ZB, int64_t M, void* prep,
                        ColMeta& cm, long long* hr, cudaStream_t st) {
  MetaList ml;
  int e = meta_list(tb, ml);
  if (e) return e;
  const int d = tb->d;
  long long* part = reinterpret_cast<long long*>(prep);
  long long* out = part + (int64_t)kRangeBlocks * 4 * MAXD;
  k_rows_ranges<<<kRangeBlocks, 256, 0, st>>>(ZA, R, ZB, M, d, part);
  k_rows_meta<<<1, 256, 0, st>>>(ml, part, d, out);
  count_launches(2);
  long long v[4 * MAXD + kMetaMax];
  int n = 4 * d;
  for (int q = 0; q < 12; q++) n += ml.n[q];
  e = cuda_status(cudaMemcpyAsync(v, out, n * sizeof(long long), cudaMemcpyDeviceToHost, st), "pair tables");
  if (!e) e = cuda_status(cudaStreamSynchronize(st), "pair tables");
  if (!e) e = parse_meta(tb, reinterpret_cast<const int64_t*>(v + 4 * d), cm);
  if (e) return e;
  for (int i = 0; i < 4 * d; i++) hr[i] = v[i];
  return extents_ok(cm, hr);
}

static int rows_tables_ok(const blml_tables* tb, const ColMeta& cm, int grad) {
  if (tb->f32 ? (!tb->T32 || (cm.G && !tb->RT32) || (grad && (!tb->dT32 || !tb->dR32)))
              : (!tb->T || (cm.G && !tb->RT) || (grad && (!tb->dT || !tb->dR)))) {
    set_error(tb->f32 ? "blml_rows: float32 tables missing" : "blml_rows: tables missing");
    return BLML_ERR_ARG;
  }
  return BLML_OK;
}

extern "C" {

// a rows plan: the tables' metadata read and the coordinates' extents checked once, for many value-row passes over
// rows of the same coordinate set (the block coordinate descent's passes of every bin against a block)
struct blml_rows_plan_s {
  blml_tables tb;
  ColMeta cm;
  long long hr[4 * MAXD];                // the coordinate set's ranges
};

int blml_rows_plan_create(const blml_tables* tb, const int64_t* Z, int64_t n, void* stream, blml_rows_plan* out) {
  if (!tb || !out || n < 0 || (n > 0 && !Z)) { set_error("blml_rows_plan_create: bad arguments"); return BLML_ERR_ARG; }
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  blml_rows_plan_s* p = new blml_rows_plan_s();
  p->tb = *tb;
  int e = read_meta(tb, p->cm, st);
  for (auto& x : p->hr) x = 0;
  if (!e && n > 0) e = check_extents(p->cm, Z, n, Z, n, st, p->hr);   // every pair within Z: min / max per column
  if (!e && (tb->f32 ? (!tb->T32 || (p->cm.G && !tb->RT32)) : (!tb->T || (p->cm.G && !tb->RT)))) {
    set_error("blml_rows_plan_create: value tables missing"); e = BLML_ERR_ARG;
  }
  if (e) { delete p; return e; }
  *out = p;
  return BLML_OK;
}

int64_t blml_rows_plan_workspace(blml_rows_plan p, int64_t R, int64_t M) {
  if (!p || R < 0 || M < 1) return -1;
  if (R == 0) return 0;
  int64_t nsl, slice;
  rows_slices(R, M, nsl, slice);
  return nsl * R * (int64_t)sizeof(double);
}

int blml_rows_plan_run(blml_rows_plan p, const int64_t* ZA, int64_t R, const int64_t* ZB, int64_t M, const double* w,
                       double* s, void* ws, int64_t ws_bytes, void* stream) {
  if (!p || R < 0 || M < 0) { set_error("blml_rows_plan_run: bad arguments"); return BLML_ERR_ARG; }
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  if (R == 0) return BLML_OK;
  if (M == 0) return cuda_status(cudaMemsetAsync(s, 0, R * sizeof(double), st), "blml_rows_plan_run");
  const int64_t need = blml_rows_plan_workspace(p, R, M);
  if (!ws || ws_bytes < need) {
    set_error("blml_rows_plan_run: workspace of %lld bytes, need %lld", (long long)ws_bytes, (long long)need);
    return BLML_ERR_WORKSPACE;
  }
  const blml_tables* tb = &p->tb;
  double* part = reinterpret_cast<double*>(ws);
  if (tb->f32)
    return rows_impl<float>(p->cm, p->hr, tb->T32, tb->RT32, nullptr, nullptr, ZA, R, ZB, M, w, 0, s, nullptr, st, part);
  return rows_impl<double>(p->cm, p->hr, tb->T, tb->RT, nullptr, nullptr, ZA, R, ZB, M, w, 0, s, nullptr, st, part);
}

int blml_rows_plan_destroy(blml_rows_plan p) {
  delete p;
  return BLML_OK;
}

int64_t blml_rows_workspace(int64_t R, int64_t M, int nW) {
  return R < 1 || M < 1 || nW < 0 ? 0 : rows_bytes(R, M, nW);
}

int blml_rows_ws(const blml_tables* tb, const int64_t* ZA, int64_t R, const int64_t* ZB, int64_t M, const double* w,
                 int grad, double* s, double* ds, void* ws, int64_t ws_bytes, void* stream) {
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  if (!tb || R < 0 || M < 0) { set_error("blml_rows: no tables, or a negative count of rows or columns"); return BLML_ERR_ARG; }
  ColMeta cm;
  if (R == 0 || M == 0) {                    // nothing to sum: the tables are checked all the same
    const int e = read_meta(tb, cm, st);
    if (e || R == 0) return e;
    return cuda_status(cudaMemsetAsync(s, 0, R * sizeof(double), st), "blml_rows");
  }
  if (tb->nW == 0) grad = 0;
  const int64_t need = rows_bytes(R, M, grad ? tb->nW : 0);
  if (!ws || ws_bytes < need) {
    set_error("blml_rows: workspace of %lld bytes, need %lld", (long long)ws_bytes, (long long)need);
    return BLML_ERR_WORKSPACE;
  }
  long long hr[4 * MAXD];
  int e = rows_prepare(tb, ZA, R, ZB, M, ws, cm, hr, st);
  if (!e) e = rows_tables_ok(tb, cm, grad);
  if (e) return e;
  double* part = reinterpret_cast<double*>(reinterpret_cast<char*>(ws) + (kPrepBytes + 255) / 256 * 256);
  if (tb->f32) return rows_impl<float>(cm, hr, tb->T32, tb->RT32, tb->dT32, tb->dR32, ZA, R, ZB, M, w, grad, s, ds, st, part);
  return rows_impl<double>(cm, hr, tb->T, tb->RT, tb->dT, tb->dR, ZA, R, ZB, M, w, grad, s, ds, st, part);
}

int blml_rows(const blml_tables* tb, const int64_t* ZA, int64_t R, const int64_t* ZB, int64_t M, const double* w,
              int grad, double* s, double* ds, void* stream) {
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  if (R <= 0 || M <= 0 || !tb) return blml_rows_ws(tb, ZA, R, ZB, M, w, grad, s, ds, nullptr, 0, stream);
  void* ws = nullptr;
  const int64_t need = rows_bytes(R, M, grad && tb->nW > 0 ? tb->nW : 0);
  int e = cuda_status(cudaMallocAsync(&ws, need, st), "blml_rows workspace");
  if (e) return e;
  e = blml_rows_ws(tb, ZA, R, ZB, M, w, grad, s, ds, ws, need, stream);
  cudaFreeAsync(ws, st);
  return e;
}

}  // extern "C"

template <typename REAL>
static int rows_multi_impl(const ColMeta& cm, const REAL* T, const REAL* RT, const int64_t* ZA, int64_t R,
                           const int64_t* ZB, int64_t M, const double* W, int Mm, const DensMasks& dm, double* s,
                           cudaStream_t st) {
  const int64_t rblocks = (R + PR_THREADS - 1) / PR_THREADS;
  int64_t nsl, slice;
  rows_slices(R, M, nsl, slice);
  double* part = nullptr;
  int e = cuda_status(cudaMallocAsync((void**)&part, std::max<size_t>((size_t)nsl * R * Mm * sizeof(double), 8), st),
                      "blml_rows_multi workspace");
  if (e) return e;
  const size_t sm = (size_t)cm.Tn * sizeof(REAL) + (size_t)cm.G * cm.LR * sizeof(REAL);
  if (sm > 200 * 1024) { cudaFreeAsync(part, st); set_error("blml_rows_multi: tables too large for shared memory"); return BLML_ERR_UNSUPPORTED; }
  cudaFuncSetAttribute(k_rows_multi<REAL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  k_rows_multi<REAL><<<dim3((unsigned)rblocks, (unsigned)nsl), PR_THREADS, sm, st>>>(cm, T, RT, ZA, R, ZB, W, Mm, dm,
                                                                                   slice, M, part);
  e = cuda_status(cudaGetLastError(), "blml_rows_multi");
  if (!e) {
    count_launches(2);
    k_sum_slices<<<std::min<int64_t>((R * Mm + 255) / 256, 4096), 256, 0, st>>>(part, (int)nsl, R * Mm, s);
    e = cuda_status(cudaGetLastError(), "blml_rows_multi finish");
  }
  cudaFreeAsync(part, st);
  return e;
}

extern "C" {

int blml_rows_multi(const blml_tables* tb, const int64_t* ZA, int64_t R, const int64_t* ZB, int64_t M,
                    const double* W, int Mm, const unsigned* umask, double* s, void* stream) {
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  if (Mm < 1 || Mm > MAXM || !umask) { set_error("blml_rows_multi: 1 to %d densities with a unit mask each", MAXM); return BLML_ERR_ARG; }
  if (R < 0 || M < 0) { set_error("blml_rows_multi: a negative count of rows or columns"); return BLML_ERR_ARG; }
  ColMeta cm;
  int e = read_meta(tb, cm, st);
  if (e) return e;
  DensMasks dm;
  for (int m = 0; m < MAXM; m++) dm.bits[m] = m < Mm ? umask[m] : 0u;
  for (int m = 0; m < Mm; m++)
    if (dm.bits[m] >> cm.U) { set_error("blml_rows_multi: density %d masks a unit beyond the tables' %d", m, cm.U); return BLML_ERR_ARG; }
  if (R == 0) return BLML_OK;
  if (M == 0) return cuda_status(cudaMemsetAsync(s, 0, R * Mm * sizeof(double), st), "blml_rows_multi");
  if (!ZA || !ZB || !W || !s) { set_error("blml_rows_multi: null pointer"); return BLML_ERR_ARG; }
  e = check_extents(cm, ZA, R, ZB, M, st);
  if (e) return e;
  if (tb->f32) {
    if (!tb->T32 || (cm.G && !tb->RT32)) { set_error("blml_rows_multi: float32 tables missing"); return BLML_ERR_ARG; }
    return rows_multi_impl<float>(cm, tb->T32, tb->RT32, ZA, R, ZB, M, W, Mm, dm, s, st);
  }
  if (!tb->T || (cm.G && !tb->RT)) { set_error("blml_rows_multi: tables missing"); return BLML_ERR_ARG; }
  return rows_multi_impl<double>(cm, tb->T, tb->RT, ZA, R, ZB, M, W, Mm, dm, s, st);
}

}  // extern "C"

// ---- blml_rows_noalloc: the value rows with a fixed scratch array instead of any device allocation ----
// Its scratch (the per-column coordinate ranges of the extent check, then the column-slice partial sums) lives in
// this file-scope device array: 4 MiB on every GPU that loads the library, held until the process exits. Host code
// must not pass the symbol itself to a kernel (on the host it names a stand-in, not device memory): the device
// address comes from cudaGetSymbolAddress, taken once per device with that device current, on the first call (and
// again if the device's context has changed since).
constexpr int64_t kRowsScratchDoubles = (int64_t)1 << 19;       // 4 MiB
constexpr int64_t kRowsScratchRangeSlots = 64;                   // 4 * d <= 32 range words, padded to 512 bytes
constexpr int64_t kRowsNoAllocMaxR = kRowsScratchDoubles - kRowsScratchRangeSlots;
static __device__ __align__(256) double g_rows_scratch[kRowsScratchDoubles];

static int rows_scratch(double** out) {
  int dev = 0;
  int e = cuda_status(cudaGetDevice(&dev), "blml_rows_noalloc");
  if (e) return e;
  if (dev < 0 || dev >= 64) { set_error("blml_rows_noalloc: device ordinal %d above 63", dev); return BLML_ERR_ARG; }
  // the address belongs to the device's current context: taken again when that context is not the one it was
  // taken in (after a cudaDeviceReset, or under another context)
  // cuCtxGetCurrent through the runtime's driver entry point, so that the library needs no link to libcuda and
  // loads on a host without a driver
  using CtxGetFn = CUresult (*)(CUcontext*);
  static CtxGetFn ctx_get = []() -> CtxGetFn {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      return reinterpret_cast<CtxGetFn>(p);
    return nullptr;
  }();
  CUcontext ctx = nullptr;
  if (!ctx_get || ctx_get(&ctx) != CUDA_SUCCESS) {
    set_error("blml_rows_noalloc: no current context"); return BLML_ERR_CUDA;
  }
  static std::mutex mu;
  static double* ptrs[64] = {nullptr};
  static CUcontext ctxs[64] = {nullptr};
  std::lock_guard<std::mutex> lock(mu);
  if (!ptrs[dev] || ctxs[dev] != ctx) {
    void* p = nullptr;
    e = cuda_status(cudaGetSymbolAddress(&p, g_rows_scratch), "blml_rows_noalloc scratch address");
    if (e) return e;
    ptrs[dev] = reinterpret_cast<double*>(p); ctxs[dev] = ctx;
  }
  *out = ptrs[dev];
  return BLML_OK;
}

template <typename REAL>
static int rows_noalloc_launch(const ColMeta& cm, const long long* hr, const REAL* T, const REAL* RT, const int64_t* ZA,
                               int64_t R, const int64_t* ZB, int64_t M, const double* w, double* part, double* s,
                               cudaStream_t st) {
  int64_t nsl, slice;
  rows_slices(R, M, nsl, slice, std::max<int64_t>(1, kRowsNoAllocMaxR / R));
  int e = rows_launch<REAL>(cm, hr, T, RT, nullptr, nullptr, ZA, R, ZB, M, w, 0, nsl, slice, part, nullptr, st,
                            "blml_rows_noalloc");
  if (!e) e = cuda_status(cudaGetLastError(), "blml_rows_noalloc");
  if (e) return e;
  k_sum_slices<<<std::min<int64_t>((R + 255) / 256, 4096), 256, 0, st>>>(part, (int)nsl, R, s);
  count_launches(2);
  return cuda_status(cudaGetLastError(), "blml_rows_noalloc finish");
}

extern "C" {

int blml_rows_noalloc(const blml_tables* tb, const int64_t* ZA, int64_t R, const int64_t* ZB, int64_t M,
                      const double* w, double* s, void* stream) {
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  ColMeta cm;
  int e = read_meta(tb, cm, st);
  if (e) return e;
  if (R < 0 || M < 0) { set_error("blml_rows_noalloc: negative sizes"); return BLML_ERR_ARG; }
  if (R > kRowsNoAllocMaxR) {
    set_error("blml_rows_noalloc: %lld rows exceed the fixed scratch (at most %lld rows)", (long long)R,
              (long long)kRowsNoAllocMaxR);
    return BLML_ERR_ARG;
  }
  if (R == 0) return BLML_OK;
  if (M == 0) return cuda_status(cudaMemsetAsync(s, 0, R * sizeof(double), st), "blml_rows_noalloc");
  double* scratch = nullptr;
  e = rows_scratch(&scratch);
  if (e) return e;
  // extent check: per-column coordinate ranges into the scratch head, read back, compared with the tables
  long long* ranges = reinterpret_cast<long long*>(scratch);
  k_coord_range<<<cm.d, 256, 0, st>>>(ZA, R, ZB, M, cm.d, ranges);
  count_launches(1);
  long long hr[4 * MAXD];
  e = cuda_status(cudaMemcpyAsync(hr, ranges, 4 * cm.d * sizeof(long long), cudaMemcpyDeviceToHost, st),
                  "blml_rows_noalloc extents");
  if (!e) e = cuda_status(cudaStreamSynchronize(st), "blml_rows_noalloc extents");
  if (e) return e;
  e = extents_ok(cm, hr);
  if (e) return e;
  double* part = scratch + kRowsScratchRangeSlots;
  if (tb->f32) {
    if (!tb->T32 || (cm.G && !tb->RT32)) { set_error("blml_rows_noalloc: float32 tables missing"); return BLML_ERR_ARG; }
    return rows_noalloc_launch<float>(cm, hr, tb->T32, tb->RT32, ZA, R, ZB, M, w, part, s, st);
  }
  if (!tb->T || (cm.G && !tb->RT)) { set_error("blml_rows_noalloc: tables missing"); return BLML_ERR_ARG; }
  return rows_noalloc_launch<double>(cm, hr, tb->T, tb->RT, ZA, R, ZB, M, w, part, s, st);
}

int blml_lattice_coords(const double* Z, int64_t n, int d, const double* h, int64_t* out, void* stream) {
  if (n < 0 || d < 1) { set_error("blml_lattice_coords: bad sizes"); return BLML_ERR_ARG; }
  if (n == 0) return BLML_OK;
  const int g = (int)std::min<int64_t>((n * d + 255) / 256, 148 * 32);
  k_lattice_coords<<<g, 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(Z, n, d, h, out);
  count_launches(1);
  return cuda_status(cudaGetLastError(), "blml_lattice_coords");
}

static int cols_launch(const blml_tables* tb, const int64_t* ZA, int64_t R, const int64_t* ZB, int64_t M, void* out,
                       void* out_m, int64_t depmask, int out_f32, void* stream, const char* who) {
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  ColMeta cm;
  int e = read_meta(tb, cm, st);
  if (e) return e;
  if (depmask < 0 || (cm.d < 63 && (depmask >> cm.d) != 0)) { set_error("%s: depmask has bits past column d", who); return BLML_ERR_ARG; }
  if (R == 0 || M == 0) return BLML_OK;
  e = check_extents(cm, ZA, R, ZB, M, st);
  if (e) return e;
  unsigned dep_units = 0;                        // a unit (column or radial group) is dep when one of its columns is
  for (int k = 0; k < cm.d; k++)              // a group column's unit is its group's
    if ((depmask >> k) & 1) dep_units |= 1u << ((cm.code[k] == 2 || cm.code[k] == 4) ? cm.grp_unit[cm.grp[k]] : cm.dim_unit[k]);
  const int64_t n = R * M;
  const int g = (int)std::min<int64_t>((n + 255) / 256, 148 * 32);
  if (tb->f32) {
    if (out_f32) k_cols<float, float><<<g, 256, 0, st>>>(cm, tb->T32, tb->RT32, ZA, R, ZB, M, (float*)out, (float*)out_m, dep_units);
    else k_cols<float, double><<<g, 256, 0, st>>>(cm, tb->T32, tb->RT32, ZA, R, ZB, M, (double*)out, (double*)out_m, dep_units);
  } else {
    if (out_f32) k_cols<double, float><<<g, 256, 0, st>>>(cm, tb->T, tb->RT, ZA, R, ZB, M, (float*)out, (float*)out_m, dep_units);
    else k_cols<double, double><<<g, 256, 0, st>>>(cm, tb->T, tb->RT, ZA, R, ZB, M, (double*)out, (double*)out_m, dep_units);
  }
  count_launches(1);
  return cuda_status(cudaGetLastError(), who);
}

int blml_cols(const blml_tables* tb, const int64_t* ZA, int64_t R, const int64_t* ZB, int64_t M, void* out,
              int out_f32, void* stream) {
  return cols_launch(tb, ZA, R, ZB, M, out, nullptr, 0, out_f32, stream, "blml_cols");
}

int blml_cols_dep(const blml_tables* tb, const int64_t* ZA, int64_t R, const int64_t* ZB, int64_t M, int64_t depmask,
                  void* out, void* out_m, int out_f32, void* stream) {
  if (!out_m) { set_error("blml_cols_dep: out_m"); return BLML_ERR_ARG; }
  return cols_launch(tb, ZA, R, ZB, M, out, out_m, depmask, out_f32, stream, "blml_cols_dep");
}

}
