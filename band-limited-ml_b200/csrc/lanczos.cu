// One Lanczos step of many certificates at once (blml_binned.py:501-518 calls ARPACK there): x = V[j] (for j > 0 first
// w / beta of the last step), w = dh S (dh x), then w orthogonalised against V[0 .. j] twice, alpha_j = V[j] . w of the
// first pass, beta_j = |w|. Each fit works on its own slice of the vectors.
//
// Bound: reading the basis from HBM, (j + 1) doubles per bin and pass. A pass needs every product before it may subtract,
// so the textbook order reads the basis four times; here the second pass's products are formed from the shared-memory copy
// of the tile that the first pass's subtraction has just read: three times, and w is read and written once per launch.
// Certificates of 64 fits (2.2 M bins, 58 steps, bases up to 49 vectors): separate inner products, finishes,
// coefficients, combinations and scalings took 30.1 ms in 18 launches a step, these 10.6 in 8 (with the mat-vec's four).
//
// Blocks take chunks of one fit (tab: launch row and chunk of each block, a row's chunks in a run), so big and small fits
// share the GPU evenly; the last block of a row to finish sums the row's partials in a fixed order.
#include <atomic>
#include "common.cuh"
#include "plan.cuh"

namespace blml {

constexpr int LZ_Q = 64;                  // vectors per launch; longer bases go in slabs of that
constexpr int LZ_T = 128;                 // bins per tile of the fused subtraction

struct LzArgs {
  const blml_seg* segs; const int* fid; const int2* tab;
  int chunk;
  double *part, *coef;                    // [q][block] partials, [fit][LZ_Q] coefficients
  int* cnt;                               // blocks of a row that are done
};

struct LzBlock {
  int row, fit, first, nblk;              // launch row, fit, the row's first block and their number
  int64_t off, lo, hi;                    // the fit's offset, the block's bins
};

__device__ __forceinline__ LzBlock lz_block(const LzArgs& A) {
  const int2 t = A.tab[blockIdx.x];
  const blml_seg S = A.segs[t.x];
  LzBlock b;
  b.row = t.x; b.fit = A.fid[t.x]; b.first = (int)blockIdx.x - t.y; b.nblk = (int)((S.B + A.chunk - 1) / A.chunk);
  b.off = S.boff; b.lo = (int64_t)t.y * A.chunk; b.hi = min(S.B, b.lo + A.chunk);
  return b;
}

// whether this block is the row's last; its partials and the others' are then visible
__device__ __forceinline__ bool lz_last(const LzArgs& A, const LzBlock& b) {
  __shared__ int last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    last = atomicAdd(A.cnt + b.row, 1) == b.nblk - 1;
    if (last) A.cnt[b.row] = 0;
  }
  __syncthreads();
  if (last) __threadfence();
  return last;
}

// the row's sum of quantity q over its blocks, in lane 0 of the calling warp
__device__ __forceinline__ double lz_total(const LzArgs& A, const LzBlock& b, int q) {
  const double* p = A.part + (int64_t)q * gridDim.x + b.first;
  double s = 0.0;
  for (int i = threadIdx.x & 31; i < b.nblk; i += 32) s += __ldcg(p + i);
  return warp_sum(s);
}

// x = V[j], tmp = dh x; scale: V[j] = scale w first
__global__ void __launch_bounds__(256) k_lz_next(LzArgs A, double* __restrict__ Vj, const double* __restrict__ scale,
                                                 const double* __restrict__ w, const double* __restrict__ dh,
                                                 double* __restrict__ tmp) {
  const LzBlock b = lz_block(A);
  const double c = scale ? scale[b.fit] : 0.0;
  for (int64_t i = b.lo + threadIdx.x; i < b.hi; i += 256) {
    double x;
    if (scale) { x = c * w[b.off + i]; Vj[b.off + i] = x; }
    else x = Vj[b.off + i];
    tmp[b.off + i] = x * dh[b.off + i];
  }
}

// the rows' coefficients from their partials: coef[fit][q] = -(V_q . w); alpha[fit] = the product of vector acol
__device__ __forceinline__ void lz_coef(const LzArgs& A, const LzBlock& b, int nq, double* alpha, int acol) {
  for (int q = threadIdx.x >> 5; q < nq; q += blockDim.x >> 5) {
    const double s = lz_total(A, b, q);
    if ((threadIdx.x & 31) == 0) {
      A.coef[(int64_t)b.fit * LZ_Q + q] = -s;
      if (alpha && q == acol) alpha[b.fit] = s;
    }
  }
}

// partials of V_q . w, q < nq <= 8 NW; FIRST: w = dh sv, formed here. Warp v takes the vectors v, v + 8, ..: each lane
// holds NW sums and has NW x 8 loads to issue per tile of 256 bins.
template <bool FIRST, int NW>
__global__ void __launch_bounds__(256) k_lz_dots(LzArgs A, const double* __restrict__ V, int64_t ldv, int nq,
                                                 const double* __restrict__ sv, const double* __restrict__ dh, double* w,
                                                 double* alpha, int acol) {
  __shared__ double ws[256];
  const LzBlock b = lz_block(A);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const double* p[NW];
  double acc[NW];
#pragma unroll
  for (int k = 0; k < NW; k++) { p[k] = V + (int64_t)min(warp + 8 * k, nq - 1) * ldv + b.off; acc[k] = 0.0; }
  for (int64_t t0 = b.lo; t0 < b.hi; t0 += 256) {
    const int64_t i = t0 + tid;
    double x = 0.0;
    if (i < b.hi) {
      if (FIRST) { x = sv[b.off + i] * dh[b.off + i]; w[b.off + i] = x; }
      else x = w[b.off + i];
    }
    __syncthreads();
    ws[tid] = x;
    __syncthreads();
    if (t0 + 256 <= b.hi) {
#pragma unroll
      for (int k = 0; k < NW; k++) {
        double v[8];
#pragma unroll
        for (int e = 0; e < 8; e++) v[e] = __ldg(p[k] + t0 + lane + 32 * e);
#pragma unroll
        for (int e = 0; e < 8; e++) acc[k] += v[e] * ws[lane + 32 * e];
      }
    } else {
#pragma unroll
      for (int k = 0; k < NW; k++)
        for (int e = 0; e < 8; e++)
          if (t0 + lane + 32 * e < b.hi) acc[k] += __ldg(p[k] + t0 + lane + 32 * e) * ws[lane + 32 * e];
    }
  }
#pragma unroll
  for (int k = 0; k < NW; k++) {
    const int q = warp + 8 * k;
    const double s = warp_sum(acc[k]);
    if (lane == 0 && q < nq) A.part[(int64_t)q * gridDim.x + blockIdx.x] = s;
  }
  if (lz_last(A, b)) lz_coef(A, b, nq, alpha, acol);
}

// w += sum_q coef_q V_q in vector order; NEXT: then the partials of V_q . w from the tile's copy in shared memory and the
// rows' new coefficients; else, with beta, |w| and 1 / |w| (0 for 0) per fit
template <bool NEXT>
__global__ void __launch_bounds__(LZ_T) k_lz_sub(LzArgs A, const double* __restrict__ V, int64_t ldv, int nq, double* w,
                                                 double* beta, double* scale) {
  extern __shared__ double vs[];                        // NEXT: [nq][LZ_T]
  __shared__ double cs[LZ_Q], ws[LZ_T], red[LZ_T / 32];
  const LzBlock b = lz_block(A);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid < nq) cs[tid] = A.coef[(int64_t)b.fit * LZ_Q + tid];
  double acc[LZ_Q / 4], nrm = 0.0;
#pragma unroll
  for (int k = 0; k < LZ_Q / 4; k++) acc[k] = 0.0;
  __syncthreads();
  for (int64_t t0 = b.lo; t0 < b.hi; t0 += LZ_T) {
    const bool in = t0 + tid < b.hi;
    const int64_t i = b.off + (in ? t0 + tid : t0);     // past the end: the tile's first bin, with a zero w
    const double* p = V + i;
    double r = in ? w[i] : 0.0;
    if (NEXT && t0 != b.lo) __syncthreads();            // the last tile's copy is done with
    int q = 0;
    for (; q + 16 <= nq; q += 16) {
      double v[16];
#pragma unroll
      for (int e = 0; e < 16; e++) v[e] = __ldg(p + (q + e) * ldv);
#pragma unroll
      for (int e = 0; e < 16; e++) { r += cs[q + e] * v[e]; if (NEXT) vs[(q + e) * LZ_T + tid] = v[e]; }
    }
    for (; q + 4 <= nq; q += 4) {
      double v[4];
#pragma unroll
      for (int e = 0; e < 4; e++) v[e] = __ldg(p + (q + e) * ldv);
#pragma unroll
      for (int e = 0; e < 4; e++) { r += cs[q + e] * v[e]; if (NEXT) vs[(q + e) * LZ_T + tid] = v[e]; }
    }
    for (; q < nq; q++) { const double v = __ldg(p + q * ldv); r += cs[q] * v; if (NEXT) vs[q * LZ_T + tid] = v; }
    if (!in) r = 0.0;
    else w[i] = r;
    if (NEXT) {
      ws[tid] = r;
      __syncthreads();
      double x[LZ_T / 32];
#pragma unroll
      for (int e = 0; e < LZ_T / 32; e++) x[e] = ws[lane + 32 * e];
#pragma unroll
      for (int k = 0; k < LZ_Q / 4; k++) {
        const int v = warp + 4 * k;
        if (v < nq) {
#pragma unroll
          for (int e = 0; e < LZ_T / 32; e++) acc[k] += vs[v * LZ_T + lane + 32 * e] * x[e];
        }
      }
    } else nrm += r * r;
  }
  if (NEXT) {
#pragma unroll
    for (int k = 0; k < LZ_Q / 4; k++) {
      const int v = warp + 4 * k;
      if (v < nq) {
        const double s = warp_sum(acc[k]);
        if (lane == 0) A.part[(int64_t)v * gridDim.x + blockIdx.x] = s;
      }
    }
    if (lz_last(A, b)) lz_coef(A, b, nq, nullptr, 0);
  } else if (beta) {
    nrm = warp_sum(nrm);
    if (lane == 0) red[warp] = nrm;
    __syncthreads();
    if (tid == 0) {
      double s = 0.0;
      for (int k = 0; k < LZ_T / 32; k++) s += red[k];
      A.part[blockIdx.x] = s;
    }
    if (lz_last(A, b) && warp == 0) {
      const double s = lz_total(A, b, 0);
      if (lane == 0) {
        const double v = sqrt(fmax(s, 0.0));
        beta[b.fit] = v;
        scale[b.fit] = v > 0.0 ? 1.0 / v : 0.0;
      }
    }
  }
}

// The two largest eigenvalues of each row's tridiagonal matrix (n square) and the last component of the top eigenvector.
// One warp a row. An eigenvalue by multisection with Sturm counts: each lane counts the eigenvalues above one of 32 points
// of the bracket from the signs of the leading minors p_k = (a_k - x) p_{k-1} - b_{k-1}^2 p_{k-2}, five bits a round. The
// last component from the twisted factorisation of T - theta (Dhillon and Parlett): the pivots d_k from the top and u_k
// from the bottom, the twist m at the smallest |d_m + u_m - (a_m - theta)|, y_m = 1, ratios b_k / d_k above and
// b_k / u_{k+1} below it; from the top alone it is lost where the vector has died out before the last step.
// Bound: the chain of n dependent multiply-adds a round (78 us for 64 fits at up to 64 square, behind which the next
// step is queued), where the host took 0.75 ms for the full decompositions, mostly with the GPU idle.
struct LzMat { const double* a; const double* b; int sa; int n; double inv; };     // entries sa apart, scaled by inv

__device__ __forceinline__ int lz_above(const LzMat& M, double x) {
  double p1 = 1.0, p = M.a[0] * M.inv - x;
  if (p == 0.0) p = -1e-290;
  int c = p > 0.0;
  for (int k = 1; k < M.n; k++) {
    const double b = M.b[(int64_t)(k - 1) * M.sa] * M.inv;
    double q = fma(M.a[(int64_t)k * M.sa] * M.inv - x, p, -(b * b) * p1);
    if (q == 0.0) q = p > 0.0 ? -1e-290 : 1e-290;
    c += (q > 0.0) == (p > 0.0);
    p1 = p; p = q;
    if ((k & 7) == 0) {                                   // back to order one (a power of two: exact)
      const double f = ldexp(1.0, -ilogb(fmax(fabs(p), fabs(p1))));
      p *= f; p1 *= f;
    }
  }
  return c;
}

// the largest x with at least `want` eigenvalues above it, in [lo, hi]
__device__ double lz_section(const LzMat& M, int want, double lo, double hi) {
  const int lane = threadIdx.x & 31;
  for (int r = 0; r < 16 && hi - lo > 2.3e-16 * fmax(fabs(lo), fabs(hi)); r++) {
    const double w = (hi - lo) / 33.0, x = lo + w * (lane + 1);
    const unsigned m = __ballot_sync(0xffffffffu, x > lo && x < hi && lz_above(M, x) >= want);
    const int top = 31 - __clz((int)m);                   // -1: none
    const double l = lo + w * (top + 1), h = lo + w * (top + 2);
    if (top >= 0) lo = l;
    if (top < 31 && h < hi) hi = h;
  }
  return 0.5 * (lo + hi);
}

constexpr int LZ_SHARED_N = 1024;
__global__ void __launch_bounds__(32) k_lz_check(const int* fid, int stride, const double* ab, int j, double* work,
                                                 double* out) {
  __shared__ double as[LZ_SHARED_N], bs[LZ_SHARED_N];
  const int f = fid[blockIdx.x], lane = threadIdx.x, n = j + 1;
  const double *a = ab + f, *b = ab + stride + f;         // alpha_i, beta_i at i * 2 stride
  LzMat M{a, b, 2 * stride, n, 1.0};
  if (n <= LZ_SHARED_N) {
    for (int i = lane; i < n; i += 32) { as[i] = a[(int64_t)i * M.sa]; bs[i] = b[(int64_t)i * M.sa]; }
    M.a = as; M.b = bs; M.sa = 1;
  }
  __syncwarp();
  double lo = INFINITY, hi = -INFINITY;                   // Gershgorin
  bool bad = false;
  for (int i = lane; i < n; i += 32) {
    const double d = M.a[(int64_t)i * M.sa];
    const double r = (i > 0 ? fabs(M.b[(int64_t)(i - 1) * M.sa]) : 0.0) + (i < n - 1 ? fabs(M.b[(int64_t)i * M.sa]) : 0.0);
    lo = fmin(lo, d - r); hi = fmax(hi, d + r);
    bad |= !isfinite(d) || !isfinite(r);
  }
  for (int o = 16; o > 0; o >>= 1) {
    lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o)); hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
  }
  bad = __any_sync(0xffffffffu, bad);
  const double size = fmax(fabs(lo), fabs(hi));
  double t1 = bad ? NAN : 0.0, t2 = bad || n == 1 ? NAN : 0.0, y = 1.0;       // (the zero matrix)
  if (!bad && size > 0.0) {
    M.inv = 1.0 / size;
    const double pad = 4e-16, l = lo * M.inv - pad, h = hi * M.inv + pad;
    t1 = lz_section(M, 1, l, h);
    if (n > 1) t2 = lz_section(M, 2, l, h);
    // lane 0 from the top, lane 1 from the bottom: pivots and the sums of (y_i / y_k)^2 up to k
    double* W = work + 4 * (int64_t)n * blockIdx.x;
    if (lane < 2) {
      double S = 1.0, d = 0.0;
      for (int k = 0; k < n; k++) {
        const int i = lane ? n - 1 - k : k;
        if (k == 0) d = M.a[(int64_t)i * M.sa] * M.inv - t1;
        else {
          const double bk = M.b[(int64_t)(lane ? i : i - 1) * M.sa] * M.inv;
          if (fabs(d) < 1e-30) d = -1e-30;
          const double r = bk / d;
          S = 1.0 + r * r * S;
          d = M.a[(int64_t)i * M.sa] * M.inv - t1 - bk * r;
        }
        W[(2 * lane) * n + i] = d; W[(2 * lane + 1) * n + i] = S;
      }
    }
    __syncwarp();
    double best = INFINITY;
    int m = n - 1;
    for (int i = lane; i < n; i += 32) {
      const double g = fabs(W[i] + W[2 * n + i] - (M.a[(int64_t)i * M.sa] * M.inv - t1));
      if (g < best) { best = g; m = i; }
    }
    for (int o = 16; o > 0; o >>= 1) {
      const double g = __shfl_xor_sync(0xffffffffu, best, o);
      const int i = __shfl_xor_sync(0xffffffffu, m, o);
      if (g < best || (g == best && i < m)) { best = g; m = i; }
    }
    y = 1.0;
    for (int i = m + lane; i < n - 1; i += 32) {
      double u = W[2 * n + i + 1];
      if (fabs(u) < 1e-30) u = -1e-30;
      y *= fabs(M.b[(int64_t)i * M.sa] * M.inv / u);
    }
    for (int o = 16; o > 0; o >>= 1) y *= __shfl_xor_sync(0xffffffffu, y, o);
    y /= sqrt(W[n + m] + W[3 * n + m] - 1.0);
    t1 *= size; t2 *= size;
  }
  if (lane == 0) {
    double* o = out + 4 * (int64_t)f;
    o[0] = t1; o[1] = t2; o[2] = y; o[3] = M.b[(int64_t)j * M.sa];
  }
}

template <bool FIRST>
static void lz_dots(int nblocks, cudaStream_t st, const LzArgs& A, const double* V, int64_t ldv, int nq, const double* sv,
                    const double* dh, double* w, double* alpha, int acol) {
  auto go = [&](auto k) { k<<<nblocks, 256, 0, st>>>(A, V, ldv, nq, sv, dh, w, alpha, acol); };
  if (nq <= 8) go(k_lz_dots<FIRST, 1>);
  else if (nq <= 16) go(k_lz_dots<FIRST, 2>);
  else if (nq <= 24) go(k_lz_dots<FIRST, 3>);
  else if (nq <= 32) go(k_lz_dots<FIRST, 4>);
  else if (nq <= 48) go(k_lz_dots<FIRST, 6>);
  else go(k_lz_dots<FIRST, 8>);
}

}  // namespace blml

using namespace blml;

extern "C" {

int blml_lanczos_step(int F, const blml_seg* segs, const int* fid, int nblocks, const int* tab, int chunk,
                      blml_group group, double* V, int64_t ldv, int j, const double* dh, double* tmp, const double* sv,
                      double* w, double* part, int* counters, double* coef, double* alpha, double* beta, double* scale,
                      void* stream) {
  if (F < 1 || F > 65535 || !segs || !fid || nblocks < F || !tab || chunk < 1 || !group || !V || j < 0 || !dh || !tmp ||
      !sv || !w || !part || !counters || !coef || !alpha || !beta || !scale ||
      (reinterpret_cast<uintptr_t>(tab) & 7)) {
    set_error("blml_lanczos_step: bad arguments (tab: 8-byte aligned)"); return BLML_ERR_ARG;
  }
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  constexpr int smem = LZ_Q * LZ_T * (int)sizeof(double);
  static std::atomic<bool> done[64];
  int dev = 0;
  int e = cuda_status(cudaGetDevice(&dev), "blml_lanczos_step");
  if (!e && (dev >= 64 || !done[dev])) {
    e = cuda_status(cudaFuncSetAttribute(k_lz_sub<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem), "blml_lanczos_step");
    if (!e && dev < 64) done[dev] = true;
  }
  if (e) return e;
  const LzArgs A{segs, fid, reinterpret_cast<const int2*>(tab), chunk, part, coef, counters};
  k_lz_next<<<nblocks, 256, 0, st>>>(A, V + (int64_t)j * ldv, j ? scale : nullptr, w, dh, tmp);
  BLML_CHECK_LAUNCH("lanczos vector");
  e = blml_group_matvec(group, stream);
  if (e) return e;
  const int n = j + 1;
  if (n <= LZ_Q) {
    lz_dots<true>(nblocks, st, A, V, ldv, n, sv, dh, w, alpha, j);
    BLML_CHECK_LAUNCH("lanczos products");
    k_lz_sub<true><<<nblocks, LZ_T, n * LZ_T * sizeof(double), st>>>(A, V, ldv, n, w, nullptr, nullptr);
    BLML_CHECK_LAUNCH("lanczos subtraction and products");
    k_lz_sub<false><<<nblocks, LZ_T, 0, st>>>(A, V, ldv, n, w, beta, scale);
    BLML_CHECK_LAUNCH("lanczos subtraction");
    return BLML_OK;
  }
  // a longer basis: each pass in slabs, every slab's products against the w that the slabs before it left
  for (int pass = 0; pass < 2; pass++)
    for (int q0 = 0; q0 < n; q0 += LZ_Q) {
      const int nq = n - q0 < LZ_Q ? n - q0 : LZ_Q;
      const double* Vq = V + (int64_t)q0 * ldv;
      const bool newest = pass == 0 && q0 + nq == n, last = pass == 1 && q0 + nq == n;
      if (pass == 0 && q0 == 0) lz_dots<true>(nblocks, st, A, Vq, ldv, nq, sv, dh, w, nullptr, 0);
      else lz_dots<false>(nblocks, st, A, Vq, ldv, nq, nullptr, nullptr, w, newest ? alpha : nullptr, j - q0);
      BLML_CHECK_LAUNCH("lanczos products");
      k_lz_sub<false><<<nblocks, LZ_T, 0, st>>>(A, Vq, ldv, nq, w, last ? beta : nullptr, last ? scale : nullptr);
      BLML_CHECK_LAUNCH("lanczos subtraction");
    }
  return BLML_OK;
}

int blml_lanczos_check(int F, const int* fid, int stride, const double* alpha_beta, int j, double* work,
                       double* out, void* stream) {
  if (F < 1 || !fid || stride < 1 || !alpha_beta || j < 0 || !work || !out) { set_error("blml_lanczos_check: bad arguments"); return BLML_ERR_ARG; }
  k_lz_check<<<F, 32, 0, reinterpret_cast<cudaStream_t>(stream)>>>(fid, stride, alpha_beta, j, work, out);
  BLML_CHECK_LAUNCH("lanczos check");
  return BLML_OK;
}

}  // extern "C"
