// The FFT route of the mat-vec for kernels that are exact DFT masks on a circular 2-D lattice.
//
// A pball group, or dirichlet columns, on a lattice whose every axis is one period (the reference's circular pad,
// blml_binned.py:130-136) has plane waves at integer harmonics: nu = k / M on an M-point axis. Then
//     S e = sum_q W_q v_q v_q^H e
// is the unnormalised inverse 2-D DFT of W times the forward DFT of e, restricted to the band's harmonics: the
// reference's rfftn -> x Kf -> irfftn (blml_binned.py:156-168) with Kf zero outside the band. Three grouped stages
// run it over every fit of a batch, each a batch of 1-D FFTs:
//   A  rows:    FFT of every lattice row (length M2), keep the H2 harmonics of axis 1 -> Z (nb, H2, M1)
//   B  columns: FFT of every Z column (length M1), times W over the band (zero elsewhere), inverse FFT -> Z
//   C  rows:    each row's H2 harmonics in a zero spectrum, inverse FFT (length M2) -> the lattice row
// The FFTs are mixed-radix Stockham passes of radix 2 to 8: sides 2^a 3^b. A thread holds one butterfly in registers;
// the first pass reads global memory, the last one writes it, and between passes the values cross shared memory once.
// The column stage multiplies by W as the forward transform's last pass leaves its values in shared memory for the
// inverse transform's first. (Fusing those two passes in registers wants the inverse radices backwards: no faster, and it
// rounds differently.)
// Small work -- one lattice of 64 x 64, a few of 128 x 128 -- runs the three stages in one launch, a thread-block cluster
// per lattice (k_fft_cluster).
// Bound: latency in small launches; in large ones issue (35-40% of slots), L1 / shared memory (50%) and FP64 (20%)
// together. Staging every row in and out of shared memory and the twiddles per CTA moved each value 8 to 10 times through
// shared memory where this moves it four times (sides 65 to 512). Radix 16 (two passes up to 256) needs 128 registers: 2
// CTAs per SM and twice the code, 15-20% slower at every size. Float64 pball fc 0.33, before -> now: 384 x 384 x 8
// 42.4 -> 34.0 us, x 64 225 -> 193 us; 256 x 256 20.7 -> 15.7; the benchmark sweep's 64 lattices 93.6 -> 73 us.
// Versus the restricted transforms (matvec.cu) this costs O(M log M) per row instead of O(M H), and in float64 it
// rounds like an FFT (~1e-16 log M relative), so the route changes no result beyond rounding.
#include <vector>
#include <algorithm>
#include <functional>
#include <cmath>
#include <cooperative_groups.h>
#include "plan.cuh"

namespace blml {

constexpr int kFT = 256;                 // threads per CTA
constexpr int kCtaBytesMax = 72 * 1024;  // the largest shared-memory budget a CTA may aim for

// launch shape of the route, chosen by blml_fft_set_shape (the project's autotuner writes a table the package applies)
// and read when a plan's descriptor is made: the shared memory a CTA aims for (several transforms per CTA; one when
// longer) and the most columns a CTA of the column stage takes
static int g_cta_bytes = kCtaBytesMax;
static int g_max_cols = 16;
constexpr int kMaxSide = 4096;           // longest side of the route
constexpr int kMaxPass = 7;              // 3^7 = 2187 = 3 x 3 x 3 x 3 x 3 x 3 x 3

// x / d for 0 <= x < 2^16 and 1 <= d < 2^16 by a multiply and a shift: m = floor((2^32 - 1) / d) + 1 (0 for d = 1)
__host__ __device__ __forceinline__ unsigned magic_of(unsigned d) { return d <= 1 ? 0u : 0xFFFFFFFFu / d + 1u; }
__device__ __forceinline__ int div_m(int x, unsigned m) { return m ? (int)__umulhi((unsigned)x, m) : x; }

static int fft_smem_once();

// The passes of one axis's transform: radix, sub-transform length ns before the pass, butterflies nbt = N / R. In
// shared memory point i lies at (i / R0) pitch + i mod R0 (R0 the first radix, pitch odd: the first pass's stores at
// stride R0 spread over the banks), a transform occupies ld slots (odd: transforms side by side start on different
// banks). The twiddle table holds, pass after pass (ns > 1), w^(r k N / (ns R)) for 1 <= r < R, k < ns at
// [(r - 1) ns + k], w = exp(-2 pi i / N): threads with consecutive k read consecutive values.
struct FftAxis {
  int N, npass, pitch, ld;
  unsigned mr0;                          // division by R0
  int8_t rad[kMaxPass];
  int ns[kMaxPass], nbt[kMaxPass], twoff[kMaxPass];
  unsigned mnbt[kMaxPass], mns[kMaxPass];
};

// per-plan data of the route (host struct holding device pointers)
struct FftPlan {
  int M1, M2, H1, H2;
  FftAxis ax1, ax2;                      // axis 0 (columns, length M1) and axis 1 (rows, length M2)
  void* tw1; void* tw2;                 // the axes' pass twiddle tables, complex of the plan's dtype
  int shift2;                            // >= 0: DFT index k of axis 1 is band position (k + shift2) mod M2 (< H2), a run
  int* map2;                             // of harmonics; else map2[k]: its position, or -1
  void* wc;                              // weights (H2, M1) over the DFT indices of axis 0, zero outside the band
};

struct FftDesc {
  const void* X; void* Y; void* Z; const void* wc;
  const void* tw1; const void* tw2; const int* map2;
  int M1, M2, H2, nb, flags, shift2;     // flags: 1 real input, 4 real output
  unsigned mM1;                          // division by M1
  int rows, cols;                        // transforms per CTA: rows (stages A, C), columns (stage B)
  unsigned mrows;                        // division by rows
  int ctasA, ctasB;                      // CTAs of this problem in stages A / C and B
  FftAxis ax1, ax2;
};

// ------------------------------------------------------------------------------------------------- butterflies
// y_s = sum_r a_r exp(sign 2 pi i r s / R), sign = +1 for the inverse transform, -1 forward.
template <typename T, bool INV> __device__ __forceinline__ cpx<T> mul_i(cpx<T> a) {   // a * (sign i)
  return INV ? cpx<T>{-a.im, a.re} : cpx<T>{a.im, -a.re};
}
template <typename T> __device__ __forceinline__ cpx<T> cadd(cpx<T> a, cpx<T> b) { return {a.re + b.re, a.im + b.im}; }
template <typename T> __device__ __forceinline__ cpx<T> csub(cpx<T> a, cpx<T> b) { return {a.re - b.re, a.im - b.im}; }

template <typename T, bool INV> __device__ __forceinline__ void dft2(cpx<T>& a0, cpx<T>& a1) {
  const cpx<T> t = a0; a0 = cadd(t, a1); a1 = csub(t, a1);
}
template <typename T, bool INV> __device__ __forceinline__ void dft4(cpx<T>& a0, cpx<T>& a1, cpx<T>& a2, cpx<T>& a3) {
  const cpx<T> t0 = cadd(a0, a2), t1 = csub(a0, a2), t2 = cadd(a1, a3), t3 = mul_i<T, INV>(csub(a1, a3));
  a0 = cadd(t0, t2); a2 = csub(t0, t2); a1 = cadd(t1, t3); a3 = csub(t1, t3);
}
template <typename T, bool INV> __device__ __forceinline__ void dft3(cpx<T>& a0, cpx<T>& a1, cpx<T>& a2) {
  const T h = T(0.8660254037844386);      // sin(pi / 3)
  const cpx<T> t = cadd(a1, a2), u = csub(a1, a2);
  const cpx<T> m = {a0.re - T(0.5) * t.re, a0.im - T(0.5) * t.im};
  const cpx<T> v = mul_i<T, INV>(cpx<T>{h * u.re, h * u.im});
  a0 = cadd(a0, t); a1 = cadd(m, v); a2 = csub(m, v);
}
template <typename T, int R, bool INV> __device__ __forceinline__ void butterfly(cpx<T> (&a)[R]) {
  if constexpr (R == 2) {
    dft2<T, INV>(a[0], a[1]);
  } else if constexpr (R == 3) {
    dft3<T, INV>(a[0], a[1], a[2]);
  } else if constexpr (R == 4) {
    dft4<T, INV>(a[0], a[1], a[2], a[3]);
  } else if constexpr (R == 6) {            // evens and odds by DFT3, joined with exp(sign 2 pi i s / 6)
    cpx<T> e0 = a[0], e1 = a[2], e2 = a[4], o0 = a[1], o1 = a[3], o2 = a[5];
    dft3<T, INV>(e0, e1, e2); dft3<T, INV>(o0, o1, o2);
    const T h = T(0.8660254037844386);
    const cpx<T> w1 = {T(0.5), INV ? h : -h}, w2 = {T(-0.5), INV ? h : -h};
    const cpx<T> p1 = cmul(o1, w1), p2 = cmul(o2, w2);
    a[0] = cadd(e0, o0); a[3] = csub(e0, o0);
    a[1] = cadd(e1, p1); a[4] = csub(e1, p1);
    a[2] = cadd(e2, p2); a[5] = csub(e2, p2);
  } else {                                  // R == 8: evens and odds by DFT4, joined with exp(sign 2 pi i s / 8)
    cpx<T> e0 = a[0], e1 = a[2], e2 = a[4], e3 = a[6], o0 = a[1], o1 = a[3], o2 = a[5], o3 = a[7];
    dft4<T, INV>(e0, e1, e2, e3); dft4<T, INV>(o0, o1, o2, o3);
    const T c = T(0.7071067811865476);       // cos(pi / 4)
    const cpx<T> p1 = INV ? cpx<T>{c * (o1.re - o1.im), c * (o1.im + o1.re)}
                          : cpx<T>{c * (o1.re + o1.im), c * (o1.im - o1.re)};
    const cpx<T> p2 = mul_i<T, INV>(o2);
    const cpx<T> p3 = INV ? cpx<T>{c * (-o3.re - o3.im), c * (o3.re - o3.im)}
                          : cpx<T>{c * (-o3.re + o3.im), c * (-o3.re - o3.im)};
    a[0] = cadd(e0, o0); a[4] = csub(e0, o0);
    a[1] = cadd(e1, p1); a[5] = csub(e1, p1);
    a[2] = cadd(e2, p2); a[6] = csub(e2, p2);
    a[3] = cadd(e3, p3); a[7] = csub(e3, p3);
  }
}

// ------------------------------------------------------------------------------------------------- passes
// Pass p of ntr transforms: butterfly j (of nbt) of transform t takes points j + r nbt (from load(t, j, r, nbt) in the
// first pass, from shared memory times w^(r (j mod ns) N / (ns R)) later), and its outputs s go to points
// (j - j mod ns) R + j mod ns + s ns: to shared memory, or in the last pass (where that is j + s ns) to
// store(t, j, s, ns, value). TF: consecutive threads take consecutive transforms (the side whose global accesses are
// contiguous over transforms), else consecutive butterflies.
// ldg_c: constants of the plan, through the read-only path. ld_c: what the kernel before may have written -- the stages may
// be resident while it still writes (stage_wait), and only ordinary loads are ordered behind that wait.
template <typename T> __device__ __forceinline__ cpx<T> ldg_c(const cpx<T>* p) {
  if constexpr (sizeof(T) == 8) { const double2 v = __ldg(reinterpret_cast<const double2*>(p)); return {v.x, v.y}; }
  else { const float2 v = __ldg(reinterpret_cast<const float2*>(p)); return {v.x, v.y}; }
}
template <typename T> __device__ __forceinline__ cpx<T> ld_c(const cpx<T>* p) {
  if constexpr (sizeof(T) == 8) { const double2 v = *reinterpret_cast<const double2*>(p); return {v.x, v.y}; }
  else { const float2 v = *reinterpret_cast<const float2*>(p); return {v.x, v.y}; }
}

// the band position of DFT index k of axis 1, or -1
__device__ __forceinline__ int band_pos(const FftDesc& D, int k) {
  if (D.shift2 < 0) return __ldg(D.map2 + k);
  int q = k + D.shift2;
  if (q >= D.M2) q -= D.M2;
  return q < D.H2 ? q : -1;
}
// row r of all nb lattices -> lattice and row within it
__device__ __forceinline__ int lattice_of(const FftDesc& D, int row) {
  return row < 65536 ? div_m(row, D.mM1) : row / D.M1;
}

// the butterfly's slot arithmetic: input slot base and step, output slot base and step
struct Slots { int in, din, out, dout, k; };
__device__ __forceinline__ Slots slots_of(const FftAxis& ax, int p, int R, int j) {
  const int R0 = ax.rad[0];
  Slots s;
  if (p == 0) {                          // (input from global memory) outputs j R0 + s
    s.in = 0; s.din = 0; s.k = 0; s.out = j * ax.pitch; s.dout = 1;
    return s;
  }
  // ns and nbt are multiples of R0 after the first pass
  const int jd = div_m(j, ax.mr0), jm = j - jd * R0;
  s.in = jd * ax.pitch + jm; s.din = div_m(ax.nbt[p], ax.mr0) * ax.pitch;
  const int k = j - div_m(j, ax.mns[p]) * ax.ns[p], kd = div_m(k, ax.mr0);
  s.k = k;
  s.out = ((jd - kd) * R + kd) * ax.pitch + jm; s.dout = div_m(ax.ns[p], ax.mr0) * ax.pitch;
  return s;
}

template <typename T, int R, bool INV>
__device__ __forceinline__ void twiddle(cpx<T> (&v)[R], const cpx<T>* tw, int ns, int k) {
#pragma unroll
  for (int r = 1; r < R; r++) {
    cpx<T> w = ldg_c(tw + (r - 1) * ns + k);
    if (INV) w.im = -w.im;
    v[r] = cmul(v[r], w);
  }
}

template <typename T, int R, bool INV, bool FIRST, bool LAST, bool TF, typename L, typename S>
__device__ __forceinline__ void pass_r(const FftAxis& ax, int p, const cpx<T>* tw, int ntr, unsigned mntr,
                                       const cpx<T>* src, cpx<T>* dst, L load, S store) {
  const int nbt = ax.nbt[p], total = nbt * ntr, ns = ax.ns[p];
  for (int b = threadIdx.x; b < total; b += blockDim.x) {
    int t, j;
    if (TF) { j = div_m(b, mntr); t = b - j * ntr; } else { t = div_m(b, ax.mnbt[p]); j = b - t * nbt; }
    const Slots sl = slots_of(ax, p, R, j);
    cpx<T> v[R];
    if (FIRST) {
#pragma unroll
      for (int r = 0; r < R; r++) v[r] = load(t, j + r * nbt);
    } else {
      const cpx<T>* s = src + t * ax.ld + sl.in;
#pragma unroll
      for (int r = 0; r < R; r++) v[r] = s[r * sl.din];
      twiddle<T, R, INV>(v, tw + ax.twoff[p], ns, sl.k);
    }
    butterfly<T, R, INV>(v);
    if (LAST) {
#pragma unroll
      for (int s = 0; s < R; s++) store(t, j + s * ns, v[s]);
    } else {
      cpx<T>* d = dst + t * ax.ld + sl.out;
#pragma unroll
      for (int s = 0; s < R; s++) d[s * sl.dout] = v[s];
    }
  }
}

#define FFT_RADIX(RAD, CALL)                                                                                        \
  switch (RAD) {                                                                                                   \
    case 8: { constexpr int R = 8; CALL; break; }                                                                  \
    case 6: { constexpr int R = 6; CALL; break; }                                                                  \
    case 4: { constexpr int R = 4; CALL; break; }                                                                  \
    case 3: { constexpr int R = 3; CALL; break; }                                                                  \
    default: { constexpr int R = 2; CALL; break; }                                                                 \
  }

struct NoIO {
  template <typename... A> __device__ void operator()(A...) const {}
};
template <typename T> struct NoLoad {
  __device__ cpx<T> operator()(int, int) const { return {T(0), T(0)}; }
};

// passes 1 .. npass - 2 (shared memory to shared memory, alternating between the two buffers); returns the buffer that
// holds the result (the first pass wrote into a)
template <typename T, bool INV>
__device__ __forceinline__ cpx<T>* middle_passes(const FftAxis& ax, const cpx<T>* tw, int ntr, cpx<T>* a, cpx<T>* b) {
  for (int p = 1; p < ax.npass - 1; p++) {
    __syncthreads();
    FFT_RADIX(ax.rad[p], (pass_r<T, R, INV, false, false, false>(ax, p, tw, ntr, 0u, a, b, NoLoad<T>(), NoIO())));
    cpx<T>* t = a; a = b; b = t;
  }
  __syncthreads();
  return a;
}

// a whole transform from load to store; TF1 / TF2: the first / last pass over transforms first
template <typename T, bool INV, bool TF1, bool TF2, typename L, typename S>
__device__ __forceinline__ void transform(const FftAxis& ax, const cpx<T>* tw, int ntr, unsigned mntr, cpx<T>* a,
                                          cpx<T>* b, L load, S store) {
  if (ax.npass == 1) {
    FFT_RADIX(ax.rad[0], (pass_r<T, R, INV, true, true, TF1>(ax, 0, tw, ntr, mntr, a, a, load, store)));
    return;
  }
  FFT_RADIX(ax.rad[0], (pass_r<T, R, INV, true, false, TF1>(ax, 0, tw, ntr, mntr, a, a, load, NoIO())));
  const cpx<T>* src = middle_passes<T, INV>(ax, tw, ntr, a, b);
  const int p = ax.npass - 1;
  FFT_RADIX(ax.rad[p], (pass_r<T, R, INV, false, true, TF2>(ax, p, tw, ntr, mntr, src, a, NoLoad<T>(), store)));
}

// The columns between the two transforms: the last forward pass leaves its outputs times W at their points in shared
// memory (natural order), the first inverse pass takes them from there.
__device__ __forceinline__ int slot_at(const FftAxis& ax, int i) {
  const int d = div_m(i, ax.mr0);
  return d * ax.pitch + (i - d * ax.rad[0]);
}

// ------------------------------------------------------------------------------------------------- stages
// Each stage is a device body over one problem's descriptor and one CTA index, behind two entry points: grouped
// (grid (max CTAs of a problem, 1, n); problem gi = subset[blockIdx.z] or blockIdx.z; problems with live[gi] == 0 and
// CTAs past the problem's own count return at once, uniformly per CTA) and single-plan (the descriptor by value).
// Dynamic shared memory: buffers of `transforms` padded transforms (rows_smem, cols_smem).
template <typename T>
__device__ __forceinline__ void rows_fwd_body(const FftDesc& D, int cta, unsigned char* smem) {
  const FftAxis& ax = D.ax2;
  const int N = D.M2, M1 = D.M1, H2 = D.H2, r0 = cta * D.rows, nr = min(D.rows, D.nb * M1 - r0);
  cpx<T>* a = reinterpret_cast<cpx<T>*>(smem);
  cpx<T>* b = a + D.rows * ax.ld;
  cpx<T>* Z = reinterpret_cast<cpx<T>*>(D.Z);
  const unsigned mnr = nr == D.rows ? D.mrows : magic_of((unsigned)nr);
  // harmonic k of row r0 + t: kept when it is in the band, at Z (b, q2, r)
  auto keep = [&](int t, int k, cpx<T> v) {
    const int q2 = band_pos(D, k);
    if (q2 >= 0) {
      const int row = r0 + t, bt = lattice_of(D, row);
      Z[((int64_t)bt * H2 + q2) * M1 + (row - bt * M1)] = v;
    }
  };
  const cpx<T>* tw = reinterpret_cast<const cpx<T>*>(D.tw2);
  const int64_t base = (int64_t)r0 * N;
  if (D.flags & 1) {
    const T* X = reinterpret_cast<const T*>(D.X) + base;
    transform<T, false, false, true>(ax, tw, nr, mnr, a, b,
                                     [&](int t, int i) { return cpx<T>{X[t * N + i], T(0)}; }, keep);
  } else {
    const cpx<T>* X = reinterpret_cast<const cpx<T>*>(D.X) + base;
    transform<T, false, false, true>(ax, tw, nr, mnr, a, b, [&](int t, int i) { return ld_c(X + t * N + i); }, keep);
  }
}

// nc columns from load to store: forward passes, times their weight rows w, inverse passes
template <typename T, typename L, typename S>
__device__ __forceinline__ void columns(const FftDesc& D, const T* w, int nc, cpx<T>* a, cpx<T>* b, L load, S store) {
  const FftAxis& ax = D.ax1;
  const cpx<T>* tw = reinterpret_cast<const cpx<T>*>(D.tw1);
  const int N = ax.N;
  auto to_smem = [&](cpx<T>* dst) {
    return [=, &ax](int t, int i, cpx<T> v) {
      const T m = w[t * N + i];
      v.re *= m; v.im *= m;
      dst[t * ax.ld + slot_at(ax, i)] = v;
    };
  };
  auto from_smem = [&](const cpx<T>* src) { return [=, &ax](int t, int i) { return src[t * ax.ld + slot_at(ax, i)]; }; };
  cpx<T>* mid = b;                                                  // where the weighted spectrum goes
  if (ax.npass == 1) {
    FFT_RADIX(ax.rad[0], (pass_r<T, R, false, true, true, false>(ax, 0, tw, nc, 0u, a, a, load, to_smem(b))));
  } else {
    FFT_RADIX(ax.rad[0], (pass_r<T, R, false, true, false, false>(ax, 0, tw, nc, 0u, a, a, load, NoIO())));
    const cpx<T>* src = middle_passes<T, false>(ax, tw, nc, a, b);
    mid = src == a ? b : a;
    const int p = ax.npass - 1;
    FFT_RADIX(ax.rad[p], (pass_r<T, R, false, false, true, false>(ax, p, tw, nc, 0u, src, a, NoLoad<T>(), to_smem(mid))));
  }
  __syncthreads();
  transform<T, true, false, false>(ax, tw, nc, 0u, mid == a ? b : a, mid, from_smem(mid), store);
}

template <typename T>
__device__ __forceinline__ void cols_body(const FftDesc& D, int cta, unsigned char* smem) {
  const int N = D.M1, H2 = D.H2, c0 = cta * D.cols, nc = min(D.cols, D.nb * H2 - c0);
  cpx<T>* a = reinterpret_cast<cpx<T>*>(smem);
  cpx<T>* b = a + D.cols * D.ax1.ld;
  cpx<T>* Z = reinterpret_cast<cpx<T>*>(D.Z) + (int64_t)c0 * N;
  const T* W = reinterpret_cast<const T*>(D.wc);
  const int q0 = c0 % H2;
  // lattice by lattice: a CTA's columns may run on into the next one, whose weights start over
  for (int t0 = 0; t0 < nc;) {
    const int q = t0 ? 0 : q0, m = min(nc - t0, H2 - q);
    cpx<T>* Zt = Z + (int64_t)t0 * N;                              // (this CTA's columns only: read before written)
    columns<T>(D, W + (int64_t)q * N, m, a, b, [&](int t, int i) { return Zt[t * N + i]; },
               [&](int t, int i, cpx<T> v) { Zt[t * N + i] = v; });
    t0 += m;
    if (t0 < nc) __syncthreads();
  }
}

template <typename T>
__device__ __forceinline__ void rows_inv_body(const FftDesc& D, int cta, unsigned char* smem) {
  const FftAxis& ax = D.ax2;
  const int N = D.M2, M1 = D.M1, H2 = D.H2, r0 = cta * D.rows, nr = min(D.rows, D.nb * M1 - r0);
  cpx<T>* a = reinterpret_cast<cpx<T>*>(smem);
  cpx<T>* b = a + D.rows * ax.ld;
  const cpx<T>* Z = reinterpret_cast<const cpx<T>*>(D.Z);
  const unsigned mnr = nr == D.rows ? D.mrows : magic_of((unsigned)nr);
  const cpx<T>* tw = reinterpret_cast<const cpx<T>*>(D.tw2);
  auto band = [&](int t, int k) {
    const int q2 = band_pos(D, k);
    if (q2 < 0) return cpx<T>{T(0), T(0)};
    const int row = r0 + t, bt = lattice_of(D, row);
    return ld_c(Z + ((int64_t)bt * H2 + q2) * M1 + (row - bt * M1));
  };
  const int64_t base = (int64_t)r0 * N;
  if (D.flags & 4) {
    T* Y = reinterpret_cast<T*>(D.Y) + base;
    transform<T, true, true, false>(ax, tw, nr, mnr, a, b, band, [&](int t, int i, cpx<T> v) { Y[t * N + i] = v.re; });
  } else {
    cpx<T>* Y = reinterpret_cast<cpx<T>*>(D.Y) + base;
    transform<T, true, true, false>(ax, tw, nr, mnr, a, b, band, [&](int t, int i, cpx<T> v) { Y[t * N + i] = v; });
  }
}

// the stages are launched with programmatic dependent launch: a stage's CTAs may be placed while the one before drains,
// and wait here for its results; every stage lets the next one in as soon as all its own CTAs have started. No memory that
// another kernel writes is read before the wait or through the read-only path (no __ldg, no const __restrict__ parameter:
// such loads are not ordered behind it)
__device__ __forceinline__ void stage_wait() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

// The three stages of one lattice in one launch, for lattices whose band fits a thread-block cluster's shared memory:
// the cluster's CTAs take M1 / CS rows each, the rows' harmonics go straight to the shared memory of the CTA that owns
// their column (distributed shared memory), each CTA runs its H2 / CS columns there, and the row transforms back read
// the harmonics from the columns' owners. Two cluster barriers in place of two launches, and the spectrum never leaves
// the SMs. Small batches, where the three launches' latencies are most of the time.
constexpr int kClThreads = 512;
struct FftCluster {
  FftDesc D;
  int cpc, zld;                          // columns per CTA, slots per column
  unsigned mcpc;
  int rpc, rows_t, cols_t;               // rows per CTA; rows / columns a CTA transforms at a time
  unsigned mrows_t;
  int off_a, off_b;                      // the exchange buffers in shared memory (complex slots)
};

template <typename T>
__global__ void __launch_bounds__(kClThreads, 1) k_fft_cluster(const __grid_constant__ FftCluster C) {
  extern __shared__ __align__(16) unsigned char fft_smem[];
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  const FftDesc& D = C.D;
  const int rank = (int)cl.block_rank(), lat = (int)blockIdx.x / (int)cl.num_blocks();
  cpx<T>* Zs = reinterpret_cast<cpx<T>*>(fft_smem);
  cpx<T>* a = Zs + C.off_a;
  cpx<T>* b = Zs + C.off_b;
  const int M1 = D.M1, N = D.M2, r_beg = rank * C.rpc, r_end = min(M1, r_beg + C.rpc);
  const int64_t base = (int64_t)lat * M1 * N;
  // harmonic q2 of lattice row r, in the shared memory of its column's CTA
  auto slot = [&](int q2, int r) {
    const int o = div_m(q2, C.mcpc);
    return cl.map_shared_rank(Zs, o) + (q2 - o * C.cpc) * C.zld + r;
  };
  const cpx<T>* tw2 = reinterpret_cast<const cpx<T>*>(D.tw2);
  stage_wait();
  cl.sync();                                                      // every CTA of the cluster has started
  for (int r0 = r_beg; r0 < r_end; r0 += C.rows_t) {
    const int nr = min(C.rows_t, r_end - r0);
    const unsigned mnr = nr == C.rows_t ? C.mrows_t : magic_of((unsigned)nr);
    auto keep = [&](int t, int k, cpx<T> v) {
      const int q2 = band_pos(D, k);
      if (q2 >= 0) *slot(q2, r0 + t) = v;
    };
    if (D.flags & 1) {
      const T* X = reinterpret_cast<const T*>(D.X) + base + (int64_t)r0 * N;
      transform<T, false, false, true>(D.ax2, tw2, nr, mnr, a, b,
                                       [&](int t, int i) { return cpx<T>{X[t * N + i], T(0)}; }, keep);
    } else {
      const cpx<T>* X = reinterpret_cast<const cpx<T>*>(D.X) + base + (int64_t)r0 * N;
      transform<T, false, false, true>(D.ax2, tw2, nr, mnr, a, b, [&](int t, int i) { return ld_c(X + t * N + i); },
                                       keep);
    }
    __syncthreads();
  }
  cl.sync();
  const int c_beg = rank * C.cpc, c_end = min(D.H2, c_beg + C.cpc);
  for (int c0 = c_beg; c0 < c_end; c0 += C.cols_t) {
    const int m = min(C.cols_t, c_end - c0), zld = C.zld;
    cpx<T>* Zt = Zs + (c0 - c_beg) * zld;
    auto ld = [&](int t, int i) { return Zt[t * zld + i]; };
    auto st = [&](int t, int i, cpx<T> v) { Zt[t * zld + i] = v; };
    columns<T>(D, reinterpret_cast<const T*>(D.wc) + (int64_t)c0 * M1, m, a, b, ld, st);
    __syncthreads();
  }
  cl.sync();
  for (int r0 = r_beg; r0 < r_end; r0 += C.rows_t) {
    const int nr = min(C.rows_t, r_end - r0);
    const unsigned mnr = nr == C.rows_t ? C.mrows_t : magic_of((unsigned)nr);
    auto band = [&](int t, int k) {
      const int q2 = band_pos(D, k);
      return q2 < 0 ? cpx<T>{T(0), T(0)} : *slot(q2, r0 + t);
    };
    if (D.flags & 4) {
      T* Y = reinterpret_cast<T*>(D.Y) + base + (int64_t)r0 * N;
      transform<T, true, true, false>(D.ax2, tw2, nr, mnr, a, b, band, [&](int t, int i, cpx<T> v) { Y[t * N + i] = v.re; });
    } else {
      cpx<T>* Y = reinterpret_cast<cpx<T>*>(D.Y) + base + (int64_t)r0 * N;
      transform<T, true, true, false>(D.ax2, tw2, nr, mnr, a, b, band, [&](int t, int i, cpx<T> v) { Y[t * N + i] = v; });
    }
    __syncthreads();
  }
  cl.sync();                                                      // no CTA leaves while others read its columns
}

// The grouped launches cover only the work of the problems taking part: k_fft_schedule (one block) lists the
// problems of the launch (subset[i], or i), drops those with live == 0, and writes the exclusive prefix sums of
// their CTA counts for stages A / C and B; CTA x of a stage finds its problem by binary search over those sums
// and returns at once when x is past the total. The grid is the host's bound: the sum of the n largest counts.
constexpr int kSchedMax = 2048;          // problems a schedule takes (a launch over more runs in chunks of 2048)

struct FftSched {
  int n;                                 // problems in the schedule
  int prob[kSchedMax];                   // their indices
  int offA[kSchedMax + 1], offB[kSchedMax + 1];
};

__global__ void k_fft_schedule(const FftDesc* __restrict__ descs, const int* __restrict__ subset, int n0, int n,
                               const int* __restrict__ live, FftSched* sch) {
  __shared__ int cA[kSchedMax], cB[kSchedMax], pr[kSchedMax];
  __shared__ int wsA[32], wsB[32];
  const int tid = threadIdx.x;
  for (int i = tid; i < n; i += blockDim.x) {
    const int g = subset ? subset[n0 + i] : n0 + i;
    const bool on = !live || live[g];
    pr[i] = g; cA[i] = on ? descs[g].ctasA : 0; cB[i] = on ? descs[g].ctasB : 0;
  }
  __syncthreads();
  if (tid < 32) {                        // one warp: a serial scan per lane chunk, then a warp scan of the chunk sums
    const int per = (n + 31) / 32, lo = tid * per, hi = min(n, lo + per);
    int sa = 0, sb = 0;
    for (int i = lo; i < hi; i++) { sa += cA[i]; sb += cB[i]; }
    int xa = sa, xb = sb;
    for (int o = 1; o < 32; o <<= 1) {
      const int ya = __shfl_up_sync(0xffffffffu, xa, o), yb = __shfl_up_sync(0xffffffffu, xb, o);
      if (tid >= o) { xa += ya; xb += yb; }
    }
    wsA[tid] = xa - sa; wsB[tid] = xb - sb;
    int ra = wsA[tid], rb = wsB[tid];
    for (int i = lo; i < hi; i++) {
      sch->offA[i] = ra; sch->offB[i] = rb; sch->prob[i] = pr[i];
      ra += cA[i]; rb += cB[i];
    }
    if (tid == 31) { sch->offA[n] = xa; sch->offB[n] = xb; sch->n = n; }
  }
}

// the problem and local CTA index of CTA x in a schedule (offsets off[0 .. n]), or -1 past the total
__device__ __forceinline__ int sched_find(const int* off, int n, int x, int& local) {
  if (x >= off[n]) return -1;
  int lo = 0, hi = n - 1;                // the last i with off[i] <= x
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (off[mid] <= x) lo = mid; else hi = mid - 1;
  }
  local = x - off[lo];
  return lo;
}

// a few plans' lattices in one launch, their descriptors by value (the modes of one fit with kernels of their own: two
// of 256 x 256 complex: 6 launches -> 3, 28 -> 19 us of kernels)
constexpr int kFew = 4;
struct FftFew { FftDesc d[kFew]; int n, offA[kFew + 1], offB[kFew + 1]; };

// 4 CTAs per SM over many problems (the sweep's lattices 78 -> 73 us, although the float64 column stage then spills 8 bytes
// at 64 registers), 3 and more registers for one plan's lattices (384 x 384 x 8: 36.1 -> 34.0 us; 80 registers, 4 bytes)
#define FFT_STAGE(NAME, BODY, OFF)                                                                                \
  template <typename T>                                                                                          \
  __global__ void __launch_bounds__(kFT, 4) NAME##_grp(const FftDesc* descs, const FftSched* sch) {                 \
    extern __shared__ __align__(16) unsigned char fft_smem[];                                                    \
    __shared__ __align__(16) FftDesc Ds;                                                                         \
    stage_wait();                                                                                                \
    int local = 0;                                                                                               \
    const int i = sched_find(sch->OFF, sch->n, (int)blockIdx.x, local);                                          \
    if (i < 0) return;                                                                                           \
    {                                   /* the problem's descriptor, staged once per CTA */                     \
      const int* src = reinterpret_cast<const int*>(descs + sch->prob[i]);                                       \
      int* dst = reinterpret_cast<int*>(&Ds);                                                                    \
      for (int q = threadIdx.x; q < (int)(sizeof(FftDesc) / 4); q += kFT) dst[q] = src[q];                       \
    }                                                                                                            \
    __syncthreads();                                                                                             \
    BODY<T>(Ds, local, fft_smem);                                                                                \
  }                                                                                                              \
  template <typename T>                                                                                          \
  __global__ void __launch_bounds__(kFT, 3) NAME##_one(const FftDesc D) {                                           \
    extern __shared__ __align__(16) unsigned char fft_smem[];                                                    \
    stage_wait();                                                                                                \
    BODY<T>(D, blockIdx.x, fft_smem);                                                                            \
  }                                                                                                              \
  template <typename T>                                                                                          \
  __global__ void __launch_bounds__(kFT, 3) NAME##_few(const __grid_constant__ FftFew P) {                          \
    extern __shared__ __align__(16) unsigned char fft_smem[];                                                    \
    int i = 0;                                                                                                   \
    while (i < P.n - 1 && (int)blockIdx.x >= P.OFF[i + 1]) i++;                                                  \
    stage_wait();                                                                                                \
    BODY<T>(P.d[i], (int)blockIdx.x - P.OFF[i], fft_smem);                                                       \
  }

FFT_STAGE(k_fft_rows_fwd, rows_fwd_body, offA)
FFT_STAGE(k_fft_cols, cols_body, offB)
FFT_STAGE(k_fft_rows_inv, rows_inv_body, offA)

// ------------------------------------------------------------------------------------------------- host side
// radices of an N = 2^a 3^b point FFT: 8s, then a 4 or 2, then 3s, a 2 and a 3 merged into a 6 (fewest passes); 0
// when N has another prime factor
static int radix_plan(int N, int8_t* rad) {
  int a = 0, b = 0, m = N;
  while (m % 2 == 0) { m /= 2; a++; }
  while (m % 3 == 0) { m /= 3; b++; }
  if (m != 1 || N < 2) return 0;
  int n = 0, two = 0;
  auto add = [&](int r) { if (n < kMaxPass) rad[n] = (int8_t)r; n++; };
  for (; a >= 3; a -= 3) add(8);
  if (a == 2) add(4);
  else if (a == 1) two = 1;
  for (int i = 0; i < b; i++) {
    if (two) { add(6); two = 0; }
    else add(3);
  }
  if (two) add(2);
  return n <= kMaxPass ? n : 0;
}

// an axis's passes and its twiddle table (float64 host values, interleaved complex); false when N has no plan
static bool axis_plan(int N, FftAxis& ax, std::vector<double>& tw) {
  ax = FftAxis{};
  ax.N = N;
  ax.npass = radix_plan(N, ax.rad);
  if (!ax.npass) return false;
  const int R0 = ax.rad[0];
  ax.pitch = R0 | 1; ax.ld = (N / R0 * ax.pitch) | 1; ax.mr0 = magic_of((unsigned)R0);
  tw.clear();
  int Ns = 1;
  for (int p = 0; p < ax.npass; p++) {
    const int R = ax.rad[p];
    ax.ns[p] = Ns; ax.nbt[p] = N / R; ax.mnbt[p] = magic_of((unsigned)(N / R)); ax.mns[p] = magic_of((unsigned)Ns);
    ax.twoff[p] = (int)(tw.size() / 2);
    if (Ns > 1) {
      const int stride = N / (Ns * R);
      for (int r = 1; r < R; r++)
        for (int k = 0; k < Ns; k++) {
          const long long e = (long long)r * k * stride % N;
          const double ph = 2.0 * M_PI * (double)e / (double)N;
          tw.push_back(std::cos(ph)); tw.push_back(-std::sin(ph));
        }
    }
    Ns *= R;
  }
  if (tw.empty()) { tw.push_back(1.0); tw.push_back(0.0); }
  return true;
}

// shared-memory buffers a row transform alternates between: none for one pass, one for two, two beyond
static int row_buffers(const FftAxis& ax) { return ax.npass <= 1 ? 0 : ax.npass == 2 ? 1 : 2; }

// transforms per CTA: as many as the shared-memory budget and one first-pass butterfly per thread hold, but no more than
// spread `total` transforms over two CTAs per SM; at least one
static int transforms_per_cta(const FftAxis& ax, int bufs, int ld, size_t esz, long long total, int most) {
  long long n = kFT / ax.nbt[0];
  if (bufs) n = std::min<long long>(n, g_cta_bytes / (long long)(esz * bufs * ld));
  n = std::min<long long>({n, (long long)most, (total + 2 * 148 - 1) / (2 * 148)});
  return (int)std::max<long long>(1, n);
}

static size_t rows_smem(const FftAxis& ax, int ntr, size_t esz) { return (size_t)row_buffers(ax) * ntr * ax.ld * esz; }
static size_t cols_smem(const FftAxis& ax, int ntr, size_t esz) {
  return 2 * (size_t)ntr * ax.ld * esz;
}

int fft_plan_init(blml_plan_s* p, const double* freqs, const double* weights) {
  p->fft = nullptr;
  if (p->d != 2 || p->engine != BLML_ENGINE_SIMT) return BLML_OK;
  const int M1 = (int)p->shape[0], M2 = (int)p->shape[1], H1 = p->nfreq[0], H2 = p->nfreq[1];
  if (M1 > kMaxSide || M2 > kMaxSide || H1 > M1 || H2 > M2) return BLML_OK;
  FftPlan fp{};
  fp.M1 = M1; fp.M2 = M2; fp.H1 = H1; fp.H2 = H2;
  std::vector<double> tws1, tws2;
  if (!axis_plan(M1, fp.ax1, tws1) || !axis_plan(M2, fp.ax2, tws2)) return BLML_OK;
  // integer harmonics, distinct modulo the side: then S is exactly the DFT mask
  std::vector<int> map1(M1, -1), map2(M2, -1);
  for (int q = 0; q < H1 + H2; q++) {
    const int M = q < H1 ? M1 : M2;
    const double x = freqs[q] * M, r = std::nearbyint(x);
    if (std::fabs(x - r) > 1e-9 * std::max(1.0, std::fabs(r))) return BLML_OK;
    const int k = (int)(((long long)r % M + M) % M);
    if (q < H1) {
      if (map1[k] >= 0) return BLML_OK;
      map1[k] = q;
    } else {
      if (map2[k] >= 0) return BLML_OK;
      map2[k] = q - H1;
    }
  }
  // a run of harmonics in ascending order (every kernel without an inner gap): positions by arithmetic
  fp.shift2 = -1;
  for (int k = 0; k < M2 && fp.shift2 < 0; k++)
    if (map2[k] == 0) fp.shift2 = (M2 - k) % M2;
  for (int k = 0; k < M2; k++) {
    const int q = (k + fp.shift2) % M2;
    if (map2[k] != (q < H2 ? q : -1)) { fp.shift2 = -1; break; }
  }
  const bool f64 = p->dtype == BLML_F64;
  const size_t esz = f64 ? 16 : 8;
  auto table = [&](const std::vector<double>& t, void** dst) -> int {
    const size_t n = t.size() / 2;
    if (cudaMalloc(dst, n * esz) != cudaSuccess) { set_error("FFT plan: device allocation"); return BLML_ERR_CUDA; }
    if (f64) return cuda_status(cudaMemcpy(*dst, t.data(), n * esz, cudaMemcpyHostToDevice), "FFT plan twiddles");
    std::vector<float> t32(t.begin(), t.end());
    return cuda_status(cudaMemcpy(*dst, t32.data(), n * esz, cudaMemcpyHostToDevice), "FFT plan twiddles");
  };
  int rc = table(tws1, &fp.tw1);
  if (!rc) rc = table(tws2, &fp.tw2);
  if (!rc && cudaMalloc(&fp.map2, M2 * sizeof(int)) != cudaSuccess) { set_error("FFT plan: device allocation"); rc = BLML_ERR_CUDA; }
  if (!rc) rc = cuda_status(cudaMemcpy(fp.map2, map2.data(), M2 * sizeof(int), cudaMemcpyHostToDevice), "FFT plan");
  if (!rc) {
    std::vector<double> wc((size_t)H2 * M1, 0.0);
    for (int q2 = 0; q2 < H2; q2++)
      for (int k = 0; k < M1; k++)
        if (map1[k] >= 0) wc[(size_t)q2 * M1 + k] = weights[(size_t)map1[k] * H2 + q2];
    const size_t n = wc.size(), b = n * (f64 ? 8 : 4);
    if (cudaMalloc(&fp.wc, b) != cudaSuccess) { set_error("FFT plan: device allocation"); rc = BLML_ERR_CUDA; }
    else if (f64) rc = cuda_status(cudaMemcpy(fp.wc, wc.data(), b, cudaMemcpyHostToDevice), "FFT plan weights");
    else {
      const std::vector<float> c32(wc.begin(), wc.end());
      rc = cuda_status(cudaMemcpy(fp.wc, c32.data(), b, cudaMemcpyHostToDevice), "FFT plan weights");
    }
  }
  if (rc) {
    cudaFree(fp.tw1); cudaFree(fp.tw2); cudaFree(fp.map2); cudaFree(fp.wc);
    return rc;
  }
  p->fft = new FftPlan(fp);
  return fft_smem_once();
}

void fft_plan_free(blml_plan_s* p) {
  FftPlan* fp = reinterpret_cast<FftPlan*>(p->fft);
  if (!fp) return;
  cudaFree(fp->tw1); cudaFree(fp->tw2); cudaFree(fp->map2); cudaFree(fp->wc);
  delete fp;
  p->fft = nullptr;
}

// rows_all, cols_all: the row and column transforms of the whole launch (this problem's and the others')
static FftDesc make_desc(const blml_plan_s* p, const void* x, void* y, void* z, int nb, int xc, long long rows_all,
                         long long cols_all) {
  const FftPlan* fp = reinterpret_cast<const FftPlan*>(p->fft);
  FftDesc D{};
  D.X = x; D.Y = y; D.Z = z; D.wc = fp->wc;
  D.tw1 = fp->tw1; D.tw2 = fp->tw2; D.map2 = fp->map2;
  D.M1 = fp->M1; D.M2 = fp->M2; D.H2 = fp->H2; D.nb = nb; D.shift2 = fp->shift2;
  D.mM1 = magic_of((unsigned)fp->M1);
  D.flags = xc ? 0 : (1 | 4);
  D.ax1 = fp->ax1; D.ax2 = fp->ax2;
  const size_t esz = p->dtype == BLML_F64 ? 16 : 8;
  D.rows = transforms_per_cta(fp->ax2, row_buffers(fp->ax2), fp->ax2.ld, esz, rows_all, kFT);
  D.cols = transforms_per_cta(fp->ax1, 2, fp->ax1.ld, esz, cols_all,
                              g_max_cols);
  D.mrows = magic_of((unsigned)D.rows);
  D.ctasA = (nb * fp->M1 + D.rows - 1) / D.rows;
  D.ctasB = (nb * fp->H2 + D.cols - 1) / D.cols;
  return D;
}

struct FftGroup {
  FftDesc* dev;                  // G descriptors
  FftSched* sch;                 // the schedule of the current launch (written by k_fft_schedule)
  std::vector<int> boundA, boundB;   // [n]: the sum of the n largest CTA counts (grid bounds), n <= kSchedMax
  size_t smemA, smemB;           // largest dynamic shared memory of a problem's stage
};

// the largest dynamic shared memory any stage asks for: two padded buffers of one kMaxSide-point float64 transform
// (first radix at least 2: at most 3 / 2 slots per point; shorter transforms stay within the CTA budget)
constexpr size_t kMaxSmem = 2 * (size_t)(kMaxSide + kMaxSide / 2 + 1) * 16;

// the six kernels' dynamic shared-memory limit, set once per device (outside any stream capture: at plan creation)
constexpr size_t kClSmem = 227 * 1024;

template <typename T>
static int set_fft_smem() {
  const int v = (int)kMaxSmem;
  int e = BLML_OK;
  auto set = [&](const void* f) {
    if (!e) e = cuda_status(cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, v), "FFT route");
  };
  set((const void*)k_fft_rows_fwd_grp<T>); set((const void*)k_fft_cols_grp<T>); set((const void*)k_fft_rows_inv_grp<T>);
  if (!e) e = cuda_status(cudaFuncSetAttribute(k_fft_cluster<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kClSmem), "FFT route");
  if (!e) e = cuda_status(cudaFuncSetAttribute(k_fft_cluster<T>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1), "FFT route");
  set((const void*)k_fft_rows_fwd_one<T>); set((const void*)k_fft_cols_one<T>); set((const void*)k_fft_rows_inv_one<T>);
  set((const void*)k_fft_rows_fwd_few<T>); set((const void*)k_fft_cols_few<T>); set((const void*)k_fft_rows_inv_few<T>);
  return e;
}

static int fft_smem_once() {
  static bool done[64] = {};
  int dev = 0;
  int e = cuda_status(cudaGetDevice(&dev), "FFT route");
  if (e || (dev < 64 && done[dev])) return e;
  e = set_fft_smem<double>();
  if (!e) e = set_fft_smem<float>();
  if (!e && dev < 64) done[dev] = true;
  return e;
}

// a launch of `grid` CTAs that may start while the kernel before it on the stream drains (stage_wait)
template <typename... P, typename... A>
static void launch_dep(void (*k)(P...), int grid, size_t smem, cudaStream_t st, A... args) {
  cudaLaunchConfig_t c{};
  c.gridDim = dim3((unsigned)grid); c.blockDim = dim3(kFT); c.dynamicSmemBytes = smem; c.stream = st;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  c.attrs = &at; c.numAttrs = 1;
  cudaLaunchKernelEx(&c, k, static_cast<P>(args)...);
}

template <typename T>
static int launch_fft_grp(const FftGroup* fg, const int* subset, int n0, int n, const int* live, cudaStream_t st) {
  k_fft_schedule<<<1, 256, 0, st>>>(fg->dev, subset, n0, n, live, fg->sch);
  BLML_CHECK_LAUNCH("FFT route: schedule");
  const int gA = fg->boundA[n], gB = fg->boundB[n];
  if (gA > 0) {
    launch_dep(k_fft_rows_fwd_grp<T>, gA, fg->smemA, st, fg->dev, fg->sch);
    BLML_CHECK_LAUNCH("FFT route: rows");
  }
  if (gB > 0) {
    launch_dep(k_fft_cols_grp<T>, gB, fg->smemB, st, fg->dev, fg->sch);
    BLML_CHECK_LAUNCH("FFT route: columns");
  }
  if (gA > 0) {
    launch_dep(k_fft_rows_inv_grp<T>, gA, fg->smemA, st, fg->dev, fg->sch);
    BLML_CHECK_LAUNCH("FFT route: inverse rows");
  }
  return BLML_OK;
}

template <typename T>
static int launch_fft_one(const FftDesc& D, size_t smA, size_t smB, cudaStream_t st) {
  launch_dep(k_fft_rows_fwd_one<T>, D.ctasA, smA, st, D);
  BLML_CHECK_LAUNCH("FFT route: rows");
  launch_dep(k_fft_cols_one<T>, D.ctasB, smB, st, D);
  BLML_CHECK_LAUNCH("FFT route: columns");
  launch_dep(k_fft_rows_inv_one<T>, D.ctasA, smA, st, D);
  BLML_CHECK_LAUNCH("FFT route: inverse rows");
  return BLML_OK;
}

static size_t desc_bytes(int G) { return ((size_t)G * sizeof(FftDesc) + 255) & ~(size_t)255; }
size_t fft_group_bytes(int G) { return desc_bytes(G) + sizeof(FftSched); }

int fft_group_init(void** out, int G, const blml_plan* plans, const int* nbatch, int xc, const void* const* x,
                   void* const* y, void* const* z, void* dev, std::vector<char>& up) {
  *out = nullptr;
  for (int g = 0; g < G; g++)
    if (!plans[g]->fft) return BLML_OK;
  const size_t esz = plans[0]->dtype == BLML_F64 ? 16 : 8;
  std::vector<FftDesc> h(G);
  FftGroup* fg = new FftGroup();
  fg->dev = nullptr; fg->sch = nullptr; fg->smemA = fg->smemB = 0;
  std::vector<int> cA(G), cB(G);
  long long rows_all = 0, cols_all = 0;
  for (int g = 0; g < G; g++) {
    const FftPlan* fp = reinterpret_cast<const FftPlan*>(plans[g]->fft);
    rows_all += (long long)nbatch[g] * fp->M1; cols_all += (long long)nbatch[g] * fp->H2;
  }
  for (int g = 0; g < G; g++) {
    h[g] = make_desc(plans[g], x[g], y[g], z[g], nbatch[g], xc, rows_all, cols_all);
    cA[g] = h[g].ctasA; cB[g] = h[g].ctasB;
    fg->smemA = std::max(fg->smemA, rows_smem(h[g].ax2, h[g].rows, esz));
    fg->smemB = std::max(fg->smemB, cols_smem(h[g].ax1, h[g].cols, esz));
  }
  std::sort(cA.begin(), cA.end(), std::greater<int>()); std::sort(cB.begin(), cB.end(), std::greater<int>());
  const int nmax = std::min(G, kSchedMax);
  fg->boundA.assign(nmax + 1, 0); fg->boundB.assign(nmax + 1, 0);
  for (int i = 0; i < nmax; i++) { fg->boundA[i + 1] = fg->boundA[i] + cA[i]; fg->boundB[i + 1] = fg->boundB[i] + cB[i]; }
  const int e = fft_smem_once();
  if (e) { delete fg; return e; }
  fg->dev = reinterpret_cast<FftDesc*>(dev);
  fg->sch = reinterpret_cast<FftSched*>(reinterpret_cast<char*>(dev) + desc_bytes(G));
  up.assign(reinterpret_cast<const char*>(h.data()), reinterpret_cast<const char*>(h.data() + G));
  *out = fg;
  return BLML_OK;
}

void fft_group_free(void* fgv) { delete reinterpret_cast<FftGroup*>(fgv); }

// problems of the launch in chunks of kSchedMax (one schedule buffer: the chunks run one after another on st)
int fft_group_launch(void* fgv, int dtype, const int* subset, int n, const int* live, cudaStream_t st) {
  const FftGroup* fg = reinterpret_cast<const FftGroup*>(fgv);
  for (int n0 = 0; n0 < n; n0 += kSchedMax) {
    const int nc = std::min(kSchedMax, n - n0);
    const int e = dtype == BLML_F64 ? launch_fft_grp<double>(fg, subset, n0, nc, live, st)
                                    : launch_fft_grp<float>(fg, subset, n0, nc, live, st);
    if (e) return e;
  }
  return BLML_OK;
}

// one plan over nb lattices: Z (nb, H2, M1) in the caller's workspace, the descriptor passed by value
int64_t fft_workspace(const blml_plan_s* p, int nb) {
  const FftPlan* fp = reinterpret_cast<const FftPlan*>(p->fft);
  const size_t esz = p->dtype == BLML_F64 ? 16 : 8;
  return (int64_t)((size_t)nb * fp->H2 * fp->M1 * esz);
}

// one cluster of cs CTAs per lattice; false when the band does not fit their shared memory
static bool cluster_args(const FftDesc& D, int cs, size_t esz, FftCluster& C, size_t& smem) {
  C.D = D;
  C.cpc = (D.H2 + cs - 1) / cs; C.mcpc = magic_of((unsigned)C.cpc); C.zld = D.M1 | 1;
  C.rpc = (D.M1 + cs - 1) / cs;
  C.rows_t = std::max(1, std::min(C.rpc, kClThreads / D.ax2.nbt[0]));
  C.cols_t = std::max(1, std::min(C.cpc, kClThreads / D.ax1.nbt[0]));
  C.mrows_t = magic_of((unsigned)C.rows_t);
  const int buf = std::max(C.rows_t * D.ax2.ld, C.cols_t * D.ax1.ld);
  C.off_a = C.cpc * C.zld; C.off_b = C.off_a + buf;
  smem = (size_t)(C.off_b + buf) * esz;
  return smem <= kClSmem;
}

template <typename T>
static int cluster_launch(const FftCluster& C, int nb, int cs, size_t smem, cudaStream_t st) {
  cudaLaunchConfig_t c{};
  c.gridDim = dim3((unsigned)(nb * cs)); c.blockDim = dim3(kClThreads); c.dynamicSmemBytes = smem; c.stream = st;
  cudaLaunchAttribute at[2] = {};
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)cs; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = 1;
  c.attrs = at; c.numAttrs = 2;
  cudaLaunchKernelEx(&c, k_fft_cluster<T>, C);
  BLML_CHECK_LAUNCH("FFT route: cluster");
  return BLML_OK;
}

static bool cluster_rule(const blml_plan_s* p, int nb, int cs) {
  return nb * cs <= 64 && p->shape[0] * p->shape[1] <= 1024LL * cs;
}

int fft_matvec(blml_plan_s* p, const void* x, void* y, int nb, int xc, void* ws, cudaStream_t st) {
  const size_t esz = p->dtype == BLML_F64 ? 16 : 8;
  const FftDesc D = make_desc(p, x, y, ws, nb, xc, (long long)nb * p->shape[0], (long long)nb * p->nfreq[1]);
  // one launch for small work: CTAs of a cluster take at most 1,024 points of their lattice each, and the clusters 64
  // CTAs together (more than the GPU's clusters of that size would run in two waves). Float64, one lattice (three
  // launches -> one): 64 x 64 12.9 -> 8.7 us, 128 x 128 12.7 -> 11.0; at 256 x 256 sixteen CTAs are too few (15.1 -> 20.5).
  for (int cs = 16; cs >= 4; cs >>= 1) {
    if (!cluster_rule(p, nb, cs)) continue;
    FftCluster C;
    size_t smem = 0;
    if (cluster_args(D, cs, esz, C, smem))
      return p->dtype == BLML_F64 ? cluster_launch<double>(C, nb, cs, smem, st) : cluster_launch<float>(C, nb, cs, smem, st);
  }
  const size_t smA = rows_smem(D.ax2, D.rows, esz), smB = cols_smem(D.ax1, D.cols, esz);
  return p->dtype == BLML_F64 ? launch_fft_one<double>(D, smA, smB, st) : launch_fft_one<float>(D, smA, smB, st);
}

template <typename T>
static int launch_fft_few(const FftFew& P, size_t smA, size_t smB, cudaStream_t st) {
  launch_dep(k_fft_rows_fwd_few<T>, P.offA[P.n], smA, st, P);
  BLML_CHECK_LAUNCH("FFT route: rows");
  launch_dep(k_fft_cols_few<T>, P.offB[P.n], smB, st, P);
  BLML_CHECK_LAUNCH("FFT route: columns");
  launch_dep(k_fft_rows_inv_few<T>, P.offA[P.n], smA, st, P);
  BLML_CHECK_LAUNCH("FFT route: inverse rows");
  return BLML_OK;
}

// whether n problems go in one launch chain: a few, and none small enough for one of its own
bool fft_few(int n, const blml_plan* plans, const int* nb) {
  if (n < 2 || n > kFew) return false;
  for (int i = 0; i < n; i++)
    if (cluster_rule(plans[i], nb[i], 16)) return false;
  return true;
}

int fft_matvec_few(int n, const blml_plan* plans, const int* nb, const void* const* x, void* const* y, void* const* z,
                   int xc, cudaStream_t st) {
  const bool f64 = plans[0]->dtype == BLML_F64;
  const size_t esz = f64 ? 16 : 8;
  long long rows = 0, cols = 0;
  for (int i = 0; i < n; i++) { rows += (long long)nb[i] * plans[i]->shape[0]; cols += (long long)nb[i] * plans[i]->nfreq[1]; }
  FftFew P{};
  size_t smA = 0, smB = 0;
  P.n = n;
  for (int i = 0; i < n; i++) {
    P.d[i] = make_desc(plans[i], x[i], y[i], z[i], nb[i], xc, rows, cols);
    P.offA[i + 1] = P.offA[i] + P.d[i].ctasA; P.offB[i + 1] = P.offB[i] + P.d[i].ctasB;
    smA = std::max(smA, rows_smem(P.d[i].ax2, P.d[i].rows, esz)); smB = std::max(smB, cols_smem(P.d[i].ax1, P.d[i].cols, esz));
  }
  return f64 ? launch_fft_few<double>(P, smA, smB, st) : launch_fft_few<float>(P, smA, smB, st);
}

}  // namespace blml

extern "C" {

int blml_fft_set_shape(int cta_bytes, int max_cols) {
  if (cta_bytes < 8 * 1024 || cta_bytes > blml::kCtaBytesMax || max_cols < 1 || max_cols > 64) {
    blml::set_error("blml_fft_set_shape: 8 KiB <= cta_bytes <= %d, 1 <= max_cols <= 64", blml::kCtaBytesMax);
    return BLML_ERR_ARG;
  }
  blml::g_cta_bytes = cta_bytes; blml::g_max_cols = max_cols;
  return BLML_OK;
}

int blml_fft_get_shape(int* cta_bytes, int* max_cols) {
  if (!cta_bytes || !max_cols) { blml::set_error("blml_fft_get_shape: null argument"); return BLML_ERR_ARG; }
  *cta_bytes = blml::g_cta_bytes; *max_cols = blml::g_max_cols;
  return BLML_OK;
}

}
