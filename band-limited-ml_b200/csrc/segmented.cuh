// Segmented-kernel helpers shared by the batched solver kernels (batched.cu) and the device-side control of the
// batched engine (batch_runner.cu): fit f owns the slice [off_f, off_f + K_f B_f) of every flat mode array and
// [boff_f, boff_f + B_f) of every flat bin array; blockIdx.y is the fit, blockIdx.x strides over its bins.
#pragma once
#include "common.cuh"

namespace blml {

// blocks per fit (gridDim.x) of a segmented launch over F fits: ~16384 blocks in all, 16 to 256 per fit. Fits differ
// in size by up to ~300x (lattice and mode count), and every fit gets the same blocks, so the block count is sized
// for the largest: their blocks then still spread over every SM while the small fits' blocks find little or no work
// and leave at once. The partials of a reduction over F fits take nq * F * seg_blocks_for(F) <= nq * SEG_PART_WIDTH(F)
// doubles.
constexpr int SEG_BLOCKS_MIN = 16, SEG_BLOCKS_MAX = 256, SEG_BLOCKS_TOTAL = 16384;
__host__ __device__ constexpr int64_t SEG_PART_WIDTH(int F) {
  return (int64_t)(SEG_BLOCKS_TOTAL > 16 * F ? SEG_BLOCKS_TOTAL : 16 * F);
}
__host__ __device__ inline int seg_blocks_for(int F) {
  int x = SEG_BLOCKS_TOTAL / (F > 0 ? F : 1);
  return x < SEG_BLOCKS_MIN ? SEG_BLOCKS_MIN : (x > SEG_BLOCKS_MAX ? SEG_BLOCKS_MAX : x);
}

// A block split: SEG_SPLIT_BLOCKS blocks in all, shared out among the fits in proportion to their element counts
// K B (at least one block per fit with work, none per fit without, and no more blocks than SEG_SPLIT_MIN_ELEMS-element
// chunks), so that big and small fits finish together and every block has several tiles to stream. The split is
// computed on the device from the segment table itself (k_seg_split), so it follows fits whose table entry the device
// changes (a converged fit's B set to 0). Its ints: bstart[F + 1] (fit f owns split blocks
// [bstart[f], bstart[f + 1])), then fit_of[G + F] (the fit of each block of a launch of G + F blocks, -1 for blocks
// past the last fit's). Partials of a split reduction: quantity q of block b at part[q * (G + F) + b].
constexpr int SEG_SPLIT_BLOCKS = BLML_SEG_SPLIT_BLOCKS, SEG_SPLIT_MIN_ELEMS = 1024;
__host__ __device__ inline int64_t seg_split_ints(int F) { return 2 * (int64_t)F + 1 + SEG_SPLIT_BLOCKS; }
int seg_split(int F, const blml_seg* segs, int* split, cudaStream_t st);

// The history slots a scan covers: slot p and the slots that hold a pair (stamp >= 0) of launch row j's fit fid[j]; the
// other slots' products are 0 and their memory is not read. stamp null: every slot. most: no fit has more slots than that.
struct HistMask {
  const int* stamp; const int* fid; int m, p, most;
  __device__ __forceinline__ bool on(int j, int q) const { return !stamp || q == p || stamp[(int64_t)fid[j] * m + q] >= 0; }
};

// the L-BFGS runner's history scans (batched.cu): state of dtype, or complex64 storage (split: seg_split's output)
// out: blml_seg_dots2's quantities of the vectors a; out2 (or null): those of a second list a2 of as many
int seg_dots2(int dtype, int F, const blml_seg* segs, int cplx, int np, const void* const* a, const void* const* a2,
              const void* b0, const void* b1, const void* x, double* part, double* out, double* out2, HistMask hm,
              cudaStream_t st);
int seg_dots2_h32(int F, const blml_seg* segs, const int* split, int np, const void* const* a, const void* const* a2,
                  const void* b0, const void* b1, const void* x, double* part, double* out, double* out2, HistMask hm,
                  cudaStream_t st);
// the two quantities of blml_seg_resid from their partials
int seg_finish_resid(int F, const double* part, double* out, cudaStream_t st);
constexpr int SEG_DOTS2_ROWS = 83;         // partials per block: two lists of 20 twice, three norms
int seg_lincomb_mixed(int F, const blml_seg* segs, const int* split, void* out, int out_f32, int nterms,
                      const double* coef, const void* const* v, unsigned long long f32mask, cudaStream_t st);

template <typename T, bool CPLX>
struct SAcc {
  static __device__ __forceinline__ void get(const void* p, int64_t i, double& re, double& im) {
    if (CPLX) { const cpx<T> v = reinterpret_cast<const cpx<T>*>(p)[i]; re = (double)v.re; im = (double)v.im; }
    else { re = (double)reinterpret_cast<const T*>(p)[i]; im = 0.0; }
  }
  static __device__ __forceinline__ void put(void* p, int64_t i, double re, double im) {
    if (CPLX) reinterpret_cast<cpx<T>*>(p)[i] = cpx<T>{(T)re, (T)im};
    else reinterpret_cast<T*>(p)[i] = (T)re;
  }
};

#define SEG_LOOP(b, sg) for (int64_t b = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; b < (sg).B; \
                             b += (int64_t)gridDim.x * blockDim.x)

// partials layout, quantity-major so it does not depend on how many accumulators a kernel carries:
// part[((q * F) + j) * nblk + bx] for block bx of the nblk blocks of row j of F
template <int NQ>
__device__ __forceinline__ void seg_partials_at(double (&v)[NQ], double* part, unsigned maxmask, int F, int j, int nblk,
                                                int bx) {
  __shared__ double sh[NQ][32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
  for (int q = 0; q < NQ; q++) {
    double x = ((maxmask >> q) & 1u) ? warp_max(v[q]) : warp_sum(v[q]);
    if (lane == 0) sh[q][wid] = x;
  }
  __syncthreads();
  if (wid == 0) {
#pragma unroll
    for (int q = 0; q < NQ; q++) {
      const bool mx = (maxmask >> q) & 1u;
      double x = lane < nw ? sh[q][lane] : (mx ? -INFINITY : 0.0);
      x = mx ? warp_max(x) : warp_sum(x);
      if (lane == 0) part[((int64_t)q * F + j) * nblk + bx] = x;
    }
  }
}

template <int NQ>
__device__ __forceinline__ void seg_partials(double (&v)[NQ], double* part, unsigned maxmask = 0u) {
  seg_partials_at<NQ>(v, part, maxmask, gridDim.y, blockIdx.y, gridDim.x, blockIdx.x);
}

// body(j, bx) for the nblk blocks bx of every row j whose flag is set, shared out among the launch's blocks (256 threads);
// the flags are listed 256 at a time. A launch of nblk blocks for each of F rows costs 25 to 40 us of blocks that leave at
// once when few flags or none are set, this one 4.
constexpr int SEG_FLAGGED_BLOCKS = 148 * 8;
template <typename Body>
__device__ __forceinline__ void seg_flagged(const int* flag, int F, int nblk, Body body) {
  __shared__ int list[256], cnt[8];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  int64_t base = 0;
  for (int j0 = 0; j0 < F; j0 += 256) {
    const bool on = j0 + tid < F && flag[j0 + tid];
    const unsigned m = __ballot_sync(0xffffffffu, on);
    if (lane == 0) cnt[warp] = __popc(m);
    __syncthreads();
    int at = __popc(m & ((1u << lane) - 1u)), total = 0;
    for (int w = 0; w < 8; w++) { at += w < warp ? cnt[w] : 0; total += cnt[w]; }
    if (on) list[at] = j0 + tid;
    __syncthreads();
    const int64_t n = (int64_t)total * nblk, g = gridDim.x, d = (int64_t)blockIdx.x - base % g;
    for (int64_t i = d < 0 ? d + g : d; i < n; i += g) {
      body(list[i / nblk], (int)(i % nblk));
      __syncthreads();                     // seg_partials_at's shared memory
    }
    base += n;
    __syncthreads();                       // list and cnt
  }
}

}  // namespace blml
