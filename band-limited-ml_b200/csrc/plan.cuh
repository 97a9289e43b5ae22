// The mat-vec plan shared by the SIMT (matvec.cu) and tensor-core (tc_matvec.cu) engines.
#pragma once
#include <vector>
#include "common.cuh"

struct blml_plan_s {
  int d, dtype, engine;
  int64_t shape[8];
  int32_t nfreq[8];
  int64_t max_elems;                 // largest intermediate tensor of one lattice (elements), SIMT schedule
  void* tf[8];                       // forward twiddles per axis: (M x H) conj(v), complex of dtype
  void* ti[8];                       // inverse twiddles per axis: (H x M) v^T
  void* W;                           // weights over the frequency grid, real of dtype
  void* tc;                          // tensor-core engine state (split-TF32 operands), or null
  void* fft;                         // FFT route state (fft_matvec.cu) when the kernel is a DFT mask, or null
  int route;                         // BLML_ROUTE_*: which route blml_matvec takes
};

namespace blml {
// fwd[a] / inv[a]: the float64 twiddles of axis a, interleaved complex, (M x H) conj(v) and (H x M) v^T
int tc_plan_init(blml_plan_s* p, const std::vector<std::vector<double>>& fwd,
                 const std::vector<std::vector<double>>& inv);
void tc_plan_free(blml_plan_s* p);
int tc_matvec(blml_plan_s* p, const void* x, void* y, int nb, int xc, void* ws, int64_t wsb, cudaStream_t st);
int64_t tc_workspace(const blml_plan_s* p, int nb);
int tc_error(blml_plan_s* p);

// the FFT route (fft_matvec.cu): set up when the plan is a 2-D DFT mask on sides 2^a 3^b (else p->fft stays null)
int fft_plan_init(blml_plan_s* p, const double* freqs, const double* weights);
void fft_plan_free(blml_plan_s* p);
int64_t fft_workspace(const blml_plan_s* p, int nb);
int fft_matvec(blml_plan_s* p, const void* x, void* y, int nb, int xc, void* ws, cudaStream_t st);
// the same for a few plans at once, when fft_few says so (z[i]: problem i's workspace)
bool fft_few(int n, const blml_plan* plans, const int* nb);
int fft_matvec_few(int n, const blml_plan* plans, const int* nb, const void* const* x, void* const* y, void* const* z,
                   int xc, cudaStream_t st);
// a group's descriptors: problem g reads x[g], writes y[g] and keeps its spectrum in z[g] (its workspace); *out stays
// null when a plan has no FFT route. dev: fft_group_bytes(G) bytes of device memory (kept); its first bytes are to be
// filled from `up`
size_t fft_group_bytes(int G);
int fft_group_init(void** out, int G, const blml_plan* plans, const int* nbatch, int xc, const void* const* x,
                   void* const* y, void* const* z, void* dev, std::vector<char>& up);
void fft_group_free(void* fg);
// blml_group_create in the caller's memory (alloc null: the library's own); ws: intermediate buffers shared with a group
// of the same problems whose launches do not overlap this one's (null: its own); fft_only: no contraction descriptors
// when every plan has the FFT route
int group_create(int G, const blml_plan* plans, const int* nbatch, int x_complex, const void* x_base,
                 const int64_t* x_off, void* y_base, const int64_t* y_off, blml_alloc_fn alloc, void* ctx,
                 cudaStream_t st, void* ws, bool fft_only, blml_group* out);
void* group_ws(blml_group g);
int fft_group_launch(void* fg, int dtype, const int* subset, int n, const int* live, cudaStream_t st);
}  // namespace blml
