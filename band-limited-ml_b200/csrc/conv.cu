// The warm start's 3 x 3 convolutions (pad 1) as implicit GEMMs on tcgen05: the nine shifted views of the NHWC
// activation are never written out. A tile of 128 output pixels is a BW x BH x BN patch (powers of two) of the
// lattice; its operand for tap (ky, kx) is the same patch moved by (kx - 1, ky - 1), one 4-D TMA box per slice of
// channels whose out-of-range pixels the copy fills with zeros -- the convolution's padding. The products run in the
// order of the explicit form (tap by tap, channels ascending, 16 at a time into one FP32 accumulator), so the results
// are those of an im2col matrix and a GEMM, bit for bit.
//
// Bound: an im2col matrix is 9 x the activation written and read again (453 MB each way for the 96-channel decoder
// layer on 16 x 128 x 128 pixels) for a product of 14.5 GFLOP; here each pixel comes from L2 nine times and from HBM
// once, so what is left is the L2 reads.
#include "nn_tc.cuh"

namespace blml {

// channels per K slice: 64 (128-byte rows, 128B swizzle), 32 (64-byte rows, 64B swizzle), 8 (the input layer: 16-byte
// rows, no swizzle; its nine taps and a zero tenth are one K = 80 slice of five MMAs, each over two taps)
__host__ __device__ constexpr int conv_taps8() { return 10; }

// a K-major operand descriptor: start address, leading (K) and stride (8-row group) byte offsets, swizzle code
__device__ __forceinline__ uint64_t conv_desc(uint32_t addr, uint32_t lead, uint32_t stride, uint32_t swz) {
  return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)(lead >> 4) << 16) | ((uint64_t)(stride >> 4) << 32) |
         ((uint64_t)1 << 46) | ((uint64_t)swz << 61);
}

__device__ __forceinline__ void nn_tma_4d(uint32_t dst, const CUtensorMap* map, int c0, int c1, int c2, int c3,
                                          uint64_t* bar) {
  asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];"
               :: "r"(dst), "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(nn_smem_u32(bar)) : "memory");
}

__device__ __forceinline__ void nn_mma_f16(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, bool acc) {
  asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
               " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n"
               :: "r"(d), "l"(a), "l"(b), "r"(idesc), "r"((uint32_t)acc));
}

__device__ __forceinline__ void nn_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
               :: "r"(nn_smem_u32(bar)) : "memory");
}

__device__ __forceinline__ void nn_tmem_ld16(uint32_t addr, uint32_t (&v)[16]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, "
               "%13, %14, %15}, [%16];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                 "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
               : "r"(addr));
}
__device__ __forceinline__ void nn_tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// how the (N, H, W) pixels are cut into patches of 2^(bw + bh + bn) pixels
struct ConvTiles {
  int bw, bh, bn;                        // log2 of the patch's sides
  int tx, ty, tn;                        // patches per axis
  int H, W, N;
};

__device__ __forceinline__ void conv_tile(const ConvTiles& g, int t, int& x0, int& y0, int& n0) {
  const int q = t / g.tx, r = q / g.ty;
  x0 = (t - q * g.tx) << g.bw; y0 = (q - r * g.ty) << g.bh; n0 = r << g.bn;
}

// the pixel of row r of a patch, or -1 outside the lattice
__device__ __forceinline__ long long conv_pixel(const ConvTiles& g, int x0, int y0, int n0, int r) {
  const int x = x0 + (r & ((1 << g.bw) - 1)), y = y0 + ((r >> g.bw) & ((1 << g.bh) - 1)), n = n0 + (r >> (g.bw + g.bh));
  return x < g.W && y < g.H && n < g.N ? ((long long)n * g.H + y) * g.W + x : -1;
}

// shared set-up and tear-down of the pipelined kernels: barriers, tensor memory
__device__ __forceinline__ uint32_t conv_begin(NNPipeShared* sh, int stages, int columns) {
  const int tid = threadIdx.x;
  if (tid < 32) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                 :: "r"(nn_smem_u32(&sh->tslot)), "r"(columns));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (tid == 32) {
    for (int s = 0; s < stages; s++) { nn_mbar_init(&sh->full[s], 1); nn_mbar_init(&sh->empty[s], 1); }
    for (int a = 0; a < 2; a++) { nn_mbar_init(&sh->tfull[a], 1); nn_mbar_init(&sh->tempty[a], 4); }
    sh->abort = 0; sh->issued = 0; sh->consumed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  return sh->tslot;
}

__device__ __forceinline__ void conv_end(NNPipeShared* sh, int stages, int columns, uint32_t taddr) {
  const int tid = threadIdx.x;
  __syncthreads();
  if (*(volatile int*)&sh->abort && tid == 0) {
    // a bounded wait gave up: the slices still loading and the MMAs last committed get one more bounded wait each
    // before the shared and tensor memory are released
    const long long iss = *(volatile long long*)&sh->issued, con = *(volatile long long*)&sh->consumed;
    for (long long g = con; g < iss; g++)
      nn_wait_or_abort(&sh->full[g % stages], (uint32_t)((g / stages) & 1), nullptr);
    if (con > 0) nn_wait_or_abort(&sh->empty[(con - 1) % stages], (uint32_t)(((con - 1) / stages) & 1), nullptr);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (tid < 32) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(taddr), "r"(columns));
}

// a ring position: stage and the parity of its current use
struct Ring {
  int s = 0; uint32_t phase = 0;
  __device__ __forceinline__ void next(int stages) { if (++s == stages) { s = 0; phase ^= 1; } }
};

// Y[p, yc0 + o] = act(bias[o] + sum_{tap, c} X[p + shift(tap), c] W[o][tap C + c]) in BF16; with Yup also the nearest
// x2 upsampled copy (a (N, 2H, 2W) buffer of channel stride ups, offset up0). Persistent, one CTA per SM, the roles of
// the plain GEMM (TMA producer, MMA issuer, four epilogue warps over two TMEM accumulators): the loads run up to
// 8 slices ahead, a tile's epilogue overlaps the next tile's MMAs.
template <int CK>
__global__ void __launch_bounds__(NN_PIPE_THREADS, 1) k_conv3x3(const __grid_constant__ CUtensorMap mX,
                                                                const __grid_constant__ CUtensorMap mW, ConvTiles geo,
                                                                int C, int Co, int tcols, int stages,
                                                                const float* __restrict__ bias, int relu,
                                                                __nv_bfloat16* __restrict__ Y, int ys, int y0c,
                                                                __nv_bfloat16* __restrict__ Yup, int ups, int up0,
                                                                int* err) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  constexpr int TAPS8 = conv_taps8();
  constexpr uint32_t a_bytes = CK == 8 ? TAPS8 * NN_BM * 16 : NN_BM * CK * 2;
  const uint32_t b_tap = (uint32_t)Co * 16, b_bytes = CK == 8 ? TAPS8 * b_tap : (uint32_t)Co * CK * 2;
  const uint32_t stage_bytes = a_bytes + ((b_bytes + 1023) & ~1023u);
  NNPipeShared* sh = reinterpret_cast<NNPipeShared*>(base + (size_t)stages * stage_bytes);
  volatile int* abort = &sh->abort;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int tiles = geo.tx * geo.ty * geo.tn;
  const uint32_t sbase = nn_smem_u32(base);
  const uint32_t taddr = conv_begin(sh, stages, 2 * tcols);
  const int nslice = CK == 8 ? 1 : 9 * (C / CK);

  if (warp == 4 && lane == 0) {                                   // ---- TMA producer
    Ring r;
    long long g = 0;
    bool ok = true;
    for (int t = blockIdx.x; t < tiles && ok; t += gridDim.x) {
      int x0, y0, n0;
      conv_tile(geo, t, x0, y0, n0);
      for (int tap = 0, sl = 0; sl < nslice && ok; tap++)
        for (int c = 0; c < C; c += CK, sl++, g++) {
          if (g >= stages && !nn_wait_or_abort(&sh->empty[r.s], r.phase ^ 1, abort)) { nn_fail(abort, err); ok = false; break; }
          const uint32_t sa = sbase + r.s * stage_bytes;
          nn_mbar_expect_tx(&sh->full[r.s], a_bytes + b_bytes);
          if (CK == 8) {
            // tap 9 lies past the last image and past the weights' columns: zeros
            for (int k = 0; k < TAPS8; k++) {
              const int ky = k / 3, kx = k - 3 * ky;
              nn_tma_4d(sa + k * NN_BM * 16, &mX, 0, x0 + kx - 1, y0 + ky - 1, k < 9 ? n0 : geo.N, &sh->full[r.s]);
              nn_tma_2d(base + r.s * stage_bytes + a_bytes + k * b_tap, &mW, 8 * k, 0, &sh->full[r.s]);
            }
          } else {
            const int ky = tap / 3, kx = tap - 3 * ky;
            nn_tma_4d(sa, &mX, c, x0 + kx - 1, y0 + ky - 1, n0, &sh->full[r.s]);
            nn_tma_2d(base + r.s * stage_bytes + a_bytes, &mW, tap * C + c, 0, &sh->full[r.s]);
          }
          *(volatile long long*)&sh->issued = g + 1;
          r.next(stages);
        }
    }
  } else if (warp == 5 && lane == 0) {                            // ---- MMA issuer
    const uint32_t idesc = idesc_bf16(Co);
    Ring r, a;
    long long g = 0;
    bool ok = true;
    int it = 0;
    for (int t = blockIdx.x; t < tiles && ok; t += gridDim.x, it++) {
      if (it >= 2 && !nn_wait_or_abort(&sh->tempty[a.s], a.phase ^ 1, abort)) { nn_fail(abort, err); break; }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t acc = taddr + (uint32_t)(a.s * tcols);
      for (int sl = 0; sl < nslice; sl++, g++) {
        if (!nn_wait_or_abort(&sh->full[r.s], r.phase, abort)) { nn_fail(abort, err); ok = false; break; }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t sa = sbase + r.s * stage_bytes, sb = sa + a_bytes;
        if (CK == 8) {
#pragma unroll
          for (int j = 0; j < TAPS8 / 2; j++)
            nn_mma_f16(acc, conv_desc(sa + 2 * j * NN_BM * 16, NN_BM * 16, 128, 0),
                       conv_desc(sb + 2 * j * b_tap, b_tap, 128, 0), idesc, j > 0);
        } else {
          constexpr uint32_t grp = CK * 16, swz = CK == 64 ? 2 : 4;        // 8 rows of CK bf16; swizzle code
#pragma unroll
          for (int j = 0; j < CK / 16; j++)
            nn_mma_f16(acc, conv_desc(sa + 32 * j, 16, grp, swz), conv_desc(sb + 32 * j, 16, grp, swz), idesc,
                       sl > 0 || j > 0);
        }
        nn_commit(&sh->empty[r.s]);
        *(volatile long long*)&sh->consumed = g + 1;
        r.next(stages);
      }
      if (!ok) break;
      nn_commit(&sh->tfull[a.s]);
      a.next(2);
    }
  } else if (warp < 4) {                                          // ---- epilogue
    Ring a;
    for (int t = blockIdx.x; t < tiles; t += gridDim.x) {
      if (__any_sync(0xffffffffu, *abort != 0)) break;            // warp-uniform: the tcgen05.ld below are .aligned
      int x0, y0, n0;
      conv_tile(geo, t, x0, y0, n0);
      const long long p = conv_pixel(geo, x0, y0, n0, 32 * warp + lane);
      const bool got = nn_wait_or_abort(&sh->tfull[a.s], a.phase, abort);
      if (!__all_sync(0xffffffffu, got)) { if (lane == 0) nn_fail(abort, err); break; }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t tm = taddr + ((uint32_t)(32 * warp) << 16) + (uint32_t)(a.s * tcols);
      __nv_bfloat16* out = Y + (p < 0 ? 0 : p) * ys + y0c;
      __nv_bfloat16* upo = nullptr;
      if (Yup && p >= 0) {
        const long long q = p / geo.W;                            // (n H + y), x: rows 2 (n H + y) and + 1 of 2W pixels
        upo = Yup + (4 * q * geo.W + 2 * (p - q * geo.W)) * ups + up0;
      }
      const long long uprow = 2LL * geo.W * ups;
      for (int c0 = 0; c0 < Co; c0 += 16) {
        uint32_t v[16];
        nn_tmem_ld16(tm + c0, v);
        nn_tmem_wait_ld();
        if (p >= 0) {
          __nv_bfloat162 h[8];
#pragma unroll
          for (int i = 0; i < 8; i++) {
            float lo = __ldg(bias + c0 + 2 * i) + __uint_as_float(v[2 * i]);
            float hi = __ldg(bias + c0 + 2 * i + 1) + __uint_as_float(v[2 * i + 1]);
            if (relu) { lo = fmaxf(lo, 0.0f); hi = fmaxf(hi, 0.0f); }
            h[i] = __floats2bfloat162_rn(lo, hi);
          }
          const uint4 w0 = *reinterpret_cast<uint4*>(&h[0]), w1 = *reinterpret_cast<uint4*>(&h[4]);
          *reinterpret_cast<uint4*>(out + c0) = w0; *reinterpret_cast<uint4*>(out + c0 + 8) = w1;
          if (upo) {
#pragma unroll
            for (int i = 0; i < 4; i++) {
              __nv_bfloat16* o = upo + (i >> 1) * uprow + (i & 1) * ups + c0;
              *reinterpret_cast<uint4*>(o) = w0; *reinterpret_cast<uint4*>(o + 8) = w1;
            }
          }
        }
      }
      // this warp's accumulator reads are done: the MMA issuer may overwrite the accumulator
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" :: "r"(nn_smem_u32(&sh->tempty[a.s])) : "memory");
      a.next(2);
    }
  }
  conv_end(sh, stages, 2 * tcols, taddr);
}

// ----------------------------------------------------------------------------------------------------- host side
// the patch of `pixels` (a power of two) pixels that covers (N, H, W) with the fewest patches, then with the fewest
// pixels in its nine shifted views together (a square one: neighbouring views share most of their lines)
static ConvTiles conv_tiles(int N, int H, int W, int pixels) {
  int lg = 0;
  while ((1 << lg) < pixels) lg++;
  auto cd = [](int a, int s) { return (a + (1 << s) - 1) >> s; };
  ConvTiles best{};
  long long bt = -1, bh_ = 0;
  for (int bw = 0; bw <= lg; bw++)
    for (int bh = 0; bh + bw <= lg; bh++) {
      const int bn = lg - bw - bh;
      const long long t = (long long)cd(W, bw) * cd(H, bh) * cd(N, bn), h = (long long)((1 << bw) + 2) * ((1 << bh) + 2) << bn;
      if (bt < 0 || t < bt || (t == bt && h < bh_) || (t == bt && h == bh_ && bw > best.bw)) {
        bt = t; bh_ = h;
        best = {bw, bh, bn, cd(W, bw), cd(H, bh), cd(N, bn), H, W, N};
      }
    }
  return best;
}

// an NHWC BF16 channel slice [c0, c0 + C) of stride Cs as a 4-D map with patches of CK channels; zeros outside
static int conv_map_x(CUtensorMap* m, const void* X, int C, int Cs, const ConvTiles& g, int CK) {
  NNEncodeFn fn = nn_encode();
  if (!fn) { set_error("conv: cuTensorMapEncodeTiled unavailable"); return BLML_ERR_CUDA; }
  cuuint64_t dims[4] = {(cuuint64_t)C, (cuuint64_t)g.W, (cuuint64_t)g.H, (cuuint64_t)g.N};
  cuuint64_t strides[3] = {(cuuint64_t)Cs * 2, (cuuint64_t)Cs * 2 * g.W, (cuuint64_t)Cs * 2 * g.W * g.H};
  cuuint32_t box[4] = {(cuuint32_t)CK, 1u << g.bw, 1u << g.bh, 1u << g.bn};
  cuuint32_t es[4] = {1, 1, 1, 1};
  const CUtensorMapSwizzle sw = CK == 64 ? CU_TENSOR_MAP_SWIZZLE_128B : CK == 32 ? CU_TENSOR_MAP_SWIZZLE_64B
                                                                                 : CU_TENSOR_MAP_SWIZZLE_NONE;
  CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(X), dims, strides, box, es,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, sw, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) { set_error("conv: tensor map encoding failed (%d)", (int)r); return BLML_ERR_CUDA; }
  return BLML_OK;
}

// a row-major BF16 matrix [rows x K], boxes of CK columns and box_rows rows
static int conv_map_w(CUtensorMap* m, const void* Wt, int64_t K, int64_t rows, int box_rows, int CK) {
  NNEncodeFn fn = nn_encode();
  if (!fn) { set_error("conv: cuTensorMapEncodeTiled unavailable"); return BLML_ERR_CUDA; }
  cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)(K * 2)};
  cuuint32_t box[2] = {(cuuint32_t)CK, (cuuint32_t)box_rows};
  cuuint32_t es[2] = {1, 1};
  const CUtensorMapSwizzle sw = CK == 64 ? CU_TENSOR_MAP_SWIZZLE_128B : CK == 32 ? CU_TENSOR_MAP_SWIZZLE_64B
                                                                                 : CU_TENSOR_MAP_SWIZZLE_NONE;
  CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(Wt), dims, strides, box, es,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, sw, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) { set_error("conv: tensor map encoding failed (%d)", (int)r); return BLML_ERR_CUDA; }
  return BLML_OK;
}

static bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

constexpr size_t kConvSmemMax = 227 * 1024;

static int conv_sms() {
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return sms;
}

// shared memory of a pipelined kernel: as many slices as fit (at most 8), more than half an SM so one CTA per SM
static size_t conv_smem(size_t stage_bytes, int& stages) {
  const size_t fixed = 1024 + sizeof(NNPipeShared);
  stages = (int)std::min<size_t>(NN_MAX_STAGES, (kConvSmemMax - fixed) / stage_bytes);
  return std::max<size_t>(fixed + (size_t)stages * stage_bytes, 120 * 1024);
}

template <typename F>
static int conv_smem_limit(F kernel) {
  return cuda_status(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kConvSmemMax), "conv");
}

}  // namespace blml

using namespace blml;

extern "C" {

int blml_nn_conv3x3(const void* X, int Nb, int H, int W, int Cs, int c0, int C, const void* Wt, const float* bias,
                    int relu, int Co, void* Y, int Ys, int y0, void* Yup, int Ups, int up0, int* err, void* stream) {
  if (!X || !Wt || !bias || !Y || !err || Nb < 1 || H < 1 || W < 1 || c0 < 0 || C < 1 || c0 + C > Cs || y0 < 0 ||
      Co < 1 || y0 + Co > Ys || (Yup && (up0 < 0 || up0 + Co > Ups))) {
    set_error("blml_nn_conv3x3: bad arguments"); return BLML_ERR_ARG;
  }
  const __nv_bfloat16* Xs = (const __nv_bfloat16*)X + c0;
  if ((C != 8 && C % 32) || Co % 16 || Co > 256 || Cs % 8 || c0 % 8 || Ys % 8 || y0 % 8 || !aligned16(X) ||
      !aligned16(Wt) || !aligned16(Y) || (Yup && (Ups % 8 || up0 % 8 || !aligned16(Yup)))) {
    set_error("blml_nn_conv3x3: 8 or a multiple of 32 input channels, a multiple of 16 (at most 256) output channels, "
              "16-byte aligned slices");
    return BLML_ERR_UNSUPPORTED;
  }
  const int CK = C == 8 ? 8 : C % 64 == 0 ? 64 : 32;
  const ConvTiles g = conv_tiles(Nb, H, W, NN_BM);
  CUtensorMap mX, mW;
  int e = conv_map_x(&mX, Xs, C, Cs, g, CK);
  if (!e) e = conv_map_w(&mW, Wt, 9LL * C, Co, Co, CK);
  if (e) return e;
  int tcols = 32;
  while (tcols < Co) tcols <<= 1;                                 // two accumulators: 2 tcols <= 512 TMEM columns
  const size_t a = CK == 8 ? (size_t)conv_taps8() * NN_BM * 16 : (size_t)NN_BM * CK * 2;
  const size_t b = CK == 8 ? (size_t)conv_taps8() * Co * 16 : (size_t)Co * CK * 2;
  int stages = 0;
  const size_t smem = conv_smem(a + ((b + 1023) & ~(size_t)1023), stages);
  auto kern = CK == 64 ? k_conv3x3<64> : CK == 32 ? k_conv3x3<32> : k_conv3x3<8>;
  e = conv_smem_limit(kern);
  if (e) return e;
  const int tiles = g.tx * g.ty * g.tn;
  kern<<<std::min(tiles, conv_sms()), NN_PIPE_THREADS, smem, reinterpret_cast<cudaStream_t>(stream)>>>(
      mX, mW, g, C, Co, tcols, stages, bias, relu, (__nv_bfloat16*)Y, Ys, y0, (__nv_bfloat16*)Yup, Ups, up0, err);
  BLML_CHECK_LAUNCH("blml_nn_conv3x3");
  return BLML_OK;
}

}
