// The warm start's 3 x 3 convolutions (pad 1) as implicit GEMMs on tcgen05: the nine shifted views of the NHWC
// activation are never written out. A tile of 128 output pixels is a BW x BH x BN patch (powers of two) of the
// lattice; its operand for tap (ky, kx) is the same patch moved by (kx - 1, ky - 1), one 4-D TMA box per slice of
// channels whose out-of-range pixels the copy fills with zeros -- the convolution's padding. The products run in the
// order of the explicit form (tap by tap, channels ascending, 16 at a time into one FP32 accumulator), so the results
// are those of an im2col matrix and a GEMM, bit for bit.
//
// Bound: an im2col matrix is 9 x the activation written and read again (453 MB each way for the 96-channel decoder
// layer on 16 x 128 x 128 pixels) for a product of 14.5 GFLOP; here each pixel comes from L2 nine times and from HBM
// once, so what is left is the L2 reads: 8-9 TB/s on the wide layers, 4-6 TB/s where a pixel is 64 bytes (32 channels:
// the copies' requests bound it). On 16 x 128 x 128 pixels: the 14 forward layers 412 us (im2col alone took 5.3 ms), a
// forward pass 6.2 -> 0.49 ms; the backward layers' gradients 1.2 ms, a training step 16.1 -> 2.4 ms.
#include "nn_tc.cuh"

namespace blml {

// channels per K slice: 64 (128-byte rows, 128B swizzle), 32 (64-byte rows, 64B swizzle), 8 (the input layer: 16-byte
// rows, no swizzle; its nine taps and a zero tenth are one K = 80 slice of five MMAs, each over two taps)
constexpr int kConvTaps8 = 10;
// one slice of the weights [Co x CK] in shared memory (Co a multiple of 16: whole swizzle atoms)
__host__ __device__ constexpr uint32_t conv_w_bytes(int CK, int Co) {
  return CK == 8 ? (uint32_t)kConvTaps8 * Co * 16 : (uint32_t)Co * CK * 2;
}

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

__device__ __forceinline__ void nn_tma_3d(uint32_t dst, const CUtensorMap* map, int c0, int c1, int c2, uint64_t* bar) {
  asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
               :: "r"(dst), "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(nn_smem_u32(bar)) : "memory");
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

// the pipeline's state: a ring of up to kConvStages slices, two accumulators, and a barrier of the operand that is
// loaded once per CTA
constexpr int kConvStages = 20;
struct ConvPipe {
  uint64_t full[kConvStages], empty[kConvStages], tfull[2], tempty[2], once;
  uint32_t tslot;
  int abort, once_issued;               // (once_issued: the load behind `once` has been started)
  long long issued, consumed;           // slices loaded by the producer / taken by the MMA issuer
};

// shared set-up and tear-down of the pipelined kernels: barriers, tensor memory
__device__ __forceinline__ uint32_t conv_begin(ConvPipe* sh, int stages, int columns) {
  const int tid = threadIdx.x;
  if (tid < 32) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                 :: "r"(nn_smem_u32(&sh->tslot)), "r"(columns));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (tid == 32) {
    for (int s = 0; s < stages; s++) { nn_mbar_init(&sh->full[s], 1); nn_mbar_init(&sh->empty[s], 1); }
    for (int a = 0; a < 2; a++) { nn_mbar_init(&sh->tfull[a], 1); nn_mbar_init(&sh->tempty[a], 4); }
    nn_mbar_init(&sh->once, 1);
    sh->abort = 0; sh->once_issued = 0; sh->issued = 0; sh->consumed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  return sh->tslot;
}

__device__ __forceinline__ void conv_end(ConvPipe* sh, int stages, int columns, uint32_t taddr) {
  const int tid = threadIdx.x;
  __syncthreads();
  if (*(volatile int*)&sh->abort && tid == 0) {
    // a bounded wait gave up: the resident operand and the slices still loading and the MMAs last committed get one more
    // bounded wait each before the shared and tensor memory are released
    if (*(volatile int*)&sh->once_issued) nn_wait_or_abort(&sh->once, 0, nullptr);
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
// 20 slices ahead, a tile's epilogue overlaps the next tile's MMAs. wonce: the whole weight matrix is loaded once per
// CTA (it fits beside enough slices) and only the activation streams.
template <int CK>
__global__ void __launch_bounds__(NN_PIPE_THREADS, 1) k_conv3x3(const __grid_constant__ CUtensorMap mX,
                                                                const __grid_constant__ CUtensorMap mW, ConvTiles geo,
                                                                int C, int Co, int tcols, int stages, int wonce,
                                                                const float* __restrict__ bias, int relu,
                                                                __nv_bfloat16* __restrict__ Y, int ys, int y0c,
                                                                __nv_bfloat16* __restrict__ Yup, int ups, int up0,
                                                                int* err) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  constexpr uint32_t a_bytes = CK == 8 ? kConvTaps8 * NN_BM * 16 : NN_BM * CK * 2;
  const int nslice = CK == 8 ? 1 : 9 * (C / CK);
  const uint32_t b_bytes = conv_w_bytes(CK, Co), stage_bytes = a_bytes + (wonce ? 0 : b_bytes);
  uint8_t* wbase = base + (size_t)stages * stage_bytes;            // the resident weights
  ConvPipe* sh = reinterpret_cast<ConvPipe*>(wbase + (wonce ? (size_t)nslice * b_bytes : 0));
  volatile int* abort = &sh->abort;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int tiles = geo.tx * geo.ty * geo.tn;
  const uint32_t sbase = nn_smem_u32(base);
  const uint32_t taddr = conv_begin(sh, stages, 2 * tcols);

  // the weights of slice sl (tap, c) to shared memory
  auto load_w = [&](uint8_t* dst, int tap, int c, uint64_t* bar) {
    if (CK == 8)                                                   // column 72 on: past the matrix, zeros
      for (int k = 0; k < kConvTaps8; k++) nn_tma_2d(dst + k * Co * 16, &mW, 8 * k, 0, bar);
    else
      nn_tma_2d(dst, &mW, tap * C + c, 0, bar);
  };
  if (warp == 4 && lane == 0) {                                   // ---- TMA producer
    Ring r;
    long long g = 0;
    bool ok = true;
    if (wonce) {
      nn_mbar_expect_tx(&sh->once, (uint32_t)nslice * b_bytes);
      *(volatile int*)&sh->once_issued = 1;
      for (int tap = 0, sl = 0; sl < nslice; tap++)
        for (int c = 0; c < C; c += CK, sl++) load_w(wbase + (size_t)sl * b_bytes, tap, c, &sh->once);
    }
    for (int t = blockIdx.x; t < tiles && ok; t += gridDim.x) {
      int x0, y0, n0;
      conv_tile(geo, t, x0, y0, n0);
      for (int tap = 0, sl = 0; sl < nslice && ok; tap++)
        for (int c = 0; c < C; c += CK, sl++, g++) {
          if (g >= stages && !nn_wait_or_abort(&sh->empty[r.s], r.phase ^ 1, abort)) { nn_fail(abort, err); ok = false; break; }
          const uint32_t sa = sbase + r.s * stage_bytes;
          nn_mbar_expect_tx(&sh->full[r.s], stage_bytes);
          if (CK == 8) {
            // a lattice row is one run of 8 W values: a shift by one pixel is a shift by 8 values (16 bytes); the tenth
            // tap lies past the last image: zeros
            for (int k = 0; k < kConvTaps8; k++) {
              const int ky = k / 3, kx = k - 3 * ky;
              nn_tma_3d(sa + k * NN_BM * 16, &mX, 8 * (x0 + kx - 1), y0 + ky - 1, k < 9 ? n0 : geo.N, &sh->full[r.s]);
            }
          } else {
            const int ky = tap / 3, kx = tap - 3 * ky;
            nn_tma_4d(sa, &mX, c, x0 + kx - 1, y0 + ky - 1, n0, &sh->full[r.s]);
          }
          if (!wonce) load_w(base + r.s * stage_bytes + a_bytes, tap, c, &sh->full[r.s]);
          *(volatile long long*)&sh->issued = g + 1;
          r.next(stages);
        }
    }
  } else if (warp == 5 && lane == 0) {                            // ---- MMA issuer
    const uint32_t idesc = idesc_bf16(Co), wsm = nn_smem_u32(wbase);
    Ring r, a;
    long long g = 0;
    bool ok = !wonce || nn_wait_or_abort(&sh->once, 0, abort);
    if (!ok) nn_fail(abort, err);
    int it = 0;
    for (int t = blockIdx.x; t < tiles && ok; t += gridDim.x, it++) {
      if (it >= 2 && !nn_wait_or_abort(&sh->tempty[a.s], a.phase ^ 1, abort)) { nn_fail(abort, err); break; }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t acc = taddr + (uint32_t)(a.s * tcols);
      for (int sl = 0; sl < nslice; sl++, g++) {
        if (!nn_wait_or_abort(&sh->full[r.s], r.phase, abort)) { nn_fail(abort, err); ok = false; break; }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t sa = sbase + r.s * stage_bytes, sb = wonce ? wsm + sl * b_bytes : sa + a_bytes;
        if (CK == 8) {
          const uint32_t b_tap = (uint32_t)Co * 16;
#pragma unroll
          for (int j = 0; j < kConvTaps8 / 2; j++)
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

// dX[p, c0 + c] = sum over taps, in tap order, of sum_o dPre[p - shift(tap), o] Wt[tap C + c][o] (FP32): the data
// gradient without its P x 9C matrix. Each tap's product goes into a TMEM accumulator of its own and the epilogue adds
// the nine in registers, in the order of the explicit form's gather (col2im), so the sums are the same bit for bit.
// NT input channels per tile; two accumulators, so a tap's MMAs overlap the previous tap's adds.
template <int CK, int NT>
__global__ void __launch_bounds__(NN_PIPE_THREADS, 1) k_conv3x3_dgrad(const __grid_constant__ CUtensorMap mD,
                                                                      const __grid_constant__ CUtensorMap mW,
                                                                      ConvTiles geo, int C, int Co, int stages,
                                                                      float* __restrict__ dX, int xs, int x0c, int* err) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  constexpr uint32_t a_bytes = NN_BM * CK * 2, stage_bytes = a_bytes + NT * CK * 2;
  constexpr int tcols = NT <= 32 ? 32 : NT <= 64 ? 64 : 128;
  ConvPipe* sh = reinterpret_cast<ConvPipe*>(base + (size_t)stages * stage_bytes);
  volatile int* abort = &sh->abort;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int nt = C / NT, tiles = geo.tx * geo.ty * geo.tn * nt;
  const uint32_t sbase = nn_smem_u32(base);
  const uint32_t taddr = conv_begin(sh, stages, 2 * tcols);

  if (warp == 4 && lane == 0) {                                   // ---- TMA producer
    Ring r;
    long long g = 0;
    bool ok = true;
    for (int t = blockIdx.x; t < tiles && ok; t += gridDim.x) {
      int x0, y0, n0;
      conv_tile(geo, t / nt, x0, y0, n0);
      const int cb = (t % nt) * NT;
      for (int tap = 0; tap < 9 && ok; tap++) {
        const int ky = tap / 3, kx = tap - 3 * ky;
        for (int o = 0; o < Co; o += CK, g++) {
          if (g >= stages && !nn_wait_or_abort(&sh->empty[r.s], r.phase ^ 1, abort)) { nn_fail(abort, err); ok = false; break; }
          nn_mbar_expect_tx(&sh->full[r.s], stage_bytes);
          nn_tma_4d(sbase + r.s * stage_bytes, &mD, o, x0 + 1 - kx, y0 + 1 - ky, n0, &sh->full[r.s]);
          nn_tma_2d(base + r.s * stage_bytes + a_bytes, &mW, o, tap * C + cb, &sh->full[r.s]);
          *(volatile long long*)&sh->issued = g + 1;
          r.next(stages);
        }
      }
    }
  } else if (warp == 5 && lane == 0) {                            // ---- MMA issuer
    constexpr uint32_t idesc = idesc_bf16(NT);
    Ring r, a;
    long long g = 0;
    bool ok = true;
    int it = 0;
    for (int t = blockIdx.x; t < tiles && ok; t += gridDim.x)
      for (int tap = 0; tap < 9 && ok; tap++, it++) {
        if (it >= 2 && !nn_wait_or_abort(&sh->tempty[a.s], a.phase ^ 1, abort)) { nn_fail(abort, err); ok = false; break; }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t acc = taddr + (uint32_t)(a.s * tcols);
        for (int o = 0; o < Co; o += CK, g++) {
          if (!nn_wait_or_abort(&sh->full[r.s], r.phase, abort)) { nn_fail(abort, err); ok = false; break; }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t sa = sbase + r.s * stage_bytes, sb = sa + a_bytes;
          constexpr uint32_t grp = CK * 16, swz = CK == 64 ? 2 : 4;
#pragma unroll
          for (int j = 0; j < CK / 16; j++)
            nn_mma_f16(acc, conv_desc(sa + 32 * j, 16, grp, swz), conv_desc(sb + 32 * j, 16, grp, swz), idesc,
                       o > 0 || j > 0);
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
    bool ok = true;
    for (int t = blockIdx.x; t < tiles && ok; t += gridDim.x) {
      int x0, y0, n0;
      conv_tile(geo, t / nt, x0, y0, n0);
      const int cb = (t % nt) * NT;
      const long long p = conv_pixel(geo, x0, y0, n0, 32 * warp + lane);
      float sum[NT];
#pragma unroll
      for (int c = 0; c < NT; c++) sum[c] = 0.0f;
      for (int tap = 0; tap < 9; tap++) {
        const bool got = nn_wait_or_abort(&sh->tfull[a.s], a.phase, abort);
        if (!__all_sync(0xffffffffu, got)) { if (lane == 0) nn_fail(abort, err); ok = false; break; }   // warp-uniform
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t tm = taddr + ((uint32_t)(32 * warp) << 16) + (uint32_t)(a.s * tcols);
#pragma unroll
        for (int c = 0; c < NT; c += 16) {
          uint32_t v[16];
          nn_tmem_ld16(tm + c, v);
          nn_tmem_wait_ld();
#pragma unroll
          for (int i = 0; i < 16; i++) sum[c + i] += __uint_as_float(v[i]);
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" :: "r"(nn_smem_u32(&sh->tempty[a.s])) : "memory");
        a.next(2);
      }
      if (ok && p >= 0) {
        float4* out = reinterpret_cast<float4*>(dX + p * xs + x0c + cb);
#pragma unroll
        for (int c = 0; c < NT / 4; c++) out[c] = make_float4(sum[4 * c], sum[4 * c + 1], sum[4 * c + 2], sum[4 * c + 3]);
      }
    }
  }
  conv_end(sh, stages, 2 * tcols, taddr);
}

// part[z][o][tap C + c] = sum over the pixels of split z of dPre[p, o] X[p + shift(tap), c]: the weight gradient with
// the pixels as K. Both operands are read as they lie (channels innermost: the MN-major operand forms), so neither is
// transposed and no im2col matrix is written. M: 128 rows of (tap, channel) -- 128 / CB blocks of CB channels of one tap
// each (64 with 128-byte rows, 32 with 64-byte rows, 8 with 16-byte rows) --, N: Co, K: blocks of 64 consecutive pixels
// (n, y, x), the last one filled up with zeros -- the explicit form's products in its order, so its sums bit for bit.
// A block of pixels is copied as runs that are boxes of the lattice (WgRuns). Rows past the ninth tap multiply what the
// slot happens to hold and are not stored. A work item is (128 rows, split of the pixel blocks).
constexpr int kWgPixels = 64;
// 64 consecutive pixels as 64 / run boxes of bw x bh x bn = run pixels, each a contiguous run of the lattice
struct WgRuns { int bw, bh, bn, run, H, W, N; };
template <int CB>
__global__ void __launch_bounds__(NN_PIPE_THREADS, 1) k_conv3x3_wgrad(const __grid_constant__ CUtensorMap mX,
                                                                      const __grid_constant__ CUtensorMap mD,
                                                                      WgRuns geo, int C, int Co, int tcols,
                                                                      int splits, int stages, float* __restrict__ part,
                                                                      int* err) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  constexpr int NB = NN_BM / CB;                                   // blocks of M
  constexpr uint32_t x_block = kWgPixels * CB * 2, a_bytes = NB * x_block;
  const int CO = Co % 64 == 0 ? 64 : 32;                           // channels per block of N
  const uint32_t d_block = kWgPixels * CO * 2, stage_bytes = a_bytes + (uint32_t)Co * kWgPixels * 2;
  ConvPipe* sh = reinterpret_cast<ConvPipe*>(base + (size_t)stages * stage_bytes);
  volatile int* abort = &sh->abort;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int per_tap = C / CB, blocks = 9 * per_tap, Mt = (blocks + NB - 1) / NB;
  const int patches = (int)(((long long)geo.N * geo.H * geo.W + kWgPixels - 1) / kWgPixels);
  const int per = (patches + splits - 1) / splits, items = Mt * splits;
  const uint32_t sbase = nn_smem_u32(base);
  const uint32_t taddr = conv_begin(sh, stages, 2 * tcols);

  if (warp == 4 && lane == 0) {                                   // ---- TMA producer
    Ring r;
    long long g = 0;
    bool ok = true;
    for (int t = blockIdx.x; t < items && ok; t += gridDim.x) {
      const int z = t / Mt, b0 = (t - z * Mt) * NB, nb = min(NB, blocks - b0);
      for (int q = z * per; q < min(patches, (z + 1) * per); q++, g++) {
        if (g >= stages && !nn_wait_or_abort(&sh->empty[r.s], r.phase ^ 1, abort)) { nn_fail(abort, err); ok = false; break; }
        const uint32_t sa = sbase + r.s * stage_bytes;
        nn_mbar_expect_tx(&sh->full[r.s], (uint32_t)nb * x_block + (uint32_t)Co * kWgPixels * 2);
        for (int i = 0; i < kWgPixels; i += geo.run) {             // run by run
          const long long p = (long long)q * kWgPixels + i, row = p / geo.W;
          const int x = (int)(p - row * geo.W), n = (int)(row / geo.H), y = (int)(row - (long long)n * geo.H);
          for (int b = 0; b < nb; b++) {
            const int tap = (b0 + b) / per_tap, c = (b0 + b - tap * per_tap) * CB, ky = tap / 3, kx = tap - 3 * ky;
            const uint32_t dst = sa + b * x_block + i * CB * 2;
            if (CB == 8) nn_tma_3d(dst, &mX, 8 * (x + kx - 1), y + ky - 1, n, &sh->full[r.s]);
            else nn_tma_4d(dst, &mX, c, x + kx - 1, y + ky - 1, n, &sh->full[r.s]);
          }
          for (int o = 0; o < Co; o += CO)
            nn_tma_4d(sa + a_bytes + (o / CO) * d_block + i * CO * 2, &mD, o, x, y, n, &sh->full[r.s]);
        }
        *(volatile long long*)&sh->issued = g + 1;
        r.next(stages);
      }
    }
  } else if (warp == 5 && lane == 0) {                            // ---- MMA issuer
    const uint32_t idesc = idesc_bf16(Co) | (1u << 15) | (1u << 16);       // both operands MN-major
    // swizzled: leading offset = the next block of channels, stride offset = the next 8 pixels; unswizzled (CB = 8)
    // the other way round
    constexpr uint32_t xr = CB * 2, xswz = CB == 64 ? 2 : CB == 32 ? 4 : 0;
    const uint32_t dr = CO * 2, dswz = CO == 64 ? 2 : 4;
    Ring r, a;
    long long g = 0;
    bool ok = true;
    int it = 0;
    for (int t = blockIdx.x; t < items && ok; t += gridDim.x) {
      const int z = t / Mt, q0 = z * per, q1 = min(patches, (z + 1) * per);
      if (q0 >= q1) continue;
      if (it >= 2 && !nn_wait_or_abort(&sh->tempty[a.s], a.phase ^ 1, abort)) { nn_fail(abort, err); break; }
      it++;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t acc = taddr + (uint32_t)(a.s * tcols);
      for (int q = q0; q < q1; q++, g++) {
        if (!nn_wait_or_abort(&sh->full[r.s], r.phase, abort)) { nn_fail(abort, err); ok = false; break; }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t sa = sbase + r.s * stage_bytes, sb = sa + a_bytes;
#pragma unroll
        for (int j = 0; j < kWgPixels / 16; j++)
          nn_mma_f16(acc, CB == 8 ? conv_desc(sa + 16 * xr * j, 8 * xr, x_block, 0) : conv_desc(sa + 16 * xr * j, x_block, 8 * xr, xswz),
                     conv_desc(sb + 16 * dr * j, d_block, 8 * dr, dswz), idesc, q > q0 || j > 0);
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
    const size_t K9 = 9 * (size_t)C;
    for (int t = blockIdx.x; t < items; t += gridDim.x) {
      if (__any_sync(0xffffffffu, *abort != 0)) break;
      const int z = t / Mt, row = (t - z * Mt) * NN_BM + 32 * warp + lane;        // (tap C + c): blocks are in that order
      float* out = part + (size_t)z * Co * K9 + row;
      const bool mine = row < (int)K9;
      if (z * per >= patches) {                                   // no pixels in this split: the partial is zero
        for (int o = 0; o < Co && mine; o++) out[o * K9] = 0.0f;
        continue;
      }
      const bool got = nn_wait_or_abort(&sh->tfull[a.s], a.phase, abort);
      if (!__all_sync(0xffffffffu, got)) { if (lane == 0) nn_fail(abort, err); break; }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t tm = taddr + ((uint32_t)(32 * warp) << 16) + (uint32_t)(a.s * tcols);
      for (int o = 0; o < Co; o += 16) {
        uint32_t v[16];
        nn_tmem_ld16(tm + o, v);
        nn_tmem_wait_ld();
        if (mine) {
#pragma unroll
          for (int i = 0; i < 16; i++) out[(o + i) * K9] = __uint_as_float(v[i]);
        }
      }
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
static ConvTiles conv_tiles(int N, int H, int W, int pixels, int max_bw = 7) {
  int lg = 0;
  while ((1 << lg) < pixels) lg++;
  auto cd = [](int a, int s) { return (a + (1 << s) - 1) >> s; };
  ConvTiles best{};
  long long bt = -1, bh_ = 0;
  for (int bw = 0; bw <= std::min(lg, max_bw); bw++)
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

// an NHWC BF16 channel slice [c0, c0 + C) of stride Cs as a 4-D map with bw x bh x bn boxes of CK channels; zeros outside
struct ConvBox { int bw, bh, bn, H, W, N; };
static int conv_map_x(CUtensorMap* m, const void* X, int C, int Cs, const ConvBox& g, int CK) {
  NNEncodeFn fn = nn_encode();
  if (!fn) { set_error("conv: cuTensorMapEncodeTiled unavailable"); return BLML_ERR_CUDA; }
  const bool runs = CK == 8;             // 8 channels: a lattice row as one run of 8 W values
  const int k = runs ? 1 : 0;
  cuuint64_t dims[4] = {(cuuint64_t)C, (cuuint64_t)g.W, (cuuint64_t)g.H, (cuuint64_t)g.N};
  cuuint64_t strides[3] = {(cuuint64_t)Cs * 2, (cuuint64_t)Cs * 2 * g.W, (cuuint64_t)Cs * 2 * g.W * g.H};
  cuuint32_t box[4] = {(cuuint32_t)CK, (cuuint32_t)g.bw, (cuuint32_t)g.bh, (cuuint32_t)g.bn};
  cuuint32_t es[4] = {1, 1, 1, 1};
  if (runs) { dims[1] *= 8; box[1] *= 8; }
  const CUtensorMapSwizzle sw = CK == 64 ? CU_TENSOR_MAP_SWIZZLE_128B : CK == 32 ? CU_TENSOR_MAP_SWIZZLE_64B
                                                                                 : CU_TENSOR_MAP_SWIZZLE_NONE;
  CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4 - k, const_cast<void*>(X), dims + k, strides + k, box + k, es,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, sw, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) { set_error("conv: tensor map encoding failed (%d)", (int)r); return BLML_ERR_CUDA; }
  return BLML_OK;
}

static ConvBox conv_box(const ConvTiles& g) { return {1 << g.bw, 1 << g.bh, 1 << g.bn, g.H, g.W, g.N}; }

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

// shared memory of a pipelined kernel: `once` bytes, as many slices as fit beside them, more than half an SM so that
// one CTA runs per SM
static size_t conv_smem(size_t once, size_t stage_bytes, int& stages) {
  const size_t fixed = 1024 + sizeof(ConvPipe) + once;
  stages = (int)std::min<size_t>(kConvStages, (kConvSmemMax - fixed) / stage_bytes);
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
  if ((C == 8 ? Cs != 8 : C % 32 != 0) || Co % 16 || Co > 256 || Cs % 8 || c0 % 8 || Ys % 8 || y0 % 8 || !aligned16(X) ||
      !aligned16(Wt) || !aligned16(Y) || (Yup && (Ups % 8 || up0 % 8 || !aligned16(Yup)))) {
    set_error("blml_nn_conv3x3: 8 input channels (a buffer of its own) or a multiple of 32, a multiple of 16 (at most 256) output channels, "
              "16-byte aligned slices");
    return BLML_ERR_UNSUPPORTED;
  }
  const int CK = C == 8 ? 8 : C % 64 == 0 ? 64 : 32;
  const ConvTiles g = conv_tiles(Nb, H, W, NN_BM, CK == 8 ? 5 : 7);
  CUtensorMap mX, mW;
  int e = conv_map_x(&mX, Xs, C, Cs, conv_box(g), CK);
  if (!e) e = conv_map_w(&mW, Wt, 9LL * C, Co, Co, CK);
  if (e) return e;
  int tcols = 32;
  while (tcols < Co) tcols <<= 1;                                 // two accumulators: 2 tcols <= 512 TMEM columns
  // the weights stay in shared memory when they leave room for 100 KB of slices
  const size_t a = CK == 8 ? (size_t)kConvTaps8 * NN_BM * 16 : (size_t)NN_BM * CK * 2, b = conv_w_bytes(CK, Co);
  const size_t wall = b * (CK == 8 ? 1 : 9 * (C / CK));
  const int wonce = wall <= 120 * 1024;
  int stages = 0;
  const size_t smem = conv_smem(wonce ? wall : 0, a + (wonce ? 0 : b), stages);
  auto kern = CK == 64 ? k_conv3x3<64> : CK == 32 ? k_conv3x3<32> : k_conv3x3<8>;
  e = conv_smem_limit(kern);
  if (e) return e;
  const int tiles = g.tx * g.ty * g.tn;
  kern<<<std::min(tiles, conv_sms()), NN_PIPE_THREADS, smem, reinterpret_cast<cudaStream_t>(stream)>>>(
      mX, mW, g, C, Co, tcols, stages, wonce, bias, relu, (__nv_bfloat16*)Y, Ys, y0, (__nv_bfloat16*)Yup, Ups, up0, err);
  BLML_CHECK_LAUNCH("blml_nn_conv3x3");
  return BLML_OK;
}

int blml_nn_conv3x3_dgrad(const void* dpre, int Nb, int H, int W, int Co, const void* Wt, int C, float* dX, int Xs,
                          int x0, int* err, void* stream) {
  if (!dpre || !Wt || !dX || !err || Nb < 1 || H < 1 || W < 1 || C < 1 || Co < 1 || x0 < 0 || x0 + C > Xs) {
    set_error("blml_nn_conv3x3_dgrad: bad arguments"); return BLML_ERR_ARG;
  }
  if (C % 32 || Co % 32 || Xs % 4 || x0 % 4 || !aligned16(dpre) || !aligned16(Wt) || !aligned16(dX)) {
    set_error("blml_nn_conv3x3_dgrad: channels in multiples of 32, 16-byte aligned slices");
    return BLML_ERR_UNSUPPORTED;
  }
  const int CK = Co % 64 == 0 ? 64 : 32;
  const int NT = C % 128 == 0 ? 128 : C % 96 == 0 ? 96 : C % 64 == 0 ? 64 : 32;     // 16 registers of a thread per 16
  const ConvTiles g = conv_tiles(Nb, H, W, NN_BM);
  CUtensorMap mD, mW;
  int e = conv_map_x(&mD, dpre, Co, Co, conv_box(g), CK);
  if (!e) e = conv_map_w(&mW, Wt, Co, 9LL * C, NT, CK);
  if (e) return e;
  int stages = 0;
  const size_t smem = conv_smem(0, (size_t)(NN_BM + NT) * CK * 2, stages);
  const int tiles = g.tx * g.ty * g.tn * (C / NT), grid = std::min(tiles, conv_sms());
  auto run = [&](auto kern) -> int {
    int er = conv_smem_limit(kern);
    if (er) return er;
    kern<<<grid, NN_PIPE_THREADS, smem, reinterpret_cast<cudaStream_t>(stream)>>>(mD, mW, g, C, Co, stages, dX, Xs, x0, err);
    BLML_CHECK_LAUNCH("blml_nn_conv3x3_dgrad");
    return BLML_OK;
  };
  if (CK == 64)
    return NT == 128 ? run(k_conv3x3_dgrad<64, 128>) : NT == 96 ? run(k_conv3x3_dgrad<64, 96>)
         : NT == 64 ? run(k_conv3x3_dgrad<64, 64>) : run(k_conv3x3_dgrad<64, 32>);
  return NT == 128 ? run(k_conv3x3_dgrad<32, 128>) : NT == 96 ? run(k_conv3x3_dgrad<32, 96>)
       : NT == 64 ? run(k_conv3x3_dgrad<32, 64>) : run(k_conv3x3_dgrad<32, 32>);
}

int blml_nn_conv3x3_wgrad(const void* X, int Nb, int H, int W, int Cs, int c0, int C, const void* dpre, int Co,
                          int splits, float* part, float* dW, int* err, void* stream) {
  if (!X || !dpre || !part || !dW || !err || Nb < 1 || H < 1 || W < 1 || c0 < 0 || C < 1 || c0 + C > Cs || Co < 1 ||
      splits < 1 || splits > 4096) {
    set_error("blml_nn_conv3x3_wgrad: bad arguments"); return BLML_ERR_ARG;
  }
  if ((C == 8 ? Cs != 8 : C % 32 != 0) || Co % 32 || Co > 256 || Cs % 8 || c0 % 8 || !aligned16(X) || !aligned16(dpre)) {
    set_error("blml_nn_conv3x3_wgrad: 8 input channels (a buffer of its own) or a multiple of 32, output channels a "
              "multiple of 32 (at most 256), 16-byte aligned slices");
    return BLML_ERR_UNSUPPORTED;
  }
  const int CB = C == 8 ? 8 : C % 64 == 0 ? 64 : 32;
  const int CO = Co % 64 == 0 ? 64 : 32;
  // the longest run of 2^k pixels that divides the rows (whole rows: the lattices' rows too, then the images)
  auto pow2_in = [](int m, int most) { int r = 1; while (r < most && m % (2 * r) == 0) r *= 2; return r; };
  WgRuns g{1, 1, 1, 1, H, W, Nb};
  g.bw = pow2_in(W, CB == 8 ? 32 : kWgPixels);                     // (CB = 8: a box row of at most 256 values)
  if (g.bw == W) {
    g.bh = pow2_in(H, kWgPixels / g.bw);
    if (g.bh == H) g.bn = kWgPixels / (g.bw * g.bh);
  }
  g.run = g.bw * g.bh * g.bn;
  if (g.run * CB * 2 % 128 || g.run * CO * 2 % 128) {              // a copy starts on a 128-byte boundary
    set_error("blml_nn_conv3x3_wgrad: lattice rows of %d pixels do not split into 128-byte runs", W);
    return BLML_ERR_UNSUPPORTED;
  }
  const ConvBox box{g.bw, g.bh, g.bn, H, W, Nb};
  CUtensorMap mX, mD;
  int e = conv_map_x(&mX, (const __nv_bfloat16*)X + c0, C, Cs, box, CB);
  if (!e) e = conv_map_x(&mD, dpre, Co, Co, box, CO);
  if (e) return e;
  int tcols = 32;
  while (tcols < Co) tcols <<= 1;
  int stages = 0;
  const size_t smem = conv_smem(0, (size_t)(NN_BM + Co) * kWgPixels * 2, stages);
  const int NB = NN_BM / CB, items = (9 * (C / CB) + NB - 1) / NB * splits;
  auto run = [&](auto kern) -> int {
    int er = conv_smem_limit(kern);
    if (er) return er;
    kern<<<std::min(items, conv_sms()), NN_PIPE_THREADS, smem, reinterpret_cast<cudaStream_t>(stream)>>>(
        mX, mD, g, C, Co, tcols, splits, stages, part, err);
    BLML_CHECK_LAUNCH("blml_nn_conv3x3_wgrad");
    return BLML_OK;
  };
  e = CB == 64 ? run(k_conv3x3_wgrad<64>) : CB == 32 ? run(k_conv3x3_wgrad<32>) : run(k_conv3x3_wgrad<8>);
  if (e) return e;
  return blml_nn_sum_splits(part, splits, 9LL * C * Co, dW, stream);
}

}
