// Kernels of the learned warm start for Liu-Shen: a small encoder-decoder CNN over
// bfloat16 NHWC activations with float32 accumulation.
//
//  of_cnn_conv3x3   3x3 convolution, zero padding, as an implicit GEMM on the 5th-gen
//                   tensor cores: M = 128 output pixels (a bh x bw patch of one image, or
//                   nb whole images when an image has fewer than 128 pixels),
//                   N = output channels (<= 256 per CTA), K = 9 taps x input channels.
//                   Warp 0 streams A (the input patch shifted by the tap; TMA fills the
//                   zero padding) and B (the tap's weights) into a 4-stage shared-memory
//                   ring; one thread of warp 1 issues tcgen05.mma into a TMEM accumulator;
//                   warps 2-5 read TMEM back (one pixel per thread) and apply bias, ReLU
//                   and the bf16 / f32 store, into a channel slice of a wider tensor when
//                   the output feeds a concatenation.  The same kernel computes the input
//                   gradient (transposed, flipped weights), with the mask of the ReLU
//                   below it in the epilogue.
//  of_cnn_conv3x3_wgrad  weight gradient (CUDA cores, f32 FMA over bf16 operands).
//  pooling, nearest upsampling, ReLU masks, loss, Adam and weight packing: elementwise.
//
// Every wait on an mbarrier is bounded by time (about one second); a CTA that gives up
// sets a bit in the caller's error word, waits (bounded) for its copies in flight and
// for its MMAs, frees its TMEM and exits.
#include <cooperative_groups.h>
#include <cuda_bf16.h>

#include "common.cuh"
#include "tma.cuh"

namespace ofb {

namespace cg = cooperative_groups;
typedef __nv_bfloat16 bf16;

constexpr int CV_M = 128;
constexpr int CV_STAGES = 4;
constexpr int CV_THREADS = 192;
constexpr unsigned long long CV_WAIT_NS = 1000000000ull;

enum { CV_RELU = 1, CV_F32 = 2 };

struct ConvParams {
  int n, H, W, ck, nchunks;
  int bw, bh, nb, tiles_x, tiles_per_group;  // a tile: nb images x bh rows x bw columns = 128 pixels
  int bn, cout_store, flags;
  const float* bias;
  void* y;
  int y_ctot, y_coff;
  const bf16* act;  // ReLU backward in the epilogue: the output is 0 where this activation is not > 0
  int act_ctot, act_coff;
  unsigned* err;
  uint32_t a_bytes, b_bytes, stage_bytes, tmem_cols;
};

__device__ __forceinline__ unsigned long long globaltimer_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ bool mbar_try(uint64_t* bar, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(done)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return done != 0;
}

// Waits for phase `parity`, a whole warp at once with one result for all its lanes; gives up
// after CV_WAIT_NS or when *abort becomes nonzero.
__device__ bool cv_wait_warp(uint64_t* bar, uint32_t parity, volatile int* abort) {
  if (__all_sync(0xffffffffu, mbar_try(bar, parity))) return true;  // the clock is read only to wait
  unsigned long long t0 = globaltimer_ns();
  while (!__all_sync(0xffffffffu, mbar_try(bar, parity))) {
    const bool stop = (abort && *abort) || globaltimer_ns() - t0 > CV_WAIT_NS;
    if (__any_sync(0xffffffffu, stop)) return false;
  }
  return true;
}

// 1 in one lane of a converged warp.  The warps that issue copies and MMAs run their loops
// converged and let this lane issue: inside a one-lane branch the operands are not uniform for
// the compiler, and moving them to uniform registers costs more than a small MMA takes
// (128 x 16 x 16 from shared memory: 171 cycles with index divisions, 53 unrolled, 39 converged).
// In a training step of 16 crops of 128 x 128: the convolutions 564 -> 505 us, the weight
// gradients 407 -> 383 us; both are now bound by the boxes they load, nine per pixel.
__device__ __forceinline__ uint32_t elect_one() {
  uint32_t e;
  asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}\n" : "=r"(e));
  return e;
}

// Shared-memory matrix descriptor (sm_100 UMMA), K-major operand with a 32/64/128-byte
// swizzle: rows of `swz` bytes, 8-row core groups `8 * swz` bytes apart.
__device__ __forceinline__ uint64_t umma_desc_k(uint32_t saddr, int swz) {
  uint64_t layout = swz == 128 ? 2ull : (swz == 64 ? 4ull : 6ull);
  uint64_t sbo = (uint64_t)(8 * swz) >> 4;
  return (uint64_t)((saddr >> 4) & 0x3FFFu) | (1ull << 16) | (sbo << 32) | (1ull << 46) | (layout << 61);
}

// Instruction descriptor: kind::f16 with bf16 A and B (both K-major), f32 accumulator.
__host__ __device__ inline uint32_t umma_idesc_bf16(int m, int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

// Issued by the lane whose `elect` is 1; all other operands are the same in every lane.
__device__ __forceinline__ void umma_bf16(uint32_t elect, uint32_t tmem_d, uint64_t adesc, uint64_t bdesc,
                                          uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p, e;\n setp.ne.b32 p, %4, 0;\n setp.ne.b32 e, %5, 0;\n"
      " @e tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem_d),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(elect)
      : "memory");
}

__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// 16 accumulator columns of the warp's 32 TMEM lanes.  Called by all 32 lanes; they converge here,
// as both instructions demand.
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  __syncwarp();
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
      "%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ float2 bf2f(unsigned int u) {
  return make_float2(__uint_as_float(u << 16), __uint_as_float(u & 0xffff0000u));
}
__device__ __forceinline__ unsigned int f2bf(float a, float b) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const unsigned int*>(&h);
}
// Two bf16 gradients g where the two activations y are > 0, else +0.
__device__ __forceinline__ unsigned int relu_mask(unsigned int g, unsigned int y) {
  const float2 a = bf2f(y);
  return (a.x > 0.f ? g & 0xffffu : 0u) | (a.y > 0.f ? g & 0xffff0000u : 0u);
}
__device__ __forceinline__ uint4 relu_mask8(uint4 g, uint4 y) {
  return make_uint4(relu_mask(g.x, y.x), relu_mask(g.y, y.y), relu_mask(g.z, y.z), relu_mask(g.w, y.w));
}

// TMEM accumulator row (this thread's pixel) -> bias, ReLU, bf16 / f32 store of the N tile
// starting at channel n0.  With p.act the gradient is masked before its store, which replaces
// a pass that read it and the activation and wrote it again.  taddr: the warp's TMEM lane quarter, column 0.
__device__ __forceinline__ void cv_epilogue(const ConvParams& p, uint32_t taddr, size_t pix, int n0) {
  for (int c = 0; c < p.bn; c += 16) {
    uint32_t r[16];
    tmem_ld16(taddr + (uint32_t)c, r);
    const int co = n0 + c;
    if (co >= p.cout_store) continue;
    float v[16];
#pragma unroll
    for (int j = 0; j < 16; j++) {
      float a = __uint_as_float(r[j]);
      if (p.bias && co + j < p.cout_store) a = __fadd_rn(a, p.bias[co + j]);
      if (p.flags & CV_RELU) a = fmaxf(a, 0.f);
      v[j] = a;
    }
    const int nvalid = p.cout_store - co < 16 ? p.cout_store - co : 16;
    if (p.flags & CV_F32) {
      float* yo = static_cast<float*>(p.y) + pix * p.y_ctot + p.y_coff + co;
#pragma unroll
      for (int j = 0; j < 16; j++)
        if (j < nvalid) yo[j] = v[j];
    } else {
      bf16* yo = static_cast<bf16*>(p.y) + pix * p.y_ctot + p.y_coff + co;
      if (nvalid == 16) {
        uint32_t w[8];
#pragma unroll
        for (int j = 0; j < 8; j++) {
          __nv_bfloat162 h2 = __floats2bfloat162_rn(v[2 * j], v[2 * j + 1]);
          w[j] = *reinterpret_cast<uint32_t*>(&h2);
        }
        uint4 lo = make_uint4(w[0], w[1], w[2], w[3]), hi = make_uint4(w[4], w[5], w[6], w[7]);
        if (p.act) {
          const uint4* ao = reinterpret_cast<const uint4*>(p.act + pix * p.act_ctot + p.act_coff + co);
          lo = relu_mask8(lo, ao[0]);
          hi = relu_mask8(hi, ao[1]);
        }
        reinterpret_cast<uint4*>(yo)[0] = lo;
        reinterpret_cast<uint4*>(yo)[1] = hi;
      } else {
        const bf16* ao = p.act ? p.act + pix * p.act_ctot + p.act_coff + co : nullptr;
#pragma unroll
        for (int j = 0; j < 16; j++)
          if (j < nvalid) yo[j] = __float2bfloat16_rn(ao && !(__bfloat162float(ao[j]) > 0.f) ? 0.f : v[j]);
      }
    }
  }
}

// KSTEPS: MMAs of 16 channels per chunk of `ck`.
template <int KSTEPS>
__global__ void __launch_bounds__(CV_THREADS, 1)
    conv3x3_tc_kernel(const __grid_constant__ CUtensorMap tm_x, const __grid_constant__ CUtensorMap tm_w,
                      const ConvParams p) {
  extern __shared__ uint8_t cv_smem_raw[];
  __shared__ __align__(8) uint64_t full[CV_STAGES], empty[CV_STAGES], accf;
  __shared__ uint32_t tmem_slot;
  __shared__ volatile int abort_flag;
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(cv_smem_raw) + 1023) & ~(uintptr_t)1023);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int grp = blockIdx.x / p.tiles_per_group, t_in = blockIdx.x - grp * p.tiles_per_group;
  const int tyi = t_in / p.tiles_x, txi = t_in - tyi * p.tiles_x, img0 = grp * p.nb;
  const int x0 = txi * p.bw, y0 = tyi * p.bh, n0 = blockIdx.y * p.bn;
  const int kiters = 9 * p.nchunks;

  if (threadIdx.x == 0) {
    for (int s = 0; s < CV_STAGES; s++) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(&accf, 1);
    // once any CTA has given up, the rest skip their work instead of timing out in turn
    abort_flag = *reinterpret_cast<volatile unsigned*>(p.err) != 0u;
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)),
                 "r"(p.tmem_cols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_slot, 0);

  if (warp == 0) {
    const uint32_t el = elect_one();
    int issued = 0, ch = 0, tap = 0;
    for (int it = 0; it < kiters && !__any_sync(0xffffffffu, abort_flag); it++) {
      const int s = it % CV_STAGES;
      if (!cv_wait_warp(&empty[s], ((uint32_t)(it / CV_STAGES) & 1u) ^ 1u, &abort_flag)) {
        if (el) atomicOr(p.err, 1u);
        abort_flag = 1;
        break;
      }
      uint8_t* a = smem + (size_t)s * p.stage_bytes;
      if (el) {
        mbar_expect_tx(&full[s], p.a_bytes + p.b_bytes);
        tma_load_4d(a, &tm_x, ch * p.ck, x0 + tap % 3 - 1, y0 + tap / 3 - 1, img0, &full[s]);
        tma_load_3d(a + p.a_bytes, &tm_w, ch * p.ck, n0, tap, &full[s]);
      }
      if (++ch == p.nchunks) {
        ch = 0;
        tap++;
      }
      issued = it + 1;
    }
    // the copies of the last stages must land before the CTA's shared memory is released
    for (int it = issued > CV_STAGES ? issued - CV_STAGES : 0; it < issued; it++) {
      const int s = it % CV_STAGES;
      if (!cv_wait_warp(&full[s], (uint32_t)(it / CV_STAGES) & 1u, nullptr) && el) atomicOr(p.err, 2u);
    }
  } else if (warp == 1) {
    const uint32_t el = elect_one();
    const uint32_t idesc = umma_idesc_bf16(CV_M, p.bn);
    const uint32_t a0 = smem_u32(smem);
    const uint64_t ad0 = umma_desc_k(a0, KSTEPS * 32), bd0 = umma_desc_k(a0 + p.a_bytes, KSTEPS * 32);
    for (int it = 0; it < kiters; it++) {
      const int s = it % CV_STAGES;
      if (!cv_wait_warp(&full[s], (uint32_t)(it / CV_STAGES) & 1u, &abort_flag)) {
        if (el) atomicOr(p.err, 4u);
        abort_flag = 1;
        break;
      }
      tc_fence_after();
      const uint64_t off = (uint64_t)(s * (p.stage_bytes >> 4));
#pragma unroll
      for (int kk = 0; kk < KSTEPS; kk++)  // +32 bytes of K per step (descriptor address unit: 16 B)
        umma_bf16(el, tmem, ad0 + off + 2ull * kk, bd0 + off + 2ull * kk, idesc, (it | kk) != 0);
      if (el) umma_commit(&empty[s]);
      __syncwarp();
    }
    if (el) umma_commit(&accf);  // arrives once every MMA issued above has completed
    __syncwarp();
  } else {
    const int q = warp & 3;  // a warp reads the TMEM lanes 32 * (warp % 4) ...
    const int m = q * 32 + lane;
    const int mi = m / (p.bh * p.bw), mr = m - mi * (p.bh * p.bw);
    const int img = img0 + mi, py = y0 + mr / p.bw, px = x0 + mr % p.bw;
    const bool ok = cv_wait_warp(&accf, 0u, nullptr);
    if (!ok) atomicOr(p.err, 8u);
    tc_fence_after();
    // one decision for the warp: cv_epilogue reads TMEM
    if (__all_sync(0xffffffffu, ok && !abort_flag))
      cv_epilogue(p, tmem + ((uint32_t)(q * 32) << 16), ((size_t)img * p.H + py) * p.W + px, n0);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(p.tmem_cols) : "memory");
  }
}

// ----------------------------------------------------------------------------- wgrad, tensor cores
// dW[tap] = sum over pixels of dY[p] (x) X[p + tap]: per tap a GEMM whose K is the pixel
// count.  NHWC keeps the channels contiguous, so both operands are MN-major: a TMA box of
// 64 channels x 64 pixels lands as 64 rows of 128 B (128-byte swizzle), which is the
// canonical MN-major layout (8-row groups 1024 B apart, 64-channel atoms 8 KB apart).
// A is the wider channel side (M = 128, channels past its end are ignored rows), B the
// narrower (N <= 256), shifted by the tap through its box coordinates (zero padding from TMA's
// out-of-bounds fill): by +tap where B is X, by -tap where B is dY.  A CTA takes `tg` taps (9, 3
// or 1) of its pixels with one TMEM accumulator each, so that A is loaded once for all of them:
// with one tap per CTA the kernel is bound by the boxes it loads, 9 x (2 + B's) per 64 pixels.
// CTAs split the pixel range; each adds its sums into dW with atomics, four input channels at
// a time where the lanes run over output channels (scalar ones touch a sector each there).
// The 12 layers of a training step of 16 crops of 128 x 128: 634 us with one tap per CTA and
// scalar atomics, 383 us here.
constexpr int WT_KP = 64;  // pixels per K chunk
constexpr int WT_STAGES = 4;

struct WgParams {
  int n, H, W, bw, bh, nb, tiles_x, tiles_per_group, nchunk;  // pixel chunk geometry
  int chunks_per_cta, mtiles, ntiles;
  int a_is_dy, a_ch, b_ch;   // channel counts of the A and B sides
  int nmma, batoms;          // MMA N and 64-channel atoms loaded for B
  int tg, cstride, stages;   // taps per CTA, TMEM columns from one tap's accumulator to the next
  int cin, cout;
  float* dw;
  unsigned* err;
  uint32_t a_bytes, b_bytes, stage_bytes, tmem_cols;
};

// Shared-memory descriptor of a MN-major operand with the 128-byte swizzle: 64-element atoms
// `lbo` bytes apart along M/N, 8-row K groups 1024 bytes apart.
__device__ __forceinline__ uint64_t umma_desc_mn128(uint32_t saddr, uint32_t lbo) {
  return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) | ((uint64_t)(1024 >> 4) << 32) |
         (1ull << 46) | (2ull << 61);
}

__host__ __device__ inline uint32_t umma_idesc_bf16_mn(int m, int n) {
  return umma_idesc_bf16(m, n) | (1u << 15) | (1u << 16);  // A and B MN-major
}

__global__ void __launch_bounds__(CV_THREADS, 1)
    wgrad_tc_kernel(const __grid_constant__ CUtensorMap tm_a, const __grid_constant__ CUtensorMap tm_b,
                    const WgParams p) {
  extern __shared__ uint8_t wg_smem_raw[];
  __shared__ __align__(8) uint64_t full[WT_STAGES], empty[WT_STAGES], accf;
  __shared__ uint32_t tmem_slot;
  __shared__ volatile int abort_flag;
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(wg_smem_raw) + 1023) & ~(uintptr_t)1023);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tap0 = blockIdx.z * p.tg, mt = blockIdx.y / p.ntiles, nt = blockIdx.y - mt * p.ntiles;
  const int m0 = mt * 128, n0 = nt * 256;
  const int c0 = blockIdx.x * p.chunks_per_cta;
  const int c1 = c0 + p.chunks_per_cta < p.nchunk ? c0 + p.chunks_per_cta : p.nchunk;
  const int kiters = c1 > c0 ? c1 - c0 : 0;
  const bool atom1 = m0 + 64 < p.a_ch;  // A's second 64 channels; absent, their rows are ignored

  if (threadIdx.x == 0) {
    for (int s = 0; s < WT_STAGES; s++) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(&accf, 1);
    abort_flag = *reinterpret_cast<volatile unsigned*>(p.err) != 0u;
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)),
                 "r"(p.tmem_cols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_slot, 0);

  if (warp == 0) {
    const uint32_t el = elect_one();
    int issued = 0, s = 0;
    uint32_t ph = 1;
    const uint32_t bytes = (atom1 ? 2u : 1u) * 8192u + p.tg * p.b_bytes;
    const int sgn = p.a_is_dy ? 1 : -1;
    for (int it = 0; it < kiters && !__any_sync(0xffffffffu, abort_flag); it++) {
      if (!cv_wait_warp(&empty[s], ph, &abort_flag)) {
        if (el) atomicOr(p.err, 1u);
        abort_flag = 1;
        break;
      }
      if (el) {
        const int ch = c0 + it, grp = ch / p.tiles_per_group, t_in = ch - grp * p.tiles_per_group;
        const int ty = t_in / p.tiles_x, tx = t_in - ty * p.tiles_x;
        const int x0 = tx * p.bw, y0 = ty * p.bh, img0 = grp * p.nb;
        uint8_t* a = smem + (size_t)s * p.stage_bytes;
        mbar_expect_tx(&full[s], bytes);
        tma_load_4d(a, &tm_a, m0, x0, y0, img0, &full[s]);
        if (atom1) tma_load_4d(a + 8192, &tm_a, m0 + 64, x0, y0, img0, &full[s]);
        uint8_t* b = a + p.a_bytes;
        for (int t = tap0; t < tap0 + p.tg; t++) {
          const int dy = sgn * (t / 3 - 1), dx = sgn * (t % 3 - 1);
          for (int j = 0; j < p.batoms; j++, b += 8192)
            tma_load_4d(b, &tm_b, n0 + 64 * j, x0 + dx, y0 + dy, img0, &full[s]);
        }
      }
      if (++s == p.stages) {
        s = 0;
        ph ^= 1u;
      }
      issued = it + 1;
    }
    for (int it = issued > p.stages ? issued - p.stages : 0; it < issued; it++)
      if (!cv_wait_warp(&full[it % p.stages], (uint32_t)(it / p.stages) & 1u, nullptr) && el) atomicOr(p.err, 2u);
  } else if (warp == 1) {
    const uint32_t el = elect_one();
    const uint32_t idesc = umma_idesc_bf16_mn(128, p.nmma);
    const uint32_t a0 = smem_u32(smem);
    const uint64_t ad0 = umma_desc_mn128(a0, 8192), bd0 = umma_desc_mn128(a0 + p.a_bytes, 8192);
    int s = 0;
    uint32_t ph = 0;
    for (int it = 0; it < kiters; it++) {
      if (!cv_wait_warp(&full[s], ph, &abort_flag)) {
        if (el) atomicOr(p.err, 4u);
        abort_flag = 1;
        break;
      }
      tc_fence_after();
      const uint64_t ad = ad0 + (uint64_t)(s * (p.stage_bytes >> 4));
      uint64_t bd = bd0 + (uint64_t)(s * (p.stage_bytes >> 4));
      uint32_t d = tmem;
      for (int t = 0; t < p.tg; t++) {
#pragma unroll
        for (int kk = 0; kk < WT_KP / 16; kk++)  // 16 pixels = two 8-row groups: +2048 B (128 descriptor units)
          umma_bf16(el, d, ad + 128ull * kk, bd + 128ull * kk, idesc, (it | kk) != 0);
        d += p.cstride;
        bd += p.b_bytes >> 4;
      }
      if (el) umma_commit(&empty[s]);
      __syncwarp();
      if (++s == p.stages) {
        s = 0;
        ph ^= 1u;
      }
    }
    if (el) umma_commit(&accf);
    __syncwarp();
  } else {
    const int q = warp & 3;
    const int m = q * 32 + lane;
    const bool ok = cv_wait_warp(&accf, 0u, nullptr);
    if (!ok) atomicOr(p.err, 8u);
    tc_fence_after();
    const int am = m0 + m;  // this thread's A-side channel
    // one decision for the warp, and no lane leaves a round early: the loads from TMEM are warp-wide
    if (__all_sync(0xffffffffu, ok && !abort_flag && kiters > 0)) {
      const bool vec = p.a_is_dy && (p.cin & 3) == 0 && (reinterpret_cast<uintptr_t>(p.dw) & 15) == 0;
      for (int t = 0; t < p.tg; t++)
        for (int c = 0; c < p.nmma; c += 16) {
          uint32_t r[16];
          tmem_ld16(tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(t * p.cstride + c), r);
          float* dw = p.dw + (size_t)(tap0 + t) * p.cout * p.cin;
          if (am < p.a_ch) {
            if (vec) {
#pragma unroll
              for (int j = 0; j < 16; j += 4)
                if (n0 + c + j < p.b_ch)
                  atomicAdd(reinterpret_cast<float4*>(dw + (size_t)am * p.cin + n0 + c + j),
                            make_float4(__uint_as_float(r[j]), __uint_as_float(r[j + 1]), __uint_as_float(r[j + 2]),
                                        __uint_as_float(r[j + 3])));
            } else {
#pragma unroll
              for (int j = 0; j < 16; j++) {
                const int bn = n0 + c + j;
                if (bn >= p.b_ch) break;
                const int co = p.a_is_dy ? am : bn, ci = p.a_is_dy ? bn : am;
                atomicAdd(&dw[(size_t)co * p.cin + ci], __uint_as_float(r[j]));
              }
            }
          }
        }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(p.tmem_cols) : "memory");
  }
}

// ----------------------------------------------------------------------------- wgrad
// dW[tap][co][ci] += sum over pixels p of dY[p][co] * X[p + tap][ci]  (zero outside the
// image).  A CTA owns a 32 (co) x 32 (ci) block of all 9 taps and walks 64-pixel row
// segments; each thread keeps 9 x 4 accumulators (one co, four ci).
constexpr int WG_SEG = 64;

__global__ void __launch_bounds__(256) conv3x3_wgrad_kernel(const bf16* __restrict__ X, int xct, int xco,
                                                            const bf16* __restrict__ dY, int dct, int dco, int n,
                                                            int H, int W, int cin, int cout, float* __restrict__ dW) {
  __shared__ __align__(16) float sx[3][WG_SEG + 2][32];
  __shared__ float sg[WG_SEG][33];
  const int t = threadIdx.x, col = t >> 3, cg = (t & 7) * 4;
  const int ci0 = blockIdx.y * 32, co0 = blockIdx.z * 32;
  const int segs = (W + WG_SEG - 1) / WG_SEG;
  const long long units = (long long)n * H * segs;
  float acc[9][4];
#pragma unroll
  for (int k = 0; k < 9; k++)
#pragma unroll
    for (int j = 0; j < 4; j++) acc[k][j] = 0.f;
  for (long long u = blockIdx.x; u < units; u += gridDim.x) {
    const int sgi = (int)(u % segs);
    const long long rowi = u / segs;
    const int y = (int)(rowi % H), img = (int)(rowi / H), xs = sgi * WG_SEG;
    __syncthreads();
    for (int e = t; e < 3 * (WG_SEG + 2) * 32; e += 256) {
      int c = e & 31, rest = e >> 5, xx = rest % (WG_SEG + 2), ky = rest / (WG_SEG + 2);
      int gy = y + ky - 1, gx = xs + xx - 1, ci = ci0 + c;
      float v = 0.f;
      if (gy >= 0 && gy < H && gx >= 0 && gx < W && ci < cin)
        v = __bfloat162float(X[(((size_t)img * H + gy) * W + gx) * xct + xco + ci]);
      sx[ky][xx][c] = v;
    }
    for (int e = t; e < WG_SEG * 32; e += 256) {
      int c = e & 31, xx = e >> 5, gx = xs + xx, co = co0 + c;
      float v = 0.f;
      if (gx < W && co < cout) v = __bfloat162float(dY[(((size_t)img * H + y) * W + gx) * dct + dco + co]);
      sg[xx][c] = v;
    }
    __syncthreads();
#pragma unroll 4
    for (int xx = 0; xx < WG_SEG; xx++) {
      const float g = sg[xx][col];
#pragma unroll
      for (int ky = 0; ky < 3; ky++)
#pragma unroll
        for (int kx = 0; kx < 3; kx++) {
          const float4 xv = *reinterpret_cast<const float4*>(&sx[ky][xx + kx][cg]);
          float* a = acc[ky * 3 + kx];
          a[0] = __fmaf_rn(g, xv.x, a[0]);
          a[1] = __fmaf_rn(g, xv.y, a[1]);
          a[2] = __fmaf_rn(g, xv.z, a[2]);
          a[3] = __fmaf_rn(g, xv.w, a[3]);
        }
    }
  }
  const int co = co0 + col;
  if (co >= cout) return;
#pragma unroll
  for (int k = 0; k < 9; k++)
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const int ci = ci0 + cg + j;
      if (ci < cin) atomicAdd(&dW[((size_t)k * cout + co) * cin + ci], acc[k][j]);
    }
}

// db[co] += sum over pixels of dY[p][co]
__global__ void bias_grad_kernel(const bf16* __restrict__ dY, int dct, int dco, long long P, int cout,
                                 float* __restrict__ db) {
  const int c = threadIdx.x;  // blockDim.x >= cout
  float s = 0.f;
  if (c < cout)
    for (long long p = blockIdx.x; p < P; p += gridDim.x) s = __fadd_rn(s, __bfloat162float(dY[p * dct + dco + c]));
  if (c < cout) atomicAdd(&db[c], s);
}

// The same sum, 8 channels (16 bytes) per thread: the scalar kernel is bound by the latency of
// one 2-byte load per pixel and thread (the 12 layers of a training step of 16 crops of
// 128 x 128: 146 us, 40 us here).  A CTA of 256 threads holds 256 / (channel groups) pixels at a time and four loads in flight per
// thread, adds the pixel rows in shared memory and issues one atomic per channel.
// A last group that is not full reads, and drops, channels of the same pixel.
constexpr int BG_THREADS = 256;
__global__ void __launch_bounds__(BG_THREADS) bias_grad_v8_kernel(const bf16* __restrict__ dY, int dct, int dco,
                                                                  long long P, int cout, float* __restrict__ db) {
  __shared__ float part[BG_THREADS][9];
  const int c8 = (cout + 7) / 8, rows = BG_THREADS / c8;
  const int row = threadIdx.x / c8, grp = threadIdx.x - row * c8;
  float s[8];
#pragma unroll
  for (int k = 0; k < 8; k++) s[k] = 0.f;
  if (row < rows) {
    const bf16* src = dY + dco + 8 * grp;
    const long long step = (long long)gridDim.x * rows;
    long long p = (long long)blockIdx.x * rows + row;
    auto add = [&](const uint4& q) {
      const unsigned int u[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
      for (int k = 0; k < 4; k++) {
        const float2 v = bf2f(u[k]);
        s[2 * k] = __fadd_rn(s[2 * k], v.x);
        s[2 * k + 1] = __fadd_rn(s[2 * k + 1], v.y);
      }
    };
    for (; p + 3 * step < P; p += 4 * step) {
      uint4 q[4];
#pragma unroll
      for (int j = 0; j < 4; j++) q[j] = *reinterpret_cast<const uint4*>(src + (p + j * step) * dct);
#pragma unroll
      for (int j = 0; j < 4; j++) add(q[j]);
    }
    for (; p < P; p += step) add(*reinterpret_cast<const uint4*>(src + p * dct));
  }
#pragma unroll
  for (int k = 0; k < 8; k++) part[threadIdx.x][k] = s[k];
  __syncthreads();
  for (int c = threadIdx.x; c < cout; c += BG_THREADS) {
    float t = 0.f;
    for (int r = 0; r < rows; r++) t = __fadd_rn(t, part[r * c8 + (c >> 3)][c & 7]);
    atomicAdd(&db[c], t);
  }
}

// ----------------------------------------------------------------------------- elementwise
// out[img][y][x][0..cpad) = (I0 / max I0, I1 / max I1, 0, ...)  in bf16; max over the frame
__global__ void frame_max_kernel(const float* __restrict__ I, int H, int W, int pitch, unsigned* __restrict__ mx) {
  float m = 0.f;
  for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < (long long)H * W;
       e += (long long)gridDim.x * blockDim.x) {
    int y = (int)(e / W), x = (int)(e - (long long)y * W);
    m = fmaxf(m, I[(size_t)y * pitch + x]);
  }
  for (int o = 16; o; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) atomicMax(mx, __float_as_uint(m));  // non-negative floats order as integers
}

// One pixel of the network input: (a, b, 0, ...) over cpad channels; 16-byte stores when
// cpad is a multiple of 8 and the pixel's channels start 16-byte aligned.
__device__ __forceinline__ void pack_store(bf16* o, int cpad, float a, float b) {
  if ((cpad & 7) == 0 && (reinterpret_cast<uintptr_t>(o) & 15) == 0) {
    const __nv_bfloat162 ab = __floats2bfloat162_rn(a, b);
    uint4 v = make_uint4(*reinterpret_cast<const unsigned int*>(&ab), 0u, 0u, 0u);
    reinterpret_cast<uint4*>(o)[0] = v;
    v.x = 0u;
    for (int c = 8; c < cpad; c += 8) reinterpret_cast<uint4*>(o + c)[0] = v;
    return;
  }
  o[0] = __float2bfloat16_rn(a);
  o[1] = __float2bfloat16_rn(b);
  for (int c = 2; c < cpad; c++) o[c] = __float2bfloat16_rn(0.f);
}

__global__ void pack_pair_kernel(const float* __restrict__ I0, const float* __restrict__ I1, int H, int W, int pitch,
                                 const unsigned* __restrict__ mx, bf16* __restrict__ out, int cpad) {
  long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= (long long)H * W) return;
  int y = (int)(e / W), x = (int)(e - (long long)y * W);
  float m0 = __uint_as_float(mx[0]), m1 = __uint_as_float(mx[1]);
  float a = m0 > 0.f ? __fdiv_rn(I0[(size_t)y * pitch + x], m0) : 0.f;
  float b = m1 > 0.f ? __fdiv_rn(I1[(size_t)y * pitch + x], m1) : 0.f;
  pack_store(out + (size_t)e * cpad, cpad, a, b);
}

// Both maxima and the packing in one cluster of 8 CTAs, for the small frames the network runs
// on (up to 64 K pixels): each CTA reduces an eighth of the pixels, the CTAs exchange their
// two maxima through distributed shared memory, and each packs its own eighth (which its L1
// still holds).  One CTA alone is bound by its own load latency: 28.5 us for a 128 x 128 pair,
// 8.3 us here; three launches (the path for larger frames) wait for each other.  The maxima are the same
// (max is exact and order-free, NaN-free through fmaxf as in frame_max_kernel) and the packing
// is pack_pair_kernel's per pixel.
constexpr int PKC_CTAS = 8, PKC_THREADS = 512, PKC_PIX = 65536;
__global__ void __cluster_dims__(PKC_CTAS, 1, 1) __launch_bounds__(PKC_THREADS)
    pack_pair_cluster_kernel(const float* __restrict__ I0, const float* __restrict__ I1, int H, int W, int pitch,
                             unsigned* __restrict__ mx, bf16* __restrict__ out, int cpad) {
  __shared__ float r0[PKC_THREADS / 32], r1[PKC_THREADS / 32];
  __shared__ float2 all[PKC_CTAS];
  cg::cluster_group cl = cg::this_cluster();
  const int rank = (int)cl.block_rank();
  const int n = H * W, per = (n + PKC_CTAS - 1) / PKC_CTAS;
  const int e0 = rank * per, e1 = e0 + per < n ? e0 + per : n;
  float m0 = 0.f, m1 = 0.f;
#pragma unroll 4
  for (int e = e0 + (int)threadIdx.x; e < e1; e += PKC_THREADS) {
    const int y = e / W, x = e - y * W;
    m0 = fmaxf(m0, I0[(size_t)y * pitch + x]);
    m1 = fmaxf(m1, I1[(size_t)y * pitch + x]);
  }
  for (int o = 16; o; o >>= 1) {
    m0 = fmaxf(m0, __shfl_xor_sync(0xffffffffu, m0, o));
    m1 = fmaxf(m1, __shfl_xor_sync(0xffffffffu, m1, o));
  }
  if ((threadIdx.x & 31) == 0) {
    r0[threadIdx.x >> 5] = m0;
    r1[threadIdx.x >> 5] = m1;
  }
  cl.sync();  // this CTA's partial maxima, and every CTA of the cluster runs
  if (threadIdx.x < PKC_CTAS) {
    m0 = r0[0];
    m1 = r1[0];
    for (int w = 1; w < PKC_THREADS / 32; w++) {
      m0 = fmaxf(m0, r0[w]);
      m1 = fmaxf(m1, r1[w]);
    }
    *cl.map_shared_rank(&all[rank], threadIdx.x) = make_float2(m0, m1);
  }
  cl.sync();  // no remote access after this one: a CTA may exit
  m0 = all[0].x;
  m1 = all[0].y;
#pragma unroll
  for (int r = 1; r < PKC_CTAS; r++) {
    m0 = fmaxf(m0, all[r].x);
    m1 = fmaxf(m1, all[r].y);
  }
  if (rank == 0 && threadIdx.x == 0) {
    mx[0] = __float_as_uint(m0);
    mx[1] = __float_as_uint(m1);
  }
#pragma unroll 4
  for (int e = e0 + (int)threadIdx.x; e < e1; e += PKC_THREADS) {
    const int y = e / W, x = e - y * W;
    const float a = m0 > 0.f ? __fdiv_rn(I0[(size_t)y * pitch + x], m0) : 0.f;
    const float b = m1 > 0.f ? __fdiv_rn(I1[(size_t)y * pitch + x], m1) : 0.f;
    pack_store(out + (size_t)e * cpad, cpad, a, b);
  }
}

__global__ void avgpool2_kernel(const bf16* __restrict__ x, int xct, int xco, int n, int H, int W, int C,
                                bf16* __restrict__ y, int yct, int yco) {
  const int h = H / 2, w = W / 2;
  long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= (long long)n * h * w * C) return;
  int c = (int)(e % C);
  long long q = e / C;
  int ox = (int)(q % w), oy = (int)((q / w) % h), img = (int)(q / ((long long)w * h));
  const bf16* b = x + (((size_t)img * H + 2 * oy) * W + 2 * ox) * xct + xco + c;
  float s = __fadd_rn(__fadd_rn(__bfloat162float(b[0]), __bfloat162float(b[xct])),
                      __fadd_rn(__bfloat162float(b[(size_t)W * xct]), __bfloat162float(b[(size_t)W * xct + xct])));
  y[(((size_t)img * h + oy) * w + ox) * yct + yco + c] = __float2bfloat16_rn(__fmul_rn(s, 0.25f));
}

// The same two kernels on 8 channels (16 bytes) per thread, one output row per blockIdx.y
// (image * rows + row) and 32-bit index arithmetic: used when the channel counts, channel
// offsets and row strides are multiples of 8 and the bases 16-byte aligned (every layer of
// the network).  Per channel the arithmetic is the scalar kernels'.
__global__ void avgpool2_v8_kernel(const bf16* __restrict__ x, int xct, int xco, int H, int W, int C,
                                   bf16* __restrict__ y, int yct, int yco) {
  const int h = H / 2, w = W / 2, c8 = C / 8;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= w * c8) return;
  const int ox = t / c8, c = 8 * (t - ox * c8);
  const int img = blockIdx.y / h, oy = blockIdx.y - img * h;
  const bf16* b = x + (((size_t)img * H + 2 * oy) * W + 2 * ox) * xct + xco + c;
  const uint4 p0 = *reinterpret_cast<const uint4*>(b), p1 = *reinterpret_cast<const uint4*>(b + xct);
  const uint4 p2 = *reinterpret_cast<const uint4*>(b + (size_t)W * xct);
  const uint4 p3 = *reinterpret_cast<const uint4*>(b + (size_t)W * xct + xct);
  const unsigned int a0[4] = {p0.x, p0.y, p0.z, p0.w}, a1[4] = {p1.x, p1.y, p1.z, p1.w};
  const unsigned int a2[4] = {p2.x, p2.y, p2.z, p2.w}, a3[4] = {p3.x, p3.y, p3.z, p3.w};
  unsigned int o[4];
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const float2 v0 = bf2f(a0[k]), v1 = bf2f(a1[k]), v2 = bf2f(a2[k]), v3 = bf2f(a3[k]);
    const float sx = __fadd_rn(__fadd_rn(v0.x, v1.x), __fadd_rn(v2.x, v3.x));
    const float sy = __fadd_rn(__fadd_rn(v0.y, v1.y), __fadd_rn(v2.y, v3.y));
    o[k] = f2bf(__fmul_rn(sx, 0.25f), __fmul_rn(sy, 0.25f));
  }
  *reinterpret_cast<uint4*>(y + (((size_t)img * h + oy) * w + ox) * yct + yco + c) = make_uint4(o[0], o[1], o[2], o[3]);
}

__global__ void upsample2_v8_kernel(const bf16* __restrict__ x, int xct, int xco, int h, int w, int C,
                                    bf16* __restrict__ y, int yct, int yco) {
  const int H = 2 * h, W = 2 * w, c8 = C / 8;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= W * c8) return;
  const int xx = t / c8, c = 8 * (t - xx * c8);
  const int img = blockIdx.y / H, yy = blockIdx.y - img * H;
  *reinterpret_cast<uint4*>(y + (((size_t)img * H + yy) * W + xx) * yct + yco + c) =
      *reinterpret_cast<const uint4*>(x + (((size_t)img * h + yy / 2) * w + xx / 2) * xct + xco + c);
}

static bool v8_ok(const void* x, int xct, int xco, const void* y, int yct, int yco, int C) {
  return C % 8 == 0 && xct % 8 == 0 && xco % 8 == 0 && yct % 8 == 0 && yco % 8 == 0 &&
         ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(y)) & 15) == 0;
}

// dx (fine) = dy (coarse parent) / 4, added to dx when accumulate
__global__ void avgpool2_bwd_kernel(const bf16* __restrict__ dy, int dct, int dco, int n, int H, int W, int C,
                                    bf16* __restrict__ dx, int xct, int xco, int accumulate,
                                    const bf16* __restrict__ act, int act_ct, int act_co) {
  long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= (long long)n * H * W * C) return;
  int c = (int)(e % C);
  long long q = e / C;
  int xx = (int)(q % W), yy = (int)((q / W) % H), img = (int)(q / ((long long)W * H));
  const int h = H / 2, w = W / 2;
  float g = __fmul_rn(__bfloat162float(dy[(((size_t)img * h + yy / 2) * w + xx / 2) * dct + dco + c]), 0.25f);
  bf16* o = dx + (((size_t)img * H + yy) * W + xx) * xct + xco + c;
  if (accumulate) g = __fadd_rn(g, __bfloat162float(*o));
  if (act && !(__bfloat162float(act[(((size_t)img * H + yy) * W + xx) * act_ct + act_co + c]) > 0.f)) g = 0.f;
  *o = __float2bfloat16_rn(g);
}

// nearest 2x upsampling of x (n, h, w, C) into a channel slice of y (n, 2h, 2w, yct)
__global__ void upsample2_kernel(const bf16* __restrict__ x, int xct, int xco, int n, int h, int w, int C,
                                 bf16* __restrict__ y, int yct, int yco) {
  const int H = 2 * h, W = 2 * w;
  long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= (long long)n * H * W * C) return;
  int c = (int)(e % C);
  long long q = e / C;
  int xx = (int)(q % W), yy = (int)((q / W) % H), img = (int)(q / ((long long)W * H));
  y[(((size_t)img * H + yy) * W + xx) * yct + yco + c] = x[(((size_t)img * h + yy / 2) * w + xx / 2) * xct + xco + c];
}

__global__ void upsample2_bwd_kernel(const bf16* __restrict__ dy, int dct, int dco, int n, int h, int w, int C,
                                     bf16* __restrict__ dx, int xct, int xco, const bf16* __restrict__ act, int act_ct,
                                     int act_co) {
  long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= (long long)n * h * w * C) return;
  int c = (int)(e % C);
  long long q = e / C;
  int ox = (int)(q % w), oy = (int)((q / w) % h), img = (int)(q / ((long long)w * h));
  const int W = 2 * w, H = 2 * h;
  const bf16* b = dy + (((size_t)img * H + 2 * oy) * W + 2 * ox) * dct + dco + c;
  float s = __fadd_rn(__fadd_rn(__bfloat162float(b[0]), __bfloat162float(b[dct])),
                      __fadd_rn(__bfloat162float(b[(size_t)W * dct]), __bfloat162float(b[(size_t)W * dct + dct])));
  if (act && !(__bfloat162float(act[(((size_t)img * h + oy) * w + ox) * act_ct + act_co + c]) > 0.f)) s = 0.f;
  dx[(((size_t)img * h + oy) * w + ox) * xct + xco + c] = __float2bfloat16_rn(s);
}

// The backward passes on 8 channels per thread, under the rule of the forward ones and with
// the same arithmetic per channel.  They should be bound by memory; one element per thread was
// bound by its 64-bit index arithmetic.  The mask of the ReLU whose output was pooled or
// upsampled goes in before the store.  The three poolings of a training step of 16 crops of
// 128 x 128: 111 us and their masks before, 26 us with the masks now; the three upsamplings
// 60 us and masks before, 17 us now; all eleven masks were 167 us.
__global__ void avgpool2_bwd_v8_kernel(const bf16* __restrict__ dy, int dct, int dco, int H, int W, int C,
                                       bf16* __restrict__ dx, int xct, int xco, int accumulate,
                                       const bf16* __restrict__ act, int act_ct, int act_co) {
  // one thread: 2 x 2 outputs of one input
  const int h = H / 2, w = W / 2, c8 = C / 8;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= w * c8) return;
  const int ox = t / c8, c = 8 * (t - ox * c8);
  const int img = blockIdx.y / h, oy = blockIdx.y - img * h;
  const size_t pix = ((size_t)img * H + 2 * oy) * W + 2 * ox;
  const uint4 q = *reinterpret_cast<const uint4*>(dy + (((size_t)img * h + oy) * w + ox) * dct + dco + c);
  const unsigned int u[4] = {q.x, q.y, q.z, q.w};
  float2 g[4];
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const float2 v = bf2f(u[k]);
    g[k] = make_float2(__fmul_rn(v.x, 0.25f), __fmul_rn(v.y, 0.25f));
  }
  uint4 old[4], a[4];
#pragma unroll
  for (int j = 0; j < 4; j++) {
    const size_t o = pix + (size_t)(j >> 1) * W + (j & 1);
    if (accumulate) old[j] = *reinterpret_cast<const uint4*>(dx + o * xct + xco + c);
    if (act) a[j] = *reinterpret_cast<const uint4*>(act + o * act_ct + act_co + c);
  }
#pragma unroll
  for (int j = 0; j < 4; j++) {
    const size_t o = pix + (size_t)(j >> 1) * W + (j & 1);
    unsigned int r[4];
    const unsigned int d[4] = {old[j].x, old[j].y, old[j].z, old[j].w};
#pragma unroll
    for (int k = 0; k < 4; k++) {
      float2 v = g[k];
      if (accumulate) {
        const float2 e = bf2f(d[k]);
        v = make_float2(__fadd_rn(v.x, e.x), __fadd_rn(v.y, e.y));
      }
      r[k] = f2bf(v.x, v.y);
    }
    uint4 out = make_uint4(r[0], r[1], r[2], r[3]);
    if (act) out = relu_mask8(out, a[j]);
    *reinterpret_cast<uint4*>(dx + o * xct + xco + c) = out;
  }
}

__global__ void upsample2_bwd_v8_kernel(const bf16* __restrict__ dy, int dct, int dco, int h, int w, int C,
                                        bf16* __restrict__ dx, int xct, int xco, const bf16* __restrict__ act,
                                        int act_ct, int act_co) {
  const int H = 2 * h, W = 2 * w, c8 = C / 8;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= w * c8) return;
  const int ox = t / c8, c = 8 * (t - ox * c8);
  const int img = blockIdx.y / h, oy = blockIdx.y - img * h;
  const bf16* b = dy + (((size_t)img * H + 2 * oy) * W + 2 * ox) * dct + dco + c;
  const size_t o = ((size_t)img * h + oy) * w + ox;
  const uint4 p0 = *reinterpret_cast<const uint4*>(b), p1 = *reinterpret_cast<const uint4*>(b + dct);
  const uint4 p2 = *reinterpret_cast<const uint4*>(b + (size_t)W * dct);
  const uint4 p3 = *reinterpret_cast<const uint4*>(b + (size_t)W * dct + dct);
  uint4 a = make_uint4(0u, 0u, 0u, 0u);
  if (act) a = *reinterpret_cast<const uint4*>(act + o * act_ct + act_co + c);
  const unsigned int a0[4] = {p0.x, p0.y, p0.z, p0.w}, a1[4] = {p1.x, p1.y, p1.z, p1.w};
  const unsigned int a2[4] = {p2.x, p2.y, p2.z, p2.w}, a3[4] = {p3.x, p3.y, p3.z, p3.w};
  unsigned int r[4];
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const float2 v0 = bf2f(a0[k]), v1 = bf2f(a1[k]), v2 = bf2f(a2[k]), v3 = bf2f(a3[k]);
    r[k] = f2bf(__fadd_rn(__fadd_rn(v0.x, v1.x), __fadd_rn(v2.x, v3.x)),
                __fadd_rn(__fadd_rn(v0.y, v1.y), __fadd_rn(v2.y, v3.y)));
  }
  uint4 out = make_uint4(r[0], r[1], r[2], r[3]);
  if (act) out = relu_mask8(out, a);
  *reinterpret_cast<uint4*>(dx + o * xct + xco + c) = out;
}

// g = g * (y > 0) over a channel slice (the ReLU derivative from the layer's output)
__global__ void relu_bwd_kernel(bf16* __restrict__ g, int gct, int gco, const bf16* __restrict__ y, int yct, int yco,
                                long long P, int C) {
  long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= P * C) return;
  long long p = e / C;
  int c = (int)(e - p * C);
  if (!(__bfloat162float(y[p * yct + yco + c]) > 0.f)) g[p * gct + gco + c] = __float2bfloat16_rn(0.f);
}

// The same, 8 channels per thread.
__global__ void relu_bwd_v8_kernel(bf16* __restrict__ g, int gct, int gco, const bf16* __restrict__ y, int yct, int yco,
                                   long long P, int C) {
  const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int c8 = C / 8;
  const long long p = e / c8;
  if (p >= P) return;
  const int c = 8 * (int)(e - p * c8);
  uint4* o = reinterpret_cast<uint4*>(g + p * gct + gco + c);
  *o = relu_mask8(*o, *reinterpret_cast<const uint4*>(y + p * yct + yco + c));
}

// mean squared flow error: loss += sum (pred - label)^2 / (2 P);  dpred = (pred - label) / P
// (bf16, padded to gct channels, the padding zeroed).  One pixel per thread; the CTA adds its warps'
// sums in double and issues one atomic (one per warp serialised on the loss's address: 16 x 128 x 128
// pixels 25.4 us, 4.8 us here).
__global__ void __launch_bounds__(256) flow_mse_kernel(const float* __restrict__ pred, const float* __restrict__ label,
                                                       long long P, bf16* __restrict__ dpred, int gct,
                                                       double* __restrict__ loss) {
  long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  float l = 0.f;
  if (p < P) {
    const float inv = __frcp_rn((float)P);
    float du = __fadd_rn(pred[2 * p], -label[2 * p]), dv = __fadd_rn(pred[2 * p + 1], -label[2 * p + 1]);
    l = __fadd_rn(__fmul_rn(du, du), __fmul_rn(dv, dv));
    if (dpred) {
      pack_store(dpred + p * gct, gct, __fmul_rn(du, inv), __fmul_rn(dv, inv));
    }
  }
  for (int o = 16; o; o >>= 1) l = __fadd_rn(l, __shfl_xor_sync(0xffffffffu, l, o));
  __shared__ double part[8];
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = (double)l / (2.0 * (double)P);
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = part[0];
    for (int w = 1; w < 8; w++) t += part[w];
    atomicAdd(loss, t);
  }
}

__global__ void adam_kernel(float* __restrict__ w, const float* __restrict__ g, float* __restrict__ m,
                            float* __restrict__ v, long long n, float lr, float b1, float b2, float eps, float bc1,
                            float bc2) {
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float gi = g[i];
  float mi = __fadd_rn(__fmul_rn(b1, m[i]), __fmul_rn(__fadd_rn(1.f, -b1), gi));
  float vi = __fadd_rn(__fmul_rn(b2, v[i]), __fmul_rn(__fadd_rn(1.f, -b2), __fmul_rn(gi, gi)));
  m[i] = mi;
  v[i] = vi;
  float mh = __fdiv_rn(mi, bc1), vh = __fdiv_rn(vi, bc2);
  w[i] = __fadd_rn(w[i], -__fdiv_rn(__fmul_rn(lr, mh), __fadd_rn(__fsqrt_rn(vh), eps)));
}

// master weights w[tap][co][ci] (f32, the wgrad layout) -> bf16 B operands:
//   forward:  out[tap][co][ci]                     (cout_pad x cin_pad rows per tap)
//   backward: out[tap'][ci][co] = w[co][ci][8-tap'] (cin_pad x cout_pad rows per tap)
__global__ void pack_weights_kernel(const float* __restrict__ w, int cout, int cin, int cout_pad, int cin_pad,
                                    int transpose_flip, bf16* __restrict__ out) {
  long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  long long total = 9LL * cout_pad * cin_pad;
  if (e >= total) return;
  int tap = (int)(e / ((long long)cout_pad * cin_pad));
  int r = (int)(e - (long long)tap * cout_pad * cin_pad);
  int cols = transpose_flip ? cout_pad : cin_pad;
  int row = r / cols, colm = r - row * cols;
  int co = transpose_flip ? colm : row, ci = transpose_flip ? row : colm;
  int k = transpose_flip ? 8 - tap : tap;
  float v = (co < cout && ci < cin) ? w[((size_t)k * cout + co) * cin + ci] : 0.f;
  out[e] = __float2bfloat16_rn(v);
}

// Every layer's operands in one launch: 23 launches of 2.5 us each (57 us, and more than that
// on the host) against 14.6 us.  blockIdx.y picks the entry, the CTAs of a row walk it.
constexpr int PW_MAX = 64;
struct PackMany {
  const float* w[PW_MAX];
  bf16* out[PW_MAX];
  short cout[PW_MAX], cin[PW_MAX], cout_pad[PW_MAX], cin_pad[PW_MAX], flip[PW_MAX];
};
__global__ void pack_weights_many_kernel(const __grid_constant__ PackMany p) {
  const int i = blockIdx.y;
  const int cp = p.cout_pad[i], ip = p.cin_pad[i], cout = p.cout[i], cin = p.cin[i], flip = p.flip[i];
  const int per = cp * ip, cols = flip ? cp : ip;
  const float* w = p.w[i];
  bf16* out = p.out[i];
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < 9 * per; e += gridDim.x * blockDim.x) {
    const int tap = e / per, r = e - tap * per, row = r / cols, col = r - row * cols;
    const int co = flip ? col : row, ci = flip ? row : col, k = flip ? 8 - tap : tap;
    out[e] = __float2bfloat16_rn(co < cout && ci < cin ? w[((size_t)k * cout + co) * cin + ci] : 0.f);
  }
}

// (h, w, 2) interleaved f32 flow -> two planes with row pitch `pitch`
__global__ void split_flow_kernel(const float* __restrict__ f, int h, int w, float* __restrict__ u,
                                  float* __restrict__ v, int pitch) {
  long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= (long long)h * w) return;
  int y = (int)(e / w), x = (int)(e - (long long)y * w);
  u[(size_t)y * pitch + x] = f[2 * e];
  v[(size_t)y * pitch + x] = f[2 * e + 1];
}

// (h, w, 2) interleaved f32 flow -> U, V planes at (f h, f w), bilinear with pixel-centre
// alignment (fine pixel X samples coarse position (X + 0.5) / f - 0.5, clamped) and the
// displacement scaled by `scale`.
__global__ void flow_up_kernel(const float* __restrict__ fl, int h, int w, int f, float* __restrict__ U,
                               float* __restrict__ V, int pitch, float scale) {
  const int X = blockIdx.x * blockDim.x + threadIdx.x, Y = blockIdx.y;
  if (X >= f * w) return;
  const float inv = __frcp_rn((float)f);
  const float sx = fmaxf(__fsub_rn(__fmul_rn(__fadd_rn((float)X, 0.5f), inv), 0.5f), 0.f);
  const float sy = fmaxf(__fsub_rn(__fmul_rn(__fadd_rn((float)Y, 0.5f), inv), 0.5f), 0.f);
  int x0 = (int)sx, y0 = (int)sy;
  x0 = x0 < w - 1 ? x0 : w - 1;
  y0 = y0 < h - 1 ? y0 : h - 1;
  const int x1 = x0 + 1 < w ? x0 + 1 : w - 1, y1 = y0 + 1 < h ? y0 + 1 : h - 1;
  const float ax = __fsub_rn(sx, (float)x0), ay = __fsub_rn(sy, (float)y0);
#pragma unroll
  for (int c = 0; c < 2; c++) {
    const float a = fl[((size_t)y0 * w + x0) * 2 + c], b = fl[((size_t)y0 * w + x1) * 2 + c];
    const float d = fl[((size_t)y1 * w + x0) * 2 + c], e = fl[((size_t)y1 * w + x1) * 2 + c];
    const float top = __fmaf_rn(ax, __fsub_rn(b, a), a), bot = __fmaf_rn(ax, __fsub_rn(e, d), d);
    const float v = __fmul_rn(__fmaf_rn(ay, __fsub_rn(bot, top), top), scale);
    (c == 0 ? U : V)[(size_t)Y * pitch + X] = v;
  }
}

static int blocks_for(long long n, int t = 256) { return (int)((n + t - 1) / t); }

}  // namespace ofb

using namespace ofb;

static int conv3x3(const void* x, int n, int H, int W, int cin, int x_ctot, int x_coff, const void* w, int cout,
                   const float* bias, int flags, void* y, int y_ctot, int y_coff, int cout_store, const void* act,
                   int act_ctot, int act_coff, unsigned* err, void* stream) {
  OF_REQUIRE(x && w && y && err && n > 0 && H > 0 && W > 0, "of_cnn_conv3x3: bad arguments");
  int ck = cin % 64 == 0 ? 64 : (cin % 32 == 0 ? 32 : (cin == 16 ? 16 : 0));
  OF_REQUIRE(ck, "of_cnn_conv3x3: input channels %d (need 16, a multiple of 32)", cin);
  OF_REQUIRE(cout % 16 == 0 && cout <= 512 && cout > 0, "of_cnn_conv3x3: output channels %d (need 16..512, /16)", cout);
  int ntile = (cout + 255) / 256, bn = cout / ntile;
  OF_REQUIRE(bn * ntile == cout && bn % 16 == 0, "of_cnn_conv3x3: output channels %d do not split into N tiles", cout);
  int bw = W < CV_M ? W : CV_M;
  OF_REQUIRE(CV_M % bw == 0 && W % bw == 0, "of_cnn_conv3x3: width %d (need a divisor of 128 or a multiple)", W);
  int bh = CV_M / bw < H ? CV_M / bw : H;
  OF_REQUIRE(H % bh == 0 && (CV_M / bw) % bh == 0, "of_cnn_conv3x3: height %d does not tile by %d", H, bh);
  int nb = CV_M / (bw * bh);  // small images: one tile spans nb whole images
  OF_REQUIRE(n % nb == 0, "of_cnn_conv3x3: %d images of %d x %d do not fill 128-pixel tiles", n, H, W);
  OF_REQUIRE(x_ctot % 8 == 0 && x_coff % 8 == 0 && x_coff + cin <= x_ctot, "of_cnn_conv3x3: input channel slice");
  // bf16 stores go out 16 bytes at a time; f32 stores are scalar
  const bool f32 = (flags & CV_F32) != 0;
  OF_REQUIRE((f32 || (y_ctot % 8 == 0 && y_coff % 8 == 0)) && cout_store <= cout && cout_store > 0 &&
                 y_coff + cout_store <= y_ctot,
             "of_cnn_conv3x3: output channel slice");
  OF_REQUIRE(f32 || ((uintptr_t)y & 15) == 0, "of_cnn_conv3x3: output not 16-byte aligned");
  CUtensorMap tmx, tmw;
  {
    uint64_t dims[4] = {(uint64_t)cin, (uint64_t)W, (uint64_t)H, (uint64_t)n};
    uint64_t st[3] = {(uint64_t)x_ctot * 2, (uint64_t)W * x_ctot * 2, (uint64_t)H * W * x_ctot * 2};
    uint32_t box[4] = {(uint32_t)ck, (uint32_t)bw, (uint32_t)bh, (uint32_t)nb};
    int rc = tmap_bf16(&tmx, static_cast<const bf16*>(x) + x_coff, 4, dims, st, box, ck * 2);
    if (rc) return rc;
  }
  {
    uint64_t dims[3] = {(uint64_t)cin, (uint64_t)cout, 9};
    uint64_t st[2] = {(uint64_t)cin * 2, (uint64_t)cout * cin * 2};
    uint32_t box[3] = {(uint32_t)ck, (uint32_t)bn, 1};
    int rc = tmap_bf16(&tmw, w, 3, dims, st, box, ck * 2);
    if (rc) return rc;
  }
  ConvParams p;
  p.n = n;
  p.H = H;
  p.W = W;
  p.ck = ck;
  p.nchunks = cin / ck;
  p.bw = bw;
  p.bh = bh;
  p.nb = nb;
  p.tiles_x = W / bw;
  p.tiles_per_group = (W / bw) * (H / bh);
  p.bn = bn;
  p.cout_store = cout_store;
  p.flags = flags;
  p.bias = bias;
  p.y = y;
  p.y_ctot = y_ctot;
  p.y_coff = y_coff;
  p.act = static_cast<const bf16*>(act);
  p.act_ctot = act_ctot;
  p.act_coff = act_coff;
  p.err = err;
  p.a_bytes = (uint32_t)(CV_M * ck * 2);
  p.b_bytes = (uint32_t)(bn * ck * 2);
  p.stage_bytes = (uint32_t)align_up(p.a_bytes + p.b_bytes, 1024);
  p.tmem_cols = bn <= 32 ? 32 : (bn <= 64 ? 64 : (bn <= 128 ? 128 : 256));
  // shared memory in proportion to the TMEM columns held, so the CTAs resident on an SM
  // never ask for more than its 512 columns
  size_t smem = 1024 + (size_t)CV_STAGES * p.stage_bytes;
  size_t floor_smem = (size_t)p.tmem_cols * 456 + 1024;
  if (smem < floor_smem) smem = floor_smem;
  cudaError_t e = ck == 64   ? OF_SMEM_OPT_IN(conv3x3_tc_kernel<4>, smem)
                  : ck == 32 ? OF_SMEM_OPT_IN(conv3x3_tc_kernel<2>, smem)
                             : OF_SMEM_OPT_IN(conv3x3_tc_kernel<1>, smem);
  if (e != cudaSuccess)
    return set_error(OF_ERR_CUDA, "of_cnn_conv3x3: %zu B of shared memory: %s", smem, cudaGetErrorString(e));
  dim3 grid((n / nb) * p.tiles_per_group, ntile);
  (ck == 64   ? conv3x3_tc_kernel<4>
   : ck == 32 ? conv3x3_tc_kernel<2>
              : conv3x3_tc_kernel<1>)<<<grid, CV_THREADS, smem, as_stream(stream)>>>(tmx, tmw, p);
  return check_launch("of_cnn_conv3x3");
}

extern "C" int of_cnn_conv3x3(const void* x, int n, int H, int W, int cin, int x_ctot, int x_coff, const void* w,
                              int cout, const float* bias, int flags, void* y, int y_ctot, int y_coff, int cout_store,
                              unsigned* err, void* stream) {
  return conv3x3(x, n, H, W, cin, x_ctot, x_coff, w, cout, bias, flags, y, y_ctot, y_coff, cout_store, nullptr, 0, 0, err,
                 stream);
}

extern "C" int of_cnn_conv3x3_relu_bwd(const void* dy, int n, int H, int W, int cin, int dy_ctot, int dy_coff,
                                       const void* w, int cout, const void* act, int act_ctot, int act_coff, void* dx,
                                       int dx_ctot, int dx_coff, int cout_store, unsigned* err, void* stream) {
  OF_REQUIRE(act && act_ctot % 8 == 0 && act_coff % 8 == 0 && act_coff >= 0 && cout_store > 0 &&
                 act_coff + cout_store <= act_ctot && ((uintptr_t)act & 15) == 0,
             "of_cnn_conv3x3_relu_bwd: activation channel slice");
  return conv3x3(dy, n, H, W, cin, dy_ctot, dy_coff, w, cout, nullptr, 0, dx, dx_ctot, dx_coff, cout_store, act, act_ctot,
                 act_coff, err, stream);
}

extern "C" int of_cnn_conv3x3_wgrad(const void* x, int x_ctot, int x_coff, const void* dy, int dy_ctot, int dy_coff,
                                    int n, int H, int W, int cin, int cout, float* dw, void* stream) {
  OF_REQUIRE(x && dy && dw && n > 0 && H > 0 && W > 0 && cin > 0 && cout > 0, "of_cnn_conv3x3_wgrad: bad arguments");
  long long units = (long long)n * H * ((W + WG_SEG - 1) / WG_SEG);
  int gx = (int)(units < 4LL * kNumSMs ? units : 4LL * kNumSMs);
  dim3 grid(gx, (cin + 31) / 32, (cout + 31) / 32);
  conv3x3_wgrad_kernel<<<grid, 256, 0, as_stream(stream)>>>(static_cast<const bf16*>(x), x_ctot, x_coff,
                                                             static_cast<const bf16*>(dy), dy_ctot, dy_coff, n, H, W,
                                                             cin, cout, dw);
  return check_launch("of_cnn_conv3x3_wgrad");
}

extern "C" int of_cnn_bias_grad(const void* dy, int dy_ctot, int dy_coff, long long P, int cout, float* db,
                                void* stream) {
  OF_REQUIRE(dy && db && P > 0 && cout > 0 && cout <= 1024, "of_cnn_bias_grad: bad arguments");
  if (dy_ctot % 8 == 0 && dy_coff % 8 == 0 && dy_coff + (cout + 7) / 8 * 8 <= dy_ctot && ((uintptr_t)dy & 15) == 0) {
    const int rows = BG_THREADS / ((cout + 7) / 8);
    // two CTAs per SM, fewer where a CTA would see less than 4 rounds of pixels
    long long g = (P + 4LL * rows - 1) / (4LL * rows);
    if (g > 2 * kNumSMs) g = 2 * kNumSMs;
    bias_grad_v8_kernel<<<(int)g, BG_THREADS, 0, as_stream(stream)>>>(static_cast<const bf16*>(dy), dy_ctot, dy_coff, P,
                                                                      cout, db);
    return check_launch("of_cnn_bias_grad");
  }
  int t = (cout + 31) / 32 * 32;
  int g = (int)(P < 2LL * kNumSMs * 8 ? P : 2LL * kNumSMs * 8);
  bias_grad_kernel<<<g, t, 0, as_stream(stream)>>>(static_cast<const bf16*>(dy), dy_ctot, dy_coff, P, cout, db);
  return check_launch("of_cnn_bias_grad");
}

extern "C" int of_cnn_pack_pair(const float* I0, const float* I1, int H, int W, int pitch, unsigned* max2, void* out,
                                int cpad, void* stream) {
  OF_REQUIRE(I0 && I1 && max2 && out && H > 0 && W > 0 && pitch >= W && cpad >= 2, "of_cnn_pack_pair: bad arguments");
  cudaStream_t st = as_stream(stream);
  if ((long long)H * W <= PKC_PIX) {
    pack_pair_cluster_kernel<<<PKC_CTAS, PKC_THREADS, 0, st>>>(I0, I1, H, W, pitch, max2, static_cast<bf16*>(out), cpad);
    return check_launch("of_cnn_pack_pair");
  }
  cudaMemsetAsync(max2, 0, 2 * sizeof(unsigned), st);
  int g = blocks_for((long long)H * W);
  int gm = g < 4 * kNumSMs ? g : 4 * kNumSMs;
  frame_max_kernel<<<gm, 256, 0, st>>>(I0, H, W, pitch, max2);
  frame_max_kernel<<<gm, 256, 0, st>>>(I1, H, W, pitch, max2 + 1);
  pack_pair_kernel<<<g, 256, 0, st>>>(I0, I1, H, W, pitch, max2, static_cast<bf16*>(out), cpad);
  return check_launch("of_cnn_pack_pair", 3);
}

extern "C" int of_cnn_avgpool2(const void* x, int x_ctot, int x_coff, int n, int H, int W, int C, void* y, int y_ctot,
                               int y_coff, void* stream) {
  OF_REQUIRE(x && y && H % 2 == 0 && W % 2 == 0 && C > 0, "of_cnn_avgpool2: bad arguments");
  if (v8_ok(x, x_ctot, x_coff, y, y_ctot, y_coff, C) && (long long)n * (H / 2) <= 65535) {
    avgpool2_v8_kernel<<<dim3(blocks_for((long long)(W / 2) * (C / 8)), n * (H / 2)), 256, 0, as_stream(stream)>>>(
        static_cast<const bf16*>(x), x_ctot, x_coff, H, W, C, static_cast<bf16*>(y), y_ctot, y_coff);
    return check_launch("of_cnn_avgpool2");
  }
  long long tot = (long long)n * (H / 2) * (W / 2) * C;
  avgpool2_kernel<<<blocks_for(tot), 256, 0, as_stream(stream)>>>(static_cast<const bf16*>(x), x_ctot, x_coff, n, H,
                                                                   W, C, static_cast<bf16*>(y), y_ctot, y_coff);
  return check_launch("of_cnn_avgpool2");
}

static int avgpool2_bwd(const void* dy, int dy_ctot, int dy_coff, int n, int H, int W, int C, void* dx, int dx_ctot,
                        int dx_coff, int accumulate, const void* act, int act_ctot, int act_coff, void* stream) {
  OF_REQUIRE(dy && dx && H % 2 == 0 && W % 2 == 0 && C > 0, "of_cnn_avgpool2_bwd: bad arguments");
  const bf16 *d = static_cast<const bf16*>(dy), *a = static_cast<const bf16*>(act);
  if (v8_ok(dy, dy_ctot, dy_coff, dx, dx_ctot, dx_coff, C) && (!act || v8_ok(act, act_ctot, act_coff, dx, 0, 0, C)) &&
      (long long)n * (H / 2) <= 65535) {
    avgpool2_bwd_v8_kernel<<<dim3(blocks_for((long long)(W / 2) * (C / 8)), n * (H / 2)), 256, 0, as_stream(stream)>>>(
        d, dy_ctot, dy_coff, H, W, C, static_cast<bf16*>(dx), dx_ctot, dx_coff, accumulate, a, act_ctot, act_coff);
    return check_launch("of_cnn_avgpool2_bwd");
  }
  long long tot = (long long)n * H * W * C;
  avgpool2_bwd_kernel<<<blocks_for(tot), 256, 0, as_stream(stream)>>>(d, dy_ctot, dy_coff, n, H, W, C,
                                                                       static_cast<bf16*>(dx), dx_ctot, dx_coff,
                                                                       accumulate, a, act_ctot, act_coff);
  return check_launch("of_cnn_avgpool2_bwd");
}

extern "C" int of_cnn_avgpool2_bwd(const void* dy, int dy_ctot, int dy_coff, int n, int H, int W, int C, void* dx,
                                   int dx_ctot, int dx_coff, int accumulate, void* stream) {
  return avgpool2_bwd(dy, dy_ctot, dy_coff, n, H, W, C, dx, dx_ctot, dx_coff, accumulate, nullptr, 0, 0, stream);
}

extern "C" int of_cnn_avgpool2_relu_bwd(const void* dy, int dy_ctot, int dy_coff, int n, int H, int W, int C, void* dx,
                                        int dx_ctot, int dx_coff, int accumulate, const void* act, int act_ctot,
                                        int act_coff, void* stream) {
  OF_REQUIRE(act, "of_cnn_avgpool2_relu_bwd: bad arguments");
  return avgpool2_bwd(dy, dy_ctot, dy_coff, n, H, W, C, dx, dx_ctot, dx_coff, accumulate, act, act_ctot, act_coff, stream);
}

extern "C" int of_cnn_upsample2(const void* x, int x_ctot, int x_coff, int n, int h, int w, int C, void* y, int y_ctot,
                                int y_coff, void* stream) {
  OF_REQUIRE(x && y && h > 0 && w > 0 && C > 0, "of_cnn_upsample2: bad arguments");
  if (v8_ok(x, x_ctot, x_coff, y, y_ctot, y_coff, C) && (long long)n * 2 * h <= 65535) {
    upsample2_v8_kernel<<<dim3(blocks_for((long long)(2 * w) * (C / 8)), n * 2 * h), 256, 0, as_stream(stream)>>>(
        static_cast<const bf16*>(x), x_ctot, x_coff, h, w, C, static_cast<bf16*>(y), y_ctot, y_coff);
    return check_launch("of_cnn_upsample2");
  }
  long long tot = (long long)n * 4 * h * w * C;
  upsample2_kernel<<<blocks_for(tot), 256, 0, as_stream(stream)>>>(static_cast<const bf16*>(x), x_ctot, x_coff, n, h,
                                                                    w, C, static_cast<bf16*>(y), y_ctot, y_coff);
  return check_launch("of_cnn_upsample2");
}

static int upsample2_bwd(const void* dy, int dy_ctot, int dy_coff, int n, int h, int w, int C, void* dx, int dx_ctot,
                         int dx_coff, const void* act, int act_ctot, int act_coff, void* stream) {
  OF_REQUIRE(dy && dx && h > 0 && w > 0 && C > 0, "of_cnn_upsample2_bwd: bad arguments");
  const bf16 *d = static_cast<const bf16*>(dy), *a = static_cast<const bf16*>(act);
  if (v8_ok(dy, dy_ctot, dy_coff, dx, dx_ctot, dx_coff, C) && (!act || v8_ok(act, act_ctot, act_coff, dx, 0, 0, C)) &&
      (long long)n * h <= 65535) {
    upsample2_bwd_v8_kernel<<<dim3(blocks_for((long long)w * (C / 8)), n * h), 256, 0, as_stream(stream)>>>(
        d, dy_ctot, dy_coff, h, w, C, static_cast<bf16*>(dx), dx_ctot, dx_coff, a, act_ctot, act_coff);
    return check_launch("of_cnn_upsample2_bwd");
  }
  long long tot = (long long)n * h * w * C;
  upsample2_bwd_kernel<<<blocks_for(tot), 256, 0, as_stream(stream)>>>(
      d, dy_ctot, dy_coff, n, h, w, C, static_cast<bf16*>(dx), dx_ctot, dx_coff, a, act_ctot, act_coff);
  return check_launch("of_cnn_upsample2_bwd");
}

extern "C" int of_cnn_upsample2_bwd(const void* dy, int dy_ctot, int dy_coff, int n, int h, int w, int C, void* dx,
                                    int dx_ctot, int dx_coff, void* stream) {
  return upsample2_bwd(dy, dy_ctot, dy_coff, n, h, w, C, dx, dx_ctot, dx_coff, nullptr, 0, 0, stream);
}

extern "C" int of_cnn_upsample2_relu_bwd(const void* dy, int dy_ctot, int dy_coff, int n, int h, int w, int C, void* dx,
                                         int dx_ctot, int dx_coff, const void* act, int act_ctot, int act_coff,
                                         void* stream) {
  OF_REQUIRE(act, "of_cnn_upsample2_relu_bwd: bad arguments");
  return upsample2_bwd(dy, dy_ctot, dy_coff, n, h, w, C, dx, dx_ctot, dx_coff, act, act_ctot, act_coff, stream);
}

extern "C" int of_cnn_relu_bwd(void* g, int g_ctot, int g_coff, const void* y, int y_ctot, int y_coff, long long P,
                               int C, void* stream) {
  OF_REQUIRE(g && y && P > 0 && C > 0, "of_cnn_relu_bwd: bad arguments");
  if (v8_ok(g, g_ctot, g_coff, y, y_ctot, y_coff, C)) {
    relu_bwd_v8_kernel<<<blocks_for(P * (C / 8)), 256, 0, as_stream(stream)>>>(
        static_cast<bf16*>(g), g_ctot, g_coff, static_cast<const bf16*>(y), y_ctot, y_coff, P, C);
    return check_launch("of_cnn_relu_bwd");
  }
  relu_bwd_kernel<<<blocks_for(P * C), 256, 0, as_stream(stream)>>>(static_cast<bf16*>(g), g_ctot, g_coff,
                                                                     static_cast<const bf16*>(y), y_ctot, y_coff, P, C);
  return check_launch("of_cnn_relu_bwd");
}

extern "C" int of_cnn_flow_mse(const float* pred, const float* label, long long P, void* dpred, int g_ctot,
                               double* loss, void* stream) {
  OF_REQUIRE(pred && label && loss && P > 0 && (!dpred || g_ctot >= 2), "of_cnn_flow_mse: bad arguments");
  flow_mse_kernel<<<blocks_for(P), 256, 0, as_stream(stream)>>>(pred, label, P, static_cast<bf16*>(dpred), g_ctot,
                                                                 loss);
  return check_launch("of_cnn_flow_mse");
}

extern "C" int of_cnn_adam(float* w, const float* g, float* m, float* v, long long n, float lr, float b1, float b2,
                           float eps, int step, void* stream) {
  OF_REQUIRE(w && g && m && v && n > 0 && step >= 1, "of_cnn_adam: bad arguments");
  float bc1 = (float)(1.0 - pow((double)b1, step)), bc2 = (float)(1.0 - pow((double)b2, step));
  adam_kernel<<<blocks_for(n), 256, 0, as_stream(stream)>>>(w, g, m, v, n, lr, b1, b2, eps, bc1, bc2);
  return check_launch("of_cnn_adam");
}

extern "C" int of_cnn_pack_weights(const float* w, int cout, int cin, int cout_pad, int cin_pad, int transpose_flip,
                                   void* out, void* stream) {
  OF_REQUIRE(w && out && cout > 0 && cin > 0 && cout_pad >= cout && cin_pad >= cin, "of_cnn_pack_weights: bad arguments");
  long long tot = 9LL * cout_pad * cin_pad;
  pack_weights_kernel<<<blocks_for(tot), 256, 0, as_stream(stream)>>>(w, cout, cin, cout_pad, cin_pad, transpose_flip,
                                                                       static_cast<bf16*>(out));
  return check_launch("of_cnn_pack_weights");
}

extern "C" int of_cnn_pack_weights_many(int count, const float* const* w, const int* dims, void* const* out,
                                        void* stream) {
  OF_REQUIRE(count > 0 && count <= PW_MAX && w && dims && out, "of_cnn_pack_weights_many: %d entries (1..%d)", count,
             PW_MAX);
  PackMany p;
  int most = 0;
  for (int i = 0; i < count; i++) {
    const int *d = dims + 5 * i, cout = d[0], cin = d[1], cp = d[2], ip = d[3];
    OF_REQUIRE(w[i] && out[i] && cout > 0 && cin > 0 && cp >= cout && ip >= cin && cp <= 4096 && ip <= 4096,
               "of_cnn_pack_weights_many: entry %d", i);
    p.w[i] = w[i];
    p.out[i] = static_cast<bf16*>(out[i]);
    p.cout[i] = (short)cout;
    p.cin[i] = (short)cin;
    p.cout_pad[i] = (short)cp;
    p.cin_pad[i] = (short)ip;
    p.flip[i] = d[4] != 0;
    if (9 * cp * ip > most) most = 9 * cp * ip;
  }
  const int g = blocks_for(most) < 2 * kNumSMs ? blocks_for(most) : 2 * kNumSMs;
  pack_weights_many_kernel<<<dim3(g, count), 256, 0, as_stream(stream)>>>(p);
  return check_launch("of_cnn_pack_weights_many");
}

extern "C" int of_cnn_split_flow(const float* flow, int h, int w, float* u, float* v, int pitch, void* stream) {
  OF_REQUIRE(flow && u && v && h > 0 && w > 0 && pitch >= w, "of_cnn_split_flow: bad arguments");
  split_flow_kernel<<<blocks_for((long long)h * w), 256, 0, as_stream(stream)>>>(flow, h, w, u, v, pitch);
  return check_launch("of_cnn_split_flow");
}

extern "C" int of_cnn_conv3x3_wgrad_tc(const void* x, int x_ctot, int x_coff, const void* dy, int dy_ctot, int dy_coff,
                                       int n, int H, int W, int cin, int cout, float* dw, unsigned* err, void* stream) {
  OF_REQUIRE(x && dy && dw && err && n > 0 && H > 0 && W > 0 && cin > 0 && cout > 0 && cin <= 512 && cout <= 512,
             "of_cnn_conv3x3_wgrad_tc: bad arguments");
  OF_REQUIRE(x_ctot % 8 == 0 && x_coff % 8 == 0 && dy_ctot % 8 == 0 && dy_coff % 8 == 0 && x_coff + cin <= x_ctot &&
                 dy_coff + cout <= dy_ctot,
             "of_cnn_conv3x3_wgrad_tc: channel slices");
  int bw = W < WT_KP ? W : WT_KP;
  OF_REQUIRE(WT_KP % bw == 0 && W % bw == 0, "of_cnn_conv3x3_wgrad_tc: width %d", W);
  int bh = WT_KP / bw < H ? WT_KP / bw : H;
  OF_REQUIRE(H % bh == 0 && (WT_KP / bw) % bh == 0, "of_cnn_conv3x3_wgrad_tc: height %d", H);
  int nb = WT_KP / (bw * bh);
  OF_REQUIRE(n % nb == 0, "of_cnn_conv3x3_wgrad_tc: %d images of %d x %d", n, H, W);
  WgParams p;
  p.n = n;
  p.H = H;
  p.W = W;
  p.bw = bw;
  p.bh = bh;
  p.nb = nb;
  p.tiles_x = W / bw;
  p.tiles_per_group = (W / bw) * (H / bh);
  p.nchunk = (n / nb) * p.tiles_per_group;
  p.a_is_dy = cout >= cin;
  p.a_ch = p.a_is_dy ? cout : cin;
  p.b_ch = p.a_is_dy ? cin : cout;
  p.mtiles = (p.a_ch + 127) / 128;
  p.ntiles = (p.b_ch + 255) / 256;
  int nb_last = p.b_ch - (p.ntiles - 1) * 256;  // every N tile uses the same MMA N: the largest needed
  int nmax = p.ntiles > 1 ? 256 : nb_last;
  p.nmma = (nmax + 15) / 16 * 16;
  p.batoms = (p.nmma + 63) / 64;
  p.cin = cin;
  p.cout = cout;
  p.dw = dw;
  p.err = err;
  p.a_bytes = 2 * 8192;
  p.b_bytes = (uint32_t)p.batoms * 8192;
  // As many taps per CTA as TMEM holds accumulators for, fewer where the chip would then not
  // have a CTA of at least 4 chunks for each SM.
  p.cstride = (p.nmma + 31) / 32 * 32;
  const int tiles_mn = p.mtiles * p.ntiles;
  p.tg = 9 * p.cstride <= 512 ? 9 : (3 * p.cstride <= 512 ? 3 : 1);
  while (p.tg > 1 && (long long)(9 / p.tg) * tiles_mn * (p.nchunk / 4) < kNumSMs) p.tg /= 3;
  p.stage_bytes = p.a_bytes + p.tg * p.b_bytes;
  p.stages = (int)(200 * 1024 / p.stage_bytes);  // at least 2: 88 KB at most
  if (p.stages > WT_STAGES) p.stages = WT_STAGES;
  const int cols = p.tg * p.cstride;
  p.tmem_cols = cols <= 32 ? 32 : (cols <= 64 ? 64 : (cols <= 128 ? 128 : (cols <= 256 ? 256 : 512)));
  size_t smem = 1024 + (size_t)p.stages * p.stage_bytes;
  size_t floor_smem = (size_t)p.tmem_cols * 448;  // resident CTAs never exceed 512 TMEM columns
  if (smem < floor_smem) smem = floor_smem;
  // split the pixel chunks over whole waves of resident CTAs
  const long long resident = 228 * 1024 / (long long)(smem + 2048);
  const long long tiles = 9LL / p.tg * tiles_mn;
  const int least = p.tg > 1 ? 4 : 8;
  long long ks = kNumSMs * (resident > 1 ? resident : 1) / tiles;
  if (ks < 1) ks = 1;
  // The tensor core truncates its running sums, so a sum's error grows with the chunks one CTA
  // adds: whole waves until there are as many splits as four CTAs per SM with a tap each would
  // make, eight chunks at least (16 x 256 x 256, 192 -> 64 channels: 500 accumulations in a chain
  // there, 683 in one wave, 342 in two).
  long long splits = (4LL * kNumSMs + 9 * tiles_mn - 1) / (9 * tiles_mn);
  if (splits > p.nchunk / 8) splits = p.nchunk / 8;
  if (ks < splits) ks *= (splits + ks - 1) / ks;
  if (ks > p.nchunk / least) ks = p.nchunk / least;
  if (ks < 1) ks = 1;
  p.chunks_per_cta = (int)((p.nchunk + ks - 1) / ks);
  ks = (p.nchunk + p.chunks_per_cta - 1) / p.chunks_per_cta;
  CUtensorMap tma, tmb;
  {
    const void* ap = p.a_is_dy ? dy : x;
    int act = p.a_is_dy ? dy_ctot : x_ctot, aco = p.a_is_dy ? dy_coff : x_coff;
    uint64_t dims[4] = {(uint64_t)p.a_ch, (uint64_t)W, (uint64_t)H, (uint64_t)n};
    uint64_t st[3] = {(uint64_t)act * 2, (uint64_t)W * act * 2, (uint64_t)H * W * act * 2};
    uint32_t box[4] = {64, (uint32_t)bw, (uint32_t)bh, (uint32_t)nb};
    int rc = tmap_bf16(&tma, static_cast<const bf16*>(ap) + aco, 4, dims, st, box, 128);
    if (rc) return rc;
  }
  {
    const void* bp = p.a_is_dy ? x : dy;
    int bct = p.a_is_dy ? x_ctot : dy_ctot, bco = p.a_is_dy ? x_coff : dy_coff;
    uint64_t dims[4] = {(uint64_t)p.b_ch, (uint64_t)W, (uint64_t)H, (uint64_t)n};
    uint64_t st[3] = {(uint64_t)bct * 2, (uint64_t)W * bct * 2, (uint64_t)H * W * bct * 2};
    uint32_t box[4] = {64, (uint32_t)bw, (uint32_t)bh, (uint32_t)nb};
    int rc = tmap_bf16(&tmb, static_cast<const bf16*>(bp) + bco, 4, dims, st, box, 128);
    if (rc) return rc;
  }
  {
    cudaError_t e = OF_SMEM_OPT_IN(wgrad_tc_kernel, smem);
    if (e != cudaSuccess)
      return set_error(OF_ERR_CUDA, "of_cnn_conv3x3_wgrad_tc: %zu B of shared memory: %s", smem, cudaGetErrorString(e));
  }
  dim3 grid((unsigned)ks, tiles_mn, 9 / p.tg);
  wgrad_tc_kernel<<<grid, CV_THREADS, smem, as_stream(stream)>>>(tma, tmb, p);
  return check_launch("of_cnn_conv3x3_wgrad_tc");
}

extern "C" int of_cnn_flow_up(const float* flow, int h, int w, int factor, float* U, float* V, int pitch, float scale,
                              void* stream) {
  OF_REQUIRE(flow && U && V && h > 0 && w > 0 && factor >= 1 && factor <= 16 && pitch >= factor * w,
             "of_cnn_flow_up: bad arguments");
  dim3 g((factor * w + 255) / 256, factor * h);
  flow_up_kernel<<<g, 256, 0, as_stream(stream)>>>(flow, h, w, factor, U, V, pitch, scale);
  return check_launch("of_cnn_flow_up");
}
