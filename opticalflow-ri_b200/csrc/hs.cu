// A6/A7 Horn-Schunck (src/HornSchunck.py:28-126), bit-exact with the reference.
//
// Derivatives: the 2x2 correlations of computeDerivatives(frame1, frame0) with scipy's
// 'mirror' border, each accumulated in double over the non-zero weights in C order and
// rounded to float32.  Sweep: the 3x3 averaging kernel (weights float32(1/12),
// float32(1/6)) accumulated the same way, then HS_helper2's float32 update.
// Layout: U, V, fx, fy, ft are H x W float32 planes with a shared pitch.  A sweep reads
// 3 coefficient planes and the two 3x3 neighbourhoods (served by L1) and writes U, V:
// 28 B per pixel of HBM/L2 traffic.
#include "common.cuh"
#include "hsweep.cuh"

namespace ofb {

__device__ __forceinline__ double dacc(double a, float v, double w) { return __dadd_rn(a, __dmul_rn((double)v, w)); }

__global__ void hs_deriv_kernel(const float* __restrict__ f0, const float* __restrict__ f1, float* __restrict__ fx,
                                float* __restrict__ fy, float* __restrict__ ft, int H, int W, int pitch) {
  int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
  if (x >= W || y >= H) return;
  int y1 = mirror1(y + 1, H), x1 = mirror1(x + 1, W);
  size_t i00 = (size_t)y * pitch + x, i01 = (size_t)y * pitch + x1, i10 = (size_t)y1 * pitch + x, i11 = (size_t)y1 * pitch + x1;
  float a00 = f1[i00], a01 = f1[i01], a10 = f1[i10], a11 = f1[i11];  // frame t1
  float b00 = f0[i00], b01 = f0[i01], b10 = f0[i10], b11 = f0[i11];  // frame t0
  // kernelX flipped: +.25 -.25 / +.25 -.25 ; kernelY flipped: +.25 +.25 / -.25 -.25
  double t;
  t = dacc(dacc(dacc(dacc(0.0, a00, 0.25), a01, -0.25), a10, 0.25), a11, -0.25);
  float gx1 = (float)t;
  t = dacc(dacc(dacc(dacc(0.0, b00, 0.25), b01, -0.25), b10, 0.25), b11, -0.25);
  float gx0 = (float)t;
  t = dacc(dacc(dacc(dacc(0.0, a00, 0.25), a01, 0.25), a10, -0.25), a11, -0.25);
  float gy1 = (float)t;
  t = dacc(dacc(dacc(dacc(0.0, b00, 0.25), b01, 0.25), b10, -0.25), b11, -0.25);
  float gy0 = (float)t;
  t = dacc(dacc(dacc(dacc(0.0, b00, 0.25), b01, 0.25), b10, 0.25), b11, 0.25);
  float gt0 = (float)t;
  t = dacc(dacc(dacc(dacc(0.0, a00, -0.25), a01, -0.25), a10, -0.25), a11, -0.25);
  float gt1 = (float)t;
  fx[i00] = __fadd_rn(gx1, gx0);
  fy[i00] = __fadd_rn(gy1, gy0);
  ft[i00] = __fadd_rn(gt0, gt1);
}

__global__ void hs_sweep_kernel(const float* __restrict__ fx, const float* __restrict__ fy,
                                const float* __restrict__ ft, const float* __restrict__ U, const float* __restrict__ V,
                                float* __restrict__ Un, float* __restrict__ Vn, int H, int W, int pitch, float a2) {
  int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
  if (x >= W || y >= H) return;
  const double wc = (double)(1.0f / 12.0f), we = (double)(1.0f / 6.0f);
  int ym = mirror1(y - 1, H), yp = mirror1(y + 1, H), xm = mirror1(x - 1, W), xp = mirror1(x + 1, W);
  const size_t rm = (size_t)ym * pitch, r0 = (size_t)y * pitch, rp = (size_t)yp * pitch;
  double su = 0.0, sv = 0.0;
  su = dacc(su, U[rm + xm], wc); sv = dacc(sv, V[rm + xm], wc);
  su = dacc(su, U[rm + x], we);  sv = dacc(sv, V[rm + x], we);
  su = dacc(su, U[rm + xp], wc); sv = dacc(sv, V[rm + xp], wc);
  su = dacc(su, U[r0 + xm], we); sv = dacc(sv, V[r0 + xm], we);
  su = dacc(su, U[r0 + xp], we); sv = dacc(sv, V[r0 + xp], we);
  su = dacc(su, U[rp + xm], wc); sv = dacc(sv, V[rp + xm], wc);
  su = dacc(su, U[rp + x], we);  sv = dacc(sv, V[rp + x], we);
  su = dacc(su, U[rp + xp], wc); sv = dacc(sv, V[rp + xp], wc);
  float ua = (float)su, va = (float)sv;
  size_t i = r0 + x;
  float gx = fx[i], gy = fy[i];
  float num = __fadd_rn(__fadd_rn(__fmul_rn(gx, ua), __fmul_rn(gy, va)), ft[i]);
  float den = __fadd_rn(__fadd_rn(a2, __fmul_rn(gx, gx)), __fmul_rn(gy, gy));
  float der = __fdiv_rn(num, den);
  Un[i] = __fsub_rn(ua, __fmul_rn(gx, der));
  Vn[i] = __fsub_rn(va, __fmul_rn(gy, der));
}

// Temporally blocked sweeps: one pass runs up to HB_T sweeps on a region of the image whose
// cells the CTA's threads hold in registers in 2 x 4 blocks (hr_sweep, hsweep.cuh), so the
// three derivative planes and (U, V) cross HBM/L2 once per HB_T sweeps.  A CTA owns
// 56 x 24 pixels and sweeps a 64 x 32 region (halo HB_T): after sweep s the cells at least
// s + 1 from the region's edge are exact, after HB_T sweeps the owned ones, which are written
// back.  A warp is one row of blocks.
//
// What bounds it: the issue slots (65 instructions per cell update, 16 of them float64
// multiply-adds) at 50 % busy, and the latency of the pass's loads and barriers behind two
// CTAs per SM (128 registers a thread).  600 sweeps, one pair alone: 256 x 256 2.75 -> 1.14 ms,
// 512 x 512 3.1 -> 1.22 ms; 100 sweeps of 2048 x 2048 3.96 -> 2.20 ms (106 -> 191 G cell updates
// per second) against the column walk with one cell per thread and row it replaces.  4 x 4
// blocks spill at 12 warps per SM (113 G/s), a 64 x 64 region in one CTA of 512 threads does
// less halo work but leaves its loads exposed (164 G/s).
constexpr int HB_T = 4, HB_RW = 64, HB_RH = 32, HB_TW = HB_RW - 2 * HB_T, HB_TH = HB_RH - 2 * HB_T;
constexpr int HB_BX = 2, HB_BY = 4;  // block of a thread
using HbGeom = HrGeom<HB_RW, HB_RH, HB_BX, HB_BY>;
constexpr size_t HB_SMEM = 2 * HbGeom::BUF;  // ping-pong: one barrier per sweep

// A block's cells of a plane, 0 outside the image.  `inside`: the whole region is, and the
// rows are 8-byte aligned: no branch between the loads, which are then all in flight at once.
__device__ __forceinline__ void hb_load(float2 out[HB_BY], const float* __restrict__ p, int gy0, int gx0, int H, int W,
                                        int pitch, bool inside) {
  const float* r = p + (ptrdiff_t)gy0 * pitch + gx0;
  if (inside) {
#pragma unroll
    for (int j = 0; j < HB_BY; j++) out[j] = *reinterpret_cast<const float2*>(r + (size_t)j * pitch);
  } else {
#pragma unroll
    for (int j = 0; j < HB_BY; j++) {
      const bool y = gy0 + j >= 0 && gy0 + j < H;
      const float* q = r + (ptrdiff_t)j * pitch;
      out[j] = make_float2(y && gx0 >= 0 && gx0 < W ? q[0] : 0.f, y && gx0 + 1 >= 0 && gx0 + 1 < W ? q[1] : 0.f);
    }
  }
}

__device__ __forceinline__ void hb_store2(float* __restrict__ p, const double v[2], int gy, int gx, int H, int W,
                                          int pitch, bool vec) {
  if (gy >= H || gx >= W) return;
  float* r = p + (size_t)gy * pitch + gx;
  if (vec && gx + 2 <= W) {
    *reinterpret_cast<float2*>(r) = make_float2((float)v[0], (float)v[1]);
  } else {
    r[0] = (float)v[0];
    if (gx + 1 < W) r[1] = (float)v[1];
  }
}

struct HbPass {
  const float *fx, *fy, *ft, *U, *V;
  float *Un, *Vn;
  int H, W, pitch, nsw, vec;
  float a2;
  float one;  // 1.0f (hr_row)
};

using HbBlock = HrBlock<HB_BX, HB_BY>;

// Loads the block's cells.  Returns whether those of two corners are so small (and not zero) that
// numerators made of such may leave the refined quotient's range: a guess, from 4 of 16 values, since
// the flow that diffuses into a region is of one size over a block.
__device__ __forceinline__ bool hb_load_uv(HbBlock& K, const HbPass& P, int gy0, int gx0, bool inside) {
  float2 u[HB_BY], v[HB_BY];
  hb_load(u, P.U, gy0, gx0, P.H, P.W, P.pitch, inside);
  hb_load(v, P.V, gy0, gx0, P.H, P.W, P.pitch, inside);
#pragma unroll
  for (int j = 0; j < HB_BY; j++) {
    K.u[j][0] = u[j].x; K.u[j][1] = u[j].y;
    K.v[j][0] = v[j].x; K.v[j][1] = v[j].y;
  }
  auto key = [](float x) { return 2u * __float_as_uint(x) - 1u; };
  return min(min(key(u[0].x), key(v[0].x)), min(key(u[HB_BY - 1].y), key(v[HB_BY - 1].y))) < HR_LO;
}

// The sweeps of a pass from the cells that the CTA's blocks have published in the first buffer; on
// return the last sweep's are in the blocks only.
template <bool RAG, int Q>
__device__ __forceinline__ void hb_sweeps(HbBlock& K, const HbPass& P, double2* sm, bool in, int r0, int c0,
                                          const HrWin& win) {
  // a warp whose rows no later sweep reads (the outermost, in the last sweep) sits out
  auto needed = [&](int k) { return in && r0 + HB_BY > 1 + k && r0 < HB_RH - 1 - k; };
#pragma unroll 1
  for (int s = 0; s < P.nsw; s += 2) {
    double2* const b0 = sm;
    double2* const b1 = sm + HB_RW * HB_RH;
    if (needed(s)) hr_sweep<HB_RW, HB_RH, HB_BX, HB_BY, RAG, Q>(K, b0, r0, c0, win);
    if (s + 1 >= P.nsw) break;
    if (needed(s)) hr_publish<HB_RW, HB_RH, HB_BX, HB_BY>(K, b1, r0, c0);
    __syncthreads();
    if (needed(s + 1)) hr_sweep<HB_RW, HB_RH, HB_BX, HB_BY, RAG, Q>(K, b1, r0, c0, win);
    if (s + 2 >= P.nsw) break;
    if (needed(s + 1)) hr_publish<HB_RW, HB_RH, HB_BX, HB_BY>(K, b0, r0, c0);
    __syncthreads();
  }
}

// The CTA's region and the thread's block in it.
struct HbPos {
  int x0, y0;    // image position of region cell (0, 0)
  int c0, r0;    // the block's first region cell
  int gx0, gy0;  // its image position
  bool in;       // the block has cells in the image
  bool inside;   // the whole region is in the image, with 8-byte aligned rows
};

__device__ __forceinline__ HbPos hb_pos(const HbPass& P) {
  HbPos p;
  p.x0 = blockIdx.x * HB_TW - HB_T;
  p.y0 = blockIdx.y * HB_TH - HB_T;
  p.c0 = ((int)threadIdx.x % HbGeom::NX) * HB_BX;
  p.r0 = ((int)threadIdx.x / HbGeom::NX) * HB_BY;
  p.gx0 = p.x0 + p.c0;
  p.gy0 = p.y0 + p.r0;
  p.in = p.gx0 + HB_BX > 0 && p.gy0 + HB_BY > 0 && p.gx0 < P.W && p.gy0 < P.H;
  p.inside = !(p.x0 < 0 || p.y0 < 0 || p.x0 + HB_RW > P.W || p.y0 + HB_RH > P.H) && P.vec;
  return p;
}

// Loads the block's derivatives; the result is hr_init_den's.
__device__ __forceinline__ bool hb_load_g(HbBlock& K, const HbPass& P, const HbPos& p) {
  float2 a[HB_BY], b[HB_BY], c[HB_BY];
  hb_load(a, P.fx, p.gy0, p.gx0, P.H, P.W, P.pitch, p.inside);
  hb_load(b, P.fy, p.gy0, p.gx0, P.H, P.W, P.pitch, p.inside);
  hb_load(c, P.ft, p.gy0, p.gx0, P.H, P.W, P.pitch, p.inside);
#pragma unroll
  for (int j = 0; j < HB_BY; j++) {
    K.g[j][0] = make_float2(a[j].x, b[j].x);
    K.g[j][1] = make_float2(a[j].y, b[j].y);
    K.gt[j][0] = c[j].x; K.gt[j][1] = c[j].y;
  }
  return hr_init_den(K, P.a2, P.one);
}

__device__ __forceinline__ void hb_store(const HbBlock& K, const HbPass& P, const HbPos& p) {
  if (p.in && p.c0 >= HB_T && p.c0 < HB_T + HB_TW && p.r0 >= HB_T && p.r0 < HB_T + HB_TH) {
#pragma unroll
    for (int j = 0; j < HB_BY; j++) {
      hb_store2(P.Un, K.u[j], p.gy0 + j, p.gx0, P.H, P.W, P.pitch, P.vec);
      hb_store2(P.Vn, K.v[j], p.gy0 + j, p.gx0, P.H, P.W, P.pitch, P.vec);
    }
  }
}

extern __shared__ __align__(16) double2 hb_sm[];

// The CTA's pass with the wide quotient, or with the divide where that one's range fails too.  A
// function of its own that starts from the image: in the kernel its registers cost every pass 1 to
// 2 % from 1024 x 1024 on.  512 x 512, 600 sweeps, one half the same texture in both frames: 1.93 ms
// (4.50 where such passes were run again with the divide, 1.22 without tiny numerators).
__device__ __noinline__ void hb_pass_wide(const HbPass& P) {
  const HbPos p = hb_pos(P);
  const HrWin win = hr_window<HB_RW, HB_RH, HB_BX, HB_BY>(p.r0, p.c0, p.gy0, p.gx0, P.H, P.W);
  HbBlock K;
  bool ok = true;
  if (p.in) {
    ok = hb_load_g(K, P, p);
    hb_load_uv(K, P, p.gy0, p.gx0, p.inside);
    hr_publish<HB_RW, HB_RH, HB_BX, HB_BY>(K, hb_sm, p.r0, p.c0);
  }
  bool bad = __syncthreads_or(p.in && !ok);
  if (!bad) {
    hb_sweeps<true, HR_WIDE>(K, P, hb_sm, p.in, p.r0, p.c0, win);
    bad = __syncthreads_or(p.in && !hr_in_range(K, HR_WIDE));
    if (bad) {
      if (p.in) {
        hb_load_uv(K, P, p.gy0, p.gx0, p.inside);
        hr_publish<HB_RW, HB_RH, HB_BX, HB_BY>(K, hb_sm, p.r0, p.c0);
      }
      __syncthreads();
    }
  }
  if (bad) hb_sweeps<true, HR_DIVIDE>(K, P, hb_sm, p.in, p.r0, p.c0, win);
  hb_store(K, P, p);
}

__global__ void __launch_bounds__(HbGeom::NT, 2) hs_pass_kernel(const __grid_constant__ HbPass P) {
  // passes after the first are programmatic dependents of the pass before them: they take the
  // SM slots its tail frees and load the derivatives, which do not change during a solve
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const HbPos p = hb_pos(P);
  HbBlock K;
  bool wide = p.in && !hb_load_g(K, P, p);
  asm volatile("griddepcontrol.wait;" ::: "memory");
  if (p.in) {
    wide = hb_load_uv(K, P, p.gy0, p.gx0, p.inside) || wide;
    hr_publish<HB_RW, HB_RH, HB_BX, HB_BY>(K, hb_sm, p.r0, p.c0);
  }
  // formed here, while the loads are on their way: behind the barrier it would stand in front of the
  // first sweep (600 sweeps of 256 x 256 1.21 -> 1.14 ms)
  HrWin win = hr_window<HB_RW, HB_RH, HB_BX, HB_BY>(p.r0, p.c0, p.gy0, p.gx0, P.H, P.W);
  // the region holds blocks that the image ends inside of
  const bool rag = (P.W % HB_BX && p.x0 + HB_RW > P.W) || (P.H % HB_BY && p.y0 + HB_RH > P.H);
  asm volatile("" : "+r"(win.cl), "+r"(win.cr), "+r"(win.rt), "+r"(win.rb));
  if (!__syncthreads_or(wide)) {
    if (rag)
      hb_sweeps<true, HR_REFINED>(K, P, hb_sm, p.in, p.r0, p.c0, win);
    else
      hb_sweeps<false, HR_REFINED>(K, P, hb_sm, p.in, p.r0, p.c0, win);
    if (!__syncthreads_or(p.in && !hr_in_range(K, HR_REFINED))) {
      hb_store(K, P, p);
      return;
    }
  }
  hb_pass_wide(P);
}

__global__ void copy2_kernel(const float* __restrict__ a, const float* __restrict__ b, float* __restrict__ ao,
                             float* __restrict__ bo, int W, int pitch) {
  int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y;
  if (x < W) {
    size_t i = (size_t)y * pitch + x;
    ao[i] = a[i];
    bo[i] = b[i];
  }
}

// sum of squared differences of two plane pairs into acc[0], acc[1] (double atomics)
__global__ void sqdiff2_kernel(const float* __restrict__ a, const float* __restrict__ a0, const float* __restrict__ b,
                               const float* __restrict__ b0, int H, int W, int pitch, double* acc) {
  double sa = 0.0, sb = 0.0;
  for (int y = blockIdx.y; y < H; y += gridDim.y)
    for (int x = blockIdx.x * blockDim.x + threadIdx.x; x < W; x += gridDim.x * blockDim.x) {
      size_t i = (size_t)y * pitch + x;
      double da = (double)a[i] - (double)a0[i], db = (double)b[i] - (double)b0[i];
      sa += da * da;
      sb += db * db;
    }
  for (int o = 16; o > 0; o >>= 1) {
    sa += __shfl_down_sync(0xffffffffu, sa, o);
    sb += __shfl_down_sync(0xffffffffu, sb, o);
  }
  __shared__ double ra[32], rb[32];
  int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) { ra[w] = sa; rb[w] = sb; }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int k = 1; k < (int)(blockDim.x >> 5); k++) { sa += ra[k]; sb += rb[k]; }
    atomicAdd(acc, sa);
    atomicAdd(acc + 1, sb);
  }
}

// status (optional): a persistent solve's status word; a solve whose bounded waits gave up
// reports a NaN error
__global__ void hs_err_kernel(const double* acc, double n, double* err_out, const int* status) {
  const bool failed = status && (*status & OF_ST_WAIT_TIMEOUT);
  *err_out = failed ? __longlong_as_double(0x7ff8000000000000ll) : (sqrt(acc[0]) + sqrt(acc[1])) / n;
}

}  // namespace ofb

using namespace ofb;

extern "C" int of_hs_derivatives(const float* I0, const float* I1, float* fx, float* fy, float* ft, int H, int W,
                                 int pitch, void* stream) {
  OF_REQUIRE(!bad_plane(I0, H, W, pitch) && I1 && fx && fy && ft, "of_hs_derivatives: bad plane");
  dim3 blk(32, 8), grd((W + 31) / 32, (H + 7) / 8);
  hs_deriv_kernel<<<grd, blk, 0, as_stream(stream)>>>(I0, I1, fx, fy, ft, H, W, pitch);
  return check_launch("of_hs_derivatives");
}

// of_hs_solve_persistent: one pair through the persistent kernels of hsq.cu (of_hs_batch,
// automatic schedule: tagged halos, or counters for up to 8 sweeps and thin images, when all
// the launch's CTAs run at once, else the device work queue, whose items only wait for items
// of running CTAs, so it is correct beside any other work on the GPU, if slower there).
constexpr int kHsSolveShape = 3;  // of_hs_batch tile shape for one pair: 32 x 32 regions, 8 sweeps per pass

static size_t hs_persistent_ws(int H, int W, int pitch) {
  OfHsBatchPair q = {nullptr, nullptr, nullptr, nullptr, H, W, pitch, 0.f, 1};
  return of_hs_batch_workspace_size(&q, 1);
}

// Whether of_hs_solve_persistent runs a size in one launch.  Images with more tiles than SMs: a
// launch per pass, whose tiles all SMs share, beats the persistent queue (600 sweeps of 512 x 512:
// 1.22 ms against 2.98).
static bool hs_one_launch(int H, int W) { return hs_halo_bytes(H, W) != 0 || H < 16 || W < 16; }

// Covers both of_hs_solve and of_hs_solve_persistent.
extern "C" size_t of_hs_workspace_size(int H, int W, int pitch) {
  size_t N = (size_t)H * pitch;
  Sizer s;  // of_hs_solve
  for (int i = 0; i < 7; i++) s.take<float>(N);
  s.take<double>(2);
  if (!hs_one_launch(H, W)) return s.off;
  Sizer q;  // of_hs_solve_persistent: initial flow (for the error), sums, status, batch workspace
  q.take<float>(2 * N);
  q.take<double>(2);
  q.take<int>(1);
  q.take<unsigned char>(hs_persistent_ws(H, W, pitch));
  q.take<unsigned char>(hs_halo_bytes(H, W));
  return s.off > q.off ? s.off : q.off;
}

extern "C" int of_hs_solve(const float* I0, const float* I1, float* U, float* V, int H, int W, int pitch, float alpha,
                           int niter, double* err_out, void* workspace, size_t workspace_bytes, void* stream) {
  OF_REQUIRE(!bad_plane(I0, H, W, pitch) && I1 && U && V, "of_hs_solve: bad plane");
  OF_REQUIRE(niter >= 0, "of_hs_solve: niter < 0");
  if (!workspace || workspace_bytes < of_hs_workspace_size(H, W, pitch))
    return set_error(OF_ERR_WORKSPACE, "of_hs_solve: workspace too small (%zu < %zu)", workspace_bytes,
                     of_hs_workspace_size(H, W, pitch));
  cudaStream_t st = as_stream(stream);
  size_t N = (size_t)H * pitch;
  Carver c(workspace, workspace_bytes);
  float *fx = c.take<float>(N), *fy = c.take<float>(N), *ft = c.take<float>(N);
  float *U0 = c.take<float>(N), *V0 = c.take<float>(N), *Ub = c.take<float>(N), *Vb = c.take<float>(N);
  double* acc = c.take<double>(2);
  dim3 blk(32, 8), grd((W + 31) / 32, (H + 7) / 8);
  dim3 rgrid((W + 255) / 256, H);
  hs_deriv_kernel<<<grd, blk, 0, st>>>(I0, I1, fx, fy, ft, H, W, pitch);
  copy2_kernel<<<rgrid, 256, 0, st>>>(U, V, U0, V0, W, pitch);
  float a2 = alpha * alpha;
  if (H >= 16 && W >= 16 && niter > 0) {  // temporally blocked: HB_T sweeps per launch
    cudaError_t e = OF_SMEM_OPT_IN(hs_pass_kernel, HB_SMEM);
    if (e != cudaSuccess) return set_error(OF_ERR_CUDA, "of_hs_solve: %s", cudaGetErrorString(e));
    const int np = (niter + HB_T - 1) / HB_T;
    dim3 pg((W + HB_TW - 1) / HB_TW, (H + HB_TH - 1) / HB_TH);
    // the workspace planes start 256-byte aligned: the callers' U, V decide
    const int vec = (pitch % 2) == 0 && ((reinterpret_cast<uintptr_t>(U) | reinterpret_cast<uintptr_t>(V)) & 7) == 0;
    for (int p = 0; p < np; p++) {
      // the last pass writes U, V; earlier ones alternate with Ub, Vb; the first reads U0, V0
      const bool to_uv = ((np - 1 - p) & 1) == 0;
      const float* su = p == 0 ? U0 : (to_uv ? Ub : U);
      const float* sv = p == 0 ? V0 : (to_uv ? Vb : V);
      const int nsw = niter - p * HB_T < HB_T ? niter - p * HB_T : HB_T;
      HbPass P{fx, fy, ft, su, sv, to_uv ? U : Ub, to_uv ? V : Vb, H, W, pitch, nsw, vec, a2, 1.0f};
      cudaLaunchAttribute pdl[1];
      pdl[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
      pdl[0].val.programmaticStreamSerializationAllowed = 1;
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = pg;
      cfg.blockDim = dim3(HbGeom::NT);
      cfg.dynamicSmemBytes = HB_SMEM;
      cfg.stream = st;
      cfg.attrs = pdl;
      cfg.numAttrs = p > 0 ? 1 : 0;
      e = cudaLaunchKernelEx(&cfg, hs_pass_kernel, P);
      if (e != cudaSuccess) return set_error(OF_ERR_CUDA, "of_hs_solve: pass launch: %s", cudaGetErrorString(e));
    }
    long long n = 2 + np;
    if (err_out) {
      cudaMemsetAsync(acc, 0, 2 * sizeof(double), st);
      dim3 g2((W + 255) / 256 < 4 ? (W + 255) / 256 : 4, H < 256 ? H : 256);
      sqdiff2_kernel<<<g2, 256, 0, st>>>(U, U0, V, V0, H, W, pitch, acc);
      hs_err_kernel<<<1, 1, 0, st>>>(acc, (double)H * (double)W, err_out, nullptr);
      n += 2;
    }
    return check_launch("of_hs_solve", n);
  }
  for (int k = 0; k < niter; k++) {
    const float *su, *sv;
    float *du, *dv;
    if (k == 0) { su = U0; sv = V0; du = U; dv = V; }
    else if (k & 1) { su = U; sv = V; du = Ub; dv = Vb; }
    else { su = Ub; sv = Vb; du = U; dv = V; }
    hs_sweep_kernel<<<grd, blk, 0, st>>>(fx, fy, ft, su, sv, du, dv, H, W, pitch, a2);
  }
  long long n = 2 + niter;
  if (niter > 0 && ((niter - 1) & 1)) {
    copy2_kernel<<<rgrid, 256, 0, st>>>(Ub, Vb, U, V, W, pitch);
    n += 1;
  }
  if (err_out) {
    cudaMemsetAsync(acc, 0, 2 * sizeof(double), st);
    dim3 g2((W + 255) / 256 < 4 ? (W + 255) / 256 : 4, H < 256 ? H : 256);
    sqdiff2_kernel<<<g2, 256, 0, st>>>(U, U0, V, V0, H, W, pitch, acc);
    hs_err_kernel<<<1, 1, 0, st>>>(acc, (double)H * (double)W, err_out, nullptr);
    n += 2;
  }
  return check_launch("of_hs_solve", n);
}

extern "C" int of_hs_solve_persistent(const float* I0, const float* I1, float* U, float* V, int H, int W, int pitch,
                                      float alpha, int niter, double* err_out, void* workspace, size_t workspace_bytes,
                                      void* stream) {
  return of_hs_solve_persistent_limit(I0, I1, U, V, H, W, pitch, alpha, niter, err_out, 1ll << 20, nullptr, workspace,
                                      workspace_bytes, stream);
}

extern "C" int of_hs_solve_persistent_limit(const float* I0, const float* I1, float* U, float* V, int H, int W, int pitch,
                                            float alpha, int niter, double* err_out, long long wait_limit,
                                            int* schedule, void* workspace, size_t workspace_bytes, void* stream) {
  OF_REQUIRE(!bad_plane(I0, H, W, pitch) && I1 && U && V, "of_hs_solve_persistent: bad plane");
  OF_REQUIRE(niter >= 0, "of_hs_solve_persistent: niter < 0");
  if (!workspace || workspace_bytes < of_hs_workspace_size(H, W, pitch))
    return set_error(OF_ERR_WORKSPACE, "of_hs_solve_persistent: workspace too small (%zu < %zu)", workspace_bytes,
                     of_hs_workspace_size(H, W, pitch));
  OF_REQUIRE(wait_limit > 0, "of_hs_solve_persistent: wait_limit must be positive");
  cudaStream_t st = as_stream(stream);
  cudaError_t e = schedule ? cudaMemsetAsync(schedule, 0, sizeof(int), st) : cudaSuccess;
  if (e != cudaSuccess) return set_error(OF_ERR_CUDA, "of_hs_solve_persistent: %s", cudaGetErrorString(e));
  if (!hs_one_launch(H, W))
    return of_hs_solve(I0, I1, U, V, H, W, pitch, alpha, niter, err_out, workspace, workspace_bytes, stream);
  const size_t hbs = hs_halo_bytes(H, W);
  const size_t N = (size_t)H * pitch;
  Carver c(workspace, workspace_bytes);
  float* U0 = c.take<float>(2 * N);
  float* V0 = U0 + N;
  double* acc = c.take<double>(2);
  int* status = c.take<int>(1);
  const size_t bws = hs_persistent_ws(H, W, pitch);
  void* bw = c.take<unsigned char>(bws);
  void* halo = hbs ? c.take<unsigned char>(hbs) : nullptr;
  long long n = 0;
  if (err_out) {
    copy2_kernel<<<dim3((W + 255) / 256, H), 256, 0, st>>>(U, V, U0, V0, W, pitch);
    n++;
  }
  e = cudaMemsetAsync(status, 0, sizeof(int), st);
  if (e != cudaSuccess) return set_error(OF_ERR_CUDA, "of_hs_solve_persistent: %s", cudaGetErrorString(e));
  OfHsBatchPair q = {I0, I1, U, V, H, W, pitch, alpha, niter};
  OfTuning tun = {kHsSolveShape, 0, OF_HS_EXACT, OF_HS_SCHED_AUTO};
  const int rc = hs_batch(&q, 1, &tun, status, wait_limit, bw, bws, halo, stream);
  if (rc != OF_OK) return rc;
  if (schedule) {
    e = cudaMemcpyAsync(schedule, hs_batch_mode(&q, 1, bw, bws), sizeof(int), cudaMemcpyDeviceToDevice, st);
    if (e != cudaSuccess) return set_error(OF_ERR_CUDA, "of_hs_solve_persistent: %s", cudaGetErrorString(e));
  }
  if (err_out) {
    cudaMemsetAsync(acc, 0, 2 * sizeof(double), st);
    dim3 g2((W + 255) / 256 < 4 ? (W + 255) / 256 : 4, H < 256 ? H : 256);
    sqdiff2_kernel<<<g2, 256, 0, st>>>(U, U0, V, V0, H, W, pitch, acc);
    hs_err_kernel<<<1, 1, 0, st>>>(acc, (double)H * (double)W, err_out, status);
    n += 2;
  }
  return check_launch("of_hs_solve_persistent", n);
}
