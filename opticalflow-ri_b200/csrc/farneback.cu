// A12-A19 Farneback kernels (src/optical_flow_farneback.cl:72-429).
//
// Arithmetic follows the OpenCL source with its multiply-adds fused the way the CPU
// oracle fixes them (`acc += a*b` -> fmaf(a, b, acc); `a*b + c*d` -> fmaf(a, b, c*d)),
// so GPU and oracle agree bit for bit.  Planar 5-coefficient fields are 5 stacked H x W
// planes sharing one pitch.
//
// Kernels
//  - fb_blur_kernel: separable Gaussian (vertical then horizontal, reflect-101), one plane
//    per blockIdx.z; the input tile with its halo is staged in shared memory once.
//  - fb_polyexp_kernel: 7- (or 5-) tap vertical moments of the clamped neighbourhood into
//    shared memory, then the horizontal combination into the 5 coefficient planes.
//  - fb_iter_tile_kernel: one solver iteration fused — blur5 of M, updateFlow, and
//    updateMatrices into the other M buffer — so M is read once per iteration and the
//    blurred M never leaves the SM (fb_iter_kernel: the same for half windows above 16).
#include "common.cuh"
#include "tma.cuh"

namespace ofb {

constexpr int FB_MAXKH = 32;
struct FbTaps {
  float g[FB_MAXKH + 1];
};

__host__ __device__ __forceinline__ int fb_low(int y, int last) { return abs(y) % (last + 1); }
__host__ __device__ __forceinline__ int fb_high(int y, int last) { return abs(last - abs(last - y)) % (last + 1); }
// reflect-101 mapping of the gaussianBlur kernels (idx_row_low / idx_row_high / idx_col)
__device__ __forceinline__ int fb_row(int y, int rows) {
  if (y < 0) return fb_low(y, rows - 1);
  if (y > rows - 1) return fb_high(y, rows - 1);
  return y;
}
__device__ __forceinline__ int fb_col(int x, int cols) { return fb_low(fb_high(x, cols - 1), cols - 1); }

constexpr int FBB_TW = 64, FBB_TH = 16;

// Blur of plane blockIdx.z: out = H(V(src)).  smem: input (TH+2kh) x (TW+2kh), vertical
// result TH x (TW+2kh).  KHC > 0: the half width is the compile-time KHC (the Farneback
// levels' frame smoothing uses 1 and 4), so the tile widths are constants and the tap
// loops unroll; KHC = 0: kh at run time.
template <int KHC = 0>
__global__ void __launch_bounds__(256) fb_blur_kernel(const float* __restrict__ src, float* __restrict__ dst, int H,
                                                      int W, int pitch, FbTaps t, int khrt) {
  extern __shared__ float sm[];
  const int kh = KHC > 0 ? KHC : khrt;
  const int iw = FBB_TW + 2 * kh, ih = FBB_TH + 2 * kh;
  float* tin = sm;
  float* tv = sm + ih * iw;
  const size_t plane = (size_t)H * pitch * blockIdx.z;
  const float* s = src + plane;
  const int x0 = blockIdx.x * FBB_TW, y0 = blockIdx.y * FBB_TH;
  // interior tiles (halo inside the image) need no reflect-101 mapping
  const bool inside = x0 >= kh && y0 >= kh && x0 + FBB_TW + kh <= W && y0 + FBB_TH + kh <= H;
  for (int i = threadIdx.x; i < ih * iw; i += blockDim.x) {
    int ly = i / iw, lx = i - ly * iw;
    const int gy = y0 - kh + ly, gx = x0 - kh + lx;
    tin[i] = inside ? s[(size_t)gy * pitch + gx] : s[(size_t)fb_row(gy, H) * pitch + fb_col(gx, W)];
  }
  __syncthreads();
  for (int i = threadIdx.x; i < FBB_TH * iw; i += blockDim.x) {
    int ly = i / iw, lx = i - ly * iw;
    const float* c = tin + (ly + kh) * iw + lx;
    float acc = __fmul_rn(c[0], t.g[0]);
#pragma unroll
    for (int j = 1; j <= (KHC > 0 ? KHC : FB_MAXKH); j++) {
      if (KHC == 0 && j > kh) break;
      acc = __fmaf_rn(__fadd_rn(c[-j * iw], c[j * iw]), t.g[j], acc);
    }
    tv[i] = acc;
  }
  __syncthreads();
  for (int i = threadIdx.x; i < FBB_TH * FBB_TW; i += blockDim.x) {
    int ly = i / FBB_TW, lx = i - ly * FBB_TW;
    int y = y0 + ly, x = x0 + lx;
    if (y >= H || x >= W) continue;
    const float* r = tv + ly * iw + lx + kh;
    float res = __fmul_rn(r[0], t.g[0]);
#pragma unroll
    for (int j = 1; j <= (KHC > 0 ? KHC : FB_MAXKH); j++) {
      if (KHC == 0 && j > kh) break;
      res = __fmaf_rn(__fadd_rn(r[-j], r[j]), t.g[j], res);
    }
    dst[plane + (size_t)y * pitch + x] = res;
  }
}

// boxFilter5 (:350-406): clamped borders, plain sums, one plane per blockIdx.z
__global__ void __launch_bounds__(256) fb_box_kernel(const float* __restrict__ src, float* __restrict__ dst, int H,
                                                     int W, int pitch, int kh, float inv) {
  extern __shared__ float sm[];
  const int iw = FBB_TW + 2 * kh, ih = FBB_TH + 2 * kh;
  float* tin = sm;
  float* tv = sm + ih * iw;
  const size_t plane = (size_t)H * pitch * blockIdx.z;
  const float* s = src + plane;
  const int x0 = blockIdx.x * FBB_TW, y0 = blockIdx.y * FBB_TH;
  for (int i = threadIdx.x; i < ih * iw; i += blockDim.x) {
    int ly = i / iw, lx = i - ly * iw;
    tin[i] = s[(size_t)clampi(y0 - kh + ly, 0, H - 1) * pitch + clampi(x0 - kh + lx, 0, W - 1)];
  }
  __syncthreads();
  for (int i = threadIdx.x; i < FBB_TH * iw; i += blockDim.x) {
    int ly = i / iw, lx = i - ly * iw;
    const float* c = tin + (ly + kh) * iw + lx;
    float acc = c[0];
    for (int j = 1; j <= kh; j++) acc = __fadd_rn(acc, __fadd_rn(c[-j * iw], c[j * iw]));
    tv[i] = acc;
  }
  __syncthreads();
  for (int i = threadIdx.x; i < FBB_TH * FBB_TW; i += blockDim.x) {
    int ly = i / FBB_TW, lx = i - ly * FBB_TW;
    int y = y0 + ly, x = x0 + lx;
    if (y >= H || x >= W) continue;
    const float* r = tv + ly * iw + lx + kh;
    float res = r[0];
    for (int j = 1; j <= kh; j++) res = __fadd_rn(res, __fadd_rn(r[-j], r[j]));
    dst[plane + (size_t)y * pitch + x] = __fmul_rn(res, inv);
  }
}

struct FbPoly {
  float g[8], xg[8], xxg[8], ig[4];
  int n;
};

// polynomialExpansion: one CTA = 1 row segment of 256-2n outputs (the reference's
// (256,1) work-group shape), vertical moments for 256 clamped columns in smem.
constexpr int FBP_T = 256;
__global__ void __launch_bounds__(FBP_T) fb_polyexp_kernel(const float* __restrict__ src, float* __restrict__ dst,
                                                           int H, int W, int pitch, FbPoly P) {
  __shared__ float row[3][FBP_T];
  const int n = P.n;
  const int y = blockIdx.y, tx = threadIdx.x;
  const int x = blockIdx.x * (FBP_T - 2 * n) + tx - n;
  const int xw = clampi(x, 0, W - 1);
  float r0 = __fmul_rn(src[(size_t)y * pitch + xw], P.g[0]), r1 = 0.f, r2 = 0.f;
  for (int k = 1; k <= n; k++) {
    float t0 = src[(size_t)max(y - k, 0) * pitch + xw];
    float t1 = src[(size_t)min(y + k, H - 1) * pitch + xw];
    r0 = __fmaf_rn(P.g[k], __fadd_rn(t0, t1), r0);
    r1 = __fmaf_rn(P.xg[k], __fsub_rn(t1, t0), r1);
    r2 = __fmaf_rn(P.xxg[k], __fadd_rn(t0, t1), r2);
  }
  row[0][tx] = r0;
  row[1][tx] = r1;
  row[2][tx] = r2;
  __syncthreads();
  if (tx >= n && tx + n < FBP_T && x < W) {
    float b1 = __fmul_rn(P.g[0], row[0][tx]), b3 = __fmul_rn(P.g[0], row[1][tx]), b5 = __fmul_rn(P.g[0], row[2][tx]);
    float b2 = 0.f, b4 = 0.f, b6 = 0.f;
    for (int k = 1; k <= n; k++) {
      float sp = __fadd_rn(row[0][tx + k], row[0][tx - k]), sm_ = __fsub_rn(row[0][tx + k], row[0][tx - k]);
      b1 = __fmaf_rn(sp, P.g[k], b1);
      b4 = __fmaf_rn(sp, P.xxg[k], b4);
      b2 = __fmaf_rn(sm_, P.xg[k], b2);
      b3 = __fmaf_rn(__fadd_rn(row[1][tx + k], row[1][tx - k]), P.g[k], b3);
      b6 = __fmaf_rn(__fsub_rn(row[1][tx + k], row[1][tx - k]), P.xg[k], b6);
      b5 = __fmaf_rn(__fadd_rn(row[2][tx + k], row[2][tx - k]), P.g[k], b5);
    }
    const size_t pl = (size_t)H * pitch, i = (size_t)y * pitch + x;
    dst[i] = __fmul_rn(b3, P.ig[0]);
    dst[pl + i] = __fmul_rn(b2, P.ig[0]);
    dst[2 * pl + i] = __fmaf_rn(b1, P.ig[1], __fmul_rn(b5, P.ig[2]));
    dst[3 * pl + i] = __fmaf_rn(b1, P.ig[1], __fmul_rn(b4, P.ig[2]));
    dst[4 * pl + i] = __fmul_rn(b6, P.ig[3]);
  }
}

// Tiled polynomial expansion for a compile-time half width N (polyN 5 and 7, the
// reference's two settings).  The row kernel above loads 2N+1 samples per output from
// global memory; here a CTA covers FBQ_R rows x FBQ_OW columns.  Each thread walks one
// column down the tile with a register window (FBQ_R + 2N loads for FBQ_R outputs) and
// leaves the three vertical moments in shared memory; then each thread takes 8 consecutive
// outputs of one row with a register window along the row.  The arithmetic of every
// output is the row kernel's, in the same order.  The moment rows are padded by one float
// per 8 columns, so the 8-column segments of a warp's lanes fall in distinct banks.
// What bounds it: the issue slots (240 instructions per pixel, three quarters of them adds
// and multiply-adds) with few warps to hide the loads in front of them.  Moments 0 and 1 are
// stored as pairs, whose sums along the row take the same taps in packed instructions (7 for 11
// per tap), and 80 registers a thread let three CTAs share an SM.  Blurred / plain, us:
// 1024 x 1024 22.8 / 15.5 -> 19.2 / 12.6, 2048 x 2048 57.7 / 43.3 -> 47.0 / 35.0; two CTAs per
// SM 20.8 / 14.3 and 54.7 / 38.9.
//
// BLUR = true fuses the level's 3-tap frame blur in front (gaussianBlur with kh = 1 and
// reflect-101 borders, :160-253, then the expansion of the blurred frame, as at the
// pyramid's full-size level where no resize lies between them).  The CTA first computes
// the vertical blur V of its rows for the CW + 2 columns around its window into shared
// memory (the storage the moments use later), then each thread forms the blurred samples
// of its column from V and its two reflect-101 neighbours.  Every blurred value is the
// blur kernel's, operation for operation, so the result equals of_fb_blur followed by
// of_fb_polyexp.  Needs H, W >= 3.
constexpr int FBQ_OW = 240, FBQ_R = 8, FBQ_SEG = 8;
__device__ __forceinline__ int fbq_col(int c) { return c + (c >> 3); }
template <int N, bool BLUR>
__global__ void __launch_bounds__(256, 3) fb_polyexp_tile_kernel(const float* __restrict__ src, float* __restrict__ dst,
                                                              int H, int W, int pitch, FbPoly P, int vec, float bg0,
                                                              float bg1) {
  constexpr int CW = FBQ_OW + 2 * N;          // columns that get vertical moments
  constexpr int CWP = CW + (CW >> 3) + 1;     // padded row length
  constexpr int WIN = FBQ_SEG + 2 * N;
  constexpr int NR = FBQ_R + 2 * N;           // rows of the vertical window
  static_assert(CW + 2 <= 256 && NR * 256 <= 3 * FBQ_R * CWP, "blur rows must fit the moment storage");
  __shared__ __align__(16) float store[3 * FBQ_R * CWP];
  float2 (*mom01)[CWP] = reinterpret_cast<float2 (*)[CWP]>(store);           // moments 0 and 1
  float (*mom2)[CWP] = reinterpret_cast<float (*)[CWP]>(store + 2 * FBQ_R * CWP);
  const int x0 = blockIdx.x * FBQ_OW, y0 = blockIdx.y * FBQ_R, tx = threadIdx.x;
  float c[NR];
  if (BLUR) {
    // V(y, x) = g1 (src[y-1] + src[y+1]) + g0 src[y] at the window's clamped rows y, for
    // the columns clamp(x0 - N - 1 + j), j <= CW + 1
    float (*vs)[256] = reinterpret_cast<float (*)[256]>(store);
    if (tx < CW + 2) {
      const float* col = src + clampi(x0 - N - 1 + tx, 0, W - 1);
      if (y0 - N - 1 >= 0 && y0 + FBQ_R + N < H) {  // rows y0-N-1 .. y0+R+N, all inside
        float r[NR + 2];
#pragma unroll
        for (int q = 0; q < NR + 2; q++) r[q] = col[(size_t)(y0 - N - 1 + q) * pitch];
#pragma unroll
        for (int q = 0; q < NR; q++) vs[q][tx] = __fmaf_rn(__fadd_rn(r[q], r[q + 2]), bg1, __fmul_rn(r[q + 1], bg0));
      } else {
#pragma unroll
        for (int q = 0; q < NR; q++) {
          const int y = clampi(y0 - N + q, 0, H - 1);
          const float up = col[(size_t)fb_row(y - 1, H) * pitch], mid = col[(size_t)y * pitch],
                      dn = col[(size_t)fb_row(y + 1, H) * pitch];
          vs[q][tx] = __fmaf_rn(__fadd_rn(up, dn), bg1, __fmul_rn(mid, bg0));
        }
      }
    }
    __syncthreads();
    if (tx < CW) {
      // column u = x0 - N + tx, clamped to xw; V's column j holds clamp(x0 - N - 1 + j)
      const int u = x0 - N + tx;
      int jl = tx, jr = tx + 2;  // xw - 1 and xw + 1 inside the image
      if (u <= 0) jl = jr = N + 2 - x0;           // xw = 0: both reflect-101 neighbours are column 1
      else if (u >= W - 1) jl = jr = W - 1 - x0 + N;  // xw = W - 1: both are column W - 2
#pragma unroll
      for (int q = 0; q < NR; q++) c[q] = __fmaf_rn(__fadd_rn(vs[q][jl], vs[q][jr]), bg1, __fmul_rn(vs[q][tx + 1], bg0));
    }
    __syncthreads();  // V is overwritten by the moments below
  }
  if (tx < CW) {
    if (!BLUR) {
      const int xw = clampi(x0 - N + tx, 0, W - 1);
#pragma unroll
      for (int q = 0; q < NR; q++) c[q] = src[(size_t)clampi(y0 - N + q, 0, H - 1) * pitch + xw];
    }
#pragma unroll
    for (int r = 0; r < FBQ_R; r++) {
      float r0 = __fmul_rn(c[r + N], P.g[0]), r1 = 0.f, r2 = 0.f;
#pragma unroll
      for (int k = 1; k <= N; k++) {
        const float t0 = c[r + N - k], t1 = c[r + N + k];
        r0 = __fmaf_rn(P.g[k], __fadd_rn(t0, t1), r0);
        r1 = __fmaf_rn(P.xg[k], __fsub_rn(t1, t0), r1);
        r2 = __fmaf_rn(P.xxg[k], __fadd_rn(t0, t1), r2);
      }
      mom01[r][fbq_col(tx)] = make_float2(r0, r1);
      mom2[r][fbq_col(tx)] = r2;
    }
  }
  __syncthreads();
  constexpr int NSEG = FBQ_OW / FBQ_SEG;
  const int r = tx / NSEG, sg = tx - r * NSEG;
  const int y = y0 + r, xs = x0 + sg * FBQ_SEG;
  const bool act = tx < FBQ_R * NSEG && y < H && xs < W;
  const size_t pl = (size_t)H * pitch;
  float o[5][FBQ_SEG];
  if (act) {
    // output column xs + i is moment column sg*8 + i + N; its window is sg*8 .. sg*8 + 7 + 2N
    float2 a01[WIN];
    float a2[WIN];
#pragma unroll
    for (int q = 0; q < WIN; q++) {
      const int cc = sg * (FBQ_SEG + 1) + q + (q >> 3);  // fbq_col(sg * 8 + q)
      a01[q] = mom01[r][cc];
      a2[q] = mom2[r][cc];
    }
#pragma unroll
    for (int i = 0; i < FBQ_SEG; i++) {
      const int t = i + N;
      float2 b13 = __fmul2_rn(make_float2(P.g[0], P.g[0]), a01[t]), b26 = make_float2(0.f, 0.f);
      float b5 = __fmul_rn(P.g[0], a2[t]), b4 = 0.f;
#pragma unroll
      for (int k = 1; k <= N; k++) {
        // sums and differences of moments 0 and 1; the product with -1 is exact
        const float2 sp = __fadd2_rn(a01[t + k], a01[t - k]);
        const float2 sm = __ffma2_rn(a01[t - k], make_float2(-1.f, -1.f), a01[t + k]);
        b13 = __ffma2_rn(sp, make_float2(P.g[k], P.g[k]), b13);
        b26 = __ffma2_rn(sm, make_float2(P.xg[k], P.xg[k]), b26);
        b4 = __fmaf_rn(sp.x, P.xxg[k], b4);
        b5 = __fmaf_rn(__fadd_rn(a2[t + k], a2[t - k]), P.g[k], b5);
      }
      o[0][i] = __fmul_rn(b13.y, P.ig[0]);
      o[1][i] = __fmul_rn(b26.x, P.ig[0]);
      o[2][i] = __fmaf_rn(b13.x, P.ig[1], __fmul_rn(b5, P.ig[2]));
      o[3][i] = __fmaf_rn(b13.x, P.ig[1], __fmul_rn(b4, P.ig[2]));
      o[4][i] = __fmul_rn(b26.y, P.ig[3]);
    }
  }
  if (vec) {  // 16-byte aligned rows
    if (!act) return;
    const size_t i0 = (size_t)y * pitch + xs;
    if (xs + FBQ_SEG <= W) {
#pragma unroll
      for (int p = 0; p < 5; p++) {
        float4* d = reinterpret_cast<float4*>(dst + p * pl + i0);
        d[0] = make_float4(o[p][0], o[p][1], o[p][2], o[p][3]);
        d[1] = make_float4(o[p][4], o[p][5], o[p][6], o[p][7]);
      }
    } else {
#pragma unroll
      for (int i = 0; i < FBQ_SEG; i++)
        if (xs + i < W) {
#pragma unroll
          for (int p = 0; p < 5; p++) dst[p * pl + i0 + i] = o[p][i];
        }
    }
    return;
  }
  // Any other rows: through shared memory, so that a warp stores consecutive words (8 apart they
  // cost a sector each: 719 x 1013, blurred, 31.0 us against 18.7).
  static_assert(3 * FBQ_R * FBQ_OW <= 3 * FBQ_R * CWP, "three planes of the tile fit");
#pragma unroll
  for (int p0 = 0; p0 < 5; p0 += 3) {
    __syncthreads();
    if (act) {
#pragma unroll
      for (int p = p0; p < p0 + 3 && p < 5; p++) {
        float4* d = reinterpret_cast<float4*>(store + ((p - p0) * FBQ_R + r) * FBQ_OW + sg * FBQ_SEG);
        d[0] = make_float4(o[p][0], o[p][1], o[p][2], o[p][3]);
        d[1] = make_float4(o[p][4], o[p][5], o[p][6], o[p][7]);
      }
    }
    __syncthreads();
    if (tx < FBQ_OW && x0 + tx < W) {
#pragma unroll
      for (int p = p0; p < p0 + 3 && p < 5; p++)
#pragma unroll
        for (int rr = 0; rr < FBQ_R; rr++)
          if (y0 + rr < H)
            dst[p * pl + (size_t)(y0 + rr) * pitch + x0 + tx] = store[((p - p0) * FBQ_R + rr) * FBQ_OW + tx];
    }
  }
}

__constant__ float c_border[6] = {0.14f, 0.14f, 0.4472f, 0.4472f, 0.4472f, 1.f};

// Element offset of a pixel in a plane.  Off unsigned (planes of less than 2^30 elements,
// fb_off32): a plane base that is the same for every thread plus a 32-bit index costs one
// instruction per address; size_t for larger planes.
template <class Off>
__device__ __forceinline__ Off fb_off(int y, int x, int pitch) {
  return (Off)y * (Off)pitch + (Off)x;
}
inline bool fb_off32(int H, int pitch) { return (long long)H * pitch < (1ll << 30); }

// updateMatrices (:256-348) for one pixel in two steps, so that a thread with several pixels
// has all their loads in flight before the first result is needed: fb_mat_load reads the
// pixel's R0 and the four R1 samples at its displaced position, fb_mat_store forms and writes
// the 5 M planes.  off: the pixel's offset in a plane; BORDER: the pixel may lie within 5
// pixels of the image border, where the M planes are scaled down (elsewhere the factor is 1).
struct FbMat {
  float dx, dy, fx, fy;
  float r0[5], r1[5][4];
  bool inside;  // the four samples lie in the image
};

template <class Off>
__device__ __forceinline__ void fb_mat_load(FbMat& m, int y, int x, Off off, float dx, float dy,
                                            const float* __restrict__ R0, const float* __restrict__ R1, int H, int W,
                                            int pitch) {
  const size_t pl = (size_t)H * pitch;
  const float fx = __fadd_rn((float)x, dx), fy = __fadd_rn((float)y, dy);
  const int x1 = __float2int_rd(fx), y1 = __float2int_rd(fy);
  m.fx = __fsub_rn(fx, (float)x1);
  m.fy = __fsub_rn(fy, (float)y1);
  m.dx = dx;
  m.dy = dy;
  m.inside = (unsigned)x1 < (unsigned)(W - 1) && (unsigned)y1 < (unsigned)(H - 1);
  const Off q = m.inside ? fb_off<Off>(y1, x1, pitch) : 0;
#pragma unroll
  for (int p = 0; p < 5; p++) {
    m.r0[p] = (R0 + p * pl)[off];
    m.r1[p][0] = m.inside ? (R1 + p * pl)[q] : 0.f;
    m.r1[p][1] = m.inside ? (R1 + p * pl + 1)[q] : 0.f;
    m.r1[p][2] = m.inside ? (R1 + p * pl + pitch)[q] : 0.f;
    m.r1[p][3] = m.inside ? (R1 + p * pl + pitch + 1)[q] : 0.f;
  }
}

template <bool BORDER, class Off>
__device__ __forceinline__ void fb_mat_store(const FbMat& m, int y, int x, Off off, float* __restrict__ M, int H,
                                             int W, int pitch) {
  const size_t pl = (size_t)H * pitch;
  const float ofx = __fsub_rn(1.f, m.fx), ofy = __fsub_rn(1.f, m.fy);
  const float a00 = __fmul_rn(ofx, ofy), a01 = __fmul_rn(m.fx, ofy), a10 = __fmul_rn(ofx, m.fy),
              a11 = __fmul_rn(m.fx, m.fy);
  float rr[5];
#pragma unroll
  for (int p = 0; p < 5; p++) {
    float tt = __fmaf_rn(a00, m.r1[p][0], __fmul_rn(a01, m.r1[p][1]));
    tt = __fmaf_rn(a10, m.r1[p][2], tt);
    rr[p] = __fmaf_rn(a11, m.r1[p][3], tt);
  }
  float r2 = m.inside ? rr[0] : 0.f, r3 = m.inside ? rr[1] : 0.f;
  float r4 = m.inside ? __fmul_rn(__fadd_rn(m.r0[2], rr[2]), 0.5f) : m.r0[2];
  float r5 = m.inside ? __fmul_rn(__fadd_rn(m.r0[3], rr[3]), 0.5f) : m.r0[3];
  float r6 = m.inside ? __fmul_rn(__fadd_rn(m.r0[4], rr[4]), 0.25f) : __fmul_rn(m.r0[4], 0.5f);
  r2 = __fmul_rn(__fsub_rn(m.r0[0], r2), 0.5f);
  r3 = __fmul_rn(__fsub_rn(m.r0[1], r3), 0.5f);
  r2 = __fadd_rn(r2, __fmaf_rn(r4, m.dy, __fmul_rn(r6, m.dx)));
  r3 = __fadd_rn(r3, __fmaf_rn(r6, m.dy, __fmul_rn(r5, m.dx)));
  if (BORDER) {
    float scale = __fmul_rn(c_border[min(x, 5)], c_border[min(y, 5)]);
    scale = __fmul_rn(scale, c_border[min(W - x - 1, 5)]);
    scale = __fmul_rn(scale, c_border[min(H - y - 1, 5)]);
    r2 = __fmul_rn(r2, scale);
    r3 = __fmul_rn(r3, scale);
    r4 = __fmul_rn(r4, scale);
    r5 = __fmul_rn(r5, scale);
    r6 = __fmul_rn(r6, scale);
  }
  M[off] = __fmaf_rn(r4, r4, __fmul_rn(r6, r6));
  (M + pl)[off] = __fmul_rn(__fadd_rn(r4, r5), r6);
  (M + 2 * pl)[off] = __fmaf_rn(r5, r5, __fmul_rn(r6, r6));
  (M + 3 * pl)[off] = __fmaf_rn(r4, r2, __fmul_rn(r6, r3));
  (M + 4 * pl)[off] = __fmaf_rn(r6, r2, __fmul_rn(r5, r3));
}

template <class Off>
__device__ __forceinline__ void fb_matrices_at(int y, int x, float dx, float dy, const float* __restrict__ R0,
                                               const float* __restrict__ R1, float* __restrict__ M, int H, int W,
                                               int pitch) {
  FbMat m;
  const Off off = fb_off<Off>(y, x, pitch);
  fb_mat_load(m, y, x, off, dx, dy, R0, R1, H, W, pitch);
  fb_mat_store<true>(m, y, x, off, M, H, W, pitch);
}

__device__ __forceinline__ void fb_flow_from(float g11, float g12, float g22, float h1, float h2, float* fx,
                                             float* fy) {
  float detInv = __frcp_rn(__fadd_rn(__fmaf_rn(g11, g22, -__fmul_rn(g12, g12)), 1e-3f));
  *fx = __fmul_rn(__fmaf_rn(g11, h2, -__fmul_rn(g12, h1)), detInv);
  *fy = __fmul_rn(__fmaf_rn(g22, h1, -__fmul_rn(g12, h2)), detInv);
}

template <class Off>
__global__ void fb_update_matrices_kernel(const float* __restrict__ flowx, const float* __restrict__ flowy,
                                          const float* __restrict__ R0, const float* __restrict__ R1,
                                          float* __restrict__ M, int H, int W, int pitch) {
  int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
  if (x >= W || y >= H) return;
  size_t i = (size_t)y * pitch + x;
  fb_matrices_at<Off>(y, x, flowx[i], flowy[i], R0, R1, M, H, W, pitch);
}

__global__ void fb_update_flow_kernel(const float* __restrict__ M, float* __restrict__ flowx, float* __restrict__ flowy,
                                      int H, int W, int pitch) {
  int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
  if (x >= W || y >= H) return;
  const size_t pl = (size_t)H * pitch, i = (size_t)y * pitch + x;
  float fx, fy;
  fb_flow_from(M[i], M[pl + i], M[2 * pl + i], M[3 * pl + i], M[4 * pl + i], &fx, &fy);
  flowx[i] = fx;
  flowy[i] = fy;
}

// Fused iteration.  CTA tile: FBI_TW x FBI_TH outputs, all 5 planes.  Per plane the input
// tile (+kh halo) is staged, blurred vertically into tv, horizontally into registers; the
// 5 blurred values of each output pixel then feed updateFlow and updateMatrices.
constexpr int FBI_TW = 32, FBI_TH = 16;
__global__ void __launch_bounds__(256) fb_iter_kernel(const float* __restrict__ Min, float* __restrict__ Mout,
                                                      const float* __restrict__ R0, const float* __restrict__ R1,
                                                      float* __restrict__ flowx, float* __restrict__ flowy, int H,
                                                      int W, int pitch, FbTaps t, int kh, int upd) {
  extern __shared__ float sm[];
  const int iw = FBI_TW + 2 * kh, ih = FBI_TH + 2 * kh;
  float* tin = sm;
  float* tv = sm + ih * iw;
  const size_t pl = (size_t)H * pitch;
  const int x0 = blockIdx.x * FBI_TW, y0 = blockIdx.y * FBI_TH;
  // each thread owns 2 output pixels of the 32x16 tile
  float res[2][5];
#pragma unroll
  for (int p = 0; p < 5; p++) {
    const float* s = Min + p * pl;
    for (int i = threadIdx.x; i < ih * iw; i += blockDim.x) {
      int ly = i / iw, lx = i - ly * iw;
      tin[i] = s[(size_t)fb_row(y0 - kh + ly, H) * pitch + fb_col(x0 - kh + lx, W)];
    }
    __syncthreads();
    for (int i = threadIdx.x; i < FBI_TH * iw; i += blockDim.x) {
      int ly = i / iw, lx = i - ly * iw;
      const float* c = tin + (ly + kh) * iw + lx;
      float acc = __fmul_rn(c[0], t.g[0]);
      for (int j = 1; j <= kh; j++) acc = __fmaf_rn(__fadd_rn(c[-j * iw], c[j * iw]), t.g[j], acc);
      tv[i] = acc;
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 2; q++) {
      int o = threadIdx.x + q * 256;
      int ly = o / FBI_TW, lx = o - ly * FBI_TW;
      const float* r = tv + ly * iw + lx + kh;
      float v = __fmul_rn(r[0], t.g[0]);
      for (int j = 1; j <= kh; j++) v = __fmaf_rn(__fadd_rn(r[-j], r[j]), t.g[j], v);
      res[q][p] = v;
    }
    __syncthreads();
  }
#pragma unroll
  for (int q = 0; q < 2; q++) {
    int o = threadIdx.x + q * 256;
    int ly = o / FBI_TW, lx = o - ly * FBI_TW;
    int y = y0 + ly, x = x0 + lx;
    if (y >= H || x >= W) continue;
    float fx, fy;
    fb_flow_from(res[q][0], res[q][1], res[q][2], res[q][3], res[q][4], &fx, &fy);
    size_t i = (size_t)y * pitch + x;
    flowx[i] = fx;
    flowy[i] = fy;
    if (upd) fb_matrices_at<size_t>(y, x, fx, fy, R0, R1, Mout, H, W, pitch);
  }
}

// Fused iteration for half windows up to 16 (FULL: exactly 16, the default windowSize 33).
// CTA: 64 x 32 outputs, 256 threads.  The 5 planes' 96 x 64 input tiles arrive one after
// another in two stages, so plane p+1 is in flight while plane p is blurred: by TMA (a 3-D map
// over the 5 stacked planes) for tiles inside the image when the strides allow it, else by
// 4-byte asynchronous copies that map the reflect-101 border (and any pitch) on the way.
// The taps run as packed f32x2 operations: the vertical pass takes two columns and 8 rows per
// thread, the horizontal pass two rows and 8 columns (its input, the vertical result, is kept
// as row pairs), each output's taps in the reference's order.  The blurred planes go to shared
// memory, and the epilogue (updateFlow, updateMatrices) runs one pixel per lane, two pixels'
// loads in flight, so its accesses and the R1 gathers fall on neighbouring addresses.
//
// What bounds it: per tile alone, 5 x 2150 cycles of the two passes (shared-memory reads and
// FMA pipe in turn) and 7000 of gather latency in the epilogue; two CTAs per SM overlap them.
// One iteration, windowSize 33: 512 x 512 29.5 -> 18.2 us, 1024 x 1024 64 -> 47 us, 2048 x 2048
// 160 -> 140 us against one scalar output per operation with a border fix-up pass; 1013 x 719
// (no TMA strides) 142 -> 40 us and windowSize 21 99 -> 36 us against the run-time-window kernel
// (fb_iter_kernel, kept for half windows above 16, images of at most 16 pixels a side and
// planes of 4 GB or more).  Tried: vertical and horizontal pass at once in different warps
// (no faster), a third stage (no faster), four pixels' loads in flight (spills, slower).
constexpr int FBK_KH = 16, FBK_TW = 64, FBK_TH = 32, FBK_R = 8;
constexpr int FBK_IW = FBK_TW + 2 * FBK_KH, FBK_IH = FBK_TH + 2 * FBK_KH;  // staged tile: 96 x 64
constexpr int FBK_STAGE = FBK_IW * FBK_IH;                                 // floats
constexpr int FBK_VITEMS = (FBK_IW / 2) * (FBK_TH / FBK_R), FBK_HITEMS = (FBK_TW / 8) * (FBK_TH / 2);
static_assert(FBK_VITEMS <= 256 && FBK_HITEMS <= 256, "one item per thread");
// Vertical result: 16-byte units of two columns of a row pair, (r, c), (r + 1, c), (r, c + 1),
// (r + 1, c + 1).  A thread of the horizontal pass reads every fourth unit's neighbours, so the
// units of a row pair are kept by u % 4, 18 units (2 banks of 16 bytes mod 8) apart: neither
// pass conflicts.
constexpr int FBK_CLS = 18, FBK_TVP = 3 * FBK_CLS + FBK_IW / 8;  // units per class, per row pair
static_assert(FBK_IW / 8 <= FBK_CLS && FBK_CLS % 8 == 2, "classes in distinct banks");
constexpr int FBK_TV = (FBK_TH / 2) * FBK_TVP * 4;               // floats
constexpr int FBK_RS = FBK_TH * FBK_TW;                          // floats of a blurred plane
constexpr size_t FBK_SMEM = (2 * (size_t)FBK_STAGE + FBK_TV + 5 * FBK_RS) * 4 + 128 + 128;
static_assert((FBK_STAGE * 4) % 128 == 0, "TMA destinations");
constexpr long long FBK_WAIT_LIMIT = 1ll << 22;
constexpr int FBK_NP = 2;  // pixels of a thread whose loads are in flight at once
static_assert(FBK_TH % (FBK_NP * (256 / FBK_TW)) == 0, "whole epilogue rounds");

struct FbTaps2 {
  float2 g[FBK_KH + 1];  // each tap twice, for the packed operations
};

// Reflect-101 position for the tile copies of an image of n > KH pixels: one reflection covers
// every position that an output reads (-KH .. n - 1 + KH); those beyond are only kept in range.
// (fb_row's general form costs two integer divisions.)
__device__ __forceinline__ int fbk_reflect(int i, int n) {
  i = abs(i);
  i = i >= n ? 2 * (n - 1) - i : i;
  return max(i, 0);
}

// Plane tile (x0 - KH, y0 - KH) into `dst` by asynchronous 4-byte copies, reflect-101 mapped:
// threads 0 .. 191 take a column (col: its address in row 0) and every second row each.
__device__ __forceinline__ void fbk_copy(float* dst, const float* __restrict__ col, int y0, int H, int pitch) {
  const int t = threadIdx.x;
  if (t < 2 * FBK_IW) {
    const int c = t % FBK_IW, r0 = t / FBK_IW, gy0 = y0 - FBK_KH + r0;
    const uint32_t d = smem_u32(dst + r0 * FBK_IW + c);
#pragma unroll 8
    for (int r = 0; r < FBK_IH; r += 2)
      asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d + r * FBK_IW * 4),
                   "l"(col + (size_t)fbk_reflect(gy0 + r, H) * pitch)
                   : "memory");
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
}

// updateFlow and (upd) updateMatrices of a tile from its blurred planes; ok false (a tile copy
// never arrived): the tile's flow is reported as NaN.
template <bool BORDER>
__device__ __forceinline__ void fbk_epilogue(const float* rs, bool ok, int x0, int y0, float* __restrict__ Mout,
                                             const float* __restrict__ R0, const float* __restrict__ R1,
                                             float* __restrict__ flowx, float* __restrict__ flowy, int H, int W,
                                             int pitch, int upd) {
  constexpr int STEP = 256 / FBK_TW;  // rows between a thread's pixels
  const int lx = threadIdx.x % FBK_TW, x = x0 + lx;
#pragma unroll 1
  for (int ly = threadIdx.x / FBK_TW; ly < FBK_TH; ly += FBK_NP * STEP) {
    FbMat m[FBK_NP];
    float fx[FBK_NP], fy[FBK_NP];
#pragma unroll
    for (int k = 0; k < FBK_NP; k++) {
      const int yl = ly + k * STEP, y = y0 + yl;
      const float* q = rs + yl * FBK_TW + lx;
      fb_flow_from(q[0], q[FBK_RS], q[2 * FBK_RS], q[3 * FBK_RS], q[4 * FBK_RS], &fx[k], &fy[k]);
      if (!ok) fx[k] = fy[k] = __int_as_float(0x7fc00000);
      if ((!BORDER || (y < H && x < W)) && upd && ok)
        fb_mat_load(m[k], y, x, fb_off<unsigned>(y, x, pitch), fx[k], fy[k], R0, R1, H, W, pitch);
    }
#pragma unroll
    for (int k = 0; k < FBK_NP; k++) {
      const int y = y0 + ly + k * STEP;
      if (BORDER && (y >= H || x >= W)) continue;
      const unsigned off = fb_off<unsigned>(y, x, pitch);
      flowx[off] = fx[k];
      flowy[off] = fy[k];
      if (upd && ok) fb_mat_store<BORDER>(m[k], y, x, off, Mout, H, W, pitch);
    }
  }
}

template <bool FULL>
__global__ void __launch_bounds__(256, 2) fb_iter_tile_kernel(const __grid_constant__ CUtensorMap tm_m, int use_tma,
                                                              const float* __restrict__ Min, float* __restrict__ Mout,
                                                              const float* __restrict__ R0,
                                                              const float* __restrict__ R1, float* __restrict__ flowx,
                                                              float* __restrict__ flowy, int H, int W, int pitch,
                                                              const __grid_constant__ FbTaps2 t, int kh, int upd) {
  constexpr int KH = FBK_KH, IW = FBK_IW;
  extern __shared__ __align__(128) unsigned char fbk_raw[];
  unsigned char* base = fbk_raw + ((128 - (smem_u32(fbk_raw) & 127)) & 127);
  float* const stage = reinterpret_cast<float*>(base);
  float4* const tv = reinterpret_cast<float4*>(stage + 2 * FBK_STAGE);
  float* const rs = stage + 2 * FBK_STAGE + FBK_TV;  // blurred planes, [5][FBK_TH][FBK_TW]
  uint64_t* const bar = reinterpret_cast<uint64_t*>(rs + 5 * FBK_RS);
  const int tid = threadIdx.x, x0 = blockIdx.x * FBK_TW, y0 = blockIdx.y * FBK_TH;
  const size_t pl = (size_t)H * pitch;
  const bool tma = use_tma && x0 >= KH && y0 >= KH && x0 + FBK_TW + KH <= W && y0 + FBK_TH + KH <= H;
  if (tma && tid == 0) {
    mbar_init(&bar[0], 1);
    mbar_init(&bar[1], 1);
  }
  if (tma) __syncthreads();
  const float* const col = Min + fbk_reflect(x0 - KH + tid % IW, W);
  auto load = [&](int p) {  // plane p into its stage, asynchronously
    float* dst = stage + (p & 1) * FBK_STAGE;
    if (!tma) {
      fbk_copy(dst, col + p * pl, y0, H, pitch);
    } else if (tid == 0) {
      mbar_expect_tx(&bar[p & 1], FBK_STAGE * 4);
      tma_load_3d(dst, &tm_m, x0 - KH, y0 - KH, p, &bar[p & 1]);
    }
  };
  load(0);
  load(1);
  bool ok = true;
#pragma unroll 1
  for (int p = 0; p < 5; p++) {
    const float* tin = stage + (p & 1) * FBK_STAGE;
    if (tma) {
      if (ok && !mbar_wait(&bar[p & 1], (p >> 1) & 1, FBK_WAIT_LIMIT)) ok = false;
    } else {
      if (p < 4)
        asm volatile("cp.async.wait_group 1;" ::: "memory");
      else
        asm volatile("cp.async.wait_group 0;" ::: "memory");
      __syncthreads();
    }
    if (tid < FBK_VITEMS) {  // vertical: two columns, 8 rows
      const int u = tid % (IW / 2), r0 = (tid / (IW / 2)) * FBK_R;
      float2 c[FBK_R + 2 * KH];
      constexpr int MID = (FBK_R + 2 * KH) / 2;
#pragma unroll
      for (int q = 0; q < MID; q++) {  // from the centre out, as the taps need them
        c[MID + q] = *reinterpret_cast<const float2*>(tin + (r0 + MID + q) * IW + 2 * u);
        c[MID - 1 - q] = *reinterpret_cast<const float2*>(tin + (r0 + MID - 1 - q) * IW + 2 * u);
      }
      float2 acc[FBK_R];  // taps outside, rows inside: 8 independent chains per tap
#pragma unroll
      for (int r = 0; r < FBK_R; r++) acc[r] = __fmul2_rn(c[r + KH], t.g[0]);
#pragma unroll
      for (int j = 1; j <= KH; j++) {
        if (!FULL && j > kh) break;
        const float2 gj = t.g[j];
#pragma unroll
        for (int r = 0; r < FBK_R; r++) acc[r] = __ffma2_rn(__fadd2_rn(c[r + KH - j], c[r + KH + j]), gj, acc[r]);
      }
      float4* d = tv + (r0 / 2) * FBK_TVP + (u >> 2) + (u & 3) * FBK_CLS;
#pragma unroll
      for (int r = 0; r < FBK_R; r += 2)
        d[(r / 2) * FBK_TVP] = make_float4(acc[r].x, acc[r + 1].x, acc[r].y, acc[r + 1].y);
    }
    __syncthreads();
    if (p + 2 < 5 && ok) load(p + 2);  // the stage is free again
    if (tid < FBK_HITEMS) {  // horizontal: a row pair, 8 columns
      const int g = tid & 7, rp = tid >> 3;
      const float4* v = tv + rp * FBK_TVP + g;
      float2 c[8 + 2 * KH];
      constexpr int MID = (4 + KH) / 2;
      auto get = [&](int k) {  // unit 4 g + k
        const float4 q = v[(k >> 2) + (k & 3) * FBK_CLS];
        c[2 * k] = make_float2(q.x, q.y);
        c[2 * k + 1] = make_float2(q.z, q.w);
      };
#pragma unroll
      for (int k = 0; k < MID; k++) {
        get(MID + k);
        get(MID - 1 - k);
      }
      float2 o[8];
#pragma unroll
      for (int i = 0; i < 8; i++) o[i] = __fmul2_rn(c[i + KH], t.g[0]);
#pragma unroll
      for (int j = 1; j <= KH; j++) {
        if (!FULL && j > kh) break;
        const float2 gj = t.g[j];
#pragma unroll
        for (int i = 0; i < 8; i++) o[i] = __ffma2_rn(__fadd2_rn(c[i + KH - j], c[i + KH + j]), gj, o[i]);
      }
      float4* d = reinterpret_cast<float4*>(rs + p * FBK_RS + 2 * rp * FBK_TW + 8 * g);
      d[0] = make_float4(o[0].x, o[1].x, o[2].x, o[3].x);
      d[1] = make_float4(o[4].x, o[5].x, o[6].x, o[7].x);
      d[FBK_TW / 4] = make_float4(o[0].y, o[1].y, o[2].y, o[3].y);
      d[FBK_TW / 4 + 1] = make_float4(o[4].y, o[5].y, o[6].y, o[7].y);
    }
    __syncthreads();
  }
  // a tile at least 5 pixels from the image border needs neither bounds nor border factors
  if (x0 >= 5 && y0 >= 5 && x0 + FBK_TW + 5 <= W && y0 + FBK_TH + 5 <= H)
    fbk_epilogue<false>(rs, ok, x0, y0, Mout, R0, R1, flowx, flowy, H, W, pitch, upd);
  else
    fbk_epilogue<true>(rs, ok, x0, y0, Mout, R0, R1, flowx, flowy, H, W, pitch, upd);
}

static FbTaps make_taps(const float* gk, int kh) {
  FbTaps t{};
  for (int j = 0; j <= kh; j++) t.g[j] = gk[j];
  return t;
}

}  // namespace ofb

using namespace ofb;

extern "C" int of_fb_blur(const float* src, float* dst, int H, int W, int pitch, int planes, const float* gk, int kh,
                          void* stream) {
  OF_REQUIRE(!bad_plane(src, H, W, pitch) && dst && src != dst, "of_fb_blur: bad plane");
  OF_REQUIRE(gk && kh >= 0 && kh <= FB_MAXKH && planes >= 1 && planes <= 65535, "of_fb_blur: bad kernel");
  size_t smem = sizeof(float) * ((size_t)(FBB_TH + 2 * kh) * (FBB_TW + 2 * kh) + (size_t)FBB_TH * (FBB_TW + 2 * kh));
  if (smem > 48 * 1024) {
    cudaError_t e = OF_SMEM_OPT_IN(fb_blur_kernel<0>, 64 * 1024);
    if (e != cudaSuccess) return set_error(OF_ERR_CUDA, "of_fb_blur: %s", cudaGetErrorString(e));
  }
  dim3 grid((W + FBB_TW - 1) / FBB_TW, (H + FBB_TH - 1) / FBB_TH, planes);
  const FbTaps tp = make_taps(gk, kh);
  if (kh == 1)
    fb_blur_kernel<1><<<grid, 256, smem, as_stream(stream)>>>(src, dst, H, W, pitch, tp, kh);
  else if (kh == 4)
    fb_blur_kernel<4><<<grid, 256, smem, as_stream(stream)>>>(src, dst, H, W, pitch, tp, kh);
  else
    fb_blur_kernel<0><<<grid, 256, smem, as_stream(stream)>>>(src, dst, H, W, pitch, tp, kh);
  return check_launch("of_fb_blur");
}

extern "C" int of_fb_box5(const float* src, float* dst, int H, int W, int pitch, int kh, void* stream) {
  OF_REQUIRE(!bad_plane(src, H, W, pitch) && dst && src != dst, "of_fb_box5: bad plane");
  OF_REQUIRE(kh >= 0 && kh <= FB_MAXKH, "of_fb_box5: bad kernel");
  size_t smem = sizeof(float) * ((size_t)(FBB_TH + 2 * kh) * (FBB_TW + 2 * kh) + (size_t)FBB_TH * (FBB_TW + 2 * kh));
  if (smem > 48 * 1024) {
    cudaError_t e = OF_SMEM_OPT_IN(fb_box_kernel, 64 * 1024);
    if (e != cudaSuccess) return set_error(OF_ERR_CUDA, "of_fb_box5: %s", cudaGetErrorString(e));
  }
  dim3 grid((W + FBB_TW - 1) / FBB_TW, (H + FBB_TH - 1) / FBB_TH, 5);
  float inv = 1.f / (float)((1 + 2 * kh) * (1 + 2 * kh));
  fb_box_kernel<<<grid, 256, smem, as_stream(stream)>>>(src, dst, H, W, pitch, kh, inv);
  return check_launch("of_fb_box5");
}

extern "C" int of_fb_polyexp(const float* src, float* dst, int H, int W, int pitch, const of_fb_poly_consts* c,
                             void* stream) {
  OF_REQUIRE(!bad_plane(src, H, W, pitch) && dst && c, "of_fb_polyexp: bad plane");
  OF_REQUIRE(c->polyN >= 1 && c->polyN <= 7, "of_fb_polyexp: polyN must be in 1..7");
  FbPoly P{};
  P.n = c->polyN;
  for (int k = 0; k <= P.n; k++) {
    P.g[k] = c->g[k];
    P.xg[k] = c->xg[k];
    P.xxg[k] = c->xxg[k];
  }
  for (int k = 0; k < 4; k++) P.ig[k] = c->ig[k];
  if (P.n == 5 || P.n == 7) {  // the reference's polyN settings: the tiled kernel
    const int vec = (pitch % 4) == 0 && (reinterpret_cast<uintptr_t>(dst) & 15) == 0;
    dim3 grid((W + FBQ_OW - 1) / FBQ_OW, (H + FBQ_R - 1) / FBQ_R);
    if (P.n == 7)
      fb_polyexp_tile_kernel<7, false><<<grid, 256, 0, as_stream(stream)>>>(src, dst, H, W, pitch, P, vec, 0.f, 0.f);
    else
      fb_polyexp_tile_kernel<5, false><<<grid, 256, 0, as_stream(stream)>>>(src, dst, H, W, pitch, P, vec, 0.f, 0.f);
    return check_launch("of_fb_polyexp");
  }
  dim3 grid((W + (FBP_T - 2 * P.n) - 1) / (FBP_T - 2 * P.n), H);
  fb_polyexp_kernel<<<grid, FBP_T, 0, as_stream(stream)>>>(src, dst, H, W, pitch, P);
  return check_launch("of_fb_polyexp");
}

extern "C" int of_fb_polyexp_blurred(const float* src, float* dst, int H, int W, int pitch, const float* gk,
                                     const of_fb_poly_consts* c, void* stream) {
  OF_REQUIRE(!bad_plane(src, H, W, pitch) && dst && c && gk, "of_fb_polyexp_blurred: bad plane");
  OF_REQUIRE(c->polyN == 5 || c->polyN == 7, "of_fb_polyexp_blurred: polyN must be 5 or 7");
  OF_REQUIRE(H >= 3 && W >= 3, "of_fb_polyexp_blurred: the frame must be at least 3 x 3");
  FbPoly P{};
  P.n = c->polyN;
  for (int k = 0; k <= P.n; k++) {
    P.g[k] = c->g[k];
    P.xg[k] = c->xg[k];
    P.xxg[k] = c->xxg[k];
  }
  for (int k = 0; k < 4; k++) P.ig[k] = c->ig[k];
  const int vec = (pitch % 4) == 0 && (reinterpret_cast<uintptr_t>(dst) & 15) == 0;
  dim3 grid((W + FBQ_OW - 1) / FBQ_OW, (H + FBQ_R - 1) / FBQ_R);
  if (P.n == 7)
    fb_polyexp_tile_kernel<7, true><<<grid, 256, 0, as_stream(stream)>>>(src, dst, H, W, pitch, P, vec, gk[0], gk[1]);
  else
    fb_polyexp_tile_kernel<5, true><<<grid, 256, 0, as_stream(stream)>>>(src, dst, H, W, pitch, P, vec, gk[0], gk[1]);
  return check_launch("of_fb_polyexp_blurred");
}

extern "C" int of_fb_update_matrices(const float* flowx, const float* flowy, const float* R0, const float* R1, float* M,
                                     int H, int W, int pitch, void* stream) {
  OF_REQUIRE(!bad_plane(flowx, H, W, pitch) && flowy && R0 && R1 && M, "of_fb_update_matrices: bad plane");
  dim3 blk(32, 8), grd((W + 31) / 32, (H + 7) / 8);
  if (fb_off32(H, pitch))
    fb_update_matrices_kernel<unsigned><<<grd, blk, 0, as_stream(stream)>>>(flowx, flowy, R0, R1, M, H, W, pitch);
  else
    fb_update_matrices_kernel<size_t><<<grd, blk, 0, as_stream(stream)>>>(flowx, flowy, R0, R1, M, H, W, pitch);
  return check_launch("of_fb_update_matrices");
}

extern "C" int of_fb_update_flow(const float* M, float* flowx, float* flowy, int H, int W, int pitch, void* stream) {
  OF_REQUIRE(!bad_plane(M, H, W, pitch) && flowx && flowy, "of_fb_update_flow: bad plane");
  dim3 blk(32, 8), grd((W + 31) / 32, (H + 7) / 8);
  fb_update_flow_kernel<<<grd, blk, 0, as_stream(stream)>>>(M, flowx, flowy, H, W, pitch);
  return check_launch("of_fb_update_flow");
}

extern "C" int of_fb_iteration(const float* M_in, float* M_out, const float* R0, const float* R1, float* flowx,
                               float* flowy, int H, int W, int pitch, const float* wk, int kh, int update_matrices,
                               void* stream) {
  OF_REQUIRE(!bad_plane(M_in, H, W, pitch) && R0 && R1 && flowx && flowy, "of_fb_iteration: bad plane");
  OF_REQUIRE(!update_matrices || (M_out && M_out != M_in), "of_fb_iteration: M_out missing or aliases M_in");
  OF_REQUIRE(wk && kh >= 0 && kh <= FB_MAXKH, "of_fb_iteration: bad kernel");
  // half windows up to 16 (the reference's default windowSize 33): the tiled, packed kernel, for
  // images with a single reflect-101 border (at 1013 x 719: 40 us against the general kernel's
  // 142 with windowSize 33, 36 against 99 with 21)
  if (kh <= FBK_KH && H > FBK_KH && W > FBK_KH && fb_off32(H, pitch)) {
    const bool tma = (pitch % 4) == 0 && (reinterpret_cast<uintptr_t>(M_in) & 15) == 0;
    CUtensorMap tm{};
    if (tma) {
      uint64_t dims[3] = {(uint64_t)W, (uint64_t)H, 5}, strides[2] = {(uint64_t)pitch * 4, (uint64_t)H * pitch * 4};
      uint32_t box[3] = {FBK_IW, FBK_IH, 1};
      int rc = tmap_f32(&tm, M_in, 3, dims, strides, box);
      if (rc) return rc;
    }
    FbTaps2 t2{};
    for (int j = 0; j <= kh; j++) t2.g[j] = make_float2(wk[j], wk[j]);
    dim3 grid((W + FBK_TW - 1) / FBK_TW, (H + FBK_TH - 1) / FBK_TH);
    auto run = [&](auto kernel, cudaError_t e) {
      if (e != cudaSuccess) return set_error(OF_ERR_CUDA, "of_fb_iteration: %s", cudaGetErrorString(e));
      kernel<<<grid, 256, FBK_SMEM, as_stream(stream)>>>(tm, tma, M_in, M_out, R0, R1, flowx, flowy, H, W, pitch, t2, kh,
                                                         update_matrices);
      return check_launch("of_fb_iteration");
    };
    return kh == FBK_KH ? run(fb_iter_tile_kernel<true>, OF_SMEM_OPT_IN(fb_iter_tile_kernel<true>, FBK_SMEM))
                        : run(fb_iter_tile_kernel<false>, OF_SMEM_OPT_IN(fb_iter_tile_kernel<false>, FBK_SMEM));
  }
  size_t smem = sizeof(float) * ((size_t)(FBI_TH + 2 * kh) * (FBI_TW + 2 * kh) + (size_t)FBI_TH * (FBI_TW + 2 * kh));
  dim3 grid((W + FBI_TW - 1) / FBI_TW, (H + FBI_TH - 1) / FBI_TH);
  fb_iter_kernel<<<grid, 256, smem, as_stream(stream)>>>(M_in, M_out, R0, R1, flowx, flowy, H, W, pitch,
                                                         make_taps(wk, kh), kh, update_matrices);
  return check_launch("of_fb_iteration");
}
