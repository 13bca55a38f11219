// A1 Gaussian prefilter (src/gaussian_filter.py:24-94), bit-exact.
//
// One CTA filters a 64x32 output tile.  The input tile (with a K/2 halo, the
// reference's border mapping applied per axis) is staged in shared memory, the row
// pass runs over every staged row (halo rows included, because the column pass of the
// reference reads row-filtered values), then the column pass writes the tile.
// Arithmetic is float32 multiply then add, taps j = 0..K-1 against t[x+2h-j]: the exact
// order of convolveDirect.  HBM traffic: one read of the frame (uint8 or float32) and
// one float32 write.
#include "common.cuh"

namespace ofb {

constexpr int PF_TW = 64, PF_TH = 32, PF_MAXK = 15;  // the pyramid's prefilters (3 and 5 taps)
constexpr int PF_MAXK_LARGE = 81;                     // the Liu-Shen warp's 73-tap smoothing

struct PfTaps {
  float k[PF_MAXK_LARGE];
};

// Border of convolveSeparableFilter (:62-66): coordinate c of a line of length n with
// half width h maps to line[-1-c] left of the line and line[c-h] right of it.
__device__ __forceinline__ int pf_map(int c, int n, int h) {
  if (c < 0) c = -1 - c;
  else if (c >= n) c = c - h;
  return clampi(c, 0, n - 1);  // only reached for outputs outside the image
}

// K taps at run time, up to MAXK.
template <typename Tin, int MAXK>
__global__ void __launch_bounds__(256) prefilter_kernel(const Tin* __restrict__ src, int sp, float* __restrict__ dst,
                                                        int dp, int H, int W, const PfTaps taps, int K) {
  extern __shared__ float sm[];
  const int h = K >> 1;
  const int iw = PF_TW + 2 * h, ih = PF_TH + 2 * h;
  float* tin = sm;             // ih x iw
  float* trow = sm + ih * iw;  // ih x PF_TW
  const int x0 = blockIdx.x * PF_TW, y0 = blockIdx.y * PF_TH;
  const int tid = threadIdx.x;
  for (int i = tid; i < ih * iw; i += blockDim.x) {
    int ly = i / iw, lx = i - ly * iw;
    int gy = pf_map(y0 - h + ly, H, h), gx = pf_map(x0 - h + lx, W, h);
    tin[i] = (float)src[(size_t)gy * sp + gx];
  }
  __syncthreads();
  // row pass: out[x] = sum_j k[j] * P(x + h - j), P(c) = tin[.][c - (x0 - h)]
  for (int i = tid; i < ih * PF_TW; i += blockDim.x) {
    int ly = i / PF_TW, lx = i - ly * PF_TW;
    const float* t = tin + ly * iw + lx + 2 * h;
    float acc = 0.0f;
#pragma unroll(MAXK <= PF_MAXK ? MAXK : 8)
    for (int j = 0; j < MAXK; j++)
      if (j < K) acc = __fadd_rn(acc, __fmul_rn(t[-j], taps.k[j]));
    trow[i] = acc;
  }
  __syncthreads();
  for (int i = tid; i < PF_TH * PF_TW; i += blockDim.x) {
    int ly = i / PF_TW, lx = i - ly * PF_TW;
    int y = y0 + ly, x = x0 + lx;
    if (y >= H || x >= W) continue;
    const float* t = trow + (ly + 2 * h) * PF_TW + lx;
    float acc = 0.0f;
#pragma unroll(MAXK <= PF_MAXK ? MAXK : 8)
    for (int j = 0; j < MAXK; j++)
      if (j < K) acc = __fadd_rn(acc, __fmul_rn(t[-j * PF_TW], taps.k[j]));
    dst[(size_t)y * dp + x] = acc;
  }
}

// The pyramid's 3- and 5-tap prefilters: the tile is staged with every load in flight at once
// (no border mapping inside the image), then a thread takes two columns and four rows: it
// filters the 4 + 2h rows it needs along the row in registers and these along the column, so the
// row pass costs no second trip through shared memory and no second barrier.  The sums are
// prefilter_kernel's.  What bounds it is the latency of a tile's loads.  5 taps, us, against
// prefilter_kernel with constants: 512 x 512 4.1 -> 2.5, 1024 x 1024 7.0 -> 5.2, 2048 x 2048 19.7 ->
// 13.3 (5.1 at the bandwidth of a copy).
struct PfTapsSmall {
  float k[5];
};
template <typename Tin, int K>
__global__ void __launch_bounds__(256) prefilter_small_kernel(const Tin* __restrict__ src, int sp,
                                                              float* __restrict__ dst, int dp, int H, int W,
                                                              const PfTapsSmall taps, int vec) {
  constexpr int h = K / 2, IW = PF_TW + 2 * h, IH = PF_TH + 2 * h, N = IW * IH, NK = (N + 255) / 256, R = 4;
  static_assert(PF_TW == 64 && PF_TH == 8 * R && IW % 2 == 0, "32 column pairs by 8 row groups");
  __shared__ __align__(8) float tin[N];
  const int x0 = blockIdx.x * PF_TW, y0 = blockIdx.y * PF_TH, tid = threadIdx.x;
  Tin v[NK];
  if (x0 >= h && y0 >= h && x0 + PF_TW + h <= W && y0 + PF_TH + h <= H) {
    const Tin* t = src + (size_t)(y0 - h) * sp + (x0 - h);
#pragma unroll
    for (int j = 0; j < NK; j++) {
      const int i = min(tid + 256 * j, N - 1), ly = i / IW;
      v[j] = t[(size_t)ly * sp + (i - ly * IW)];
    }
  } else {
#pragma unroll
    for (int j = 0; j < NK; j++) {
      const int i = min(tid + 256 * j, N - 1), ly = i / IW;
      v[j] = src[(size_t)pf_map(y0 - h + ly, H, h) * sp + pf_map(x0 - h + i - ly * IW, W, h)];
    }
  }
#pragma unroll
  for (int j = 0; j < NK; j++) tin[min(tid + 256 * j, N - 1)] = (float)v[j];
  __syncthreads();
  const int c = 2 * (tid & 31), r0 = R * (tid >> 5);
  const int x = x0 + c;
  if (x >= W) return;
  float2 row[R + 2 * h];  // row-filtered pairs
#pragma unroll
  for (int r = 0; r < R + 2 * h; r++) {
    float t[2 + 2 * h];
#pragma unroll
    for (int q = 0; q < 1 + h; q++) {
      const float2 p = *reinterpret_cast<const float2*>(&tin[(r0 + r) * IW + c + 2 * q]);
      t[2 * q] = p.x;
      t[2 * q + 1] = p.y;
    }
    float a = 0.0f, b = 0.0f;
#pragma unroll
    for (int j = 0; j < K; j++) {
      a = __fadd_rn(a, __fmul_rn(t[2 * h - j], taps.k[j]));
      b = __fadd_rn(b, __fmul_rn(t[2 * h + 1 - j], taps.k[j]));
    }
    row[r] = make_float2(a, b);
  }
#pragma unroll
  for (int r = 0; r < R; r++) {
    const int y = y0 + r0 + r;
    if (y >= H) return;
    float a = 0.0f, b = 0.0f;
#pragma unroll
    for (int j = 0; j < K; j++) {
      a = __fadd_rn(a, __fmul_rn(row[r + 2 * h - j].x, taps.k[j]));
      b = __fadd_rn(b, __fmul_rn(row[r + 2 * h - j].y, taps.k[j]));
    }
    float* o = dst + (size_t)y * dp + x;
    if (vec && x + 1 < W) {
      *reinterpret_cast<float2*>(o) = make_float2(a, b);
    } else {
      o[0] = a;
      if (x + 1 < W) o[1] = b;
    }
  }
}

template <typename Tin>
static int launch_prefilter(const Tin* src, int sp, float* dst, int dp, int H, int W, const float* taps, int K,
                            void* stream, const char* name) {
  OF_REQUIRE(!bad_plane(src, H, W, sp) && !bad_plane(dst, H, W, dp), "%s: bad plane", name);
  OF_REQUIRE(taps && K >= 1 && K <= PF_MAXK_LARGE && (K & 1), "%s: K must be odd and <= %d", name, PF_MAXK_LARGE);
  OF_REQUIRE(H >= K / 2 && W >= K / 2, "%s: image smaller than the half kernel", name);
  OF_REQUIRE((const void*)src != (const void*)dst, "%s: src and dst alias", name);
  PfTaps t{};
  for (int j = 0; j < K; j++) t.k[j] = taps[j];
  int h = K / 2;
  size_t smem = sizeof(float) * ((size_t)(PF_TH + 2 * h) * (PF_TW + 2 * h) + (size_t)(PF_TH + 2 * h) * PF_TW);
  dim3 grid((W + PF_TW - 1) / PF_TW, (H + PF_TH - 1) / PF_TH);
  if (K <= PF_MAXK) {
    if (K == 3 || K == 5) {
      PfTapsSmall s{};
      for (int j = 0; j < K; j++) s.k[j] = taps[j];
      const int vec = dp % 2 == 0 && (reinterpret_cast<uintptr_t>(dst) & 7) == 0;
      if (K == 5)
        prefilter_small_kernel<Tin, 5><<<grid, 256, 0, as_stream(stream)>>>(src, sp, dst, dp, H, W, s, vec);
      else
        prefilter_small_kernel<Tin, 3><<<grid, 256, 0, as_stream(stream)>>>(src, sp, dst, dp, H, W, s, vec);
      return check_launch(name);
    }
    prefilter_kernel<Tin, PF_MAXK><<<grid, 256, smem, as_stream(stream)>>>(src, sp, dst, dp, H, W, t, K);
  } else {
    // up to 83 KB of staged tile for 81 taps
    cudaError_t e = OF_SMEM_OPT_IN((prefilter_kernel<Tin, PF_MAXK_LARGE>), 96 * 1024);
    if (e != cudaSuccess) return set_error(OF_ERR_CUDA, "%s: %s", name, cudaGetErrorString(e));
    prefilter_kernel<Tin, PF_MAXK_LARGE><<<grid, 256, smem, as_stream(stream)>>>(src, sp, dst, dp, H, W, t, K);
  }
  return check_launch(name);
}

}  // namespace ofb

using namespace ofb;

extern "C" int of_prefilter_f32(const float* src, int src_pitch, float* dst, int dst_pitch, int H, int W,
                                const float* taps, int K, void* stream) {
  return launch_prefilter<float>(src, src_pitch, dst, dst_pitch, H, W, taps, K, stream, "of_prefilter_f32");
}

extern "C" int of_prefilter_u8(const uint8_t* src, int src_pitch, float* dst, int dst_pitch, int H, int W,
                               const float* taps, int K, void* stream) {
  return launch_prefilter<uint8_t>(src, src_pitch, dst, dst_pitch, H, W, taps, K, stream, "of_prefilter_u8");
}
