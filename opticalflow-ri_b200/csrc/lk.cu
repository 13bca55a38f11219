// A10/A11 dense pyramidal Lucas-Kanade (src/pyrlkDenseLargeW.cl:304-669 with
// -DWSX/-DWSY as set by src/denseLucasKanade_PyCL.py:57-71).
//
// The reference runs one 64-work-item group per pixel.  Here one WARP handles one pixel
// and a CTA handles an 8x8 pixel tile whose window data is shared: the intensity patch
// (41x41 with the Scharr border, clamp-to-edge) and its unweighted Scharr gradients
// (39x39) are staged once per CTA in shared memory.  Lane l plays the reference's work
// items l and l+32 (xid = l&7, yid = l>>3 and yid+4), so the first level of the
// reference's 64->1 reduction tree is an in-lane add and the rest are warp shuffles in
// the same pairing: A, b and the error are reduced in exactly the reference's order.
// J is sampled with exact float32 bilinear weights (pixel-centre convention, clamp to
// edge) from a 64x64 region staged per CTA around the tile's mean displaced window, stored
// as (J[y][x], J[y+4][x]) pairs: the two work items of a lane lie 4 rows apart, so the four
// 64-bit loads of a footprint feed both of them and the blend, the difference and the sums
// run as packed f32x2 operations (each half rounds as the scalar operation does).
//
// What bounds it: shared-memory reads and issue slots.  A sample needs 16 bytes of J on every
// Newton step, and the 27 x 27 window's intensities and gradients another 12; those do not
// change between the steps of a pixel, so each lane keeps its samples' 84 values in
// registers (the reason for 128-thread CTAs at 168 registers, 3 per SM).  The footprints of
// a lane's samples lie at fixed steps of 8 texels unless a position rounds across a texel,
// which the step's fractions show; so all addresses are one base plus constants.  A warp with
// such a position (where a flow is close to a whole number of pixels, a third of them) reads
// each tile's texels from their own place, 32 bits at a time; one with footprints outside the
// region tests every sample.  The error takes the same two ways.
// One 512x512 level from a smooth field (4.5 steps per pixel): 1.10 -> 0.93 ms (shared-memory
// pipe 72 %, FMA pipe 60 %, issue 67 % busy), with status and error 2.63 -> 1.44; from within
// 1e-5 of the frames' 2-pixel shift 0.44 -> 0.41 and 1.30 -> 0.84; a 301x413 level with a
// 19 x 19 window, status and error: 1.23 -> 0.46 ms.
#include <float.h>

#include "common.cuh"

namespace ofb {

constexpr int LK_PT = 8;            // pixel tile edge
constexpr int LK_G = LK_PT + 31;    // gradient positions per axis
constexpr int LK_I = LK_G + 2;      // intensity positions per axis
// Row strides of the staged patches: a warp reads 4 rows of 8 consecutive columns at once,
// so a stride of 8 or 24 (mod 32) banks puts the 4 rows in disjoint banks.
constexpr int LK_IP = 56, LK_GP = 40;  // LK_GP counts float2 (dx, dy) pairs
static_assert(LK_IP >= LK_I && LK_GP >= LK_G && LK_IP % 32 == 24 && LK_GP % 16 == 8, "patch strides");
// J region staged per CTA for the Newton steps: LK_JR x LK_JR texels centred on the tile's
// mean displaced window, row stride LK_JP (72: the 4 rows a warp reads at once fall in
// distinct banks).  Texels hold clamped-coordinate values, so a bilinear footprint inside
// the region reads exactly what the clamped global path reads.
constexpr int LK_JR = 64, LK_JP = 72;  // LK_JP counts float2 texel pairs
static_assert(LK_JP % 16 == 8, "J pair stride");
// dynamic shared memory of the kernel: sJ2 pairs, sD2 pairs, sI
constexpr size_t LK_SMEM = (size_t)LK_JR * LK_JP * 8 + (size_t)LK_G * LK_GP * 8 + (size_t)LK_I * LK_IP * 4;

// Whether a lane holds its window samples in registers, 3 values each, 2 NT^2 samples (28 of the
// default window): not the 32 of the other windows above 24, with which 8 warps fit an SM (a 31 x 31
// window on the smooth field above: 1.53 ms, 1.31 with the samples read again in every step).
constexpr bool lk_hold(int nt, bool def) { return nt < 4 || def; }
// Threads and CTAs per SM of the kernel.
constexpr int lk_threads(int nt, bool def) { return nt == 4 && def ? 128 : 256; }
constexpr int lk_ctas(int nt, bool def) { return nt == 4 && def ? 3 : 2; }

struct LkParams {
  int ws, hw, aL, aR, aT, aB, niter;
};

// per-axis tile weights of work item `id` (:339-373); base[] feeds the error guards
__device__ __forceinline__ void lk_weights(int id, int ws, int lo, int hi, float w[4], int base[2]) {
  if (ws >= 16) {
    base[0] = 16 + id;
    base[1] = 24 + id;
    w[0] = 1.f;
    w[1] = id == 0 ? (float)(1 - lo) : 1.f;
    w[2] = base[0] < ws - hi ? 1.f : 0.f;
    w[3] = base[1] < ws - hi ? 1.f : 0.f;
  } else {
    base[0] = 8 + id;
    base[1] = 16 + id;
    w[0] = 1.f;
    w[1] = id == 0 ? (float)(1 - lo) : (base[0] < ws - hi ? 1.f : 0.f);
    w[2] = 0.f;
    w[3] = 0.f;
  }
}

// A texel index from a floored position.  The error of a pixel whose flow is infinite (or
// merely huge) is evaluated there too; its index is held within 2^22 of the origin, beyond
// every image (H, W < 2^21), so that the index arithmetic that follows cannot overflow.
__device__ __forceinline__ int lk_texel(float f) { return (int)fminf(fmaxf(f, -4194304.f), 4194304.f); }

// The texels (clamp to edge) of the 2 x 2 footprint at (rx, ry) relative to the region: from it when
// they lie inside, else from global memory.
__device__ __forceinline__ void lk_texels(const float2* __restrict__ sJ, const float* __restrict__ J, int H, int W,
                                          int pitch, int rx, int ry, int ox, int oy, float (&t)[4]) {
  if ((unsigned)rx <= (unsigned)(LK_JR - 2) && (unsigned)ry <= (unsigned)(LK_JR - 2)) {
    const float2* q = sJ + ry * LK_JP + rx;
    t[0] = q[0].x;
    t[1] = q[1].x;
    t[2] = q[LK_JP].x;
    t[3] = q[LK_JP + 1].x;
  } else {
    const int i0 = rx + ox, j0 = ry + oy;
    const int xa = clampi(i0, 0, W - 1), xb = clampi(i0 + 1, 0, W - 1);
    const int ya = clampi(j0, 0, H - 1), yb = clampi(j0 + 1, 0, H - 1);
    t[0] = __ldg(J + (size_t)ya * pitch + xa);
    t[1] = __ldg(J + (size_t)ya * pitch + xb);
    t[2] = __ldg(J + (size_t)yb * pitch + xa);
    t[3] = __ldg(J + (size_t)yb * pitch + xb);
  }
}

__device__ __forceinline__ float lk_blend(float a, float oa, float b, float ob, const float (&t)[4]) {
  float r = __fmul_rn(__fmul_rn(oa, ob), t[0]);
  r = __fmaf_rn(__fmul_rn(a, ob), t[1], r);
  r = __fmaf_rn(__fmul_rn(oa, b), t[2], r);
  return __fmaf_rn(__fmul_rn(a, b), t[3], r);
}

// A bilinear sample at any position.
__device__ __forceinline__ float lk_bilinear_s(const float2* __restrict__ sJ, const float* __restrict__ J, int H, int W,
                                               int pitch, float x, float y, int ox, int oy) {
  const float xs = __fsub_rn(x, 0.5f), ys = __fsub_rn(y, 0.5f);
  const float fx0 = floorf(xs), fy0 = floorf(ys);
  const float a = __fsub_rn(xs, fx0), b = __fsub_rn(ys, fy0);
  float t[4];
  lk_texels(sJ, J, H, W, pitch, lk_texel(fx0) - ox, lk_texel(fy0) - oy, ox, oy, t);
  return lk_blend(a, __fsub_rn(1.f, a), b, __fsub_rn(1.f, b), t);
}

// floor(x) for |x| < 2^22, as a float and as an int, on the FMA pipe: x + 1.5 * 2^23 rounded
// toward -inf is floor(x) + 1.5 * 2^23 (that binade's unit is 1), and its low mantissa bits
// hold the integer.
__device__ __forceinline__ float lk_floor(float x, int& i) {
  const float t = __fadd_rd(x, 12582912.0f);
  i = (int)(__float_as_uint(t) - 0x4B400000u);
  return __fsub_rn(t, 12582912.0f);
}

// the reference's reduce tree: (t, t+32) in-lane, then 16, 8, 4, (0+1)+(2+3)
__device__ __forceinline__ float lk_tree(float lo, float hi) {
  float q = __fadd_rn(lo, hi);
  q = __fadd_rn(q, __shfl_down_sync(0xffffffffu, q, 16));
  q = __fadd_rn(q, __shfl_down_sync(0xffffffffu, q, 8));
  q = __fadd_rn(q, __shfl_down_sync(0xffffffffu, q, 4));
  float a = __fadd_rn(q, __shfl_down_sync(0xffffffffu, q, 1));
  float t = __fadd_rn(a, __shfl_down_sync(0xffffffffu, a, 2));
  return __shfl_sync(0xffffffffu, t, 0);
}

// Two sums by the same tree in half the shuffles: after the first exchange lanes 0-15 carry
// the first and lanes 16-31 the second (float32 addition commutes, so the pairing is all
// that matters).  Both results reach every lane.
__device__ __forceinline__ void lk_tree2(float2 a, float2 b, float& sa, float& sb) {
  const float qa = __fadd_rn(a.x, a.y), qb = __fadd_rn(b.x, b.y);
  const bool hi = (threadIdx.x & 16) != 0;
  float q = __fadd_rn(hi ? qb : qa, __shfl_xor_sync(0xffffffffu, hi ? qa : qb, 16));
  q = __fadd_rn(q, __shfl_down_sync(0xffffffffu, q, 8));
  q = __fadd_rn(q, __shfl_down_sync(0xffffffffu, q, 4));
  q = __fadd_rn(q, __shfl_down_sync(0xffffffffu, q, 1));
  q = __fadd_rn(q, __shfl_down_sync(0xffffffffu, q, 2));
  sa = __shfl_sync(0xffffffffu, q, 0);
  sb = __shfl_sync(0xffffffffu, q, 16);
}

// Whether sample (v, ty, tx) of lane (xid, yid) has a non-zero tile weight.
template <bool DEF>
__device__ __forceinline__ bool lk_on(unsigned act, int v, int ty, int tx, int xid, int yid) {
  if (DEF) return (tx < 3 || xid < 3) && (ty < 3 || (v == 0 && yid < 3));
  return (act >> (16 * v + 4 * ty + tx)) & 1u;
}

// NT: the window's tiles of 8 per axis (ceil(ws / 8)); tiles past it have no weight.  DEF: the
// default window (27 x 27, no asymmetric mask), whose tile-weight pattern is known at compile
// time: lane (xid, yid)'s 4th column tile is used when xid < 3, its 4th row tile of the first
// half when yid < 3, the 4th row tile of the second half never.
template <int NT, bool DEF>
__global__ void __launch_bounds__(lk_threads(NT, DEF), lk_ctas(NT, DEF)) lk_dense_kernel(
    const float* __restrict__ I, const float* __restrict__ J, float* __restrict__ U, float* __restrict__ V, int H, int W,
    int pitch, LkParams p, uint8_t* __restrict__ status, float* __restrict__ err) {
  constexpr int LK_THREADS = lk_threads(NT, DEF);
  constexpr bool HOLD = lk_hold(NT, DEF);
  extern __shared__ float4 lk_dyn[];
  float2* const sJ = reinterpret_cast<float2*>(lk_dyn);  // (J[y][x], J[y + 4][x]) pairs
  float2* const sD = sJ + LK_JR * LK_JP;                 // (dx, dy) pairs
  float* const sI = reinterpret_cast<float*>(sD + LK_G * LK_GP);
  const int i0 = blockIdx.y * LK_PT, j0 = blockIdx.x * LK_PT;
  const int oy = i0 - p.hw - 1, ox = j0 - p.hw - 1;  // image position of sI[0][0]
  for (int t = threadIdx.x; t < LK_I * LK_I; t += LK_THREADS) {
    int ly = t / LK_I, lx = t - ly * LK_I;
    sI[ly * LK_IP + lx] = I[(size_t)clampi(oy + ly, 0, H - 1) * pitch + clampi(ox + lx, 0, W - 1)];
  }
  // J region: centred on the tile centre displaced by the mean initial flow of the tile
  __shared__ float red_u[2], red_v[2];
  if (threadIdx.x < LK_PT * LK_PT) {
    const int yy = min(i0 + (int)(threadIdx.x >> 3), H - 1), xx = min(j0 + (int)(threadIdx.x & 7), W - 1);
    float su = U[(size_t)yy * pitch + xx], sv = V[(size_t)yy * pitch + xx];
    su = isfinite(su) ? fminf(fmaxf(su, -1e6f), 1e6f) : 0.f;
    sv = isfinite(sv) ? fminf(fmaxf(sv, -1e6f), 1e6f) : 0.f;
    for (int o = 16; o > 0; o >>= 1) {
      su += __shfl_down_sync(0xffffffffu, su, o);
      sv += __shfl_down_sync(0xffffffffu, sv, o);
    }
    if ((threadIdx.x & 31) == 0) {
      red_u[threadIdx.x >> 5] = su;
      red_v[threadIdx.x >> 5] = sv;
    }
  }
  __syncthreads();
  const float mu = (red_u[0] + red_u[1]) * (1.f / 64.f), mv = (red_v[0] + red_v[1]) * (1.f / 64.f);
  const int jox = j0 + LK_PT / 2 + (int)floorf(mu) - LK_JR / 2, joy = i0 + LK_PT / 2 + (int)floorf(mv) - LK_JR / 2;
#pragma unroll 4
  for (int t = threadIdx.x; t < LK_JR * LK_JR; t += LK_THREADS) {
    const int ly = t / LK_JR, lx = t - ly * LK_JR;
    const float* col = J + clampi(jox + lx, 0, W - 1);
    sJ[ly * LK_JP + lx] = make_float2(__ldg(col + (size_t)clampi(joy + ly, 0, H - 1) * pitch),
                                      __ldg(col + (size_t)clampi(joy + ly + 4, 0, H - 1) * pitch));
  }
  for (int t = threadIdx.x; t < LK_G * LK_G; t += LK_THREADS) {
    int gy = t / LK_G, gx = t - gy * LK_G;
    const float* c = sI + (gy + 1) * LK_IP + gx + 1;
#define P(dy, dx) c[(dy) * LK_IP + (dx)]
    float ddx, ddy;
    ddx = __fmaf_rn(__fsub_rn(__fsub_rn(__fadd_rn(P(-1, 1), P(1, 1)), P(-1, -1)), P(1, -1)), 3.0f,
                       __fmul_rn(__fsub_rn(P(0, 1), P(0, -1)), 10.0f));
    ddy = __fmaf_rn(__fsub_rn(__fsub_rn(__fadd_rn(P(1, -1), P(1, 1)), P(-1, -1)), P(-1, 1)), 3.0f,
                       __fmul_rn(__fsub_rn(P(1, 0), P(-1, 0)), 10.0f));
#undef P
    sD[gy * LK_GP + gx] = make_float2(ddx, ddy);
  }
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int xid = lane & 7, yid = lane >> 3;
  // A single texel (y, x) as a float index from sJ's pair (y, x): its first part, or for the lanes of
  // rows 2 and 3 the second part of the pair 4 rows up, so that a warp's reads fall in distinct banks.
  const unsigned row_lo = yid >= 2 ? 4 : 0;
  const int row_part = yid >= 2 ? 1 - 8 * LK_JP : 0;
  const float* const texel = reinterpret_cast<const float*>(sJ) + row_part;
  unsigned act = 0;  // bit 16 v + 4 ty + tx: the sample's tile weight is not 0
  unsigned any = 0;  // the same bit set when it is for some lane of the warp
  if (!DEF) {
    float wx[4], wy0[4], wy1[4];
    int bx[2], by0[2], by1[2];
    lk_weights(xid, p.ws, p.aL, p.aR, wx, bx);
    lk_weights(yid, p.ws, p.aT, p.aB, wy0, by0);
    lk_weights(yid + 4, p.ws, p.aT, p.aB, wy1, by1);
#pragma unroll
    for (int v = 0; v < 2; v++)
#pragma unroll
      for (int ty = 0; ty < 4; ty++)
#pragma unroll
        for (int tx = 0; tx < 4; tx++)
          act |= (unsigned)(__fmul_rn(wx[tx], (v ? wy1 : wy0)[ty]) != 0.f) << (16 * v + 4 * ty + tx);
    any = __reduce_or_sync(0xffffffffu, act);
  }
  // samples no lane has (row tile ty of half v, column tile tx): warp-uniform
#define LK_SKIP(v, ty, tx) (DEF ? ((v) == 1 && (ty) == 3) : !((any >> (16 * (v) + 4 * (ty) + (tx))) & 1u))
#define LK_SKIP2(ty, tx) (LK_SKIP(0, ty, tx) && LK_SKIP(1, ty, tx))
  const float hw = (float)p.hw;
  const float2 m1 = make_float2(-1.f, -1.f);  // a - b as one fused multiply-add
#pragma unroll 1
  for (int i = i0 + warp; i < min(i0 + LK_PT, H); i += LK_THREADS / 32) {
    const int gyb = i - i0;
    // the row's initial flow, one pixel per lane
    const int jl = min(j0 + (lane & (LK_PT - 1)), W - 1);
    const float row_u = U[(size_t)i * pitch + jl], row_v = V[(size_t)i * pitch + jl];
#pragma unroll 1
    for (int c = 0; c < LK_PT; c++) {
      const int j = j0 + c;
      if (j >= W) break;
      const int gxb = c;  // (gyb, gxb): gradient-tile origin of this pixel's window
      const float* const pI = sI + (gyb + yid + 1) * LK_IP + gxb + xid + 1;
      const float2* const pD = sD + (gyb + yid) * LK_GP + gxb + xid;
      // A window sample's intensities (negated) and gradients, as pairs over the two row halves.
      // Samples without weight hold 0.
      struct Sample {
        float2 nI, Dx, Dy;
      };
      auto window = [&](int ty, int tx) {
        float iv[2], dx[2], dy[2];
#pragma unroll
        for (int v = 0; v < 2; v++) {
          iv[v] = dx[v] = dy[v] = 0.f;
          if (LK_SKIP(v, ty, tx)) continue;
          iv[v] = -pI[(ty * 8 + 4 * v) * LK_IP + tx * 8];
          const float2 d = pD[(ty * 8 + 4 * v) * LK_GP + tx * 8];
          const bool on = lk_on<DEF>(act, v, ty, tx, xid, yid);
          dx[v] = on ? d.x : 0.f;
          dy[v] = on ? d.y : 0.f;
        }
        return Sample{make_float2(iv[0], iv[1]), make_float2(dx[0], dx[1]), make_float2(dy[0], dy[1])};
      };
      Sample held[HOLD ? NT : 1][HOLD ? NT : 1] = {};  // stay in registers for every Newton step
      auto sample = [&](int ty, int tx) {
        if constexpr (HOLD)
          return held[ty][tx];
        else
          return window(ty, tx);
      };
      float2 a11 = make_float2(0.f, 0.f), a12 = a11, a22 = a11;
#pragma unroll
      for (int ty = 0; ty < NT; ty++)
#pragma unroll
        for (int tx = 0; tx < NT; tx++) {
          if (!HOLD && LK_SKIP2(ty, tx)) continue;
          const Sample w = window(ty, tx);
          // the tile weights are products of 0 / 1 values, so the reference's multiplications by
          // them are exact identities; + 0 * 0 changes no sum
          if (DEF) {
            if (ty < NT - 1) {
              a11.y = __fmaf_rn(w.Dx.y, w.Dx.y, a11.y);
              a12.y = __fmaf_rn(w.Dx.y, w.Dy.y, a12.y);
              a22.y = __fmaf_rn(w.Dy.y, w.Dy.y, a22.y);
            }
            a11.x = __fmaf_rn(w.Dx.x, w.Dx.x, a11.x);
            a12.x = __fmaf_rn(w.Dx.x, w.Dy.x, a12.x);
            a22.x = __fmaf_rn(w.Dy.x, w.Dy.x, a22.x);
          } else {
            a11 = __ffma2_rn(w.Dx, w.Dx, a11);
            a12 = __ffma2_rn(w.Dx, w.Dy, a12);
            a22 = __ffma2_rn(w.Dy, w.Dy, a22);
          }
          if constexpr (HOLD) held[ty][tx] = w;
        }
      float A11, A12, A22;
      lk_tree2(a11, a12, A11, A12);
      A22 = lk_tree(a22.x, a22.y);
      const size_t gid = (size_t)i * pitch + j;
      float D = __fmaf_rn(A11, A22, -__fmul_rn(A12, A12));
      if (D < 1.192092896e-07f) {
        if (lane == 0) {
          if (status) status[gid] = 0;
          if (err) err[gid] = 0.f;
        }
        continue;
      }
      A11 = __fdiv_rn(A11, D);
      A12 = __fdiv_rn(A12, D);
      A22 = __fdiv_rn(A22, D);
      float ptx = __fsub_rn(__fadd_rn((float)j, __shfl_sync(0xffffffffu, row_u, c)), hw);
      float pty = __fsub_rn(__fadd_rn((float)i, __shfl_sync(0xffffffffu, row_v, c)), hw);
      // sample positions: x per column tile, y per row tile as pairs over the two row halves
      float lx[NT];
      float2 ly[NT];
      lx[0] = __fadd_rn(ptx, __fadd_rn((float)xid, 0.5f));
      ly[0].x = __fadd_rn(pty, __fadd_rn((float)yid, 0.5f));
      ly[0].y = __fadd_rn(pty, __fadd_rn((float)(yid + 4), 0.5f));
#pragma unroll
      for (int t = 1; t < NT; t++) {
        lx[t] = __fadd_rn(lx[t - 1], 8.0f);
        ly[t].x = __fadd_rn(ly[t - 1].x, 8.0f);
        ly[t].y = __fadd_rn(ly[t - 1].y, 8.0f);
      }
      // The fractions of every tile's position and the texels of their footprints relative to the
      // region; whether those of the whole warp lie in it.  Of use for positions below 2^22.
      auto footprints = [&](float2(&xa)[NT], float2(&xo)[NT], float2(&yb)[NT], float2(&yo)[NT], int(&xi)[NT],
                            int(&yi)[2][NT]) {
        unsigned xout = 0, yout = 0;
#pragma unroll
        for (int t = 0; t < NT; t++) {
          const float xs = __fsub_rn(lx[t], 0.5f), y0 = __fsub_rn(ly[t].x, 0.5f), y1 = __fsub_rn(ly[t].y, 0.5f);
          const float a = __fsub_rn(xs, lk_floor(xs, xi[t])), oa = __fsub_rn(1.f, a);
          xa[t] = make_float2(a, a);
          xo[t] = make_float2(oa, oa);
          yb[t] = make_float2(__fsub_rn(y0, lk_floor(y0, yi[0][t])), __fsub_rn(y1, lk_floor(y1, yi[1][t])));
          yo[t] = __ffma2_rn(yb[t], m1, make_float2(1.f, 1.f));
          // unsigned: the texels of a position that is out of reach may wrap, but not overflow
          xi[t] = (int)((unsigned)xi[t] - (unsigned)jox);
          yi[0][t] = (int)((unsigned)yi[0][t] - (unsigned)joy);
          yi[1][t] = (int)((unsigned)yi[1][t] - (unsigned)joy);
          xout = max(xout, (unsigned)xi[t]);
          yout = max(yout, max((unsigned)yi[0][t] - row_lo, (unsigned)yi[1][t] - row_lo));
        }
        return __all_sync(0xffffffffu, xout <= LK_JR - 2 && yout <= LK_JR - 2 - row_lo) != 0;
      };
      uint8_t st = 1;
#pragma unroll 1
      for (int k = 0; k < p.niter; k++) {
        if (ptx < -hw || ptx >= (float)W || pty < -hw || pty >= (float)H) {
          st = 0;
          break;
        }
        // positions here are within a window of the image (the step's range test), so
        // |xs|, |ys| < 2^22 (the ABI caps H, W) and lk_floor is floorf
        int rx, ry;
        const float fx = lk_floor(__fsub_rn(lx[0], 0.5f), rx), fy = lk_floor(__fsub_rn(ly[0].x, 0.5f), ry);
        // The fractions of every position against the first one's floor plus the tile step: a
        // fraction in [0, 1) is the position's own (the float32 difference is exact), so a
        // lane whose fractions all are has its footprints at fixed steps from the first.
        float2 xa[NT], xo[NT], yb[NT], yo[NT];
        unsigned worst = 0;
#pragma unroll
        for (int t = 0; t < NT; t++) {
          const float a = __fsub_rn(__fsub_rn(lx[t], 0.5f), __fadd_rn(fx, 8.f * t)), oa = __fsub_rn(1.f, a);
          xa[t] = make_float2(a, a);
          xo[t] = make_float2(oa, oa);
          const float2 f = __fadd2_rn(make_float2(fy, fy), make_float2(8.f * t, 8.f * t + 4.f));
          yb[t] = __ffma2_rn(f, m1, __fadd2_rn(ly[t], make_float2(-0.5f, -0.5f)));
          yo[t] = __ffma2_rn(yb[t], m1, make_float2(1.f, 1.f));
          worst = max(max(worst, __float_as_uint(a)), max(__float_as_uint(yb[t].x), __float_as_uint(yb[t].y)));
        }
        rx -= jox;
        ry -= joy;
        const bool regular = worst < 0x3f800000u && (unsigned)rx <= (unsigned)(LK_JR - 2 - 8 * (NT - 1)) &&
                             (unsigned)ry <= (unsigned)(LK_JR - 2 - 8 * (NT - 1) - 4);
        float2 b1 = make_float2(0.f, 0.f), b2 = b1;
        // sample (ty, tx) of both row halves from the texels of its footprint
        auto add = [&](int ty, int tx, float2 t00, float2 t10, float2 t01, float2 t11) {
          const float2 w00 = __fmul2_rn(xo[tx], yo[ty]), w10 = __fmul2_rn(xa[tx], yo[ty]);
          const float2 w01 = __fmul2_rn(xo[tx], yb[ty]), w11 = __fmul2_rn(xa[tx], yb[ty]);
          float2 Jv = __fmul2_rn(w00, t00);
          Jv = __ffma2_rn(w10, t10, Jv);
          Jv = __ffma2_rn(w01, t01, Jv);
          Jv = __ffma2_rn(w11, t11, Jv);
          const Sample w = sample(ty, tx);
          float2 d = __fadd2_rn(Jv, w.nI);  // (Jv - Iv) * w with w == 1
          if (!DEF || tx == NT - 1) {
            if (!lk_on<DEF>(act, 0, ty, tx, xid, yid)) d.x = 0.f;
            if (!lk_on<DEF>(act, 1, ty, tx, xid, yid)) d.y = 0.f;
          }
          b1 = __ffma2_rn(d, w.Dx, b1);
          b2 = __ffma2_rn(d, w.Dy, b2);
        };
        // the same for the first half alone
        auto add0 = [&](int ty, int tx, float t00, float t10, float t01, float t11) {
          float Jv = __fmul_rn(__fmul_rn(xo[tx].x, yo[ty].x), t00);
          Jv = __fmaf_rn(__fmul_rn(xa[tx].x, yo[ty].x), t10, Jv);
          Jv = __fmaf_rn(__fmul_rn(xo[tx].x, yb[ty].x), t01, Jv);
          Jv = __fmaf_rn(__fmul_rn(xa[tx].x, yb[ty].x), t11, Jv);
          const Sample w = sample(ty, tx);
          float d = __fadd_rn(Jv, w.nI.x);
          if (!lk_on<DEF>(act, 0, ty, tx, xid, yid)) d = 0.f;
          b1.x = __fmaf_rn(d, w.Dx.x, b1.x);
          b2.x = __fmaf_rn(d, w.Dy.x, b2.x);
        };
        if (__all_sync(0xffffffffu, regular)) {
          const float2* const q = sJ + ry * LK_JP + rx;
#pragma unroll
          for (int ty = 0; ty < NT; ty++)
#pragma unroll
            for (int tx = 0; tx < NT; tx++) {
              if (LK_SKIP2(ty, tx)) continue;
              const float2* const s = q + (8 * ty) * LK_JP + 8 * tx;
              if (DEF && ty == NT - 1)  // 32-bit reads, scalar arithmetic
                add0(ty, tx, s[0].x, s[1].x, s[LK_JP].x, s[LK_JP + 1].x);
              else
                add(ty, tx, s[0], s[1], s[LK_JP], s[LK_JP + 1]);
            }
        } else {
          // some footprint rounds to another texel or leaves the region: each tile's own
          int xi[NT], yi[2][NT];
          if (footprints(xa, xo, yb, yo, xi, yi)) {
#pragma unroll
            for (int ty = 0; ty < NT; ty++)
#pragma unroll
              for (int tx = 0; tx < NT; tx++) {
                if (LK_SKIP2(ty, tx)) continue;
                const float* const s = texel + 2 * (yi[0][ty] * LK_JP + xi[tx]);
                if (DEF && ty == NT - 1) {
                  add0(ty, tx, s[0], s[2], s[2 * LK_JP], s[2 * LK_JP + 2]);
                } else {
                  const float* const r = texel + 2 * (yi[1][ty] * LK_JP + xi[tx]);
                  add(ty, tx, make_float2(s[0], r[0]), make_float2(s[2], r[2]),
                      make_float2(s[2 * LK_JP], r[2 * LK_JP]), make_float2(s[2 * LK_JP + 2], r[2 * LK_JP + 2]));
                }
              }
          } else {
            auto half = [&](int v, float& s1, float& s2) {
#pragma unroll
              for (int ty = 0; ty < NT; ty++)
#pragma unroll
                for (int tx = 0; tx < NT; tx++) {
                  if (LK_SKIP(v, ty, tx) || !lk_on<DEF>(act, v, ty, tx, xid, yid)) continue;
                  float t[4];
                  int y;
                  const float ys = __fsub_rn(v ? ly[ty].y : ly[ty].x, 0.5f), b = __fsub_rn(ys, lk_floor(ys, y));
                  const float ob = __fsub_rn(1.f, b);
                  lk_texels(sJ, J, H, W, pitch, xi[tx], y - joy, jox, joy, t);
                  const float Jv = lk_blend(xa[tx].x, xo[tx].x, b, ob, t);
                  const Sample w = sample(ty, tx);
                  const float d = __fadd_rn(Jv, v ? w.nI.y : w.nI.x);
                  s1 = __fmaf_rn(d, v ? w.Dx.y : w.Dx.x, s1);
                  s2 = __fmaf_rn(d, v ? w.Dy.y : w.Dy.x, s2);
                }
            };
            half(0, b1.x, b2.x);
            half(1, b1.y, b2.y);
          }
        }
        float B1, B2;
        lk_tree2(b1, b2, B1, B2);
        float dx = __fmul_rn(__fmaf_rn(A12, B2, -__fmul_rn(A22, B1)), 32.0f);
        float dy = __fmul_rn(__fmaf_rn(A12, B1, -__fmul_rn(A11, B2)), 32.0f);
        ptx = __fadd_rn(ptx, dx);
        pty = __fadd_rn(pty, dy);
#pragma unroll
        for (int t = 0; t < NT; t++) {
          lx[t] = __fadd_rn(lx[t], dx);
          ly[t] = __fadd2_rn(ly[t], make_float2(dy, dy));
        }
        if (fabsf(dx) < 0.01f && fabsf(dy) < 0.01f) break;
      }
      if (err) {
        // GetError visiting order and guards (:620-653); bits: 1 xBase, 2 yBase, 4 xBase2, 8 yBase2
        const int ord[16] = {0x000, 0x010, 0x100, 0x110, 0x021, 0x121, 0x202, 0x212,
                             0x223, 0x034, 0x134, 0x234, 0x308, 0x318, 0x328, 0x33c};
        float wx[4], wy0[4], wy1[4];  // recomputed here rather than kept live through the steps
        int bx[2], by0[2], by1[2];
        lk_weights(xid, p.ws, p.aL, p.aR, wx, bx);
        lk_weights(yid, p.ws, p.aT, p.aB, wy0, by0);
        lk_weights(yid + 4, p.ws, p.aT, p.aB, wy1, by1);
        float2 xa[NT], xo[NT], yb[NT], yo[NT];
        int xi[NT], yi[2][NT];
        // the positions of an infinite or huge flow are beyond footprints' reach
        const bool inside = footprints(xa, xo, yb, yo, xi, yi) &
                            (__all_sync(0xffffffffu, fabsf(lx[0]) < 2097152.f && fabsf(ly[0].x) < 2097152.f) != 0);
        float e0 = 0.f, e1 = 0.f;
#pragma unroll
        for (int o = 0; o < 16; o++) {
          const int ty = ord[o] >> 8, tx = (ord[o] >> 4) & 15, gb = ord[o] & 15;
          if (ty >= NT || tx >= NT) continue;  // beyond the window: their guards are false
          if ((gb & 1) && !(bx[0] < p.ws)) continue;
          if ((gb & 4) && !(bx[1] < p.ws)) continue;
          const bool on0 = (!(gb & 2) || by0[0] < p.ws) && (!(gb & 8) || by0[1] < p.ws);
          const bool on1 = (!(gb & 2) || by1[0] < p.ws) && (!(gb & 8) || by1[1] < p.ws);
          float2 Jv;
          if (inside) {
            const float* const s = texel + 2 * (yi[0][ty] * LK_JP + xi[tx]);
            const float* const r = texel + 2 * (yi[1][ty] * LK_JP + xi[tx]);
            Jv = __fmul2_rn(__fmul2_rn(xo[tx], yo[ty]), make_float2(s[0], r[0]));
            Jv = __ffma2_rn(__fmul2_rn(xa[tx], yo[ty]), make_float2(s[2], r[2]), Jv);
            Jv = __ffma2_rn(__fmul2_rn(xo[tx], yb[ty]), make_float2(s[2 * LK_JP], r[2 * LK_JP]), Jv);
            Jv = __ffma2_rn(__fmul2_rn(xa[tx], yb[ty]), make_float2(s[2 * LK_JP + 2], r[2 * LK_JP + 2]), Jv);
          } else {
            Jv.x = lk_bilinear_s(sJ, J, H, W, pitch, lx[tx], ly[ty].x, jox, joy);
            Jv.y = lk_bilinear_s(sJ, J, H, W, pitch, lx[tx], ly[ty].y, jox, joy);
          }
          const float2 Iv = make_float2(pI[ty * 8 * LK_IP + tx * 8], pI[(ty * 8 + 4) * LK_IP + tx * 8]);
          // the reference's divisions by 512 are exact scalings
          const float2 big = make_float2(16384.f, 16384.f), half = make_float2(256.f, 256.f);
          const float2 inv = make_float2(1.f / 512.f, 1.f / 512.f);
          float2 d = __ffma2_rn(__fmul2_rn(__ffma2_rn(Iv, big, half), inv), m1, __fmul2_rn(__ffma2_rn(Jv, big, half), inv));
          d = __fmul2_rn(d, make_float2(__fmul_rn(wx[tx], wy0[ty]), __fmul_rn(wx[tx], wy1[ty])));
          if (on0) e0 = __fadd_rn(e0, fabsf(d.x));
          if (on1) e1 = __fadd_rn(e1, fabsf(d.y));
        }
        float E = lk_tree(e0, e1);
        if (lane == 0) err[gid] = __fdiv_rn(E, (float)(32 * p.ws * p.ws));
      }
      if (lane == 0) {
        U[gid] = __fsub_rn(__fadd_rn(ptx, hw), (float)j);
        V[gid] = __fsub_rn(__fadd_rn(pty, hw), (float)i);
        if (status) status[gid] = st;
      }
    }
  }
#undef LK_SKIP2
#undef LK_SKIP
}

}  // namespace ofb

using namespace ofb;

extern "C" int of_lk_dense(const float* I, const float* J, float* U, float* V, int H, int W, int pitch, int half_win,
                           int niter, const int* asym, uint8_t* status, float* err, void* stream) {
  OF_REQUIRE(!bad_plane(I, H, W, pitch) && J && U && V, "of_lk_dense: bad plane");
  OF_REQUIRE(half_win >= 1 && half_win <= 15, "of_lk_dense: half_win must be in 1..15");
  OF_REQUIRE(niter >= 0, "of_lk_dense: niter < 0");
  OF_REQUIRE(H < (1 << 21) && W < (1 << 21), "of_lk_dense: H and W must be below 2^21");
  LkParams p;
  p.ws = 2 * half_win + 1;
  p.hw = (p.ws - 1) >> 1;
  p.aL = asym ? asym[0] : 0;
  p.aR = asym ? asym[1] : 0;
  p.aT = asym ? asym[2] : 0;
  p.aB = asym ? asym[3] : 0;
  // the reference's window masks are 0 / 1 (denseLucasKanade_PyCL.py:75-92); the kernel's
  // tile weights rely on it
  OF_REQUIRE(((p.aL | p.aR | p.aT | p.aB) & ~1) == 0, "of_lk_dense: asym entries must be 0 or 1");
  p.niter = niter;
  dim3 grid((W + LK_PT - 1) / LK_PT, (H + LK_PT - 1) / LK_PT);
  const bool def = p.ws == 27 && !(p.aL | p.aR | p.aT | p.aB);
  // tiles with weight per axis; the error visits one more (of weight 0) when ws < 16
  const int nt = p.ws > 24 ? 4 : (p.ws > 16 || err) ? 3 : 2;
  auto run = [&](auto kernel, int threads, cudaError_t e) {
    if (e != cudaSuccess) return set_error(OF_ERR_CUDA, "of_lk_dense: %s", cudaGetErrorString(e));
    kernel<<<grid, threads, LK_SMEM, as_stream(stream)>>>(I, J, U, V, H, W, pitch, p, status, err);
    return check_launch("of_lk_dense");
  };
#define LK_RUN(NT, DEF) \
  run(lk_dense_kernel<NT, DEF>, lk_threads(NT, DEF), OF_SMEM_OPT_IN((lk_dense_kernel<NT, DEF>), LK_SMEM))
  if (def) return LK_RUN(4, true);
  if (nt == 4) return LK_RUN(4, false);
  return nt == 3 ? LK_RUN(3, false) : LK_RUN(2, false);
#undef LK_RUN
}
