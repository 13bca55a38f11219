// The Horn-Schunck sweep on a region held in shared memory, shared by the multi-launch pass
// (hs.cu) and the persistent kernels (hsq.cu): src/HornSchunck.py:61-70 (HS_helper), cell
// for cell the arithmetic of hs_sweep_kernel.
#pragma once

#include <type_traits>

#include "common.cuh"

namespace ofb {

constexpr int HQ_THREADS = 256;  // threads per CTA of the region sweeps

// of_hs_batch with a scratch buffer of hs_halo_bytes(H, W) bytes (0: the size has none) through
// which one pair may run by the tagged-halo schedule.
int hs_batch(const OfHsBatchPair* pairs, int n, const OfTuning* tuning, int* status, long long wait_limit,
             void* workspace, size_t workspace_bytes, void* halo, void* stream);
size_t hs_halo_bytes(int H, int W);
// The device word in the workspace that says which schedule the last such launch ran.
const int* hs_batch_mode(const OfHsBatchPair* pairs, int n, void* workspace, size_t workspace_bytes);

// (u, v) as held in shared memory: float64 copies of the float32 values for the bit-exact
// arithmetic (the reference's float64 stencil sums then need no conversion per
// neighbour), float32 for the float32 averaging.
template <bool FAST>
using HqVal = typename std::conditional<FAST, float, double>::type;

// A thread's window row: the values of columns c - 1, c, c + 1 (mirrored on image borders)
// of one region row, for u and v.
template <bool FAST>
struct HqRow {
  HqVal<FAST> ul, um, ur, vl, vm, vr;
};

template <int RW, bool FAST>
__device__ __forceinline__ void hq_load(HqRow<FAST>& R, const HqVal<FAST>* __restrict__ su,
                                        const HqVal<FAST>* __restrict__ sv, int row, int cm, int c, int cp) {
  const int o = row * RW;
  R.ul = su[o + cm];
  R.um = su[o + c];
  R.ur = su[o + cp];
  R.vl = sv[o + cm];
  R.vm = sv[o + c];
  R.vr = sv[o + cp];
}

// The float32 quotient num / den, correctly rounded, from rd = 1 / (double)den rounded to
// float64: RN32(RN64(num * rd)).  RN64(num * rd) lies within 2^-52 (relative) of num / den.
// A quotient of two float32 values is never that close to a midpoint m = M 2^e (M odd, 25
// bits) of two normal float32 neighbours unless it equals it, which it cannot: den * m would
// need 25 significant bits for num to have 24, and a non-zero num - den * m is a multiple of
// 2^e ulp(den), i.e. at least 2^-49 of m relative.  So the last rounding falls on the side of
// num / den (the innocuous-double-rounding argument of S. Figueroa, "When is double rounding
// innocuous?", SIGNUM Newsletter 30(3), 1995).  A midpoint of the subnormal range has fewer bits,
// and the quotient may equal it: there the product is first rounded to a multiple of 2^-177, which
// makes a quotient on a midpoint exact (its product is within 2^-179) and keeps any other, at
// least 2^-174 away, on its side.  Zeros, infinities and NaNs give IEEE's answers (rd = inf for
// den = 0, 0 for den = inf), and float64's range holds every product.  No branch: the rows of a
// sweep are one basic block the scheduler interleaves.
__device__ __forceinline__ float hq_div(float num, double rd) {
  const double q = __dmul_rn((double)num, rd), c = 0x1.8p-125, s = __dadd_rn(__dadd_rn(q, c), -c);
  // 2^-151 <= |q| < 2^-126, by the exponent
  const unsigned e = (unsigned)__double2hiint(q) & 0x7ff00000u;
  return __double2float_rn(e - ((1023u - 151u) << 20) < (25u << 20) ? s : q);
}

// The update of region cell i from its window rows U (above), C and D (below):
// hs_sweep_kernel's arithmetic, the 8 neighbours summed in its order.  RD: the quotient
// from the cell's float64 reciprocal srd[i] of the denominator (hq_div), else __fdiv_rn;
// both are the correctly rounded float32 quotient.
template <bool FAST, bool RD>
__device__ __forceinline__ void hq_cell(const HqRow<FAST>& U, const HqRow<FAST>& C, const HqRow<FAST>& D, int i,
                                        const float* __restrict__ sfx, const float* __restrict__ sfy,
                                        const float* __restrict__ sft, const double* __restrict__ srd, float a2,
                                        HqVal<FAST>& uo, HqVal<FAST>& vo) {
  float ua, va;
  if constexpr (FAST) {  // float32 averaging: corner and edge sums, one multiply-add each
    const float wcf = 1.0f / 12.0f, wef = 1.0f / 6.0f;
    const float cu = __fadd_rn(__fadd_rn(U.ul, U.ur), __fadd_rn(D.ul, D.ur));
    const float eu = __fadd_rn(__fadd_rn(U.um, D.um), __fadd_rn(C.ul, C.ur));
    const float cv = __fadd_rn(__fadd_rn(U.vl, U.vr), __fadd_rn(D.vl, D.vr));
    const float ev = __fadd_rn(__fadd_rn(U.vm, D.vm), __fadd_rn(C.vl, C.vr));
    ua = __fmaf_rn(cu, wcf, __fmul_rn(eu, wef));
    va = __fmaf_rn(cv, wcf, __fmul_rn(ev, wef));
  } else {
    const double wc = (double)(1.0f / 12.0f), we = (double)(1.0f / 6.0f);
    double a = 0.0, b = 0.0;  // float32 values held as float64: no conversions here
    a = __fma_rn(U.ul, wc, a); b = __fma_rn(U.vl, wc, b);
    a = __fma_rn(U.um, we, a); b = __fma_rn(U.vm, we, b);
    a = __fma_rn(U.ur, wc, a); b = __fma_rn(U.vr, wc, b);
    a = __fma_rn(C.ul, we, a); b = __fma_rn(C.vl, we, b);
    a = __fma_rn(C.ur, we, a); b = __fma_rn(C.vr, we, b);
    a = __fma_rn(D.ul, wc, a); b = __fma_rn(D.vl, wc, b);
    a = __fma_rn(D.um, we, a); b = __fma_rn(D.vm, we, b);
    a = __fma_rn(D.ur, wc, a); b = __fma_rn(D.vr, wc, b);
    ua = (float)a;
    va = (float)b;
  }
  const float gxv = sfx[i], gyv = sfy[i];
  const float num = __fadd_rn(__fadd_rn(__fmul_rn(gxv, ua), __fmul_rn(gyv, va)), sft[i]);
  float der;
  if constexpr (RD) {
    der = hq_div(num, srd[i]);
  } else {
    const float den = __fadd_rn(__fadd_rn(a2, __fmul_rn(gxv, gxv)), __fmul_rn(gyv, gyv));
    der = __fdiv_rn(num, den);
  }
  uo = (HqVal<FAST>)__fsub_rn(ua, __fmul_rn(gxv, der));
  vo = (HqVal<FAST>)__fsub_rn(va, __fmul_rn(gyv, der));
}

// The float64 reciprocal of a cell's denominator a2 + fx^2 + fy^2 (float32 operations in
// hs_sweep_kernel's order), for hq_div.
__device__ __forceinline__ double hq_recip_den(float gx, float gy, float a2) {
  const float den = __fadd_rn(__fadd_rn(a2, __fmul_rn(gx, gx)), __fmul_rn(gy, gy));
  return __drcp_rn((double)den);
}

template <bool FAST>
__device__ __forceinline__ void hq_update(const HqRow<FAST>& U, const HqRow<FAST>& C, const HqRow<FAST>& D, int i,
                                          const float* __restrict__ sfx, const float* __restrict__ sfy,
                                          const float* __restrict__ sft, HqVal<FAST>* __restrict__ du,
                                          HqVal<FAST>* __restrict__ dv, float a2) {
  hq_cell<FAST, false>(U, C, D, i, sfx, sfy, sft, nullptr, a2, du[i], dv[i]);
}

// K consecutive rows r0 .. r0 + K - 1 of a thread's column in one basic block: rows r0 - 1
// .. r0 + K are loaded, the K cells computed and stored, so the scheduler overlaps the
// rows' float64 chains instead of running them one after another.
template <int RW, int K, bool EDGE, bool FAST, bool RD, class RowOf>
__device__ __forceinline__ void hq_rows(const float* __restrict__ sfx, const float* __restrict__ sfy,
                                        const float* __restrict__ sft, const double* __restrict__ srd,
                                        const HqVal<FAST>* __restrict__ su, const HqVal<FAST>* __restrict__ sv,
                                        HqVal<FAST>* __restrict__ du, HqVal<FAST>* __restrict__ dv, int r0, int cm,
                                        int c, int cp, float a2, const RowOf& row_of) {
  HqRow<FAST> w[K + 2];
#pragma unroll
  for (int j = 0; j < K + 2; j++) hq_load<RW, FAST>(w[j], su, sv, row_of(r0 - 1 + j), cm, c, cp);
#pragma unroll
  for (int j = 0; j < K; j++) {
    const int i = (r0 + j) * RW + c;
    hq_cell<FAST, RD>(w[j], w[j + 1], w[j + 2], i, sfx, sfy, sft, srd, a2, du[i], dv[i]);
  }
}

// Sweep s of the region: thread t owns column t % RW and a band of the rows the sweep computes
// (band t / RW of NT / RW, NT the CTA's threads), walked in chunks of up to HQ_CHUNK rows
// (hq_rows).  A band is a whole number of warps (RW a multiple of 32), so the chunk lengths are
// warp-uniform.  The input and output buffers are distinct (ping-pong), so the pointers are
// restrict.  On image borders the neighbour columns and the outer rows go through the 'mirror'
// map; inside the image the mapped row is the row.  RD as in hq_cell.
constexpr int HQ_CHUNK = 4;

template <int RW, int RH, int T, bool EDGE, bool FAST, int NT, bool RD>
__device__ __forceinline__ void hq_sweep2(const float* __restrict__ sfx, const float* __restrict__ sfy,
                                          const float* __restrict__ sft, const double* __restrict__ srd,
                                          const HqVal<FAST>* __restrict__ su, const HqVal<FAST>* __restrict__ sv,
                                          HqVal<FAST>* __restrict__ du, HqVal<FAST>* __restrict__ dv, int s, int x0,
                                          int y0, int H, int W, float a2) {
  static_assert(NT % RW == 0 && RW % 32 == 0, "whole bands of whole warps");
  constexpr int NB = NT / RW;
  const int c = (int)threadIdx.x % RW, band = (int)threadIdx.x / RW;
  if (c < 1 + s || c >= RW - 1 - s) return;
  const int gx = x0 - T + c;
  if (EDGE && (gx < 0 || gx >= W)) return;
  int cm = c - 1, cp = c + 1;
  if (EDGE) {
    cm = mirror1(gx - 1, W) - (x0 - T);
    cp = mirror1(gx + 1, W) - (x0 - T);
  }
  int lo = 1 + s, hi = RH - 1 - s;
  if (EDGE) {
    lo = max(lo, T - y0);
    hi = min(hi, H + T - y0);
  }
  const int n = hi - lo;
  if (n <= 0) return;
  const int ra = lo + (n * band) / NB, rb = lo + (n * (band + 1)) / NB;
  auto row_of = [&](int r) { return EDGE ? mirror1(y0 - T + r, H) - (y0 - T) : r; };
#pragma unroll 1
  for (int r0 = ra; r0 < rb; r0 += HQ_CHUNK) {
    switch (min(HQ_CHUNK, rb - r0)) {
      case 4: hq_rows<RW, 4, EDGE, FAST, RD>(sfx, sfy, sft, srd, su, sv, du, dv, r0, cm, c, cp, a2, row_of); break;
      case 3: hq_rows<RW, 3, EDGE, FAST, RD>(sfx, sfy, sft, srd, su, sv, du, dv, r0, cm, c, cp, a2, row_of); break;
      case 2: hq_rows<RW, 2, EDGE, FAST, RD>(sfx, sfy, sft, srd, su, sv, du, dv, r0, cm, c, cp, a2, row_of); break;
      default: hq_rows<RW, 1, EDGE, FAST, RD>(sfx, sfy, sft, srd, su, sv, du, dv, r0, cm, c, cp, a2, row_of); break;
    }
  }
}

// ---- Register-blocked sweep (bit-exact arithmetic) ---------------------------------------
// A thread owns a BX x BY block of region cells and keeps their (u, v), as float64 copies of
// the float32 values, and their derivatives in registers through all sweeps of a pass; a sweep
// exchanges the cells through shared memory (all of them: one side of a block is 2).  A cell update
// then writes 16 bytes and reads 48 at 2 x 2, 32 at 2 x 4, where a column walk writes 16 and reads 72.
// The exchange buffer holds region cell (r, c) as a double2 (u, v) at [r][c % BX][c / BX], so
// that the threads of a row, BX cells apart, access consecutive 16-byte words.
template <int RW, int RH, int BX, int BY>
struct HrGeom {
  static_assert(RW % BX == 0 && RH % BY == 0, "whole blocks");
  static constexpr int NX = RW / BX, NY = RH / BY, NT = NX * NY;
  static constexpr size_t BUF = (size_t)RW * RH * sizeof(double2);
  static __device__ __forceinline__ int at(int r, int c) { return r * RW + (c % BX) * NX + c / BX; }
};

// One window row of a block: its BX cells and the cell to either side.
template <int BX>
struct HrRow {
  double u[BX + 2], v[BX + 2];
};

template <int BX, int BY>
struct HrBlock {
  double u[BY][BX], v[BY][BX];
  float2 g[BY][BX];    // spatial derivatives (fx, fy)
  float gt[BY][BX];    // temporal derivative
  float y[BY][BX];     // 1 / den, correctly rounded
  static constexpr bool DEN = BX * BY <= 4;  // a small block has registers for the denominators too
  float den[DEN ? BY : 1][DEN ? BX : 1];
  float a2;            // alpha^2
  float one;           // 1.0f, unknown to the assembler (see hr_row)
  unsigned lo;         // range of the numerators seen: smallest 2 |num| (bits) - 1
  float hi;            // and largest |num|
};

// Where the quotient by refinement (hr_div) is the correctly rounded one: for den in [2^-40,
// 2^40] and |num| in [2^-80, 2^60] no intermediate leaves the normal range and the residuals
// are exact (multiples of 2^-47 |num|; the quotients are at least 2^-120); and for num = +0,
// which is what a zero numerator is unless gt is -0.
constexpr float HR_DEN = 0x1p40f, HR_NUM = 0x1p60f;
constexpr unsigned HR_LO = 2u * 0x17800000u - 1u;  // 2^-80

__device__ __forceinline__ float hr_max_nan(float a, float b) {  // NaN if either is
  float r;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}

__device__ __forceinline__ float hr_den(float2 g, float a2) {
  const float2 q = __fmul2_rn(g, g);
  return __fadd_rn(__fadd_rn(a2, q.x), q.y);
}

enum HrQuot { HR_REFINED, HR_WIDE, HR_DIVIDE };  // see hr_row

template <int BX, int BY>
__device__ __forceinline__ void hr_reset_range(HrBlock<BX, BY>& K) {
  K.lo = 0xffffffffu;
  K.hi = 0.f;
}

// The block's reciprocals; false when a denominator or gt is outside the ranges above.
template <int BX, int BY>
__device__ __forceinline__ bool hr_init_den(HrBlock<BX, BY>& K, float a2, float one) {
  K.a2 = a2;
  K.one = one;
  hr_reset_range(K);
  bool ok = true;
#pragma unroll
  for (int j = 0; j < BY; j++)
#pragma unroll
    for (int i = 0; i < BX; i++) {
      const float den = hr_den(K.g[j][i], a2);
      ok = ok && den >= 1.f / HR_DEN && den <= HR_DEN && __float_as_uint(K.gt[j][i]) != 0x80000000u;
      K.y[j][i] = __frcp_rn(den);
      if constexpr (HrBlock<BX, BY>::DEN) K.den[j][i] = den;
    }
  return ok;
}

// Whether every numerator since the last reset was in the range of quotient q (HR_REFINED or HR_WIDE).
template <int BX, int BY>
__device__ __forceinline__ bool hr_in_range(const HrBlock<BX, BY>& K, int q) {
  return (K.lo >= HR_LO || q == HR_WIDE) && K.hi <= HR_NUM;
}

// num / den by two residual corrections of num * y, y = 1 / den correctly rounded; the last is
// correctly rounded (P. Markstein, "Computation of elementary functions on the IBM RISC System/6000
// processor", IBM J. Res. Develop. 34(1), 1990) for operands in the ranges above.
__device__ __forceinline__ float hr_div(float num, float den, float y) {
  float q = __fmul_rn(num, y);
  q = __fmaf_rn(__fmaf_rn(-q, den, num), y, q);
  return __fmaf_rn(__fmaf_rn(-q, den, num), y, q);
}

// The same for |num| down to the smallest subnormal.  A numerator below 2^-60 is divided at 2^64
// times its size, which is exact.  So is the way back unless the quotient is subnormal: there it is a
// second rounding, wrong where the first one's result lies midway between two subnormal numbers and
// its residual points to the other one.  No branch, and no divide, which is slow for such operands.
__device__ __forceinline__ float hr_div_wide(float num, float den, float y) {
  const bool tiny = fabsf(num) < 0x1p-60f;
  const float up = tiny ? 0x1p64f : 1.f, down = tiny ? 0x1p-64f : 1.f;
  const float n = __fmul_rn(num, up), q = hr_div(n, den, y), der = __fmul_rn(q, down);
  const float e = __fmaf_rn(der, up, -q), r = __fmaf_rn(-q, den, n);  // exact; e: what the way back added
  const float fix = e == 0x1p-86f && r < 0.f ? -0x1p-149f : e == -0x1p-86f && r > 0.f ? 0x1p-149f : 0.f;
  return fix != 0.f ? __fadd_rn(der, fix) : der;
}

// The update of a block's row j from the old window rows U (above), C, D (below):
// hs_sweep_kernel's arithmetic, the 8 neighbours summed in its order; the results replace the
// block's cells.  The quotient by Q; the range of the numerators is only recorded here, for one check
// per pass, and a CTA that fails it repeats the pass with the next Q:
//   HR_REFINED  hr_div
//   HR_WIDE     hr_div_wide.  Tiny numerators are common where both frames show the same texture:
//               the flow that diffuses in shrinks by a factor of 6 to 12 a cell, down to the
//               subnormal numbers.  So a CTA that has reason to expect them (its last pass, or the
//               flow it starts from) begins with this one.  256 x 256, 600 sweeps, one half the
//               same texture in both frames: 0.60 ms (0.54 where no numerator is tiny); every such
//               pass run again with the divide 1.99, with this one's scaling but the divide for
//               subnormal quotients 1.76, in float64 0.60 but 5 % on every pass of hs.cu in spills.
//   HR_DIVIDE   __fdiv_rn, for all operands.
template <int BX, int BY, int Q>
__device__ __forceinline__ void hr_row(HrBlock<BX, BY>& K, int j, const HrRow<BX>& U, const HrRow<BX>& C,
                                       const HrRow<BX>& D) {
  const double wc = (double)(1.0f / 12.0f), we = (double)(1.0f / 6.0f);
#pragma unroll
  for (int i = 0; i < BX; i++) {
    double a = 0.0, b = 0.0;  // float32 values held as float64: no conversions here
    a = __fma_rn(U.u[i], wc, a);     b = __fma_rn(U.v[i], wc, b);
    a = __fma_rn(U.u[i + 1], we, a); b = __fma_rn(U.v[i + 1], we, b);
    a = __fma_rn(U.u[i + 2], wc, a); b = __fma_rn(U.v[i + 2], wc, b);
    a = __fma_rn(C.u[i], we, a);     b = __fma_rn(C.v[i], we, b);
    a = __fma_rn(C.u[i + 2], we, a); b = __fma_rn(C.v[i + 2], we, b);
    a = __fma_rn(D.u[i], wc, a);     b = __fma_rn(D.v[i], wc, b);
    a = __fma_rn(D.u[i + 1], we, a); b = __fma_rn(D.v[i + 1], we, b);
    a = __fma_rn(D.u[i + 2], wc, a); b = __fma_rn(D.v[i + 2], wc, b);
    const float2 m = make_float2((float)a, (float)b), g = K.g[j][i];
    const float2 gm = __fmul2_rn(g, m);
    const float num = __fadd_rn(__fadd_rn(gm.x, gm.y), K.gt[j][i]);
    float den;
    if constexpr (HrBlock<BX, BY>::DEN)
      den = K.den[j][i];
    else
      den = hr_den(g, K.a2);
    const float der = Q == HR_REFINED ? hr_div(num, den, K.y[j][i])
                      : Q == HR_WIDE  ? hr_div_wide(num, den, K.y[j][i])
                                      : __fdiv_rn(num, den);
    K.lo = min(K.lo, 2u * __float_as_uint(num) - 1u);
    K.hi = hr_max_nan(K.hi, fabsf(num));
    // m - g der with two roundings: the assembler would fuse a packed product into a packed
    // sum, so the product goes through a multiply-add by minus one that it cannot see
    const float2 r = __ffma2_rn(__fmul2_rn(g, make_float2(der, der)), make_float2(-K.one, -K.one), m);
    K.u[j][i] = (double)r.x;
    K.v[j][i] = (double)r.y;
  }
}

// The block's boundary cells into the exchange buffer (r0, c0: its first region cell).
template <int RW, int RH, int BX, int BY>
__device__ __forceinline__ void hr_publish(const HrBlock<BX, BY>& K, double2* buf, int r0, int c0) {
  using G = HrGeom<RW, RH, BX, BY>;
#pragma unroll
  for (int j = 0; j < BY; j++)
#pragma unroll
    for (int i = 0; i < BX; i++)
      if (j == 0 || j == BY - 1 || i == 0 || i == BX - 1)
        buf[r0 * RW + c0 / BX + j * RW + i * G::NX] = make_double2(K.u[j][i], K.v[j][i]);
}

// Where a block finds its window in the exchange buffer.  Neighbours beyond an image border are
// the mirror cells (-1 shows 1, n shows n - 2), which is only another index: every cell is
// published (BX or BY is 2), and with blocks aligned to the image's first row and column
// (T a multiple of BX and BY) a border lies between blocks, except the last row or column of an
// image whose sides are no multiple of the block.  There the neighbour is an outside cell of
// the block itself, and hr_sweep's RAG form takes the cell on the other side instead.
// Neighbours beyond the region are held at its rim.  H, W >= 2.
struct HrWin {
  int cl, cr;  // columns beside the block, as offsets in a row
  int rt, rb;  // row offsets above and below it
  int jr, ir;  // RAG: the block's last row and column in the image when others follow, else -1
};

template <int RW, int RH, int BX, int BY>
__device__ __forceinline__ HrWin hr_window(int r0, int c0, int gy0, int gx0, int H, int W) {
  static_assert(BX == 2 || BY == 2, "every cell of a block is published");
  using G = HrGeom<RW, RH, BX, BY>;
  HrWin w;
  const int l = gx0 == 0 ? c0 + 1 : (c0 > 0 ? c0 - 1 : 0);
  const int r = gx0 + BX == W ? c0 + BX - 2 : (c0 + BX < RW ? c0 + BX : RW - 1);
  w.cl = G::at(0, l);
  w.cr = G::at(0, r);
  w.rt = (gy0 == 0 ? r0 + 1 : (r0 > 0 ? r0 - 1 : 0)) * RW;
  w.rb = (gy0 + BY == H ? r0 + BY - 2 : (r0 + BY < RH ? r0 + BY : RH - 1)) * RW;
  w.jr = gy0 + BY > H ? H - 1 - gy0 : -1;
  w.ir = gx0 + BX > W ? W - 1 - gx0 : -1;
  return w;
}

// One sweep of the block from the exchange buffer `buf` (the other blocks' cells before the
// sweep).  Cells outside the image or on the region's rim get values that no exact cell reads.
template <int RW, int RH, int BX, int BY, bool RAG, int Q>
__device__ __forceinline__ void hr_sweep(HrBlock<BX, BY>& K, const double2* buf, int r0, int c0, const HrWin& win) {
  using G = HrGeom<RW, RH, BX, BY>;
  const int cb = c0 / BX;
  auto fix = [&](HrRow<BX>& R) {
    if constexpr (RAG) {
#pragma unroll
      for (int i = 0; i + 1 < BX; i++) {
        const bool p = win.ir == i;
        R.u[i + 2] = p ? R.u[i] : R.u[i + 2];
        R.v[i + 2] = p ? R.v[i] : R.v[i + 2];
      }
    }
  };
  auto ring = [&](HrRow<BX>& R, int row) {  // a row above or below the block
    const double2* b = buf + row;
    double2 t = b[win.cl];
    R.u[0] = t.x;
    R.v[0] = t.y;
#pragma unroll
    for (int i = 0; i < BX; i++) {
      t = b[i * G::NX + cb];
      R.u[i + 1] = t.x;
      R.v[i + 1] = t.y;
    }
    t = b[win.cr];
    R.u[BX + 1] = t.x;
    R.v[BX + 1] = t.y;
    fix(R);
  };
  auto own = [&](HrRow<BX>& R, int j) {  // the block's row j with the cells beside it
    const double2* b = buf + (r0 + j) * RW;
    const double2 l = b[win.cl], r = b[win.cr];
    R.u[0] = l.x;
    R.v[0] = l.y;
#pragma unroll
    for (int i = 0; i < BX; i++) {
      R.u[i + 1] = K.u[j][i];
      R.v[i + 1] = K.v[j][i];
    }
    R.u[BX + 1] = r.x;
    R.v[BX + 1] = r.y;
    fix(R);
  };
  HrRow<BX> w[3];
  ring(w[0], win.rt);
  own(w[1], 0);
#pragma unroll
  for (int j = 0; j < BY; j++) {
    HrRow<BX>&U = w[j % 3], &C = w[(j + 1) % 3], &D = w[(j + 2) % 3];
    if (j + 1 < BY)
      own(D, j + 1);
    else
      ring(D, win.rb);
    if (RAG && j + 1 < BY) {
      const bool p = win.jr == j;
      HrRow<BX> M;
#pragma unroll
      for (int i = 0; i < BX + 2; i++) {
        M.u[i] = p ? U.u[i] : D.u[i];
        M.v[i] = p ? U.v[i] : D.v[i];
      }
      hr_row<BX, BY, Q>(K, j, U, C, M);
    } else {
      hr_row<BX, BY, Q>(K, j, U, C, D);
    }
  }
}

}  // namespace ofb
