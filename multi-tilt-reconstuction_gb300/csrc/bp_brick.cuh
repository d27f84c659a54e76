// Device side of the TMA-windowed back-projection (bp_tma.cu, bp_pairs.cu):
// the brick routine, its kernel and the templated launch helpers.  Included by
// the two translation units that instantiate the FP32-window and the
// residual-pair variants, so that they compile in parallel.
#pragma once

#include <algorithm>
#include <atomic>
#include <type_traits>

#include "mtr_internal.h"
#include "tma.cuh"

namespace mtr {

// Arguments of one windowed back-projection launch (shared by both units).
struct BpArgs {
  AxisDev ax;
  VolDev vol;
  int z0, z1;
  int WX, WY;       // window box (elements)
  int align;        // TMA x alignment (elements)
  int mode;         // 0 WBP, 1 SIRT
  float step;
  float* vol_out;
  float* cbp;
  void* vol_copy;
  int copy_kind;
  int* err;
  unsigned wait_iters;  // polls of a pipeline wait before it gives up
};

// The SIRT update over residual-pair windows (bp_pairs.cu).
cudaError_t launch_backproject_tma_pairs(const CUtensorMap& map, const BpPlan& plan, const BpArgs& P,
                                         cudaStream_t st);
// WBP and SIRT update over windows of plain rows (bp_rows.cu).
cudaError_t launch_backproject_tma_rows(const CUtensorMap& map, const BpPlan& plan, const BpArgs& P,
                                        cudaStream_t st);

namespace {

constexpr int NST = 4;             // pipeline stages
constexpr int kConsumerWarps = 8;  // 256 consumer threads
constexpr int kThreads = (kConsumerWarps + 1) * 32;
// Polls of the pipeline waits (producer on a free stage, consumers on a
// loaded window) before they give up are a launch argument, so that a test
// can make them give up at once.  The drain of the producer's own copies in
// flight always has the full bound: a CTA never exits with a copy pending.
constexpr uint32_t kDrainIters = 1u << 24;
constexpr float kMagic = 12582912.0f;  // 1.5 * 2^23: x + kMagic holds round(x) in its low bits
constexpr int kMagicBits = 0x4B400000;

struct __align__(16) WinConst {
  float xf, a1, a2, a3;  // x map relative to the CTA base voxel (fractional base)
  float yf, b1, b2, b3;
  int lxm, lym;          // window-local integer base minus the magic bits
  int ox, oy;            // window origin on the detector (ox aligned for TMA)
  int flags, pad[3];     // row pairs: kHolds, kOnDetector
};
// The window holds every tap of the brick at this angle (else the plan is wrong:
// the angle is skipped and the launch flagged); every tap lies on the detector.
constexpr int kHolds = 1, kOnDetector = 2;

// A fractional base that the clamp to +-1e9 px left large: the position is
// beyond what its integer part and the windows' float arithmetic hold.
__device__ __forceinline__ bool far(float f) { return !(fabsf(f) <= 65536.f); }
__device__ __forceinline__ int floor_div(int a, int b) { return (a >= 0) ? a / b : -((-a + b - 1) / b); }

__device__ __forceinline__ int magic_int(float integral) { return __float_as_int(__fadd_rn(integral, kMagic)); }

// Shared-memory loads at a 32-bit shared address plus a constant byte offset:
// the column gathers step their tap address in this form (one 32-bit add per
// pixel crossed) instead of a generic pointer.  Volatile keeps them after the
// pipeline's mbarrier waits.
template <int OFF> __device__ __forceinline__ float lds_f32(uint32_t a) {
  float v;
  asm volatile("ld.shared.f32 %0, [%1+%2];" : "=f"(v) : "r"(a), "n"(OFF));
  return v;
}
template <int OFF> __device__ __forceinline__ float2 lds_f32x2(uint32_t a) {
  float2 v;
  asm volatile("ld.shared.v2.f32 {%0, %1}, [%2+%3];" : "=f"(v.x), "=f"(v.y) : "r"(a), "n"(OFF));
  return v;
}
template <int OFF> __device__ __forceinline__ float2 lds_h2_widened(uint32_t a) {
  __half2 h;
  asm volatile("ld.shared.b32 %0, [%1+%2];" : "=r"(*reinterpret_cast<unsigned*>(&h)) : "r"(a), "n"(OFF));
  return __half22float2(h);
}

// Gather of one voxel column (fixed X, Y; y-map without a Z term) from a row of
// row pairs (`row0`: elements (r[y], r[y + 1]) of one detector row), adding
// into s[0..NZ).  x advances by |a3| < 1 per voxel.  The column carries the
// y-interpolated value at its current pixel (B0) and the step to the next (D),
// so a voxel costs two operations beside its fraction, and a pixel is loaded
// (one 8-byte load for both rows, a crossing ahead of its use) and interpolated
// in y once per pixel entered instead of at every voxel.  Some lane of a warp
// crosses at almost every voxel, so the crossing is a few predicated
// instructions and the load is not conditional (the next pixel's again where
// the column stayed).  Bound by issue, 12 instructions a voxel where the four
// taps took 17: 512x512x64 at 60 degrees, 61 angles, 0.52 against 0.70 ms; WBP
// 0.55 against 0.89 ms.  The walk
// runs z upwards; where a3 < 0 in the mirrored coordinate u = -x, whose pixels
// p and p + 1 are the window's columns -p and -p - 1, so that one copy of the
// code serves both signs.  Rounding of the stepped fraction stays below 4e-6 px
// over 32 voxels; the window has one pixel of slack for it.
//
// ROWS: the window holds plain rows of `pitch` pixels and a pixel of both rows is
// two 4-byte loads, one instruction more a voxel and half the shared memory.
template <int NZ, bool ROWS, typename WT>
__device__ __forceinline__ void bp_column_rows(float (&s)[NZ], const WT* row0, int pitch, float xr, float a3, int lxm,
                                               float fy) {
  const bool up = a3 >= 0.f;
  const float u = up ? xr : -xr;
  const float tu = __fadd_rd(u, kMagic);  // floor, in the low bits
  float fx = u - (tu - kMagic);
  const float step = fabsf(a3);
  const int pix = __float_as_int(tu) - kMagicBits;
  constexpr uint32_t kEs = ROWS ? 4u : 8u;
  const uint32_t dp = up ? kEs : 0u - kEs;
  uint32_t p = smem_u32(row0) + kEs * (uint32_t)((lxm + kMagicBits) + (up ? pix : -pix));
  const uint32_t dr = 4u * (uint32_t)pitch;
  auto pixel = [&](uint32_t q) {
    if constexpr (ROWS) return make_float2(lds_f32<0>(q), lds_f32<0>(q + dr));
    else return lds_f32x2<0>(q);
  };
  const float2 q0 = pixel(p), q1 = pixel(p + dp);
  p += 2u * dp;
  float2 n = pixel(p);  // the pixel after the next (not used unless the column reaches it)
  float b0 = fmaf(fy, q0.y - q0.x, q0.x), b1 = fmaf(fy, q1.y - q1.x, q1.x);
  float d = b1 - b0;
#pragma unroll
  for (int z = 0; z < NZ; ++z) {
    if (z > 0) {
      fx += step;
      if (fx >= 1.f) {
        fx -= 1.f;
        b0 = b1;
        b1 = fmaf(fy, n.y - n.x, n.x);
        p += dp;
      }
      d = b1 - b0;
      n = pixel(p);
    }
    s[z] = fmaf(fx, d, s[z] + b0);
  }
}

// The SIRT update's windows hold (value, next value - value) pairs of the
// residual (residual_pairs_kernel): a tap pair of one detector row is one
// 8-byte load and its x interpolation one FFMA.
template <bool ASC, int NZ>
__device__ __forceinline__ void bp_column(float (&s)[NZ], const float2* row0, int WX, float xr, float a3, int lxm,
                                          float wy0, float wy1) {
  constexpr int zf = ASC ? 0 : NZ - 1;
  const float x = fmaf(a3, (float)zf, xr);
  const float flx = floorf(x);
  float fx = x - flx;
  const float step = fabsf(a3);
  uint32_t p = smem_u32(row0) + 8u * (uint32_t)(magic_int(flx) + lxm);
  const uint32_t dr = 8u * (uint32_t)WX;
#pragma unroll
  for (int i = 0; i < NZ; ++i) {
    const int z = ASC ? i : NZ - 1 - i;
    if (i > 0) {
      fx += step;
      const bool adv = fx >= 1.f;
      fx = adv ? fx - 1.f : fx;
      p += adv ? 8u : 0u;
    }
    const float2 q0 = lds_f32x2<0>(p), q1 = lds_f32x2<0>(p + dr);
    s[z] = fmaf(wy0, fmaf(fx, q0.y, q0.x), s[z]);
    s[z] = fmaf(wy1, fmaf(fx, q1.y, q1.x), s[z]);
  }
}

// The same from planar pair windows: a detector row's values, then its
// differences, WX floats each, so a voxel's row r reads p[0] and p[WX] and
// row r + 1 reads p[2 WX] and p[3 WX] (four 4-byte loads, two FFMAs).
template <bool ASC, int NZ>
__device__ __forceinline__ void bp_column_planar(float (&s)[NZ], const float* row0, int WX, float xr, float a3,
                                                 int lxm, float wy0, float wy1) {
  constexpr int zf = ASC ? 0 : NZ - 1;
  const float x = fmaf(a3, (float)zf, xr);
  const float flx = floorf(x);
  float fx = x - flx;
  const float step = fabsf(a3);
  uint32_t p = smem_u32(row0) + 4u * (uint32_t)(magic_int(flx) + lxm);
  const uint32_t d1 = 4u * (uint32_t)WX, d2 = 2u * d1, d3 = 3u * d1;
#pragma unroll
  for (int i = 0; i < NZ; ++i) {
    const int z = ASC ? i : NZ - 1 - i;
    if (i > 0) {
      fx += step;
      const bool adv = fx >= 1.f;
      fx = adv ? fx - 1.f : fx;
      p += adv ? 4u : 0u;
    }
    s[z] = fmaf(wy0, fmaf(fx, lds_f32<0>(p + d1), lds_f32<0>(p)), s[z]);
    s[z] = fmaf(wy1, fmaf(fx, lds_f32<0>(p + d3), lds_f32<0>(p + d2)), s[z]);
  }
}

// The same from FP16 pair windows (mixed precision): a detector row's tap
// pair is one 4-byte load of (value, next - value) in FP16, widened to FP32
// before the interpolation.  Half the shared-memory bytes of the FP32 formats.
template <bool ASC, int NZ>
__device__ __forceinline__ void bp_column_half(float (&s)[NZ], const __half2* row0, int WX, float xr, float a3,
                                               int lxm, float wy0, float wy1) {
  constexpr int zf = ASC ? 0 : NZ - 1;
  const float x = fmaf(a3, (float)zf, xr);
  const float flx = floorf(x);
  float fx = x - flx;
  const float step = fabsf(a3);
  uint32_t p = smem_u32(row0) + 4u * (uint32_t)(magic_int(flx) + lxm);
  const uint32_t dr = 4u * (uint32_t)WX;
#pragma unroll
  for (int i = 0; i < NZ; ++i) {
    const int z = ASC ? i : NZ - 1 - i;
    if (i > 0) {
      fx += step;
      const bool adv = fx >= 1.f;
      fx = adv ? fx - 1.f : fx;
      p += adv ? 4u : 0u;
    }
    const float2 q0 = lds_h2_widened<0>(p), q1 = lds_h2_widened<0>(p + dr);
    s[z] = fmaf(wy0, fmaf(fx, q0.y, q0.x), s[z]);
    s[z] = fmaf(wy1, fmaf(fx, q1.y, q1.x), s[z]);
  }
}

// The same column gather from a row pre-blended by the warp: b[i] holds the
// y-interpolated pair of window column i.
template <bool ASC, int NZ>
__device__ __forceinline__ void bp_column_blended(float (&s)[NZ], const float2* b, float xr, float a3, int lxm) {
  constexpr int zf = ASC ? 0 : NZ - 1;
  const float x = fmaf(a3, (float)zf, xr);
  const float flx = floorf(x);
  float fx = x - flx;
  const float step = fabsf(a3);
  uint32_t p = smem_u32(b) + 8u * (uint32_t)(magic_int(flx) + lxm);
#pragma unroll
  for (int i = 0; i < NZ; ++i) {
    const int z = ASC ? i : NZ - 1 - i;
    if (i > 0) {
      fx += step;
      const bool adv = fx >= 1.f;
      fx = adv ? fx - 1.f : fx;
      p += adv ? 8u : 0u;
    }
    const float2 q = lds_f32x2<0>(p);
    s[z] += fmaf(fx, q.y, q.x);
  }
}

// A column whose y-map has a Z term and whose taps all lie in the window: a
// position, its floor (one addition that rounds down) and its fraction per
// coordinate and voxel, and the taps without a check of their own.
template <int NZ, bool PAIR, bool HALF, typename WT>
__device__ __forceinline__ void bp_column_zy(float (&s)[NZ], const WT* win, int WX, float xr, float yr,
                                             const WinConst& k) {
  const uint32_t base = smem_u32(win);
  const uint32_t es = sizeof(WT), dr = es * (uint32_t)WX;
#pragma unroll
  for (int z = 0; z < NZ; ++z) {
    asm volatile("" : "+f"(xr), "+f"(yr));  // (one voxel's position at a time: no registers for all of them)
    const float x = fmaf(k.a3, (float)z, xr), y = fmaf(k.b3, (float)z, yr);
    const float tx = __fadd_rd(x, kMagic), ty = __fadd_rd(y, kMagic);  // floor, in the low bits
    const float fx = x - (tx - kMagic), fy = y - (ty - kMagic);
    const uint32_t p = base + es * (uint32_t)((__float_as_int(ty) + k.lym) * WX + (__float_as_int(tx) + k.lxm));
    float r0, r1;
    if constexpr (HALF) {
      const float2 q0 = lds_h2_widened<0>(p), q1 = lds_h2_widened<0>(p + dr);
      r0 = fmaf(fx, q0.y, q0.x);
      r1 = fmaf(fx, q1.y, q1.x);
    } else if constexpr (PAIR) {
      const float2 q0 = lds_f32x2<0>(p), q1 = lds_f32x2<0>(p + dr);
      r0 = fmaf(fx, q0.y, q0.x);
      r1 = fmaf(fx, q1.y, q1.x);
    } else if constexpr (sizeof(WT) == 4) {  // plain rows
      const float p00 = lds_f32<0>(p), p10 = lds_f32<4>(p), p01 = lds_f32<0>(p + dr), p11 = lds_f32<4>(p + dr);
      r0 = fmaf(fx, p10 - p00, p00);
      r1 = fmaf(fx, p11 - p01, p01);
    } else {
      const float2 q0 = lds_f32x2<0>(p), q1 = lds_f32x2<8>(p);  // both rows at two pixels
      r0 = fmaf(fx, q1.x - q0.x, q0.x);
      r1 = fmaf(fx, q1.y - q0.y, q0.y);
    }
    s[z] = fmaf(fy, r1 - r0, s[z] + r0);
  }
}

// Weight of a coordinate's two taps that lie on [0, n) (off: its integer base
// minus the magic bits).
__device__ __forceinline__ float tap_weight(float x, int off, int n) {
  const float t = __fadd_rd(x, kMagic);
  const float f = x - (t - kMagic);
  const int i = __float_as_int(t) + off;
  const bool in0 = (unsigned)i < (unsigned)n, in1 = (unsigned)(i + 1) < (unsigned)n;
  return in0 ? (in1 ? 1.f : 1.f - f) : in1 ? f : 0.f;
}

// One brick (bx, by, bz) of one axis.  LANES: 0 = each warp a line of 32
// voxels along X (brick 32x8), 1 = a line along Y (brick 8x32, used when the
// detector x follows Y), 2 = an 8x4 patch (on oblique axes the taps of a line
// fall on a diagonal of the window that maps several lanes to one shared-memory
// bank; a patch keeps them compact).  Patches fill a 16x16 square, the smallest
// footprint, or with the smaller elements of pairs along x a 32x8 brick (FP16
// pairs, 512x512x64 at 60 degrees: 0.60 against 0.63 ms; row pairs 0.52).  `smem` is the CTA's
// dynamic shared memory; `reinit` re-initialises the mbarriers of a CTA that
// already ran a brick.  PF (pair format, with PAIR): 0 interleaved FP32
// pairs; 1 planar FP32 pairs, each detector row as two FP32 rows, its values
// and then its differences; 2 FP16 pairs (value, next - value) in 32 bits.
// Without PAIR: 0 row pairs, 3 plain rows.
template <typename PT, int MODE, bool PAIR, int LANES, bool BZ0, int NZ, int PF = 0>
__device__ __forceinline__ void bp_brick(const CUtensorMap* tmap, const BpArgs& P, int bx, int by, int bz,
                                         unsigned char* smem, bool reinit) {
  constexpr int BX = bp_brick_x(LANES, PAIR), BY = bp_brick_y(LANES, PAIR);
  // Windows hold row pairs (of the residual, or for the WBP of the
  // projections), an element (x, y) the pixels (x, y) and (x, y + 1), or its plain
  // rows; or, with PAIR, residual pairs along x (value, next - value), one per pixel, from a
  // pair array whose column c is pixel c - 1.
  static_assert(!PAIR || MODE == 1, "residual pairs feed the SIRT update only");
  constexpr bool PLANAR = PAIR && PF == 1, HALF = PAIR && PF == 2, ROWS = !PAIR && PF == 3;
  static_assert(!PLANAR || BZ0, "planar windows are a pair format, for y-maps without a Z term");
  using WT = typename std::conditional<
      PLANAR || ROWS, float,
      typename std::conditional<HALF, __half2, float2>::type>::type;
  uint64_t* full = reinterpret_cast<uint64_t*>(smem);
  uint64_t* empty = full + NST;
  WinConst* kc = reinterpret_cast<WinConst*>(smem + 128);
  const int A = P.ax.A;
  const size_t kc_bytes = ((size_t)A * sizeof(WinConst) + 127) & ~(size_t)127;
  const int win_elems = P.WX * P.WY * (PLANAR ? 2 : 1);
  const size_t stage_bytes = (((size_t)win_elems * sizeof(WT)) + 127) & ~(size_t)127;
  WT* win0 = reinterpret_cast<WT*>(smem + 128 + kc_bytes);
  // per-warp blended row (uniform-row angles)
  float2* blend = reinterpret_cast<float2*>(smem + 128 + kc_bytes + NST * stage_bytes) + (threadIdx.x >> 5) * P.WX;

  const int tid = threadIdx.x;
  const int warp = tid >> 5, lane = tid & 31;
  const int X0 = P.vol.Xs + bx * BX;
  const int Y0 = P.vol.Ys + by * BY;
  const int Z0 = P.z0 + bz * NZ;

  if (tid == 0) {
    for (int s = 0; s < NST; ++s) {
      if (reinit) {
        mbar_inval(&full[s]);
        mbar_inval(&empty[s]);
      }
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], kConsumerWarps);
    }
    mbar_fence_init();
  }
  // Per-angle constants: FP64 map at the base voxel, split into int + float.
  for (int a = tid; a < A; a += kThreads) {
    const double* cx = P.ax.xc + 4 * a;
    const double* cy = P.ax.yc + 4 * a;
    const double xb = cx[0] + cx[1] * X0 + cx[2] * Y0 + cx[3] * Z0 - 1.0;
    const double yb = cy[0] + cy[1] * X0 + cy[2] * Y0 + cy[3] * Z0 - 1.0;
    const double fxb = floor(fmin(fmax(xb, -1.0e9), 1.0e9)), fyb = floor(fmin(fmax(yb, -1.0e9), 1.0e9));
    WinConst k;
    k.xf = (float)(xb - fxb);
    k.yf = (float)(yb - fyb);
    k.a1 = (float)cx[1]; k.a2 = (float)cx[2]; k.a3 = (float)cx[3];
    k.b1 = (float)cy[1]; k.b2 = (float)cy[2]; k.b3 = (float)cy[3];
    const int xi = (int)fxb, yi = (int)fyb;
    const float xmin = k.xf + fminf(0.f, k.a1 * (BX - 1)) + fminf(0.f, k.a2 * (BY - 1)) + fminf(0.f, k.a3 * (NZ - 1));
    const float ymin = k.yf + fminf(0.f, k.b1 * (BX - 1)) + fminf(0.f, k.b2 * (BY - 1)) + fminf(0.f, k.b3 * (NZ - 1));
    // leftmost tap pixel xi + floor(xmin) - 1; for pairs the window's first
    // pair column (pixel + 1) is rounded down to an even one (TMA alignment)
    const int ox = PAIR ? floor_div(xi + (int)floorf(xmin), P.align) * P.align - 1
                        : floor_div(xi + (int)floorf(xmin) - 1, P.align) * P.align;
    const int oy = yi + (int)floorf(ymin) - 1;
    k.ox = ox;
    k.oy = oy;
    k.lxm = xi - ox - kMagicBits;
    k.lym = yi - oy - kMagicBits;
    k.flags = 0;
    if (!PAIR) {
      const float xmax = k.xf + fmaxf(0.f, k.a1 * (BX - 1)) + fmaxf(0.f, k.a2 * (BY - 1)) + fmaxf(0.f, k.a3 * (NZ - 1));
      const float ymax = k.yf + fmaxf(0.f, k.b1 * (BX - 1)) + fmaxf(0.f, k.b2 * (BY - 1)) + fmaxf(0.f, k.b3 * (NZ - 1));
      // first and last tap, with a pixel of slack for the rounding of a thread's own position
      const int x0 = xi + (int)floorf(xmin) - 1, x1 = xi + (int)floorf(xmax) + 2;
      const int y0 = yi + (int)floorf(ymin) - 1, y1 = yi + (int)floorf(ymax) + 2;
      // The window's rows are the extent's ceiling and three more (a pixel of slack
      // below, the last pixel's row, a pixel above; for plain rows the row after it),
      // as the host planned them, which
      // no rounding of the two ends decides: ymin and ymax rounded apart reach a row
      // further where the extent is whole and the fraction a few 1e-7 below one.
      // The extent in FP32 is off by less than 1e-4 of the host's; the slack of 1e-3 is
      // part of the pixel above.  (In FP64 the check cost 1.4 us a launch: 52x61x6
      // voxels, 119 angles, 8 iterations on host buffers 742 against 731 us.)
      const float ey = fabsf(k.b1) * (BX - 1) + fabsf(k.b2) * (BY - 1) + fabsf(k.b3) * (NZ - 1);
      // (far(): integers and positions beyond their range say nothing about the window)
      if (!far(k.xf) && !far(k.yf) && x0 >= ox && x1 < ox + P.WX && (int)ceilf(ey - 1e-3f) + (ROWS ? 4 : 3) <= P.WY)
        k.flags |= kHolds;
      if (x0 >= 0 && x1 < P.ax.PX && y0 >= 0 && y1 < P.ax.PY) k.flags |= kOnDetector;
    }
    kc[a] = k;
  }
  __syncthreads();
  stream_wait();

  if (warp == kConsumerWarps) {
    // ---------------- producer warp: one elected lane issues the TMA loads
    if (lane == 0) {
      prefetch_tensormap(tmap);
      const uint32_t bytes = (uint32_t)(win_elems * sizeof(WT));
      int issued = 0;  // angles whose window load has been issued
      for (int a = 0; a < A; ++a) {
        const int s = a % NST;
        const int n = a / NST;
        if (n > 0 && !mbar_wait_bounded(&empty[s], (uint32_t)((n - 1) & 1), P.wait_iters)) {
          atomicExch(P.err, 2);
          break;
        }
        WT* dst = reinterpret_cast<WT*>(reinterpret_cast<unsigned char*>(win0) + s * stage_bytes);
        mbar_arrive_expect_tx(&full[s], bytes);
        // arrays of FP32 pairs are mapped as their floats: x = 2 * (first
        // column), a multiple of 4; planar ones as two FP32 rows per detector
        // row; row pairs have a row above the detector's first
        tma_load_3d(dst, tmap, ROWS ? kc[a].ox : (PLANAR || HALF) ? kc[a].ox + 1 : PAIR ? 2 * (kc[a].ox + 1) : 2 * kc[a].ox,
                    PLANAR ? 2 * kc[a].oy : PAIR || ROWS ? kc[a].oy : kc[a].oy + 1, a, &full[s]);
        issued = a + 1;
      }
      // Drain: the last load issued into each stage must land before exit
      // (earlier ones into that stage completed before it could be reissued).
      for (int s = 0; s < NST && s < issued; ++s) {
        const int n_last = (issued - 1 - s) / NST;
        if (!mbar_wait_bounded(&full[s], (uint32_t)(n_last & 1), kDrainIters)) atomicExch(P.err, 3);
      }
    }
    return;
  }

  // ---------------- consumer warps
  constexpr int kAcross = BX / 8;  // patches along X
  const int tx = LANES == 0 ? lane : LANES == 1 ? warp : (warp % kAcross) * 8 + (lane & 7);
  const int ty = LANES == 0 ? warp : LANES == 1 ? lane : (warp / kAcross) * 4 + (lane >> 3);
  const bool active = (X0 + tx < P.vol.Xs + P.vol.NX) && (Y0 + ty < P.vol.Ys + P.vol.NY);
  const int WX = P.WX;
  // pairs along x: a tap at window (ix, iy) reads one pair of rows iy and iy + 1
  const unsigned lim_x = (unsigned)WX, lim_y = (unsigned)(P.WY - 1);
  const long long sx = P.vol.NX, sxy = (long long)P.vol.NX * P.vol.NY;
  const long long base = (long long)(X0 + tx - P.vol.Xs) + (long long)(Y0 + ty - P.vol.Ys) * sx;
  // WBP: the in-detector weight sums.  They depend on the geometry alone, and the
  // weights of a voxel whose taps all lie on the detector sum to one, so they are
  // formed first, from the angles at which the brick leaves the detector, and
  // wait in cbp: the loop over the windows carries no second accumulator.
  int n_inside = 0;  // angles at which the whole brick lies on the detector
  if (MODE == 0) {
    for (int a = 0; a < A; ++a) n_inside += (kc[a].flags & kOnDetector) ? 1 : 0;
    if (n_inside < A) {
      float c[NZ];
#pragma unroll
      for (int z = 0; z < NZ; ++z) c[z] = (float)n_inside;
      for (int a = 0; a < A; ++a) {
        const WinConst k = kc[a];
        if (k.flags & kOnDetector) continue;
        const float xr = fmaf(k.a2, (float)ty, fmaf(k.a1, (float)tx, k.xf));
        const float yr = fmaf(k.b2, (float)ty, fmaf(k.b1, (float)tx, k.yf));
#pragma unroll
        for (int z = 0; z < NZ; ++z)
          c[z] = fmaf(tap_weight(fmaf(k.a3, (float)z, xr), k.lxm + k.ox, P.ax.PX),
                      tap_weight(fmaf(k.b3, (float)z, yr), k.lym + k.oy, P.ax.PY), c[z]);
      }
#pragma unroll
      for (int z = 0; z < NZ; ++z)
        if (active && Z0 + z < P.z1) P.cbp[base + (long long)(Z0 + z - P.z0) * sxy] = c[z];
    }
  }
  float s[NZ];
#pragma unroll
  for (int z = 0; z < NZ; ++z) s[z] = 0.f;
  bool bad = false;

  for (int a = 0; a < A; ++a) {
    const int st = a % NST;
    // every lane of the warp takes the same branch (the warp syncs below)
    if (!__all_sync(0xffffffffu, mbar_wait_bounded(&full[st], (uint32_t)((a / NST) & 1), P.wait_iters))) {
      if (lane == 0) atomicExch(P.err, 4);
      break;
    }
    const WT* w = reinterpret_cast<const WT*>(reinterpret_cast<const unsigned char*>(win0) + st * stage_bytes);
    const WinConst k = kc[a];
    float xr = fmaf(k.a2, (float)ty, fmaf(k.a1, (float)tx, k.xf));
    float yr = fmaf(k.b2, (float)ty, fmaf(k.b1, (float)tx, k.yf));
    if constexpr (!PAIR) {
      if (!(k.flags & kHolds)) {
        bad = true;
      } else if (active) {
        if (BZ0 && fabsf(k.a3) < 0.999f) {
          const float ty = __fadd_rd(yr, kMagic);  // floor, in the low bits
          const float fy = yr - (ty - kMagic);
          const WT* row0 = w + (__float_as_int(ty) + k.lym) * WX;
          bp_column_rows<NZ, ROWS>(s, row0, WX, xr, k.a3, k.lxm, fy);
        } else {
          bp_column_zy<NZ, false, false>(s, w, WX, xr, yr, k);
        }
      }
    } else {
      // Uniform rows: the detector y does not move along the lanes (|slope| * 31
      // below 1e-6 px), so every lane of the warp reads the same two rows with
      // the same weights; the warp blends them once per angle.
      const bool uni = BZ0 && LANES != 2 && fabsf(LANES == 1 ? k.b2 : k.b1) < 3e-8f;
      bool blended = false;
      if (uni) {
        yr = __shfl_sync(0xffffffffu, yr, 0);
        const float fly = floorf(yr);
        const float fy = yr - fly;
        const int rowi = magic_int(fly) + k.lym;
        if ((unsigned)rowi < lim_y) {
          const WT* row0 = w + rowi * WX * (PLANAR ? 2 : 1);
          for (int i = lane; i < WX; i += 32) {
            if constexpr (PLANAR) {
              const float v0 = row0[i], d0 = row0[i + WX], v1 = row0[i + 2 * WX], d1 = row0[i + 3 * WX];
              blend[i] = make_float2(fmaf(fy, v1 - v0, v0), fmaf(fy, d1 - d0, d0));
            } else if constexpr (HALF) {
              const float2 q0 = __half22float2(row0[i]), q1 = __half22float2(row0[i + WX]);
              blend[i] = make_float2(fmaf(fy, q1.x - q0.x, q0.x), fmaf(fy, q1.y - q0.y, q0.y));
            } else {
              const float2 q0 = row0[i], q1 = row0[i + WX];
              blend[i] = make_float2(fmaf(fy, q1.x - q0.x, q0.x), fmaf(fy, q1.y - q0.y, q0.y));
            }
          }
          blended = true;
        }
        __syncwarp();
      }
      bool done = !active;
      if (active && !BZ0) {
        // x and y are affine in z: the column's end voxels bound every tap, so
        // the window is checked once per column
        const float xe = fmaf(k.a3, (float)(NZ - 1), xr), ye = fmaf(k.b3, (float)(NZ - 1), yr);
        const int ixa = magic_int(floorf(xr)) + k.lxm, ixb = magic_int(floorf(xe)) + k.lxm;
        const int iya = magic_int(floorf(yr)) + k.lym, iyb = magic_int(floorf(ye)) + k.lym;
        bool inside = (unsigned)min(ixa, ixb) < lim_x && (unsigned)max(ixa, ixb) < lim_x &&
                      (unsigned)min(iya, iyb) < lim_y && (unsigned)max(iya, iyb) < lim_y;
        if (inside) {
          bp_column_zy<NZ, PAIR, HALF>(s, w, WX, xr, yr, k);
          done = true;
        }
      }
      if (active && BZ0 && fabsf(k.a3) < 0.999f) {
        // x is affine in z: the column's end voxels bound every tap index, so
        // the window bound is checked once per column instead of per voxel; the
        // stepped tap may run one pixel past the exact last one.
        const float fly = floorf(yr);
        const float fy = yr - fly;
        const int rowi = magic_int(fly) + k.lym;
        const int ixa = magic_int(floorf(xr)) + k.lxm;
        const int ixb = magic_int(floorf(fmaf(k.a3, (float)(NZ - 1), xr))) + k.lxm;
        bool inside = (unsigned)rowi < lim_y && (unsigned)min(ixa, ixb) < lim_x && (unsigned)(max(ixa, ixb) + 1) < lim_x;
        if (inside) {
          if (blended) {
            if (k.a3 >= 0.f) bp_column_blended<true, NZ>(s, blend, xr, k.a3, k.lxm);
            else bp_column_blended<false, NZ>(s, blend, xr, k.a3, k.lxm);
          } else if constexpr (PLANAR) {
            const float* row0 = w + rowi * 2 * WX;
            if (k.a3 >= 0.f) bp_column_planar<true, NZ>(s, row0, WX, xr, k.a3, k.lxm, 1.f - fy, fy);
            else bp_column_planar<false, NZ>(s, row0, WX, xr, k.a3, k.lxm, 1.f - fy, fy);
          } else if constexpr (HALF) {
            const __half2* row0 = w + rowi * WX;
            if (k.a3 >= 0.f) bp_column_half<true, NZ>(s, row0, WX, xr, k.a3, k.lxm, 1.f - fy, fy);
            else bp_column_half<false, NZ>(s, row0, WX, xr, k.a3, k.lxm, 1.f - fy, fy);
          } else {
            const WT* row0 = w + rowi * WX;
            if (k.a3 >= 0.f) bp_column<true, NZ>(s, row0, WX, xr, k.a3, k.lxm, 1.f - fy, fy);
            else bp_column<false, NZ>(s, row0, WX, xr, k.a3, k.lxm, 1.f - fy, fy);
          }
          done = true;
        }
      }
      if (!done) {
        // y part (per column when the map has no Z term)
        float fy = 0.f, wy0 = 0.f, wy1 = 0.f;
        int rowi = 0;
        if (BZ0) {
          const float fly = floorf(yr);
          fy = yr - fly;
          rowi = magic_int(fly) + k.lym;
          if ((unsigned)rowi >= lim_y) bad = true;
          wy0 = 1.f - fy;
          wy1 = fy;
        }
#pragma unroll
        for (int z = 0; z < NZ; ++z) {
          if (!BZ0) {
            const float y = fmaf(k.b3, (float)z, yr);
            const float fly = floorf(y);
            fy = y - fly;
            rowi = magic_int(fly) + k.lym;
            if ((unsigned)rowi >= lim_y) bad = true;
            wy0 = 1.f - fy;
            wy1 = fy;
          }
          const float x = fmaf(k.a3, (float)z, xr);
          const float flx = floorf(x);
          const float fx = x - flx;
          const int ix = magic_int(flx) + k.lxm;
          if ((unsigned)ix >= lim_x) bad = true;
          const int i0 = bad ? 0 : ix + rowi * WX * (PLANAR ? 2 : 1);  // never index outside the window
          float r0, r1;
          if constexpr (PLANAR) {
            r0 = fmaf(fx, w[i0 + WX], w[i0]);
            r1 = fmaf(fx, w[i0 + 3 * WX], w[i0 + 2 * WX]);
          } else if constexpr (HALF) {
            const float2 q0 = __half22float2(w[i0]), q1 = __half22float2(w[i0 + WX]);
            r0 = fmaf(fx, q0.y, q0.x);
            r1 = fmaf(fx, q1.y, q1.x);
          } else {
            const float2 q0 = w[i0], q1 = w[i0 + WX];
            r0 = fmaf(fx, q0.y, q0.x);
            r1 = fmaf(fx, q1.y, q1.x);
          }
          s[z] = fmaf(wy0, r0, s[z]);
          s[z] = fmaf(wy1, r1, s[z]);
        }
      }
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(&empty[st]);
  }
  if (bad) atomicExch(P.err, 5);
  if (!active) return;
#pragma unroll
  for (int z = 0; z < NZ; ++z) {
    const int zz = Z0 + z;
    if (zz >= P.z1) break;
    const long long vi = base + (long long)(zz - P.z0) * sxy;
    float out;
    if (MODE == 0) {
      const float c = n_inside < A ? P.cbp[vi] : (float)A;
      out = c != 0.f ? s[z] / c : 0.f;
      P.vol_out[vi] = out;
      if (n_inside == A) P.cbp[vi] = c;
    } else {
      const float cv = P.cbp[vi];
      out = P.vol_out[vi];
      if (cv != 0.f) {
        out = fmaf(P.step, s[z] / cv, out);
        P.vol_out[vi] = out;
      }
    }
    if (P.copy_kind == 1) static_cast<__nv_bfloat16*>(P.vol_copy)[vi] = __float2bfloat16_rn(out);
    else if (P.copy_kind == 2) static_cast<__half*>(P.vol_copy)[vi] = __float2half_rn(out);
  }
}

// One CTA per brick of one axis.  The grid runs x fastest, then z, then y:
// bricks of the same rows at all depths run together, so the detector rows
// they read stay in L2 instead of being re-read from DRAM once per z layer.
template <typename PT, int MODE, bool PAIR, int LANES, bool BZ0, int NZ, int PF = 0>
// (registers: 4 CTAs per SM leave 56, enough for 32 accumulators over x pairs;
// the walk over row pairs takes 72 at depth 32)
__global__ void __launch_bounds__(kThreads, !PAIR && NZ >= 32 ? 3 : MODE == 1 && NZ < 32 && PAIR && PF == 2 ? 5 : 4)
bp_tma_kernel(const __grid_constant__ CUtensorMap tmap, const BpArgs P) {
  extern __shared__ __align__(128) unsigned char smem[];
  bp_brick<PT, MODE, PAIR, LANES, BZ0, NZ, PF>(&tmap, P, blockIdx.x, blockIdx.z, blockIdx.y, smem, false);
}

template <typename PT, int MODE, bool PAIR, int LANES, bool BZ0, int NZ, int PF = 0>
cudaError_t launch_one(const CUtensorMap& map, const BpArgs& P, size_t smem, cudaStream_t st) {
  auto kern = bp_tma_kernel<PT, MODE, PAIR, LANES, BZ0, NZ, PF>;
  cudaError_t e = allow_shared_memory(kern, smem);
  if (e != cudaSuccess) return e;
  constexpr int BX = bp_brick_x(LANES, PAIR), BY = bp_brick_y(LANES, PAIR);
  const dim3 grid((P.vol.NX + BX - 1) / BX, (P.z1 - P.z0 + NZ - 1) / NZ, (P.vol.NY + BY - 1) / BY);
  launch_overlapped(kern, grid, kThreads, smem, st, map, P);
  const cudaError_t le = cudaGetLastError();
  if (le == cudaSuccess) g_windowed_launches.fetch_add(1, std::memory_order_relaxed);
  return le;
}

template <typename PT, int MODE, bool PAIR, int LANES, bool BZ0, int PF = 0>
cudaError_t launch_nz(const CUtensorMap& map, const BpArgs& P, const BpPlan& plan, cudaStream_t st) {
  if constexpr (MODE == 0) {  // the WBP has no depth 4
    if (plan.nz == 32) return launch_one<PT, 0, PAIR, LANES, BZ0, 32, PF>(map, P, plan.smem, st);
    if (plan.nz == 16) return launch_one<PT, 0, PAIR, LANES, BZ0, 16, PF>(map, P, plan.smem, st);
    return launch_one<PT, 0, PAIR, LANES, BZ0, 8, PF>(map, P, plan.smem, st);
  } else {
    if (plan.nz == 8) return launch_one<PT, MODE, PAIR, LANES, BZ0, 8, PF>(map, P, plan.smem, st);
    if (plan.nz == 4) return launch_one<PT, MODE, PAIR, LANES, BZ0, 4, PF>(map, P, plan.smem, st);
    if (plan.nz == 16) return launch_one<PT, MODE, PAIR, LANES, BZ0, 16, PF>(map, P, plan.smem, st);
    if (plan.nz == 32) return launch_one<PT, MODE, PAIR, LANES, BZ0, 32, PF>(map, P, plan.smem, st);
    return cudaErrorInvalidValue;
  }
}

}  // namespace
}  // namespace mtr
