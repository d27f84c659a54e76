// Forward projection (bilinear splat) with shared-memory detector windows
// and TMA bulk reduce-add (sm_103a).
//
// The reference adds every voxel's four bilinear weights into the projection
// with global float atomics (FunctionOnGPU.cu:27-52, 316-333): eight atomics
// per voxel and angle, contending along every ray.  Here one CTA owns a
// brick of BX x BY x NZ voxels for the whole launch (prefix sums in shared
// memory, or voxels in registers where the y-map has a Z term or a warp sums
// rows of its own).  For each of
// its angles it splats the brick into a private detector window in shared
// memory, then one thread flushes the window into the ray-sum array with a
// single 3-D tiled cp.reduce.async.bulk.tensor add (the L2 reduces whole
// sectors).  Three window stages rotate: the flush of one angle
// overlaps the splat of the next, and the stage after it is zeroed during the
// conversion pass, so an angle costs two block barriers.
//
// Window accumulation is fixed point: shared-memory float atomicAdd is not a
// single native operation on this part, integer adds are.  Each CTA scales
// its values by a power of two S with S * max|v| < 2^b and b <= 21 - log2(weight
// one pixel can receive from one column), so every added value rounds to an
// integer below 2^21 (rounded with the 1.5*2^23 trick, no float->int
// conversion) with an absolute error of at most 2^-(b+1) * max|v|.  The host bounds the weight one pixel can receive from
// one brick by 2^mass_shift (lattice points in the preimage of a 2x2-pixel
// square, times the brick depth) and b <= 30 - mass_shift keeps every window
// sum below 2^30.  Before the flush the window is converted back to float and
// divided by S (exact: S is a power of two).
//
// A voxel column is merged along its length before it is added: pixel by pixel
// from prefix sums, or voxel by voxel in registers where the y-map has a Z term
// (2-16x fewer shared-memory adds than four per voxel, depending on the tilt);
// bricks at the detector edge check each add against the window.
//
// Windows are clamped inside the detector (TMA reduces must not start at a
// negative coordinate), so a tap is on the detector iff it lies in the valid
// part of the window; taps off the detector are dropped as in the reference.
#include "mtr_internal.h"
#include "tma.cuh"

namespace mtr {
namespace {

constexpr int kWarps = 8;
constexpr int kThreads = kWarps * 32;
constexpr int kStages = 3;  // window stages in flight (splat, flush, next)
constexpr float kMagic = 12582912.0f;  // 1.5 * 2^23
constexpr int kMagicBits = 0x4B400000;

struct FwdConst {
  float xf, a1, a2, a3;
  float yf, b1, b2, b3;
  int lxm, lym;  // window-local integer base minus the magic bits
  int ox, oy;    // window origin (clamped inside the detector, ox aligned)
  int wlx;       // valid window columns (left of the detector's right edge)
  int interior;  // window not clamped and inside the detector: every tap is valid
  int pad[2];
};

struct FwdArgs {
  AxisDev ax;
  VolDev vol;
  int z0, z1;
  int WX, WY;
  int groups;      // angle groups (grid.z = z-blocks * groups)
  int max_angles;  // angles per group (shared-memory constants sized for it)
  int mass_shift;  // log2 bound of one pixel's total weight from one brick
  int nz;          // brick depth (voxels per column)
  const void* x;   // volume (nullptr: ones)
};

__device__ __forceinline__ int magic_int(float integral) { return __float_as_int(__fadd_rn(integral, kMagic)); }
// Zeroes a window stage (16-byte aligned) with all threads of the block.
__device__ __forceinline__ void zero_window(int* w, int n) {
  for (int i = threadIdx.x * 4; i < n; i += kThreads * 4) {
    if (i + 3 < n) *reinterpret_cast<int4*>(w + i) = make_int4(0, 0, 0, 0);
    else
      for (int q = i; q < n; ++q) w[q] = 0;
  }
}
__device__ __forceinline__ int floor_div(int a, int b) { return (a >= 0) ? a / b : -((-a + b - 1) / b); }
// round(w * v) for |w*v| < 2^22, as an integer, without a conversion instruction
__device__ __forceinline__ int fixq(float w, float v) { return __float_as_int(fmaf(w, v, kMagic)) - kMagicBits; }
// Integer add to the shared-memory word at 32-bit shared address `addr`
// (no value returned; the column walks keep their addresses in this form).
__device__ __forceinline__ void red_shared(uint32_t addr, int v) {
  asm volatile("red.shared.add.s32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}

// Ends an angle's splat into window stage `wi`: the fixed-point sums are
// converted in place and reduced into the ray sums with one bulk reduce-add;
// `next`, the stage of the following angle, is zeroed meanwhile (the bulk
// reduce of angle j - 2, its last reader, must be done reading).
__device__ __forceinline__ void flush_window(const CUtensorMap* smap, int* wi, int* next, int win_elems, float invS,
                                             int j, bool more, int ox, int oy, int a) {
  float* wf = reinterpret_cast<float*>(wi);
  if (threadIdx.x == 0 && j >= 2) bulk_wait_read<1>();
  __syncthreads();
  // fixed point -> float (exact power-of-two scale), in place, 16 bytes a step
  for (int i = threadIdx.x * 4; i < win_elems; i += kThreads * 4) {  // (WX is a multiple of 4)
    const int4 q = *reinterpret_cast<const int4*>(wi + i);
    *reinterpret_cast<float4*>(wf + i) =
        make_float4((float)q.x * invS, (float)q.y * invS, (float)q.z * invS, (float)q.w * invS);
    if (more) *reinterpret_cast<int4*>(next + i) = make_int4(0, 0, 0, 0);
  }
  fence_proxy_async_smem();
  __syncthreads();
  if (threadIdx.x == 0) {
    tma_reduce_add_3d(smap, wf, ox, oy, a);
    bulk_commit();
  }
}
template <int N> struct Off { static constexpr int value = N; };

template <typename VT> __device__ __forceinline__ float ldv(const void* p, long long i);
template <> __device__ __forceinline__ float ldv<float>(const void* p, long long i) {
  return __ldg(static_cast<const float*>(p) + i);
}
template <> __device__ __forceinline__ float ldv<__nv_bfloat16>(const void* p, long long i) {
  return __bfloat162float(__ldg(static_cast<const __nv_bfloat16*>(p) + i));
}
template <> __device__ __forceinline__ float ldv<__half>(const void* p, long long i) {
  return __half2float(__ldg(static_cast<const __half*>(p) + i));
}

// Integer add with a constant byte offset.
template <int OFF> __device__ __forceinline__ void red_shared_at(uint32_t addr, int v) {
  asm volatile("red.shared.add.s32 [%0+%2], %1;" ::"r"(addr), "r"(v), "n"(OFF) : "memory");
}

// ---- y-maps without a Z term: pixel by pixel over prefix sums ----------------
//
// A thread owns one voxel column and splats it pixel by pixel, not voxel by
// voxel.  Along the column the detector x is affine in z, so the voxels that
// fall between two neighbouring pixels p and p + 1 are a run of z, and what
// the run adds to the two pixels needs only its sums of v and of z v: two
// differences of prefix sums, which the CTA forms once, before its angles, and
// keeps in shared memory ([index][thread]: conflict-free whatever index each
// lane reads).  With z_p the place where x reaches p,
//     G = D1 - z_p D0,   part on p + 1: a3 G,   part on p: D0 - a3 G,
// and a pixel is added to the window when its right neighbour's run ends:
// E = D0 + a3 (G of the run before - G).  All lanes run in step (their pixel
// counts differ by at most one), where a walk along the voxels diverges at
// every pixel crossing.  A voxel that rounding puts on the wrong side of a
// boundary is harmless: its weights run on linearly past it.
//
// Bound by shared-memory wavefronts (4.3 per 32 voxels and angle at depth 32:
// 2.2 for the adds, which conflict 2.1 times whatever the window's pitch or
// the lanes' layout, 1.1 for the prefix, the rest the window and constants)
// with 14 instructions per voxel and angle, where the walk along the voxels was
// bound by the issue of 22.  512x512x64 at 60 degrees, 61 angles: 0.675 against
// 0.70 ms; 320x288x48, 45 angles: 0.16 against 0.21 ms; 512x512x128 read from
// FP16: 1.34 against 1.49 ms.
struct __align__(16) PreConst {  // per-angle constants of a brick
  float xf, a1, a2, a3;   // (|a3| at least 1e-7: 2e-6 px over a column)
  float yf, b1, b2, inv;  // inv = 1 / a3
  int lxm, lym;           // window-local integer base minus the magic bits
  int nx;                 // pixel boundaries that every column crosses: floor(|a3| (depth - 1))
  float scale;            // fixed-point scale of this angle (power of two)
  int ox, oy;             // window origin (clamped inside the detector, ox aligned)
  int wlx;                // valid window columns; negative where every tap is valid (window not clamped)
  float inv_scale;
};
constexpr uint32_t kPreStride = kThreads * 8u;  // bytes from one prefix index to the next
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 lds_pair(uint32_t a) {
  f32x2 v;
  asm volatile("ld.shared.b64 %0, [%1];" : "=l"(v) : "r"(a));
  return v;
}
__device__ __forceinline__ float lds_float(uint32_t a) {
  float v;
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a));
  return v;
}
__device__ __forceinline__ float2 sub2(f32x2 a, f32x2 b) {  // a - b in one packed instruction
  f32x2 r;
  float2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(b), "l"(0xBF800000BF800000ull), "l"(a));
  asm("mov.b64 {%0, %1}, %2;" : "=f"(d.x), "=f"(d.y) : "l"(r));
  return d;
}

// One column of depth nz at one angle: its prefix sums at `pre` (index i: sums
// over voxels z < i of v and (z - nz / 2) v), detector rows at shared address
// `row` and `row` + drow with weights wy0, wy1 (scaled).  CHK: the brick's
// window is clamped at the detector edge (or reaches past it): each addition
// checks its window column against the valid columns (span, in bytes) and each
// detector row against the window, and drops what falls outside, as the
// reference drops off-detector taps.
template <bool CHK>
__device__ __forceinline__ void splat_column(uint32_t pre, int nz, uint32_t row, uint32_t drow, float xr,
                                             const PreConst& k, float wy0, float wy1, uint32_t span, bool y0ok,
                                             bool y1ok) {
  const bool asc = k.a3 >= 0.f;
  const int c0 = nz >> 1;  // origin of the moments
  const float lo = (float)-c0, hi = (float)(nz - c0);  // the column's ends, in centred z
  const float xs = asc ? xr : fmaf(k.a3, (float)(nz - 1), xr);  // x of the first voxel met
  const float fl = floorf(xs);
  float zp = fmaf(fl - xr, k.inv, lo);  // where x reaches the current pixel
  float tb = zp + k.inv;                // and the next one
  const float ceil_at = kMagic + (float)c0;  // rounding up to an index, in the low bits
  const uint32_t base = pre - (uint32_t)kMagicBits * kPreStride;
  const uint32_t end = pre + (asc ? (uint32_t)nz * kPreStride : 0u);
  f32x2 prev = 0ull;
  if (!asc) {  // read backwards, the prefix gives the negated sums
    prev = lds_pair(pre + (uint32_t)nz * kPreStride);
    wy0 = -wy0;
    wy1 = -wy1;
  }
  uint32_t at = row + 4u * (uint32_t)((k.lxm + kMagicBits) + (magic_int(fl) - kMagicBits)), at1 = at + drow;
  float before = 0.f;  // G of the run before
  auto index_at = [&](float t) { return base + __float_as_uint(__fadd_ru(t, ceil_at)) * kPreStride; };
  auto add = [&](auto off, float e) {
    constexpr int OFF = decltype(off)::value;
    if (CHK) {
      const bool xok = at + (uint32_t)OFF - row < span;  // (a column left of the window wraps to a large offset)
      if (xok && y0ok) red_shared_at<OFF>(at, fixq(wy0, e));
      if (xok && y1ok) red_shared_at<OFF>(at1, fixq(wy1, e));
    } else {
      red_shared_at<OFF>(at, fixq(wy0, e));
      red_shared_at<OFF>(at1, fixq(wy1, e));
    }
  };
  auto run = [&](auto off, f32x2 s, float z) {  // the run from z (the current pixel's place) to prefix s
    const float2 d = sub2(s, prev);
    prev = s;
    const float g = fmaf(-z, d.x, d.y);
    add(off, fmaf(k.a3, before - g, d.x));
    before = g;
  };
  // The boundaries that every column crosses lie inside it; four prefix loads
  // are in flight at a time.
  int n = k.nx;
#pragma unroll 1
  for (; n >= 4; n -= 4) {
    const float t1 = tb + k.inv, t2 = fmaf(2.f, k.inv, tb), t3 = fmaf(3.f, k.inv, tb);
    const f32x2 s0 = lds_pair(index_at(tb)), s1 = lds_pair(index_at(t1)), s2 = lds_pair(index_at(t2)),
                s3 = lds_pair(index_at(t3));
    run(Off<0>{}, s0, zp);
    run(Off<4>{}, s1, tb);
    run(Off<8>{}, s2, t1);
    run(Off<12>{}, s3, t2);
    zp = t3;
    tb = fmaf(4.f, k.inv, tb);
    at += 16u;
    at1 += 16u;
  }
  if (n & 2) {
    const float t1 = tb + k.inv;
    const f32x2 s0 = lds_pair(index_at(tb)), s1 = lds_pair(index_at(t1));
    run(Off<0>{}, s0, zp);
    run(Off<4>{}, s1, tb);
    zp = t1;
    tb = t1 + k.inv;
    at += 8u;
    at1 += 8u;
  }
  if (n & 1) {
    run(Off<0>{}, lds_pair(index_at(tb)), zp);
    zp = tb;
    tb += k.inv;
    at += 4u;
    at1 += 4u;
  }
  // Some columns cross one more; the next run ends the column, and where the
  // one before ended it already, its pixel has only the carried part.
  const uint32_t last = index_at(asc ? fminf(tb, hi) : fmaxf(tb, lo));
  const f32x2 s0 = lds_pair(last), s1 = lds_pair(end);
  run(Off<0>{}, s0, zp);
  run(Off<4>{}, s1, tb);
  if (last != end) add(Off<8>{}, k.a3 * before);
}

// The same column voxel by voxel: its values are the differences of the prefix
// sums, its four taps are added one by one.  A pixel costs splat_column 14
// instructions and 4-6 shared wavefronts, a voxel costs this 20 and 6-10, so it
// takes the slopes of kSteep pixels per voxel and more (detectors finer than the
// volume): 256x256x64, 61 angles, 45 degrees, 3 and 4 pixels per voxel, 0.60 and
// 0.85 ms against 0.66 and 1.02 (0.60 and 0.86 from 1.3 and from 2.0).
constexpr float kSteep = 1.6f;
template <bool CHK>
__device__ __forceinline__ void splat_voxels(uint32_t pre, int nz, uint32_t row, uint32_t drow, float xr,
                                             const PreConst& k, float wy0, float wy1, uint32_t span, bool y0ok,
                                             bool y1ok) {
  float prev = 0.f;
#pragma unroll 4
  for (int z = 0; z < nz; ++z) {
    pre += kPreStride;
    const float s = lds_float(pre), v = s - prev;
    prev = s;
    const float x = fmaf(k.a3, (float)z, xr);
    const float t = __fadd_rd(x, kMagic);  // floor, in the low bits
    const float fx = x - (t - kMagic);
    const uint32_t at = row + 4u * (uint32_t)(__float_as_int(t) + k.lxm), at1 = at + drow;
    const float v1 = fx * v, v0 = v - v1;
    const bool x0ok = !CHK || at - row < span, x1ok = !CHK || at + 4u - row < span;
    if (x0ok && (!CHK || y0ok)) red_shared_at<0>(at, fixq(wy0, v0));
    if (x1ok && (!CHK || y0ok)) red_shared_at<4>(at, fixq(wy0, v1));
    if (x0ok && (!CHK || y1ok)) red_shared_at<0>(at1, fixq(wy1, v0));
    if (x1ok && (!CHK || y1ok)) red_shared_at<4>(at1, fixq(wy1, v1));
  }
}

// One brick (bx, by, zb) and angle group g of one axis whose y-map has no Z
// term; `smem` is the CTA's dynamic shared memory.  On return every bulk
// reduce it issued is complete.  STEEP: some angles may reach kSteep.
template <typename VT, bool STEEP>
__device__ __forceinline__ void prefix_brick(const CUtensorMap* smap, const FwdArgs& P, int lanes, int bx, int by,
                                             int zb, int g, unsigned char* smem) {
  const int BX = brick_x(lanes), BY = brick_y(lanes), NZ = P.nz;
  PreConst* kc = reinterpret_cast<PreConst*>(smem);
  const size_t kc_bytes = ((size_t)P.max_angles * sizeof(PreConst) + 127) & ~(size_t)127;
  const int WX = P.WX, WY = P.WY;
  const int win_elems = WX * WY;
  const size_t stage_bytes = ((size_t)win_elems * 4 + 127) & ~(size_t)127;
  unsigned char* win0 = smem + kc_bytes + 128;
  float* red = reinterpret_cast<float*>(smem + kc_bytes);  // 32 floats for the block max
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int A = P.ax.A;
  const int a_begin = (int)((long long)A * g / P.groups), a_end = (int)((long long)A * (g + 1) / P.groups);
  const int na = a_end - a_begin;
  const int X0 = P.vol.Xs + bx * BX, Y0 = P.vol.Ys + by * BY, Z0 = P.z0 + zb * NZ;

  // own column, read once (coalesced along lanes): prefix sums, and the brick's max |v|
  const int tx = lanes == 0 ? lane : lanes == 1 ? warp : (warp & 1) * 8 + (lane & 7);
  const int ty = lanes == 0 ? warp : lanes == 1 ? lane : (warp >> 1) * 4 + (lane >> 3);
  const bool active = (X0 + tx < P.vol.Xs + P.vol.NX) && (Y0 + ty < P.vol.Ys + P.vol.NY);
  float2* pre = reinterpret_cast<float2*>(win0 + kStages * stage_bytes) + tid;
  float vmax = 0.f;
  {
    const long long sx = P.vol.NX, sxy = (long long)P.vol.NX * P.vol.NY;
    const long long base = (long long)(X0 + tx - P.vol.Xs) + (long long)(Y0 + ty - P.vol.Ys) * sx + stream_wait();
    const int c0 = NZ >> 1;
    float s0 = 0.f, s1 = 0.f;
    pre[0] = make_float2(0.f, 0.f);
#pragma unroll 1
    for (int z8 = 0; z8 < NZ; z8 += 8) {  // eight loads in flight
      float v[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const int z = z8 + q;
        v[q] = 0.f;
        if (active && z < NZ && Z0 + z < P.z1)
          v[q] = P.x ? ldv<VT>(P.x, base + (long long)(Z0 + z - P.z0) * sxy) : 1.f;
      }
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const int z = z8 + q;
        if (z < NZ) {
          vmax = fmaxf(vmax, fabsf(v[q]));
          s0 += v[q];
          s1 = fmaf((float)(z - c0), v[q], s1);
          pre[(z + 1) * kThreads] = make_float2(s0, s1);
        }
      }
    }
  }
  for (int o = 16; o > 0; o >>= 1) vmax = fmaxf(vmax, __shfl_xor_sync(0xffffffffu, vmax, o));
  if (lane == 0) red[warp] = vmax;
  zero_window(reinterpret_cast<int*>(win0), win_elems);  // the first angle's stage
  if (tid == 0) prefetch_tensormap(smap);
  __syncthreads();
  vmax = red[0];
  for (int w = 1; w < kWarps; ++w) vmax = fmaxf(vmax, red[w]);
  int e2 = 0;
  if (vmax > 0.f && isfinite(vmax)) frexpf(vmax, &e2);

  for (int j = tid; j < na; j += kThreads) {
    const int a = a_begin + j;
    const double* cx = P.ax.xc + 4 * a;
    const double* cy = P.ax.yc + 4 * a;
    const double xb = cx[0] + cx[1] * X0 + cx[2] * Y0 + cx[3] * Z0 - 1.0;
    const double yb = cy[0] + cy[1] * X0 + cy[2] * Y0 + cy[3] * Z0 - 1.0;
    const double fxb = floor(fmin(fmax(xb, -1.0e9), 1.0e9)), fyb = floor(fmin(fmax(yb, -1.0e9), 1.0e9));
    PreConst k;
    k.xf = (float)(xb - fxb);
    k.yf = (float)(yb - fyb);
    k.a1 = (float)cx[1]; k.a2 = (float)cx[2];
    const float st = fmaxf(fabsf((float)cx[3]), 1e-7f);
    k.a3 = cx[3] >= 0.0 ? st : -st;
    k.b1 = (float)cy[1]; k.b2 = (float)cy[2];
    k.inv = 1.f / k.a3;
    const int xi = (int)fxb, yi = (int)fyb;
    const float xmin = k.xf + fminf(0.f, k.a1 * (BX - 1)) + fminf(0.f, k.a2 * (BY - 1)) + fminf(0.f, k.a3 * (NZ - 1));
    const float ymin = k.yf + fminf(0.f, k.b1 * (BX - 1)) + fminf(0.f, k.b2 * (BY - 1));
    const int ox0 = floor_div(xi + (int)floorf(xmin) - 1, 4) * 4;
    const int oy0 = yi + (int)floorf(ymin) - 1;
    // clamp inside [0, pitch - WX] x [0, PY - WY]; the host checked both ranges exist
    k.ox = min(max(ox0, 0), P.ax.pitch - WX);
    k.oy = min(max(oy0, 0), P.ax.PY - WY);
    k.lxm = xi - k.ox - kMagicBits;
    k.lym = yi - k.oy - kMagicBits;
    // An unclamped window holds the whole footprint; inside the detector every tap is kept.
    const bool interior = k.ox == ox0 && k.oy == oy0 && k.ox + WX <= P.ax.PX;
    k.wlx = interior ? -1 : max(0, min(WX, P.ax.PX - k.ox));
    k.nx = (int)(st * (float)(NZ - 1));
    // A base that the clamp to +-1e9 px left large: no tap near the detector, and
    // its float positions must index neither the prefix sums nor the window.  The
    // columns walk from zero instead, over no valid window column.
    if (!(fabsf(k.xf) <= 65536.f && fabsf(k.yf) <= 65536.f)) {
      k.xf = k.yf = 0.f;
      k.wlx = 0;
    }
    // S = 2^(b-e) with max |v| < 2^e, so |v S| < 2^b.  A pixel receives at most
    // the weight w = min(depth, 1 + 1/slope) <= 2^lw from one column:
    // |addition| < 2^(b + lw) <= 2^21, the range of the magic rounding.  A
    // pixel's window sum stays below 2^(b + mass_shift) <= 2^30 (no overflow).
    const int lw = log2_ceil(fminf((float)NZ, 1.f + 1.f / st));
    const int bits = min(21 - lw, 30 - P.mass_shift);
    const int sexp = max(-120, min(120, bits - e2));
    k.scale = ldexpf(1.f, sexp);
    k.inv_scale = ldexpf(1.f, -sexp);
    kc[j] = k;
  }
  __syncthreads();

  // Three window stages as in fwd_brick.
  const uint32_t pre_a = smem_u32(pre);
#pragma unroll 1
  for (int j = 0; j < na; ++j) {
    const int st = j % kStages;
    int* wi = reinterpret_cast<int*>(win0 + st * stage_bytes);
    const PreConst k = kc[j];  // (a copy: the adds order memory)
    if (active) {
      const float xr = fmaf(k.a2, (float)ty, fmaf(k.a1, (float)tx, k.xf));
      const float yr = fmaf(k.b2, (float)ty, fmaf(k.b1, (float)tx, k.yf));
      const float fly = floorf(yr);
      const float fy = yr - fly;
      const int rowi = magic_int(fly) + k.lym;
      const uint32_t rowa = smem_u32(wi) + 4u * (uint32_t)(rowi * WX);
      const float wy0 = (1.f - fy) * k.scale, wy1 = fy * k.scale;
      if (STEEP && fabsf(k.a3) >= kSteep) {
        if (k.wlx < 0)
          splat_voxels<false>(pre_a, NZ, rowa, 4u * (uint32_t)WX, xr, k, wy0, wy1, 0u, true, true);
        else
          splat_voxels<true>(pre_a, NZ, rowa, 4u * (uint32_t)WX, xr, k, wy0, wy1, 4u * (uint32_t)k.wlx,
                             (unsigned)rowi < (unsigned)WY, (unsigned)(rowi + 1) < (unsigned)WY);
      } else if (k.wlx < 0)
        splat_column<false>(pre_a, NZ, rowa, 4u * (uint32_t)WX, xr, k, wy0, wy1, 0u, true, true);
      else
        splat_column<true>(pre_a, NZ, rowa, 4u * (uint32_t)WX, xr, k, wy0, wy1, 4u * (uint32_t)k.wlx,
                           (unsigned)rowi < (unsigned)WY, (unsigned)(rowi + 1) < (unsigned)WY);
    }
    flush_window(smap, wi, reinterpret_cast<int*>(win0 + ((j + 1) % kStages) * stage_bytes), win_elems, k.inv_scale, j,
                 j + 1 < na, k.ox, k.oy, a_begin + j);
  }
  if (tid == 0) bulk_wait_all();
}

// ---- y-maps with a Z term: voxel by voxel ---------------------------------------
//
// Streaming splat of one voxel column (fixed X, Y), held in registers: its
// detector x moves by |a3| < 1 and its y by |b3| < 1 per voxel, so consecutive
// voxels reach at most one new pixel and one new row.  The walk always runs z
// upwards; where a3 < 0 it runs in the mirrored coordinate u = -x, which grows
// by |a3| per voxel (a voxel at u with fraction f splats (1 - f, f) onto
// mirrored pixels (p, p + 1), which are the original pixels (-p, -p - 1) with
// the original weights), and likewise in y.  Four sums are carried: the weight
// not yet emitted of the current row and the next (S0, S1), and its parts on
// the next pixel (X0, X1).  At a pixel
// crossing one pixel is emitted in both rows; at a row crossing the two pixels
// of the row left are, and the next row's sums move down.  Two shared-memory
// adds per pixel and two per row crossed, against four per voxel tap by tap:
// 320x300x72 voxels, 51 angles, rows crossed every ~100 voxels, 0.55 ms
// against 0.72 ms (bound by issue: 40 instructions per voxel and angle, half
// of them in the crossings that some lane of a warp takes at almost every voxel).
// CHK as in splat_column.
template <int NZ, bool CHK>
__device__ __forceinline__ void stream_column_zy(uint32_t win, int WX, int WY, const float (&v)[NZ], float xr,
                                                 float yr, const FwdConst& k) {
  const int dir = k.a3 >= 0.f ? 1 : -1, diry = k.b3 >= 0.f ? 1 : -1;
  const float u = dir > 0 ? xr : -xr, t = diry > 0 ? yr : -yr;
  const float flu = floorf(u), flt = floorf(t);
  float fx = u - flu, fy = t - flt;
  const float step = fabsf(k.a3), stepy = fabsf(k.b3);
  const int col = (k.lxm + kMagicBits) + dir * (magic_int(flu) - kMagicBits);
  int row = (k.lym + kMagicBits) + diry * (magic_int(flt) - kMagicBits);
  uint32_t rowa = win + 4u * (uint32_t)(row * WX);  // address of the current row
  uint32_t at = rowa + 4u * (uint32_t)col;
  const uint32_t dstep = dir > 0 ? 4u : 0xFFFFFFFCu;
  const uint32_t drow = diry > 0 ? 4u * (uint32_t)WX : 0u - 4u * (uint32_t)WX;
  const uint32_t span = 4u * (uint32_t)k.wlx;
  auto emit0 = [&](uint32_t q, float e) {  // current row
    if (!CHK || (q - rowa < span && (unsigned)row < (unsigned)WY)) red_shared(q, fixq(1.f, e));
  };
  auto emit1 = [&](uint32_t q, float e) {  // next row
    if (!CHK || (q - rowa < span && (unsigned)(row + diry) < (unsigned)WY)) red_shared(q + drow, fixq(1.f, e));
  };
  float g1 = fy * v[0], g0 = v[0] - g1;
  float S0 = g0, S1 = g1, X0 = fx * g0, X1 = fx * g1;
#pragma unroll
  for (int z = 1; z < NZ; ++z) {
    fx += step;
    fy += stepy;
    if (fy >= 1.f) {  // the column left the current row
      emit0(at, S0 - X0);
      emit0(at + dstep, X0);
      S0 = S1;
      X0 = X1;
      S1 = X1 = 0.f;
      fy -= 1.f;
      at += drow;
      rowa += drow;
      if (CHK) row += diry;
    }
    if (fx >= 1.f) {  // the column left the current pixel
      emit0(at, S0 - X0);
      emit1(at, S1 - X1);
      S0 = X0;
      S1 = X1;
      X0 = X1 = 0.f;
      fx -= 1.f;
      at += dstep;
    }
    g1 = fy * v[z];
    g0 = v[z] - g1;
    S0 += g0;
    S1 += g1;
    X0 = fmaf(fx, g0, X0);
    X1 = fmaf(fx, g1, X1);
  }
  emit0(at, S0 - X0);
  emit1(at, S1 - X1);
  emit0(at + dstep, X0);
  emit1(at + dstep, X1);
}

// ---- rows shared by a warp: voxel by voxel into one row ---------------------------
//
// Axes along a volume axis whose columns are too steep for the line kernels: the
// lanes of a warp share their two detector rows and weights, so the warp sums its
// columns into one row of its own, which is split over the two detector rows once
// per angle.  The columns stay in registers; prefix sums would take the shared
// memory that the wide windows of such an axis need (one CTA an SM against three).
//
// One column (fixed X, Y) whose x moves by |a3| < 1 per voxel, upwards in z and
// where a3 < 0 in the mirrored coordinate u = -x, from fraction fx of the pixel at
// shared address `at`: a pixel is emitted when the column has left it.  L > 1
// (slope below 1 / L): a chunk of L voxels crosses one boundary at most, so it
// accumulates without a branch.  S is the weight not yet emitted, a1 its part on
// the next pixel; inside a chunk the fraction runs on past 1, and C collects
// (f - 1) v of the voxels beyond the crossing, which moves them to their true
// pixels when the chunk ends.
template <int NZ, int L, typename Emit>
__device__ __forceinline__ void walk_column(const float (&v)[NZ], uint32_t at, uint32_t dstep, float fx, float step,
                                            const Emit& emit) {
  float S = v[0], a1 = fx * v[0];
#pragma unroll
  for (int z0 = 1; z0 < NZ; z0 += L) {
    float C = 0.f;
#pragma unroll
    for (int j = 0; j < L; ++j) {
      if (z0 + j < NZ) {
        fx += step;
        S += v[z0 + j];
        a1 = fmaf(fx, v[z0 + j], a1);
        C = fmaf(__saturatef(fx - 1.f), v[z0 + j], C);
      }
    }
    if (fx >= 1.f) {
      emit(at, (S - a1) + C);
      S = a1 - C;
      a1 = C;
      fx -= 1.f;
      at += dstep;
    }
  }
  emit(at, S - a1);
  emit(at + dstep, a1);
}
// One column at any slope, with the longest chunk its slope allows.
template <int NZ, typename Emit>
__device__ __forceinline__ void splat_walk(const float (&v)[NZ], uint32_t row, float xr, float a3, int lxm,
                                           const Emit& emit) {
  const float st = fabsf(a3);
  if (st < 0.999f) {
    const float u = a3 >= 0.f ? xr : -xr;
    const float fl = floorf(u);
    const int p = magic_int(fl) - kMagicBits;
    const uint32_t at = row + 4u * (uint32_t)((lxm + kMagicBits) + (a3 >= 0.f ? p : -p));
    const uint32_t dstep = a3 >= 0.f ? 4u : 0xFFFFFFFCu;
    if (st < 0.2499f) walk_column<NZ, 4>(v, at, dstep, u - fl, st, emit);
    else if (st < 0.4999f) walk_column<NZ, 2>(v, at, dstep, u - fl, st, emit);
    else walk_column<NZ, 1>(v, at, dstep, u - fl, st, emit);
    return;
  }
#pragma unroll
  for (int z = 0; z < NZ; ++z) {
    const float x = fmaf(a3, (float)z, xr);
    const float t = __fadd_rd(x, kMagic);  // floor, in the low bits
    const float fx = x - (t - kMagic);
    const uint32_t at = row + 4u * (uint32_t)(__float_as_int(t) + lxm);
    const float v1 = fx * v[z];
    emit(at, v[z] - v1);
    emit(at + 4u, v1);
  }
}
// Adds the warp's row of WX fixed-point sums (to 24 bits) to the two detector rows
// at `row` with weights 1 - fy and fy, and zeroes it.
__device__ __forceinline__ void split_row(int* urow, int WX, uint32_t row, float fy) {
  __syncwarp();
  for (int i = threadIdx.x & 31; i < WX; i += 32) {
    const int q = urow[i];
    if (q != 0) {
      const float f = (float)q;
      red_shared(row + 4u * (uint32_t)i, __float2int_rn((1.f - fy) * f));
      red_shared(row + 4u * (uint32_t)(WX + i), __float2int_rn(fy * f));
      urow[i] = 0;
    }
  }
  __syncwarp();
}

// One brick (bx, by, zb) and angle group g of one axis; `smem` is the CTA's
// dynamic shared memory.  On return every bulk reduce it issued is complete.
// ROWS: the lanes of a warp share their rows at every angle.
template <typename VT, int NZ, bool ROWS>
__device__ __forceinline__ void fwd_brick(const CUtensorMap* smap, const FwdArgs& P, int lanes, int bx, int by, int zb, int g,
                                          unsigned char* smem) {
  const int BX = brick_x(lanes), BY = brick_y(lanes);
  FwdConst* kc = reinterpret_cast<FwdConst*>(smem);
  const size_t kc_bytes = ((size_t)P.max_angles * sizeof(FwdConst) + 127) & ~(size_t)127;
  const int WX = P.WX, WY = P.WY;
  const int win_elems = WX * WY;
  const size_t stage_bytes = ((size_t)win_elems * 4 + 127) & ~(size_t)127;
  unsigned char* win0 = smem + kc_bytes + 128;
  float* red = reinterpret_cast<float*>(smem + kc_bytes);  // 32 floats for the block max

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  int* urow = reinterpret_cast<int*>(win0 + kStages * stage_bytes) + warp * WX;  // kept zero between uses
  for (int i = lane; ROWS && i < WX; i += 32) urow[i] = 0;
  const int A = P.ax.A;
  const int a_begin = (int)((long long)A * g / P.groups), a_end = (int)((long long)A * (g + 1) / P.groups);
  const int na = a_end - a_begin;
  const int X0 = P.vol.Xs + bx * BX;
  const int Y0 = P.vol.Ys + by * BY;
  const int Z0 = P.z0 + zb * NZ;
  const int PX = P.ax.PX, PY = P.ax.PY;

  for (int j = tid; j < na; j += kThreads) {
    const int a = a_begin + j;
    const double* cx = P.ax.xc + 4 * a;
    const double* cy = P.ax.yc + 4 * a;
    const double xb = cx[0] + cx[1] * X0 + cx[2] * Y0 + cx[3] * Z0 - 1.0;
    const double yb = cy[0] + cy[1] * X0 + cy[2] * Y0 + cy[3] * Z0 - 1.0;
    const double fxb = floor(fmin(fmax(xb, -1.0e9), 1.0e9)), fyb = floor(fmin(fmax(yb, -1.0e9), 1.0e9));
    FwdConst k;
    k.xf = (float)(xb - fxb);
    k.yf = (float)(yb - fyb);
    k.a1 = (float)cx[1]; k.a2 = (float)cx[2]; k.a3 = (float)cx[3];
    k.b1 = (float)cy[1]; k.b2 = (float)cy[2]; k.b3 = (float)cy[3];
    const int xi = (int)fxb, yi = (int)fyb;
    const float xmin = k.xf + fminf(0.f, k.a1 * (BX - 1)) + fminf(0.f, k.a2 * (BY - 1)) + fminf(0.f, k.a3 * (NZ - 1));
    const float ymin = k.yf + fminf(0.f, k.b1 * (BX - 1)) + fminf(0.f, k.b2 * (BY - 1)) + fminf(0.f, k.b3 * (NZ - 1));
    const int ox0 = floor_div(xi + (int)floorf(xmin) - 1, 4) * 4;
    const int oy0 = yi + (int)floorf(ymin) - 1;
    // clamp inside [0, pitch - WX] x [0, PY - WY]; the host checked both ranges exist
    const int ox = min(max(ox0, 0), P.ax.pitch - WX);
    const int oy = min(max(oy0, 0), PY - WY);
    k.ox = ox;
    k.oy = oy;
    k.lxm = xi - ox - kMagicBits;
    k.lym = yi - oy - kMagicBits;
    k.wlx = min(WX, PX - ox);
    // An unclamped window holds the whole footprint; inside the detector every tap is kept.
    k.interior = (ox == ox0 && oy == oy0 && ox + WX <= PX) ? 1 : 0;
    kc[j] = k;
  }

  // own voxels, loaded once (coalesced along lanes), and the brick's max |v|
  // lanes: 0 each warp a line along X, 1 a line along Y, 2 an 8x4 patch
  const int tx = lanes == 0 ? lane : lanes == 1 ? warp : (warp & 1) * 8 + (lane & 7);
  const int ty = lanes == 0 ? warp : lanes == 1 ? lane : (warp >> 1) * 4 + (lane >> 3);
  const bool active = (X0 + tx < P.vol.Xs + P.vol.NX) && (Y0 + ty < P.vol.Ys + P.vol.NY);
  float v[NZ];
  float vmax = 0.f;
  {
    const long long sx = P.vol.NX, sxy = (long long)P.vol.NX * P.vol.NY;
    const long long base = (long long)(X0 + tx - P.vol.Xs) + (long long)(Y0 + ty - P.vol.Ys) * sx + stream_wait();
#pragma unroll
    for (int z = 0; z < NZ; ++z) {
      const int zz = Z0 + z;
      v[z] = 0.f;
      if (active && zz < P.z1) v[z] = P.x ? ldv<VT>(P.x, base + (long long)(zz - P.z0) * sxy) : 1.f;
      vmax = fmaxf(vmax, fabsf(v[z]));
    }
  }
  for (int o = 16; o > 0; o >>= 1) vmax = fmaxf(vmax, __shfl_xor_sync(0xffffffffu, vmax, o));
  if (lane == 0) red[warp] = vmax;
  zero_window(reinterpret_cast<int*>(win0), win_elems);  // the first angle's stage
  __syncthreads();
  vmax = red[0];
  for (int w = 1; w < kWarps; ++w) vmax = fmaxf(vmax, red[w]);
  // S = 2^(b-e) with vmax < 2^e, so |v*S| < 2^b.  One emitted value merges at
  // most NZ voxels of weight <= 1 each: |emission| < 2^(b + log2 NZ) <= 2^21,
  // the range of the magic rounding.  A pixel's window sum stays below
  // 2^(b + mass_shift) <= 2^30 (no int overflow).
  int e2 = 0;
  if (vmax > 0.f && isfinite(vmax)) frexpf(vmax, &e2);
  constexpr int kLog2NZ = NZ >= 32 ? 5 : NZ >= 16 ? 4 : 3;
  const int bits = min(21 - kLog2NZ, 30 - P.mass_shift);
  const int sexp = max(-120, min(120, bits - e2));
  const float S = ldexpf(1.f, sexp), invS = ldexpf(1.f, -sexp);
#pragma unroll
  for (int z = 0; z < NZ; ++z) v[z] *= S;
  if (tid == 0) prefetch_tensormap(smap);

  // Three window stages: angle j splats into stage j % 3 (zeroed while angle
  // j - 1 was flushed), then converts it while zeroing the stage of angle
  // j + 1, whose last reader (the bulk reduce of angle j - 2) has finished.
  // Two block barriers per angle.
  for (int j = 0; j < na; ++j) {
    const int a = a_begin + j;
    const int st = j % kStages;
    int* wi = reinterpret_cast<int*>(win0 + st * stage_bytes);
    const FwdConst k = kc[j];
    if constexpr (ROWS) {
      const float xr = fmaf(k.a2, (float)ty, fmaf(k.a1, (float)tx, k.xf));
      const float yr = lanes == 1 ? fmaf(k.b1, (float)tx, k.yf) : fmaf(k.b2, (float)ty, k.yf);  // (the warp's)
      const float fly = floorf(yr);
      const float fy = yr - fly;
      const int rowi = magic_int(fly) + k.lym;
      const uint32_t row = smem_u32(wi) + 4u * (uint32_t)(rowi * WX);
      if (k.interior) {
        if (active) splat_walk<NZ>(v, smem_u32(urow), xr, k.a3, k.lxm, [](uint32_t q, float e) { red_shared(q, fixq(1.f, e)); });
        split_row(urow, WX, row, fy);
      } else if (active) {  // clamped at the detector edge: taps off it are dropped
        const uint32_t span = 4u * (uint32_t)k.wlx, drow = 4u * (uint32_t)WX;
        const bool y0ok = (unsigned)rowi < (unsigned)WY, y1ok = (unsigned)(rowi + 1) < (unsigned)WY;
        splat_walk<NZ>(v, row, xr, k.a3, k.lxm, [&](uint32_t q, float e) {
          const bool xok = q - row < span;
          if (xok && y0ok) red_shared(q, fixq(1.f - fy, e));
          if (xok && y1ok) red_shared(q + drow, fixq(fy, e));
        });
      }
    } else if (active && fabsf(k.a3) < 0.999f && fabsf(k.b3) < 0.999f) {
      const float xr = fmaf(k.a2, (float)ty, fmaf(k.a1, (float)tx, k.xf));
      const float yr = fmaf(k.b2, (float)ty, fmaf(k.b1, (float)tx, k.yf));
      if (k.interior) stream_column_zy<NZ, false>(smem_u32(wi), WX, WY, v, xr, yr, k);
      else stream_column_zy<NZ, true>(smem_u32(wi), WX, WY, v, xr, yr, k);
    } else if (active) {
      const float xr = fmaf(k.a2, (float)ty, fmaf(k.a1, (float)tx, k.xf));
      const float yr = fmaf(k.b2, (float)ty, fmaf(k.b1, (float)tx, k.yf));
#pragma unroll
      for (int z = 0; z < NZ; ++z) {
        const float y = fmaf(k.b3, (float)z, yr);
        const float fly = floorf(y);
        const float fy = y - fly;
        const int rowi = magic_int(fly) + k.lym;
        const float wy0 = 1.f - fy, wy1 = fy;
        const bool y0ok = (unsigned)rowi < (unsigned)WY;
        const bool y1ok = (unsigned)(rowi + 1) < (unsigned)WY;
        const float x = fmaf(k.a3, (float)z, xr);
        const float flx = floorf(x);
        const float fx = x - flx;
        const int ix = magic_int(flx) + k.lxm;
        const bool x0ok = (unsigned)ix < (unsigned)k.wlx;
        const bool x1ok = (unsigned)(ix + 1) < (unsigned)k.wlx;
        const float g0 = wy0 * v[z], g1 = wy1 * v[z];
        const float wx0 = 1.f - fx;
        int* r0 = wi + (rowi * WX + ix);
        if (y0ok) {
          if (x0ok) red_shared(smem_u32(r0), fixq(wx0, g0));
          if (x1ok) red_shared(smem_u32(r0 + 1), fixq(fx, g0));
        }
        if (y1ok) {
          if (x0ok) red_shared(smem_u32(r0 + WX), fixq(wx0, g1));
          if (x1ok) red_shared(smem_u32(r0 + WX + 1), fixq(fx, g1));
        }
      }
    }
    flush_window(smap, wi, reinterpret_cast<int*>(win0 + ((j + 1) % kStages) * stage_bytes), win_elems, invS, j,
                 j + 1 < na, k.ox, k.oy, a);
  }
  if (tid == 0) bulk_wait_all();
}

// One CTA per (brick, angle group) of one axis.  NZ: the depth of the voxel
// walk (z-dependent y-maps), or for the prefix sums, whose depth is P.nz, 0, or
// kSteepAxis with the voxel by voxel path (which costs the others 0.5 %).
constexpr int kSteepAxis = -1;
template <typename VT, int NZ, bool ROWS>
__global__ void __launch_bounds__(kThreads)
fwd_tma_kernel(const __grid_constant__ CUtensorMap smap, const __grid_constant__ FwdArgs P, int lanes) {
  extern __shared__ __align__(128) unsigned char smem[];
  if constexpr (NZ <= 0)
    prefix_brick<VT, NZ == kSteepAxis>(&smap, P, lanes, blockIdx.x, blockIdx.y, blockIdx.z / P.groups, blockIdx.z % P.groups, smem);
  else
    fwd_brick<VT, NZ, ROWS>(&smap, P, lanes, blockIdx.x, blockIdx.y, blockIdx.z / P.groups, blockIdx.z % P.groups, smem);
}

// Dynamic shared memory: per-angle constants, block-max scratch, window stages
// and the columns' prefix sums or (rows) a row per warp.
size_t fwd_smem(int WX, int WY, int nz, bool prefix, bool rows, int angles) {
  const size_t stage = (((size_t)WX * WY * 4) + 127) & ~(size_t)127;
  const size_t k = (size_t)angles * (prefix ? sizeof(PreConst) : sizeof(FwdConst));
  return ((k + 127) & ~(size_t)127) + 128 + kStages * stage + (prefix ? (size_t)(nz + 1) * kPreStride : 0) +
         (rows ? (size_t)kWarps * WX * 4 : 0);
}

template <typename VT, int NZ, bool ROWS = false>
cudaError_t launch_one(const CUtensorMap& map, FwdArgs P, int lanes, int num_sms, cudaStream_t st) {
  auto kern = fwd_tma_kernel<VT, NZ, ROWS>;
  const int BX = brick_x(lanes), BY = brick_y(lanes);
  const dim3 b3((P.vol.NX + BX - 1) / BX, (P.vol.NY + BY - 1) / BY, (P.z1 - P.z0 + P.nz - 1) / P.nz);
  const long long bricks = (long long)b3.x * b3.y * b3.z;
  // split the angles over several CTAs when there are too few bricks to fill the GPU
  const long long target = (long long)num_sms * 8;
  int groups = (int)std::min<long long>((target + bricks - 1) / bricks, (long long)P.ax.A);
  if (groups < 1) groups = 1;
  P.groups = groups;
  P.max_angles = (P.ax.A + groups - 1) / groups;
  const size_t smem = fwd_smem(P.WX, P.WY, P.nz, NZ <= 0, ROWS, P.max_angles);
  cudaError_t e = allow_shared_memory(kern, smem);
  if (e != cudaSuccess) return e;
  launch_overlapped(kern, dim3(b3.x, b3.y, b3.z * groups), kThreads, smem, st, map, P, lanes);
  const cudaError_t le = cudaGetLastError();
  if (le == cudaSuccess) g_windowed_launches.fetch_add(1, std::memory_order_relaxed);
  return le;
}

}  // namespace

namespace {

// Persistent forward splat over the bricks of many axes (one angle group per
// brick): each CTA takes items blockIdx.x, blockIdx.x + gridDim.x, ...; every
// brick ends with its bulk reduces complete, so the next one reuses the
// shared-memory windows after a barrier.
template <typename VT>
__global__ void __launch_bounds__(kThreads)
fwd_batch_kernel(const FwdBatchDesc* __restrict__ descs, const long long* __restrict__ first, int n_desc,
                 long long n_items) {
  extern __shared__ __align__(128) unsigned char smem[];
  // The item's arguments are staged in shared memory (no registers held).
  __shared__ FwdArgs sP;
  __shared__ const CUtensorMap* sMap;
  __shared__ int sB[5];  // brick x, y, z, depth, lanes * 2 + bz0
  for (long long it = blockIdx.x; it < n_items; it += gridDim.x) {
    __syncthreads();
    if (threadIdx.x == 0) {
      const int2 item = work_item(first, n_desc, it);
      const FwdBatchDesc& D = descs[item.x];
      sP = FwdArgs{D.ax, D.vol, D.vol.Zs, D.vol.Zs + D.vol.NZ, D.WX, D.WY, 1, D.ax.A, D.mass_shift, D.nz, D.x};
      sMap = D.map;
      sB[0] = item.y % D.gx;
      sB[1] = (item.y / D.gx) % D.gy;
      sB[2] = item.y / (D.gx * D.gy);
      sB[3] = D.nz;
      sB[4] = D.lanes * 2 + D.bz0;
    }
    __syncthreads();
    if (sB[4] & 1) prefix_brick<VT, true>(sMap, sP, sB[4] >> 1, sB[0], sB[1], sB[2], 0, smem);
    else if (sB[3] == 8) fwd_brick<VT, 8, false>(sMap, sP, sB[4] >> 1, sB[0], sB[1], sB[2], 0, smem);
    else if (sB[3] == 32) fwd_brick<VT, 32, false>(sMap, sP, sB[4] >> 1, sB[0], sB[1], sB[2], 0, smem);
    else fwd_brick<VT, 16, false>(sMap, sP, sB[4] >> 1, sB[0], sB[1], sB[2], 0, smem);
  }
}

}  // namespace

template <typename VT>
int forward_batch_ctas_per_sm(size_t smem) {
  int n = 0;
  if (allow_shared_memory(fwd_batch_kernel<VT>, smem) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, fwd_batch_kernel<VT>, kThreads, smem) != cudaSuccess) {
    cudaGetLastError();
    return 1;
  }
  return n > 0 ? n : 1;
}

template <typename VT>
cudaError_t launch_forward_batch(const FwdBatchDesc* descs, const long long* first, int n_desc, long long n_items,
                                 size_t smem, int grid, cudaStream_t st) {
  cudaError_t e = allow_shared_memory(fwd_batch_kernel<VT>, smem);
  if (e != cudaSuccess) return e;
  launch_overlapped(fwd_batch_kernel<VT>, grid, kThreads, smem, st, descs, first, n_desc, n_items);
  const cudaError_t le = cudaGetLastError();
  if (le == cudaSuccess) g_windowed_launches.fetch_add(1, std::memory_order_relaxed);
  return le;
}

template int forward_batch_ctas_per_sm<float>(size_t);
template int forward_batch_ctas_per_sm<__nv_bfloat16>(size_t);
template int forward_batch_ctas_per_sm<__half>(size_t);
template cudaError_t launch_forward_batch<float>(const FwdBatchDesc*, const long long*, int, long long, size_t,
                                                  int, cudaStream_t);
template cudaError_t launch_forward_batch<__nv_bfloat16>(const FwdBatchDesc*, const long long*, int, long long,
                                                          size_t, int, cudaStream_t);
template cudaError_t launch_forward_batch<__half>(const FwdBatchDesc*, const long long*, int, long long, size_t,
                                                   int, cudaStream_t);

namespace {

// Largest z slope from which an axis along a volume axis sums rows per warp (those
// below 0.999 run on lines): at 1.04, 1.30, 1.73, 2.6 and 3.5 pixels per voxel
// (256x256x64, 61 angles) 0.200, 0.188, 0.186, 0.219 and 0.303 ms against 0.172,
// 0.203, 0.245, 0.331 and 0.455 over prefix sums.
constexpr double kRowsSlope = 1.2;
FwdPlan plan_forward_uncached(const std::vector<double>& xc, const std::vector<double>& yc, int A, int PX, int PY,
                              int pitch, int nz, int lane) {
  FwdPlan p;
  double sx = 0, sy = 0;
  bool bz0 = true;
  for (int a = 0; a < A; ++a) {
    sx += std::fabs(xc[4 * a + 1]) - std::fabs(yc[4 * a + 1]);
    sy += std::fabs(xc[4 * a + 2]) - std::fabs(yc[4 * a + 2]);
    if (yc[4 * a + 3] != 0.0) bz0 = false;
  }
  // lane: -1 heuristic (lines along X or Y), 0 lines along X, 1 along Y, 2 8x4 patches
  p.lanes = lane < 0 ? (sy > sx ? 1 : 0) : std::min(lane, 2);
  p.bz0 = bz0;
  for (int a = 0; a < A; ++a)
    if (std::fabs((float)xc[4 * a + 3]) >= kSteep) p.steep = true;
  p.nz = nz;
  // the rows are the warp's own (their y moves by less than 1e-6 px along the lanes)
  double top = 0.0;
  p.rows = bz0 && p.lanes != 2 && (nz == 8 || nz == 16 || nz == 32);
  for (int a = 0; a < A; ++a) {
    top = std::max(top, std::fabs(xc[4 * a + 3]));
    if (!(std::fabs(yc[4 * a + (p.lanes == 1 ? 2 : 1)]) < 3e-8)) p.rows = false;
  }
  if (!(top >= kRowsSlope)) p.rows = false;
  const int BX = brick_x(p.lanes), BY = brick_y(p.lanes), BZ = p.nz;
  double ex = 0, ey = 0;
  for (int a = 0; a < A; ++a) {
    ex = std::max(ex, std::fabs(xc[4 * a + 1]) * (BX - 1) + std::fabs(xc[4 * a + 2]) * (BY - 1) +
                          std::fabs(xc[4 * a + 3]) * (BZ - 1));
    ey = std::max(ey, std::fabs(yc[4 * a + 1]) * (BX - 1) + std::fabs(yc[4 * a + 2]) * (BY - 1) +
                          std::fabs(yc[4 * a + 3]) * (BZ - 1));
  }
  const int wx_min = ((int)std::ceil(ex) + 4 + 4 + 3) / 4 * 4;
  p.WY = (int)std::ceil(ey) + 4;
  auto smem_for = [&](int WX) { return fwd_smem(WX, p.WY, p.nz, bz0 && !p.rows, p.rows, A); };  // (one angle group)
  // Row pitch (= box width) with the fewest shared-memory bank conflicts of
  // the warp's splat atomics, searched over a few widths only: a wider window
  // leaves the interior fast path at more bricks near the detector edge.
  p.WX = wx_min;
  double best = 1e30;
  for (int WX = wx_min; WX <= std::min(std::min(256, pitch), wx_min + 16); WX += 4) {
    if (WX > wx_min && smem_for(WX) > (size_t)(228 * 1024 / 4 - 1024)) break;
    const double c = window_bank_cost(xc, yc, A, p.lanes, p.nz, WX);
    if (c < best - 1e-9) {
      best = c;
      p.WX = WX;
    }
  }
  p.smem = smem_for(p.WX);
  // Weight a pixel can receive from one brick: per Z plane at most the number
  // of voxels whose taps reach it, i.e. lattice points in the preimage of a
  // 2x2-pixel square under the in-plane map J (bounding box of J^-1 [-1,1]^2).
  double count = 0;
  bool singular = false;
  for (int a = 0; a < A; ++a) {
    const double j00 = xc[4 * a + 1], j01 = xc[4 * a + 2], j10 = yc[4 * a + 1], j11 = yc[4 * a + 2];
    const double det = j00 * j11 - j01 * j10;
    if (std::fabs(det) < 1e-3) { singular = true; break; }
    const double wx = 2.0 * (std::fabs(j11) + std::fabs(j01)) / std::fabs(det);
    const double wy = 2.0 * (std::fabs(j10) + std::fabs(j00)) / std::fabs(det);
    count = std::max(count, (wx + 1.0) * (wy + 1.0));
  }
  p.mass_shift = (int)std::ceil(std::log2(std::max(1.0, count * BZ)));
  p.ok = !singular && p.mass_shift <= 16 && p.WX <= 256 && p.WY <= 256 && p.WX <= pitch && p.WY <= PY &&
         p.smem <= 227 * 1024 && (bz0 ? p.nz >= 1 && p.nz <= 32 : p.nz == 8 || p.nz == 16 || p.nz == 32);
  (void)PX;
  return p;
}

PlanMemo<FwdPlan> g_fwd_plans;

}  // namespace

FwdPlan plan_forward(const std::vector<double>& xc, const std::vector<double>& yc, int A, int PX, int PY, int pitch,
                     int nz, int lane) {
  return g_fwd_plans.get(plan_key(xc, yc, A, {PX, PY, pitch, nz, lane}),
                         [&] { return plan_forward_uncached(xc, yc, A, PX, PY, pitch, nz, lane); });
}

template <typename VT>
cudaError_t launch_forward_tma(const CUtensorMap& smap, const FwdPlan& plan, const AxisDev& ax, const VolDev& vol,
                               const VT* x, int z0, int z1, cudaStream_t st) {
  const int sms = device_sm_count();
  const FwdArgs P{ax, vol, z0, z1, plan.WX, plan.WY, 1, ax.A, plan.mass_shift, plan.nz, x};
  if (plan.rows) {
    if (plan.nz == 8) return launch_one<VT, 8, true>(smap, P, plan.lanes, sms, st);
    if (plan.nz == 32) return launch_one<VT, 32, true>(smap, P, plan.lanes, sms, st);
    return launch_one<VT, 16, true>(smap, P, plan.lanes, sms, st);
  }
  if (plan.bz0 && plan.steep) return launch_one<VT, kSteepAxis>(smap, P, plan.lanes, sms, st);
  if (plan.bz0) return launch_one<VT, 0>(smap, P, plan.lanes, sms, st);
  if (plan.nz == 8) return launch_one<VT, 8>(smap, P, plan.lanes, sms, st);
  if (plan.nz == 32) return launch_one<VT, 32>(smap, P, plan.lanes, sms, st);
  return launch_one<VT, 16>(smap, P, plan.lanes, sms, st);
}

template cudaError_t launch_forward_tma<float>(const CUtensorMap&, const FwdPlan&, const AxisDev&, const VolDev&,
                                               const float*, int, int, cudaStream_t);
template cudaError_t launch_forward_tma<__nv_bfloat16>(const CUtensorMap&, const FwdPlan&, const AxisDev&,
                                                       const VolDev&, const __nv_bfloat16*, int, int, cudaStream_t);
template cudaError_t launch_forward_tma<__half>(const CUtensorMap&, const FwdPlan&, const AxisDev&, const VolDev&,
                                                const __half*, int, int, cudaStream_t);

}  // namespace mtr
