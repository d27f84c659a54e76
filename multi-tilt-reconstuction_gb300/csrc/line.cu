// Projector pair on line images (see line.cuh): forward line sums, line
// back-projection and the step between line images and the detector.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <type_traits>

#include "line.cuh"
#include "tma.cuh"

namespace mtr {

namespace {

constexpr int kWarps = 8;            // compute warps: one m position each
constexpr int kThreads = kWarps * 32;
constexpr int kFwdStages = 3;        // window stages in flight (splat, flush, next)
constexpr int kBpStages = 4;         // loaded windows in flight
constexpr int kBpThreads = kThreads + 32;  // and a producer warp
constexpr uint32_t kDrainIters = 1u << 24;
constexpr float kMagic = 12582912.0f;  // 1.5 * 2^23
constexpr int kMagicBits = 0x4B400000;
constexpr int kMaxRows = 128;  // window rows at most

// Pairs of FP32 values in one 64-bit register: Blackwell's FFMA2 takes one
// issue slot for two fused multiply-adds.
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float a, float b) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float2 unpack2(f32x2 v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 sub2(f32x2 a, f32x2 b) { return fma2(b, 0xBF800000BF800000ull, a); }
__device__ __forceinline__ f32x2 lds_pair(uint32_t a) {
  f32x2 v;
  asm volatile("ld.shared.b64 %0, [%1];" : "=l"(v) : "r"(a));
  return v;
}
struct Weights {  // {1 - f, 1 - f} and {f, f} of one plane of a column
  f32x2 a, b;
};
__device__ __forceinline__ Weights lds_weights(uint32_t at) {
  Weights w;
  asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(w.a), "=l"(w.b) : "r"(at));
  return w;
}
__device__ __forceinline__ void red_shared(uint32_t addr, int v) {
  asm volatile("red.shared.add.s32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}
template <typename VT> __device__ __forceinline__ float ldv(const VT* p, long long i);
template <> __device__ __forceinline__ float ldv<float>(const float* p, long long i) { return __ldg(p + i); }
template <> __device__ __forceinline__ float ldv<__nv_bfloat16>(const __nv_bfloat16* p, long long i) {
  return __bfloat162float(__ldg(p + i));
}
template <> __device__ __forceinline__ float ldv<__half>(const __half* p, long long i) {
  return __half2float(__ldg(p + i));
}
template <typename BT> __device__ __forceinline__ float ldb(const BT* p);
template <> __device__ __forceinline__ float ldb<float>(const float* p) { return __ldg(p); }
template <> __device__ __forceinline__ float ldb<__half>(const __half* p) { return __half2float(__ldg(p)); }

struct LineArgs {
  AxisDev ax;
  VolDev vol;
  int along_x, z0, z1;
  int rows;        // window rows (detector columns x)
  int groups;      // forward: angle groups (grid.z = z blocks * groups)
  int max_angles;
};

// Per-angle constants of a brick.  A column (fixed m) is walked with z
// growing; where a3 < 0 in the mirrored coordinate u = -x, whose pixel p is
// detector column -p, so that one walk serves both signs.
struct __align__(16) LineConst {
  float xf, am, a3;  // x at (m0, z0) relative to base, and its slopes
  int base;          // detector column of xf = 0 minus the window origin
  int ox;            // window origin
  int interior;      // forward: the window holds the whole footprint
  float scale, inv_scale;
};

struct LineBase {  // x of the brick's first column and plane
  double x;
  double am, a3;
};
__device__ __forceinline__ LineBase line_base(const LineArgs& P, int a, int wc, int m0, int z0) {
  const double* c = P.ax.xc + 4 * a;
  const double X = P.along_x ? P.vol.Xs + wc : P.vol.Xs + m0, Y = P.along_x ? P.vol.Ys + m0 : P.vol.Ys + wc;
  LineBase b;
  b.x = c[0] + c[1] * X + c[2] * Y + c[3] * z0 - 1.0;
  b.am = P.along_x ? c[2] : c[1];
  b.a3 = c[3];
  return b;
}
// Integer part of the base, window origin (one column of slack) and fraction.
template <int NZ>
__device__ __forceinline__ int line_origin(const LineBase& b, float& xf, int& xi) {
  const double fl = floor(fmin(fmax(b.x, -1.0e9), 1.0e9));
  xf = (float)(b.x - fl);
  xi = (int)fl;
  const float am = (float)b.am, a3 = (float)b.a3;
  const float xmin = xf + fminf(0.f, am * (kWarps - 1)) + fminf(0.f, a3 * (NZ - 1));
  return xi + (int)floorf(xmin) - 1;
}

// A column's walk at one angle.  Its position is the same for all lanes, so
// the lanes share the work of laying it out: lane z takes plane z, writes the
// plane's two weights to the warp's table (16 bytes, read back by all lanes
// with one broadcast load per plane, already paired), and votes whether the
// column enters a new pixel there; the vote is uniform, and so are the
// branches on it.
struct Walk {
  int pix, dir;        // first detector column relative to the window, direction
  unsigned cross;      // bit z: plane z lies one pixel further than plane z - 1
  int lane_pix;        // the lane's plane: its detector column relative to the window,
  float lane_f;        // and its fraction towards the next
};
template <int NZ>
__device__ __forceinline__ Walk lay_out_walk(const LineConst& k, int m, int lane, float4* table) {
  Walk w;
  w.dir = k.a3 >= 0.f ? 1 : -1;
  const float x = fmaf(k.am, (float)m, k.xf);
  const float u = w.dir > 0 ? x : -x;
  const float uz = fmaf(fabsf(k.a3), (float)min(lane, NZ - 1), u);
  const float fl = floorf(uz), f = uz - fl;
  __syncwarp();  // the table's last reads are done
  if (lane < NZ) table[lane] = make_float4(1.f - f, 1.f - f, f, f);
  const float before = __shfl_up_sync(0xffffffffu, fl, 1);
  w.cross = __ballot_sync(0xffffffffu, lane > 0 && fl != before);
  w.pix = k.base + w.dir * (__float_as_int(__fadd_rn(floorf(u), kMagic)) - kMagicBits);
  w.lane_pix = k.base + w.dir * (__float_as_int(__fadd_rn(fl, kMagic)) - kMagicBits);
  w.lane_f = f;
  __syncwarp();
  return w;
}

// ---- forward -----------------------------------------------------------------
// Line sums of a brick of 32*VL line positions x 8 columns x NZ planes, held
// in registers for all angles of the CTA's group.  Per angle each warp walks
// its column: the two running sums of the current pixel and the next are
// updated with two packed multiply-adds per pair of values, and a pixel is
// added to the shared window (one red.shared per value: fixed point, as there
// is no native shared float add) when the column leaves it.  The value is
// added with the rounding constant's bits still on it, 0x4B400000 per
// addition; a counter per window row says how many to take off again.  The
// window is converted and flushed with one TMA reduce-add, three stages
// rotating as in fwd_tma_kernel.
//
// 16 planes x 4 values fill the registers of 16 warps per SM; bound by the
// issue of those warps (6.7 warp instructions per 32 visits at half the issue
// slots, 1.9 shared wavefronts) against 20 in the general splat.  512x512x64,
// 61 angles: 0.34 ms against 0.62 ms; 1024x1024x96, 121 angles: 3.5 against 6.8 ms.
template <typename VT, int VL, int NZ>
__global__ void __launch_bounds__(kThreads, VL * NZ >= 64 ? 2 : VL * NZ >= 32 ? 4 : 5)
line_forward_kernel(const __grid_constant__ CUtensorMap map, const LineArgs P, const VT* __restrict__ x) {
  extern __shared__ __align__(128) unsigned char smem[];
  constexpr int BW = 32 * VL;
  constexpr int VP = VL / 2;
  LineConst* kc = reinterpret_cast<LineConst*>(smem);
  const size_t kc_bytes = ((size_t)P.max_angles * sizeof(LineConst) + 127) & ~(size_t)127;
  float* red = reinterpret_cast<float*>(smem + kc_bytes);
  float4* table = reinterpret_cast<float4*>(smem + kc_bytes + 128) + (threadIdx.x >> 5) * NZ;
  int* count0 = reinterpret_cast<int*>(smem + kc_bytes + 128 + kWarps * NZ * sizeof(float4));  // [stages][kMaxRows]
  unsigned char* win0 = reinterpret_cast<unsigned char*>(count0 + kFwdStages * kMaxRows);
  const int win_elems = P.rows * BW;
  const size_t stage_bytes = (size_t)win_elems * 4;  // a multiple of 128: BW >= 64

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int w0 = blockIdx.x * BW, m0 = blockIdx.y * kWarps;
  const int zb = blockIdx.z / P.groups, g = blockIdx.z % P.groups;
  const int Z0 = P.z0 + zb * NZ;
  const int A = P.ax.A;
  const int a_begin = (int)((long long)A * g / P.groups), a_end = (int)((long long)A * (g + 1) / P.groups);
  const int na = a_end - a_begin;
  const int W = P.along_x ? P.vol.NX : P.vol.NY, M = P.along_x ? P.vol.NY : P.vol.NX;
  const long long sx = P.vol.NX, sxy = (long long)P.vol.NX * P.vol.NY;

  const long long after = stream_wait();  // (added to the loads' index)
  // own voxels: value j of a lane is line position w0 + 32 j + lane
  f32x2 v[NZ][VP];
  float vmax = 0.f;
  if (P.along_x) {
    const bool col = m0 + warp < M;
    const long long base = (long long)(m0 + warp) * sx + w0 + lane + after;
#pragma unroll
    for (int z = 0; z < NZ; ++z) {
      float t[VL];
#pragma unroll
      for (int j = 0; j < VL; ++j) {
        t[j] = 0.f;
        if (col && Z0 + z < P.z1 && w0 + 32 * j + lane < W)
          t[j] = x ? ldv<VT>(x, base + 32 * j + (long long)(Z0 + z - P.z0) * sxy) : 1.f;
        vmax = fmaxf(vmax, fabsf(t[j]));
      }
#pragma unroll
      for (int q = 0; q < VP; ++q) v[z][q] = pack2(t[2 * q], t[2 * q + 1]);
    }
  } else {
    // lines along Y: the eight columns are eight neighbours in memory; a plane
    // is read in 32-byte runs, two planes ahead, and handed to the warps through
    // one of two shared-memory tiles
    const int tm = tid & 7, tw = tid >> 3;
    auto load = [&](int z, float (&t)[VL]) {
#pragma unroll
      for (int j = 0; j < VL; ++j) {
        t[j] = 0.f;
        const int w = w0 + 32 * j + tw;
        if (z < NZ && m0 + tm < M && Z0 + z < P.z1 && w < W)
          t[j] = x ? ldv<VT>(x, (long long)w * sx + (m0 + tm) + after + (long long)(Z0 + z - P.z0) * sxy) : 1.f;
        vmax = fmaxf(vmax, fabsf(t[j]));
      }
    };
    float ta[VL], tb[VL];
    load(0, ta);
    load(1, tb);
#pragma unroll
    for (int z = 0; z < NZ; ++z) {
      float* tile = reinterpret_cast<float*>(win0) + (z & 1) * BW * 9;  // [BW][9]
      float(&t)[VL] = z & 1 ? tb : ta;
#pragma unroll
      for (int j = 0; j < VL; ++j) tile[(32 * j + tw) * 9 + tm] = t[j];
      load(z + 2, t);
      __syncthreads();
#pragma unroll
      for (int q = 0; q < VP; ++q)
        v[z][q] = pack2(tile[(64 * q + lane) * 9 + warp], tile[(64 * q + 32 + lane) * 9 + warp]);
    }
    __syncthreads();
  }
  for (int o = 16; o > 0; o >>= 1) vmax = fmaxf(vmax, __shfl_xor_sync(0xffffffffu, vmax, o));
  if (lane == 0) red[warp] = vmax;
  for (int i = tid * 4; i < win_elems; i += kThreads * 4)
    *reinterpret_cast<int4*>(reinterpret_cast<int*>(win0) + i) = make_int4(0, 0, 0, 0);
  for (int i = tid; i < P.rows; i += kThreads) count0[i] = 0;
  if (tid == 0) prefetch_tensormap(&map);
  __syncthreads();
  vmax = red[0];
  for (int w = 1; w < kWarps; ++w) vmax = fmaxf(vmax, red[w]);
  int e2 = 0;
  if (vmax > 0.f && isfinite(vmax)) frexpf(vmax, &e2);
  for (int j = tid; j < na; j += kThreads) {
    LineConst k;
    int xi;
    const LineBase b = line_base(P, a_begin + j, w0 + BW / 2, m0, Z0);
    const int ox0 = line_origin<NZ>(b, k.xf, xi);
    k.am = (float)b.am;
    k.a3 = (float)b.a3;
    // the window stays inside the detector (a TMA reduce may not start below 0)
    k.ox = min(max(ox0, 0), P.ax.PX - P.rows);
    k.interior = k.ox == ox0;
    k.base = xi - k.ox;
    // |v| < 2^e; an emission sums at most w = min(NZ, 1 + 1/slope) <= 2^lw of
    // them and stays below 2^21 (the rounding addition's range); a window
    // element gathers at most 8 NZ voxels, so its sum stays below 2^29
    const float st = fabsf(k.a3);
    const int lw = log2_ceil(fminf((float)NZ, 1.f + (st > 1e-30f ? 1.f / st : 1e30f)));
    const int sexp = max(-120, min(120, 21 - lw - e2));
    k.scale = ldexpf(1.f, sexp);
    k.inv_scale = ldexpf(1.f, -sexp);
    kc[j] = k;
  }
  __syncthreads();

  const bool active = m0 + warp < M;
#pragma unroll 1
  for (int j = 0; j < na; ++j) {
    int* wi = reinterpret_cast<int*>(win0 + (j % kFwdStages) * stage_bytes);
    float* wf = reinterpret_cast<float*>(wi);
    const LineConst k = kc[j];
    int* count = count0 + (j % kFwdStages) * kMaxRows;
    if (active) {
      const Walk s = lay_out_walk<NZ>(k, warp, lane, table);
      const uint32_t tab = smem_u32(table);
      uint32_t at = smem_u32(wi) + 4u * (uint32_t)(s.pix * BW + lane);
      const uint32_t dstep = s.dir > 0 ? 4u * BW : 0u - 4u * BW;
      const f32x2 scale = pack2(k.scale, k.scale), magic = pack2(kMagic, kMagic);
      {  // every pixel from the first to one past the last is added to once
        const int row = s.pix + s.dir * lane;
        if (lane < __popc(s.cross) + 2 && (unsigned)row < (unsigned)P.rows) red_shared(smem_u32(count + row), 1);
      }
      // CHK: the window is clamped at the detector edge, and pixels off it are dropped
      auto walk = [&](auto chk) {
        constexpr bool CHK = decltype(chk)::value;
        int pix = s.pix;
        auto emit = [&](uint32_t q, int row, const f32x2 (&e)[VP]) {
          if (CHK && (unsigned)row >= (unsigned)P.rows) return;
#pragma unroll
          for (int p = 0; p < VP; ++p) {
            const float2 t = unpack2(fma2(scale, e[p], magic));
            red_shared(q + 256u * p, __float_as_int(t.x));
            red_shared(q + 256u * p + 128u, __float_as_int(t.y));
          }
        };
        f32x2 c0[VP], c1[VP];  // sums of the current pixel and the next
        Weights w = lds_weights(tab), next = lds_weights(tab + 16u);  // (a plane ahead of their use)
#pragma unroll
        for (int p = 0; p < VP; ++p) {
          c0[p] = mul2(w.a, v[0][p]);
          c1[p] = mul2(w.b, v[0][p]);
        }
#pragma unroll
        for (int z = 1; z < NZ; ++z) {
          w = next;
          if (z + 1 < NZ) next = lds_weights(tab + 16u * (z + 1));
          if (s.cross & (1u << z)) {  // the column left the pixel
            emit(at, pix, c0);
            at += dstep;
            if (CHK) pix += s.dir;
#pragma unroll
            for (int p = 0; p < VP; ++p) {
              c0[p] = fma2(w.a, v[z][p], c1[p]);
              c1[p] = mul2(w.b, v[z][p]);
            }
          } else {
#pragma unroll
            for (int p = 0; p < VP; ++p) {
              c0[p] = fma2(w.a, v[z][p], c0[p]);
              c1[p] = fma2(w.b, v[z][p], c1[p]);
            }
          }
        }
        emit(at, pix, c0);
        emit(at + dstep, pix + s.dir, c1);
      };
      if (k.interior) walk(std::false_type{});
      else walk(std::true_type{});
    }
    // the bulk reduce of angle j - 2 (the next stage's last reader) must be done reading
    if (tid == 0 && j >= 2) bulk_wait_read<1>();
    __syncthreads();
    const float inv = k.inv_scale;
    const bool more = j + 1 < na;
    int* wn = reinterpret_cast<int*>(win0 + ((j + 1) % kFwdStages) * stage_bytes);
    for (int i = tid; more && i < P.rows; i += kThreads) count0[((j + 1) % kFwdStages) * kMaxRows + i] = 0;
    for (int i = tid * 4; i < win_elems; i += kThreads * 4) {
      int4 q = *reinterpret_cast<const int4*>(wi + i);
      const int off = (int)((uint32_t)count[i / BW] * (uint32_t)kMagicBits);
      q.x -= off; q.y -= off; q.z -= off; q.w -= off;
      *reinterpret_cast<float4*>(wf + i) =
          make_float4((float)q.x * inv, (float)q.y * inv, (float)q.z * inv, (float)q.w * inv);
      if (more) *reinterpret_cast<int4*>(wn + i) = make_int4(0, 0, 0, 0);
    }
    fence_proxy_async_smem();
    __syncthreads();
    if (tid == 0) {
      tma_reduce_add_3d(&map, wf, w0, k.ox, a_begin + j);
      bulk_commit();
    }
  }
  if (tid == 0) bulk_wait_all();
}

// ---- back-projection -----------------------------------------------------------
// Line back-projection of a brick of 32*VL positions x 8 columns x NZ planes
// over all angles.  A producer warp streams the line image's windows ([rows]
// [32*VL], one TMA box per angle) through a ring of stages; each consumer warp
// walks its column with the values of two neighbouring detector columns in
// registers and loads a new one only when the column crosses a pixel.
//
// Bound by instruction issue: two packed multiply-adds per pair of values, one
// broadcast load of the plane's weights and a load per crossing.  8 planes x 4
// values leave 3 CTAs per SM, faster than 16 x 4 at two.  512x512x64, 61
// angles: 0.25 ms against 0.47 ms for the windowed gather; 1024x1024x96, 121
// angles: 2.5 against 4.9-5.5 ms.
//
// The WBP also sums the weights, which separate too: with one row table for all
// angles, sum_a cx(a, m, z) * cy(w).  Lane z keeps the sum of plane z, one
// register in place of one per voxel, and the WBP takes the update's shapes:
// 512x512x64, 61 angles, 0.32 / 0.31 ms (lines along Y / X) against 0.43 / 0.42
// with a sum per voxel, which only maps with a row table per angle still need.
// Its values are interpolated before they are added, from the taps' difference
// formed at each crossing: one rounding per angle at the size of the sum in place
// of two (400x384x40, 61 angles: 1.2e-7 of the 64-bit result against 1.7e-7), 0.31 /
// 0.30 ms.  The update keeps the two multiply-adds, 1 % faster on small volumes.
struct LineBpArgs {
  LineArgs l;
  LineTab tab;
  int Wp;
  float step;
  float* vol_out;
  float* cbp;
  void* vol_copy;
  int copy_kind;
  int* err;
  unsigned wait_iters;
};

// Modes of the back-projection: WBP whose line positions keep their detector
// weight at every angle, SIRT update, WBP with a row table per angle.
constexpr int kWbp = 0, kSirt = 1, kWbpTables = 2;

// The results of N voxels at offsets i from the brick's first voxel (negative:
// none): WBP s/c (0 where c is 0), or the SIRT update, whose N loads are all
// issued before the first use.
struct BrickOut {
  float *x, *cbp;
  void* copy;
  int copy_kind;
  float step;
};
template <int MODE, int N>
__device__ __forceinline__ void finish_voxels(const BrickOut& B, const int (&i)[N], const float (&s)[N],
                                              const float (&c)[N]) {
  float cv[N], xv[N];
#pragma unroll
  for (int q = 0; q < N; ++q) {
    cv[q] = MODE != kSirt ? c[q] : i[q] >= 0 ? B.cbp[i[q]] : 0.f;
    xv[q] = MODE != kSirt || i[q] < 0 ? 0.f : B.x[i[q]];
  }
#pragma unroll
  for (int q = 0; q < N; ++q) {
    if (i[q] < 0) continue;
    float out = xv[q];
    if (cv[q] != 0.f) out = MODE != kSirt ? s[q] / cv[q] : fmaf(B.step, s[q] / cv[q], out);
    if (MODE != kSirt) B.cbp[i[q]] = cv[q];
    if (MODE != kSirt || cv[q] != 0.f) B.x[i[q]] = out;
    if (B.copy_kind == 1) static_cast<__nv_bfloat16*>(B.copy)[i[q]] = __float2bfloat16_rn(out);
    else if (B.copy_kind == 2) static_cast<__half*>(B.copy)[i[q]] = __float2half_rn(out);
  }
}

__host__ __device__ constexpr size_t bp_table_bytes(int nz) { return (size_t)kWarps * nz * sizeof(float4); }

template <int MODE, int VL, int NZ>
__global__ void __launch_bounds__(kBpThreads, VL * NZ >= 64 || (MODE == kWbpTables && VL * NZ >= 32) ? 2 : VL * NZ >= 32 || MODE == kWbpTables ? 3 : 4)
line_bp_kernel(const __grid_constant__ CUtensorMap map, const LineBpArgs P) {
  extern __shared__ __align__(128) unsigned char smem[];
  constexpr int BW = 32 * VL;
  constexpr int VP = VL / 2;
  uint64_t* full = reinterpret_cast<uint64_t*>(smem);
  uint64_t* empty = full + kBpStages;
  LineConst* kc = reinterpret_cast<LineConst*>(smem + 128);
  const LineArgs& L = P.l;
  const int A = L.ax.A;
  const size_t kc_bytes = ((size_t)A * sizeof(LineConst) + 127) & ~(size_t)127;
  float4* table = reinterpret_cast<float4*>(smem + 128 + kc_bytes) + (threadIdx.x >> 5) * NZ;
  unsigned char* win0 = smem + 128 + kc_bytes + bp_table_bytes(NZ);
  const uint32_t stage_bytes = (uint32_t)(L.rows * BW * 4);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // x fastest, then z, then the columns: bricks that read the same windows run together
  const int w0 = blockIdx.x * BW, m0 = blockIdx.z * kWarps;
  const int Z0 = L.z0 + blockIdx.y * NZ;
  const int W = L.along_x ? L.vol.NX : L.vol.NY, M = L.along_x ? L.vol.NY : L.vol.NX;

  if (tid == 0) {
    for (int s = 0; s < kBpStages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], kWarps);
    }
    mbar_fence_init();
  }
  for (int a = tid; a < A; a += kBpThreads) {
    LineConst k;
    int xi;
    const LineBase b = line_base(L, a, w0 + BW / 2, m0, Z0);
    k.ox = line_origin<NZ>(b, k.xf, xi);
    k.am = (float)b.am;
    k.a3 = (float)b.a3;
    k.base = xi - k.ox;
    k.interior = 1;
    k.scale = k.inv_scale = 1.f;
    kc[a] = k;
  }
  __syncthreads();
  stream_wait();

  if (warp == kWarps) {  // producer: one elected lane issues the loads
    if (lane == 0) {
      prefetch_tensormap(&map);
      int issued = 0;
      for (int a = 0; a < A; ++a) {
        const int s = a % kBpStages, n = a / kBpStages;
        if (n > 0 && !mbar_wait_bounded(&empty[s], (uint32_t)((n - 1) & 1), P.wait_iters)) {
          atomicExch(P.err, 2);
          break;
        }
        mbar_arrive_expect_tx(&full[s], stage_bytes);
        tma_load_3d(win0 + (size_t)s * stage_bytes, &map, w0, kc[a].ox, a, &full[s]);
        issued = a + 1;
      }
      // every load issued lands before exit
      for (int s = 0; s < kBpStages && s < issued; ++s) {
        const int n_last = (issued - 1 - s) / kBpStages;
        if (!mbar_wait_bounded(&full[s], (uint32_t)(n_last & 1), kDrainIters)) atomicExch(P.err, 3);
      }
    }
    __syncwarp();
    __syncthreads();  // (the windows' memory is reused by the epilogue)
    return;
  }

  // value pair q of a lane: line positions w0 + 64 q + 2 lane and the next one
  f32x2 acc[NZ][VP];
  constexpr bool kTables = MODE == kWbpTables;
  float c[kTables ? NZ : 1][kTables ? VL : 1];  // weight sums with a row table per angle
  float csum = 0.f;  // with a shared one: the sum over the angles of the x weights of plane `lane`
#pragma unroll
  for (int z = 0; z < NZ; ++z) {
#pragma unroll
    for (int q = 0; q < VP; ++q) acc[z][q] = 0ull;
    if (kTables) {
#pragma unroll
      for (int q = 0; q < VL; ++q) c[kTables ? z : 0][kTables ? q : 0] = 0.f;
    }
  }
  float cy[VL];  // WBP: detector weights along y of the lane's line positions
  auto load_weights = [&](int a) {
    const float* wt = P.tab.weight + (long long)a * P.tab.stride * P.Wp;
#pragma unroll
    for (int q = 0; q < VL; ++q) {
      const int w = w0 + 64 * (q >> 1) + 2 * lane + (q & 1);
      cy[q] = w < W ? __ldg(wt + w) : 0.f;
    }
  };
#pragma unroll 1
  for (int a = 0; a < A; ++a) {
    const int st = a % kBpStages;
    if (!__all_sync(0xffffffffu, mbar_wait_bounded(&full[st], (uint32_t)((a / kBpStages) & 1), P.wait_iters))) {
      if (lane == 0) atomicExch(P.err, 4);
      break;
    }
    const LineConst k = kc[a];
    const Walk s = lay_out_walk<NZ>(k, warp, lane, table);
    const uint32_t tab = smem_u32(table);
    const uint32_t dstep = s.dir > 0 ? 4u * BW : 0u - 4u * BW;
    uint32_t at = smem_u32(win0 + (size_t)st * stage_bytes) + 4u * (uint32_t)(s.pix * BW) + 8u * lane;
    f32x2 p0[VP], p1[VP], d[VP];
#pragma unroll
    for (int q = 0; q < VP; ++q) {
      p0[q] = lds_pair(at + 256u * q);
      p1[q] = lds_pair(at + dstep + 256u * q);
      if (MODE != kSirt) d[q] = sub2(p1[q], p0[q]);
    }
    if (MODE != kSirt) {
      // weight of the lane's plane: its two taps where they lie on the detector (both: exactly one)
      const int p = s.lane_pix + k.ox;
      const bool in0 = (unsigned)p < (unsigned)L.ax.PX, in1 = (unsigned)(p + s.dir) < (unsigned)L.ax.PX;
      const float cx = in0 ? (in1 ? 1.f : 1.f - s.lane_f) : in1 ? s.lane_f : 0.f;
      if (MODE == kWbp) csum += cx;
      if (kTables) {
        load_weights(a);
#pragma unroll
        for (int z = 0; z < NZ; ++z) {
          const float t = __shfl_sync(0xffffffffu, cx, z);
#pragma unroll
          for (int q = 0; q < VL; ++q) c[kTables ? z : 0][kTables ? q : 0] = fmaf(t, cy[q], c[kTables ? z : 0][kTables ? q : 0]);
        }
      }
    }
#pragma unroll
    for (int z = 0; z < NZ; ++z) {
      if (z > 0 && (s.cross & (1u << z))) {  // the column left the pixel
        at += dstep;
#pragma unroll
        for (int q = 0; q < VP; ++q) {
          p0[q] = p1[q];
          p1[q] = lds_pair(at + dstep + 256u * q);
          if (MODE != kSirt) d[q] = sub2(p1[q], p0[q]);
        }
      }
      if (MODE == kSirt) {
        const Weights w = lds_weights(tab + 16u * z);
#pragma unroll
        for (int q = 0; q < VP; ++q) acc[z][q] = fma2(w.b, p1[q], fma2(w.a, p0[q], acc[z][q]));
      } else {  // (interpolated first: the sums of the projections round once per angle)
        const f32x2 f = lds_pair(tab + 16u * z + 8u);
#pragma unroll
        for (int q = 0; q < VP; ++q) acc[z][q] = add2(acc[z][q], fma2(f, d[q], p0[q]));
      }
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(&empty[st]);
  }

  __syncthreads();  // every warp is done with the windows, and the producer with its loads
  const int sx = L.vol.NX, sxy = L.vol.NX * L.vol.NY;  // (16 planes stay below 2^31 voxels: plan_lines)
  const long long first = (long long)(Z0 - L.z0) * sxy + (L.along_x ? (long long)m0 * sx + w0 : (long long)w0 * sx + m0);
  const BrickOut B{P.vol_out + first, P.cbp + first,
                   static_cast<char*>(P.vol_copy) + (P.copy_kind ? 2 * first : 0), P.copy_kind, P.step};
  constexpr int ZB = VL == 4 ? 1 : 2;  // planes per batch: 4 voxels a lane
  const int nz = min(NZ, L.z1 - Z0);
  if (MODE == kWbp) load_weights(0);
  auto weight = [&](int z, int q) {  // WBP: weight sum of value q in plane z (every lane calls it)
    if (kTables) return c[kTables ? z : 0][kTables ? q : 0];
    return MODE == kWbp ? __shfl_sync(0xffffffffu, csum, z) * cy[q] : 0.f;
  };
  if (L.along_x) {
    if (m0 + warp >= M) return;
#pragma unroll
    for (int zb = 0; zb < NZ; zb += ZB) {
      int at[ZB * VL];
      float sv[ZB * VL], cv[ZB * VL];
#pragma unroll
      for (int e = 0; e < ZB * VL; ++e) {
        const int z = zb + e / VL, q = e % VL, w = 64 * (q >> 1) + 2 * lane + (q & 1);
        const float2 t = unpack2(acc[z][q >> 1]);
        at[e] = z < nz && w0 + w < W ? z * sxy + warp * sx + w : -1;
        sv[e] = q & 1 ? t.y : t.x;
        cv[e] = weight(z, q);
      }
      finish_voxels<MODE>(B, at, sv, cv);
    }
  } else {
    // lines along Y: the eight columns are neighbours in memory; each plane
    // goes through shared memory so that it is updated in 32-byte runs
    float* tile = reinterpret_cast<float*>(win0);  // [BW][9], sums (then weights) of ZB planes
    constexpr int kTile = BW * 9;
    const int tm = tid & 7, tw = tid >> 3;
#pragma unroll
    for (int zb = 0; zb < NZ; zb += ZB) {
      if (zb >= nz) break;
      int at[ZB * VL];
      float sv[ZB * VL], cv[ZB * VL];
#pragma unroll
      for (int pass = 0; pass < (MODE == kSirt ? 1 : 2); ++pass) {
#pragma unroll
        for (int e = 0; e < ZB * VL; ++e) {
          const int z = zb + e / VL, q = e % VL;
          const float2 t = unpack2(acc[z][q >> 1]);
          tile[(z - zb) * kTile + (64 * (q >> 1) + 2 * lane + (q & 1)) * 9 + warp] =
              pass ? weight(z, q) : q & 1 ? t.y : t.x;
        }
        named_sync(1, kThreads);
#pragma unroll
        for (int e = 0; e < ZB * VL; ++e) {
          const int z = zb + e / VL, w = 32 * (e % VL) + tw;
          const float t = tile[(e / VL) * kTile + w * 9 + tm];
          if (pass) {
            cv[e] = t;
          } else {
            sv[e] = t;
            at[e] = z < nz && w0 + w < W && m0 + tm < M ? z * sxy + w * sx + tm : -1;
            if (MODE == kSirt) cv[e] = 0.f;
          }
        }
        named_sync(1, kThreads);
      }
      finish_voxels<MODE>(B, at, sv, cv);
    }
  }
}

// ---- between line images and the detector ---------------------------------------
// One CTA per angle and kCols detector columns: the columns' line sums and
// residuals pass through shared memory, so that the line images are accessed
// along w and the detector arrays in 32-byte runs along x.  20 bytes per pixel
// as the plain residual, but bound by the latency of its three dependent
// phases: 0.10 ms against 0.05 ms for 512x512 px and 61 angles.
constexpr int kCols = 8;
constexpr int kBatch = 4;  // loads in flight per thread and array

template <int MODE, typename BT, bool NORM>
__global__ void __launch_bounds__(256, 5)
line_rows_kernel(AxisDev ax, int W, int Wp, LineTab tab, const BT* __restrict__ b, float* __restrict__ sums,
                 float* __restrict__ cf, float* __restrict__ image, double* __restrict__ norm2) {
  extern __shared__ __align__(16) float sh[];
  const int ws = (W + 31) / 32 * 32 + 4, ys = (ax.PY + 31) / 32 * 32 + 4;
  int2* trow = reinterpret_cast<int2*>(sh);  // [W] the angle's row table (the streams evict it from L1)
  float* lt = sh + 2 * ws;                   // [kCols][ws] line sums
  float* lr = lt + kCols * ws;               // [kCols][ys] detector rows
  const int a = blockIdx.y, x0 = blockIdx.x * kCols;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long plane = (long long)ax.pitch * ax.PY;
  const int2* row = tab.row + (long long)a * tab.stride * Wp;
  const int2* span = tab.span + (long long)a * tab.stride * ax.PY;
  double acc = 0.0;
  for (int w = threadIdx.x; w < W; w += 256) trow[w] = __ldg(row + w);
  const long long after = stream_wait();
  b += after;
  sums += after;
  cf += after;
  if (MODE != 2) {
    if (x0 + warp < ax.PX) {
      float* src = sums + ((long long)a * ax.PX + x0 + warp) * Wp;
      for (int w = lane; w < W; w += 32 * kBatch) {
        float t[kBatch];
#pragma unroll
        for (int q = 0; q < kBatch; ++q) t[q] = w + 32 * q < W ? src[w + 32 * q] : 0.f;
#pragma unroll
        for (int q = 0; q < kBatch; ++q) {
          if (w + 32 * q < W) {
            lt[warp * ws + w + 32 * q] = t[q];
          }
        }
      }
    }
    __syncthreads();
  }
  const int tx = threadIdx.x & 7;
  if (x0 + tx < ax.PX) {
    for (int y0 = threadIdx.x >> 3; y0 < ax.PY; y0 += 32 * kBatch) {
      float bv[kBatch], cv[kBatch];
      int2 sp[kBatch];
#pragma unroll
      for (int q = 0; q < kBatch; ++q) {
        const int y = min(y0 + 32 * q, ax.PY - 1);
        const long long i = a * plane + (long long)y * ax.pitch + x0 + tx;
        if (MODE != 1) bv[q] = ldb<BT>(b + i);
        if (MODE == 0) cv[q] = __ldg(cf + i);
        if (MODE != 2) sp[q] = __ldg(span + y);  // line positions whose rows touch y
      }
#pragma unroll
      for (int q = 0; q < kBatch; ++q) {
        const int y = y0 + 32 * q;
        if (y >= ax.PY) break;
        float s = 0.f;
        if (MODE != 2) {
          for (int w = sp[q].x; w < sp[q].x + sp[q].y; ++w) {
            const int2 e = trow[w];
            const float fy = __int_as_float(e.y);
            s = fmaf(e.x == y ? 1.f - fy : fy, lt[tx * ws + w], s);
          }
        }
        if (MODE == 1) {
          cf[a * plane + (long long)y * ax.pitch + x0 + tx] = s;
        } else {
          float r = bv[q];
          if (MODE == 0) {
            r -= cv[q] != 0.f ? s / cv[q] : s;
            if (NORM) acc += (double)(r * r);
          }
          lr[tx * ys + y] = r;
        }
      }
    }
  }
  if (MODE != 1) {
    __syncthreads();
    if (x0 + warp < ax.PX) {
      float* dst = image + ((long long)a * ax.PX + x0 + warp) * Wp;
      const float* r = lr + warp * ys;
#pragma unroll 4
      for (int w = lane; w < W; w += 32) {
        const int2 e = trow[w];
        const float fy = __int_as_float(e.y);
        const float r0 = (unsigned)e.x < (unsigned)ax.PY ? r[e.x] : 0.f;
        const float r1 = (unsigned)(e.x + 1) < (unsigned)ax.PY ? r[e.x + 1] : 0.f;
        dst[w] = fmaf(fy, r1 - r0, r0);
      }
    }
  }
  if (MODE != 2) {
    // zeroed at the end and 16 bytes a store: between the loads the stores cost
    // three times the rest of the kernel (315 against 100 us, 512x512 px, 61 angles)
    float4* z = reinterpret_cast<float4*>(sums + ((long long)a * ax.PX + x0) * Wp);
    const int n4 = min(kCols, ax.PX - x0) * Wp / 4;
    for (int i = threadIdx.x; i < n4; i += 256) z[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  if (NORM) {
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane == 0) atomicAdd(norm2, acc);
  }
}

size_t rows_smem(int W, int PY) {
  return ((size_t)(kCols + 2) * ((W + 31) / 32 * 32 + 4) + (size_t)kCols * ((PY + 31) / 32 * 32 + 4)) * sizeof(float);
}
size_t fwd_smem(const LinePlan& p, int angles) {
  return (((size_t)angles * sizeof(LineConst) + 127) & ~(size_t)127) + 128 +
         kWarps * p.fwd_nz * sizeof(float4) + kFwdStages * kMaxRows * sizeof(int) +
         std::max((size_t)kFwdStages * p.fwd_rows * 32 * p.fwd_vl * 4, (size_t)2 * 32 * p.fwd_vl * 9 * 4);
}
size_t bp_smem(int rows, int vl, int nz, int A) {
  return 128 + (((size_t)A * sizeof(LineConst) + 127) & ~(size_t)127) + bp_table_bytes(nz) +
         std::max((size_t)kBpStages * rows * 32 * vl * 4, (size_t)(vl == 4 ? 1 : 2) * 32 * vl * 9 * 4);
}

template <typename VT, int VL, int NZ>
cudaError_t run_forward(const CUtensorMap& map, const LinePlan& p, LineArgs L, const VT* x, cudaStream_t st) {
  auto kern = line_forward_kernel<VT, VL, NZ>;
  const int W = L.along_x ? L.vol.NX : L.vol.NY, M = L.along_x ? L.vol.NY : L.vol.NX;
  const int gx = (W + 32 * VL - 1) / (32 * VL), gy = (M + kWarps - 1) / kWarps, gz = (L.z1 - L.z0 + NZ - 1) / NZ;
  // split the angles over several CTAs when there are too few bricks to fill
  // the GPU; each group reads the brick again, worth a few angles' work
  const long long bricks = (long long)gx * gy * gz, target = 6LL * device_sm_count();
  const int groups = (int)std::max(1LL, std::min<long long>((target + bricks - 1) / bricks, (L.ax.A + 3) / 4));
  L.groups = groups;
  L.max_angles = (L.ax.A + groups - 1) / groups;
  const size_t smem = fwd_smem(p, L.max_angles);
  cudaError_t e = allow_shared_memory(kern, smem);
  if (e != cudaSuccess) return e;
  launch_overlapped(kern, dim3(gx, gy, gz * groups), kThreads, smem, st, map, L, x);
  e = cudaGetLastError();
  if (e == cudaSuccess) g_windowed_launches.fetch_add(1, std::memory_order_relaxed);
  return e;
}

template <int MODE, int VL, int NZ>
cudaError_t run_bp(const CUtensorMap& map, LineBpArgs P, cudaStream_t st) {
  auto kern = line_bp_kernel<MODE, VL, NZ>;
  const LineArgs& L = P.l;
  const int W = L.along_x ? L.vol.NX : L.vol.NY, M = L.along_x ? L.vol.NY : L.vol.NX;
  const size_t smem = bp_smem(L.rows, VL, NZ, L.ax.A);
  cudaError_t e = allow_shared_memory(kern, smem);
  if (e != cudaSuccess) return e;
  const dim3 grid((W + 32 * VL - 1) / (32 * VL), (L.z1 - L.z0 + NZ - 1) / NZ, (M + kWarps - 1) / kWarps);
  launch_overlapped(kern, grid, kBpThreads, smem, st, map, P);
  e = cudaGetLastError();
  if (e == cudaSuccess) g_windowed_launches.fetch_add(1, std::memory_order_relaxed);
  return e;
}

template <int MODE>
cudaError_t run_bp_shape(int vl, int nz, const CUtensorMap& map, const LineBpArgs& P, cudaStream_t st) {
  if (vl == 4) return run_bp<MODE, 4, 8>(map, P, st);
  return nz == 16 ? run_bp<MODE, 2, 16>(map, P, st) : nz == 8 ? run_bp<MODE, 2, 8>(map, P, st) : run_bp<MODE, 2, 4>(map, P, st);
}

template <int MODE, typename BT, bool NORM>
cudaError_t run_rows(const LinePlan& p, const LineTab& tab, const AxisDev& ax, const BT* b, float* sums, float* cf,
                     float* image, double* norm2, cudaStream_t st) {
  auto kern = line_rows_kernel<MODE, BT, NORM>;
  const size_t smem = rows_smem(p.W, ax.PY);
  cudaError_t e = allow_shared_memory(kern, smem);
  if (e != cudaSuccess) return e;
  launch_overlapped(kern, dim3((ax.PX + kCols - 1) / kCols, ax.A), 256, smem, st, ax, p.W, p.Wp, tab, b, sums, cf, image,
                    norm2);
  return cudaGetLastError();
}

}  // namespace

template <typename VT>
cudaError_t launch_line_forward(const CUtensorMap& map, const LinePlan& p, const AxisDev& ax, const VolDev& vol,
                                const VT* x, int z0, int z1, cudaStream_t st) {
  const LineArgs L{ax, vol, p.along_x, z0, z1, p.fwd_rows, 1, ax.A};
  if (p.fwd_vl == 4) return p.fwd_nz == 16 ? run_forward<VT, 4, 16>(map, p, L, x, st) : run_forward<VT, 4, 8>(map, p, L, x, st);
  return p.fwd_nz == 16 ? run_forward<VT, 2, 16>(map, p, L, x, st) : run_forward<VT, 2, 8>(map, p, L, x, st);
}

cudaError_t launch_line_backproject(const CUtensorMap& map, const LinePlan& p, const LineTab& tab, const AxisDev& ax,
                                    const VolDev& vol, int mode, float step, float* vol_out, float* cbp,
                                    void* vol_copy, int copy_kind, int z0, int z1, int* err, cudaStream_t st) {
  const LineArgs L{ax, vol, p.along_x, z0, z1, mode == 0 ? p.wbp_rows : p.bp_rows, 1, ax.A};
  const LineBpArgs P{L, tab, p.Wp, step, vol_out, cbp, vol_copy, copy_kind, err, pipeline_wait_limit()};
  if (mode == 0) {
    if (p.n_tab == 1) return run_bp_shape<kWbp>(p.wbp_vl, p.wbp_nz, map, P, st);
    if (p.wbp_vl == 4) return run_bp<kWbpTables, 4, 8>(map, P, st);
    return p.wbp_nz == 8 ? run_bp<kWbpTables, 2, 8>(map, P, st) : run_bp<kWbpTables, 2, 4>(map, P, st);
  }
  return run_bp_shape<kSirt>(p.bp_vl, p.bp_nz, map, P, st);
}

template <typename BT>
cudaError_t launch_line_rows(int mode, const LinePlan& p, const LineTab& tab, const AxisDev& ax, const BT* b,
                             float* sums, float* cf, float* image, double* norm2, cudaStream_t st) {
  if (mode == 1) return run_rows<1, BT, false>(p, tab, ax, b, sums, cf, image, nullptr, st);
  if (mode == 2) return run_rows<2, BT, false>(p, tab, ax, b, sums, cf, image, nullptr, st);
  if (norm2) return run_rows<0, BT, true>(p, tab, ax, b, sums, cf, image, norm2, st);
  return run_rows<0, BT, false>(p, tab, ax, b, sums, cf, image, nullptr, st);
}

template cudaError_t launch_line_forward<float>(const CUtensorMap&, const LinePlan&, const AxisDev&, const VolDev&,
                                                const float*, int, int, cudaStream_t);
template cudaError_t launch_line_forward<__nv_bfloat16>(const CUtensorMap&, const LinePlan&, const AxisDev&,
                                                        const VolDev&, const __nv_bfloat16*, int, int, cudaStream_t);
template cudaError_t launch_line_forward<__half>(const CUtensorMap&, const LinePlan&, const AxisDev&, const VolDev&,
                                                 const __half*, int, int, cudaStream_t);
template cudaError_t launch_line_rows<float>(int, const LinePlan&, const LineTab&, const AxisDev&, const float*,
                                             float*, float*, float*, double*, cudaStream_t);
template cudaError_t launch_line_rows<__half>(int, const LinePlan&, const LineTab&, const AxisDev&, const __half*,
                                              float*, float*, float*, double*, cudaStream_t);

LinePlan plan_lines(const std::vector<double>& xc, const std::vector<double>& yc, int A, int PX, int PY, int pitch,
                    const VolDev& vol, int depth, int sms) {
  LinePlan p;
  for (int along_x = 1; along_x >= 0 && !p.ok; --along_x) {
    const int cw = along_x ? 1 : 2, cm = along_x ? 2 : 1;
    const int W = along_x ? vol.NX : vol.NY, M = along_x ? vol.NY : vol.NX;
    bool sep = true;
    for (int a = 0; a < A && sep; ++a) {
      const double* cx = &xc[4 * (size_t)a];
      const double* cy = &yc[4 * (size_t)a];
      // (negated comparisons: NaN and infinite maps do not separate)
      sep = std::fabs(cx[cw]) <= 1e-8 && std::fabs(cy[cm]) * M + std::fabs(cy[3]) * vol.NZ <= 1e-6 &&
            std::fabs(cy[cw]) >= 0.5 && std::fabs(cy[cw]) <= 2.0 && std::fabs(cx[cm]) <= 4.0 &&
            std::fabs(cx[3]) < 0.999 && std::fabs(cx[0]) < 1e9 && std::fabs(cy[0]) < 1e9;
    }
    // (positions stay within the integers and floats that the kernels index with)
    const double m0 = along_x ? vol.Ys : vol.Xs, w0 = along_x ? vol.Xs : vol.Ys;
    for (int a = 0; a < A && sep; ++a)
      for (int c = 0; c < 8 && sep; ++c) {
        const double* cx = &xc[4 * (size_t)a];
        const double x = cx[0] + cx[cw] * (w0 + (c & 1 ? W : 0)) + cx[cm] * (m0 + (c & 2 ? M : 0)) +
                         cx[3] * ((double)vol.Zs + (c & 4 ? vol.NZ : 0));
        sep = std::fabs(x) < 9e8;
      }
    if (!sep) continue;
    p.along_x = along_x;
    p.W = W;
    p.Wp = (W + 3) / 4 * 4;
    // Values per lane and depth: the least padded work at the measured cost per
    // voxel (1024x1024x96, 121 angles, forward 3.5 / 3.8 / 4.0 / 5.0 ms and SIRT
    // update 2.9 / 2.5 / 3.1 / 3.6 ms for 4x16, 4x8, 2x16, 2x8) among the shapes
    // with a CTA or more for every SM; small volumes take the smallest bricks
    // (128x128x32: SIRT update 66 / 35 / 43 / 29 and 27 us for 2x4).
    auto ctas = [&](int vl, int nz) {
      return (long long)((W + 32 * vl - 1) / (32 * vl)) * ((M + kWarps - 1) / kWarps) * ((depth + nz - 1) / nz);
    };
    auto work = [&](int vl, int nz) {
      return (double)((W + 32 * vl - 1) / (32 * vl) * 32 * vl) * ((depth + nz - 1) / nz * nz);
    };
    static const struct { int vl, nz; double fwd, bp, wbp; } kShapes[] = {
        {4, 16, 1.00, 0., 0.}, {4, 8, 1.08, 1.00, 1.00}, {2, 16, 1.12, 1.23, 0.}, {2, 8, 1.41, 1.40, 1.10}};
    double bf = 1e300, bb = 1e300, bw = 1e300;
    p.fwd_vl = p.bp_vl = p.wbp_vl = 2;
    p.fwd_nz = 8;  // (the forward splits the angles of few bricks over more CTAs)
    p.bp_nz = p.wbp_nz = 4;
    for (const auto& sh : kShapes) {
      const double wk = work(sh.vl, sh.nz);
      if (wk * sh.fwd < bf) { bf = wk * sh.fwd; p.fwd_vl = sh.vl; p.fwd_nz = sh.nz; }
      if (ctas(sh.vl, sh.nz) < 2 * sms) continue;
      if (sh.bp > 0 && wk * sh.bp < bb) { bb = wk * sh.bp; p.bp_vl = sh.vl; p.bp_nz = sh.nz; }
      if (sh.wbp > 0 && wk * sh.wbp < bw) { bw = wk * sh.wbp; p.wbp_vl = sh.vl; p.wbp_nz = sh.nz; }
    }
    p.n_tab = 1;
    for (int a = 1; a < A; ++a)
      for (int c = 0; c < 4; ++c)
        if (yc[4 * (size_t)a + c] != yc[c]) p.n_tab = A;
    if (p.n_tab == 1) {  // (a WBP without weight sums to carry: as the SIRT update)
      p.wbp_vl = p.bp_vl;
      p.wbp_nz = p.bp_nz;
    }
    auto rows = [&](int nz) {  // detector columns of a brick, at the widest angle
      double e = 0;
      for (int a = 0; a < A; ++a)
        e = std::max(e, std::fabs(xc[4 * (size_t)a + cm]) * (kWarps - 1) + std::fabs(xc[4 * (size_t)a + 3]) * (nz - 1));
      return (int)std::ceil(e) + 4;
    };
    p.fwd_rows = rows(p.fwd_nz);
    p.bp_rows = rows(p.bp_nz);
    p.wbp_rows = rows(p.wbp_nz);
    // the line images live in the axis' ray-sum and residual arrays
    p.ok = (long long)PX * p.Wp <= (long long)PY * pitch && p.fwd_rows <= PX && p.fwd_rows <= kMaxRows &&
           (long long)vol.NX * vol.NY < (1LL << 27) &&
           fwd_smem(p, A) <= 100 * 1024 && bp_smem(p.bp_rows, p.bp_vl, p.bp_nz, A) <= 110 * 1024 &&
           bp_smem(p.wbp_rows, p.wbp_vl, p.wbp_nz, A) <= 110 * 1024 && rows_smem(W, PY) <= 200 * 1024;
    if (!p.ok) continue;
    const int ws = along_x ? vol.Xs : vol.Ys, ms = along_x ? vol.Ys : vol.Xs;
    const size_t nw = (size_t)p.n_tab * p.Wp, ny = (size_t)p.n_tab * PY;
    p.off_rows = 2 * nw;
    p.off_weight = p.off_rows + 2 * ny;
    p.tables.assign(p.off_weight + nw, 0);
    for (int t = 0; t < p.n_tab; ++t) {
      const double* cy = &yc[4 * (size_t)t];
      int* rw = &p.tables[2 * (size_t)t * p.Wp];
      int* sp = &p.tables[p.off_rows + 2 * (size_t)t * PY];
      for (int w = 0; w < p.Wp; ++w) {
        const double y = cy[0] + cy[cw] * (ws + w) + cy[cm] * (ms + 0.5 * (M - 1)) + cy[3] * (vol.Zs + 0.5 * (vol.NZ - 1)) - 1.0;
        double iy = std::floor(y);
        float fy = (float)(y - iy);
        if (fy >= 1.f) {
          iy += 1.0;
          fy = 0.f;
        }
        const int r = (int)std::min(std::max(iy, -2.0), (double)PY + 1.0);
        const bool in0 = r >= 0 && r < PY, in1 = r + 1 >= 0 && r + 1 < PY;
        const float c = in0 && in1 ? 1.f : in0 ? 1.f - fy : in1 ? fy : 0.f;
        rw[2 * w] = r;
        std::copy_n(reinterpret_cast<const int*>(&fy), 1, &rw[2 * w + 1]);
        std::copy_n(reinterpret_cast<const int*>(&c), 1, &p.tables[p.off_weight + (size_t)t * p.Wp + w]);
        if (w >= W) continue;
        for (int q = 0; q < 2; ++q) {  // rows are monotonic in w: the positions of a row are consecutive
          const int y1 = r + q;
          if (y1 < 0 || y1 >= PY) continue;
          if (sp[2 * y1 + 1] == 0) sp[2 * y1] = w;
          sp[2 * y1 + 1] = w - sp[2 * y1] + 1;
        }
      }
    }
  }
  return p;
}

}  // namespace mtr
