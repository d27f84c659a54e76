// Elementwise and MACE consensus kernels (sm_103a).  These are HBM-bound:
// grid-stride loops over the volume, sized to a multiple of the SM count.
#include <algorithm>
#include <atomic>
#include <map>
#include <mutex>
#include <utility>

#include "mtr_internal.h"

namespace mtr {
namespace {

constexpr int kThreads = 256;

unsigned grid_for(long long n) {
  long long b = (n + kThreads - 1) / kThreads;
  const long long cap = (long long)device_sm_count() * 8;  // 8 resident CTAs per SM
  if (b > cap) b = cap;
  if (b < 1) b = 1;
  return (unsigned)b;
}

__global__ void fill_kernel(float* __restrict__ p, long long n, float v) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    p[i] = v;
}

__global__ void add_kernel(float* __restrict__ dst, const float* __restrict__ src, long long n) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    dst[i] = __fadd_rn(dst[i], src[i]);
}

// z = 2*w_avg - w (FunctionOnGPU.cu:268-276).
__global__ void initial_z_kernel(const float* __restrict__ w, const float* __restrict__ wavg, float* __restrict__ z,
                                 long long n) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    z[i] = __fsub_rn(2.f * wavg[i], w[i]);
}

// Mixed precision stores each MACE state as its FP16 deviation from the FP32
// consensus, d_k = w_k - w_avg: the axes' states differ from their consensus
// by much less than they differ from zero, so FP16 rounds d_k far more finely
// than it would round w_k.  The state's value is w_avg + d_k (one FP32 add).
__device__ __forceinline__ float state_of(float wavg, __half d) { return __fadd_rn(wavg, __half2float(d)); }

// z = 2*w_avg - w from a deviation state, w = w_avg + d.
__global__ void initial_z_half_kernel(const __half* __restrict__ d, const float* __restrict__ wavg,
                                      float* __restrict__ z, long long n) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const float wa = wavg[i];
    z[i] = __fsub_rn(2.f * wa, state_of(wa, d[i]));
  }
}

// d = fp16(w - w_avg) and w = w_avg + d (state to and from its stored form).
__global__ void state_dev_kernel(const float* __restrict__ w, const float* __restrict__ wavg, __half* __restrict__ d,
                                 long long n) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    d[i] = __float2half_rn(__fsub_rn(w[i], wavg[i]));
}
__global__ void state_value_kernel(const __half* __restrict__ d, const float* __restrict__ wavg, float* __restrict__ w,
                                   long long n) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    w[i] = state_of(wavg[i], d[i]);
}

// w = step*(2v - z) + (1-step)*w, with the reference host loop's float
// rounding (MultiAxis.cpp:33-38; no fused multiply-add).
__device__ __forceinline__ float mann(float v, float z, float w, float step) {
  const float t1 = __fsub_rn(2.f * v, z);
  const float t2 = __fmul_rn(step, t1);
  const float t3 = __fmul_rn(__fsub_rn(1.f, step), w);
  return __fadd_rn(t2, t3);
}

__global__ void update_w_kernel(const float* __restrict__ v, const float* __restrict__ z, float* __restrict__ w,
                                long long n, float step) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    w[i] = mann(v[i], z[i], w[i], step);
}

__global__ void convert_kernel(const float* __restrict__ src, void* __restrict__ dst, int kind, long long n) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    if (kind == 1) static_cast<__nv_bfloat16*>(dst)[i] = __float2bfloat16_rn(src[i]);
    else static_cast<__half*>(dst)[i] = __float2half_rn(src[i]);
  }
}

__global__ void widen_kernel(const __half* __restrict__ src, float* __restrict__ dst, long long n) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    dst[i] = __half2float(src[i]);
}

// One MACE outer step for all K axes at once, replacing the reference's
// initialZdata + runMaceOnCPU + Reduce/Bcast consensus (FunctionOnGPU.cu:268-313,
// MultiAxis.cpp:48-67).  On entry x[k] holds v_k = SIRT(z_k), w[k] the state
// w_k and wavg the consensus that z_k was formed from (z_k = 2 wavg - w_k,
// recomputed here instead of stored).  On exit:
//   w[k] = rho*(2 v_k - z_k) + (1-rho) w_k
//   wavg = (sum_k w[k]) / K      (summed in FP64)
//   x[k] = 2 wavg - w[k]         (the next outer iteration's z_k)
// and, when copy_kind != 0, x_copy[k] = x[k] in bf16/f16 for the forward pass.
// With WH (mixed precision) w[k] holds the FP16 deviation d_k = w_k - w_avg
// (state_of): the new states are computed in FP32, the consensus averages
// them unrounded (so the output carries no rounding of the step that made
// it), then each is stored as fp16(w_k - w_avg_new) and the next z_k is formed
// from the stored value, exactly as the next step recomputes it.  REC: dchange
// (2 doubles) accumulates sum (wavg_new - wavg_old)^2 and sum wavg_new^2 in
// FP64, the convergence test's relative change (without it those FP64
// operations are not run).
constexpr int kMaxK = MTR_MAX_AXES;
struct MacePtrs {
  void* w[kMaxK];
  float* x[kMaxK];
  void* xc[kMaxK];
};

// The state w_k at voxel i (consensus wa at that voxel).
template <bool WH>
__device__ __forceinline__ float ld_state(const void* w, long long i, float wa) {
  if constexpr (WH) return state_of(wa, static_cast<const __half*>(w)[i]);
  else return static_cast<const float*>(w)[i];
}
// Stores the new state v against the new consensus na and returns the state
// as it will be read back.
template <bool WH>
__device__ __forceinline__ float st_state(void* w, long long i, float v, float na) {
  if constexpr (WH) {
    const __half h = __float2half_rn(__fsub_rn(v, na));
    static_cast<__half*>(w)[i] = h;
    return state_of(na, h);
  } else {
    static_cast<float*>(w)[i] = v;
    return v;
  }
}

// Mean of K states, rounded once to FP32 as an FP64 sum times 1/K is.  The
// FP64 pipe of this part runs at 1/64 of the FP32 rate and bound the whole
// step, so the sum is carried as an unevaluated pair of floats (error-free
// two-term sums: Knuth's TwoSum) and multiplied by 1/K held as a pair, with
// the product's rounding error recovered by a fused multiply-add: 48 bits
// before the final rounding.  Sums near the ends of the FP32 range, where the
// pair would overflow or its low part underflow, infinities and NaN, and sums
// that cancel take the FP64 form.  The two forms may still round apart near a
// midpoint of two floats; of 36 million drawn means of 2-4 states none did, and
// both stay within half an ulp.
__device__ __noinline__ float mean_states_fp64(int K, const float* w) {
  double sum = 0.0;
  for (int k = 0; k < K; ++k) sum += (double)w[k];
  return (float)(sum * (1.0 / (double)K));
}
template <int KC>
__device__ __forceinline__ float mean_states(int K, const float (&w)[KC], float ck, float ckl) {
  if (KC == 1) return w[0];
  float s = w[0], e = 0.f;
#pragma unroll
  for (int k = 1; k < KC; ++k) {
    if (k < K) {
      const float t = __fadd_rn(s, w[k]);
      const float bb = __fsub_rn(t, s);
      e = __fadd_rn(e, __fadd_rn(__fsub_rn(s, __fsub_rn(t, bb)), __fsub_rn(w[k], bb)));
      s = t;
    }
  }
  const float hi = __fadd_rn(s, e), lo = __fsub_rn(e, __fsub_rn(hi, s));
  const float p = __fmul_rn(hi, ck);
  const float pe = __fmaf_rn(hi, ck, -p);
  float corr = __fadd_rn(pe, __fmaf_rn(hi, ckl, __fmul_rn(lo, ck)));
  if (KC > 2) {
    // K times a midpoint of two floats is a common sum, and the pair's last
    // bits would break the tie: the correction is snapped to 2^-40 of the
    // product, so that such a mean rounds to even as the FP64 one does.
    const float grid = __fmul_rn(p, 0x1p-17f);
    corr = __fsub_rn(__fadd_rn(corr, grid), grid);
  }
  const float r = __fadd_rn(p, corr);
  const float m = fabsf(hi);
  // (the low parts of three or more states are summed in FP32: exact enough
  // unless the states cancel, so a sum far below the largest state is redone)
  float top = 0.f;
  if (KC > 2) {
#pragma unroll
    for (int k = 0; k < KC; ++k) top = fmaxf(top, fabsf(w[k]));
  }
  if ((m >= 1e-28f && m <= 1e37f && m >= top * 0x1p-16f) || (hi == 0.f && lo == 0.f && top == 0.f)) return r;
  float v[KC];
#pragma unroll
  for (int k = 0; k < KC; ++k) v[k] = w[k];
  return mean_states_fp64(K, v);
}

// V voxels i .. i + V - 1 of K states (KC: K's compile-time bound).
template <int KC, int V, bool REC, bool WH>
__device__ __forceinline__ void mace_voxels(int K, void* const* w, float* const* x, void* const* xc,
                                            float* __restrict__ wavg, long long i, float rho, int copy_kind, float ck,
                                            float ckl, double& acc, double& acc2) {
  float wa[V], na[V], wn[V][KC];
  if constexpr (V == 4) {
    const float4 t = *reinterpret_cast<const float4*>(wavg + i);
    wa[0] = t.x; wa[1] = t.y; wa[2] = t.z; wa[3] = t.w;
  } else {
    wa[0] = wavg[i];
  }
#pragma unroll
  for (int k = 0; k < KC; ++k) {
    if (k < K) {
      float wk[V], xk[V];
      if constexpr (V == 4) {
        const float4 t = *reinterpret_cast<const float4*>(x[k] + i);
        xk[0] = t.x; xk[1] = t.y; xk[2] = t.z; xk[3] = t.w;
        if constexpr (WH) {
          const uint2 h = *reinterpret_cast<const uint2*>(static_cast<const __half*>(w[k]) + i);
          const __half* hp = reinterpret_cast<const __half*>(&h);
#pragma unroll
          for (int q = 0; q < 4; ++q) wk[q] = state_of(wa[q], hp[q]);
        } else {
          const float4 u = *reinterpret_cast<const float4*>(static_cast<const float*>(w[k]) + i);
          wk[0] = u.x; wk[1] = u.y; wk[2] = u.z; wk[3] = u.w;
        }
      } else {
        wk[0] = ld_state<WH>(w[k], i, wa[0]);
        xk[0] = x[k][i];
      }
#pragma unroll
      for (int q = 0; q < V; ++q) wn[q][k] = mann(xk[q], __fsub_rn(2.f * wa[q], wk[q]), wk[q], rho);
    } else {
#pragma unroll
      for (int q = 0; q < V; ++q) wn[q][k] = 0.f;
    }
  }
#pragma unroll
  for (int q = 0; q < V; ++q) {
    na[q] = mean_states<KC>(K, wn[q], ck, ckl);
    if (REC) {
      const double d = (double)na[q] - (double)wa[q];
      acc += d * d;
      acc2 += (double)na[q] * (double)na[q];
    }
  }
  if constexpr (V == 4) *reinterpret_cast<float4*>(wavg + i) = make_float4(na[0], na[1], na[2], na[3]);
  else wavg[i] = na[0];
#pragma unroll
  for (int k = 0; k < KC; ++k) {
    if (k < K) {
      float zn[V];
      if constexpr (V == 4) {
        if constexpr (WH) {
          uint2 h;
          __half* hp = reinterpret_cast<__half*>(&h);
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            hp[q] = __float2half_rn(__fsub_rn(wn[q][k], na[q]));
            zn[q] = __fsub_rn(2.f * na[q], state_of(na[q], hp[q]));
          }
          *reinterpret_cast<uint2*>(static_cast<__half*>(w[k]) + i) = h;
        } else {
          *reinterpret_cast<float4*>(static_cast<float*>(w[k]) + i) =
              make_float4(wn[0][k], wn[1][k], wn[2][k], wn[3][k]);
#pragma unroll
          for (int q = 0; q < 4; ++q) zn[q] = __fsub_rn(2.f * na[q], wn[q][k]);
        }
        *reinterpret_cast<float4*>(x[k] + i) = make_float4(zn[0], zn[1], zn[2], zn[3]);
        if (copy_kind == 1) {
          uint2 h;
          __nv_bfloat16* hp = reinterpret_cast<__nv_bfloat16*>(&h);
#pragma unroll
          for (int q = 0; q < 4; ++q) hp[q] = __float2bfloat16_rn(zn[q]);
          *reinterpret_cast<uint2*>(static_cast<__nv_bfloat16*>(xc[k]) + i) = h;
        } else if (copy_kind == 2) {
          uint2 h;
          __half* hp = reinterpret_cast<__half*>(&h);
#pragma unroll
          for (int q = 0; q < 4; ++q) hp[q] = __float2half_rn(zn[q]);
          *reinterpret_cast<uint2*>(static_cast<__half*>(xc[k]) + i) = h;
        }
      } else {
        zn[0] = __fsub_rn(2.f * na[0], st_state<WH>(w[k], i, wn[0][k], na[0]));
        x[k][i] = zn[0];
        if (copy_kind == 1) static_cast<__nv_bfloat16*>(xc[k])[i] = __float2bfloat16_rn(zn[0]);
        else if (copy_kind == 2) static_cast<__half*>(xc[k])[i] = __float2half_rn(zn[0]);
      }
    }
  }
}

// Bound by HBM (each state, iterate and the consensus read and written once).
// One axis of 320x300x72 voxels (166 MB): 0.02 ms against 0.44 ms when the
// mean ran on the FP64 pipe; three axes of 256x256x64: 0.04 ms against 0.27 ms.
// 4 voxels per thread and step, 16-byte accesses; n4 = 0 where an array is not
// 16-byte aligned (a slab of an odd plane size), then one voxel per step.
// KC = K for the usual 1-4 axes, else the maximum (one voxel per step).
template <int KC, bool REC, bool WH>
__global__ void __launch_bounds__(kThreads)
mace_kernel(int K, const __grid_constant__ MacePtrs P, float* __restrict__ wavg, long long n, long long n4, float rho,
            int copy_kind, float ck, float ckl, double* __restrict__ dchange) {
  double acc = 0.0, acc2 = 0.0;
  const long long t0 = blockIdx.x * (long long)blockDim.x + threadIdx.x, stride = (long long)gridDim.x * blockDim.x;
  if constexpr (KC <= 4)
    for (long long q = t0; q < n4; q += stride)
      mace_voxels<KC, 4, REC, WH>(K, P.w, P.x, P.xc, wavg, 4 * q, rho, copy_kind, ck, ckl, acc, acc2);
  for (long long i = 4 * n4 + t0; i < n; i += stride)
    mace_voxels<KC, 1, REC, WH>(K, P.w, P.x, P.xc, wavg, i, rho, copy_kind, ck, ckl, acc, acc2);
  if (REC) {
    for (int o = 16; o > 0; o >>= 1) {
      acc += __shfl_xor_sync(0xffffffffu, acc, o);
      acc2 += __shfl_xor_sync(0xffffffffu, acc2, o);
    }
    __shared__ double red[2][kThreads / 32];
    if ((threadIdx.x & 31) == 0) {
      red[0][threadIdx.x >> 5] = acc;
      red[1][threadIdx.x >> 5] = acc2;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      double t = 0.0, t2 = 0.0;
      for (int w = 0; w < kThreads / 32; ++w) {
        t += red[0][w];
        t2 += red[1][w];
      }
      atomicAdd(dchange, t);
      atomicAdd(dchange + 1, t2);
    }
  }
}

template <int KC>
void launch_mace_k(int K, const MacePtrs& P, int w_half, float* wavg, long long n, long long n4, float rho,
                   int copy_kind, double* dchange, cudaStream_t st) {
  const double inv_k = 1.0 / (double)K;
  const float ck = (float)inv_k, ckl = (float)(inv_k - (double)ck);
  const unsigned g = grid_for(n4 > 0 ? n4 : n);
  if (dchange) {
    if (w_half) mace_kernel<KC, true, true><<<g, kThreads, 0, st>>>(K, P, wavg, n, n4, rho, copy_kind, ck, ckl, dchange);
    else mace_kernel<KC, true, false><<<g, kThreads, 0, st>>>(K, P, wavg, n, n4, rho, copy_kind, ck, ckl, dchange);
  } else {
    if (w_half) mace_kernel<KC, false, true><<<g, kThreads, 0, st>>>(K, P, wavg, n, n4, rho, copy_kind, ck, ckl, dchange);
    else mace_kernel<KC, false, false><<<g, kThreads, 0, st>>>(K, P, wavg, n, n4, rho, copy_kind, ck, ckl, dchange);
  }
}

// The voxels [i0, i1) of one reconstruction (its arrays are whole allocations,
// so the chunk starts 16-byte aligned).
template <int KC>
__device__ __forceinline__ void mace_batch_item(const MaceBatchDesc& D, long long i0, long long i1) {
  double acc = 0.0, acc2 = 0.0;
  const double inv_k = 1.0 / (double)D.K;
  const float ck = (float)inv_k, ckl = (float)(inv_k - (double)ck);
  long long i4 = i0;
  if constexpr (KC <= 4) {
    i4 = i0 + (i1 - i0) / 4 * 4;
    for (long long i = i0 + 4 * threadIdx.x; i < i4; i += 4 * blockDim.x) {
      if (D.w_half) mace_voxels<KC, 4, false, true>(D.K, D.w, D.x, D.xc, D.wavg, i, D.rho, D.copy_kind, ck, ckl, acc, acc2);
      else mace_voxels<KC, 4, false, false>(D.K, D.w, D.x, D.xc, D.wavg, i, D.rho, D.copy_kind, ck, ckl, acc, acc2);
    }
  }
  for (long long i = i4 + threadIdx.x; i < i1; i += blockDim.x) {
    if (D.w_half) mace_voxels<KC, 1, false, true>(D.K, D.w, D.x, D.xc, D.wavg, i, D.rho, D.copy_kind, ck, ckl, acc, acc2);
    else mace_voxels<KC, 1, false, false>(D.K, D.w, D.x, D.xc, D.wavg, i, D.rho, D.copy_kind, ck, ckl, acc, acc2);
  }
}

// MACE step over many reconstructions: item = (descriptor, chunk of voxels);
// the arithmetic is mace_kernel's (reference float rounding, mean_states).
__global__ void __launch_bounds__(kThreads)
mace_batch_kernel(const MaceBatchDesc* __restrict__ descs, const long long* __restrict__ first, int n_desc,
                  long long n_items) {
  for (long long it = blockIdx.x; it < n_items; it += gridDim.x) {
    const int2 item = work_item(first, n_desc, it);
    const MaceBatchDesc& D = descs[item.x];
    const long long i0 = (long long)item.y * kBatchChunk;
    const long long i1 = min(D.n, i0 + kBatchChunk);
    if (D.K == 1) mace_batch_item<1>(D, i0, i1);
    else if (D.K == 2) mace_batch_item<2>(D, i0, i1);
    else if (D.K == 3) mace_batch_item<3>(D, i0, i1);
    else if (D.K == 4) mace_batch_item<4>(D, i0, i1);
    else mace_batch_item<kMaxK>(D, i0, i1);
  }
}

}  // namespace

cudaError_t raise_shared_memory_limit(const void* kern, size_t bytes) {
  static std::mutex mu;
  static std::map<std::pair<int, const void*>, size_t> limit;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  std::lock_guard<std::mutex> lock(mu);
  size_t& top = limit[{dev, kern}];
  const size_t want = std::max(top, bytes);
  e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)want);
  if (e == cudaSuccess) top = want;
  return e;
}

int device_sm_count() {
  constexpr int kMaxDevices = 64;
  static std::atomic<int> cached[kMaxDevices];  // 0 = not yet queried
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) {
    cudaGetLastError();
    dev = -1;
  }
  if (dev >= 0) {
    const int c = cached[dev].load(std::memory_order_relaxed);
    if (c > 0) return c;
  }
  int n = 0;
  if (dev < 0 || cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) {
    cudaGetLastError();
    return 1;  // a one-SM grid still covers everything through its grid-stride loop
  }
  cached[dev].store(n, std::memory_order_relaxed);
  return n;
}

void launch_mace_batch(const MaceBatchDesc* descs, const long long* first, int n_desc, long long n_items, int grid,
                       cudaStream_t st) {
  mace_batch_kernel<<<grid, kThreads, 0, st>>>(descs, first, n_desc, n_items);
}

void launch_fill(float* p, long long n, float v, cudaStream_t st) {
  fill_kernel<<<grid_for(n), kThreads, 0, st>>>(p, n, v);
}
void launch_axpy_acc(float* dst, const float* src, long long n, cudaStream_t st) {
  add_kernel<<<grid_for(n), kThreads, 0, st>>>(dst, src, n);
}
void launch_initial_z(const float* w, const float* wavg, float* z, long long n, cudaStream_t st) {
  initial_z_kernel<<<grid_for(n), kThreads, 0, st>>>(w, wavg, z, n);
}
void launch_initial_z_half(const __half* d, const float* wavg, float* z, long long n, cudaStream_t st) {
  initial_z_half_kernel<<<grid_for(n), kThreads, 0, st>>>(d, wavg, z, n);
}
void launch_state_dev(const float* w, const float* wavg, __half* d, long long n, cudaStream_t st) {
  state_dev_kernel<<<grid_for(n), kThreads, 0, st>>>(w, wavg, d, n);
}
void launch_state_value(const __half* d, const float* wavg, float* w, long long n, cudaStream_t st) {
  state_value_kernel<<<grid_for(n), kThreads, 0, st>>>(d, wavg, w, n);
}
void launch_update_w(const float* v, const float* z, float* w, long long n, float step, cudaStream_t st) {
  update_w_kernel<<<grid_for(n), kThreads, 0, st>>>(v, z, w, n, step);
}
void launch_convert_copy(const float* src, void* dst, int copy_kind, long long n, cudaStream_t st) {
  convert_kernel<<<grid_for(n), kThreads, 0, st>>>(src, dst, copy_kind, n);
}
void launch_widen(const __half* src, float* dst, long long n, cudaStream_t st) {
  widen_kernel<<<grid_for(n), kThreads, 0, st>>>(src, dst, n);
}
void launch_mace(int K, void* const* w, int w_half, float* const* x, float* wavg, long long n, float rho,
                 void* const* x_copy, int copy_kind, double* dchange, cudaStream_t st) {
  MacePtrs P{};
  for (int k = 0; k < K && k < kMaxK; ++k) {
    P.w[k] = w[k];
    P.x[k] = x[k];
    P.xc[k] = x_copy ? x_copy[k] : nullptr;
  }
  uintptr_t low = reinterpret_cast<uintptr_t>(wavg);
  for (int k = 0; k < K && k < kMaxK; ++k)
    low |= reinterpret_cast<uintptr_t>(P.w[k]) | reinterpret_cast<uintptr_t>(P.x[k]) |
           (copy_kind ? reinterpret_cast<uintptr_t>(P.xc[k]) : 0);
  const long long n4 = (low & 15) == 0 && K <= 4 ? n / 4 : 0;
  switch (K) {
    case 1: launch_mace_k<1>(K, P, w_half, wavg, n, n4, rho, copy_kind, dchange, st); break;
    case 2: launch_mace_k<2>(K, P, w_half, wavg, n, n4, rho, copy_kind, dchange, st); break;
    case 3: launch_mace_k<3>(K, P, w_half, wavg, n, n4, rho, copy_kind, dchange, st); break;
    case 4: launch_mace_k<4>(K, P, w_half, wavg, n, n4, rho, copy_kind, dchange, st); break;
    default: launch_mace_k<kMaxK>(K, P, w_half, wavg, n, n4, rho, copy_kind, dchange, st); break;
  }
}

}  // namespace mtr
