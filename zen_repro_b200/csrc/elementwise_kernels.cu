// Memory-bound model ops for sm_100a: norms (with the residual add fused in), gated activations,
// RoPE, embedding forward / row-sparse backward, cross-entropy (loss and dlogits in one kernel),
// column sums, and a multi-tensor AdamW.  All are bandwidth kernels: 16-byte accesses, one pass over
// each operand, fp32 math, bf16 / fp32 / fp16 storage.
//
// The reference takes these from HuggingFace modules and ColossalAI's HybridAdam
// (train.py:149-157); nothing of them is in its tree.
#include "act_common.cuh"
#include "launch.cuh"
#include "tc_common.cuh"
#include "xent_common.cuh"
#include "zen_common.cuh"

namespace {

using namespace zen_act;
using namespace zen_xe;

template <typename T> struct Vec8;   // 8 elements of T <-> 8 floats
template <> struct Vec8<__nv_bfloat16> {
  static __device__ __forceinline__ void load(const __nv_bfloat16* p, float (&v)[8]) {
    uint4 r = *reinterpret_cast<const uint4*>(p);
    uint32_t w[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) { v[2 * i] = __uint_as_float(w[i] << 16); v[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u); }
  }
  static __device__ __forceinline__ void store(__nv_bfloat16* p, const float (&v)[8]) {
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
      w[i] = *reinterpret_cast<uint32_t*>(&h);
    }
    *reinterpret_cast<uint4*>(p) = make_uint4(w[0], w[1], w[2], w[3]);
  }
};
template <> struct Vec8<__half> {
  static __device__ __forceinline__ void load(const __half* p, float (&v)[8]) {
    uint4 r = *reinterpret_cast<const uint4*>(p);
    const __half2* h = reinterpret_cast<const __half2*>(&r);
#pragma unroll
    for (int i = 0; i < 4; ++i) { float2 f = __half22float2(h[i]); v[2 * i] = f.x; v[2 * i + 1] = f.y; }
  }
  static __device__ __forceinline__ void store(__half* p, const float (&v)[8]) {
    uint4 r;
    __half2* h = reinterpret_cast<__half2*>(&r);
#pragma unroll
    for (int i = 0; i < 4; ++i) h[i] = __floats2half2_rn(v[2 * i], v[2 * i + 1]);
    *reinterpret_cast<uint4*>(p) = r;
  }
};
template <> struct Vec8<float> {
  static __device__ __forceinline__ void load(const float* p, float (&v)[8]) {
    float4 a = *reinterpret_cast<const float4*>(p), b = *reinterpret_cast<const float4*>(p + 4);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
  }
  static __device__ __forceinline__ void store(float* p, const float (&v)[8]) {
    *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
    *reinterpret_cast<float4*>(p + 4) = make_float4(v[4], v[5], v[6], v[7]);
  }
};

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int d = 16; d; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int d = 16; d; d >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, d));
  return v;
}
// Sum over the CTA (blockDim.x a multiple of 32, at most 1024); every thread gets the result.
__device__ __forceinline__ float block_sum(float v, float* sh) {
  v = warp_sum(v);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  __syncthreads();
  if (lane == 0) sh[w] = v;
  __syncthreads();
  float t = (lane < nw) ? sh[lane] : 0.f;
  return warp_sum(t);
}
__device__ __forceinline__ float block_max(float v, float* sh) {
  v = warp_max(v);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  __syncthreads();
  if (lane == 0) sh[w] = v;
  __syncthreads();
  float t = (lane < nw) ? sh[lane] : -INFINITY;
  return warp_max(t);
}

#define NORM_THREADS 128
#define NORM_MAXV 8   // up to 128 * 8 * 8 = 8192 columns held in registers; kernels are instantiated for 1, 2, 4, 8

// --------------------------------------------------------------------------------------------
// Norm forward.  h = x (+ res); y = (h - mean) * rstd * wgt + bias   (LayerNorm, kLayer)
//                                y = h * rstd * (wgt or 1 + wgt)     (RMSNorm)
// `hout` (optional) receives h, the new residual stream.  stats: rstd[rows] (+ mean[rows]).
template <typename T, bool kLayer, int NV>
__global__ void __launch_bounds__(NORM_THREADS)
norm_fwd_kernel(const T* x, const T* res, const T* wgt,
                const T* bias, T* __restrict__ y, T* __restrict__ hout, float* __restrict__ rstd_out,
                float* __restrict__ mean_out, int rows, int cols, float eps, int unit_offset) {
  zen_pdl::enter();
  __shared__ float sh[32];
  const int nv = cols / 8;                         // cols % 8 == 0 checked on the host
  for (int row = blockIdx.x; row < rows; row += gridDim.x) {
    const size_t base = (size_t)row * cols;
    float h[NV][8];
    float s = 0.f, ss = 0.f;
#pragma unroll
    for (int j = 0; j < NV; ++j) {
      const int v = threadIdx.x + j * NORM_THREADS;
      if (v < nv) {
        Vec8<T>::load(x + base + (size_t)v * 8, h[j]);
        if (res) {
          float r[8];
          Vec8<T>::load(res + base + (size_t)v * 8, r);
#pragma unroll
          for (int i = 0; i < 8; ++i) h[j][i] += r[i];
        }
        if (hout) {
          Vec8<T>::store(hout + base + (size_t)v * 8, h[j]);
          // keep exactly what was stored so that forward and backward see the same h
          Vec8<T>::load(hout + base + (size_t)v * 8, h[j]);
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) { s += h[j][i]; ss += h[j][i] * h[j][i]; }
      }
    }
    float mean = 0.f, var;
    if (kLayer) {
      mean = block_sum(s, sh) / cols;
      float d2 = 0.f;
#pragma unroll
      for (int j = 0; j < NV; ++j) {
        const int v = threadIdx.x + j * NORM_THREADS;
        if (v < nv) {
#pragma unroll
          for (int i = 0; i < 8; ++i) { const float d = h[j][i] - mean; d2 += d * d; }
        }
      }
      var = block_sum(d2, sh) / cols;
    } else {
      var = block_sum(ss, sh) / cols;
    }
    const float rstd = rsqrtf(var + eps);
    if (threadIdx.x == 0) { rstd_out[row] = rstd; if (kLayer) mean_out[row] = mean; }
#pragma unroll
    for (int j = 0; j < NV; ++j) {
      const int v = threadIdx.x + j * NORM_THREADS;
      if (v < nv) {
        float w[8], o[8];
        Vec8<T>::load(wgt + (size_t)v * 8, w);
        if (kLayer) {
          float b[8];
          if (bias) Vec8<T>::load(bias + (size_t)v * 8, b);
#pragma unroll
          for (int i = 0; i < 8; ++i) o[i] = (h[j][i] - mean) * rstd * w[i] + (bias ? b[i] : 0.f);
        } else {
#pragma unroll
          for (int i = 0; i < 8; ++i) o[i] = h[j][i] * rstd * (unit_offset ? 1.f + w[i] : w[i]);
        }
        Vec8<T>::store(y + base + (size_t)v * 8, o);
      }
    }
  }
}

// Rows kept as raw 16-byte vectors (8 registers per vector for fp32, 4 for 16-bit types) and unpacked on use.
template <typename T> struct Pack;
template <> struct Pack<float> {
  struct raw_t { float4 a, b; };
  static __device__ __forceinline__ raw_t load(const float* p) { raw_t r; r.a = *reinterpret_cast<const float4*>(p); r.b = *reinterpret_cast<const float4*>(p + 4); return r; }
  static __device__ __forceinline__ void unpack(const raw_t& r, float (&v)[8]) { v[0] = r.a.x; v[1] = r.a.y; v[2] = r.a.z; v[3] = r.a.w; v[4] = r.b.x; v[5] = r.b.y; v[6] = r.b.z; v[7] = r.b.w; }
};
template <> struct Pack<__nv_bfloat16> {
  typedef uint4 raw_t;
  static __device__ __forceinline__ raw_t load(const __nv_bfloat16* p) { return *reinterpret_cast<const uint4*>(p); }
  static __device__ __forceinline__ void unpack(const raw_t& r, float (&v)[8]) {
    const uint32_t w[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) { v[2 * i] = __uint_as_float(w[i] << 16); v[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u); }
  }
};
template <> struct Pack<__half> {
  typedef uint4 raw_t;
  static __device__ __forceinline__ raw_t load(const __half* p) { return *reinterpret_cast<const uint4*>(p); }
  static __device__ __forceinline__ void unpack(const raw_t& r, float (&v)[8]) {
    const __half2* h = reinterpret_cast<const __half2*>(&r);
#pragma unroll
    for (int i = 0; i < 4; ++i) { float2 f = __half22float2(h[i]); v[2 * i] = f.x; v[2 * i + 1] = f.y; }
  }
};

// Norm backward.  dh = grad through the norm (+ dres, the gradient arriving on the residual stream).
// Per-CTA partial sums of dw (and db) go to part_dw/part_db [gridDim.x][cols] (fp32 scratch) and are
// folded by colreduce_kernel.
template <typename T, bool kLayer, int NV, bool kParams>
__global__ void __launch_bounds__(NORM_THREADS)
norm_bwd_kernel(const T* dy, const T* h, const T* wgt,
                const float* rstd_in, const float* mean_in, const T* dres,
                T* __restrict__ dh, float* __restrict__ part_dw, float* __restrict__ part_db, int rows, int cols,
                int unit_offset) {
  zen_pdl::enter();
  __shared__ float sh[32];
  const int nv = cols / 8;
  // kParams = false: only dh here (the parameter gradients come from norm_dwdb_partial_kernel), which frees the
  // 16 * NV accumulator registers and lets several CTAs share an SM
  float aw[kParams ? NV : 1][8], ab[kParams ? NV : 1][8];
  if (kParams) {
#pragma unroll
    for (int j = 0; j < NV; ++j)
#pragma unroll
      for (int i = 0; i < 8; ++i) { aw[j][i] = 0.f; ab[j][i] = 0.f; }
  }
  for (int row = blockIdx.x; row < rows; row += gridDim.x) {
    const size_t base = (size_t)row * cols;
    const float rstd = rstd_in[row];
    const float mean = kLayer ? mean_in[row] : 0.f;
    float g[NV][8], xh[NV][8];
    typename Pack<T>::raw_t rres[NV];               // residual-stream gradient, fetched with the first loads
    float s1 = 0.f, s2 = 0.f;                       // sum(g), sum(g * xhat)
#pragma unroll
    for (int j = 0; j < NV; ++j) {
      const int v = threadIdx.x + j * NORM_THREADS;
      if (v < nv && dres) rres[j] = Pack<T>::load(dres + base + (size_t)v * 8);
    }
#pragma unroll
    for (int j = 0; j < NV; ++j) {
      const int v = threadIdx.x + j * NORM_THREADS;
      if (v < nv) {
        float d[8], w[8];
        Vec8<T>::load(dy + base + (size_t)v * 8, d);
        Vec8<T>::load(h + base + (size_t)v * 8, xh[j]);
        Vec8<T>::load(wgt + (size_t)v * 8, w);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          xh[j][i] = (xh[j][i] - mean) * rstd;
          if (kParams) { aw[j][i] += d[i] * xh[j][i]; ab[j][i] += d[i]; }
          g[j][i] = d[i] * (kLayer ? w[i] : (unit_offset ? 1.f + w[i] : w[i]));
          s1 += g[j][i];
          s2 += g[j][i] * xh[j][i];
        }
      }
    }
    s2 = block_sum(s2, sh) / cols;
    if (kLayer) s1 = block_sum(s1, sh) / cols; else s1 = 0.f;
#pragma unroll
    for (int j = 0; j < NV; ++j) {
      const int v = threadIdx.x + j * NORM_THREADS;
      if (v < nv) {
        float o[8];
        if (dres) Pack<T>::unpack(rres[j], o);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float t = rstd * (g[j][i] - s1 - xh[j][i] * s2);
          o[i] = dres ? o[i] + t : t;
        }
        Vec8<T>::store(dh + base + (size_t)v * 8, o);
      }
    }
  }
  if (!kParams) return;
#pragma unroll
  for (int j = 0; j < NV; ++j) {
    const int v = threadIdx.x + j * NORM_THREADS;
    if (v < nv) {
      Vec8<float>::store(part_dw + (size_t)blockIdx.x * cols + (size_t)v * 8, aw[j]);
      if (kLayer && part_db) Vec8<float>::store(part_db + (size_t)blockIdx.x * cols + (size_t)v * 8, ab[j]);
    }
  }
}

// ---- warp-per-row variants for narrow rows (cols <= 256 * NV): no block barriers, many rows in flight per SM.
// Rows are kept as raw 16-byte vectors (8 registers per vector for fp32, 4 for 16-bit types) and unpacked on use.
#define NORMW_WARPS 8

template <typename T, bool kLayer, int NV>
__global__ void __launch_bounds__(NORMW_WARPS * 32, 4)      // 64 registers: four CTAs (32 warps, a row each) per SM
norm_fwd_warp_kernel(const T* x, const T* res, const T* wgt,
                     const T* bias, T* __restrict__ y, T* __restrict__ hout, float* __restrict__ rstd_out,
                     float* __restrict__ mean_out, int rows, int cols, float eps, int unit_offset) {
  zen_pdl::enter();
  const int lane = threadIdx.x & 31;
  const int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = (gridDim.x * blockDim.x) >> 5;
  const int nv = cols / 8;
  for (int row = gw; row < rows; row += nw) {
    const size_t base = (size_t)row * cols;
    float h[NV][8];
    float s = 0.f, ss = 0.f;
#pragma unroll
    for (int j = 0; j < NV; ++j) {
      const int v = lane + 32 * j;
      if (v < nv) {
        Vec8<T>::load(x + base + (size_t)v * 8, h[j]);
        if (res) {
          float r[8];
          Vec8<T>::load(res + base + (size_t)v * 8, r);
#pragma unroll
          for (int i = 0; i < 8; ++i) h[j][i] += r[i];
        }
        if (hout) {
          Vec8<T>::store(hout + base + (size_t)v * 8, h[j]);
          if (sizeof(T) == 2) {   // continue with exactly what was stored
#pragma unroll
            for (int i = 0; i < 8; ++i) h[j][i] = ZenVal<T>::to_f(ZenVal<T>::from_f(h[j][i]));
          }
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) { s += h[j][i]; ss += h[j][i] * h[j][i]; }
      }
    }
    float mean = 0.f, var;
    if (kLayer) {
      mean = warp_sum(s) / cols;
      float d2 = 0.f;
#pragma unroll
      for (int j = 0; j < NV; ++j) {
        if (lane + 32 * j < nv) {
#pragma unroll
          for (int i = 0; i < 8; ++i) { const float d = h[j][i] - mean; d2 += d * d; }
        }
      }
      var = warp_sum(d2) / cols;
    } else {
      var = warp_sum(ss) / cols;
    }
    const float rstd = rsqrtf(var + eps);
    if (lane == 0) { rstd_out[row] = rstd; if (kLayer) mean_out[row] = mean; }
#pragma unroll
    for (int j = 0; j < NV; ++j) {
      const int v = lane + 32 * j;
      if (v < nv) {
        float w[8], o[8];
        Vec8<T>::load(wgt + (size_t)v * 8, w);
        if (kLayer) {
          float b[8];
          if (bias) Vec8<T>::load(bias + (size_t)v * 8, b);
#pragma unroll
          for (int i = 0; i < 8; ++i) o[i] = (h[j][i] - mean) * rstd * w[i] + (bias ? b[i] : 0.f);
        } else {
#pragma unroll
          for (int i = 0; i < 8; ++i) o[i] = h[j][i] * rstd * (unit_offset ? 1.f + w[i] : w[i]);
        }
        Vec8<T>::store(y + base + (size_t)v * 8, o);
      }
    }
  }
}

template <typename T, bool kLayer, int NV, bool kParams>
__global__ void __launch_bounds__(NORMW_WARPS * 32, (NV <= 3 && !kParams) ? 4 : 2)   // up to 768 columns: four CTAs per SM
norm_bwd_warp_kernel(const T* dy, const T* h, const T* wgt,
                     const float* rstd_in, const float* mean_in, const T* dres,
                     T* __restrict__ dh, float* __restrict__ part_dw, float* __restrict__ part_db, int rows, int cols,
                     int unit_offset) {
  zen_pdl::enter();
  extern __shared__ float sm_acc[];                 // [2][cols]: dw and db sums of this CTA
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = (gridDim.x * blockDim.x) >> 5;
  const int nv = cols / 8;
  float aw[kParams ? NV : 1][8], ab[(kLayer && kParams) ? NV : 1][8];
  // the weights stay packed (a warp usually handles one or two rows: half the registers of an unpacked copy, and with
  // them a fourth CTA per SM)
  typename Pack<T>::raw_t rw[NV];
  const float woff = (!kLayer && unit_offset) ? 1.f : 0.f;
#pragma unroll
  for (int j = 0; j < NV; ++j) {
#pragma unroll
    for (int i = 0; i < 8; ++i) { if (kParams) { aw[j][i] = 0.f; if (kLayer) ab[j][i] = 0.f; } }
    if (lane + 32 * j < nv) rw[j] = Pack<T>::load(wgt + (size_t)(lane + 32 * j) * 8);
  }
  for (int row = gw; row < rows; row += nw) {
    const size_t base = (size_t)row * cols;
    const float rstd = rstd_in[row];
    const float mean = kLayer ? mean_in[row] : 0.f;
    typename Pack<T>::raw_t rd[NV], rh[NV];
    float s1 = 0.f, s2 = 0.f;
#pragma unroll
    for (int j = 0; j < NV; ++j) {
      if (lane + 32 * j < nv) {
        rd[j] = Pack<T>::load(dy + base + (size_t)(lane + 32 * j) * 8);
        rh[j] = Pack<T>::load(h + base + (size_t)(lane + 32 * j) * 8);
      }
    }
#pragma unroll
    for (int j = 0; j < NV; ++j) {
      if (lane + 32 * j < nv) {
        float d[8], xh[8], wv[8];
        Pack<T>::unpack(rd[j], d);
        Pack<T>::unpack(rh[j], xh);
        Pack<T>::unpack(rw[j], wv);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          xh[i] = (xh[i] - mean) * rstd;
          if (kParams) { aw[j][i] += d[i] * xh[i]; if (kLayer) ab[j][i] += d[i]; }
          const float g = d[i] * (wv[i] + woff);
          s1 += g;
          s2 += g * xh[i];
        }
      }
    }
    s2 = warp_sum(s2) / cols;
    s1 = kLayer ? warp_sum(s1) / cols : 0.f;
#pragma unroll
    for (int j = 0; j < NV; ++j) {
      const int v = lane + 32 * j;
      if (v < nv) {
        float d[8], xh[8], o[8], wv[8];
        Pack<T>::unpack(rd[j], d);
        Pack<T>::unpack(rh[j], xh);
        Pack<T>::unpack(rw[j], wv);
        if (dres) Vec8<T>::load(dres + base + (size_t)v * 8, o);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float xhat = (xh[i] - mean) * rstd;
          const float t = rstd * (d[i] * (wv[i] + woff) - s1 - xhat * s2);
          o[i] = dres ? o[i] + t : t;
        }
        Vec8<T>::store(dh + base + (size_t)v * 8, o);
      }
    }
  }
  if (!kParams) return;
  // fold the warps' partial dw / db through shared memory, one warp at a time (fixed order)
  float* sdw = sm_acc;
  float* sdb = sm_acc + cols;
  for (int wsel = 0; wsel < NORMW_WARPS; ++wsel) {
    if (warp == wsel) {
#pragma unroll
      for (int j = 0; j < NV; ++j) {
        const int v = lane + 32 * j;
        if (v < nv) {
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            sdw[v * 8 + i] = (wsel == 0 ? 0.f : sdw[v * 8 + i]) + aw[j][i];
            if (kLayer) sdb[v * 8 + i] = (wsel == 0 ? 0.f : sdb[v * 8 + i]) + ab[j][i];
          }
        }
      }
    }
    __syncthreads();
  }
  for (int c = threadIdx.x; c < cols; c += blockDim.x) {
    part_dw[(size_t)blockIdx.x * cols + c] = sdw[c];
    if (kLayer && part_db) part_db[(size_t)blockIdx.x * cols + c] = sdb[c];
  }
}

// Norm backward in one pass: dh, the partial sums of dw and db, and (part_dh) the column sums of dh itself, which are the bias
// gradient of the layer before.  CTA b takes rows [b * chunk, (b + 1) * chunk), RS at a time: dy, h and dres arrive through a
// ring of stages (bulk copies; rows lie end to end, so a stage is one copy an array), 8 / RS warps work out a row's sums and
// its dh, then every thread adds its columns' share of the RS rows to sums that stay in registers until the chunk ends.
//
// What bounds it: memory, each operand once.  As separate kernels dh read dy, h and dres, the parameter sums dy and h again
// and the bias sums dh, each at two thirds of the L2's rate and with a launch of its own.
// us, two kernels / one (without the bias sums): 8192 x 768 18.8 / 13.4, 64 x 768 8.5 / 5.0, 4096 x 3072 37.2 / 24.3, 3000 x 2560
// 24.9 / 19.1, 8192 x 2048 43.3 / 35.1, 2048 x 2304 without a residual gradient 15.0 / 11.1.
constexpr int NF_STAGES = 3, NF_COLS = 3072;
__device__ int g_norm_error = 0;                        // a copy that never arrived (zen_norm_error)
template <typename T, bool kLayer, int RS>
__global__ void __launch_bounds__(256, 2)
norm_bwd_fused_kernel(const T* dy, const T* h, const T* wgt, const float* rstd_in, const float* mean_in, const T* dres, T* __restrict__ dh,
                      float* __restrict__ part_dw, float* __restrict__ part_db, float* __restrict__ part_dh, int rows, int cols, int chunk,
                      int unit_offset) {
  constexpr int WPR = 8 / RS, NIT = 3, NVT = RS >= 4 ? 1 : 2;   // warps to a row; vectors of a lane; of a thread's columns
  extern __shared__ __align__(128) unsigned char nf_smem[];
  __shared__ __align__(8) uint64_t full[NF_STAGES];
  __shared__ float red[8][2], srs[NF_STAGES][8], smu[NF_STAGES][8];
  __shared__ volatile int s_abort;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nv = cols / 8;
  const bool keep = part_dh != nullptr, third = dres != nullptr || keep;
  const uint32_t row_bytes = (uint32_t)cols * sizeof(T), arr = RS * row_bytes, stage_bytes = arr * (third ? 3 : 2);
  if (tid == 0) {
    s_abort = 0;
    for (int s = 0; s < NF_STAGES; ++s) tc::mbar_init(&full[s], 1);
    tc::fence_barrier_init();
  }
  __syncthreads();
  zen_pdl::enter();
  const int row0 = blockIdx.x * chunk, nrows = min(chunk, rows - row0), nsb = (nrows + RS - 1) / RS;
  auto issue = [&](int sb) {                            // thread 0
    const int s = sb % NF_STAGES, n = min(RS, nrows - sb * RS);
    const size_t at = (size_t)(row0 + sb * RS) * cols;
    unsigned char* st = nf_smem + s * stage_bytes;
    const uint32_t bytes = n * row_bytes;
    tc::mbar_expect_tx(&full[s], bytes * (dres ? 3 : 2));
    tc::bulk_load_1d(st, dy + at, bytes, &full[s]);
    tc::bulk_load_1d(st + arr, h + at, bytes, &full[s]);
    if (dres) tc::bulk_load_1d(st + 2 * arr, dres + at, bytes, &full[s]);
  };
  auto stats = [&](int sb) {                            // a thread per row of the stage
    if (tid < RS && sb * RS + tid < nrows) {
      const int r = row0 + sb * RS + tid;
      srs[sb % NF_STAGES][tid] = rstd_in[r];
      smu[sb % NF_STAGES][tid] = kLayer ? mean_in[r] : 0.f;
    }
  };
  if (tid == 0)
    for (int sb = 0; sb < min(nsb, NF_STAGES); ++sb) issue(sb);
  for (int sb = 0; sb < min(nsb, NF_STAGES); ++sb) stats(sb);
  const float woff = (!kLayer && unit_offset) ? 1.f : 0.f;
  const int row = warp / WPR, wsub = warp % WPR;
  typename Pack<T>::raw_t rw[NIT];
#pragma unroll
  for (int k = 0; k < NIT; ++k) {
    const int v = wsub * 32 + lane + k * 32 * WPR;
    if (v < nv) rw[k] = Pack<T>::load(wgt + (size_t)v * 8);
  }
  // column sums: threads in groups that walk interleaved rows where the columns do not take them all
  const int groups = nv <= 128 ? min(256 / nv, RS) : 1, g = groups > 1 ? tid / nv : 0, c0 = groups > 1 ? tid % nv : tid;
  float aw[NVT][8], ab[NVT][8], ah[NVT][8];
#pragma unroll
  for (int j = 0; j < NVT; ++j)
#pragma unroll
    for (int i = 0; i < 8; ++i) aw[j][i] = ab[j][i] = ah[j][i] = 0.f;
  __syncthreads();
  for (int sb = 0; sb < nsb; ++sb) {
    const int s = sb % NF_STAGES, n = min(RS, nrows - sb * RS);
    unsigned char* st = nf_smem + s * stage_bytes;
    T *sdy = reinterpret_cast<T*>(st), *shh = reinterpret_cast<T*>(st + arr), *sx = reinterpret_cast<T*>(st + 2 * arr);
    if (!tc::mbar_test(&full[s], (sb / NF_STAGES) & 1)) {
      const uint64_t t0 = tc::gtimer();
      while (!tc::mbar_test(&full[s], (sb / NF_STAGES) & 1))
        if (s_abort || tc::gtimer() - t0 > tc::WAIT_NS) { s_abort = 1; atomicCAS(&g_norm_error, 0, 1); break; }
    }
    const bool mine = row < n;
    float s1 = 0.f, s2 = 0.f;
    typename Pack<T>::raw_t rd[NIT], rh[NIT];
    const float rstd = mine ? srs[s][row] : 0.f, mean = mine ? smu[s][row] : 0.f;
    if (mine) {
#pragma unroll
      for (int k = 0; k < NIT; ++k) {
        const int v = wsub * 32 + lane + k * 32 * WPR;
        if (v < nv) {
          rd[k] = Pack<T>::load(sdy + (size_t)row * cols + v * 8);
          rh[k] = Pack<T>::load(shh + (size_t)row * cols + v * 8);
          float d[8], x[8], w[8];
          Pack<T>::unpack(rd[k], d);
          Pack<T>::unpack(rh[k], x);
          Pack<T>::unpack(rw[k], w);
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const float gr = d[i] * (w[i] + woff);
            s1 += gr;
            s2 += gr * ((x[i] - mean) * rstd);
          }
        }
      }
    }
    s1 = kLayer ? warp_sum(s1) : 0.f;
    s2 = warp_sum(s2);
    if (WPR > 1) {
      if (lane == 0) { red[warp][0] = s1; red[warp][1] = s2; }
      __syncthreads();
      s1 = s2 = 0.f;
#pragma unroll
      for (int k = 0; k < WPR; ++k) { s1 += red[row * WPR + k][0]; s2 += red[row * WPR + k][1]; }
    }
    s1 /= cols;
    s2 /= cols;
    if (mine) {
      T* out = dh + (size_t)(row0 + sb * RS + row) * cols;
#pragma unroll
      for (int k = 0; k < NIT; ++k) {
        const int v = wsub * 32 + lane + k * 32 * WPR;
        if (v < nv) {
          float d[8], x[8], w[8], o[8];
          Pack<T>::unpack(rd[k], d);
          Pack<T>::unpack(rh[k], x);
          Pack<T>::unpack(rw[k], w);
          if (dres) Vec8<T>::load(sx + (size_t)row * cols + v * 8, o);
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const float t = rstd * (d[i] * (w[i] + woff) - s1 - (x[i] - mean) * rstd * s2);
            o[i] = dres ? o[i] + t : t;
          }
          Vec8<T>::store(out + v * 8, o);
          if (keep) Vec8<T>::store(sx + (size_t)row * cols + v * 8, o);
        }
      }
    }
    if (keep) tc::fence_async_smem();                   // the next copy into this place comes after these stores
    __syncthreads();
    if (g < groups) {
#pragma unroll
      for (int j = 0; j < NVT; ++j) {
        const int c = c0 + j * 256;
        if (c >= nv) continue;
        for (int r = g; r < n; r += groups) {
          float d[8], x[8];
          Vec8<T>::load(sdy + (size_t)r * cols + c * 8, d);
          Vec8<T>::load(shh + (size_t)r * cols + c * 8, x);
          const float rs = srs[s][r], mu = smu[s][r];
#pragma unroll
          for (int i = 0; i < 8; ++i) { aw[j][i] += d[i] * (x[i] - mu) * rs; if (kLayer) ab[j][i] += d[i]; }
          if (keep) {
            float o[8];
            Vec8<T>::load(sx + (size_t)r * cols + c * 8, o);
#pragma unroll
            for (int i = 0; i < 8; ++i) ah[j][i] += o[i];
          }
        }
      }
    }
    // The stage of the step before this one is filled again.  A barrier does not wait for loads that have only been issued, so the
    // step's own stage would be too early.  The loads of the step before have all arrived: every warp has added what it read to its
    // sums, in program order before it came to the barrier in the middle of this step.
    const int next = sb - 1 + NF_STAGES;
    if (sb >= 1 && next < nsb) {
      if (tid == 0) issue(next);
      stats(next);
    }
    __syncthreads();
  }
  if (s_abort) {                                        // copies in flight are given time to land
    const uint64_t t0 = tc::gtimer();
    while (tc::gtimer() - t0 < 200000ull) __nanosleep(1000);
    return;
  }
  // groups fold into the first through shared memory, in group order
  float* fold = reinterpret_cast<float*>(nf_smem);
  for (int k = 1; k < groups; ++k) {
    if (g == k && c0 < nv) {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        fold[c0 * 8 + i] = aw[0][i];
        if (kLayer) fold[cols + c0 * 8 + i] = ab[0][i];
        if (keep) fold[2 * cols + c0 * 8 + i] = ah[0][i];
      }
    }
    __syncthreads();
    if (g == 0) {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        aw[0][i] += fold[c0 * 8 + i];
        if (kLayer) ab[0][i] += fold[cols + c0 * 8 + i];
        if (keep) ah[0][i] += fold[2 * cols + c0 * 8 + i];
      }
    }
    __syncthreads();
  }
  if (g == 0) {
#pragma unroll
    for (int j = 0; j < NVT; ++j) {
      const int c = c0 + j * 256;
      if (c >= nv) continue;
      const size_t at = (size_t)blockIdx.x * cols + c * 8;
      Vec8<float>::store(part_dw + at, aw[j]);
      if (kLayer && part_db) Vec8<float>::store(part_db + at, ab[j]);
      if (keep) Vec8<float>::store(part_dh + at, ah[j]);
    }
  }
}

// Norm forward through the same ring of stages: x and the residual arrive while earlier rows are worked on, and few enough CTAs
// start under their predecessor.  What bounds the kernels above, which it replaces up to NF_COLS columns of a 16-bit type: one
// row per warp or CTA, read, summed and written in turn, and (a CTA per row) h read back from where it had just been stored.
// us, before / now, with a residual: 8192 x 768 10.5 / 8.8, 20 000 x 768 28.8 / 20.5, 4096 x 3072 18.2 / 13.9, 8192 x 2048 25.2 / 21.0,
// 777 x 3072 6.2 / 4.5, 64 x 768 5.0 / 4.8.
template <typename T, bool kLayer, int RS, int NIT>
__global__ void __launch_bounds__(256, 2)
norm_fwd_staged_kernel(const T* x, const T* res, const T* wgt, const T* bias, T* __restrict__ y, T* __restrict__ hout, float* __restrict__ rstd_out,
                       float* __restrict__ mean_out, int rows, int cols, int chunk, float eps, int unit_offset) {
  constexpr int WPR = 8 / RS;
  extern __shared__ __align__(128) unsigned char nf_smem[];
  __shared__ __align__(8) uint64_t full[NF_STAGES];
  __shared__ float red[2][8];
  __shared__ volatile int s_abort;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nv = cols / 8;
  const uint32_t row_bytes = (uint32_t)cols * sizeof(T), arr = RS * row_bytes, stage_bytes = arr * (res ? 2 : 1);
  if (tid == 0) {
    s_abort = 0;
    for (int s = 0; s < NF_STAGES; ++s) tc::mbar_init(&full[s], 1);
    tc::fence_barrier_init();
  }
  __syncthreads();
  zen_pdl::enter();
  const int row0 = blockIdx.x * chunk, nrows = min(chunk, rows - row0), nsb = (nrows + RS - 1) / RS;
  auto issue = [&](int sb) {                            // thread 0
    const int s = sb % NF_STAGES, n = min(RS, nrows - sb * RS);
    const size_t at = (size_t)(row0 + sb * RS) * cols;
    unsigned char* st = nf_smem + s * stage_bytes;
    const uint32_t bytes = n * row_bytes;
    tc::mbar_expect_tx(&full[s], bytes * (res ? 2 : 1));
    tc::bulk_load_1d(st, x + at, bytes, &full[s]);
    if (res) tc::bulk_load_1d(st + arr, res + at, bytes, &full[s]);
  };
  if (tid == 0)
    for (int sb = 0; sb < min(nsb, NF_STAGES); ++sb) issue(sb);
  const int row = warp / WPR, wsub = warp % WPR;
  typename Pack<T>::raw_t rw[NIT], rb[kLayer ? NIT : 1];
#pragma unroll
  for (int k = 0; k < NIT; ++k) {
    const int v = wsub * 32 + lane + k * 32 * WPR;
    if (v < nv) {
      rw[k] = Pack<T>::load(wgt + (size_t)v * 8);
      if (kLayer && bias) rb[k] = Pack<T>::load(bias + (size_t)v * 8);
    }
  }
  // Sum over a row's warps, in the order of norm_fwd_warp_kernel up to 1024 columns and of norm_fwd_kernel above: a
  // last bit of one row's statistics flips one rounding in 400 000, which four layers of a Llama amplify to 0.9 % of the
  // logits, and the kernel that a call takes should not decide that.  `slot` alternates so that one barrier a sum is enough
  auto row_sum = [&](float v, int slot) {
    v = warp_sum(v);
    if constexpr (WPR == 1) return v;
    if (lane == 0) red[slot][warp] = v;
    __syncthreads();
    const float* r = &red[slot][row * WPR];
    return (r[0] + r[2]) + (r[1] + r[3]);                // as block_sum adds four warps
  };
  for (int sb = 0; sb < nsb; ++sb) {
    const int s = sb % NF_STAGES, n = min(RS, nrows - sb * RS);
    const T* sx = reinterpret_cast<const T*>(nf_smem + s * stage_bytes);
    const T* sr = reinterpret_cast<const T*>(nf_smem + s * stage_bytes + arr);
    if (!tc::mbar_test(&full[s], (sb / NF_STAGES) & 1)) {
      const uint64_t t0 = tc::gtimer();
      while (!tc::mbar_test(&full[s], (sb / NF_STAGES) & 1))
        if (s_abort || tc::gtimer() - t0 > tc::WAIT_NS) { s_abort = 1; atomicCAS(&g_norm_error, 0, 2); break; }
    }
    const bool mine = row < n;
    const size_t base = (size_t)(row0 + sb * RS + row) * cols;
    float h[NIT][8], sum = 0.f;
    if (mine) {
#pragma unroll
      for (int k = 0; k < NIT; ++k) {
        const int v = wsub * 32 + lane + k * 32 * WPR;
        if (v < nv) {
          Vec8<T>::load(sx + (size_t)row * cols + v * 8, h[k]);
          if (res) {
            float r[8];
            Vec8<T>::load(sr + (size_t)row * cols + v * 8, r);
#pragma unroll
            for (int i = 0; i < 8; ++i) h[k][i] += r[i];
          }
          if (hout) {                                   // continue with exactly what is stored
            Vec8<T>::store(hout + base + v * 8, h[k]);
#pragma unroll
            for (int i = 0; i < 8; ++i) h[k][i] = ZenVal<T>::to_f(ZenVal<T>::from_f(h[k][i]));
          }
#pragma unroll
          for (int i = 0; i < 8; ++i) sum += kLayer ? h[k][i] : h[k][i] * h[k][i];
        }
      }
    }
    float mean = 0.f, var = row_sum(sum, 0) / cols;
    if (kLayer) {
      mean = var;
      float d2 = 0.f;
      if (mine) {
#pragma unroll
        for (int k = 0; k < NIT; ++k)
          if (wsub * 32 + lane + k * 32 * WPR < nv) {
#pragma unroll
            for (int i = 0; i < 8; ++i) { const float d = h[k][i] - mean; d2 += d * d; }
          }
      }
      var = row_sum(d2, 1) / cols;
    }
    const float rstd = rsqrtf(var + eps);
    if (mine) {
      if (wsub == 0 && lane == 0) {
        rstd_out[row0 + sb * RS + row] = rstd;
        if (kLayer) mean_out[row0 + sb * RS + row] = mean;
      }
#pragma unroll
      for (int k = 0; k < NIT; ++k) {
        const int v = wsub * 32 + lane + k * 32 * WPR;
        if (v < nv) {
          float w[8], b[8], o[8];
          Pack<T>::unpack(rw[k], w);
          if (kLayer && bias) Pack<T>::unpack(rb[k], b);
#pragma unroll
          for (int i = 0; i < 8; ++i)
            o[i] = kLayer ? (h[k][i] - mean) * rstd * w[i] + (bias ? b[i] : 0.f) : h[k][i] * rstd * (unit_offset ? 1.f + w[i] : w[i]);
          Vec8<T>::store(y + base + v * 8, o);
        }
      }
    }
    __syncthreads();
    // this step's rows have been summed, so none of its loads is still on its way: sums went through shuffles before the barrier
    if (tid == 0 && sb + NF_STAGES < nsb) issue(sb + NF_STAGES);
  }
  if (s_abort) {                                        // copies in flight are given time to land
    const uint64_t t0 = tc::gtimer();
    while (tc::gtimer() - t0 < 200000ull) __nanosleep(1000);
  }
}

// Parameter gradients of a norm, column-sum style: CTA b covers rows [32 b, 32 b + 32) and every column (a thread
// owns 8 columns, loads are coalesced along the row): part_dw[b][c] = sum_r dy * xhat, part_db[b][c] = sum_r dy.
template <typename T, bool kLayer>
__global__ void __launch_bounds__(256)
norm_dwdb_partial_kernel(const T* dy, const T* h, const float* rstd_in,
                         const float* mean_in, float* __restrict__ part_dw, float* __restrict__ part_db,
                         int rows, int cols, int rows_per_cta) {
  zen_pdl::enter();
  // Wide matrices: blockIdx.y selects a 2048-column slice (one vector per thread), blockIdx.x a group of rows.
  // Narrow matrices (fewer 8-column vectors than threads): the threads form `groups` row groups that walk
  // interleaved rows of the CTA's 32 and meet in shared memory, group by group, so that no thread idles.
  __shared__ float red_w[2048], red_b[2048];
  const int r0 = blockIdx.x * rows_per_cta, r1 = min(rows, r0 + rows_per_cta);
  const int vpr = cols / 8;
  const int groups = vpr <= 128 ? 256 / vpr : 1;
  const int g = groups > 1 ? threadIdx.x / vpr : 0;
  const int c8 = groups > 1 ? (threadIdx.x % vpr) * 8 : (blockIdx.y * 256 + threadIdx.x) * 8;   // this thread's one vector
  // threads left over when 256 is not a multiple of vpr stay with their warp for the barriers
  const bool live = g < groups && c8 < cols;
  float aw[8] = {0, 0, 0, 0, 0, 0, 0, 0}, ab[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  if (live) {
#pragma unroll 4
    for (int r = r0 + g; r < r1; r += groups) {
      float d[8], x[8];
      Vec8<T>::load(dy + (size_t)r * cols + c8, d);
      Vec8<T>::load(h + (size_t)r * cols + c8, x);
      const float rs = rstd_in[r], mu = kLayer ? mean_in[r] : 0.f;
#pragma unroll
      for (int i = 0; i < 8; ++i) { aw[i] += d[i] * (x[i] - mu) * rs; ab[i] += d[i]; }
    }
  }
  for (int k = 1; k < groups; ++k) {                         // fold group k into group 0, in group order
    if (live && g == k) {
#pragma unroll
      for (int i = 0; i < 8; ++i) { red_w[c8 + i] = aw[i]; red_b[c8 + i] = ab[i]; }
    }
    __syncthreads();
    if (live && g == 0) {
#pragma unroll
      for (int i = 0; i < 8; ++i) { aw[i] += red_w[c8 + i]; ab[i] += red_b[c8 + i]; }
    }
    __syncthreads();
  }
  if (live && g == 0) {
    Vec8<float>::store(part_dw + (size_t)blockIdx.x * cols + c8, aw);
    if (kLayer && part_db) Vec8<float>::store(part_db + (size_t)blockIdx.x * cols + c8, ab);
  }
}

// out[c] (+)= sum_p part[p][c], cast to T.  CTA = 32 columns x 32 part-lanes; fixed summation order.
// blockIdx.y == 1 reduces a second (part, out) pair of the same shape in the same launch (dw and db of a LayerNorm).
template <typename T>
__global__ void __launch_bounds__(1024)
colreduce_kernel(const float* part, T* __restrict__ out, int nparts, int cols, int accumulate,
                 const float* part2 = nullptr, T* __restrict__ out2 = nullptr) {
  zen_pdl::enter();
  if (blockIdx.y == 1) { part = part2; out = out2; }
  __shared__ float sh[32][33];
  const int x = threadIdx.x & 31, y = threadIdx.x >> 5;
  const int c = blockIdx.x * 32 + x;
  float s = 0.f;
  if (c < cols)
    for (int p = y; p < nparts; p += 32) s += part[(size_t)p * cols + c];
  sh[y][x] = s;
  __syncthreads();
  if (y == 0 && c < cols) {
    float t = 0.f;
#pragma unroll
    for (int i = 0; i < 32; ++i) t += sh[i][x];
    if (accumulate) t += ZenVal<T>::to_f(out[c]);
    out[c] = ZenVal<T>::from_f(t);
  }
}

// Several reductions of that kind in one launch (the bias and norm-parameter gradients of a layer): blockIdx.y = 2 * job
// (+ 1 for the job's second pair, if it has one), blockIdx.x = 32-column block of that job.
#define COLREDUCE_MAX_JOBS 8
struct ColReduceJob {
  const float* part;
  void* out;
  const float* part2;             // optional second (part, out) pair of the same shape (dw and db of a LayerNorm)
  void* out2;
  int nparts, cols, accumulate, pad;
};
struct ColReduceJobs {
  ColReduceJob j[COLREDUCE_MAX_JOBS];
  int n;
};
template <typename T>
__global__ void __launch_bounds__(1024)
colreduce_multi_kernel(const ColReduceJobs jobs) {
  zen_pdl::enter();
  const ColReduceJob& jb = jobs.j[blockIdx.y >> 1];
  const float* part = (blockIdx.y & 1) ? jb.part2 : jb.part;
  T* out = reinterpret_cast<T*>((blockIdx.y & 1) ? jb.out2 : jb.out);
  if (!part || !out || (int)blockIdx.x * 32 >= jb.cols) return;                // uniform over the CTA
  __shared__ float sh[32][33];
  const int x = threadIdx.x & 31, y = threadIdx.x >> 5;
  const int c = blockIdx.x * 32 + x;
  float s = 0.f;
  if (c < jb.cols)
    for (int p = y; p < jb.nparts; p += 32) s += part[(size_t)p * jb.cols + c];
  sh[y][x] = s;
  __syncthreads();
  if (y == 0 && c < jb.cols) {
    float t = 0.f;
#pragma unroll
    for (int i = 0; i < 32; ++i) t += sh[i][x];
    if (jb.accumulate) t += ZenVal<T>::to_f(out[c]);
    out[c] = ZenVal<T>::from_f(t);
  }
}

// Column sums of a [rows, cols] matrix: CTA b sums rows [b * rows_per_cta, ...) for every column (thread = one
// 8-column vector, coalesced along the row) into part[b][cols] (bias gradients).
template <typename T>
__global__ void __launch_bounds__(256) colsum_partial_kernel(const T* a, float* __restrict__ part, int rows, int cols, int rows_per_cta) {
  zen_pdl::enter();
  __shared__ float red[2048];                                // see norm_dwdb_partial_kernel: row groups for narrow matrices
  const int r0 = blockIdx.x * rows_per_cta, r1 = min(rows, r0 + rows_per_cta);
  const int vpr = cols / 8;
  const int groups = vpr <= 128 ? 256 / vpr : 1;
  if (groups == 1) {                                          // wide matrix: every thread has columns of its own
    for (int c8 = threadIdx.x * 8; c8 < cols; c8 += blockDim.x * 8) {
      float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll 8
      for (int r = r0; r < r1; ++r) {
        float v[8];
        Vec8<T>::load(a + (size_t)r * cols + c8, v);
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[i] += v[i];
      }
      Vec8<float>::store(part + (size_t)blockIdx.x * cols + c8, acc);
    }
    return;
  }
  const int g = threadIdx.x / vpr, c8 = (threadIdx.x % vpr) * 8;
  const bool live = g < groups;                               // leftover threads stay with their warp for the barriers
  float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  if (live) {
#pragma unroll 8
    for (int r = r0 + g; r < r1; r += groups) {
      float v[8];
      Vec8<T>::load(a + (size_t)r * cols + c8, v);
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[i] += v[i];
    }
  }
  for (int k = 1; k < groups; ++k) {
    if (live && g == k) {
#pragma unroll
      for (int i = 0; i < 8; ++i) red[c8 + i] = acc[i];
    }
    __syncthreads();
    if (live && g == 0) {
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[i] += red[c8 + i];
    }
    __syncthreads();
  }
  if (live && g == 0) Vec8<float>::store(part + (size_t)blockIdx.x * cols + c8, acc);
}

// --------------------------------------------------------------------------------------------
__device__ __forceinline__ float gelu_tanh_grad(float x) {
  const float k = 0.7978845608028654f;
  const float t = tanh_fast(k * (x + 0.044715f * x * x * x));
  return 0.5f * (1.f + t) + 0.5f * x * (1.f - t * t) * k * (1.f + 3.f * 0.044715f * x * x);
}

// a and b may be the two halves of one [rows, 2 * inner] matrix (strided) or separate tensors.
//
// What bounds these: memory, if enough of it is asked for at once.  One vector per thread and trip, and an index taken apart with a 64-bit
// division, left them at half of the copy rate: the loads of a trip cannot pass the stores of the one before (the pointers
// promise nothing).  ACT_U vectors per thread are loaded before any is stored, 512 threads on two CTAs per SM, which start
// under their predecessor.  us, before / now, forward: 4096 x 8192 SwiGLU 49.4 / 38.5, 2048 x 9216 GeGLU 24.7 / 17.4, 8192 x 16 384
// 151 / 139; backward 63.8 / 59.0, 35.0 / 31.6, 215 / 204.  (The same for the column-sum form below and for the rotation of heads,
// which walk rows or heads that the compiler unrolls: nothing gained, 5 to 20 % lost.)
constexpr int ACT_U = 4, ACT_THREADS = 512;
struct ActPos { int r, c; };                            // row, vector of the row
__device__ __forceinline__ ActPos act_pos(uint32_t v, uint32_t vpr) {
  const uint32_t r = v / vpr;
  return ActPos{(int)r, (int)(v - r * vpr)};
}
template <typename T, int MODE>
__global__ void __launch_bounds__(ACT_THREADS, 2)
act_fwd_kernel(const T* a, const T* b, T* __restrict__ out, int rows, int inner, int lda, int ldb) {
  zen_pdl::enter();
  const uint32_t vpr = inner / 8, nvec = (uint32_t)rows * vpr;
  for (uint32_t v0 = blockIdx.x * (ACT_THREADS * ACT_U) + threadIdx.x; v0 < nvec; v0 += gridDim.x * (ACT_THREADS * ACT_U)) {
    typename Pack<T>::raw_t x[ACT_U], y[ACT_U];
    size_t at[ACT_U];
#pragma unroll
    for (int u = 0; u < ACT_U; ++u) {
      const uint32_t v = v0 + u * ACT_THREADS;
      if (v >= nvec) break;
      const ActPos p = act_pos(v, vpr);
      at[u] = (size_t)p.r * inner + p.c * 8;
      x[u] = Pack<T>::load(a + (size_t)p.r * lda + p.c * 8);
      if (MODE >= 2) y[u] = Pack<T>::load(b + (size_t)p.r * ldb + p.c * 8);
    }
#pragma unroll
    for (int u = 0; u < ACT_U; ++u) {
      if (v0 + u * ACT_THREADS >= nvec) break;
      float xv[8], yv[8], o[8];
      Pack<T>::unpack(x[u], xv);
      if (MODE >= 2) Pack<T>::unpack(y[u], yv);
#pragma unroll
      for (int i = 0; i < 8; ++i) o[i] = zen_act::value(MODE, xv[i], MODE >= 2 ? yv[i] : 0.f);
      Vec8<T>::store(out + at[u], o);
    }
  }
}

template <typename T, int MODE>
__global__ void __launch_bounds__(ACT_THREADS, 2)
act_bwd_kernel(const T* a, const T* b, const T* dout, T* __restrict__ da, T* __restrict__ db, int rows, int inner, int lda, int ldb) {
  zen_pdl::enter();
  constexpr int U = 2;                                  // three operands: six loads under way
  const uint32_t vpr = inner / 8, nvec = (uint32_t)rows * vpr;
  for (uint32_t v0 = blockIdx.x * (ACT_THREADS * U) + threadIdx.x; v0 < nvec; v0 += gridDim.x * (ACT_THREADS * U)) {
    typename Pack<T>::raw_t xr[U], yr[U], gr[U];
    ActPos p[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const uint32_t v = v0 + u * ACT_THREADS;
      if (v >= nvec) break;
      p[u] = act_pos(v, vpr);
      xr[u] = Pack<T>::load(a + (size_t)p[u].r * lda + p[u].c * 8);
      gr[u] = Pack<T>::load(dout + (size_t)p[u].r * inner + p[u].c * 8);
      if (MODE >= 2) yr[u] = Pack<T>::load(b + (size_t)p[u].r * ldb + p[u].c * 8);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (v0 + u * ACT_THREADS >= nvec) break;
      float x[8], y[8], g[8], ga[8], gb[8];
      Pack<T>::unpack(xr[u], x);
      Pack<T>::unpack(gr[u], g);
      if (MODE >= 2) Pack<T>::unpack(yr[u], y);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        if (MODE == 0) ga[i] = g[i] * gelu_tanh_grad(x[i]);
        else if (MODE == 1) ga[i] = x[i] > 0.f ? g[i] : 0.f;
        else if (MODE == 2) {
          const float s = sigmoidf_(x[i]);
          ga[i] = g[i] * y[i] * s * (1.f + x[i] * (1.f - s));
          gb[i] = g[i] * x[i] * s;
        } else {
          ga[i] = g[i] * y[i] * gelu_tanh_grad(x[i]);
          gb[i] = g[i] * gelu_tanh(x[i]);
        }
      }
      Vec8<T>::store(da + (size_t)p[u].r * lda + p[u].c * 8, ga);
      if (MODE >= 2) Vec8<T>::store(db + (size_t)p[u].r * ldb + p[u].c * 8, gb);
    }
  }
}

// Backward of an ungated activation (mode 0 / 1) that also leaves the column sums of its result, the bias gradient of
// the linear layer that produced the activation's input: CTA b handles rows [b * rows_per_cta, ...) of every column and
// writes part[b][inner], the layout that colreduce_kernel sums.  The separate column-sum kernel would read da again.
template <typename T>
__global__ void __launch_bounds__(512)
act_bwd_colsum_kernel(const T* a, const T* dout, T* __restrict__ da, float* __restrict__ part,
                      int rows, int inner, int mode, int rows_per_cta) {
  zen_pdl::enter();
  const int r0 = blockIdx.x * rows_per_cta, r1 = min(rows, r0 + rows_per_cta);
  for (int c8 = threadIdx.x * 8; c8 < inner; c8 += blockDim.x * 8) {
    float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll 4
    for (int r = r0; r < r1; ++r) {
      float x[8], g[8], ga[8];
      Vec8<T>::load(a + (size_t)r * inner + c8, x);
      Vec8<T>::load(dout + (size_t)r * inner + c8, g);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float v = (mode == 0) ? g[i] * gelu_tanh_grad(x[i]) : (x[i] > 0.f ? g[i] : 0.f);
        ga[i] = ZenVal<T>::to_f(ZenVal<T>::from_f(v));       // the sum is that of the stored values
        acc[i] += ga[i];
      }
      Vec8<T>::store(da + (size_t)r * inner + c8, ga);
    }
    Vec8<float>::store(part + (size_t)blockIdx.x * inner + c8, acc);
  }
}

// --------------------------------------------------------------------------------------------
// RoPE (rotate-half convention): x is [tokens, heads, hd] with row stride `ld` elements between
// tokens; token t sits at position pos0 + t % seq.  sign = -1 applies the inverse rotation
// (the backward pass).  In place.
template <typename T>
__global__ void __launch_bounds__(256)
rope_kernel(T* __restrict__ x, int tokens, int heads, int hd, int ld, int seq, int pos0, float log2_theta, float sign) {
  zen_pdl::enter();
  const int half = hd / 2;
  const size_t n = (size_t)tokens * heads * half;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const int j = (int)(i % half);
    const int hh = (int)((i / half) % heads);
    const int t = (int)(i / ((size_t)half * heads));
    const float inv_freq = exp2f(-log2_theta * (2.f * j / hd));
    float s, c;
    sincosf((float)(pos0 + t % seq) * inv_freq, &s, &c);
    s *= sign;
    T* p = x + (size_t)t * ld + (size_t)hh * hd;
    const float a = ZenVal<T>::to_f(p[j]), b = ZenVal<T>::to_f(p[j + half]);
    p[j] = ZenVal<T>::from_f(a * c - b * s);
    p[j + half] = ZenVal<T>::from_f(b * c + a * s);
  }
}

// Vectorised form for hd / 2 a multiple of 8: a thread owns 8 consecutive frequencies of one token, computes their
// sines and cosines once and walks all heads with 16-byte loads and stores (the scalar kernel above recomputes the
// trigonometry for every head and moves two bytes per access).  With few tokens the heads are split over hgroups threads so
// that the GPU fills up (777 tokens, 24 + 8 heads of 128: 24 CTAs, 11 us before; the trigonometry is then repeated, which
// idle SMs do for nothing).
template <typename T>
__global__ void __launch_bounds__(256)
rope_vec_kernel(T* __restrict__ x, int tokens, int heads, int hd, int ld, int seq, int pos0, float log2_theta, float sign, int hgroups) {
  zen_pdl::enter();
  const int half = hd / 2, vph = half / 8;
  const size_t n = (size_t)tokens * vph * hgroups;
  for (size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x; idx < n; idx += (size_t)gridDim.x * blockDim.x) {
    const int jv = (int)(idx % vph);
    const int hg = (int)((idx / vph) % hgroups);
    const int t = (int)(idx / ((size_t)vph * hgroups));
    const float pos = (float)(pos0 + t % seq);
    float c[8], sn[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float inv_freq = exp2f(-log2_theta * (2.f * (jv * 8 + i) / hd));
      sincosf(pos * inv_freq, &sn[i], &c[i]);
      sn[i] *= sign;
    }
    T* p = x + (size_t)t * ld + jv * 8;
#pragma unroll 4
    for (int hh = heads * hg / hgroups; hh < heads * (hg + 1) / hgroups; ++hh) {
      float a[8], b[8], oa[8], ob[8];
      Vec8<T>::load(p + (size_t)hh * hd, a);
      Vec8<T>::load(p + (size_t)hh * hd + half, b);
#pragma unroll
      for (int i = 0; i < 8; ++i) { oa[i] = a[i] * c[i] - b[i] * sn[i]; ob[i] = b[i] * c[i] + a[i] * sn[i]; }
      Vec8<T>::store(p + (size_t)hh * hd, oa);
      Vec8<T>::store(p + (size_t)hh * hd + half, ob);
    }
  }
}

// --------------------------------------------------------------------------------------------
// Embedding forward: out[t] = wte[ids[t]] * scale (+ wpe[pos_offset + t % seq]).
template <typename T>
__global__ void __launch_bounds__(128)
embedding_fwd_kernel(const int64_t* ids, const T* wte, const T* wpe,
                     T* __restrict__ out, int tokens, int d, int seq, int pos_offset, float scale, int vocab) {
  zen_pdl::enter();
  for (int t = blockIdx.x; t < tokens; t += gridDim.x) {
    int64_t id = ids[t];
    if (id < 0 || id >= vocab) id = 0;
    for (int c = threadIdx.x * 8; c < d; c += blockDim.x * 8) {
      float v[8];
      Vec8<T>::load(wte + (size_t)id * d + c, v);
      if (scale != 1.f) {
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = ZenVal<T>::to_f(ZenVal<T>::from_f(v[i] * scale));
      }
      if (wpe) {
        float p[8];
        Vec8<T>::load(wpe + (size_t)(pos_offset + t % seq) * d + c, p);
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] += p[i];
      }
      Vec8<T>::store(out + (size_t)t * d + c, v);
    }
  }
}

// Row-sparse embedding backward, four kernels over a bitmap of the vocabulary (bit r of word r / 32 = row r is touched) with
// one prefix count per word, both in the caller's flag buffer ([words | prefixes], zero between calls):
//   mark    : set the bits of the token ids
//   compact : one CTA scans the words (8 000 for a 256 000-row table; as one flag per row the scan took 185 us):
//             prefix[w] = touched rows before word w, rows[] ascending, *count
//   accum   : acc[rank(id)][:] += dy[t][:] * scale   (fp32 atomics into a [U, d] scratch)
//   finish  : vals = T(acc); acc and the bitmap are zeroed for the next call
__global__ void embed_mark_kernel(const int64_t* ids, uint32_t* __restrict__ bits, int tokens, int vocab) {
  zen_pdl::enter();
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < tokens; t += gridDim.x * blockDim.x) {
    const int64_t id = ids[t];
    if (id >= 0 && id < vocab) atomicOr(bits + (id >> 5), 1u << (id & 31));
  }
}

// Thread t owns words [t * per, (t + 1) * per).
__global__ void __launch_bounds__(1024)
embed_compact_kernel(const uint32_t* bits, uint32_t* __restrict__ prefix, int32_t* __restrict__ rows, int32_t* __restrict__ count,
                     int words) {
  zen_pdl::enter();
  __shared__ uint32_t wtot[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int per = (words + 1023) / 1024, b = threadIdx.x * per, e = min(words, b + per);
  uint32_t s = 0;
  for (int i = b; i < e; ++i) s += __popc(bits[i]);
  uint32_t pre = s;                                                   // inclusive scan over the warp, then over the warps
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t t = __shfl_up_sync(0xffffffffu, pre, d);
    if (lane >= d) pre += t;
  }
  if (lane == 31) wtot[warp] = pre;
  __syncthreads();
  uint32_t wp = wtot[lane];
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t t = __shfl_up_sync(0xffffffffu, wp, d);
    if (lane >= d) wp += t;
  }
  const uint32_t total = __shfl_sync(0xffffffffu, wp, 31);
  uint32_t run = __shfl_sync(0xffffffffu, wp, warp) - wtot[warp] + pre - s;
  for (int i = b; i < e; ++i) {
    prefix[i] = run;
    for (uint32_t w = bits[i]; w; w &= w - 1) rows[run++] = i * 32 + __ffs((int)w) - 1;
  }
  if (threadIdx.x == 0) *count = (int32_t)total;
}

template <typename T>
__global__ void __launch_bounds__(128)
embed_accum_kernel(const int64_t* ids, const uint32_t* bits, const uint32_t* prefix,
                   const T* dy, float* __restrict__ acc, int tokens, int d, int vocab, float scale) {
  zen_pdl::enter();
  for (int t = blockIdx.x; t < tokens; t += gridDim.x) {
    const int64_t id = ids[t];
    if (id < 0 || id >= vocab) continue;
    const uint32_t u = prefix[id >> 5] + __popc(bits[id >> 5] & ((1u << (id & 31)) - 1u));
    for (int c = threadIdx.x * 8; c < d; c += blockDim.x * 8) {
      float v[8];
      Vec8<T>::load(dy + (size_t)t * d + c, v);
      float* a = acc + (size_t)u * d + c;
      atomicAdd(reinterpret_cast<float4*>(a), make_float4(v[0] * scale, v[1] * scale, v[2] * scale, v[3] * scale));
      atomicAdd(reinterpret_cast<float4*>(a + 4), make_float4(v[4] * scale, v[5] * scale, v[6] * scale, v[7] * scale));
    }
  }
}

template <typename T>
__global__ void __launch_bounds__(128)
embed_finish_kernel(float* __restrict__ acc, uint32_t* __restrict__ bits, int words, const int32_t* count, T* __restrict__ vals, int d) {
  zen_pdl::enter();
  const int n = *count;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < words; i += gridDim.x * blockDim.x) bits[i] = 0u;
  for (int u = blockIdx.x; u < n; u += gridDim.x) {
    for (int c = threadIdx.x * 8; c < d; c += blockDim.x * 8) {
      float v[8];
      Vec8<float>::load(acc + (size_t)u * d + c, v);
      Vec8<T>::store(vals + (size_t)u * d + c, v);
      const float z[8] = {0, 0, 0, 0, 0, 0, 0, 0};
      Vec8<float>::store(acc + (size_t)u * d + c, z);
    }
  }
}

// Gradient of learned position embeddings: out[s][:] (+)= sum over the batch of dy[b * S + s][:].
template <typename T>
__global__ void __launch_bounds__(256)
pos_grad_kernel(const T* dy, T* __restrict__ out, int B, int S, int d, int accumulate) {
  zen_pdl::enter();
  const size_t n = (size_t)S * (d / 8);
  for (size_t v = (size_t)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += (size_t)gridDim.x * blockDim.x) {
    float a[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll 4
    for (int b = 0; b < B; ++b) {
      float x[8];
      Vec8<T>::load(dy + ((size_t)b * n + v) * 8, x);
#pragma unroll
      for (int i = 0; i < 8; ++i) a[i] += x[i];
    }
    if (accumulate) {
      float x[8];
      Vec8<T>::load(out + v * 8, x);
#pragma unroll
      for (int i = 0; i < 8; ++i) a[i] = ZenVal<T>::to_f(ZenVal<T>::from_f(a[i])) + x[i];
    }
    Vec8<T>::store(out + v * 8, a);
  }
}

// lab[b][s] = labels[b][s + shift] (ignore beyond the sequence); *inv = 1 / max(1, labels that count).  One CTA.
__global__ void __launch_bounds__(1024)
label_prep_kernel(const int64_t* labels, int64_t* __restrict__ lab, float* __restrict__ inv, int B, int S, int shift, int64_t ignore) {
  zen_pdl::enter();
  __shared__ uint32_t tot;
  if (threadIdx.x == 0) tot = 0;
  __syncthreads();
  uint32_t c = 0;
  for (int i = threadIdx.x; i < B * S; i += 1024) {
    const int64_t v = (i % S) + shift < S ? labels[i + shift] : ignore;
    if (lab) lab[i] = v;
    c += v != ignore;
  }
#pragma unroll
  for (int d = 16; d; d >>= 1) c += __shfl_xor_sync(0xffffffffu, c, d);
  if ((threadIdx.x & 31) == 0) atomicAdd(&tot, c);
  __syncthreads();
  if (threadIdx.x == 0) *inv = 1.f / (float)(tot ? tot : 1u);
}

// *out = (sum of x) * scale.  One CTA, fixed order.
__global__ void __launch_bounds__(1024)
sum_scale_kernel(const float* x, int n, const float* scale, float* __restrict__ out) {
  zen_pdl::enter();
  __shared__ float sh[32];
  float s = 0.f;
  for (int i = threadIdx.x; i < n; i += 1024) s += x[i];
  s = block_sum(s, sh);
  if (threadIdx.x == 0) *out = s * *scale;
}

// out = cap * tanh(x / cap) in fp32 from [rows, cols] logits (row stride ld) to a dense matrix.
template <typename T>
__global__ void __launch_bounds__(256)
softcap_kernel(const T* x, float* __restrict__ out, int rows, int cols, int ld, float cap) {
  zen_pdl::enter();
  const size_t n = (size_t)rows * cols;
  for (size_t i = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) * 4; i < n; i += (size_t)gridDim.x * blockDim.x * 4)
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (i + k < n) {
        const size_t r = (i + k) / cols, c = (i + k) % cols;
        out[i + k] = cap * tanhf(ZenVal<T>::to_f(x[r * ld + c]) / cap);
      }
}

// grad[rows[u]][:] += vals[u][:] for u < *count (rows unique): applies a row-sparse gradient to a dense one.
template <typename T>
__global__ void __launch_bounds__(128)
rows_add_kernel(T* __restrict__ grad, const int32_t* rows, const int32_t* count,
                const T* vals, int d, int vocab, int max_rows) {
  zen_pdl::enter();
  const int n = min(*count, max_rows);
  for (int u = blockIdx.x; u < n; u += gridDim.x) {
    const int r = rows[u];
    if (r < 0 || r >= vocab) continue;
    for (int c = threadIdx.x * 8; c < d; c += blockDim.x * 8) {
      float a[8], b[8];
      Vec8<T>::load(grad + (size_t)r * d + c, a);
      Vec8<T>::load(vals + (size_t)u * d + c, b);
#pragma unroll
      for (int i = 0; i < 8; ++i) a[i] += b[i];
      Vec8<T>::store(grad + (size_t)r * d + c, a);
    }
  }
}

// --------------------------------------------------------------------------------------------
// Cross-entropy over [rows, vocab] logits, one CTA per row, two passes: maximum and sum of exponentials, then dlogits =
// (softmax - onehot) * gscale written in place (or to `dlogits`).  loss[row] = lse - logit[label]; rows with label == ignore
// give loss 0 and zero gradient.  `ld` = row stride in elements.  CAP: the logits are soft-capped on the way,
// y = cap tanh(x / cap), and the gradient goes back through it.
//
// What bounds it: memory, if the second pass finds the row in L2.  512-thread CTAs, four to an SM, had 592 rows under way (300 MB
// at a vocabulary of 256 000, the L2 holds 126) and one 16-byte load per thread in flight: 2.88 ms for 8192 rows, 3.3 TB/s
// of the three passes.  Now as many threads to a row as keep the rows under way within the L2 (the launcher decides), two to
// four loads in flight per thread, one rescaling of the running sum per 16 elements, no label test per element.
constexpr int XENT_U = 2;

// Eight elements as loaded; unpacked only where they are used (the loads in flight then take half the registers).
template <typename T> struct Raw8v {
  uint4 q[sizeof(T) / 2];
  __device__ __forceinline__ void load(const T* p) {
#pragma unroll
    for (int i = 0; i < (int)(sizeof(T) / 2); ++i) q[i] = reinterpret_cast<const uint4*>(p)[i];
  }
  __device__ __forceinline__ float at(int i) const {
    const uint32_t* w = reinterpret_cast<const uint32_t*>(q);
    if constexpr (sizeof(T) == 4) return __uint_as_float(w[i]);
    else return ZenVal<T>::unbits((i & 1) ? w[i >> 1] >> 16 : w[i >> 1] & 0xffffu);
  }
};

template <typename T, bool CAP, int XENT_THREADS>
__global__ void __launch_bounds__(XENT_THREADS, XENT_THREADS == 512 ? 2 : 1)
xent_kernel(const T* logits, const int64_t* labels, float* __restrict__ loss,
            T* __restrict__ dlogits, int rows, int vocab, int ld, float gscale_host, const float* gscale_dev,
            int64_t ignore_index, float cap) {
  zen_pdl::enter();
  __shared__ float sh[32];
  const float gscale = gscale_dev ? gscale_host * (*gscale_dev) : gscale_host;
  const float k2 = CAP ? 2.f * L2E / cap : 0.f;
  const bool vec_ok = ld % 8 == 0 && (reinterpret_cast<uintptr_t>(logits) | reinterpret_cast<uintptr_t>(dlogits)) % 16 == 0;
  const int nv = vec_ok ? vocab / 8 : 0;                // vector body; tail handled scalar
  for (int row = blockIdx.x; row < rows; row += gridDim.x) {
    const T* lp = logits + (size_t)row * ld;
    T* dp = dlogits ? dlogits + (size_t)row * ld : nullptr;
    const int64_t label = labels[row];
    const bool valid = label != ignore_index && label >= 0 && label < vocab;
    float slope_label = 1.f;                            // thread 0: the label's logit and, soft-capped, the cap's slope there
    const float at_label = valid && threadIdx.x == 0 ? xent_cap<T, CAP>(ZenVal<T>::to_f(lp[label]), cap, k2, &slope_label) : 0.f;
    float m = -INFINITY, s = 0.f;
    // the next XENT_U vectors of the thread are on their way while the current ones are worked on; beyond the row's end the
    // last vector is read again and not used
    auto fetch = [&](Raw8v<T>(&x)[XENT_U], int v0) {
#pragma unroll
      for (int u = 0; u < XENT_U; ++u) x[u].load(lp + (size_t)min(v0 + u * XENT_THREADS, nv - 1) * 8);
    };
    if ((int)threadIdx.x < nv) {
      Raw8v<T> x[XENT_U], y[XENT_U];
      fetch(x, threadIdx.x);
      for (int v0 = threadIdx.x; v0 < nv; v0 += XENT_THREADS * XENT_U) {
        fetch(y, v0 + XENT_THREADS * XENT_U);
        float mx = -INFINITY;
#pragma unroll
        for (int u = 0; u < XENT_U; ++u)
#pragma unroll
          for (int i = 0; i < 8; ++i) mx = fmaxf(mx, x[u].at(i));
        if (CAP) mx = xent_cap<T, CAP>(mx, cap, k2);  // monotonic
        const float nm = fmaxf(m, mx);
        // exponents are made of differences: with x * L2E - nm * L2E in one FMA a maximum of the type's lowest value (masked
        // logits) overflows, and large logits lose the bits that cancel.  Nothing but -inf so far: exp(-inf - 0) = 0.
        const float ref = nm == -INFINITY ? 0.f : nm;
        float add[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int u = 0; u < XENT_U; ++u)
          if (v0 + u * XENT_THREADS < nv) {
#pragma unroll
            for (int i = 0; i < 8; ++i) add[i & 3] += ex2_fast((xent_cap<T, CAP>(x[u].at(i), cap, k2) - ref) * L2E);
          }
        s = s * ex2_fast((m - ref) * L2E) + ((add[0] + add[1]) + (add[2] + add[3]));
        m = nm;
#pragma unroll
        for (int u = 0; u < XENT_U; ++u) x[u] = y[u];
      }
    }
    for (int c = nv * 8 + threadIdx.x; c < vocab; c += XENT_THREADS) {
      const float x = xent_cap<T, CAP>(ZenVal<T>::to_f(lp[c]), cap, k2);
      const float nm = fmaxf(m, x), ref = nm == -INFINITY ? 0.f : nm;
      s = s * __expf(m - ref) + __expf(x - ref);
      m = nm;
    }
    const float gm = block_max(m, sh);
    s = (m == -INFINITY) ? 0.f : s * __expf(m - gm);
    const float gs = block_sum(s, sh);
    const float lse = gm + logf(gs);
    if (threadIdx.x == 0) loss[row] = valid ? lse - at_label : 0.f;
    if (dp) {
      const float sc = valid ? gscale : 0.f;
      if ((int)threadIdx.x < nv) {
        Raw8v<T> x[XENT_U], y[XENT_U];
        fetch(x, threadIdx.x);
        for (int v0 = threadIdx.x; v0 < nv; v0 += XENT_THREADS * XENT_U) {
          fetch(y, v0 + XENT_THREADS * XENT_U);
#pragma unroll
          for (int u = 0; u < XENT_U; ++u)
            if (v0 + u * XENT_THREADS < nv) {
              float o[8];
#pragma unroll
              for (int i = 0; i < 8; ++i) {
                float slope = 1.f;
                const float p = ex2_fast((xent_cap<T, CAP>(x[u].at(i), cap, k2, &slope) - lse) * L2E);
                o[i] = CAP ? p * sc * slope : p * sc;
              }
              Vec8<T>::store(dp + (size_t)(v0 + u * XENT_THREADS) * 8, o);
            }
#pragma unroll
          for (int u = 0; u < XENT_U; ++u) x[u] = y[u];
        }
      }
      for (int c = nv * 8 + threadIdx.x; c < vocab; c += XENT_THREADS) {
        float slope = 1.f;
        const float p = __expf(xent_cap<T, CAP>(ZenVal<T>::to_f(lp[c]), cap, k2, &slope) - lse);
        dp[c] = ZenVal<T>::from_f(CAP ? p * sc * slope : p * sc);
      }
      __syncthreads();
      if (valid && threadIdx.x == 0) {                  // the label's own entry: softmax - 1
        const float g = (ex2_fast((at_label - lse) * L2E) - 1.f) * sc;
        dp[label] = ZenVal<T>::from_f(CAP ? g * slope_label : g);
      }
    }
  }
}

// --------------------------------------------------------------------------------------------
// Cross-entropy whose row statistics come out of the product that makes the logits (zen_gemm_bf16_2cta_loss):
//   xent_finish_kernel : lse and loss of each row from the (maximum, sum of exponentials) of its 128-column pieces
//   xent_grad_kernel   : dlogits = (exp(y - lse) - onehot) * gscale in place, one pass
// xent_kernel makes the same out of the logits alone, but reads them twice and has two exponentials an element to do (three
// times two special functions when soft-capped) between which nothing overlaps within a row.  us, xent_kernel / finish + grad:
// 8192 x 50 257 397 / 11 + 296, 4096 x 128 256 539 / 23 + 360, 8192 x 256 000 2 210 / 47 + 1 493, 2048 x 256 000 soft-capped 972 / 39 + 558
// (memory alone, read and write once: 251, 320, 1 280, 320).  Without a gradient the logits are not even written: 215 / 11.
constexpr int XF_ROWS = 16, XF_G = 32;                  // rows of a CTA (128 bytes of a piece) and pieces side by side
template <bool CAP>
__global__ void __launch_bounds__(XF_ROWS * XF_G)
xent_finish_kernel(const float2* part, int nparts, int part_ld, const float* target, const int64_t* labels, float* loss, float* lse_out,
                   int rows, int vocab, int64_t ignore_index, float cap) {
  zen_pdl::enter();
  __shared__ float2 sh[XF_G][XF_ROWS];
  const int r = threadIdx.x % XF_ROWS, g = threadIdx.x / XF_ROWS, row = blockIdx.x * XF_ROWS + r;
  float m = -INFINITY, s = 0.f;
  if (row < rows) {
    for (int p0 = g; p0 < nparts; p0 += XF_G * 8) {
      float2 x[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) x[u] = p0 + u * XF_G < nparts ? part[(size_t)(p0 + u * XF_G) * part_ld + row] : make_float2(-INFINITY, 0.f);
      float nm = m;
#pragma unroll
      for (int u = 0; u < 8; ++u) nm = fmaxf(nm, x[u].x);
      const float ref = nm == -INFINITY ? 0.f : nm;
      s *= __expf(m - ref);
#pragma unroll
      for (int u = 0; u < 8; ++u) s += x[u].y * __expf(x[u].x - ref);
      m = nm;
    }
  }
  sh[g][r] = make_float2(m, s);
  __syncthreads();
  if (g == 0 && row < rows) {
#pragma unroll
    for (int k = 0; k < XF_G; ++k) m = fmaxf(m, sh[k][r].x);
    const float ref = m == -INFINITY ? 0.f : m;
    s = 0.f;
#pragma unroll
    for (int k = 0; k < XF_G; ++k) s += sh[k][r].y * __expf(sh[k][r].x - ref);
    const float lse = m + logf(s);
    const int64_t label = labels[row];
    const bool valid = label != ignore_index && label >= 0 && label < vocab;
    lse_out[row] = lse;
    loss[row] = valid ? lse - xent_cap<__nv_bfloat16, CAP>(target[row], cap, CAP ? 2.f * L2E / cap : 0.f) : 0.f;
  }
}

constexpr int XG_U = 4;                                 // vectors of eight in flight per thread
template <bool CAP>
__global__ void __launch_bounds__(256)
xent_grad_kernel(__nv_bfloat16* logits, const int64_t* labels, const float* lse_in, int rows, int vocab, int ld, float gscale_host,
                 const float* gscale_dev, int64_t ignore_index, float cap) {
  typedef __nv_bfloat16 T;
  zen_pdl::enter();
  const float gscale = gscale_dev ? gscale_host * (*gscale_dev) : gscale_host;
  const float k2 = CAP ? 2.f * L2E / cap : 0.f;
  const int nv = vocab / 8;                             // ld % 8 == 0 and the base on 16 bytes: checked by the launcher
  for (int row = blockIdx.x; row < rows; row += gridDim.x) {
    T* lp = logits + (size_t)row * ld;
    const int64_t label = labels[row];
    const bool valid = label != ignore_index && label >= 0 && label < vocab;
    const float lse = lse_in[row], sc = valid ? gscale : 0.f;
    const int at = valid ? (int)label : -1;
    auto grad = [&](float x, bool hit) -> float {
      float slope = 1.f;
      const float p = ex2_fast((xent_cap<T, CAP>(x, cap, k2, &slope) - lse) * L2E);
      const float g = (hit ? p - 1.f : p) * sc;
      return CAP ? g * slope : g;
    };
    for (int v0 = threadIdx.x; v0 < nv; v0 += 256 * XG_U) {
      Raw8v<T> x[XG_U];
#pragma unroll
      for (int u = 0; u < XG_U; ++u)
        if (v0 + u * 256 < nv) x[u].load(lp + (size_t)(v0 + u * 256) * 8);
#pragma unroll
      for (int u = 0; u < XG_U; ++u) {
        const int v = v0 + u * 256;
        if (v >= nv) continue;
        float o[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) o[i] = grad(x[u].at(i), false);
        if ((at >> 3) == v && at >= 0) {
          float slope = 1.f;
          const float y = xent_cap<T, CAP>(ZenVal<T>::to_f(lp[at]), cap, k2, &slope);
          const float g = (ex2_fast((y - lse) * L2E) - 1.f) * sc;
#pragma unroll
          for (int i = 0; i < 8; ++i)
            if ((at & 7) == i) o[i] = CAP ? g * slope : g;
        }
        Vec8<T>::store(lp + (size_t)v * 8, o);
      }
    }
    for (int c = nv * 8 + threadIdx.x; c < vocab; c += 256) lp[c] = ZenVal<T>::from_f(grad(ZenVal<T>::to_f(lp[c]), c == at));
  }
}

// Vocabulary-parallel cross-entropy, two kernels around the small cross-rank reductions:
//   xent_partial_kernel : per row, max and sum-exp over this rank's vocabulary shard (columns >= valid_cols are
//                         padding and ignored), plus the target logit when the label falls in the shard
//   xent_apply_kernel   : dlogits = (exp(x - lse) - onehot) * scale in place, with the global lse of each row
template <typename T>
__global__ void __launch_bounds__(512)
xent_partial_kernel(const T* logits, const int64_t* labels, float* __restrict__ rowmax,
                    float* __restrict__ sumexp, float* __restrict__ target, int rows, int valid_cols, int ld,
                    int64_t vocab_start, int64_t ignore_index) {
  zen_pdl::enter();
  __shared__ float sh[32];
  for (int row = blockIdx.x; row < rows; row += gridDim.x) {
    const T* lp = logits + (size_t)row * ld;
    float m = -INFINITY, s = 0.f;
    for (int c = threadIdx.x; c < valid_cols; c += blockDim.x) {
      const float x = ZenVal<T>::to_f(lp[c]);
      const float nm = fmaxf(m, x);
      s = s * __expf(m - nm) + __expf(x - nm);
      m = nm;
    }
    const float gm = block_max(m, sh);
    s = (m == -INFINITY) ? 0.f : s * __expf(m - gm);
    const float gs = block_sum(s, sh);
    if (threadIdx.x == 0) {
      rowmax[row] = gm;
      sumexp[row] = gs;
      const int64_t lab = labels[row] - vocab_start;
      target[row] = (labels[row] != ignore_index && lab >= 0 && lab < valid_cols) ? ZenVal<T>::to_f(lp[lab]) : 0.f;
    }
  }
}

template <typename T>
__global__ void __launch_bounds__(512)
xent_apply_kernel(T* __restrict__ logits, const int64_t* labels, const float* lse,
                  int rows, int cols, int valid_cols, int ld, float gscale_host, const float* gscale_dev,
                  int64_t vocab_start, int64_t ignore_index) {
  zen_pdl::enter();
  const float gscale = gscale_dev ? gscale_host * (*gscale_dev) : gscale_host;
  for (int row = blockIdx.x; row < rows; row += gridDim.x) {
    T* lp = logits + (size_t)row * ld;
    const bool valid = labels[row] != ignore_index;
    const int64_t lab = labels[row] - vocab_start;
    const float l = lse[row], sc = valid ? gscale : 0.f;
    for (int c = threadIdx.x; c < cols; c += blockDim.x) {
      float pr = (c < valid_cols) ? __expf(ZenVal<T>::to_f(lp[c]) - l) : 0.f;
      if (c == lab) pr -= 1.f;
      lp[c] = ZenVal<T>::from_f(pr * sc);
    }
  }
}

// --------------------------------------------------------------------------------------------
// Multi-tensor AdamW.  One table entry per tensor; CTAs walk a flat list of 64K-element chunks.
struct AdamTensor {
  void* param;       // T (bf16 / fp32) weights used by the model
  float* master;     // optional fp32 master copy (null when param is fp32)
  void* grad;        // T gradient
  float* m;
  float* v;
  uint64_t numel;
  uint64_t chunk0;   // index of this tensor's first chunk
  float wd;          // weight decay for this tensor
  int32_t clear;     // leave zeros in the gradient (2 bytes written beside the 28 moved, instead of a fill of its own later)
};
#define ADAM_CHUNK 65536

// One AdamW element update.  The square root and the quotient use the approximate units (about 2 ulp): the update is
// rounded to bf16 (or added to an fp32 master) right after, and the exact sequences cost several times the
// instructions, enough to show against the 22 bytes per element this kernel moves.
__device__ __forceinline__ void adam_update(float& p, float& m, float& v, float g, float b1, float b2, float eps,
                                            float ibc1, float isb2, float decay, float lr) {
  m = b1 * m + (1.f - b1) * g;
  v = b2 * v + (1.f - b2) * g * g;
  float sq;
  asm("sqrt.approx.f32 %0, %1;" : "=f"(sq) : "f"(v));
  const float den = fmaf(sq, isb2, eps);
  p = fmaf(-lr, __fdividef(m * ibc1, den), p * decay);
}

// Eight floats in one access (32-byte aligned).  As two accesses of 16 bytes each lane's half-sectors are 32 bytes apart: the loads ask
// for every sector twice, and the stores reach L2 as partial sectors.  AdamW over 58 M parameters 350 -> 320 us, over 50 M in fp32 276 ->
// 269; over 700 M and more it stays at 6.0 TB/s, 92 % of a copy's rate, either way.
__device__ __forceinline__ void load256(const float* p, float (&v)[8]) {
  asm volatile("ld.global.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]) : "l"(p));
}
__device__ __forceinline__ void store256(float* p, const float (&v)[8]) {
  asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
               ::"l"(p), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7]) : "memory");
}

template <typename T>
__global__ void __launch_bounds__(256)
adamw_kernel(const AdamTensor* tab, int ntensors, const int32_t* chunk_tensor,
             uint64_t nchunks, float lr, float b1, float b2, float eps, float bc1, float bc2, float gscale,
             const int32_t* step_dev) {
  zen_pdl::enter();
  if (step_dev) {                        // step count kept on the device (CUDA-graph replay): derive the bias corrections here
    const float t = (float)(*step_dev);
    bc1 = 1.f - powf(b1, t);
    bc2 = 1.f - powf(b2, t);
  }
  const float ibc1 = 1.f / bc1, isb2 = rsqrtf(bc2);
  for (uint64_t ch = blockIdx.x; ch < nchunks; ch += gridDim.x) {
    const AdamTensor t = tab[chunk_tensor[ch]];
    const uint64_t start = (ch - t.chunk0) * ADAM_CHUNK;
    const uint64_t end = min(t.numel, start + ADAM_CHUNK);
    T* p = reinterpret_cast<T*>(t.param);
    T* g = reinterpret_cast<T*>(t.grad);
    const float zeros[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    const float decay = 1.f - lr * t.wd;
    const bool wide = ((reinterpret_cast<uintptr_t>(t.master) | reinterpret_cast<uintptr_t>(t.m) | reinterpret_cast<uintptr_t>(t.v)) & 31) == 0;
    // two 8-element vectors per thread and trip, all loads issued before the arithmetic
    for (uint64_t i0 = start + (uint64_t)threadIdx.x * 8; i0 < end; i0 += 2 * 256 * 8) {
      const uint64_t i1 = i0 + 256 * 8;
      if (i1 + 8 <= end) {
        float pv[2][8], gv[2][8], mv[2][8], vv[2][8];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const uint64_t i = u ? i1 : i0;
          if (t.master && wide) load256(t.master + i, pv[u]);
          else if (t.master) Vec8<float>::load(t.master + i, pv[u]);
          else Vec8<T>::load(p + i, pv[u]);
          Vec8<T>::load(g + i, gv[u]);
          if (wide) {
            load256(t.m + i, mv[u]);
            load256(t.v + i, vv[u]);
          } else {
            Vec8<float>::load(t.m + i, mv[u]);
            Vec8<float>::load(t.v + i, vv[u]);
          }
        }
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const uint64_t i = u ? i1 : i0;
#pragma unroll
          for (int k = 0; k < 8; ++k) adam_update(pv[u][k], mv[u][k], vv[u][k], gv[u][k] * gscale, b1, b2, eps, ibc1, isb2, decay, lr);
          if (wide) {
            store256(t.m + i, mv[u]);
            store256(t.v + i, vv[u]);
            if (t.master) store256(t.master + i, pv[u]);
          } else {
            Vec8<float>::store(t.m + i, mv[u]);
            Vec8<float>::store(t.v + i, vv[u]);
            if (t.master) Vec8<float>::store(t.master + i, pv[u]);
          }
          Vec8<T>::store(p + i, pv[u]);
          if (t.clear) Vec8<T>::store(g + i, zeros);
        }
        continue;
      }
      for (int u = 0; u < 2; ++u) {
        const uint64_t i = u ? i1 : i0;
        if (i >= end) break;
        if (i + 8 <= end) {
          float pv[8], gv[8], mv[8], vv[8];
          if (t.master) Vec8<float>::load(t.master + i, pv); else Vec8<T>::load(p + i, pv);
          Vec8<T>::load(g + i, gv);
          Vec8<float>::load(t.m + i, mv);
          Vec8<float>::load(t.v + i, vv);
#pragma unroll
          for (int k = 0; k < 8; ++k) adam_update(pv[k], mv[k], vv[k], gv[k] * gscale, b1, b2, eps, ibc1, isb2, decay, lr);
          Vec8<float>::store(t.m + i, mv);
          Vec8<float>::store(t.v + i, vv);
          if (t.master) Vec8<float>::store(t.master + i, pv);
          Vec8<T>::store(p + i, pv);
          if (t.clear) Vec8<T>::store(g + i, zeros);
        } else {
          for (uint64_t k = i; k < end; ++k) {
            float pv = t.master ? t.master[k] : ZenVal<T>::to_f(p[k]);
            float mm = t.m[k], vv = t.v[k];
            adam_update(pv, mm, vv, ZenVal<T>::to_f(g[k]) * gscale, b1, b2, eps, ibc1, isb2, decay, lr);
            t.m[k] = mm; t.v[k] = vv;
            if (t.master) t.master[k] = pv;
            p[k] = ZenVal<T>::from_f(pv);
            if (t.clear) g[k] = ZenVal<T>::from_f(0.f);
          }
        }
      }
    }
  }
}

int sm_count_e() {
  static int n = 0;
  if (!n) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    if (n <= 0) n = 148;
  }
  return n;
}
// Rows per CTA of the column-sum passes: two CTAs per SM, 32 rows at most (64 rows of 768 columns on two CTAs of 32 rows took
// 7 us, all of it the latency of the rows one after the other).
inline int colsum_rpc(int rows) {
  const int rpc = (rows + 2 * sm_count_e() - 1) / (2 * sm_count_e());
  return rpc < 1 ? 1 : (rpc > 32 ? 32 : rpc);
}
inline int cap_grid(size_t want, int mult) {
  size_t mx = (size_t)sm_count_e() * mult;
  return (int)(want < 1 ? 1 : (want > mx ? mx : want));
}

}  // namespace

#define DISPATCH_T(dtype, ...)                                             \
  switch (dtype) {                                                         \
    case ZEN_DTYPE_F32: { using T = float; __VA_ARGS__; } break;           \
    case ZEN_DTYPE_BF16: { using T = __nv_bfloat16; __VA_ARGS__; } break;  \
    case ZEN_DTYPE_F16: { using T = __half; __VA_ARGS__; } break;          \
    default: return -1;                                                    \
  }

extern "C" {

// Rows of at most NORMW_MAXCOLS columns use the warp-per-row kernels, wider rows the CTA-per-row kernels.

#define NORMW_MAXCOLS 1024
static inline bool norm_warp_path(int cols, int dtype) { (void)dtype; return cols <= NORMW_MAXCOLS; }

// Number of per-CTA partial rows the norm backward writes (the caller sizes its scratch with this).
int zen_norm_bwd_parts(int rows) { const int a = cap_grid((size_t)rows, 2), b = (rows + 7) / 8; return a > b ? a : b; }

#define NORM_NV_DISPATCH(cols, ...)                                   \
  if (cols <= NORM_THREADS * 8) { constexpr int NV = 1; __VA_ARGS__; } \
  else if (cols <= NORM_THREADS * 16) { constexpr int NV = 2; __VA_ARGS__; } \
  else if (cols <= NORM_THREADS * 32) { constexpr int NV = 4; __VA_ARGS__; } \
  else { constexpr int NV = 8; __VA_ARGS__; }
#define NORMW_NV_DISPATCH(cols, ...)                        \
  if (cols <= 256) { constexpr int NV = 1; __VA_ARGS__; }   \
  else if (cols <= 512) { constexpr int NV = 2; __VA_ARGS__; } \
  else if (cols <= 768) { constexpr int NV = 3; __VA_ARGS__; } \
  else { constexpr int NV = 4; __VA_ARGS__; }

int zen_norm_fwd(const void* x, const void* res, const void* w, const void* b, void* y, void* hout, float* rstd,
                 float* mean, int rows, int cols, float eps, int layer, int unit_offset, int dtype, void* stream) {
  if (cols % 8 || cols > NORM_THREADS * NORM_MAXV * 8) return -2;
  cudaStream_t st = (cudaStream_t)stream;
  const uintptr_t ptrs = reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(res) | reinterpret_cast<uintptr_t>(w) |
                         reinterpret_cast<uintptr_t>(b) | reinterpret_cast<uintptr_t>(y) | reinterpret_cast<uintptr_t>(hout);
  if (ptrs % 16) return -3;                             // every kernel below reads and writes 16 bytes at a time
  if (dtype != ZEN_DTYPE_F32 && cols <= NF_COLS && rows > 0) {
    const int chunk = (rows + 2 * sm_count_e() - 1) / (2 * sm_count_e()), grid = (rows + chunk - 1) / chunk;
#define NORM_STAGED(L_, RS_, NIT_)                                                                                                      \
  do {                                                                                                                                  \
    const size_t smem = (size_t)NF_STAGES * (res ? 2 : 1) * RS_ * cols * 2;                                                             \
    static const int rc = (int)cudaFuncSetAttribute(norm_fwd_staged_kernel<T, L_, RS_, NIT_>, cudaFuncAttributeMaxDynamicSharedMemorySize, \
                                                    NF_STAGES * 2 * 8 * 1024 * 2);                                                      \
    if (rc) return rc;                                                                                                                  \
    zen_pdl::launch_small(norm_fwd_staged_kernel<T, L_, RS_, NIT_>, grid, 256, smem, st, (const T*)x, (const T*)res, (const T*)w, (const T*)b,  \
                          (T*)y, (T*)hout, rstd, mean, rows, cols, chunk, eps, unit_offset);                                            \
  } while (0)
#define NORM_STAGED_RS(L_)                                   \
  do {                                                       \
    if (cols <= 768) NORM_STAGED(L_, 8, 3);                  \
    else if (cols <= 1024) NORM_STAGED(L_, 8, 4);            \
    else NORM_STAGED(L_, 2, 3);                              \
  } while (0)
    const auto run = [&](auto zero) -> int {
      typedef decltype(zero) T;
      if (layer) NORM_STAGED_RS(true); else NORM_STAGED_RS(false);
      return (int)cudaGetLastError();
    };
#undef NORM_STAGED_RS
#undef NORM_STAGED
    return dtype == ZEN_DTYPE_BF16 ? run(__nv_bfloat16()) : run(__half());
  }
  if (norm_warp_path(cols, dtype)) {
    const int grid = cap_grid((size_t)(rows + NORMW_WARPS - 1) / NORMW_WARPS, 8);
    DISPATCH_T(dtype, {
      NORMW_NV_DISPATCH(cols, {
        if (layer) zen_pdl::launch_small(norm_fwd_warp_kernel<T, true, NV>, grid, NORMW_WARPS * 32, 0, st, (const T*)x, (const T*)res, (const T*)w, (const T*)b, (T*)y, (T*)hout, rstd, mean, rows, cols, eps, unit_offset);
        else zen_pdl::launch_small(norm_fwd_warp_kernel<T, false, NV>, grid, NORMW_WARPS * 32, 0, st, (const T*)x, (const T*)res, (const T*)w, (const T*)b, (T*)y, (T*)hout, rstd, mean, rows, cols, eps, unit_offset);
      });
    });
    return (int)cudaGetLastError();
  }
  const int grid = cap_grid((size_t)rows, 16);
  DISPATCH_T(dtype, {
    NORM_NV_DISPATCH(cols, {
      if (layer) zen_pdl::launch_small(norm_fwd_kernel<T, true, NV>, grid, NORM_THREADS, 0, st, (const T*)x, (const T*)res, (const T*)w, (const T*)b, (T*)y, (T*)hout, rstd, mean, rows, cols, eps, unit_offset);
      else zen_pdl::launch_small(norm_fwd_kernel<T, false, NV>, grid, NORM_THREADS, 0, st, (const T*)x, (const T*)res, (const T*)w, (const T*)b, (T*)y, (T*)hout, rstd, mean, rows, cols, eps, unit_offset);
    });
  });
  return (int)cudaGetLastError();
}

// part_dw / part_db: fp32 scratch of zen_norm_bwd_parts(rows) * cols each.  dw / db are written (or
// accumulated into when accumulate != 0) in dtype.
int zen_norm_bwd_ex(const void* dy, const void* h, const void* w, const float* rstd, const float* mean, const void* dres,
                    void* dh, float* part_dw, float* part_db, void* dw, void* db, int rows, int cols, int layer,
                    int unit_offset, int accumulate, int dtype, int skip_reduce, void* stream);

int zen_norm_bwd(const void* dy, const void* h, const void* w, const float* rstd, const float* mean, const void* dres,
                 void* dh, float* part_dw, float* part_db, void* dw, void* db, int rows, int cols, int layer,
                 int unit_offset, int accumulate, int dtype, void* stream) {
  return zen_norm_bwd_ex(dy, h, w, rstd, mean, dres, dh, part_dw, part_db, dw, db, rows, cols, layer, unit_offset, accumulate,
                         dtype, 0, stream);
}

int zen_colsum_partial(const void* x, float* part, int rows, int cols, int dtype, void* stream);
int zen_norm_bwd_sums(const void* dy, const void* h, const void* w, const float* rstd, const float* mean, const void* dres,
                      void* dh, float* part_dw, float* part_db, float* part_dh, void* dw, void* db, int rows, int cols, int layer,
                      int unit_offset, int accumulate, int dtype, int skip_reduce, void* stream);

int zen_norm_bwd_ex(const void* dy, const void* h, const void* w, const float* rstd, const float* mean, const void* dres,
                    void* dh, float* part_dw, float* part_db, void* dw, void* db, int rows, int cols, int layer,
                    int unit_offset, int accumulate, int dtype, int skip_reduce, void* stream) {
  return zen_norm_bwd_sums(dy, h, w, rstd, mean, dres, dh, part_dw, part_db, nullptr, dw, db, rows, cols, layer, unit_offset, accumulate, dtype,
                           skip_reduce, stream);
}

int zen_norm_error() {
  int v = 0, zero = 0;
  if (cudaMemcpyFromSymbol(&v, g_norm_error, sizeof(int)) != cudaSuccess) return -1;
  if (v) cudaMemcpyToSymbol(g_norm_error, &zero, sizeof(int));
  return v;
}

// Partial rows that zen_norm_bwd_ex leaves in part_dw / part_db for a matrix of this shape.
int zen_norm_bwd_parts_used(int rows, int cols) { (void)cols; const int rpc = colsum_rpc(rows); return (rows + rpc - 1) / rpc; }

// skip_reduce != 0: leave the partial sums in part_dw / part_db (zen_norm_bwd_parts_used(rows, cols) rows of cols floats)
// for a later zen_colreduce_multi; dw / db are not touched.
// part_dh (may be null): column sums of dh, as many partial rows.
int zen_norm_bwd_sums(const void* dy, const void* h, const void* w, const float* rstd, const float* mean, const void* dres,
                      void* dh, float* part_dw, float* part_db, float* part_dh, void* dw, void* db, int rows, int cols, int layer,
                      int unit_offset, int accumulate, int dtype, int skip_reduce, void* stream) {
  if (cols % 8 || cols > NORM_THREADS * NORM_MAXV * 8) return -2;
  cudaStream_t st = (cudaStream_t)stream;
  const uintptr_t ptrs = reinterpret_cast<uintptr_t>(dy) | reinterpret_cast<uintptr_t>(h) | reinterpret_cast<uintptr_t>(dres) |
                         reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(dh);
  if (ptrs % 16) return -3;                             // as in the forward
  // One pass up to NF_COLS columns of a 16-bit type (wider rows leave the sums of a thread's columns no registers: 4096 x 5120 90 us as
  // two kernels, 102 as one).
  if (dtype != ZEN_DTYPE_F32 && cols <= NF_COLS) {
    const int chunk = colsum_rpc(rows), parts = (rows + chunk - 1) / chunk;
    // rows to a stage: three stages in 108 KB, so that two CTAs fit an SM (8 x 1024 rows of 2048 columns take 56 us with one CTA to an SM,
    // 46 with two), and three vectors of a row to a lane
#define NORM_FUSED(L_, RS_)                                                                                                             \
  do {                                                                                                                                  \
    const size_t smem = (size_t)NF_STAGES * 3 * RS_ * cols * 2;                                                                         \
    static const int rc = (int)cudaFuncSetAttribute(norm_bwd_fused_kernel<T, L_, RS_>, cudaFuncAttributeMaxDynamicSharedMemorySize,     \
                                                    NF_STAGES * 3 * 2 * NF_COLS * 2);                                                          \
    if (rc) return rc;                                                                                                                  \
    zen_pdl::launch_small(norm_bwd_fused_kernel<T, L_, RS_>, parts, 256, smem, st, (const T*)dy, (const T*)h, (const T*)w, rstd, mean,  \
                          (const T*)dres, (T*)dh, part_dw, part_db, part_dh, rows, cols, chunk, unit_offset);                           \
  } while (0)
#define NORM_FUSED_RS(L_)                                                                                        \
  do {                                                                                                           \
    if (cols <= 768) NORM_FUSED(L_, 8);                                                                          \
    else if (cols <= 1536) NORM_FUSED(L_, 4);                                                                    \
    else NORM_FUSED(L_, 2);                                                                                      \
  } while (0)
    const auto run = [&](auto zero) -> int {
      typedef decltype(zero) T;
      if (layer) NORM_FUSED_RS(true); else NORM_FUSED_RS(false);
      if (skip_reduce) {}
      else if (layer && db) zen_pdl::launch_small(colreduce_kernel<T>, dim3((cols + 31) / 32, 2), 1024, 0, st, part_dw, (T*)dw, parts, cols, accumulate, part_db, (T*)db);
      else zen_pdl::launch_small(colreduce_kernel<T>, (cols + 31) / 32, 1024, 0, st, part_dw, (T*)dw, parts, cols, accumulate, (const float*)nullptr, (T*)nullptr);
      return (int)cudaGetLastError();
    };
#undef NORM_FUSED_RS
#undef NORM_FUSED
    return dtype == ZEN_DTYPE_BF16 ? run(__nv_bfloat16()) : run(__half());
  }
  if (part_dh) {
    const int rc = zen_norm_bwd_sums(dy, h, w, rstd, mean, dres, dh, part_dw, part_db, nullptr, dw, db, rows, cols, layer, unit_offset, accumulate, dtype,
                                     skip_reduce, stream);
    return rc ? rc : zen_colsum_partial(dh, part_dh, rows, cols, dtype, stream);
  }
  const int grid = cap_grid((size_t)rows, 2);
  if (norm_warp_path(cols, dtype)) {
    // dh by warp-per-row (light on registers, many rows in flight), then dw / db by a column-sum pass
    const int g1 = cap_grid((size_t)(rows + NORMW_WARPS - 1) / NORMW_WARPS, 8);
    const int rpc = colsum_rpc(rows), parts = (rows + rpc - 1) / rpc;
    DISPATCH_T(dtype, {
      NORMW_NV_DISPATCH(cols, {
        if (layer) zen_pdl::launch_small(norm_bwd_warp_kernel<T, true, NV, false>, g1, NORMW_WARPS * 32, 0, st, (const T*)dy, (const T*)h, (const T*)w, rstd, mean, (const T*)dres, (T*)dh, part_dw, part_db, rows, cols, unit_offset);
        else zen_pdl::launch_small(norm_bwd_warp_kernel<T, false, NV, false>, g1, NORMW_WARPS * 32, 0, st, (const T*)dy, (const T*)h, (const T*)w, rstd, mean, (const T*)dres, (T*)dh, part_dw, part_db, rows, cols, unit_offset);
      });
      if (layer) zen_pdl::launch_small(norm_dwdb_partial_kernel<T, true>, dim3(parts, (cols + 2047) / 2048), 256, 0, st, (const T*)dy, (const T*)h, rstd, mean, part_dw, part_db, rows, cols, rpc);
      else zen_pdl::launch_small(norm_dwdb_partial_kernel<T, false>, dim3(parts, (cols + 2047) / 2048), 256, 0, st, (const T*)dy, (const T*)h, rstd, mean, part_dw, part_db, rows, cols, rpc);
      if (skip_reduce) {}
      else if (layer && db) zen_pdl::launch_small(colreduce_kernel<T>, dim3((cols + 31) / 32, 2), 1024, 0, st, part_dw, (T*)dw, parts, cols, accumulate, part_db, (T*)db);
      else zen_pdl::launch_small(colreduce_kernel<T>, (cols + 31) / 32, 1024, 0, st, part_dw, (T*)dw, parts, cols, accumulate, (const float*)nullptr, (T*)nullptr);
    });
    return (int)cudaGetLastError();
  }
  (void)grid;
  // wide rows: dh by one CTA per row (no parameter accumulators, so several CTAs fit an SM), then dw / db by the
  // column-sum pass, as on the warp path
  const int g2 = cap_grid((size_t)rows, 6);
  const int rpc = colsum_rpc(rows);
  const int parts = (rows + rpc - 1) / rpc;
  DISPATCH_T(dtype, {
    NORM_NV_DISPATCH(cols, {
      if (layer) zen_pdl::launch_small(norm_bwd_kernel<T, true, NV, false>, g2, NORM_THREADS, 0, st, (const T*)dy, (const T*)h, (const T*)w, rstd, mean, (const T*)dres, (T*)dh, part_dw, part_db, rows, cols, unit_offset);
      else zen_pdl::launch_small(norm_bwd_kernel<T, false, NV, false>, g2, NORM_THREADS, 0, st, (const T*)dy, (const T*)h, (const T*)w, rstd, mean, (const T*)dres, (T*)dh, part_dw, part_db, rows, cols, unit_offset);
    });
    if (layer) zen_pdl::launch_small(norm_dwdb_partial_kernel<T, true>, dim3(parts, (cols + 2047) / 2048), 256, 0, st, (const T*)dy, (const T*)h, rstd, mean, part_dw, part_db, rows, cols, rpc);
    else zen_pdl::launch_small(norm_dwdb_partial_kernel<T, false>, dim3(parts, (cols + 2047) / 2048), 256, 0, st, (const T*)dy, (const T*)h, rstd, mean, part_dw, part_db, rows, cols, rpc);
    if (skip_reduce) {}
    else if (layer && db) zen_pdl::launch_small(colreduce_kernel<T>, dim3((cols + 31) / 32, 2), 1024, 0, st, part_dw, (T*)dw, parts, cols, accumulate, part_db, (T*)db);
    else zen_pdl::launch_small(colreduce_kernel<T>, (cols + 31) / 32, 1024, 0, st, part_dw, (T*)dw, parts, cols, accumulate, (const float*)nullptr, (T*)nullptr);
  });
  return (int)cudaGetLastError();
}

int zen_colsum_parts(int rows) { const int rpc = colsum_rpc(rows); return (rows + rpc - 1) / rpc; }

// out[c] (+)= sum_r a[r][c]; part: fp32 scratch zen_colsum_parts(rows) * cols.
int zen_colsum(const void* a, float* part, void* out, int rows, int cols, int accumulate, int dtype, void* stream) {
  if (cols % 8) return -2;
  cudaStream_t st = (cudaStream_t)stream;
  const int parts = zen_colsum_parts(rows);
  DISPATCH_T(dtype, {
    zen_pdl::launch_small(colsum_partial_kernel<T>, parts, 256, 0, st, (const T*)a, part, rows, cols, colsum_rpc(rows));
    zen_pdl::launch_small(colreduce_kernel<T>, (cols + 31) / 32, 1024, 0, st, part, (T*)out, parts, cols, accumulate, (const float*)nullptr, (T*)nullptr);
  });
  return (int)cudaGetLastError();
}

// Rows of one launch: the kernels count vectors in 32 bits.
static int act_rows(int inner) { return (int)(((size_t)1 << 31) / (inner / 8)) - 1; }
// Two CTAs per SM at most, and small outputs spread over all SMs.
static int act_grid(size_t nvec, int u) { return cap_grid((nvec + (size_t)ACT_THREADS * u - 1) / ((size_t)ACT_THREADS * u), 2); }

int zen_act_fwd(const void* a, const void* b, void* out, int rows, int inner, int lda, int ldb, int mode, int dtype,
                void* stream) {
  if (inner % 8 || lda % 8 || ldb % 8) return -2;
  if (rows <= 0 || inner <= 0) return 0;
  const int step = act_rows(inner);
  for (int r0 = 0; r0 < rows; r0 += step) {
    const int n = rows - r0 < step ? rows - r0 : step, grid = act_grid((size_t)n * (inner / 8), ACT_U);
#define ACT_FWD(M_)                                                                                                              \
  zen_pdl::launch_small(act_fwd_kernel<T, M_>, grid, ACT_THREADS, 0, (cudaStream_t)stream, (const T*)a + (size_t)r0 * lda,     \
                        b ? (const T*)b + (size_t)r0 * ldb : nullptr, (T*)out + (size_t)r0 * inner, n, inner, lda, ldb)
    DISPATCH_T(dtype, if (mode == 0) ACT_FWD(0); else if (mode == 1) ACT_FWD(1); else if (mode == 2) ACT_FWD(2); else ACT_FWD(3));
#undef ACT_FWD
  }
  return (int)cudaGetLastError();
}

int zen_act_bwd(const void* a, const void* b, const void* dout, void* da, void* db, int rows, int inner, int lda,
                int ldb, int mode, int dtype, void* stream) {
  if (inner % 8 || lda % 8 || ldb % 8) return -2;
  if (rows <= 0 || inner <= 0) return 0;
  const int step = act_rows(inner);
  for (int r0 = 0; r0 < rows; r0 += step) {
    const int n = rows - r0 < step ? rows - r0 : step, grid = act_grid((size_t)n * (inner / 8), 2);
#define ACT_BWD(M_)                                                                                                              \
  zen_pdl::launch_small(act_bwd_kernel<T, M_>, grid, ACT_THREADS, 0, (cudaStream_t)stream, (const T*)a + (size_t)r0 * lda,     \
                        b ? (const T*)b + (size_t)r0 * ldb : nullptr, (const T*)dout + (size_t)r0 * inner, (T*)da + (size_t)r0 * lda, \
                        db ? (T*)db + (size_t)r0 * ldb : nullptr, n, inner, lda, ldb)
    DISPATCH_T(dtype, if (mode == 0) ACT_BWD(0); else if (mode == 1) ACT_BWD(1); else if (mode == 2) ACT_BWD(2); else ACT_BWD(3));
#undef ACT_BWD
  }
  return (int)cudaGetLastError();
}

// Rows per CTA of zen_act_bwd_colsum: three CTAs per SM, all resident at once and evenly loaded.
static int act_colsum_rows_per_cta(int rows) {
  const int target = sm_count_e() * 3;
  const int rpc = (rows + target - 1) / target;
  return rpc < 1 ? 1 : rpc;
}
int zen_act_colsum_parts(int rows) { const int rpc = act_colsum_rows_per_cta(rows); return (rows + rpc - 1) / rpc; }

// Ungated activation backward (mode 0 gelu_tanh, 1 relu) on dense [rows, inner] tensors that also writes the partial
// column sums of da: part[zen_act_colsum_parts(rows)][inner] floats, to be summed by zen_colsum_reduce.
int zen_act_bwd_colsum(const void* a, const void* dout, void* da, float* part, int rows, int inner, int mode, int dtype,
                       void* stream) {
  if (inner % 8 || mode < 0 || mode > 1) return -2;
  if (rows <= 0) return 0;
  int threads = ((inner / 8 + 31) / 32) * 32;
  if (threads > 512) threads = 512;
  const int rpc = act_colsum_rows_per_cta(rows);
  DISPATCH_T(dtype, zen_pdl::launch_small(act_bwd_colsum_kernel<T>, (rows + rpc - 1) / rpc, threads, 0, (cudaStream_t)stream, (const T*)a, (const T*)dout, (T*)da, part, rows, inner, mode, rpc));
  return (int)cudaGetLastError();
}

// First half of zen_colsum only: part[zen_colsum_parts(rows)][cols] partial column sums of a.
int zen_colsum_partial(const void* a, float* part, int rows, int cols, int dtype, void* stream) {
  if (cols % 8) return -2;
  DISPATCH_T(dtype, zen_pdl::launch_small(colsum_partial_kernel<T>, zen_colsum_parts(rows), 256, 0, (cudaStream_t)stream, (const T*)a, part, rows, cols, colsum_rpc(rows)));
  return (int)cudaGetLastError();
}

// Up to COLREDUCE_MAX_JOBS reductions out[c] (+)= sum_p part[p][c] in ONE launch; a job may carry a second (part2, out2)
// pair of the same shape.  All outputs have type `dtype`.
int zen_colreduce_job_size() { return (int)sizeof(ColReduceJob); }
int zen_colreduce_max_jobs() { return COLREDUCE_MAX_JOBS; }
int zen_colreduce_multi(const void* jobs_, int n, int dtype, void* stream) {
  const ColReduceJob* jobs = static_cast<const ColReduceJob*>(jobs_);      // records of zen_colreduce_job_size() bytes
  if (!jobs || n < 1 || n > COLREDUCE_MAX_JOBS) return -2;
  ColReduceJobs t;
  int max_cols = 0;
  for (int i = 0; i < n; ++i) {
    t.j[i] = jobs[i];
    if (jobs[i].nparts <= 0 || jobs[i].cols <= 0 || !jobs[i].part || !jobs[i].out) return -2;
    if (jobs[i].cols > max_cols) max_cols = jobs[i].cols;
  }
  for (int i = n; i < COLREDUCE_MAX_JOBS; ++i) t.j[i] = ColReduceJob{nullptr, nullptr, nullptr, nullptr, 0, 0, 0, 0};
  t.n = n;
  DISPATCH_T(dtype, zen_pdl::launch_small(colreduce_multi_kernel<T>, dim3((max_cols + 31) / 32, 2 * n), 1024, 0, (cudaStream_t)stream, t));
  return (int)cudaGetLastError();
}

// out[c] (+)= sum over p of part[p][c]: the second half of zen_colsum for partial sums that another kernel produced.
int zen_colsum_reduce(const float* part, void* out, int parts, int cols, int accumulate, int dtype, void* stream) {
  if (parts <= 0 || cols <= 0) return -2;
  DISPATCH_T(dtype, zen_pdl::launch_small(colreduce_kernel<T>, (cols + 31) / 32, 1024, 0, (cudaStream_t)stream, part, (T*)out, parts, cols, accumulate, (const float*)nullptr, (T*)nullptr));
  return (int)cudaGetLastError();
}

int zen_rope(void* x, int tokens, int heads, int hd, int ld, int seq, int pos0, float theta, int inverse, int dtype,
             void* stream) {
  if (hd % 2) return -2;
  const size_t n = (size_t)tokens * heads * (hd / 2);
  const int grid = cap_grid((n + 255) / 256, 16);
  if ((hd / 2) % 8 == 0 && (ld % 8) == 0 && (reinterpret_cast<uintptr_t>(x) % 16) == 0) {
    int hgroups = 1;
    while (hgroups < heads && (size_t)tokens * (hd / 16) * hgroups < (size_t)sm_count_e() * 1024) hgroups *= 2;
    if (hgroups > heads) hgroups = heads;
    const size_t nvec = (size_t)tokens * (hd / 16) * hgroups;
    const int gv = cap_grid((nvec + 255) / 256, 16);
    DISPATCH_T(dtype, zen_pdl::launch_small(rope_vec_kernel<T>, gv, 256, 0, (cudaStream_t)stream, (T*)x, tokens, heads, hd, ld, seq, pos0, log2f(theta), inverse ? -1.f : 1.f, hgroups));
    return (int)cudaGetLastError();
  }
  DISPATCH_T(dtype, zen_pdl::launch_small(rope_kernel<T>, grid, 256, 0, (cudaStream_t)stream, (T*)x, tokens, heads, hd, ld, seq, pos0, log2f(theta), inverse ? -1.f : 1.f));
  return (int)cudaGetLastError();
}

int zen_embedding_fwd(const int64_t* ids, const void* wte, const void* wpe, void* out, int tokens, int d, int seq,
                      int pos_offset, float scale, int vocab, int dtype, void* stream) {
  if (d % 8) return -2;
  DISPATCH_T(dtype, zen_pdl::launch_small(embedding_fwd_kernel<T>, cap_grid((size_t)tokens, 32), 128, 0, (cudaStream_t)stream, ids, (const T*)wte, (const T*)wpe, (T*)out, tokens, d, seq, pos_offset, scale, vocab));
  return (int)cudaGetLastError();
}

// Row-sparse gradient of an embedding lookup.  flag: int32 scratch of zen_embedding_flag_words(vocab) words, zero on entry (the
// call leaves its first half zero again); acc fp32[max_rows][d], zero on entry and exit.  Outputs: rows int32[max_rows]
// (ascending unique ids), count int32[1], vals T[max_rows][d].  max_rows >= min(tokens, vocab).
int zen_embedding_flag_words(int vocab) { return 2 * ((vocab + 31) / 32); }
int zen_embedding_bwd_rows(const int64_t* ids, const void* dy, int32_t* flag, float* acc, int32_t* rows,
                           int32_t* count, void* vals, int tokens, int d, int vocab, float scale, int dtype,
                           void* stream) {
  if (d % 8) return -2;
  cudaStream_t st = (cudaStream_t)stream;
  const int words = (vocab + 31) / 32;
  uint32_t *bits = reinterpret_cast<uint32_t*>(flag), *prefix = bits + words;
  zen_pdl::launch_small(embed_mark_kernel, cap_grid(((size_t)tokens + 255) / 256, 8), 256, 0, st, ids, bits, tokens, vocab);
  zen_pdl::launch_small(embed_compact_kernel, 1, 1024, 0, st, bits, prefix, rows, count, words);
  DISPATCH_T(dtype, {
    zen_pdl::launch_small(embed_accum_kernel<T>, cap_grid((size_t)tokens, 32), 128, 0, st, ids, bits, prefix, (const T*)dy, acc, tokens, d, vocab, scale);
    zen_pdl::launch_small(embed_finish_kernel<T>, cap_grid((size_t)(tokens < vocab ? tokens : vocab), 32), 128, 0, st, acc, bits, words, count, (T*)vals, d);
  });
  return (int)cudaGetLastError();
}

// Gradient of learned position embeddings (see pos_grad_kernel); out: the first of the S rows that were added.
int zen_pos_grad(const void* dy, void* out, int B, int S, int d, int accumulate, int dtype, void* stream) {
  if (d % 8) return -2;
  DISPATCH_T(dtype, zen_pdl::launch_small(pos_grad_kernel<T>, cap_grid(((size_t)S * (d / 8) + 255) / 256, 8), 256, 0, (cudaStream_t)stream, (const T*)dy, (T*)out, B, S, d, accumulate));
  return (int)cudaGetLastError();
}

// Labels moved `shift` positions to the left within each sequence (lab may be null: only counted) and 1 / (labels that count).
int zen_label_prep(const int64_t* labels, int64_t* lab, float* inv, int B, int S, int shift, int64_t ignore, void* stream) {
  zen_pdl::launch_small(label_prep_kernel, 1, 1024, 0, (cudaStream_t)stream, labels, lab, inv, B, S, shift, ignore);
  return (int)cudaGetLastError();
}
int zen_sum_scale(const float* x, int n, const float* scale, float* out, void* stream) {
  zen_pdl::launch_small(sum_scale_kernel, 1, 1024, 0, (cudaStream_t)stream, x, n, scale, out);
  return (int)cudaGetLastError();
}
int zen_softcap(const void* x, float* out, int rows, int cols, int ld, float cap, int dtype, void* stream) {
  DISPATCH_T(dtype, zen_pdl::launch_small(softcap_kernel<T>, cap_grid(((size_t)rows * cols + 1023) / 1024, 16), 256, 0, (cudaStream_t)stream, (const T*)x, out, rows, cols, ld, cap));
  return (int)cudaGetLastError();
}

int zen_rows_add(void* grad, const int32_t* rows, const int32_t* count, const void* vals, int d, int vocab,
                 int max_rows, int dtype, void* stream) {
  if (d % 8) return -2;
  DISPATCH_T(dtype, zen_pdl::launch_small(rows_add_kernel<T>, cap_grid((size_t)max_rows, 32), 128, 0, (cudaStream_t)stream, (T*)grad, rows, count, (const T*)vals, d, vocab, max_rows));
  return (int)cudaGetLastError();
}

// gscale_dev (optional device float) multiplies gscale; lets the caller scale by 1 / (valid tokens) without a host sync.
// softcap > 0: the logits are soft-capped (see xent_kernel), which the gradient takes into account.
int zen_xent(const void* logits, const int64_t* labels, float* loss, void* dlogits, int rows, int vocab, int ld,
             float gscale, const float* gscale_dev, int64_t ignore_index, int dtype, float softcap, void* stream) {
  // two rows of 512 threads per SM while the rows of all SMs stay within 96 MB of the L2, else one row of 1024 threads
  const size_t row_bytes = (size_t)ld * (dtype == ZEN_DTYPE_F32 ? 4 : 2);
  const bool two = row_bytes * 2 * sm_count_e() <= ((size_t)96 << 20);
  const int grid = cap_grid((size_t)rows, two ? 2 : 1);
  cudaStream_t st = (cudaStream_t)stream;
#define XENT(CAP_, TH_) zen_pdl::launch_small(xent_kernel<T, CAP_, TH_>, grid, TH_, 0, st, (const T*)logits, labels, loss, (T*)dlogits, rows, vocab, ld, gscale, gscale_dev, ignore_index, softcap)
  DISPATCH_T(dtype, {
    if (softcap > 0.f) { if (two) XENT(true, 512); else XENT(true, 1024); }
    else { if (two) XENT(false, 512); else XENT(false, 1024); }
  });
#undef XENT
  return (int)cudaGetLastError();
}

// Loss and log-sum-exp of rows from their 128-column pieces; part: [nparts][part_ld] (maximum, sum of exponentials).
int zen_xent_finish(const void* part, int nparts, int part_ld, const float* target, const int64_t* labels, float* loss, float* lse, int rows,
                    int vocab, int64_t ignore_index, float softcap, void* stream) {
  const int grid = (rows + XF_ROWS - 1) / XF_ROWS;
  cudaStream_t st = (cudaStream_t)stream;
  if (softcap > 0.f) zen_pdl::launch_small(xent_finish_kernel<true>, grid, XF_ROWS * XF_G, 0, st, (const float2*)part, nparts, part_ld, target, labels, loss, lse, rows, vocab, ignore_index, softcap);
  else zen_pdl::launch_small(xent_finish_kernel<false>, grid, XF_ROWS * XF_G, 0, st, (const float2*)part, nparts, part_ld, target, labels, loss, lse, rows, vocab, ignore_index, softcap);
  return (int)cudaGetLastError();
}
// In place: bf16 logits <- (softmax - onehot) * gscale (* *gscale_dev), from each row's log-sum-exp.
int zen_xent_grad(void* logits, const int64_t* labels, const float* lse, int rows, int vocab, int ld, float gscale, const float* gscale_dev,
                  int64_t ignore_index, float softcap, void* stream) {
  if (ld % 8 || reinterpret_cast<uintptr_t>(logits) % 16) return -2;
  const int grid = cap_grid((size_t)rows, 8);
  cudaStream_t st = (cudaStream_t)stream;
  if (softcap > 0.f) zen_pdl::launch_small(xent_grad_kernel<true>, grid, 256, 0, st, (__nv_bfloat16*)logits, labels, lse, rows, vocab, ld, gscale, gscale_dev, ignore_index, softcap);
  else zen_pdl::launch_small(xent_grad_kernel<false>, grid, 256, 0, st, (__nv_bfloat16*)logits, labels, lse, rows, vocab, ld, gscale, gscale_dev, ignore_index, softcap);
  return (int)cudaGetLastError();
}

int zen_xent_partial(const void* logits, const int64_t* labels, float* rowmax, float* sumexp, float* target, int rows,
                     int valid_cols, int ld, int64_t vocab_start, int64_t ignore_index, int dtype, void* stream) {
  DISPATCH_T(dtype, zen_pdl::launch_small(xent_partial_kernel<T>, cap_grid((size_t)rows, 8), 512, 0, (cudaStream_t)stream, (const T*)logits, labels, rowmax, sumexp, target, rows, valid_cols, ld, vocab_start, ignore_index));
  return (int)cudaGetLastError();
}

int zen_xent_apply(void* logits, const int64_t* labels, const float* lse, int rows, int cols, int valid_cols, int ld,
                   float gscale, const float* gscale_dev, int64_t vocab_start, int64_t ignore_index, int dtype, void* stream) {
  DISPATCH_T(dtype, zen_pdl::launch_small(xent_apply_kernel<T>, cap_grid((size_t)rows, 8), 512, 0, (cudaStream_t)stream, (T*)logits, labels, lse, rows, cols, valid_cols, ld, gscale, gscale_dev, vocab_start, ignore_index));
  return (int)cudaGetLastError();
}

int zen_adam_tensor_size() { return (int)sizeof(AdamTensor); }

// step_dev (optional): device int32 holding the 1-based step count; when given, bc1 / bc2 are ignored and computed
// from it inside the kernel, so that a captured launch stays correct across replays.
int zen_adamw(const void* table, int ntensors, const int32_t* chunk_tensor, uint64_t nchunks, float lr, float b1,
              float b2, float eps, float bc1, float bc2, float gscale, const int32_t* step_dev, int dtype, void* stream) {
  const int grid = cap_grid((size_t)nchunks, 8);
  DISPATCH_T(dtype, zen_pdl::launch_small(adamw_kernel<T>, grid, 256, 0, (cudaStream_t)stream, (const AdamTensor*)table, ntensors, chunk_tensor, nchunks, lr, b1, b2, eps, bc1, bc2, gscale, step_dev));
  return (int)cudaGetLastError();
}

}  // extern "C"

// ------------------------------------------------------------------------------------------------
// Allocation-free column sum (declared in zen_noalloc.h, which says who needs it and why).
#include "zen_noalloc.h"

#include <mutex>
#include <stdio.h>

// Scratch of the allocation-free entry point: per-CTA partial sums, [ceil(rows / 32)][cols] floats.
// In host code this name is only a handle for cudaGetSymbolAddress, never a pointer to hand to a kernel.
static __device__ __align__(256) float g_colsum_noalloc_scratch[ZEN_COLSUM_NOALLOC_MAX_FLOATS];

namespace {
constexpr int kMaxDevices = 64;
float* g_noalloc_ptr[kMaxDevices] = {nullptr};   // device address of the scratch, per device
std::mutex g_noalloc_mu;
thread_local char g_noalloc_err[256] = "";

int noalloc_fail(int code, const char* what) {
  snprintf(g_noalloc_err, sizeof(g_noalloc_err), "%s", what);
  return code;
}

// Device address of the scratch array on the current device; looked up once per device.
int noalloc_scratch(float** out) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return noalloc_fail((int)e, cudaGetErrorString(e));
  if (dev < 0 || dev >= kMaxDevices) return noalloc_fail(ZEN_NOALLOC_BAD_ARG, "device index out of range");
  std::lock_guard<std::mutex> g(g_noalloc_mu);
  if (!g_noalloc_ptr[dev]) {
    float* p = nullptr;
    e = cudaGetSymbolAddress((void**)&p, g_colsum_noalloc_scratch);
    if (e != cudaSuccess) return noalloc_fail((int)e, cudaGetErrorString(e));
    g_noalloc_ptr[dev] = p;
  }
  *out = g_noalloc_ptr[dev];
  return 0;
}
}  // namespace

extern "C" {

const char* zen_noalloc_last_error(void) { return g_noalloc_err; }

int zen_colsum_noalloc(const void* a, void* out, int rows, int cols, int accumulate, int dtype, void* stream) {
  if (!a || !out || rows <= 0 || cols <= 0) return noalloc_fail(ZEN_NOALLOC_BAD_ARG, "null pointer or empty matrix");
  if (cols % 8) return noalloc_fail(ZEN_NOALLOC_BAD_ARG, "cols must be a multiple of 8");
  if (reinterpret_cast<uintptr_t>(a) % 16) return noalloc_fail(ZEN_NOALLOC_BAD_ARG, "input must be 16-byte aligned");
  if (dtype < 0 || dtype > 2) return noalloc_fail(ZEN_NOALLOC_BAD_ARG, "dtype must be 0 (fp32), 1 (bf16) or 2 (fp16)");
  constexpr int RPC = 32;                                     // bounds the scratch; zen_colsum takes fewer rows for few rows
  const int parts = (rows + RPC - 1) / RPC;
  if ((uint64_t)parts * (uint64_t)cols > (uint64_t)ZEN_COLSUM_NOALLOC_MAX_FLOATS) {
    snprintf(g_noalloc_err, sizeof(g_noalloc_err),
             "scratch of %llu floats needed for %d x %d, the built-in array holds %u: use zen_colsum with caller scratch",
             (unsigned long long)parts * cols, rows, cols, (unsigned)ZEN_COLSUM_NOALLOC_MAX_FLOATS);
    return ZEN_NOALLOC_TOO_LARGE;
  }
  float* part = nullptr;
  int rc = noalloc_scratch(&part);
  if (rc) return rc;
  cudaStream_t st = (cudaStream_t)stream;
  DISPATCH_T(dtype, {
    zen_pdl::plain(colsum_partial_kernel<T>, parts, 256, 0, st, (const T*)a, part, rows, cols, RPC);
    zen_pdl::plain(colreduce_kernel<T>, (cols + 31) / 32, 1024, 0, st, part, (T*)out, parts, cols, accumulate, (const float*)nullptr, (T*)nullptr);
  });
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return noalloc_fail((int)e, cudaGetErrorString(e));
  return 0;
}

}  // extern "C"
