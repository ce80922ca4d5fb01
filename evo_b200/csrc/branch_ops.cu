// Row kernels of designs whose layers run several branches side by side on norms of the same fp32 stream:
//   evo_sum_norm          x += sum of (optionally RMS-normed) branch outputs, then one or two norms of the new x
//   evo_conv_act          short causal convolution per channel on columns of a projection, with carried inputs, then SiLU
//   evo_xielu             the xIELU activation between the two feed-forward products
//   evo_gated_group_norm  y * silu(gate), RMS norm in equal parts of the row, weight
// Sums of squares, norms and the stream are fp32 whatever the activation type.
#include "common.cuh"
#include "conv_rows.h"
#include "../../include/evo_b200.h"
#include <math.h>
#include <algorithm>
#include <stdint.h>

using namespace evo;

namespace {

template <typename T> __device__ __forceinline__ float ldf(const T* p);
template <> __device__ __forceinline__ float ldf<float>(const float* p) { return *p; }
template <> __device__ __forceinline__ float ldf<bf16>(const bf16* p) { return __bfloat162float(*p); }
template <typename T> __device__ __forceinline__ void stf(T* p, float v);
template <> __device__ __forceinline__ void stf<float>(float* p, float v) { *p = v; }
template <> __device__ __forceinline__ void stf<bf16>(bf16* p, float v) { *p = __float2bfloat16_rn(v); }

__device__ __forceinline__ float silu_f(float v) { return v / (1.f + expf(-v)); }

// four consecutive elements (16 bytes of fp32, 8 of bf16) as floats, and back
template <typename T> struct Vec4;
template <> struct Vec4<float> {
  static __device__ __forceinline__ void load(const float* p, float* o) { const float4 u = *reinterpret_cast<const float4*>(p); o[0] = u.x; o[1] = u.y; o[2] = u.z; o[3] = u.w; }
  static __device__ __forceinline__ void store(float* p, const float* v) { *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]); }
};
template <> struct Vec4<bf16> {
  static __device__ __forceinline__ void load(const bf16* p, float* o) {
    const uint2 u = *reinterpret_cast<const uint2*>(p);
    o[0] = __uint_as_float(u.x << 16); o[1] = __uint_as_float(u.x & 0xffff0000u); o[2] = __uint_as_float(u.y << 16); o[3] = __uint_as_float(u.y & 0xffff0000u);
  }
  static __device__ __forceinline__ void store(bf16* p, const float* v) {
    const __nv_bfloat162 a = __floats2bfloat162_rn(v[0], v[1]), b = __floats2bfloat162_rn(v[2], v[3]);
    uint2 u; u.x = *reinterpret_cast<const uint32_t*>(&a); u.y = *reinterpret_cast<const uint32_t*>(&b);
    *reinterpret_cast<uint2*>(p) = u;
  }
};
template <typename T> inline bool aligned4(const void* p) { return ((uintptr_t)p & (4 * sizeof(T) - 1)) == 0; }

// sum over the CTA (blockDim.x a multiple of 32, at most 1024); every thread gets the result; red: 33 floats
__device__ __forceinline__ float block_sum(float v, float* red) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  __syncthreads();                       // red may still be read from the previous sum
  if (lane == 0) red[w] = v;
  __syncthreads();
  if (w == 0) {
    float t = lane < nw ? red[lane] : 0.f;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (lane == 0) red[32] = t;
  }
  __syncthreads();
  return red[32];
}

// ---- evo_sum_norm: one CTA per row; the new row of x is kept in shared memory between the passes
template <typename T, bool VEC>
__global__ void __launch_bounds__(256) sum_norm_kernel(evo_sum_norm_params p) {
  pdl_wait();
  extern __shared__ float xs[];          // [D] + 33
  float* red = xs + p.D;
  const int64_t r = blockIdx.x;
  const int64_t src = p.gather ? p.gather[r] : r;
  const int D = p.D, tid = threadIdx.x, nt = blockDim.x;
  float rstd[EVO_SUM_NORM_BRANCHES];
#pragma unroll
  for (int b = 0; b < EVO_SUM_NORM_BRANCHES; ++b) {
    rstd[b] = 1.f;
    if (b < p.n_branches && p.norm_w[b]) {
      const T* y = (const T*)p.y[b] + src * p.ldy[b];
      float ss = 0.f;
      if (VEC) {
        for (int c = tid * 4; c < D; c += nt * 4) { float v[4]; Vec4<T>::load(y + c, v); ss = fmaf(v[0], v[0], fmaf(v[1], v[1], fmaf(v[2], v[2], fmaf(v[3], v[3], ss)))); }
      } else {
        for (int c = tid; c < D; c += nt) { const float v = ldf(y + c); ss = fmaf(v, v, ss); }
      }
      rstd[b] = 1.0f / sqrtf(block_sum(ss, red) / (float)D + p.eps);
    }
  }
  float* xr = p.x + src * D;
  const bf16* cs = (const bf16*)p.col_scale;
  float ss = 0.f;
  if (VEC) {
    for (int c = tid * 4; c < D; c += nt * 4) {
      float v[4], add[4] = {0.f, 0.f, 0.f, 0.f}, cw[4];
      Vec4<float>::load(xr + c, v);
      if (cs) Vec4<bf16>::load(cs + c, cw);
#pragma unroll
      for (int b = 0; b < EVO_SUM_NORM_BRANCHES; ++b) {
        if (b < p.n_branches) {
          float y[4];
          Vec4<T>::load((const T*)p.y[b] + src * p.ldy[b] + c, y);
          if (p.norm_w[b]) {
            float w[4];
            Vec4<bf16>::load((const bf16*)p.norm_w[b] + c, w);
#pragma unroll
            for (int u = 0; u < 4; ++u) y[u] = y[u] * rstd[b] * w[u];
          }
#pragma unroll
          for (int u = 0; u < 4; ++u) add[u] = fmaf(p.scale[b], y[u], add[u]);
        }
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) { v[u] = cs ? fmaf(cw[u], add[u], v[u]) : v[u] + add[u]; ss = fmaf(v[u], v[u], ss); }
      Vec4<float>::store(xs + c, v);
      if (p.n_branches > 0 && !p.gather) Vec4<float>::store(xr + c, v);
    }
  } else
  for (int c = tid; c < D; c += nt) {
    float v = xr[c];
    float add = 0.f;
#pragma unroll
    for (int b = 0; b < EVO_SUM_NORM_BRANCHES; ++b) {
      if (b < p.n_branches) {
        float y = ldf((const T*)p.y[b] + src * p.ldy[b] + c);
        if (p.norm_w[b]) y = y * rstd[b] * __bfloat162float(((const bf16*)p.norm_w[b])[c]);
        add = fmaf(p.scale[b], y, add);
      }
    }
    v = cs ? fmaf(__bfloat162float(cs[c]), add, v) : v + add;
    xs[c] = v;
    if (p.n_branches > 0 && !p.gather) xr[c] = v;
    ss = fmaf(v, v, ss);
  }
  if (!p.out[0] && !p.out[1]) return;
  const float rs = 1.0f / sqrtf(block_sum(ss, red) / (float)D + p.eps);
#pragma unroll
  for (int n = 0; n < 2; ++n) {
    if (!p.out[n]) continue;
    T* o = (T*)p.out[n] + r * p.ldo;
    const bf16* w = (const bf16*)p.w[n];
    if (VEC) {
      for (int c = tid * 4; c < p.ldo; c += nt * 4) {
        float v[4] = {0.f, 0.f, 0.f, 0.f};
        if (c < D) {                     // D % 4 == 0: a group of four lies inside the row or in the padding
          float wv[4];
          Vec4<bf16>::load(w + c, wv);
#pragma unroll
          for (int u = 0; u < 4; ++u) v[u] = xs[c + u] * rs * wv[u];
        }
        Vec4<T>::store(o + c, v);
      }
    } else
    for (int c = tid; c < p.ldo; c += nt) stf(o + c, c < D ? xs[c] * rs * __bfloat162float(w[c]) : 0.f);
  }
}

// The same for rows of up to 1024 NV elements that can be read four at a time: the row stays in registers (NV groups of four per thread), all loads of a
// pass are issued together, and a sum over the CTA costs one barrier.  One CTA per row, 256 threads.  8190 x 4096, two bf16 branches, two norms: 87 us = 6.2 TB/s (116 through
// shared memory; 112 with the branches unpacked, whose registers left three rows per SM instead of four).
__device__ __forceinline__ float cta_sum(float v, float* red) {          // red: 8 floats of this sum's own
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  const float4 a = reinterpret_cast<const float4*>(red)[0], b = reinterpret_cast<const float4*>(red)[1];
  return ((a.x + a.y) + (a.z + a.w)) + ((b.x + b.y) + (b.z + b.w));
}

// four elements as they lie in memory
template <typename T> struct Raw4;
template <> struct Raw4<float> {
  float4 v;
  __device__ __forceinline__ void load(const float* p) { v = *reinterpret_cast<const float4*>(p); }
  __device__ __forceinline__ void get(float* o) const { o[0] = v.x; o[1] = v.y; o[2] = v.z; o[3] = v.w; }
  __device__ __forceinline__ void clear() { v = make_float4(0.f, 0.f, 0.f, 0.f); }
};
template <> struct Raw4<bf16> {
  uint2 v;
  __device__ __forceinline__ void load(const bf16* p) { v = *reinterpret_cast<const uint2*>(p); }
  __device__ __forceinline__ void get(float* o) const { o[0] = bf_lo(v.x); o[1] = bf_hi(v.x); o[2] = bf_lo(v.y); o[3] = bf_hi(v.y); }
  __device__ __forceinline__ void clear() { v = make_uint2(0u, 0u); }
};

template <typename T, int NV, int NB>
__global__ void __launch_bounds__(256) sum_norm_row_kernel(const evo_sum_norm_params p) {
  pdl_wait();
  __shared__ __align__(16) float red[4][8];
  const int64_t r = blockIdx.x;
  const int64_t src = p.gather ? p.gather[r] : r;
  const int D = p.D, c0 = threadIdx.x * 4;
  float* xr = p.x + src * D;
  float v[NV][4];
  Raw4<T> y[NB > 0 ? NB : 1][NV];                         // packed: more rows fit an SM
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int c = c0 + i * 1024;
    if (c < D) {
      Vec4<float>::load(xr + c, v[i]);
#pragma unroll
      for (int b = 0; b < NB; ++b) y[b][i].load((const T*)p.y[b] + src * p.ldy[b] + c);
    } else {
      v[i][0] = v[i][1] = v[i][2] = v[i][3] = 0.f;
#pragma unroll
      for (int b = 0; b < NB; ++b) y[b][i].clear();
    }
  }
  float rstd[NB > 0 ? NB : 1];
#pragma unroll
  for (int b = 0; b < NB; ++b) {
    rstd[b] = 1.f;
    if (p.norm_w[b]) {
      float ss = 0.f;
#pragma unroll
      for (int i = 0; i < NV; ++i) { float q[4]; y[b][i].get(q); ss = fmaf(q[0], q[0], fmaf(q[1], q[1], fmaf(q[2], q[2], fmaf(q[3], q[3], ss)))); }
      rstd[b] = 1.0f / sqrtf(cta_sum(ss, red[b]) / (float)D + p.eps);
    }
  }
  const bf16* cs = (const bf16*)p.col_scale;
  float ss = 0.f;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int c = c0 + i * 1024;
    if (c < D) {
      float add[4] = {0.f, 0.f, 0.f, 0.f}, cw[4];
      if (cs) Vec4<bf16>::load(cs + c, cw);
#pragma unroll
      for (int b = 0; b < NB; ++b) {
        float q[4], w[4];
        y[b][i].get(q);
        if (p.norm_w[b]) {
          Vec4<bf16>::load((const bf16*)p.norm_w[b] + c, w);
#pragma unroll
          for (int u = 0; u < 4; ++u) q[u] = q[u] * rstd[b] * w[u];
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) add[u] = fmaf(p.scale[b], q[u], add[u]);
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        if (NB > 0) v[i][u] = cs ? fmaf(cw[u], add[u], v[i][u]) : v[i][u] + add[u];
        ss = fmaf(v[i][u], v[i][u], ss);
      }
      if (NB > 0 && !p.gather) Vec4<float>::store(xr + c, v[i]);
    }
  }
  if (!p.out[0] && !p.out[1]) return;
  const float rs = 1.0f / sqrtf(cta_sum(ss, red[3]) / (float)D + p.eps);
#pragma unroll
  for (int n = 0; n < 2; ++n) {
    if (!p.out[n]) continue;
    T* o = (T*)p.out[n] + r * p.ldo;
    const bf16* w = (const bf16*)p.w[n];
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int c = c0 + i * 1024;
      if (c < D) {
        float wv[4], q[4];
        Vec4<bf16>::load(w + c, wv);
#pragma unroll
        for (int u = 0; u < 4; ++u) q[u] = v[i][u] * rs * wv[u];
        Vec4<T>::store(o + c, q);
      }
    }
    for (int64_t c = D + c0; c < p.ldo; c += 1024) { const float z[4] = {0.f, 0.f, 0.f, 0.f}; Vec4<T>::store(o + c, z); }      // D and ldo are multiples of four
  }
}

// ---- evo_conv_act: a thread owns one channel of one sequence over RT consecutive rows, its last taps inputs in registers
constexpr int CONV_RT = 32, CONV_MAX_TAPS = 8, CONV_CTAS = 4;

// silu(4 v) of two values, as silu2_bf16 (common.cuh) does it, for sums whose weights were made a quarter beforehand (exact): the factor that keeps the reciprocal from being flushed
// then costs nothing, and every constant is four times its own
__device__ __forceinline__ float2 silu2_of_quarter(float2 v) {
  constexpr float LOG2E = 1.44269502f, LOG2E_REST = 1.92596303e-8f, QUARTER_LN2 = 0.25f * 0.693147182f;
  const float2 x = make_float2(fminf(v.x, 25.f), fminf(v.y, 25.f)), up = make_float2(-4.f * LOG2E, -4.f * LOG2E), quarter = make_float2(0.25f, 0.25f);
  const float2 t = __fmul2_rn(x, up);
  const float2 lo = __ffma2_rn(x, make_float2(-4.f * LOG2E_REST, -4.f * LOG2E_REST), __ffma2_rn(x, up, make_float2(-t.x, -t.y)));
  float2 e, r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e.x) : "f"(t.x));
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e.y) : "f"(t.y));
  const float2 d = __ffma2_rn(e, __ffma2_rn(lo, make_float2(QUARTER_LN2, QUARTER_LN2), quarter), quarter);
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r.x) : "f"(d.x));
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r.y) : "f"(d.y));
  return __fmul2_rn(v, r);
}
template <typename T, bool ACT> __device__ __forceinline__ float2 conv_finish(float2 v) {
  if constexpr (!ACT) return v;
  else if constexpr (sizeof(T) == 2) return silu2_of_quarter(v);
  else return make_float2(silu_f(v.x), silu_f(v.y));
}

// four channels per thread (8- or 16-byte accesses), taps and activation known at compile time.  Two special functions per element are 46 us for 4 x 4096 rows of 6144 channels, the
// bytes 64 (a plain copy): 79 us with cold L2 (88 to 92 as CTAs of 32 rows with four rows in work and four under way).  What it takes: bytes under way -- eight bf16 rows in work and
// eight under way, four CTAs per SM of 128 registers (with SiLU and two to four taps 8 to 16 bytes of a thread spill; four rows and six CTAs 83, five 90, four 97) -- and one wave of CTAs (conv_rows.h).  fp32 rows, four and four: 148 us (162).
template <typename T, int TAPS, bool ACT>
__global__ void __launch_bounds__(128, CONV_CTAS) conv_act4_kernel(evo_conv_act_params p, int write_carry, int rows_per) {
  pdl_wait();
  const int c = (blockIdx.x * blockDim.x + threadIdx.x) * 4;
  if (c >= p.C) return;
  constexpr int HALO = TAPS - 1, NB = sizeof(T) == 2 ? 8 : 4;
  const int b = blockIdx.z;
  const int64_t t0 = (int64_t)blockIdx.y * rows_per, ld = p.ld, ldo = p.ldo;
  const int rows = (int)min((int64_t)rows_per, p.L - t0);
  const T* src = (const T*)p.in + ((int64_t)b * p.L + t0) * ld + c;
  T* dst = (T*)p.out + ((int64_t)b * p.L + t0) * ldo + c;
  float* carry = p.carry ? p.carry + (int64_t)b * HALO * p.C + c : nullptr;
  constexpr float SCALE = ACT && sizeof(T) == 2 ? 0.25f : 1.f;
  float2 w[TAPS][2], bias[2];                             // channel pairs: one packed multiply-add serves two channels
  {
    // the four channels' taps lie one behind the other: 8 TAPS bytes, which start on 8 wherever the first channel's do
    const bf16* wp = (const bf16*)p.weight + (int64_t)c * TAPS;
    float f[4 * TAPS];
    if (((uintptr_t)p.weight & 7) == 0) {
#pragma unroll
      for (int j = 0; j < TAPS; ++j) Vec4<bf16>::load(wp + 4 * j, f + 4 * j);
    } else {
#pragma unroll
      for (int j = 0; j < 4 * TAPS; ++j) f[j] = __bfloat162float(wp[j]);
    }
#pragma unroll
    for (int u = 0; u < 2; ++u)
#pragma unroll
      for (int j = 0; j < TAPS; ++j) w[j][u] = make_float2(SCALE * f[2 * u * TAPS + j], SCALE * f[(2 * u + 1) * TAPS + j]);
  }
  bias[0] = bias[1] = make_float2(0.f, 0.f);
  if (p.bias) {
    float v[4];
    Vec4<bf16>::load((const bf16*)p.bias + c, v);
    bias[0] = make_float2(SCALE * v[0], SCALE * v[1]); bias[1] = make_float2(SCALE * v[2], SCALE * v[3]);
  }
  // rows travel packed, as they lie in memory: NB in work, NB under way
  Raw4<T> next[NB];
#pragma unroll
  for (int i = 0; i < NB; ++i)
    if (i < rows) next[i].load(src + i * ld);
  float2 x[HALO + NB][2];                            // the inputs in front, and the rows in work
#pragma unroll
  for (int j = 0; j < HALO; ++j) {
    float v[4] = {0.f, 0.f, 0.f, 0.f};
    if (t0 - HALO + j >= 0) Vec4<T>::load(src + (j - HALO) * ld, v);
    else if (carry && !p.zero_start) Vec4<float>::load(carry + (t0 + j) * p.C, v);
    x[j][0] = make_float2(v[0], v[1]); x[j][1] = make_float2(v[2], v[3]);
  }
  const auto take = [&](int i) {                          // row i of the group under way
    float v[4];
    next[i].get(v);
    x[HALO + i][0] = make_float2(v[0], v[1]); x[HALO + i][1] = make_float2(v[2], v[3]);
  };
  const auto row = [&](int i) {
    float v[4];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      float2 a = __ffma2_rn(w[HALO][u], x[HALO + i][u], bias[u]);
#pragma unroll
      for (int j = 0; j < HALO; ++j) a = __ffma2_rn(w[j][u], x[i + j][u], a);
      a = conv_finish<T, ACT>(a);
      v[2 * u] = a.x; v[2 * u + 1] = a.y;
    }
    Vec4<T>::store(dst + i * ldo, v);
  };
  int left = rows;
  for (; left >= NB; left -= NB) {
#pragma unroll
    for (int i = 0; i < NB; ++i) take(i);
    src += NB * ld;
    // the next rows are under way while these are worked on
    if (left >= 2 * NB) {
#pragma unroll
      for (int i = 0; i < NB; ++i) next[i].load(src + i * ld);
    } else {
#pragma unroll
      for (int i = 0; i < NB; ++i)
        if (NB + i < left) next[i].load(src + i * ld);
    }
#pragma unroll
    for (int i = 0; i < NB; ++i) row(i);
    dst += NB * ldo;
#pragma unroll
    for (int j = 0; j < HALO; ++j) { x[j][0] = x[j + NB][0]; x[j][1] = x[j + NB][1]; }
  }
#pragma unroll
  for (int i = 0; i + 1 < NB; ++i)                        // fewer than NB rows
    if (i < left) { take(i); row(i); }
  if (write_carry && carry && t0 + rows == p.L) {         // the last HALO inputs: x[left ..]
#pragma unroll
    for (int j = 0; j < HALO; ++j) {
      float2 lo = x[j][0], hi = x[j][1];
#pragma unroll
      for (int i = 1; i < NB; ++i)
        if (left == i) { lo = x[j + i][0]; hi = x[j + i][1]; }
      const float v[4] = {lo.x, lo.y, hi.x, hi.y};
      Vec4<float>::store(carry + (int64_t)j * p.C, v);
    }
  }
}

template <typename T>
__global__ void __launch_bounds__(128) conv_act_kernel(evo_conv_act_params p, int write_carry) {
  pdl_wait();
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= p.C) return;
  const int b = blockIdx.z, taps = p.taps, halo = taps - 1;
  const int64_t t0 = (int64_t)blockIdx.y * CONV_RT, t1 = min(p.L, t0 + CONV_RT);
  const T* in = (const T*)p.in + (int64_t)b * p.L * p.ld + c;
  float* carry = p.carry ? p.carry + (int64_t)b * halo * p.C + c : nullptr;
  float w[CONV_MAX_TAPS], win[CONV_MAX_TAPS];
#pragma unroll
  for (int j = 0; j < CONV_MAX_TAPS; ++j) w[j] = j < taps ? __bfloat162float(((const bf16*)p.weight)[(int64_t)c * taps + j]) : 0.f;
  const float bias = p.bias ? __bfloat162float(((const bf16*)p.bias)[c]) : 0.f;
  // win[j] = input at t - halo + j for the row t about to be computed; filled for j < halo here, win[halo] in the loop
#pragma unroll
  for (int j = 0; j < CONV_MAX_TAPS - 1; ++j) {
    win[j] = 0.f;
    if (j < halo) {
      const int64_t s = t0 - halo + j;
      if (s >= 0) win[j] = ldf(in + s * p.ld);
      else if (carry && !p.zero_start) win[j] = carry[(int64_t)(halo + s) * p.C];
    }
  }
  win[CONV_MAX_TAPS - 1] = 0.f;
  for (int64_t t = t0; t < t1; ++t) {
    const float cur = ldf(in + t * p.ld);
    float acc = bias;
#pragma unroll
    for (int j = 0; j < CONV_MAX_TAPS; ++j) {
      if (j < halo) acc = fmaf(w[j], win[j], acc);
      else if (j == halo) acc = fmaf(w[j], cur, acc);
    }
    if (p.act == 1) acc = silu_f(acc);
    stf((T*)p.out + ((int64_t)b * p.L + t) * p.ldo + c, acc);
#pragma unroll
    for (int j = 0; j < CONV_MAX_TAPS - 1; ++j) {
      if (j + 1 < halo) win[j] = win[j + 1];
      else if (j + 1 == halo) win[j] = cur;
    }
  }
  // after the last row win[0 .. halo) holds the last halo inputs (carried ones included when L < halo)
  if (write_carry && carry && t1 == p.L) {
#pragma unroll
    for (int j = 0; j < CONV_MAX_TAPS - 1; ++j)
      if (j < halo) carry[(int64_t)j * p.C] = win[j];
  }
}

// the carried inputs of a call whose rows were spread over several threads per channel: written after every row has been read
template <typename T>
__global__ void __launch_bounds__(128) conv_carry_kernel(evo_conv_act_params p) {
  pdl_wait();
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= p.C) return;
  const int b = blockIdx.z, halo = p.taps - 1;
  const T* in = (const T*)p.in + (int64_t)b * p.L * p.ld + c;
  float* carry = p.carry + (int64_t)b * halo * p.C + c;
  float keep[CONV_MAX_TAPS];
#pragma unroll
  for (int j = 0; j < CONV_MAX_TAPS - 1; ++j) {
    keep[j] = 0.f;
    if (j < halo) {
      const int64_t s = p.L - halo + j;
      if (s >= 0) keep[j] = ldf(in + s * p.ld);
      else if (!p.zero_start) keep[j] = carry[(int64_t)(halo + s) * p.C];
    }
  }
#pragma unroll
  for (int j = 0; j < CONV_MAX_TAPS - 1; ++j)
    if (j < halo) carry[(int64_t)j * p.C] = keep[j];
}

// ---- evo_xielu
template <typename T>
__global__ void __launch_bounds__(256) xielu_kernel(const T* __restrict__ z, int64_t ldz, const bf16* __restrict__ coef, T* __restrict__ out, int64_t ldo,
                                                    int64_t rows, int F) {
  const float pa = __bfloat162float(coef[0]), qa = __bfloat162float(coef[1]);
  // softplus in the form that neither overflows nor loses small values
  const float ap = fmaxf(pa, 0.f) + log1pf(expf(-fabsf(pa)));
  const float an = 0.5f + fmaxf(qa, 0.f) + log1pf(expf(-fabsf(qa)));
  const int64_t total = rows * ldo;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = i / ldo; const int c = (int)(i - r * ldo);
    float o = 0.f;
    if (c < F) {
      const float v = ldf(z + r * ldz + c);
      o = v > 0.f ? fmaf(ap * v, v, 0.5f * v) : fmaf(an, expm1f(v) - v, 0.5f * v);
    }
    stf(out + i, o);
  }
}

// four columns per thread, rows along grid.y: no division per element
template <typename T>
__global__ void __launch_bounds__(256) xielu4_kernel(const T* __restrict__ z, int64_t ldz, const bf16* __restrict__ coef, T* __restrict__ out, int64_t ldo,
                                                     int64_t rows, int F) {
  const float pa = __bfloat162float(coef[0]), qa = __bfloat162float(coef[1]);
  const float ap = fmaxf(pa, 0.f) + log1pf(expf(-fabsf(pa)));
  const float an = 0.5f + fmaxf(qa, 0.f) + log1pf(expf(-fabsf(qa)));
  const int c = (blockIdx.x * blockDim.x + threadIdx.x) * 4;
  if (c >= ldo) return;
  for (int64_t r = blockIdx.y; r < rows; r += gridDim.y) {
    float v[4] = {0.f, 0.f, 0.f, 0.f}, o[4];
    if (c < F) Vec4<T>::load(z + r * ldz + c, v);           // ldz >= F rounded up to four: the group may read pad columns of z, masked below
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const float x = v[u];
      // bf16 activations: e^x - 1 from the fast exponential (its absolute error is far below the output's rounding step)
      const float em1 = sizeof(T) == 2 ? __expf(x) - 1.f : expm1f(x);
      o[u] = c + u < F ? (x > 0.f ? fmaf(ap * x, x, 0.5f * x) : fmaf(an, em1 - x, 0.5f * x)) : 0.f;
    }
    Vec4<T>::store(out + r * ldo + c, o);
  }
}

// ---- evo_gated_group_norm: one warp per (row, part)
// the same with four entries per access (part size, strides and bases multiples of four entries)
template <typename T>
__global__ void __launch_bounds__(256) gated_group_norm4_kernel(const float* __restrict__ y, const T* __restrict__ gate, int64_t ldg, const bf16* __restrict__ nw,
                                                                T* __restrict__ out, int64_t ldo, int64_t rows, int width, int groups, float eps) {
  const int64_t wid = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (wid >= rows * groups) return;
  const int64_t r = wid / groups; const int g = (int)(wid % groups);
  const int gs = width / groups, c0 = g * gs;
  const float* yr = y + r * width + c0;
  const T* gr = gate + r * ldg + c0;
  float ss = 0.f;
  for (int c = lane * 4; c < gs; c += 128) {
    float a[4], b[4];
    Vec4<float>::load(yr + c, a); Vec4<T>::load(gr + c, b);
#pragma unroll
    for (int u = 0; u < 4; ++u) { const float v = a[u] * silu_f(b[u]); ss = fmaf(v, v, ss); }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
  const float rs = 1.0f / sqrtf(ss / (float)gs + eps);
  T* orow = out + r * ldo;
  for (int c = lane * 4; c < gs; c += 128) {
    float a[4], b[4], w[4];
    Vec4<float>::load(yr + c, a); Vec4<T>::load(gr + c, b); Vec4<bf16>::load(nw + c0 + c, w);
#pragma unroll
    for (int u = 0; u < 4; ++u) a[u] = a[u] * silu_f(b[u]) * rs * w[u];
    Vec4<T>::store(orow + c0 + c, a);
  }
  if (g == groups - 1)
    for (int64_t c = width + lane; c < ldo; c += 32) stf(orow + c, 0.f);
}

template <typename T>
__global__ void __launch_bounds__(256) gated_group_norm_kernel(const float* __restrict__ y, const T* __restrict__ gate, int64_t ldg, const bf16* __restrict__ nw,
                                                               T* __restrict__ out, int64_t ldo, int64_t rows, int width, int groups, float eps) {
  const int64_t wid = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (wid >= rows * groups) return;
  const int64_t r = wid / groups; const int g = (int)(wid % groups);
  const int gs = width / groups, c0 = g * gs;
  const float* yr = y + r * width + c0;
  const T* gr = gate + r * ldg + c0;
  float ss = 0.f;
  for (int c = lane; c < gs; c += 32) { const float v = yr[c] * silu_f(ldf(gr + c)); ss = fmaf(v, v, ss); }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
  const float rs = 1.0f / sqrtf(ss / (float)gs + eps);
  T* orow = out + r * ldo;
  for (int c = lane; c < gs; c += 32) stf(orow + c0 + c, yr[c] * silu_f(ldf(gr + c)) * rs * __bfloat162float(nw[c0 + c]));
  if (g == groups - 1)
    for (int64_t c = width + lane; c < ldo; c += 32) stf(orow + c, 0.f);
}

}  // namespace

extern "C" int evo_sum_norm(const evo_sum_norm_params* p, void* stream) {
  EVO_REQUIRE(p->x && p->D > 0 && p->rows >= 0 && p->n_branches >= 0 && p->n_branches <= EVO_SUM_NORM_BRANCHES, "evo_sum_norm: bad arguments");
  for (int b = 0; b < p->n_branches; ++b) EVO_REQUIRE(p->y[b] && p->ldy[b] >= p->D, "evo_sum_norm: branch %d missing or too narrow", b);
  for (int n = 0; n < 2; ++n) EVO_REQUIRE(!p->out[n] || (p->w[n] && p->ldo >= p->D), "evo_sum_norm: output %d without weight or too narrow", n);
  if (p->rows == 0) return 0;
  const size_t smem = sizeof(float) * ((size_t)p->D + 33);
  EVO_REQUIRE(smem <= 200 * 1024, "evo_sum_norm: width %d too large for one CTA's shared memory", p->D);
  cudaStream_t st = (cudaStream_t)stream;
  // four elements per access when every row of every operand starts on a multiple of four elements
  bool vec = p->D % 4 == 0 && p->ldo % 4 == 0 && ((uintptr_t)p->x & 15) == 0;
  for (int b = 0; b < p->n_branches; ++b) {
    vec = vec && p->ldy[b] % 4 == 0 && (p->dtype ? aligned4<float>(p->y[b]) : aligned4<bf16>(p->y[b]));
    if (p->norm_w[b]) vec = vec && aligned4<bf16>(p->norm_w[b]);
  }
  vec = vec && (!p->col_scale || aligned4<bf16>(p->col_scale));
  for (int n = 0; n < 2; ++n)
    if (p->out[n]) vec = vec && aligned4<bf16>(p->w[n]) && (p->dtype ? aligned4<float>(p->out[n]) : aligned4<bf16>(p->out[n]));
  if (vec && p->D <= 4096) {
    static_assert(EVO_SUM_NORM_BRANCHES == 3, "the switch below");
    // rows in registers: (groups of four per thread) x (branches)
#define EVO_SUM_NORM(TT, NV) \
    switch (p->n_branches) { \
      case 0: EVO_CUDA(launch_dependent(sum_norm_row_kernel<TT, NV, 0>, dim3((unsigned)p->rows), dim3(256), 0, st, *p)); break; \
      case 1: EVO_CUDA(launch_dependent(sum_norm_row_kernel<TT, NV, 1>, dim3((unsigned)p->rows), dim3(256), 0, st, *p)); break; \
      case 2: EVO_CUDA(launch_dependent(sum_norm_row_kernel<TT, NV, 2>, dim3((unsigned)p->rows), dim3(256), 0, st, *p)); break; \
      default: EVO_CUDA(launch_dependent(sum_norm_row_kernel<TT, NV, 3>, dim3((unsigned)p->rows), dim3(256), 0, st, *p)); break; \
    }
    if (p->dtype) { if (p->D <= 1024) { EVO_SUM_NORM(float, 1) } else if (p->D <= 2048) { EVO_SUM_NORM(float, 2) } else { EVO_SUM_NORM(float, 4) } }
    else { if (p->D <= 1024) { EVO_SUM_NORM(bf16, 1) } else if (p->D <= 2048) { EVO_SUM_NORM(bf16, 2) } else { EVO_SUM_NORM(bf16, 4) } }
#undef EVO_SUM_NORM
    return check_launch("evo_sum_norm");
  }
  auto kern = p->dtype ? (vec ? sum_norm_kernel<float, true> : sum_norm_kernel<float, false>) : (vec ? sum_norm_kernel<bf16, true> : sum_norm_kernel<bf16, false>);
  if (smem > 48 * 1024) EVO_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  EVO_CUDA(launch_dependent(kern, dim3((unsigned)p->rows), dim3(256), smem, st, *p));
  return check_launch("evo_sum_norm");
}

extern "C" int evo_conv_act(const evo_conv_act_params* p, void* stream) {
  EVO_REQUIRE(p->in && p->weight && p->out && p->C > 0 && p->taps >= 1 && p->taps <= CONV_MAX_TAPS, "evo_conv_act: bad arguments (taps 1..%d)", CONV_MAX_TAPS);
  EVO_REQUIRE(p->ld >= p->C && p->ldo >= p->C && p->B >= 0 && p->L >= 0, "evo_conv_act: bad shape");
  if (p->B == 0 || p->L == 0) return 0;
  cudaStream_t st = (cudaStream_t)stream;
  const bool vec = p->C % 4 == 0 && p->ld % 4 == 0 && p->ldo % 4 == 0 && p->taps <= 4 && (!p->carry || ((uintptr_t)p->carry & 15) == 0) &&
                   (!p->bias || aligned4<bf16>(p->bias)) &&
                   (p->dtype ? aligned4<float>(p->in) && aligned4<float>(p->out) : aligned4<bf16>(p->in) && aligned4<bf16>(p->out));
  const int64_t rows_per = vec ? conv_rows(p->L, (p->C / 4 + 127) / 128 * (int64_t)p->B, (int64_t)device_sm_count() * CONV_CTAS, CONV_RT) : CONV_RT;
  const unsigned chunks = (unsigned)((p->L + rows_per - 1) / rows_per);
  const dim3 grid((p->C + 127) / 128, chunks, p->B);
  // with one thread per (sequence, channel) that thread reads the carried inputs before it replaces them, and where none are read (zero_start) the thread of the last
  // rows may replace them; otherwise a second launch does
  const int own = chunks == 1 || p->zero_start;
  if (vec) {
    const dim3 g4((p->C / 4 + 127) / 128, chunks, p->B);
#define EVO_CONV4(TT, ACT) \
    switch (p->taps) { \
      case 1: EVO_CUDA(launch_dependent(conv_act4_kernel<TT, 1, ACT>, g4, dim3(128), 0, st, *p, own, (int)rows_per)); break; \
      case 2: EVO_CUDA(launch_dependent(conv_act4_kernel<TT, 2, ACT>, g4, dim3(128), 0, st, *p, own, (int)rows_per)); break; \
      case 3: EVO_CUDA(launch_dependent(conv_act4_kernel<TT, 3, ACT>, g4, dim3(128), 0, st, *p, own, (int)rows_per)); break; \
      default: EVO_CUDA(launch_dependent(conv_act4_kernel<TT, 4, ACT>, g4, dim3(128), 0, st, *p, own, (int)rows_per)); break; \
    }
    if (p->dtype) { if (p->act == 1) { EVO_CONV4(float, true) } else { EVO_CONV4(float, false) } }
    else if (p->act == 1) { EVO_CONV4(bf16, true) } else { EVO_CONV4(bf16, false) }
#undef EVO_CONV4
  } else EVO_CUDA(launch_dependent(p->dtype ? conv_act_kernel<float> : conv_act_kernel<bf16>, grid, dim3(128), 0, st, *p, own));
  int rc = check_launch("evo_conv_act");
  if (rc || own || !p->carry || p->taps == 1) return rc;
  const dim3 g2((p->C + 127) / 128, 1, p->B);
  EVO_CUDA(launch_dependent(p->dtype ? conv_carry_kernel<float> : conv_carry_kernel<bf16>, g2, dim3(128), 0, st, *p));
  return check_launch("evo_conv_act");
}

extern "C" int evo_xielu(const void* z, int64_t ldz, const void* coef, void* out, int64_t ldo, int64_t rows, int F, int dtype, void* stream) {
  EVO_REQUIRE(z && coef && out && F > 0 && ldz >= F && ldo >= F && rows >= 0, "evo_xielu: bad arguments");
  if (rows == 0) return 0;
  const int64_t total = rows * ldo;
  const unsigned grid = (unsigned)std::min<int64_t>((total + 255) / 256, (int64_t)device_sm_count() * 16);
  cudaStream_t st = (cudaStream_t)stream;
  if (ldz % 4 == 0 && ldo % 4 == 0 && ldz >= (F + 3) / 4 * 4 && (dtype ? aligned4<float>(z) && aligned4<float>(out) : aligned4<bf16>(z) && aligned4<bf16>(out))) {
    // a thread walks several rows of its four columns, so that the two softplus of the coefficients are paid once per many elements
    const dim3 g4((unsigned)((ldo / 4 + 255) / 256), (unsigned)std::min<int64_t>(rows, std::max<int64_t>(1, (int64_t)device_sm_count() * 8 / ((ldo / 4 + 255) / 256))));
    if (dtype) xielu4_kernel<float><<<g4, 256, 0, st>>>((const float*)z, ldz, (const bf16*)coef, (float*)out, ldo, rows, F);
    else xielu4_kernel<bf16><<<g4, 256, 0, st>>>((const bf16*)z, ldz, (const bf16*)coef, (bf16*)out, ldo, rows, F);
    return check_launch("evo_xielu");
  }
  if (dtype) xielu_kernel<float><<<grid, 256, 0, st>>>((const float*)z, ldz, (const bf16*)coef, (float*)out, ldo, rows, F);
  else xielu_kernel<bf16><<<grid, 256, 0, st>>>((const bf16*)z, ldz, (const bf16*)coef, (bf16*)out, ldo, rows, F);
  return check_launch("evo_xielu");
}

extern "C" int evo_gated_group_norm(const float* y, const void* gate, int64_t ldg, const void* norm_w, void* out, int64_t ldo,
                                    int64_t rows, int width, int groups, float eps, int dtype, void* stream) {
  EVO_REQUIRE(y && gate && norm_w && out && width > 0 && groups > 0 && width % groups == 0 && ldo >= width && ldg >= width, "evo_gated_group_norm: bad arguments");
  if (rows == 0) return 0;
  const int64_t warps = rows * groups;
  cudaStream_t st = (cudaStream_t)stream;
  const unsigned grid = (unsigned)((warps + 7) / 8);
  if ((width / groups) % 4 == 0 && ldg % 4 == 0 && ldo % 4 == 0 && ((uintptr_t)y & 15) == 0 && aligned4<bf16>(norm_w) &&
      (dtype ? aligned4<float>(gate) && aligned4<float>(out) : aligned4<bf16>(gate) && aligned4<bf16>(out))) {
    if (dtype) gated_group_norm4_kernel<float><<<grid, 256, 0, st>>>(y, (const float*)gate, ldg, (const bf16*)norm_w, (float*)out, ldo, rows, width, groups, eps);
    else gated_group_norm4_kernel<bf16><<<grid, 256, 0, st>>>(y, (const bf16*)gate, ldg, (const bf16*)norm_w, (bf16*)out, ldo, rows, width, groups, eps);
    return check_launch("evo_gated_group_norm");
  }
  if (dtype) gated_group_norm_kernel<float><<<grid, 256, 0, st>>>(y, (const float*)gate, ldg, (const bf16*)norm_w, (float*)out, ldo, rows, width, groups, eps);
  else gated_group_norm_kernel<bf16><<<grid, 256, 0, st>>>(y, (const bf16*)gate, ldg, (const bf16*)norm_w, (bf16*)out, ldo, rows, width, groups, eps);
  return check_launch("evo_gated_group_norm");
}
