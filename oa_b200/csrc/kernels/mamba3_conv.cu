// Causal depthwise convolution + SiLU over a column range of the projected rows of a Mamba block, in place, and the
// learned-decay fill of the dd_A columns.  These are the options of the benchmark's Mamba-3 configuration (convolution
// width 4 before the scan, A = -exp(A_log)); the reference's mixer has neither (Source/Private/Oa/Ml/Nn/Mamba3/Mamba3.cpp).
//
//   forward   y[t, c] = silu(sum_k w[k, c] * x[t - k, c])   (x = 0 before the start of the sequence), written over x
//   backward  g[t, c] = dy[t, c] * silu'(pre[t, c]) with pre recomputed from the saved x;
//             dx[t, c] = sum_k w[k, c] * g[t + k, c];  dw[k, c] = sum_t g[t, c] * x[t - k, c]
// One thread owns one column and walks a block of TB tokens with the last K-1 inputs in registers, so global memory is read
// in whole rows; weight-gradient partials are written per token block and reduced in a fixed order by the caller.
#include "common.cuh"
#include "api.h"

namespace oa {

constexpr int MC_TB = 64;      // tokens per block
constexpr int MC_MAXK = 8;

template <typename T> __device__ __forceinline__ float mc_ld(const T* p);
template <> __device__ __forceinline__ float mc_ld<float>(const float* p) { return *p; }
template <> __device__ __forceinline__ float mc_ld<__nv_bfloat16>(const __nv_bfloat16* p) { return __bfloat162float(*p); }
template <typename T> __device__ __forceinline__ void mc_st(T* p, float v);
template <> __device__ __forceinline__ void mc_st<float>(float* p, float v) { *p = v; }
template <> __device__ __forceinline__ void mc_st<__nv_bfloat16>(__nv_bfloat16* p, float v) { *p = __float2bfloat16_rn(v); }

// grid (ceil(C / 128), B * ceil(L / TB)); x: [B*L, ld] column range [col0, col0 + C); saved: [B*L, C] copy of the inputs
template <typename T>
__global__ void __launch_bounds__(128)
mamba3_conv_fwd_kernel(T* __restrict__ x, long long ld, int col0, T* __restrict__ saved, const float* __restrict__ w, int B, int L, int C,
                       int Kw) {
  const int c = blockIdx.x * 128 + threadIdx.x;
  if (c >= C) return;
  const int nb = (L + MC_TB - 1) / MC_TB;
  const int b = blockIdx.y / nb, t0 = (blockIdx.y % nb) * MC_TB;
  float wk[MC_MAXK], win[MC_MAXK];
#pragma unroll
  for (int k = 0; k < MC_MAXK; ++k) {
    wk[k] = k < Kw ? w[(long long)k * C + c] : 0.f;
    const int t = t0 - 1 - k;                    // win[k] = x[t0 - 1 - k]
    win[k] = (k < Kw - 1 && t >= 0) ? mc_ld(saved + ((long long)b * L + t) * C + c) : 0.f;
  }
  // Inputs (also the halo, which another block overwrites) are read from `saved`, the copy made by the launch before this one.
  const int t1 = min(L, t0 + MC_TB);
  for (int t = t0; t < t1; ++t) {
    const long long row = (long long)b * L + t;
    const float xt = mc_ld(saved + row * C + c);
    float acc = wk[0] * xt;
#pragma unroll
    for (int k = 1; k < MC_MAXK; ++k) acc = fmaf(wk[k], win[k - 1], acc);
#pragma unroll
    for (int k = MC_MAXK - 1; k > 0; --k) win[k] = win[k - 1];
    win[0] = xt;
    mc_st(x + row * ld + col0 + c, silu_f(acc));
  }
}

template <typename T>
__global__ void mamba3_cols_copy_kernel(const T* __restrict__ x, long long ld, int col0, T* __restrict__ out, long long rows, int C) {
  const long long total = rows * C;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride)
    out[i] = x[(i / C) * ld + col0 + (i % C)];
}

// dy: [B*L, ld] column range (gradient of the convolved columns), overwritten by dx; saved: the forward inputs;
// dw_part: float[B * nb][Kw][C]
template <typename T>
__global__ void __launch_bounds__(128)
mamba3_conv_bwd_kernel(T* __restrict__ dy, long long ld, int col0, const T* __restrict__ saved, const float* __restrict__ w,
                       float* __restrict__ dw_part, T* __restrict__ gbuf, int B, int L, int C, int Kw) {
  // pass A (gbuf != null, dy read-only): g = dy * silu'(pre) -> gbuf [B*L, C];   pass B (gbuf read-only): dx and dw from g
  const int c = blockIdx.x * 128 + threadIdx.x;
  if (c >= C) return;
  const int nb = (L + MC_TB - 1) / MC_TB;
  const int b = blockIdx.y / nb, t0 = (blockIdx.y % nb) * MC_TB;
  const int t1 = min(L, t0 + MC_TB);
  float wk[MC_MAXK];
#pragma unroll
  for (int k = 0; k < MC_MAXK; ++k) wk[k] = k < Kw ? w[(long long)k * C + c] : 0.f;
  if (dw_part == nullptr) {
    float win[MC_MAXK];
#pragma unroll
    for (int k = 0; k < MC_MAXK; ++k) {
      const int t = t0 - 1 - k;
      win[k] = (k < Kw - 1 && t >= 0) ? mc_ld(saved + ((long long)b * L + t) * C + c) : 0.f;
    }
    for (int t = t0; t < t1; ++t) {
      const long long row = (long long)b * L + t;
      const float xt = mc_ld(saved + row * C + c);
      float pre = wk[0] * xt;
#pragma unroll
      for (int k = 1; k < MC_MAXK; ++k) pre = fmaf(wk[k], win[k - 1], pre);
#pragma unroll
      for (int k = MC_MAXK - 1; k > 0; --k) win[k] = win[k - 1];
      win[0] = xt;
      const float sg = sigmoid_f(pre);
      mc_st(gbuf + row * C + c, mc_ld(dy + row * ld + col0 + c) * sg * (1.f + pre * (1.f - sg)));
    }
    return;
  }
  // pass B: dx[t] = sum_k w[k] g[t + k];  dw[k] += g[t] x[t - k]
  float dwk[MC_MAXK];
#pragma unroll
  for (int k = 0; k < MC_MAXK; ++k) dwk[k] = 0.f;
  for (int t = t0; t < t1; ++t) {
    const long long row = (long long)b * L + t;
    float dx = 0.f;
    const float gt = mc_ld(gbuf + row * C + c);
#pragma unroll
    for (int k = 0; k < MC_MAXK; ++k) {
      if (k < Kw) {
        if (t + k < L) dx = fmaf(wk[k], mc_ld(gbuf + (row + k) * C + c), dx);
        if (t - k >= 0) dwk[k] = fmaf(gt, mc_ld(saved + (row - k) * C + c), dwk[k]);
      }
    }
    mc_st(dy + row * ld + col0 + c, dx);
  }
  for (int k = 0; k < Kw; ++k) dw_part[((long long)blockIdx.y * Kw + k) * C + c] = dwk[k];
}

// Width-4 convolution of bf16 columns in 16-byte pieces: a thread owns eight neighbouring columns.  The kernels above move two
// bytes per lane and access and fetch every tap again: 2 x 4096 tokens x 3328 columns: forward 177 -> 76 us,
// backward 306 -> 130 us.
constexpr int MC_KW = 4;
__device__ __forceinline__ void mc_ld8(const __nv_bfloat16* p, float (&v)[8]) {
  const uint4 u = *reinterpret_cast<const uint4*>(p);
  const float2 a = unpack_bf16x2(u.x), b = unpack_bf16x2(u.y), c = unpack_bf16x2(u.z), d = unpack_bf16x2(u.w);
  v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y; v[4] = c.x; v[5] = c.y; v[6] = d.x; v[7] = d.y;
}
__device__ __forceinline__ void mc_st8(__nv_bfloat16* p, const float (&v)[8]) {
  *reinterpret_cast<uint4*>(p) = make_uint4(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]), pack_bf16x2(v[4], v[5]), pack_bf16x2(v[6], v[7]));
}

__global__ void __launch_bounds__(256)
mamba3_cols_copy_vec_kernel(const __nv_bfloat16* __restrict__ x, long long ld, int col0, __nv_bfloat16* __restrict__ out, long long rows, int C) {
  const int c8 = C >> 3;
  const long long total = rows * c8, stride = (long long)gridDim.x * blockDim.x;
#pragma unroll 4
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
    const long long r = i / c8;
    *reinterpret_cast<uint4*>(out + i * 8) = *reinterpret_cast<const uint4*>(x + r * ld + col0 + (i - r * c8) * 8);
  }
}

// MODE 0: y = silu(conv) over x;  1: g = dy silu'(pre) into gbuf;  2: dx from g over dy, and the weight-gradient partials.
// Grid as above with 128 x 8 columns per block; MODE 2 walks a window of g forwards and of the inputs backwards.
template <int MODE>
__global__ void __launch_bounds__(128)
mamba3_conv4_vec_kernel(__nv_bfloat16* __restrict__ x, long long ld, int col0, const __nv_bfloat16* __restrict__ saved, const float* __restrict__ w,
                        __nv_bfloat16* __restrict__ gbuf, float* __restrict__ dw_part, int L, int C, int tb) {
  const int c = (blockIdx.x * 128 + threadIdx.x) * 8;
  if (c >= C) return;
  const int nb = (L + tb - 1) / tb;
  const int b = blockIdx.y / nb, t0 = (blockIdx.y % nb) * tb, t1 = min(L, t0 + tb);
  const long long base = (long long)b * L;
  float wk[MC_KW][8], win[MC_KW - 1][8];                     // win[k] = input at t - 1 - k
#pragma unroll
  for (int k = 0; k < MC_KW; ++k)
#pragma unroll
    for (int j = 0; j < 8; ++j) wk[k][j] = w[(long long)k * C + c + j];
#pragma unroll
  for (int k = 0; k < MC_KW - 1; ++k) {
    if (t0 - 1 - k >= 0) mc_ld8(saved + (base + t0 - 1 - k) * C + c, win[k]);
    else
#pragma unroll
      for (int j = 0; j < 8; ++j) win[k][j] = 0.f;
  }
  if (MODE != 2) {
#pragma unroll 4
    for (int t = t0; t < t1; ++t) {
      const long long row = base + t;
      float xt[8], d[8], o[8];
      mc_ld8(saved + row * C + c, xt);
      if (MODE == 1) mc_ld8(x + row * ld + col0 + c, d);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        float pre = wk[0][j] * xt[j];
        pre = fmaf(wk[1][j], win[0][j], pre);
        pre = fmaf(wk[2][j], win[1][j], pre);
        pre = fmaf(wk[3][j], win[2][j], pre);
        win[2][j] = win[1][j]; win[1][j] = win[0][j]; win[0][j] = xt[j];
        if (MODE == 0) o[j] = silu_f(pre);
        else {
          const float sg = sigmoid_f(pre);
          o[j] = d[j] * sg * (1.f + pre * (1.f - sg));
        }
      }
      if (MODE == 0) mc_st8(x + row * ld + col0 + c, o);
      else mc_st8(gbuf + row * C + c, o);
    }
  } else {
    float dwk[MC_KW][8], g[MC_KW][8];                        // g[k] = g[t + k]
#pragma unroll
    for (int k = 0; k < MC_KW; ++k)
#pragma unroll
      for (int j = 0; j < 8; ++j) dwk[k][j] = g[k][j] = 0.f;
#pragma unroll
    for (int k = 0; k < MC_KW - 1; ++k)
      if (t0 + k < L) mc_ld8(gbuf + (base + t0 + k) * C + c, g[k]);
#pragma unroll 2
    for (int t = t0; t < t1; ++t) {
      const long long row = base + t;
      float xt[8], o[8];
      mc_ld8(saved + row * C + c, xt);
      if (t + MC_KW - 1 < L) mc_ld8(gbuf + (row + MC_KW - 1) * C + c, g[MC_KW - 1]);
      else
#pragma unroll
        for (int j = 0; j < 8; ++j) g[MC_KW - 1][j] = 0.f;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        float dx = wk[0][j] * g[0][j];
        dx = fmaf(wk[1][j], g[1][j], dx);
        dx = fmaf(wk[2][j], g[2][j], dx);
        o[j] = fmaf(wk[3][j], g[3][j], dx);
        dwk[0][j] = fmaf(g[0][j], xt[j], dwk[0][j]);
        dwk[1][j] = fmaf(g[0][j], win[0][j], dwk[1][j]);
        dwk[2][j] = fmaf(g[0][j], win[1][j], dwk[2][j]);
        dwk[3][j] = fmaf(g[0][j], win[2][j], dwk[3][j]);
        win[2][j] = win[1][j]; win[1][j] = win[0][j]; win[0][j] = xt[j];
        g[0][j] = g[1][j]; g[1][j] = g[2][j]; g[2][j] = g[3][j];
      }
      mc_st8(x + row * ld + col0 + c, o);
    }
#pragma unroll
    for (int k = 0; k < MC_KW; ++k)
#pragma unroll
      for (int j = 0; j < 8; ++j) dw_part[((long long)blockIdx.y * MC_KW + k) * C + c + j] = dwk[k][j];
  }
}

// A step of the serial walk over tokens costs more with eight columns to a thread, which the better loads repay once there are many
// threads, or tokens enough for the shorter blocks.  Scalar against vector, forward: 1 x 16 x 768 8.0 / 14 us, 1 x 32 x 3328 13.5 / 15.9,
// 1 x 48 x 768 and 64 x 1 x 3328 the other way (6.9 / 5.5); backward: 1 x 16 x 768 15 / 19, 64 x 1 x 3328 8.8 / 11.1, 64 x 8 x 3328 22.5 / 19.6.
inline bool mc_vec_fwd_pays(long long rows, int L, int C) { return L >= 48 || rows * (C >> 3) > 24576; }
inline bool mc_vec_bwd_pays(long long rows, int L, int C) { return L >= 32 || rows * (C >> 3) > 131072; }

inline bool mc_vec_ok(int dtype, int C, int Kw, long long ld, int col0, const void* a, const void* b, const void* c) {
  return dtype == OA_BF16 && Kw == MC_KW && (C & 7) == 0 && (ld & 7) == 0 && (col0 & 7) == 0 &&
         ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b) | reinterpret_cast<uintptr_t>(c)) & 15) == 0;
}

// x[row, col0 + h] = exp(a_log[h]) - 1
template <typename T>
__global__ void mamba3_alog_fill_kernel(T* __restrict__ x, long long ld, int col0, const float* __restrict__ a_log, long long rows, int H) {
  const long long total = rows * H;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
    const int h = (int)(i % H);
    mc_st(x + (i / H) * ld + col0 + h, __expf(a_log[h]) - 1.f);
  }
}

static inline int mc_grid(long long n) {
  long long b = (n + 255) / 256;
  if (b > 148 * 8) b = 148 * 8;
  return (int)(b < 1 ? 1 : b);
}

}  // namespace oa

using namespace oa;
#define ST ((cudaStream_t)stream)
#define CHECK_LAUNCH() (cudaGetLastError() == cudaSuccess ? OA_OK : OA_ERR_LAUNCH)

extern "C" int oa_mamba3_conv_fwd(int dtype, void* x, long long ld, int col0, void* saved, const float* w, int B, int L, int C,
                                  int Kw, void* stream) {
  if (Kw < 1 || Kw > MC_MAXK || B <= 0 || L <= 0 || C <= 0) return OA_ERR_ARG;
  const long long rows = (long long)B * L;
  dim3 grid((C + 127) / 128, B * ((L + MC_TB - 1) / MC_TB));
  const int tb = 16; // short blocks: three halo rows each, but enough of them to fill the SMs
  if (mc_vec_ok(dtype, C, Kw, ld, col0, x, saved, nullptr) && mc_vec_fwd_pays(rows, L, C) && (long long)B * ((L + tb - 1) / tb) <= 65535) {
    mamba3_cols_copy_vec_kernel<<<mc_grid(rows * (C / 8)), 256, 0, ST>>>((const __nv_bfloat16*)x, ld, col0, (__nv_bfloat16*)saved, rows, C);
    mamba3_conv4_vec_kernel<0><<<dim3((C / 8 + 127) / 128, B * ((L + tb - 1) / tb)), 128, 0, ST>>>((__nv_bfloat16*)x, ld, col0,
        (const __nv_bfloat16*)saved, w, nullptr, nullptr, L, C, tb);
    return CHECK_LAUNCH();
  }
  if (dtype == OA_F32) {
    mamba3_cols_copy_kernel<float><<<mc_grid(rows * C), 256, 0, ST>>>((const float*)x, ld, col0, (float*)saved, rows, C);
    mamba3_conv_fwd_kernel<float><<<grid, 128, 0, ST>>>((float*)x, ld, col0, (float*)saved, w, B, L, C, Kw);
  } else if (dtype == OA_BF16) {
    mamba3_cols_copy_kernel<__nv_bfloat16><<<mc_grid(rows * C), 256, 0, ST>>>((const __nv_bfloat16*)x, ld, col0, (__nv_bfloat16*)saved, rows, C);
    mamba3_conv_fwd_kernel<__nv_bfloat16><<<grid, 128, 0, ST>>>((__nv_bfloat16*)x, ld, col0, (__nv_bfloat16*)saved, w, B, L, C, Kw);
  } else return OA_ERR_UNSUPPORTED;
  return CHECK_LAUNCH();
}

// gbuf: [B*L, C] scratch of the data type; dw_part: float[B * ceil(L / 64) * Kw * C] (reduce over its first axis afterwards)
extern "C" int oa_mamba3_conv_bwd(int dtype, void* dy, long long ld, int col0, const void* saved, const float* w, float* dw_part,
                                  void* gbuf, int B, int L, int C, int Kw, void* stream) {
  if (Kw < 1 || Kw > MC_MAXK || B <= 0 || L <= 0 || C <= 0) return OA_ERR_ARG;
  dim3 grid((C + 127) / 128, B * ((L + MC_TB - 1) / MC_TB));
  const int tb = 16;
  if (mc_vec_ok(dtype, C, Kw, ld, col0, dy, saved, gbuf) && mc_vec_bwd_pays((long long)B * L, L, C) && (long long)B * ((L + tb - 1) / tb) <= 65535) {
    mamba3_conv4_vec_kernel<1><<<dim3((C / 8 + 127) / 128, B * ((L + tb - 1) / tb)), 128, 0, ST>>>((__nv_bfloat16*)dy, ld, col0,
        (const __nv_bfloat16*)saved, w, (__nv_bfloat16*)gbuf, nullptr, L, C, tb);
    mamba3_conv4_vec_kernel<2><<<dim3((C / 8 + 127) / 128, B * ((L + MC_TB - 1) / MC_TB)), 128, 0, ST>>>((__nv_bfloat16*)dy, ld, col0,
        (const __nv_bfloat16*)saved, w, (__nv_bfloat16*)gbuf, dw_part, L, C, MC_TB);
    return CHECK_LAUNCH();
  }
  if (dtype == OA_F32) {
    mamba3_conv_bwd_kernel<float><<<grid, 128, 0, ST>>>((float*)dy, ld, col0, (const float*)saved, w, nullptr, (float*)gbuf, B, L, C, Kw);
    mamba3_conv_bwd_kernel<float><<<grid, 128, 0, ST>>>((float*)dy, ld, col0, (const float*)saved, w, dw_part, (float*)gbuf, B, L, C, Kw);
  } else if (dtype == OA_BF16) {
    mamba3_conv_bwd_kernel<__nv_bfloat16><<<grid, 128, 0, ST>>>((__nv_bfloat16*)dy, ld, col0, (const __nv_bfloat16*)saved, w, nullptr,
                                                                (__nv_bfloat16*)gbuf, B, L, C, Kw);
    mamba3_conv_bwd_kernel<__nv_bfloat16><<<grid, 128, 0, ST>>>((__nv_bfloat16*)dy, ld, col0, (const __nv_bfloat16*)saved, w, dw_part,
                                                                (__nv_bfloat16*)gbuf, B, L, C, Kw);
  } else return OA_ERR_UNSUPPORTED;
  return CHECK_LAUNCH();
}

extern "C" int oa_mamba3_alog_fill(int dtype, void* x, long long ld, int col0, const float* a_log, long long rows, int H, void* stream) {
  if (rows <= 0 || H <= 0) return OA_OK;
  if (dtype == OA_F32) mamba3_alog_fill_kernel<float><<<mc_grid(rows * H), 256, 0, ST>>>((float*)x, ld, col0, a_log, rows, H);
  else if (dtype == OA_BF16) mamba3_alog_fill_kernel<__nv_bfloat16><<<mc_grid(rows * H), 256, 0, ST>>>((__nv_bfloat16*)x, ld, col0, a_log, rows, H);
  else return OA_ERR_UNSUPPORTED;
  return CHECK_LAUNCH();
}
