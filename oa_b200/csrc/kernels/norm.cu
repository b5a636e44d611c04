// RMSNorm and LayerNorm, forward and backward (fp32 or bf16 storage, fp32 math).
//   RMSNorm:   y = x * rsqrt(mean(x^2) + eps) * w                  (Nn/RmsNorm/RmsNorm.slang:26-30)
//   LayerNorm: y = (x - mean) * rsqrt(var + eps) * w + b, biased variance, two passes
//              (Nn/LayerNorm/LayerNorm.slang:41-58)
// One warp per row.  The forward can add a residual stream first (ResidualRmsNorm); the backward
// can add the gradient that arrives through the residual path, so that no separate add kernels run.
// Weight / bias gradients: each warp keeps private column partials in shared memory over the rows it
// owns, each CTA writes one partial row to a scratch buffer, and a second kernel sums the partial
// rows in a fixed order (deterministic, no atomics).
#include "common.cuh"
#include "api.h"

namespace oa {

template <typename T> struct NIO;
template <> struct NIO<float> {
  static constexpr int VEC = 4;
  __device__ static void load(const float* p, float* v) {
    float4 x = *reinterpret_cast<const float4*>(p);
    v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
  }
  __device__ static void store(float* p, const float* v) { *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]); }
};
template <> struct NIO<__nv_bfloat16> {
  static constexpr int VEC = 8;
  __device__ static void load(const __nv_bfloat16* p, float* v) {
    uint4 x = *reinterpret_cast<const uint4*>(p);
    float2 a = unpack_bf16x2(x.x), b = unpack_bf16x2(x.y), c = unpack_bf16x2(x.z), d = unpack_bf16x2(x.w);
    v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y; v[4] = c.x; v[5] = c.y; v[6] = d.x; v[7] = d.y;
  }
  __device__ static void store(__nv_bfloat16* p, const float* v) {
    *reinterpret_cast<uint4*>(p) = make_uint4(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]), pack_bf16x2(v[4], v[5]),
                                              pack_bf16x2(v[6], v[7]));
  }
};

constexpr int NORM_THREADS = 256;
constexpr int NORM_WARPS = NORM_THREADS / 32;

// Rows of up to 32 * VEC * NV columns: the row stays in registers (packed as it is stored) between the sum of squares and the
// output, so memory is read once and all of a lane's loads are in flight together.  16384 x 1024 is at the copy rate either way
// (9.5 and 9.0 us out of L2); with few rows two dependent passes were all latency: 149 x 4096 went from 6.8 to 4.4 us.  Where rows
// are many and wide the registers leave too few warps (4736 x 2880: 9.4 us in two passes, 12.3 here), the more so with a residual,
// whose loads wait behind the row's (33.6 and 54.3 us at 4736 x 4096): see rmsnorm_in_registers.
template <typename T, int NV>
__global__ void __launch_bounds__(NORM_THREADS)
rmsnorm_fwd_reg_kernel(const T* __restrict__ x, const T* __restrict__ w, T* __restrict__ y, float* __restrict__ rstd_out,
                       long long rows, int cols, float eps, const T* __restrict__ res_in, T* __restrict__ res_out) {
  pdl_launch_dependents();
  pdl_wait();
  constexpr int V = NIO<T>::VEC;
  const int lane = threadIdx.x & 31;
  const long long row = (long long)blockIdx.x * NORM_WARPS + (threadIdx.x >> 5);
  if (row >= rows) return;
  const int nv = cols / V;
  const T* px = x + row * cols;
  uint4 xp[NV], wp[NV];
#pragma unroll
  for (int i = 0; i < NV; ++i)
    if (i * 32 + lane < nv) xp[i] = *reinterpret_cast<const uint4*>(px + (i * 32 + lane) * V);
#pragma unroll
  for (int i = 0; i < NV; ++i)
    if (i * 32 + lane < nv) wp[i] = *reinterpret_cast<const uint4*>(w + (i * 32 + lane) * V);
  float ss = 0.f;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    if (i * 32 + lane < nv) {
      float v[V];
      NIO<T>::load(reinterpret_cast<const T*>(&xp[i]), v);
      if (res_in) {
        float r[V];
        NIO<T>::load(res_in + row * cols + (i * 32 + lane) * V, r);
#pragma unroll
        for (int j = 0; j < V; ++j) v[j] += r[j];
        NIO<T>::store(reinterpret_cast<T*>(&xp[i]), v);
        *reinterpret_cast<uint4*>(res_out + row * cols + (i * 32 + lane) * V) = xp[i];
      }
#pragma unroll
      for (int j = 0; j < V; ++j) ss += v[j] * v[j];
    }
  }
  ss = warp_sum(ss);
  const float rstd = rsqrtf(ss / (float)cols + eps);
  if (lane == 0 && rstd_out) rstd_out[row] = rstd;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    if (i * 32 + lane < nv) {
      float v[V], g[V];
      NIO<T>::load(reinterpret_cast<const T*>(&xp[i]), v);
      NIO<T>::load(reinterpret_cast<const T*>(&wp[i]), g);
#pragma unroll
      for (int j = 0; j < V; ++j) v[j] = v[j] * rstd * g[j];
      NIO<T>::store(y + row * cols + (i * 32 + lane) * V, v);
    }
  }
}

// A block per row while there are fewer rows than SMs (decoding steps): a lane has at most two 16-byte pieces per operand instead of
// sixteen, and the loads of the weight and of the row are one round trip.  32 x 4096: 5.2 us with a warp per
// row, 2.2 us here.  The squares are added in another order than by a warp, so the last bits of a row depend on whether it comes with
// more than 147 others (as between a prompt and the steps that follow it).
template <typename T>
__global__ void __launch_bounds__(NORM_THREADS)
rmsnorm_fwd_row_kernel(const T* __restrict__ x, const T* __restrict__ w, T* __restrict__ y, float* __restrict__ rstd_out, int cols, float eps,
                       const T* __restrict__ res_in, T* __restrict__ res_out) {
  pdl_launch_dependents();
  pdl_wait();
  constexpr int V = NIO<T>::VEC, NV = 2;                  // rows of up to NORM_THREADS * NV vectors
  __shared__ float s_sum[NORM_WARPS];
  const int nv = cols / V;
  const long long base = (long long)blockIdx.x * cols;
  uint4 xp[NV], wp[NV], rp[NV];
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int c = i * NORM_THREADS + threadIdx.x;
    if (c < nv) {
      xp[i] = *reinterpret_cast<const uint4*>(x + base + c * V);
      wp[i] = *reinterpret_cast<const uint4*>(w + c * V);
      if (res_in) rp[i] = *reinterpret_cast<const uint4*>(res_in + base + c * V);
    }
  }
  float ss = 0.f;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int c = i * NORM_THREADS + threadIdx.x;
    if (c < nv) {
      float v[V];
      NIO<T>::load(reinterpret_cast<const T*>(&xp[i]), v);
      if (res_in) {
        float r[V];
        NIO<T>::load(reinterpret_cast<const T*>(&rp[i]), r);
#pragma unroll
        for (int j = 0; j < V; ++j) v[j] += r[j];
        NIO<T>::store(reinterpret_cast<T*>(&xp[i]), v);
        *reinterpret_cast<uint4*>(res_out + base + c * V) = xp[i];
      }
#pragma unroll
      for (int j = 0; j < V; ++j) ss += v[j] * v[j];
    }
  }
  ss = warp_sum(ss);
  if ((threadIdx.x & 31) == 0) s_sum[threadIdx.x >> 5] = ss;
  __syncthreads();
  ss = 0.f;
#pragma unroll
  for (int k = 0; k < NORM_WARPS; ++k) ss += s_sum[k];
  const float rstd = rsqrtf(ss / (float)cols + eps);
  if (threadIdx.x == 0 && rstd_out) rstd_out[blockIdx.x] = rstd;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int c = i * NORM_THREADS + threadIdx.x;
    if (c < nv) {
      float v[V], g[V];
      NIO<T>::load(reinterpret_cast<const T*>(&xp[i]), v);
      NIO<T>::load(reinterpret_cast<const T*>(&wp[i]), g);
#pragma unroll
      for (int j = 0; j < V; ++j) v[j] = v[j] * rstd * g[j];
      NIO<T>::store(y + base + c * V, v);
    }
  }
}

template <typename T>
__global__ void __launch_bounds__(NORM_THREADS)
rmsnorm_fwd_kernel(const T* __restrict__ x, const T* __restrict__ w, T* __restrict__ y, float* __restrict__ rstd_out,
                   long long rows, int cols, float eps, const T* __restrict__ res_in, T* __restrict__ res_out) {
  pdl_launch_dependents();
  pdl_wait();
  constexpr int V = NIO<T>::VEC;
  const int lane = threadIdx.x & 31;
  const long long warp_global = (long long)blockIdx.x * NORM_WARPS + (threadIdx.x >> 5);
  const long long warp_stride = (long long)gridDim.x * NORM_WARPS;
  for (long long row = warp_global; row < rows; row += warp_stride) {
    const T* px = x + row * cols;
    float ss = 0.f;
    for (int c = lane * V; c < cols; c += 32 * V) {
      float v[V];
      NIO<T>::load(px + c, v);
      if (res_in) {
        float r[V];
        NIO<T>::load(res_in + row * cols + c, r);
#pragma unroll
        for (int j = 0; j < V; ++j) v[j] += r[j];
        NIO<T>::store(res_out + row * cols + c, v);
      }
#pragma unroll
      for (int j = 0; j < V; ++j) ss += v[j] * v[j];
    }
    ss = warp_sum(ss);
    float rstd = rsqrtf(ss / (float)cols + eps);
    if (lane == 0 && rstd_out) rstd_out[row] = rstd;
    const T* src = res_in ? res_out + row * cols : px;
    if (res_in) __syncwarp();
    for (int c = lane * V; c < cols; c += 32 * V) {
      float v[V], g[V];
      NIO<T>::load(src + c, v);
      NIO<T>::load(w + c, g);
#pragma unroll
      for (int j = 0; j < V; ++j) v[j] = v[j] * rstd * g[j];
      NIO<T>::store(y + row * cols + c, v);
    }
  }
}

// dx = rstd * (dy*w - xhat * mean(dy*w*xhat)) (+ dres);   dw partial += dy * xhat
template <typename T>
__global__ void __launch_bounds__(NORM_THREADS)
rmsnorm_bwd_kernel(const T* __restrict__ x, const T* __restrict__ w, const T* __restrict__ dy,
                   const float* __restrict__ rstd_in, T* __restrict__ dx, long long rows, int cols,
                   const T* __restrict__ dres, float* __restrict__ partial, int warps_used) {
  pdl_launch_dependents();
  pdl_wait();
  extern __shared__ float s_dw[];  // [warps_used][cols]
  constexpr int V = NIO<T>::VEC;
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  for (int i = threadIdx.x; i < warps_used * cols; i += blockDim.x) s_dw[i] = 0.f;
  __syncthreads();
  if (warp < warps_used) {
    float* my = s_dw + (size_t)warp * cols;
    const long long warp_global = (long long)blockIdx.x * warps_used + warp;
    const long long warp_stride = (long long)gridDim.x * warps_used;
    for (long long row = warp_global; row < rows; row += warp_stride) {
      const T* px = x + row * cols;
      const T* pd = dy + row * cols;
      const float rstd = rstd_in[row];
      float dot = 0.f;
      for (int c = lane * V; c < cols; c += 32 * V) {
        float v[V], d[V], g[V];
        NIO<T>::load(px + c, v);
        NIO<T>::load(pd + c, d);
        NIO<T>::load(w + c, g);
#pragma unroll
        for (int j = 0; j < V; ++j) dot += d[j] * g[j] * v[j] * rstd;
      }
      dot = warp_sum(dot) / (float)cols;
      for (int c = lane * V; c < cols; c += 32 * V) {
        float v[V], d[V], g[V], o[V];
        NIO<T>::load(px + c, v);
        NIO<T>::load(pd + c, d);
        NIO<T>::load(w + c, g);
        if (dres) NIO<T>::load(dres + row * cols + c, o);
#pragma unroll
        for (int j = 0; j < V; ++j) {
          float xh = v[j] * rstd;
          my[c + j] += d[j] * xh;
          float r = rstd * (d[j] * g[j] - xh * dot);
          o[j] = dres ? o[j] + r : r;
        }
        NIO<T>::store(dx + row * cols + c, o);
      }
    }
  }
  __syncthreads();
  for (int c = threadIdx.x; c < cols; c += blockDim.x) {
    float s = 0.f;
    for (int k = 0; k < warps_used; ++k) s += s_dw[(size_t)k * cols + c];
    partial[(size_t)blockIdx.x * cols + c] = s;
  }
}

// bf16 fast path for cols = ITER * 256: a lane always owns the same 8 * ITER columns, so the row stays in registers
// between the two passes (packed bf16), the weight is loaded once, and the dw partial sums live in registers across all
// rows of the warp instead of read-modify-write traffic on shared memory.  Taken while a warp has one row at most and SMs are free: there
// is nothing to fetch ahead, and the ring below is a detour through shared memory (512 x 1024: 4.95 us here, 5.5 us there).
template <int ITER>
__global__ void __launch_bounds__(NORM_THREADS)
rmsnorm_bwd_reg_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ w, const __nv_bfloat16* __restrict__ dy,
                       const float* __restrict__ rstd_in, __nv_bfloat16* __restrict__ dx, long long rows, const __nv_bfloat16* __restrict__ dres,
                       float* __restrict__ partial) {
  pdl_launch_dependents();
  pdl_wait();
  extern __shared__ float s_dw[];  // [NORM_WARPS][cols]
  constexpr int cols = ITER * 256;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint4 wp[ITER];
  float acc[ITER][8];
#pragma unroll
  for (int it = 0; it < ITER; ++it) {
    wp[it] = *reinterpret_cast<const uint4*>(w + it * 256 + lane * 8);
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[it][j] = 0.f;
  }
  const long long warp_global = (long long)blockIdx.x * NORM_WARPS + warp;
  const long long warp_stride = (long long)gridDim.x * NORM_WARPS;
  for (long long row = warp_global; row < rows; row += warp_stride) {
    uint4 xp[ITER], dp[ITER], rp[ITER];
#pragma unroll
    for (int it = 0; it < ITER; ++it) {
      xp[it] = *reinterpret_cast<const uint4*>(x + row * cols + it * 256 + lane * 8);
      dp[it] = *reinterpret_cast<const uint4*>(dy + row * cols + it * 256 + lane * 8);
      if (dres) rp[it] = *reinterpret_cast<const uint4*>(dres + row * cols + it * 256 + lane * 8);
    }
    const float rstd = rstd_in[row];
    float dot = 0.f;
#pragma unroll
    for (int it = 0; it < ITER; ++it) {
      const uint32_t xs[4] = {xp[it].x, xp[it].y, xp[it].z, xp[it].w}, ds[4] = {dp[it].x, dp[it].y, dp[it].z, dp[it].w},
                     ws[4] = {wp[it].x, wp[it].y, wp[it].z, wp[it].w};
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float2 xv = unpack_bf16x2(xs[k]), dv = unpack_bf16x2(ds[k]), wv = unpack_bf16x2(ws[k]);
        dot += dv.x * wv.x * xv.x + dv.y * wv.y * xv.y;
      }
    }
    dot = warp_sum(dot) * rstd / (float)cols;
#pragma unroll
    for (int it = 0; it < ITER; ++it) {
      const uint32_t xs[4] = {xp[it].x, xp[it].y, xp[it].z, xp[it].w}, ds[4] = {dp[it].x, dp[it].y, dp[it].z, dp[it].w},
                     ws[4] = {wp[it].x, wp[it].y, wp[it].z, wp[it].w}, rs[4] = {rp[it].x, rp[it].y, rp[it].z, rp[it].w};
      uint32_t o[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float2 xv = unpack_bf16x2(xs[k]), dv = unpack_bf16x2(ds[k]), wv = unpack_bf16x2(ws[k]);
        const float xh0 = xv.x * rstd, xh1 = xv.y * rstd;
        acc[it][2 * k] += dv.x * xh0;
        acc[it][2 * k + 1] += dv.y * xh1;
        float r0 = rstd * (dv.x * wv.x - xh0 * dot), r1 = rstd * (dv.y * wv.y - xh1 * dot);
        if (dres) { const float2 rv = unpack_bf16x2(rs[k]); r0 += rv.x; r1 += rv.y; }
        o[k] = pack_bf16x2(r0, r1);
      }
      *reinterpret_cast<uint4*>(dx + row * cols + it * 256 + lane * 8) = make_uint4(o[0], o[1], o[2], o[3]);
    }
  }
#pragma unroll
  for (int it = 0; it < ITER; ++it)
#pragma unroll
    for (int j = 0; j < 8; ++j) s_dw[(size_t)warp * cols + it * 256 + lane * 8 + j] = acc[it][j];
  __syncthreads();
  for (int c = threadIdx.x; c < cols; c += blockDim.x) {
    float s = 0.f;
#pragma unroll
    for (int k = 0; k < NORM_WARPS; ++k) s += s_dw[(size_t)k * cols + c];
    partial[(size_t)blockIdx.x * cols + c] = s;
  }
}

__device__ __forceinline__ void cp_async16(void* smem_dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(smem_dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

__device__ __forceinline__ uint4 ld_shared_v4(const uint4* p) {
  uint4 v;
  asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(smem_u32(p)) : "memory");
  return v;
}

// bf16 rows of up to WPR * 256 * NV columns: WPR warps share a row, a lane always owns the same NV * 8 columns, so the weight
// is loaded once and the dw partial sums live in registers across all rows of the warp.  The rows arrive through a ring of
// three rows per warp (two when a residual gradient is read too: 98 KB, two CTAs per SM) filled with cp.async: every lane reads back only what it copied itself, so the ring needs no
// barrier, and the loads of the next rows are in flight while this row's dot product is reduced.
// 16384 x 1024, no residual: 24.0 us with the row loaded when its turn came, 18.8 us (5.4 TB/s) with the ring; 8192 x 2048 with a
// residual: 52.4 -> 20.3 us (the old kernel added its partial sums through shared memory there).
constexpr int RMS_BWD_SMEM_MAX = NORM_WARPS * 6 * 4 * 512;
template <int NV, int WPR>
__global__ void __launch_bounds__(NORM_THREADS, 2)
rmsnorm_bwd_ring_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ w, const __nv_bfloat16* __restrict__ dy,
                        const float* __restrict__ rstd_in, __nv_bfloat16* __restrict__ dx, long long rows, int cols,
                        const __nv_bfloat16* __restrict__ dres, float* __restrict__ partial) {
  pdl_launch_dependents();
  pdl_wait();
  constexpr int GROUPS = NORM_WARPS / WPR;
  extern __shared__ __align__(16) unsigned char s_raw[];   // ring, then reused as [GROUPS][cols] floats
  __shared__ float s_dot[2][NORM_WARPS];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int group = warp / WPR, part = warp % WPR;
  const int nv = cols >> 3;
  const int v0 = part * NV * 32 + lane;                    // this lane's vectors: v0 + 32 i
  const int streams = dres ? 3 : 2, stages = dres ? 2 : 3;
  uint4* ring = reinterpret_cast<uint4*>(s_raw) + (size_t)warp * stages * streams * NV * 32;
  uint4 wp[NV];
  float acc[NV][8];
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    wp[i] = make_uint4(0, 0, 0, 0);
    if (v0 + 32 * i < nv) wp[i] = *reinterpret_cast<const uint4*>(w + (v0 + 32 * i) * 8);
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[i][j] = 0.f;
  }
  const long long first = (long long)blockIdx.x * GROUPS + group, stride = (long long)gridDim.x * GROUPS;
  auto fetch = [&](long long row, int st) {
    if (row < rows) {
      uint4* d = ring + (size_t)st * streams * NV * 32 + lane;
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        if (v0 + 32 * i < nv) {
          const long long at = row * cols + (v0 + 32 * i) * 8;
          cp_async16(d + i * 32, x + at);
          cp_async16(d + (NV + i) * 32, dy + at);
          if (dres) cp_async16(d + (2 * NV + i) * 32, dres + at);
        }
      }
    }
    cp_async_commit();
  };
  for (int s = 0; s < stages; ++s) fetch(first + s * stride, s);
  float rstd = first < rows ? rstd_in[first] : 0.f;
  int st = 0, par = 0;
  for (long long row = first; row < rows; row += stride) {
    const float rstd_next = row + stride < rows ? rstd_in[row + stride] : 0.f;
    if (dres) cp_async_wait<1>();
    else cp_async_wait<2>();
    const uint4* d = ring + (size_t)st * streams * NV * 32 + lane;
    float dot = 0.f;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      if (v0 + 32 * i >= nv) continue;
      const uint4 xp = ld_shared_v4(d + i * 32), dp = ld_shared_v4(d + (NV + i) * 32);
      const uint32_t xs[4] = {xp.x, xp.y, xp.z, xp.w}, ds[4] = {dp.x, dp.y, dp.z, dp.w},
                     ws[4] = {wp[i].x, wp[i].y, wp[i].z, wp[i].w};
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float2 xv = unpack_bf16x2(xs[k]), dv = unpack_bf16x2(ds[k]), wv = unpack_bf16x2(ws[k]);
        dot += dv.x * wv.x * xv.x + dv.y * wv.y * xv.y;
      }
    }
    dot = warp_sum(dot);
    if (WPR > 1) {                                         // the row's other warps; two slots, so one barrier per row is enough
      if (lane == 0) s_dot[par][warp] = dot;
      asm volatile("bar.sync %0, %1;" ::"r"(group + 1), "n"(WPR * 32) : "memory");
      dot = 0.f;
#pragma unroll
      for (int k = 0; k < WPR; ++k) dot += s_dot[par][group * WPR + k];
      par ^= 1;
    }
    dot = dot * rstd / (float)cols;
    // read the row from the ring again: keeping it unpacked across the reduction spills at four vectors a lane
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      if (v0 + 32 * i >= nv) continue;
      const uint4 xp = ld_shared_v4(d + i * 32), dp = ld_shared_v4(d + (NV + i) * 32);
      const uint4 rp = dres ? ld_shared_v4(d + (2 * NV + i) * 32) : make_uint4(0, 0, 0, 0);
      const uint32_t xs[4] = {xp.x, xp.y, xp.z, xp.w}, ds[4] = {dp.x, dp.y, dp.z, dp.w},
                     ws[4] = {wp[i].x, wp[i].y, wp[i].z, wp[i].w}, rs[4] = {rp.x, rp.y, rp.z, rp.w};
      uint32_t o[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float2 xv = unpack_bf16x2(xs[k]), dv = unpack_bf16x2(ds[k]), wv = unpack_bf16x2(ws[k]);
        const float xh0 = xv.x * rstd, xh1 = xv.y * rstd;
        acc[i][2 * k] += dv.x * xh0;
        acc[i][2 * k + 1] += dv.y * xh1;
        float r0 = rstd * (dv.x * wv.x - xh0 * dot), r1 = rstd * (dv.y * wv.y - xh1 * dot);
        if (dres) { const float2 rv = unpack_bf16x2(rs[k]); r0 += rv.x; r1 += rv.y; }
        o[k] = pack_bf16x2(r0, r1);
      }
      *reinterpret_cast<uint4*>(dx + row * cols + (v0 + 32 * i) * 8) = make_uint4(o[0], o[1], o[2], o[3]);
    }
    fetch(row + stages * stride, st);              // the stage has been read and used above
    st = st + 1 == stages ? 0 : st + 1;
    rstd = rstd_next;
  }
  cp_async_wait<0>();
  __syncthreads();                                         // the ring is free: it becomes the dw staging
  float* s_dw = reinterpret_cast<float*>(s_raw);
#pragma unroll
  for (int i = 0; i < NV; ++i)
    if (v0 + 32 * i < nv) {
      float4* t = reinterpret_cast<float4*>(s_dw + (size_t)group * cols + (v0 + 32 * i) * 8);
      t[0] = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
      t[1] = make_float4(acc[i][4], acc[i][5], acc[i][6], acc[i][7]);
    }
  __syncthreads();
  for (int c = threadIdx.x; c < cols; c += blockDim.x) {
    float s = 0.f;
#pragma unroll
    for (int k = 0; k < GROUPS; ++k) s += s_dw[(size_t)k * cols + c];
    partial[(size_t)blockIdx.x * cols + c] = s;
  }
}

template <typename T>
__global__ void __launch_bounds__(NORM_THREADS)
layernorm_fwd_kernel(const T* __restrict__ x, const T* __restrict__ w, const T* __restrict__ b, T* __restrict__ y,
                     float* __restrict__ mean_out, float* __restrict__ rstd_out, long long rows, int cols, float eps) {
  pdl_wait();
  constexpr int V = NIO<T>::VEC;
  const int lane = threadIdx.x & 31;
  const long long warp_global = (long long)blockIdx.x * NORM_WARPS + (threadIdx.x >> 5);
  const long long warp_stride = (long long)gridDim.x * NORM_WARPS;
  for (long long row = warp_global; row < rows; row += warp_stride) {
    const T* px = x + row * cols;
    float s = 0.f;
    for (int c = lane * V; c < cols; c += 32 * V) {
      float v[V];
      NIO<T>::load(px + c, v);
#pragma unroll
      for (int j = 0; j < V; ++j) s += v[j];
    }
    float mean = warp_sum(s) / (float)cols;
    float ss = 0.f;
    for (int c = lane * V; c < cols; c += 32 * V) {
      float v[V];
      NIO<T>::load(px + c, v);
#pragma unroll
      for (int j = 0; j < V; ++j) ss += (v[j] - mean) * (v[j] - mean);
    }
    float rstd = rsqrtf(warp_sum(ss) / (float)cols + eps);
    if (lane == 0) {
      if (mean_out) mean_out[row] = mean;
      if (rstd_out) rstd_out[row] = rstd;
    }
    for (int c = lane * V; c < cols; c += 32 * V) {
      float v[V], g[V], bb[V];
      NIO<T>::load(px + c, v);
      NIO<T>::load(w + c, g);
      if (b) NIO<T>::load(b + c, bb);
#pragma unroll
      for (int j = 0; j < V; ++j) v[j] = (v[j] - mean) * rstd * g[j] + (b ? bb[j] : 0.f);
      NIO<T>::store(y + row * cols + c, v);
    }
  }
}

// dx = rstd * (g - mean(g) - xhat * mean(g * xhat)) with g = dy * w;  dw += dy * xhat;  db += dy
template <typename T>
__global__ void __launch_bounds__(NORM_THREADS)
layernorm_bwd_kernel(const T* __restrict__ x, const T* __restrict__ w, const T* __restrict__ dy,
                     const float* __restrict__ mean_in, const float* __restrict__ rstd_in, T* __restrict__ dx,
                     long long rows, int cols, const T* __restrict__ dres, float* __restrict__ partial, int warps_used, int nblocks_total) {
  extern __shared__ float s_acc[];  // [warps_used][2][cols]
  constexpr int V = NIO<T>::VEC;
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  for (int i = threadIdx.x; i < warps_used * 2 * cols; i += blockDim.x) s_acc[i] = 0.f;
  __syncthreads();
  pdl_wait();
  if (warp < warps_used) {
    float* my_dw = s_acc + (size_t)warp * 2 * cols;
    float* my_db = my_dw + cols;
    const long long warp_global = (long long)blockIdx.x * warps_used + warp;
    const long long warp_stride = (long long)gridDim.x * warps_used;
    for (long long row = warp_global; row < rows; row += warp_stride) {
      const T* px = x + row * cols;
      const T* pd = dy + row * cols;
      const float mean = mean_in[row], rstd = rstd_in[row];
      float sg = 0.f, sgx = 0.f;
      for (int c = lane * V; c < cols; c += 32 * V) {
        float v[V], d[V], g[V];
        NIO<T>::load(px + c, v);
        NIO<T>::load(pd + c, d);
        NIO<T>::load(w + c, g);
#pragma unroll
        for (int j = 0; j < V; ++j) {
          float gg = d[j] * g[j];
          sg += gg;
          sgx += gg * (v[j] - mean) * rstd;
        }
      }
      sg = warp_sum(sg) / (float)cols;
      sgx = warp_sum(sgx) / (float)cols;
      for (int c = lane * V; c < cols; c += 32 * V) {
        float v[V], d[V], g[V], o[V];
        NIO<T>::load(px + c, v);
        NIO<T>::load(pd + c, d);
        NIO<T>::load(w + c, g);
#pragma unroll
        for (int j = 0; j < V; ++j) {
          float xh = (v[j] - mean) * rstd;
          my_dw[c + j] += d[j] * xh;
          my_db[c + j] += d[j];
          o[j] = rstd * (d[j] * g[j] - sg - xh * sgx);
        }
        if (dres) {                                  // what x has collected through the residual stream
          float q[V];
          NIO<T>::load(dres + row * cols + c, q);
#pragma unroll
          for (int j = 0; j < V; ++j) o[j] += q[j];
        }
        NIO<T>::store(dx + row * cols + c, o);
      }
    }
  }
  __syncthreads();
  for (int c = threadIdx.x; c < cols; c += blockDim.x) {
    float s0 = 0.f, s1 = 0.f;
    for (int k = 0; k < warps_used; ++k) {
      s0 += s_acc[(size_t)k * 2 * cols + c];
      s1 += s_acc[(size_t)k * 2 * cols + cols + c];
    }
    partial[(size_t)blockIdx.x * cols + c] = s0;
    partial[((size_t)nblocks_total + blockIdx.x) * cols + c] = s1;
  }
}

// out[c] (+)= sum_p partial[p, c]: 32 columns x 32 row groups per CTA, shared-memory reduce over the groups.  With 296 partial
// rows a thread adds about nine loads; eight row groups made it 37 dependent ones.  Up to PSUM_FEW partial rows eight groups do.
constexpr int PSUM_FEW = 64;
template <typename D, int THREADS>
__global__ void __launch_bounds__(THREADS)
partial_rows_sum_kernel(const float* __restrict__ partial, D* __restrict__ out, D* __restrict__ out2, int nparts, int cols, int accumulate) {
  pdl_launch_dependents();
  pdl_wait();
  if (blockIdx.y) { partial += (size_t)nparts * cols; out = out2; }      // a second set of sums, behind the first
  constexpr int NG = THREADS / 32;
  __shared__ float red[NG][33];
  const int cx = threadIdx.x & 31, ry = threadIdx.x >> 5;
  const int c = blockIdx.x * 32 + cx;
  float s = 0.f;
  if (c < cols)
    for (int p = ry; p < nparts; p += NG) s += partial[(size_t)p * cols + c];
  red[ry][cx] = s;
  __syncthreads();
  if (ry == 0 && c < cols) {
    float t = 0.f;
#pragma unroll
    for (int k = 0; k < NG; ++k) t += red[k][cx];
    if constexpr (sizeof(D) == 4) {
      if (accumulate) t += out[c];
      out[c] = t;
    } else {
      if (accumulate) t += __bfloat162float(out[c]);
      out[c] = __float2bfloat16_rn(t);
    }
  }
}

static int norm_bwd_blocks(long long rows) {
  long long b = (rows + NORM_WARPS - 1) / NORM_WARPS;
  if (b > 148 * 2) b = 148 * 2;
  if (b < 1) b = 1;
  return (int)b;
}

}  // namespace oa

using namespace oa;
#define ST ((cudaStream_t)stream)
#define CHECK_LAUNCH() (cudaGetLastError() == cudaSuccess ? OA_OK : OA_ERR_LAUNCH)

// Scratch for the weight (and bias) gradient partial rows: float[2 * blocks * cols].
extern "C" size_t oa_norm_bwd_scratch_bytes(long long rows, int cols) {
  return (size_t)2 * norm_bwd_blocks(rows) * cols * sizeof(float);
}

// Whether the row-in-registers kernel beats the two passes, by the 16-byte vectors per lane (nv) and the blocks of eight rows.  Up to
// one block per SM it is latency that counts and registers win at any width.  Beyond, two passes against registers: 9472 x 1536 bf16
// 9.1 / 9.7 us (nv 6), 16384 x 1024 fp32 24.2 / 20.2 (8), 2368 x 4096 bf16 7.4 / 8.2 (16); with a residual 16384 x 1024 23.1 / 24.5 (4), 4736 x 1536 7.4 / 8.2 (6),
// 1200 x 2880 8.1 / 10.9 (12).
static bool rmsnorm_in_registers(int nv, long long blocks, bool residual) {
  if (nv <= 2) return true;
  if (nv <= 4) return !residual || blocks <= 8 * 148;
  if (nv <= 8) return residual ? blocks <= 2 * 148 : (nv > 6 || blocks <= 7 * 148);
  return nv <= 16 && blocks <= 148;
}

extern "C" int oa_rmsnorm_fwd(int dtype, const void* x, const void* w, void* y, float* rstd, long long rows, int cols,
                              float eps, const void* residual_in, void* residual_out, void* stream) {
  if (rows <= 0) return OA_OK;
  if (cols % 8) return OA_ERR_ALIGN;
  const int vec = dtype == OA_F32 ? 4 : 8;
  const uintptr_t at = reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(y) |
                       reinterpret_cast<uintptr_t>(residual_in) | reinterpret_cast<uintptr_t>(residual_out);
  if (dtype != OA_F32 && dtype != OA_BF16) return OA_ERR_UNSUPPORTED;
  long long b = (rows + NORM_WARPS - 1) / NORM_WARPS;
  const int nv = (cols + 32 * vec - 1) / (32 * vec);
  if ((at & 15) == 0 && rows <= 148 && nv > 2 && cols / vec <= 2 * NORM_THREADS) {
    if (dtype == OA_F32)
      launch_short(rmsnorm_fwd_row_kernel<float>, dim3((unsigned)rows), dim3(NORM_THREADS), 0, ST, (const float*)x, (const float*)w, (float*)y, rstd, cols, eps,
                 (const float*)residual_in, (float*)residual_out);
    else
      launch_short(rmsnorm_fwd_row_kernel<__nv_bfloat16>, dim3((unsigned)rows), dim3(NORM_THREADS), 0, ST, (const __nv_bfloat16*)x, (const __nv_bfloat16*)w,
                 (__nv_bfloat16*)y, rstd, cols, eps, (const __nv_bfloat16*)residual_in, (__nv_bfloat16*)residual_out);
    return CHECK_LAUNCH();
  }
  if (rmsnorm_in_registers(nv, b, residual_in != nullptr) && (at & 15) == 0 && b < 0x7fffffffLL) {
#define OA_RMS_FWD_REG(T, NV)                                                                                                   \
    launch_pdl(rmsnorm_fwd_reg_kernel<T, NV>, dim3((unsigned)b), dim3(NORM_THREADS), 0, ST, (const T*)x, (const T*)w, (T*)y, rstd, \
               rows, cols, eps, (const T*)residual_in, (T*)residual_out)
#define OA_RMS_FWD_PICK(T)                                 \
    if (nv <= 1) OA_RMS_FWD_REG(T, 1);                     \
    else if (nv <= 2) OA_RMS_FWD_REG(T, 2);                \
    else if (nv <= 4) OA_RMS_FWD_REG(T, 4);                \
    else if (nv <= 8) OA_RMS_FWD_REG(T, 8);                \
    else OA_RMS_FWD_REG(T, 16)
    if (dtype == OA_F32) { OA_RMS_FWD_PICK(float); }
    else { OA_RMS_FWD_PICK(__nv_bfloat16); }
#undef OA_RMS_FWD_PICK
#undef OA_RMS_FWD_REG
    return CHECK_LAUNCH();
  }
  if (b > 148 * 8) b = 148 * 8;
  if (dtype == OA_F32)
    rmsnorm_fwd_kernel<float><<<(int)b, NORM_THREADS, 0, ST>>>((const float*)x, (const float*)w, (float*)y, rstd, rows, cols, eps, (const float*)residual_in, (float*)residual_out);
  else
    launch_pdl(rmsnorm_fwd_kernel<__nv_bfloat16>, dim3((unsigned)b), dim3(NORM_THREADS), 0, ST, (const __nv_bfloat16*)x, (const __nv_bfloat16*)w, (__nv_bfloat16*)y, rstd, rows, cols, eps, (const __nv_bfloat16*)residual_in, (__nv_bfloat16*)residual_out);
  return CHECK_LAUNCH();
}

template <typename K>
static int set_smem(K kernel, size_t bytes) {
  if (bytes > 48 * 1024) {
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) != cudaSuccess) return OA_ERR_LAUNCH;
  }
  return OA_OK;
}

// One launch for both of LayerNorm's sums (second set in blockIdx.y): at 1000 x 128 a sum is 2.4-2.9 us of launch and of one pass over
// the partial rows, for each of nine norms.  With the pending gradient added in the kernel above it (an add of 3.4 us less for
// eight of them) a character model's step of 954 us takes 926.
static void partial_rows_sum(const float* partial, void* out, void* out2, int out_dtype, int nparts, int cols, int accumulate, cudaStream_t st) {
  const dim3 grid((cols + 31) / 32, out2 ? 2 : 1);
#define OA_PSUM(D, THREADS) launch_short(partial_rows_sum_kernel<D, THREADS>, grid, dim3(THREADS), 0, st, partial, (D*)out, (D*)out2, nparts, cols, accumulate)
  if (out_dtype == OA_F32) {
    if (nparts <= PSUM_FEW) OA_PSUM(float, 256);
    else OA_PSUM(float, 1024);
  } else {
    if (nparts <= PSUM_FEW) OA_PSUM(__nv_bfloat16, 256);
    else OA_PSUM(__nv_bfloat16, 1024);
  }
#undef OA_PSUM
}

extern "C" int oa_rmsnorm_bwd(int dtype, const void* x, const void* w, const void* dy, const float* rstd, void* dx,
                              void* dw, int dw_dtype, long long rows, int cols, const void* dres, float* scratch,
                              int accumulate_dw, void* stream) {
  if (rows <= 0) return OA_OK;
  if (cols % 8) return OA_ERR_ALIGN;
  int warps = NORM_WARPS;
  while (warps > 1 && (size_t)warps * cols * 4 > 200 * 1024) warps >>= 1;
  size_t smem = (size_t)warps * cols * 4;
  if (smem > 200 * 1024) return OA_ERR_TOO_LARGE;
  int blocks = norm_bwd_blocks(rows);
  int rc;
  if (dtype == OA_F32) {
    if ((rc = set_smem(rmsnorm_bwd_kernel<float>, smem))) return rc;
    rmsnorm_bwd_kernel<float><<<blocks, NORM_THREADS, smem, ST>>>((const float*)x, (const float*)w, (const float*)dy, rstd, (float*)dx, rows, cols, (const float*)dres, scratch, warps);
  } else if (dtype == OA_BF16 && cols <= 4096 &&
             ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(dy) | reinterpret_cast<uintptr_t>(dx) | reinterpret_cast<uintptr_t>(w) |
               reinterpret_cast<uintptr_t>(dres)) & 15) == 0) {
    const __nv_bfloat16 *bx = (const __nv_bfloat16*)x, *bw = (const __nv_bfloat16*)w, *bd = (const __nv_bfloat16*)dy, *br = (const __nv_bfloat16*)dres;
    __nv_bfloat16* bo = (__nv_bfloat16*)dx;
#define OA_RMS_BWD_REG(IT)                                                                          \
    launch_pdl(rmsnorm_bwd_reg_kernel<IT>, dim3(blocks), dim3(NORM_THREADS), smem, ST, bx, bw, bd, rstd, bo, rows, br, scratch)
    // a lane carries at most four 8-column vectors (32 partial sums): wider rows are shared by two or four warps
    const int wpr = cols <= 1024 ? 1 : cols <= 2048 ? 2 : 4;
    const int nv = (cols + wpr * 256 - 1) / (wpr * 256);
    const size_t ring = (size_t)NORM_WARPS * 6 * nv * 512, stage = (size_t)(NORM_WARPS / wpr) * cols * 4;
    const size_t rsm = ring > stage ? ring : stage;
#define OA_RMS_BWD_RING(NV, WPR)                                                                                               \
    {                                                                                                                         \
      if ((rc = set_smem(rmsnorm_bwd_ring_kernel<NV, WPR>, RMS_BWD_SMEM_MAX))) return rc;                                                  \
      launch_pdl(rmsnorm_bwd_ring_kernel<NV, WPR>, dim3(blocks), dim3(NORM_THREADS), rsm, ST, bx, bw, bd, rstd, bo, rows, cols, br, scratch); \
    }
    if (blocks <= 148 && cols % 256 == 0 && cols <= 1024) {
      if (nv == 1) OA_RMS_BWD_REG(1);
      else if (nv == 2) OA_RMS_BWD_REG(2);
      else if (nv == 3) OA_RMS_BWD_REG(3);
      else OA_RMS_BWD_REG(4);
    }
    else if (wpr == 4) { if (nv == 3) OA_RMS_BWD_RING(3, 4) else OA_RMS_BWD_RING(4, 4) }
    else if (wpr == 2) { if (nv == 3) OA_RMS_BWD_RING(3, 2) else OA_RMS_BWD_RING(4, 2) }
    else if (nv == 1) OA_RMS_BWD_RING(1, 1)
    else if (nv == 2) OA_RMS_BWD_RING(2, 1)
    else if (nv == 3) OA_RMS_BWD_RING(3, 1)
    else OA_RMS_BWD_RING(4, 1)
#undef OA_RMS_BWD_RING
#undef OA_RMS_BWD_REG
  } else if (dtype == OA_BF16) {
    if ((rc = set_smem(rmsnorm_bwd_kernel<__nv_bfloat16>, smem))) return rc;
    rmsnorm_bwd_kernel<__nv_bfloat16><<<blocks, NORM_THREADS, smem, ST>>>((const __nv_bfloat16*)x, (const __nv_bfloat16*)w, (const __nv_bfloat16*)dy, rstd, (__nv_bfloat16*)dx, rows, cols, (const __nv_bfloat16*)dres, scratch, warps);
  } else return OA_ERR_UNSUPPORTED;
  if (dw) partial_rows_sum(scratch, dw, nullptr, dw_dtype, blocks, cols, accumulate_dw, ST);
  return CHECK_LAUNCH();
}

extern "C" int oa_layernorm_fwd(int dtype, const void* x, const void* w, const void* b, void* y, float* mean,
                                float* rstd, long long rows, int cols, float eps, void* stream) {
  if (rows <= 0) return OA_OK;
  if (cols % 8) return OA_ERR_ALIGN;
  long long nb = (rows + NORM_WARPS - 1) / NORM_WARPS;
  if (nb > 148 * 8) nb = 148 * 8;
  if (dtype == OA_F32)
    launch_short(layernorm_fwd_kernel<float>, dim3((unsigned)nb), dim3(NORM_THREADS), 0, ST, (const float*)x, (const float*)w, (const float*)b, (float*)y, mean, rstd, rows, cols, eps);
  else if (dtype == OA_BF16)
    launch_short(layernorm_fwd_kernel<__nv_bfloat16>, dim3((unsigned)nb), dim3(NORM_THREADS), 0, ST, (const __nv_bfloat16*)x, (const __nv_bfloat16*)w, (const __nv_bfloat16*)b, (__nv_bfloat16*)y, mean, rstd, rows, cols, eps);
  else return OA_ERR_UNSUPPORTED;
  return CHECK_LAUNCH();
}

extern "C" int oa_layernorm_bwd(int dtype, const void* x, const void* w, const void* dy, const float* mean,
                                const float* rstd, void* dx, void* dw, void* db, int dw_dtype, long long rows, int cols, const void* dres,
                                float* scratch, int accumulate_dw, void* stream) {
  if (rows <= 0) return OA_OK;
  if (cols % 8) return OA_ERR_ALIGN;
  int warps = NORM_WARPS;
  while (warps > 1 && (size_t)warps * 2 * cols * 4 > 200 * 1024) warps >>= 1;
  size_t smem = (size_t)warps * 2 * cols * 4;
  if (smem > 200 * 1024) return OA_ERR_TOO_LARGE;
  int blocks = norm_bwd_blocks(rows);
  int rc;
  if (dtype == OA_F32) {
    if ((rc = set_smem(layernorm_bwd_kernel<float>, smem))) return rc;
    launch_short(layernorm_bwd_kernel<float>, dim3(blocks), dim3(NORM_THREADS), smem, ST, (const float*)x, (const float*)w, (const float*)dy, mean, rstd, (float*)dx, rows, cols, (const float*)dres, scratch, warps, blocks);
  } else if (dtype == OA_BF16) {
    if ((rc = set_smem(layernorm_bwd_kernel<__nv_bfloat16>, smem))) return rc;
    launch_short(layernorm_bwd_kernel<__nv_bfloat16>, dim3(blocks), dim3(NORM_THREADS), smem, ST, (const __nv_bfloat16*)x, (const __nv_bfloat16*)w, (const __nv_bfloat16*)dy, mean, rstd, (__nv_bfloat16*)dx, rows, cols, (const __nv_bfloat16*)dres, scratch, warps, blocks);
  } else return OA_ERR_UNSUPPORTED;
  if (dw) partial_rows_sum(scratch, dw, db, dw_dtype, blocks, cols, accumulate_dw, ST);
  else if (db) partial_rows_sum(scratch + (size_t)blocks * cols, db, nullptr, dw_dtype, blocks, cols, accumulate_dw, ST);
  return CHECK_LAUNCH();
}
