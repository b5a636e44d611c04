// Fused softmax cross-entropy: per-row fp32 loss (lse - logit[target]) and, in the same kernel,
// the logits gradient (softmax - onehot) * grad_scale, optionally written over the logits.
// An out-of-range target gives a NaN row loss instead of an out-of-bounds read, and a target
// equal to `ignore_index` gives loss 0 and a zero gradient row (masked cross-entropy).
// Reference semantics: Source/Private/Oa/Ml/Shader/Compute/Nn/CrossEntropy/CrossEntropy.slang:58-75,
// CrossEntropyBwd.slang:69-78 and the fused CrossEntropyLossGradBwd registry entry.
#include <cfloat>
#include "common.cuh"
#include "api.h"

namespace oa {

template <typename T> struct XIO;
template <> struct XIO<float> {
  static constexpr int VEC = 4;
  __device__ static void load(const float* p, float* v) {
    float4 x = *reinterpret_cast<const float4*>(p);
    v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
  }
  __device__ static void store(float* p, const float* v) { *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]); }
  __device__ static float ld1(const float* p) { return *p; }
};
template <> struct XIO<__nv_bfloat16> {
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
  __device__ static float ld1(const __nv_bfloat16* p) { return __bfloat162float(*p); }
};

constexpr int XENT_THREADS = 256;

template <typename T>
__global__ void __launch_bounds__(XENT_THREADS)
xent_kernel(const T* __restrict__ logits, const int* __restrict__ targets, float* __restrict__ row_loss, T* dlogits,
            int vocab, int ld, float grad_scale, int ignore_index, int vec_ok) {
  constexpr int V = XIO<T>::VEC;
  __shared__ float red_m[XENT_THREADS / 32], red_s[XENT_THREADS / 32];
  const long long row = blockIdx.x;
  const T* p = logits + row * ld;
  const int tgt = targets[row];
  const int nvec = vec_ok ? vocab / V : 0;        // rows that do not start on a 16-byte boundary take the scalar loops
  const bool ignored = (tgt == ignore_index);
  const bool oor = !ignored && (tgt < 0 || tgt >= vocab);
  // read before any thread can overwrite the logits with the gradient (dlogits may alias logits)
  const float tgt_logit = (threadIdx.x == 0 && !ignored && !oor) ? XIO<T>::ld1(p + tgt) : 0.f;
  float m = -FLT_MAX, s = 0.f;                     // finite: a masked logit (-inf) adds exp(-inf) = 0 whatever came before it
  for (int i = threadIdx.x; i < nvec; i += XENT_THREADS) {
    float v[V];
    XIO<T>::load(p + i * V, v);
    float mx = v[0];
#pragma unroll
    for (int j = 1; j < V; ++j) mx = fmaxf(mx, v[j]);
    if (mx > m) { s *= __expf(m - mx); m = mx; }
#pragma unroll
    for (int j = 0; j < V; ++j) s += __expf(v[j] - m);
  }
  for (int c = nvec * V + threadIdx.x; c < vocab; c += XENT_THREADS) {
    float v = XIO<T>::ld1(p + c);
    if (v > m) { s *= __expf(m - v); m = v; }
    s += __expf(v - m);
  }
  // block combine of (m, s)
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    float om = __shfl_xor_sync(0xffffffffu, m, o), os = __shfl_xor_sync(0xffffffffu, s, o);
    float nm = fmaxf(m, om);
    s = s * __expf(m - nm) + os * __expf(om - nm);
    m = nm;
  }
  if ((threadIdx.x & 31) == 0) { red_m[threadIdx.x >> 5] = m; red_s[threadIdx.x >> 5] = s; }
  __syncthreads();
  m = red_m[0]; s = red_s[0];
#pragma unroll
  for (int w = 1; w < XENT_THREADS / 32; ++w) {
    float om = red_m[w], os = red_s[w];
    float nm = fmaxf(m, om);
    s = s * __expf(m - nm) + os * __expf(om - nm);
    m = nm;
  }
  const float lse = m + logf(s);
  if (threadIdx.x == 0) {
    float l = ignored ? 0.f : (oor ? __int_as_float(0x7fc00000) : lse - tgt_logit);
    row_loss[row] = l;
  }
  if (!dlogits) return;
  T* d = dlogits + row * ld;
  const float gs = ignored ? 0.f : grad_scale;
  for (int i = threadIdx.x; i < nvec; i += XENT_THREADS) {
    float v[V];
    XIO<T>::load(p + i * V, v);
#pragma unroll
    for (int j = 0; j < V; ++j) {
      float pr = __expf(v[j] - lse);
      v[j] = (pr - ((i * V + j) == tgt ? 1.f : 0.f)) * gs;
    }
    XIO<T>::store(d + i * V, v);
  }
  for (int c = nvec * V + threadIdx.x; c < vocab; c += XENT_THREADS) {
    float pr = __expf(XIO<T>::ld1(p + c) - lse);
    float g = (pr - (c == tgt ? 1.f : 0.f)) * gs;
    if constexpr (sizeof(T) == 4) d[c] = g; else d[c] = __float2bfloat16_rn(g);
  }
}

// The same with the row kept on the chip, so that the logits are read once.  Rows of up to XENT_SMEM_MAX bytes: the row goes
// to shared memory through cp.async; every thread reads back only the 16-byte vectors that it copied itself, so no barrier
// stands between the copy and its use, and the gradient can be written over the logits.  A thread takes the exponentials of its vectors
// against a maximum of its own, in one pass.  What bounds it: one read and one write of the logits, beside the exponentials (two to a logit,
// 230 us of 16384 x 32000 by themselves) and the instructions around them, of which few are left: with a subtraction, a product and the other
// steps one element at a time they were 177 per 8 logits and the issue slots 82 % taken.  The CTAs of an SM (three at 64,000-byte rows) cover
// one another's waits; with the copy in four groups, each worked on as it landed, rows took longer (the figures below), short ones and fp32 most.
// us, two passes over the row on the chip one element at a time / one pass, packed, in four groups / now: 16384 x 32000 bf16 401 / 357 / 332 (6.3 TB/s;
// 475 with two reads of the logits), 8192 x 50264 338 / 302 / 300, 32768 x 8192 209 / 175 / 165, 16384 x 4096 65 / 60 / 52, 500 x 32000 19.6 / 18.6 / 16.5; fp32
// 4096 x 16384 83.3 / 83.9 / 82.5, 8192 x 2048 24.7 / 26.8 / 22.7, 2048 x 5000 14.6 / 16.5 / 14.5.
// A quarter of the exponentials on the multiply-add pipe made it slower (382 -> 406).
// Errors against 64 bits, standard deviation 2, subtraction first and probabilities from the rounded log-sum-exp / now: fp32 gradients over
// 4096 columns 3.3e-7 / 1.3e-7, over 32000 3.8e-7 / 1.7e-7; losses 4.6e-7 / 4.2e-7.  With a product of m and log2(e) rounded into every term the
// gradients were at 5.5e-7, and wrong far from zero.
__device__ __forceinline__ void xent_cp16(void* smem_dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(smem_dst)), "l"(src) : "memory");
}
constexpr int XENT_SMEM_MAX = 200 * 1024;
constexpr float XENT_LOG2E = 1.4426950408889634f;

template <typename T> __device__ __forceinline__ float xent_vec_max(const T* p);
template <> __device__ __forceinline__ float xent_vec_max<float>(const float* p) {
  const float4 x = *reinterpret_cast<const float4*>(p);
  return fmaxf(fmaxf(x.x, x.y), fmaxf(x.z, x.w));
}
template <> __device__ __forceinline__ float xent_vec_max<__nv_bfloat16>(const __nv_bfloat16* p) {
  const uint4 x = *reinterpret_cast<const uint4*>(p);
  const __nv_bfloat162 *a = reinterpret_cast<const __nv_bfloat162*>(&x);
  const float2 m = __bfloat1622float2(__hmax2(__hmax2(a[0], a[1]), __hmax2(a[2], a[3])));
  return fmaxf(m.x, m.y);
}

// (softmax - onehot) * gs of one vector; `hit` = position of the target inside it, or a value outside [0, VEC)
template <typename T>
__device__ __forceinline__ void xent_vec_grad(const T* src, T* dst, float lse, float gs, int hit) {
  constexpr int V = XIO<T>::VEC;
  float v[V];
  XIO<T>::load(src, v);
  const unsigned long long nl = f2_of(__float_as_uint(-lse), __float_as_uint(-lse)), l2 = f2_of(__float_as_uint(XENT_LOG2E), __float_as_uint(XENT_LOG2E));
#pragma unroll
  for (int j = 0; j < V; j += 2) {
    uint32_t a, b;
    f2_to(f2_mul(f2_add(f2_of(__float_as_uint(v[j]), __float_as_uint(v[j + 1])), nl), l2), a, b);
    v[j] = fast_exp2(__uint_as_float(a));
    v[j + 1] = fast_exp2(__uint_as_float(b));
  }
  if ((unsigned)hit < (unsigned)V) {
#pragma unroll
    for (int j = 0; j < V; ++j) v[j] -= j == hit ? 1.f : 0.f;
  }
#pragma unroll
  for (int j = 0; j < V; ++j) v[j] *= gs;
  XIO<T>::store(dst, v);
}

// The vector's elements as fp32 pairs
__device__ __forceinline__ void xent_pairs(const float* p, unsigned long long* v) {
  const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(p);
  v[0] = x.x; v[1] = x.y;
}
__device__ __forceinline__ void xent_pairs(const __nv_bfloat16* p, unsigned long long* v) {
  const uint4 x = *reinterpret_cast<const uint4*>(p);
  v[0] = f2_bf16x2(x.x); v[1] = f2_bf16x2(x.y); v[2] = f2_bf16x2(x.z); v[3] = f2_bf16x2(x.w);
}
__device__ __forceinline__ unsigned long long xent_splat(float v) { return f2_of(__float_as_uint(v), __float_as_uint(v)); }
// 2^(v log2(e) + b): one multiply-add where a subtraction and a product stood.  b is the whole number beside -m log2(e): a row's terms pass
// from one maximum to another, and from threads to the row, by powers of two, and nothing is lost on the way.  A probability is a term over
// the sum of terms, whatever b is; the loss, which needs the sum as it counts from m, is given what lies between (xent_rest).
// Rows whose maximum lies beyond XENT_WIDE either way are worked out apart (xent_wide_row), by subtraction: far out, the product is
// rounded to more than a whole number.
__device__ __forceinline__ unsigned long long xent_exp2(unsigned long long v, unsigned long long b) {
  uint32_t x0, x1;
  f2_to(f2_fma(v, xent_splat(XENT_LOG2E), b), x0, x1);
  return f2_of(__float_as_uint(fast_exp2(__uint_as_float(x0))), __float_as_uint(fast_exp2(__uint_as_float(x1))));
}
constexpr float XENT_WIDE = 1048576.f;
// By adding 1.5 * 2^23 and taking it off: whole numbers up to 2^22
__device__ __forceinline__ float xent_base(float m) { return fmaf(-m, XENT_LOG2E, 12582912.f) - 12582912.f; }
// 2^(-m log2(e) - b), b within 1/2 of the exponent's first part: the Taylor series of the exponential up to x^7 (x^8 / 8! is 5e-9)
__device__ __forceinline__ float xent_rest(float m, float b) {
  const float x = fmaf(-m, XENT_LOG2E, -b) * 0.693147181f;
  float r = fmaf(x, 1.f / 5040.f, 1.f / 720.f);
  r = fmaf(x, r, 1.f / 120.f);
  r = fmaf(x, r, 1.f / 24.f);
  r = fmaf(x, r, 1.f / 6.f);
  r = fmaf(x, r, 0.5f);
  r = fmaf(x, r, 1.f);
  return fmaf(x, r, 1.f);
}

// The running maximum raised to mx: terms added so far count from the new b on
__device__ __forceinline__ void xent_raise(float mx, float& m, float& b, unsigned long long& s) {
  const float nb = xent_base(mx);
  s = f2_mul(s, xent_splat(fast_exp2(nb - b)));
  m = mx;
  b = nb;
}

// s += sum exp(v - m) of one vector, m (and b) raised to its largest element first
template <typename T>
__device__ __forceinline__ void xent_vec_add(const T* p, float& m, float& b, unsigned long long& s) {
  constexpr int NP = XIO<T>::VEC / 2;
  const float mx = xent_vec_max<T>(p);
  if (mx > m) xent_raise(mx, m, b, s);
  unsigned long long v[NP];
  xent_pairs(p, v);
#pragma unroll
  for (int j = 0; j < NP; ++j) s = f2_add(s, xent_exp2(v[j], xent_splat(b)));
}

__device__ __forceinline__ void xent_store_pairs(float* p, const unsigned long long* v) { *reinterpret_cast<ulonglong2*>(p) = make_ulonglong2(v[0], v[1]); }
__device__ __forceinline__ void xent_store_pairs(__nv_bfloat16* p, const unsigned long long* v) {
  uint32_t w[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    uint32_t a, b;
    f2_to(v[j], a, b);
    w[j] = pack_bf16x2(__uint_as_float(a), __uint_as_float(b));
  }
  *reinterpret_cast<uint4*>(p) = make_uint4(w[0], w[1], w[2], w[3]);
}

// Sum of exp(v - m) over a row in shared memory whose maximum lies beyond XENT_WIDE (every logit masked by a finite value, or one far above
// what a model gives): m and the sum, found one after the other.  The block calls it together.
template <typename T, int THREADS>
__device__ __noinline__ float2 xent_wide_row(const T* srow, const T* p, int nvec, int vocab, float* red) {
  constexpr int V = XIO<T>::VEC, W = THREADS / 32;
  const int tid = threadIdx.x;
  float m = -INFINITY, s = 0.f;
  for (int i = tid; i < nvec; i += THREADS) m = fmaxf(m, xent_vec_max<T>(srow + i * V));
  for (int c = nvec * V + tid; c < vocab; c += THREADS) m = fmaxf(m, XIO<T>::ld1(p + c));
  m = warp_max(m);
  __syncthreads();
  if ((tid & 31) == 0) red[tid >> 5] = m;
  __syncthreads();
  for (int w = 0; w < W; ++w) m = fmaxf(m, red[w]);
  for (int i = tid; i < nvec; i += THREADS) {
    float v[V];
    XIO<T>::load(srow + i * V, v);
    for (int j = 0; j < V; ++j) s += __expf(v[j] - m);
  }
  for (int c = nvec * V + tid; c < vocab; c += THREADS) s += __expf(XIO<T>::ld1(p + c) - m);
  s = warp_sum(s);
  __syncthreads();
  if ((tid & 31) == 0) red[tid >> 5] = s;
  __syncthreads();
  s = 0.f;
  for (int w = 0; w < W; ++w) s += red[w];
  return make_float2(m, s);
}

template <typename T, int THREADS>
__global__ void __launch_bounds__(THREADS)
xent_smem_kernel(const T* __restrict__ logits, const int* __restrict__ targets, float* __restrict__ row_loss, T* dlogits,
                 int vocab, int ld, float grad_scale, int ignore_index) {
  constexpr int V = XIO<T>::VEC, W = THREADS / 32;
  extern __shared__ __align__(16) unsigned char xs_raw[];
  __shared__ float red_m[W], red_s[W];
  T* srow = reinterpret_cast<T*>(xs_raw);
  const long long row = blockIdx.x;
  const T* p = logits + row * ld;
  const int tid = threadIdx.x, nvec = vocab / V;
  for (int i = tid; i < nvec; i += THREADS) xent_cp16(srow + i * V, p + i * V);
  asm volatile("cp.async.commit_group;" ::: "memory");
  const int tgt = targets[row];
  const bool ignored = (tgt == ignore_index);
  const bool oor = !ignored && (tgt < 0 || tgt >= vocab);
  const float tgt_logit = (tid == 0 && !ignored && !oor) ? XIO<T>::ld1(p + tgt) : 0.f;   // before any thread overwrites the row
  // finite: a masked logit (-inf, or any value below) adds 0 whatever came before it
  float m = -XENT_WIDE, b = xent_base(m);
  unsigned long long s2 = 0;
  for (int c = nvec * V + tid; c < vocab; c += THREADS) {
    const float v = XIO<T>::ld1(p + c);
    if (v > m) xent_raise(v, m, b, s2);
    s2 = f2_add(s2, f2_of(__float_as_uint(fast_exp2(fmaf(v, XENT_LOG2E, b))), 0u));
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll 2
  for (int i = tid; i < nvec; i += THREADS) xent_vec_add<T>(srow + i * V, m, b, s2);
  uint32_t s_lo, s_hi;
  f2_to(s2, s_lo, s_hi);
  const float mw = warp_max(m), bw = xent_base(mw);
  float s = warp_sum((__uint_as_float(s_lo) + __uint_as_float(s_hi)) * fast_exp2(bw - b));
  if ((tid & 31) == 0) { red_m[tid >> 5] = mw; red_s[tid >> 5] = s; }
  __syncthreads();
  m = red_m[0];
#pragma unroll
  for (int w = 1; w < W; ++w) m = fmaxf(m, red_m[w]);
  b = xent_base(m);
  s = 0.f;
#pragma unroll
  for (int w = 0; w < W; ++w) s += red_s[w] * fast_exp2(b - xent_base(red_m[w]));
  const bool wide = !(fabsf(m) < XENT_WIDE);             // the same in every thread; whatever s is then
  float lse = 0.f;
  if (wide) {
    const float2 ms = xent_wide_row<T, THREADS>(srow, p, nvec, vocab, red_m);
    lse = ms.x + logf(ms.y);
  }
  if (tid == 0)
    row_loss[row] = ignored ? 0.f : oor ? __int_as_float(0x7fc00000) : wide ? lse - tgt_logit : (m - tgt_logit) + logf(s * xent_rest(m, b));
  if (!dlogits) return;
  T* d = dlogits + row * ld;
  const float gs = ignored ? 0.f : grad_scale;
  // probabilities: terms counted from the sum's own power of two, 2^e <= s < 2^(e + 1), over s 2^-e
  const int e = (__float_as_int(s) >> 23) - 127;
  const float sn = s * __int_as_float((127 - e) << 23), inv = 1.f / sn;
  b -= (float)e;
  const unsigned long long b2 = xent_splat(b), gs2 = xent_splat(gs * inv);
  const int hit = tgt >= 0 ? tgt / V : -1;               // the vector that holds the target, or none
#pragma unroll 2
  for (int i = tid; i < nvec; i += THREADS) {
    if (wide) {
      xent_vec_grad<T>(srow + i * V, d + i * V, lse, gs, tgt - i * V);
      continue;
    }
    unsigned long long v[V / 2];
    xent_pairs(srow + i * V, v);
#pragma unroll
    for (int j = 0; j < V / 2; ++j) v[j] = xent_exp2(v[j], b2);
    if (i == hit) {
#pragma unroll
      for (int j = 0; j < V / 2; ++j) {
        const int k = tgt - i * V - 2 * j;
        v[j] = f2_add(v[j], f2_of(__float_as_uint(k == 0 ? -sn : 0.f), __float_as_uint(k == 1 ? -sn : 0.f)));
      }
    }
#pragma unroll
    for (int j = 0; j < V / 2; ++j) v[j] = f2_mul(v[j], gs2);
    xent_store_pairs(d + i * V, v);
  }
  for (int c = nvec * V + tid; c < vocab; c += THREADS) {
    const float v = XIO<T>::ld1(p + c), pr = wide ? __expf(v - lse) : fast_exp2(fmaf(v, XENT_LOG2E, b)) * inv;
    const float g = (pr - (c == tgt ? 1.f : 0.f)) * gs;
    if constexpr (sizeof(T) == 4) d[c] = g; else d[c] = __float2bfloat16_rn(g);
  }
}

// Short rows (whole vectors, at most XENT_WARP_VECS * 32 of them): one warp per row, the row in registers.  A CTA per row left
// seven of eight warps idle at 256 columns.
constexpr int XENT_WARP_VECS = 4;
template <typename T>
__global__ void __launch_bounds__(XENT_THREADS)
xent_warp_kernel(const T* __restrict__ logits, const int* __restrict__ targets, float* __restrict__ row_loss, T* dlogits,
                 long long rows, int vocab, int ld, float grad_scale, int ignore_index) {
  constexpr int V = XIO<T>::VEC, NV = XENT_WARP_VECS;
  pdl_wait();
  const long long row = (long long)blockIdx.x * (XENT_THREADS / 32) + (threadIdx.x >> 5);
  if (row >= rows) return;
  const int lane = threadIdx.x & 31, nvec = vocab / V;
  const T* p = logits + row * ld;
  uint4 x[NV];
#pragma unroll
  for (int k = 0; k < NV; ++k)
    if (k * 32 + lane < nvec) x[k] = *reinterpret_cast<const uint4*>(p + (k * 32 + lane) * V);
  const int tgt = targets[row];
  const bool ignored = (tgt == ignore_index);
  const bool oor = !ignored && (tgt < 0 || tgt >= vocab);
  float tgt_logit = (lane == 0 && !ignored && !oor) ? XIO<T>::ld1(p + tgt) : 0.f;
  float m = -INFINITY, s = 0.f;
#pragma unroll
  for (int k = 0; k < NV; ++k)
    if (k * 32 + lane < nvec) m = fmaxf(m, xent_vec_max<T>(reinterpret_cast<const T*>(&x[k])));
  m = warp_max(m);
#pragma unroll
  for (int k = 0; k < NV; ++k)
    if (k * 32 + lane < nvec) {
      float v[V];
      XIO<T>::load(reinterpret_cast<const T*>(&x[k]), v);
#pragma unroll
      for (int j = 0; j < V; ++j) s += __expf(v[j] - m);
    }
  s = warp_sum(s);
  const float lse = m + logf(s);
  if (lane == 0) row_loss[row] = ignored ? 0.f : (oor ? __int_as_float(0x7fc00000) : lse - tgt_logit);
  if (!dlogits) return;
  __syncwarp();                                          // lane 0 has read the target's logit
  T* d = dlogits + row * ld;
  const float gs = ignored ? 0.f : grad_scale;
#pragma unroll
  for (int k = 0; k < NV; ++k)
    if (k * 32 + lane < nvec)
      xent_vec_grad<T>(reinterpret_cast<const T*>(&x[k]), d + (k * 32 + lane) * V, lse, gs, tgt - (k * 32 + lane) * V);
}

// Whether the row in shared memory beats the online kernel.  With the gradient it saves a read of the logits: always, except for 16-bit
// rows of which only one fits an SM (2048 x 65536 139.6 us online, 143.6 on the chip).  The loss alone reads them once either way, and the
// online kernel keeps more loads in flight when rows are long: 8192 x 16384 bf16 72.3 / 60.5 us, fp32 88.2 / 83.9; 2048 x 32000 bf16
// 33.1 / 34.9, 2048 x 50264 46.7 / 55.2, 8192 x 20480 fp32 108 / 118, 8192 x 32000 162 / 247.  One wave of rows is latency, not
// bandwidth: 148 x 50264 8.2 / 6.8.
static bool xent_row_on_chip(size_t bytes, long long rows, bool grad, size_t elem) {
  if (rows <= 148) return true;
  return grad ? elem == 4 || bytes <= 112 * 1024 : bytes <= 16384 * elem;
}

template <typename T>
static int launch_xent(const T* logits, const int* targets, float* row_loss, T* dlogits, long long rows, int vocab, int ld, float grad_scale,
                       int ignore_index, int vec_ok, cudaStream_t st) {
  constexpr int V = XIO<T>::VEC;
  const int nvec = vocab / V;
  const size_t smem = (size_t)nvec * 16;
  if (vec_ok && vocab % V == 0 && nvec <= XENT_WARP_VECS * 32) {
    const unsigned blocks = (unsigned)((rows + XENT_THREADS / 32 - 1) / (XENT_THREADS / 32));
    launch_short(xent_warp_kernel<T>, dim3(blocks), dim3(XENT_THREADS), 0, st, logits, targets, row_loss, dlogits, rows, vocab, ld, grad_scale, ignore_index);
  } else if (vec_ok && smem > 0 && smem <= XENT_SMEM_MAX && xent_row_on_chip(smem, rows, dlogits != nullptr, sizeof(T))) {
    // eight vectors or so per thread: fewer threads leave the copies of short rows in flight together with the next CTA's
    auto go = [&](auto kernel, int threads) -> int {
      if (smem > 40 * 1024 && cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, XENT_SMEM_MAX) != cudaSuccess) return OA_ERR_LAUNCH;
      kernel<<<(unsigned)rows, threads, smem, st>>>(logits, targets, row_loss, dlogits, vocab, ld, grad_scale, ignore_index);
      return OA_OK;
    };
    int rc;
    if (nvec <= 1024) rc = go(xent_smem_kernel<T, 128>, 128);
    else if (nvec <= 2048) rc = go(xent_smem_kernel<T, 256>, 256);
    else rc = go(xent_smem_kernel<T, 512>, 512);
    if (rc) return rc;
  } else {
    xent_kernel<T><<<(unsigned)rows, XENT_THREADS, 0, st>>>(logits, targets, row_loss, dlogits, vocab, ld, grad_scale, ignore_index, vec_ok);
  }
  return cudaGetLastError() == cudaSuccess ? OA_OK : OA_ERR_LAUNCH;
}

// out[0] = scale * sum(x), one CTA, fixed reduction order.  Latency: eight loads on their way together, one at a time / so: 16384 values 2.33 /
// 2.12 us, 32768 3.13 / 2.92, 65536 4.65 / 3.81, 2048 1.83 either way.
__global__ void mean_f32_kernel(const float* __restrict__ x, float* __restrict__ out, long long n, float scale) {
  __shared__ float red[32];
  pdl_wait();
  float s = 0.f;
  long long i = threadIdx.x;
  for (; i + 7LL * blockDim.x < n; i += 8LL * blockDim.x) {
    float v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) v[u] = x[i + (long long)u * blockDim.x];
#pragma unroll
    for (int u = 0; u < 8; ++u) s += v[u];
  }
  for (; i < n; i += blockDim.x) s += x[i];
  s = warp_sum(s);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    float t = 0.f;
    for (int w = 0; w < (blockDim.x >> 5); ++w) t += red[w];
    out[0] = t * scale;
  }
}

}  // namespace oa

using namespace oa;

extern "C" int oa_xent_fwd_bwd(int dtype, const void* logits, const int* targets, float* row_loss, void* dlogits,
                               long long rows, int vocab, int ld, float grad_scale, int ignore_index, void* stream) {
  if (rows <= 0) return OA_OK;
  const int es = dtype == OA_F32 ? 4 : 2;
  const int vec_ok = ((long long)ld * es) % 16 == 0 && (reinterpret_cast<uintptr_t>(logits) & 15) == 0 &&
                     (!dlogits || (reinterpret_cast<uintptr_t>(dlogits) & 15) == 0);
  cudaStream_t st = (cudaStream_t)stream;
  if (dtype == OA_F32)
    return launch_xent<float>((const float*)logits, targets, row_loss, (float*)dlogits, rows, vocab, ld, grad_scale, ignore_index, vec_ok, st);
  if (dtype == OA_BF16)
    return launch_xent<__nv_bfloat16>((const __nv_bfloat16*)logits, targets, row_loss, (__nv_bfloat16*)dlogits, rows, vocab, ld, grad_scale,
                                      ignore_index, vec_ok, st);
  return OA_ERR_UNSUPPORTED;
}

// ---- vocabulary-parallel cross-entropy (tensor parallel head): every rank holds [rows, vocab / W] logits.
// stats: (max, sum exp(l - max), target logit if the target falls into this shard else 0) per row;
// finish: global lse from all ranks' stats, row loss, and dlogits = (exp(l - lse) - onehot) * scale written in place.
namespace oa {

template <typename T>
__global__ void __launch_bounds__(XENT_THREADS)
vp_xent_stats_kernel(const T* __restrict__ logits, const int* __restrict__ targets, float* __restrict__ stats, int vocab, int v0) {
  constexpr int V = XIO<T>::VEC;
  __shared__ float red_m[XENT_THREADS / 32], red_s[XENT_THREADS / 32];
  const long long row = blockIdx.x;
  const T* p = logits + row * vocab;
  float m = -INFINITY, s = 0.f;
  for (int i = threadIdx.x; i < vocab / V; i += XENT_THREADS) {
    float v[V];
    XIO<T>::load(p + i * V, v);
    float mx = v[0];
#pragma unroll
    for (int j = 1; j < V; ++j) mx = fmaxf(mx, v[j]);
    if (mx > m) { s *= __expf(m - mx); m = mx; }
#pragma unroll
    for (int j = 0; j < V; ++j) s += __expf(v[j] - m);
  }
  // combine (m, s) pairs: warp, then block
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float m2 = __shfl_xor_sync(0xffffffffu, m, o), s2 = __shfl_xor_sync(0xffffffffu, s, o);
    const float mm = fmaxf(m, m2);
    s = (m == -INFINITY ? 0.f : s * __expf(m - mm)) + (m2 == -INFINITY ? 0.f : s2 * __expf(m2 - mm));
    m = mm;
  }
  if ((threadIdx.x & 31) == 0) { red_m[threadIdx.x >> 5] = m; red_s[threadIdx.x >> 5] = s; }
  __syncthreads();
  if (threadIdx.x == 0) {
    float M = red_m[0], S = red_s[0];
    for (int w = 1; w < XENT_THREADS / 32; ++w) {
      const float mm = fmaxf(M, red_m[w]);
      S = (M == -INFINITY ? 0.f : S * __expf(M - mm)) + (red_m[w] == -INFINITY ? 0.f : red_s[w] * __expf(red_m[w] - mm));
      M = mm;
    }
    const int t = targets[row] - v0;
    stats[row * 3 + 0] = M;
    stats[row * 3 + 1] = S;
    stats[row * 3 + 2] = (t >= 0 && t < vocab) ? XIO<T>::ld1(p + t) : 0.f;
  }
}

template <typename T>
__global__ void __launch_bounds__(XENT_THREADS)
vp_xent_finish_kernel(T* __restrict__ logits, const int* __restrict__ targets, const float* all_stats, float* __restrict__ row_loss,
                      long long rows, int vocab, int v0, int world, float scale, int want_grad) {
  constexpr int V = XIO<T>::VEC;
  const long long row = blockIdx.x;
  float M = -INFINITY;
  // peers wrote these: read through L2 (L1 may hold the previous step's values)
  for (int r = 0; r < world; ++r) M = fmaxf(M, __ldcg(all_stats + ((long long)r * rows + row) * 3));
  float S = 0.f, tl = 0.f;
  for (int r = 0; r < world; ++r) {
    const float* st = all_stats + ((long long)r * rows + row) * 3;
    S += __ldcg(st + 1) * __expf(__ldcg(st) - M);
    tl += __ldcg(st + 2);
  }
  const float lse = M + __logf(S);
  if (threadIdx.x == 0) row_loss[row] = lse - tl;
  if (!want_grad) return;
  T* p = logits + row * vocab;
  const int t = targets[row] - v0;
  for (int i = threadIdx.x; i < vocab / V; i += XENT_THREADS) {
    float v[V];
    XIO<T>::load(p + i * V, v);
#pragma unroll
    for (int j = 0; j < V; ++j) v[j] = (__expf(v[j] - lse) - ((i * V + j) == t ? 1.f : 0.f)) * scale;
    XIO<T>::store(p + i * V, v);
  }
}

}  // namespace oa

extern "C" int oa_vp_xent_stats(int dtype, const void* logits, const int* targets, float* stats, long long rows, int vocab, int v0,
                                void* stream) {
  if (rows <= 0) return OA_OK;
  if (vocab % 8 || (reinterpret_cast<uintptr_t>(logits) & 15)) return OA_ERR_ALIGN;
  cudaStream_t st = (cudaStream_t)stream;
  if (dtype == OA_F32) oa::vp_xent_stats_kernel<float><<<(unsigned)rows, oa::XENT_THREADS, 0, st>>>((const float*)logits, targets, stats, vocab, v0);
  else if (dtype == OA_BF16)
    oa::vp_xent_stats_kernel<__nv_bfloat16><<<(unsigned)rows, oa::XENT_THREADS, 0, st>>>((const __nv_bfloat16*)logits, targets, stats, vocab, v0);
  else return OA_ERR_UNSUPPORTED;
  return cudaGetLastError() == cudaSuccess ? OA_OK : OA_ERR_LAUNCH;
}

extern "C" int oa_vp_xent_finish(int dtype, void* logits, const int* targets, const float* all_stats, float* row_loss, long long rows,
                                 int vocab, int v0, int world, float scale, int want_grad, void* stream) {
  if (rows <= 0) return OA_OK;
  if (vocab % 8 || (reinterpret_cast<uintptr_t>(logits) & 15)) return OA_ERR_ALIGN;
  cudaStream_t st = (cudaStream_t)stream;
  if (dtype == OA_F32)
    oa::vp_xent_finish_kernel<float><<<(unsigned)rows, oa::XENT_THREADS, 0, st>>>((float*)logits, targets, all_stats, row_loss, rows, vocab, v0, world, scale, want_grad);
  else if (dtype == OA_BF16)
    oa::vp_xent_finish_kernel<__nv_bfloat16><<<(unsigned)rows, oa::XENT_THREADS, 0, st>>>((__nv_bfloat16*)logits, targets, all_stats, row_loss, rows, vocab, v0, world, scale, want_grad);
  else return OA_ERR_UNSUPPORTED;
  return cudaGetLastError() == cudaSuccess ? OA_OK : OA_ERR_LAUNCH;
}

extern "C" int oa_mean_f32(const float* x, float* out, long long n, float scale, void* stream) {
  oa::launch_short(mean_f32_kernel, dim3(1), dim3(1024), 0, (cudaStream_t)stream, x, out, n, scale);
  return cudaGetLastError() == cudaSuccess ? OA_OK : OA_ERR_LAUNCH;
}
