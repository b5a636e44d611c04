// Exact-fp32 attention (forward and backward) for the engine's FP32 precision mode and for gradient
// checks.  Same contract as the bf16 tensor-core kernels in flash_attn.cu: q, k, v are [B*S, row_stride]
// views with head h at column h*head_dim, o is [B*S, H*head_dim], lse is [B, H, S] (natural log).
//
// Every output element has a single writer, like the reference's FlashCausal / FlashCausalBwdQ /
// FlashCausalBwdKV (Source/Private/Oa/Ml/Shader/Compute/Nn/Attention/*.slang), but the other side of the
// product is streamed through shared memory 32 rows at a time with an online softmax, so there is no
// sequence-length cap and global memory is read in whole rows.
//
// Work split (forward and both gradients): a CTA of 128 threads owns 128 / (DS KS) rows of one (batch, head).  A row is shared by DS threads that
// keep 32 head dimensions each in registers (their partial dot products meet in shuffles) and by KS groups of those that take every
// KS-th row of the other side, with a running maximum and sums of their own that meet once, at the end.  KS = 1 does the least
// work per score; KS = 4 makes four times as many, shorter CTAs (which under the causal mask also skip more of the other side), lets
// the next tile arrive through cp.async under this one, and is taken while KS = 1 would leave SMs idle (af_split).
// 16 x 4 heads of 32 dimensions and 128 positions are 64 CTAs with KS = 1, one warp per scheduler: 29 us forward
// and 83 us both gradients.  With KS = 4: 12.6 us, and 25.7 for both gradients (eight dimensions per thread, whose dot products each took
// two shuffles, were 2.5 and 15 us slower).
// What bounds it: eight to twelve warps per SM, whose reads of shared memory and dot products wait for one another.  So the two gradients,
// neither of which needs the other, share one launch: the blocks of dQ fill the room that those of dK and dV leave.  A row's own dimensions
// come in 16-byte pieces where the operands allow it, and under the causal mask the longest blocks of each kind start first.  Both gradients
// as two launches one after the other / as one, us: 16 x 128 of 4 x 32 causal 37.8 / 25.7, 16 x 512 of 4 x 32 causal 270 / 224, 8 x 256 of 4 x 128
// causal 254 / 179, 2 x 1024 of 4 x 64 full 469 / 358.  (As two launches of which the second began without a wait they took 31, 255, 201 and
// 319; but what a kernel reads that does not wait for those before it, nothing promises.)
// Forward and dQ rows are queries (keys / values stream through shared memory), dK / dV rows are keys (queries and output gradients
// stream through shared memory together with their log-sum-exp and delta = rowsum(dO * O)).
#include "common.cuh"
#include "api.h"

namespace oa {

constexpr int AF_THREADS = 128;
constexpr int AF_TILE = 32;     // streamed rows per step

constexpr int AF_W = 32;        // head dimensions per thread
constexpr int AF_SEG = AF_W + 4;   // floats per such segment in shared memory (padded: rows and segments land in different banks)

// A streamed tile of rows [r0, r0 + 32) of a [rows, stride] matrix, columns [col0, col0 + hd), as [32][DS][AF_SEG]; rows >= limit and
// dimensions >= hd become 0.  `vec`: 16-byte pieces (hd, stride and the pointer allow it), asynchronously when ASYNC.
template <int DS, bool ASYNC>
__device__ __forceinline__ void af_load_tile(float* sm, const float* __restrict__ g, long long stride, long long row_base, int r0, int limit, int col0,
                                             int hd, bool vec) {
  constexpr int COLS = DS * AF_W;
  if (vec) {
#pragma unroll
    for (int idx = threadIdx.x; idx < AF_TILE * COLS / 4; idx += AF_THREADS) {
      const int r = idx / (COLS / 4), c = idx % (COLS / 4) * 4;
      const bool ok = r0 + r < limit && c < hd;
      const float* src = ok ? g + (row_base + r0 + r) * stride + col0 + c : g;
      float* dst = sm + (r * DS + c / AF_W) * AF_SEG + c % AF_W;
      if (ASYNC) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(ok ? 16 : 0) : "memory");
      else *reinterpret_cast<float4*>(dst) = ok ? *reinterpret_cast<const float4*>(src) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
  } else {
#pragma unroll 4
    for (int idx = threadIdx.x; idx < AF_TILE * COLS; idx += AF_THREADS) {
      const int r = idx / COLS, c = idx % COLS;
      float x = 0.f;
      if (r0 + r < limit && c < hd) x = g[(row_base + r0 + r) * stride + col0 + c];
      sm[(r * DS + c / AF_W) * AF_SEG + c % AF_W] = x;
    }
  }
}
__device__ __forceinline__ void af_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void af_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// A thread's 32 dimensions of its own row, zeros beyond hd and for rows that are not there
__device__ __forceinline__ void af_own(float* dst, const float* __restrict__ row, int left, bool ok, bool vec) {
  if (!ok) left = 0;
  if (vec) {
#pragma unroll
    for (int t = 0; t < AF_W; t += 4) *reinterpret_cast<float4*>(dst + t) = t < left ? *reinterpret_cast<const float4*>(row + t) : make_float4(0.f, 0.f, 0.f, 0.f);
  } else {
#pragma unroll
    for (int t = 0; t < AF_W; ++t) dst[t] = t < left ? row[t] : 0.f;
  }
}

// sum over the DS threads that share a row's dot products (neighbouring lanes)
template <int DS>
__device__ __forceinline__ float af_reduce(float x) {
  if (DS >= 2) x += __shfl_xor_sync(0xffffffffu, x, 1);
  if (DS >= 4) x += __shfl_xor_sync(0xffffffffu, x, 2);
  return x;
}
// Sums of v[0..31] over the KS groups of a row: every group ends up with 32 / KS of them, v[0 .. 32 / KS), which are dimensions
// af_first<KS>(ks) and on.
template <int DS, int KS>
__device__ __forceinline__ void af_scatter_sum(float* v, int ks) {
  if constexpr (KS == 4) {
#pragma unroll
    for (int t = 0; t < 16; ++t) {
      const float mine = ks & 1 ? v[t + 16] : v[t], theirs = ks & 1 ? v[t] : v[t + 16];
      v[t] = mine + __shfl_xor_sync(0xffffffffu, theirs, DS);
    }
#pragma unroll
    for (int t = 0; t < 8; ++t) {
      const float mine = ks & 2 ? v[t + 8] : v[t], theirs = ks & 2 ? v[t] : v[t + 8];
      v[t] = mine + __shfl_xor_sync(0xffffffffu, theirs, 2 * DS);
    }
  }
}
template <int KS>
__device__ __forceinline__ int af_first(int ks) { return KS == 4 ? (ks & 1) * 16 + (ks >> 1) * 8 : 0; }

__device__ __forceinline__ float af_dot(const float* a, const float* __restrict__ sm_row) {
  float d0 = 0.f, d1 = 0.f, d2 = 0.f, d3 = 0.f;
#pragma unroll
  for (int t = 0; t < AF_W; t += 4) {
    const float4 x = *reinterpret_cast<const float4*>(sm_row + t);
    d0 = fmaf(a[t], x.x, d0); d1 = fmaf(a[t + 1], x.y, d1); d2 = fmaf(a[t + 2], x.z, d2); d3 = fmaf(a[t + 3], x.w, d3);
  }
  return (d0 + d1) + (d2 + d3);
}

__device__ __forceinline__ void af_axpy(float* acc, float a, const float* __restrict__ sm_row) {
#pragma unroll
  for (int t = 0; t < AF_W; t += 4) {
    const float4 x = *reinterpret_cast<const float4*>(sm_row + t);
    acc[t] = fmaf(a, x.x, acc[t]); acc[t + 1] = fmaf(a, x.y, acc[t + 1]);
    acc[t + 2] = fmaf(a, x.z, acc[t + 2]); acc[t + 3] = fmaf(a, x.w, acc[t + 3]);
  }
}

template <int DS, int KS>
struct AfCfg {
  static constexpr int TPR = DS * KS, ROWS = AF_THREADS / TPR;
  static constexpr bool ASYNC = KS > 1;                        // two buffers, the next tile in flight
  static constexpr int BUFS = ASYNC ? 2 : 1, TILE = AF_TILE * DS * AF_SEG;
};

// The two streamed matrices of each pass, tile by tile: body(j0, x tile, y tile) for j0 in [lo, hi) in steps of 32.
template <int DS, int KS, typename Body>
__device__ __forceinline__ void af_stream(float* sx, float* sy, const float* __restrict__ x, long long xs, const float* __restrict__ y, long long ys,
                                          long long row0, int lo, int hi, int limit, int col0, int hd, bool vec, Body body) {
  using Cfg = AfCfg<DS, KS>;
  auto load = [&](int j0, int buf) {
    af_load_tile<DS, Cfg::ASYNC>(sx + buf * Cfg::TILE, x, xs, row0, j0, limit, col0, hd, vec);
    af_load_tile<DS, Cfg::ASYNC>(sy + buf * Cfg::TILE, y, ys, row0, j0, limit, col0, hd, vec);
    if (Cfg::ASYNC) af_commit();
  };
  if constexpr (Cfg::ASYNC) {
    load(lo, 0);
    for (int j0 = lo, buf = 0; j0 < hi; j0 += AF_TILE, buf ^= 1) {
      if (j0 + AF_TILE < hi) { load(j0 + AF_TILE, buf ^ 1); af_wait<1>(); } else { af_wait<0>(); }
      __syncthreads();
      body(j0, sx + buf * Cfg::TILE, sy + buf * Cfg::TILE);
      __syncthreads();                                         // the buffer may be filled again
    }
  } else {
    for (int j0 = lo; j0 < hi; j0 += AF_TILE) {
      __syncthreads();
      load(j0, 0);
      __syncthreads();
      body(j0, sx, sy);
    }
  }
}

template <int DS, int KS>
__global__ void __launch_bounds__(AF_THREADS)
attn_f32_fwd_kernel(const float* __restrict__ q, const float* __restrict__ k, const float* __restrict__ v,
                    float* __restrict__ o, float* __restrict__ lse, int heads, int seq, int hd, long long rs, long long os,
                    float scale, int causal, int vec) {
  using Cfg = AfCfg<DS, KS>;
  constexpr int NJ = AF_TILE / KS;                             // keys of a tile that this thread takes: ks, ks + KS, ...
  __shared__ __align__(16) float sK[Cfg::BUFS * Cfg::TILE], sV[Cfg::BUFS * Cfg::TILE];
  pdl_wait();
  const int h = blockIdx.y, b = blockIdx.z;
  const int i0 = (gridDim.x - 1 - blockIdx.x) * Cfg::ROWS;       // under the causal mask the longest first
  const int i = i0 + threadIdx.x / Cfg::TPR, seg = threadIdx.x % DS, ks = threadIdx.x % Cfg::TPR / DS;
  const long long row0 = (long long)b * seq;
  const bool row_ok = i < seq;
  float qr[AF_W], acc[AF_W];
  af_own(qr, q + (row0 + i) * rs + h * hd + seg * AF_W, hd - seg * AF_W, row_ok, vec);
#pragma unroll
  for (int t = 0; t < AF_W; ++t) {
    qr[t] *= scale;
    acc[t] = 0.f;
  }
  float m = -INFINITY, l = 0.f;
  const int kend = causal ? min(seq, i0 + Cfg::ROWS) : seq;       // keys this CTA needs
  af_stream<DS, KS>(sK, sV, k, rs, v, rs, row0, 0, kend, seq, h * hd, hd, vec, [&](int j0, const float* tk, const float* tv) {
    float s[NJ];
    float mt = -INFINITY;
#pragma unroll
    for (int jj = 0; jj < NJ; ++jj) {
      const int j = jj * KS + ks;
      const float d = af_reduce<DS>(af_dot(qr, tk + (j * DS + seg) * AF_SEG));
      const int kj = j0 + j;
      const bool alive = kj < seq && (!causal || kj <= i);
      s[jj] = alive ? d : -INFINITY;
      mt = fmaxf(mt, s[jj]);
    }
    const float mn = fmaxf(m, mt);
    const float mu = (mn == -INFINITY) ? 0.f : mn;
    const float alpha = __expf(m - mu);
    float ls = 0.f;
#pragma unroll
    for (int t = 0; t < AF_W; ++t) acc[t] *= alpha;
#pragma unroll
    for (int jj = 0; jj < NJ; ++jj) {
      const float p = __expf(s[jj] - mu);
      ls += p;
      af_axpy(acc, p, tv + ((jj * KS + ks) * DS + seg) * AF_SEG);
    }
    l = l * alpha + ls;
    m = mn;
  });
  if constexpr (KS == 4) {
    // the groups' maxima and sums meet
    float mx = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, DS));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2 * DS));
    const float w = __expf(m - (mx == -INFINITY ? 0.f : mx));
    l *= w;
    l += __shfl_xor_sync(0xffffffffu, l, DS);
    l += __shfl_xor_sync(0xffffffffu, l, 2 * DS);
#pragma unroll
    for (int t = 0; t < AF_W; ++t) acc[t] *= w;
    m = mx;
    af_scatter_sum<DS, KS>(acc, ks);
  }
  if (!row_ok) return;
  const float inv = l > 0.f ? 1.f / l : 0.f;
#pragma unroll
  for (int t = 0; t < AF_W / KS; ++t) {
    const int d = seg * AF_W + af_first<KS>(ks) + t;
    if (d < hd) o[(row0 + i) * os + h * hd + d] = acc[t] * inv;
  }
  if (seg == 0 && ks == 0 && lse) lse[((long long)b * heads + h) * seq + i] = m + logf(l);
}

// dQ: rows are queries; K and V stream through shared memory.
template <int DS, int KS>
__device__ __forceinline__ void af_bwd_q(float* sK, float* sV, int b, const float* __restrict__ q, const float* __restrict__ k, const float* __restrict__ v,
                                         const float* __restrict__ o, const float* __restrict__ dout, const float* __restrict__ lse,
                                         float* __restrict__ dq, int heads, int seq, int hd, long long rs, long long os, long long ds_, float scale,
                                         int causal, int vec) {
  using Cfg = AfCfg<DS, KS>;
  constexpr int NJ = AF_TILE / KS;
  const int h = blockIdx.y;
  const int i0 = (gridDim.x - 1 - blockIdx.x) * Cfg::ROWS;       // under the causal mask the longest first
  const int i = i0 + threadIdx.x / Cfg::TPR, seg = threadIdx.x % DS, ks = threadIdx.x % Cfg::TPR / DS;
  const long long row0 = (long long)b * seq;
  const bool row_ok = i < seq;
  float qr[AF_W], dor[AF_W], acc[AF_W];
  float delta = 0.f;
  const int left = hd - seg * AF_W;
  af_own(acc, o + (row0 + i) * os + h * hd + seg * AF_W, left, row_ok, vec);
  af_own(dor, dout + (row0 + i) * os + h * hd + seg * AF_W, left, row_ok, vec);
  af_own(qr, q + (row0 + i) * rs + h * hd + seg * AF_W, left, row_ok, vec);
#pragma unroll
  for (int t = 0; t < AF_W; ++t) {
    qr[t] *= scale;
    if (t < left) delta = fmaf(dor[t], acc[t], delta);
    acc[t] = 0.f;
  }
  delta = af_reduce<DS>(delta);
  const float L = row_ok ? lse[((long long)b * heads + h) * seq + i] : 0.f;
  const int kend = causal ? min(seq, i0 + Cfg::ROWS) : seq;
  af_stream<DS, KS>(sK, sV, k, rs, v, rs, row0, 0, kend, seq, h * hd, hd, vec, [&](int j0, const float* tk, const float* tv) {
#pragma unroll 4
    for (int jj = 0; jj < NJ; ++jj) {
      const int j = jj * KS + ks;
      const float* kr = tk + (j * DS + seg) * AF_SEG;
      const float d = af_reduce<DS>(af_dot(qr, kr));
      const float dp = af_reduce<DS>(af_dot(dor, tv + (j * DS + seg) * AF_SEG));
      const int kj = j0 + j;
      const bool alive = row_ok && kj < seq && (!causal || kj <= i);
      const float ds = alive ? __expf(d - L) * (dp - delta) * scale : 0.f;
      af_axpy(acc, ds, kr);
    }
  });
  af_scatter_sum<DS, KS>(acc, ks);
  if (!row_ok) return;
#pragma unroll
  for (int t = 0; t < AF_W / KS; ++t) {
    const int d = seg * AF_W + af_first<KS>(ks) + t;
    if (d < hd) dq[(row0 + i) * ds_ + h * hd + d] = acc[t];
  }
}

// dK, dV: rows are keys; Q and dO stream through shared memory with the queries' log-sum-exp and delta.
template <int DS, int KS>
__device__ __forceinline__ void af_bwd_kv(float* sQ, float* sDO, int b, const float* __restrict__ q, const float* __restrict__ k, const float* __restrict__ v,
                                          const float* __restrict__ o, const float* __restrict__ dout, const float* __restrict__ lse,
                                          float* __restrict__ dk, float* __restrict__ dv, int heads, int seq, int hd, long long rs, long long os,
                                          long long ds_, float scale, int causal, int vec) {
  using Cfg = AfCfg<DS, KS>;
  constexpr int NI = AF_TILE / KS;
  __shared__ float sL[2][AF_TILE], sDelta[2][AF_TILE];
  const int h = blockIdx.y;
  const int j0 = blockIdx.x * Cfg::ROWS;
  const int j = j0 + threadIdx.x / Cfg::TPR, seg = threadIdx.x % DS, ks = threadIdx.x % Cfg::TPR / DS;
  const long long row0 = (long long)b * seq;
  const bool row_ok = j < seq;
  float kr[AF_W], vr[AF_W], acck[AF_W], accv[AF_W];
  af_own(kr, k + (row0 + j) * rs + h * hd + seg * AF_W, hd - seg * AF_W, row_ok, vec);
  af_own(vr, v + (row0 + j) * rs + h * hd + seg * AF_W, hd - seg * AF_W, row_ok, vec);
#pragma unroll
  for (int t = 0; t < AF_W; ++t) {
    kr[t] *= scale;
    acck[t] = 0.f; accv[t] = 0.f;
  }
  // delta and log-sum-exp of the 32 queries of a tile: 4 threads per query, shuffle-combined.  Tiles alternate between two slots, so
  // those of the next tile can be written while the last warps still read this one's.
  auto stats = [&](int i0, int slot) {
    const int r = threadIdx.x >> 2, part = threadIdx.x & 3;
    float dl = 0.f;
    if (i0 + r < seq) {
      const float *pd = dout + (row0 + i0 + r) * os + h * hd, *po = o + (row0 + i0 + r) * os + h * hd;
      if (vec) {
        for (int d = part * 4; d < hd; d += 16) {
          const float4 a = *reinterpret_cast<const float4*>(pd + d), c = *reinterpret_cast<const float4*>(po + d);
          dl = fmaf(a.x, c.x, fmaf(a.y, c.y, fmaf(a.z, c.z, fmaf(a.w, c.w, dl))));
        }
      } else {
        for (int d = part; d < hd; d += 4) dl = fmaf(pd[d], po[d], dl);
      }
    }
    dl += __shfl_xor_sync(0xffffffffu, dl, 1);
    dl += __shfl_xor_sync(0xffffffffu, dl, 2);
    if (part == 0) {
      sDelta[slot][r] = dl;
      sL[slot][r] = (i0 + r < seq) ? lse[((long long)b * heads + h) * seq + i0 + r] : INFINITY;
    }
  };
  const int istart = causal ? (j0 / AF_TILE) * AF_TILE : 0;    // first query tile any key of this CTA can see
  int slot = 0;
  stats(istart, 0);
  af_stream<DS, KS>(sQ, sDO, q, rs, dout, os, row0, istart, seq, seq, h * hd, hd, vec, [&](int i0, const float* tq, const float* td) {
    if (i0 + AF_TILE < seq) stats(i0 + AF_TILE, slot ^ 1);
#pragma unroll 4
    for (int jj = 0; jj < NI; ++jj) {
      const int ii = jj * KS + ks;
      const float* qrow = tq + (ii * DS + seg) * AF_SEG;
      const float* dorow = td + (ii * DS + seg) * AF_SEG;
      const float d = af_reduce<DS>(af_dot(kr, qrow));
      const float dp = af_reduce<DS>(af_dot(vr, dorow));
      const int qi = i0 + ii;
      const bool alive = row_ok && qi < seq && (!causal || j <= qi);
      const float p = alive ? __expf(d - sL[slot][ii]) : 0.f;
      const float ds = p * (dp - sDelta[slot][ii]);     // the key registers carry the scale: dK = scale * dS^T Q restored below
      af_axpy(accv, p, dorow);
      af_axpy(acck, ds, qrow);
    }
    slot ^= 1;
  });
  af_scatter_sum<DS, KS>(acck, ks);
  af_scatter_sum<DS, KS>(accv, ks);
  if (!row_ok) return;
#pragma unroll
  for (int t = 0; t < AF_W / KS; ++t) {
    const int d = seg * AF_W + af_first<KS>(ks) + t;
    if (d < hd) {
      dk[(row0 + j) * ds_ + h * hd + d] = acck[t] * scale;
      dv[(row0 + j) * ds_ + h * hd + d] = accv[t];
    }
  }
}

// Both gradients in one launch: the first half of the grid takes dK and dV, the second dQ.  (The halves of a sequence beside one another
// put two of a kind on some SMs: 2 x 1024 of 4 x 64, full mask, 380 us for 358.)
template <int DS, int KS>
__global__ void __launch_bounds__(AF_THREADS)
attn_f32_bwd_kernel(const float* __restrict__ q, const float* __restrict__ k, const float* __restrict__ v,
                    const float* __restrict__ o, const float* __restrict__ dout, const float* __restrict__ lse, float* __restrict__ dq,
                    float* __restrict__ dk, float* __restrict__ dv, int heads, int seq, int hd, long long rs, long long os,
                    long long ds_, float scale, int causal, int vec) {
  using Cfg = AfCfg<DS, KS>;
  __shared__ __align__(16) float sx[Cfg::BUFS * Cfg::TILE], sy[Cfg::BUFS * Cfg::TILE];
  pdl_wait();
  const int batch = gridDim.z >> 1, b = blockIdx.z;
  if (b < batch) af_bwd_kv<DS, KS>(sx, sy, b, q, k, v, o, dout, lse, dk, dv, heads, seq, hd, rs, os, ds_, scale, causal, vec);
  else af_bwd_q<DS, KS>(sx, sy, b - batch, q, k, v, o, dout, lse, dq, heads, seq, hd, rs, os, ds_, scale, causal, vec);
}

// One gradient to a launch
template <int DS, int KS, bool KV>
__global__ void __launch_bounds__(AF_THREADS)
attn_f32_bwd_part_kernel(const float* __restrict__ q, const float* __restrict__ k, const float* __restrict__ v,
                         const float* __restrict__ o, const float* __restrict__ dout, const float* __restrict__ lse, float* __restrict__ dq,
                         float* __restrict__ dk, float* __restrict__ dv, int heads, int seq, int hd, long long rs, long long os,
                         long long ds_, float scale, int causal, int vec) {
  using Cfg = AfCfg<DS, KS>;
  __shared__ __align__(16) float sx[Cfg::BUFS * Cfg::TILE], sy[Cfg::BUFS * Cfg::TILE];
  pdl_wait();
  if (KV) af_bwd_kv<DS, KS>(sx, sy, blockIdx.z, q, k, v, o, dout, lse, dk, dv, heads, seq, hd, rs, os, ds_, scale, causal, vec);
  else af_bwd_q<DS, KS>(sx, sy, blockIdx.z, q, k, v, o, dout, lse, dq, heads, seq, hd, rs, os, ds_, scale, causal, vec);
}

}  // namespace oa

using namespace oa;

// CTAs of the KS = 1 form
static inline long long af_ctas(int hd, int batch, int heads, int seq) {
  const int rows = AF_THREADS / (hd <= 32 ? 1 : (hd <= 64 ? 2 : 4));
  return (long long)((seq + rows - 1) / rows) * heads * batch;
}

// DS, or -4 DS for KS = 4, which is taken up to `limit` CTAs of the KS = 1 form: one per SM, or somewhat more where the causal mask lets the
// shorter CTAs skip work, and wherever a sequence would leave most rows of a wide CTA empty.  KS = 1 against 4 (4 heads, us), forward, full mask,
// 14 x 128 of 64 dimensions (112 CTAs) 32.2 / 22.4, 48 x 128 of 32 (192) 29.8 / 31.0, 28 x 128 of 64 (224) 34.4 / 37.7; causal 16 x 512 of 32 (256) 104 / 93,
// 36 x 128 of 64 (288) 35.2 / 35.6.  Backward, where a launch has twice the CTAs, full, 18 x 128 of 32 (72) 38.0 / 33.2, 24 x 128 of 32 (96) 49.9 / 45.6,
// 3 x 1024 of 32 (96) 296 / 306, 3 x 512 of 64 (96) 185 / 179, 28 x 128 of 32 (112) 50.2 / 54.8, 14 x 128 of 64 (112) 55.5 / 61.2, 2 x 1024 of 64 (128) 359 / 480,
// 48 x 128 of 32 (192) 73 / 86; causal 16 x 512 of 32 (256) 237 / 224, 64 x 128 of 32 (256) 93 / 77, 36 x 128 of 64 (288) 104 / 96, 48 x 128 of 64 (384) 129 / 125, but
// 5 x 512 of 64 (160) 178 / 169, 8 x 512 of 64 (256) 247 / 254, 2 x 2048 of 64 (256) 856 / 914.
static inline int af_split(int hd, int batch, int heads, int seq, int limit) {
  const int wide = hd <= 32 ? 1 : (hd <= 64 ? 2 : 4);
  return hd <= 64 && (seq <= AF_TILE || af_ctas(hd, batch, heads, seq) <= limit) ? -4 * wide : wide;
}

// Whether every row of the streamed operands can be read in 16-byte pieces.
static int af_vec(int hd, long long rs, long long os, const void* a, const void* b, const void* c, const void* d, const void* e) {
  const uintptr_t at = reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b) | reinterpret_cast<uintptr_t>(c) |
                       reinterpret_cast<uintptr_t>(d) | reinterpret_cast<uintptr_t>(e);
  return ((hd | rs | os) & 3) == 0 && (at & 15) == 0;
}

extern "C" int oa_attn_f32(const float* q, const float* k, const float* v, float* o, float* lse, int batch, int heads,
                           int seq, int head_dim, long long row_stride, long long o_row_stride, float scale, int causal,
                           void* stream) {
  if (head_dim < 1 || head_dim > 128) return OA_ERR_UNSUPPORTED;
  if (batch <= 0 || heads <= 0 || seq <= 0) return OA_OK;
  if (heads > 65535 || batch > 65535) return OA_ERR_ARG;
  cudaStream_t st = (cudaStream_t)stream;
  const int split = af_split(head_dim, batch, heads, seq, causal ? 260 : 192), rows = AF_THREADS / (split < 0 ? -split : split);
  dim3 grid((seq + rows - 1) / rows, heads, batch);
  const int vec = af_vec(head_dim, row_stride, o_row_stride, q, k, v, o, o);
#define AF_FWD(D, S) launch_short(attn_f32_fwd_kernel<D, S>, grid, dim3(AF_THREADS), 0, st, q, k, v, o, lse, heads, seq, head_dim, row_stride, \
                                  o_row_stride, scale, causal, vec)
  if (split == -4) AF_FWD(1, 4);
  else if (split == -8) AF_FWD(2, 4);
  else if (split == 1) AF_FWD(1, 1);
  else if (split == 2) AF_FWD(2, 1);
  else AF_FWD(4, 1);
#undef AF_FWD
  return cudaGetLastError() == cudaSuccess ? OA_OK : OA_ERR_LAUNCH;
}

extern "C" int oa_attn_f32_bwd(const float* q, const float* k, const float* v, const float* o, const float* dout,
                               const float* lse, float* dq, float* dk, float* dv, int batch, int heads, int seq,
                               int head_dim, long long row_stride, long long o_row_stride, long long d_row_stride,
                               float scale, int causal, void* stream) {
  if (head_dim < 1 || head_dim > 128) return OA_ERR_UNSUPPORTED;
  if (batch <= 0 || heads <= 0 || seq <= 0) return OA_OK;
  if (heads > 65535 || batch > 65535) return OA_ERR_ARG;
  cudaStream_t st = (cudaStream_t)stream;
  const int limit = !causal ? 96 : (head_dim > 32 && seq > 128 ? 240 : 300);
  const int split = af_split(head_dim, batch, heads, seq, limit), rows = AF_THREADS / (split < 0 ? -split : split);
  const int vec = af_vec(head_dim, row_stride, o_row_stride, q, k, v, o, dout);
  // The registers of dK and dV leave room for two CTAs on an SM, those of dQ alone for three.  With a full mask and several waves that outweighs
  // what the two kinds gain beside one another.  One launch / two, 4 heads of 64: 16 x 512 (512 CTAs) 691 / 661 us, 8 x 1024 1333 / 1233, 24 x 512 1018 / 904,
  // but 12 x 512 (384) 506 / 524, 5 x 512 265 / 330; causal 24 x 512 629 / 631, 16 x 512 430 / 452; of 128, full, 16 x 512 1676 / 1732; of 32 433 / 536 for 24 x 512.
  const bool apart = split == 2 && !causal && af_ctas(head_dim, batch, heads, seq) > 400;
  const int most = apart ? 65535 : 32767;                // sequences in a grid, which holds each once or twice
  for (int b0 = 0; b0 < batch; b0 += most) {
    const int nb = batch - b0 < most ? batch - b0 : most;
    const dim3 grid((seq + rows - 1) / rows, heads, apart ? nb : 2 * nb);
    const long long at = (long long)b0 * seq, qa = at * row_stride, oa = at * o_row_stride, da = at * d_row_stride;
#define AF_BWD(...)                                                                                                                          \
  launch_short(__VA_ARGS__, grid, dim3(AF_THREADS), 0, st, q + qa, k + qa, v + qa, o + oa, dout + oa, lse + at * heads, dq + da, dk + da, dv + da, \
               heads, seq, head_dim, row_stride, o_row_stride, d_row_stride, scale, causal, vec)
    if (apart) {
      AF_BWD((attn_f32_bwd_part_kernel<2, 1, true>));
      AF_BWD((attn_f32_bwd_part_kernel<2, 1, false>));
    } else if (split == -4) AF_BWD((attn_f32_bwd_kernel<1, 4>));
    else if (split == -8) AF_BWD((attn_f32_bwd_kernel<2, 4>));
    else if (split == 1) AF_BWD((attn_f32_bwd_kernel<1, 1>));
    else if (split == 2) AF_BWD((attn_f32_bwd_kernel<2, 1>));
    else AF_BWD((attn_f32_bwd_kernel<4, 1>));
  }
#undef AF_BWD
  return cudaGetLastError() == cudaSuccess ? OA_OK : OA_ERR_LAUNCH;
}
