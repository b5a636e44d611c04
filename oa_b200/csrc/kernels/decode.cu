// KV-cache serving kernels.  The reference has no KV cache: its generation loop re-runs the whole window for every new
// token (Tutorial/Cpp/Ml/Nlp/TutorialNlpCommon.h:145-177), so these are new.
//   oa_kv_append   copies the (already rotated) key and value rows of new tokens into the per-layer cache
//                  [batch, heads, max_seq, head_dim];
//   oa_decode_attn one query token per sequence against the cache: one CTA per (sequence, head), four warps stride over
//                  the cached positions with a running softmax (lane = position for q.k, lane = head-dim slice for p.v),
//                  the four partial states are merged through shared memory.  Bandwidth bound: it reads the cache once.
#include "common.cuh"
#include "api.h"

namespace oa {

__global__ void kv_append_kernel(const __nv_bfloat16* __restrict__ k_src, const __nv_bfloat16* __restrict__ v_src, long long src_stride,
                                 __nv_bfloat16* __restrict__ kc, __nv_bfloat16* __restrict__ vc, int batch, int s_new, int heads, int hd,
                                 int pos0, int max_seq, const int* __restrict__ pos_dev) {
  pdl_launch_dependents();
  pdl_wait();
  // one thread per 8 elements of one (token, head) row; pos_dev (optional) adds a device-resident offset so that a decode
  // step captured in a CUDA graph advances without host-side parameters
  if (pos_dev) pos0 += *pos_dev;
  const int vec = hd >> 3;
  const long long total = (long long)batch * s_new * heads * vec;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const int v = (int)(i % vec);
    long long r = i / vec;
    const int h = (int)(r % heads); r /= heads;
    const int s = (int)(r % s_new);
    const int b = (int)(r / s_new);
    const long long src = ((long long)b * s_new + s) * src_stride + h * hd + v * 8;
    if (pos0 + s >= max_seq) continue;           // a full cache drops the token (the host checks capacity before replaying)
    const long long dst = (((long long)b * heads + h) * max_seq + pos0 + s) * hd + v * 8;
    *reinterpret_cast<uint4*>(kc + dst) = *reinterpret_cast<const uint4*>(k_src + src);
    *reinterpret_cast<uint4*>(vc + dst) = *reinterpret_cast<const uint4*>(v_src + src);
  }
}

template <int HD>
__global__ void __launch_bounds__(128)
decode_attn_kernel(const __nv_bfloat16* __restrict__ q, long long q_stride, const __nv_bfloat16* __restrict__ kc,
                   const __nv_bfloat16* __restrict__ vc, __nv_bfloat16* __restrict__ out, long long out_stride, int heads, int len,
                   int max_seq, float scale_log2, const int* __restrict__ pos_dev) {
  pdl_launch_dependents();
  pdl_wait();
  if (pos_dev) len = min(len + *pos_dev, max_seq);
  constexpr int PER = HD / 32;                  // head-dim elements per lane in the p.v phase
  __shared__ float s_q[HD];
  __shared__ float s_m[4], s_l[4];
  __shared__ float s_acc[4][HD];
  const int b = blockIdx.x / heads, h = blockIdx.x % heads;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int d = threadIdx.x; d < HD; d += 128) s_q[d] = __bfloat162float(q[(long long)b * q_stride + h * HD + d]);
  __syncthreads();
  const __nv_bfloat16* kb = kc + ((long long)b * heads + h) * max_seq * HD;
  const __nv_bfloat16* vb = vc + ((long long)b * heads + h) * max_seq * HD;
  float m = -INFINITY, l = 0.f, acc[PER];
#pragma unroll
  for (int i = 0; i < PER; ++i) acc[i] = 0.f;
  for (int s0 = warp * 32; s0 < len; s0 += 128) {
    const int s = s0 + lane;
    float sc = -INFINITY;
    if (s < len) {
      const uint4* kr = reinterpret_cast<const uint4*>(kb + (long long)s * HD);
      float dot = 0.f;
#pragma unroll
      for (int j = 0; j < HD / 8; ++j) {
        const uint4 kv = kr[j];
        const float2 a = unpack_bf16x2(kv.x), c = unpack_bf16x2(kv.y), e = unpack_bf16x2(kv.z), g = unpack_bf16x2(kv.w);
        const float* qq = s_q + j * 8;
        dot += a.x * qq[0] + a.y * qq[1] + c.x * qq[2] + c.y * qq[3] + e.x * qq[4] + e.y * qq[5] + g.x * qq[6] + g.y * qq[7];
      }
      sc = dot * scale_log2;
    }
    const float m_new = fmaxf(m, warp_max(sc));
    const float p = s < len ? fast_exp2(sc - m_new) : 0.f;
    const float corr = m == -INFINITY ? 0.f : fast_exp2(m - m_new);
    l = l * corr + warp_sum(p);
    m = m_new;
#pragma unroll
    for (int i = 0; i < PER; ++i) acc[i] *= corr;
    const int n = min(32, len - s0);
    // p.v: eight value rows are loaded before the first multiply-add so that their latencies overlap
#pragma unroll 1
    for (int j0 = 0; j0 < n; j0 += 8) {
      uint2 vv[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int j = min(j0 + u, n - 1);
        const __nv_bfloat16* vr = vb + (long long)(s0 + j) * HD + lane * PER;
        if (PER == 4) vv[u] = *reinterpret_cast<const uint2*>(vr);
        else vv[u] = make_uint2(*reinterpret_cast<const uint32_t*>(vr), 0u);
      }
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const float pj = (j0 + u < n) ? __shfl_sync(0xffffffffu, p, (j0 + u) & 31) : 0.f;
        const float2 a = unpack_bf16x2(vv[u].x);
        acc[0] += pj * a.x; acc[1] += pj * a.y;
        if (PER == 4) {
          const float2 c = unpack_bf16x2(vv[u].y);
          acc[2] += pj * c.x; acc[3] += pj * c.y;
        }
      }
    }
  }
  if (lane == 0) { s_m[warp] = m; s_l[warp] = l; }
#pragma unroll
  for (int i = 0; i < PER; ++i) s_acc[warp][lane * PER + i] = acc[i];
  __syncthreads();
  const float M = fmaxf(fmaxf(s_m[0], s_m[1]), fmaxf(s_m[2], s_m[3]));
  float L = 0.f;
  float w[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) { w[k] = s_m[k] == -INFINITY ? 0.f : fast_exp2(s_m[k] - M); L += s_l[k] * w[k]; }
  for (int d = threadIdx.x; d < HD; d += 128) {
    const float v = s_acc[0][d] * w[0] + s_acc[1][d] * w[1] + s_acc[2][d] * w[2] + s_acc[3][d] * w[3];
    out[(long long)b * out_stride + h * HD + d] = __float2bfloat16_rn(L > 0.f ? v / L : 0.f);
  }
}


// ------------------------------------------------------------------------------------------------ streamed decode attention
// The cache of one (sequence, head) is contiguous, so a tile of TILE positions is one 16 KB block of K and one of V.  A
// producer thread streams those blocks into a 3-stage shared-memory ring with bulk asynchronous copies (completion counted
// on an mbarrier), four consumer warps compute out of shared memory: the memory system always has about 96 KB per CTA in
// flight, independent of how fast the arithmetic warps issue.  CTAs are persistent over (sequence, head, split) items; each
// item leaves an unnormalised partial (acc, m, l) that `decode_merge_kernel` combines; positions in one piece leave the result itself.
// Short contexts are bound by the warps' arithmetic on a tile, long ones by the cache's bytes: with packed multiply-adds and no branch on a
// probability (which kept a row's load behind the row before) 32 rows x 32 heads of 128 at 300 positions 36.0 -> 29.3 us (5.4 TB/s), at 2048
// 169.6 -> 162.8 (6.6 TB/s), 16 rows at 700 37.8 -> 32.7, 1 row at 130 6.2 -> 4.7; 64 rows x 16 heads of 64 at 512 33.5 -> 29.5.
// Merging only several pieces:
// (prompt of 100 and 32 steps of two 7B-class blocks with one row: 8.01 ms, 8.13 with the merge).
__device__ __forceinline__ void bulk_load_1d(void* smem_dst, const void* gsrc, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(smem_dst)),
               "l"(gsrc), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}
__device__ __forceinline__ void consumer_sync() { asm volatile("bar.sync 1, 128;" ::: "memory"); }

constexpr int DA_STAGES = 3;
constexpr int DA_TILE_BYTES = 16384;

template <int HD>
__global__ void __launch_bounds__(160)
decode_attn_stream_kernel(const __nv_bfloat16* __restrict__ q, long long q_stride, const __nv_bfloat16* __restrict__ kc,
                          const __nv_bfloat16* __restrict__ vc, float* __restrict__ partial, __nv_bfloat16* __restrict__ out, long long out_stride,
                          int heads, int n_bh, int splits, int len, int max_seq, float scale_log2, const int* __restrict__ pos_dev, int* __restrict__ status) {
  constexpr int LPR = HD / 64;            // lanes that share one row in the q.k phase (64 head-dim elements each)
  constexpr int RW = 32 / LPR;            // rows per warp and tile
  constexpr int TILE = 4 * RW;            // positions per tile: 64 (HD 128) or 128 (HD 64) -> 16 KB of K and of V
  constexpr int CH = HD / 8;              // 16-byte chunks per row
  constexpr int RG = 32 / CH;             // rows handled at once in the p.v phase
  static_assert(TILE * HD * 2 == DA_TILE_BYTES, "tile size");
  extern __shared__ __align__(128) unsigned char da_smem[];
  __shared__ uint64_t full_bar[DA_STAGES], empty_bar[DA_STAGES];
  __shared__ float4 s_qlo[16], s_qhi[16];
  __shared__ float s_m[4], s_l[4];
  __shared__ float s_acc[4][HD];
  __shared__ int s_fail;
  pdl_launch_dependents();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n_items = n_bh * splits;
  if (threadIdx.x == 0) {
    for (int i = 0; i < DA_STAGES; ++i) { mbar_init(&full_bar[i], 1); mbar_init(&empty_bar[i], 4); }
    mbar_fence_init();
    s_fail = 0;
  }
  __syncthreads();
  pdl_wait();
  if (pos_dev) len = min(len + *pos_dev, max_seq);
  const int per = (((len + splits - 1) / splits + TILE - 1) / TILE) * TILE;     // positions per split, whole tiles
  unsigned char* tiles = da_smem;

  if (warp == 4) {
    // ---------------------------------------------------------------- producer (one thread)
    if (lane == 0) {
      uint32_t it = 0;
      bool ok = true;
      for (int item = blockIdx.x; item < n_items && ok; item += gridDim.x) {
        const int bh = item / splits, sp = item - bh * splits;
        const int lo = sp * per, hi = min(len, lo + per);
        const __nv_bfloat16* kb = kc + (long long)bh * max_seq * HD;
        const __nv_bfloat16* vb = vc + (long long)bh * max_seq * HD;
        for (int pos = lo; pos < hi; pos += TILE, ++it) {
          const uint32_t stage = it % DA_STAGES, phase = (it / DA_STAGES) & 1u;
          if (!mbar_wait(&empty_bar[stage], phase ^ 1u)) { report_error(status, OA_KERR_WAIT_EMPTY); ok = false; break; }
          const uint32_t bytes = (uint32_t)min(TILE, hi - pos) * HD * 2u;
          mbar_expect_tx(&full_bar[stage], 2u * bytes);
          bulk_load_1d(tiles + stage * 2 * DA_TILE_BYTES, kb + (long long)pos * HD, bytes, &full_bar[stage]);
          bulk_load_1d(tiles + stage * 2 * DA_TILE_BYTES + DA_TILE_BYTES, vb + (long long)pos * HD, bytes, &full_bar[stage]);
        }
      }
    }
  } else {
    // ---------------------------------------------------------------- consumers (four warps)
    const int r = lane % RW, hh = lane / RW;            // q.k: row within the warp's rows, 64-element half of the row
    const int pc = lane % CH, pg = lane / CH;           // p.v: 16-byte chunk of the head dim, row group
    uint32_t it = 0;
    bool ok = true;
    for (int item = blockIdx.x; item < n_items; item += gridDim.x) {
      const int bh = item / splits, sp = item - bh * splits;
      const int b = bh / heads, h = bh - b * heads;
      const int lo = sp * per, hi = min(len, lo + per);
      if (threadIdx.x < HD / 4) {
        const __nv_bfloat16* qp = q + (long long)b * q_stride + h * HD + threadIdx.x * 4;
        const float4 v = make_float4(__bfloat162float(qp[0]), __bfloat162float(qp[1]), __bfloat162float(qp[2]), __bfloat162float(qp[3]));
        if (threadIdx.x & 1) s_qhi[threadIdx.x >> 1] = v; else s_qlo[threadIdx.x >> 1] = v;
      }
      consumer_sync();
      float m = -INFINITY, l = 0.f;
      unsigned long long acc2[4] = {0, 0, 0, 0};
      for (int pos = lo; pos < hi && ok; pos += TILE, ++it) {
        const uint32_t stage = it % DA_STAGES, phase = (it / DA_STAGES) & 1u;
        if (!warp_wait(&full_bar[stage], phase)) { report_error(status, OA_KERR_WAIT_FULL); ok = false; break; }
        const unsigned char* sk = tiles + stage * 2 * DA_TILE_BYTES;
        const unsigned char* sv = sk + DA_TILE_BYTES;
        const int row0 = warp * RW;                       // this warp's first row of the tile
        const int valid_rows = min(TILE, hi - pos) - row0; // rows of this warp that hold cached positions (may be <= 0)
        // q.k: each lane takes eight 16-byte chunks of its row, starting at a row-dependent chunk (no bank conflicts)
        unsigned long long d0 = 0, d1 = 0;
        const unsigned char* krow = sk + (row0 + r) * (HD * 2);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const int c = 8 * hh + ((j + r) & 7);
          const uint4 kv = *reinterpret_cast<const uint4*>(krow + c * 16);
          const ulonglong2 ql = *reinterpret_cast<const ulonglong2*>(&s_qlo[c]), qh = *reinterpret_cast<const ulonglong2*>(&s_qhi[c]);
          d0 = f2_fma(f2_bf16x2(kv.x), ql.x, d0);
          d1 = f2_fma(f2_bf16x2(kv.y), ql.y, d1);
          d0 = f2_fma(f2_bf16x2(kv.z), qh.x, d0);
          d1 = f2_fma(f2_bf16x2(kv.w), qh.y, d1);
        }
        uint32_t dw[2];
        f2_to(f2_add(d0, d1), dw[0], dw[1]);
        float dot = __uint_as_float(dw[0]) + __uint_as_float(dw[1]);
        if (LPR == 2) dot += __shfl_xor_sync(0xffffffffu, dot, 16);
        const bool live = r < valid_rows;
        const float sc = live ? dot * scale_log2 : -INFINITY;
        const float m_new = fmaxf(m, warp_max(sc));
        const float p = (live && m_new != -INFINITY) ? fast_exp2(sc - m_new) : 0.f;
        const float corr = (m == -INFINITY) ? 0.f : fast_exp2(m - m_new);
        l = l * corr + warp_sum(p) * (1.f / LPR);
        m = m_new;
        const unsigned long long corr2 = f2_of(__float_as_uint(corr), __float_as_uint(corr));
#pragma unroll
        for (int i = 0; i < 4; ++i) acc2[i] = f2_mul(acc2[i], corr2);
        // p.v: a quarter warp reads 128 contiguous bytes of one value row.  A row of probability 0 counts as zeros, whatever it holds (rows past
        // the end are what the ring held before); chosen and not branched on, so that the rows' loads are on their way together.
#pragma unroll
        for (int i = 0; i < RW / RG; ++i) {
          const int row = i * RG + pg;
          const float pj = __shfl_sync(0xffffffffu, p, row);
          uint4 vv = *reinterpret_cast<const uint4*>(sv + (row0 + row) * (HD * 2) + pc * 16);
          if (pj == 0.f) vv = make_uint4(0, 0, 0, 0);
          const unsigned long long pj2 = f2_of(__float_as_uint(pj), __float_as_uint(pj));
          acc2[0] = f2_fma(f2_bf16x2(vv.x), pj2, acc2[0]);
          acc2[1] = f2_fma(f2_bf16x2(vv.y), pj2, acc2[1]);
          acc2[2] = f2_fma(f2_bf16x2(vv.z), pj2, acc2[2]);
          acc2[3] = f2_fma(f2_bf16x2(vv.w), pj2, acc2[3]);
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&empty_bar[stage]);
      }
      float acc[8];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        uint32_t lo, hi;
        f2_to(acc2[i], lo, hi);
        acc[2 * i] = __uint_as_float(lo); acc[2 * i + 1] = __uint_as_float(hi);
      }
      // row groups of the p.v phase hold partial sums of the same chunk
#pragma unroll
      for (int o = CH; o < 32; o <<= 1)
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[i] += __shfl_xor_sync(0xffffffffu, acc[i], o);
      if (lane == 0) { s_m[warp] = m; s_l[warp] = l; if (!ok) s_fail = 1; }
      if (pg == 0) {
#pragma unroll
        for (int i = 0; i < 8; ++i) s_acc[warp][pc * 8 + i] = acc[i];
      }
      consumer_sync();
      const float M = fmaxf(fmaxf(s_m[0], s_m[1]), fmaxf(s_m[2], s_m[3]));
      float w[4], L = 0.f;
#pragma unroll
      for (int k = 0; k < 4; ++k) { w[k] = s_m[k] == -INFINITY ? 0.f : fast_exp2(s_m[k] - M); L += s_l[k] * w[k]; }
      if (threadIdx.x < HD) {
        const int d = threadIdx.x;
        const float v = s_acc[0][d] * w[0] + s_acc[1][d] * w[1] + s_acc[2][d] * w[2] + s_acc[3][d] * w[3];
        float* dst = partial + (long long)item * (HD + 2);
        if (splits == 1) {                                // the only piece: nothing to merge
          out[(long long)b * out_stride + h * HD + d] = __float2bfloat16_rn(L > 0.f ? v / L : 0.f);
        } else {
          dst[d] = v;
          if (d == 0) { dst[HD] = M; dst[HD + 1] = L; }
        }
      }
      const bool stop = s_fail != 0;                      // the same for all four warps: they leave together
      consumer_sync();
      if (stop) break;
    }
  }
  __syncthreads();
}

// out[b, h, :] = sum_s acc_s * 2^(m_s - M) / sum_s l_s * 2^(m_s - M)
template <int HD>
__global__ void decode_merge_kernel(const float* __restrict__ partial, __nv_bfloat16* __restrict__ out, long long out_stride, int heads,
                                    int splits) {
  pdl_launch_dependents();
  pdl_wait();
  const int bh = blockIdx.x, b = bh / heads, h = bh - b * heads, d = threadIdx.x;
  const float* src = partial + (long long)bh * splits * (HD + 2);
  float M = -INFINITY;
  for (int s = 0; s < splits; ++s) M = fmaxf(M, src[s * (HD + 2) + HD]);
  float L = 0.f, v = 0.f;
  for (int s = 0; s < splits; ++s) {
    const float ms = src[s * (HD + 2) + HD];
    const float w = ms == -INFINITY ? 0.f : fast_exp2(ms - M);
    L += src[s * (HD + 2) + HD + 1] * w;
    v += src[s * (HD + 2) + d] * w;
  }
  out[(long long)b * out_stride + h * HD + d] = __float2bfloat16_rn(L > 0.f ? v / L : 0.f);
}

// One new token per sequence: the rotate-half embedding of q and k in place and the append of k and v to the cache, which as launches of
// their own cost a decoding step 4.2 and 1.9 us (the same 32 steps: 8.14 ms, 8.33 with two launches; 32 rows, 48 steps 20.1 and 20.4).  A block takes eight of a row's 2 H rotated heads (and the v heads beside its k
// heads); its first hd / 2 threads compute one angle each, the same for every head, where the general kernel's threads compute
// eight one after the other.
constexpr int RA_HEADS = 8;
__global__ void __launch_bounds__(128)
rope_kv_append_kernel(__nv_bfloat16* x, long long row_stride, int heads, int hd, int pos, float theta, const int* __restrict__ pos_dev,
                      __nv_bfloat16* __restrict__ kc, __nv_bfloat16* __restrict__ vc, int max_seq) {
  __shared__ float s_cos[64], s_sin[64];
  pdl_launch_dependents();
  pdl_wait();
  if (pos_dev) pos += *pos_dev;
  const int b = blockIdx.x, half = hd >> 1;
  if ((int)threadIdx.x < half) {
    const float freq = __powf(theta, -2.f * (float)threadIdx.x / (float)hd);
    sincosf((float)pos * freq, &s_sin[threadIdx.x], &s_cos[threadIdx.x]);
  }
  __syncthreads();
  const bool fits = pos < max_seq;               // a full cache drops the token (the host checks capacity before replaying)
  const int jv = half >> 3;                      // 8-wide vectors per half head
  for (int i = threadIdx.x; i < RA_HEADS * jv; i += blockDim.x) {
    const int head = blockIdx.y * RA_HEADS + i / jv, j = (i % jv) * 8;
    if (head >= 2 * heads) break;
    __nv_bfloat16* row = x + b * row_stride + (long long)head * hd + j;
    const uint4 ua = *reinterpret_cast<const uint4*>(row), ub = *reinterpret_cast<const uint4*>(row + half);
    const uint32_t wa[4] = {ua.x, ua.y, ua.z, ua.w}, wb[4] = {ub.x, ub.y, ub.z, ub.w};
    uint32_t oa[4], ob[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float2 p = unpack_bf16x2(wa[k]), q = unpack_bf16x2(wb[k]);
      const float c0 = s_cos[j + 2 * k], c1 = s_cos[j + 2 * k + 1], s0 = s_sin[j + 2 * k], s1 = s_sin[j + 2 * k + 1];
      oa[k] = pack_bf16x2(p.x * c0 - q.x * s0, p.y * c1 - q.y * s1);
      ob[k] = pack_bf16x2(q.x * c0 + p.x * s0, q.y * c1 + p.y * s1);
    }
    const uint4 ra = make_uint4(oa[0], oa[1], oa[2], oa[3]), rb = make_uint4(ob[0], ob[1], ob[2], ob[3]);
    *reinterpret_cast<uint4*>(row) = ra;
    *reinterpret_cast<uint4*>(row + half) = rb;
    if (head >= heads && fits) {
      const long long at = (((long long)b * heads + head - heads) * max_seq + pos) * hd + j;
      const __nv_bfloat16* v = row + (long long)heads * hd;
      *reinterpret_cast<uint4*>(kc + at) = ra;
      *reinterpret_cast<uint4*>(kc + at + half) = rb;
      *reinterpret_cast<uint4*>(vc + at) = *reinterpret_cast<const uint4*>(v);
      *reinterpret_cast<uint4*>(vc + at + half) = *reinterpret_cast<const uint4*>(v + half);
    }
  }
}

// What comes before a replayed decoding step: the rows of the new tokens, fetched by the caller's ids into the step's own input, and the
// position moved on by one.  As nodes of the graph these are a copy of the ids, a gather and an addition of one number, three links of
// the step's chain; prompt of 100 and 32 steps of two 7B-class blocks with one row 8.15 -> 8.05 ms, 256 and 48 steps with 32 rows 19.92 -> 19.65.
__global__ void __launch_bounds__(256)
decode_begin_kernel(const uint4* __restrict__ table, const int* __restrict__ ids, uint4* __restrict__ x, int* pos, int vecs, int vocab,
                    const uint4* __restrict__ norm_w, uint4* __restrict__ x_w, float* __restrict__ squares) {
  __shared__ float red[8];
  pdl_launch_dependents();
  pdl_wait();
  const uint32_t nan2 = pack_bf16x2(__int_as_float(0x7fc00000), __int_as_float(0x7fc00000));
  const int row = blockIdx.x, id = ids[row];
  float ss = 0.f;
  for (int i = threadIdx.x; i < vecs; i += blockDim.x) {
    const uint4 v = id >= 0 && id < vocab ? table[(long long)id * vecs + i] : make_uint4(nan2, nan2, nan2, nan2);
    x[(long long)row * vecs + i] = v;
    if (!norm_w) continue;
    const uint4 w = norm_w[i];
    const uint32_t vs[4] = {v.x, v.y, v.z, v.w}, ws[4] = {w.x, w.y, w.z, w.w};
    uint32_t o[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float2 a = unpack_bf16x2(vs[k]), b = unpack_bf16x2(ws[k]);
      ss += a.x * a.x + a.y * a.y;
      o[k] = pack_bf16x2(a.x * b.x, a.y * b.y);
    }
    x_w[(long long)row * vecs + i] = make_uint4(o[0], o[1], o[2], o[3]);
  }
  if (row == 0 && threadIdx.x == 0) *pos += 1;
  if (!norm_w) return;
  ss = warp_sum(ss);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ss;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int k = 1; k < 8; ++k) ss += red[k];
    squares[row] = ss;
  }
}

}  // namespace oa

using namespace oa;

// x [n_ids, dim] = table[ids] (bf16; an id outside [0, vocab) gives a row of NaN), *pos += 1.  With norm_w [dim] also x_w = x * norm_w and
// squares [n_ids], the sums of the rows' squares.
extern "C" int oa_decode_begin(const void* table, const int* ids, void* x, int* pos, int n_ids, int dim, int vocab, const void* norm_w, void* x_w,
                               float* squares, void* stream) {
  if (dim % 8 || ((reinterpret_cast<uintptr_t>(table) | reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(norm_w) | reinterpret_cast<uintptr_t>(x_w)) & 15))
    return OA_ERR_ALIGN;
  if (n_ids <= 0 || dim <= 0 || (norm_w && (!x_w || !squares))) return OA_ERR_ARG;
  launch_short(decode_begin_kernel, dim3((unsigned)n_ids), dim3(256), 0, (cudaStream_t)stream, (const uint4*)table, ids, (uint4*)x, pos, dim / 8, vocab,
               (const uint4*)norm_w, (uint4*)x_w, squares);
  return cudaGetLastError() == cudaSuccess ? OA_OK : OA_ERR_LAUNCH;
}

// x: [batch, row_stride] rows q | k | v of `heads` heads each.  OA_ERR_UNSUPPORTED for head dims the vector path does not take.
extern "C" int oa_rope_kv_append(void* x, long long row_stride, int batch, int heads, int head_dim, int pos, float theta, const int* pos_dev, void* k_cache,
                                 void* v_cache, int max_seq, void* stream) {
  if (head_dim % 16 || head_dim < 16 || head_dim > 128 || heads <= 0 || batch > 0x7fffffff / 4) return OA_ERR_UNSUPPORTED;
  if (row_stride % 8 || ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(k_cache) | reinterpret_cast<uintptr_t>(v_cache)) & 15)) return OA_ERR_ALIGN;
  if (pos < 0 || (!pos_dev && pos >= max_seq)) return OA_ERR_ARG;
  if (batch <= 0) return OA_OK;
  launch_short(rope_kv_append_kernel, dim3((unsigned)batch, (unsigned)((2 * heads + RA_HEADS - 1) / RA_HEADS)), dim3(128), 0, (cudaStream_t)stream,
               (__nv_bfloat16*)x, row_stride, heads, head_dim, pos, theta, pos_dev, (__nv_bfloat16*)k_cache, (__nv_bfloat16*)v_cache, max_seq);
  return cudaGetLastError() == cudaSuccess ? OA_OK : OA_ERR_LAUNCH;
}

extern "C" int oa_kv_append(const void* k_src, const void* v_src, long long src_stride, void* k_cache, void* v_cache, int batch,
                            int s_new, int heads, int head_dim, int pos0, int max_seq, const int* pos_dev, void* stream) {
  if (head_dim % 8 || src_stride % 8) return OA_ERR_ALIGN;
  if (pos0 < 0 || (!pos_dev && pos0 + s_new > max_seq)) return OA_ERR_ARG;
  if (batch <= 0 || s_new <= 0) return OA_OK;
  const long long total = (long long)batch * s_new * heads * (head_dim / 8);
  const int threads = 256;
  const int blocks = (int)((total + threads - 1) / threads < 148 * 16 ? (total + threads - 1) / threads : 148 * 16);
  launch_short(kv_append_kernel, dim3(blocks), dim3(threads), 0, (cudaStream_t)stream, (const __nv_bfloat16*)k_src, (const __nv_bfloat16*)v_src,
               src_stride, (__nv_bfloat16*)k_cache, (__nv_bfloat16*)v_cache, batch, s_new, heads, head_dim, pos0, max_seq, pos_dev);
  return cudaGetLastError() == cudaSuccess ? OA_OK : OA_ERR_LAUNCH;
}

extern "C" int oa_decode_attn(const void* q, long long q_stride, const void* k_cache, const void* v_cache, void* out, long long out_stride,
                              int batch, int heads, int head_dim, int len, int max_seq, float scale, const int* pos_dev,
                              void* stream) {
  if (len <= 0 || len > max_seq) return OA_ERR_ARG;
  if (batch <= 0) return OA_OK;
  const float sl2 = scale * 1.4426950408889634f;
  cudaStream_t st = (cudaStream_t)stream;
  const int grid = batch * heads;
  if (head_dim == 128)
    decode_attn_kernel<128><<<grid, 128, 0, st>>>((const __nv_bfloat16*)q, q_stride, (const __nv_bfloat16*)k_cache, (const __nv_bfloat16*)v_cache,
                                                  (__nv_bfloat16*)out, out_stride, heads, len, max_seq, sl2, pos_dev);
  else if (head_dim == 64)
    decode_attn_kernel<64><<<grid, 128, 0, st>>>((const __nv_bfloat16*)q, q_stride, (const __nv_bfloat16*)k_cache, (const __nv_bfloat16*)v_cache,
                                                 (__nv_bfloat16*)out, out_stride, heads, len, max_seq, sl2, pos_dev);
  else return OA_ERR_UNSUPPORTED;
  return cudaGetLastError() == cudaSuccess ? OA_OK : OA_ERR_LAUNCH;
}

// Streamed variant: `partial` holds batch*heads*splits*(head_dim+2) floats.  Both kernels are captured together in a graph.
extern "C" size_t oa_decode_attn_stream_scratch_bytes(int batch, int heads, int head_dim, int splits) {
  return (size_t)batch * heads * splits * (head_dim + 2) * sizeof(float);
}

template <int HD>
static int launch_decode_stream(const void* q, long long q_stride, const void* kc, const void* vc, void* out, long long out_stride, int batch,
                                int heads, int len, int max_seq, float sl2, const int* pos_dev, void* partial, int splits, int* status,
                                cudaStream_t st) {
  static bool set = false;
  const int smem = DA_STAGES * 2 * DA_TILE_BYTES;
  if (!set) {
    if (cudaFuncSetAttribute(decode_attn_stream_kernel<HD>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) return OA_ERR_LAUNCH;
    set = true;
  }
  const int n_bh = batch * heads, items = n_bh * splits;
  const int grid = items < 2 * 148 ? items : 2 * 148;
  // Early launch only while a CTA has one item and most SMs have two CTAs.  CTAs that become resident as the launch before them drains
  // do not sit as a launch on a free chip places them: up to one per SM they come in pairs, and beyond 2 x 148 items the CTAs with an item
  // more share SMs (1024 items are four or three per CTA).  Prompt of 100 and 24 steps at the 7B-class width, 32 heads, with / without
  // the flag: 2 rows (64 items) 6.33 / 6.26 ms, 4 (128) 6.43 / 6.43, 6 (192) 6.71 / 6.76, 8 (256) 6.80 / 6.87, 10 (320) 6.85 / 6.81, 16
  // (512) 7.52 / 7.42, 32 (1024) 9.24 / 8.78, 40 10.2 / 9.59; 2600 positions, 2 rows (256) 10.1 / 10.4, 5 (1120) 17.0 / 16.9.
  const bool early = items > 148 && items <= 2 * 148;
  launch_pdl_if(pdl_on(early), decode_attn_stream_kernel<HD>, dim3(grid), dim3(160), smem, st, (const __nv_bfloat16*)q, q_stride, (const __nv_bfloat16*)kc,
               (const __nv_bfloat16*)vc, (float*)partial, (__nv_bfloat16*)out, out_stride, heads, n_bh, splits, len, max_seq, sl2, pos_dev, status);
  if (splits > 1) launch_short(decode_merge_kernel<HD>, dim3(n_bh), dim3(HD), 0, st, (const float*)partial, (__nv_bfloat16*)out, out_stride, heads, splits);
  return cudaGetLastError() == cudaSuccess ? OA_OK : OA_ERR_LAUNCH;
}

extern "C" int oa_decode_attn_stream(const void* q, long long q_stride, const void* k_cache, const void* v_cache, void* out,
                                     long long out_stride, int batch, int heads, int head_dim, int len, int max_seq, float scale,
                                     const int* pos_dev, void* partial, int splits, int* status, void* stream) {
  if (len <= 0 || len > max_seq || splits < 1 || splits > 64) return OA_ERR_ARG;
  if ((((uintptr_t)k_cache | (uintptr_t)v_cache) & 15) != 0) return OA_ERR_ALIGN;
  if (batch <= 0) return OA_OK;
  const float sl2 = scale * 1.4426950408889634f;
  if (head_dim == 128)
    return launch_decode_stream<128>(q, q_stride, k_cache, v_cache, out, out_stride, batch, heads, len, max_seq, sl2, pos_dev, partial, splits,
                                     status, (cudaStream_t)stream);
  if (head_dim == 64)
    return launch_decode_stream<64>(q, q_stride, k_cache, v_cache, out, out_stride, batch, heads, len, max_seq, sl2, pos_dev, partial, splits,
                                    status, (cudaStream_t)stream);
  return OA_ERR_UNSUPPORTED;
}
