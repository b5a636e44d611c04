// Exact-fp32 SIMT GEMM with arbitrary element strides, a batch dimension and the bias / activation
// epilogues.  It backs the engine's FP32 precision mode (the reference's only fully exercised
// precision) and the finite-difference gradient checks, where TF32/bf16 rounding is not acceptable.
// The bf16 path uses gemm_tcgen05.cu instead.
//   v = alpha * sum_k A[b][m*sam + k*sak] * B[b][n*sbn + k*sbk] + bias[n];  aux_out = v;  v = act(v) or v * act'(aux_in);
//   C[b][m,n] = v + residual (+ C)
// The epilogue carries what the bf16 kernel's does, so that a Transformer layer in fp32 launches no pass of its own for the saved
// pre-activation, the activation's gradient or the residual sum.
// Three kernels of 256 threads and 64 x 64 (or 32 x 64) output tiles, the tiling class of the reference's GemmTiled
// (Source/Private/Oa/Core/Shader/Compute/Blas/Gemm/GemmTiled.slang:1-110), with runtime strides so that NT / NN / TN products and
// Bmm need no transposed copies: gemm_f32_tile_kernel where each operand has one contiguous direction and 16-byte rows (an
// asynchronous ring of K tiles), gemm_f32_brief_kernel for short reductions of such operands, gemm_f32_kernel for any other strides (the next K tile prefetched into registers).  Few tiles with a
// long reduction: K is sliced over more blocks, and the kernel that adds the slices up carries the epilogue.
#include <type_traits>

#include "common.cuh"
#include "api.h"

namespace oa {

constexpr int FT = 64, FK = 16;   // output tile width (and height of the plain kernel), columns of K per stage of the plain kernel

struct F32Epi {
  const float *bias, *residual, *aux_in;
  float* aux_out;
  int ldr, ldaux, act, accumulate;
  float alpha;
  float* a_sum = nullptr;        // [M]: also the sums of A over K (bias gradient beside a weight gradient), by the blocks of the first columns
  int a_sum_accumulate = 0;
};

// Not inlined: sixteen copies of tanhf and its gradient made the epilogue some tens of kilobytes of code, and a launch of a few
// microseconds waited for the instruction fetches of the copies it jumped over.
__device__ __noinline__ float f32_activation(int act, float v, float z) {
  if (act == OA_ACT_GELU) return gelu_tanh(v);
  if (act == OA_ACT_RELU) return fmaxf(v, 0.f);
  if (act == OA_ACT_SILU) return silu_f(v);
  if (act == OA_ACT_GELU_BWD) return v * gelu_tanh_grad(z);
  if (act == OA_ACT_RELU_BWD) return z > 0.f ? v : 0.f;
  return v;
}

__device__ __forceinline__ float f32_epilogue(const F32Epi& e, float acc, int m, int n, float* c) {
  float v = acc * e.alpha;
  if (e.bias) v += e.bias[n];
  if (e.aux_out) e.aux_out[(long long)m * e.ldaux + n] = v;
  if (e.act != OA_ACT_NONE) v = f32_activation(e.act, v, e.aux_in ? e.aux_in[(long long)m * e.ldaux + n] : 0.f);
  if (e.residual) v += e.residual[(long long)m * e.ldr + n];
  if (e.accumulate) v += *c;
  return v;
}

// sum += v with what the addition loses carried on (Kahan): a thread adds up all of K, where separate column sums had short chains, and
// one after the other 500 terms lost four times as much
__device__ __forceinline__ void f32_add_kept(float& sum, float& lost, float v) {
  const float y = v - lost, t = sum + y;
  const float e = (t - sum) - y;
  lost = fabsf(e) <= 3.4028235e38f ? e : 0.f;            // an infinite sum stays one
  sum = t;
}
__device__ __forceinline__ void f32_store_sum(const F32Epi& e, float s, int m, int M, int slice) {
  if (m >= M) return;
  float* o = e.a_sum + (long long)slice * M + m;
  *o = e.a_sum_accumulate ? *o + s : s;
}

__global__ void __launch_bounds__(256)
gemm_f32_kernel(const float* __restrict__ A, const float* __restrict__ B, float* __restrict__ C, int M, int N, int K,
                long long sam, long long sak, long long sbn, long long sbk, int ldc, long long batch_a,
                long long batch_b, long long batch_c, const F32Epi epi, int k_chunk) {
  __shared__ __align__(16) float sA[FK][FT + 4];
  __shared__ __align__(16) float sB[FK][FT + 4];
  const int b = blockIdx.z;
  // k_chunk > 0: split-K mode - blockIdx.z is the K slice (batch 1) and C is the slice's own [M, ldc] partial buffer
  const int k_lo = k_chunk > 0 ? b * k_chunk : 0;
  const int k_hi = k_chunk > 0 ? min(K, k_lo + k_chunk) : K;
  if (k_chunk > 0) {
    C += (long long)b * batch_c;
  } else {
    A += (long long)b * batch_a;
    B += (long long)b * batch_b;
    C += (long long)b * batch_c;
  }
  const int m0 = blockIdx.y * FT, n0 = blockIdx.x * FT;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  // 64x16 elements per operand, 256 threads -> 4 loads each; the faster-varying index follows the contiguous dimension
  int ar[4], ak[4], br[4], bk[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int idx = threadIdx.x + i * 256;
    if (sak == 1) { ak[i] = idx & 15; ar[i] = idx >> 4; } else { ar[i] = idx & 63; ak[i] = idx >> 6; }
    if (sbk == 1) { bk[i] = idx & 15; br[i] = idx >> 4; } else { br[i] = idx & 63; bk[i] = idx >> 6; }
  }
  float ra[4], rb[4];
  auto fetch = [&](int k0) {       // global -> registers (the next tile is in flight while this one is multiplied)
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int gm = m0 + ar[i], gka = k0 + ak[i], gn = n0 + br[i], gkb = k0 + bk[i];
      ra[i] = (gm < M && gka < k_hi) ? A[gm * sam + gka * sak] : 0.f;
      rb[i] = (gn < N && gkb < k_hi) ? B[gn * sbn + gkb * sbk] : 0.f;
    }
  };
  auto stash = [&]() {
#pragma unroll
    for (int i = 0; i < 4; ++i) { sA[ak[i]][ar[i]] = ra[i]; sB[bk[i]][br[i]] = rb[i]; }
  };
  float acc[4][4] = {};
  if (k_lo < k_hi) fetch(k_lo);
  for (int k0 = k_lo; k0 < k_hi; k0 += FK) {
    stash();
    __syncthreads();
    if (k0 + FK < k_hi) fetch(k0 + FK);
#pragma unroll
    for (int kk = 0; kk < FK; ++kk) {
      const float4 a4 = *reinterpret_cast<const float4*>(&sA[kk][ty * 4]);
      const float4 b4 = *reinterpret_cast<const float4*>(&sB[kk][tx * 4]);
      const float a[4] = {a4.x, a4.y, a4.z, a4.w}, bb[4] = {b4.x, b4.y, b4.z, b4.w};
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], bb[j], acc[i][j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    int gm = m0 + ty * 4 + i;
    if (gm >= M) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      int gn = n0 + tx * 4 + j;
      if (gn >= N) continue;
      float* c = C + (long long)gm * ldc + gn;
      *c = f32_epilogue(epi, acc[i][j], gm, gn, c);
    }
  }
}

// Operands with one contiguous direction and 16-byte rows: the tile arrives through a ring of 16-byte cp.async stages, so that a block
// waits for memory once instead of once per stage.  An operand keeps the layout it has in memory ([row][k], or [k][row], with
// four floats of padding); the columns a thread owns follow it, which leaves its 16-byte reads free of bank conflicts.
// A thread owns 8 x 4 outputs, whatever the tile: 64 threads cover 32 x 64, 128 cover 64 x 64, and the block's 256 threads are KG = 4 or
// 2 such groups that each take their own eight columns of a stage and add their sums up, in group order, through shared memory at the
// end.  That is twelve 16-byte reads per 128 multiply-adds; two or four rows per thread over all of K, the shape of the tile kernel
// before this one, read six or eight per 32 or 64, ran at 320 clocks per four columns of K where the reads alone need 80, and left a
// block of 2048 x 128 x 512 with 8 warps in step and nothing to hide their latencies.
// What bounds it: multiply-adds at half their rate in long reductions, the ramp of a launch and the two passes through the epilogue's
// shared memory in short ones.  Before -> now: 2048 x 128 x 512 20.3 -> 13.1 us,
// 512 x 512 x 512 20.5 -> 13.2, 128 x 128 x 4096 in slices 14.2 -> 11.6 to 13.3, 4096^3 with both operands row-contiguous 3.50 -> 2.72 ms,
// with both K-contiguous 3.57 -> 3.4 (there the pairs of a register file's double width do not lie side by side).
// No early trigger for the next launch: its blocks would sit in pairs where this kernel has left room, not one per SM, and two blocks
// of products share the multiply-add pipe.  A feed-forward of 2048 x 128 and 512 inner columns (two products) in a captured chain: 29.4 us
// without a trigger, 38.7 with one before the epilogue (30.0 without the flag on the launches); a data and weight gradient 28.8 and 40.9.
constexpr int F_THREADS = 256;
template <int ROWS, int MN, int KW>   // a [ROWS x KW] tile: [k][row] when MN, else [row][k]
struct F32Tile {
  static constexpr int PITCH = (MN ? ROWS : KW) + 4;
  static constexpr int FLOATS = (MN ? KW : ROWS) * PITCH;
  static constexpr int PIECES = ROWS * KW / 4 / F_THREADS;      // 16-byte pieces per thread
  static_assert(PIECES * 4 * F_THREADS == ROWS * KW, "whole pieces per thread");
  const float* src[PIECES];        // this thread's pieces of the next stage (rows outside the matrix: any valid address, no bytes)
  uint32_t dst[PIECES];            // byte offset inside a stage
  int bytes[PIECES], left[PIECES]; // bytes of a whole stage; columns of K from the piece to the end of the slice
  long long step;
  __device__ __forceinline__ void start(const float* __restrict__ g, long long ld, int r0, int k_lo, int rows, int k_hi) {
    step = MN ? (long long)KW * ld : KW;
#pragma unroll
    for (int q = 0; q < PIECES; ++q) {
      const int i = threadIdx.x + q * F_THREADS;
      constexpr int PER = (MN ? ROWS : KW) / 4;
      const int major = i / PER, minor = (i % PER) * 4, r = MN ? minor : major, k = MN ? major : minor;
      bytes[q] = max(0, min(4, MN ? rows - (r0 + r) : (r0 + r < rows ? 4 : 0))) * 4;
      left[q] = k_hi - (k_lo + k);
      dst[q] = (uint32_t)(major * PITCH + minor) * 4u;
      src[q] = bytes[q] ? g + (MN ? (long long)(k_lo + k) * ld + r0 + r : (long long)(r0 + r) * ld + k_lo + k) : g;
    }
  }
  __device__ __forceinline__ void fetch(uint32_t stage, const float* g, bool whole) {
#pragma unroll
    for (int q = 0; q < PIECES; ++q) {
      int n = bytes[q];
      const float* p = src[q];
      if (!whole) {                                             // the slice ends inside this stage
        n = MN ? (left[q] > 0 ? n : 0) : min(n, max(0, min(4, left[q])) * 4);
        if (n == 0) p = g;
      }
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(stage + dst[q]), "l"(p), "r"(n) : "memory");
      if (bytes[q]) src[q] += step;
      left[q] -= KW;
    }
  }
};

template <int A_MN, int B_MN, int ROWS>
__global__ void __launch_bounds__(F_THREADS, 2)
gemm_f32_tile_kernel(const float* __restrict__ A, const float* __restrict__ B, float* __restrict__ C, int M, int N, int K, long long lda,
                     long long ldb, int ldc, long long batch_a, long long batch_b, long long batch_c, const F32Epi epi, int k_chunk) {
  constexpr int KG = 128 / ROWS, KW = 8 * KG, STAGES = ROWS == 32 ? 3 : 4, TY = ROWS / 8;
  using TA = F32Tile<ROWS, A_MN, KW>;
  using TB = F32Tile<FT, B_MN, KW>;
  constexpr int STAGE = TA::FLOATS + TB::FLOATS;
  __shared__ __align__(16) float ring[STAGES * STAGE];
  static_assert(KG * ROWS * FT <= STAGES * STAGE, "the groups' sums reuse the ring");
  const int b = blockIdx.z;
  const int k_lo = k_chunk > 0 ? b * k_chunk : 0, k_hi = k_chunk > 0 ? min(K, k_lo + k_chunk) : K;
  if (k_chunk == 0) { A += (long long)b * batch_a; B += (long long)b * batch_b; }
  C += (long long)b * batch_c;
  const int m0 = blockIdx.y * ROWS, n0 = blockIdx.x * FT;
  const int group = threadIdx.x / (F_THREADS / KG), t = threadIdx.x % (F_THREADS / KG);
  const int tx = t & 15, ty = t >> 4;
  const int steps = (k_hi - k_lo + KW - 1) / KW, whole = (k_hi - k_lo) / KW;
  TA ta;
  TB tb;
  ta.start(A, lda, m0, k_lo, M, k_hi);
  tb.start(B, ldb, n0, k_lo, N, k_hi);
  const uint32_t ring0 = smem_u32(ring);
  int filled = 0, slot = 0;                           // stages requested so far, and the place of the next
  auto load = [&]() {
    if (filled < steps) {
      const uint32_t st = ring0 + slot * (STAGE * 4);
      ta.fetch(st, A, filled < whole);
      tb.fetch(st + TA::FLOATS * 4, B, filled < whole);
    }
    ++filled;
    if (++slot == STAGES) slot = 0;
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  pdl_wait();
#pragma unroll
  for (int i = 0; i < STAGES - 1; ++i) load();
  // Sums of two outputs, or of the even and the odd columns of K of one output, per register pair: whichever way the operands' 16-byte
  // reads leave pairs side by side (K-major both: along K; A row-contiguous: two rows; else two columns).
  constexpr int PAIR = A_MN ? 1 : (B_MN ? 2 : 0);
  constexpr int PR = PAIR == 1 ? 4 : 8, PC = PAIR == 2 ? 2 : 4;
  using Acc = typename std::conditional<PAIR == 0, float, unsigned long long>::type;
  Acc acc[PR][PC] = {};
  const bool sums = A_MN && epi.a_sum && blockIdx.x == 0 && threadIdx.x < ROWS;
  float a_sum = 0.f, a_lost = 0.f;
  int at = 0;
  for (int i = 0; i < steps; ++i) {
    asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
    __syncthreads();                                  // stage i has landed everywhere, stage i - 1 has been read
    load();
    const float *pa = ring + at * STAGE, *pb = pa + TA::FLOATS;
    if (++at == STAGES) at = 0;
    if constexpr (A_MN) {
      if (sums) {
        float v = 0.f;
#pragma unroll
        for (int k = 0; k < KW; ++k) v += pa[k * TA::PITCH + threadIdx.x];
        f32_add_kept(a_sum, a_lost, v);
      }
    }
#pragma unroll
    for (int kk = 0; kk < 8; kk += 4) {
      const int k0 = group * 8 + kk;
      if constexpr (PAIR == 0) {
        float a[8][4], bb[4][4];                      // [row][k], [column][k]
#pragma unroll
        for (int c = 0; c < 4; ++c) *reinterpret_cast<float4*>(bb[c]) = *reinterpret_cast<const float4*>(pb + (tx + 16 * c) * TB::PITCH + k0);
#pragma unroll
        for (int r = 0; r < 8; ++r) *reinterpret_cast<float4*>(a[r]) = *reinterpret_cast<const float4*>(pa + (ty + TY * r) * TA::PITCH + k0);
#pragma unroll
        for (int k = 0; k < 4; ++k)
#pragma unroll
          for (int r = 0; r < 8; ++r)
#pragma unroll
            for (int c = 0; c < 4; ++c) acc[r][c] = fmaf(a[r][k], bb[c][k], acc[r][c]);
      } else if constexpr (PAIR == 1) {
        float bk[4][4];                               // [column][k]
        if constexpr (!B_MN) {
#pragma unroll
          for (int c = 0; c < 4; ++c) *reinterpret_cast<float4*>(bk[c]) = *reinterpret_cast<const float4*>(pb + (tx + 16 * c) * TB::PITCH + k0);
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const ulonglong2 lo = *reinterpret_cast<const ulonglong2*>(pa + (k0 + k) * TA::PITCH + ty * 8);
          const ulonglong2 hi = *reinterpret_cast<const ulonglong2*>(pa + (k0 + k) * TA::PITCH + ty * 8 + 4);
          const unsigned long long a[4] = {lo.x, lo.y, hi.x, hi.y};
          float b[4];
          if constexpr (B_MN) *reinterpret_cast<float4*>(b) = *reinterpret_cast<const float4*>(pb + (k0 + k) * TB::PITCH + tx * 4);
          else { b[0] = bk[0][k]; b[1] = bk[1][k]; b[2] = bk[2][k]; b[3] = bk[3][k]; }
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            const unsigned long long b2 = f2_of(__float_as_uint(b[c]), __float_as_uint(b[c]));
#pragma unroll
            for (int r = 0; r < 4; ++r) acc[r][c] = f2_fma(a[r], b2, acc[r][c]);
          }
        }
      } else {
        ulonglong2 b[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) b[k] = *reinterpret_cast<const ulonglong2*>(pb + (k0 + k) * TB::PITCH + tx * 4);
#pragma unroll
        for (int r = 0; r < 8; ++r) {
          const float4 v = *reinterpret_cast<const float4*>(pa + (ty + TY * r) * TA::PITCH + k0);
          const float a[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const unsigned long long a2 = f2_of(__float_as_uint(a[k]), __float_as_uint(a[k]));
            acc[r][0] = f2_fma(a2, b[k].x, acc[r][0]);
            acc[r][1] = f2_fma(a2, b[k].y, acc[r][1]);
          }
        }
      }
    }
  }
  if (A_MN && sums) f32_store_sum(epi, a_sum, m0 + threadIdx.x, M, k_chunk > 0 ? b : 0);
  __syncthreads();                                    // the last stage has been read; the copies still counted are empty
  {
    float* mine = ring + group * (ROWS * FT);
    auto half = [](unsigned long long v, int h) -> float { return __uint_as_float((uint32_t)(h ? v >> 32 : v)); };
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      float* row = mine + (A_MN ? ty * 8 + r : ty + TY * r) * FT;
      float v[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        if constexpr (PAIR == 0) v[c] = acc[r][c];
        else if constexpr (PAIR == 1) v[c] = half(acc[r >> 1][c], r & 1);
        else v[c] = half(acc[r][c >> 1], c & 1);
      }
      if (B_MN) {
        *reinterpret_cast<float4*>(row + tx * 4) = make_float4(v[0], v[1], v[2], v[3]);
      } else {
#pragma unroll
        for (int c = 0; c < 4; ++c) row[tx + 16 * c] = v[c];
      }
    }
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < ROWS * FT / F_THREADS; ++i) {
    const int e = i * F_THREADS + threadIdx.x, gm = m0 + e / FT, gn = n0 + e % FT;
    if (gm >= M || gn >= N) continue;
    float v = ring[e];
#pragma unroll
    for (int g = 1; g < KG; ++g) v += ring[g * (ROWS * FT) + e];
    float* o = C + (long long)gm * ldc + gn;
    *o = f32_epilogue(epi, v, gm, gn, o);
  }
}

// The same products over fewer than F_BRIEF_K columns of K with tiles for every SM: 4 x 4 outputs per thread over all of K, stored from
// registers.  Fewer registers leave room for more blocks per SM, and of a few stages of arithmetic what counts is how many blocks
// overlap their loads and stores.  Against the kernel above: 2048 x 512 x 128 11.9 / 12.9 us, 8192 x 384 x 64 17 / 24, 4096 x 1024 x 160
// 40 / 48, 50000 x 32 x 32 10.5 / 17; 1024 x 1024 x 256 21.1 / 20.6 (18 with both operands row-contiguous), 512 x 512 x 512 20.5 / 13.2.
constexpr int F_BRIEF_K = 192;
constexpr int FS = 4, FP_K = FK + 4, FP_MN = FT + 4, F_STAGE = FT * FP_K;
__device__ __forceinline__ void f32_cp16(float* dst, const float* src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(bytes) : "memory");
}
// the 16-byte pieces of a [ROWS x 16] tile; `ld` is the pitch of the direction that is not contiguous
template <int MN, int ROWS>
__device__ __forceinline__ void f32_fetch(float* sm, const float* __restrict__ g, long long ld, int r0, int k0, int rows, int k_hi) {
#pragma unroll
  for (int i = threadIdx.x; i < ROWS * 4; i += F_THREADS) {
    if (MN) {
      constexpr int PER = ROWS / 4;
      const int k = i / PER, r = (i % PER) * 4, left = rows - (r0 + r);
      const int bytes = k0 + k < k_hi ? max(0, min(4, left)) * 4 : 0;
      f32_cp16(sm + k * FP_MN + r, bytes ? g + (long long)(k0 + k) * ld + r0 + r : g, bytes);
    } else {
      const int r = i >> 2, k = (i & 3) * 4, left = k_hi - (k0 + k);
      const int bytes = r0 + r < rows ? max(0, min(4, left)) * 4 : 0;
      f32_cp16(sm + r * FP_K + k, bytes ? g + (long long)(r0 + r) * ld + k0 + k : g, bytes);
    }
  }
}

template <int A_MN, int B_MN>
__global__ void __launch_bounds__(F_THREADS)
gemm_f32_brief_kernel(const float* __restrict__ A, const float* __restrict__ B, float* __restrict__ C, int M, int N, int K, long long lda,
                     long long ldb, int ldc, long long batch_a, long long batch_b, long long batch_c, const F32Epi epi, int k_chunk) {
  constexpr int TM = 4, TY = F_THREADS / 16, ROWS = TY * TM;
  __shared__ __align__(16) float sA[FS][F_STAGE], sB[FS][F_STAGE];
  const int b = blockIdx.z;
  pdl_wait();
  const int k_lo = k_chunk > 0 ? b * k_chunk : 0, k_hi = k_chunk > 0 ? min(K, k_lo + k_chunk) : K;
  if (k_chunk == 0) { A += (long long)b * batch_a; B += (long long)b * batch_b; }
  C += (long long)b * batch_c;
  const int m0 = blockIdx.y * ROWS, n0 = blockIdx.x * FT;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const int steps = (k_hi - k_lo + FK - 1) / FK;
  auto load = [&](int i) {
    if (i < steps) {
      f32_fetch<A_MN, ROWS>(sA[i % FS], A, lda, m0, k_lo + i * FK, M, k_hi);
      f32_fetch<B_MN, FT>(sB[i % FS], B, ldb, n0, k_lo + i * FK, N, k_hi);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (int i = 0; i < FS - 1; ++i) load(i);
  float acc[TM][4] = {};
  const bool sums = A_MN && epi.a_sum && blockIdx.x == 0 && threadIdx.x < ROWS;
  float a_sum = 0.f, a_lost = 0.f;
  for (int i = 0; i < steps; ++i) {
    asm volatile("cp.async.wait_group %0;" ::"n"(FS - 2) : "memory");
    __syncthreads();                                  // stage i has landed everywhere, stage i - 1 has been read
    load(i + FS - 1);
    const float *pa = sA[i % FS], *pb = sB[i % FS];
    if constexpr (A_MN) {
      if (sums) {
        float v = 0.f;
#pragma unroll
        for (int k = 0; k < FK; ++k) v += pa[k * FP_MN + threadIdx.x];
        f32_add_kept(a_sum, a_lost, v);
      }
    }
#pragma unroll
    for (int kk = 0; kk < FK; kk += 4) {
      float a[4][TM], bb[4][4];                       // [k][row], [k][column]
      if (A_MN) {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
#pragma unroll
          for (int r = 0; r < TM; r += 2) {
            const float2 v = *reinterpret_cast<const float2*>(pa + (kk + k) * FP_MN + ty * TM + r);
            a[k][r] = v.x; a[k][r + 1] = v.y;
          }
        }
      } else {
#pragma unroll
        for (int r = 0; r < TM; ++r) {
          const float4 v = *reinterpret_cast<const float4*>(pa + (ty + TY * r) * FP_K + kk);
          a[0][r] = v.x; a[1][r] = v.y; a[2][r] = v.z; a[3][r] = v.w;
        }
      }
      if (B_MN) {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const float4 v = *reinterpret_cast<const float4*>(pb + (kk + k) * FP_MN + tx * 4);
          bb[k][0] = v.x; bb[k][1] = v.y; bb[k][2] = v.z; bb[k][3] = v.w;
        }
      } else {
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const float4 v = *reinterpret_cast<const float4*>(pb + (tx + 16 * c) * FP_K + kk);
          bb[0][c] = v.x; bb[1][c] = v.y; bb[2][c] = v.z; bb[3][c] = v.w;
        }
      }
#pragma unroll
      for (int k = 0; k < 4; ++k)
#pragma unroll
        for (int r = 0; r < TM; ++r)
#pragma unroll
          for (int c = 0; c < 4; ++c) acc[r][c] = fmaf(a[k][r], bb[k][c], acc[r][c]);
    }
  }
  if (A_MN && sums) f32_store_sum(epi, a_sum, m0 + threadIdx.x, M, k_chunk > 0 ? b : 0);
#pragma unroll
  for (int r = 0; r < TM; ++r) {
    const int gm = m0 + (A_MN ? ty * TM + r : ty + TY * r);
    if (gm >= M) continue;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int gn = n0 + (B_MN ? tx * 4 + c : tx + 16 * c);
      if (gn >= N) continue;
      float* o = C + (long long)gm * ldc + gn;
      *o = f32_epilogue(epi, acc[r][c], gm, gn, o);
    }
  }
}

// false: the operands do not fit the tile kernel
static bool gemm_f32_tiles(const float* A, const float* B, float* C, int M, int N, int K, long long sam, long long sak, long long sbn, long long sbk,
                           int ldc, int batch, long long batch_a, long long batch_b, long long batch_c, const F32Epi& epi, int k_chunk, int slices,
                           cudaStream_t st) {
  const bool a_k = sak == 1, b_k = sbk == 1;
  const long long lda = a_k ? sam : sak, ldb = b_k ? sbn : sbk;
  if ((!a_k && sam != 1) || (!b_k && sbn != 1) || ((lda | ldb | batch_a | batch_b) & 3) || lda < 0 || ldb < 0 || K <= 0 ||
      ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(B)) & 15))
    return false;
  const int z = k_chunk > 0 ? slices : batch;
  const long long tiles = (long long)((N + FT - 1) / FT) * ((M + FT - 1) / FT) * z;
  const int rows = tiles >= 148 ? 64 : 32;
  const bool brief = rows == 64 && (k_chunk > 0 ? k_chunk : K) < F_BRIEF_K;
  const dim3 grid((N + FT - 1) / FT, (M + rows - 1) / rows, z);
  if (grid.y > 65535) return false;
#define OA_F32_RUN(KERNEL) launch_short(KERNEL, grid, dim3(F_THREADS), 0, st, A, B, C, M, N, K, lda, ldb, ldc, batch_a, batch_b, batch_c, epi, k_chunk)
#define OA_F32_TILE(AM, BMN)                                              \
  if (brief) OA_F32_RUN((gemm_f32_brief_kernel<AM, BMN>));                \
  else if (rows == 64) OA_F32_RUN((gemm_f32_tile_kernel<AM, BMN, 64>));   \
  else OA_F32_RUN((gemm_f32_tile_kernel<AM, BMN, 32>))
  if (a_k && b_k) { OA_F32_TILE(0, 0); }
  else if (a_k) { OA_F32_TILE(0, 1); }
  else if (b_k) { OA_F32_TILE(1, 0); }
  else { OA_F32_TILE(1, 1); }
#undef OA_F32_TILE
#undef OA_F32_RUN
  return true;
}

// C[m,n] = epilogue(sum_s part[s][m,n]): fixed slice order, so the split-K result is reproducible
__global__ void gemm_f32_splitk_reduce_kernel(const float* __restrict__ part, const float* __restrict__ part_sum, float* __restrict__ C, int M, int N, int ldc,
                                              int splits, const F32Epi epi) {
  pdl_wait();
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (epi.a_sum && i < M) {
    float s = 0.f;
    for (int k = 0; k < splits; ++k) s += part_sum[(long long)k * M + i];
    f32_store_sum(epi, s, (int)i, M, 0);
  }
  if (i >= (long long)M * N) return;
  const int m = (int)(i / N), n = (int)(i % N);
  float s = 0.f;
  for (int k = 0; k < splits; ++k) s += part[((long long)k * M + m) * N + n];
  float* c = C + (long long)m * ldc + n;
  *c = f32_epilogue(epi, s, m, n, c);
}

// Slices of K for a product with few output tiles and a long reduction (weight gradients of small models); 1: not sliced.  At most
// 63 tiles and 64 slices: the partial sums take 64 MB at most.  The kernel that adds the slices up carries the epilogue: 128 x 128 x 4096
// with a residual takes 148 us in one piece, 15 us in 32 slices.
static int f32_splits(int M, int N, int K, int batch, int* k_chunk) {
  const long long tiles = (long long)((N + FT - 1) / FT) * ((M + FT - 1) / FT);
  if (batch != 1 || tiles >= 64 || K < 512) return 1;
  int splits = (int)((256 + tiles - 1) / tiles);
  if (splits > K / 128) splits = K / 128;
  if (splits > 64) splits = 64;
  if (splits < 2) return 1;
  *k_chunk = (((K + splits - 1) / splits) + FK - 1) / FK * FK;
  return (K + *k_chunk - 1) / *k_chunk;
}

}  // namespace oa

static int gemm_f32(const float* A, const float* B, float* C, int M, int N, int K, long long sam, long long sak, long long sbn, long long sbk,
                    int ldc, int batch, long long batch_a, long long batch_b, long long batch_c, const oa::F32Epi& epi, float* scratch, void* stream) {
  if (M <= 0 || N <= 0 || batch <= 0) return OA_OK;
  if (K < 0 || batch > 65535) return OA_ERR_ARG;
  oa::F32Epi part_epi{nullptr, nullptr, nullptr, nullptr, 0, 0, OA_ACT_NONE, 0, 1.0f};
  dim3 grid((N + oa::FT - 1) / oa::FT, (M + oa::FT - 1) / oa::FT, batch);
  cudaStream_t st = (cudaStream_t)stream;
  int k_chunk = 0;
  const int splits = scratch ? oa::f32_splits(M, N, K, batch, &k_chunk) : 1;
  if (splits >= 2) {
    grid.z = splits;
    float* part_sum = scratch + (long long)splits * M * N;
    if (epi.a_sum) part_epi.a_sum = part_sum;
    if (!oa::gemm_f32_tiles(A, B, scratch, M, N, K, sam, sak, sbn, sbk, N, 1, 0, 0, (long long)M * N, part_epi, k_chunk, splits, st))
      oa::gemm_f32_kernel<<<grid, 256, 0, st>>>(A, B, scratch, M, N, K, sam, sak, sbn, sbk, N, 0, 0, (long long)M * N, part_epi, k_chunk);
    const long long n = (long long)M * N;
    oa::launch_short(oa::gemm_f32_splitk_reduce_kernel, dim3((unsigned)((n + 255) / 256)), dim3(256), 0, st, (const float*)scratch, (const float*)part_sum, C, M, N, ldc, splits, epi);
    return cudaGetLastError() == cudaSuccess ? OA_OK : OA_ERR_LAUNCH;
  }
  if (!oa::gemm_f32_tiles(A, B, C, M, N, K, sam, sak, sbn, sbk, ldc, batch, batch_a, batch_b, batch_c, epi, 0, 0, st))
    oa::gemm_f32_kernel<<<grid, 256, 0, st>>>(A, B, C, M, N, K, sam, sak, sbn, sbk, ldc, batch_a, batch_b, batch_c, epi, 0);
  return cudaGetLastError() == cudaSuccess ? OA_OK : OA_ERR_LAUNCH;
}

// Floats of scratch with which the product's reduction is sliced (0: it never is).  The caller owns the scratch, so products on several
// streams or devices never share partial sums.
extern "C" size_t oa_gemm_f32_scratch_floats(int M, int N, int K, int batch) {
  int k_chunk = 0;
  if (M <= 0 || N <= 0) return 0;
  const int splits = oa::f32_splits(M, N, K, batch, &k_chunk);
  return splits >= 2 ? (size_t)splits * M * (N + 1) : 0;   // + the sums of A, when they are asked for
}

extern "C" int oa_gemm_f32(const float* A, const float* B, float* C, int M, int N, int K, long long sam, long long sak,
                           long long sbn, long long sbk, int ldc, int batch, long long batch_a, long long batch_b,
                           long long batch_c, const float* bias, int act, int accumulate, float alpha, float* scratch, void* stream) {
  if (act == OA_ACT_GELU_BWD || act == OA_ACT_RELU_BWD) return OA_ERR_UNSUPPORTED;
  return gemm_f32(A, B, C, M, N, K, sam, sak, sbn, sbk, ldc, batch, batch_a, batch_b, batch_c,
                  oa::F32Epi{bias, nullptr, nullptr, nullptr, 0, 0, act, accumulate, alpha}, scratch, stream);
}

extern "C" int oa_gemm_f32_epi(const float* A, const float* B, float* C, int M, int N, int K, long long sam, long long sak, long long sbn,
                               long long sbk, int ldc, const float* bias, const float* residual, int ldr, float* aux_out, const float* aux_in,
                               int ldaux, int act, int accumulate, float alpha, float* scratch, void* stream) {
  if ((act == OA_ACT_GELU_BWD || act == OA_ACT_RELU_BWD) && !aux_in) return OA_ERR_ARG;
  return gemm_f32(A, B, C, M, N, K, sam, sak, sbn, sbk, ldc, 1, 0, 0, 0, oa::F32Epi{bias, residual, aux_in, aux_out, ldr, ldaux, act, accumulate, alpha},
                  scratch, stream);
}

// C[M, N] (+)= A^T B for row-contiguous A [K, M] and B [K, N] (a weight gradient), and a_sum[M] (+)= the column sums of A (the bias
// gradient) from the same tiles.  OA_ERR_UNSUPPORTED: the operands do not fit the tile kernels, nothing was done.
extern "C" int oa_gemm_f32_weight_grad(const float* A, const float* B, float* C, int M, int N, int K, long long lda, long long ldb, int ldc, int accumulate,
                                       float* a_sum, int a_sum_accumulate, float* scratch, void* stream) {
  if (M <= 0 || N <= 0 || K <= 0 || ((lda | ldb) & 3) || lda < 0 || ldb < 0 || ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(B)) & 15) ||
      (M + 31) / 32 > 65535)
    return OA_ERR_UNSUPPORTED;
  oa::F32Epi epi{nullptr, nullptr, nullptr, nullptr, 0, 0, OA_ACT_NONE, accumulate, 1.0f};
  epi.a_sum = a_sum;
  epi.a_sum_accumulate = a_sum_accumulate;
  return gemm_f32(A, B, C, M, N, K, 1, lda, 1, ldb, ldc, 1, 0, 0, 0, epi, scratch, stream);
}
