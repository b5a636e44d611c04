// Exact-fp32 SIMT GEMM with arbitrary element strides, a batch dimension and the bias / activation
// epilogues.  It backs the engine's FP32 precision mode (the reference's only fully exercised
// precision) and the finite-difference gradient checks, where TF32/bf16 rounding is not acceptable.
// The bf16 path uses gemm_tcgen05.cu instead.
//   v = alpha * sum_k A[b][m*sam + k*sak] * B[b][n*sbn + k*sbk] + bias[n];  aux_out = v;  v = act(v) or v * act'(aux_in);
//   C[b][m,n] = v + residual (+ C)
// The epilogue carries what the bf16 kernel's does, so that a Transformer layer in fp32 launches no pass of its own for the saved
// pre-activation, the activation's gradient or the residual sum.
// Kernels of 256 threads and 64 x 64 (or 32 x 64) output tiles, the tiling class of the reference's GemmTiled
// (Source/Private/Oa/Core/Shader/Compute/Blas/Gemm/GemmTiled.slang:1-110), with runtime strides so that NT / NN / TN products and
// Bmm need no transposed copies.  Where each operand has one contiguous direction and 16-byte rows, an asynchronous ring of K tiles:
// gemm_f32_wide_kernel when one wave of blocks holds all tiles, else gemm_f32_tile_kernel, or gemm_f32_brief_kernel for short reductions;
// gemm_f32_kernel for any other strides (the next K tile prefetched into registers).  Few tiles with a long reduction: K is sliced over
// the blocks of a cluster, which add their sums up among themselves, or over more blocks still, and a second kernel adds the slices up;
// whichever adds up carries the epilogue.
#include <atomic>
#include <type_traits>

#include "common.cuh"
#include "api.h"

namespace oa {

constexpr int FT = 64, FK = 16;   // output tile width (and height of the plain kernel), columns of K per stage of the plain kernel
int num_sms();

struct F32Epi {
  const float *bias, *residual, *aux_in;
  float* aux_out;
  int ldr, ldaux, act, accumulate;
  float alpha;
  float* a_sum = nullptr;        // [M]: also the sums of A over K (bias gradient beside a weight gradient), by the blocks of the first columns
  int a_sum_accumulate = 0;
  int vec = 0;                   // wide kernel: rows of C and of all that the epilogue reads start on 16 bytes
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

// Four neighbouring columns at once.  `vec`: every row of C and of what the epilogue reads starts on 16 bytes (set by the host).
__device__ __forceinline__ void f32_epilogue4(const F32Epi& e, float4 acc, int m, int n, int M, int N, float* __restrict__ C, int ldc) {
  if (m >= M || n >= N) return;
  float* c = C + (long long)m * ldc + n;
  float v[4] = {acc.x, acc.y, acc.z, acc.w};
  if (!e.vec || n + 4 > N) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (n + i < N) c[i] = f32_epilogue(e, v[i], m, n + i, c + i);
    return;
  }
  auto get = [](const float* p, float* q) { *reinterpret_cast<float4*>(q) = *reinterpret_cast<const float4*>(p); };
  float u[4], z[4] = {0.f, 0.f, 0.f, 0.f};
  if (e.aux_in) get(e.aux_in + (long long)m * e.ldaux + n, z);
#pragma unroll
  for (int i = 0; i < 4; ++i) v[i] *= e.alpha;
  if (e.bias) {
    get(e.bias + n, u);
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] += u[i];
  }
  if (e.aux_out) *reinterpret_cast<float4*>(e.aux_out + (long long)m * e.ldaux + n) = make_float4(v[0], v[1], v[2], v[3]);
  if (e.act != OA_ACT_NONE) {
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = f32_activation(e.act, v[i], z[i]);
  }
  if (e.residual) {
    get(e.residual + (long long)m * e.ldr + n, u);
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] += u[i];
  }
  if (e.accumulate) {
    get(c, u);
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] += u[i];
  }
  *reinterpret_cast<float4*>(c) = make_float4(v[0], v[1], v[2], v[3]);
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
// four floats of padding); the columns a thread owns follow it, which leaves its 16-byte reads free of bank conflicts.  A thread's pieces of
// a stage are a fixed distance apart, so it carries one address per operand: with one for each piece 4096 x 4096 x 1024 took 2 % longer.
constexpr int F_THREADS = 256;
template <int ROWS, int MN, int KW>   // a [ROWS x KW] tile: [k][row] when MN, else [row][k]
struct F32Tile {
  static constexpr int PITCH = (MN ? ROWS : KW) + 4;
  static constexpr int FLOATS = (MN ? KW : ROWS) * PITCH;
  static constexpr int PIECES = ROWS * KW / 4 / F_THREADS;      // 16-byte pieces per thread
  static constexpr int PER = (MN ? ROWS : KW) / 4, JUMP = F_THREADS / PER;   // pieces side by side; rows (of either kind) from one piece of a thread to its next
  static_assert(PIECES * 4 * F_THREADS == ROWS * KW && JUMP * PER == F_THREADS, "whole pieces per thread");
  const float* src;                // this thread's first piece of the next stage
  long long jump, step;
  uint32_t dst;                    // byte offset inside a stage
  int along, across;               // floats from the piece to the end of its row; rows from the piece to the last
  __device__ __forceinline__ void start(const float* __restrict__ g, long long ld, int r0, int k_lo, int rows, int k_hi) {
    const int major = threadIdx.x / PER, minor = (threadIdx.x % PER) * 4, r = r0 + (MN ? minor : major), k = k_lo + (MN ? major : minor);
    step = MN ? (long long)KW * ld : KW;
    jump = (long long)JUMP * ld;
    along = MN ? rows - r : k_hi - k;
    across = MN ? k_hi - k : rows - r;
    dst = (uint32_t)(major * PITCH + minor) * 4u;
    src = g + (MN ? (long long)k * ld + r : (long long)r * ld + k);
  }
  __device__ __forceinline__ void fetch(uint32_t stage, const float* g) {      // pieces outside the matrix: any valid address, no bytes
    const int in = max(0, min(4, along)) * 4;
    const float* p = src;
#pragma unroll
    for (int q = 0; q < PIECES; ++q) {
      const int n = across > q * JUMP ? in : 0;
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(stage + dst + q * JUMP * PITCH * 4), "l"(n ? p : g), "r"(n) : "memory");
      p += jump;
    }
    src += step;
    if (MN) across -= KW;
    else along -= KW;
  }
};

// Tiles for more than one wave.  A thread owns 8 x 4 outputs: 128 threads cover 64 x 64, and the block's 256 threads are two such groups that
// each take their own eight columns of a stage and add their sums up, in group order, through shared memory at the end.  That is twelve
// 16-byte reads per 128 multiply-adds.
// What bounds it: multiply-adds at 55 to 70 % of their rate (4096 x 4096 x 1024 with both operands row-contiguous 706 us, 870 with both
// K-contiguous, where the pairs of a register file's double width do not lie side by side).  8 x 8 outputs per thread read less, but two
// such blocks do not fit the registers of an SM without spilling, and one leaves two waves of blocks nothing to overlap: 934 and 775 us for 725.
// No early trigger for the next launch: its blocks would sit in pairs where this kernel has left room, not one per SM, and two blocks
// of products share the multiply-add pipe.  A feed-forward of 2048 x 128 and 512 inner columns (two products) in a captured chain: 29.4 us
// without a trigger, 38.7 with one before the epilogue (30.0 without the flag on the launches); a data and weight gradient 28.8 and 40.9.
template <int A_MN, int B_MN>
__global__ void __launch_bounds__(F_THREADS, 2)
gemm_f32_tile_kernel(const float* __restrict__ A, const float* __restrict__ B, float* __restrict__ C, int M, int N, int K, long long lda,
                     long long ldb, int ldc, long long batch_a, long long batch_b, long long batch_c, const F32Epi epi, int k_chunk) {
  constexpr int ROWS = 64, KG = 2, KW = 8 * KG, STAGES = 4, TY = ROWS / 8;
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
  const int steps = (k_hi - k_lo + KW - 1) / KW;
  TA ta;
  TB tb;
  ta.start(A, lda, m0, k_lo, M, k_hi);
  tb.start(B, ldb, n0, k_lo, N, k_hi);
  const uint32_t ring0 = smem_u32(ring);
  int filled = 0, slot = 0;                           // stages requested so far, and the place of the next
  auto load = [&]() {
    if (filled < steps) {
      const uint32_t st = ring0 + slot * (STAGE * 4);
      ta.fetch(st, A);
      tb.fetch(st + TA::FLOATS * 4, B);
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

// Products over fewer than F_BRIEF_K columns of K with tiles for more than one wave: 4 x 4 outputs per thread over all of K, stored from
// registers.  Fewer registers leave room for more blocks per SM, and of a few stages of arithmetic what counts is how many blocks
// overlap their loads and stores.  Against the tile kernel: 2048 x 512 x 128 11.9 / 12.9 us, 8192 x 384 x 64 17 / 24, 4096 x 1024 x 160
// 40 / 48, 50000 x 32 x 32 10.5 / 17; 1024 x 1024 x 256 21.1 / 20.6 (18 with both operands row-contiguous).
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

template <int A_MN, int B_MN, int ROWS>
struct F32Wide {
  static constexpr int KG = 256 / ROWS, KW = 8 * KG, STAGES = 4;
  static constexpr int STAGE = F32Tile<ROWS, A_MN, KW>::FLOATS + F32Tile<FT, B_MN, KW>::FLOATS;
  static constexpr int PITCH = FT + (A_MN && !B_MN ? 4 : 8);    // of the groups' sums: the rows that a warp stores to at once fall into different banks
  static constexpr int SUMS = KG * ROWS * PITCH;
  static constexpr int SMEM = (STAGES * STAGE > SUMS ? STAGES * STAGE : SUMS) * 4;
};

// One block per SM and all tiles in one wave: 8 x 8 outputs per thread, 32 or 64 threads to a tile and 8 or 4 such groups on their own columns
// of K.  That is sixteen 16-byte reads per 256 multiply-adds, two thirds of the tile kernel's, and with an SM's registers for one block
// (150 to 230 a thread) the next reads are under way while these are multiplied; at the 128 registers of two blocks per SM, 2048 x 128 x 512
// took 13.0 us, no less than with 8 x 4 outputs.  Results leave in 16-byte pieces where C and what the epilogue reads allow it.
// What bounds it: 3.3 us of launch, first loads and epilogue, then 3.6 us per 256 columns of a 32-row tile, of which the multiply-adds need 2.2.
// 8 x 4 outputs / now, both operands K-contiguous, us: 2048 x 128 x 512 13.1 / 10.8, x 384 10.6 / 8.8, x 128 5.4 / 4.6, 2048 x 256 x 128
// 8.0 / 6.7, x 512 20.4 / 19.2, 300 x 300 x 300 9.2 / 7.4; both row-contiguous 11.2 / 10.1, 9.4 / 8.4, 5.0 / 4.5, 7.2 / 6.3, 18.0 / 17.0, 7.8 / 7.1.
// CLUSTER: blockIdx.z counts the slices of K, and the blocks of a cluster hold all of them: each adds its groups up, then finishes its
// share of the rows from everyone's shared memory, in slice order, so the result is reproducible.
template <int A_MN, int B_MN, int ROWS, int CLUSTER>
__global__ void __launch_bounds__(F_THREADS, 1)
gemm_f32_wide_kernel(const float* __restrict__ A, const float* __restrict__ B, float* __restrict__ C, int M, int N, int K, long long lda,
                     long long ldb, int ldc, long long batch_a, long long batch_b, long long batch_c, const F32Epi epi, int k_chunk) {
  using S = F32Wide<A_MN, B_MN, ROWS>;
  constexpr int KG = S::KG, KW = S::KW, STAGES = S::STAGES, STAGE = S::STAGE, TY = ROWS / 8, TX = FT / 8;
  using TA = F32Tile<ROWS, A_MN, KW>;
  using TB = F32Tile<FT, B_MN, KW>;
  extern __shared__ __align__(16) float ring[];
  __shared__ float slice_sum[ROWS];
  const int b = blockIdx.z;
  const int k_lo = k_chunk > 0 ? b * k_chunk : 0, k_hi = k_chunk > 0 ? min(K, k_lo + k_chunk) : K;
  if (k_chunk == 0) { A += (long long)b * batch_a; B += (long long)b * batch_b; }
  if (!CLUSTER) C += (long long)b * batch_c;
  const int m0 = blockIdx.y * ROWS, n0 = blockIdx.x * FT;
  const int group = threadIdx.x / (F_THREADS / KG), t = threadIdx.x % (F_THREADS / KG);
  const int tx = t % TX, ty = t / TX;
  const int steps = (k_hi - k_lo + KW - 1) / KW;
  TA ta;
  TB tb;
  ta.start(A, lda, m0, k_lo, M, k_hi);
  tb.start(B, ldb, n0, k_lo, N, k_hi);
  const uint32_t ring0 = smem_u32(ring);
  int filled = 0, slot = 0;                           // stages requested so far, and the place of the next
  auto load = [&]() {
    if (filled < steps) {
      const uint32_t st = ring0 + slot * (STAGE * 4);
      ta.fetch(st, A);
      tb.fetch(st + TA::FLOATS * 4, B);
    }
    ++filled;
    if (++slot == STAGES) slot = 0;
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  pdl_wait();
#pragma unroll
  for (int i = 0; i < STAGES - 1; ++i) load();
  // Two outputs per register pair where an operand's 16-byte reads leave two of its rows side by side (A row-contiguous: two rows of the
  // result, else B: two columns); one each where both operands are K-contiguous.
  constexpr int PAIR = A_MN ? 1 : (B_MN ? 2 : 0);
  constexpr int PR = PAIR == 1 ? 4 : 8, PC = PAIR == 2 ? 4 : 8;
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
#pragma unroll 8
        for (int k = 0; k < KW; ++k) {
          v += pa[k * TA::PITCH + threadIdx.x];
          if (k % 16 == 15) { f32_add_kept(a_sum, a_lost, v); v = 0.f; }
        }
      }
    }
#pragma unroll
    for (int kk = 0; kk < 8; kk += 4) {
      const int k0 = group * 8 + kk;
      if constexpr (PAIR == 0) {
        float bb[8][4];                               // [column][k]
#pragma unroll
        for (int c = 0; c < 8; ++c) *reinterpret_cast<float4*>(bb[c]) = *reinterpret_cast<const float4*>(pb + (tx + TX * c) * TB::PITCH + k0);
#pragma unroll
        for (int r = 0; r < 8; ++r) {
          const float4 v = *reinterpret_cast<const float4*>(pa + (ty + TY * r) * TA::PITCH + k0);
          const float a[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
          for (int k = 0; k < 4; ++k)
#pragma unroll
            for (int c = 0; c < 8; ++c) acc[r][c] = fmaf(a[k], bb[c][k], acc[r][c]);
        }
      } else if constexpr (PAIR == 1) {
        float bk[8][4];                               // [column][k]
        if constexpr (!B_MN) {
#pragma unroll
          for (int c = 0; c < 8; ++c) *reinterpret_cast<float4*>(bk[c]) = *reinterpret_cast<const float4*>(pb + (tx + TX * c) * TB::PITCH + k0);
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const ulonglong2 lo = *reinterpret_cast<const ulonglong2*>(pa + (k0 + k) * TA::PITCH + ty * 4);
          const ulonglong2 hi = *reinterpret_cast<const ulonglong2*>(pa + (k0 + k) * TA::PITCH + ROWS / 2 + ty * 4);
          const unsigned long long a[4] = {lo.x, lo.y, hi.x, hi.y};
          float b[8];
          if constexpr (B_MN) {
            *reinterpret_cast<float4*>(b) = *reinterpret_cast<const float4*>(pb + (k0 + k) * TB::PITCH + tx * 4);
            *reinterpret_cast<float4*>(b + 4) = *reinterpret_cast<const float4*>(pb + (k0 + k) * TB::PITCH + FT / 2 + tx * 4);
          } else {
#pragma unroll
            for (int c = 0; c < 8; ++c) b[c] = bk[c][k];
          }
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            const unsigned long long b2 = f2_of(__float_as_uint(b[c]), __float_as_uint(b[c]));
#pragma unroll
            for (int r = 0; r < 4; ++r) acc[r][c] = f2_fma(a[r], b2, acc[r][c]);
          }
        }
      } else {
        float a[8][4];                                // [row][k]
#pragma unroll
        for (int r = 0; r < 8; ++r) *reinterpret_cast<float4*>(a[r]) = *reinterpret_cast<const float4*>(pa + (ty + TY * r) * TA::PITCH + k0);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const ulonglong2 lo = *reinterpret_cast<const ulonglong2*>(pb + (k0 + k) * TB::PITCH + tx * 4);
          const ulonglong2 hi = *reinterpret_cast<const ulonglong2*>(pb + (k0 + k) * TB::PITCH + FT / 2 + tx * 4);
          const unsigned long long b[4] = {lo.x, lo.y, hi.x, hi.y};
#pragma unroll
          for (int r = 0; r < 8; ++r) {
            const unsigned long long a2 = f2_of(__float_as_uint(a[r][k]), __float_as_uint(a[r][k]));
#pragma unroll
            for (int c = 0; c < 4; ++c) acc[r][c] = f2_fma(a2, b[c], acc[r][c]);
          }
        }
      }
    }
  }
  if constexpr (CLUSTER) {
    if (A_MN && threadIdx.x < ROWS) slice_sum[threadIdx.x] = a_sum;
  } else if (A_MN && sums) {
    f32_store_sum(epi, a_sum, m0 + threadIdx.x, M, k_chunk > 0 ? b : 0);
  }
  __syncthreads();                                    // the last stage has been read; the copies still counted are empty
  constexpr int PITCH = S::PITCH;
  {
    float* mine = ring + group * (ROWS * PITCH);
    auto half = [](unsigned long long v, int h) -> float { return __uint_as_float((uint32_t)(h ? v >> 32 : v)); };
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      float* row = mine + (A_MN ? (r / 4) * (ROWS / 2) + ty * 4 + r % 4 : ty + TY * r) * PITCH;
      float v[8];
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        if constexpr (PAIR == 0) v[c] = acc[r][c];
        else if constexpr (PAIR == 1) v[c] = half(acc[r >> 1][c], r & 1);
        else v[c] = half(acc[r][c >> 1], c & 1);
      }
      if (B_MN) {
        *reinterpret_cast<float4*>(row + tx * 4) = make_float4(v[0], v[1], v[2], v[3]);
        *reinterpret_cast<float4*>(row + FT / 2 + tx * 4) = make_float4(v[4], v[5], v[6], v[7]);
      } else {
#pragma unroll
        for (int c = 0; c < 8; ++c) row[tx + TX * c] = v[c];
      }
    }
  }
  __syncthreads();
  auto group_sum = [&](int row, int col) -> float4 {
    const float* p = ring + row * PITCH + col;
    float4 v = *reinterpret_cast<const float4*>(p);
#pragma unroll
    for (int g = 1; g < KG; ++g) {
      const float4 u = *reinterpret_cast<const float4*>(p + g * (ROWS * PITCH));
      v.x += u.x; v.y += u.y; v.z += u.z; v.w += u.w;
    }
    return v;
  };
  if constexpr (CLUSTER) {
#pragma unroll
    for (int i = 0; i < ROWS * FT / 4 / F_THREADS; ++i) {
      const int e = i * F_THREADS + threadIdx.x, row = e / (FT / 4), col = e % (FT / 4) * 4;
      *reinterpret_cast<float4*>(ring + row * PITCH + col) = group_sum(row, col);
    }
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    const int slices = gridDim.z;                     // 2, 4 or 8: each block finishes an equal part of the rows
    const int rows = ROWS / slices;
    auto remote = [](uint32_t at, int rank) -> uint32_t {
      uint32_t a;
      asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(at), "r"(rank));
      return a;
    };
    for (int e = threadIdx.x; e < rows * (FT / 4); e += F_THREADS) {
      const int row = b * rows + e / (FT / 4), col = e % (FT / 4) * 4;
      const uint32_t own = ring0 + (uint32_t)(row * PITCH + col) * 4u;
      float4 part[8];
#pragma unroll
      for (int s = 0; s < 8; ++s)
        if (s < slices)
          asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(part[s].x), "=f"(part[s].y), "=f"(part[s].z), "=f"(part[s].w) : "r"(remote(own, s)));
      float4 v = part[0];
#pragma unroll
      for (int s = 1; s < 8; ++s)
        if (s < slices) { v.x += part[s].x; v.y += part[s].y; v.z += part[s].z; v.w += part[s].w; }
      f32_epilogue4(epi, v, m0 + row, n0 + col, M, N, C, ldc);
    }
    if (A_MN && epi.a_sum && blockIdx.x == 0 && b == 0 && threadIdx.x < ROWS) {
      float s = 0.f;
      for (int i = 0; i < slices; ++i) {
        float u;
        asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(u) : "r"(remote(smem_u32(slice_sum + threadIdx.x), i)));
        s += u;
      }
      f32_store_sum(epi, s, m0 + threadIdx.x, M, 0);
    }
    // no block leaves while another may still read its sums
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  } else {
#pragma unroll
    for (int i = 0; i < ROWS * FT / 4 / F_THREADS; ++i) {
      const int e = i * F_THREADS + threadIdx.x, row = e / (FT / 4), col = e % (FT / 4) * 4;
      f32_epilogue4(epi, group_sum(row, col), m0 + row, n0 + col, M, N, C, ldc);
    }
  }
}

template <int AM, int BMN, int ROWS, int CLUSTER>
static cudaError_t launch_f32_wide(dim3 grid, cudaStream_t st, const float* A, const float* B, float* C, int M, int N, int K, long long lda, long long ldb, int ldc,
                                   long long batch_a, long long batch_b, long long batch_c, const F32Epi& epi, int k_chunk) {
  constexpr int smem = F32Wide<AM, BMN, ROWS>::SMEM;
  auto kernel = gemm_f32_wide_kernel<AM, BMN, ROWS, CLUSTER>;
  // Devices on which the kernel may have this much shared memory already: asked before every launch, an eager product took 8.95 us of host time,
  // 8.78 since it is asked once (8.72 with a static ring)
  static std::atomic<unsigned long long> allowed{0};
  int dev = 0;
  if (cudaError_t rc = cudaGetDevice(&dev)) return rc;
  const unsigned long long bit = dev < 64 ? 1ull << dev : 0;
  if (!(allowed.load(std::memory_order_relaxed) & bit)) {
    if (cudaError_t rc = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem)) return rc;
    allowed.fetch_or(bit, std::memory_order_relaxed);
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(F_THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  int n = 0;
  if (pdl_on((long long)grid.x * grid.y * grid.z <= PDL_SHORT_BLOCKS)) {
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n++].val.programmaticStreamSerializationAllowed = 1;
  }
  if (CLUSTER) {
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = attr[n].val.clusterDim.y = 1;
    attr[n++].val.clusterDim.z = grid.z;
  }
  cfg.attrs = attr;
  cfg.numAttrs = n;
  return cudaLaunchKernelEx(&cfg, kernel, A, B, C, M, N, K, lda, ldb, ldc, batch_a, batch_b, batch_c, epi, k_chunk);
}

// false: the operands do not fit the tile kernels.  k_chunk > 0: slices of K, each with its own C (`batch_c` apart), or, with
// `cluster`, added up by the blocks themselves.
static bool gemm_f32_tiles(const float* A, const float* B, float* C, int M, int N, int K, long long sam, long long sak, long long sbn, long long sbk,
                           int ldc, int batch, long long batch_a, long long batch_b, long long batch_c, F32Epi epi, int k_chunk, int slices, bool cluster,
                           cudaStream_t st) {
  const bool a_k = sak == 1, b_k = sbk == 1;
  const long long lda = a_k ? sam : sak, ldb = b_k ? sbn : sbk;
  if ((!a_k && sam != 1) || (!b_k && sbn != 1) || ((lda | ldb | batch_a | batch_b) & 3) || lda < 0 || ldb < 0 || K <= 0 ||
      ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(B)) & 15))
    return false;
  const int z = k_chunk > 0 ? slices : batch;
  const long long wide = (N + FT - 1) / FT, tiles = wide * ((M + 63) / 64) * z, tiles32 = wide * ((M + 31) / 32) * z;
  // Beyond one wave two blocks on an SM share it better than one after the other: 2048 x 384 x 128 11.3 us in the brief kernel, 12.3 in the
  // wide one, 2048 x 384 x 192 14.5 to 16.0 against 13.3 with two blocks.  Up to eight columns of K one of the wide kernel's groups has all the
  // work and the others' sums are only added up: 20 x 48 x 8 2.77 us wide, 2.07 brief (the same sums), 2048 x 128 x 4 3.49 / 2.95; with A
  // row-contiguous 2.65 / 2.62 and, 64 x 64, 2.70 / 2.79.
  const bool one_wave = tiles <= num_sms() && (K > 8 || !a_k);
  const int rows = one_wave && (cluster || tiles32 <= num_sms()) ? 32 : 64;
  const bool brief = !one_wave && (k_chunk > 0 ? k_chunk : K) < F_BRIEF_K;
  const dim3 grid((unsigned)wide, (M + rows - 1) / rows, z);
  if (grid.y > 65535) return false;
  epi.vec = ((reinterpret_cast<uintptr_t>(C) | reinterpret_cast<uintptr_t>(epi.bias) | reinterpret_cast<uintptr_t>(epi.residual) | reinterpret_cast<uintptr_t>(epi.aux_in) |
              reinterpret_cast<uintptr_t>(epi.aux_out)) & 15) == 0 &&
            ((ldc | batch_c | (epi.residual ? epi.ldr : 0) | (epi.aux_in || epi.aux_out ? epi.ldaux : 0)) & 3) == 0;
#define OA_F32_RUN(KERNEL) launch_short(KERNEL, grid, dim3(F_THREADS), 0, st, A, B, C, M, N, K, lda, ldb, ldc, batch_a, batch_b, batch_c, epi, k_chunk)
#define OA_F32_WIDE(AM, BMN, ROWS, CL) launch_f32_wide<AM, BMN, ROWS, CL>(grid, st, A, B, C, M, N, K, lda, ldb, ldc, batch_a, batch_b, batch_c, epi, k_chunk)
#define OA_F32_TILE(AM, BMN)                                              \
  if (cluster) OA_F32_WIDE(AM, BMN, 32, 1);                               \
  else if (one_wave && rows == 32) OA_F32_WIDE(AM, BMN, 32, 0);           \
  else if (one_wave) OA_F32_WIDE(AM, BMN, 64, 0);                         \
  else if (brief) OA_F32_RUN((gemm_f32_brief_kernel<AM, BMN>));           \
  else OA_F32_RUN((gemm_f32_tile_kernel<AM, BMN>))
  if (a_k && b_k) { OA_F32_TILE(0, 0); }
  else if (a_k) { OA_F32_TILE(0, 1); }
  else if (b_k) { OA_F32_TILE(1, 0); }
  else { OA_F32_TILE(1, 1); }
#undef OA_F32_TILE
#undef OA_F32_WIDE
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
// 63 tiles and 64 slices: the partial sums take 64 MB at most.  128 x 128 x 4096 with a residual takes 148 us in one piece, 15 us in 32 slices.
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

// Slices of K that the blocks of a cluster add up themselves; 1: not sliced so.  A cluster's blocks have an SM each, so eight members for
// at most eight tiles (sixteen such clusters ran in two waves: 128 x 256 x 1024 10.5 us, 6.7 in two kernels), and 128 blocks at most.
// Two kernels slice finer, so where the cluster's blocks leave much of the chip idle or are long the line is the time of a slice (3.6 us
// per 256 columns).  Two kernels / a cluster, us: 128 x 128 x 512 5.4 / 4.8, x 1024 5.9 / 5.7, x 1536 6.1 / 6.7; 128 x 384 x 512 5.8 / 5.6,
// x 1024 8.5 / 7.7, x 1536 9.0 / 9.6; with more slices than the chip has SMs 512 x 128 x 1536 12.8 / 9.7, x 2048 13.1 / 11.6,
// x 3072 16.5 / 15.5, 384 x 256 x 1024 12.6 / 11.3.
static int f32_cluster(int M, int N, int K, int batch, int* k_chunk) {
  const long long tiles = (long long)((N + FT - 1) / FT) * ((M + 31) / 32);
  if (batch != 1 || K < 512 || tiles > 64) return 1;
  const int s = tiles <= 8 ? 8 : tiles <= 32 ? 4 : 2;
  const bool filled = tiles * s >= 96;
  int unused = 0;
  const long long tiles64 = (long long)((N + FT - 1) / FT) * ((M + FT - 1) / FT);
  const int chunk = ((K + s - 1) / s + 3) / 4 * 4;
  const int most = !filled ? 128 : tiles64 * f32_splits(M, N, K, batch, &unused) > num_sms() ? 768 : s >= 4 ? 256 : 0;
  if (chunk > most) return 1;
  *k_chunk = chunk;
  return s;
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
  const int members = oa::f32_cluster(M, N, K, batch, &k_chunk);
  if (members >= 2 && oa::gemm_f32_tiles(A, B, C, M, N, K, sam, sak, sbn, sbk, ldc, 1, 0, 0, 0, epi, k_chunk, members, true, st))
    return cudaGetLastError() == cudaSuccess ? OA_OK : OA_ERR_LAUNCH;
  k_chunk = 0;
  const int splits = scratch ? oa::f32_splits(M, N, K, batch, &k_chunk) : 1;
  if (splits >= 2) {
    grid.z = splits;
    float* part_sum = scratch + (long long)splits * M * N;
    if (epi.a_sum) part_epi.a_sum = part_sum;
    if (!oa::gemm_f32_tiles(A, B, scratch, M, N, K, sam, sak, sbn, sbk, N, 1, 0, 0, (long long)M * N, part_epi, k_chunk, splits, false, st))
      oa::gemm_f32_kernel<<<grid, 256, 0, st>>>(A, B, scratch, M, N, K, sam, sak, sbn, sbk, N, 0, 0, (long long)M * N, part_epi, k_chunk);
    const long long n = (long long)M * N;
    oa::launch_short(oa::gemm_f32_splitk_reduce_kernel, dim3((unsigned)((n + 255) / 256)), dim3(256), 0, st, (const float*)scratch, (const float*)part_sum, C, M, N, ldc, splits, epi);
    return cudaGetLastError() == cudaSuccess ? OA_OK : OA_ERR_LAUNCH;
  }
  if (!oa::gemm_f32_tiles(A, B, C, M, N, K, sam, sak, sbn, sbk, ldc, batch, batch_a, batch_b, batch_c, epi, 0, 0, false, st))
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
