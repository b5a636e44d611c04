// y[M, N] = act(alpha * x[M, K] W[N, K]^T + bias) + residual for a handful of rows (M <= 64): the products of token-by-token
// decoding, where the time is that of reading W once.
//
// W fills the 128-row side of the MMA (a tile is 128 output columns), the few rows of x are its N side, so that no tensor work
// or shared memory is spent on padding rows.  K is cut over the CTAs of a cluster (up to 8): every CTA streams its share of the
// tile's weights through a TMA ring into one TMEM accumulator, the partial tiles meet in distributed shared memory and every CTA
// sums, in rank order, and writes its share of the rows.  No workspace, no second kernel, no transposed copy.
//
// Two CTAs of about 100 KB per SM keep some 160 KB of weights per SM on their way.  Up to 2 x 128 columns per SM (37,888) one wave
// holds the whole grid: CTAs get equal shares of the bandwidth and of the bytes, whatever their number, so the cluster size only has
// to be large enough to have enough bytes in flight.  Wider products run further waves, whose tiles do not overlap their epilogues
// with the next tile's loads as the persistent tile kernel does; gemm_skinny_wins says where that costs more than it saves.
//
// What bounds it: the weights' bytes, at 5.6 TB/s in a long product (128-byte pieces of 128 rows), plus 4 to 6 us to start, to meet in
// the cluster and to store.  The start is taken off where the caller knows that nothing in flight writes W (w_at_rest, a decoding
// step replayed as a graph): a CTA fills its ring, 27 MB over the chip, under the kernels between two products, which are chained the
// same way (launch_short).  A prompt of 100 and 32 steps of two 7B-class blocks with one row: 8.84 ms with ordinary launches, 8.86 with
// chained ones alone, 8.14 with the weights requested ahead as well; 256 and 48 steps with 32 rows: 21.0, 20.8 and 20.1 ms (before what follows).
// A decoding step's norms and gates ride on the products (SkinnyParams): one row 8.08 -> 7.75 ms, 256 and 48 steps with 32 rows 18.92 -> 18.99
// (24 steps after a prompt of 100 8.50 -> 8.42).  The factors of the rows are worked out by the two warps that have nothing else to do, and
// bias, residual and the norm's weight requested, before the last product is waited for; after it they cost more than the norm's launch.
// One row against 12288 x 4096 / 4096 x 4096 / 32000 x 4096: 31 / 18 / 66 us, with the tile kernel 38 / 22 / 69; a decoding step of
// two 7B-class blocks and the head with 32 rows: 233 us of products, 336 us before (tile kernel on the transposed product, split-K
// reduction, transposing copy and residual add as launches of their own).  Below 512 columns of K or 256 of N the tile kernel's
// single tile is as fast (11 us either way), above 64 rows its padding is no longer waste.
#include "common.cuh"
#include "api.h"

namespace oa {

int make_tmap_3d_bf16(CUtensorMap* out, const void* ptr, uint64_t inner, uint64_t outer, uint64_t batch, uint64_t ld, uint64_t batch_stride,
                      uint32_t box_inner, uint32_t box_outer);
int num_sms();

constexpr int SK_BN = 128, SK_BK = 64, SK_THREADS = 128, SK_MAX_CLUSTER = 8;

struct SkinnyParams {
  int M, N, K, ldc, ldr, act, out_f32, cluster, w_at_rest;
  float alpha;
  void* out;
  const __nv_bfloat16 *bias, *residual;
  int* status;
  // Between the products of a decoding step stands an RMS norm, whose factor is one number per row: the product in front of it also leaves
  // its rows times the norm's weight and the sums of their squares by tile, and the one behind scales its result by the factor.
  const __nv_bfloat16* norm_w;     // [N] or null
  __nv_bfloat16* out_w;            // [M, N] out * norm_w
  float* squares_out;              // [tiles, M]
  const float* squares_in;         // [n_squares, M] or null: results are scaled by rsqrt(sum / K + eps)
  int n_squares;
  float eps;
  int gated;                       // > 0: W holds `gated` rows of gates and as many of values; out [M, gated] = silu(gate) * value
};

template <int MT>   // rows of x, padded to 16
struct SkinnyCfg {
  static constexpr int W_BYTES = SK_BN * SK_BK * 2, X_BYTES = MT * SK_BK * 2, STAGE_BYTES = W_BYTES + X_BYTES;
  static constexpr int STAGES = MT <= 16 ? 6 : MT <= 48 ? 5 : 4;
  static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024;   // + alignment slack
  static constexpr int TMEM_COLS = MT <= 32 ? 32 : 64;
  static_assert(SK_BN * MT * 4 <= STAGES * STAGE_BYTES, "the partial tile reuses the ring");
  static_assert(2 * (SMEM_BYTES + 1024 + 256) <= 228 * 1024, "two CTAs per SM");
};

// FUSED: the fields from norm_w on may be set; apart, because the plain kernel's epilogue is on the chain of every product.
template <int MT, bool FUSED>
__global__ void __launch_bounds__(SK_THREADS, 2)
gemm_skinny_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX, const SkinnyParams p) {
  using Cfg = SkinnyCfg<MT>;
  constexpr int NS = Cfg::STAGES;
  extern __shared__ uint8_t sk_raw[];
  __shared__ uint64_t full[NS], empty[NS], done;
  __shared__ uint32_t tmem_slot;
  __shared__ float s_factor[FUSED ? 64 : 1];         // of the norm in front, by row
  uint8_t* ring = sk_raw + ((1024u - (smem_u32(sk_raw) & 1023u)) & 1023u);   // the same offset in every CTA of the kernel
  pdl_launch_dependents();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int c = p.cluster, rank = (int)cluster_ctarank();
  const bool gated = FUSED && p.gated > 0;
  const int n0 = (int)(blockIdx.x / c) * (gated ? SK_BN / 2 : SK_BN);
  auto load_w = [&](uint8_t* d, uint64_t* bar, int k) {
    if (gated) {                                     // 64 rows of gates, the 64 rows of values that belong to them
      tma_load_3d(d, &tmW, bar, k, n0, 0);
      tma_load_3d(d + Cfg::W_BYTES / 2, &tmW, bar, k, p.gated + n0, 0);
    } else {
      tma_load_3d(d, &tmW, bar, k, n0, 0);
    }
  };
  const int kb = (p.K + SK_BK - 1) / SK_BK;
  const int kb0 = (int)((long long)kb * rank / c), kb1 = (int)((long long)kb * (rank + 1) / c);
  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmW); tma_prefetch_desc(&tmX);
    for (int s = 0; s < NS; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    mbar_init(&done, 1);
    mbar_fence_init();
    // The ring is empty: fill it before the block meets, and with weights that no kernel still in flight writes even before the
    // previous kernel has finished (only x comes from it).
    if (!p.w_at_rest) pdl_wait();
    for (int j = 0; j < NS && kb0 + j < kb1; ++j) {
      mbar_expect_tx(&full[j], Cfg::STAGE_BYTES);
      load_w(ring + j * Cfg::STAGE_BYTES, &full[j], (kb0 + j) * SK_BK);
    }
    pdl_wait();
    for (int j = 0; j < NS && kb0 + j < kb1; ++j)
      tma_load_3d(ring + j * Cfg::STAGE_BYTES + Cfg::W_BYTES, &tmX, &full[j], (kb0 + j) * SK_BK, 0, 0);
  }
  if (warp == 1) { tmem_alloc<Cfg::TMEM_COLS>(&tmem_slot); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t acc = tmem_slot;
  pdl_wait();                                       // the residual and the output are touched by all threads

  if (warp == 0) {
    for (int i = kb0 + NS; i < kb1; ++i) {
      const int j = i - kb0, st = j % NS;
      if (!warp_wait(&empty[st], ((j / NS) & 1) ^ 1)) { if (lane == 0) report_error(p.status, OA_KERR_WAIT_EMPTY); break; }
      if (elect_one()) {
        uint8_t* d = ring + st * Cfg::STAGE_BYTES;
        mbar_expect_tx(&full[st], Cfg::STAGE_BYTES);
        load_w(d, &full[st], i * SK_BK);
        tma_load_3d(d + Cfg::W_BYTES, &tmX, &full[st], i * SK_BK, 0, 0);
      }
      __syncwarp();
    }
  } else if (warp == 1) {
    constexpr uint32_t idesc = umma_idesc_bf16(SK_BN, MT, 0, 0);
    for (int i = kb0; i < kb1; ++i) {
      const int j = i - kb0, st = j % NS;
      if (!warp_wait(&full[st], (j / NS) & 1)) { if (lane == 0) report_error(p.status, OA_KERR_WAIT_FULL); break; }
      tc_fence_after();
      if (elect_one()) {
        const uint32_t wa = smem_u32(ring + st * Cfg::STAGE_BYTES), xa = wa + Cfg::W_BYTES;
#pragma unroll
        for (int ks = 0; ks < SK_BK / 16; ++ks)
          umma_f16(acc, umma_smem_desc_sw128(wa + ks * 32, 16, 1024), umma_smem_desc_sw128(xa + ks * 32, 16, 1024), idesc, (j > 0 || ks > 0) ? 1u : 0u);
        umma_commit(&empty[st]);
        if (i + 1 == kb1) umma_commit(&done);
      }
      __syncwarp();
    }
  } else if (FUSED && p.squares_in) {                // the other two warps, under the products
#pragma unroll 4
    for (int t = warp - 2; t < p.M; t += 2) {
      float ss = 0.f;
      for (int i = lane; i < p.n_squares; i += 32) ss += p.squares_in[(long long)i * p.M + t];
      ss = warp_sum(ss);
      if (lane == 0) s_factor[t] = rsqrtf(ss / (float)p.K + p.eps);
    }
  }
  __syncwarp();
  // what the results are added to and multiplied with, requested before the last product is waited for: of a warp's first row
  const int col = lane * 4, n = n0 + col;
  const bool in = gated || n < p.N;                  // N is a multiple of 8: the four columns of a lane are inside or outside together
  const int t0 = rank + c * warp;
  uint2 bias_w = make_uint2(0, 0), norm_w = make_uint2(0, 0), res_w = make_uint2(0, 0);
  if (in && !gated) {
    if (p.bias) bias_w = *reinterpret_cast<const uint2*>(p.bias + n);
    if (FUSED && p.norm_w) norm_w = *reinterpret_cast<const uint2*>(p.norm_w + n);
    if (p.residual && t0 < p.M) res_w = *reinterpret_cast<const uint2*>(p.residual + (long long)t0 * p.ldr + n);
  }
  if (!warp_wait(&done, 0)) { if (lane == 0) report_error(p.status, OA_KERR_WAIT_TMEM_FULL); }
  tc_fence_after();
  // partial tile [rows of x][128 output columns], fp32, over the drained ring
  float* part = reinterpret_cast<float*>(ring);
#pragma unroll
  for (int q = 0; q < MT / 16; ++q) {
    uint32_t r[16];
    tmem_ld16(acc + ((uint32_t)(warp * 32) << 16) + q * 16, r);
    tmem_ld_wait();
#pragma unroll
    for (int t = 0; t < 16; ++t) part[(q * 16 + t) * SK_BN + warp * 32 + lane] = __uint_as_float(r[t]);
  }
  tc_fence_before();
  cluster_sync_all();
  {
    // one warp per row, four columns per lane; all partial tiles of a piece are requested before the first one is added
    const uint32_t base = smem_u32(part);
    if (in || FUSED) {
      const float2 b01 = unpack_bf16x2(bias_w.x), b23 = unpack_bf16x2(bias_w.y), w01 = unpack_bf16x2(norm_w.x), w23 = unpack_bf16x2(norm_w.y);
      const float bias[4] = {b01.x, b01.y, b23.x, b23.y}, nw[4] = {w01.x, w01.y, w23.x, w23.y};
#pragma unroll 2
      for (int t = t0; t < p.M; t += 4 * c) {
        float4 u[SK_MAX_CLUSTER];
        const float alpha = FUSED && p.squares_in ? p.alpha * s_factor[t] : p.alpha;
        if (c == 1) {
          u[0] = *reinterpret_cast<const float4*>(part + t * SK_BN + col);
        } else {
#pragma unroll
          for (int j = 0; j < SK_MAX_CLUSTER; ++j)
            if (j < c)
              asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                           : "=f"(u[j].x), "=f"(u[j].y), "=f"(u[j].z), "=f"(u[j].w)
                           : "r"(map_to_cta(base + (uint32_t)(t * SK_BN + col) * 4u, (uint32_t)j)) : "memory");
        }
        float v[4] = {u[0].x, u[0].y, u[0].z, u[0].w};
#pragma unroll
        for (int j = 1; j < SK_MAX_CLUSTER; ++j)
          if (j < c) { v[0] += u[j].x; v[1] += u[j].y; v[2] += u[j].z; v[3] += u[j].w; }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          v[k] = v[k] * alpha + bias[k];
          if (p.act == OA_ACT_GELU) v[k] = gelu_tanh_fast(v[k]);
          else if (p.act == OA_ACT_RELU) v[k] = fmaxf(v[k], 0.f);
          else if (p.act == OA_ACT_SILU) v[k] = silu_f(v[k]);
        }
        if (gated) {                                // lanes 0..15 hold gates, 16..31 the values beside them
#pragma unroll
          for (int k = 0; k < 4; ++k) v[k] = silu_f(v[k]) * __shfl_down_sync(0xffffffffu, v[k], 16);
          if (lane < 16 && n < p.gated)
            *reinterpret_cast<uint2*>(reinterpret_cast<__nv_bfloat16*>(p.out) + (long long)t * p.ldc + n) = make_uint2(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]));
          continue;
        }
        if (p.residual && in) {
          const float2 r0 = unpack_bf16x2(res_w.x), r1 = unpack_bf16x2(res_w.y);
          if (t + 4 * c < p.M) res_w = *reinterpret_cast<const uint2*>(p.residual + (long long)(t + 4 * c) * p.ldr + n);
          v[0] += r0.x; v[1] += r0.y; v[2] += r1.x; v[3] += r1.y;
        }
        const uint2 o2 = make_uint2(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]));
        if (in) {
          if (p.out_f32) *reinterpret_cast<float4*>(reinterpret_cast<float*>(p.out) + (long long)t * p.ldc + n) = make_float4(v[0], v[1], v[2], v[3]);
          else *reinterpret_cast<uint2*>(reinterpret_cast<__nv_bfloat16*>(p.out) + (long long)t * p.ldc + n) = o2;
        }
        if (FUSED && p.norm_w) {                    // of the rounded rows, as a norm that reads them sees them
          const float2 a = unpack_bf16x2(o2.x), b = unpack_bf16x2(o2.y);
          const float ss = warp_sum(in ? a.x * a.x + a.y * a.y + b.x * b.x + b.y * b.y : 0.f);
          if (in) *reinterpret_cast<uint2*>(p.out_w + (long long)t * p.N + n) = make_uint2(pack_bf16x2(a.x * nw[0], a.y * nw[1]), pack_bf16x2(b.x * nw[2], b.y * nw[3]));
          if (lane == 0) p.squares_out[(long long)(blockIdx.x / c) * p.M + t] = ss;
        }
      }
    }
  }
  cluster_sync_all();                               // no CTA leaves while another one still reads its partial tile
  if (warp == 1) { tc_fence_after(); tmem_dealloc<Cfg::TMEM_COLS>(acc); }
}

template <int MT, bool FUSED>
static int launch_skinny(const CUtensorMap& tw, const CUtensorMap& tx, const SkinnyParams& p, int tiles, cudaStream_t st) {
  if (cudaFuncSetAttribute(gemm_skinny_kernel<MT, FUSED>, cudaFuncAttributeMaxDynamicSharedMemorySize, SkinnyCfg<MT>::SMEM_BYTES) != cudaSuccess) return OA_ERR_LAUNCH;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(tiles * p.cluster));
  cfg.blockDim = dim3(SK_THREADS);
  cfg.dynamicSmemBytes = SkinnyCfg<MT>::SMEM_BYTES;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)p.cluster;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl_mode() == PDL_NONE ? 1 : 2;
  return cudaLaunchKernelEx(&cfg, gemm_skinny_kernel<MT, FUSED>, tw, tx, p) == cudaSuccess && cudaGetLastError() == cudaSuccess ? OA_OK : OA_ERR_LAUNCH;
}

// Whether reading the weight this way beats the tile kernel: it depends on the weight's bytes against the output's, which a CTA writes
// after its last product and under nothing else.  While the tiles leave half of the SMs free it always does.  Up to one full wave, tile
// kernel against this one: 32 x 32000 x 512 12.8 / 12.1 us, 64 x 12288 x 512 9.0 / 10.7, 64 x 32000 x 1024 18.0 / 19.1, 48 x 18944 x 1024
// 14.4 / 13.3, 64 x 32000 x 4096 70 / 50.  Further waves: 64 x 50264 x 1024 27 / 32, 32 x 128256 x 2048 90 / 96, 16 x 50264 x 512 17 / 18,
// 48 x 50264 x 4096 80 / 79, 8 x 50264 x 1024 27 / 26.
bool gemm_skinny_wins(int M, int N, int K) {
  const long long tiles = (N + SK_BN - 1) / SK_BN, sms = num_sms();
  if (2 * tiles < sms) return true;
  if (tiles <= 2 * sms) return M <= 32 || K > 32 * M;
  return K > 64 * M;
}

static int run_skinny(const void* x, const void* w, int ldx, int ldw, int w_rows, SkinnyParams p, cudaStream_t st) {
  const int tile = p.gated ? SK_BN / 2 : SK_BN, cols = p.gated ? p.gated : p.N;
  const int mt = (p.M + 15) / 16 * 16, tiles = (cols + tile - 1) / tile, kb = (p.K + SK_BK - 1) / SK_BK;
  int c = 1;                                        // powers of two: a cluster of three left holes in the SMs' slots and a second wave
  while (c < SK_MAX_CLUSTER && 2 * c * tiles <= 2 * num_sms() && 2 * c <= kb / 4) c *= 2;
  CUtensorMap tw, tx;
  int rc;
  if ((rc = make_tmap_3d_bf16(&tw, w, (uint64_t)p.K, (uint64_t)w_rows, 1, (uint64_t)ldw, 0, SK_BK, (uint32_t)tile))) return rc;
  if ((rc = make_tmap_3d_bf16(&tx, x, (uint64_t)p.K, (uint64_t)p.M, 1, (uint64_t)ldx, 0, SK_BK, (uint32_t)mt))) return rc;
  p.cluster = c;
  const bool fused = p.norm_w || p.squares_in || p.gated;
#define OA_SK(MT) return fused ? launch_skinny<MT, true>(tw, tx, p, tiles, st) : launch_skinny<MT, false>(tw, tx, p, tiles, st)
  if (mt == 16) OA_SK(16);
  if (mt == 32) OA_SK(32);
  if (mt == 48) OA_SK(48);
  OA_SK(64);
#undef OA_SK
}

// Called by oa_gemm_bf16 for the shapes its dispatch names; the arguments have passed its checks.
int gemm_skinny(const void* x, const void* w, void* out, int M, int N, int K, int ldx, int ldw, int ldc, const void* bias, const void* residual,
                int ldr, int act, int out_f32, float alpha, int w_at_rest, int* status, cudaStream_t st) {
  SkinnyParams p = {};
  p.M = M; p.N = N; p.K = K; p.ldc = ldc; p.ldr = ldr; p.act = act; p.out_f32 = out_f32; p.alpha = alpha; p.w_at_rest = w_at_rest;
  p.out = out; p.bias = (const __nv_bfloat16*)bias; p.residual = (const __nv_bfloat16*)residual; p.status = status;
  return run_skinny(x, w, ldx, ldw, N, p, st);
}

}  // namespace oa

using namespace oa;

// Sums of squares by tile that oa_few_rows_step leaves for N columns
extern "C" int oa_few_rows_tiles(int N) { return (N + SK_BN - 1) / SK_BN; }

// One product of a decoding step, few rows of bf16, with what the RMS norms around it need:
//   scale = squares_in ? rsqrt(sum_i squares_in[i, t] / K + eps) : 1, x being rows times the norm's weight, before its factor;
//   gated == 0: out [M, N] = scale x W^T + bias + residual; with norm_w also out_w [M, N] = out * norm_w and squares_out [tiles, M];
//   gated > 0: W [2 gated, K] holds gates and values, out [M, gated] = silu(scale x Wg^T) * (scale x Wu^T).
// OA_ERR_UNSUPPORTED for shapes that the few-row kernel leaves to the tile kernels.
extern "C" int oa_few_rows_step(const void* x, const void* w, void* out, int M, int N, int K, int ldx, int ldw, int ldc, const void* bias, const void* residual,
                                int ldr, int gated, const void* norm_w, void* out_w, float* squares_out, const float* squares_in, int n_squares, float eps,
                                int w_at_rest, int* status, void* stream) {
  if (M <= 0 || N <= 0 || K <= 0 || gated < 0 || (gated && N != 2 * gated)) return OA_ERR_ARG;
  if ((N & 7) || (K & 7) || (gated & 7) || (ldc & 7) || (residual && (ldr & 7)) || (norm_w && (!out_w || !squares_out)) || (squares_in && n_squares < 1)) return OA_ERR_ALIGN;
  if ((reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(bias) | reinterpret_cast<uintptr_t>(residual) | reinterpret_cast<uintptr_t>(norm_w) |
       reinterpret_cast<uintptr_t>(out_w)) & 15)
    return OA_ERR_ALIGN;
  if (M > 64 || N < 256 || K < 512 || !gemm_skinny_wins(M, N, K) || (gated && (bias || residual || norm_w))) return OA_ERR_UNSUPPORTED;
  SkinnyParams p = {};
  p.M = M; p.N = N; p.K = K; p.ldc = ldc; p.ldr = ldr; p.act = OA_ACT_NONE; p.alpha = 1.f; p.w_at_rest = w_at_rest; p.status = status;
  p.out = out; p.bias = (const __nv_bfloat16*)bias; p.residual = (const __nv_bfloat16*)residual;
  p.norm_w = (const __nv_bfloat16*)norm_w; p.out_w = (__nv_bfloat16*)out_w; p.squares_out = squares_out;
  p.squares_in = squares_in; p.n_squares = n_squares; p.eps = eps; p.gated = gated;
  return run_skinny(x, w, ldx, ldw, N, p, (cudaStream_t)stream);
}
