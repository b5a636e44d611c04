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
// chained ones alone, 8.14 with the weights requested ahead as well; 256 and 48 steps with 32 rows: 21.0, 20.8 and 20.1 ms.
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

template <int MT>
__global__ void __launch_bounds__(SK_THREADS, 2)
gemm_skinny_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX, const SkinnyParams p) {
  using Cfg = SkinnyCfg<MT>;
  constexpr int NS = Cfg::STAGES;
  extern __shared__ uint8_t sk_raw[];
  __shared__ uint64_t full[NS], empty[NS], done;
  __shared__ uint32_t tmem_slot;
  uint8_t* ring = sk_raw + ((1024u - (smem_u32(sk_raw) & 1023u)) & 1023u);   // the same offset in every CTA of the kernel
  pdl_launch_dependents();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int c = p.cluster, rank = (int)cluster_ctarank();
  const int n0 = (int)(blockIdx.x / c) * SK_BN;
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
      tma_load_3d(ring + j * Cfg::STAGE_BYTES, &tmW, &full[j], (kb0 + j) * SK_BK, n0, 0);
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
        tma_load_3d(d, &tmW, &full[st], i * SK_BK, n0, 0);
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
  }
  __syncwarp();
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
    const int col = lane * 4, n = n0 + col;
    const uint32_t base = smem_u32(part);
    if (n < p.N) {                                  // N is a multiple of 8: the four columns of a lane are inside or outside together
      float bias[4] = {0.f, 0.f, 0.f, 0.f};
      if (p.bias) {
        const uint2 bw = *reinterpret_cast<const uint2*>(p.bias + n);
        const float2 b0 = unpack_bf16x2(bw.x), b1 = unpack_bf16x2(bw.y);
        bias[0] = b0.x; bias[1] = b0.y; bias[2] = b1.x; bias[3] = b1.y;
      }
#pragma unroll 2
      for (int t = rank + c * warp; t < p.M; t += 4 * c) {
        float4 u[SK_MAX_CLUSTER];
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
          v[k] = v[k] * p.alpha + bias[k];
          if (p.act == OA_ACT_GELU) v[k] = gelu_tanh_fast(v[k]);
          else if (p.act == OA_ACT_RELU) v[k] = fmaxf(v[k], 0.f);
          else if (p.act == OA_ACT_SILU) v[k] = silu_f(v[k]);
        }
        if (p.residual) {
          const uint2 rw = *reinterpret_cast<const uint2*>(p.residual + (long long)t * p.ldr + n);
          const float2 r0 = unpack_bf16x2(rw.x), r1 = unpack_bf16x2(rw.y);
          v[0] += r0.x; v[1] += r0.y; v[2] += r1.x; v[3] += r1.y;
        }
        if (p.out_f32) *reinterpret_cast<float4*>(reinterpret_cast<float*>(p.out) + (long long)t * p.ldc + n) = make_float4(v[0], v[1], v[2], v[3]);
        else *reinterpret_cast<uint2*>(reinterpret_cast<__nv_bfloat16*>(p.out) + (long long)t * p.ldc + n) = make_uint2(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]));
      }
    }
  }
  cluster_sync_all();                               // no CTA leaves while another one still reads its partial tile
  if (warp == 1) { tc_fence_after(); tmem_dealloc<Cfg::TMEM_COLS>(acc); }
}

template <int MT>
static int launch_skinny(const CUtensorMap& tw, const CUtensorMap& tx, const SkinnyParams& p, int tiles, cudaStream_t st) {
  if (cudaFuncSetAttribute(gemm_skinny_kernel<MT>, cudaFuncAttributeMaxDynamicSharedMemorySize, SkinnyCfg<MT>::SMEM_BYTES) != cudaSuccess) return OA_ERR_LAUNCH;
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
  return cudaLaunchKernelEx(&cfg, gemm_skinny_kernel<MT>, tw, tx, p) == cudaSuccess && cudaGetLastError() == cudaSuccess ? OA_OK : OA_ERR_LAUNCH;
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

// Called by oa_gemm_bf16 for the shapes its dispatch names; the arguments have passed its checks.
int gemm_skinny(const void* x, const void* w, void* out, int M, int N, int K, int ldx, int ldw, int ldc, const void* bias, const void* residual,
                int ldr, int act, int out_f32, float alpha, int w_at_rest, int* status, cudaStream_t st) {
  const int mt = (M + 15) / 16 * 16, tiles = (N + SK_BN - 1) / SK_BN, kb = (K + SK_BK - 1) / SK_BK;
  int c = 1;                                        // powers of two: a cluster of three left holes in the SMs' slots and a second wave
  while (c < SK_MAX_CLUSTER && 2 * c * tiles <= 2 * num_sms() && 2 * c <= kb / 4) c *= 2;
  CUtensorMap tw, tx;
  int rc;
  if ((rc = make_tmap_3d_bf16(&tw, w, (uint64_t)K, (uint64_t)N, 1, (uint64_t)ldw, 0, SK_BK, SK_BN))) return rc;
  if ((rc = make_tmap_3d_bf16(&tx, x, (uint64_t)K, (uint64_t)M, 1, (uint64_t)ldx, 0, SK_BK, (uint32_t)mt))) return rc;
  SkinnyParams p;
  p.M = M; p.N = N; p.K = K; p.ldc = ldc; p.ldr = ldr; p.act = act; p.out_f32 = out_f32; p.cluster = c; p.alpha = alpha; p.w_at_rest = w_at_rest;
  p.out = out; p.bias = (const __nv_bfloat16*)bias; p.residual = (const __nv_bfloat16*)residual; p.status = status;
  if (mt == 16) return launch_skinny<16>(tw, tx, p, tiles, st);
  if (mt == 32) return launch_skinny<32>(tw, tx, p, tiles, st);
  if (mt == 48) return launch_skinny<48>(tw, tx, p, tiles, st);
  return launch_skinny<64>(tw, tx, p, tiles, st);
}

}  // namespace oa
