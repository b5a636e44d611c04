// The chunk products of the Mamba-3 scan with everything between them, on the tensor cores: one CTA owns one chunk of 128 tokens
// of one (batch, head), state width 128, head width 64 (ops/mamba3_ssd.py states the algebra; other widths run the batched GEMMs
// and the kernels of mamba3_ssd.cu).
//
//   ssd_chunk_fwd   G = C~ B~^T -> M (decayed strict lower triangle + exact diagonal) -> y = M X + e^cum (C~ Hin^T), gate, token
//                   layout.  G and M live in TMEM: the fp32 score matrix (64 KB a chunk), the mask and the fp32 output never
//                   reach memory.
//   ssd_chunk_bwd   recomputes M, then dM = dY X^T and every product of the backward pass that needs only this chunk:
//                   dX = M^T dY + w (B~ dH^T), dC~ = dG B~ + e^cum (dY Hin) + dqk B~, dB~ = dG^T C~ + (w X) dH + dqk C~, and the row
//                   and column sums that carry d cum, d scale, d gamma, d w.  dC~ and dB~ leave once, in fp32.
// What bounds them: the bytes of the operands and, backward, the serial chain of a chunk (scores, mask, products, stores) on one CTA
// per SM.  2 x 4096 tokens x 48 heads: forward 77 -> 72 us, backward 337 -> 280 us since a row's results leave as 64 bytes at a time (16 bytes
// of a row to a lane touch 32 lines a store, and a chunk has 8,000 of them) and the next C~ and B~ arrive under the epilogue, 187 us
// with the mask in packed arithmetic, its blocks below the diagonal without a choice per element (the scheduler of the last 32 tokens, which
// meets every block of columns, took 7,800 of a chunk's 24,600 clocks for it), and a token's scalars and X requested ahead; the batched
// products and elementwise kernels they replace took 0.42 and 1.0 ms.
#include "common.cuh"
#include "api.h"

namespace oa {

int make_tmap_2d_bf16(CUtensorMap* out, const void* ptr, uint64_t inner, uint64_t outer, uint64_t ld, uint32_t box_inner, uint32_t box_outer);

constexpr int CQ = 128, CN = 128, CP = 64;          // tokens of a chunk, state width, head width
constexpr uint32_t HALF = CQ * 128;                 // bytes of one [128 rows x 64 bf16] half of a 128-column operand

// K-major step ks (16 columns) of a 128-column operand stored as 64-column halves of `rows` rows
__device__ __forceinline__ uint64_t desc_k(uint32_t addr, int ks, uint32_t half) { return umma_smem_desc_sw128(addr + (ks >> 2) * half + (ks & 3) * 32, 16, 1024); }
// MN-major step ks (16 rows); `half` = distance between 64-column groups
__device__ __forceinline__ uint64_t desc_mn(uint32_t addr, int ks, uint32_t half) { return umma_smem_desc_sw128(addr + ks * 2048, half, 1024); }

// ------------------------------------------------------------------------------------------------------------- forward
struct SsdChunkFwd {
  const float *cum, *scale, *gamma, *qk;            // [G, 128]
  const float* D;                                   // [H] or null
  const __nv_bfloat16* z; long long ldz;            // gate columns of the projection, null without the in-scan gate
  __nv_bfloat16 *y, *yraw; long long ldy;           // token layout [B*L, H*64]
  int H, nC, L;
  int* status;
};

struct ChunkFwdSmem {
  static constexpr int OFF_C = 0, OFF_B = 2 * HALF, OFF_X = 4 * HALF, OFF_H = 5 * HALF, OFF_F = 6 * HALF;   // Hin: two [64 x 64] boxes
  static constexpr int BYTES = OFF_F + 2 * CQ * 4 + 1024;
};

__global__ void __launch_bounds__(160, 2)
ssd_chunk_fwd_kernel(const __grid_constant__ CUtensorMap tmC, const __grid_constant__ CUtensorMap tmB, const __grid_constant__ CUtensorMap tmX,
                     const __grid_constant__ CUtensorMap tmH, const SsdChunkFwd p) {
  using S = ChunkFwdSmem;
  extern __shared__ uint8_t raw[];
  __shared__ uint64_t cb_full, h_full, x_full, g_full, m_full, y_full;
  __shared__ uint32_t tmem_slot;
  uint8_t* sm = raw + ((1024u - (smem_u32(raw) & 1023u)) & 1023u);
  float* s_cum = reinterpret_cast<float*>(sm + S::OFF_F);
  float* s_scale = s_cum + CQ;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = blockIdx.x;
  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmC); tma_prefetch_desc(&tmB); tma_prefetch_desc(&tmX); tma_prefetch_desc(&tmH);
    mbar_init(&cb_full, 1); mbar_init(&h_full, 1); mbar_init(&x_full, 1); mbar_init(&g_full, 1); mbar_init(&m_full, 4); mbar_init(&y_full, 1);
    mbar_fence_init();
  }
  if (warp == 4) { tmem_alloc<256>(&tmem_slot); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tm = tmem_slot;                    // G (M over its first half) | M X | C~ Hin^T = 128 + 64 + 64 columns

  if (warp == 4) {
    if (elect_one()) {
      mbar_expect_tx(&cb_full, 4 * HALF);
      for (int x = 0; x < 2; ++x) {
        tma_load_2d(sm + S::OFF_C + x * HALF, &tmC, &cb_full, x * 64, g * CQ);
        tma_load_2d(sm + S::OFF_B + x * HALF, &tmB, &cb_full, x * 64, g * CQ);
      }
      mbar_expect_tx(&h_full, HALF);
      for (int x = 0; x < 2; ++x) tma_load_2d(sm + S::OFF_H + x * (HALF / 2), &tmH, &h_full, x * 64, g * CP);
      mbar_expect_tx(&x_full, HALF);
      tma_load_2d(sm + S::OFF_X, &tmX, &x_full, 0, g * CQ);
    }
    __syncwarp();
    const uint32_t c_addr = smem_u32(sm + S::OFF_C), b_addr = smem_u32(sm + S::OFF_B), x_addr = smem_u32(sm + S::OFF_X), h_addr = smem_u32(sm + S::OFF_H);
    bool ok = warp_wait(&cb_full, 0);
    if (ok) {
      tc_fence_after();
      if (elect_one()) {
#pragma unroll
        for (int ks = 0; ks < CN / 16; ++ks)
          umma_f16(tm, desc_k(c_addr, ks, HALF), desc_k(b_addr, ks, HALF), umma_idesc_bf16(CQ, CQ, 0, 0), ks > 0);
        umma_commit(&g_full);
      }
      __syncwarp();
      ok = warp_wait(&h_full, 0);
    }
    if (ok) {
      tc_fence_after();
      if (elect_one())
#pragma unroll
        for (int ks = 0; ks < CN / 16; ++ks)
          umma_f16(tm + 192, desc_k(c_addr, ks, HALF), desc_k(h_addr, ks, HALF / 2), umma_idesc_bf16(CQ, CP, 0, 0), ks > 0);
      __syncwarp();
      ok = warp_wait(&x_full, 0) && warp_wait(&m_full, 0);
    }
    if (ok) {
      tc_fence_after();
      if (elect_one()) {
#pragma unroll
        for (int ks = 0; ks < CQ / 16; ++ks)
          umma_f16_ts(tm + 128, tm + ks * 8, desc_mn(x_addr, ks, HALF), umma_idesc_bf16(CQ, CP, 0, 1), ks > 0);
        umma_commit(&y_full);
      }
      __syncwarp();
    } else if (lane == 0) {
      report_error(p.status, OA_KERR_WAIT_FULL);
    }
  } else {
    const int t = threadIdx.x;                       // token of the chunk = TMEM lane
    const uint32_t t_lane = (uint32_t)(warp * 32) << 16;
    const long long gi = (long long)g * CQ + t;
    const int c = g % p.nC, bh = g / p.nC, h = bh % p.H, b = bh / p.H;
    const float ct = p.cum[gi];
    s_cum[t] = ct;
    s_scale[t] = p.scale[gi];
    const float diag = (p.D ? p.D[h] : 0.f) + p.gamma[gi] * p.qk[gi];
    asm volatile("bar.sync 1, 128;" ::: "memory");
    bool ok = warp_wait(&g_full, 0);
    tc_fence_after();
    if (ok) {
#pragma unroll 1
      for (int q = 0; q < 4; ++q) {                  // 32 columns at a time; those past the warp's rows are zero
        uint32_t m[16];
        if (q > warp) {
#pragma unroll
          for (int i = 0; i < 16; ++i) m[i] = 0u;
        } else {
          uint32_t v[32];
          tmem_ld32(tm + t_lane + q * 32, v);
          tmem_ld_wait();
          const float4 *cs4 = reinterpret_cast<const float4*>(s_cum + q * 32), *sc4 = reinterpret_cast<const float4*>(s_scale + q * 32);
          const int lim = t - q * 32;                // columns below it are decayed, itself is the diagonal
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const float4 cs = cs4[i], sc = sc4[i];
            float r[4] = {__uint_as_float(v[4 * i]) * __expf(ct - cs.x) * sc.x, __uint_as_float(v[4 * i + 1]) * __expf(ct - cs.y) * sc.y,
                          __uint_as_float(v[4 * i + 2]) * __expf(ct - cs.z) * sc.z, __uint_as_float(v[4 * i + 3]) * __expf(ct - cs.w) * sc.w};
            if (q == warp) {
#pragma unroll
              for (int j = 0; j < 4; ++j) r[j] = 4 * i + j < lim ? r[j] : (4 * i + j == lim ? diag : 0.f);
            }
            m[2 * i] = pack_bf16x2(r[0], r[1]);
            m[2 * i + 1] = pack_bf16x2(r[2], r[3]);
          }
        }
        tmem_st16(tm + t_lane + q * 16, m);          // M_q covers columns of G that this lane has already read
      }
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&m_full);
      ok = warp_wait(&y_full, 0);
    }
    if (ok) {
      tc_fence_after();
      const long long row = (long long)b * p.L + (long long)c * CQ + t;
      const float e = __expf(ct);
      const long long row4 = row - (lane & 3);           // rows of this lane's group of four: accesses cover 64 bytes of eight rows
      const int col4 = h * CP + (lane & 3) * 8;
#pragma unroll 1
      for (int q = 0; q < 2; ++q) {
        uint32_t u[32], v[32];
        uint4 zv[4], o[4], gated[4];
        if (p.z) {
#pragma unroll
          for (int k = 0; k < 4; ++k) zv[k] = *reinterpret_cast<const uint4*>(p.z + (row4 + k) * p.ldz + col4 + q * 32);
          exchange4(zv, lane);
        }
        tmem_ld32(tm + t_lane + 128 + q * 32, u);
        tmem_ld32(tm + t_lane + 192 + q * 32, v);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          float r[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) r[j] = fmaf(e, __uint_as_float(v[8 * i + j]), __uint_as_float(u[8 * i + j]));
          o[i] = make_uint4(pack_bf16x2(r[0], r[1]), pack_bf16x2(r[2], r[3]), pack_bf16x2(r[4], r[5]), pack_bf16x2(r[6], r[7]));
          if (p.z) {
            const uint32_t zs[4] = {zv[i].x, zv[i].y, zv[i].z, zv[i].w};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const float2 zf = unpack_bf16x2(zs[j]);
              r[2 * j] *= silu_f(zf.x); r[2 * j + 1] *= silu_f(zf.y);
            }
            gated[i] = make_uint4(pack_bf16x2(r[0], r[1]), pack_bf16x2(r[2], r[3]), pack_bf16x2(r[4], r[5]), pack_bf16x2(r[6], r[7]));
          }
        }
        exchange4(o, lane);
        __nv_bfloat16* raw_out = p.z ? p.yraw : p.y;
#pragma unroll
        for (int k = 0; k < 4; ++k) *reinterpret_cast<uint4*>(raw_out + (row4 + k) * p.ldy + col4 + q * 32) = o[k];
        if (p.z) {
          exchange4(gated, lane);
#pragma unroll
          for (int k = 0; k < 4; ++k) *reinterpret_cast<uint4*>(p.y + (row4 + k) * p.ldy + col4 + q * 32) = gated[k];
        }
      }
    } else if (lane == 0) {
      report_error(p.status, OA_KERR_WAIT_TMEM_FULL);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 4) { tc_fence_after(); tmem_dealloc<256>(tm); }
}

// ------------------------------------------------------------------------------------------------------------ backward
struct SsdChunkBwd {
  const float *cum, *scale, *gamma, *qk, *w;        // [G, 128]
  const float* D;
  const __nv_bfloat16* X;                           // [G, 128, 64]
  float *dC, *dB;                                   // [G, 128, 128]
  float *row_mm, *col_mm, *col_ge, *diag, *dcum_ce, *dw;   // [G, 128]
  __nv_bfloat16* dx; long long lddx;                // x columns of the projection gradient
  int H, nC, L, G;
  int* status;
};

struct ChunkBwdSmem {
  // Two regions of 64 KB change roles from chunk to chunk: one holds C~ | B~, the other M | dG (bf16, in the swizzle of the operands).  The
  // next chunk's C~ and B~ land where M and dG were as soon as the products have read those, under this chunk's epilogue.
  static constexpr int OFF_R0 = 0, OFF_X = 4 * HALF, OFF_XW = 5 * HALF, OFF_DY = 6 * HALF, OFF_H = 7 * HALF, OFF_DH = 8 * HALF, OFF_R1 = 9 * HALF;
  static constexpr int OFF_F = 13 * HALF;
  static constexpr int BYTES = OFF_F + (3 + 4 + 2 + 2) * CQ * 4 + 1024;
  static_assert(BYTES <= 227 * 1024, "shared memory");
};

// Sum over the 32 lanes of v[0..31]: lane l returns the total of column l.
__device__ __forceinline__ float lane_transpose_sum(float* v, int lane) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const bool up = lane & o;
#pragma unroll
    for (int i = 0; i < o; ++i) {
      const float send = up ? v[i] : v[i + o], keep = up ? v[i + o] : v[i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  }
  return v[0];
}

constexpr int CB_THREADS = 288;                     // 8 worker warps (two threads per token), 1 warp that loads and issues products
__global__ void __launch_bounds__(CB_THREADS, 1)
ssd_chunk_bwd_kernel(const __grid_constant__ CUtensorMap tmC, const __grid_constant__ CUtensorMap tmB, const __grid_constant__ CUtensorMap tmX,
                     const __grid_constant__ CUtensorMap tmXw, const __grid_constant__ CUtensorMap tmDY, const __grid_constant__ CUtensorMap tmH,
                     const __grid_constant__ CUtensorMap tmDH, const SsdChunkBwd p) {
  using S = ChunkBwdSmem;
  extern __shared__ uint8_t raw[];
  __shared__ uint64_t cb_full, ops_full, s_full, m_full, fin_full, acc_free, ops_free;
  __shared__ uint32_t tmem_slot;
  uint8_t* sm = raw + ((1024u - (smem_u32(raw) & 1023u)) & 1023u);
  float* s_ncum = reinterpret_cast<float*>(sm + S::OFF_F);
  float* s_scale = s_ncum + CQ;
  float* s_dqk = s_scale + CQ;
  float* s_col = s_dqk + CQ;                        // [4 row quadrants][128]
  float* s_row = s_col + 4 * CQ;                    // [2 column halves][128]
  float* s_fin = s_row + 2 * CQ;                    // [2][128]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmC); tma_prefetch_desc(&tmB); tma_prefetch_desc(&tmX); tma_prefetch_desc(&tmXw);
    tma_prefetch_desc(&tmDY); tma_prefetch_desc(&tmH); tma_prefetch_desc(&tmDH);
    mbar_init(&cb_full, 1); mbar_init(&ops_full, 1); mbar_init(&s_full, 1); mbar_init(&m_full, 8); mbar_init(&fin_full, 1);
    mbar_init(&acc_free, 8); mbar_init(&ops_free, 1);
    mbar_fence_init();
  }
  if (warp == 8) { tmem_alloc<512>(&tmem_slot); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tm = tmem_slot;
  // TMEM: G, then dC~ | dM, then dB~ | dY Hin | B~ dH^T | M^T dY
  constexpr uint32_t TM_A = 0, TM_B = 128, TM_CE = 256, TM_XW = 384, TM_X = 448;

  if (warp == 8) {
    const uint32_t x_a = smem_u32(sm + S::OFF_X), xw_a = smem_u32(sm + S::OFF_XW), dy_a = smem_u32(sm + S::OFF_DY), h_a = smem_u32(sm + S::OFF_H),
                   dh_a = smem_u32(sm + S::OFF_DH);
    uint32_t n = 0;
    bool ok = true;
    for (int g = blockIdx.x; g < p.G && ok; g += gridDim.x, ++n) {
      uint8_t* cb = sm + ((n & 1) ? S::OFF_R1 : S::OFF_R0);
      const uint32_t c_a = smem_u32(cb), b_a = c_a + 2 * HALF, m_a = smem_u32(sm + ((n & 1) ? S::OFF_R0 : S::OFF_R1)), dg_a = m_a + 2 * HALF;
      // the previous chunk's products have read their operands, M and dG
      ok = warp_wait(&ops_free, (n & 1) ^ 1);
      if (ok && elect_one()) {
        mbar_expect_tx(&cb_full, 4 * HALF);
        for (int x = 0; x < 2; ++x) {
          tma_load_2d(cb + x * HALF, &tmC, &cb_full, x * 64, g * CQ);
          tma_load_2d(cb + (2 + x) * HALF, &tmB, &cb_full, x * 64, g * CQ);
        }
        mbar_expect_tx(&ops_full, 5 * HALF);
        tma_load_2d(sm + S::OFF_DY, &tmDY, &ops_full, 0, g * CQ);
        tma_load_2d(sm + S::OFF_X, &tmX, &ops_full, 0, g * CQ);
        tma_load_2d(sm + S::OFF_XW, &tmXw, &ops_full, 0, g * CQ);
        for (int x = 0; x < 2; ++x) {
          tma_load_2d(sm + S::OFF_H + x * (HALF / 2), &tmH, &ops_full, x * 64, g * CP);
          tma_load_2d(sm + S::OFF_DH + x * (HALF / 2), &tmDH, &ops_full, x * 64, g * CP);
        }
      }
      __syncwarp();
      // the accumulators are free when the previous chunk's epilogue has read them
      ok = ok && warp_wait(&cb_full, n & 1) && warp_wait(&ops_full, n & 1) && warp_wait(&acc_free, (n & 1) ^ 1);
      if (!ok) break;
      tc_fence_after();
      if (elect_one()) {
#pragma unroll
        for (int ks = 0; ks < CN / 16; ++ks)        // G = C~ B~^T
          umma_f16(tm + TM_A, desc_k(c_a, ks, HALF), desc_k(b_a, ks, HALF), umma_idesc_bf16(CQ, CQ, 0, 0), ks > 0);
#pragma unroll
        for (int ks = 0; ks < CP / 16; ++ks)        // dM = dY X^T
          umma_f16(tm + TM_B, desc_k(dy_a, ks, HALF), desc_k(x_a, ks, HALF), umma_idesc_bf16(CQ, CQ, 0, 0), ks > 0);
        umma_commit(&s_full);
#pragma unroll
        for (int ks = 0; ks < CP / 16; ++ks)        // dY Hin: reduction over the head width = the rows of Hin
          umma_f16(tm + TM_CE, desc_k(dy_a, ks, HALF), desc_mn(h_a, ks, HALF / 2), umma_idesc_bf16(CQ, CN, 0, 1), ks > 0);
#pragma unroll
        for (int ks = 0; ks < CN / 16; ++ks)        // B~ dH^T
          umma_f16(tm + TM_XW, desc_k(b_a, ks, HALF), desc_k(dh_a, ks, HALF / 2), umma_idesc_bf16(CQ, CP, 0, 0), ks > 0);
      }
      __syncwarp();
      ok = warp_wait(&m_full, n & 1);
      if (!ok) break;
      tc_fence_after();
      if (elect_one()) {
#pragma unroll
        for (int ks = 0; ks < CQ / 16; ++ks)        // M^T dY
          umma_f16(tm + TM_X, desc_mn(m_a, ks, HALF), desc_mn(dy_a, ks, HALF), umma_idesc_bf16(CQ, CP, 1, 1), ks > 0);
#pragma unroll
        for (int ks = 0; ks < CQ / 16; ++ks)        // dG B~
          umma_f16(tm + TM_A, desc_k(dg_a, ks, HALF), desc_mn(b_a, ks, HALF), umma_idesc_bf16(CQ, CN, 0, 1), ks > 0);
#pragma unroll
        for (int ks = 0; ks < CQ / 16; ++ks)        // dG^T C~
          umma_f16(tm + TM_B, desc_mn(dg_a, ks, HALF), desc_mn(c_a, ks, HALF), umma_idesc_bf16(CQ, CN, 1, 1), ks > 0);
#pragma unroll
        for (int ks = 0; ks < CP / 16; ++ks)        // + (w X) dH
          umma_f16(tm + TM_B, desc_k(xw_a, ks, HALF), desc_mn(dh_a, ks, HALF / 2), umma_idesc_bf16(CQ, CN, 0, 1), 1u);
        umma_commit(&fin_full);
        umma_commit(&ops_free);
      }
      __syncwarp();
    }
    if (!ok && lane == 0) report_error(p.status, OA_KERR_WAIT_FULL);
  } else {
    const int quad = warp & 3, half = warp >> 2;
    const int t = quad * 32 + lane;                  // token of this thread = TMEM lane; columns [64 half, 64 half + 64)
    const uint32_t t_lane = (uint32_t)(quad * 32) << 16;
    const uint32_t sw = (uint32_t)(t & 7) << 4;      // 128-byte swizzle of the thread's row
    uint32_t n = 0;
    bool ok = true;
    // the scalars of a token, requested a chunk ahead
    float n_cum = 0.f, n_gam = 0.f, n_qk = 0.f, n_scale = 0.f, n_w = 0.f, n_d = 0.f;
    auto request = [&](int g) {
      if (g >= p.G) return;
      const long long gi = (long long)g * CQ + t;
      n_cum = p.cum[gi]; n_gam = p.gamma[gi]; n_qk = p.qk[gi]; n_scale = p.scale[gi]; n_w = p.w[gi];
      n_d = p.D ? p.D[(g / p.nC) % p.H] : 0.f;
    };
    request(blockIdx.x);
    for (int g = blockIdx.x; g < p.G; g += gridDim.x, ++n) {
      const long long gi = (long long)g * CQ + t;
      const int c = g % p.nC, bh = g / p.nC, h = bh % p.H, b = bh / p.H;
      const float ct = n_cum, gam = n_gam, wv = n_w;
      const float dval = n_d + gam * n_qk;
      if (half == 0) { s_ncum[t] = -ct; s_scale[t] = n_scale; }
      asm volatile("bar.sync 1, 256;" ::: "memory");   // also: the previous chunk's sums have been read
      // a wait that runs out is not left early: the worker warps meet at barriers, so they all finish the loop (without waiting again)
      // C~ and B~ are waited for here: the barrier of the next chunk's may complete once this chunk's products are done
      ok = ok && warp_wait(&s_full, n & 1) && warp_wait(&cb_full, n & 1);
      tc_fence_after();
      const uint8_t* cb = sm + ((n & 1) ? S::OFF_R1 : S::OFF_R0);
      const uint32_t m_a = smem_u32(sm + ((n & 1) ? S::OFF_R0 : S::OFF_R1));
      float rsum = 0.f;
#pragma unroll 1
      for (int q = 0; q < 2; ++q) {
        const int qc = half * 2 + q;                 // 32-column group: below, on or above the diagonal block of this warp
        uint32_t m[16], dg[16];
        if (qc > quad) {
#pragma unroll
          for (int i = 0; i < 16; ++i) m[i] = dg[i] = 0u;
          s_col[quad * CQ + qc * 32 + lane] = 0.f;
        } else {
          uint32_t gv[32], dv[32];
          tmem_ld32(tm + t_lane + TM_A + qc * 32, gv);
          tmem_ld32(tm + t_lane + TM_B + qc * 32, dv);
          tmem_ld_wait();
          const ulonglong2 *nc2 = reinterpret_cast<const ulonglong2*>(s_ncum + qc * 32), *sc2 = reinterpret_cast<const ulonglong2*>(s_scale + qc * 32);
          const unsigned long long ct2 = f2_of(__float_as_uint(ct), __float_as_uint(ct)), l2e = f2_of(0x3fb8aa3bu, 0x3fb8aa3bu);   // log2 e
          float ge[32];
          // two columns: decay e, then e scale, G and dM times it, G dM e
          auto pair = [&](int k, unsigned long long nc, unsigned long long sc, unsigned long long& ge2, uint32_t* mv, uint32_t* g2) {
            uint32_t x0, x1;
            f2_to(f2_mul(f2_add(ct2, nc), l2e), x0, x1);
            const unsigned long long e = f2_of(__float_as_uint(fast_exp2(__uint_as_float(x0))), __float_as_uint(fast_exp2(__uint_as_float(x1))));
            const unsigned long long es = f2_mul(e, sc), gg = f2_of(gv[k], gv[k + 1]), dm = f2_of(dv[k], dv[k + 1]);
            f2_to(f2_mul(gg, es), mv[0], mv[1]);
            f2_to(f2_mul(dm, es), g2[0], g2[1]);
            ge2 = f2_mul(f2_mul(dm, gg), e);
          };
          if (qc < quad) {                            // every column is an earlier token
            unsigned long long rs = 0;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              const ulonglong2 nc = nc2[i], sc = sc2[i];
#pragma unroll
              for (int j = 0; j < 2; ++j) {
                const int k = 4 * i + 2 * j;
                uint32_t mv[2], g2[2], u0, u1;
                unsigned long long ge2;
                pair(k, j ? nc.y : nc.x, j ? sc.y : sc.x, ge2, mv, g2);
                m[k >> 1] = pack_bf16x2(__uint_as_float(mv[0]), __uint_as_float(mv[1]));
                dg[k >> 1] = pack_bf16x2(__uint_as_float(g2[0]), __uint_as_float(g2[1]));
                rs = f2_fma(ge2, j ? sc.y : sc.x, rs);
                f2_to(ge2, u0, u1);
                ge[k] = __uint_as_float(u0); ge[k + 1] = __uint_as_float(u1);
              }
            }
            uint32_t r0, r1;
            f2_to(rs, r0, r1);
            rsum += __uint_as_float(r0) + __uint_as_float(r1);
          } else {                                    // the block on the diagonal: columns below `lane`, itself, and none
            float dmd = 0.f;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              const ulonglong2 nc = nc2[i], sc = sc2[i];
              const float4 scf = reinterpret_cast<const float4*>(sc2)[i];
              const float scv[4] = {scf.x, scf.y, scf.z, scf.w};
#pragma unroll
              for (int j = 0; j < 2; ++j) {
                const int k = 4 * i + 2 * j;
                uint32_t mv[2], g2[2], u[2];
                unsigned long long ge2;
                pair(k, j ? nc.y : nc.x, j ? sc.y : sc.x, ge2, mv, g2);
                f2_to(ge2, u[0], u[1]);
#pragma unroll
                for (int z = 0; z < 2; ++z) {         // chosen, not multiplied by 0: a later token may hold an infinity
                  mv[z] = k + z < lane ? mv[z] : (k + z == lane ? __float_as_uint(dval) : 0u);
                  g2[z] = k + z < lane ? g2[z] : 0u;
                  ge[k + z] = k + z < lane ? __uint_as_float(u[z]) : 0.f;
                  rsum += ge[k + z] * scv[2 * j + z];
                  dmd = k + z == lane ? __uint_as_float(dv[k + z]) : dmd;
                }
                m[k >> 1] = pack_bf16x2(__uint_as_float(mv[0]), __uint_as_float(mv[1]));
                dg[k >> 1] = pack_bf16x2(__uint_as_float(g2[0]), __uint_as_float(g2[1]));
              }
            }
            p.diag[gi] = dmd;
            s_dqk[t] = dmd * gam;
          }
          s_col[quad * CQ + qc * 32 + lane] = lane_transpose_sum(ge, lane);
        }
        const uint32_t off = half * HALF + t * 128 + q * 64;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          st_shared_v4(m_a + ((off + i * 16) ^ sw), make_uint4(m[4 * i], m[4 * i + 1], m[4 * i + 2], m[4 * i + 3]));
          st_shared_v4(m_a + 2 * HALF + ((off + i * 16) ^ sw), make_uint4(dg[4 * i], dg[4 * i + 1], dg[4 * i + 2], dg[4 * i + 3]));
        }
      }
      s_row[half * CQ + t] = rsum;
      fence_proxy_async_smem();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&m_full);
      asm volatile("bar.sync 1, 256;" ::: "memory");
      if (half == 0) {
        p.row_mm[gi] = s_row[t] + s_row[CQ + t];
        const float cg = (s_col[t] + s_col[CQ + t]) + (s_col[2 * CQ + t] + s_col[3 * CQ + t]);
        p.col_ge[gi] = cg;
        p.col_mm[gi] = cg * s_scale[t];
      }
      const float dqk = s_dqk[t], e = __expf(ct);
      const long long g4 = gi - (lane & 3);             // first row of this lane's group of four: accesses cover 64 bytes of eight rows
      const uint4* xp = reinterpret_cast<const uint4*>(p.X + g4 * CP + half * 32) + (lane & 3);
      uint4 xv[4], o[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) xv[k] = xp[k * (CP / 8)];
      request(g + gridDim.x);
      ok = ok && warp_wait(&fin_full, n & 1);
      tc_fence_after();
      // dC~ (row t) and dB~ (row t as a key); this thread's half of the state columns
      float dce = 0.f;
      float* dc_out = p.dC + g4 * CN + half * 64 + (lane & 3) * 4;
      float* db_out = p.dB + g4 * CN + half * 64 + (lane & 3) * 4;
#pragma unroll 1
      for (int q = 0; q < 4; ++q) {
        uint32_t a[16], ce[16], d2[16];
        tmem_ld16(tm + t_lane + TM_A + half * 64 + q * 16, a);
        tmem_ld16(tm + t_lane + TM_CE + half * 64 + q * 16, ce);
        tmem_ld16(tm + t_lane + TM_B + half * 64 + q * 16, d2);
        tmem_ld_wait();
        const uint32_t off = half * HALF + t * 128 + q * 32;
        uint4 oc[4], ob[4];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const uint4 cp = *reinterpret_cast<const uint4*>(cb + ((off + i * 16) ^ sw));
          const uint4 bp = *reinterpret_cast<const uint4*>(cb + 2 * HALF + ((off + i * 16) ^ sw));
          const uint32_t cw[4] = {cp.x, cp.y, cp.z, cp.w}, bw[4] = {bp.x, bp.y, bp.z, bp.w};
          float fc[8], fb[8];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float2 cv = unpack_bf16x2(cw[j]), bv = unpack_bf16x2(bw[j]);
            const int k = i * 8 + 2 * j;
            const float c0 = __uint_as_float(ce[k]), c1 = __uint_as_float(ce[k + 1]);
            dce += c0 * cv.x + c1 * cv.y;
            fc[2 * j] = __uint_as_float(a[k]) + c0 * e + dqk * bv.x;
            fc[2 * j + 1] = __uint_as_float(a[k + 1]) + c1 * e + dqk * bv.y;
            fb[2 * j] = __uint_as_float(d2[k]) + dqk * cv.x;
            fb[2 * j + 1] = __uint_as_float(d2[k + 1]) + dqk * cv.y;
          }
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            oc[2 * i + j] = make_uint4(__float_as_uint(fc[4 * j]), __float_as_uint(fc[4 * j + 1]), __float_as_uint(fc[4 * j + 2]), __float_as_uint(fc[4 * j + 3]));
            ob[2 * i + j] = make_uint4(__float_as_uint(fb[4 * j]), __float_as_uint(fb[4 * j + 1]), __float_as_uint(fb[4 * j + 2]), __float_as_uint(fb[4 * j + 3]));
          }
        }
        exchange4(oc, lane);
        exchange4(ob, lane);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          *reinterpret_cast<uint4*>(dc_out + k * CN + q * 16) = oc[k];
          *reinterpret_cast<uint4*>(db_out + k * CN + q * 16) = ob[k];
        }
      }
      // dx and dw: this thread's 32 of the head's 64 columns
      float dwv = 0.f;
      const long long row = (long long)b * p.L + (long long)c * CQ + t;
      {
        uint32_t u[32], v[32];
        tmem_ld32(tm + t_lane + TM_X + half * 32, u);
        tmem_ld32(tm + t_lane + TM_XW + half * 32, v);
        tmem_ld_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&acc_free);        // C~, B~ and the accumulators may be replaced
        exchange4(xv, lane);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const uint32_t xs[4] = {xv[i].x, xv[i].y, xv[i].z, xv[i].w};
          uint32_t r[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float2 xf = unpack_bf16x2(xs[j]);
            const float b0 = __uint_as_float(v[8 * i + 2 * j]), b1 = __uint_as_float(v[8 * i + 2 * j + 1]);
            dwv += b0 * xf.x + b1 * xf.y;
            r[j] = pack_bf16x2(__uint_as_float(u[8 * i + 2 * j]) + b0 * wv, __uint_as_float(u[8 * i + 2 * j + 1]) + b1 * wv);
          }
          o[i] = make_uint4(r[0], r[1], r[2], r[3]);
        }
        exchange4(o, lane);
        __nv_bfloat16* dxo = p.dx + (row - (lane & 3)) * p.lddx + h * CP + half * 32 + (lane & 3) * 8;
#pragma unroll
        for (int k = 0; k < 4; ++k) *reinterpret_cast<uint4*>(dxo + k * p.lddx) = o[k];
      }
      // both halves of a token meet: the half 1 threads leave their sums in shared memory
      if (half == 1) { s_fin[t] = dce; s_fin[CQ + t] = dwv; }
      asm volatile("bar.sync 1, 256;" ::: "memory");
      if (half == 0) {
        p.dcum_ce[gi] = (dce + s_fin[t]) * e;
        p.dw[gi] = dwv + s_fin[CQ + t];
      }
    }
    if (!ok && lane == 0) report_error(p.status, OA_KERR_WAIT_TMEM_FULL);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 8) { tc_fence_after(); tmem_dealloc<512>(tm); }
}

int num_sms();

}  // namespace oa

using namespace oa;

extern "C" {

// C~, B~ [G, 128, 128], X [G, 128, 64], Hin [G, 64, 128] bf16; cum, scale, gamma, qk [G, 128] fp32 -> y (and yraw, with z) token layout.
int oa_ssd_chunk_fwd(const void* C, const void* Bt, const void* X, const void* Hin, const void* cum, const void* scale, const void* gamma,
                     const void* qk, const void* D, const void* z, long long ldz, void* y, void* yraw, long long ldy, int B, int L, int H,
                     void* status, void* stream) {
  if (B <= 0 || H <= 0 || L <= 0 || L % CQ || (z && !yraw)) return OA_ERR_ARG;
  const int nC = L / CQ;
  const long long G = (long long)B * H * nC;
  if (G * CQ > 0x7fffffffLL) return OA_ERR_TOO_LARGE;
  if ((ldy & 7) || (ldz & 7) || ((reinterpret_cast<uintptr_t>(y) | reinterpret_cast<uintptr_t>(yraw) | reinterpret_cast<uintptr_t>(z)) & 15)) return OA_ERR_ALIGN;
  CUtensorMap tc, tb, tx, th;
  int rc;
  if ((rc = make_tmap_2d_bf16(&tc, C, CN, G * CQ, CN, 64, CQ)) || (rc = make_tmap_2d_bf16(&tb, Bt, CN, G * CQ, CN, 64, CQ)) ||
      (rc = make_tmap_2d_bf16(&tx, X, CP, G * CQ, CP, 64, CQ)) || (rc = make_tmap_2d_bf16(&th, Hin, CN, G * CP, CN, 64, CP)))
    return rc;
  SsdChunkFwd p{(const float*)cum, (const float*)scale, (const float*)gamma, (const float*)qk, (const float*)D, (const __nv_bfloat16*)z, ldz,
                (__nv_bfloat16*)y, (__nv_bfloat16*)yraw, ldy, H, nC, L, (int*)status};
  if (cudaFuncSetAttribute(ssd_chunk_fwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, ChunkFwdSmem::BYTES) != cudaSuccess) return OA_ERR_LAUNCH;
  ssd_chunk_fwd_kernel<<<(unsigned)G, 160, ChunkFwdSmem::BYTES, (cudaStream_t)stream>>>(tc, tb, tx, th, p);
  return cudaGetLastError() == cudaSuccess ? OA_OK : OA_ERR_LAUNCH;
}

// One chunk's share of the backward pass; dC, dB [G, 128, 128] fp32, row_mm, col_mm, col_ge, diag, dcum_ce, dw [G, 128] fp32, dx
// token layout.
int oa_ssd_chunk_bwd(const void* C, const void* Bt, const void* X, const void* Xw, const void* dY, const void* Hin, const void* dH,
                     const void* cum, const void* scale, const void* gamma, const void* qk, const void* w, const void* D, void* dC, void* dB,
                     void* row_mm, void* col_mm, void* col_ge, void* diag, void* dcum_ce, void* dw, void* dx, long long lddx, int B, int L, int H,
                     void* status, void* stream) {
  if (B <= 0 || H <= 0 || L <= 0 || L % CQ) return OA_ERR_ARG;
  const int nC = L / CQ;
  const long long G = (long long)B * H * nC;
  if (G * CQ > 0x7fffffffLL) return OA_ERR_TOO_LARGE;
  if ((lddx & 7) || ((reinterpret_cast<uintptr_t>(dx) | reinterpret_cast<uintptr_t>(dC) | reinterpret_cast<uintptr_t>(dB)) & 15)) return OA_ERR_ALIGN;
  CUtensorMap tc, tb, tx, txw, tdy, th, tdh;
  int rc;
  if ((rc = make_tmap_2d_bf16(&tc, C, CN, G * CQ, CN, 64, CQ)) || (rc = make_tmap_2d_bf16(&tb, Bt, CN, G * CQ, CN, 64, CQ)) ||
      (rc = make_tmap_2d_bf16(&tx, X, CP, G * CQ, CP, 64, CQ)) || (rc = make_tmap_2d_bf16(&txw, Xw, CP, G * CQ, CP, 64, CQ)) ||
      (rc = make_tmap_2d_bf16(&tdy, dY, CP, G * CQ, CP, 64, CQ)) || (rc = make_tmap_2d_bf16(&th, Hin, CN, G * CP, CN, 64, CP)) ||
      (rc = make_tmap_2d_bf16(&tdh, dH, CN, G * CP, CN, 64, CP)))
    return rc;
  SsdChunkBwd p{(const float*)cum, (const float*)scale, (const float*)gamma, (const float*)qk, (const float*)w, (const float*)D,
                (const __nv_bfloat16*)X, (float*)dC, (float*)dB, (float*)row_mm, (float*)col_mm, (float*)col_ge,
                (float*)diag, (float*)dcum_ce, (float*)dw, (__nv_bfloat16*)dx, lddx, H, nC, L, (int)G, (int*)status};
  if (cudaFuncSetAttribute(ssd_chunk_bwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, ChunkBwdSmem::BYTES) != cudaSuccess) return OA_ERR_LAUNCH;
  const int grid = (int)(G < num_sms() ? G : num_sms());
  ssd_chunk_bwd_kernel<<<grid, CB_THREADS, ChunkBwdSmem::BYTES, (cudaStream_t)stream>>>(tc, tb, tx, txw, tdy, th, tdh, p);
  return cudaGetLastError() == cudaSuccess ? OA_OK : OA_ERR_LAUNCH;
}

}  // extern "C"
