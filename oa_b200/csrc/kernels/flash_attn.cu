// Causal / full scaled-dot-product attention for sm_100a, forward and backward, bf16 in / fp32 accumulate.
//
// The reference's FlashCausal kernels (Source/Private/Oa/Ml/Shader/Compute/Nn/Attention/FlashCausal*.slang)
// run one work-group per query row with all scores of the row in shared memory (S <= 1024, fp32 only, no
// tensor cores).  Here the work is tiled 128 queries x 128 keys, every matrix product of a tile runs on
// tcgen05 with accumulators in TMEM, tiles arrive through TMA, and the probabilities (and their gradients) are
// written back to TMEM as bf16 and read from there as the A operand of the next product: nothing but Q, K, V, dO
// passes through shared memory.  Q, K, V are read in place from a packed projection output ([B*S, row_stride] with
// head h at column h*head_dim), and O is written merged ([B*S, H*head_dim]), so there are no SplitHeads / MergeHeads
// passes.
//
// Measured facts that shape the kernels (clocks of one tcgen05.mma in a row of them): both operands from shared memory 66 at N = 128, 50 at
// N = 64; A from TMEM 64 and 33; two warps that issue at once share the pipe evenly; a group of eight is seen complete 330 clocks
// after its last product.  An MUFU exponential occupies its pipe for 8 clocks per warp (1024 per 128 x 128 tile).  Hence: where the
// columns allow it score tiles are copied to registers and released at once so the next score product is issued under this block's
// exponentials; where they do not, the issuing order sees to it that a tile's products run under another's exponentials; descriptors are
// made once; and every kernel but the single-tile forward is persistent (one CTA per SM walks its work items in snake order, heaviest
// causal items first), so TMEM, barriers and the operand rings live across items.
//
// Backward is two kernels, both deterministic (single writer per output element, like the reference's
// FlashCausalBwdQ / FlashCausalBwdKV): one accumulates dK, dV in TMEM over the query blocks of a key block, the other dQ
// over the key blocks of a query block.  Probabilities are recomputed from the saved log-sum-exp.
// Every wait is bounded and reports to a status word.
#include "common.cuh"
#include "api.h"

namespace oa {

constexpr int FA_BM = 128;   // queries per tile
constexpr int FA_BN = 128;   // keys per tile
constexpr float LOG2E = 1.4426950408889634f;
constexpr int FA_THREADS = 320;   // single-tile forward: 8 softmax warps + MMA warp + TMA warp

// The descriptor of an operand that starts `bytes` further (the address is in units of 16 bytes in the low bits): an issuing warp makes
// its descriptors once and only adds to them between products.
__device__ __forceinline__ uint64_t desc_at(uint64_t desc, uint32_t bytes) { return desc + (bytes >> 4); }
__device__ __forceinline__ uint64_t desc_k(const void* smem) { return umma_smem_desc_sw128(smem_u32(smem), 16, 1024); }             // reduction contiguous
__device__ __forceinline__ uint64_t desc_mn(const void* smem) { return umma_smem_desc_sw128(smem_u32(smem), FA_BN * 128, 1024); }   // 128 rows of the reduction

// 64-thread named barrier shared by the two warps that own the same 32 query rows.
__device__ __forceinline__ void pair_sync(int quad) {
  asm volatile("bar.sync %0, 64;" ::"r"(quad + 1) : "memory");
}

// Two exponentials 2^x on the multiply-add pipe: x = n + f with n the nearest integer (added and taken off at 1.5 * 2^23), 2^f by the
// minimax polynomial of degree 5 on [-1/2, 1/2] (Remez exchange on the relative error: 7.5e-8, with coefficients rounded to fp32 1.55e-7,
// 2.1e-7 with the rounding of its steps; ex2.approx states 2^-22 = 2.4e-7), 2^n as an exponent field, which is zero at n = -127: below that, -inf included, the result is 0 as ex2.approx.ftz gives it.
// NaN stays NaN; x up to 127.
__device__ __forceinline__ unsigned long long f2_splat(float v) { return f2_of(__float_as_uint(v), __float_as_uint(v)); }
__device__ __forceinline__ float max_nan(float a, float b) {
  float d;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(d) : "f"(a), "f"(b));
  return d;
}
__device__ __forceinline__ unsigned long long exp2_fma2(unsigned long long x) {
  uint32_t a, b;
  f2_to(x, a, b);
  x = f2_of(__float_as_uint(max_nan(__uint_as_float(a), -127.f)), __float_as_uint(max_nan(__uint_as_float(b), -127.f)));
  const unsigned long long t = f2_add(x, f2_splat(12582912.f));
  const unsigned long long f = f2_fma(f2_add(t, f2_splat(-12582912.f)), f2_splat(-1.f), x);
  unsigned long long r = f2_fma(f2_splat(0.00132764725f), f, f2_splat(0.00967554096f));
  r = f2_fma(r, f, f2_splat(0.0555071309f));
  r = f2_fma(r, f, f2_splat(0.240221202f));
  r = f2_fma(r, f, f2_splat(0.693146944f));
  r = f2_fma(r, f, f2_splat(1.00000012f));
  f2_to(t, a, b);
  return f2_mul(r, f2_of((a << 23) + 0x3f800000u, (b << 23) + 0x3f800000u));
}
__device__ __forceinline__ unsigned long long exp2_mufu2(unsigned long long x) {
  uint32_t a, b;
  f2_to(x, a, b);
  return f2_of(__float_as_uint(fast_exp2(__uint_as_float(a))), __float_as_uint(fast_exp2(__uint_as_float(b))));
}
__device__ __forceinline__ uint32_t f2_bf16(unsigned long long v) {
  uint32_t a, b;
  f2_to(v, a, b);
  return pack_bf16x2(__uint_as_float(a), __uint_as_float(b));
}
// How many of eight pairs of exponentials go to the multiply-add pipe: one in the forward pass, one and two in the backward pass, where
// two warps of a scheduler reach their exponentials together.  The pipe relieves the special-function units and costs issue slots.  Zero /
// one / two / three, forward: 8 x 2048 x 16 heads of 64 causal 121.9 / 113.7 / 119.0 / 126.7 us, 1 x 4096 x 16 full 103.7 / 106.7 / 114.0 / 119.9,
// 2 x 3001 x 16 of 128 80.4 / 79.5 / - / 83.7.  Backward, one / two / three / four: 8 x 2048 x 16 of 64 341 / 330 / 336 / 349; of 128, one / two /
// three: 1 x 4096 x 32 423 / 424 / 433.
constexpr int FA_FMA_PAIRS = 1;
template <int HD> constexpr int FA_BWD_FMA_PAIRS = HD == 64 ? 2 : 1;

// 32 fp32 columns of a warp's 32 rows (one row to a lane) as bf16, 64 bytes of eight rows to a store (the rows lie apart by a whole
// projection).  `at`: the row of this warp's first lane; rows from `rows` on are not written.
__device__ __forceinline__ void store_rows(__nv_bfloat16* at, long long stride, int rows, const uint32_t* a, float mul, int lane) {
  uint4 v[4];
#pragma unroll
  for (int g = 0; g < 4; ++g) {
    const float* f = reinterpret_cast<const float*>(a) + g * 8;
    v[g] = make_uint4(pack_bf16x2(f[0] * mul, f[1] * mul), pack_bf16x2(f[2] * mul, f[3] * mul), pack_bf16x2(f[4] * mul, f[5] * mul), pack_bf16x2(f[6] * mul, f[7] * mul));
  }
  exchange4(v, lane);
  const int r0 = lane & ~3;
  at += (long long)r0 * stride + (lane & 3) * 8;
#pragma unroll
  for (int k = 0; k < 4; ++k)
    if (r0 + k < rows) *reinterpret_cast<uint4*>(at + k * stride) = v[k];
}

struct FlashParams {
  int batch, heads, seq, head_dim;
  float scale;
  int causal;
  __nv_bfloat16* o;
  long long o_stride;
  float* lse;            // [B, H, S]
  int* status;
};

// ===================================================================================== forward, S double-buffered in TMEM
// One CTA owns one 128-query tile of one (batch, head).  S = Q K_j^T alternates between two TMEM buffers, and the MMA warp
// always runs two key blocks ahead of the softmax (Q K_{j+2}^T is issued right after P_j V_j), so the softmax warps never
// wait for the tensor pipe: they go from block j straight to block j+1 and the SFU stays busy.
//   warps 0-7  softmax: two threads per query row (warp w: TMEM lane quadrant w % 4, key columns [64 * (w / 4), +64)), the
//              64 scores of a thread are read from TMEM once, the row maximum is exchanged with the partner thread through
//              a parity-double-buffered slot, probabilities go back to TMEM as packed bf16 over the columns of S_j;
//   warp 8     MMA issuer: P is the A operand straight from TMEM, V the B operand from shared memory, O accumulates in
//              TMEM over all key blocks and is read once at the end;
//   warp 9     TMA producer (Q once, K / V rings).
// The running maximum is updated lazily: while the new row maximum exceeds the one in use by less than 2^8 the old one is
// kept (probabilities then stay below 256), so O in TMEM is rescaled only in the rare iterations where some row of a warp
// jumps by more than that; the final 1/l uses the same maxima, so the result is the exact softmax.
// TMEM: S0 | S1 | O = 128 + 128 + head_dim columns.
template <int HD>
struct Fwd2Cfg {
  static constexpr int NSK = 3;                            // K ring depth (K runs two blocks ahead of V)
  static constexpr int NSV = (HD == 64) ? 3 : 2;           // V ring depth
  static constexpr int Q_BYTES = FA_BM * HD * 2;
  static constexpr int KV_BYTES = FA_BN * HD * 2;
  static constexpr int OFF_Q = 0;
  static constexpr int OFF_K = OFF_Q + Q_BYTES;
  static constexpr int OFF_V = OFF_K + NSK * KV_BYTES;
  static constexpr int OFF_X = OFF_V + NSV * KV_BYTES;     // float[2 parities][2 halves][128 rows]: row-maximum exchange
  static constexpr int OFF_BAR = OFF_X + 2 * 2 * FA_BM * 4;
  static constexpr int SMEM_BYTES = OFF_BAR + 256;
  static constexpr int TMEM_COLS = 512;
  static constexpr int TM_S = 0;                           // + 128 * (j & 1)
  static constexpr int TM_O = 256;
};

constexpr float FA_RESCALE_THRESHOLD = 8.f;                // log2 units


template <int HD>
__global__ void __launch_bounds__(FA_THREADS, 1)
flash_fwd2_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                  const __grid_constant__ CUtensorMap tmV, const FlashParams p) {
  using Cfg = Fwd2Cfg<HD>;
  constexpr int NSK = Cfg::NSK, NSV = Cfg::NSV;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + Cfg::OFF_BAR);
  uint64_t* q_full = bars + 0;
  uint64_t* k_full = bars + 1;                 // [NSK]
  uint64_t* k_empty = k_full + NSK;            // [NSK]
  uint64_t* v_full = k_empty + NSK;            // [NSV]
  uint64_t* v_empty = v_full + NSV;            // [NSV]
  uint64_t* s_full = v_empty + NSV;            // [2]  S buffer holds Q K_j^T
  uint64_t* p_full = s_full + 2;               // [2]  P_j written over S buffer (and O rescaled if needed)
  uint64_t* o_done = s_full + 4;               //      O += P_j V_j finished
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(s_full + 5);
  float* xch = reinterpret_cast<float*>(smem + Cfg::OFF_X);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nblk = (p.seq + FA_BM - 1) / FA_BM;
  const int qb = nblk - 1 - blockIdx.x;        // heaviest causal tiles first
  const int h = blockIdx.y, b = blockIdx.z;
  const int n_kv = p.causal ? (qb + 1) : nblk;
  const int row0 = b * p.seq;

  if ((smem_u32(smem) & 1023u) != 0) {
    if (threadIdx.x == 0) report_error(p.status, OA_KERR_BAD_ARG);
    return;
  }
  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmQ); tma_prefetch_desc(&tmK); tma_prefetch_desc(&tmV);
    mbar_init(q_full, 1);
    for (int s = 0; s < NSK; ++s) { mbar_init(&k_full[s], 1); mbar_init(&k_empty[s], 1); }
    for (int s = 0; s < NSV; ++s) { mbar_init(&v_full[s], 1); mbar_init(&v_empty[s], 1); }
    for (int t = 0; t < 2; ++t) { mbar_init(&s_full[t], 1); mbar_init(&p_full[t], 8); }
    mbar_init(o_done, 1);
    mbar_fence_init();
  }
  if (warp == 8) { tmem_alloc<Cfg::TMEM_COLS>(tmem_slot); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_wait();                            // the prologue above ran under the previous kernel's tail; global memory from here on

  if (warp == 9) {
    // ------------- producer: the whole warp walks the loop and waits together; one lane issues the copies.  K block i is
    // loaded two iterations before V block i - 2... both rings are simply filled in order, K first.
    if (elect_one()) {
      mbar_expect_tx(q_full, Cfg::Q_BYTES);
#pragma unroll
      for (int x = 0; x < HD / 64; ++x)
        tma_load_2d(smem + Cfg::OFF_Q + x * (FA_BM * 128), &tmQ, q_full, h * HD + x * 64, row0 + qb * FA_BM);
    }
    for (int i = 0; i < n_kv + 2; ++i) {
      if (i < n_kv) {
        const int st = i % NSK;
        if (!warp_wait(&k_empty[st], ((i / NSK) & 1) ^ 1)) { if (lane == 0) report_error(p.status, OA_KERR_WAIT_EMPTY); break; }
        if (elect_one()) {
          mbar_expect_tx(&k_full[st], Cfg::KV_BYTES);
#pragma unroll
          for (int x = 0; x < HD / 64; ++x)
            tma_load_2d(smem + Cfg::OFF_K + st * Cfg::KV_BYTES + x * (FA_BN * 128), &tmK, &k_full[st], h * HD + x * 64, row0 + i * FA_BN);
        }
      }
      const int jv = i - 2;                    // V lags K by two blocks, like its consumer
      if (jv >= 0) {
        const int st = jv % NSV;
        if (!warp_wait(&v_empty[st], ((jv / NSV) & 1) ^ 1)) { if (lane == 0) report_error(p.status, OA_KERR_WAIT_EMPTY); break; }
        if (elect_one()) {
          mbar_expect_tx(&v_full[st], Cfg::KV_BYTES);
#pragma unroll
          for (int x = 0; x < HD / 64; ++x)
            tma_load_2d(smem + Cfg::OFF_V + st * Cfg::KV_BYTES + x * (FA_BN * 128), &tmV, &v_full[st], h * HD + x * 64, row0 + jv * FA_BN);
        }
      }
      __syncwarp();
    }
  } else if (warp == 8) {
    // ------------- MMA issuer (warp-uniform waits, lane 0 issues)
    constexpr uint32_t idesc_qk = umma_idesc_bf16(FA_BM, FA_BN, 0, 0);
    constexpr uint32_t idesc_pv = umma_idesc_bf16(FA_BM, HD, 0, 1);
    const uint32_t q_addr = smem_u32(smem + Cfg::OFF_Q);
    auto issue_qk = [&](int i) -> bool {       // S[i & 1] = Q K_i^T
      const int st = i % NSK;
      if (!warp_wait(&k_full[st], (i / NSK) & 1)) { if (lane == 0) report_error(p.status, OA_KERR_WAIT_FULL); return false; }
      tc_fence_after();
      if (elect_one()) {
        const uint32_t k_addr = smem_u32(smem + Cfg::OFF_K + st * Cfg::KV_BYTES);
#pragma unroll
        for (int ks = 0; ks < HD / 16; ++ks) {
          const uint32_t off = (ks >> 2) * (FA_BM * 128) + (ks & 3) * 32;
          umma_f16(tmem_base + Cfg::TM_S + (i & 1) * FA_BN, umma_smem_desc_sw128(q_addr + off, 16, 1024),
                   umma_smem_desc_sw128(k_addr + off, 16, 1024), idesc_qk, ks > 0 ? 1u : 0u);
        }
        umma_commit(&k_empty[st]);
        umma_commit(&s_full[i & 1]);
      }
      __syncwarp();
      return true;
    };
    bool ok = warp_wait(q_full, 0);
    if (!ok && lane == 0) report_error(p.status, OA_KERR_WAIT_FULL);
    if (ok) ok = issue_qk(0);
    if (ok && n_kv > 1) ok = issue_qk(1);
    for (int j = 0; j < n_kv && ok; ++j) {
      const int st = j % NSV;
      if (!warp_wait(&v_full[st], (j / NSV) & 1)) { if (lane == 0) report_error(p.status, OA_KERR_WAIT_FULL); break; }
      if (!warp_wait(&p_full[j & 1], (j >> 1) & 1)) { if (lane == 0) report_error(p.status, OA_KERR_WAIT_SOFTMAX); break; }
      tc_fence_after();
      if (elect_one()) {
        const uint32_t v_addr = smem_u32(smem + Cfg::OFF_V + st * Cfg::KV_BYTES);
#pragma unroll
        for (int ks = 0; ks < FA_BN / 16; ++ks)
          umma_f16_ts(tmem_base + Cfg::TM_O, tmem_base + Cfg::TM_S + (j & 1) * FA_BN + ks * 8,
                      umma_smem_desc_sw128(v_addr + ks * 2048, FA_BN * 128, 1024), idesc_pv, (j > 0 || ks > 0) ? 1u : 0u);
        umma_commit(&v_empty[st]);
        umma_commit(o_done);
      }
      __syncwarp();
      if (j + 2 < n_kv) ok = issue_qk(j + 2);  // overwrites S[j & 1] = P_j: ordered after P_j V_j by the pipe
    }
  } else {
    // ------------- softmax + output: two threads per query row (key columns split in halves)
    constexpr int OC = HD / 2;                   // output columns owned by this thread
    const int quad = warp & 3;
    const int half = warp >> 2;
    const int r = quad * 32 + lane;
    const int qi = qb * FA_BM + r;               // query index inside the sequence
    const uint32_t t_lane = (uint32_t)(quad * 32) << 16;
    const uint32_t o_addr = tmem_base + t_lane + Cfg::TM_O + half * OC;
    const float sl2 = p.scale * LOG2E;
    float m_run = -INFINITY, l_run = 0.f;
    bool ok = true;
    for (int j = 0; j < n_kv; ++j) {
      ok = warp_wait(&s_full[j & 1], (j >> 1) & 1);
      if (!ok) { if (lane == 0) report_error(p.status, OA_KERR_WAIT_TMEM_FULL); break; }
      tc_fence_after();
      const uint32_t s_addr = tmem_base + t_lane + Cfg::TM_S + (j & 1) * FA_BN;
      uint32_t sv[64];
      tmem_ld32(s_addr + half * 64, sv);
      tmem_ld32(s_addr + half * 64 + 32, sv + 32);
      tmem_ld_wait();
      const bool need_mask = (p.causal && j == qb) || (j * FA_BN + FA_BN > p.seq);
      if (need_mask) {
        const int lim = min(p.causal ? qi : 0x7fffffff, p.seq - 1) - j * FA_BN - half * 64;   // columns i <= lim are alive
#pragma unroll
        for (int i = 0; i < 64; ++i) sv[i] = (i <= lim) ? sv[i] : 0xff800000u;                 // -inf
      }
      float m0 = __uint_as_float(sv[0]), m1 = __uint_as_float(sv[1]), m2 = __uint_as_float(sv[2]), m3 = __uint_as_float(sv[3]);
#pragma unroll
      for (int i = 4; i < 64; i += 4) {
        m0 = fmaxf(m0, __uint_as_float(sv[i])); m1 = fmaxf(m1, __uint_as_float(sv[i + 1]));
        m2 = fmaxf(m2, __uint_as_float(sv[i + 2])); m3 = fmaxf(m3, __uint_as_float(sv[i + 3]));
      }
      float mx = fmaxf(fmaxf(m0, m1), fmaxf(m2, m3));
      // Exchange with the partner thread of this row.  Both threads now hold their scores in registers, so after this
      // barrier the S buffer may be overwritten by either of them.
      float* slots = xch + (j & 1) * (2 * FA_BM);
      slots[(half ^ 1) * FA_BM + r] = mx;
      pair_sync(quad);
      mx = fmaxf(mx, slots[half * FA_BM + r]) * sl2;
      const float m_new = fmaxf(m_run, mx);
      const bool grow = (m_new - m_run) > FA_RESCALE_THRESHOLD;           // first block: m_run = -inf -> true
      const float m_cand = grow ? m_new : m_run;
      const float m_use = (m_cand == -INFINITY) ? 0.f : m_cand;           // row fully masked so far
      const float alpha = grow ? fast_exp2(m_run - m_use) : 1.f;           // m_run = -inf -> 0
      const float neg_m = -m_use;
      float l0 = 0.f, l1 = 0.f, l2 = 0.f, l3 = 0.f;
      uint32_t pk[32];
#pragma unroll
      for (int i = 0; i < 64; i += 4) {
        const float e0 = fast_exp2(fmaf(__uint_as_float(sv[i]), sl2, neg_m));
        const float e1 = fast_exp2(fmaf(__uint_as_float(sv[i + 1]), sl2, neg_m));
        const float e2 = fast_exp2(fmaf(__uint_as_float(sv[i + 2]), sl2, neg_m));
        const float e3 = fast_exp2(fmaf(__uint_as_float(sv[i + 3]), sl2, neg_m));
        l0 += e0; l1 += e1; l2 += e2; l3 += e3;
        pk[i >> 1] = pack_bf16x2(e0, e1);
        pk[(i >> 1) + 1] = pack_bf16x2(e2, e3);
      }
      tmem_st32(s_addr + half * 32, pk);          // P over the first 64 columns of S (two keys per column)
      l_run = l_run * alpha + ((l0 + l1) + (l2 + l3));
      m_run = m_cand;
      if (j > 0 && __any_sync(0xffffffffu, grow)) {
        // some row of this warp moved its maximum: rescale O (needs the previous P*V finished)
        ok = warp_wait(o_done, (j - 1) & 1);
        if (!ok) { if (lane == 0) report_error(p.status, OA_KERR_WAIT_TMEM_FULL); break; }
        tc_fence_after();
#pragma unroll
        for (int c = 0; c < OC / 32; ++c) {
          uint32_t o[32];
          tmem_ld32(o_addr + c * 32, o);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
          tmem_st32(o_addr + c * 32, o);
        }
      }
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&p_full[j & 1]);
    }
    // combine the two partial row sums (parity slot of an iteration that is two behind any reader)
    {
      float* slots = xch + (n_kv & 1) * (2 * FA_BM);
      slots[(half ^ 1) * FA_BM + r] = l_run;
      pair_sync(quad);
      l_run += slots[half * FA_BM + r];
    }
    if (ok) {
      ok = warp_wait(o_done, (n_kv - 1) & 1);
      if (!ok && lane == 0) report_error(p.status, OA_KERR_WAIT_TMEM_FULL);
    }
    if (ok) {
      tc_fence_after();
      const float inv = l_run > 0.f ? 1.f / l_run : 0.f;
      __nv_bfloat16* op = p.o + (long long)(row0 + qi) * p.o_stride + h * HD + half * OC;
#pragma unroll
      for (int c = 0; c < OC / 32; ++c) {
        uint32_t o[32];
        tmem_ld32(o_addr + c * 32, o);
        tmem_ld_wait();
        if (qi < p.seq) {
#pragma unroll
          for (int g = 0; g < 4; ++g)
            *reinterpret_cast<uint4*>(op + c * 32 + g * 8) = make_uint4(
                pack_bf16x2(__uint_as_float(o[g * 8]) * inv, __uint_as_float(o[g * 8 + 1]) * inv),
                pack_bf16x2(__uint_as_float(o[g * 8 + 2]) * inv, __uint_as_float(o[g * 8 + 3]) * inv),
                pack_bf16x2(__uint_as_float(o[g * 8 + 4]) * inv, __uint_as_float(o[g * 8 + 5]) * inv),
                pack_bf16x2(__uint_as_float(o[g * 8 + 6]) * inv, __uint_as_float(o[g * 8 + 7]) * inv));
        }
      }
      if (p.lse && half == 0 && qi < p.seq) p.lse[((long long)b * p.heads + h) * p.seq + qi] = (m_run + log2f(l_run)) / LOG2E;
    }
  }
  pdl_launch_dependents();
  tc_fence_before();
  __syncthreads();
  if (warp == 8) { tc_fence_after(); tmem_dealloc<Cfg::TMEM_COLS>(tmem_base); }
}

// ===================================================================================== forward: two tiles per CTA
// Two adjacent 128-query tiles of one (batch, head) share a CTA and the K / V rings, softmax warps 0-3 for tile 0, warps 4-7 for
// tile 1, and the exponentials of one tile cover the TMEM traffic, row maxima and barrier hand-offs of the other.  One thread owns one
// query row (all 128 key columns: no partner exchange).  The running maximum is updated lazily, as above.
// Two threads per row (sixteen softmax warps, maxima exchanged through shared memory) measured 127.7 instead of 121.7 us at head
// dim 64 (8 x 2048 x 16).
// Head dim 64: the score tile is copied to registers and RELEASED at once, so Q K_{j+1}^T is issued while the exponentials of block j
// run; probabilities have their own TMEM columns, S0 | S1 | P0 | P1 | O0 | O1 = 128 + 128 + 64 + 64 + 64 + 64, and each tile an issuing
// warp (one warp for both: 125 us against 116, 8 x 2048 x 16 causal).  Bound by the exponentials, 2048 clocks of about 3,000 a pair of blocks.
// Head dim 128: O takes the columns of P, so P_t overwrites the first half of S_t (S0 | S1 | O0 | O1 = 4 x 128 columns), and Q K_{j+1}^T
// of a tile can only follow its P V_j.  What counts is that the tiles take turns: ONE warp issues P V and the next scores of one tile and
// then those of the other, so that a tile's products run at the full rate under the other's exponentials.  With a warp for each tile the
// products of both were in the pipe together and the exponentials of both after them: 4,870 clocks a pair of blocks, 3,510 in turns, of which the
// products need 2,080 (and more while copies and operands share the 128 bytes a clock of shared memory).  P is handed over in halves of
// the keys.  Measured 1 x 4096 x 32 / 2 x 3001 x 16 causal: 168 / 108 us before, 134 / 86 in turns, 130 / 84 with P in halves, 124 / 79.5 with
// packed arithmetic and a part of the exponentials on the multiply-add pipe.  A wait more in the issuing warp, even for a
// barrier that is complete, costs (141 / 90 us with the ring waits and arrivals made once per tile and not once for both).
template <int HD_>
struct FwdPairCfg {
  static constexpr int HD = HD_;
  static constexpr bool ALIAS = HD == 128;
  static constexpr int NS = ALIAS ? 2 : 3;
  static constexpr int Q_BYTES = FA_BM * HD * 2;
  static constexpr int KV_BYTES = FA_BN * HD * 2;
  static constexpr int OFF_Q = 0;
  static constexpr int OFF_K = OFF_Q + 2 * Q_BYTES;
  static constexpr int OFF_V = OFF_K + NS * KV_BYTES;
  static constexpr int OFF_BAR = OFF_V + NS * KV_BYTES;
  static constexpr int SMEM_BYTES = OFF_BAR + 256;
  static constexpr int TMEM_COLS = 512;
  static constexpr int TM_S = 0, TM_P = ALIAS ? 0 : 256, P_STEP = ALIAS ? FA_BN : 64, TM_O = ALIAS ? 256 : 384;   // S: + 128 * tile, O: + HD * tile
  static constexpr int MMA_WARPS = ALIAS ? 1 : 2, TMA_WARP = 8 + MMA_WARPS;   // after 8 softmax warps
  static constexpr int THREADS = (TMA_WARP + 1) * 32;
};

__device__ __forceinline__ float fmax3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}

// Persistent: one CTA per SM walks the work items (tile pair, head, batch) it owns, heaviest causal pairs first and items
// dealt in snake order (round r: CTA c takes item r G + c, or r G + G-1-c when r is odd; within 3 % of the greedy optimum), so TMEM, barriers and the K / V rings live across items, the producer and the MMA warps run ahead
// into the next item while the softmax warps write the previous output, and no SM pays a CTA launch per item.  Every
// barrier phase is derived from a running count kept identically by its producers and consumers.
template <int HD>
__global__ void __launch_bounds__(FwdPairCfg<HD>::THREADS, 1)
flash_fwd_pair_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                      const __grid_constant__ CUtensorMap tmV, const FlashParams p) {
  using Cfg = FwdPairCfg<HD>;
  constexpr int NS = Cfg::NS;
  constexpr bool ALIAS = Cfg::ALIAS;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + Cfg::OFF_BAR);
  uint64_t* q_full = bars + 0;
  uint64_t* q_empty = bars + 1;            // the MMA warps are done with the Q tiles of the item
  uint64_t* k_full = bars + 2;             // [NS]
  uint64_t* k_empty = k_full + NS;         // [NS]  one arrival per MMA warp
  uint64_t* v_full = k_empty + NS;         // [NS]
  uint64_t* v_empty = v_full + NS;         // [NS]  one arrival per MMA warp
  uint64_t* s_full = v_empty + NS;         // [2]   S_t holds Q_t K_j^T
  uint64_t* s_empty = s_full + 2;          // [2]   ... and is in registers (4 warps)
  uint64_t* p_full = s_full + 4;           // [2][2]  P_t written, by half of the keys (the first: O_t rescaled if needed) (4 warps)
  uint64_t* o_done = s_full + 8;           // [2]   O_t += P_t V_j finished: P_t may be overwritten, O_t may be rescaled
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(s_full + 10);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nblk = (p.seq + FA_BM - 1) / FA_BM;
  const int npair = (nblk + 1) >> 1;
  const int hb = p.heads * p.batch;
  const int n_items = npair * hb;
  const int n_rounds = (n_items + (int)gridDim.x - 1) / (int)gridDim.x;
  auto item_of = [&](int round) -> int {     // snake order; >= n_items: this CTA sits the round out
    return round * (int)gridDim.x + ((round & 1) ? (int)gridDim.x - 1 - (int)blockIdx.x : (int)blockIdx.x);
  };

  if ((smem_u32(smem) & 1023u) != 0) {
    if (threadIdx.x == 0) report_error(p.status, OA_KERR_BAD_ARG);
    return;
  }
  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmQ); tma_prefetch_desc(&tmK); tma_prefetch_desc(&tmV);
    mbar_init(q_full, 1);
    mbar_init(q_empty, Cfg::MMA_WARPS);
    for (int s = 0; s < NS; ++s) { mbar_init(&k_full[s], 1); mbar_init(&v_full[s], 1); mbar_init(&k_empty[s], Cfg::MMA_WARPS); mbar_init(&v_empty[s], Cfg::MMA_WARPS); }
    for (int t = 0; t < 2; ++t) { mbar_init(&s_full[t], 1); mbar_init(&s_empty[t], 4); mbar_init(&p_full[2 * t], 4); mbar_init(&p_full[2 * t + 1], 4); mbar_init(&o_done[t], 1); }
    mbar_fence_init();
  }
  if (warp == 8) { tmem_alloc<Cfg::TMEM_COLS>(tmem_slot); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_wait();                            // the prologue above ran under the previous kernel's tail; global memory from here on

  // item -> (pair, head, batch) and the block counts of its two tiles (tile 1 absent: 0)
  auto decode = [&](int item, int& pr, int& h, int& b, int& nkv0, int& nkv1) {
    pr = npair - 1 - item / hb;
    const int rem = item % hb;
    h = rem % p.heads;
    b = rem / p.heads;
    nkv0 = p.causal ? (2 * pr + 1) : nblk;
    nkv1 = (2 * pr + 1 < nblk) ? (p.causal ? (2 * pr + 2) : nblk) : 0;
  };

  if (warp == Cfg::TMA_WARP) {
    // ------------- producer
    uint32_t blk = 0, itc = 0;   // K / V blocks and items loaded so far
    bool ok = true;
    for (int round = 0; round < n_rounds && ok; ++round) {
      const int item = item_of(round);
      if (item >= n_items) continue;
      int pr, h, b, nkv0, nkv1;
      decode(item, pr, h, b, nkv0, nkv1);
      const int n_it = max(nkv0, nkv1), row0 = b * p.seq;
      if (!warp_wait(q_empty, (itc & 1) ^ 1)) { if (lane == 0) report_error(p.status, OA_KERR_WAIT_EMPTY); break; }
      if (elect_one()) {
        const int tiles = nkv1 > 0 ? 2 : 1;
        mbar_expect_tx(q_full, tiles * Cfg::Q_BYTES);
        for (int t = 0; t < tiles; ++t)
#pragma unroll
          for (int x = 0; x < HD / 64; ++x)
            tma_load_2d(smem + Cfg::OFF_Q + t * Cfg::Q_BYTES + x * (FA_BM * 128), &tmQ, q_full, h * HD + x * 64, row0 + (2 * pr + t) * FA_BM);
      }
      for (int j = 0; j < n_it; ++j, ++blk) {
        const int st = blk % NS;
        const uint32_t ph = (blk / NS) & 1;
        if (!warp_wait(&k_empty[st], ph ^ 1)) { if (lane == 0) report_error(p.status, OA_KERR_WAIT_EMPTY); ok = false; break; }
        if (elect_one()) {
          mbar_expect_tx(&k_full[st], Cfg::KV_BYTES);
#pragma unroll
          for (int x = 0; x < HD / 64; ++x)
            tma_load_2d(smem + Cfg::OFF_K + st * Cfg::KV_BYTES + x * (FA_BN * 128), &tmK, &k_full[st], h * HD + x * 64, row0 + j * FA_BN);
        }
        if (!warp_wait(&v_empty[st], ph ^ 1)) { if (lane == 0) report_error(p.status, OA_KERR_WAIT_EMPTY); ok = false; break; }
        if (elect_one()) {
          mbar_expect_tx(&v_full[st], Cfg::KV_BYTES);
#pragma unroll
          for (int x = 0; x < HD / 64; ++x)
            tma_load_2d(smem + Cfg::OFF_V + st * Cfg::KV_BYTES + x * (FA_BN * 128), &tmV, &v_full[st], h * HD + x * 64, row0 + j * FA_BN);
        }
        __syncwarp();
      }
      ++itc;
    }
  } else if (ALIAS && warp == 8) {
    // ------------- MMA issuer of both tiles, in turn (warp-uniform waits, one lane issues)
    constexpr uint32_t idesc_qk = umma_idesc_bf16(FA_BM, FA_BN, 0, 0);
    constexpr uint32_t idesc_pv = umma_idesc_bf16(FA_BM, HD, 0, 1);
    uint32_t base = 0, itc = 0, pc[2] = {0, 0};   // K / V blocks before this item, items, P V products of each tile so far
    bool ok = true;
    const uint64_t q_desc = desc_k(smem + Cfg::OFF_Q), k_desc = desc_k(smem + Cfg::OFF_K), v_desc = desc_mn(smem + Cfg::OFF_V);
    // S_t = Q_t K^T of ring block `blk`; `first` / `last`: of the tiles that read it, `end`: nothing reads Q after it
    auto issue_qk = [&](int t, uint32_t blk, bool first, bool last, bool end) -> bool {
      const int st = blk % NS;
      if (first && !warp_wait(&k_full[st], (blk / NS) & 1)) { if (lane == 0) report_error(p.status, OA_KERR_WAIT_FULL); return false; }
      tc_fence_after();
      if (elect_one()) {
        const uint64_t qd = desc_at(q_desc, t * Cfg::Q_BYTES), kd = desc_at(k_desc, st * Cfg::KV_BYTES);
#pragma unroll
        for (int ks = 0; ks < HD / 16; ++ks) {
          const uint32_t off = (ks >> 2) * (FA_BM * 128) + (ks & 3) * 32;
          umma_f16(tmem_base + Cfg::TM_S + t * FA_BN, desc_at(qd, off), desc_at(kd, off), idesc_qk, ks > 0 ? 1u : 0u);
        }
        umma_commit(&s_full[t]);
        if (last) umma_commit(&k_empty[st]);
        if (end) umma_commit(q_empty);
      }
      __syncwarp();
      return true;
    };
    for (int round = 0; round < n_rounds && ok; ++round) {
      const int item = item_of(round);
      if (item >= n_items) continue;
      int pr, h, b, n[2];
      decode(item, pr, h, b, n[0], n[1]);
      const int n_it = max(n[0], n[1]);
      if (!warp_wait(q_full, itc & 1)) { if (lane == 0) report_error(p.status, OA_KERR_WAIT_FULL); break; }
      // a block's tiles: both, or the one whose row of blocks is longer (tile 1, unless it is absent)
      auto qk = [&](int t, int j) -> bool {
        const bool last = j >= n[1 - t] || t == 1;
        return issue_qk(t, base + j, t == 0 || j >= n[0], last, last && j + 1 == n_it);
      };
      if (n[0] > 0) ok = qk(0, 0);
      if (ok && n[1] > 0) ok = qk(1, 0);
      for (int j = 0; j < n_it && ok; ++j) {
        const int st = (base + j) % NS;
        if (!warp_wait(&v_full[st], ((base + j) / NS) & 1)) { if (lane == 0) report_error(p.status, OA_KERR_WAIT_FULL); ok = false; break; }
#pragma unroll
        for (int t = 0; t < 2; ++t) {
          if (j >= n[t]) continue;
#pragma unroll
          for (int half = 0; half < 2; ++half) {
            if (!warp_wait(&p_full[2 * t + half], pc[t] & 1)) { if (lane == 0) report_error(p.status, OA_KERR_WAIT_SOFTMAX); ok = false; break; }
            tc_fence_after();
            if (elect_one()) {
              const uint64_t vd = desc_at(v_desc, st * Cfg::KV_BYTES);
              const uint32_t p_tm = tmem_base + Cfg::TM_P + t * Cfg::P_STEP, o_tm = tmem_base + Cfg::TM_O + t * HD;
#pragma unroll
              for (int ks = half * 4; ks < half * 4 + 4; ++ks)
                umma_f16_ts(o_tm, p_tm + ks * 8, desc_at(vd, ks * 2048), idesc_pv, (j > 0 || ks > 0) ? 1u : 0u);
              if (half == 1) {
                if (t == 1 || j >= n[1]) umma_commit(&v_empty[st]);
                if (j + 1 == n[t]) umma_commit(&o_done[t]);
              }
            }
            __syncwarp();
          }
          if (!ok) break;
          ++pc[t];
          if (j + 1 < n[t]) { ok = qk(t, j + 1); if (!ok) break; }   // overwrites P_j: ordered after P_j V_j by the pipe
        }
      }
      base += n_it;
      ++itc;
    }
  } else if (!ALIAS && warp >= 8) {
    // ------------- MMA issuer of tile t (warp-uniform waits, lane 0 issues)
    const int t = warp - 8;
    constexpr uint32_t idesc_qk = umma_idesc_bf16(FA_BM, FA_BN, 0, 0);
    constexpr uint32_t idesc_pv = umma_idesc_bf16(FA_BM, HD, 0, 1);
    const uint64_t qd = desc_k(smem + Cfg::OFF_Q + t * Cfg::Q_BYTES), k_desc = desc_k(smem + Cfg::OFF_K), v_desc = desc_mn(smem + Cfg::OFF_V);
    const uint32_t s_tm = tmem_base + Cfg::TM_S + t * FA_BN, p_tm = tmem_base + Cfg::TM_P + t * Cfg::P_STEP, o_tm = tmem_base + Cfg::TM_O + t * HD;
    uint32_t base = 0, itc = 0, sc = 0, pc = 0;   // K / V blocks before this item, items, S products and P V products of this tile so far
    bool ok = true;
    auto issue_qk = [&](uint32_t blk, bool last) -> bool {       // S_t = Q_t K^T of ring block `blk`
      const int st = blk % NS;
      if (!warp_wait(&k_full[st], (blk / NS) & 1)) { if (lane == 0) report_error(p.status, OA_KERR_WAIT_FULL); return false; }
      if (sc > 0 && !warp_wait(&s_empty[t], (sc - 1) & 1)) { if (lane == 0) report_error(p.status, OA_KERR_WAIT_TMEM_EMPTY); return false; }
      tc_fence_after();
      if (elect_one()) {
        const uint64_t kd = desc_at(k_desc, st * Cfg::KV_BYTES);
#pragma unroll
        for (int ks = 0; ks < HD / 16; ++ks) {
          const uint32_t off = (ks >> 2) * (FA_BM * 128) + (ks & 3) * 32;
          umma_f16(s_tm, desc_at(qd, off), desc_at(kd, off), idesc_qk, ks > 0 ? 1u : 0u);
        }
        umma_commit(&k_empty[st]);
        umma_commit(&s_full[t]);
        if (last) umma_commit(q_empty);
      }
      __syncwarp();
      ++sc;
      return true;
    };
    for (int round = 0; round < n_rounds && ok; ++round) {
      const int item = item_of(round);
      if (item >= n_items) continue;
      int pr, h, b, nkv0, nkv1;
      decode(item, pr, h, b, nkv0, nkv1);
      const int n_it = max(nkv0, nkv1);
      const int n = t == 0 ? nkv0 : nkv1;
      if (!warp_wait(q_full, itc & 1)) { if (lane == 0) report_error(p.status, OA_KERR_WAIT_FULL); break; }
      if (n > 0) ok = issue_qk(base, n == 1);
      for (int j = 0; j < n && ok; ++j) {
        if (j + 1 < n) { ok = issue_qk(base + j + 1, j + 2 == n); if (!ok) break; }
        const int st = (base + j) % NS;
        if (!warp_wait(&v_full[st], ((base + j) / NS) & 1)) { if (lane == 0) report_error(p.status, OA_KERR_WAIT_FULL); ok = false; break; }
        if (!warp_wait(&p_full[2 * t], pc & 1)) { if (lane == 0) report_error(p.status, OA_KERR_WAIT_SOFTMAX); ok = false; break; }
        tc_fence_after();
        if (elect_one()) {
          const uint64_t vd = desc_at(v_desc, st * Cfg::KV_BYTES);
#pragma unroll
          for (int ks = 0; ks < FA_BN / 16; ++ks)
            umma_f16_ts(o_tm, p_tm + ks * 8, desc_at(vd, ks * 2048), idesc_pv, (j > 0 || ks > 0) ? 1u : 0u);
          umma_commit(&v_empty[st]);
          umma_commit(&o_done[t]);
        }
        __syncwarp();
        ++pc;
      }
      // blocks of this item that this tile does not use (the last one of the pair's shorter tile, or all of an absent tile):
      // the rings still expect one arrival per MMA warp, given once the block has landed
      for (int j = n; j < n_it && ok; ++j) {
        const int st = (base + j) % NS;
        const uint32_t ph = ((base + j) / NS) & 1;
        if (!warp_wait(&k_full[st], ph)) { if (lane == 0) report_error(p.status, OA_KERR_WAIT_FULL); ok = false; break; }
        if (lane == 0) mbar_arrive(&k_empty[st]);
        if (!warp_wait(&v_full[st], ph)) { if (lane == 0) report_error(p.status, OA_KERR_WAIT_FULL); ok = false; break; }
        if (lane == 0) mbar_arrive(&v_empty[st]);
        __syncwarp();
      }
      if (n == 0 && ok && lane == 0) mbar_arrive(q_empty);
      __syncwarp();
      base += n_it;
      ++itc;
    }
  } else {
    // ------------- softmax + output of tile t: one thread per query row
    const int t = warp >> 2;
    const int quad = warp & 3;
    const int r = quad * 32 + lane;
    const uint32_t t_lane = (uint32_t)(quad * 32) << 16;
    const uint32_t s_addr = tmem_base + t_lane + Cfg::TM_S + t * FA_BN;
    const uint32_t p_addr = tmem_base + t_lane + Cfg::TM_P + t * Cfg::P_STEP;
    const uint32_t o_addr = tmem_base + t_lane + Cfg::TM_O + t * HD;
    const float sl2 = p.scale * LOG2E;
    uint32_t sc = 0, pc = 0;     // score tiles consumed and P V completions awaited so far
    bool ok = true;
    for (int round = 0; round < n_rounds && ok; ++round) {
      const int item = item_of(round);
      if (item >= n_items) continue;
      int pr, h, b, nkv0, nkv1;
      decode(item, pr, h, b, nkv0, nkv1);
      const int n = t == 0 ? nkv0 : nkv1;
      if (n == 0) continue;
      const int row0 = b * p.seq;
      const int qbt = 2 * pr + t;
      const int qi = qbt * FA_BM + r;               // query index inside the sequence
      float m_run = -INFINITY, l_run = 0.f;
      for (int j = 0; j < n; ++j, ++sc) {
        ok = warp_wait(&s_full[t], sc & 1);
        if (!ok) { if (lane == 0) report_error(p.status, OA_KERR_WAIT_TMEM_FULL); break; }
        tc_fence_after();
        uint32_t sv[FA_BN];
#pragma unroll
        for (int c = 0; c < FA_BN / 32; ++c) tmem_ld32(s_addr + c * 32, sv + c * 32);
        tmem_ld_wait();
        if (!ALIAS) {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&s_empty[t]);   // the next block's scores may overwrite S_t now
        }
        const bool need_mask = (p.causal && j == qbt) || (j * FA_BN + FA_BN > p.seq);
        if (need_mask) {
          const int lim = min(p.causal ? qi : 0x7fffffff, p.seq - 1) - j * FA_BN;   // columns i <= lim are alive
#pragma unroll
          for (int i = 0; i < FA_BN; ++i) sv[i] = (i <= lim) ? sv[i] : 0xff800000u;  // -inf
        }
        float m0 = __uint_as_float(sv[0]), m1 = __uint_as_float(sv[1]);
#pragma unroll
        for (int i = 2; i < FA_BN - 2; i += 4) {
          m0 = fmax3(m0, __uint_as_float(sv[i]), __uint_as_float(sv[i + 1]));
          m1 = fmax3(m1, __uint_as_float(sv[i + 2]), __uint_as_float(sv[i + 3]));
        }
        const float mx = fmax3(m0, m1, fmaxf(__uint_as_float(sv[FA_BN - 2]), __uint_as_float(sv[FA_BN - 1]))) * sl2;
        const float m_new = fmaxf(m_run, mx);
        const bool grow = (m_new - m_run) > FA_RESCALE_THRESHOLD;           // first block: m_run = -inf -> true
        const float m_cand = grow ? m_new : m_run;
        const float m_use = (m_cand == -INFINITY) ? 0.f : m_cand;           // row fully masked so far
        const float alpha = grow ? fast_exp2(m_run - m_use) : 1.f;           // m_run = -inf -> 0
        const float neg_m = -m_use;
        // P_t is free and O_t is complete once the previous P V has finished (head dim 128: s_full already says so, the scores were
        // issued behind it)
        if (!ALIAS && j > 0) {
          ok = warp_wait(&o_done[t], pc & 1);
          if (!ok) { if (lane == 0) report_error(p.status, OA_KERR_WAIT_TMEM_FULL); break; }
          ++pc;
          tc_fence_after();
        }
        auto rescale = [&]() {                               // some row of this warp moved its maximum: rescale O
          if (j == 0 || !__any_sync(0xffffffffu, grow)) return;
#pragma unroll 1
          for (int q = 0; q < HD / 32; ++q) {
            uint32_t o[32];
            tmem_ld32(o_addr + q * 32, o);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
            tmem_st32(o_addr + q * 32, o);
          }
        };
        auto hand_over = [&](int half) {
          tmem_st_wait();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&p_full[2 * t + half]);
        };
        unsigned long long l01 = 0, l23 = 0;
        const unsigned long long sl22 = f2_splat(sl2), neg_m2 = f2_splat(neg_m);
#pragma unroll
        for (int c = 0; c < FA_BN / 32; ++c) {
          uint32_t pk[16];
#pragma unroll
          for (int i = 0; i < 32; i += 4) {
            const uint32_t* sc4 = sv + c * 32 + i;
            const unsigned long long x01 = f2_fma(f2_of(sc4[0], sc4[1]), sl22, neg_m2), x23 = f2_fma(f2_of(sc4[2], sc4[3]), sl22, neg_m2);
            const unsigned long long e01 = exp2_mufu2(x01), e23 = (i >> 2) % 4 < FA_FMA_PAIRS ? exp2_fma2(x23) : exp2_mufu2(x23);
            l01 = f2_add(l01, e01);
            l23 = f2_add(l23, e23);
            pk[i >> 1] = f2_bf16(e01);
            pk[(i >> 1) + 1] = f2_bf16(e23);
          }
          tmem_st16(p_addr + c * 16, pk);
          if (ALIAS && (c & 1)) {                        // the products of half of the keys start under the other half's exponentials
            if (c == 1) rescale();
            hand_over(c >> 1);
          }
        }
        if (!ALIAS) {
          rescale();
          hand_over(0);
        }
        uint32_t lw[4];
        f2_to(l01, lw[0], lw[1]);
        f2_to(l23, lw[2], lw[3]);
        l_run = l_run * alpha + ((__uint_as_float(lw[0]) + __uint_as_float(lw[1])) + (__uint_as_float(lw[2]) + __uint_as_float(lw[3])));
        m_run = m_cand;
      }
      if (!ok) break;
      ok = warp_wait(&o_done[t], pc & 1);
      if (!ok) { if (lane == 0) report_error(p.status, OA_KERR_WAIT_TMEM_FULL); break; }
      ++pc;
      tc_fence_after();
      const float inv = l_run > 0.f ? 1.f / l_run : 0.f;
      const int q0 = qbt * FA_BM + quad * 32;
      __nv_bfloat16* op = p.o + (long long)(row0 + q0) * p.o_stride + h * HD;
#pragma unroll
      for (int c = 0; c < HD / 32; ++c) {
        uint32_t o[32];
        tmem_ld32(o_addr + c * 32, o);
        tmem_ld_wait();
        // At head dim 64 a row's 16 bytes to a lane are the faster: 8 x 2048 x 16 causal 109.0 us (115.6 through store_rows), 1 x 4096 x 16 full
        // 103.2 (114.3), 32 x 256 x 16 23.0 (24.1), 64 x 128 x 16 full 21.2 (22.8)
        if (ALIAS) store_rows(op + c * 32, p.o_stride, p.seq - q0, o, inv, lane);
        else if (qi < p.seq) {
          __nv_bfloat16* od = p.o + (long long)(row0 + qi) * p.o_stride + h * HD + c * 32;
#pragma unroll
          for (int g = 0; g < 4; ++g)
            *reinterpret_cast<uint4*>(od + g * 8) = make_uint4(
                pack_bf16x2(__uint_as_float(o[g * 8]) * inv, __uint_as_float(o[g * 8 + 1]) * inv),
                pack_bf16x2(__uint_as_float(o[g * 8 + 2]) * inv, __uint_as_float(o[g * 8 + 3]) * inv),
                pack_bf16x2(__uint_as_float(o[g * 8 + 4]) * inv, __uint_as_float(o[g * 8 + 5]) * inv),
                pack_bf16x2(__uint_as_float(o[g * 8 + 6]) * inv, __uint_as_float(o[g * 8 + 7]) * inv));
        }
      }
      if (p.lse && qi < p.seq) p.lse[((long long)b * p.heads + h) * p.seq + qi] = (m_run + log2f(l_run)) / LOG2E;
      tc_fence_before();   // the O reads above complete before this warp's next p_full arrival lets the next item's first P V overwrite O
    }
  }
  pdl_launch_dependents();
  tc_fence_before();
  __syncthreads();
  if (warp == 8) { tc_fence_after(); tmem_dealloc<Cfg::TMEM_COLS>(tmem_base); }
}

template <int HD>
static int launch_fwd2(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const FlashParams& p, dim3 grid, cudaStream_t st) {
  static bool set = false;
  if (!set) {
    if (cudaFuncSetAttribute(flash_fwd2_kernel<HD>, cudaFuncAttributeMaxDynamicSharedMemorySize, Fwd2Cfg<HD>::SMEM_BYTES) != cudaSuccess) return OA_ERR_LAUNCH;
    set = true;
  }
  launch_pdl(flash_fwd2_kernel<HD>, grid, dim3(FA_THREADS), Fwd2Cfg<HD>::SMEM_BYTES, st, tq, tk, tv, p);
  return cudaGetLastError() == cudaSuccess ? OA_OK : OA_ERR_LAUNCH;
}

// Head dim 128: whether the pair kernel beats one tile per CTA.  A pair of tiles takes 1.55 times as long as one, so it loses only where
// pairs leave SMs free that single tiles would fill.  Full rows are a matter of whole waves: single tile against pair, us, at 8 key blocks
// 60 / 148 / 200 / 300 pairs 17.1 / 22.0, 30.6 / 24.2, 41.6 / 38.5, 67.7 / 54.0; at 32 64 / 96 / 160 / 304 / 992 pairs 43 / 62, 79 / 63, 112 / 114,
// 184 / 171, 508 / 378; at 64 96 / 192 / 448 141 / 115, 210 / 227, 480 / 444.  Causal rows even out over the SMs: 4 blocks 60 / 148 / 300 pairs
// 19.7 / 20.5, 22.0 / 19.7, 39.6 / 28.2; 9 blocks 60 / 100 / 150 / 445 21.0 / 22.1, 24.2 / 22.0, 30.0 / 24.0, 69.1 / 50.5; 16 blocks 96 / 144 / 600 34.2 / 35.8,
// 42.7 / 36.3, 127 / 88; 32 blocks 96 / 144 / 992 50 / 61, 67 / 63, 306 / 207.
static bool flash_pair_hd128(int nblk, long long heads, long long batch, int causal, int sms) {
  if (heads > 65535 || batch > 65535) return true;       // beyond the single-tile kernel's grid
  const long long rows = heads * batch, items = (long long)((nblk + 1) / 2) * rows;
  if (causal) return nblk <= 7 || (nblk <= 12 ? 3 * items >= 2 * sms : items >= sms);
  const long long pair_rounds = (items + sms - 1) / sms, tile_waves = (nblk * rows + sms - 1) / sms;
  return 2 * tile_waves > 3 * pair_rounds || (tile_waves > pair_rounds && nblk < 24);
}

template <int HD>
static int launch_fwd_pair(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const FlashParams& p, cudaStream_t st) {
  static int sms = 0;
  if (sms == 0) {
    int dev = 0, n = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return OA_ERR_DRIVER;
    if (cudaFuncSetAttribute(flash_fwd_pair_kernel<HD>, cudaFuncAttributeMaxDynamicSharedMemorySize, FwdPairCfg<HD>::SMEM_BYTES) != cudaSuccess) return OA_ERR_LAUNCH;
    sms = n;
  }
  const int nblk = (p.seq + FA_BM - 1) / FA_BM;
  if constexpr (HD == 128)
    if (!flash_pair_hd128(nblk, p.heads, p.batch, p.causal, sms)) return launch_fwd2<HD>(tq, tk, tv, p, dim3(nblk, p.heads, p.batch), st);
  const long long items = (long long)((nblk + 1) / 2) * p.heads * p.batch;
  const int ctas = (int)(items < sms ? items : sms);
  launch_pdl(flash_fwd_pair_kernel<HD>, dim3(ctas), dim3(FwdPairCfg<HD>::THREADS), FwdPairCfg<HD>::SMEM_BYTES, st, tq, tk, tv, p);
  return cudaGetLastError() == cudaSuccess ? OA_OK : OA_ERR_LAUNCH;
}

// ===================================================================================== backward
struct FlashBwdParams {
  int batch, heads, seq, head_dim;
  float scale;
  int causal;
  const float* lse;      // [B, H, S]
  const float* delta;    // [B, H, S]  sum_d dO * O
  __nv_bfloat16* dq; long long dq_stride;
  __nv_bfloat16* dk; __nv_bfloat16* dv; long long dkv_stride;
  int* status;
};

// delta[b,h,i] = sum_d dO[i, h*hd + d] * O[i, h*hd + d]; hd / 8 lanes per (row, head), 16-byte loads.
__global__ void __launch_bounds__(256)
flash_delta_kernel(const __nv_bfloat16* __restrict__ o, const __nv_bfloat16* __restrict__ dout, float* __restrict__ delta, int batch,
                   int heads, int seq, int hd, long long o_stride, long long do_stride) {
  pdl_launch_dependents();
  pdl_wait();
  const int lpi = hd >> 3;                                   // lanes per item: 8 (hd 64) or 16 (hd 128)
  const long long total = (long long)batch * seq * heads;
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long item = t / lpi;
  const int sub = (int)(t % lpi);
  float s = 0.f;
  int h = 0;
  long long row = 0;
  if (item < total) {
    h = (int)(item % heads);
    row = item / heads;
    const uint4 a = *reinterpret_cast<const uint4*>(o + row * o_stride + h * hd + sub * 8);
    const uint4 b = *reinterpret_cast<const uint4*>(dout + row * do_stride + h * hd + sub * 8);
    const float2 a0 = unpack_bf16x2(a.x), a1 = unpack_bf16x2(a.y), a2 = unpack_bf16x2(a.z), a3 = unpack_bf16x2(a.w);
    const float2 b0 = unpack_bf16x2(b.x), b1 = unpack_bf16x2(b.y), b2 = unpack_bf16x2(b.z), b3 = unpack_bf16x2(b.w);
    s = a0.x * b0.x + a0.y * b0.y + a1.x * b1.x + a1.y * b1.y + a2.x * b2.x + a2.y * b2.y + a3.x * b3.x + a3.y * b3.y;
  }
  for (int off = lpi >> 1; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
  if (item < total && sub == 0) {
    const int bi = (int)(row / seq), si = (int)(row % seq);
    delta[((long long)bi * heads + h) * seq + si] = s;
  }
}

constexpr int FA_BWD_THREADS = 352;   // 8 softmax warps + 2 MMA issuer warps + 1 TMA warp

// Backward pipeline (both kernels).  A tile passes through two phases in the eight softmax warps (two threads per TMEM lane, 64 columns
// each): scores -> probabilities, then dP -> dS.  The phases have barriers of their own, so the tensor pipe always has the other
// phase's products to run: under the exponentials of tile i it works on dS_{i-1}'s gradient product and on dP_i, and under
// the dS phase of tile i it consumes P_i and forms the scores of tile i + 1.  One warp issues the products that hang on the
// probabilities (scores and dV), the other those that hang on dS (dP and dK, or dP and dQ); within a warp the products that reuse
// tensor-memory columns are ordered by the pipe.  The bf16 results overwrite the columns they were computed from, each half of the
// columns within its own 64, so neither half waits for the other before it stores, and the gradient products start on the first half.
// At head dim 128 the columns leave room for one score tile, so the scores of tile i + 1 can only follow dV of tile i, and the next
// exponentials wait for both: the issuer of dK and dP waits its turn until those scores are in the pipe (`turn`), and its products run under
// the exponentials.  Left to themselves they ran beside dV and the scores, which took twice as long, and nothing under the exponentials.
// A turn is given once per tile but an item's last, which has no scores behind it.  That the giver cannot be two turns ahead, when the barrier's
// parity would read as none, follows from the ring: turn i + 1 is given behind the scores of tile i + 2, whose Q takes the place that dK of tile
// i has left, and across items from the end of an item, which waits for the last dK.
// The kernels are bound by that chain: at head dim 64 the exponentials take 1024 of about 2,400 clocks per tile, at head dim 128 the
// products 2,080 of about 3,500, and a barrier that is already complete costs a warp 100 clocks or more while the pipes are busy.
// dK, dV and dQ leave through store_rows; with 16-byte stores of a row to a lane the end of an item took 4,000 to 5,000 clocks, 15 to 20 %.
// Measured, us of the whole backward pass: before / dK, dP in turn / rows by store_rows / part of the exponentials on the multiply-add pipe
// 1 x 4096 x 32 heads of 128 468 / 448 / 430 / 423, 2 x 3001 x 16 of 128 282 / 270 / 254 / 247, 8 x 2048 x 16 of 64 369 / 369 / 344 / 330, 8 x 512 x 16
// of 64 60 / 60 / 55 / 53.
// dK/dV and dQ kernel, with one barrier for both phases (scores and dP issued together, both read before either was computed on) -> with
// two: 2 x 3001 x 16 heads of 128 194 and 129 -> 161 and 109 us, 8 x 2048 x 16 of 64 195 and 164 -> 191 and 160.  Slower: one issuing warp for all
// four products (172 us, 260 us at head dim 64), sixteen softmax warps (300 us at head dim 64 with the two phases merged into one pass;
// every wait is made by twice the warps), one lane waiting for its warp (261 us), partner warps of a scheduler taking turns at the
// exponentials (212 us), and the halves of a tile as pipelines of their own (128 478, 64 365: a product of 64 columns takes 50 clocks, one of 128 66).
//
// The dK/dV kernel works on the TRANSPOSED tile, S^T = K Q^T with keys on the TMEM lanes, because dV = P^T dO and
// dK = dS^T Q need P^T / dS^T with keys as the M dimension.  Per-query statistics (log-sum-exp, delta) are then per
// COLUMN: the producer warp stages them in shared memory beside the Q tile and they are read as broadcasts.
template <int HD>
struct BwdKvCfg {
  static constexpr int NST = (HD == 64) ? 3 : 2;       // Q and dO rings
  static constexpr int NS = (HD == 64) ? 2 : 1;        // score buffers in TMEM (P^T lies over S^T, dS^T over dP^T)
  static constexpr int T_BYTES = FA_BM * HD * 2;        // one [128 x HD] tile
  static constexpr int OFF_K = 0;
  static constexpr int OFF_V = OFF_K + T_BYTES;
  static constexpr int OFF_Q = OFF_V + T_BYTES;
  static constexpr int OFF_DO = OFF_Q + NST * T_BYTES;
  static constexpr int OFF_STAT = OFF_DO + NST * T_BYTES;   // float[NST][256]: -lse*log2e | -delta*scale of the query block
  static constexpr int OFF_BAR = OFF_STAT + NST * 256 * 4;
  static constexpr int SMEM_BYTES = OFF_BAR + 208;
  static constexpr int TMEM_COLS = 512;
  static constexpr int TM_S = 0, TM_DP = NS * FA_BN, TM_DV = TM_DP + FA_BN, TM_DK = TM_DV + HD;
};

// Two probabilities exp2(s sl2 + nl), over the scores; two p (dp scale + nd), over the probabilities
template <bool FMA = false>
__device__ __forceinline__ void bwd_prob2(uint32_t& a, uint32_t& b, unsigned long long sl2, unsigned long long nl) {
  const unsigned long long x = f2_fma(f2_of(a, b), sl2, nl);
  f2_to(FMA ? exp2_fma2(x) : exp2_mufu2(x), a, b);
}
__device__ __forceinline__ void bwd_ds2(uint32_t& a, uint32_t& b, uint32_t d0, uint32_t d1, unsigned long long scale, unsigned long long nd) {
  f2_to(f2_mul(f2_of(a, b), f2_fma(f2_of(d0, d1), scale, nd)), a, b);
}
// 32 values of a lane as bf16 over 16 columns
__device__ __forceinline__ void bwd_store16(uint32_t taddr, const uint32_t* v) {
  uint32_t w[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) w[i] = pack_bf16x2(__uint_as_float(v[2 * i]), __uint_as_float(v[2 * i + 1]));
  tmem_st16(taddr, w);
}

// Persistent: one CTA per SM walks the work items (key block, head, batch) it owns, heaviest causal key blocks first, items
// dealt in snake order; dK, dV of an item accumulate in TMEM over its query blocks.  Barrier phases come from running counts.
template <int HD>
__global__ void __launch_bounds__(FA_BWD_THREADS, 1)
flash_bwd_kv_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                    const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmDO,
                    const FlashBwdParams p) {
  using Cfg = BwdKvCfg<HD>;
  constexpr int NST = Cfg::NST, NS = Cfg::NS;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + Cfg::OFF_BAR);
  uint64_t* kv_full = bars + 0;
  uint64_t* kv_empty = bars + 1;   // the item's last score and dP products have read K, V
  uint64_t* q_full = bars + 2;     // [3]  Q bytes and the statistics
  uint64_t* q_empty = bars + 5;    // [3]  dK has read Q (the scores and the statistics were read before)
  uint64_t* do_full = bars + 8;    // [3]
  uint64_t* do_empty = bars + 11;  // [3]  dP and dV have read dO
  uint64_t* s_full = bars + 14;    // [2]  S^T of this tile is in TMEM
  uint64_t* p_full = bars + 16;    // [2][2]  P^T, by score buffer and column half (4 warps each)
  uint64_t* dp_full = bars + 20;   // dP^T
  uint64_t* ds_full = bars + 21;   // [2]  dS^T, by column half (4 warps each)
  uint64_t* fin_full = bars + 23;  // dV, dK of the item are complete (both issuers arrive)
  uint64_t* turn = bars + 24;      // NS == 1: the next tile's scores are in the pipe, dK and dP may follow (not for an item's last tile)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 25);
  float* stat = reinterpret_cast<float*>(smem + Cfg::OFF_STAT);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nblk = (p.seq + FA_BM - 1) / FA_BM;
  const int hb = p.heads * p.batch;
  const int n_items = nblk * hb;
  const int n_rounds = (n_items + (int)gridDim.x - 1) / (int)gridDim.x;
  auto item_of = [&](int round) -> int {     // snake order; >= n_items: this CTA sits the round out
    return round * (int)gridDim.x + ((round & 1) ? (int)gridDim.x - 1 - (int)blockIdx.x : (int)blockIdx.x);
  };
  auto decode = [&](int item, int& jb, int& h, int& b) {   // key block 0 has the most query blocks under the causal mask
    jb = item / hb;
    const int rem = item % hb;
    h = rem % p.heads;
    b = rem / p.heads;
  };

  if ((smem_u32(smem) & 1023u) != 0) {
    if (threadIdx.x == 0) report_error(p.status, OA_KERR_BAD_ARG);
    return;
  }
  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmQ); tma_prefetch_desc(&tmK); tma_prefetch_desc(&tmV); tma_prefetch_desc(&tmDO);
    mbar_init(kv_full, 1);
    mbar_init(kv_empty, 2);
    for (int s = 0; s < NST; ++s) { mbar_init(&q_full[s], 2); mbar_init(&q_empty[s], 1); mbar_init(&do_full[s], 1); mbar_init(&do_empty[s], 2); }
    for (int s = 0; s < 2; ++s) { mbar_init(&s_full[s], 1); mbar_init(&ds_full[s], 4); }
    for (int s = 0; s < 4; ++s) mbar_init(&p_full[s], 4);
    mbar_init(dp_full, 1);
    mbar_init(fin_full, 2);
    mbar_init(turn, 1);
    mbar_fence_init();
  }
  if (warp == 8) { tmem_alloc<Cfg::TMEM_COLS>(tmem_slot); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_wait();                            // the prologue above ran under the previous kernel's tail; global memory from here on

  if (warp == 10) {
    // ------------- TMA producer (also stages the per-query statistics of each block)
    uint32_t itc = 0, qc = 0;       // items and Q / dO blocks loaded so far
    bool ok = true;
    for (int round = 0; round < n_rounds && ok; ++round) {
      const int item = item_of(round);
      if (item >= n_items) continue;
      int jb, h, b;
      decode(item, jb, h, b);
      const int i0 = p.causal ? jb : 0, n_it = nblk - i0, row0 = b * p.seq;
      const long long stat_base = ((long long)b * p.heads + h) * p.seq;
      if (!warp_wait(kv_empty, (itc & 1) ^ 1)) { if (lane == 0) report_error(p.status, OA_KERR_WAIT_EMPTY); break; }
      if (elect_one()) {
        mbar_expect_tx(kv_full, 2 * Cfg::T_BYTES);
#pragma unroll
        for (int x = 0; x < HD / 64; ++x) {
          tma_load_2d(smem + Cfg::OFF_K + x * (FA_BN * 128), &tmK, kv_full, h * HD + x * 64, row0 + jb * FA_BN);
          tma_load_2d(smem + Cfg::OFF_V + x * (FA_BN * 128), &tmV, kv_full, h * HD + x * 64, row0 + jb * FA_BN);
        }
      }
      for (int it = 0; it < n_it; ++it, ++qc) {
        const int st = qc % NST;
        const uint32_t ph = (qc / NST) & 1;
        const int qrow = row0 + (i0 + it) * FA_BM;
        if (!warp_wait(&q_empty[st], ph ^ 1)) { if (lane == 0) report_error(p.status, OA_KERR_WAIT_EMPTY); ok = false; break; }
        if (elect_one()) {
          mbar_expect_tx(&q_full[st], Cfg::T_BYTES);
#pragma unroll
          for (int x = 0; x < HD / 64; ++x)
            tma_load_2d(smem + Cfg::OFF_Q + st * Cfg::T_BYTES + x * (FA_BM * 128), &tmQ, &q_full[st], h * HD + x * 64, qrow);
        }
        if (!warp_wait(&do_empty[st], ph ^ 1)) { if (lane == 0) report_error(p.status, OA_KERR_WAIT_EMPTY); ok = false; break; }
        if (elect_one()) {
          mbar_expect_tx(&do_full[st], Cfg::T_BYTES);
#pragma unroll
          for (int x = 0; x < HD / 64; ++x)
            tma_load_2d(smem + Cfg::OFF_DO + st * Cfg::T_BYTES + x * (FA_BM * 128), &tmDO, &do_full[st], h * HD + x * 64, qrow);
        }
        // per-query statistics of this block, negated and pre-scaled: lane l stages queries 4l .. 4l+3
        {
          float4 nl, nd;
          float* nlp = reinterpret_cast<float*>(&nl);
          float* ndp = reinterpret_cast<float*>(&nd);
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const int qi = (i0 + it) * FA_BM + lane * 4 + u;
            const bool okq = qi < p.seq;
            nlp[u] = okq ? -p.lse[stat_base + qi] * LOG2E : -INFINITY;
            ndp[u] = okq ? -p.delta[stat_base + qi] * p.scale : 0.f;
          }
          float* dst = stat + st * 256;
          reinterpret_cast<float4*>(dst)[lane] = nl;
          reinterpret_cast<float4*>(dst + 128)[lane] = nd;
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&q_full[st]);
        __syncwarp();
      }
      ++itc;
    }
  } else if (warp == 8) {
    // ------------- MMA issuer A: S^T = K Q^T and dV += P^T dO.  S^T of a tile goes over the P^T that dV read NS tiles ago.
    constexpr uint32_t idesc_s = umma_idesc_bf16(FA_BN, FA_BM, 0, 0);
    constexpr uint32_t idesc_g = umma_idesc_bf16(FA_BN, HD, 0, 1);   // [keys x HD] += X^T[keys x q] (TMEM) * Y[q x HD]
    const uint64_t k_desc = desc_k(smem + Cfg::OFF_K), q_desc = desc_k(smem + Cfg::OFF_Q), do_desc = desc_mn(smem + Cfg::OFF_DO);
    uint32_t itc = 0, qc = 0;
    bool ok = true;
    auto issue_s = [&](uint32_t n, bool last) -> bool {
      const int st = n % NST;
      if (!warp_wait(&q_full[st], (n / NST) & 1)) { if (lane == 0) report_error(p.status, OA_KERR_WAIT_FULL); return false; }
      tc_fence_after();
      if (elect_one()) {
        const uint64_t qd = desc_at(q_desc, st * Cfg::T_BYTES);
        const uint32_t s_tm = tmem_base + Cfg::TM_S + (n % NS) * FA_BN;
#pragma unroll
        for (int ks = 0; ks < HD / 16; ++ks) {
          const uint32_t off = (ks >> 2) * (FA_BM * 128) + (ks & 3) * 32;
          umma_f16(s_tm, desc_at(k_desc, off), desc_at(qd, off), idesc_s, ks > 0 ? 1u : 0u);
        }
        umma_commit(&s_full[n % NS]);
        if (last) umma_commit(kv_empty);
      }
      __syncwarp();
      return true;
    };
    for (int round = 0; round < n_rounds && ok; ++round) {
      const int item = item_of(round);
      if (item >= n_items) continue;
      int jb, h, b;
      decode(item, jb, h, b);
      const int n_it = nblk - (p.causal ? jb : 0);
      if (!warp_wait(kv_full, itc & 1)) { if (lane == 0) report_error(p.status, OA_KERR_WAIT_FULL); break; }
      ok = issue_s(qc, n_it == 1);
      // the previous item's dV / dK were read by the softmax warps before they produced this item's first P^T, dS^T
      for (int it = 0; it < n_it && ok; ++it, ++qc) {
        if (NS == 2 && it + 1 < n_it) { ok = issue_s(qc + 1, it + 2 == n_it); if (!ok) break; }
        const int st = qc % NST;
        if (!warp_wait(&do_full[st], (qc / NST) & 1)) { if (lane == 0) report_error(p.status, OA_KERR_WAIT_FULL); ok = false; break; }
        const uint64_t bd = desc_at(do_desc, st * Cfg::T_BYTES);
        const uint32_t a_addr = tmem_base + Cfg::TM_S + (qc % NS) * FA_BN;
        for (int half = 0; half < 2; ++half) {
          // an item's first product replaces the accumulator: wait until both halves' warps have read the previous item's
          if (it == 0 && half == 0) ok = warp_wait(&p_full[(qc % NS) * 2 + 1], (qc / NS) & 1);
          if (!ok || !warp_wait(&p_full[(qc % NS) * 2 + half], (qc / NS) & 1)) { if (lane == 0) report_error(p.status, OA_KERR_WAIT_SOFTMAX); ok = false; break; }
          tc_fence_after();
          if (elect_one()) {
#pragma unroll
            for (int ks = 0; ks < 4; ++ks)    // reduction over the 64 queries of this half
              umma_f16_ts(tmem_base + Cfg::TM_DV, a_addr + half * 64 + ks * 8, desc_at(bd, (half * 4 + ks) * 2048),
                          idesc_g, (it > 0 || half > 0 || ks > 0) ? 1u : 0u);
            if (half == 1) {
              umma_commit(&do_empty[st]);
              if (it + 1 == n_it) umma_commit(fin_full);
            }
          }
          __syncwarp();
        }
        if (!ok) break;
        if (NS == 1 && it + 1 < n_it) {
          ok = issue_s(qc + 1, it + 2 == n_it);
          if (lane == 0) mbar_arrive(turn);
        }
      }
      ++itc;
    }
  } else if (warp == 9) {
    // ------------- MMA issuer B: dP^T = V dO^T and dK += dS^T Q.  dP^T of a tile goes over the dS^T that dK has read.
    constexpr uint32_t idesc_s = umma_idesc_bf16(FA_BN, FA_BM, 0, 0);
    constexpr uint32_t idesc_g = umma_idesc_bf16(FA_BN, HD, 0, 1);
    const uint64_t v_desc = desc_k(smem + Cfg::OFF_V), do_desc = desc_k(smem + Cfg::OFF_DO), q_desc = desc_mn(smem + Cfg::OFF_Q);
    const uint32_t dp_tm = tmem_base + Cfg::TM_DP;
    uint32_t itc = 0, qc = 0, turns = 0;
    bool ok = true;
    auto issue_dp = [&](uint32_t n, bool last) -> bool {
      const int st = n % NST;
      if (!warp_wait(&do_full[st], (n / NST) & 1)) { if (lane == 0) report_error(p.status, OA_KERR_WAIT_FULL); return false; }
      tc_fence_after();
      if (elect_one()) {
        const uint64_t dd = desc_at(do_desc, st * Cfg::T_BYTES);
#pragma unroll
        for (int ks = 0; ks < HD / 16; ++ks) {
          const uint32_t off = (ks >> 2) * (FA_BM * 128) + (ks & 3) * 32;
          umma_f16(dp_tm, desc_at(v_desc, off), desc_at(dd, off), idesc_s, ks > 0 ? 1u : 0u);
        }
        umma_commit(dp_full);
        umma_commit(&do_empty[st]);
        if (last) umma_commit(kv_empty);
      }
      __syncwarp();
      return true;
    };
    for (int round = 0; round < n_rounds && ok; ++round) {
      const int item = item_of(round);
      if (item >= n_items) continue;
      int jb, h, b;
      decode(item, jb, h, b);
      const int n_it = nblk - (p.causal ? jb : 0);
      if (!warp_wait(kv_full, itc & 1)) { if (lane == 0) report_error(p.status, OA_KERR_WAIT_FULL); break; }
      ok = issue_dp(qc, n_it == 1);
      for (int it = 0; it < n_it && ok; ++it, ++qc) {
        const int st = qc % NST;
        if (!warp_wait(&q_full[st], (qc / NST) & 1)) { if (lane == 0) report_error(p.status, OA_KERR_WAIT_FULL); ok = false; break; }
        const uint64_t bd = desc_at(q_desc, st * Cfg::T_BYTES);
        if (NS == 1 && it + 1 < n_it) {
          if (!warp_wait(turn, turns & 1)) { if (lane == 0) report_error(p.status, OA_KERR_WAIT_EMPTY); ok = false; break; }
          ++turns;
        }
        for (int half = 0; half < 2; ++half) {
          if (it == 0 && half == 0) ok = warp_wait(&ds_full[1], qc & 1);   // as for dV
          if (!ok || !warp_wait(&ds_full[half], qc & 1)) { if (lane == 0) report_error(p.status, OA_KERR_WAIT_SOFTMAX); ok = false; break; }
          tc_fence_after();
          if (elect_one()) {
#pragma unroll
            for (int ks = 0; ks < 4; ++ks)
              umma_f16_ts(tmem_base + Cfg::TM_DK, dp_tm + half * 64 + ks * 8, desc_at(bd, (half * 4 + ks) * 2048),
                          idesc_g, (it > 0 || half > 0 || ks > 0) ? 1u : 0u);
            if (half == 1) {
              umma_commit(&q_empty[st]);
              if (it + 1 == n_it) umma_commit(fin_full);
            }
          }
          __syncwarp();
        }
        if (!ok) break;
        if (it + 1 < n_it) ok = issue_dp(qc + 1, it + 2 == n_it);
      }
      ++itc;
    }
  } else {
    const int quad = warp & 3;
    const int half = warp >> 2;                  // this thread owns query columns [64*half, 64*half+64) of the tile
    const int r = quad * 32 + lane;              // key row inside the block = TMEM lane
    const uint32_t t_lane = tmem_base + ((uint32_t)(quad * 32) << 16);
    const float sl2 = p.scale * LOG2E, scale = p.scale;
    const unsigned long long sl22 = f2_of(__float_as_uint(sl2), __float_as_uint(sl2)), scale2 = f2_of(__float_as_uint(scale), __float_as_uint(scale));
    uint32_t itc = 0, qc = 0;
    bool ok = true;
    for (int round = 0; round < n_rounds && ok; ++round) {
      const int item = item_of(round);
      if (item >= n_items) continue;
      int jb, h, b;
      decode(item, jb, h, b);
      const int i0 = p.causal ? jb : 0, n_it = nblk - i0, row0 = b * p.seq;
      for (int it = 0; it < n_it; ++it, ++qc) {
        const int st = qc % NST;
        const float* st_cur = stat + st * 256 + half * 64;
        ok = warp_wait(&q_full[st], (qc / NST) & 1);   // statistics of this block are staged
        if (ok) ok = warp_wait(&s_full[qc % NS], (qc / NS) & 1);
        if (!ok) { if (lane == 0) report_error(p.status, OA_KERR_WAIT_TMEM_FULL); break; }
        tc_fence_after();
        const uint32_t s_addr = t_lane + Cfg::TM_S + (qc % NS) * FA_BN + half * 64;
        const uint32_t dp_addr = t_lane + Cfg::TM_DP + half * 64;
        uint32_t s[64];
        tmem_ld32(s_addr, s);
        tmem_ld32(s_addr + 32, s + 32);
        tmem_ld_wait();
        const ulonglong2* nl4 = reinterpret_cast<const ulonglong2*>(st_cur);
        const ulonglong2* nd4 = reinterpret_cast<const ulonglong2*>(st_cur + 128);
        const bool diag = p.causal && it == 0;     // alive iff key <= query: column >= row
        const int first = r - half * 64;           // first alive column of this thread on the diagonal tile
#pragma unroll
        for (int c = 0; c < 2; ++c) {
#pragma unroll
          for (int i = 0; i < 32; i += 4) {
            const ulonglong2 nl = nl4[c * 8 + (i >> 2)];
            uint32_t* sc = s + c * 32 + i;
            bwd_prob2(sc[0], sc[1], sl22, nl.x);
            if ((i >> 2) % 4 < FA_BWD_FMA_PAIRS<HD>) bwd_prob2<true>(sc[2], sc[3], sl22, nl.y);
            else bwd_prob2(sc[2], sc[3], sl22, nl.y);
          }
          if (diag) {
#pragma unroll
            for (int i = 0; i < 32; ++i) s[c * 32 + i] = (c * 32 + i >= first) ? s[c * 32 + i] : 0u;
          }
          bwd_store16(s_addr + c * 16, s + c * 32);
        }
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&p_full[(qc % NS) * 2 + half]);
        ok = warp_wait(dp_full, qc & 1);
        if (!ok) { if (lane == 0) report_error(p.status, OA_KERR_WAIT_TMEM_FULL); break; }
        tc_fence_after();
        uint32_t dp[64];
        tmem_ld32(dp_addr, dp);
        tmem_ld32(dp_addr + 32, dp + 32);
        tmem_ld_wait();
#pragma unroll
        for (int c = 0; c < 2; ++c) {
#pragma unroll
          for (int i = 0; i < 32; i += 4) {
            const ulonglong2 nd = nd4[c * 8 + (i >> 2)];
            uint32_t *sc = s + c * 32 + i, *dc = dp + c * 32 + i;
            bwd_ds2(sc[0], sc[1], dc[0], dc[1], scale2, nd.x);
            bwd_ds2(sc[2], sc[3], dc[2], dc[3], scale2, nd.y);
          }
          bwd_store16(dp_addr + c * 16, s + c * 32);
        }
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&ds_full[half]);
      }
      if (!ok) break;
      ok = warp_wait(fin_full, itc & 1);
      if (!ok) { if (lane == 0) report_error(p.status, OA_KERR_WAIT_TMEM_FULL); break; }
      ++itc;
      tc_fence_after();
      const int k0 = jb * FA_BN + quad * 32;   // accumulator rows are keys
#pragma unroll 1
      for (int which = 0; which < 2; ++which) {
        __nv_bfloat16* base = (which == 0 ? p.dv : p.dk) + (long long)(row0 + k0) * p.dkv_stride + h * HD + half * (HD / 2);
        const uint32_t tcol = t_lane + (which == 0 ? Cfg::TM_DV : Cfg::TM_DK) + half * (HD / 2);
        uint32_t a[HD / 2];
#pragma unroll
        for (int c = 0; c < HD / 64; ++c) tmem_ld32(tcol + c * 32, a + c * 32);
        tmem_ld_wait();
#pragma unroll
        for (int c = 0; c < HD / 64; ++c) store_rows(base + c * 32, p.dkv_stride, p.seq - k0, a + c * 32, 1.f, lane);
      }
      tc_fence_before();   // dV / dK are read before this warp's next p_full / ds_full arrivals let the next item's products overwrite them
    }
  }
  pdl_launch_dependents();
  tc_fence_before();
  __syncthreads();
  if (warp == 8) { tc_fence_after(); tmem_dealloc<Cfg::TMEM_COLS>(tmem_base); }
}

template <int HD>
struct BwdQCfg {
  static constexpr int NK = (HD == 64) ? 4 : 3;        // K ring: a tile is held from its scores to dQ
  static constexpr int NV = (HD == 64) ? 3 : 2;        // V ring: held for dP only
  static constexpr int T_BYTES = FA_BM * HD * 2;
  static constexpr int OFF_Q = 0;
  static constexpr int OFF_DO = OFF_Q + T_BYTES;
  static constexpr int OFF_K = OFF_DO + T_BYTES;
  static constexpr int OFF_V = OFF_K + NK * T_BYTES;
  static constexpr int OFF_BAR = OFF_V + NV * T_BYTES;
  static constexpr int SMEM_BYTES = OFF_BAR + 208;
  static constexpr int TMEM_COLS = 512;
  static constexpr int TM_S = 0, TM_DP = 256, TM_DQ = 384;   // two score buffers; dS over dP
};

// Persistent, like the dK / dV kernel: items are (query block, head, batch), heaviest causal query blocks first; dQ of an item
// accumulates in TMEM over its key blocks.  P is needed in registers only, so a score buffer is free once it has been read.
template <int HD>
__global__ void __launch_bounds__(FA_BWD_THREADS, 1)
flash_bwd_q_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                   const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmDO,
                   const FlashBwdParams p) {
  using Cfg = BwdQCfg<HD>;
  constexpr int NK = Cfg::NK, NV = Cfg::NV;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + Cfg::OFF_BAR);
  uint64_t* q_full = bars + 0;
  uint64_t* q_empty = bars + 1;    // the item's last score and dP products have read Q, dO
  uint64_t* k_full = bars + 2;     // [4]
  uint64_t* k_empty = bars + 6;    // [4]  dQ has read K
  uint64_t* v_full = bars + 10;    // [3]
  uint64_t* v_empty = bars + 13;   // [3]
  uint64_t* s_full = bars + 16;    // [2]
  uint64_t* s_empty = bars + 18;   // [2]  (8 warps)
  uint64_t* dp_full = bars + 20;
  uint64_t* ds_full = bars + 21;   // [2]  by column half (4 warps each)
  uint64_t* fin_full = bars + 23;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 24);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nblk = (p.seq + FA_BM - 1) / FA_BM;
  const int hb = p.heads * p.batch;
  const int n_items = nblk * hb;
  const int n_rounds = (n_items + (int)gridDim.x - 1) / (int)gridDim.x;
  auto item_of = [&](int round) -> int {
    return round * (int)gridDim.x + ((round & 1) ? (int)gridDim.x - 1 - (int)blockIdx.x : (int)blockIdx.x);
  };
  auto decode = [&](int item, int& ib, int& h, int& b) {   // the last query block has the most key blocks under the causal mask
    ib = nblk - 1 - item / hb;
    const int rem = item % hb;
    h = rem % p.heads;
    b = rem / p.heads;
  };

  if ((smem_u32(smem) & 1023u) != 0) {
    if (threadIdx.x == 0) report_error(p.status, OA_KERR_BAD_ARG);
    return;
  }
  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmQ); tma_prefetch_desc(&tmK); tma_prefetch_desc(&tmV); tma_prefetch_desc(&tmDO);
    mbar_init(q_full, 1);
    mbar_init(q_empty, 2);
    for (int s = 0; s < NK; ++s) { mbar_init(&k_full[s], 1); mbar_init(&k_empty[s], 1); }
    for (int s = 0; s < NV; ++s) { mbar_init(&v_full[s], 1); mbar_init(&v_empty[s], 1); }
    for (int s = 0; s < 2; ++s) { mbar_init(&s_full[s], 1); mbar_init(&s_empty[s], 8); mbar_init(&ds_full[s], 4); }
    mbar_init(dp_full, 1);
    mbar_init(fin_full, 1);
    mbar_fence_init();
  }
  if (warp == 8) { tmem_alloc<Cfg::TMEM_COLS>(tmem_slot); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_wait();                            // the prologue above ran under the previous kernel's tail; global memory from here on

  if (warp == 10) {
    uint32_t itc = 0, kc = 0;
    bool ok = true;
    for (int round = 0; round < n_rounds && ok; ++round) {
      const int item = item_of(round);
      if (item >= n_items) continue;
      int ib, h, b;
      decode(item, ib, h, b);
      const int n_kv = p.causal ? (ib + 1) : nblk, row0 = b * p.seq;
      if (!warp_wait(q_empty, (itc & 1) ^ 1)) { if (lane == 0) report_error(p.status, OA_KERR_WAIT_EMPTY); break; }
      if (elect_one()) {
        mbar_expect_tx(q_full, 2 * Cfg::T_BYTES);
#pragma unroll
        for (int x = 0; x < HD / 64; ++x) {
          tma_load_2d(smem + Cfg::OFF_Q + x * (FA_BM * 128), &tmQ, q_full, h * HD + x * 64, row0 + ib * FA_BM);
          tma_load_2d(smem + Cfg::OFF_DO + x * (FA_BM * 128), &tmDO, q_full, h * HD + x * 64, row0 + ib * FA_BM);
        }
      }
      for (int j = 0; j < n_kv; ++j, ++kc) {
        const int sk = kc % NK, sv = kc % NV;
        if (!warp_wait(&k_empty[sk], ((kc / NK) & 1) ^ 1)) { if (lane == 0) report_error(p.status, OA_KERR_WAIT_EMPTY); ok = false; break; }
        if (elect_one()) {
          mbar_expect_tx(&k_full[sk], Cfg::T_BYTES);
#pragma unroll
          for (int x = 0; x < HD / 64; ++x)
            tma_load_2d(smem + Cfg::OFF_K + sk * Cfg::T_BYTES + x * (FA_BN * 128), &tmK, &k_full[sk], h * HD + x * 64, row0 + j * FA_BN);
        }
        if (!warp_wait(&v_empty[sv], ((kc / NV) & 1) ^ 1)) { if (lane == 0) report_error(p.status, OA_KERR_WAIT_EMPTY); ok = false; break; }
        if (elect_one()) {
          mbar_expect_tx(&v_full[sv], Cfg::T_BYTES);
#pragma unroll
          for (int x = 0; x < HD / 64; ++x)
            tma_load_2d(smem + Cfg::OFF_V + sv * Cfg::T_BYTES + x * (FA_BN * 128), &tmV, &v_full[sv], h * HD + x * 64, row0 + j * FA_BN);
        }
        __syncwarp();
      }
      ++itc;
    }
  } else if (warp == 8) {
    // ------------- MMA issuer A: S = Q K_j^T
    constexpr uint32_t idesc_s = umma_idesc_bf16(FA_BM, FA_BN, 0, 0);
    const uint64_t q_desc = desc_k(smem + Cfg::OFF_Q), k_desc = desc_k(smem + Cfg::OFF_K);
    uint32_t itc = 0, kc = 0;
    bool ok = true;
    for (int round = 0; round < n_rounds && ok; ++round) {
      const int item = item_of(round);
      if (item >= n_items) continue;
      int ib, h, b;
      decode(item, ib, h, b);
      const int n_kv = p.causal ? (ib + 1) : nblk;
      if (!warp_wait(q_full, itc & 1)) { if (lane == 0) report_error(p.status, OA_KERR_WAIT_FULL); break; }
      for (int j = 0; j < n_kv; ++j, ++kc) {
        const int st = kc % NK;
        if (!warp_wait(&k_full[st], (kc / NK) & 1)) { if (lane == 0) report_error(p.status, OA_KERR_WAIT_FULL); ok = false; break; }
        if (kc > 1 && !warp_wait(&s_empty[kc & 1], ((kc >> 1) - 1) & 1)) { if (lane == 0) report_error(p.status, OA_KERR_WAIT_TMEM_EMPTY); ok = false; break; }
        tc_fence_after();
        if (elect_one()) {
          const uint64_t kd = desc_at(k_desc, st * Cfg::T_BYTES);
#pragma unroll
          for (int ks = 0; ks < HD / 16; ++ks) {
            const uint32_t off = (ks >> 2) * (FA_BM * 128) + (ks & 3) * 32;
            umma_f16(tmem_base + Cfg::TM_S + (kc & 1) * FA_BN, desc_at(q_desc, off), desc_at(kd, off), idesc_s, ks > 0 ? 1u : 0u);
          }
          umma_commit(&s_full[kc & 1]);
          if (j + 1 == n_kv) umma_commit(q_empty);
        }
        __syncwarp();
      }
      ++itc;
    }
  } else if (warp == 9) {
    // ------------- MMA issuer B: dP = dO V_j^T and dQ += dS K_j (dS from TMEM, over dP)
    constexpr uint32_t idesc_s = umma_idesc_bf16(FA_BM, FA_BN, 0, 0);
    constexpr uint32_t idesc_q = umma_idesc_bf16(FA_BM, HD, 0, 1);   // dQ[q x HD] += dS[q x keys] * K[keys x HD]
    const uint64_t do_desc = desc_k(smem + Cfg::OFF_DO), v_desc = desc_k(smem + Cfg::OFF_V), k_desc = desc_mn(smem + Cfg::OFF_K);
    const uint32_t dp_tm = tmem_base + Cfg::TM_DP;
    uint32_t itc = 0, kc = 0;
    bool ok = true;
    auto issue_dp = [&](uint32_t n, bool last) -> bool {
      const int st = n % NV;
      if (!warp_wait(&v_full[st], (n / NV) & 1)) { if (lane == 0) report_error(p.status, OA_KERR_WAIT_FULL); return false; }
      tc_fence_after();
      if (elect_one()) {
        const uint64_t vd = desc_at(v_desc, st * Cfg::T_BYTES);
#pragma unroll
        for (int ks = 0; ks < HD / 16; ++ks) {
          const uint32_t off = (ks >> 2) * (FA_BM * 128) + (ks & 3) * 32;
          umma_f16(dp_tm, desc_at(do_desc, off), desc_at(vd, off), idesc_s, ks > 0 ? 1u : 0u);
        }
        umma_commit(dp_full);
        umma_commit(&v_empty[st]);
        if (last) umma_commit(q_empty);
      }
      __syncwarp();
      return true;
    };
    for (int round = 0; round < n_rounds && ok; ++round) {
      const int item = item_of(round);
      if (item >= n_items) continue;
      int ib, h, b;
      decode(item, ib, h, b);
      const int n_kv = p.causal ? (ib + 1) : nblk;
      if (!warp_wait(q_full, itc & 1)) { if (lane == 0) report_error(p.status, OA_KERR_WAIT_FULL); break; }
      ok = issue_dp(kc, n_kv == 1);
      for (int j = 0; j < n_kv && ok; ++j, ++kc) {
        const int st = kc % NK;
        if (!warp_wait(&k_full[st], (kc / NK) & 1)) { if (lane == 0) report_error(p.status, OA_KERR_WAIT_FULL); ok = false; break; }
        const uint64_t kd = desc_at(k_desc, st * Cfg::T_BYTES);
        for (int half = 0; half < 2; ++half) {
          // an item's first product replaces the accumulator: wait until both halves' warps have read the previous item's
          if (j == 0 && half == 0) ok = warp_wait(&ds_full[1], kc & 1);
          if (!ok || !warp_wait(&ds_full[half], kc & 1)) { if (lane == 0) report_error(p.status, OA_KERR_WAIT_SOFTMAX); ok = false; break; }
          tc_fence_after();
          if (elect_one()) {
#pragma unroll
            for (int ks = 0; ks < 4; ++ks)
              umma_f16_ts(tmem_base + Cfg::TM_DQ, dp_tm + half * 64 + ks * 8, desc_at(kd, (half * 4 + ks) * 2048),
                          idesc_q, (j > 0 || half > 0 || ks > 0) ? 1u : 0u);
            if (half == 1) {
              umma_commit(&k_empty[st]);
              if (j + 1 == n_kv) umma_commit(fin_full);
            }
          }
          __syncwarp();
        }
        if (!ok) break;
        if (j + 1 < n_kv) ok = issue_dp(kc + 1, j + 2 == n_kv);
      }
      ++itc;
    }
  } else if (warp < 8) {
    const int quad = warp & 3;
    const int half = warp >> 2;
    const int r = quad * 32 + lane;
    const uint32_t t_lane = tmem_base + ((uint32_t)(quad * 32) << 16);
    const float sl2 = p.scale * LOG2E, scale = p.scale;
    const unsigned long long sl22 = f2_of(__float_as_uint(sl2), __float_as_uint(sl2)), scale2 = f2_of(__float_as_uint(scale), __float_as_uint(scale));
    uint32_t itc = 0, kc = 0;
    bool ok = true;
    for (int round = 0; round < n_rounds && ok; ++round) {
      const int item = item_of(round);
      if (item >= n_items) continue;
      int ib, h, b;
      decode(item, ib, h, b);
      const int n_kv = p.causal ? (ib + 1) : nblk, row0 = b * p.seq;
      const long long stat_base = ((long long)b * p.heads + h) * p.seq;
      const int qi = ib * FA_BM + r;
      const bool q_ok = qi < p.seq;
      const float nlse = q_ok ? -p.lse[stat_base + qi] * LOG2E : -INFINITY;
      const float ndlt = q_ok ? -p.delta[stat_base + qi] * scale : 0.f;
      const unsigned long long nlse2 = f2_of(__float_as_uint(nlse), __float_as_uint(nlse)), ndlt2 = f2_of(__float_as_uint(ndlt), __float_as_uint(ndlt));
      for (int j = 0; j < n_kv; ++j, ++kc) {
        ok = warp_wait(&s_full[kc & 1], (kc >> 1) & 1);
        if (!ok) { if (lane == 0) report_error(p.status, OA_KERR_WAIT_TMEM_FULL); break; }
        tc_fence_after();
        const uint32_t s_addr = t_lane + Cfg::TM_S + (kc & 1) * FA_BN + half * 64;
        const uint32_t dp_addr = t_lane + Cfg::TM_DP + half * 64;
        uint32_t s[64];
        tmem_ld32(s_addr, s);
        tmem_ld32(s_addr + 32, s + 32);
        tmem_ld_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&s_empty[kc & 1]);
        const int k0 = j * FA_BN;
        const bool need_mask = (p.causal && j == ib) || (k0 + FA_BN > p.seq) || !q_ok;
#pragma unroll
        for (int i = 0; i < 64; i += 4) {
          bwd_prob2(s[i], s[i + 1], sl22, nlse2);
          if ((i >> 2) % 4 < FA_BWD_FMA_PAIRS<HD>) bwd_prob2<true>(s[i + 2], s[i + 3], sl22, nlse2);
          else bwd_prob2(s[i + 2], s[i + 3], sl22, nlse2);
        }
        if (need_mask) {
          const int lim = q_ok ? (min(p.causal ? qi : 0x7fffffff, p.seq - 1) - (k0 + half * 64)) : -1;
#pragma unroll
          for (int i = 0; i < 64; ++i) s[i] = (i <= lim) ? s[i] : 0u;
        }
        ok = warp_wait(dp_full, kc & 1);
        if (!ok) { if (lane == 0) report_error(p.status, OA_KERR_WAIT_TMEM_FULL); break; }
        tc_fence_after();
        uint32_t dp[64];
        tmem_ld32(dp_addr, dp);
        tmem_ld32(dp_addr + 32, dp + 32);
        tmem_ld_wait();
#pragma unroll
        for (int c = 0; c < 2; ++c) {
#pragma unroll
          for (int i = c * 32; i < c * 32 + 32; i += 2) bwd_ds2(s[i], s[i + 1], dp[i], dp[i + 1], scale2, ndlt2);
          bwd_store16(dp_addr + c * 16, s + c * 32);
        }
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&ds_full[half]);
      }
      if (!ok) break;
      ok = warp_wait(fin_full, itc & 1);
      if (!ok) { if (lane == 0) report_error(p.status, OA_KERR_WAIT_TMEM_FULL); break; }
      ++itc;
      tc_fence_after();
      const int q0 = ib * FA_BM + quad * 32;
      __nv_bfloat16* base = p.dq + (long long)(row0 + q0) * p.dq_stride + h * HD + half * (HD / 2);
      uint32_t a[HD / 2];
#pragma unroll
      for (int c = 0; c < HD / 64; ++c) tmem_ld32(t_lane + Cfg::TM_DQ + half * (HD / 2) + c * 32, a + c * 32);
      tmem_ld_wait();
#pragma unroll
      for (int c = 0; c < HD / 64; ++c) store_rows(base + c * 32, p.dq_stride, p.seq - q0, a + c * 32, 1.f, lane);
      tc_fence_before();   // dQ is read before this warp's next ds_full arrival lets the next item's products overwrite it
    }
  }
  pdl_launch_dependents();
  tc_fence_before();
  __syncthreads();
  if (warp == 8) { tc_fence_after(); tmem_dealloc<Cfg::TMEM_COLS>(tmem_base); }
}

int make_tmap_2d_bf16(CUtensorMap* out, const void* ptr, uint64_t inner, uint64_t outer, uint64_t ld,
                      uint32_t box_inner, uint32_t box_outer);

}  // namespace oa

using namespace oa;

extern "C" int oa_flash_fwd(const void* q, const void* k, const void* v, void* o, float* lse, int batch, int heads,
                            int seq, int head_dim, long long q_row_stride, long long kv_row_stride,
                            long long o_row_stride, float scale, int causal, int* status, void* stream) {
  if (head_dim != 64 && head_dim != 128) return OA_ERR_UNSUPPORTED;
  if (batch <= 0 || heads <= 0 || seq <= 0) return OA_ERR_ARG;
  if ((o_row_stride & 7) || (reinterpret_cast<uintptr_t>(o) & 15)) return OA_ERR_ALIGN;
  CUtensorMap tq, tk, tv;
  int rc;
  uint64_t rows = (uint64_t)batch * seq, width = (uint64_t)heads * head_dim;
  if ((rc = make_tmap_2d_bf16(&tq, q, width, rows, (uint64_t)q_row_stride, 64, FA_BM))) return rc;
  if ((rc = make_tmap_2d_bf16(&tk, k, width, rows, (uint64_t)kv_row_stride, 64, FA_BN))) return rc;
  if ((rc = make_tmap_2d_bf16(&tv, v, width, rows, (uint64_t)kv_row_stride, 64, FA_BN))) return rc;
  FlashParams p;
  p.batch = batch; p.heads = heads; p.seq = seq; p.head_dim = head_dim; p.scale = scale; p.causal = causal;
  p.o = (__nv_bfloat16*)o; p.o_stride = o_row_stride; p.lse = lse; p.status = status;
  cudaStream_t st = (cudaStream_t)stream;
  return head_dim == 64 ? launch_fwd_pair<64>(tq, tk, tv, p, st) : launch_fwd_pair<128>(tq, tk, tv, p, st);
}

// scratch: float[B*H*S] for delta
extern "C" size_t oa_flash_bwd_scratch_bytes(int batch, int heads, int seq, int head_dim) {
  (void)head_dim;
  return (size_t)batch * heads * seq * sizeof(float);
}

template <typename K>
static int set_max_smem(K kernel, int bytes) {
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) == cudaSuccess ? OA_OK : OA_ERR_LAUNCH;
}

extern "C" int oa_flash_bwd(const void* q, const void* k, const void* v, const void* o, const void* dout,
                            const float* lse, void* dq, void* dk, void* dv, int batch, int heads, int seq, int head_dim,
                            long long q_row_stride, long long kv_row_stride, long long o_row_stride,
                            long long dq_row_stride, long long dkv_row_stride, float scale, int causal, float* scratch,
                            int* status, void* stream) {
  if (head_dim != 64 && head_dim != 128) return OA_ERR_UNSUPPORTED;
  if (batch <= 0 || heads <= 0 || seq <= 0) return OA_ERR_ARG;
  if ((dq_row_stride & 7) || (dkv_row_stride & 7) || (reinterpret_cast<uintptr_t>(dq) & 15) ||
      (reinterpret_cast<uintptr_t>(dk) & 15) || (reinterpret_cast<uintptr_t>(dv) & 15))
    return OA_ERR_ALIGN;
  cudaStream_t st = (cudaStream_t)stream;
  CUtensorMap tq, tk, tv, tdo;
  int rc;
  uint64_t rows = (uint64_t)batch * seq, width = (uint64_t)heads * head_dim;
  if ((rc = make_tmap_2d_bf16(&tq, q, width, rows, (uint64_t)q_row_stride, 64, FA_BM))) return rc;
  if ((rc = make_tmap_2d_bf16(&tk, k, width, rows, (uint64_t)kv_row_stride, 64, FA_BN))) return rc;
  if ((rc = make_tmap_2d_bf16(&tv, v, width, rows, (uint64_t)kv_row_stride, 64, FA_BN))) return rc;
  if ((rc = make_tmap_2d_bf16(&tdo, dout, width, rows, (uint64_t)o_row_stride, 64, FA_BM))) return rc;
  {
    long long threads = (long long)batch * seq * heads * (head_dim / 8);
    unsigned blocks = (unsigned)((threads + 255) / 256);
    launch_pdl(flash_delta_kernel, dim3(blocks), dim3(256), 0, st, (const __nv_bfloat16*)o, (const __nv_bfloat16*)dout, scratch, batch, heads,
               seq, head_dim, o_row_stride, o_row_stride);
  }
  FlashBwdParams p;
  p.batch = batch; p.heads = heads; p.seq = seq; p.head_dim = head_dim; p.scale = scale; p.causal = causal;
  p.lse = lse; p.delta = scratch;
  p.dq = (__nv_bfloat16*)dq; p.dq_stride = dq_row_stride;
  p.dk = (__nv_bfloat16*)dk; p.dv = (__nv_bfloat16*)dv; p.dkv_stride = dkv_row_stride;
  p.status = status;
  static int sms = 0;
  if (sms == 0) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return OA_ERR_DRIVER;
  }
  const long long items = (long long)((seq + FA_BM - 1) / FA_BM) * heads * batch;
  const dim3 grid((unsigned)(items < sms ? items : sms));     // persistent: one CTA per SM walks its items
  if (head_dim == 64) {
    static bool set = false;
    if (!set) {
      if ((rc = set_max_smem(flash_bwd_kv_kernel<64>, BwdKvCfg<64>::SMEM_BYTES))) return rc;
      if ((rc = set_max_smem(flash_bwd_q_kernel<64>, BwdQCfg<64>::SMEM_BYTES))) return rc;
      set = true;
    }
    launch_pdl(flash_bwd_kv_kernel<64>, dim3(grid), dim3(FA_BWD_THREADS), BwdKvCfg<64>::SMEM_BYTES, st, tq, tk, tv, tdo, p);
    launch_pdl(flash_bwd_q_kernel<64>, dim3(grid), dim3(FA_BWD_THREADS), BwdQCfg<64>::SMEM_BYTES, st, tq, tk, tv, tdo, p);
  } else {
    static bool set = false;
    if (!set) {
      if ((rc = set_max_smem(flash_bwd_kv_kernel<128>, BwdKvCfg<128>::SMEM_BYTES))) return rc;
      if ((rc = set_max_smem(flash_bwd_q_kernel<128>, BwdQCfg<128>::SMEM_BYTES))) return rc;
      set = true;
    }
    launch_pdl(flash_bwd_kv_kernel<128>, dim3(grid), dim3(FA_BWD_THREADS), BwdKvCfg<128>::SMEM_BYTES, st, tq, tk, tv, tdo, p);
    launch_pdl(flash_bwd_q_kernel<128>, dim3(grid), dim3(FA_BWD_THREADS), BwdQCfg<128>::SMEM_BYTES, st, tq, tk, tv, tdo, p);
  }
  return cudaGetLastError() == cudaSuccess ? OA_OK : OA_ERR_LAUNCH;
}
