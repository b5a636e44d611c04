// Whole-sequence GRU / RNN recurrent scans, forward and backward, one launch per layer.
//
// Contracts (Source/Private/Oa/Ml/Shader/Compute/Nn/Gru/GruScan.slang:8-15,73-86, Nn/Rnn/RnnScan.slang:8-12):
//   GRU:  r = sigmoid(i_r + h_r); z = sigmoid(i_z + h_z); n = tanh(i_n + r * h_n); h' = (1 - z) * n + z * h
//         with [h_r | h_z | h_n] = W_hh h + b_hh, gate order reset | update | candidate, h(0) = 0
//   RNN:  h' = tanh(i + W_hh h + b_hh)
// The input projection i = W_ih x + b_ih for all time steps is one GEMM done by the caller; only the serial part
// runs here.  The reference runs one work-group per batch element with h in shared memory.  Hidden widths up to 128 that
// are multiples of 8 (rnn_reg_ok) do likewise, with W_hh in registers for the whole sequence (rnn_reg_*_kernel, further
// down); for other widths (rnn_scan_*_kernel) a CTA owns a tile of BT batch rows so that every W_hh row fetched from L2 /
// shared memory is reused BT times, and h and the gate pre-activations live in shared memory.  Math is fp32.  The backward pass walks time in reverse from the saved
// h(t-1), emits the gate gradients dGi (for the input projection) and dGh; the weight gradient
// dW_hh = dGh^T Hprev and db_hh are then ordinary (tensor-core) GEMM / column-sum calls.
#include "common.cuh"
#include "api.h"

namespace oa {

template <typename T> __device__ __forceinline__ float rld(const T* p);
template <> __device__ __forceinline__ float rld<float>(const float* p) { return *p; }
template <> __device__ __forceinline__ float rld<__nv_bfloat16>(const __nv_bfloat16* p) { return __bfloat162float(*p); }
template <typename T> __device__ __forceinline__ void rst(T* p, float v);
template <> __device__ __forceinline__ void rst<float>(float* p, float v) { *p = v; }
template <> __device__ __forceinline__ void rst<__nv_bfloat16>(__nv_bfloat16* p, float v) { *p = __float2bfloat16_rn(v); }

constexpr int RNN_BT = 4;        // batch rows per CTA
constexpr int RNN_THREADS = 256;

// G = number of gates (3 = GRU, 1 = RNN).  Shared: h[BT][H], gh[BT][G*H].
template <typename T, int G>
__global__ void __launch_bounds__(RNN_THREADS)
rnn_scan_fwd_kernel(const T* __restrict__ gates_i, const T* __restrict__ w_hh, const T* __restrict__ b_hh, const T* __restrict__ h0,
                    T* __restrict__ out, T* __restrict__ hprev, int batch, int seq, int H) {
  extern __shared__ float sm[];
  float* sh = sm;                       // [BT][H]
  float* sg = sm + RNN_BT * H;          // [BT][G*H]
  const int b0 = blockIdx.x * RNN_BT;
  const int nb = min(RNN_BT, batch - b0);
  for (int i = threadIdx.x; i < RNN_BT * H; i += blockDim.x) {
    int bb = i / H, j = i % H;
    sh[i] = (h0 && bb < nb) ? rld<T>(h0 + (long long)(b0 + bb) * H + j) : 0.f;
  }
  __syncthreads();
  for (int t = 0; t < seq; ++t) {
    // recurrent projection: gh[b][j] = b_hh[j] + sum_k W_hh[j][k] * h[b][k]
    for (int j = threadIdx.x; j < G * H; j += blockDim.x) {
      float acc[RNN_BT];
      const float bj = b_hh ? rld<T>(b_hh + j) : 0.f;
#pragma unroll
      for (int bb = 0; bb < RNN_BT; ++bb) acc[bb] = bj;
      const T* wr = w_hh + (long long)j * H;
      for (int k = 0; k < H; ++k) {
        const float w = rld<T>(wr + k);
#pragma unroll
        for (int bb = 0; bb < RNN_BT; ++bb) acc[bb] = fmaf(w, sh[bb * H + k], acc[bb]);
      }
#pragma unroll
      for (int bb = 0; bb < RNN_BT; ++bb) sg[bb * G * H + j] = acc[bb];
    }
    __syncthreads();
    for (int i = threadIdx.x; i < nb * H; i += blockDim.x) {
      const int bb = i / H, j = i % H;
      const long long row = ((long long)(b0 + bb) * seq + t);
      const T* gi = gates_i + row * G * H;
      const float hp = sh[bb * H + j];
      float hn;
      if (G == 3) {
        const float r = sigmoid_f(rld<T>(gi + j) + sg[bb * 3 * H + j]);
        const float z = sigmoid_f(rld<T>(gi + H + j) + sg[bb * 3 * H + H + j]);
        const float n = tanhf(rld<T>(gi + 2 * H + j) + r * sg[bb * 3 * H + 2 * H + j]);
        hn = (1.f - z) * n + z * hp;
      } else {
        hn = tanhf(rld<T>(gi + j) + sg[bb * H + j]);
      }
      if (hprev) rst<T>(hprev + row * H + j, hp);
      rst<T>(out + row * H + j, hn);
      sh[bb * H + j] = hn;
    }
    __syncthreads();
  }
}

// Shared: h[BT][H] (saved h(t-1)), gh[BT][G*H], dh[BT][H] (running gradient), dgh[BT][G*H].
template <typename T, int G>
__global__ void __launch_bounds__(RNN_THREADS)
rnn_scan_bwd_kernel(const T* __restrict__ gates_i, const T* __restrict__ w_hh, const T* __restrict__ b_hh,
                    const T* __restrict__ hprev, const T* __restrict__ dout, T* __restrict__ dgi, T* __restrict__ dgh,
                    T* __restrict__ dh0, int batch, int seq, int H) {
  extern __shared__ float sm[];
  float* sh = sm;
  float* sg = sh + RNN_BT * H;
  float* sdh = sg + RNN_BT * G * H;
  float* sdg = sdh + RNN_BT * H;
  const int b0 = blockIdx.x * RNN_BT;
  const int nb = min(RNN_BT, batch - b0);
  for (int i = threadIdx.x; i < RNN_BT * H; i += blockDim.x) sdh[i] = 0.f;
  for (int i = threadIdx.x; i < RNN_BT * G * H; i += blockDim.x) sdg[i] = 0.f;
  __syncthreads();
  for (int t = seq - 1; t >= 0; --t) {
    for (int i = threadIdx.x; i < RNN_BT * H; i += blockDim.x) {
      int bb = i / H, j = i % H;
      sh[i] = bb < nb ? rld<T>(hprev + ((long long)(b0 + bb) * seq + t) * H + j) : 0.f;
    }
    __syncthreads();
    for (int j = threadIdx.x; j < G * H; j += blockDim.x) {
      float acc[RNN_BT];
      const float bj = b_hh ? rld<T>(b_hh + j) : 0.f;
#pragma unroll
      for (int bb = 0; bb < RNN_BT; ++bb) acc[bb] = bj;
      const T* wr = w_hh + (long long)j * H;
      for (int k = 0; k < H; ++k) {
        const float w = rld<T>(wr + k);
#pragma unroll
        for (int bb = 0; bb < RNN_BT; ++bb) acc[bb] = fmaf(w, sh[bb * H + k], acc[bb]);
      }
#pragma unroll
      for (int bb = 0; bb < RNN_BT; ++bb) sg[bb * G * H + j] = acc[bb];
    }
    __syncthreads();
    // pointwise backward; dh_total = dout[t] + carried dh
    for (int i = threadIdx.x; i < nb * H; i += blockDim.x) {
      const int bb = i / H, j = i % H;
      const long long row = ((long long)(b0 + bb) * seq + t);
      const T* gi = gates_i + row * G * H;
      const float hp = sh[bb * H + j];
      const float d = rld<T>(dout + row * H + j) + sdh[bb * H + j];
      if (G == 3) {
        const float hr = sg[bb * 3 * H + j], hz = sg[bb * 3 * H + H + j], hn_ = sg[bb * 3 * H + 2 * H + j];
        const float r = sigmoid_f(rld<T>(gi + j) + hr);
        const float z = sigmoid_f(rld<T>(gi + H + j) + hz);
        const float n = tanhf(rld<T>(gi + 2 * H + j) + r * hn_);
        const float dn = d * (1.f - z);
        const float dz = d * (hp - n);
        const float dn_pre = dn * (1.f - n * n);
        const float dr = dn_pre * hn_;
        const float dr_pre = dr * r * (1.f - r);
        const float dz_pre = dz * z * (1.f - z);
        rst<T>(dgi + row * 3 * H + j, dr_pre);
        rst<T>(dgi + row * 3 * H + H + j, dz_pre);
        rst<T>(dgi + row * 3 * H + 2 * H + j, dn_pre);
        const float dhn = dn_pre * r;
        rst<T>(dgh + row * 3 * H + j, dr_pre);
        rst<T>(dgh + row * 3 * H + H + j, dz_pre);
        rst<T>(dgh + row * 3 * H + 2 * H + j, dhn);
        sdg[bb * 3 * H + j] = dr_pre; sdg[bb * 3 * H + H + j] = dz_pre; sdg[bb * 3 * H + 2 * H + j] = dhn;
        sdh[bb * H + j] = d * z;          // direct path h -> h'
      } else {
        const float hn = tanhf(rld<T>(gi + j) + sg[bb * H + j]);
        const float dpre = d * (1.f - hn * hn);
        rst<T>(dgi + row * H + j, dpre);
        rst<T>(dgh + row * H + j, dpre);
        sdg[bb * H + j] = dpre;
        sdh[bb * H + j] = 0.f;
      }
    }
    __syncthreads();
    // dh(t-1) += W_hh^T dgh
    for (int k = threadIdx.x; k < H; k += blockDim.x) {
      float acc[RNN_BT];
#pragma unroll
      for (int bb = 0; bb < RNN_BT; ++bb) acc[bb] = 0.f;
      for (int j = 0; j < G * H; ++j) {
        const float w = rld<T>(w_hh + (long long)j * H + k);
#pragma unroll
        for (int bb = 0; bb < RNN_BT; ++bb) acc[bb] = fmaf(w, sdg[bb * G * H + j], acc[bb]);
      }
#pragma unroll
      for (int bb = 0; bb < RNN_BT; ++bb) sdh[bb * H + k] += acc[bb];
    }
    __syncthreads();
  }
  if (dh0)
    for (int i = threadIdx.x; i < nb * H; i += blockDim.x) rst<T>(dh0 + (long long)(b0 + i / H) * H + i % H, sdh[(i / H) * H + i % H]);
}

// ------------------------------------------------------------------------------------------------ hidden width up to 128
// The recurrent weights stay in registers for the whole sequence: the kernels above fetch W_hh again in every time step, and that
// fetch is what the step waits for.  One CTA owns one sequence; four neighbouring lanes own one hidden unit and a quarter of
// its reduction each (interleaved 16-byte pieces, so the shared-memory reads of a warp are broadcasts without conflicts), the
// quarters meet in two shuffles and a step costs one block barrier.  Products are packed pairs (fma.rn.f32x2).
// NM: 16-wide pieces of the hidden width, G * NM * 4 weights per thread.
// What bounds it: the serial chain of a step (dot product, two shuffles, activations, one barrier), about 1 us.  A GRU layer of
// 128 units over 64 sequences of 128 steps, forward and backward with its products: 13.7 ms before, 0.51 ms now (scans 127 us
// and 151 us, coefficients 74 us).  The line lies at 128 units because the weights of a thread are 96 registers there; wider
// layers take the kernels above.
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ unsigned long long pack2(float lo, float hi) {
  unsigned long long d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
  return d;
}
__device__ __forceinline__ float sum2(unsigned long long a) {
  float lo, hi;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(a));
  return lo + hi;
}
__device__ __forceinline__ float quad_sum(float v) {
  v += __shfl_xor_sync(0xffffffffu, v, 1);
  return v + __shfl_xor_sync(0xffffffffu, v, 2);
}

// this lane's quarter of sum_k w[k] h[k] for G rows; h is zero beyond the hidden width
template <int G, int NM>
__device__ __forceinline__ void quad_dot(const unsigned long long (&w)[G][NM][2], const float* h, int p, float (&out)[G]) {
  unsigned long long acc[G][2];
#pragma unroll
  for (int g = 0; g < G; ++g) acc[g][0] = acc[g][1] = 0ull;
#pragma unroll
  for (int m = 0; m < NM; ++m) {
    const ulonglong2 hv = *reinterpret_cast<const ulonglong2*>(h + 4 * (p + 4 * m));
#pragma unroll
    for (int g = 0; g < G; ++g) {
      acc[g][0] = fma2(w[g][m][0], hv.x, acc[g][0]);
      acc[g][1] = fma2(w[g][m][1], hv.y, acc[g][1]);
    }
  }
#pragma unroll
  for (int g = 0; g < G; ++g) out[g] = quad_sum(sum2(acc[g][0]) + sum2(acc[g][1]));
}

// w[g][m] = the lane's pieces of row g * H + i of W_hh (by_row) or of the columns i of gate g (W_hh^T)
template <typename T, int G, int NM>
__device__ __forceinline__ void quad_load(unsigned long long (&w)[G][NM][2], const T* __restrict__ w_hh, int i, int p, int H, bool by_row) {
#pragma unroll
  for (int g = 0; g < G; ++g)
#pragma unroll
    for (int m = 0; m < NM; ++m) {
      float v[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int k = 4 * (p + 4 * m) + c;
        v[c] = k < H ? (by_row ? rld<T>(w_hh + (long long)(g * H + i) * H + k) : rld<T>(w_hh + (long long)(g * H + k) * H + i)) : 0.f;
      }
      w[g][m][0] = pack2(v[0], v[1]);
      w[g][m][1] = pack2(v[2], v[3]);
    }
}

template <typename T, int G, int NM>
__global__ void __launch_bounds__(64 * NM, 1)
rnn_reg_fwd_kernel(const T* __restrict__ gates_i, const T* __restrict__ w_hh, const T* __restrict__ b_hh, const T* __restrict__ h0,
                   T* __restrict__ out, T* __restrict__ hprev, int seq, int H) {
  __shared__ __align__(16) float sh[2][16 * NM];
  const int i = threadIdx.x >> 2, p = threadIdx.x & 3, b = blockIdx.x;
  unsigned long long w[G][NM][2];
  quad_load<T, G, NM>(w, w_hh, i, p, H, true);
  float bias[G];
#pragma unroll
  for (int g = 0; g < G; ++g) bias[g] = b_hh ? rld<T>(b_hh + g * H + i) : 0.f;
  float hp = h0 ? rld<T>(h0 + (long long)b * H + i) : 0.f;
  for (int k = threadIdx.x; k < 16 * NM; k += blockDim.x) sh[0][k] = sh[1][k] = 0.f;
  __syncthreads();
  if (p == 0) sh[0][i] = hp;
  __syncthreads();
  constexpr int PF = 4;                                       // input gates are fetched four steps ahead, lane p brings gate p
  const T* gi = gates_i + (long long)b * seq * G * H + (p < G ? p : 0) * H + i;
  float pf[PF];
#pragma unroll
  for (int u = 0; u < PF; ++u) pf[u] = u < seq ? rld<T>(gi + (long long)u * G * H) : 0.f;
  const int q0 = threadIdx.x & 28;                            // first lane of the quad
  for (int t0 = 0; t0 < seq; t0 += PF) {
#pragma unroll
    for (int u = 0; u < PF; ++u) {
      const int t = t0 + u;
      if (t >= seq) break;
      float gh[G], x[G];
      quad_dot<G, NM>(w, sh[u & 1], p, gh);
      const float mine = pf[u];
      if (t + PF < seq) pf[u] = rld<T>(gi + (long long)(t + PF) * G * H);
#pragma unroll
      for (int g = 0; g < G; ++g) { x[g] = __shfl_sync(0xffffffffu, mine, q0 + g); gh[g] += bias[g]; }
      float hn;
      if constexpr (G == 3) {
        const float r = sigmoid_f(x[0] + gh[0]), z = sigmoid_f(x[1] + gh[1]), n = tanhf(x[2] + r * gh[2]);
        hn = (1.f - z) * n + z * hp;
      } else {
        hn = tanhf(x[0] + gh[0]);
      }
      const long long row = (long long)b * seq + t;
      if (p == 0) sh[(u & 1) ^ 1][i] = hn;
      if (p == 1) rst<T>(out + row * H + i, hn);
      if (p == 2 && hprev) rst<T>(hprev + row * H + i, hp);
      hp = hn;
      __syncthreads();
    }
  }
}

// Everything of the backward step that does not depend on the running gradient, for all time steps at once.  The gate
// gradients are the running gradient d times coef[row][i] = {c_r, c_z, c_n r, c_n} (RNN: {1 - h'^2}), and zg[row][i] = z is the
// direct path h -> h'.
template <typename T, int G, int NM>
__global__ void __launch_bounds__(64 * NM, 1)
rnn_reg_coef_kernel(const T* __restrict__ gates_i, const T* __restrict__ w_hh, const T* __restrict__ b_hh, const T* __restrict__ hprev,
                    float* __restrict__ coef, float* __restrict__ zg, long long rows, int H) {
  __shared__ __align__(16) float sh[2][16 * NM];
  const int i = threadIdx.x >> 2, p = threadIdx.x & 3;
  unsigned long long w[G][NM][2];
  quad_load<T, G, NM>(w, w_hh, i, p, H, true);
  float bias[G];
#pragma unroll
  for (int g = 0; g < G; ++g) bias[g] = b_hh ? rld<T>(b_hh + g * H + i) : 0.f;
  for (int k = threadIdx.x; k < 16 * NM; k += blockDim.x) sh[0][k] = sh[1][k] = 0.f;
  __syncthreads();
  float hp = blockIdx.x < rows ? rld<T>(hprev + (long long)blockIdx.x * H + i) : 0.f;
  int buf = 0;
  for (long long row = blockIdx.x; row < rows; row += gridDim.x, buf ^= 1) {
    if (p == 0) sh[buf][i] = hp;
    const float h_in = hp;
    if (row + gridDim.x < rows) hp = rld<T>(hprev + (row + gridDim.x) * H + i);
    float x[G], gh[G];
#pragma unroll
    for (int g = 0; g < G; ++g) x[g] = rld<T>(gates_i + (row * G + g) * H + i);
    __syncthreads();                                          // two buffers: the previous row's readers are past this row's writes
    quad_dot<G, NM>(w, sh[buf], p, gh);
#pragma unroll
    for (int g = 0; g < G; ++g) gh[g] += bias[g];
    if constexpr (G == 3) {
      const float r = sigmoid_f(x[0] + gh[0]), z = sigmoid_f(x[1] + gh[1]), n = tanhf(x[2] + r * gh[2]);
      const float cn = (1.f - z) * (1.f - n * n);
      const float v = p == 0 ? cn * gh[2] * r * (1.f - r) : p == 1 ? (h_in - n) * z * (1.f - z) : p == 2 ? cn * r : cn;
      coef[(row * H + i) * 4 + p] = v;
      if (p == 0) zg[row * H + i] = z;
    } else {
      const float hn = tanhf(x[0] + gh[0]);
      if (p == 0) coef[row * H + i] = 1.f - hn * hn;
    }
  }
}

template <typename T, int G, int NM>
__global__ void __launch_bounds__(64 * NM, 1)
rnn_reg_bwd_kernel(const float* __restrict__ coef, const float* __restrict__ zg, const T* __restrict__ w_hh, const T* __restrict__ dout,
                   T* __restrict__ dgi, T* __restrict__ dgh, T* __restrict__ dh0, int seq, int H) {
  __shared__ __align__(16) float sg[2][G][16 * NM];
  const int i = threadIdx.x >> 2, p = threadIdx.x & 3, b = blockIdx.x;
  unsigned long long w[G][NM][2];
  quad_load<T, G, NM>(w, w_hh, i, p, H, false);
  for (int k = threadIdx.x; k < 2 * G * 16 * NM; k += blockDim.x) (&sg[0][0][0])[k] = 0.f;
  __syncthreads();
  constexpr int PF = 2, CW = G == 3 ? 4 : 1;
  const long long row0 = (long long)b * seq;
  float cf[PF], zf[PF], df[PF];
  auto fetch = [&](int t, float& c, float& z, float& d) {
    const long long row = row0 + t;
    c = coef[(row * H + i) * CW + (G == 3 ? p : 0)];
    z = G == 3 ? zg[row * H + i] : 0.f;
    d = rld<T>(dout + row * H + i);
  };
#pragma unroll
  for (int u = 0; u < PF; ++u)
    if (seq - 1 - u >= 0) fetch(seq - 1 - u, cf[u], zf[u], df[u]);
  float carry = 0.f;
  for (int t0 = seq - 1; t0 >= 0; t0 -= PF) {
#pragma unroll
    for (int u = 0; u < PF; ++u) {
      const int t = t0 - u;
      if (t < 0) break;
      const float d = df[u] + carry, g = d * cf[u], direct = d * zf[u];
      if (t - PF >= 0) fetch(t - PF, cf[u], zf[u], df[u]);
      const long long row = row0 + t;
      if constexpr (G == 3) {
        if (p < 3) sg[u & 1][p][i] = g;
        if (p != 3) rst<T>(dgh + (row * 3 + p) * H + i, g);
        if (p != 2) rst<T>(dgi + (row * 3 + (p == 3 ? 2 : p)) * H + i, g);
      } else {
        if (p == 0) { sg[u & 1][0][i] = g; rst<T>(dgi + row * H + i, g); }
        if (p == 1) rst<T>(dgh + row * H + i, g);
      }
      __syncthreads();
      // W_hh^T dgh: this lane's quarter of every gate's rows
      unsigned long long acc[2] = {0ull, 0ull};
#pragma unroll
      for (int gg = 0; gg < G; ++gg)
#pragma unroll
        for (int m = 0; m < NM; ++m) {
          const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(&sg[u & 1][gg][4 * (p + 4 * m)]);
          acc[0] = fma2(w[gg][m][0], v.x, acc[0]);
          acc[1] = fma2(w[gg][m][1], v.y, acc[1]);
        }
      carry = direct + quad_sum(sum2(acc[0]) + sum2(acc[1]));
    }
  }
  if (dh0 && p == 0) rst<T>(dh0 + (long long)b * H + i, carry);
}

// GRU layers of 80, 96, 112 and 128 units: four lanes own TWO units, which halves the warps, and with them the passes through
// the activations that all lanes of a quad make together, and the shared-memory reads per product.  After a reduce-scatter over the
// quad two lanes hold each unit.  A thread's weights are 192 registers.  Whole warps need multiples of 16 units; up to 64 units and at
// 72, 88, 104 and 120 the kernels above stay.
// 64 sequences of 128 steps, 128 units, fp32: forward 129 -> 85 us, backward with the coefficients of rnn_reg_coef_kernel 228 -> 162.
// Forward at 80 units 109 -> 80, 96: 113 -> 81, 112: 124 -> 83, in bf16 125 -> 93, 129 -> 95, 140 -> 95; one sequence alike, 600 sequences
// of 64 steps 273 -> 201 at 80 units.  The products are padded to 128 columns: instantiations by 16 measured 68 us at 80, 74 at 96.
// A forward scan may also write those coefficients, by-products of its step (+ 2 us), instead of leaving the coefficient kernel to
// run the recurrent products of all steps again: backward 162 -> 87.  They are five fp32 values per unit and step that live from the
// forward to the backward pass, beside the 20 bytes (fp32) or 10 (bf16) that a layer keeps there anyway, so the caller bounds them.
constexpr int GRU2_NM = 8;
template <typename T>
__device__ __forceinline__ void gru2_load(unsigned long long (&w)[2][3][GRU2_NM][2], const T* __restrict__ w_hh, int i0, int p, int H, bool by_row) {
#pragma unroll
  for (int u = 0; u < 2; ++u)
#pragma unroll
    for (int g = 0; g < 3; ++g)
#pragma unroll
      for (int m = 0; m < GRU2_NM; ++m) {
        float v[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const int k = 4 * (p + 4 * m) + c;
          v[c] = k < H ? (by_row ? rld<T>(w_hh + (long long)(g * H + i0 + u) * H + k) : rld<T>(w_hh + (long long)(g * H + k) * H + i0 + u)) : 0.f;
        }
        w[u][g][m][0] = pack2(v[0], v[1]);
        w[u][g][m][1] = pack2(v[2], v[3]);
      }
}
// the quad's sum of each of two units; lanes 0, 1 get the first one's, lanes 2, 3 the second one's
__device__ __forceinline__ float gru2_sum(float a, float b, int p) {
  const float mine = p & 2 ? b : a, theirs = p & 2 ? a : b;
  const float v = mine + __shfl_xor_sync(0xffffffffu, theirs, 2);
  return v + __shfl_xor_sync(0xffffffffu, v, 1);
}

template <typename T>
__global__ void __launch_bounds__(256, 1)
gru2_fwd_kernel(const T* __restrict__ gates_i, const T* __restrict__ w_hh, const T* __restrict__ b_hh, const T* __restrict__ h0, T* __restrict__ out,
                T* __restrict__ hprev, float* __restrict__ coef, float* __restrict__ zg, int seq, int H) {
  __shared__ __align__(16) float sh[2][16 * GRU2_NM];
  const int p = threadIdx.x & 3, q = p & 1, i0 = (threadIdx.x >> 2) * 2, i = i0 + (p >> 1), b = blockIdx.x;
  unsigned long long w[2][3][GRU2_NM][2];
  gru2_load<T>(w, w_hh, i0, p, H, true);
  float bias[3];
#pragma unroll
  for (int g = 0; g < 3; ++g) bias[g] = b_hh ? rld<T>(b_hh + g * H + i) : 0.f;
  float hp = h0 ? rld<T>(h0 + (long long)b * H + i) : 0.f;
  for (int k = threadIdx.x; k < 16 * GRU2_NM; k += blockDim.x) sh[0][k] = sh[1][k] = 0.f;
  __syncthreads();
  if (q == 0) sh[0][i] = hp;
  __syncthreads();
  constexpr int PF = 2;                                       // input gates are fetched two steps ahead
  const T* gi = gates_i + (long long)b * seq * 3 * H + i;
  float pf[PF][3];
#pragma unroll
  for (int u = 0; u < PF; ++u)
#pragma unroll
    for (int g = 0; g < 3; ++g) pf[u][g] = u < seq ? rld<T>(gi + ((long long)u * 3 + g) * H) : 0.f;
  for (int t0 = 0; t0 < seq; t0 += PF) {
#pragma unroll
    for (int u = 0; u < PF; ++u) {
      const int t = t0 + u;
      if (t >= seq) break;
      unsigned long long acc[2][3] = {};
#pragma unroll
      for (int m = 0; m < GRU2_NM; ++m) {
        const ulonglong2 hv = *reinterpret_cast<const ulonglong2*>(&sh[u & 1][4 * (p + 4 * m)]);
#pragma unroll
        for (int v = 0; v < 2; ++v)
#pragma unroll
          for (int g = 0; g < 3; ++g) acc[v][g] = fma2(w[v][g][m][1], hv.y, fma2(w[v][g][m][0], hv.x, acc[v][g]));
      }
      float x[3], gh[3];
#pragma unroll
      for (int g = 0; g < 3; ++g) {
        x[g] = pf[u][g];
        if (t + PF < seq) pf[u][g] = rld<T>(gi + ((long long)(t + PF) * 3 + g) * H);
        gh[g] = gru2_sum(sum2(acc[0][g]), sum2(acc[1][g]), p) + bias[g];
      }
      const float r = sigmoid_f(x[0] + gh[0]), z = sigmoid_f(x[1] + gh[1]), n = tanhf(x[2] + r * gh[2]);
      const float hn = (1.f - z) * n + z * hp;
      const long long at = ((long long)b * seq + t) * H + i;
      if (q == 0) sh[(u & 1) ^ 1][i] = hn;
      else rst<T>(out + at, hn);
      if (q == 0 && hprev) rst<T>(hprev + at, hp);
      if (coef) {
        const float cn = (1.f - z) * (1.f - n * n);
        const float2 c = q == 0 ? make_float2(cn * gh[2] * r * (1.f - r), (hp - n) * z * (1.f - z)) : make_float2(cn * r, cn);
        *reinterpret_cast<float2*>(coef + at * 4 + 2 * q) = c;
        if (q == 1) zg[at] = z;
      }
      hp = hn;
      __syncthreads();
    }
  }
}

template <typename T>
__global__ void __launch_bounds__(256, 1)
gru2_bwd_kernel(const float* __restrict__ coef, const float* __restrict__ zg, const T* __restrict__ w_hh, const T* __restrict__ dout, T* __restrict__ dgi,
                T* __restrict__ dgh, T* __restrict__ dh0, int seq, int H) {
  __shared__ __align__(16) float sg[2][3][16 * GRU2_NM];
  const int p = threadIdx.x & 3, q = p & 1, i0 = (threadIdx.x >> 2) * 2, i = i0 + (p >> 1), b = blockIdx.x;
  unsigned long long w[2][3][GRU2_NM][2];
  gru2_load<T>(w, w_hh, i0, p, H, false);
  for (int k = threadIdx.x; k < 2 * 3 * 16 * GRU2_NM; k += blockDim.x) (&sg[0][0][0])[k] = 0.f;
  __syncthreads();
  constexpr int PF = 2;
  const long long row0 = (long long)b * seq;
  float2 cf[PF];
  float zf[PF], df[PF];
  auto fetch = [&](int t, float2& c, float& z, float& d) {
    const long long at = (row0 + t) * H + i;
    c = *reinterpret_cast<const float2*>(coef + at * 4 + 2 * q);
    z = zg[at];
    d = rld<T>(dout + at);
  };
#pragma unroll
  for (int u = 0; u < PF; ++u)
    if (seq - 1 - u >= 0) fetch(seq - 1 - u, cf[u], zf[u], df[u]);
  float carry = 0.f;
  for (int t0 = seq - 1; t0 >= 0; t0 -= PF) {
#pragma unroll
    for (int u = 0; u < PF; ++u) {
      const int t = t0 - u;
      if (t < 0) break;
      const float d = df[u] + carry, g0 = d * cf[u].x, g1 = d * cf[u].y, direct = d * zf[u];
      if (t - PF >= 0) fetch(t - PF, cf[u], zf[u], df[u]);
      const long long at = (row0 + t) * 3 * H + i;
      if (q == 0) {                                            // reset and update gate
        sg[u & 1][0][i] = g0;
        sg[u & 1][1][i] = g1;
        rst<T>(dgh + at, g0); rst<T>(dgh + at + H, g1);
        rst<T>(dgi + at, g0); rst<T>(dgi + at + H, g1);
      } else {                                                 // candidate: through the recurrent and through the input projection
        sg[u & 1][2][i] = g0;
        rst<T>(dgh + at + 2 * H, g0);
        rst<T>(dgi + at + 2 * H, g1);
      }
      __syncthreads();
      unsigned long long acc[2][3] = {};
#pragma unroll
      for (int g = 0; g < 3; ++g)
#pragma unroll
        for (int m = 0; m < GRU2_NM; ++m) {
          const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(&sg[u & 1][g][4 * (p + 4 * m)]);
#pragma unroll
          for (int x = 0; x < 2; ++x) acc[x][g] = fma2(w[x][g][m][1], v.y, fma2(w[x][g][m][0], v.x, acc[x][g]));
        }
      float s[2];
#pragma unroll
      for (int x = 0; x < 2; ++x) s[x] = sum2(acc[x][0]) + sum2(acc[x][1]) + sum2(acc[x][2]);
      carry = direct + gru2_sum(s[0], s[1], p);
    }
  }
  if (dh0 && q == 0) rst<T>(dh0 + (long long)b * H + i, carry);
}

constexpr int RNN_REG_MAX_H = 128;
inline bool gru2_ok(int gates, int H) { return gates == 3 && H > 64 && H <= RNN_REG_MAX_H && H % 16 == 0; }
inline bool rnn_reg_ok(int H) { return H >= 8 && H <= RNN_REG_MAX_H && H % 8 == 0; }   // whole warps of four lanes per unit
#define OA_RNN_REG_NM(T, G, CALL)                                        \
  {                                                                      \
    if (H <= 32) { constexpr int NM = 2; CALL(T, G, NM); }               \
    else if (H <= 64) { constexpr int NM = 4; CALL(T, G, NM); }          \
    else { constexpr int NM = 8; CALL(T, G, NM); }                       \
  }
#define OA_RNN_REG_PICK(CALL)                                            \
  if (dtype == OA_F32) { if (gates == 3) OA_RNN_REG_NM(float, 3, CALL) else OA_RNN_REG_NM(float, 1, CALL) }          \
  else { if (gates == 3) OA_RNN_REG_NM(__nv_bfloat16, 3, CALL) else OA_RNN_REG_NM(__nv_bfloat16, 1, CALL) }

template <typename K>
static int rnn_set_smem(K kernel, size_t bytes) {
  if (bytes > 48 * 1024 && cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) != cudaSuccess) return OA_ERR_LAUNCH;
  return OA_OK;
}

}  // namespace oa

using namespace oa;
#define ST ((cudaStream_t)stream)

static void gru2_fwd(int dtype, const void* gates_i, const void* w_hh, const void* b_hh, const void* h0, void* out, void* hprev, float* coef, int batch, int seq,
                     int H, cudaStream_t st) {
  float* zg = coef ? coef + (size_t)batch * seq * H * 4 : nullptr;
  if (dtype == OA_F32)
    gru2_fwd_kernel<float><<<batch, 2 * H, 0, st>>>((const float*)gates_i, (const float*)w_hh, (const float*)b_hh, (const float*)h0, (float*)out, (float*)hprev,
                                                    coef, zg, seq, H);
  else
    gru2_fwd_kernel<__nv_bfloat16><<<batch, 2 * H, 0, st>>>((const __nv_bfloat16*)gates_i, (const __nv_bfloat16*)w_hh, (const __nv_bfloat16*)b_hh,
                                                            (const __nv_bfloat16*)h0, (__nv_bfloat16*)out, (__nv_bfloat16*)hprev, coef, zg, seq, H);
}
static void gru2_bwd(int dtype, const float* coef, const void* w_hh, const void* dout, void* dgi, void* dgh, void* dh0, int batch, int seq, int H,
                     cudaStream_t st) {
  const float* zg = coef + (size_t)batch * seq * H * 4;
  if (dtype == OA_F32)
    gru2_bwd_kernel<float><<<batch, 2 * H, 0, st>>>(coef, zg, (const float*)w_hh, (const float*)dout, (float*)dgi, (float*)dgh, (float*)dh0, seq, H);
  else
    gru2_bwd_kernel<__nv_bfloat16><<<batch, 2 * H, 0, st>>>(coef, zg, (const __nv_bfloat16*)w_hh, (const __nv_bfloat16*)dout, (__nv_bfloat16*)dgi,
                                                            (__nv_bfloat16*)dgh, (__nv_bfloat16*)dh0, seq, H);
}

// Floats that a forward scan can leave for the backward one (0: it leaves none), and the two scans with them.
extern "C" size_t oa_gru_coef_floats(int gates, int batch, int seq, int H) { return gru2_ok(gates, H) ? (size_t)batch * seq * H * 5 : 0; }
extern "C" int oa_gru_scan_fwd_coef(int dtype, const void* gates_i, const void* w_hh, const void* b_hh, const void* h0, void* out, void* hprev, float* coef,
                                    int batch, int seq, int H, void* stream) {
  if (batch <= 0 || seq <= 0) return OA_OK;
  if ((dtype != OA_F32 && dtype != OA_BF16) || !gru2_ok(3, H)) return OA_ERR_UNSUPPORTED;
  if (!coef) return OA_ERR_ARG;
  gru2_fwd(dtype, gates_i, w_hh, b_hh, h0, out, hprev, coef, batch, seq, H, ST);
  return cudaGetLastError() == cudaSuccess ? OA_OK : OA_ERR_LAUNCH;
}
extern "C" int oa_gru_scan_bwd_coef(int dtype, const float* coef, const void* w_hh, const void* dout, void* dgi, void* dgh, void* dh0, int batch, int seq,
                                    int H, void* stream) {
  if (batch <= 0 || seq <= 0) return OA_OK;
  if ((dtype != OA_F32 && dtype != OA_BF16) || !gru2_ok(3, H)) return OA_ERR_UNSUPPORTED;
  if (!coef) return OA_ERR_ARG;
  gru2_bwd(dtype, coef, w_hh, dout, dgi, dgh, dh0, batch, seq, H, ST);
  return cudaGetLastError() == cudaSuccess ? OA_OK : OA_ERR_LAUNCH;
}

// gates = 3 (GRU) or 1 (RNN).  gates_i [B, S, gates*H], w_hh [gates*H, H], b_hh [gates*H] or null, h0 [B, H] or null,
// out [B, S, H], hprev [B, S, H] or null (needed for the backward pass).
extern "C" int oa_rnn_scan_fwd(int dtype, int gates, const void* gates_i, const void* w_hh, const void* b_hh, const void* h0,
                               void* out, void* hprev, int batch, int seq, int H, void* stream) {
  if (gates != 1 && gates != 3) return OA_ERR_ARG;
  if (batch <= 0 || seq <= 0) return OA_OK;
  if (dtype != OA_F32 && dtype != OA_BF16) return OA_ERR_UNSUPPORTED;
  if (gru2_ok(gates, H)) {
    gru2_fwd(dtype, gates_i, w_hh, b_hh, h0, out, hprev, nullptr, batch, seq, H, ST);
    return cudaGetLastError() == cudaSuccess ? OA_OK : OA_ERR_LAUNCH;
  }
  if (rnn_reg_ok(H)) {
#define CALL_REG_FWD(T, G, NM)                                                                                              \
    rnn_reg_fwd_kernel<T, G, NM><<<batch, 4 * H, 0, ST>>>((const T*)gates_i, (const T*)w_hh, (const T*)b_hh, (const T*)h0, \
                                                          (T*)out, (T*)hprev, seq, H)
    OA_RNN_REG_PICK(CALL_REG_FWD)
    return cudaGetLastError() == cudaSuccess ? OA_OK : OA_ERR_LAUNCH;
  }
  size_t smem = (size_t)RNN_BT * H * (1 + gates) * sizeof(float);
  if (smem > 200 * 1024) return OA_ERR_TOO_LARGE;
  int blocks = (batch + RNN_BT - 1) / RNN_BT, rc;
#define LAUNCH_FWD(T, G)                                                                                         \
  {                                                                                                              \
    if ((rc = rnn_set_smem(rnn_scan_fwd_kernel<T, G>, smem))) return rc;                                         \
    rnn_scan_fwd_kernel<T, G><<<blocks, RNN_THREADS, smem, ST>>>((const T*)gates_i, (const T*)w_hh, (const T*)b_hh, \
                                                                 (const T*)h0, (T*)out, (T*)hprev, batch, seq, H); \
  }
  if (dtype == OA_F32) { if (gates == 3) LAUNCH_FWD(float, 3) else LAUNCH_FWD(float, 1) }
  else if (dtype == OA_BF16) { if (gates == 3) LAUNCH_FWD(__nv_bfloat16, 3) else LAUNCH_FWD(__nv_bfloat16, 1) }
  else return OA_ERR_UNSUPPORTED;
  return cudaGetLastError() == cudaSuccess ? OA_OK : OA_ERR_LAUNCH;
}

// Floats of scratch that oa_rnn_scan_bwd wants (0: none): the per-step coefficients of the register-resident path.
extern "C" size_t oa_rnn_scan_bwd_scratch_floats(int gates, int batch, int seq, int H) {
  return rnn_reg_ok(H) ? (size_t)batch * seq * H * (gates == 3 ? 5 : 1) : 0;
}

extern "C" int oa_rnn_scan_bwd(int dtype, int gates, const void* gates_i, const void* w_hh, const void* b_hh, const void* hprev,
                               const void* dout, void* dgi, void* dgh, void* dh0, float* scratch, int batch, int seq, int H, void* stream) {
  if (gates != 1 && gates != 3) return OA_ERR_ARG;
  if (batch <= 0 || seq <= 0) return OA_OK;
  if (dtype != OA_F32 && dtype != OA_BF16) return OA_ERR_UNSUPPORTED;
  if (rnn_reg_ok(H)) {
    if (!scratch) return OA_ERR_ARG;
    const long long rows = (long long)batch * seq;
    float* zg = scratch + rows * H * 4;                       // GRU only
    const int grid = rows < 148 * 4 ? (int)rows : 148 * 4;
    if (gru2_ok(gates, H)) {
      if (dtype == OA_F32)
        rnn_reg_coef_kernel<float, 3, 8><<<grid, 4 * H, 0, ST>>>((const float*)gates_i, (const float*)w_hh, (const float*)b_hh, (const float*)hprev, scratch, zg,
                                                                 rows, H);
      else
        rnn_reg_coef_kernel<__nv_bfloat16, 3, 8><<<grid, 4 * H, 0, ST>>>((const __nv_bfloat16*)gates_i, (const __nv_bfloat16*)w_hh, (const __nv_bfloat16*)b_hh,
                                                                         (const __nv_bfloat16*)hprev, scratch, zg, rows, H);
      gru2_bwd(dtype, scratch, w_hh, dout, dgi, dgh, dh0, batch, seq, H, ST);
      return cudaGetLastError() == cudaSuccess ? OA_OK : OA_ERR_LAUNCH;
    }
#define CALL_REG_BWD(T, G, NM)                                                                                               \
    rnn_reg_coef_kernel<T, G, NM><<<grid, 4 * H, 0, ST>>>((const T*)gates_i, (const T*)w_hh, (const T*)b_hh, (const T*)hprev, \
                                                          scratch, zg, rows, H);                                              \
    rnn_reg_bwd_kernel<T, G, NM><<<batch, 4 * H, 0, ST>>>(scratch, zg, (const T*)w_hh, (const T*)dout, (T*)dgi, (T*)dgh,      \
                                                          (T*)dh0, seq, H)
    OA_RNN_REG_PICK(CALL_REG_BWD)
    return cudaGetLastError() == cudaSuccess ? OA_OK : OA_ERR_LAUNCH;
  }
  size_t smem = (size_t)RNN_BT * H * (2 + 2 * gates) * sizeof(float);
  if (smem > 200 * 1024) return OA_ERR_TOO_LARGE;
  int blocks = (batch + RNN_BT - 1) / RNN_BT, rc;
#define LAUNCH_BWD(T, G)                                                                                           \
  {                                                                                                                \
    if ((rc = rnn_set_smem(rnn_scan_bwd_kernel<T, G>, smem))) return rc;                                           \
    rnn_scan_bwd_kernel<T, G><<<blocks, RNN_THREADS, smem, ST>>>((const T*)gates_i, (const T*)w_hh, (const T*)b_hh,   \
                                                                 (const T*)hprev, (const T*)dout, (T*)dgi, (T*)dgh,  \
                                                                 (T*)dh0, batch, seq, H);                           \
  }
  if (dtype == OA_F32) { if (gates == 3) LAUNCH_BWD(float, 3) else LAUNCH_BWD(float, 1) }
  else if (dtype == OA_BF16) { if (gates == 3) LAUNCH_BWD(__nv_bfloat16, 3) else LAUNCH_BWD(__nv_bfloat16, 1) }
  else return OA_ERR_UNSUPPORTED;
  return cudaGetLastError() == cudaSuccess ? OA_OK : OA_ERR_LAUNCH;
}
