// Real-gated linear recurrent unit, fp32 state, one channel per thread:
//   r = sigmoid(gr + br), i = sigmoid(gi + bi), log a = -8 r softplus(lam), a = exp(log a)
//   S <- a S + sqrt(1 - a^2) i u,     out = S * gelu_tanh(y)
// gr, gi are the fp32 products of the block-diagonal gate matrices with u (biases are added here).  Any L; a call
// whose first token is position 0 starts from zero whatever the state buffer holds.
//
//  * rglru: the recurrence alone, u and the gate products given.
//  * rglru_step: a decode step from the packed projection to the gated output in ONE launch (bf16): short convolution over the
//    input ring, both gate products, recurrence.  All of it is latency (0.6 MB of weights and state at 16 rows of 1024): a
//    block has 32 channels of one gate block and 16 rows, takes the convolution of the whole gate block for itself (a few KB,
//    cheaper than a second launch that shares it) and multiplies it by its 64 rows of the gate matrices, one 8-row tile per
//    warp, whose loads are in flight before the convolution.  Three launches, the middle one a library product that ends a
//    chain of programmatic launches, took 6.5 us in a chain of their own at 16 rows of 1024 (7.2 without programmatic launches),
//    this one 4.2; a step of 17 such layers 731 -> 662 us.
#include <initializer_list>

#include "seq_common.cuh"

namespace based {
namespace {

using namespace seq;

struct RgP {
  const void *u, *y, *rb, *ib;
  const float *gates, *lam;
  float* state;                  // [B, W]
  void* out;
  const int32_t* offsets;
  int offset, B, L, W, bw;       // bw: width of one block
  Strides2 su, sy, so;           // .b batch, .h token
  int64_t g_block, g_row;        // gates: (block, row = b L + l, r_0..r_bw-1 i_0..i_bw-1)
};

constexpr int kThreads = 64;

template <typename T, int U>
__global__ void __launch_bounds__(kThreads) rglru_kernel(const RgP p) {
  pdl_trigger();
  pdl_wait();
  const int c = blockIdx.x * kThreads + threadIdx.x, b = blockIdx.y;
  if (c >= p.W) return;
  const int blk = c / p.bw, j = c - blk * p.bw;
  const T* u = static_cast<const T*>(p.u) + b * p.su.b + c;
  const T* y = static_cast<const T*>(p.y) + b * p.sy.b + c;
  T* out = static_cast<T*>(p.out) + b * p.so.b + c;
  const float* gt = p.gates + blk * p.g_block + (int64_t)b * p.L * p.g_row + j;
  const float rb = to_float<T>(static_cast<const T*>(p.rb)[c]), ib = to_float<T>(static_cast<const T*>(p.ib)[c]);
  const float decay = -8.0f * softplus_acc(p.lam[c]);
  float S = position0(p.offsets, p.offset, b) == 0 ? 0.f : p.state[(int64_t)b * p.W + c];
  for (int l0 = 0; l0 < p.L; l0 += U) {
    float uv[U], yv[U], gr[U], gi[U];
#pragma unroll
    for (int t = 0; t < U; ++t)
      if (l0 + t < p.L) {
        uv[t] = to_float<T>(u[(l0 + t) * p.su.h]);
        yv[t] = to_float<T>(y[(l0 + t) * p.sy.h]);
        gr[t] = gt[(l0 + t) * p.g_row];
        gi[t] = gt[(l0 + t) * p.g_row + p.bw];
      }
#pragma unroll
    for (int t = 0; t < U; ++t)
      if (l0 + t < p.L) {
        const float la = decay * sigmoid_acc(gr[t] + rb);
        const float in = sqrtf(-expm1f(2.0f * la)) * sigmoid_acc(gi[t] + ib) * uv[t];
        S = fmaf(expf(la), S, in);
        out[(l0 + t) * p.so.h] = from_float<T>(S * gelu_tanh_t<T>(yv[t]));
      }
  }
  p.state[(int64_t)b * p.W + c] = S;
}

// ------------------------------------------------------------------ decode step
constexpr int kStepCh = 32, kStepThreads = 256, kMaxN = 256;

struct RgStepP {
  const __nv_bfloat16 *x, *y, *cw, *cb, *gw, *rb, *ib;   // x, y: rows sx, sy apart; cw [W, taps], cb [W] or null; gw [blocks][2][n][n]
  const float* lam;
  __nv_bfloat16 *ring, *out;                             // ring [B, taps, W]
  float* state;                                          // [B, W]
  const int32_t* offsets;
  int64_t sx, sy, so;
  int offset, B, W, n, taps;
};

// grid (W / 32, ceil(B / 16))
template <int TAPS>
__global__ void __launch_bounds__(kStepThreads) rglru_step_kernel(const RgStepP p) {
  pdl_trigger();
  constexpr int LD = kMaxN + 8;
  __shared__ __align__(16) __nv_bfloat16 us[16 * LD];
  __shared__ float gates[2][16][kStepCh];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  const int c0 = blockIdx.x * kStepCh, blk = c0 / p.n, in0 = c0 - blk * p.n, base = blk * p.n, row0 = blockIdx.y * 16;
  const __nv_bfloat16* w = p.gw + ((int64_t)blk * 2 + (warp >> 2)) * p.n * p.n + (int64_t)(in0 + (warp & 3) * 8 + g) * p.n;   // r: warps 0-3, i: 4-7
  if (t == 0) prefetch_l2(w, p.n * 2);
  pdl_wait();
  uint4 wv[kMaxN / 32];
#pragma unroll
  for (int k = 0; k < kMaxN / 32; ++k)
    if (k * 32 < p.n) wv[k] = __ldg(reinterpret_cast<const uint4*>(w + k * 32 + 8 * t));
  // what the recurrence of this thread's two (row, channel) will need
  const int ch = c0 + lane;
  float yv[2], S[2];
  int at[2];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int b = row0 + warp + 8 * i;
    yv[i] = S[i] = 0.f;
    if (b < p.B) {
      yv[i] = __bfloat162float(p.y[b * p.sy + ch]);
      if (position0(p.offsets, p.offset, b) > 0) S[i] = p.state[(int64_t)b * p.W + ch];
    }
    at[i] = b;
  }
  const float rb = __bfloat162float(p.rb[ch]), ib = __bfloat162float(p.ib[ch]), lam = p.lam[ch];
  // the convolution of the gate block's channels, eight of a row per thread
  const int vecs = p.n / 8;
  for (int v = tid; v < 16 * vecs; v += kStepThreads) {
    const int r = v / vecs, c = (v - r * vecs) * 8, b = row0 + r;
    float acc[8] = {};
    if (b < p.B) {
      const int pos = position0(p.offsets, p.offset, b);
      const __nv_bfloat16* x = p.x + b * p.sx + base + c;
      __nv_bfloat16* ring = p.ring + (int64_t)b * TAPS * p.W + base + c;
      float in[TAPS][8], taps[8 * TAPS];
      const uint4 now = *reinterpret_cast<const uint4*>(x);
#pragma unroll
      for (int j = 0; j < TAPS - 1; ++j) {
        const int pp = pos - (TAPS - 1) + j;
#pragma unroll
        for (int i = 0; i < 8; ++i) in[j][i] = 0.f;
        if (pp >= 0) Pack<__nv_bfloat16, 8>::load(ring + (int64_t)(pp % TAPS) * p.W, in[j]);
      }
      Pack<__nv_bfloat16, 8>::load(x, in[TAPS - 1]);
#pragma unroll
      for (int q = 0; q < TAPS; ++q) {
        float f[8];
        Pack<__nv_bfloat16, 8>::load(p.cw + (int64_t)(base + c) * TAPS + 8 * q, f);
#pragma unroll
        for (int i = 0; i < 8; ++i) taps[8 * q + i] = f[i];
      }
      if (p.cb) Pack<__nv_bfloat16, 8>::load(p.cb + base + c, acc);
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < TAPS; ++j) acc[i] = fmaf(taps[i * TAPS + j], in[j][i], acc[i]);
      // the slot nobody reads; one of the gate block's blocks writes it
      if (in0 == 0) *reinterpret_cast<uint4*>(ring + (int64_t)(pos % TAPS) * p.W) = now;
    }
    Pack<__nv_bfloat16, 8>::store(us + r * LD + c, acc);
  }
  __syncthreads();
  float acc[4] = {};
#pragma unroll
  for (int k = 0; k < kMaxN / 32; ++k)
    if (k * 32 < p.n) {   // 32 of K: 8 consecutive values per lane, permuted alike in both operands
      const uint4 lo = *reinterpret_cast<const uint4*>(us + g * LD + k * 32 + 8 * t), hi = *reinterpret_cast<const uint4*>(us + (g + 8) * LD + k * 32 + 8 * t);
      const uint4 b = wv[k];
      asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                   : "+f"(acc[0]), "+f"(acc[1]), "+f"(acc[2]), "+f"(acc[3]) : "r"(lo.x), "r"(hi.x), "r"(lo.y), "r"(hi.y), "r"(b.x), "r"(b.y));
      asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                   : "+f"(acc[0]), "+f"(acc[1]), "+f"(acc[2]), "+f"(acc[3]) : "r"(lo.z), "r"(hi.z), "r"(lo.w), "r"(hi.w), "r"(b.z), "r"(b.w));
    }
  {
    const int col = (warp & 3) * 8 + 2 * t;
    *reinterpret_cast<float2*>(&gates[warp >> 2][g][col]) = make_float2(acc[0], acc[1]);
    *reinterpret_cast<float2*>(&gates[warp >> 2][g + 8][col]) = make_float2(acc[2], acc[3]);
  }
  __syncthreads();
  const float decay = -8.0f * softplus_acc(lam);
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    if (at[i] >= p.B) continue;
    const int r = warp + 8 * i;
    const float la = decay * sigmoid_acc(gates[0][r][lane] + rb);
    const float in = sqrtf(-expm1f(2.0f * la)) * sigmoid_acc(gates[1][r][lane] + ib) * __bfloat162float(us[r * LD + in0 + lane]);
    const float s = fmaf(expf(la), S[i], in);
    p.out[at[i] * p.so + ch] = __float2bfloat16_rn(s * gelu_tanh_t<__nv_bfloat16>(yv[i]));
    p.state[(int64_t)at[i] * p.W + ch] = s;
  }
}

}  // namespace

// BASED_ERR_IMPL: sizes or alignments the step kernel does not take.
int launch_rglru_step(const void* x, const void* y, const void* cw, const void* cb, void* ring, const void* gw, const void* rb,
                      const void* ib, const float* lam, float* state, void* out, int B, int W, int n, int taps, int64_t sx,
                      int64_t sy, int64_t so, const int32_t* offsets, int offset, cudaStream_t stream) {
  if (n % kStepCh || n > kMaxN || taps < 2 || taps > 4 || sx % 8 || B > 16 * 65535) return BASED_ERR_IMPL;
  for (const void* q : {x, cw, cb, static_cast<const void*>(ring), gw})
    if (!aligned16(q)) return BASED_ERR_IMPL;
  using T = __nv_bfloat16;
  const RgStepP p{static_cast<const T*>(x), static_cast<const T*>(y), static_cast<const T*>(cw), static_cast<const T*>(cb),
                  static_cast<const T*>(gw), static_cast<const T*>(rb), static_cast<const T*>(ib), lam, static_cast<T*>(ring),
                  static_cast<T*>(out), state, offsets, sx, sy, so, offset, B, W, n, taps};
  auto kern = taps == 2 ? rglru_step_kernel<2> : taps == 3 ? rglru_step_kernel<3> : rglru_step_kernel<4>;
  return launched(launch_pdl(kern, dim3(W / kStepCh, (B + 15) / 16), dim3(kStepThreads), 0, stream, p));
}

int launch_rglru(const void* u, const void* y, const float* gates, const void* rb, const void* ib, const float* lam,
                 float* state, void* out, int B, int L, int W, int bw, Strides2 su, Strides2 sy, Strides2 so,
                 int64_t g_block, int64_t g_row, const int32_t* offsets, int offset, int io_dtype, cudaStream_t stream) {
  if (B > 65535) return BASED_ERR_TOO_LARGE;
  const RgP p{u, y, rb, ib, gates, lam, state, out, offsets, offset, B, L, W, bw, su, sy, so, g_block, g_row};
  const dim3 grid((W + kThreads - 1) / kThreads, B);
  if (io_dtype == BASED_BF16) {
    if (L == 1) launch_pdl(rglru_kernel<__nv_bfloat16, 1>, grid, kThreads, 0, stream, p);
    else launch_pdl(rglru_kernel<__nv_bfloat16, 8>, grid, kThreads, 0, stream, p);
  } else {
    if (L == 1) launch_pdl(rglru_kernel<float, 1>, grid, kThreads, 0, stream, p);
    else launch_pdl(rglru_kernel<float, 8>, grid, kThreads, 0, stream, p);
  }
  return (int)cudaGetLastError();
}

}  // namespace based
