// Linear layers of a decode step: y[M, N] = x[M, K] W[N, K]^T (+ bias) for a handful of rows
// (M = batch of single tokens), bf16 in, fp32 accumulation, with the elementwise step that
// follows the projection in the Based blocks fused into the epilogue:
//   PLAIN   y = x W^T + b                                   (out_proj, fc2, Wqkv, q/k/v projections)
//   SWIGLU  out = (x W1^T) * act(x W2^T), W = [W1; W2]      fc1 + `y * act(gate)` of GatedMlp.forward
//                                                           (based/models/mlp.py:141-154)
//   CONV    u = x W^T + b, [u1 | u2] = u; the BaseConv decode step on u1 (shift the [B, d, k] state,
//           append, dot with the taps), silu, gate by u2       in_proj + ShortConvolution.step + gate
//                                                           (based/models/mixers/convolution.py:88-109, :205-211)
//   F32     PLAIN with an fp32 result
//   ADD     y = x W^T + b joins the fp32 residual stream in place (z = residual + y), and z times the weights of the
//           norm that comes next goes out in bf16, with the sums of z^2 over 8 columns beside it
// A product of up to 16 rows may take ADD's outputs for x: the norm's 1 / rms is one factor per row, so it is applied to the
// sums (row_ss), and no launch stands between the product before a norm and the one after it.
// The work is reading W once, 2 to 26 MB: 0.3 to 4 us at the HBM rate, so a launch of its own is mostly latency: the launch, the
// first bytes from HBM, the sum over the split of K.  Two things against that:
//  * The launch is programmatic: the blocks start while the kernel before still runs, bring their part of W into L2 (a hint;
//    nothing is read that an earlier kernel may still write), and only then wait for that kernel's end.  The HBM stream of a
//    chain of such launches does not stop between them.
//  * All or half of a warp's loads are in flight at once for the usual K: eight or sixteen warps split K, a block owns 8 output
//    columns (for two halves that an epilogue combines 8 of each; two or four times that where N would need more blocks than
//    the device holds) and 16, 32 or 64 rows (m16n8k16 tiles, W read once for all).  Each lane reads 16 contiguous
//    bytes of one weight row per step -- the K order inside a 32-wide block is permuted identically for x and W, which a dot
//    product does not notice -- so a warp's load covers 8 rows x 64 bytes; x (a few KB, L2 resident) is read the same way.
// In a chain of such launches, W from HBM, 16 rows (us; cuBLAS's kernel, this one, W at the HBM rate): 1024 x 1024 4.6, 2.9, 0.3;
// 1024 x 2048 6.6, 2.6, 0.6; 4096 x 1024 4.7, 3.1, 1.3 (with the gated activation 6.8, 3.1); 7168 x 1792 7.4, 6.9, 3.9.
#include "common.cuh"

namespace based {
namespace {

constexpr int kSms = 148;
enum Epi { EPI_PLAIN = 0, EPI_SWIGLU = 1, EPI_CONV = 2, EPI_F32 = 3, EPI_ADD = 4 };

struct LinParams {
  const __nv_bfloat16 *x, *w, *bias;
  void* out;
  int M, N, K;          // N = rows of W (SWIGLU / CONV: 2 x outputs)
  int64_t sx, so;       // row strides of x and out
  int act;              // SWIGLU: 0 silu, 1 sigmoid
  // CONV
  __nv_bfloat16* state;            // [M, N/2, ck]
  const void *cw, *cb;             // taps [N/2, ck], bias [N/2] or null
  int ck, cw_bf16;
  // x is scaled per row by 1 / sqrt(sum of the row's n_ss entries / K + eps); null: it is not
  const float* row_ss;             // [M, n_ss]
  int n_ss;
  float eps;
  // ADD
  float *residual, *ss;            // [M, N] fp32; [M, N / 8]
  const __nv_bfloat16* norm;       // [N]
};

__device__ __forceinline__ void mma_16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ float sigmoid_f(float x) { return __fdividef(1.0f, 1.0f + __expf(-x)); }
__device__ __forceinline__ float bf16_round(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }
__device__ __forceinline__ float ld_w(const void* p, int bf16, int i) {
  return bf16 ? __bfloat162float(static_cast<const __nv_bfloat16*>(p)[i]) : static_cast<const float*>(p)[i];
}

// CT: 8-column tiles of outputs per block; an epilogue of two halves reads two tiles of W for each, N/2 rows apart.
// MT: tiles of 16 rows of x.  U: 32-wide blocks of K whose loads are issued together.
// grid = (ceil(outputs / (8 CT)), ceil(M / (16 MT))), block = WARPS x 32
template <int CT, int EPI, int MT, int U, int WARPS>
__global__ void __launch_bounds__(WARPS * 32, WARPS > 8 ? 1 : 2) decode_linear_kernel(const LinParams p) {
  pdl_trigger();
  constexpr bool kTwo = EPI == EPI_SWIGLU || EPI == EPI_CONV;
  constexpr int kCols = 8 * CT, NT8 = kTwo ? 2 * CT : CT;   // output columns of the block, tiles of W: tile i of a second half is CT + i
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int n0 = blockIdx.x * kCols, m0 = blockIdx.y * 16 * MT;
  const int half = p.N / 2, outputs = kTwo ? half : p.N;
  // first row of W of a tile; the last block's may not be full
  auto w_row = [&](int tile) { return min(n0 + (tile % CT) * 8, outputs - 8) + (tile >= CT ? half : 0); };
  // K slice of this warp, in blocks of 32
  const int kblocks = p.K / 32, per = (kblocks + WARPS - 1) / WARPS;
  const int kb0 = warp * per, kb1 = min(kb0 + per, kblocks);
  const __nv_bfloat16* wr[NT8];
#pragma unroll
  for (int i = 0; i < NT8; ++i) wr[i] = p.w + (int64_t)(w_row(i) + g) * p.K + 8 * t;
  // This warp's part of W into L2, a row segment per lane.  Not for two row tiles a block and more than 32 rows: the library's product
  // is ahead then, nothing overlaps, and W comes twice anyway (MLP of 512 x 1024, 33 rows: 7.3 us with it, 6.6 without).
  if ((MT != 2 || p.M <= 32) && lane < 8 * NT8 && kb0 < kb1) prefetch_l2(p.w + (int64_t)(w_row(lane >> 3) + (lane & 7)) * p.K + kb0 * 32, (kb1 - kb0) * 64);
  pdl_wait();
  const __nv_bfloat16* xr[2 * MT];
  bool live[2 * MT];
#pragma unroll
  for (int m = 0; m < 2 * MT; ++m) {
    live[m] = m0 + g + 8 * m < p.M;
    xr[m] = p.x + (int64_t)(live[m] ? m0 + g + 8 * m : 0) * p.sx + 8 * t;
  }
  float acc[NT8][MT][4];
#pragma unroll
  for (int i = 0; i < NT8; ++i)
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[i][m][e] = 0.f;
  const uint4 zero = make_uint4(0, 0, 0, 0);
  for (int kb = kb0; kb < kb1; kb += U) {
    uint4 wv[U][NT8], xv[U][2 * MT];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const bool ok = kb + u < kb1;
      const int ko = (kb + u) * 32;
#pragma unroll
      for (int i = 0; i < NT8; ++i) wv[u][i] = ok ? __ldg(reinterpret_cast<const uint4*>(wr[i] + ko)) : zero;
#pragma unroll
      for (int m = 0; m < 2 * MT; ++m) xv[u][m] = ok && live[m] ? *reinterpret_cast<const uint4*>(xr[m] + ko) : zero;
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int m = 0; m < MT; ++m) {
        const uint4 lo = xv[u][2 * m], hi = xv[u][2 * m + 1];
        const uint32_t fa[4] = {lo.x, hi.x, lo.y, hi.y}, fb[4] = {lo.z, hi.z, lo.w, hi.w};
#pragma unroll
        for (int i = 0; i < NT8; ++i) {
          mma_16816(acc[i][m], fa, wv[u][i].x, wv[u][i].y);
          mma_16816(acc[i][m], fb, wv[u][i].z, wv[u][i].w);
        }
      }
  }
  // ---- the rows' factors, a few threads to a row
  __shared__ float factor[16 * MT];
  if (MT == 1 && p.row_ss) {
    constexpr int kTo = WARPS * 2;   // threads per row
    const int row = tid / kTo, j0 = tid % kTo;
    float sum = 0.f;
    if (m0 + row < p.M)
      for (int j = j0; j < p.n_ss; j += kTo) sum += p.row_ss[(int64_t)(m0 + row) * p.n_ss + j];
#pragma unroll
    for (int o = kTo / 2; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (j0 == 0) factor[row] = rsqrtf(sum / (float)p.K + p.eps);
  }
  // ---- the K slices' sums meet in shared memory, [warp][tile][row][column]; lanes hold rows g, g + 8 and columns 2t, 2t + 1
  __shared__ float red[WARPS][NT8][16 * MT * 8];
#pragma unroll
  for (int i = 0; i < NT8; ++i)
#pragma unroll
    for (int m = 0; m < MT; ++m) {
      *reinterpret_cast<float2*>(&red[warp][i][(16 * m + g) * 8 + 2 * t]) = make_float2(acc[i][m][0], acc[i][m][1]);
      *reinterpret_cast<float2*>(&red[warp][i][(16 * m + g + 8) * 8 + 2 * t]) = make_float2(acc[i][m][2], acc[i][m][3]);
    }
  // outputs (tile, row, column) over the threads
  constexpr int kIn = 16 * MT * 8, kOut = kIn * CT, kThreads = WARPS * 32, kPer = (kOut + kThreads - 1) / kThreads;
  float bias[kPer][2], cs[kPer][8], cw[kPer][8], cb[kPer];
#pragma unroll
  for (int r = 0; r < kPer; ++r) {
    const int o = tid + r * kThreads, in = o % kIn, col = n0 + o / kIn * 8 + (in & 7), row = m0 + (in >> 3);
    bias[r][0] = bias[r][1] = cb[r] = 0.f;
    if (o < kOut && col < outputs && p.bias) {
      bias[r][0] = __bfloat162float(p.bias[col]);
      if (kTwo) bias[r][1] = __bfloat162float(p.bias[col + half]);
    }
    if (EPI == EPI_CONV && o < kOut && row < p.M && col < outputs) {   // these loads' latency passes with the barrier
      const __nv_bfloat16* st = p.state + ((int64_t)row * half + col) * p.ck;
      if (p.cb) cb[r] = ld_w(p.cb, p.cw_bf16, col);
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (j < p.ck) {
          cs[r][j] = __bfloat162float(st[j]);
          cw[r][j] = ld_w(p.cw, p.cw_bf16, col * p.ck + j);
        }
    }
    if (EPI == EPI_ADD && o < kOut && row < p.M && col < outputs) {
      cs[r][0] = p.residual[(int64_t)row * p.N + col];
      cw[r][0] = __bfloat162float(p.norm[col]);
    }
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < kPer; ++r) {
    const int o = tid + r * kThreads, tile = o / kIn, in = o % kIn, col = n0 + tile * 8 + (in & 7), row = m0 + (in >> 3);
    if (o >= kOut || row >= p.M || col >= outputs) continue;
    float y = 0.f, y2 = 0.f;
#pragma unroll
    for (int w = 0; w < WARPS; ++w) {
      y += red[w][tile][in];
      if (kTwo) y2 += red[w][(kTwo ? CT : 0) + tile][in];
    }
    if (MT == 1 && p.row_ss) {
      y *= factor[in >> 3];
      y2 *= factor[in >> 3];
    }
    y += bias[r][0];
    y2 += bias[r][1];
    const int64_t at = (int64_t)row * p.so + col;
    if (EPI == EPI_F32) {
      static_cast<float*>(p.out)[at] = y;
      continue;
    }
    __nv_bfloat16* out = static_cast<__nv_bfloat16*>(p.out) + at;
    if (EPI == EPI_ADD) {
      const float z = cs[r][0] + y;     // fp32: the branch is not rounded on its way
      p.residual[(int64_t)row * p.N + col] = z;
      *out = __float2bfloat16_rn(z * cw[r][0]);
      float ss = z * z;            // eight neighbouring threads have a row's eight columns, and take this way together
#pragma unroll
      for (int d = 1; d < 8; d <<= 1) ss += __shfl_xor_sync(0xffu << (lane & 24), ss, d);
      if ((in & 7) == 0) p.ss[(int64_t)row * (p.N / 8) + col / 8] = ss;
    } else if (EPI == EPI_PLAIN) {
      *out = __float2bfloat16_rn(y);
    } else if (EPI == EPI_SWIGLU) {
      y = bf16_round(y);                          // fc1's output is a bf16 tensor in the unfused sequence
      const float gt = bf16_round(y2), s = sigmoid_f(gt);
      *out = __float2bfloat16_rn(y * (p.act == 0 ? gt * s : s));
    } else {
      __nv_bfloat16* st = p.state + ((int64_t)row * half + col) * p.ck;
      const __nv_bfloat16 u1 = __float2bfloat16_rn(y);
      float c = cb[r];
#pragma unroll
      for (int j = 0; j < 7; ++j)
        if (j < p.ck - 1) {
          st[j] = __float2bfloat16_rn(cs[r][j + 1]);   // exact: it was a bf16 value
          c = fmaf(cw[r][j], cs[r][j + 1], c);
        }
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (j == p.ck - 1) {
          st[j] = u1;
          c = fmaf(cw[r][j], __bfloat162float(u1), c);
        }
      *out = __float2bfloat16_rn(c * sigmoid_f(c) * bf16_round(y2));
    }
  }
}

template <int EPI, int CT>
int launch_tiles(const LinParams& p, int outputs, cudaStream_t stream) {
  constexpr int NT8 = (EPI == EPI_SWIGLU || EPI == EPI_CONV ? 2 : 1) * CT;
  constexpr int U1 = NT8 == 1 ? 8 : NT8 == 2 ? 4 : 2, U2 = NT8 == 1 ? 4 : 2;
  const int gx = (outputs / 8 + CT - 1) / CT;
  const dim3 g1(gx, 1), g2(gx, (p.M + 31) / 32);
  // More rows: four tiles of 16, W read once for all of them, where registers and shared memory allow it (64 rows, us with two tiles
  // and W read twice / like this: 4096 x 1024 8.2 / 6.3, with the gated activation the same; 1792 x 1792 10.8 / 7.1).  Not with the
  // gated activation while two tiles need no second round of blocks: 2048 x 1024 4.2 / 5.2 (33 rows), 4.2 / 6.0 (64).
  if constexpr (NT8 <= 2 && EPI != EPI_CONV && EPI != EPI_ADD) {
    const int resident = CT == 1 && p.K > 1024 && gx <= kSms ? kSms : 2 * kSms;
    const bool once = EPI == EPI_SWIGLU && (int64_t)gx * g2.y <= resident;
    if (p.M > 32 && !once) return launch_pdl(decode_linear_kernel<CT, EPI, 4, 1, 8>, dim3(gx, (p.M + 63) / 64), dim3(256), 0, stream, p);
  }
  // 16 warps to a block where K is long and every block has an SM: a warp's loads are one round again
  if constexpr (CT == 1) {
    if (p.K > 1024 && gx <= kSms) {
      if (p.M <= 16) return launch_pdl(decode_linear_kernel<CT, EPI, 1, 4, 16>, g1, dim3(512), 0, stream, p);
      return launch_pdl(decode_linear_kernel<CT, EPI, 2, U2, 16>, g2, dim3(512), 0, stream, p);
    }
  }
  if (p.M <= 16) return launch_pdl(decode_linear_kernel<CT, EPI, 1, U1, 8>, g1, dim3(256), 0, stream, p);
  return launch_pdl(decode_linear_kernel<CT, EPI, 2, U2, 8>, g2, dim3(256), 0, stream, p);
}

// Column tiles per block: as few as let all blocks be on the device at once, two to an SM; a block that starts later starts
// its share of W later, and the kernel after this one cannot start its own before it.
template <int EPI>
int launch_epi(const LinParams& p, int outputs, cudaStream_t stream) {
  const int tiles = outputs / 8;
  if constexpr (EPI == EPI_PLAIN || EPI == EPI_F32 || EPI == EPI_ADD)
    if (tiles > 4 * kSms) return launch_tiles<EPI, 4>(p, outputs, stream);
  return tiles > 2 * kSms ? launch_tiles<EPI, 2>(p, outputs, stream) : launch_tiles<EPI, 1>(p, outputs, stream);
}

}  // namespace

int launch_decode_linear(const void* x, const void* w, const void* bias, void* out, int M, int N, int K, int64_t sx,
                         int64_t so, int epilogue, int act, void* conv_state, const void* conv_weight,
                         const void* conv_bias, int conv_k, int conv_w_dtype, const float* row_ss, int n_ss, float eps,
                         cudaStream_t stream) {
  if (K % 32 != 0 || sx % 8 != 0 || !aligned16(x) || !aligned16(w)) return BASED_ERR_ALIGN;
  const bool two = epilogue == EPI_SWIGLU || epilogue == EPI_CONV;
  const int outputs = two ? N / 2 : N;
  if (outputs % 8 != 0 || (two && N % 2 != 0) || (row_ss && M > 16)) return BASED_ERR_SHAPE;
  LinParams p{static_cast<const __nv_bfloat16*>(x), static_cast<const __nv_bfloat16*>(w),
              static_cast<const __nv_bfloat16*>(bias), out, M, N, K, sx, so, act,
              static_cast<__nv_bfloat16*>(conv_state), conv_weight, conv_bias, conv_k, conv_w_dtype == BASED_BF16,
              row_ss, n_ss, eps, nullptr, nullptr, nullptr};
  if (epilogue == EPI_PLAIN) return launched(launch_epi<EPI_PLAIN>(p, outputs, stream));
  if (epilogue == EPI_SWIGLU) return launched(launch_epi<EPI_SWIGLU>(p, outputs, stream));
  if (epilogue == EPI_CONV) return launched(launch_epi<EPI_CONV>(p, outputs, stream));
  if (epilogue == EPI_F32) return launched(launch_epi<EPI_F32>(p, outputs, stream));
  return BASED_ERR_SHAPE;
}

int launch_decode_linear_add(const void* x, const void* w, const void* bias, int M, int N, int K, int64_t sx, float* residual,
                             const void* norm, void* out, float* ss,
                             cudaStream_t stream) {
  if (K % 32 != 0 || sx % 8 != 0 || !aligned16(x) || !aligned16(w)) return BASED_ERR_ALIGN;
  if (N % 8 != 0 || M > 16) return BASED_ERR_SHAPE;
  LinParams p{static_cast<const __nv_bfloat16*>(x), static_cast<const __nv_bfloat16*>(w),
              static_cast<const __nv_bfloat16*>(bias), out, M, N, K, sx, N, 0, nullptr, nullptr, nullptr, 0, 0,
              nullptr, 0, 0.f, residual, ss, static_cast<const __nv_bfloat16*>(norm)};
  return launched(launch_epi<EPI_ADD>(p, N, stream));
}

}  // namespace based
