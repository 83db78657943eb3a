// A layer's token input for the rows of a prompt in one launch: residual += norm(W_proj (gelu_tanh(W_gate x) * table[token, column ..])) *
// norm_weight, and the new residual in bf16.  bf16 operands, fp32 sums in TMEM; nothing is rounded between the steps but the middle
// product's operand.
//
// Bound by the stream: 12 bytes an element (x read, the residual read and written, its bf16 form written), while the products are 64 wide
// on one side.  As two library products, a gate and a norm it was four launches and 20 bytes more.  A CTA takes 128 rows at a time: the
// first product (K = the model's width, 64 columns) through a ring of TMA stages; its rows, gated, become the second product's left
// operand in shared memory.  That one is taken twice, 128 columns at a time through two TMEM buffers: once for the sums of squares, once
// for the output, because a row of it (1024 columns and more) fits neither TMEM nor registers and 64 multiply-adds an element are
// cheaper than keeping it.  Where there are fewer row tiles than SMs each is shared out by its output columns; the first product and
// the sums of squares are then made by every share, at the price of more reads of L2.  The stream comes and goes by TMA through slabs of
// a warp's own, as in prompt_linear's ADD.
// Measured at width 1024, 64 values, us as four launches / here, one after the other in a graph: 512 rows 10.0 / 12.6, 2048 12.7 / 13.2, 4096
// 16.4 / 16.3, 6001 19.8 / 19.4, 7168 24.0 / 22.4, 18944 57 / 48.  Up to some 4000 rows a prompt of 27 such layers is bound by its launches
// instead: 5.55 to 5.9 ms / 4.85 to 5.2 (6001: 6.23 / 6.09); hence also the fewer rows, from where one round of token_side.cu's clusters ends
// (128 rows there 6.8 us, 12.4 here).  Three stages and a third slab of the stream: 13 at 128 rows, 19.9 at 6001.
#include "common.cuh"
#include "seq_common.cuh"
#include "tc_pair.cuh"

#include <algorithm>

namespace based {
namespace {

using namespace tc;

__device__ unsigned int g_tc_status_side;

constexpr int kWarps = 8, kThreads = (kWarps + 2) * 32, kStages = 4, kBK = 64, kValues = 64, kCols = 128, kRes = 2;
constexpr uint32_t kA = 128 * kBK * 2, kStage = kA + kValues * kBK * 2, kSlab = 4096, kStaging = (kRes + 1) * kSlab;   // bytes; the last two of a warp
constexpr uint32_t kLeft = kStages * kStage, kSlabs = kLeft + 128 * kValues * 2, kBars = kSlabs + kWarps * kStaging;
constexpr uint32_t kSmem = kBars + 8 * (2 * kStages + 6 + kRes * kWarps) + 1024;
constexpr unsigned kCode = 1u << 15;
static_assert(kCols * kValues * 2 <= kStage && kSmem <= 226 * 1024, "shared memory");

struct SideParams {
  const int64_t* tokens;
  const __nv_bfloat16 *table, *norm;
  int64_t V, st;       // rows of the table, elements between them (at the layer's column already)
  int M, W, n, items, parts, col_tiles, part_tiles;   // an item: 128 rows and one of `parts` equal shares of the column tiles
  float eps;
  unsigned int* status;
};

__global__ void __launch_bounds__(kThreads, 1)
    token_side_tc_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_gate, const __grid_constant__ CUtensorMap map_proj,
                         const __grid_constant__ CUtensorMap map_res, const __grid_constant__ CUtensorMap map_out, const SideParams p) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag;
  __shared__ float squares[2][128];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u, left = base + kLeft, bars = base + kBars;
  const uint32_t full = bars, empty = full + 8 * kStages, mid_full = empty + 8 * kStages, left_full = mid_full + 8, acc_full = left_full + 8,
                 acc_empty = acc_full + 16, res_full = acc_empty + 16;
  if (tid == 0) {
    abort_flag = 0;
    for (int i = 0; i < kStages; ++i) {
      mbar_init(full + 8 * i, 1);
      mbar_init(empty + 8 * i, 1);
    }
    mbar_init(mid_full, 1);
    mbar_init(left_full, kWarps);
    for (int i = 0; i < 2; ++i) {
      mbar_init(acc_full + 8 * i, 1);
      mbar_init(acc_empty + 8 * i, kWarps);
    }
    for (int i = 0; i < kRes * kWarps; ++i) mbar_init(res_full + 8 * i, 1);
    fence_mbar_init();
    tma::prefetch_map(&map_x);
    tma::prefetch_map(&map_gate);
    tma::prefetch_map(&map_proj);
  }
  pdl_trigger();
  pdl_wait();
  if (warp == kWarps + 1) tmem_alloc(smem_u32(&tmem_slot), 512);   // 64 columns of the first product, two buffers of 128 of the second
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  const uint32_t tmem = tmem_slot, second = tmem + kValues;
  const int kblocks = (p.W + kBK - 1) / kBK;

  if (warp == kWarps) {   // ---- TMA producer
    if (elect_one_sync()) {
      int s = 0;
      uint32_t phase = 0;
      auto stage = [&](uint32_t bytes) {
        mbar_wait_bounded<false>(empty + 8 * s, phase ^ 1, &abort_flag, p.status, kCode);
        tma::mbar_expect_tx(full + 8 * s, bytes);
        return base + s * kStage;
      };
      auto advance = [&] {
        if (++s == kStages) { s = 0; phase ^= 1; }
      };
      for (int t = blockIdx.x; t < p.items; t += gridDim.x) {
        const int row0 = t / p.parts * 128, first = t % p.parts * p.part_tiles, last = min(first + p.part_tiles, p.col_tiles);
        for (int kb = 0; kb < kblocks; ++kb) {
          const uint32_t at = stage(kStage);
          load_2d<1>(at, &map_x, full + 8 * s, kb * kBK, row0);
          load_2d<1>(at + kA, &map_gate, full + 8 * s, kb * kBK, 0);
          advance();
        }
        for (int i = 0; i < p.col_tiles + last - first; ++i) {
          const uint32_t at = stage(kCols * kValues * 2);
          load_2d<1>(at, &map_proj, full + 8 * s, 0, (i < p.col_tiles ? i : i - p.col_tiles + first) * kCols);
          advance();
        }
      }
      for (int i = 0; i < kStages; ++i) {   // every stage read: the last products' signals have come in
        mbar_wait_bounded<false>(empty + 8 * s, phase ^ 1, &abort_flag, p.status, kCode);
        advance();
      }
    }
    __syncwarp();
  } else if (warp == kWarps + 1) {   // ---- MMA
    if (elect_one_sync()) {
      constexpr uint32_t id1 = make_idesc_bf16(128, kValues, 0, 0), id2 = make_idesc_bf16(128, kCols, 0, 0);
      int s = 0, use = 0, it = 0;
      uint32_t phase = 0;
      auto advance = [&] {
        mma_commit(empty + 8 * s);
        if (++s == kStages) { s = 0; phase ^= 1; }
      };
      for (int t = blockIdx.x; t < p.items; t += gridDim.x, ++it) {
        const int first = t % p.parts * p.part_tiles, last = min(first + p.part_tiles, p.col_tiles);
        for (int kb = 0; kb < kblocks; ++kb) {   // (the tile before's were read when its left operand was written)
          mbar_wait_bounded<false>(full + 8 * s, phase, &abort_flag, p.status, kCode);
          fence_after_sync();
          const uint32_t at = base + s * kStage;
          const uint64_t a = make_smem_desc_sw128(at, 16, 1024), b = make_smem_desc_sw128(at + kA, 16, 1024);
#pragma unroll
          for (int k = 0; k < kBK / 16; ++k) mma_ss(tmem, a + 2 * k, b + 2 * k, id1, kb | k);
          advance();
        }
        mma_commit(mid_full);
        mbar_wait_bounded<false>(left_full, it & 1, &abort_flag, p.status, kCode);
        for (int i = 0; i < p.col_tiles + last - first; ++i, ++use) {
          mbar_wait_bounded<false>(acc_empty + 8 * (use & 1), ((use >> 1) & 1) ^ 1, &abort_flag, p.status, kCode);
          mbar_wait_bounded<false>(full + 8 * s, phase, &abort_flag, p.status, kCode);
          fence_after_sync();
          const uint64_t a = make_smem_desc_sw128(left, 16, 1024), b = make_smem_desc_sw128(base + s * kStage, 16, 1024);
#pragma unroll
          for (int k = 0; k < kValues / 16; ++k) mma_ss(second + (use & 1) * kCols, a + 2 * k, b + 2 * k, id2, k);
          advance();
          mma_commit(acc_full + 8 * (use & 1));
        }
      }
    }
    __syncwarp();
  } else {   // ---- rows of the warp's quadrant, half of the columns
    const int quad = warp & 3, half = warp >> 2;
    const uint32_t lanes = (uint32_t)quad << 21, mine = base + kSlabs + warp * kStaging, outs = mine + kRes * kSlab, res_bar = res_full + 8 * kRes * warp;
    const int steps = 2 * p.part_tiles;   // of 32 columns, in an item
    auto col_of = [&](int t, int j) { return (t % p.parts * p.part_tiles + (j >> 1)) * kCols + half * 64 + (j & 1) * 32; };
    auto row_of = [&](int t) { return t / p.parts * 128 + quad * 32; };
    auto live = [&](int t, int j) { return col_of(t, j) < p.W && row_of(t) < p.M; };
    auto next = [&](int& t, int& j) {
      do {
        if (++j == steps) { j = 0; t += gridDim.x; }
      } while (t < p.items && !live(t, j));
    };
    auto fetch = [&](int t, int j, int at) {   // by one lane: 32 columns of the stream
      tma::mbar_expect_tx(res_bar + 8 * at, kSlab);
      load_2d<1>(mine + at * kSlab, &map_res, res_bar + 8 * at, col_of(t, j), row_of(t));
    };
    int ft = blockIdx.x, fj = -1, step = 0, use = 0, it = 0, at = 0;   // at, round: step's slab, how often it has been used
    uint32_t round = 0;
    for (int i = 0; i < kRes - 1; ++i) {
      if (ft < p.items) next(ft, fj);
      if (ft < p.items && lane == 0) fetch(ft, fj, i);
    }
    for (int t = blockIdx.x; t < p.items; t += gridDim.x, ++it) {
      const int row0 = row_of(t), row = row0 + lane;
      // ---- the gate, 32 of its values
      uint4 e[4];
      {
        const int64_t tok = row < p.M ? p.tokens[row] : -1;
        const bool known = tok >= 0 && tok < p.V;
        const __nv_bfloat16* src = p.table + (known ? tok : 0) * p.st + half * 32;
#pragma unroll
        for (int q = 0; q < 4; ++q)
          e[q] = known && half * 32 + 8 * q < p.n ? *reinterpret_cast<const uint4*>(src + 8 * q) : make_uint4(0, 0, 0, 0);
      }
      mbar_wait_bounded(mid_full, it & 1, &abort_flag, p.status, kCode);
      fence_after_sync();
      {
        uint32_t r[32];
        tmem_ld32(tmem + lanes + half * 32, r);
        tmem_ld_wait();
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const uint32_t w[4] = {e[q].x, e[q].y, e[q].z, e[q].w};
          uint32_t h[4];
#pragma unroll
          for (int i = 0; i < 4; ++i)
            h[i] = pack_bf16(seq::gelu_tanh_t<__nv_bfloat16>(__uint_as_float(r[8 * q + 2 * i])) * __uint_as_float(w[i] << 16),
                             seq::gelu_tanh_t<__nv_bfloat16>(__uint_as_float(r[8 * q + 2 * i + 1])) * __uint_as_float(w[i] & 0xffff0000u));
          st_shared16(left + tma::sw128_offset(quad * 32 + lane, half * 4 + q), h[0], h[1], h[2], h[3]);
        }
      }
      fence_proxy_async();
      fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(left_full);
      // ---- the second product for its rows' sums of squares
      float ss[4] = {0.f, 0.f, 0.f, 0.f};
      for (int i = 0; i < p.col_tiles; ++i, ++use) {
        mbar_wait_bounded(acc_full + 8 * (use & 1), (use >> 1) & 1, &abort_flag, p.status, kCode);
        fence_after_sync();
        uint32_t r[2][32];
        tmem_ld32(second + lanes + (use & 1) * kCols + half * 64, r[0]);
        tmem_ld32(second + lanes + (use & 1) * kCols + half * 64 + 32, r[1]);
        tmem_ld_wait();
        fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(acc_empty + 8 * (use & 1));
#pragma unroll
        for (int k = 0; k < 64; ++k) {
          const float y = __uint_as_float(r[k >> 5][k & 31]);
          ss[k & 3] = fmaf(y, y, ss[k & 3]);
        }
      }
      squares[half][quad * 32 + lane] = (ss[0] + ss[1]) + (ss[2] + ss[3]);
      asm volatile("bar.sync %0, 64;\n" ::"r"(1 + quad) : "memory");   // the two warps of these rows
      const float rstd = rsqrtf((squares[0][quad * 32 + lane] + squares[1][quad * 32 + lane]) / (float)p.W + p.eps);
      // ---- and for the stream
      for (int j = 0; j < steps && col_of(t, j & ~1) - half * 64 < p.W; ++j) {
        const int c0 = col_of(t, j);
        const bool on = c0 < p.W && row0 < p.M;
        if (on && lane == 0) {   // what was stored a step ago has been read: its slab takes the columns that come next
          bulk_wait_read_all();
          if (ft < p.items) next(ft, fj);
          if (ft < p.items) fetch(ft, fj, at == 0 ? kRes - 1 : at - 1);
        }
        __syncwarp();
        if ((j & 1) == 0) {
          mbar_wait_bounded(acc_full + 8 * (use & 1), (use >> 1) & 1, &abort_flag, p.status, kCode);
          fence_after_sync();
        }
        uint32_t r[32];
        tmem_ld32(second + lanes + (use & 1) * kCols + half * 64 + (j & 1) * 32, r);
        tmem_ld_wait();
        if (j & 1) {
          fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive(acc_empty + 8 * (use & 1));
          ++use;
        }
        if (!on) continue;
        uint4 w[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) w[q] = *reinterpret_cast<const uint4*>(p.norm + min(c0 + 8 * q, p.W - 8));
        const uint32_t res = mine + at * kSlab, to = outs + (step & 1) * (kSlab / 2);
        mbar_wait_bounded(res_bar + 8 * at, round & 1, &abort_flag, p.status, kCode);
        float4 old[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) old[q] = ld_shared16(res + tma::sw128_offset(lane, q));
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const float was[8] = {old[2 * q].x, old[2 * q].y, old[2 * q].z, old[2 * q].w, old[2 * q + 1].x, old[2 * q + 1].y, old[2 * q + 1].z, old[2 * q + 1].w};
          const uint32_t ww[4] = {w[q].x, w[q].y, w[q].z, w[q].w};
          float z[8];
#pragma unroll
          for (int i = 0; i < 8; ++i)
            z[i] = fmaf(__uint_as_float(r[8 * q + i]) * rstd, __uint_as_float(i & 1 ? ww[i / 2] & 0xffff0000u : ww[i / 2] << 16), was[i]);
          st_shared16(res + tma::sw128_offset(lane, 2 * q), __float_as_uint(z[0]), __float_as_uint(z[1]), __float_as_uint(z[2]), __float_as_uint(z[3]));
          st_shared16(res + tma::sw128_offset(lane, 2 * q + 1), __float_as_uint(z[4]), __float_as_uint(z[5]), __float_as_uint(z[6]), __float_as_uint(z[7]));
          st_shared16(to + (uint32_t)lane * 64u + (uint32_t)((q ^ ((lane >> 1) & 3)) << 4), pack_bf16(z[0], z[1]), pack_bf16(z[2], z[3]), pack_bf16(z[4], z[5]),
                      pack_bf16(z[6], z[7]));
        }
        fence_proxy_async();
        __syncwarp();
        if (lane == 0) {
          store_2d(&map_res, res, c0, row0);
          store_2d(&map_out, to, c0, row0);
          bulk_commit();
        }
        ++step;
        if (++at == kRes) { at = 0; ++round; }
      }
    }
    if (lane == 0) bulk_wait_all();
    __syncwarp();
  }
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  if (warp == kWarps + 1) tmem_dealloc(tmem, 512);
}

}  // namespace

int read_tc_status_side(unsigned int* out, int reset) {
  const cudaError_t e = cudaMemcpyFromSymbol(out, g_tc_status_side, sizeof(unsigned int));
  if (e != cudaSuccess) return (int)e;
  if (reset && *out != 0) {
    const unsigned int zero = 0;
    return (int)cudaMemcpyToSymbol(g_tc_status_side, &zero, sizeof(zero));
  }
  return 0;
}

// BASED_ERR_IMPL: sizes or strides this kernel does not take.
int launch_token_side_tc(const void* x, int64_t sx, const int64_t* tokens, const void* gate, const void* proj, const void* table, int64_t V, int64_t st,
                         int64_t column, const void* norm, float* residual, void* out, int M, int W, int n, float eps, cudaStream_t stream) {
  if (n % 8 != 0 || n > kValues || W % 8 != 0 || sx % 8 != 0 || st % 8 != 0 || column % 8 != 0 || M > 2147483647 - 128) return BASED_ERR_IMPL;
  for (const void* q : {x, gate, proj, table, norm, static_cast<const void*>(residual), static_cast<const void*>(out)})
    if (!aligned16(q)) return BASED_ERR_IMPL;
  SideParams p{tokens, static_cast<const __nv_bfloat16*>(table) + column, static_cast<const __nv_bfloat16*>(norm), V, st, M, W, n, 0, 1,
               (W + kCols - 1) / kCols, 0, eps, nullptr};
  const int row_tiles = (M + 127) / 128;
  p.parts = std::max(1, std::min(148 / row_tiles, p.col_tiles));
  p.part_tiles = (p.col_tiles + p.parts - 1) / p.parts;
  p.parts = (p.col_tiles + p.part_tiles - 1) / p.part_tiles;
  p.items = row_tiles * p.parts;
  constexpr int kMaxDevices = 64;
  static std::mutex mu;
  static unsigned int* status[kMaxDevices] = {};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return (int)e;
  if (dev < 0 || dev >= kMaxDevices) return BASED_ERR_TOO_LARGE;
  {
    std::lock_guard<std::mutex> lock(mu);
    if (status[dev] == nullptr) {
      unsigned int* addr = nullptr;
      e = cudaGetSymbolAddress(reinterpret_cast<void**>(&addr), g_tc_status_side);
      if (e == cudaSuccess) e = cudaFuncSetAttribute(token_side_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem);
      if (e != cudaSuccess) return (int)e;
      status[dev] = addr;
    }
    p.status = status[dev];
  }
  CUtensorMap mx, mg, mp, mr, mo;
  int rc = tma::encode_2d(&mx, x, false, W, M, sx, kBK, 128);
  if (rc == 0) rc = tma::encode_2d(&mg, gate, false, W, n, W, kBK, kValues);
  if (rc == 0) rc = tma::encode_2d(&mp, proj, false, n, W, n, kValues, kCols);
  if (rc == 0) rc = tma::encode_2d(&mr, residual, true, W, M, W, 32, 32);
  if (rc == 0) rc = tma::encode_2d(&mo, out, false, W, M, W, 32, 32);
  if (rc != 0) return BASED_ERR_IMPL;
  return launched(launch_pdl(token_side_tc_kernel, dim3((unsigned)std::min(p.items, 148)), dim3(kThreads), kSmem, stream, mx, mg, mp, mr, mo, p));
}

}  // namespace based
