// Linear layers of a prompt in float32, on the tensor cores: y[M, N] = x[M, K] W[N, K]^T (+ bias), W in up to four matrices one after the
// other (the projections of one input are one product).
//
// A row of x or W is scaled by the power of two that takes its largest value to [1, 2), and a value's 24 significant bits are exactly the
// sum of three bf16 values of 8 bits, each what is left rounded to nearest: h + m + l, |m| <= 2^-8 and |l| <= 2^-17 of the value's power of
// two.  A product is then nine bf16 products, exact in the tensor cores' float32 sums; six of them are computed (h h, h m, m h, m m, h l,
// l h).  The other three come to at most 2^-24 of the product, of either sign: as much as rounding it once.  (Values merely cut leave 2^-21,
// always of the product's sign.)  Values below 2^-110 of their row's largest lose bits of m and l, which end at 2^-133 of it; small and
// large rows lose none, and nothing overflows that the result does not.  What is left is the sum: the tensor cores cut a sum's low bits at
// every step (1e-9 K of it at K = 1024), so the h h products leave TMEM after every 128 values of K and are added up in registers, rounded
// to nearest; the small ones, 2^-8 of them and less, stay in an accumulator of their own.  Relative error against 64 bits (2-norm, normal
// values, K = 256 to 1024) 1.25e-7 to 1.4e-7, the library's float32 product 2.9e-7 to 5.8e-7; the largest of an element in 2^-24 of its
// products' absolute sum 0.8 to 2.2 and 4.5 to 6.7, all of one sign (K = 72 to 2048) 2.0 to 5.3 and 10 to 52.
//
// linear_f32_split_kernel writes the three planes of x and W; linear_f32_kernel multiplies them: a pair of CTAs per tile, a TMA producer, an
// MMA issuer, eight warps that add.  The library's float32 product runs on the CUDA cores; us with it / here, one after the other in a graph
// (rows; outputs x K): 512 29 / 25, 2048 83 / 28.5, 8192 329 / 89 (1024 x 1024); 2048 141 / 42 (1536 x 1024); 2048 24.5 / 17.4 (512 x 512).  Of
// the 28.5, 6 are the split, 19 the products: 1.2 a chunk of 64 values of K, 1.0 of it products at full rate.  The rows' scales take 1 to 2
// of it (27 without): a row's largest value is found before its first is split, and each output is multiplied by two powers of two.
#include "common.cuh"
#include "tc_pair.cuh"

#include <algorithm>

namespace based {
namespace {

using namespace tc;

__device__ unsigned int g_tc_status_f32;

constexpr int kBM = 256, kBK = 64, kStages = 2, kRun = 2, kAddWarps = 8, kThreads = (kAddWarps + 2) * 32, kMaxParts = 5, kHeld = 4;
constexpr uint32_t kPlane = 128 * kBK * 2, kSlab = 4096;   // bytes of a plane's 128 rows in a stage; of 32 x 32 outputs
constexpr unsigned kCode = 1u << 13;

struct SplitParams {   // up to kMaxParts matrices of K columns: row r of part i goes to row at[i] + r of its planes
  const float* src[kMaxParts];
  __nv_bfloat16* dst[kMaxParts];
  int64_t stride[kMaxParts], plane[kMaxParts];   // elements between rows of src, between planes of dst
  int first[kMaxParts + 1], at[kMaxParts];       // rows before the part, row of its first in dst
  float2* power[kMaxParts];                      // of the planes' rows: the power of two to multiply them by, in two factors of some half of it
  int K, parts;
};

// A warp splits a row.  Not a finite number: all in h (the products of its m and l would be NaN where the sum is infinite).
__global__ void __launch_bounds__(256) linear_f32_split_kernel(const __grid_constant__ SplitParams p) {
  pdl_trigger();
  pdl_wait();
  const int groups = p.K / 8, lane = threadIdx.x & 31;
  int row = blockIdx.x * 8 + (threadIdx.x >> 5);
  if (row >= p.first[p.parts]) return;
  int part = 0;
  while (row >= p.first[part + 1]) ++part;
  row -= p.first[part];
  const float4* src = reinterpret_cast<const float4*>(p.src[part] + row * p.stride[part]);
  uint32_t most = 0;   // of the finite values' bits without the sign
  auto see = [&](const float4& v) {
    for (float e : {v.x, v.y, v.z, v.w}) {
      const uint32_t x = __float_as_uint(e) & 0x7fffffffu;
      most = max(most, x < 0x7f800000u ? x : 0u);
    }
  };
  // up to 1024 values of a row stay in registers; what is behind them is read again
  float4 held[2 * kHeld];
#pragma unroll
  for (int i = 0; i < kHeld; ++i) {
    const int at = lane + 32 * i;
    held[2 * i] = held[2 * i + 1] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (at < groups) {
      held[2 * i] = src[2 * at];
      held[2 * i + 1] = src[2 * at + 1];
    }
  }
  for (int at = 64 * kHeld + lane; at < 2 * groups; at += 32) see(src[at]);
#pragma unroll
  for (int i = 0; i < 2 * kHeld; ++i) see(held[i]);
  most = __reduce_max_sync(0xffffffffu, most);
  const int e = most ? min(max((int)(most >> 23) - 127, -126), 126) : 0;   // 2^-e is a normal number
  const float scale = __uint_as_float((uint32_t)(127 - e) << 23);
  if (lane == 0) {   // 2^e in two factors
    const int half = e >> 1;
    p.power[part][p.at[part] + row] = make_float2(__uint_as_float((uint32_t)(127 + half) << 23), __uint_as_float((uint32_t)(127 + e - half) << 23));
  }
  __nv_bfloat16* dst = p.dst[part] + (int64_t)(p.at[part] + row) * p.K;
  auto split = [&](int at, const float4& lo, const float4& hi) {
    const float v[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
    float h[8], m[8], l[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float x = v[j] * scale;
      h[j] = __bfloat162float(__float2bfloat16_rn(x));
      const float r = fabsf(x) < __int_as_float(0x7f800000) ? x - h[j] : 0.f;
      m[j] = __bfloat162float(__float2bfloat16_rn(r));
      l[j] = r - m[j];
    }
    auto pack = [](const float (&x)[8]) { return make_uint4(pack_bf16(x[0], x[1]), pack_bf16(x[2], x[3]), pack_bf16(x[4], x[5]), pack_bf16(x[6], x[7])); };
    *reinterpret_cast<uint4*>(dst + 8 * at) = pack(h);
    *reinterpret_cast<uint4*>(dst + p.plane[part] + 8 * at) = pack(m);
    *reinterpret_cast<uint4*>(dst + 2 * p.plane[part] + 8 * at) = pack(l);
  };
#pragma unroll
  for (int i = 0; i < kHeld; ++i)
    if (lane + 32 * i < groups) split(lane + 32 * i, held[2 * i], held[2 * i + 1]);
  for (int at = 32 * kHeld + lane; at < groups; at += 32) split(at, src[2 * at], src[2 * at + 1]);
}

struct F32Params {
  int M, N, K, col_tiles;
  const float2 *px, *pw;   // powers of the rows of x and of W
  const float* bias;
  unsigned int* status;
};

// WIDE: 256 x 256 tiles, a product of every pair of planes.  Not: 256 x 128 tiles for fewer of them; a product of 128 columns takes nearly
// the time of one of 256 (120 cycles of 128: the left operand's bytes are the same), so [h h | h m] and [m h | m m] are one product each,
// of W's planes h and m side by side (six products of 128 columns: 1.6 us a chunk instead of 1.2).
template <bool WIDE>
struct F32Tile {
  static constexpr int kBN = WIDE ? 256 : 128, kSpan = kBN / 2;   // columns of a tile, of a warp
  // right operand in shared memory, per CTA.  WIDE: 128 rows of each plane.  Not: 128 rows of h (first CTA) or m (second); 64 of h; 64 of l
  static constexpr uint32_t kRight = WIDE ? 3 * kPlane : 2 * kPlane, kStage = 3 * kPlane + kRight;
  static constexpr uint32_t kSmem = kStages * kStage + 8 * (2 * kStages + 2) + 1024;
  static_assert(kSmem <= 227 * 1024 && kAddWarps * kSpan / 32 * kSlab <= kStages * kStage, "tile");
};

template <bool WIDE>
__global__ void __launch_bounds__(kThreads, 1)
    linear_f32_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_half,
                      const __grid_constant__ CUtensorMap map_out, const F32Params p) {
  using T = F32Tile<WIDE>;
  constexpr int kBN = T::kBN, kSpan = T::kSpan;
  constexpr uint32_t kStage = T::kStage;
  extern __shared__ uint8_t smem_raw[];
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag;
  __shared__ __align__(16) float2 powers[kAddWarps][kSpan];   // of a warp's columns
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u, bars = base + kStages * kStage;
  const uint32_t full = bars, empty = full + 8 * kStages, sum_full = empty + 8 * kStages, sum_empty = sum_full + 8;
  const uint32_t rank = cluster_rank();
  const int tile = blockIdx.x >> 1, m0 = tile / p.col_tiles * kBM + (int)rank * 128, n0 = tile % p.col_tiles * kBN;
  const int chunks = (p.K + kBK - 1) / kBK, runs = (chunks + kRun - 1) / kRun;
  if (tid == 0) {
    abort_flag = 0;
    for (int i = 0; i < kStages; ++i) {
      mbar_init(full + 8 * i, 1);
      mbar_init(empty + 8 * i, 1);
    }
    mbar_init(sum_full, 1);
    mbar_init(sum_empty, 2 * kAddWarps);
    fence_mbar_init();
    tma::prefetch_map(&map_x);
    tma::prefetch_map(&map_w);
  }
  pdl_trigger();
  pdl_wait();
  // TMEM.  WIDE: the h h sums of a chunk, the small products' sums.  Not: h h of a chunk, h m + m h of a chunk, the rest.
  if (warp == kAddWarps + 1) alloc<2>(smem_u32(&tmem_slot), 512);
  fence_before_sync();
  __syncthreads();
  cluster_sync();
  fence_after_sync();
  const uint32_t tmem = tmem_slot;
  if (warp == kAddWarps) {   // ---- TMA producer
    if (elect_one_sync()) {
      int s = 0;
      uint32_t phase = 0;
      for (int c = 0; c < chunks; ++c) {
        mbar_wait_bounded<false>(empty + 8 * s, phase ^ 1, &abort_flag, p.status, kCode);
        const uint32_t at = base + s * kStage, right = at + 3 * kPlane, bar = map_rank(full + 8 * s, 0);
        if (rank == 0) tma::mbar_expect_tx(full + 8 * s, 2 * kStage);
        for (int i = 0; i < 3; ++i) load_pair_3d(at + i * kPlane, &map_x, bar, c * kBK, m0, i);
        if constexpr (WIDE) {
          for (int i = 0; i < 3; ++i) load_pair_3d(right + i * kPlane, &map_w, bar, c * kBK, n0 + (int)rank * 128, i);
        } else {
          load_pair_3d(right, &map_w, bar, c * kBK, n0, (int)rank);
          load_pair_3d(right + kPlane, &map_half, bar, c * kBK, n0 + (int)rank * 64, 0);
          load_pair_3d(right + kPlane + kPlane / 2, &map_half, bar, c * kBK, n0 + (int)rank * 64, 2);
        }
        if (++s == kStages) { s = 0; phase ^= 1; }
      }
      for (int i = 0; i < kStages; ++i) {   // every stage read: the last products' signals have come in
        mbar_wait_bounded<false>(empty + 8 * s, phase ^ 1, &abort_flag, p.status, kCode);
        if (++s == kStages) { s = 0; phase ^= 1; }
      }
    }
    __syncwarp();
  } else if (warp == kAddWarps + 1) {   // ---- MMA
    if (rank == 0 && elect_one_sync()) {
      constexpr uint32_t id256 = make_idesc_bf16(kBM, 256, 0, 0), id128 = make_idesc_bf16(kBM, 128, 0, 0);
      int s = 0;
      uint32_t phase = 0;
      for (int c = 0; c < chunks; ++c) {
        const bool first = c % kRun == 0, last = c % kRun == kRun - 1 || c == chunks - 1;   // of a run of chunks
        if (first) mbar_wait_bounded<false>(sum_empty, (c / kRun & 1) ^ 1, &abort_flag, p.status, kCode);
        mbar_wait_bounded<false>(full + 8 * s, phase, &abort_flag, p.status, kCode);
        fence_after_sync();
        const uint32_t left = base + s * kStage, right = left + 3 * kPlane;
        // the stage's products of two tiles; `fresh`: the first overwrites what the accumulator held
        auto product = [&](uint32_t d, uint32_t a, uint32_t b, uint32_t idesc, bool fresh) {
          const uint64_t da = make_smem_desc_sw128(a, 16, 1024), db = make_smem_desc_sw128(b, 16, 1024);
#pragma unroll
          for (int k = 0; k < kBK / 16; ++k) mma<2>(d, da + 2 * k, db + 2 * k, idesc, k > 0 || !fresh);
        };
        if constexpr (WIDE) {
          constexpr int kLeft[5] = {0, 1, 1, 0, 2}, kRight[5] = {1, 0, 1, 2, 0};   // planes of x and W
          product(tmem, left, right, id256, first);
          if (last) commit<2>(sum_full);
#pragma unroll
          for (int i = 0; i < 5; ++i) product(tmem + 256, left + kLeft[i] * kPlane, right + kRight[i] * kPlane, id256, c == 0 && i == 0);
        } else {
          const uint32_t h64 = right + kPlane, l64 = h64 + kPlane / 2;
          if (c == 0) product(tmem + 256, left, l64, id128, true);
          product(tmem, left, right, id256, first);
          product(tmem + 128, left + kPlane, right, id256, false);
          if (last) commit<2>(sum_full);
          if (c > 0) product(tmem + 256, left, l64, id128, false);
          product(tmem + 256, left + 2 * kPlane, h64, id128, false);
        }
        commit<2>(empty + 8 * s);
        if (++s == kStages) { s = 0; phase ^= 1; }
      }
      mbar_wait_bounded<false>(sum_empty, (runs & 1) ^ 1, &abort_flag, p.status, kCode);
      commit<2>(sum_full);   // the accumulator that stayed to the end
    }
    __syncwarp();
  } else {   // ---- sums: rows of the warp's quadrant, half of the columns
    const int part = (warp >> 2) * kSpan;
    const uint32_t at = tmem + ((uint32_t)(warp & 3) << 21) + part, done = map_rank(sum_empty, 0);
    const float inf = __int_as_float(0x7f800000);
    const int own = m0 + (warp & 3) * 32 + lane;
    const float2 px = own < p.M ? p.px[own] : make_float2(1.f, 1.f);
    for (int i = lane; i < kSpan; i += 32) powers[warp][i] = n0 + part + i < p.N ? p.pw[n0 + part + i] : make_float2(1.f, 1.f);
    __syncwarp();
    float sum[kSpan];
#pragma unroll
    for (int i = 0; i < kSpan; ++i) sum[i] = 0.f;
    for (int c = 0; c < runs; ++c) {
      mbar_wait_bounded(sum_full, c & 1, &abort_flag, p.status, kCode);
      fence_after_sync();
#pragma unroll
      for (int j = 0; j < kSpan; j += 16) {
        uint32_t r[16], q[16];
        tmem_ld16(at + j, r);
        if constexpr (!WIDE) tmem_ld16(at + 128 + j, q);
        tmem_ld_wait();
        if (j == kSpan - 16) {
          fence_before_sync();
          __syncwarp();
          if (lane == 0) arrive_at(done);
        }
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const float big = __uint_as_float(r[i]);
          if constexpr (WIDE) sum[j + i] += big;
          else sum[j + i] += fabsf(big) < inf ? big + __uint_as_float(q[i]) : big;   // infinite: the small products may be NaN
        }
      }
    }
    mbar_wait_bounded(sum_full, runs & 1, &abort_flag, p.status, kCode);
    fence_after_sync();
    // All products are done, so the stages are free: 32 rows x 32 columns at a time through them, out by TMA.
    const int row0 = m0 + (warp & 3) * 32;
#pragma unroll
    for (int j = 0; j < kSpan / 32; ++j) {
      uint32_t r[32];
      tmem_ld32(at + 256 + 32 * j, r);
      tmem_ld_wait();
      const uint32_t slab = base + (warp * (kSpan / 32) + j) * kSlab;
      const int c0 = n0 + part + 32 * j;
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        float y[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int col = 4 * q + i;
          const float big = sum[32 * j + col];
          const float2 pw = powers[warp][32 * j + col];
          // as one rounding: the factors are near one another, so where the first product is subnormal the second is nothing
          y[i] = (fabsf(big) < inf ? big + __uint_as_float(r[col]) : big) * (px.x * pw.x) * (px.y * pw.y);
          if (p.bias && c0 + col < p.N) y[i] += p.bias[c0 + col];
        }
        st_shared16(slab + tma::sw128_offset(lane, q), __float_as_uint(y[0]), __float_as_uint(y[1]), __float_as_uint(y[2]), __float_as_uint(y[3]));
      }
      fence_proxy_async();
      __syncwarp();
      if (lane == 0 && c0 < p.N && row0 < p.M) {
        store_2d(&map_out, slab, c0, row0);
        bulk_commit();
      }
    }
    if (lane == 0) bulk_wait_all();
    __syncwarp();
  }
  fence_before_sync();
  __syncthreads();
  cluster_sync();
  fence_after_sync();
  if (warp == kAddWarps + 1) dealloc<2>(tmem, 512);
}

template <bool WIDE>
int run_f32(F32Params p, const void* px, const void* pw, float* out, cudaStream_t stream) {
  using T = F32Tile<WIDE>;
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
      e = cudaGetSymbolAddress(reinterpret_cast<void**>(&addr), g_tc_status_f32);
      if (e != cudaSuccess) return (int)e;
      e = cudaFuncSetAttribute(linear_f32_kernel<WIDE>, cudaFuncAttributeMaxDynamicSharedMemorySize, T::kSmem);
      if (e != cudaSuccess) return (int)e;
      status[dev] = addr;
    }
    p.status = status[dev];
  }
  p.col_tiles = (p.N + T::kBN - 1) / T::kBN;
  CUtensorMap mx, mw, mh, mo;
  int rc = tma::encode_planes(&mx, px, p.K, p.M, 3, 128);
  if (rc == 0) rc = tma::encode_planes(&mw, pw, p.K, p.N, 3, 128);
  if (rc == 0) rc = tma::encode_planes(&mh, pw, p.K, p.N, 3, 64);
  if (rc == 0) rc = tma::encode_2d(&mo, out, true, p.N, p.M, p.N, 32, 32);
  if (rc != 0) return rc;
  const int64_t tiles = (int64_t)((p.M + kBM - 1) / kBM) * p.col_tiles;
  if (tiles > 1 << 30) return BASED_ERR_TOO_LARGE;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = 2;
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(2 * tiles));
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = T::kSmem;
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  return launched((int)cudaLaunchKernelEx(&cfg, linear_f32_kernel<WIDE>, mx, mw, mh, mo, p));
}

// three planes of bf16, and a row's power of two
size_t row_bytes(int K) { return 6 * (size_t)K + sizeof(float2); }

// Rows of x that are split at a time: all of them, or whole tiles that fit in what kScratch leaves beside W (kLeast, whatever W takes), as many
// as make the fewest rounds of wide tiles over all parts.  us with all rows' planes at once
// / in parts: 32768 rows 463 / 465, 65536 896 / 922 (1536 x 1024), 665 / 738 (1024 x 1024; the parts' last rounds are not full).
constexpr size_t kScratch = (size_t)128 << 20;
constexpr int kLeast = 2048;
int rows_at_a_time(int M, int N, int K) {
  const size_t w = row_bytes(K) * N;
  const int64_t fit = std::max<int64_t>(w < kScratch ? (kScratch - w) / row_bytes(K) : 0, kLeast);
  if (M <= fit) return M;
  const int64_t most = fit / kBM, all = ((int64_t)M + kBM - 1) / kBM, cols = (N + 255) / 256;   // tiles
  int64_t best = most, least = INT64_MAX;
  for (int64_t t = most; t > most / 2; --t) {
    const int64_t cost = all / t * ((t * cols + 73) / 74) + (all % t * cols + 73) / 74;
    if (cost < least) { best = t; least = cost; }
  }
  return (int)(best * kBM);
}

}  // namespace

int read_tc_status_f32(unsigned int* out, int reset) {
  const cudaError_t e = cudaMemcpyFromSymbol(out, g_tc_status_f32, sizeof(unsigned int));
  if (e != cudaSuccess) return (int)e;
  if (reset && *out != 0) {
    const unsigned int zero = 0;
    return (int)cudaMemcpyToSymbol(g_tc_status_f32, &zero, sizeof(zero));
  }
  return 0;
}

size_t linear_f32_scratch_bytes(int M, int N, int K) { return row_bytes(K) * ((size_t)rows_at_a_time(M, N, K) + N); }

int launch_linear_f32(const float* x, const float* const* w, const int* rows, int parts, const float* bias, float* out, int M, int N, int K, int64_t sx,
                      void* scratch, size_t scratch_bytes, cudaStream_t stream) {
  if (K % 8 != 0 || N % 4 != 0) return BASED_ERR_SHAPE;
  if (sx % 4 != 0 || !aligned16(x) || !aligned16(out) || !aligned16(scratch)) return BASED_ERR_ALIGN;
  if (scratch_bytes < linear_f32_scratch_bytes(M, N, K)) return BASED_ERR_SCRATCH;
  const int step = rows_at_a_time(M, N, K);
  if (((int64_t)step + N + 7) / 8 > 2147483647LL / 8) return BASED_ERR_TOO_LARGE;
  for (int i = 0; i < parts; ++i)
    if (!aligned16(w[i])) return BASED_ERR_ALIGN;
  __nv_bfloat16 *px = static_cast<__nv_bfloat16*>(scratch), *pw = px + 3 * (size_t)step * K;
  float2 *power_w = reinterpret_cast<float2*>(pw + 3 * (size_t)N * K), *power_x = power_w + N;
  for (int64_t m0 = 0; m0 < M; m0 += step) {   // W is split with the first rows; a launch waits for the one before, so px is free again
    const int m = (int)std::min<int64_t>(step, M - m0);
    SplitParams sp{};
    sp.K = K;
    sp.parts = 1;
    sp.src[0] = x + m0 * sx; sp.dst[0] = px; sp.stride[0] = sx; sp.plane[0] = (int64_t)m * K; sp.first[1] = m; sp.power[0] = power_x;
    for (int i = 0, at = 0; i < parts && m0 == 0; at += rows[i++]) {
      sp.parts = i + 2;
      sp.src[i + 1] = w[i]; sp.dst[i + 1] = pw; sp.stride[i + 1] = K; sp.plane[i + 1] = (int64_t)N * K; sp.power[i + 1] = power_w;
      sp.at[i + 1] = at; sp.first[i + 2] = m + at + rows[i];
    }
    int rc = launch_pdl(linear_f32_split_kernel, dim3((unsigned)((sp.first[sp.parts] + 7) / 8)), dim3(256), 0, stream, sp);
    if (rc != 0) return launched(rc);
    // the wide tile has more products to a byte, the other one fills the chip sooner: 2.15 and 1.2 us a round for 64 values of K
    const int64_t rounds = (m + kBM - 1) / kBM, wide = (rounds * ((N + 255) / 256) + 73) / 74, narrow = (rounds * ((N + 127) / 128) + 73) / 74;
    const F32Params p{m, N, K, 0, power_x, power_w, bias, nullptr};
    float* y = out + m0 * N;
    rc = wide * 215 <= narrow * 120 ? run_f32<true>(p, px, pw, y, stream) : run_f32<false>(p, px, pw, y, stream);
    if (rc != 0) return rc;
  }
  return 0;
}

}  // namespace based
