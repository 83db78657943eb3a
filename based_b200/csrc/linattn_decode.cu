// Recurrent decode step of Taylor linear attention: feature map, rank-1 state update and
// normalised readout in ONE pass over the state (HBM-bound: the state is read once and
// written once).
//
// Replaces TaylorExp.forward on q, k (based/models/mixers/linear_attention.py:67-75, called
// at :139) and LinearAttention.recurrent_forward (:230-251) up to out_proj.
//
// State layout (unchanged from the reference, linear_attention.py:261-266):
//   kv_state [B, H, 1, dv, 273]  feature index fastest, k_state [B, H, 1, 1, 273].
// One row of 273 elements is not 16-byte aligned, but RPG = 16/sizeof(state) consecutive rows
// are exactly 273 sixteen-byte vectors.  A warp owns such a row group: 128-bit coalesced
// loads, FMA, 128-bit stores, and a per-row dot product with phi(q) reduced by shuffles.
#include "common.cuh"

namespace based {
namespace {

// Bound by HBM with fp32 states, by instructions with bf16 ones.  A block's loads of its first row groups and of the row of sums are in
// flight while it builds the feature tables; the 32 vectors of a step lie in two rows known at compile time, so a product is added to one
// of two sums (to one of all rows of a group: 16 instructions more a vector for bf16).
// CTA size: 192 threads, four CTAs per SM, for many (batch, head) blocks with fp32 states, 128 and five with bf16 ones (their row
// groups are half as many).  us at B=256, H=16, dv=64, one launch after the other in a graph (the bytes at the HBM rate; a lone call takes
// some 5 more): fp32 93 (89), with three CTAs, their first loads behind the tables, 102.5; bf16 73 (45), 163 then; dv=112 161 (155) and 122
// (77).  256 threads (two per SM) for few blocks, where one block's latency counts (B=16, H=16, bf16 state 7.5); 512 where every block has
// an SM of its own and more than eight row groups (B=8, H=16, dv=112, bf16 state, in a chain of launches: 10.5 us with 256, 6.6 with 512).
constexpr int kTab = 288;     // table length: 273 + wrap-around + padding, multiple of 4
constexpr int kVecPerGroup = kExpandedDim;  // 273 vectors of 16 B per row group
constexpr int kIters = (kVecPerGroup + 31) / 32;  // 9

template <typename ST> struct VecOps;
template <> struct VecOps<float> {
  static constexpr int kVec = 4;
  static __device__ __forceinline__ void unpack(const uint4& r, float* e) {
    e[0] = __uint_as_float(r.x); e[1] = __uint_as_float(r.y);
    e[2] = __uint_as_float(r.z); e[3] = __uint_as_float(r.w);
  }
  // e as it is stored, rounded in place
  static __device__ __forceinline__ uint4 pack(float* e) {
    return make_uint4(__float_as_uint(e[0]), __float_as_uint(e[1]), __float_as_uint(e[2]), __float_as_uint(e[3]));
  }
  static __device__ __forceinline__ float round(float x) { return x; }
};
template <> struct VecOps<__nv_bfloat16> {
  static constexpr int kVec = 8;
  static __device__ __forceinline__ void unpack(const uint4& r, float* e) {
    const uint32_t w[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      e[2 * i] = __uint_as_float(w[i] << 16);
      e[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
    }
  }
  static __device__ __forceinline__ uint4 pack(float* e) {
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const __nv_bfloat162 pair = __floats2bfloat162_rn(e[2 * i], e[2 * i + 1]);
      w[i] = *reinterpret_cast<const uint32_t*>(&pair);
    }
    unpack(make_uint4(w[0], w[1], w[2], w[3]), e);
    return make_uint4(w[0], w[1], w[2], w[3]);
  }
  static __device__ __forceinline__ float round(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }
};

template <typename IO, typename ST, int kThreads>
__global__ void __launch_bounds__(kThreads, kThreads == 128 ? 5 : kThreads == 192 ? 4 : kThreads == 256 ? 2 : 1)
linattn_decode_kernel(const IO* q, const IO* k, const IO* v,
                      IO* y, ST* kv_state, ST* k_state,
                      int H, int dv, Strides2 sq, Strides2 sk, Strides2 sv, Strides2 sy, float eps) {
  pdl_trigger();
  // Few blocks: their state into L2 before the kernel ahead has ended; whole 16-byte vectors.  More blocks than two per SM start behind others,
  // where it only asks twice (a mixer's step, 16 heads of 64: 16 rows 15.5 -> 14.8 us with it, 40 rows 30.6 -> 32.8).
  if (kThreads > 192 && threadIdx.x < 32 && gridDim.x <= 2 * 148) {
    const uint32_t bytes = dv * kExpandedDim * sizeof(ST), piece = (bytes / 32 + 15) & ~15u, at = threadIdx.x * piece;
    if (at < bytes) prefetch_l2(reinterpret_cast<const char*>(kv_state) + (size_t)blockIdx.x * bytes + at, min(piece, bytes - at));
  }
  pdl_wait();
  using VO = VecOps<ST>;
  constexpr int VEC = VO::kVec;
  constexpr int RPG = VEC;  // rows per 16-byte-aligned group
  constexpr int kWarps = kThreads / 32;

  // s_t*[s][i] = phi[(i + s) % 273]: four shifted copies so that phi[f0 .. f0+VEC) can be
  // fetched with aligned 128-bit shared loads whatever f0 mod 4 is.
  __shared__ __align__(16) float s_tq[4][kTab];
  __shared__ __align__(16) float s_tk[4][kTab];
  __shared__ float s_x[2][kFeatureDim];
  __shared__ float s_v[128];
  __shared__ float s_num[128];
  __shared__ float s_den;

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int bh = blockIdx.x;
  const int b = bh / H, h = bh - b * H;

  // a warp's first rows of the state are in flight while the feature tables are built
  const int ngroups = dv / RPG;
  uint4 r[kIters];
  auto fetch = [&](int g) {
    const uint4* base = reinterpret_cast<const uint4*>(kv_state + ((size_t)bh * dv + (size_t)g * RPG) * kExpandedDim);
#pragma unroll
    for (int n = 0; n < kIters; ++n)
      if (lane + 32 * n < kVecPerGroup) r[n] = __ldcs(base + lane + 32 * n);
  };
  if (warp < ngroups) fetch(warp);
  // the last warp has the row of sums, too
  ST* ks = k_state + (size_t)bh * kExpandedDim;
  float z[kIters];
  if (warp == kWarps - 1) {
#pragma unroll
    for (int n = 0; n < kIters; ++n) z[n] = lane + 32 * n < kExpandedDim ? to_float(ks[lane + 32 * n]) : 0.f;
  }
  if (tid < kFeatureDim) {
    s_x[0][tid] = to_float(q[b * sq.b + h * sq.h + tid]);
  } else if (tid < 2 * kFeatureDim) {
    s_x[1][tid - kFeatureDim] = to_float(k[b * sk.b + h * sk.h + tid - kFeatureDim]);
  } else {   // (128 threads: more values than there are threads left)
    for (int i = tid - 2 * kFeatureDim; i < dv; i += kThreads - 2 * kFeatureDim) s_v[i] = to_float(v[b * sv.b + h * sv.h + i]);
  }
  __syncthreads();
  for (int idx = tid; idx < 2 * kExpandedDim; idx += kThreads) {   // a feature once, into its places in the four copies
    const int which = idx >= kExpandedDim, f = idx - which * kExpandedDim;
    const float val = taylor_feature(s_x[which], f);
    float(*tab)[kTab] = which == 0 ? s_tq : s_tk;
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      const int i = f - s;
      if (i >= 0) tab[s][i] = val;
      if (i + kExpandedDim < kTab) tab[s][i + kExpandedDim] = val;
    }
  }
  __syncthreads();

  // k_state: last warp, scalar accesses (a 273-element row is only element-aligned).
  if (warp == kWarps - 1) {
    float den = 0.f;
#pragma unroll
    for (int n = 0; n < kIters; ++n) {
      const int f = lane + 32 * n;
      if (f < kExpandedDim) {
        const float nw = VO::round(z[n] + s_tk[0][f]);
        ks[f] = from_float<ST>(nw);
        den += s_tq[0][f] * nw;
      }
    }
    den = warp_sum(den);
    if (lane == 0) s_den = den;
  }

  for (int g = warp; g < ngroups; g += kWarps) {
    uint4* base = reinterpret_cast<uint4*>(kv_state + ((size_t)bh * dv + (size_t)g * RPG) * kExpandedDim);
    if (g != warp) fetch(g);
    float acc[RPG];
#pragma unroll
    for (int rr = 0; rr < RPG; ++rr) acc[rr] = 0.f;
#pragma unroll
    for (int n = 0; n < kIters; ++n) {
      const int idx = lane + 32 * n;
      if (idx < kVecPerGroup) {
        // the 32 vectors of a step lie in two rows at most, and which two is known when this is compiled
        const int first = 32 * VEC * n / kExpandedDim, e0 = idx * VEC;
        const bool second = e0 >= (first + 1) * kExpandedDim;
        const int row0 = first + second, f0 = e0 - row0 * kExpandedDim;
        const int s = f0 & 3, i = f0 - s;
        float pk[VEC], pq[VEC], e[VEC];
#pragma unroll
        for (int c4 = 0; c4 < VEC / 4; ++c4) {
          const float4 a = *reinterpret_cast<const float4*>(&s_tk[s][i + 4 * c4]);
          const float4 bq = *reinterpret_cast<const float4*>(&s_tq[s][i + 4 * c4]);
          pk[4 * c4] = a.x; pk[4 * c4 + 1] = a.y; pk[4 * c4 + 2] = a.z; pk[4 * c4 + 3] = a.w;
          pq[4 * c4] = bq.x; pq[4 * c4 + 1] = bq.y; pq[4 * c4 + 2] = bq.z; pq[4 * c4 + 3] = bq.w;
        }
        VO::unpack(r[n], e);
        const int rbase = g * RPG + row0;
        const float v0 = s_v[rbase];
        const float v1 = s_v[min(rbase + 1, dv - 1)];
        const int cwrap = kExpandedDim - f0;  // elements c >= cwrap belong to row0 + 1
        float a0 = 0.f, a1 = 0.f;
#pragma unroll
        for (int c = 0; c < VEC; ++c) {
          const bool hi = c >= cwrap;
          e[c] = fmaf(pk[c], hi ? v1 : v0, e[c]);
        }
        __stcs(base + idx, VO::pack(e));
#pragma unroll
        for (int c = 0; c < VEC; ++c) {
          const bool hi = c >= cwrap;
          const float contrib = pq[c] * e[c];
          a0 += hi ? 0.f : contrib;
          a1 += hi ? contrib : 0.f;
        }
        acc[first] += second ? 0.f : a0;
        if (first + 1 < RPG) acc[first + 1] += second ? a0 : a1;   // (a vector that begins in the second row ends there)
      }
    }
#pragma unroll
    for (int rr = 0; rr < RPG; ++rr) {
      const float t = warp_sum(acc[rr]);
      if (lane == 0) s_num[g * RPG + rr] = t;
    }
  }
  __syncthreads();
  static_assert(kThreads >= 128, "a thread per value of the output");
  if (tid < dv) {
    y[b * sy.b + h * sy.h + tid] = from_float<IO>(s_num[tid] / (s_den + eps));
  }
}

template <typename IO, typename ST>
int launch_typed(const void* q, const void* k, const void* v, void* y, void* kv_state, void* k_state, int B, int H,
                 int dv, Strides2 sq, Strides2 sk, Strides2 sv, Strides2 sy, float eps, cudaStream_t stream) {
  int dev = 0, sms = 148;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if ((long long)B * H >= 6LL * sms) {  // at least a wave and a half
    constexpr int kThreads = sizeof(ST) == 4 ? 192 : 128;
    launch_pdl(linattn_decode_kernel<IO, ST, kThreads>, B * H, kThreads, 0, stream,
        static_cast<const IO*>(q), static_cast<const IO*>(k), static_cast<const IO*>(v), static_cast<IO*>(y),
        static_cast<ST*>(kv_state), static_cast<ST*>(k_state), H, dv, sq, sk, sv, sy, eps);
  } else if ((long long)B * H <= sms && dv / VecOps<ST>::kVec > 8) {   // a block per SM: all its row groups at once
    launch_pdl(linattn_decode_kernel<IO, ST, 512>, B * H, 512, 0, stream,
        static_cast<const IO*>(q), static_cast<const IO*>(k), static_cast<const IO*>(v), static_cast<IO*>(y),
        static_cast<ST*>(kv_state), static_cast<ST*>(k_state), H, dv, sq, sk, sv, sy, eps);
  } else {
    launch_pdl(linattn_decode_kernel<IO, ST, 256>, B * H, 256, 0, stream, 
        static_cast<const IO*>(q), static_cast<const IO*>(k), static_cast<const IO*>(v), static_cast<IO*>(y),
        static_cast<ST*>(kv_state), static_cast<ST*>(k_state), H, dv, sq, sk, sv, sy, eps);
  }
  return static_cast<int>(cudaGetLastError());
}

}  // namespace

int launch_linattn_decode(const void* q, const void* k, const void* v, void* y, void* kv_state, void* k_state,
                          int B, int H, int dv, Strides2 sq, Strides2 sk, Strides2 sv, Strides2 sy,
                          int io_dtype, int state_dtype, float eps, cudaStream_t stream) {
  using bf16 = __nv_bfloat16;
  if (io_dtype == BASED_BF16 && state_dtype == BASED_F32)
    return launch_typed<bf16, float>(q, k, v, y, kv_state, k_state, B, H, dv, sq, sk, sv, sy, eps, stream);
  if (io_dtype == BASED_BF16 && state_dtype == BASED_BF16)
    return launch_typed<bf16, bf16>(q, k, v, y, kv_state, k_state, B, H, dv, sq, sk, sv, sy, eps, stream);
  if (io_dtype == BASED_F32 && state_dtype == BASED_F32)
    return launch_typed<float, float>(q, k, v, y, kv_state, k_state, B, H, dv, sq, sk, sv, sy, eps, stream);
  if (io_dtype == BASED_F32 && state_dtype == BASED_BF16)
    return launch_typed<float, bf16>(q, k, v, y, kv_state, k_state, B, H, dv, sq, sk, sv, sy, eps, stream);
  return BASED_ERR_DTYPE;
}

}  // namespace based
