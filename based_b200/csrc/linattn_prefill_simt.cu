// Causal Taylor linear attention over a whole sequence, CUDA-core version with fp32
// arithmetic throughout.  It is the fp32-I/O path (tf32/bf16 tensor-core operands cannot
// hold 1e-4 relative error) and the reference point for the tensor-core kernel.
//
// Replaces LinearAttention.parallel_forward's "quadratic" branch
// (based/models/mixers/linear_attention.py:171-182) and the state hand-off (:220-222) in
// O(L) memory: the sequence is walked in chunks of 64 tokens; within a chunk the causal part
// uses phi(q).phi(k) = 1 + s + s^2/2 (s = q.k/4), across chunks the state is carried in registers.
//
// Bound by the fp32 FMA rate.  The 256 products x_i x_j of the feature map are symmetric: the kernel keeps 153 features (1, x/2,
// products i <= j) with phi(k) scaled as in the 273 and the products i < j of phi(q) doubled, so that its state is the 273-feature
// state and every step has 56 % of the multiply-adds.  Per chunk and 64 value columns three register-tiled products run
// (256 threads, operands in shared memory): O = phi(q) S (4 x 4 per thread), O += P V (4 x 4), S += phi(k)^T V (20 x 2, the
// accumulators ARE the state): 1.6 M multiply-adds, 12 k cycles at the FMA rate; issue
// slots are 50 % used (two warps per scheduler, products in registers at 207 of them), so a chunk takes about 25 k.
//
// One CTA walks one (batch, head) and up to 64 value columns; with few of those a CLUSTER of 2 to 8 CTAs shares the sequence,
// a run of chunks each: first what the run adds to the state (the state product alone, 45 % of the work), then, from the sum
// of the runs before it, read over distributed shared memory in order, the output.  K CTAs take 1.45 / K of the time.
// B = 2, H = 16, L = 1024, dv = 64: 925 us with a CTA per head and 16-token blocks over 273 features, 99 us like this.
#include <mutex>
#include <utility>

#include "common.cuh"

namespace based {
namespace {

constexpr int T = 64;          // tokens per chunk
constexpr int CW = 64;         // value columns per CTA
constexpr int FP = 160;        // packed features: 153, padded
constexpr int kPacked = 153;
constexpr int SP = 68;         // row pitch of the state in shared memory
constexpr int KP = FP + 4;     // row pitch of phi(k): eight tokens' 16-byte pieces are in different banks
constexpr int NT = 256;
constexpr int kMaxCluster = 8;

struct Smem {
  float phi[KP * T];           // phi(q) as [feature][token], then phi(k) as [token][feature]
  float S[FP * SP];            // [feature][column]
  float v[T * CW];             // [token][column]
  float p[T * T];              // [key][query]
  float qt[kFeatureDim * T];   // [dim][token]
  float k[T * kFeatureDim];    // [token][dim]
  float den[4 * T];
  float z[FP];                 // normaliser's state
  unsigned char at[kExpandedDim + 3];   // packed place of each of the 273
};

// Dims of packed feature f >= 17, the products i <= j in rows of i.
__host__ __device__ constexpr int pair_i(int f) {
  int i = 0, left = f - 1 - kFeatureDim;
  while (left >= kFeatureDim - i) left -= kFeatureDim - i++;
  return i;
}
__host__ __device__ constexpr int pair_j(int f) {
  int i = 0, left = f - 1 - kFeatureDim;
  while (left >= kFeatureDim - i) left -= kFeatureDim - i++;
  return i + left;
}
// Packed feature F of the 16 values in x (registers: every index is known here); QUERY: products i < j twice, for (j, i) too.
template <int F, bool QUERY>
__device__ __forceinline__ float feature(const float (&x)[kFeatureDim]) {
  if constexpr (F == 0) return 1.f;
  else if constexpr (F <= kFeatureDim) return x[F - 1] * kC1;
  else if constexpr (F >= kPacked) return 0.f;
  else {
    constexpr int i = pair_i(F), j = pair_j(F);
    return x[i] * x[j] * (QUERY && i != j ? 2.f * kC2 : kC2);
  }
}
// Features [F0, F0 + 40) of one token: of phi(q) at dst[f * T], of phi(k) at dst[f].
template <int F0, int... I>
__device__ __forceinline__ void put_query(float* dst, const float (&x)[kFeatureDim], std::integer_sequence<int, I...>) {
  ((dst[(F0 + I) * T] = feature<F0 + I, true>(x)), ...);
}
template <int F0, int... I>
__device__ __forceinline__ void put_key(float* dst, const float (&x)[kFeatureDim], bool live, std::integer_sequence<int, I...>) {
  ((*reinterpret_cast<float4*>(dst + F0 + 4 * I) =
        live ? make_float4(feature<F0 + 4 * I, false>(x), feature<F0 + 4 * I + 1, false>(x), feature<F0 + 4 * I + 2, false>(x), feature<F0 + 4 * I + 3, false>(x))
             : make_float4(0.f, 0.f, 0.f, 0.f)), ...);
}

template <typename IO>
struct Args {
  const IO *q, *k, *v;
  IO* y;
  void *kv_state, *k_state;
  int H, L, dv, K, vec_out, state_bf16;   // K: CTAs per sequence
  int run;                                // tokens whose products are summed before they join the state: 8, 16, 32 or 64
  Strides3 sq, sk, sv, sy;
  float eps;
};

__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}
__device__ __forceinline__ uint32_t peer_addr(const void* own, uint32_t rank) {
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(a) : "r"((uint32_t)__cvta_generic_to_shared(own)), "r"(rank));
  return a;
}
__device__ __forceinline__ float ld_peer(uint32_t a) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];\n" : "=f"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ float2 ld_peer2(uint32_t a) {
  float2 v;
  asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];\n" : "=f"(v.x), "=f"(v.y) : "r"(a) : "memory");
  return v;
}

// acc[a][b] += x[a] * y[b]
__device__ __forceinline__ void outer4(float (&acc)[4][4], const float4& x, const float4& y) {
  const float xs[4] = {x.x, x.y, x.z, x.w}, ys[4] = {y.x, y.y, y.z, y.w};
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b) acc[a][b] = fmaf(xs[a], ys[b], acc[a][b]);
}

template <typename IO>
__global__ void __launch_bounds__(NT, 1) linattn_prefill_simt_kernel(const Args<IO> p) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Smem& s = *reinterpret_cast<Smem*>(smem_raw);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int rank = blockIdx.x % p.K, bh = blockIdx.x / p.K, b = bh / p.H, h = bh - b * p.H;
  const int c0 = blockIdx.y * CW, cols = min(CW, p.dv - c0);
  const int chunks = (p.L + T - 1) / T, first = (int)((int64_t)chunks * rank / p.K), n = (int)((int64_t)chunks * (rank + 1) / p.K) - first;
  const IO* qb = p.q + b * p.sq.b + h * p.sq.h;
  const IO* kb = p.k + b * p.sk.b + h * p.sk.h;
  const IO* vb = p.v + b * p.sv.b + h * p.sv.h + c0;
  for (int f = tid; f < kExpandedDim; f += NT) {
    if (f <= kFeatureDim) { s.at[f] = (unsigned char)f; continue; }
    const int i = (f - 1 - kFeatureDim) >> 4, j = (f - 1 - kFeatureDim) & 15, lo = min(i, j), hi = max(i, j);
    const int at = 1 + kFeatureDim + lo * kFeatureDim - lo * (lo - 1) / 2 + (hi - lo);
    s.at[f] = (unsigned char)at;
  }
  if (tid < FP) s.z[tid] = 0.f;

  // a chunk's inputs wait in registers while the one before is worked on; tokens and columns outside are zero
  float rq[4], rk[4], rv[16];
  auto load = [&](int chunk, bool with_q) {
    const int t0 = chunk * T;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int t = (tid >> 4) + 16 * i, c = tid & 15;
      const bool ok = t0 + t < p.L;
      rk[i] = ok ? to_float(kb[(int64_t)(t0 + t) * p.sk.l + c]) : 0.f;
      if (with_q) rq[i] = ok ? to_float(qb[(int64_t)(t0 + t) * p.sq.l + c]) : 0.f;
    }
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const int t = (tid >> 6) + 4 * i, c = tid & 63;
      rv[i] = t0 + t < p.L && c < cols ? to_float(vb[(int64_t)(t0 + t) * p.sv.l + c]) : 0.f;
    }
  };
  auto put = [&](bool with_q) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int t = (tid >> 4) + 16 * i, c = tid & 15;
      s.k[t * kFeatureDim + c] = rk[i];
      if (with_q) s.qt[c * T + t] = rq[i];
    }
#pragma unroll
    for (int i = 0; i < 16; ++i) s.v[((tid >> 6) + 4 * i) * CW + (tid & 63)] = rv[i];
  };
  // phi(k) of `nt` tokens as [token][feature]; tokens past the end must not reach the state
  auto build_k = [&](int nt) {
    const int t = tid & 63, part = tid >> 6;
    float x[kFeatureDim];
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      const float4 y = *reinterpret_cast<const float4*>(s.k + t * kFeatureDim + 4 * m);
      x[4 * m] = y.x; x[4 * m + 1] = y.y; x[4 * m + 2] = y.z; x[4 * m + 3] = y.w;
    }
    float* dst = s.phi + t * KP;
    constexpr std::make_integer_sequence<int, 10> ten;
    if (part == 0) put_key<0>(dst, x, t < nt, ten);
    else if (part == 1) put_key<40>(dst, x, t < nt, ten);
    else if (part == 2) put_key<80>(dst, x, t < nt, ten);
    else put_key<120>(dst, x, t < nt, ten);
  };
  // the state of this thread: features 20 warp .., columns 2 lane ..
  float S[20][2];
#pragma unroll
  for (int i = 0; i < 20; ++i) S[i][0] = S[i][1] = 0.f;
  auto update = [&]() {
    const float* a = s.phi + 20 * warp;
    const float* v = s.v + 2 * lane;
    float U[20][2];   // the sum of a run of tokens on its own: fewer roundings at the size of the whole sum
#pragma unroll
    for (int i = 0; i < 20; ++i) U[i][0] = U[i][1] = 0.f;
#pragma unroll 1
    for (int t0 = 0; t0 < T; t0 += 8) {
#pragma unroll 4
      for (int t = t0; t < t0 + 8; ++t) {
        const float2 y = *reinterpret_cast<const float2*>(v + t * CW);
#pragma unroll
        for (int i = 0; i < 5; ++i) {
          const float4 x = *reinterpret_cast<const float4*>(a + t * KP + 4 * i);
          U[4 * i][0] = fmaf(x.x, y.x, U[4 * i][0]); U[4 * i][1] = fmaf(x.x, y.y, U[4 * i][1]);
          U[4 * i + 1][0] = fmaf(x.y, y.x, U[4 * i + 1][0]); U[4 * i + 1][1] = fmaf(x.y, y.y, U[4 * i + 1][1]);
          U[4 * i + 2][0] = fmaf(x.z, y.x, U[4 * i + 2][0]); U[4 * i + 2][1] = fmaf(x.z, y.y, U[4 * i + 2][1]);
          U[4 * i + 3][0] = fmaf(x.w, y.x, U[4 * i + 3][0]); U[4 * i + 3][1] = fmaf(x.w, y.y, U[4 * i + 3][1]);
        }
      }
      if (((t0 + 8) & (p.run - 1)) == 0) {
#pragma unroll
        for (int i = 0; i < 20; ++i) {
          S[i][0] += U[i][0]; S[i][1] += U[i][1];
          U[i][0] = U[i][1] = 0.f;
        }
      }
    }
    if (tid < FP) {
      float z[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
      for (int t = 0; t < T; t += 4)
#pragma unroll
        for (int i = 0; i < 4; ++i) z[i] += s.phi[(t + i) * KP + tid];
      s.z[tid] += (z[0] + z[1]) + (z[2] + z[3]);
    }
  };
  auto put_state = [&]() {
#pragma unroll
    for (int i = 0; i < 20; ++i) *reinterpret_cast<float2*>(s.S + (20 * warp + i) * SP + 2 * lane) = make_float2(S[i][0], S[i][1]);
  };

  if (p.K > 1) {
    // ---- what this run of chunks adds to the state (nobody asks the last one)
    if (rank < p.K - 1) {
      load(first, false);
      for (int c = 0; c < n; ++c) {
        put(false);
        if (c + 1 < n) load(first + c + 1, false);
        __syncthreads();
        build_k(T);            // only the last CTA has a chunk that is not whole
        __syncthreads();
        update();
        __syncthreads();
      }
      put_state();
    }
    cluster_sync();
    // ---- the state before this run: the sum of the runs before it, in order
#pragma unroll
    for (int i = 0; i < 20; ++i) S[i][0] = S[i][1] = 0.f;
    float z = 0.f;
    for (int r = 0; r < rank; ++r) {
      const uint32_t at = peer_addr(s.S + 20 * warp * SP + 2 * lane, r);
#pragma unroll
      for (int i = 0; i < 20; ++i) {
        const float2 x = ld_peer2(at + i * SP * 4);
        S[i][0] += x.x;
        S[i][1] += x.y;
      }
      if (tid < FP) z += ld_peer(peer_addr(s.z + tid, r));
    }
    cluster_sync();
    if (tid < FP) s.z[tid] = z;
  }

  // ---- the output
  // this thread's tile of a chunk: tokens ta .., columns ca ..
  const int ta = (warp & 1) * 32 + (lane >> 2) * 4, ca = (warp >> 1) * 16 + (lane & 3) * 4;
  load(first, true);
  for (int c = 0; c < n; ++c) {
    const int t0 = (first + c) * T, nt = min(T, p.L - t0);
    const bool some = first + c > 0;   // there is a state
    put(true);
    if (c + 1 < n) load(first + c + 1, true);
    if (some) put_state();
    __syncthreads();
    {  // phi(q), scores: a thread has one token, and a quarter of the features and of the keys
      const int t = tid & 63, part = tid >> 6;
      float x[kFeatureDim];
#pragma unroll
      for (int i = 0; i < kFeatureDim; ++i) x[i] = s.qt[i * T + t];
      if (some) {
        float* dst = s.phi + t;
        constexpr std::make_integer_sequence<int, 40> forty;
        if (part == 0) put_query<0>(dst, x, forty);
        else if (part == 1) put_query<40>(dst, x, forty);
        else if (part == 2) put_query<80>(dst, x, forty);
        else put_query<120>(dst, x, forty);
      }
#pragma unroll 4
      for (int i = 0; i < 16; ++i) {
        const int key = part * 16 + i;
        const float4* kk = reinterpret_cast<const float4*>(s.k + key * kFeatureDim);
        float d = 0.f;
#pragma unroll
        for (int m = 0; m < 4; ++m) {
          const float4 y = kk[m];
          d = fmaf(x[4 * m], y.x, d); d = fmaf(x[4 * m + 1], y.y, d); d = fmaf(x[4 * m + 2], y.z, d); d = fmaf(x[4 * m + 3], y.w, d);
        }
        d *= 0.25f;
        s.p[key * T + t] = key <= t ? 1.f + d + 0.5f * d * d : 0.f;
      }
    }
    __syncthreads();
    float o[4][4], o1[4][4];   // two sums: half the roundings at full size
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) o[i][j] = o1[i][j] = 0.f;
    if (some) {
#pragma unroll 4
      for (int f = 0; f < FP / 2; ++f) {
        outer4(o, *reinterpret_cast<const float4*>(s.phi + f * T + ta), *reinterpret_cast<const float4*>(s.S + f * SP + ca));
        outer4(o1, *reinterpret_cast<const float4*>(s.phi + (f + FP / 2) * T + ta), *reinterpret_cast<const float4*>(s.S + (f + FP / 2) * SP + ca));
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) { o[i][j] += o1[i][j]; o1[i][j] = 0.f; }
    }
    // a later value must not reach an earlier token, not even times zero: it may be infinite
#pragma unroll 4
    for (int t = 0; t < ta; ++t)
      outer4(o1, *reinterpret_cast<const float4*>(s.p + t * T + ta), *reinterpret_cast<const float4*>(s.v + t * CW + ca));
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float4 y = *reinterpret_cast<const float4*>(s.v + (ta + j) * CW + ca);
#pragma unroll
      for (int i = j; i < 4; ++i) {
        const float x = s.p[(ta + j) * T + ta + i];
        o1[i][0] = fmaf(x, y.x, o1[i][0]); o1[i][1] = fmaf(x, y.y, o1[i][1]); o1[i][2] = fmaf(x, y.z, o1[i][2]); o1[i][3] = fmaf(x, y.w, o1[i][3]);
      }
    }
    {
      const int t = tid & 63, part = tid >> 6;
      float d0 = 0.f, d1 = 0.f;
      if (some)
#pragma unroll 10
        for (int f = part * 40; f < part * 40 + 40; f += 2) {
          d0 = fmaf(s.phi[f * T + t], s.z[f], d0);
          d1 = fmaf(s.phi[(f + 1) * T + t], s.z[f + 1], d1);
        }
#pragma unroll
      for (int i = 0; i < 16; i += 2) {
        d0 += s.p[(part * 16 + i) * T + t];
        d1 += s.p[(part * 16 + i + 1) * T + t];
      }
      s.den[part * T + t] = d0 + d1;
    }
    __syncthreads();
    build_k(nt);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int t = ta + i;
      if (t < nt) {
        const float den = (s.den[t] + s.den[T + t]) + (s.den[2 * T + t] + s.den[3 * T + t]) + p.eps;
        IO* y = p.y + b * p.sy.b + h * p.sy.h + (int64_t)(t0 + t) * p.sy.l + c0 + ca;
        IO r[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) r[j] = from_float<IO>((o[i][j] + o1[i][j]) / den);
        if (p.vec_out) {
          if (ca < cols) {
            if (sizeof(IO) == 4) *reinterpret_cast<float4*>(y) = *reinterpret_cast<const float4*>(r);
            else *reinterpret_cast<uint2*>(y) = *reinterpret_cast<const uint2*>(r);
          }
        } else {
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (ca + j < cols) y[j] = r[j];
        }
      }
    }
    __syncthreads();
    update();
    __syncthreads();
  }
  if (rank != p.K - 1) return;   // peers read this CTA's memory before the second cluster_sync only
  // ---- the state after the last token, all 273 features
  put_state();
  __syncthreads();
  if (p.kv_state != nullptr)
    for (int i = tid; i < cols * kExpandedDim; i += NT) {
      const int c = i / kExpandedDim, f = i - c * kExpandedDim;
      const float x = s.S[s.at[f] * SP + c];
      const int64_t to = ((int64_t)bh * p.dv + c0) * kExpandedDim + i;
      if (p.state_bf16) static_cast<__nv_bfloat16*>(p.kv_state)[to] = __float2bfloat16_rn(x);
      else static_cast<float*>(p.kv_state)[to] = x;
    }
  if (p.k_state != nullptr && blockIdx.y == 0)
    for (int f = tid; f < kExpandedDim; f += NT) {
      const float x = s.z[s.at[f]];
      const int64_t to = (int64_t)bh * kExpandedDim + f;
      if (p.state_bf16) static_cast<__nv_bfloat16*>(p.k_state)[to] = __float2bfloat16_rn(x);
      else static_cast<float*>(p.k_state)[to] = x;
    }
}

template <typename IO>
int launch_typed(const void* q, const void* k, const void* v, void* y, void* kv_state, void* k_state, int B, int H,
                 int L, int dv, Strides3 sq, Strides3 sk, Strides3 sv, Strides3 sy, int state_bf16, float eps,
                 cudaStream_t stream) {
  auto kern = linattn_prefill_simt_kernel<IO>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(Smem));
  if (e != cudaSuccess) return (int)e;
  const bool vec = reinterpret_cast<uintptr_t>(y) % (4 * sizeof(IO)) == 0 && dv % 4 == 0 && sy.b % 4 == 0 && sy.h % 4 == 0 && sy.l % 4 == 0;
  const int slices = (dv + CW - 1) / CW, chunks = (L + T - 1) / T;
  if (slices > 65535 || (int64_t)B * H > 0x7fffffff / kMaxCluster) return BASED_ERR_TOO_LARGE;
  // The largest cluster of which all fit the device at once and whose CTAs have a chunk each: two CTAs with a chunk each take
  // 1.45 of a chunk's time instead of 2.
  int K = 1;
  {
    constexpr int kMaxDevices = 64;
    static std::mutex mu;
    static short room[kMaxDevices][kMaxCluster + 1] = {};   // clusters of a size on the device at once, + 1
    int dev = 0;
    e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return (int)e;
    if (dev < 0 || dev >= kMaxDevices) return BASED_ERR_TOO_LARGE;
    std::lock_guard<std::mutex> lock(mu);
    const int64_t units = (int64_t)B * H * slices;
    for (int k = chunks < kMaxCluster ? chunks : kMaxCluster; k > 1; --k) {
      if (units * k > 148) continue;
      short& r = room[dev][k];
      if (r == 0) r = (short)(1 + max_active_clusters(kern, k, NT, (int)sizeof(Smem)));
      if (r - 1 < units) continue;
      K = k;
      break;
    }
  }
  // A state entry is rounded `run` times on the way to a run's sum and L / run times on the way to the whole: the error is least at
  // run = sqrt(L).  Off the exact state by 2-norm, B = 4, H = 16, dv = 64, with 8 / 16 / 32 / 64: L = 60 0.84 / 0.89 / 1.08 / 1.44 e-7,
  // 300 1.31 / 1.16 / 1.24 / 1.52, 1024 2.15 / 1.67 / 1.51 / 1.67, 2048 2.95 / 2.20 / 1.82 / 1.82; the time changes by 2 % at most.
  const int run = L <= 128 ? 8 : L <= 512 ? 16 : L <= 2048 ? 32 : 64;
  const Args<IO> args{static_cast<const IO*>(q), static_cast<const IO*>(k), static_cast<const IO*>(v), static_cast<IO*>(y), kv_state, k_state,
                      H, L, dv, K, vec, state_bf16, run, sq, sk, sv, sy, eps};
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = K;
  attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(B * H * K, slices);
  cfg.blockDim = dim3(NT);
  cfg.dynamicSmemBytes = sizeof(Smem);
  cfg.stream = stream;
  cfg.attrs = &attr;
  cfg.numAttrs = K > 1 ? 1 : 0;
  return launched((int)cudaLaunchKernelEx(&cfg, kern, args));
}

}  // namespace

int launch_linattn_prefill_simt(const void* q, const void* k, const void* v, void* y, void* kv_state, void* k_state,
                                int B, int H, int L, int dv, Strides3 sq, Strides3 sk, Strides3 sv, Strides3 sy,
                                int io_dtype, int state_dtype, float eps, cudaStream_t stream) {
  if (state_dtype != BASED_F32 && state_dtype != BASED_BF16) return BASED_ERR_DTYPE;
  const int sb = state_dtype == BASED_BF16;
  if (io_dtype == BASED_F32) return launch_typed<float>(q, k, v, y, kv_state, k_state, B, H, L, dv, sq, sk, sv, sy, sb, eps, stream);
  if (io_dtype == BASED_BF16) return launch_typed<__nv_bfloat16>(q, k, v, y, kv_state, k_state, B, H, L, dv, sq, sk, sv, sy, sb, eps, stream);
  return BASED_ERR_DTYPE;
}

}  // namespace based
