// Sliding-window causal softmax attention on CUDA cores: the prefill kernel used for fp32 I/O
// and as the reference point of the tensor-core kernel, and the decode-step kernel (RoPE on
// q/k at the new position, append to the KV cache, attend over <= window_left+1 cached keys),
// which is latency/bandwidth-bound and needs no tensor cores.
//
// Semantics follow the reference's calls into flash-attn:
//   prefill  based/models/mixers/slide_attention.py:100-106, :206-213
//            (causal=True, window_size=(window_left, 0): keys [i - window_left, i])
//   decode   slide_attention.py:414-427, :471-481 (append at cache_seqlens, then attend)
//   RoPE     based/ops/triton/rotary.py:75-105 (non-interleaved halves, fp32 math)
#include "common.cuh"

namespace based {
namespace {

constexpr int kWarpsPerBlock = 4;
constexpr int kMaxHd = 128;
constexpr int kMaxKeysPerLane = 9;  // supports window_left + 1 <= 288

// One warp per query.  Lane l scores keys lo + l, lo + l + 32, ...; then the lanes switch to
// owning output channels for the weighted sum of value rows.
template <typename IO>
__global__ void __launch_bounds__(kWarpsPerBlock * 32)
swa_prefill_simt_kernel(const IO* __restrict__ q, const IO* __restrict__ k, const IO* __restrict__ v,
                        IO* __restrict__ o, int L, int H, int hd, Strides3 sq, Strides3 sk, Strides3 sv,
                        Strides3 so, int window_left, float scale) {
  __shared__ float s_q[kWarpsPerBlock][kMaxHd];
  __shared__ float s_p[kWarpsPerBlock][kMaxKeysPerLane * 32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int i = blockIdx.x * kWarpsPerBlock + warp;  // query position
  const int h = blockIdx.y, b = blockIdx.z;
  if (i >= L) return;
  const IO* qp = q + b * sq.b + (int64_t)i * sq.l + h * sq.h;
  for (int c = lane; c < hd; c += 32) s_q[warp][c] = to_float(qp[c]);
  __syncwarp();
  const int lo = max(0, i - window_left);
  const int nk = i - lo + 1;
  float sc[kMaxKeysPerLane];
  float m = -INFINITY;
#pragma unroll
  for (int n = 0; n < kMaxKeysPerLane; ++n) {
    const int jj = lane + 32 * n;
    sc[n] = -INFINITY;
    if (jj < nk) {
      const IO* kp = k + b * sk.b + (int64_t)(lo + jj) * sk.l + h * sk.h;
      float dot = 0.f;
      for (int c = 0; c < hd; ++c) dot = fmaf(s_q[warp][c], to_float(kp[c]), dot);
      sc[n] = dot * scale;
      m = fmaxf(m, sc[n]);
    }
  }
  m = warp_max(m);
  float sum = 0.f;
#pragma unroll
  for (int n = 0; n < kMaxKeysPerLane; ++n) {
    const int jj = lane + 32 * n;
    if (jj < nk) {
      const float p = __expf(sc[n] - m);
      s_p[warp][jj] = p;
      sum += p;
    }
  }
  sum = warp_sum(sum);
  __syncwarp();
  const float inv = 1.f / sum;
  for (int c = lane; c < hd; c += 32) {
    float acc = 0.f;
    for (int jj = 0; jj < nk; ++jj) {
      acc = fmaf(s_p[warp][jj], to_float(v[b * sv.b + (int64_t)(lo + jj) * sv.l + h * sv.h + c]), acc);
    }
    o[b * so.b + (int64_t)i * so.l + h * so.h + c] = from_float<IO>(acc * inv);
  }
}

// 8 consecutive values of a cached row
struct Row8 {
  float x[8];
};
__device__ __forceinline__ void load8(const __nv_bfloat16* p, uint4 (&r)[1]) { r[0] = *reinterpret_cast<const uint4*>(p); }
__device__ __forceinline__ void load8(const float* p, uint4 (&r)[2]) {
  r[0] = *reinterpret_cast<const uint4*>(p);
  r[1] = *reinterpret_cast<const uint4*>(p + 4);
}
__device__ __forceinline__ Row8 unpack8(const uint4 (&r)[1]) {
  const uint32_t w[4] = {r[0].x, r[0].y, r[0].z, r[0].w};
  Row8 y;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    y.x[2 * i] = __uint_as_float(w[i] << 16);
    y.x[2 * i + 1] = __uint_as_float(w[i] & 0xFFFF0000u);
  }
  return y;
}
__device__ __forceinline__ Row8 unpack8(const uint4 (&r)[2]) {
  return Row8{{__uint_as_float(r[0].x), __uint_as_float(r[0].y), __uint_as_float(r[0].z), __uint_as_float(r[0].w),
               __uint_as_float(r[1].x), __uint_as_float(r[1].y), __uint_as_float(r[1].z), __uint_as_float(r[1].w)}};
}

// A (batch, head) has a block of WARPS warps, or HEADS of them share a block, a warp each.  A step's bytes (a window of keys and
// values, 16 KB a head) take less than a microsecond; what it takes is the chain load - scores - softmax - values.  So the window
// is spread over the warps: LPK lanes share a cached row, 8 values (16 or 32 bytes) each, a group of lanes has every
// (32 / LPK * WARPS)-th key, and its first four keys AND values are in flight before the query is rotated.  Each group keeps a
// running maximum, sum and weighted row of its own keys; the groups meet once at the end.  16 heads, 16 rows, hd = 64, 64 keys: 6.5 us
// with one warp per head (keys, softmax, values in turn), 3.6 us like this, in a chain of such launches.  hd is a multiple of 8 and
// the cache 16-byte aligned (checked by the launcher).
template <typename IO, int LPK, int WARPS, int HEADS>
__global__ void __launch_bounds__(WARPS * HEADS * 32)
swa_decode_kernel(const IO* q, const IO* k_new, const IO* v_new,
                  IO* o, IO* kv_cache, const int32_t* cache_seqlens,
                  int cache_seqlen_scalar, const IO* rcos, const IO* rsin, int rotary_dim,
                  int BH, int H, int hd, int max_seqlen, Strides2 sq, Strides2 sk, Strides2 sv, Strides2 so,
                  int window_left, float scale) {
  pdl_trigger();
  pdl_wait();
  constexpr int kGroups = WARPS * 32 / LPK, U = 4, kVec = sizeof(IO) / 2;
  static_assert(HEADS == 1 || WARPS == 1, "heads of a block leave it on their own");
  __shared__ float sq_[HEADS][kMaxHd], sk_[HEADS][kMaxHd], sv_[HEADS][kMaxHd], sr_[HEADS][2][kMaxHd];
  __shared__ float so_[HEADS][WARPS][kMaxHd], sm_[HEADS][WARPS], sl_[HEADS][WARPS];
  const int slot = HEADS == 1 ? 0 : threadIdx.x >> 5, tid = HEADS == 1 ? threadIdx.x : threadIdx.x & 31, lane = tid & 31, warp = tid >> 5;
  float *s_q = sq_[slot], *s_k = sk_[slot], *s_v = sv_[slot], *s_m = sm_[slot], *s_l = sl_[slot];
  float (*s_r)[kMaxHd] = sr_[slot], (*s_o)[kMaxHd] = so_[slot];
  auto sync = [] {
    if constexpr (WARPS == 1) __syncwarp();
    else __syncthreads();
  };
  const int bh = blockIdx.x * HEADS + slot;
  if (bh >= BH) return;
  const int b = bh / H, h = bh - b * H;
  const int pos = cache_seqlens ? cache_seqlens[b] : cache_seqlen_scalar;
  if (pos < 0 || pos >= max_seqlen) return;  // nothing sensible to do; the host validates the scalar case
  const size_t row = (size_t)2 * H * hd;  // elements per cached position
  IO* cache_b = kv_cache + (size_t)b * max_seqlen * row;
  const int lo = max(0, pos - window_left), old = pos - lo;   // cached keys; the new one comes on top
  const int group = tid / LPK, c = 8 * (tid % LPK);
  const bool on = c < hd;
  const IO* kc = cache_b + (size_t)lo * row + (size_t)h * hd + c;
  uint4 kx[U][kVec], vx[U][kVec];
  auto fetch = [&](int j0) {
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int j = j0 + u * kGroups + group;
      if (on && j < old) {
        load8(kc + (size_t)j * row, kx[u]);
        load8(kc + (size_t)j * row + (size_t)H * hd, vx[u]);
      }
    }
  };
  fetch(0);
  // the new token: RoPE in fp32, result rounded to the I/O dtype like the reference kernel's store, and its row of the cache
  const IO* qp = q + b * sq.b + h * sq.h;
  const IO* kp = k_new + b * sk.b + h * sk.h;
  const IO* vp = v_new + b * sv.b + h * sv.h;
  for (int i = tid; i < hd; i += WARPS * 32) {
    s_r[0][i] = to_float(qp[i]);
    s_r[1][i] = to_float(kp[i]);
    s_v[i] = to_float(vp[i]);
  }
  sync();
  const int half = rcos ? rotary_dim / 2 : 0;
  for (int i = tid; i < 2 * hd; i += WARPS * 32) {
    const int which = i >= hd, cc = which ? i - hd : i;
    const float* x = s_r[which];
    float y = x[cc];
    if (cc < 2 * half) {
      const int a = cc < half ? cc : cc - half;
      const float cs = to_float(rcos[(size_t)pos * half + a]), sn = to_float(rsin[(size_t)pos * half + a]);
      y = cc < half ? x[cc] * cs - x[cc + half] * sn : x[cc - half] * sn + x[cc] * cs;
    }
    const IO r = from_float<IO>(y);
    (which ? s_k : s_q)[cc] = to_float(r);
    if (which) {
      IO* knew = cache_b + (size_t)pos * row + (size_t)h * hd;
      knew[cc] = r;
      knew[(size_t)H * hd + cc] = vp[cc];
    }
  }
  sync();
  float qv[8], acc[8], m = -INFINITY, l = 0.f;
#pragma unroll
  for (int i = 0; i < 8; ++i) { qv[i] = on ? s_q[c + i] : 0.f; acc[i] = 0.f; }
  auto score = [&](const Row8& x) {
    float d = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) d = fmaf(qv[i], x.x[i], d);
#pragma unroll
    for (int x2 = LPK / 2; x2 > 0; x2 >>= 1) d += __shfl_xor_sync(0xffffffffu, d, x2);
    return d * scale;
  };
  auto take = [&](const float (&sc)[U], const Row8 (&x)[U]) {   // scores of -inf stand for no key
    float top = m;
#pragma unroll
    for (int u = 0; u < U; ++u) top = fmaxf(top, sc[u]);
    const float base = top == -INFINITY ? 0.f : top, f = __expf(m - base);
    m = top;
    l *= f;
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i] *= f;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const float w = __expf(sc[u] - base);
      l += w;
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[i] = fmaf(w, x[u].x[i], acc[i]);
    }
  };
  const Row8 none{};
  for (int j0 = 0; j0 < old; j0 += U * kGroups) {
    if (j0 > 0) fetch(j0);
    float sc[U];
    Row8 x[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const bool live = j0 + u * kGroups + group < old;
      const float d = score(on && live ? unpack8(kx[u]) : none);
      sc[u] = live ? d : -INFINITY;
      x[u] = on && live ? unpack8(vx[u]) : none;
    }
    take(sc, x);
  }
  {  // the new key belongs to the first group
    Row8 x = none, y = none;
    if (on)
#pragma unroll
      for (int i = 0; i < 8; ++i) { x.x[i] = s_k[c + i]; y.x[i] = s_v[c + i]; }
    const float d = score(x), ninf = -INFINITY;
    const float sc[U] = {group == 0 ? d : ninf, ninf, ninf, ninf};
    const Row8 v[U] = {group == 0 ? y : none, none, none, none};
    take(sc, v);
  }
  // groups of a warp, then the warps
  float top = m;
#pragma unroll
  for (int x = LPK; x < 32; x <<= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, x));
  float f = m == -INFINITY ? 0.f : __expf(m - top);
  l *= f;
#pragma unroll
  for (int i = 0; i < 8; ++i) acc[i] *= f;
#pragma unroll
  for (int x = LPK; x < 32; x <<= 1) {
    l += __shfl_xor_sync(0xffffffffu, l, x);
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i] += __shfl_xor_sync(0xffffffffu, acc[i], x);
  }
  if (lane < LPK && on)
#pragma unroll
    for (int i = 0; i < 8; ++i) s_o[warp][c + i] = acc[i];
  if (lane == 0) { s_m[warp] = top; s_l[warp] = l; }
  sync();
  for (int i = tid; i < hd; i += WARPS * 32) {
    float mm = s_m[0], sum = 0.f, y = 0.f;
#pragma unroll
    for (int w = 1; w < WARPS; ++w) mm = fmaxf(mm, s_m[w]);
#pragma unroll
    for (int w = 0; w < WARPS; ++w) {
      const float g = s_m[w] == -INFINITY ? 0.f : __expf(s_m[w] - mm);
      sum = fmaf(g, s_l[w], sum);
      y = fmaf(g, s_o[w][i], y);
    }
    o[b * so.b + h * so.h + i] = from_float<IO>(y * (1.f / sum));
  }
}

// In-place non-interleaved RoPE on x [B, L, H, hd]: one thread per rotated pair.
template <typename IO>
__global__ void rotary_kernel(IO* __restrict__ x, int L, int H, Strides3 sx, const IO* __restrict__ rcos,
                              const IO* __restrict__ rsin, int half, const int32_t* __restrict__ offsets,
                              int offset_scalar, long long total) {
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= total) return;
  const int c = (int)(idx % half);
  long long r = idx / half;
  const int h = (int)(r % H); r /= H;
  const int l = (int)(r % L);
  const int b = (int)(r / L);
  const int pos = l + (offsets ? offsets[b] : offset_scalar);
  IO* px = x + b * sx.b + (int64_t)l * sx.l + h * sx.h;
  const float cs = to_float(rcos[(size_t)pos * half + c]), sn = to_float(rsin[(size_t)pos * half + c]);
  const float x0 = to_float(px[c]), x1 = to_float(px[c + half]);
  px[c] = from_float<IO>(x0 * cs - x1 * sn);
  px[c + half] = from_float<IO>(x0 * sn + x1 * cs);
}

// The same with 16-byte accesses: one thread per group of 8 (bf16) / 4 (fp32) rotated pairs.
template <typename IO>
__global__ void rotary_vec_kernel(IO* __restrict__ x, int L, int H, Strides3 sx, const IO* __restrict__ rcos,
                                  const IO* __restrict__ rsin, int half, const int32_t* __restrict__ offsets,
                                  int offset_scalar, long long total) {
  constexpr int N = 16 / sizeof(IO);
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= total) return;
  const int groups = half / N;
  const int c = (int)(idx % groups) * N;
  long long r = idx / groups;
  const int h = (int)(r % H); r /= H;
  const int l = (int)(r % L);
  const int b = (int)(r / L);
  const int pos = l + (offsets ? offsets[b] : offset_scalar);
  IO* px = x + b * sx.b + (int64_t)l * sx.l + h * sx.h + c;
  union V { uint4 u; IO e[N]; } x0, x1, cs, sn;
  x0.u = *reinterpret_cast<const uint4*>(px);
  x1.u = *reinterpret_cast<const uint4*>(px + half);
  cs.u = __ldg(reinterpret_cast<const uint4*>(rcos + (size_t)pos * half + c));
  sn.u = __ldg(reinterpret_cast<const uint4*>(rsin + (size_t)pos * half + c));
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const float a = to_float(x0.e[i]), bb = to_float(x1.e[i]), cc = to_float(cs.e[i]), ss = to_float(sn.e[i]);
    x0.e[i] = from_float<IO>(a * cc - bb * ss);
    x1.e[i] = from_float<IO>(a * ss + bb * cc);
  }
  *reinterpret_cast<uint4*>(px) = x0.u;
  *reinterpret_cast<uint4*>(px + half) = x1.u;
}

// Prompt pass of the sliding-window mixer on the packed projection qkv [B, L, 3, H, hd] (bf16): q and k rotated in
// place (whole head, non-interleaved), and the rotated k and v written to the layer's cache [*, max_seqlen, 2, H, hd]
// in the same pass.  One thread per 16-byte piece: q and k pieces carry a rotated pair of 8-element groups, v pieces
// a plain copy.  Pieces per head: hd/16 (q) + hd/16 (k) + hd/8 (v) = hd/4.
__global__ void __launch_bounds__(256)
rotary_qkv_cache_kernel(__nv_bfloat16* __restrict__ qkv, int L, int H, int hd, int64_t sb, int64_t sl, int64_t s3,
                        int64_t sh, const __nv_bfloat16* __restrict__ rcos, const __nv_bfloat16* __restrict__ rsin,
                        __nv_bfloat16* __restrict__ cache, int64_t cb, int64_t cl, long long total) {
  pdl_trigger();
  pdl_wait();
  using IO = __nv_bfloat16;
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= total) return;
  const int half = hd / 2, gq = half / 8, per_head = 2 * gq + hd / 8;
  const int piece = (int)(idx % per_head);
  long long r = idx / per_head;
  const int h = (int)(r % H); r /= H;
  const int l = (int)(r % L);
  const int b = (int)(r / L);
  IO* base = qkv + b * sb + (int64_t)l * sl + h * sh;
  IO* crow = cache + b * cb + (int64_t)l * cl + (int64_t)h * hd;  // k part; the v part is H * hd further
  if (piece >= 2 * gq) {  // v: copy
    const int c = (piece - 2 * gq) * 8;
    *reinterpret_cast<uint4*>(crow + (int64_t)H * hd + c) = *reinterpret_cast<const uint4*>(base + 2 * s3 + c);
    return;
  }
  const int part = piece / gq, c = (piece - part * gq) * 8;  // part 0 = q, 1 = k
  IO* px = base + part * s3 + c;
  union V { uint4 u; IO e[8]; } x0, x1, cs, sn;
  x0.u = *reinterpret_cast<const uint4*>(px);
  x1.u = *reinterpret_cast<const uint4*>(px + half);
  cs.u = __ldg(reinterpret_cast<const uint4*>(rcos + (size_t)l * half + c));
  sn.u = __ldg(reinterpret_cast<const uint4*>(rsin + (size_t)l * half + c));
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const float a = to_float(x0.e[i]), bb = to_float(x1.e[i]), cc = to_float(cs.e[i]), ss = to_float(sn.e[i]);
    x0.e[i] = from_float<IO>(a * cc - bb * ss);
    x1.e[i] = from_float<IO>(a * ss + bb * cc);
  }
  *reinterpret_cast<uint4*>(px) = x0.u;
  *reinterpret_cast<uint4*>(px + half) = x1.u;
  if (part == 1) {
    *reinterpret_cast<uint4*>(crow + c) = x0.u;
    *reinterpret_cast<uint4*>(crow + c + half) = x1.u;
  }
}

}  // namespace

int launch_rotary_qkv_cache(void* qkv, int B, int L, int H, int hd, int64_t sb, int64_t sl, int64_t s3, int64_t sh,
                            const void* rcos, const void* rsin, void* cache, int64_t cb, int64_t cl,
                            cudaStream_t stream) {
  if (hd % 16 != 0) return BASED_ERR_SHAPE;
  const int64_t strides[] = {sb, sl, s3, sh, cb, cl};
  for (int64_t s : strides)
    if (s % 8 != 0) return BASED_ERR_ALIGN;
  if (!aligned16(qkv) || !aligned16(rcos) || !aligned16(rsin) || !aligned16(cache)) return BASED_ERR_ALIGN;
  const long long total = (long long)B * L * H * (hd / 4);
  if (total == 0) return 0;
  const long long blocks = (total + 255) / 256;
  if (blocks > 2147483647LL) return BASED_ERR_TOO_LARGE;
  launch_pdl(rotary_qkv_cache_kernel, (unsigned)blocks, 256, 0, stream, 
      static_cast<__nv_bfloat16*>(qkv), L, H, hd, sb, sl, s3, sh, static_cast<const __nv_bfloat16*>(rcos),
      static_cast<const __nv_bfloat16*>(rsin), static_cast<__nv_bfloat16*>(cache), cb, cl, total);
  return (int)cudaGetLastError();
}

int launch_rotary(void* x, int B, int L, int H, Strides3 sx, const void* rcos, const void* rsin, int rotary_dim,
                  const int32_t* offsets, int offset_scalar, int io_dtype, cudaStream_t stream) {
  const int half = rotary_dim / 2;
  const int threads = 256;
  if (io_dtype != BASED_BF16 && io_dtype != BASED_F32) return BASED_ERR_DTYPE;
  {
    // 16-byte path when every access it makes is aligned
    const int N = io_dtype == BASED_BF16 ? 8 : 4;
    if (half % N == 0 && sx.b % N == 0 && sx.l % N == 0 && sx.h % N == 0 && aligned16(x) && aligned16(rcos) &&
        aligned16(rsin)) {
      const long long total = (long long)B * L * H * (half / N);
      if (total == 0) return 0;
      const long long blocks = (total + threads - 1) / threads;
      if (blocks > 2147483647LL) return BASED_ERR_TOO_LARGE;
      if (io_dtype == BASED_BF16) {
        using T = __nv_bfloat16;
        rotary_vec_kernel<T><<<(unsigned)blocks, threads, 0, stream>>>(
            static_cast<T*>(x), L, H, sx, static_cast<const T*>(rcos), static_cast<const T*>(rsin), half, offsets,
            offset_scalar, total);
      } else {
        rotary_vec_kernel<float><<<(unsigned)blocks, threads, 0, stream>>>(
            static_cast<float*>(x), L, H, sx, static_cast<const float*>(rcos), static_cast<const float*>(rsin), half,
            offsets, offset_scalar, total);
      }
      return (int)cudaGetLastError();
    }
  }
  const long long total = (long long)B * L * H * half;
  if (total == 0) return 0;
  const long long blocks = (total + threads - 1) / threads;
  if (blocks > 2147483647LL) return BASED_ERR_TOO_LARGE;
  if (io_dtype == BASED_BF16) {
    using T = __nv_bfloat16;
    rotary_kernel<T><<<(unsigned)blocks, threads, 0, stream>>>(static_cast<T*>(x), L, H, sx, static_cast<const T*>(rcos),
                                                              static_cast<const T*>(rsin), half, offsets,
                                                              offset_scalar, total);
  } else if (io_dtype == BASED_F32) {
    rotary_kernel<float><<<(unsigned)blocks, threads, 0, stream>>>(
        static_cast<float*>(x), L, H, sx, static_cast<const float*>(rcos), static_cast<const float*>(rsin), half,
        offsets, offset_scalar, total);
  } else {
    return BASED_ERR_DTYPE;
  }
  return (int)cudaGetLastError();
}

int launch_swa_prefill_simt(const void* q, const void* k, const void* v, void* o, int B, int L, int H, int hd,
                            Strides3 sq, Strides3 sk, Strides3 sv, Strides3 so, int window_left, float scale,
                            int io_dtype, cudaStream_t stream) {
  if (window_left + 1 > kMaxKeysPerLane * 32) return BASED_ERR_TOO_LARGE;
  const dim3 grid((L + kWarpsPerBlock - 1) / kWarpsPerBlock, H, B);
  if (io_dtype == BASED_BF16) {
    using T = __nv_bfloat16;
    swa_prefill_simt_kernel<T><<<grid, kWarpsPerBlock * 32, 0, stream>>>(
        static_cast<const T*>(q), static_cast<const T*>(k), static_cast<const T*>(v), static_cast<T*>(o), L, H, hd,
        sq, sk, sv, so, window_left, scale);
  } else if (io_dtype == BASED_F32) {
    swa_prefill_simt_kernel<float><<<grid, kWarpsPerBlock * 32, 0, stream>>>(
        static_cast<const float*>(q), static_cast<const float*>(k), static_cast<const float*>(v),
        static_cast<float*>(o), L, H, hd, sq, sk, sv, so, window_left, scale);
  } else {
    return BASED_ERR_DTYPE;
  }
  return (int)cudaGetLastError();
}

int launch_swa_decode(const void* q, const void* k_new, const void* v_new, void* o, void* kv_cache,
                      const int32_t* cache_seqlens, int cache_seqlen_scalar, const void* rotary_cos,
                      const void* rotary_sin, int rotary_dim, int B, int H, int hd, int max_seqlen, Strides2 sq,
                      Strides2 sk, Strides2 sv, Strides2 so, int window_left, float scale, int io_dtype,
                      cudaStream_t stream) {
  if (window_left + 1 > kMaxKeysPerLane * 32) return BASED_ERR_TOO_LARGE;
  if (!aligned16(kv_cache) || hd % 8 != 0) return BASED_ERR_ALIGN;  // 16-byte reads of cached rows
  if ((int64_t)B * H > 0x7fffffff) return BASED_ERR_TOO_LARGE;
  const int BH = B * H;
  auto run = [&](auto zero) {
    using T = decltype(zero);
    auto go = [&](auto kern, int warps, int heads) {
      return launch_pdl(kern, dim3((BH - 1) / heads + 1), dim3(warps * heads * 32), 0, stream,
          static_cast<const T*>(q), static_cast<const T*>(k_new), static_cast<const T*>(v_new), static_cast<T*>(o),
          static_cast<T*>(kv_cache), cache_seqlens, cache_seqlen_scalar, static_cast<const T*>(rotary_cos),
          static_cast<const T*>(rotary_sin), rotary_dim, BH, H, hd, max_seqlen, sq, sk, sv, so, window_left, scale);
    };
    // Warps per head: few heads want the window in flight at once, many heads fewer blocks and warps.  us with 1 / 2 / 4 / 8 warps (one
    // warp: four heads to a block), windows of 16, 32, 64, 128 keys.  hd = 64: 16 heads 3.2 / 2.6 / 2.6, 3.7 / 2.7 / 2.7, 5.0 / 3.2 / 2.7,
    // 7.5 / 4.2 / 3.2; 512 heads 3.5 / 4.0 / 4.5, 4.2 / 4.0 / 4.6, 5.5 / 4.9 / 4.6, 8.2 / 6.8 / 6.0; 4096 heads 7.6 / 10.6 / 16, 9.5 / 10.8 / 17,
    // 15.9 / 15.1 / 17.6, 31 / 28 / 28.  hd = 112: 16 heads - / 3.0 / 2.8 / 3.2, - / 3.6 / 2.8 / 3.4, - / 4.8 / 3.4 / 3.4, - / 7.1 / 4.6 / 4.0; 4096 heads
    // 12.5 / 12.4 / 19 / 36, 18.5 / 16.7 / 20 / 37, 33 / 27 / 29 / 41, 56 / 47 / 46 / 56.
    const int keys = window_left + 1;
    const bool many = BH > 5 * 148;
    if (hd <= 64) {
      const int warps = many ? (keys <= 40 ? 1 : keys <= 80 ? 2 : 4) : (keys <= 40 ? 2 : 4);
      if (warps == 1) return go(swa_decode_kernel<T, 8, 1, 4>, 1, 4);
      if (warps == 2) return go(swa_decode_kernel<T, 8, 2, 1>, 2, 1);
      return go(swa_decode_kernel<T, 8, 4, 1>, 4, 1);
    }
    const int warps = many ? (keys <= 9 ? 1 : keys <= 40 ? 2 : 4) : (keys <= 80 ? 4 : 8);
    if (warps == 1) return go(swa_decode_kernel<T, 16, 1, 4>, 1, 4);
    if (warps == 2) return go(swa_decode_kernel<T, 16, 2, 1>, 2, 1);
    if (warps == 4) return go(swa_decode_kernel<T, 16, 4, 1>, 4, 1);
    return go(swa_decode_kernel<T, 16, 8, 1>, 8, 1);
  };
  if (io_dtype == BASED_BF16) return launched(run(__nv_bfloat16{}));
  if (io_dtype == BASED_F32) return launched(run(float{}));
  return BASED_ERR_DTYPE;
}

}  // namespace based
