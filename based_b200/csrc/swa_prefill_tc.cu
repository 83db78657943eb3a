// Causal sliding-window softmax attention over a whole sequence on the sm_100a tensor cores
// (tcgen05.mma, accumulators in TMEM), bf16 I/O: a banded, one-pass flash-style kernel.
//
// Replaces the flash-attn calls of the reference's SlidingAttention
// (based/models/mixers/slide_attention.py:100-106, :206-213: causal=True,
// window_size=(window_left, 0), i.e. query i attends keys [i - window_left, i]).
//
// A tile is 128 queries of one (batch, head) and the NK = 128 + window_left keys that any of them can see:
//   S = Q K^T            (M128, N = NK, K = head_dim)          -> TMEM, fp32
//   P = exp2(scale*(S - rowmax)) under the band mask           CUDA cores, two threads per query
//       row, half of its visible keys each, all of them in registers; all keys of a row are present, so the
//       softmax is exact in one pass; P (bf16) overwrites S in place and becomes the A operand
//   O = P V              (M128, N = head_dim, K = NK)          -> TMEM, over the columns of S that P left
//   out = O / rowsum
// Q, K, V tiles arrive by TMA (128-byte swizzle, zero fill outside the sequence) and the output tile leaves by TMA.
// A tile's life is a chain, and HBM is busy only while enough tiles are on their way: persistent CTAs, two to an SM (256 TMEM columns
// hold S and O of every size taken here), eight softmax warps and one warp that issues the copies and the products.  Q and K of the
// next tile are asked for when S is done, V when O is done, and the output leaves under the next S.  A tile takes a CTA 3.7 us; with
// the copies issued by a softmax warp it took 4.7 (700 to 900 cycles each time: coordinates, descriptors, the wait for the store), and
// as a CTA of its own, three to an SM, 4.1 for two at a time.
// us, one after the other in a graph, a CTA per tile with O beside S and a thread per row / now (B x H x L, head, window; floor at the HBM
// rate): 8x16x8192, 64, 64 116.8 / 104 (82; a lone call 125); 4x16x8192, 64, 32 57 / 46 (41); 64, 128 123 / 93 (41); 112, 64 174 / 91 (72);
// 2x16x8192, 128, 128 106 / 61 (41).
#include "common.cuh"
#include "tcgen05.cuh"
#include "tma.cuh"

#include <algorithm>
#include <mutex>

namespace based {

__device__ unsigned int g_tc_status_swa = 0;


namespace {

using namespace tc;

constexpr int TQ = 128;  // queries per tile
constexpr int kCompute = 8, NT = (kCompute + 1) * 32;  // softmax warps; threads per CTA
constexpr uint32_t kTmem = 256;   // columns: S, then P in the first half of them and O behind it

struct Params {
  CUtensorMap mq, mk, mv, mo;  // [B][H][L][hd] views, box = (<= 64 columns) x (rows), 128-byte swizzle
  int L, H, hd, W, tiles_per_seq, tiles;
  float scale_log2e;
  unsigned int* status;
};

// PC: pieces of 16 keys of a thread, (W + 32) / 32
template <int PC>
__global__ void __launch_bounds__(NT, PC <= 3 ? 2 : 1) swa_prefill_tc_kernel(const __grid_constant__ Params p) {
  extern __shared__ uint8_t smem_raw[];
  // the swizzled tiles need a 1024-byte aligned base
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  const uint32_t sb = smem_u32(smem);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int W = 32 * (PC - 1), NK = TQ + W;
  const int hd = p.hd, quad = warp & 3, half = warp >> 2;   // rows of a warp, which of the two warps they have
  // shared memory: per 64-column atom a of the head dimension, a 128-byte-swizzled tile with
  // 128-byte rows: Q[a] 128 rows, K[a] and V[a] NK rows, and the output tile.
  const int natom = (hd + 63) >> 6;
  const uint32_t q_atom = TQ * 128, kv_atom = (uint32_t)NK * 128;
  const uint32_t SM_Q = 0, SM_K = natom * q_atom, SM_V = SM_K + natom * kv_atom, SM_O = SM_V + natom * kv_atom, SM_BAR = SM_O + natom * q_atom;
  // loads landed; S, O computed; P written (by all warps); O read and the output tile written; the output tile read by its store
  const uint32_t bars = sb + SM_BAR, bar_qk = bars, bar_v = bars + 8, bar_s = bars + 16, bar_o = bars + 24, bar_p = bars + 32, bar_out = bars + 40, bar_free = bars + 48;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + SM_BAR + 56);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + SM_BAR + 60);
  float* rowmax = reinterpret_cast<float*>(smem + SM_BAR + 64);   // [2][128], then the sums
  if (tid == 0) {
    for (uint32_t bar : {bar_qk, bar_v, bar_s, bar_o, bar_free}) mbar_init(bar, 1);
    mbar_init(bar_p, kCompute);
    mbar_init(bar_out, kCompute);
    *abort_flag = 0;
    fence_mbar_init();
    fence_proxy_async();
  }
  // A tile's operands, one TMA tile each and column atom; rows outside [0, L) read as zero.  Every box is 64 columns wide (columns past
  // hd are out of bounds: zero-filled, and counted).  Head index fastest: CTAs that run at the same time then read the SAME token rows
  // of the packed projection (H x 128 contiguous bytes per row and part) instead of one 128-byte piece out of every row's 6 KB.
  auto load_qk = [&](int h, int t0, int b) {
    tma::mbar_expect_tx(bar_qk, (uint32_t)natom * 128u * (TQ + NK));
    for (int a = 0; a < natom; ++a) {
      tma::load_4d(sb + SM_Q + a * q_atom, &p.mq, bar_qk, 64 * a, t0, h, b);
      tma::load_4d(sb + SM_K + a * kv_atom, &p.mk, bar_qk, 64 * a, t0 - W, h, b);
    }
  };
  auto load_v = [&](int h, int t0, int b) {
    tma::mbar_expect_tx(bar_v, (uint32_t)natom * 128u * NK);
    for (int a = 0; a < natom; ++a) tma::load_4d(sb + SM_V + a * kv_atom, &p.mv, bar_v, 64 * a, t0 - W, h, b);
  };
  auto place = [&](int tile, int& h, int& t0, int& b) {
    h = tile % p.H;
    tile /= p.H;
    t0 = tile % p.tiles_per_seq * TQ;
    b = tile / p.tiles_per_seq;
  };
  __syncthreads();
  if (warp == kCompute && elect_one_sync() && (int)blockIdx.x < p.tiles) {   // the first loads do not wait for TMEM
    int h, t0, b;
    place(blockIdx.x, h, t0, b);
    load_qk(h, t0, b);
    load_v(h, t0, b);
  }
  __syncwarp();
  if (warp == 0) tmem_alloc(smem_u32(tmem_slot), kTmem);
  fence_before_sync();
  __syncthreads();  // TMEM base published
  fence_after_sync();
  const uint32_t tmem = *tmem_slot;
  const uint32_t tlane = tmem + ((uint32_t)(quad * 32) << 16);
  const uint32_t TM_S = 0, TM_O = NK / 2;
  uint32_t phase = 0;   // every barrier completes once a tile

  if (warp == kCompute) {
    // ---- copies and products.  Converged, one elected lane issues: the descriptors are then values the compiler can keep in uniform
    // registers, instead of being moved there, several moves per MMA, by a single diverged lane.
    const uint32_t tmem_u = __shfl_sync(0xffffffffu, tmem, 0);
    const bool leader = elect_one_sync();
    int h, t0, b, ph = 0, pt = 0, pb = 0;   // the next tile; the one before
    for (int tile = blockIdx.x; tile < p.tiles; tile += gridDim.x, phase ^= 1) {
      const int next = tile + gridDim.x;
      mbar_wait_bounded(bar_qk, phase, abort_flag, p.status, 64u);
      if (tile != (int)blockIdx.x) mbar_wait_bounded(bar_out, phase ^ 1, abort_flag, p.status, 256u);
      fence_after_sync();
      {
        const uint32_t idesc = make_idesc_bf16(128, NK, 0, 0);
        int first = 1;
        for (int a = 0; a < natom; ++a) {
          const int ksteps = (min(64, hd - 64 * a)) >> 4;
          for (int ks = 0; ks < ksteps; ++ks) {  // a K-step of 16 elements = 32 bytes inside the swizzled row
            const uint64_t da = make_smem_desc_sw128(sb + SM_Q + a * q_atom + ks * 32, 16, 1024);
            const uint64_t db = make_smem_desc_sw128(sb + SM_K + a * kv_atom + ks * 32, 16, 1024);
            if (leader) mma_ss(tmem_u + TM_S, da, db, idesc, first ? 0u : 1u);
            first = 0;
          }
        }
        if (leader) mma_commit(bar_s);
      }
      if (tile != (int)blockIdx.x && leader) {   // the tile before leaves
        for (int a = 0; a < natom; ++a) tma::store_4d(&p.mo, sb + SM_O + a * q_atom, 64 * a, pt, ph, pb);
        bulk_commit();
      }
      place(tile, ph, pt, pb);
      if (next < p.tiles) place(next, h, t0, b);
      if (tile != (int)blockIdx.x && leader) {
        bulk_wait_read_all();
        mbar_arrive(bar_free);
      }
      __syncwarp();
      mbar_wait_bounded(bar_s, phase, abort_flag, p.status, 16u);
      if (next < p.tiles && leader) load_qk(h, t0, b);   // Q and K have been read
      __syncwarp();
      mbar_wait_bounded(bar_v, phase, abort_flag, p.status, 128u);
      mbar_wait_bounded(bar_p, phase, abort_flag, p.status, 256u);
      fence_after_sync();
      {
        // V tiles are MN-major: 64-column atoms kv_atom apart (LBO), groups of 8 keys 1024 B apart (SBO)
        const uint32_t idesc = make_idesc_bf16(128, hd, 0, 1);
        for (int ks = 0; ks < (NK >> 4); ++ks) {
          const uint64_t dvd = make_smem_desc_sw128(sb + SM_V + ks * 2048, kv_atom, 1024);
          if (leader) mma_ts(tmem_u + TM_O, tmem_u + TM_S + 8 * ks, dvd, idesc, ks > 0);
        }
        if (leader) mma_commit(bar_o);
      }
      __syncwarp();
      mbar_wait_bounded(bar_o, phase, abort_flag, p.status, 32u);
      if (next < p.tiles && leader) load_v(h, t0, b);
      __syncwarp();
    }
    if ((int)blockIdx.x < p.tiles) {
      mbar_wait_bounded(bar_out, phase ^ 1, abort_flag, p.status, 256u);
      if (leader) {
        for (int a = 0; a < natom; ++a) tma::store_4d(&p.mo, sb + SM_O + a * q_atom, 64 * a, pt, ph, pb);
        bulk_commit();
        bulk_wait_read_all();   // shared memory must stay intact until the TMA unit has read it
      }
      __syncwarp();
    }
  } else {
  for (int tile = blockIdx.x; tile < p.tiles; tile += gridDim.x, phase ^= 1) {
  const int t0 = tile / p.H % p.tiles_per_seq * TQ, k0 = t0 - W;   // position of key column 0 (may be negative)
  // ---- softmax of row t over the band: this warp's rows need W + 32 key columns, from c_lo on; this thread has the half from lo_col ----
  // Relative to the first of them, row `lane` sees columns [lane, lane + W]; only the first tile of a sequence also has keys before
  // position 0 (columns below first_col).
  const int c_lo = quad * 32, lo_col = half * 16 * PC, first_col = -k0 - c_lo;
  mbar_wait_bounded(bar_s, phase, abort_flag, p.status, 16u);
  fence_after_sync();
  uint32_t r[PC][16], mask[PC];   // bit i of a mask: column i of the piece is visible
#pragma unroll
  for (int pc = 0; pc < PC; ++pc) tmem_ld16(tlane + TM_S + c_lo + lo_col + 16 * pc, r[pc]);
#pragma unroll
  for (int pc = 0; pc < PC; ++pc) {
    const int at = lo_col + 16 * pc, lo = max(max(lane, first_col) - at, 0), hi = min(lane + W - at, 15);
    mask[pc] = lo <= hi ? (0xFFFFFFFFu << lo) & (0xFFFFFFFFu >> (31 - hi)) : 0u;
  }
  tmem_ld_wait();
  // maximum and sum in four independent lanes each, so that neither is a chain of all the columns
  float m4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY}, sum4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int pc = 0; pc < PC; ++pc)
#pragma unroll
    for (int i = 0; i < 16; ++i) m4[i & 3] = fmaxf(m4[i & 3], (mask[pc] & (1u << i)) ? __uint_as_float(r[pc][i]) : -INFINITY);
  const int row = quad * 32 + lane;
  const float mine = fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3]));
  rowmax[half * TQ + row] = mine;
  fence_before_sync();   // the other warp's P goes over the scores that this one has read
  asm volatile("bar.sync %0, 64;\n" ::"r"(1 + quad) : "memory");   // the two warps of these rows
  fence_after_sync();
  const float msc = fmaxf(mine, rowmax[(half ^ 1) * TQ + row]) * p.scale_log2e;
#pragma unroll
  for (int pc = 0; pc < PC; ++pc) {
    uint32_t pk[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      float e[2];
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int ii = 2 * i + j;
        float val;
        asm("ex2.approx.ftz.f32 %0, %1;\n" : "=f"(val) : "f"(fmaf(__uint_as_float(r[pc][ii]), p.scale_log2e, -msc)));
        e[j] = (mask[pc] & (1u << ii)) ? val : 0.f;
      }
      pk[i] = pack_bf16(e[0], e[1]);
      // the normaliser sums what the MMA will see: the bf16-rounded probabilities
      sum4[i & 3] += __uint_as_float(pk[i] << 16) + __uint_as_float(pk[i] & 0xffff0000u);
    }
    tmem_st8(tlane + TM_S + ((c_lo + lo_col + 16 * pc) >> 1), pk);
  }
  float* rowsum = rowmax + 2 * TQ;
  rowsum[half * TQ + row] = (sum4[0] + sum4[1]) + (sum4[2] + sum4[3]);
  // zero the P columns of keys this warp's rows cannot see: 16 data columns at a time, every second one this thread's
  {
    uint32_t z[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) z[i] = 0;
    const int p_lo = c_lo >> 1, p_hi = p_lo + 16 * PC;  // data columns [p_lo, p_hi)
    int mine_next = half;
    for (int c = 0; c < (NK >> 1); c += 16)
      if ((c < p_lo || c >= p_hi) && (mine_next ^= 1)) tmem_st16(tlane + TM_S + c, z);
  }
  tmem_st_wait();
  fence_before_sync();
  __syncwarp();
  if (lane == 0) mbar_arrive(bar_p);

  // ---- epilogue ----
  mbar_wait_bounded(bar_o, phase, abort_flag, p.status, 32u);
  fence_after_sync();
  if (tile != (int)blockIdx.x) mbar_wait_bounded(bar_free, phase ^ 1, abort_flag, p.status, 256u);   // the tile before has left the output tile
  {
    // Each thread writes its normalised row into the output tile in the 128-byte-swizzled layout; it leaves by TMA,
    // which clips rows past the end of the sequence.
    const float inv = 1.0f / (rowsum[row] + rowsum[TQ + row]);
    const int t = row;
    auto put = [&](int i, const uint32_t (&r)[16]) {
      uint4 lo, hi;
      lo.x = pack_bf16(__uint_as_float(r[0]) * inv, __uint_as_float(r[1]) * inv);
      lo.y = pack_bf16(__uint_as_float(r[2]) * inv, __uint_as_float(r[3]) * inv);
      lo.z = pack_bf16(__uint_as_float(r[4]) * inv, __uint_as_float(r[5]) * inv);
      lo.w = pack_bf16(__uint_as_float(r[6]) * inv, __uint_as_float(r[7]) * inv);
      hi.x = pack_bf16(__uint_as_float(r[8]) * inv, __uint_as_float(r[9]) * inv);
      hi.y = pack_bf16(__uint_as_float(r[10]) * inv, __uint_as_float(r[11]) * inv);
      hi.z = pack_bf16(__uint_as_float(r[12]) * inv, __uint_as_float(r[13]) * inv);
      hi.w = pack_bf16(__uint_as_float(r[14]) * inv, __uint_as_float(r[15]) * inv);
      uint8_t* atom = smem + SM_O + (i >> 2) * q_atom;  // 16 columns = 2 chunks; 4 such pieces per 64-column atom
      *reinterpret_cast<uint4*>(atom + tma::sw128_offset(t, 2 * (i & 3))) = lo;
      *reinterpret_cast<uint4*>(atom + tma::sw128_offset(t, 2 * (i & 3) + 1)) = hi;
    };
    const int np = hd >> 4;   // pieces of 16 columns: every second one this thread's, two loads in flight
    for (int i0 = half; i0 < np; i0 += 4) {
      uint32_t ra[16], rb[16];
      tmem_ld16(tlane + TM_O + 16 * i0, ra);
      if (i0 + 2 < np) tmem_ld16(tlane + TM_O + 16 * (i0 + 2), rb);
      tmem_ld_wait();
      put(i0, ra);
      if (i0 + 2 < np) put(i0 + 2, rb);
    }
    fence_proxy_async();  // generic-proxy writes -> visible to the TMA unit
    fence_before_sync();  // the accumulators may be overwritten
    __syncwarp();
    if (lane == 0) mbar_arrive(bar_out);
  }
  }
  }
  fence_before_sync();
  __syncthreads();
  if (warp == 0) {
    fence_after_sync();
    tmem_dealloc(tmem, kTmem);
  }
}

}  // namespace


int read_tc_status_swa(unsigned int* out, int reset) {
  unsigned int v = 0;
  cudaError_t e = cudaMemcpyFromSymbol(&v, g_tc_status_swa, sizeof(v));
  if (e != cudaSuccess) return (int)e;
  if (out) *out = v;
  if (reset && v != 0) {
    v = 0;
    e = cudaMemcpyToSymbol(g_tc_status_swa, &v, sizeof(v));
  }
  return (int)e;
}

int launch_swa_prefill_tc(const void* q, const void* k, const void* v, void* o, int B, int L, int H, int hd,
                          Strides3 sq, Strides3 sk, Strides3 sv, Strides3 so, int window_left, float scale,
                          cudaStream_t stream) {
  // Requirements of this kernel; the caller may fall back to the CUDA-core kernel on ERR_IMPL.
  if (window_left % 32 != 0 || window_left < 0 || window_left > 128) return BASED_ERR_IMPL;
  if (!aligned16(q) || !aligned16(k) || !aligned16(v) || !aligned16(o)) return BASED_ERR_IMPL;
  const int64_t all[] = {sq.b, sq.h, sq.l, sk.b, sk.h, sk.l, sv.b, sv.h, sv.l, so.b, so.h, so.l};
  for (int64_t s : all)
    if (s % 8 != 0 || s <= 0) return BASED_ERR_IMPL;  // TMA strides: positive multiples of 16 bytes
  if (hd > 128 || hd % 16 != 0) return BASED_ERR_IMPL;   // S and O share kTmem columns
  static constexpr void (*kKernels[5])(const Params) = {swa_prefill_tc_kernel<1>, swa_prefill_tc_kernel<2>, swa_prefill_tc_kernel<3>, swa_prefill_tc_kernel<4>,
                                                        swa_prefill_tc_kernel<5>};
  const int NK = TQ + window_left;
  const int tiles_per_seq = (L + TQ - 1) / TQ;
  const long long tiles = (long long)B * H * tiles_per_seq;
  if (tiles > 2147483647LL) return BASED_ERR_TOO_LARGE;
  Params p;
  // tensor maps over [B][H][L][hd] (dims innermost first: hd, L, H, B); a batch or head extent of 1
  // may come with any stride, so give those a harmless one.  Maps are cached by pointer and geometry.
  static tma::MapCache cache;
  auto fix = [&](int64_t s, int extent) { return extent == 1 ? (int64_t)8 : s; };
  auto get_map = [&](CUtensorMap* out, const void* base, Strides3 s, int rows) -> int {
    const tma::MapKey key = tma::make_key(base, (uint64_t)hd, (uint64_t)L, (uint64_t)H, (uint64_t)B, 0, s.l, fix(s.h, H),
                                          fix(s.b, B), 0, 64, (uint32_t)rows, 0, 4);
    if (cache.find(key, out)) return 0;
    if (tma::encode_bf16_4d_sw128(out, base, hd, L, H, B, s.l, fix(s.h, H), fix(s.b, B), 64, rows)) return BASED_ERR_IMPL;
    cache.put(key, *out);
    return 0;
  };
  if (get_map(&p.mq, q, sq, TQ) || get_map(&p.mk, k, sk, NK) || get_map(&p.mv, v, sv, NK) || get_map(&p.mo, o, so, TQ))
    return BASED_ERR_IMPL;
  p.L = L; p.H = H; p.hd = hd; p.W = window_left; p.tiles_per_seq = tiles_per_seq;
  p.scale_log2e = scale * 1.4426950408889634f;
  const int natom = (hd + 63) / 64;
  const int smem = natom * (2 * TQ + 2 * NK) * 128 + 64 + 4 * TQ * 4 + 1024;  // + slack to align the tiles to 1024 bytes
  {
    // once per device: the status word's address and the largest shared-memory size this kernel is launched with
    constexpr int kMaxDevices = 64;
    static std::mutex mu;
    static unsigned int* status[kMaxDevices] = {};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return (int)e;
    if (dev < 0 || dev >= kMaxDevices) return BASED_ERR_TOO_LARGE;
    std::lock_guard<std::mutex> lock(mu);
    if (status[dev] == nullptr) {
      unsigned int* addr = nullptr;
      e = cudaGetSymbolAddress(reinterpret_cast<void**>(&addr), g_tc_status_swa);
      if (e != cudaSuccess) return (int)e;
      for (int i = 0; i < 5; ++i) {
        const int max_smem = 2 * (2 * TQ + 2 * (TQ + 32 * i)) * 128 + 64 + 4 * TQ * 4 + 1024;   // head_dim 128
        e = cudaFuncSetAttribute(kKernels[i], cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem);
        if (e != cudaSuccess) return (int)e;
      }
      status[dev] = addr;
    }
    p.status = status[dev];
  }
  p.tiles = (int)tiles;
  // (a window of more than 64 keys: 80 scores a thread, which leave no registers for a second CTA)
  const int resident = 148 * (smem <= 113 * 1024 && window_left <= 64 ? 2 : 1);
  kKernels[window_left / 32]<<<(unsigned)std::min<long long>(tiles, resident), NT, smem, stream>>>(p);
  return (int)cudaGetLastError();
}

}  // namespace based
