// Packed keys and values -> fp16 rows in the original coordinates, as operand tiles of the dense attention kernel.
//
//   K'[k] = n_k C[idx_k] Pi_k + sqrt(pi/2)/d rn_k (+-1)_k (S_eff Pi_k)      V'[k] = n_k C_v[idx_k] Pi_v
//
// so that <q, K'> is the estimator's score and softmax . V' the output: 4 d products per (query, key) pair instead of the
// 6 d of rotated and sketched queries against the two halves of a key, no rotation per query or output row, and one decode
// per key instead of one per tile of queries (a key of a 4096-token prompt is otherwise decoded by 64 clusters).
//
// Tiles of 128 rows: centroids (fp16, as in the SM-pair kernel's tables) and signs are A operands in shared memory, the
// matrices (fp16, scaled by a power of two) B operands that stay there for the CTA's life; two accumulators per key tile,
// so that both norms and the scales are applied in fp32 and a result is rounded to fp16 once.  Against the SM-pair kernel
// (bf16 matrices, fp16 products n C, bf16 output rows) the rounding of everything but the centroids is 8 times finer.
// A CTA does key tiles or value tiles: eight warps decode, one issues the MMAs, eight store, with two operand and two
// accumulator slots between them.  Output tiles have the canonical core-matrix layout (16 bytes of eight consecutive rows
// adjacent), which is the K-major operand of q K'^T and the MN-major operand of P V' at once: one contiguous copy each.
#include <limits.h>

#include <algorithm>
#include <type_traits>

#include "tq_attention.cuh"
#include "tq_common.cuh"
#include "tq_dense.cuh"
#include "tq_simt.cuh"
#include "tq_tcgen05.cuh"

namespace tq {

__device__ unsigned long long g_expand_faults = 0ull;
// this device's slot of the host-visible status page (NULL until the first call on the device installs it)
__device__ unsigned long long* g_fault_mailbox_expand = nullptr;
int set_fault_mailbox_expand(unsigned long long* slot) {
  TQ_CUDA_OK(cudaMemcpyToSymbol(g_fault_mailbox_expand, &slot, sizeof(slot)));
  return TQ_OK;
}
int read_expand_faults(unsigned long long* out) {
  TQ_CUDA_OK(cudaMemcpyFromSymbol(out, g_expand_faults, sizeof(*out)));
  return TQ_OK;
}

namespace {

constexpr int kDecodeWarps = 8, kStoreWarps = 8, kMmaWarp = kDecodeWarps + kStoreWarps, kThreads = 32 * (kMmaWarp + 1);

// 8 B-bit indices in `bits` -> 8 fp16 centroids through the pair table
template <int B>
__device__ __forceinline__ uint4 centroids8(const uint32_t* lut, uint32_t bits) {
  uint32_t o[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) o[q] = lut[(bits >> (2 * q * B)) & ((1u << (2 * B)) - 1)];
  return make_uint4(o[0], o[1], o[2], o[3]);
}
// 8 sign bits -> 8 fp16 +-1 (a set bit is +1)
__device__ __forceinline__ uint4 signs8(uint32_t bits) {
  uint32_t o[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) o[q] = 0x3c003c00u ^ ((((~bits >> (2 * q)) & 3u) * 0x40008000u) & 0x80008000u);
  return make_uint4(o[0], o[1], o[2], o[3]);
}

// Limits of a call whose hidden tiles are left out: tiles of a CTA, words of the map of tiles that are computed, and what a CTA
// reads of the mask's summary to draw it.
constexpr int kOwnTiles = 256, kLiveWords = 256, kListMapThreads = 384, kSummaryReads = 30 * kThreads;

struct LiveMap {
  uint32_t words[kLiveWords];  // [batch elements][(T + 31) / 32]: some query sees a key of the tile
  uint8_t all[kLiveWords];     // [batch elements]: a row sees nothing and averages all keys of its causal range
  int count[kLiveWords];       // [batch elements]: tiles that are computed
  int tile[kOwnTiles + 1];     // this CTA's tiles, then one past the last of all
};
// This CTA's share of the tiles that some query computes, spread evenly over the CTAs.  `m.words` and `m.all` are zeros.  The
// expansion waits for it, so the two halves of the summary are read side by side, and threads find their tiles without diverging.
__device__ __forceinline__ void list_tiles(const ExpandArgs& a, int cta, int ctas, LiveMap& m) {
  const int tid = threadIdx.x, W = (a.T + 31) / 32, b0 = a.mb.batch ? (int)(a.pair0 / a.Hkv) : 0;
  const int nb = a.mb.batch ? (int)((a.pair0 + a.pairs - 1) / a.Hkv) - b0 + 1 : 1;
  if (tid < kListMapThreads) {
    for (int e = tid; e < nb * a.T * a.parts; e += kListMapThreads) {
      const int bt = e / a.parts, bi = bt / a.T, t = bt - bi * a.T;
      const uint8_t* cls = a.mb.tiles + (int64_t)(b0 + bi) * a.mb.NG * a.T + t;
      uint32_t seen = 0;
#pragma unroll 8
      for (int g = e - bt * a.parts; g < a.mb.NG; g += a.parts) seen |= cls[(int64_t)g * a.T];
      if ((seen & 1u) != 0u) atomicOr(&m.words[bi * W + t / 32], 1u << (t % 32));
    }
  } else {
    for (int e = tid - kListMapThreads; e < nb * a.mb.NG; e += kThreads - kListMapThreads) {
      const int bi = e / a.mb.NG, g = e - bi * a.mb.NG;
      const uint32_t* rows = a.mb.rows + ((int64_t)b0 * a.mb.NG + e) * a.mb.NC;
      uint32_t seen = 0;
#pragma unroll 8
      for (int c = 0; c < a.mb.NC; ++c) seen |= rows[c];
      if ((~seen & ((1u << min(16, a.Sq - 16 * g)) - 1u)) != 0u) m.all[bi] = 1;
    }
  }
  __syncthreads();
  if (tid < nb) {
    int n = 0;
    for (int w = 0; w < W; ++w) n += __popc(m.words[tid * W + w]);
    m.count[tid] = m.all[tid] ? a.T : n;
  }
  __syncthreads();
  if (tid <= kOwnTiles) {
    const int Hkv = (int)a.Hkv, head0 = a.mb.batch ? (int)(a.pair0 - (int64_t)b0 * Hkv) : 0;  // (of the first pair)
    int at = tid < kOwnTiles ? cta + tid * ctas : INT_MAX, pair = 0, bi = 0, n = 1;
    for (; bi < nb; ++bi) {
      const int next = a.mb.batch ? min(a.pairs, (bi + 1) * Hkv - head0) : a.pairs;
      n = m.count[bi];
      if (at < n * (next - pair)) break;
      at -= n * (next - pair);
      pair = next;
    }
    int tile = a.pairs * a.T;
    if (bi < nb) {
      int t = at % n;
      tile = (pair + at / n) * a.T;
      if (!m.all[bi]) {  // the t-th bit of the map
        int w = bi * W;
        for (int c; (c = __popc(m.words[w])) <= t; ++w) t -= c;
        uint32_t bits = m.words[w];
        for (; t > 0; --t) bits &= bits - 1u;
        t = (w - bi * W) * 32 + __ffs((int)bits) - 1;
      }
      tile += t;
    }
    m.tile[tid] = tile;
  }
}

struct ExpandBars {
  uint32_t base;
  __device__ uint32_t a_full(int s) const { return base + 8u * s; }         // operand decoded: a decoding warp's arrival each
  __device__ uint32_t a_empty(int s) const { return base + 8u * (2 + s); }  // ... read by the MMAs
  __device__ uint32_t d_full(int s) const { return base + 8u * (4 + s); }   // accumulators complete
  __device__ uint32_t d_empty(int s) const { return base + 8u * (6 + s); }  // ... read: a storing warp's arrival each
  __device__ uint32_t constants() const { return base + 8u * 8; }
};

// The tiles of a CTA: cta, cta + ctas, ..., or those of a list; `tiles` or more behind the last.
template <bool LIST>
struct OwnTiles {
  int cta, ctas, tiles;
  const int* list;
  __device__ __forceinline__ int at(int i) const { return LIST ? list[i] : cta + i * ctas; }
};

template <int D, int BITS, bool KEY, bool LIST>
__device__ __forceinline__ bool expand_tiles(const ExpandArgs& a, uint8_t* smem, const uint32_t* lut, const ExpandBars bar, uint32_t tmem,
                                             volatile int* abort_flag, const OwnTiles<LIST> own) {
  constexpr int G = D / 8, NB = D / 32, B = KEY ? BITS - 1 : BITS;  // chunks and 32-coordinate blocks of a row, bits of an index
  constexpr int W = B + (KEY ? 1 : 0), NI = 128 * NB / (32 * kDecodeWarps);  // words of a block, blocks per decoding thread
  constexpr uint32_t MAT = D * D * 2, TILE = 128 * D * 2, SBO = G * 128;
  constexpr uint32_t kA = (KEY ? 2 : 1) * MAT, kASlot = (KEY ? 2 : 1) * TILE;  // operand slots behind the matrices
  const int tid = threadIdx.x, lane = tid % 32;
  const int warp = __shfl_sync(0xffffffffu, tid / 32, 0);
  const int tiles = own.tiles;
  bool ok = true;
  if (warp < kDecodeWarps) {
    uint32_t w[NI][W];
    auto load = [&](int tile) {
      const int64_t pair = a.pair0 + tile / a.T;
      const int k0 = tile % a.T * 128;
#pragma unroll
      for (int i = 0; i < NI; ++i) {
        const int e = i * 32 * kDecodeWarps + tid, r = e % 8 + 8 * (e / (8 * NB)), c = (e / 8) % NB;
        const int64_t row = pair * a.kv_stride + k0 + r;
        const bool live = k0 + r < a.Sk;
        const uint32_t* src = reinterpret_cast<const uint32_t*>((KEY ? a.key_idx : a.val_idx) + row * (G * B)) + c * B;
#pragma unroll
        for (int x = 0; x < B; ++x) w[i][x] = live ? src[x] : 0u;
        if (KEY) w[i][B] = live ? reinterpret_cast<const uint32_t*>(a.key_sgn + row * G)[c] : 0u;
      }
    };
    int tile = own.at(0);
    if (tile < tiles) load(tile);
    for (int i = 0; tile < tiles && ok; ++i) {
      const int s = i & 1;
      if (i >= 2 && !(ok = tc::mbar_spin_or_abort(bar.a_empty(s), ((i >> 1) - 1) & 1, abort_flag))) break;
#pragma unroll
      for (int n = 0; n < NI; ++n) {
        const int e = n * 32 * kDecodeWarps + tid, r = e % 8 + 8 * (e / (8 * NB)), c = (e / 8) % NB;
        uint8_t* dst = smem + kA + s * kASlot + (r / 8) * SBO + c * 512 + (r % 8) * 16;
#pragma unroll
        for (int x = 0; x < 4; ++x) {  // 8 coordinates: bits [8 B x, 8 B (x + 1)) of the block
          const int word = 8 * B * x / 32, shift = 8 * B * x % 32;
          const uint32_t bits = shift + 8 * B > 32 ? __funnelshift_r(w[n][word], w[n][word + 1 < B ? word + 1 : word], shift) : w[n][word] >> shift;
          *reinterpret_cast<uint4*>(dst + x * 128) = centroids8<B>(lut, bits);
          if (KEY) *reinterpret_cast<uint4*>(dst + TILE + x * 128) = signs8(w[n][B] >> (8 * x));
        }
      }
      tile = own.at(i + 1);
      if (tile < tiles) load(tile);
      tc::fence_async_smem();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(bar.a_full(s));
    }
  } else if (warp < kMmaWarp) {
    const int quad = warp % 4, half = (warp - kDecodeWarps) / 4, row = quad * 32 + lane;
    const float scale0 = a.scales[KEY ? 0 : 2], scale1 = KEY ? a.scales[1] : 0.f;
    uint16_t n0 = 0, n1 = 0;  // the row's norms
    auto load = [&](int tile) {
      const int key = tile % a.T * 128 + row;
      const int64_t at = (a.pair0 + tile / a.T) * a.kv_stride + key;
      n0 = key < a.Sk ? (KEY ? a.key_vn : a.val_vn)[at] : (uint16_t)0;
      if (KEY) n1 = key < a.Sk ? a.key_rn[at] : (uint16_t)0;
    };
    int tile = own.at(0);
    if (tile < tiles) load(tile);
    for (int i = 0, ahead; tile < tiles && ok; ++i, tile = ahead) {
      const int s = i & 1;
      const float f0 = fp16_value(n0) * scale0, f1 = fp16_value(n1) * scale1;
      // results stay finite where the norms are (a key of length 6e4 may come out a little longer than fp16 reaches)
      const bool finite = (n0 & 0x7c00u) != 0x7c00u && (n1 & 0x7c00u) != 0x7c00u;
      const bool live = tile % a.T * 128 + row < a.Sk;
      ahead = own.at(i + 1);
      if (ahead < tiles) load(ahead);
      if (!(ok = tc::mbar_spin_or_abort(bar.d_full(s), (i >> 1) & 1, abort_flag))) break;
      tc::fence_after_sync();
      uint8_t* out = a.dst + ((int64_t)tile * 2 + (KEY ? 0 : 1)) * TILE + (row / 8) * SBO + (row % 8) * 16;
#pragma unroll
      for (int c0 = 0; c0 < D / 2; c0 += 32) {
        const int col = half * (D / 2) + c0;
        const uint32_t addr = tmem + s * 2 * D + ((uint32_t)(quad * 32) << 16) + col;
        uint32_t u[32], v[32], o[16];
        tc::tmem_ld32(addr, u);
        if (KEY) tc::tmem_ld32(addr + D, v);
        tc::wait_ld();
        if (c0 + 32 == D / 2) {
          tc::fence_before_sync();
          __syncwarp();
          if (lane == 0) tc::mbar_arrive(bar.d_empty(s));
        }
        float y[32];
#pragma unroll
        for (int x = 0; x < 32; ++x) {
          y[x] = __uint_as_float(u[x]) * f0;
          if (KEY) y[x] = fmaf(__uint_as_float(v[x]), f1, y[x]);
        }
        if (finite) {
#pragma unroll
          for (int x = 0; x < 16; ++x) o[x] = tc::pack_f16x2_sat(y[2 * x], y[2 * x + 1]);
        } else {
#pragma unroll
          for (int x = 0; x < 16; ++x) o[x] = tc::pack_f16x2(y[2 * x], y[2 * x + 1]);
        }
#pragma unroll
        for (int x = 0; x < 4; ++x)  // rows past the last key are zeros: a probability of 0 meets them
          *reinterpret_cast<uint4*>(out + (col / 8 + x) * 128) =
              live ? make_uint4(o[4 * x], o[4 * x + 1], o[4 * x + 2], o[4 * x + 3]) : make_uint4(0u, 0u, 0u, 0u);
      }
    }
  } else {
    // the whole warp runs this loop and one elected lane issues: operands stay in uniform registers
    const uint64_t a0 = tc::smem_desc(tc::smem_u32(smem + kA), 128, SBO);
    const uint64_t b0 = tc::smem_desc(tc::smem_u32(smem), 128, SBO), b1 = tc::smem_desc(tc::smem_u32(smem + MAT), 128, SBO);
    constexpr uint32_t idesc = tc::idesc_f16(128, D, false, false);
    const bool leader = tc::elect_one();
    ok = tc::mbar_wait_or_abort(bar.constants(), 0, abort_flag);
    int i = 0;
    for (int tile = own.at(0); tile < tiles && ok; tile = own.at(++i)) {
      const int s = i & 1;
      if (!(ok = tc::mbar_spin_or_abort(bar.a_full(s), (i >> 1) & 1, abort_flag))) break;
      if (i >= 2 && !(ok = tc::mbar_spin_or_abort(bar.d_empty(s), ((i >> 1) - 1) & 1, abort_flag))) break;
      tc::fence_after_sync();
      const uint64_t ad = a0 + (uint64_t)(s * (kASlot >> 4));
      const uint32_t d = tmem + s * 2 * D;
      if (leader) {
#pragma unroll
        for (int ks = 0; ks < D / 16; ++ks) tc::mma_bf16(d, ad + (uint64_t)(ks * 256 >> 4), b0 + (uint64_t)(ks * 256 >> 4), idesc, ks > 0);
        if (KEY) {
#pragma unroll
          for (int ks = 0; ks < D / 16; ++ks)
            tc::mma_bf16(d + D, ad + (uint64_t)((TILE + ks * 256) >> 4), b1 + (uint64_t)(ks * 256 >> 4), idesc, ks > 0);
        }
        tc::mma_commit(bar.a_empty(s));
        tc::mma_commit(bar.d_full(s));
      }
      __syncwarp();
    }
    // a CTA that gave up does not leave under its own MMAs
    if (i > 0) tc::mbar_wait_bounded(bar.d_full((i - 1) & 1), ((i - 1) >> 1) & 1, 400000000ll);
  }
  return ok;
}

template <int D, int BITS, bool LIST>
__global__ void __launch_bounds__(kThreads, 1) expand_kv_kernel(const ExpandArgs a) {
  constexpr uint32_t MAT = D * D * 2;
  constexpr int NK = 1 << (2 * (BITS - 1)), NV = 1 << (2 * BITS);
  extern __shared__ __align__(1024) uint8_t smem[];
  __shared__ uint32_t lut[NV];
  __shared__ __align__(8) uint64_t bars[9];
  __shared__ uint32_t tmem_slot;
  __shared__ int s_abort, s_dead;
  __shared__ std::conditional_t<LIST, LiveMap, int> live;
  const int tid = threadIdx.x, warp = tid / 32;
  const bool key = (int)blockIdx.x < a.key_ctas;
  const int cta = key ? blockIdx.x : blockIdx.x - a.key_ctas, ctas = key ? a.key_ctas : gridDim.x - a.key_ctas;
  const ExpandBars bar{tc::smem_u32(&bars[0])};
  if (tid == 0) {
    for (int i = 0; i < 9; ++i) tc::mbar_init(bar.base + 8 * i, i < 2 ? kDecodeWarps : i == 6 || i == 7 ? kStoreWarps : 1);
    tc::fence_mbar_init();
    tc::fence_async_smem();
  }
  if (warp == kMmaWarp) tc::tmem_alloc(tc::smem_u32(&tmem_slot), 4 * D);
  if constexpr (LIST) {
    if (tid < kLiveWords) live.words[tid] = live.all[tid] = 0;
    __syncthreads();
  }
  grid_dependency_wait();
  if (tid == 0) {
    s_dead = *reinterpret_cast<volatile unsigned long long*>(&g_expand_faults) != 0ull ? 1 : 0;  // an earlier launch gave up
    s_abort = 0;
    const uint32_t bytes = (key ? 2 : 1) * MAT;
    tc::mbar_arrive_expect_tx(bar.constants(), bytes);
    tc::bulk_load(tc::smem_u32(smem), key ? a.w_key : a.w_val, bytes, bar.constants());
  }
  for (int e = tid; e < (key ? NK : NV); e += kThreads) lut[e] = a.luts[(key ? 0 : NK) + e];
  if constexpr (LIST) list_tiles(a, cta, ctas, live);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  // The attention kernel may start: what it reads before it waits for this one (the queries) was there before this line.  It
  // takes all tensor memory of its SM at once and keeps it until it ends, so the barrier between the allocation above and this
  // line has to stay: a CTA of this kernel that found none left would wait for a kernel that waits for it.
  grid_launch_dependents();
  const uint32_t tmem = tmem_slot;
  bool ok = true;
  if (!s_dead) {
    OwnTiles<LIST> own{cta, ctas, a.pairs * a.T, nullptr};
    if constexpr (LIST) own.list = live.tile;
    if (key) ok = expand_tiles<D, BITS, true>(a, smem, lut, bar, tmem, &s_abort, own);
    else ok = expand_tiles<D, BITS, false>(a, smem, lut, bar, tmem, &s_abort, own);
  }
  if (warp == kMmaWarp) tc::mbar_wait_bounded(bar.constants(), 0, 400000000ll);  // (landed long ago but for a CTA that gave up)
  if (!ok && atomicExch(&s_abort, 2) != 2) {  // one fault per CTA
    atomicAdd(&g_expand_faults, 1ull);
    notify_host_of_fault(g_fault_mailbox_expand);
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == kMmaWarp) tc::tmem_dealloc(tmem, 4 * D);
}

template <int D, int BITS, bool LIST>
int launch(ExpandArgs a, cudaStream_t stream) {
  constexpr size_t smem = (size_t)2 * D * D * 2 + (size_t)2 * 2 * 128 * D * 2;
  auto kern = expand_kv_kernel<D, BITS, LIST>;
  TQ_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const int64_t tiles = (int64_t)a.pairs * a.T;
  // A CTA per tile where that many fit the chip; otherwise three fifths of the CTAs take the keys, which cost twice the
  // MMAs and half as much again of everything else.
  const int sms = sm_count();
  int grid;
  if (2 * tiles <= sms) {
    grid = (int)(2 * tiles);
    a.key_ctas = (int)tiles;
  } else {
    grid = sms;
    a.key_ctas = sms * 3 / 5;
  }
  TQ_CUDA_OK(launch_dependent(kern, dim3((unsigned)grid), dim3(kThreads), smem, stream, a));
  return TQ_OK;
}

// Tiles that a mask hides from every query are left out where a KV head has 16 tiles and more, expanding all of them takes 10 us
// (300 tiles at head_dim 128), and the map of them is drawn in a few rounds of loads: about 2 us, most of it the latency of the
// first.  Us with all tiles expanded and so, 32 / 8 heads of 128 (nothing hidden / half of the prefix / all but a window of 64): 300
// tokens behind 2700, 2 sequences, 78 and 81 / 60 and 60 / 37 and 31; 256 behind 7936, 4 sequences, 212 and 218 / 152 and 129 / 93
// and 37; 64 behind 29936 124 and 128 / 109 and 85 / 89 and 36; 164 behind 582, 3 sequences, 144 tiles, 35 and 37 / 33 and 33 / 27
// and 27; 12 behind 15, 25 sequences, 12 / 12 heads, a tile each, 39 and 43 under any.  Listing them under a CTA's first tile took 3
// to 7 us longer.  The summary of more queries takes longer to look through than its tiles are worth beside the attention over them.
bool lists_tiles(ExpandArgs& a, int d) {
  if (a.mb.words == nullptr) return false;
  const int64_t tiles = (int64_t)a.pairs * a.T, sms = sm_count();
  const int64_t nb = a.mb.batch ? (a.pair0 + a.pairs - 1) / a.Hkv - a.pair0 / a.Hkv + 1 : 1;
  a.parts = (int)std::max<int64_t>(1, std::min<int64_t>(a.mb.NG, kListMapThreads / (nb * a.T)));
  return a.T >= 16 && tiles * d >= 300 * 128 && tiles <= kOwnTiles * (sms - sms * 3 / 5) && nb * ((a.T + 31) / 32) <= kLiveWords &&
         nb * a.mb.NG * ((int64_t)a.T + a.mb.NC) <= kSummaryReads;
}
template <int D>
int launch_bits(ExpandArgs a, int bits, cudaStream_t stream) {
  if (lists_tiles(a, D)) return bits == 2 ? launch<D, 2, true>(a, stream) : bits == 3 ? launch<D, 3, true>(a, stream) : launch<D, 4, true>(a, stream);
  return bits == 2 ? launch<D, 2, false>(a, stream) : bits == 3 ? launch<D, 3, false>(a, stream) : launch<D, 4, false>(a, stream);
}

}  // namespace

int expand_kv(const ExpandArgs& a, int d, int bits, cudaStream_t stream) {
  return d == 128 ? launch_bits<128>(a, bits, stream) : launch_bits<64>(a, bits, stream);
}

}  // namespace tq
