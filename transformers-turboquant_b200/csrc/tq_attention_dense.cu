// Flash attention over expanded keys and values (tq_expand.cu) on tcgen05.
//
// The rows of a KV head's query group are one list, row r = position r / G of query head r % G: a tile is 128 rows of it,
// whatever G and Sq are, so that few positions of several heads fill a tile and the heads of a group share every key tile.
// A CTA has two tiles, 256 rows, whose softmax warps take turns with the tensor pipe: while one tile's scores are turned into
// probabilities, the pipe works for the other one.
//
// Roles (12 warps): warps 0-3 and 4-7 softmax of the first and the second tile, one thread per row (no exchange between
// threads: a row's 128 scores are one thread's); one thread of warp 8 copies tiles of K' and V' (contiguous bulk copies, a
// ring of five slots); warps 9 and 10 issue the MMAs of either tile.
// Tensor memory: per tile 128 score columns, of which the first 64 are then the packed probabilities, and D output columns.
// Shared memory: two query tiles and the ring, 5 x 32 + 2 x 32 KB at head_dim 128.
//
// Queries are read once, scaled row by row by a power of two (undone in the exponent's factor) and rounded to fp16: exact for
// bf16 and fp16 inputs within 2^28 of the row's largest.
//
// MMAs of one thread run in issue order: S of key tile j + 1 of a tile is issued behind P V' of key tile j, which frees its
// columns, and its completion says that O is at rest -- the rescaling of O, rare, needs no wait of its own.
//
// Bound: at head_dim 128 the pipe needs 1024 cycles per tile and key tile and the 16384 exponentials another 1024 of the
// special-function units; scores -> probabilities -> P V' and the next scores is a chain of about 3000 cycles, in which the
// two tiles overlap.
#include <math.h>

#include <algorithm>

#include "tq_common.cuh"
#include "tq_dense.cuh"
#include "tq_rows.cuh"
#include "tq_simt.cuh"
#include "tq_tcgen05.cuh"

namespace tq {

__device__ unsigned long long g_dense_faults = 0ull;
// this device's slot of the host-visible status page (NULL until the first call on the device installs it)
__device__ unsigned long long* g_fault_mailbox_dense = nullptr;
int set_fault_mailbox_dense(unsigned long long* slot) {
  TQ_CUDA_OK(cudaMemcpyToSymbol(g_fault_mailbox_dense, &slot, sizeof(slot)));
  return TQ_OK;
}
int read_dense_faults(unsigned long long* out) {
  TQ_CUDA_OK(cudaMemcpyFromSymbol(out, g_dense_faults, sizeof(*out)));
  return TQ_OK;
}

namespace {

constexpr int kBM = 128, kBN = 128;   // query rows of a tile, keys of a tile
constexpr int kRows = 2 * kBM;        // rows of a CTA
constexpr int kSlots = 5;             // ring of K' and V' tiles
constexpr int kThreads = 384;
constexpr int kLoadWarp = 8, kMmaWarp = 9;
constexpr int kMapWords = kMapTiles / 32;  // masks of more keys are read without skipping
constexpr int kBars = 2 * kSlots + 21;

struct DenseArgs {
  const void* q;
  int q_dtype;
  int64_t qs_b, qs_h, qs_s;
  const uint8_t* kv;  // expanded tiles of this launch's pairs
  int T, rows;        // key tiles; rows G * Sq of a pair
  FastDiv G, Hkv;     // query heads per KV head; KV heads
  int64_t pair0;
  int blocks, pairs;  // blocks of a pair's rows, pairs of this launch
  int nsplit;
  FastDiv per_group, last_group, div_group, div_split;  // CTAs of a group; pairs of the last and of a group; nsplit
  float* part_o;   // [pairs][blocks][2][nsplit][128][D], unnormalised
  float* part_ml;  // ... [2]: running maximum (log2 units), row sum
};

template <int D>
struct DenseSmem {
  static constexpr uint32_t kTile = kBN * D * 2;
  static constexpr uint32_t kSbo = D / 8 * 128;
  static constexpr uint32_t kQOff = 0, kRing = 2 * kTile, kTotal = kRing + kSlots * kTile;
  static constexpr uint32_t kColO = 2 * kBN, kCols = 512;  // S[2] from column 0, O[2]
};

template <int D, bool MASK, bool SPLIT>
__global__ void __launch_bounds__(kThreads, 1) attention_dense_kernel(const AttnArgs a, const DenseArgs x) {
  using L = DenseSmem<D>;
  constexpr float kLog2e = 1.4426950408889634f;
  extern __shared__ __align__(1024) uint8_t smem[];
  __shared__ __align__(8) uint64_t bars[kBars];
  __shared__ uint32_t tmem_slot;
  __shared__ int s_abort, s_dead;
  // bit t: key tile t is computed at all / has hidden keys / has additive values that are neither 0 nor minus infinity
  __shared__ uint32_t map_live[MASK ? kMapWords : 1], map_hidden[MASK ? kMapWords : 1], map_other[MASK ? kMapWords : 1];
  volatile int* abort_flag = &s_abort;
  const int tid = threadIdx.x, lane = tid % 32;
  const int warp = __shfl_sync(0xffffffffu, tid / 32, 0);  // (uniform for the compiler too)
  const uint32_t bar0 = tc::smem_u32(&bars[0]);
  auto full = [&](int i) { return bar0 + 8u * i; };
  auto empty = [&](int i) { return bar0 + 8u * (kSlots + i); };
  auto s_full = [&](int w) { return bar0 + 8u * (2 * kSlots + w); };
  auto p_full = [&](int w) { return bar0 + 8u * (2 * kSlots + 2 + w); };
  auto q_full = [&](int w) { return bar0 + 8u * (2 * kSlots + 4 + w); };
  auto o_done = [&](int w) { return bar0 + 8u * (2 * kSlots + 6 + w); };
  const uint32_t drained = bar0 + 8u * (2 * kSlots + 8);
  auto p_half = [&](int w) { return bar0 + 8u * (2 * kSlots + 9 + w); };
  auto turn = [&](int w) { return bar0 + 8u * (2 * kSlots + 11 + w); };
  auto e_done = [&](int i) { return bar0 + 8u * (2 * kSlots + 13 + i); };  // exponentials of softmax warp i

  // ---- which rows and which keys ----
  // CTAs in the order of their index: groups of pairs, in a group the heaviest (latest) blocks of all its pairs first
  int lp, block, split = 0;  // pair of this launch, block of its rows, share of the keys
  {
    uint32_t at = blockIdx.x;
    if (SPLIT) {
      const uint32_t q = x.div_split.div(at);
      split = (int)(at - q * x.div_split.d);
      at = q;
    }
    const uint32_t group = x.per_group.div(at), first = group * x.div_group.d;
    at -= group * x.per_group.d;
    const bool whole = (int)(first + x.div_group.d) <= x.pairs;
    const uint32_t rank = whole ? x.div_group.div(at) : x.last_group.div(at);  // from the last block
    lp = (int)(first + at - rank * (whole ? x.div_group.d : x.last_group.d));
    block = x.blocks - 1 - (int)rank;
  }
  const uint32_t pair = (uint32_t)(x.pair0 + lp), b32 = x.Hkv.div(pair);
  const int64_t b = b32, kvh = pair - b32 * x.Hkv.d;
  const int row0 = block * kRows;
  const int shift = (int)(a.Sk - a.Sq);
  int nt0, nt1;  // key tiles in the range of either tile's last row
  {
    auto end = [&](int first) {
      if (first >= x.rows) return 0;
      int k = (int)a.Sk;
      if (a.causal) k = min(k, (int)x.G.div(min(first + kBM, x.rows) - 1) + shift + 1);
      return (k + kBN - 1) / kBN;
    };
    nt0 = end(row0);
    nt1 = end(row0 + kBM);
  }
  const int nt = max(nt0, nt1);

  if (warp == kMmaWarp) {
    for (int i = lane; i < kBars; i += 32) {
      const int r = i - 2 * kSlots;
      // p_full, q_full, p_half: the tile's softmax warps; empty, drained: both MMA warps
      tc::mbar_init(bar0 + 8u * i, (r >= 2 && r < 6) || r == 9 || r == 10 ? 4 : r == 8 || (r < 0 && i >= kSlots) ? 2 : 1);
    }
    tc::fence_mbar_init();
    tc::fence_async_smem();
  }
  if (warp == kLoadWarp) {
    tc::tmem_alloc(tc::smem_u32(&tmem_slot), L::kCols);
    if (lane == 0) {
      s_abort = 0;
      s_dead = *reinterpret_cast<volatile unsigned long long*>(&g_dense_faults) != 0ull ? 1 : 0;  // an earlier launch gave up
    }
  }

  const int w = warp / 4, r = tid % kBM, row = row0 + w * kBM + r;  // (softmax warps: a row per thread)
  const int pos = (int)x.G.div(row), head = (int)kvh * (int)x.G.d + row - pos * (int)x.G.d;
  const bool live_row = warp < 8 && row < x.rows;
  // ---- queries: a warp loads its 32 rows, eight rows by 64 bytes at a time (a thread per row: 12700 cycles until all were
  // there); 16-bit ones are on their way during the set-up ----
  const int64_t q_off = b * x.qs_b + head * x.qs_h + pos * x.qs_s;
  constexpr int QC = D / 32;  // 16-byte chunks a thread has of a row
  uint4 qv[4][QC];
  if (warp < 8 && x.q_dtype != TQ_F32) {
#pragma unroll
    for (int g = 0; g < 4; ++g) {
      const int64_t off = __shfl_sync(0xffffffffu, q_off, g * 8 + lane % 8);
      const uint4* src = reinterpret_cast<const uint4*>(static_cast<const uint16_t*>(x.q) + off) + lane / 8;
      const bool live = row - lane + g * 8 + lane % 8 < x.rows;
#pragma unroll
      for (int c = 0; c < QC; ++c) qv[g][c] = live ? src[4 * c] : make_uint4(0u, 0u, 0u, 0u);
    }
  }

  grid_dependency_wait();  // the expanded tiles (and a mask's summary)
  // Maps of the masked key tiles (32 at a time per warp).  Rows without a visible key average all keys of their causal
  // range: a CTA that has one computes every tile.
  const bool mapped = MASK && a.mb.words != nullptr && nt <= 32 * kMapWords;
  if (mapped && warp < 8) {
    const int p0 = (int)x.G.div(row0), p1 = (int)x.G.div(min(row0 + kRows, x.rows) - 1);
    const int g0 = p0 / 16, ng = p1 / 16 - g0 + 1;
    const int64_t gb = (a.mb.batch ? b * a.mb.NG : 0) + g0;
    bool blind = false;
    for (int g = lane; g < ng; g += 32) {
      uint32_t seen = 0;
      for (int c = 0; c < a.mb.NC; ++c) seen |= a.mb.rows[(gb + g) * a.mb.NC + c];
      const int n = min(16, (int)a.Sq - 16 * (g0 + g));
      blind = blind || (~seen & ((1u << n) - 1u)) != 0u;
    }
    blind = __any_sync(0xffffffffu, blind);
    for (int i = warp; i * 32 < nt; i += 8) {
      const int t = i * 32 + lane;
      uint32_t cls = 0;
      if (t < nt) {
        for (int g = 0; g < ng; ++g) cls |= a.mb.tiles[(gb + g) * a.mb.T + t];
        if (blind) cls |= 1u;
      }
      const uint32_t live = __ballot_sync(0xffffffffu, (cls & 1u) != 0u);
      const uint32_t hidden = __ballot_sync(0xffffffffu, (cls & 2u) != 0u);
      const uint32_t other = __ballot_sync(0xffffffffu, (cls & 4u) != 0u);
      if (lane == 0) {
        map_live[i] = live;
        map_hidden[i] = hidden;
        map_other[i] = other;
      }
    }
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();

  // tiles [lo, lo + n) of the live ones, of which the first n0 and n1 are computed for either query tile
  auto live_below = [&](int t) {
    if (!mapped) return t;
    int n = 0;
    for (int i = 0; i * 32 < t; ++i) n += __popc(map_live[i] & (t - i * 32 >= 32 ? 0xffffffffu : (1u << (t - i * 32)) - 1u));
    return n;
  };
  int n = s_dead ? 0 : live_below(nt), lo = 0;
  if (SPLIT) {
    lo = (int)((int64_t)n * split / x.nsplit);
    n = (int)((int64_t)n * (split + 1) / x.nsplit) - lo;
  }
  const int n0 = min(n, max(0, live_below(nt0) - lo)), n1 = min(n, max(0, live_below(nt1) - lo));
  n = max(n0, n1);
  // the key tile computed after tile t (-1: the first one)
  auto next_tile = [&](int t) -> int {
    if (SPLIT && t < 0) {
      if (!mapped) return lo;
      int left = lo;
      for (int i = 0; i * 32 < nt; ++i) {
        uint32_t bits = map_live[i];
        const int c = __popc(bits);
        if (left >= c) { left -= c; continue; }
        for (; left > 0; --left) bits &= bits - 1u;
        return i * 32 + __ffs((int)bits) - 1;
      }
      return nt;
    }
    ++t;
    if (mapped) {
      for (; t < nt; t = (t | 31) + 1) {
        const uint32_t bits = map_live[t >> 5] >> (t & 31);
        if (bits != 0u) return t + __ffs((int)bits) - 1;
      }
    }
    return t;
  };
  const uint32_t tmem = tmem_slot;
  bool ok = true;

  if (warp < 8) {
    // =============================== softmax warps ===============================
    const int nw = w == 0 ? n0 : n1;
    const uint32_t lanes = (uint32_t)(warp % 4 * 32) << 16;
    const uint32_t tmem_s = tmem + w * kBN + lanes, tmem_o = tmem + L::kColO + w * D + lanes;
    float cexp = a.sm_scale * kLog2e;
    {
      // rows scaled by a power of two to fp16, into the operand tile
      // 2^(13 - exponent of m), 1 for a row of zeros or with an infinity; at most 2^64 cexp, so that 1 / cexp and with it the
      // hidden keys' floor and the mask's unit stay finite.  A smaller row has scores below 2^-64: fp16 may flush it.
      const uint32_t most = (__float_as_uint(cexp) >> 23) + 64u;
      auto scale_of = [&](float m) {
        const uint32_t e = __float_as_uint(m) >> 23;
        return __uint_as_float(min(e == 0u || e >= 255u ? 127u : 267u - max(e, 14u), most) << 23);
      };
      float scale = 1.f;
      uint8_t* q_rows = smem + L::kQOff + w * L::kTile + warp % 4 * 4 * L::kSbo;  // this warp's 32 rows
      if (x.q_dtype == TQ_F32) {
        const float4* p = reinterpret_cast<const float4*>(static_cast<const float*>(x.q) + q_off);
        const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
        float top = 0.f;
#pragma unroll 4
        for (int i = 0; i < D / 4; ++i) {
          const float4 u = live_row ? p[i] : zero;
          top = fmaxf(top, fmaxf(fmaxf(fabsf(u.x), fabsf(u.y)), fmaxf(fabsf(u.z), fabsf(u.w))));
        }
        scale = scale_of(top);
#pragma unroll 2
        for (int i = 0; i < D / 8; ++i) {
          const float4 u = live_row ? p[2 * i] : zero, v = live_row ? p[2 * i + 1] : zero;
          *reinterpret_cast<uint4*>(q_rows + lane / 8 * L::kSbo + lane % 8 * 16 + i * 128) =
              make_uint4(tc::pack_f16x2(u.x * scale, u.y * scale), tc::pack_f16x2(u.z * scale, u.w * scale),
                         tc::pack_f16x2(v.x * scale, v.y * scale), tc::pack_f16x2(v.z * scale, v.w * scale));
        }
      } else {
        const bool bf16 = x.q_dtype == TQ_BF16;
        auto halves = [&](uint32_t u) {
          return bf16 ? make_float2(__uint_as_float(u << 16), __uint_as_float(u & 0xffff0000u))
                      : __half22float2(*reinterpret_cast<const __half2*>(&u));
        };
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          uint32_t top = 0u;  // of the magnitudes' bit patterns, two at a time
#pragma unroll
          for (int c = 0; c < QC; ++c) {
            const uint4 u = qv[g][c];
            top = __vmaxu2(__vmaxu2(top, u.x & 0x7fff7fffu), __vmaxu2(u.y & 0x7fff7fffu, __vmaxu2(u.z & 0x7fff7fffu, u.w & 0x7fff7fffu)));
          }
          top = __vmaxu2(top, __shfl_xor_sync(0xffffffffu, top, 8));
          top = __vmaxu2(top, __shfl_xor_sync(0xffffffffu, top, 16));
          const float f = scale_of(halves(max(top & 0xffffu, top >> 16)).x);  // of row g * 8 + lane % 8
          if (lane / 8 == g) scale = f;
          auto scaled = [&](uint32_t v) {
            const float2 h = halves(v);
            return tc::pack_f16x2(h.x * f, h.y * f);
          };
#pragma unroll
          for (int c = 0; c < QC; ++c) {
            const uint4 u = qv[g][c];
            *reinterpret_cast<uint4*>(q_rows + g * L::kSbo + (lane / 8 + 4 * c) * 128 + lane % 8 * 16) =
                make_uint4(scaled(u.x), scaled(u.y), scaled(u.z), scaled(u.w));
          }
        }
      }
      cexp *= 1.f / scale;  // a power of two
      tc::fence_async_smem();
    }
    __syncwarp();
    if (lane == 0) tc::mbar_arrive(q_full(w));
    const int pos0 = (int)x.G.div(row0 + w * kBM);  // the tile's first position
    const float rcexp = 1.f / cexp;
    float m_run = -INFINITY, l_run = 0.f;
    const bool mask_by_4 = MASK && ((reinterpret_cast<uintptr_t>(a.mask) | (uintptr_t)(4 * a.mask_stride_b) | (uintptr_t)(4 * a.mask_stride_q)) & 15u) == 0;
    int kt = next_tile(-1);
    for (int j = 0; j < nw && ok; ++j, kt = next_tile(kt)) {
      const int k0 = kt * kBN;
      bool hidden = false, other = MASK && a.mask != nullptr;
      uint4 seen = make_uint4(0u, 0u, 0u, 0u);  // visibility bits of the row's 128 columns
      if (MASK && a.mb.words != nullptr) {
        hidden = !mapped || ((map_hidden[kt >> 5] >> (kt & 31)) & 1u) != 0u;
        other = other && (!mapped || ((map_other[kt >> 5] >> (kt & 31)) & 1u) != 0u);
        if (hidden && !other && live_row)
          seen = *reinterpret_cast<const uint4*>(a.mb.words + ((a.mb.batch ? b * a.Sq : 0) + pos) * (4 * (int64_t)a.mb.T) + 4 * kt);
      }
      if (!(ok = tc::mbar_spin_or_abort(s_full(w), j & 1, abort_flag))) break;
      tc::fence_after_sync();
      float t[kBN];
      {
        uint32_t raw[kBN / 32][32];
#pragma unroll
        for (int c = 0; c < kBN / 32; ++c) tc::tmem_ld32(tmem_s + 32 * c, raw[c]);
        tc::wait_ld();
#pragma unroll
        for (int c = 0; c < kBN; ++c) t[c] = __uint_as_float(raw[c / 32][c % 32]);
      }
      const bool edge = k0 + kBN > a.Sk || (a.causal && k0 + kBN - 1 > pos0 + shift) || hidden || other;
      if (edge) {
        // Tiles that cross the end of the keys or the causal diagonal, and masked ones.  `vis`: the last column this row may
        // see.  A hidden key's score is the floor (-60000 in log2 units: its probability is exactly 0 beside any real score),
        // which stays finite, so that a row of hidden keys averages them as a softmax of equal scores does.
        const int vsk = (int)a.Sk - 1 - k0;
        const int vis = a.causal ? min(vsk, pos + shift - k0) : vsk;
        const float floor_raw = -60000.f * rcexp;
        if (MASK && other && live_row) {
          const float* mrow = a.mask + b * a.mask_stride_b + (int64_t)pos * a.mask_stride_q + k0;
          const float m_unit = kLog2e * rcexp;
#pragma unroll
          for (int c0 = 0; c0 < kBN; c0 += 16) {
            float mv[16];
            if (mask_by_4 && c0 + 15 <= vsk) {
#pragma unroll
              for (int i = 0; i < 16; i += 4) {
                const float4 m4 = __ldg(reinterpret_cast<const float4*>(mrow + c0 + i));
                mv[i] = m4.x; mv[i + 1] = m4.y; mv[i + 2] = m4.z; mv[i + 3] = m4.w;
              }
            } else {
#pragma unroll
              for (int i = 0; i < 16; ++i) mv[i] = c0 + i <= vsk ? __ldg(mrow + c0 + i) : 0.f;
            }
#pragma unroll
            for (int i = 0; i < 16; ++i) t[c0 + i] = fmaxf(fmaf(mv[i], m_unit, t[c0 + i]), floor_raw);
          }
        } else if (MASK && hidden) {
          const uint32_t sw[4] = {seen.x, seen.y, seen.z, seen.w};
#pragma unroll
          for (int c = 0; c < kBN; ++c) t[c] = ((sw[c / 32] >> (c & 31)) & 1u) != 0u ? fmaxf(t[c], floor_raw) : floor_raw;
        }
#pragma unroll
        for (int c = 0; c < kBN; ++c) t[c] = c <= vis ? t[c] : -INFINITY;
      }
      float mx;
      {
        float m0 = -INFINITY, m1 = -INFINITY, m2 = -INFINITY, m3 = -INFINITY;
#pragma unroll
        for (int c = 0; c < kBN; c += 8) {
          m0 = tc::fmax3(m0, t[c], t[c + 1]);
          m1 = tc::fmax3(m1, t[c + 2], t[c + 3]);
          m2 = tc::fmax3(m2, t[c + 4], t[c + 5]);
          m3 = tc::fmax3(m3, t[c + 6], t[c + 7]);
        }
        mx = fmaxf(tc::fmax3(m0, m1, m2), m3) * cexp;
      }
      if (MASK && !edge && a.mb.words != nullptr && mx < -59000.f) {
        // scores as low as the hidden keys' floor: clamped there in every tile of a masked call
        const float floor_raw = -60000.f * rcexp;
#pragma unroll
        for (int c = 0; c < kBN; ++c) t[c] = fmaxf(t[c], floor_raw);
        mx = fmaxf(mx, -60000.f);
      }
      // The maximum in use trails the row's by at most 8: probabilities reach 2^8, and O is rescaled rarely.
      const float m_cand = fmaxf(m_run, mx);
      if (__any_sync(0xffffffffu, m_cand > m_run + 8.f)) {
        const float alpha = m_run == -INFINITY ? 0.f : tc::fast_exp2(m_run - m_cand);
        m_run = m_cand;
        l_run *= alpha;
        if (j > 0) {
#pragma unroll 1
          for (int c0 = 0; c0 < D; c0 += 16) {
            uint32_t o[16];
            tc::tmem_ld16(tmem_o + c0, o);
            tc::wait_ld();
#pragma unroll
            for (int c = 0; c < 16; ++c) o[c] = __float_as_uint(__uint_as_float(o[c]) * alpha);
            tc::tmem_st16(tmem_o + c0, o);
          }
        }
      }
      const float m_use = m_run == -INFINITY ? 0.f : m_run;
      // The two warps that share a scheduler and its special-function unit take turns.
      {
        const int k = w == 0 ? j - 1 : j;  // the other one's tile that comes first
        if (k >= 0 && k < (w == 0 ? n1 : n0) && !(ok = tc::mbar_spin_or_abort(e_done((warp + 4) % 8), k & 1, abort_flag))) break;
      }
      float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
#pragma unroll
      for (int c0 = 0; c0 < kBN; c0 += 32) {
        uint32_t pw[16];
#pragma unroll
        for (int c = 0; c < 16; c += 2) {
          const float p0 = tc::fast_exp2(fmaf(t[c0 + 2 * c], cexp, -m_use)), p1 = tc::fast_exp2(fmaf(t[c0 + 2 * c + 1], cexp, -m_use));
          const float p2 = tc::fast_exp2(fmaf(t[c0 + 2 * c + 2], cexp, -m_use)), p3 = tc::fast_exp2(fmaf(t[c0 + 2 * c + 3], cexp, -m_use));
          s0 += p0; s1 += p1; s2 += p2; s3 += p3;
          pw[c] = tc::pack_f16x2(p0, p1);
          pw[c + 1] = tc::pack_f16x2(p2, p3);
        }
        tc::tmem_st16(tmem_s + c0 / 2, pw);
        if (c0 == kBN - 32 && lane == 0) tc::mbar_arrive(e_done(warp));
        if (c0 == kBN / 2 - 32) {  // the first half of P V' starts under the second half's exponentials
          tc::wait_st();
          tc::fence_before_sync();
          __syncwarp();
          if (lane == 0) tc::mbar_arrive(p_half(w));
        }
      }
      l_run += (s0 + s1) + (s2 + s3);
      tc::wait_st();
      tc::fence_before_sync();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(p_full(w));
    }
    if (ok && nw > 0) {
      ok = tc::mbar_wait_or_abort(o_done(w), 0, abort_flag);
      tc::fence_after_sync();
    }
    if (SPLIT && ok) {
      const int64_t prow = ((((int64_t)lp * x.blocks + block) * 2 + w) * x.nsplit + split) * kBM + r;
      if (live_row) *reinterpret_cast<float2*>(x.part_ml + prow * 2) = make_float2(m_run, l_run);
      if (nw > 0) {
#pragma unroll 1
        for (int c0 = 0; c0 < D; c0 += 32) {
          uint32_t o[32];
          tc::tmem_ld32(tmem_o + c0, o);
          tc::wait_ld();
          if (live_row) {
            uint4* dst = reinterpret_cast<uint4*>(x.part_o + prow * D + c0);
#pragma unroll
            for (int i = 0; i < 8; ++i) dst[i] = make_uint4(o[4 * i], o[4 * i + 1], o[4 * i + 2], o[4 * i + 3]);
          }
        }
      }
    } else if (!SPLIT && ok && nw > 0) {
      const float inv = l_run > 0.f ? 1.f / l_run : 0.f;
      const bool wide = a.out_dtype == TQ_F32;
      const int64_t ooff = b * a.o_stride_b + head * a.o_stride_h + pos * a.o_stride_s;
      // 16-bit rows go through the query tile's shared memory (its MMAs are done), a warp's 32 rows at a time, chunks
      // rotated by the row so that neither side meets in a bank
      constexpr int CH = D / 8;  // 16-byte chunks of a row
      uint8_t* stage = smem + L::kQOff + w * L::kTile + warp % 4 * 32 * D * 2;
#pragma unroll 1
      for (int c0 = 0; c0 < D; c0 += 32) {
        uint32_t o[32];
        tc::tmem_ld32(tmem_o + c0, o);
        tc::wait_ld();
#pragma unroll
        for (int c = 0; c < 32; ++c) o[c] = __float_as_uint(__uint_as_float(o[c]) * inv);
        if (wide) {
          if (live_row) store_row_chunk(a.out, TQ_F32, ooff + c0, o);
        } else {
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            uint32_t v[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const float lo_ = __uint_as_float(o[8 * i + 2 * e]), hi_ = __uint_as_float(o[8 * i + 2 * e + 1]);
              v[e] = a.out_dtype == TQ_BF16 ? tc::pack_bf16x2(lo_, hi_) : tc::pack_f16x2(lo_, hi_);
            }
            *reinterpret_cast<uint4*>(stage + lane * (D * 2) + ((c0 / 8 + i + lane) % CH) * 16) = make_uint4(v[0], v[1], v[2], v[3]);
          }
        }
      }
      if (!wide) {
        __syncwarp();
        constexpr int RPI = 32 / CH;  // rows stored per instruction
#pragma unroll 4
        for (int i = 0; i < 32; i += RPI) {
          const int rr = i + lane / CH, c = lane % CH, grow = row - lane + rr;
          const uint4 v = *reinterpret_cast<const uint4*>(stage + rr * (D * 2) + (c + rr) % CH * 16);
          const int64_t off = __shfl_sync(0xffffffffu, ooff, rr);
          if (grow < x.rows) *reinterpret_cast<uint4*>(static_cast<uint16_t*>(a.out) + off + c * 8) = v;
        }
      }
    }
  } else if (warp == kLoadWarp && lane == 0) {
    // =============================== tile copies ===============================
    const uint8_t* src = x.kv + (int64_t)lp * x.T * 2 * L::kTile;
    int kt = next_tile(-1), i = 0;
    for (int j = 0; j < n && ok; ++j, kt = next_tile(kt)) {
#pragma unroll 1
      for (int v = 0; v < 2; ++v, ++i) {
        const int s = i % kSlots, u = i / kSlots;
        if (u >= 1 && !(ok = tc::mbar_wait_or_abort(empty(s), (u - 1) & 1, abort_flag))) break;
        tc::mbar_arrive_expect_tx(full(s), L::kTile);
        tc::bulk_load(tc::smem_u32(smem + L::kRing + s * L::kTile), src + ((int64_t)kt * 2 + v) * L::kTile, L::kTile, full(s));
      }
    }
    // a CTA that gave up does not leave before its copies have landed
    for (int k = max(0, i - kSlots); k < i; ++k) tc::mbar_wait_bounded(full(k % kSlots), (k / kSlots) & 1, 400000000ll);
  } else if (warp == kMmaWarp || warp == kMmaWarp + 1) {
    // =============================== MMAs of either tile ===============================
    // The whole warp runs this loop and one elected lane issues: operands stay in uniform registers (4100 cycles per key tile
    // of both with a branch to one thread, 3310 so).
    constexpr uint32_t idesc_s = tc::idesc_f16(kBM, kBN, false, false), idesc_o = tc::idesc_f16(kBM, D, false, true);
    const int v = warp - kMmaWarp, nv = v == 0 ? n0 : n1;
    const uint64_t qdesc = tc::smem_desc(tc::smem_u32(smem + L::kQOff + v * L::kTile), 128, L::kSbo);
    const uint64_t kdesc = tc::smem_desc(tc::smem_u32(smem + L::kRing), 128, L::kSbo);
    const uint64_t vdesc = tc::smem_desc(tc::smem_u32(smem + L::kRing), L::kSbo, 128);
    const uint32_t tmem_s = tmem + v * kBN, tmem_o = tmem + L::kColO + v * D;
    const bool leader = tc::elect_one();
    if (nv > 0) ok = tc::mbar_wait_or_abort(q_full(v), 0, abort_flag);
    // K' of tile j is item 2 j of the ring, V' item 2 j + 1; a slot is free when both warps' MMAs have read it.  The warps
    // take turns: P V' of one key tile and S of the next are issued as one batch.  (Interleaved batches of both tiles end
    // together, and the softmax warps of both then work at the same time, with the pipe idle: 4400 cycles.)
    for (int j = 0; j <= n && ok; ++j) {
      const int iv = 2 * j - 1, sv = iv % kSlots, ik = 2 * j, sk = ik % kSlots;
      const bool pv = j > 0 && j <= nv, qk = j < nv;
      if (j > 0 && !(ok = tc::mbar_wait_or_abort(full(sv), (iv / kSlots) & 1, abort_flag))) break;
      if (pv && !(ok = tc::mbar_spin_or_abort(p_half(v), (j - 1) & 1, abort_flag))) break;
      if ((v == 1 || j > 0) && !(ok = tc::mbar_spin_or_abort(turn(v), (v == 0 ? j - 1 : j) & 1, abort_flag))) break;
      tc::fence_after_sync();
      if (pv) {  // O += P V' of tile j - 1
        const uint64_t vd = vdesc + (uint64_t)(sv * (L::kTile >> 4));
        if (leader) {
#pragma unroll
          for (int ks = 0; ks < kBN / 32; ++ks)
            tc::mma_bf16_ts(tmem_o, tmem_s + ks * 8, vd + (uint64_t)(ks * 2 * (L::kSbo >> 4)), idesc_o, (j > 1 || ks > 0) ? 1u : 0u);
        }
        __syncwarp();
        if (!(ok = tc::mbar_spin_or_abort(p_full(v), (j - 1) & 1, abort_flag))) break;
        tc::fence_after_sync();
        if (leader) {
#pragma unroll
          for (int ks = kBN / 32; ks < kBN / 16; ++ks)
            tc::mma_bf16_ts(tmem_o, tmem_s + ks * 8, vd + (uint64_t)(ks * 2 * (L::kSbo >> 4)), idesc_o, 1u);
          if (j == nv) tc::mma_commit(o_done(v));
        }
        __syncwarp();
      }
      if (leader && j > 0) tc::mma_commit(empty(sv));
      if (j < n) {  // S = Q K'^T of tile j
        if (!(ok = tc::mbar_wait_or_abort(full(sk), (ik / kSlots) & 1, abort_flag))) break;
        const uint64_t kd = kdesc + (uint64_t)(sk * (L::kTile >> 4));
        if (leader) {
          if (qk) {
#pragma unroll
            for (int ks = 0; ks < D / 16; ++ks)
              tc::mma_bf16(tmem_s, qdesc + (uint64_t)(ks * 256 >> 4), kd + (uint64_t)(ks * 256 >> 4), idesc_s, ks > 0);
            tc::mma_commit(s_full(v));
          }
          tc::mbar_arrive(turn(1 - v));
          tc::mma_commit(empty(sk));
        }
        __syncwarp();
      } else if (leader && v == 0) {
        tc::mbar_arrive(turn(1));
      }
    }
    // nothing of this CTA's is in flight when its tensor memory is given back
    if (leader) tc::mma_commit(drained);
    tc::mbar_wait_bounded(drained, 0, 400000000ll);
  }
  if (!ok && atomicExch(&s_abort, 2) != 2) {  // one fault per CTA
    atomicAdd(&g_dense_faults, 1ull);
    notify_host_of_fault(g_fault_mailbox_dense);
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == kLoadWarp) tc::tmem_dealloc(tmem, L::kCols);
}

// out = sum_s 2^(m_s - m) O_s / sum_s 2^(m_s - m) l_s; a warp per row.
template <int D>
__global__ void __launch_bounds__(256) merge_dense_kernel(const AttnArgs a, const DenseArgs x) {
  constexpr int E = D / 32;
  grid_dependency_wait();
  const int row = blockIdx.x * 8 + threadIdx.x / 32, lane = threadIdx.x % 32;
  if (row >= x.rows) return;
  const uint32_t pair = (uint32_t)x.pair0 + blockIdx.y, b32 = x.Hkv.div(pair), pos = x.G.div(row);
  const int64_t b = b32, kvh = pair - b32 * x.Hkv.d;
  const int64_t p0 = ((int64_t)blockIdx.y * x.blocks * 2 + row / kBM) * x.nsplit * kBM + row % kBM;
  float m = -INFINITY;
  for (int s = 0; s < x.nsplit; ++s) m = fmaxf(m, x.part_ml[(p0 + (int64_t)s * kBM) * 2]);
  const float m_use = m == -INFINITY ? 0.f : m;
  float l = 0.f, o[E] = {};
  for (int s = 0; s < x.nsplit; ++s) {
    const float2 ml = *reinterpret_cast<const float2*>(x.part_ml + (p0 + (int64_t)s * kBM) * 2);
    if (ml.y == 0.f) continue;  // no keys here (a sum of NaN has no maximum either, but goes on)
    const float f = ml.x == -INFINITY ? 1.f : tc::fast_exp2(ml.x - m_use);
    l = fmaf(f, ml.y, l);
    const float* src = x.part_o + (p0 + (int64_t)s * kBM) * D + lane * E;
    if constexpr (E == 4) {
      const float4 v = *reinterpret_cast<const float4*>(src);
      o[0] = fmaf(f, v.x, o[0]); o[1] = fmaf(f, v.y, o[1]); o[2] = fmaf(f, v.z, o[2]); o[3] = fmaf(f, v.w, o[3]);
    } else {
      const float2 v = *reinterpret_cast<const float2*>(src);
      o[0] = fmaf(f, v.x, o[0]); o[1] = fmaf(f, v.y, o[1]);
    }
  }
  const float inv = l > 0.f ? 1.f / l : (l == 0.f ? 0.f : l);
  const int64_t off = b * a.o_stride_b + (kvh * x.G.d + row - pos * x.G.d) * a.o_stride_h + pos * a.o_stride_s + lane * E;
#pragma unroll
  for (int e = 0; e < E; e += 2) {
    const float u = o[e] * inv, v = o[e + 1] * inv;
    if (a.out_dtype == TQ_F32) *reinterpret_cast<float2*>(static_cast<float*>(a.out) + off + e) = make_float2(u, v);
    else *reinterpret_cast<uint32_t*>(static_cast<uint16_t*>(a.out) + off + e) = a.out_dtype == TQ_BF16 ? tc::pack_bf16x2(u, v) : tc::pack_f16x2(u, v);
  }
}

template <int D, bool MASK, bool SPLIT>
int launch_dense(const AttnArgs& a, const DenseArgs& x, cudaStream_t stream) {
  using L = DenseSmem<D>;
  auto kern = attention_dense_kernel<D, MASK, SPLIT>;
  TQ_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)L::kTotal));
  TQ_CUDA_OK(launch_dependent(kern, dim3((unsigned)(x.pairs * x.blocks * x.nsplit)), dim3(kThreads), L::kTotal, stream, a, x));
  if (SPLIT)
    TQ_CUDA_OK(launch_dependent(merge_dense_kernel<D>, dim3((unsigned)((x.rows + 7) / 8), (unsigned)x.pairs), dim3(256), 0, stream, a, x));
  return TQ_OK;
}
template <int D>
int launch_kind(const AttnArgs& a, const DenseArgs& x, cudaStream_t stream) {
  const bool masked = a.mask != nullptr || a.mb.words != nullptr;
  if (x.nsplit > 1) return masked ? launch_dense<D, true, true>(a, x, stream) : launch_dense<D, false, true>(a, x, stream);
  return masked ? launch_dense<D, true, false>(a, x, stream) : launch_dense<D, false, false>(a, x, stream);
}

inline size_t round256(size_t v) { return (v + 255) & ~(size_t)255; }

// The plan of a call: pairs expanded at a time, splits of the keys, bytes of either.
struct DensePlan {
  int64_t T, rows, blocks, pairs;  // key tiles, rows of a pair and their blocks; pairs at a time
  int nsplit;
  size_t kv_bytes, part_bytes;
  double us;  // what the call is expected to take
};
// Expanded keys and values take 4 d bytes a token and KV head: 128 MiB at a time, about what the L2 holds.
constexpr size_t kExpandBytes = (size_t)128 << 20;
// Pairs whose blocks run side by side, heaviest first: their tiles are read by all of them and should stay in the L2 (4 x 8192
// tokens, 32 / 8 heads: 1960 us with 16 or 32 MB, 1988 with 64, 2039 with all 128).
constexpr int64_t kGroupBytes = (int64_t)32 << 20;

DensePlan dense_plan(int64_t B, int64_t Hq, int64_t Sq, int64_t Hkv, int64_t Sk, int d) {
  DensePlan p{};
  p.T = (Sk + kBN - 1) / kBN;
  p.rows = Hq / Hkv * Sq;
  p.blocks = (p.rows + kRows - 1) / kRows;
  const size_t pair_bytes = (size_t)p.T * 2 * kBN * d * 2;
  const int64_t all = B * Hkv, most = (int64_t)(kExpandBytes / pair_bytes);
  if (most < 1) return p;
  const int64_t groups = (all + most - 1) / most;
  p.pairs = (all + groups - 1) / groups;
  p.kv_bytes = round256((size_t)p.pairs * pair_bytes);
  // Few blocks of many key tiles are split over the keys: the number with the least (waves of CTAs) x (tiles + set-up) +
  // merge, in periods of a key tile of both query tiles.
  constexpr double kFixed = 4.0, kMerge = 4.0, kPeriodUs = 1.75, kExpandUs = 0.033 / 128, kLaunchUs = 8.0;
  const int64_t units = p.pairs * p.blocks, slots = sm_count();
  const int64_t free_tiles = (Sk > Sq ? Sk - Sq : 0) / kBN / 4;  // (in front of the first query: no split is empty)
  p.nsplit = 1;
  double cost = (double)((units + slots - 1) / slots) * ((double)p.T + kFixed);
  for (int64_t s = 2; s <= free_tiles && s <= 32 && units < slots; ++s) {
    const double c = (double)((units * s + slots - 1) / slots) * ((double)((p.T + s - 1) / s) + kFixed + 1.0) + kMerge;
    if (c < cost) {
      cost = c;
      p.nsplit = (int)s;
    }
  }
  // (causal prompts: the average block walks fewer tiles than the first ones)
  if (4 * Sq >= Sk && units > slots)
    cost = (double)p.T + kFixed + ((double)units / (double)slots - 1.0) * (attention_walked_keys(Sq, Sk) / kBN + kFixed);
  p.us = kLaunchUs + (double)groups * cost * kPeriodUs + (double)(all * p.T * d) * kExpandUs;
  if (p.nsplit > 1) p.part_bytes = round256((size_t)units * 2 * p.nsplit * kBM * (d + 2) * sizeof(float));
  return p;
}

}  // namespace

bool attention_dense_applies(int64_t B, int64_t Hq, int64_t Sq, int64_t Hkv, int64_t Sk, int d) {
  if (B <= 0 || Hkv <= 0 || Sk <= 0 || Sq <= 0 || Hq % Hkv != 0 || (d != 64 && d != 128)) return false;
  const DensePlan p = dense_plan(B, Hq, Sq, Hkv, Sk, d);
  // Expansion pays where a key is met by many tiles of queries.  Few queries behind a prefix, and calls of one or two key tiles,
  // are the SM-pair kernel's: either one's time is estimated (over 533 calls of 1 to 512 tokens behind 0 to 30000, 2 to 32 KV
  // heads and 1 to 16 sequences both estimates are right within 10 % (rms), no call goes to the slower kernel by more than 3 %
  // here, and what the rule leaves to the SM-pair kernel would gain 0.7 % in the mean).  SM-pair kernel and expansion: 64 tokens
  // behind 2000 (1 sequence, 32 / 8 heads) 37 and 38 us; 128 behind 8000 (4 sequences) 113 and 148; 512 behind 8000 (4 sequences,
  // 16 / 2 heads) 217 and 161; 16 x 64 tokens 41 and 24; 8192 over 512 keys (8 sequences, not causal) 1455 and 826.
  const int64_t most = (int64_t)1 << 31;
  return p.kv_bytes > 0 && p.us < 0.98 * attention_c2_us(B, Hq, Sq, Hkv, Sk, d) && B * Hkv < most && p.rows < most - kRows &&
         p.pairs * p.blocks * 32 < most && p.pairs <= 65535;
}
size_t attention_dense_bytes(int64_t B, int64_t Hq, int64_t Sq, int64_t Hkv, int64_t Sk, int d) {
  const DensePlan p = dense_plan(B, Hq, Sq, Hkv, Sk, d);
  return p.kv_bytes + p.part_bytes;
}

int attention_dense(const AttnArgs& a, int64_t B, int d, int bits, const void* q, int q_dtype, int64_t sb, int64_t sh, int64_t ss,
                    const uint8_t* constants, void* workspace, cudaStream_t stream) {
  const DensePlan p = dense_plan(B, a.Hq, a.Sq, a.Hkv, a.Sk, d);
  const ConstLayout L = const_layout(d);
  uint8_t* ws = static_cast<uint8_t*>(workspace);
  // Key tiles that a mask hides from every query are not expanded, where there are any to speak of and the expansion is: in front of
  // a chunk of few queries.  (Prompts have those of their padding, whose rows average all keys of their causal range.)
  const bool skip = a.mb.words != nullptr && p.T <= kMapTiles && a.Sk >= 6 * a.Sq;
  for (int64_t p0 = 0; p0 < B * a.Hkv; p0 += p.pairs) {
    const int pairs = (int)std::min<int64_t>(B * a.Hkv - p0, p.pairs);
    const ExpandArgs e{a.key_idx, a.key_sgn, a.key_vn, a.key_rn, a.val_idx, a.val_vn, a.kv_stride, a.Sk, constants + L.x_key,
                       constants + L.x_val, reinterpret_cast<const uint32_t*>(constants + L.luts),
                       reinterpret_cast<const float*>(constants + L.header) + kExpandScaleWord, p0, pairs, (int)p.T, 0,
                       skip ? a.mb : MaskBits{}, (int)a.Sq, 0, a.Hkv, ws};
    {
      ProfScope prof(kProfPrepareQueries, stream);
      if (int st = expand_kv(e, d, bits, stream)) return st;
    }
    const int group = (int)std::min<int64_t>(pairs, std::max<int64_t>(1, kGroupBytes / (p.T * 2 * kBN * d * 2)));
    DenseArgs x{q, q_dtype, sb, sh, ss, ws, (int)p.T, (int)p.rows, FastDiv((uint32_t)(a.Hq / a.Hkv)), FastDiv((uint32_t)a.Hkv), p0,
                (int)p.blocks, pairs, p.nsplit, FastDiv((uint32_t)(group * p.blocks)),
                FastDiv((uint32_t)(pairs % group ? pairs % group : group)), FastDiv((uint32_t)group), FastDiv((uint32_t)p.nsplit),
                nullptr, nullptr};
    if (p.nsplit > 1) {
      x.part_o = reinterpret_cast<float*>(ws + p.kv_bytes);
      x.part_ml = x.part_o + (size_t)p.pairs * p.blocks * 2 * p.nsplit * kBM * d;
    }
    ProfScope prof(kProfAttention, stream);
    if (int st = d == 128 ? launch_kind<128>(a, x, stream) : launch_kind<64>(a, x, stream)) return st;
  }
  return TQ_OK;
}

}  // namespace tq
