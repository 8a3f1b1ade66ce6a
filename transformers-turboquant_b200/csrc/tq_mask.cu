// Summary of an attention mask: one bit per (row, key) and one class per 16 rows x 128 keys.
//
// Every query head reads the same mask, and the attention kernels hold one query row per thread: reading the mask
// itself there is one 4-byte load per score, each lane of a warp in another row (32 sectors per load), repeated for
// every head.  This kernel reads the mask once -- boolean bytes as they are, or additive fp32 -- and leaves
//   * words: bit k of row s set where key k is visible (rows padded to whole 128-key tiles with zeros),
//   * tiles: per 16 rows and 128 keys, whether some key is visible, some hidden, some anything else (an additive
//     value that is neither 0 nor "minus infinity": those tiles still read the mask itself),
//   * rows:  which of the 16 rows have a visible key at all, the causal limit included.
// A thread of the attention kernels then loads 64 columns as one 8-byte word pair, tiles without hidden keys take the
// unmasked path, and tiles nobody can see are not computed: a hidden score weighs exactly 0 beside a visible one.
// (Rows with no visible key average all keys of their causal range, so nothing is skipped for their tiles.)
//
// A layer's prefill of 6 x 777 padded tokens (32 heads, boolean mask) takes 371 us with it and 507 us with the mask made
// additive by three elementwise kernels (12 us) and read as floats, 64 scattered loads per thread and tile (the other
// kernels of that pass being equal).
//
// Bound by the mask's bytes, or for the few rows of a generation step by the latency of one load: one warp per row, several
// where a group has fewer rows than warps, 128 keys (four per lane) per step, four steps in flight.  The kernels that read
// the summary start their own set-up under it (programmatic dependent launch).
#include "tq_attention.cuh"
#include "tq_common.cuh"

namespace tq {
namespace {

constexpr int kTileKeys = 128, kGroupRows = 16, kChunkTiles = 16;  // keys per tile, rows per group, tiles per CTA

struct MaskArgs {
  const void* mask;
  int64_t stride_b, stride_q;  // elements
  int Sq, Sk, shift, causal;
  int warps_per_row;  // a power of two
  uint32_t* words;
  uint8_t* tiles;
  uint32_t* rows;
  int T, NG, NC;
};

template <bool BOOL>
__global__ void __launch_bounds__(kGroupRows * 32) mask_summary_kernel(const MaskArgs a) {
  __shared__ uint32_t s_cls[kChunkTiles];
  __shared__ uint32_t s_rows;
  const int tid = threadIdx.x, warp = tid / 32, lane = tid % 32;
  const int64_t b = blockIdx.z;
  const int group = blockIdx.y, chunk = blockIdx.x;
  const int t0 = chunk * kChunkTiles, t1 = min(a.T, t0 + kChunkTiles);
  grid_launch_dependents();
  if (tid < kChunkTiles) s_cls[tid] = 0;
  if (tid == 0) s_rows = 0;
  __syncthreads();
  const int row = warp / a.warps_per_row, s = group * kGroupRows + row;
  if (s < a.Sq) {
    const int last = a.causal ? min(a.Sk - 1, s + a.shift) : a.Sk - 1;  // last key of the row's causal range
    const int64_t row_off = b * a.stride_b + (int64_t)s * a.stride_q;
    bool any_row = false;
    // kAhead tiles' loads in flight: a row is a chain of latencies otherwise (4000 keys: 23 us)
    constexpr int kAhead = 4;
    for (int ta = t0 + warp % a.warps_per_row * kAhead; ta < t1; ta += a.warps_per_row * kAhead) {
    uint32_t raw[kAhead][BOOL ? 2 : 4];
#pragma unroll
    for (int x = 0; x < kAhead; ++x) {
      const int k = (ta + x) * kTileKeys + 4 * lane;  // this lane's four keys
      const int n = ta + x < t1 ? a.Sk - k : 0;       // how many of them (and after them) exist
      if constexpr (BOOL) {
        // four bytes at any alignment: the aligned words around them, each loaded only if it holds a byte of the row
        const uint8_t* p = static_cast<const uint8_t*>(a.mask) + row_off + k;
        const uint32_t m = (uint32_t)(reinterpret_cast<uintptr_t>(p) & 3u);
        const uint32_t* w = reinterpret_cast<const uint32_t*>(p - m);
        raw[x][0] = n > 0 ? __ldg(w) : 0u;
        raw[x][1] = (m != 0 && n > (int)(4 - m)) ? __ldg(w + 1) : 0u;
      } else {
        const float* p = static_cast<const float*>(a.mask) + row_off + k;
        if (n >= 4 && (reinterpret_cast<uintptr_t>(p) & 15u) == 0) {
          const uint4 q = __ldg(reinterpret_cast<const uint4*>(p));
          raw[x][0] = q.x; raw[x][1] = q.y; raw[x][2] = q.z; raw[x][3] = q.w;
        } else {
#pragma unroll
          for (int e = 0; e < 4; ++e) raw[x][e] = e < n ? __float_as_uint(__ldg(p + e)) : 0xff800000u;
        }
      }
    }
#pragma unroll
    for (int x = 0; x < kAhead; ++x) {
      const int t = ta + x;
      if (t >= t1) break;
      const int k = t * kTileKeys + 4 * lane, n = a.Sk - k;
      uint32_t vis = 0, oth = 0;
      if constexpr (BOOL) {
        const uint32_t m = (uint32_t)((reinterpret_cast<uintptr_t>(a.mask) + (uintptr_t)(row_off + k)) & 3u);
        const uint32_t v = __funnelshift_r(raw[x][0], raw[x][1], 8 * m);
#pragma unroll
        for (int e = 0; e < 4; ++e) vis |= (e < n && ((v >> (8 * e)) & 0xffu) != 0u) ? 1u << e : 0u;
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float f = __uint_as_float(raw[x][e]);
          vis |= f == 0.f ? 1u << e : 0u;
          oth |= (f == 0.f || f <= -1e30f) ? 0u : 1u << e;  // (a NaN is neither)
        }
      }
      const uint32_t seen = vis | oth;  // keys that are not hidden
#pragma unroll
      for (int e = 0; e < 4; ++e) any_row |= ((seen >> e) & 1u) != 0u && k + e <= last;
      const uint32_t live = k >= a.Sk ? 0u : (a.Sk - k >= 4 ? 15u : (1u << (a.Sk - k)) - 1u);  // keys that exist
      const uint32_t cls = (seen ? 1u : 0u) | ((live & ~seen) ? 2u : 0u) | (oth ? 4u : 0u);
      const uint32_t all = __reduce_or_sync(0xffffffffu, cls);
      uint32_t w = seen << (4 * (lane % 8));
      w |= __shfl_xor_sync(0xffffffffu, w, 1);
      w |= __shfl_xor_sync(0xffffffffu, w, 2);
      w |= __shfl_xor_sync(0xffffffffu, w, 4);
      if (lane % 8 == 0) a.words[(b * a.Sq + s) * (4 * (int64_t)a.T) + 4 * t + lane / 8] = w;
      if (lane == 0 && all != 0u) atomicOr(&s_cls[t - t0], all);
    }
    }
    if (__any_sync(0xffffffffu, any_row) && lane == 0) atomicOr(&s_rows, 1u << row);
  }
  __syncthreads();
  if (t0 + tid < t1) a.tiles[(b * a.NG + group) * (int64_t)a.T + t0 + tid] = (uint8_t)s_cls[tid];
  if (tid == 0) a.rows[(b * a.NG + group) * (int64_t)a.NC + chunk] = s_rows;
}

inline size_t round16(size_t v) { return (v + 15) & ~(size_t)15; }

}  // namespace

MaskBits mask_bits_layout(int64_t nb, int64_t Sq, int64_t Sk, void* base, size_t* bytes) {
  MaskBits m{};
  m.T = (int)((Sk + kTileKeys - 1) / kTileKeys);
  m.NG = (int)((Sq + kGroupRows - 1) / kGroupRows);
  m.NC = (m.T + kChunkTiles - 1) / kChunkTiles;
  m.batch = nb > 1 ? 1 : 0;
  uint8_t* p = static_cast<uint8_t*>(base);
  m.words = reinterpret_cast<const uint32_t*>(p);
  size_t off = round16((size_t)nb * Sq * m.T * 16);
  m.rows = reinterpret_cast<const uint32_t*>(p + off);
  off += round16((size_t)nb * m.NG * m.NC * 4);
  m.tiles = p + off;
  off += round16((size_t)nb * m.NG * m.T);
  if (bytes != nullptr) *bytes = (off + 255) & ~(size_t)255;
  return m;
}

int summarize_mask(const void* mask, bool boolean, int64_t nb, int64_t stride_b, int64_t stride_q, int64_t Sq, int64_t Sk,
                   int causal, const MaskBits& m, cudaStream_t stream) {
  TQ_REQUIRE(nb <= 65535 && m.NG <= 65535, "mask of %lld x %lld rows is too large", (long long)nb, (long long)Sq);
  int per_row = 1;
  while (2 * per_row * Sq <= kGroupRows) per_row *= 2;
  const MaskArgs a{mask, nb > 1 ? stride_b : 0, stride_q, (int)Sq, (int)Sk, (int)(Sk - Sq), causal, per_row,
                   const_cast<uint32_t*>(m.words), const_cast<uint8_t*>(m.tiles), const_cast<uint32_t*>(m.rows),
                   m.T, m.NG, m.NC};
  const dim3 grid((unsigned)m.NC, (unsigned)m.NG, (unsigned)nb);
  if (boolean) mask_summary_kernel<true><<<grid, kGroupRows * 32, 0, stream>>>(a);
  else mask_summary_kernel<false><<<grid, kGroupRows * 32, 0, stream>>>(a);
  TQ_CUDA_OK(cudaGetLastError());
  return TQ_OK;
}

}  // namespace tq
