// Fused key + value compression, one launch (TQ_MODE_BF16, bf16 or fp16 inputs).
//
// Replaces TurboQuantCompressorV2.compress and TurboQuantCompressorMSE.compress of the reference
// (src/turboquant_pytorch/compressors.py:98-161, :270-294) with the packed result layout of compressors.py:132-138,
// :281-285.  The arithmetic is that of tq_compress_tc.cu (rotation and sketch projection on tcgen05 from split-bf16
// operands, index by boundary counting, residual in rotated coordinates); what differs is how a CTA is organised:
//
//   * work units are 128-vector tiles of one (batch, head): all key tiles, then all value tiles, dealt round-robin
//     to a persistent grid of one CTA per SM, so every CTA handles its key tiles first and then its value tiles
//     (one switch of the constant operands in between);
//   * a control warp stages tiles with TMA (cp.async.bulk.tensor, 128-byte swizzle, three slots; a tensor map
//     over the caller's [B, H, S, d] view, so any 16-byte-aligned strides work and rows past S arrive as zeros)
//     and issues the MMAs; the raw bf16 tile is the A operand as it lands;
//   * 16 epilogue warps (row = tensor-memory lane, 32 coordinates per thread) turn accumulators into packed bytes;
//   * three accumulator slots in tensor memory: the rotation of tile i+1 runs under the epilogue of tile i.  The
//     key residual (fp32, split into bf16 hi + lo) goes back to TENSOR MEMORY and is the A operand of the sketch
//     MMA there, so it costs no shared memory and no proxy fence; its projection overwrites the rotated
//     coordinates it came from.  The sign pass of tile i runs after the index pass of tile i+1, under which the
//     sketch MMA of tile i has finished;
//   * fp16 inputs are exact operands of fp16 MMAs against fp16 hi + lo images of the rotations (scaled to rows of norm
//     128, to keep the low parts out of the subnormals) and of the sketch: 22 mantissa bits, small products first.  Against fp64 as many
//     indices and signs differ as with the fp32 CUDA-core kernel (53 / 113 / 132 of 4e8 key indices, signs and value
//     indices; fp32: 53 / 110 / 131), and with the repair below the same ones: 48 us instead of 171 us for the 6 x 8 x 777
//     keys and values of a padded prompt;
//   * head_dim 64 takes half of tensor and shared memory, so two CTAs share an SM (8 x 12 x 1024 keys and values: 15 us
//     instead of 38 us for a launch per side of the kernel in tq_compress_tc.cu);
//   * the constant operands (Pi hi/lo, S_eff hi/lo for keys; Pi_v hi/lo for values) are bulk-copied from images
//     built once per compressor pair (tq_prepare_constants).
//
// Every wait is bounded; on expiry the CTA raises its abort flag, all roles leave their loops at their next wait,
// outstanding copies are waited for (bounded), tensor memory is freed and the fault is counted and reported.
#include <cuda.h>

#include <type_traits>

#include "tq_attention.cuh"
#include "tq_compress.cuh"
#include "tq_simt.cuh"
#include "tq_tcgen05.cuh"

namespace tq {

__device__ unsigned long long g_compress_kv_faults = 0ull;
__device__ unsigned long long* g_fault_mailbox_compress_kv = nullptr;
int set_fault_mailbox_compress_kv(unsigned long long* slot) {
  TQ_CUDA_OK(cudaMemcpyToSymbol(g_fault_mailbox_compress_kv, &slot, sizeof(slot)));
  return TQ_OK;
}
int read_compress_kv_faults(unsigned long long* out) {
  TQ_CUDA_OK(cudaMemcpyFromSymbol(out, g_compress_kv_faults, sizeof(*out)));
  return TQ_OK;
}

namespace {

constexpr int kSlots = 3;
template <int D>
struct KvShape {
  static constexpr int kParts = D / 32;                 // threads per row
  static constexpr int kEpiWarps = 4 * kParts;
  static constexpr int kThreads = (kEpiWarps + 1) * 32;
  // head_dim 128: all of tensor memory, nearly all of shared memory; head_dim 64: half of either
  static constexpr int kCtasPerSm = D == 64 ? 2 : 1;
  static constexpr uint32_t kTileBytes = 128 * D * 2;   // one 16-bit tile: one or two 64-column boxes of 16 KB
  static constexpr uint32_t kBoxBytes = 128 * 64 * 2;
  static constexpr uint32_t kMatBytes = D * D * 2;      // one 16-bit operand image
  static constexpr uint32_t kOffX = 0;
  static constexpr uint32_t kOffConst = kSlots * kTileBytes;
  static constexpr uint32_t kOffExch = kOffConst + 4 * kMatBytes;
  static constexpr uint32_t kOffMisc = kOffExch + kParts * 128 * 4;  // barriers, tensor-memory slot, abort flag, centroids
  static constexpr uint32_t kSmemBytes = kOffMisc + 256;
  // tensor memory: three accumulator slots (rotated coordinates, later the sketch projection), residual hi, lo
  static constexpr uint32_t kColYP = 0, kColRH = 3 * D, kColRL = 3 * D + D / 2, kCols = 4 * D;
  static_assert(kCtasPerSm * (kSmemBytes + 1024) <= 228 * 1024, "shared memory over-subscribed");
};

struct KvArgs {
  uint32_t units_k, units_v;  // tiles on either side (32-bit: unit arithmetic runs per thread and tile)
  uint32_t tiles_s, tiles_h;  // tiles along the positions and along the heads (times those along the batch)
  uint32_t box_s, box_h, box_b;  // positions x heads x batch elements of one tile, at most 128 vectors
  uint32_t S, H, B;
  const uint8_t* consts;      // constants buffer of tq_prepare_constants
  uint8_t* key_idx;
  uint8_t* key_sgn;
  uint16_t* key_vn;
  uint16_t* key_rn;
  uint8_t* val_idx;
  uint16_t* val_vn;
  const void *k, *v;             // the inputs and their element strides (batch, head, position): fp16 repair only
  int64_t k_stride[3], v_stride[3];
  int64_t out_stride, out_offset;  // vector (bh, s) -> output row bh * out_stride + out_offset + s
  ConstLayout L;
};

__device__ __forceinline__ uint32_t bf16_bits(float v) {
  return static_cast<uint32_t>(__bfloat16_as_ushort(__float2bfloat16_rn(v)));
}
__device__ __forceinline__ float bf16_value(uint32_t b) { return __uint_as_float(b << 16); }

// Number of ascending boundaries strictly below y (the Lloyd-Max index), without compares or selects: the sign
// bit of (b - y) is set exactly when y > b (b - y == 0 gives +0), and mad.hi by 2 adds that bit to the count.  Both
// instructions run on the FMA pipe, which issues at twice the rate of the integer/compare pipe this epilogue would
// otherwise saturate.
// Codebooks of 8 and more levels use the symmetry of the boundaries (b[NB-1-j] = -b[j], b[(NB-1)/2] = 0): the sign
// of y and the count m of positive boundaries below |y| give idx = h + m for y > 0 and h - 1 - m otherwise
// (h = (NB+1)/2), with half the subtractions.  The one difference: a NEGATIVE y that equals a boundary exactly
// lands one level higher than the strict count would put it (part of the documented tie budget).  SYM false: boundaries
// that a caller replaced by ones without that symmetry, counted as they are.
template <int NB, bool SYM>
__device__ __forceinline__ uint32_t index_of(float y, const float (&bd)[NB]) {
  if constexpr (NB < 7 || !SYM) {
    uint32_t idx = 0;
#pragma unroll
    for (int j = 0; j < NB; ++j) {
      const uint32_t d = __float_as_uint(bd[j] - y);
      asm("mad.hi.u32 %0, %1, 2, %2;" : "=r"(idx) : "r"(d), "r"(idx));
    }
    return idx;
  } else {
    constexpr int h = (NB + 1) / 2;
    uint32_t m = 0, pos = 0;
    const uint32_t dz = __float_as_uint(0.f - y);  // sign set iff y > 0
    asm("mad.hi.u32 %0, %1, 2, %2;" : "=r"(pos) : "r"(dz), "r"(pos));
    const float ay = fabsf(y);
#pragma unroll
    for (int j = 0; j < h - 1; ++j) {
      const uint32_t d = __float_as_uint(bd[h + j] - ay);
      asm("mad.hi.u32 %0, %1, 2, %2;" : "=r"(m) : "r"(d), "r"(m));
    }
    return (uint32_t)(h - 1) - m + pos * (2u * m + 1u);
  }
}
template <int NB>
__device__ __forceinline__ bool symmetric(const float (&b)[NB]) {
  bool s = NB < 7 || b[NB / 2] == 0.f;
#pragma unroll
  for (int j = 0; NB >= 7 && j < NB / 2; ++j) s = s && b[j] == -b[NB - 1 - j];
  return s;
}
// OR the B-bit field of coordinate E (of this thread's 32) into the thread's B packed words (LSB-first bit stream)
template <int B, int E>
__device__ __forceinline__ void put_field(uint32_t (&w)[B], uint32_t idx) {
  constexpr int pos = E * B, k = pos / 32, sh = pos % 32;
  w[k] = idx * (1u << sh) + w[k];  // the field's bits are still zero there: + is |
  if constexpr (sh + B > 32) w[k + 1] = (idx >> (32 - sh)) + w[k + 1];
}
template <int B, int E>
__device__ __forceinline__ uint32_t get_field(const uint32_t (&w)[B]) {
  constexpr int pos = E * B, k = pos / 32, sh = pos % 32;
  uint32_t v = w[k] >> sh;
  if constexpr (sh + B > 32) v |= w[k + 1] << (32 - sh);
  return v & ((1u << B) - 1);
}
// fp16 inputs: passes over a warp's 32 rows x 32 coordinates (in tensor memory at `col`) for boundaries that are counted as
// they are, scaled by `den`.  Not inlined: inside the kernel they would cost the passes for symmetric boundaries registers
// (4 bits, 8 x 8 x 4096 keys and values: 227 us inlined, 185 us so).
template <int B>
__device__ __noinline__ void index_any(uint32_t col, const float* __restrict__ bnd, float den, uint32_t (&packed)[B]) {
  constexpr int NB = (1 << B) - 1;
  uint32_t raw[32];
  tc::tmem_ld32(col, raw);
  tc::wait_ld();
  uint64_t word = 0;
#pragma unroll
  for (int j = 0; j < B; ++j) packed[j] = 0;
#pragma unroll
  for (int e = 0; e < 32; ++e) {
    uint32_t idx = 0;
#pragma unroll 1
    for (int j = 0; j < NB; ++j) idx += __uint_as_float(raw[e]) > __ldg(bnd + j) * den ? 1u : 0u;
    const int bit = e * B, k = bit / 32, sh = bit % 32;
    word = (uint64_t)idx << sh;
    packed[k] |= (uint32_t)word;
    if (sh + B > 32) packed[k + 1 < B ? k + 1 : k] |= (uint32_t)(word >> 32);
  }
}
// ... bit e set where coordinate e lies within `band` of a boundary
template <int NB>
__device__ __noinline__ uint32_t open_any(uint32_t col, const float* __restrict__ bnd, float den, float band) {
  uint32_t raw[32], open = 0;
  tc::tmem_ld32(col, raw);
  tc::wait_ld();
#pragma unroll
  for (int e = 0; e < 32; ++e) {
    float near = INFINITY;
#pragma unroll 1
    for (int j = 0; j < NB; ++j) near = fminf(near, fabsf(__ldg(bnd + j) * den - __uint_as_float(raw[e])));
    open |= near < band ? 1u << e : 0u;
  }
  return open;
}

// Repair of fp16 decisions that the tensor-core sums leave open.
//
// An index or a sign whose coordinate lies within the sums' rounding of its boundary may fall either way, and a single
// moved index moves about seven sign bytes of its vector.  A 16-bit input type with exact operands should not differ from
// the fp32 kernel in that way, so coordinates within kOpenIndex (in units of the norm) and projections within kOpenSign (in
// units of the residual's norm) are decided by the fp32 kernel's own arithmetic: the functions below, one warp per open
// coordinate, with its order of operations.  The bands follow from that kernel's rounding, the larger of the two: a sum of d
// multiply-adds whose partial sums are about as large as the boundary is off by 2^-25 of it sqrt(d) / 2 times or so, 1.8e-8 rms
// near a boundary (measured against fp64: 1.6e-8 to 1.8e-8 at 3 and 4 bits, either head_dim), and passes that error on to a
// projection sqrt(d) fold against a residual of 0.1 to 0.4 of the norm (0.5e-6 to 1.3e-6 rms measured; the tensor-core
// sums: 1e-8).  Nine and five times that leave less than one decision in 1e10 to chance.  About one
// vector in 700 has one; the compression of 6 x 8 x 777 keys and values takes 48 us with the
// repair and 22 us without (171 us on the fp32 kernels).
constexpr float kOpenIndex = 1.6e-7f, kOpenSign = 6e-6f;

// The fp32 kernel's norm of an fp16 row (sums of eight, then a butterfly) and this lane's normalised coordinates.
template <int D>
struct ExactRow {
  static constexpr int N = D / 32;  // coordinates per lane: N lane .. N lane + N - 1
  float x[N], norm;
  __device__ explicit ExactRow(const __half* row) {
    const int lane = threadIdx.x % 32, g = lane % (D / 8);
    float ss = 0.f;
    for (int e = 0; e < 8; ++e) {
      const float f = __half2float(row[8 * g + e]);
      ss = fmaf(f, f, ss);
    }
    for (int off = D / 16; off > 0; off >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, off);
    norm = sqrtf(ss);
    const float den = norm + 1e-8f;
#pragma unroll
    for (int e = 0; e < N; ++e) x[e] = __half2float(row[N * lane + e]) / den;
  }
};
// sum over i = 0 .. D - 1, in that order, of in[i] * m[i]; `in` spread over the lanes as in ExactRow
template <int D>
__device__ __forceinline__ float exact_dot(const float (&in)[D / 32], const float* __restrict__ m) {
  constexpr int N = D / 32;
  float w[N];
#pragma unroll
  for (int e = 0; e < N; ++e) w[e] = __ldg(m + N * (threadIdx.x % 32) + e);
  float acc = 0.f;
#pragma unroll 4
  for (int l = 0; l < 32; ++l)
#pragma unroll
    for (int e = 0; e < N; ++e)
      acc = fmaf(__shfl_sync(0xffffffffu, in[e], l), __shfl_sync(0xffffffffu, w[e], l), acc);
  return acc;
}
// Rotated coordinate of a row, as the fp32 kernel computes it (`m` is that row of the rotation).
template <int D>
__device__ __noinline__ float exact_coordinate(const __half* row, const float* __restrict__ m) {
  const ExactRow<D> r(row);
  return exact_dot<D>(r.x, m);
}
// Projection j of the residual of a key row, as the fp32 kernel computes it.
template <int D, int NB>
__device__ __noinline__ float exact_projection(const __half* row, const float* __restrict__ Pi,
                                               const float* __restrict__ S_eff, const float* __restrict__ bnd,
                                               const float* __restrict__ cen, int j) {
  constexpr int N = D / 32;
  const ExactRow<D> r(row);
  const float np = r.norm + 1e-8f;
  const int lane = threadIdx.x % 32;
  float y[N];
#pragma unroll
  for (int e = 0; e < N; ++e) y[e] = 0.f;
  // this lane's N rotated coordinates, sums over i in order
#pragma unroll 1
  for (int l0 = 0; l0 < 32; l0 += 4) {
    float w[N][4 * N];  // 4 N columns of this lane's N rows, all loads in flight
#pragma unroll
    for (int o = 0; o < N; ++o)
#pragma unroll
      for (int c = 0; c < 4 * N; c += 4) {
        const float4 v = __ldg(reinterpret_cast<const float4*>(Pi + (N * lane + o) * D + N * l0 + c));
        w[o][c] = v.x; w[o][c + 1] = v.y; w[o][c + 2] = v.z; w[o][c + 3] = v.w;
      }
#pragma unroll
    for (int c = 0; c < 4 * N; ++c) {
      const float xs = __shfl_sync(0xffffffffu, r.x[c % N], l0 + c / N);
#pragma unroll
      for (int o = 0; o < N; ++o) y[o] = fmaf(xs, w[o][c], y[o]);
    }
  }
#pragma unroll
  for (int o = 0; o < N; ++o) {
    int idx = 0;
    for (int b = 0; b < NB; ++b) idx += y[o] > __ldg(bnd + b) ? 1 : 0;
    y[o] = fmaf(np, y[o], -r.norm * __ldg(cen + idx));
  }
  return exact_dot<D>(y, S_eff + j * D);
}

template <int FROM, int TO, class F>
__device__ __forceinline__ void static_for(F&& f) {
  if constexpr (FROM < TO) {
    f(std::integral_constant<int, FROM>{});
    static_for<FROM + 1, TO>(f);
  }
}

// One box of a rank-4 tiled tensor map (64 columns x 128 rows of one (batch, head)) -> shared memory, completion
// counted in bytes on `bar` of this CTA.  No multicast.
__device__ __forceinline__ void tma_load_tile(uint32_t dst, const CUtensorMap* map, int c0, int c1, int c2, int c3,
                                              uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
      :
      : "r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
      : "memory");
}
// Shared-memory descriptor of a K-major operand in the 128-byte-swizzled layout TMA writes (rows of 128 bytes,
// 8-row groups 1024 bytes apart); `saddr` is the tile base (1024-byte aligned) plus 32 bytes per K step of 16.
__device__ __forceinline__ uint64_t smem_desc_sw128(uint32_t saddr) {
  return static_cast<uint64_t>((saddr >> 4) & 0x3FFFu) | (1ull << 16) | (static_cast<uint64_t>(1024 >> 4) << 32) |
         (1ull << 46) | (2ull << 61);
}

// F16: fp16 inputs (and fp16 operand images of the rotations), else bf16.
template <int D, int BITS, bool F16>
__global__ void __launch_bounds__(KvShape<D>::kThreads, KvShape<D>::kCtasPerSm)
compress_kv_kernel(const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v, const KvArgs a) {
  using L = KvShape<D>;
  constexpr int kD = D, kParts = L::kParts, kEpiWarps = L::kEpiWarps;
  constexpr uint32_t kTileBytes = L::kTileBytes, kMatBytes = L::kMatBytes, kOffX = L::kOffX, kOffConst = L::kOffConst;
  constexpr uint32_t kOffExch = L::kOffExch, kOffMisc = L::kOffMisc;
  constexpr uint32_t kColYP = L::kColYP, kColRH = L::kColRH, kColRL = L::kColRL;
  // Split of the residual for the sketch: fp16 hi + lo of the residual scaled by a power of two (22 mantissa bits), or
  // bf16 hi + lo (16 bits), which needs no scaling and two operations fewer per coordinate.
  constexpr bool SK16 = F16 || D == 64;
  // the rotated coordinates come out times these powers of two
  const float* const scales = reinterpret_cast<const float*>(a.consts + a.L.header) + kScaleWord;
  const float yscale_k = F16 ? __ldg(scales) : 1.f, yscale_v = F16 ? __ldg(scales + 1) : 1.f;
  constexpr int KB = BITS - 1, VB = BITS;
  constexpr uint32_t SBO = (kD / 8) * 128;  // canonical (unswizzled) K-major images of the constant operands
  extern __shared__ __align__(1024) uint8_t smem[];
  float (*exch)[128] = reinterpret_cast<float (*)[128]>(smem + kOffExch);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + kOffMisc);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + kOffMisc + 208);
  int* s_abort_p = reinterpret_cast<int*>(smem + kOffMisc + 212);
  float* cen_s = reinterpret_cast<float*>(smem + kOffMisc + 216);  // 2^KB <= 8 key centroids
  volatile int* abort_flag = s_abort_p;
  const uint32_t bar0 = tc::smem_u32(bars);
  auto bar = [&](int i) { return bar0 + 8u * i; };
  // 0: constants landed; 1-3: tile landed; 4-6: rotation done; 7-9: sketch done; 10-12: accumulator slot read out;
  // 13: residual operand written; 14-17: row-part exchange per lane quarter; 18-21: exchange buffer read out;
  // 22-24: tile read out of shared memory by the epilogue (its slot may be refilled once the rotation is done too)
  const uint32_t const_full = bar(0), r_full = bar(13);
  auto x_full = [&](int s) { return bar(1 + s); };
  auto y_done = [&](int s) { return bar(4 + s); };
  auto p_done = [&](int s) { return bar(7 + s); };
  auto yp_free = [&](int s) { return bar(10 + s); };
  auto xch = [&](int q) { return bar(14 + q); };
  auto xfree = [&](int q) { return bar(18 + q); };
  auto x_read = [&](int s) { return bar(22 + s); };

  const int tid = threadIdx.x, warp = tid / 32, lane = tid % 32;
  const uint32_t total = a.units_k + a.units_v;
  const uint32_t G = gridDim.x, c = blockIdx.x;
  const int n = (int)((total - c + G - 1) / G);                                  // units of this CTA
  const int nk = c < a.units_k ? (int)((a.units_k - c + G - 1) / G) : 0;         // ... of which key tiles (first)

  if (tid == 0) {
    *s_abort_p = 0;
    tc::mbar_init(const_full, 1);
    for (int s = 0; s < kSlots; ++s) {
      tc::mbar_init(x_full(s), 1);
      tc::mbar_init(y_done(s), 1);
      tc::mbar_init(p_done(s), 1);
      tc::mbar_init(yp_free(s), kEpiWarps);
      tc::mbar_init(x_read(s), kEpiWarps);
    }
    tc::mbar_init(r_full, kEpiWarps);
    for (int q = 0; q < 4; ++q) {
      tc::mbar_init(xch(q), kParts);
      tc::mbar_init(xfree(q), kParts);
    }
    tc::fence_mbar_init();
  }
  if (tid < (1 << KB)) cen_s[tid] = __ldg(reinterpret_cast<const float*>(a.consts + a.L.cen_k) + tid);
  if (warp == kEpiWarps) tc::tmem_alloc(tc::smem_u32(tmem_slot), L::kCols);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = *tmem_slot;
  bool ok = true;

  // this CTA's i-th unit -> side, first batch element, head and position of the tile
  auto unit_of = [&](int i, bool& is_key, uint32_t& b0, uint32_t& h0, uint32_t& s0) {
    const uint32_t g = c + (uint32_t)i * G;
    is_key = g < a.units_k;
    const uint32_t t = is_key ? g : g - a.units_k;
    const uint32_t th = t / a.tiles_s;
    s0 = (t - th * a.tiles_s) * a.box_s;
    b0 = th / a.tiles_h;
    h0 = (th - b0 * a.tiles_h) * a.box_h;
    b0 *= a.box_b;
  };

  if (warp == kEpiWarps) {
    // ======================================= control warp =======================================
    if (lane == 0 && n > 0) {
      int issued = 0;  // tiles whose copies have been issued
      auto issue_tile = [&](int i) {
        bool is_key;
        uint32_t b0, h0, s0;
        unit_of(i, is_key, b0, h0, s0);
        const int s = i % kSlots;
        const CUtensorMap* map = is_key ? &map_k : &map_v;
        const uint32_t dst = tc::smem_u32(smem + kOffX + s * kTileBytes);
        tc::mbar_arrive_expect_tx(x_full(s), a.box_s * a.box_h * a.box_b * (D * 2));
#pragma unroll
        for (int x = 0; x < D / 64; ++x)
          tma_load_tile(dst + x * L::kBoxBytes, map, 64 * x, (int)s0, (int)h0, (int)b0, x_full(s));
        issued = i + 1;
      };
      auto load_consts = [&](bool keys) {
        const uint32_t dst = tc::smem_u32(smem + kOffConst);
        if (keys) {
          tc::mbar_arrive_expect_tx(const_full, 4 * kMatBytes);
          tc::bulk_load(dst, a.consts + (F16 ? a.L.pik16_hi : a.L.pik_hi), kMatBytes, const_full);
          tc::bulk_load(dst + kMatBytes, a.consts + (F16 ? a.L.pik16_lo : a.L.pik_lo), kMatBytes, const_full);
          tc::bulk_load(dst + 2 * kMatBytes, a.consts + (SK16 ? a.L.se16_hi : a.L.se_hi), kMatBytes, const_full);
          tc::bulk_load(dst + 3 * kMatBytes, a.consts + (SK16 ? a.L.se16_lo : a.L.se_lo), kMatBytes, const_full);
        } else {
          tc::mbar_arrive_expect_tx(const_full, 2 * kMatBytes);
          tc::bulk_load(dst, a.consts + (F16 ? a.L.piv16_hi : a.L.piv_hi), kMatBytes, const_full);
          tc::bulk_load(dst + kMatBytes, a.consts + (F16 ? a.L.piv16_lo : a.L.piv_lo), kMatBytes, const_full);
        }
      };
      constexpr uint32_t idesc = F16 ? tc::idesc_f16(128, kD, false, false) : tc::idesc_bf16(128, kD, false, false);
      constexpr uint32_t idesc_p = SK16 ? tc::idesc_f16(128, kD, false, false) : tc::idesc_bf16(128, kD, false, false);
      const uint32_t cbase = tc::smem_u32(smem + kOffConst);
      const uint64_t b_hi = tc::smem_desc(cbase, 128, SBO), b_lo = tc::smem_desc(cbase + kMatBytes, 128, SBO);
      const uint64_t se_hi = tc::smem_desc(cbase + 2 * kMatBytes, 128, SBO);
      const uint64_t se_lo = tc::smem_desc(cbase + 3 * kMatBytes, 128, SBO);
      // sketch of key tile i: P = r_hi Se_hi^T + r_hi Se_lo^T + r_lo Se_hi^T, A from tensor memory, into the slot
      // whose rotated coordinates the residual was computed from
      auto issue_sketch = [&](int i) {
        if (!(ok = tc::mbar_wait_or_abort(r_full, i & 1, abort_flag))) return;
        tc::fence_after_sync();
        const uint32_t d_p = tmem + kColYP + (i % kSlots) * kD;
        auto product = [&](uint32_t col, uint64_t b, uint32_t first) {
#pragma unroll
          for (int ks = 0; ks < kD / 16; ++ks)
            tc::mma_bf16_ts(d_p, tmem + col + ks * 8, b + (uint64_t)(ks * 256 >> 4), idesc_p, ks > 0 ? 1u : first ^ 1u);
        };
        // the accumulator is truncated at every step, so the 22-bit form adds the large product to the small ones
        if constexpr (SK16) {
          product(kColRL, se_hi, 1u);
          product(kColRH, se_lo, 0u);
          product(kColRH, se_hi, 0u);
        } else {
          product(kColRH, se_hi, 1u);
          product(kColRH, se_lo, 0u);
          product(kColRL, se_hi, 0u);
        }
        tc::mma_commit(p_done(i % kSlots));
      };
      bool keys_loaded = nk > 0;
      int const_phase = 0;
      load_consts(keys_loaded);
      for (int t = 0; t < kSlots && t < n; ++t) issue_tile(t);
      ok = tc::mbar_wait_or_abort(const_full, const_phase, abort_flag);
      bool sketch_pending = false;  // the sketch of tile i-1 has not been issued yet
      for (int i = 0; i < n && ok; ++i) {
        const int s = i % kSlots, u = i / kSlots;
        const bool is_key = i < nk;
        if (!is_key && keys_loaded) {
          // last key tile behind us: finish its sketch, wait until no MMA reads the key operands, swap them
          if (sketch_pending) {
            issue_sketch(i - 1);
            sketch_pending = false;
            if (!ok) break;
          }
          if (nk > 0 && !(ok = tc::mbar_wait_or_abort(p_done((nk - 1) % kSlots), ((nk - 1) / kSlots) & 1, abort_flag))) break;
          keys_loaded = false;
          const_phase ^= 1;
          load_consts(false);
          if (!(ok = tc::mbar_wait_or_abort(const_full, const_phase, abort_flag))) break;
        }
        if (!(ok = tc::mbar_wait_or_abort(x_full(s), u & 1, abort_flag))) break;
        if (i >= kSlots && !(ok = tc::mbar_wait_or_abort(yp_free(s), (u - 1) & 1, abort_flag))) break;
        tc::fence_after_sync();
        {
          // rotation: Y_raw = X Pi_hi^T + X Pi_lo^T; K step ks reads 32 bytes of each 128-byte row of half ks / 4
          const uint32_t xb = tc::smem_u32(smem + kOffX + s * kTileBytes);
          const uint32_t d_y = tmem + kColYP + s * kD;
          auto product = [&](uint64_t b, uint32_t first) {
#pragma unroll
            for (int ks = 0; ks < kD / 16; ++ks)
              tc::mma_bf16(d_y, smem_desc_sw128(xb + (ks / 4) * L::kBoxBytes + (ks % 4) * 32), b + (uint64_t)(ks * 256 >> 4),
                           idesc, ks > 0 ? 1u : first ^ 1u);
          };
          product(F16 ? b_lo : b_hi, 1u);
          product(F16 ? b_hi : b_lo, 0u);
          tc::mma_commit(y_done(s));
        }
        if (sketch_pending) {
          issue_sketch(i - 1);
          sketch_pending = false;
          if (!ok) break;
        }
        sketch_pending = is_key;
        // the slot tile i-1 came from is free once its rotation has completed AND the epilogue has read its rows
        // for the norms (the control warp runs ahead of the epilogue; a refill before that read would also let
        // the slot's barrier run two phases ahead of a waiter): refill it with tile i+2
        if (i >= 1 && i + 2 < n) {
          if (!(ok = tc::mbar_wait_or_abort(y_done((i - 1) % kSlots), ((i - 1) / kSlots) & 1, abort_flag))) break;
          if (!(ok = tc::mbar_wait_or_abort(x_read((i - 1) % kSlots), ((i - 1) / kSlots) & 1, abort_flag))) break;
          issue_tile(i + 2);
        }
      }
      if (ok && sketch_pending) issue_sketch(n - 1);
      if (!ok) {
        // give the copies in flight a bounded time to land before the CTA's shared memory goes away
        for (int i = 0; i < issued; ++i) tc::mbar_wait_bounded(x_full(i % kSlots), (i / kSlots) & 1, 20000000ll);
      }
    }
  } else {
    // ======================================= epilogue warps =======================================
    const int q = warp % 4, part = warp / 4;  // lane quarter of tensor memory; coordinates [32 part, 32 part + 32)
    const int row = q * 32 + lane;
    const uint32_t lane_base = (uint32_t)(q * 32) << 16;
    float bnd_k[(1 << KB) - 1], bnd_v[(1 << VB) - 1];
#pragma unroll
    for (int j = 0; j < (1 << KB) - 1; ++j) bnd_k[j] = __ldg(reinterpret_cast<const float*>(a.consts + a.L.bnd_k) + j);
#pragma unroll
    for (int j = 0; j < (1 << VB) - 1; ++j) bnd_v[j] = __ldg(reinterpret_cast<const float*>(a.consts + a.L.bnd_v) + j);
    const bool sym_k = symmetric(bnd_k), sym_v = symmetric(bnd_v);
    // boundaries scaled for a tile's pass: from registers where symmetry needs half of them only, else loaded again
    auto scaled = [](auto sym, const float* src, const auto& bnd, float den, auto& bden) {
#pragma unroll
      for (int j = 0; j < (int)(sizeof(bden) / sizeof(float)); ++j) {
        if constexpr (decltype(sym)::value) bden[j] = bnd[j] * den;
        else bden[j] = *static_cast<const volatile float*>(src + j) * den;
      }
    };
    // this row of a tile: batch element, head and position relative to the tile's first (rows past the box hold nothing)
    const uint32_t row_h = (uint32_t)row / a.box_s, row_s = (uint32_t)row - row_h * a.box_s;
    const uint32_t row_b = row_h / a.box_h, row_hh = row_h - row_b * a.box_h;
    auto live_row = [&](uint32_t b0, uint32_t h0, uint32_t s0) {
      return row_b < a.box_b && b0 + row_b < a.B && h0 + row_hh < a.H && s0 + row_s < a.S;
    };
    auto out_row = [&](uint32_t b0, uint32_t h0, uint32_t s0) {
      return ((int64_t)(b0 + row_b) * a.H + h0 + row_hh) * a.out_stride + a.out_offset + s0 + row_s;
    };
    // where this row is in the input (fp16 repair), as one address per lane
    auto row_address = [&](bool key, uint32_t b0, uint32_t h0, uint32_t s0) {
      const int64_t* st = key ? a.k_stride : a.v_stride;
      return reinterpret_cast<unsigned long long>(static_cast<const __half*>(key ? a.k : a.v) + (int64_t)(b0 + row_b) * st[0] +
                                                  (int64_t)(h0 + row_hh) * st[1] + (int64_t)(s0 + row_s) * st[2]);
    };
    // Distance of a rotated coordinate to the nearest of the scaled boundaries (codebooks of 8 and more levels by symmetry,
    // as in index_of).
    auto distance = [](auto nb, const float (&bden)[decltype(nb)::value], float y) {
      constexpr int NB = decltype(nb)::value, h = (NB + 1) / 2;
      float near = NB < 7 ? fabsf(bden[0] - y) : fabsf(y);
      if constexpr (NB < 7) {
#pragma unroll
        for (int j = 1; j < NB; ++j) near = fminf(near, fabsf(bden[j] - y));
      } else {
#pragma unroll
        for (int j = h; j < NB; ++j) near = fminf(near, fabsf(bden[j] - fabsf(y)));
      }
      return near;
    };
    // Rotated coordinates of this warp's 32 rows x 32 coordinates in tensor memory at `col`: the open ones (a mask per
    // lane) are moved to the side of their boundary that the fp32 kernel finds them on.
    auto settle = [&](auto nb, uint32_t open, const float* Pi, const float* bnd, float den, uint32_t col, unsigned long long addr) {
      constexpr int NB = decltype(nb)::value;
      const float mine = lane < NB ? __ldg(bnd + lane) : INFINITY;  // a boundary per lane
      uint32_t lanes;
      while ((lanes = __ballot_sync(0xffffffffu, open != 0u)) != 0u) {
        const int l = __ffs((int)lanes) - 1;
        const int e = __ffs((int)__shfl_sync(0xffffffffu, open, l)) - 1;
        const float exact = exact_coordinate<D>(reinterpret_cast<const __half*>(__shfl_sync(0xffffffffu, addr, l)),
                                                Pi + (32 * part + e) * D);
        float y = tc::tmem_ld1(col + e);
        // the boundary nearest lane l's coordinate
        const float den_l = __shfl_sync(0xffffffffu, den, l);
        const uint32_t d = __float_as_uint(fabsf(mine * den_l - __shfl_sync(0xffffffffu, y, l)));  // (ordered as the floats are)
        const uint32_t nearest = __ballot_sync(0xffffffffu, d == __reduce_min_sync(0xffffffffu, d));
        const float b = __shfl_sync(0xffffffffu, mine, __ffs((int)nearest) - 1), at = b * den_l;
        if (lane == l) {
          open &= open - 1u;
          // the neighbour of the scaled boundary on that side
          const float step = fmaxf(fabsf(at) * 2.4e-7f, 1e-30f);
          y = exact > b ? at + step : at - step;
        }
        tc::tmem_st1(col + e, y);
      }
    };
    // size of a residual's coordinates, in units of the vector's norm: of a rotated coordinate or of a centroid
    float r_size = F16 ? kPi16Scale : SK16 ? kPi16Scale * __ldg(scales + 2) : 1.f;
    if constexpr (SK16) {
#pragma unroll
      for (int j = 0; j < (1 << KB); ++j) r_size = fmaxf(r_size, yscale_k * fabsf(cen_s[j]));
    }
    float band_p = 0.f;  // of the previous key tile's projections
    int n_xch = 0;    // exchanges through `exch` so far in this quarter (phase of xch / xfree)
    // sum of the four parts' values of this row, in a fixed order; every part gets the same total
    auto exchange = [&](float mine, float& total_out) -> bool {
      // the buffer must have been read out by everyone since the previous exchange
      if (n_xch >= 1 && !tc::mbar_wait_or_abort(xfree(q), (n_xch - 1) & 1, abort_flag)) return false;
      exch[part][row] = mine;
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(xch(q));
      if (!tc::mbar_wait_or_abort(xch(q), n_xch & 1, abort_flag)) return false;
      total_out = exch[0][row] + exch[1][row];
      if constexpr (kParts == 4) total_out = (total_out + exch[2][row]) + exch[3][row];
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(xfree(q));
      ++n_xch;
      return true;
    };
    for (int i = 0; i <= n && ok; ++i) {
      float band_next = 0.f;
      if (i < n) {
        const int s = i % kSlots, u = i / kSlots;
        bool is_key;
        uint32_t b0, h0, s0;
        unit_of(i, is_key, b0, h0, s0);
        const bool live = live_row(b0, h0, s0);
        const int64_t no = out_row(b0, h0, s0);
        // ---- norm of the row: this thread's 64 bytes of the tile as it landed (128-byte swizzle) ----
        if (!(ok = tc::mbar_wait_or_abort(x_full(s), u & 1, abort_flag))) break;
        float ss = 0.f;
        {
          const uint8_t* xrow = smem + kOffX + s * kTileBytes + (part / 2) * L::kBoxBytes + row * 128;
#pragma unroll
          for (int cc = 0; cc < 4; ++cc) {
            const int chunk = 4 * (part % 2) + cc;  // 16-byte chunk of the row's half
            const uint4 v = *reinterpret_cast<const uint4*>(xrow + ((chunk ^ (row & 7)) << 4));
            const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              float lo, hi;
              if constexpr (F16) {
                const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[e]));
                lo = f.x;
                hi = f.y;
              } else {
                lo = __uint_as_float(w[e] << 16);
                hi = __uint_as_float(w[e] & 0xffff0000u);
              }
              ss = fmaf(lo, lo, ss);
              ss = fmaf(hi, hi, ss);
            }
          }
        }
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(x_read(s));
        float ss_tot;
        if (!(ok = exchange(ss, ss_tot))) break;
        const float nv = sqrtf(ss_tot), den1 = nv + 1e-8f, den = (is_key ? yscale_k : yscale_v) * den1;
        if (!(ok = tc::mbar_wait_or_abort(y_done(s), u & 1, abort_flag))) break;
        tc::fence_after_sync();
        uint32_t raw[32];
        const uint32_t col_y = tmem + kColYP + s * kD + lane_base + 32 * part;
        tc::tmem_ld32(col_y, raw);
        tc::wait_ld();
        if constexpr (F16) {
          // any coordinate too close to a boundary to call?
          const bool sure = !live || !(ss_tot > 0.f) || !(den < 1e30f);
          const float band = sure ? 0.f : kOpenIndex * kPi16Scale * den1;  // (the scaled rotation's rows have norm 128)
          auto settle_side = [&](auto nb, bool sym, const float* Pi, const float* src, const float (&bnd)[decltype(nb)::value]) {
            constexpr int NB = decltype(nb)::value;
            uint32_t open = 0;
            if (NB < 7 || sym) {
              float bden[NB], near = INFINITY;
#pragma unroll
              for (int j = 0; j < NB; ++j) bden[j] = bnd[j] * den;
#pragma unroll
              for (int e = 0; e < 32; ++e) near = fminf(near, distance(nb, bden, __uint_as_float(raw[e])));
              if (!__any_sync(0xffffffffu, near < band)) return;
#pragma unroll
              for (int e = 0; e < 32; ++e) open |= distance(nb, bden, __uint_as_float(raw[e])) < band ? 1u << e : 0u;
            } else {
              open = open_any<NB>(col_y, src, den, band);
              if (!__any_sync(0xffffffffu, open != 0u)) return;
            }
            settle(nb, open, Pi, src, den, col_y, row_address(is_key, b0, h0, s0));
            tc::tmem_ld32(col_y, raw);
            tc::wait_ld();
          };
          if (is_key)
            settle_side(std::integral_constant<int, (1 << KB) - 1>{}, sym_k, reinterpret_cast<const float*>(a.consts + a.L.pi_k),
                        reinterpret_cast<const float*>(a.consts + a.L.bnd_k), bnd_k);
          else
            settle_side(std::integral_constant<int, (1 << VB) - 1>{}, sym_v, reinterpret_cast<const float*>(a.consts + a.L.pi_v),
                        reinterpret_cast<const float*>(a.consts + a.L.bnd_v), bnd_v);
        }
        if (is_key) {
          // y = y_raw / den is compared with the boundaries as y_raw > b * den (den > 0)
          float rr = 0.f;
          uint32_t packed[KB], rh[16], rl[16];
#pragma unroll
          for (int j = 0; j < KB; ++j) packed[j] = 0;
          const float neg_nv = -yscale_k * nv;
          // brings the residual's coordinates to at most about 64: a power of two
          const float r_scale = __uint_as_float((uint32_t)max(127 + 6 + 127 - (int)(__float_as_uint(r_size * den1) >> 23), 1) << 23);
          auto index_pass = [&](auto sym, auto given) {
            constexpr bool GIVEN = decltype(given)::value;  // the indices are in `packed` already
            float bden[(1 << KB) - 1];
            scaled(sym, reinterpret_cast<const float*>(a.consts + a.L.bnd_k), bnd_k, den, bden);
            static_for<0, 16>([&](auto pc) {
              constexpr int pr = decltype(pc)::value;  // coordinates 2 pr, 2 pr + 1 of this thread's 32
              float res[2];
  #pragma unroll
              for (int h = 0; h < 2; ++h) {
                const float yr = __uint_as_float(raw[2 * pr + h]);
                uint32_t idx;
                if constexpr (GIVEN) {
                  idx = h == 0 ? get_field<KB, 2 * pr>(packed) : get_field<KB, 2 * pr + 1>(packed);
                } else {
                  idx = index_of<(1 << KB) - 1, decltype(sym)::value>(yr, bden);
                  if (h == 0) put_field<KB, 2 * pr>(packed, idx);
                  else put_field<KB, 2 * pr + 1>(packed, idx);
                }
                res[h] = fmaf(neg_nv, cen_s[idx], yr);   // residual in rotated coordinates
                rr = fmaf(res[h], res[h], rr);
              }
              // split into bf16 hi (truncated: the upper halves of the two words, one byte permute) and lo = the
              // exact remainder, rounded; hi + lo carries ~16 mantissa bits
              if constexpr (SK16) {
                const float r0 = res[0] * r_scale, r1 = res[1] * r_scale;
                rh[pr] = tc::pack_f16x2(r0, r1);
                const float2 h = __half22float2(*reinterpret_cast<const __half2*>(&rh[pr]));
                rl[pr] = tc::pack_f16x2(r0 - h.x, r1 - h.y);
              } else {
                const uint32_t w0 = __float_as_uint(res[0]), w1 = __float_as_uint(res[1]);
                rh[pr] = __byte_perm(w0, w1, 0x7632);
                rl[pr] = tc::pack_bf16x2(res[0] - __uint_as_float(w0 & 0xffff0000u), res[1] - __uint_as_float(w1 & 0xffff0000u));
              }
            });
          };
          if (KB < 3 || sym_k) {
            index_pass(std::true_type{}, std::false_type{});
          } else if constexpr (KB >= 3 && F16) {
            uint32_t given[KB];
            index_any<KB>(col_y, reinterpret_cast<const float*>(a.consts + a.L.bnd_k), den, given);
#pragma unroll
            for (int j = 0; j < KB; ++j) packed[j] = given[j];
            index_pass(std::true_type{}, std::true_type{});
          } else if constexpr (KB >= 3) {
            index_pass(std::false_type{}, std::false_type{});
          }
          if (live) {
            uint32_t* dst = reinterpret_cast<uint32_t*>(a.key_idx + no * (kD * KB / 8) + 4 * KB * part);
            if constexpr (KB == 2) *reinterpret_cast<uint2*>(dst) = make_uint2(packed[0], packed[1]);
            else {
#pragma unroll
              for (int j = 0; j < KB; ++j) dst[j] = packed[j];
            }
            if (part == 0) a.key_vn[no] = fp16_bits(nv);
          }
          float rr_tot;
          if (!(ok = exchange(rr, rr_tot))) break;
          if (live && part == 0) a.key_rn[no] = fp16_bits(sqrtf(rr_tot) * (F16 ? __ldg(scales + 2) : 1.f));
          const float next_band = F16 && live && den < 1e30f ? kOpenSign * sqrtf(rr_tot) * r_scale : 0.f;
          // the residual operand of the previous key tile must have been consumed by its sketch MMAs
          if (i >= 1 && !(ok = tc::mbar_wait_or_abort(p_done((i - 1) % kSlots), ((i - 1) / kSlots) & 1, abort_flag))) break;
          tc::tmem_st16(tmem + kColRH + lane_base + 16 * part, rh);
          tc::tmem_st16(tmem + kColRL + lane_base + 16 * part, rl);
          tc::wait_st();
          tc::fence_before_sync();
          __syncwarp();
          if (lane == 0) tc::mbar_arrive(r_full);
          band_next = next_band;
        } else {
          uint32_t given[VB];
          if constexpr (VB >= 3 && F16)
            if (!sym_v) index_any<VB>(col_y, reinterpret_cast<const float*>(a.consts + a.L.bnd_v), den, given);
          tc::fence_before_sync();
          __syncwarp();
          if (lane == 0) tc::mbar_arrive(yp_free(s));  // the accumulator slot is in registers now
          uint32_t packed[VB];
#pragma unroll
          for (int j = 0; j < VB; ++j) packed[j] = 0;
          auto index_pass = [&](auto sym) {
            float bden[(1 << VB) - 1];
            scaled(sym, reinterpret_cast<const float*>(a.consts + a.L.bnd_v), bnd_v, den, bden);
            static_for<0, 32>([&](auto ec) {
              constexpr int e = decltype(ec)::value;
              put_field<VB, e>(packed, index_of<(1 << VB) - 1, decltype(sym)::value>(__uint_as_float(raw[e]), bden));
            });
          };
          if (VB < 3 || sym_v) {
            index_pass(std::true_type{});
          } else if constexpr (VB >= 3 && F16) {
#pragma unroll
            for (int j = 0; j < VB; ++j) packed[j] = given[j];
          } else if constexpr (VB >= 3) {
            index_pass(std::false_type{});
          }
          if (live) {
            uint32_t* dst = reinterpret_cast<uint32_t*>(a.val_idx + no * (kD * VB / 8) + 4 * VB * part);
            if constexpr (VB == 4) *reinterpret_cast<uint4*>(dst) = make_uint4(packed[0], packed[1], packed[2], packed[3]);
            else if constexpr (VB == 2) *reinterpret_cast<uint2*>(dst) = make_uint2(packed[0], packed[1]);
            else {
#pragma unroll
              for (int j = 0; j < VB; ++j) dst[j] = packed[j];
            }
            if (part == 0) a.val_vn[no] = fp16_bits(nv);
          }
        }
      }
      // ---- sign pass of the key tile before: its sketch MMA ran under the index pass above ----
      if (i >= 1 && i - 1 < nk) {
        const int s1 = (i - 1) % kSlots;
        bool is_key;
        uint32_t b0, h0, s0;
        unit_of(i - 1, is_key, b0, h0, s0);
        if (!(ok = tc::mbar_wait_or_abort(p_done(s1), ((i - 1) / kSlots) & 1, abort_flag))) break;
        tc::fence_after_sync();
        uint32_t raw[32];
        const uint32_t col_p = tmem + kColYP + s1 * kD + lane_base + 32 * part;
        tc::tmem_ld32(col_p, raw);
        tc::wait_ld();
        if constexpr (F16) {
          float near = INFINITY;
#pragma unroll
          for (int e = 0; e < 32; ++e) near = fminf(near, fabsf(__uint_as_float(raw[e])));
          if (__any_sync(0xffffffffu, near < band_p)) {
            const unsigned long long addr = row_address(true, b0, h0, s0);
            uint32_t open = 0, lanes;
#pragma unroll
            for (int e = 0; e < 32; ++e) open |= fabsf(__uint_as_float(raw[e])) < band_p ? 1u << e : 0u;
            while ((lanes = __ballot_sync(0xffffffffu, open != 0u)) != 0u) {
              const int l = __ffs((int)lanes) - 1;
              const int e = __ffs((int)__shfl_sync(0xffffffffu, open, l)) - 1;
              const float exact = exact_projection<D, (1 << KB) - 1>(
                  reinterpret_cast<const __half*>(__shfl_sync(0xffffffffu, addr, l)),
                  reinterpret_cast<const float*>(a.consts + a.L.pi_k), reinterpret_cast<const float*>(a.consts + a.L.s_eff),
                  reinterpret_cast<const float*>(a.consts + a.L.bnd_k), reinterpret_cast<const float*>(a.consts + a.L.cen_k),
                  32 * part + e);
              float p = tc::tmem_ld1(col_p + e);
              if (lane == l) {
                open &= open - 1u;
                p = exact >= 0.f ? 1.f : -1.f;
              }
              tc::tmem_st1(col_p + e, p);
            }
            tc::tmem_ld32(col_p, raw);
            tc::wait_ld();
          }
        }
        tc::fence_before_sync();
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(yp_free(s1));
        // bit e = (projection >= 0) = complement of its sign bit (a projection is never -0: sums of products that
        // start from +0); the sign bits are gathered with one mask and one mad.hi each
        uint32_t neg = 0;
#pragma unroll
        for (int e = 0; e < 32; ++e) {
          const uint32_t sb = raw[e] & 0x80000000u;
          neg = (e == 31 ? sb : __umulhi(sb, 2u << e)) + neg;
        }
        if (live_row(b0, h0, s0))
          *reinterpret_cast<uint32_t*>(a.key_sgn + out_row(b0, h0, s0) * (kD / 8) + 4 * part) = ~neg;
      }
      band_p = band_next;
    }
  }
  if (!ok && atomicExch(s_abort_p, 2) != 2) {  // one fault per CTA
    atomicAdd(&g_compress_kv_faults, 1ull);
    notify_host_of_fault(g_fault_mailbox_compress_kv);
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == kEpiWarps) tc::tmem_dealloc(tmem, L::kCols);
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// The driver's tensor-map encoder, looked up through the runtime (the library does not link against libcuda).
EncodeTiledFn encode_tiled() {
  static EncodeTiledFn fn = nullptr;
  if (fn == nullptr) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qres) == cudaSuccess &&
        qres == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(p);
    else
      cudaGetLastError();
  }
  return fn;
}

// Tensor map over a 16-bit [B, H, S, d] view with element strides (sb, sh, ss): box = 64 columns x the positions, heads
// and batch elements of a tile, 128-byte swizzle, zero fill past the ends.
int make_map(CUtensorMap* map, const void* base, bool f16, int d, const KvArgs& a, const int64_t* st) {
  EncodeTiledFn enc = encode_tiled();
  if (enc == nullptr) return fail(TQ_ERR_CUDA, "cuTensorMapEncodeTiled is not available from this driver");
  const cuuint64_t dims[4] = {(cuuint64_t)d, a.S, a.H, a.B};
  // a dimension of extent 1 may carry any stride; the encoder still wants a multiple of 16 bytes
  const cuuint64_t strides[3] = {(cuuint64_t)(a.S > 1 ? st[2] : d) * 2, (cuuint64_t)(a.H > 1 ? st[1] : d) * 2,
                                 (cuuint64_t)(a.B > 1 ? st[0] : d) * 2};
  const cuuint32_t box[4] = {64, a.box_s, a.box_h, a.box_b}, estr[4] = {1, 1, 1, 1};
  const CUresult r = enc(map, f16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4,
                         const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                         CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(TQ_ERR_UNSUPPORTED, "tensor map for strides (%lld, %lld, %lld) refused (CUresult %d)",
                                     (long long)st[0], (long long)st[1], (long long)st[2], (int)r);
  return TQ_OK;
}

template <int D, int BITS, bool F16>
int launch_kv(const CUtensorMap& map_k, const CUtensorMap& map_v, const KvArgs& a, cudaStream_t stream) {
  auto kern = compress_kv_kernel<D, BITS, F16>;
  constexpr uint32_t smem = KvShape<D>::kSmemBytes;
  TQ_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const int64_t total = (int64_t)a.units_k + a.units_v;
  int grid = sm_count() * KvShape<D>::kCtasPerSm;
  if (grid > total) grid = (int)total;
  {
    ProfScope prof(a.units_k != 0 ? kProfCompressKeys : kProfCompressValues, stream);
    kern<<<grid, KvShape<D>::kThreads, smem, stream>>>(map_k, map_v, a);
  }
  TQ_CUDA_OK(cudaGetLastError());
  return TQ_OK;
}
template <int D, bool F16>
int launch_bits(int bits, const CUtensorMap& map_k, const CUtensorMap& map_v, const KvArgs& a, cudaStream_t stream) {
  return bits == 2 ? launch_kv<D, 2, F16>(map_k, map_v, a, stream)
         : bits == 3 ? launch_kv<D, 3, F16>(map_k, map_v, a, stream) : launch_kv<D, 4, F16>(map_k, map_v, a, stream);
}

}  // namespace

bool compress_kv_applies(int dtype, int d, int mode) {
  return (dtype == TQ_BF16 || dtype == TQ_F16) && (d == 128 || d == 64) && mode == TQ_MODE_BF16;
}

int compress_kv(const void* k, const void* v, int dtype, int d, int64_t B, int64_t H, int64_t S, const int64_t* k_strides,
                const int64_t* v_strides, const uint8_t* consts, int bits, uint8_t* key_idx, uint8_t* key_sgn,
                uint16_t* key_vn, uint16_t* key_rn, uint8_t* val_idx, uint16_t* val_vn, int64_t out_stride,
                int64_t out_offset, cudaStream_t stream) {
  const bool f16 = dtype == TQ_F16;
  TQ_REQUIRE(S < ((int64_t)1 << 31) && H < ((int64_t)1 << 31) && B < ((int64_t)1 << 31), "problem too large");
  // A tile is up to 128 vectors of one head, or whole short sequences of several heads and batch elements (a generation
  // step of 16 x 32 heads: 24 us with a tile per head).
  const int64_t bs = S < 128 ? S : 128, bh = H < 128 / bs ? H : 128 / bs, bb = B < 128 / (bs * bh) ? B : 128 / (bs * bh);
  const int64_t tiles_s = (S + bs - 1) / bs, tiles_h = (H + bh - 1) / bh, tiles_b = (B + bb - 1) / bb;
  const int64_t units = tiles_s * tiles_h * tiles_b;
  TQ_REQUIRE(tiles_s * tiles_h < ((int64_t)1 << 31) && 2 * units < ((int64_t)1 << 31), "problem too large");
  const KvArgs a{(uint32_t)(k != nullptr ? units : 0), (uint32_t)(v != nullptr ? units : 0), (uint32_t)tiles_s,
                 (uint32_t)tiles_h, (uint32_t)bs, (uint32_t)bh, (uint32_t)bb, (uint32_t)S, (uint32_t)H, (uint32_t)B, consts,
                 key_idx, key_sgn, key_vn, key_rn, val_idx, val_vn, k, v, {k_strides[0], k_strides[1], k_strides[2]},
                 {v_strides[0], v_strides[1], v_strides[2]}, out_stride, out_offset, const_layout(d)};
  CUtensorMap map_k, map_v;
  if (int st = make_map(&map_k, k != nullptr ? k : v, f16, d, a, k != nullptr ? k_strides : v_strides)) return st;
  if (int st = make_map(&map_v, v != nullptr ? v : k, f16, d, a, v != nullptr ? v_strides : k_strides)) return st;
  if (d == 64) return f16 ? launch_bits<64, true>(bits, map_k, map_v, a, stream) : launch_bits<64, false>(bits, map_k, map_v, a, stream);
  return f16 ? launch_bits<128, true>(bits, map_k, map_v, a, stream) : launch_bits<128, false>(bits, map_k, map_v, a, stream);
}

}  // namespace tq
