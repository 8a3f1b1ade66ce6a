// Rotary position embedding of the query and key heads of one attention layer in ONE launch.
//
// The reference's adapters call HF's apply_rotary_pos_emb before they compress the keys
// (src/transformers_turboquant/families/llama.py:98, qwen2.py:98): q*cos + rotate_half(q)*sin as four
// elementwise torch kernels and a concatenation per tensor, i.e. about ten passes over q and k.  This
// kernel reads every element once and writes it once, in the [B, H, S, D] layout the compression and
// attention kernels like best, and reproduces torch's arithmetic to the bit: every product and the sum
// are rounded to the tensor dtype, as the separate torch kernels round them.
//
// HBM-bound: 2 x (B (Hq + Hkv) S D) elements in + out, plus the cos/sin rows (shared by all heads: L2).
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <string.h>

#include "tq_common.cuh"

namespace tq {
namespace {

struct RopeArgs {
  const void *q, *k, *cos, *sin;
  void *q_out, *k_out;
  int64_t B, Hq, Hkv, S;
  int64_t qsb, qsh, qss, ksb, ksh, kss, csb, css;  // element strides
  int d;
  FastDiv div_c, div_h, div_s;  // chunks of half a row, heads, positions
};

// Two elements (fp32: one) as a unit of arithmetic.  The packed 16-bit instructions round each product and sum once, which is
// what rounding the fp32 result does: a product of 16-bit numbers is exact in fp32, and 24 bits are enough (2 p + 2) for the
// second rounding of a sum to change nothing.  `_rn` forms: never contracted to a fused multiply-add.
template <int DTYPE>
struct Pair;
template <>
struct Pair<TQ_BF16> {
  using T = __nv_bfloat162;
  static __device__ __forceinline__ T mul(T a, T b) { return __hmul2_rn(a, b); }
  static __device__ __forceinline__ T add(T a, T b) { return __hadd2_rn(a, b); }
  static __device__ __forceinline__ T sub(T a, T b) { return __hsub2_rn(a, b); }
};
template <>
struct Pair<TQ_F16> {
  using T = __half2;
  static __device__ __forceinline__ T mul(T a, T b) { return __hmul2_rn(a, b); }
  static __device__ __forceinline__ T add(T a, T b) { return __hadd2_rn(a, b); }
  static __device__ __forceinline__ T sub(T a, T b) { return __hsub2_rn(a, b); }
};
template <>
struct Pair<TQ_F32> {
  using T = float;
  static __device__ __forceinline__ T mul(T a, T b) { return __fmul_rn(a, b); }
  static __device__ __forceinline__ T add(T a, T b) { return __fadd_rn(a, b); }
  static __device__ __forceinline__ T sub(T a, T b) { return __fsub_rn(a, b); }
};

// 16 bytes of a row.  They move as one vector: a copy of the struct is four copies of its elements, whose stores leave half-filled
// lines behind where half a row is less than a line (8 x 1024 tokens, 12 + 12 heads of 64, bf16: 18.2 us so, 8.7 as vectors;
// 4 x 4096, 32 + 8 heads of 64: 52 and 32).
template <int DTYPE>
struct Chunk {
  typename Pair<DTYPE>::T v[4];
  static __device__ __forceinline__ Chunk load(const uint8_t* p) {
    const uint4 u = *reinterpret_cast<const uint4*>(p);
    Chunk c;
    memcpy(&c, &u, 16);
    return c;
  }
  __device__ __forceinline__ void store(uint8_t* p) const {
    uint4 u;
    memcpy(&u, this, 16);
    *reinterpret_cast<uint4*>(p) = u;
  }
};

// One work item = one 16-byte chunk of the first half of a row and its partner in the second half.
// Items are numbered in the memory order of the projection output ([B, S, H, D]: consecutive threads read
// consecutive bytes); each output row is written in two 16-byte-per-thread runs.
// IDX: uint32_t when the item count fits (64-bit divisions would otherwise dominate the instruction stream).
// Eight CTAs per SM at 32 registers (8 x 4096 tokens of 32 + 8 heads of 128: 119 us, as six at 40 or four at 44; 1000 tokens: 4.1
// us, and 4.3 or 4.4).
template <int DTYPE, typename IDX>
__global__ void __launch_bounds__(256, 8) rope_kernel(const RopeArgs a) {
  using P = Pair<DTYPE>;
  using C = Chunk<DTYPE>;
  constexpr int64_t E = DTYPE == TQ_F32 ? 4 : 2;  // bytes of an element
  const int half = a.d / 2 * (int)E;  // bytes of half a row
  const IDX cpr = (IDX)a.div_c.d, H = (IDX)(a.Hq + a.Hkv), S = (IDX)a.S;
  const IDX items = (IDX)a.B * S * H * cpr;
  for (IDX it = (IDX)blockIdx.x * blockDim.x + threadIdx.x; it < items; it += (IDX)gridDim.x * blockDim.x) {
    IDX row, pos, b;
    if constexpr (sizeof(IDX) == 4) {
      row = a.div_c.div(it);
      pos = a.div_h.div(row);
      b = a.div_s.div(pos);
    } else {
      row = it / cpr;
      pos = row / H;
      b = pos / S;
    }
    const int c = (int)(it - row * cpr) * 16;
    const int64_t h = (int64_t)(row - pos * H), s = (int64_t)(pos - b * S), bb = (int64_t)b;
    const bool is_q = h < a.Hq;
    const int64_t hh = is_q ? h : h - a.Hq;
    const uint8_t* src = static_cast<const uint8_t*>(is_q ? a.q : a.k) +
                         (is_q ? bb * a.qsb + hh * a.qsh + s * a.qss : bb * a.ksb + hh * a.ksh + s * a.kss) * E + c;
    uint8_t* dst = static_cast<uint8_t*>(is_q ? a.q_out : a.k_out) + ((bb * (is_q ? a.Hq : a.Hkv) + hh) * a.S + s) * a.d * E + c;
    const int64_t at = (bb * a.csb + s * a.css) * E + c;
    const uint8_t *cs = static_cast<const uint8_t*>(a.cos) + at, *sn = static_cast<const uint8_t*>(a.sin) + at;
    const C xlo = C::load(src), xhi = C::load(src + half);
    const C clo = C::load(cs), chi = C::load(cs + half), slo = C::load(sn), shi = C::load(sn + half);
    C olo, ohi;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      // out[i] = x[i] cos[i] - x[i + d/2] sin[i];  out[i + d/2] = x[i + d/2] cos[i + d/2] + x[i] sin[i + d/2]
      olo.v[e] = P::sub(P::mul(xlo.v[e], clo.v[e]), P::mul(xhi.v[e], slo.v[e]));
      ohi.v[e] = P::add(P::mul(xhi.v[e], chi.v[e]), P::mul(xlo.v[e], shi.v[e]));
    }
    olo.store(dst);
    ohi.store(dst + half);
  }
}

inline bool aligned16p(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

}  // namespace
}  // namespace tq

using namespace tq;

extern "C" int tq_rope(const void* q, const void* k, int dtype, int64_t B, int64_t Hq, int64_t Hkv, int64_t S, int d,
                       int64_t q_stride_b, int64_t q_stride_h, int64_t q_stride_s, int64_t k_stride_b,
                       int64_t k_stride_h, int64_t k_stride_s, const void* cos, const void* sin, int64_t cs_stride_b,
                       int64_t cs_stride_s, void* q_out, void* k_out, void* stream) {
  TQ_REQUIRE(dtype == TQ_F32 || dtype == TQ_BF16 || dtype == TQ_F16, "unknown dtype %d", dtype);
  TQ_REQUIRE(B >= 0 && Hq >= 0 && Hkv >= 0 && S >= 0, "negative extent");
  TQ_REQUIRE(d > 0 && d % 32 == 0, "head_dim %d must be a positive multiple of 32", d);
  if (B == 0 || S == 0 || Hq + Hkv == 0) return TQ_OK;
  TQ_REQUIRE(cos && sin, "NULL cos / sin");
  TQ_REQUIRE((Hq == 0 || (q && q_out)) && (Hkv == 0 || (k && k_out)), "NULL pointer");
  const int n = dtype == TQ_F32 ? 4 : 8;  // elements per 16 bytes
  TQ_REQUIRE(aligned16p(q) && aligned16p(k) && aligned16p(cos) && aligned16p(sin) && aligned16p(q_out) && aligned16p(k_out),
             "all tensors must be 16-byte aligned");
  TQ_REQUIRE(q_stride_b % n == 0 && q_stride_h % n == 0 && q_stride_s % n == 0 && k_stride_b % n == 0 &&
                 k_stride_h % n == 0 && k_stride_s % n == 0 && cs_stride_b % n == 0 && cs_stride_s % n == 0,
             "strides must keep rows 16-byte aligned");
  TQ_REQUIRE(q_out != q && k_out != k, "outputs must not alias the inputs");
  const cudaStream_t s = static_cast<cudaStream_t>(stream);
  CallScope scope(Hq > 0 ? q : k, "q", s);
  if (scope.status()) return scope.status();
  const RopeArgs a{q, k, cos, sin, q_out, k_out, B, Hq, Hkv, S, q_stride_b, q_stride_h, q_stride_s,
                   k_stride_b, k_stride_h, k_stride_s, cs_stride_b, cs_stride_s, d,
                   FastDiv((uint32_t)(d / 2 / n)), FastDiv((uint32_t)(Hq + Hkv)), FastDiv((uint32_t)S)};
  const int64_t items = B * S * (Hq + Hkv) * (d / 2 / n);
  int dev = 0, sms = 148;
  TQ_CUDA_OK(cudaGetDevice(&dev));
  TQ_CUDA_OK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  const int64_t want = (items + 255) / 256, cap = (int64_t)sms * 8;  // 8 resident CTAs of 256 threads per SM
  const unsigned grid = (unsigned)(want < cap ? want : cap);
  const bool small = items + (int64_t)grid * 256 < (int64_t)0xffffffffu;  // the loop counter may overshoot once
  if (dtype == TQ_BF16) {
    if (small) rope_kernel<TQ_BF16, uint32_t><<<grid, 256, 0, s>>>(a);
    else rope_kernel<TQ_BF16, int64_t><<<grid, 256, 0, s>>>(a);
  } else if (dtype == TQ_F16) {
    if (small) rope_kernel<TQ_F16, uint32_t><<<grid, 256, 0, s>>>(a);
    else rope_kernel<TQ_F16, int64_t><<<grid, 256, 0, s>>>(a);
  } else {
    if (small) rope_kernel<TQ_F32, uint32_t><<<grid, 256, 0, s>>>(a);
    else rope_kernel<TQ_F32, int64_t><<<grid, 256, 0, s>>>(a);
  }
  TQ_CUDA_OK(cudaGetLastError());
  return TQ_OK;
}
