// fp32 attention of few query rows per KV head (generation steps in fp32 mode), split over the keys.
//
// The tile kernel of tq_attention_simt.cu gives every (batch, query head) one CTA that decodes 64 keys at a time for 64
// query rows: with one query row 63 of them are not there, and the keys are walked by one CTA.  A generation
// step of 32 / 8 heads over 2000 keys took 633 us that way and takes 96 us, 16 / 2 heads over 16000 keys 3934 and 109 us.
// Here the keys of a (batch, KV head) are split over CTAs and nothing is staged:
//   * four lanes share a key, a warp works on eight; each lane decodes a quarter of the key's coordinates and signs from the
//     packed words in its registers (the next eight keys' words are loaded meanwhile) and multiplies them by up to four
//     query rows in shared memory; two shuffles complete the scores;
//   * a group of four lanes keeps its own running maximum, row sum and a quarter of the output row for the keys it sees,
//     so the value half needs no exchange at all; lane groups, warps and splits are merged at the end (the splits and the
//     back-rotation by the finishing kernel of the split-KV path).
// fp32 throughout; bound by instruction issue (about 36 + 9 R warp instructions per key for R query rows), as the 16-bit
// split-KV kernel is.
#include <math.h>

#include "tq_attention.cuh"
#include "tq_common.cuh"
#include "tq_simt.cuh"

namespace tq {
namespace {

constexpr int kWarps = 4;
constexpr int kStepKeys = 8 * kWarps;  // keys per CTA and iteration

struct RowsArgs {
  AttnArgs a;
  float* part_o;   // [B*Hkv][nsplit][rows][D]
  float* part_ml;  // [B*Hkv][nsplit][rows][2]: running maximum (log2 units), row sum
  int nsplit, keys_per_split, rows, chunks;
};

// N bits at a 2-byte (N % 32 != 0) or 4-byte aligned address as little-endian words
template <int N>
__device__ __forceinline__ void load_bits(const uint8_t* p, uint32_t (&w)[(N + 31) / 32]) {
  if constexpr (N % 32 == 0) {
#pragma unroll
    for (int i = 0; i < N / 32; ++i) w[i] = __ldg(reinterpret_cast<const uint32_t*>(p) + i);
  } else {
#pragma unroll
    for (int i = 0; i < (N + 31) / 32; ++i) {
      w[i] = __ldg(reinterpret_cast<const uint16_t*>(p) + 2 * i);
      if (2 * i + 1 < N / 16) w[i] |= (uint32_t)__ldg(reinterpret_cast<const uint16_t*>(p) + 2 * i + 1) << 16;
    }
  }
}
template <int B, int W>
__device__ __forceinline__ uint32_t field(const uint32_t (&w)[W], int e) {  // e is a constant after unrolling
  const int bit = e * B, k = bit / 32, sh = bit % 32;
  const uint32_t v = sh + B <= 32 ? w[k] >> sh : __funnelshift_r(w[k], w[k + 1 < W ? k + 1 : k], sh);
  return v & ((1u << B) - 1);
}
__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

template <int D, int BITS, int R, bool MASK>
__global__ void __launch_bounds__(kWarps * 32) attention_rows_kernel(const RowsArgs x) {
  constexpr int KB = BITS - 1, VB = BITS, PER = D / 4;  // coordinates per lane
  constexpr int QP = PER + 4;                           // pitch of a quarter row: the four quarters hit different banks
  constexpr float kLog2e = 1.4426950408889634f;
  __shared__ __align__(16) float q_s[R][2][4 * QP];
  __shared__ float cen_k[1 << KB], cen_v[1 << VB];
  __shared__ float mrg_o[kWarps][R][D];
  __shared__ float mrg_ml[kWarps][R][2];
  const AttnArgs& a = x.a;
  const int tid = threadIdx.x, warp = tid / 32, lane = tid % 32, kg = lane / 4, part = lane % 4;
  const int split = blockIdx.x, kvh = blockIdx.y / x.chunks, r0 = (blockIdx.y % x.chunks) * R;
  const int64_t b = blockIdx.z;
  const int G = (int)(a.Hq / a.Hkv), Sq = (int)a.Sq, Sk = (int)a.Sk, shift = Sk - Sq;
  const int64_t kv_base = (b * a.Hkv + kvh) * a.kv_stride;
  if (tid < (1 << KB)) cen_k[tid] = a.cen_k[tid];
  if (tid < (1 << VB)) cen_v[tid] = a.cen_v[tid];
  for (int e = tid; e < R * 2 * D; e += kWarps * 32) {
    const int r = e / (2 * D), half = e / D % 2, c = e % D, row = r0 + r;
    float v = 0.f;
    if (row < x.rows)
      v = static_cast<const float*>(a.q_cat)[((b * a.Hq + kvh * G + row / Sq) * Sq + row % Sq) * 2 * D + half * D + c];
    q_s[r][half][(c / PER) * QP + c % PER] = v;
  }
  __syncthreads();
  int last[R];  // last visible key of the row
#pragma unroll
  for (int r = 0; r < R; ++r) last[r] = a.causal && r0 + r < x.rows ? (r0 + r) % Sq + shift : Sk - 1;
  const float scale = a.sm_scale * kLog2e;
  float m[R], l[R], o[R][PER];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    m[r] = -INFINITY;
    l[r] = 0.f;
#pragma unroll
    for (int c = 0; c < PER; ++c) o[r][c] = 0.f;
  }
  const int k_lo = split * x.keys_per_split, k_hi = min(Sk, k_lo + x.keys_per_split);
  uint32_t kw[(PER * KB + 31) / 32], sw[(PER + 31) / 32], vw[(PER * VB + 31) / 32];
  uint32_t n_raw[3];
  auto fetch = [&](int k) {
    const int64_t n = kv_base + (k < k_hi ? k : k_lo);  // past the end: any key of the range, not used
    load_bits<PER * KB>(a.key_idx + n * (D * KB / 8) + part * (PER * KB / 8), kw);
    load_bits<PER>(a.key_sgn + n * (D / 8) + part * (PER / 8), sw);
    load_bits<PER * VB>(a.val_idx + n * (D * VB / 8) + part * (PER * VB / 8), vw);
    n_raw[0] = __ldg(a.key_vn + n);
    n_raw[1] = __ldg(a.key_rn + n);
    n_raw[2] = __ldg(a.val_vn + n);
  };
  int kb = k_lo + 8 * warp;  // first of this warp's eight keys
  if (kb < k_hi) fetch(kb + kg);
  for (; kb < k_hi; kb += kStepKeys) {
    const int k = kb + kg;
    float a1[R], a2[R];
#pragma unroll
    for (int r = 0; r < R; ++r) a1[r] = a2[r] = 0.f;
#pragma unroll
    for (int c4 = 0; c4 < PER; c4 += 4) {
      float v[4], sg[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        v[e] = cen_k[field<KB>(kw, c4 + e)];
        sg[e] = __uint_as_float(0xbf800000u ^ (field<1>(sw, c4 + e) << 31));  // a set bit is +1
      }
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const float4 q1 = *reinterpret_cast<const float4*>(&q_s[r][0][part * QP + c4]);
        const float4 q2 = *reinterpret_cast<const float4*>(&q_s[r][1][part * QP + c4]);
        a1[r] = fmaf(q1.x, v[0], fmaf(q1.y, v[1], fmaf(q1.z, v[2], fmaf(q1.w, v[3], a1[r]))));
        a2[r] = fmaf(q2.x, sg[0], fmaf(q2.y, sg[1], fmaf(q2.z, sg[2], fmaf(q2.w, sg[3], a2[r]))));
      }
    }
    const float n1 = fp16_value((uint16_t)n_raw[0]), n2 = fp16_value((uint16_t)n_raw[1]), nv = fp16_value((uint16_t)n_raw[2]);
    uint32_t vcur[(PER * VB + 31) / 32];
#pragma unroll
    for (int i = 0; i < (PER * VB + 31) / 32; ++i) vcur[i] = vw[i];
    if (kb + kStepKeys < k_hi) fetch(kb + kStepKeys + kg);
    float pv[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      float t = fmaf(n1, a1[r], n2 * a2[r]);
      t += __shfl_xor_sync(0xffffffffu, t, 1);
      t += __shfl_xor_sync(0xffffffffu, t, 2);
      t *= scale;
      if constexpr (MASK) {
        const int row = r0 + r;
        if (row < x.rows && k < k_hi) {
          if (a.mask != nullptr) {
            // kept finite (a row whose keys are all masked with the most negative float averages them), but for -inf
            const float v = __ldg(a.mask + b * a.mask_stride_b + (int64_t)(row % Sq) * a.mask_stride_q + k);
            t += v == -INFINITY ? v : fmaxf(v * kLog2e, -3.0e38f);
          } else {
            const uint32_t w = a.mb.words[((a.mb.batch ? b * a.Sq : 0) + row % Sq) * (4 * (int64_t)a.mb.T) + k / 32];
            if (((w >> (k & 31)) & 1u) == 0u) t = -3.0e38f;
          }
        }
      }
      if (k >= k_hi || k > last[r]) t = -INFINITY;
      if (__any_sync(0xffffffffu, t > m[r])) {  // some lane group's maximum grows: O and l follow
        const float m_new = fmaxf(m[r], t), alpha = m[r] == -INFINITY ? 0.f : ex2(m[r] - m_new);
        m[r] = m_new;
        l[r] *= alpha;
#pragma unroll
        for (int c = 0; c < PER; ++c) o[r][c] *= alpha;
      }
      const float p = t == -INFINITY ? 0.f : ex2(t - m[r]);
      l[r] += p;
      pv[r] = p * nv;
    }
#pragma unroll
    for (int c = 0; c < PER; ++c) {
      const float v = cen_v[field<VB>(vcur, c)];
#pragma unroll
      for (int r = 0; r < R; ++r) o[r][c] = fmaf(pv[r], v, o[r][c]);
    }
  }
  // merge the eight lane groups, then the warps
#pragma unroll
  for (int r = 0; r < R; ++r) {
    float mx = m[r];
#pragma unroll
    for (int d = 4; d < 32; d <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, d));
    const float f = m[r] == -INFINITY ? 0.f : ex2(m[r] - mx);
    float lt = l[r] * f;
#pragma unroll
    for (int d = 4; d < 32; d <<= 1) lt += __shfl_xor_sync(0xffffffffu, lt, d);
#pragma unroll
    for (int c = 0; c < PER; ++c) {
      float v = o[r][c] * f;
#pragma unroll
      for (int d = 4; d < 32; d <<= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
      if (kg == 0) mrg_o[warp][r][part * PER + c] = v;
    }
    if (lane == 0) {
      mrg_ml[warp][r][0] = mx;
      mrg_ml[warp][r][1] = lt;
    }
  }
  __syncthreads();
  const int64_t unit = (b * a.Hkv + kvh) * x.nsplit + split;
  for (int e = tid; e < R * D; e += kWarps * 32) {
    const int r = e / D, c = e % D;
    if (r0 + r >= x.rows) break;
    float mx = -INFINITY;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) mx = fmaxf(mx, mrg_ml[w][r][0]);
    float acc = 0.f, lt = 0.f;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
      const float f = mrg_ml[w][r][0] == -INFINITY ? 0.f : ex2(mrg_ml[w][r][0] - mx);
      acc = fmaf(mrg_o[w][r][c], f, acc);
      lt = fmaf(mrg_ml[w][r][1], f, lt);
    }
    x.part_o[(unit * x.rows + r0 + r) * D + c] = acc;
    if (c == 0) {
      x.part_ml[(unit * x.rows + r0 + r) * 2] = mx;
      x.part_ml[(unit * x.rows + r0 + r) * 2 + 1] = lt;
    }
  }
}

template <int D, int BITS, int R>
int launch_rows(const RowsArgs& x, int64_t B, cudaStream_t stream) {
  const bool masked = x.a.mask != nullptr || x.a.mb.words != nullptr;
  auto kern = masked ? attention_rows_kernel<D, BITS, R, true> : attention_rows_kernel<D, BITS, R, false>;
  ProfScope prof(kProfAttention, stream);
  kern<<<dim3((unsigned)x.nsplit, (unsigned)(x.a.Hkv * x.chunks), (unsigned)B), kWarps * 32, 0, stream>>>(x);
  TQ_CUDA_OK(cudaGetLastError());
  return TQ_OK;
}
template <int D, int BITS>
int launch_r(int r, const RowsArgs& x, int64_t B, cudaStream_t stream) {
  return r == 1 ? launch_rows<D, BITS, 1>(x, B, stream) : r == 2 ? launch_rows<D, BITS, 2>(x, B, stream) : launch_rows<D, BITS, 4>(x, B, stream);
}
template <int D>
int launch_bits(int bits, int r, const RowsArgs& x, int64_t B, cudaStream_t stream) {
  return bits == 2 ? launch_r<D, 2>(r, x, B, stream) : bits == 3 ? launch_r<D, 3>(r, x, B, stream) : launch_r<D, 4>(r, x, B, stream);
}

// Query rows per CTA, CTAs' row chunks and splits of a call.
struct RowsPlan {
  int rows, r, chunks, nsplit, per;
};
RowsPlan rows_plan(int64_t B, int64_t Hq, int64_t Sq, int64_t Hkv, int64_t Sk) {
  RowsPlan p{};
  p.rows = (int)(Hq / Hkv * Sq);
  p.r = p.rows == 1 ? 1 : p.rows == 2 ? 2 : 4;
  p.chunks = (p.rows + p.r - 1) / p.r;
  // one wave of CTAs (the output rows fill the registers: four CTAs per SM for one row, two for four), of at least 64 keys
  const int64_t ctas = (int64_t)sm_count() * (p.r == 1 ? 4 : p.r == 2 ? 3 : 2), units = B * Hkv * p.chunks;
  int64_t n = (ctas + units - 1) / units;
  const int64_t most = (Sk + 63) / 64;
  n = n < most ? n : most;
  n = n < 512 ? n : 512;  // the finishing kernel's table of splits
  p.per = (int)(((Sk + n - 1) / n + kStepKeys - 1) / kStepKeys * kStepKeys);
  p.nsplit = (int)((Sk + p.per - 1) / p.per);
  return p;
}

}  // namespace

// Behind many query heads that fill the chip, short key ranges are left to the tile kernel: the finishing kernel reads Pi_v
// once for every query row, the tile kernel rotates 64 rows back at a time.  Costs in us on 148 SMs, measured at head_dim
// 128 / 64: this path 15 + 0.0215 / 0.008 per query row + 1.75e-4 / 1.1e-4 per key and chunk of rows, the tile kernel
// 30 / 25 + 0.1 / 0.05 per query head and for each of its tiles of 64 keys.  32 x 32 heads of 16 rows, 64 keys: 370 us here
// and 234 there; 500 keys: 697 and 957; 8 rows, 64 keys: 198 and 234.
bool attention_rows_applies(int64_t B, int64_t Hq, int64_t Sq, int64_t Hkv, int64_t Sk, int d) {
  if (Hkv <= 0 || Hq / Hkv * Sq > 16) return false;
  if (B * Hq < sm_count()) return true;
  const RowsPlan p = rows_plan(B, Hq, Sq, Hkv, Sk);
  const bool wide = d == 128;
  const double heads = (double)(B * Hq), chunk_keys = (double)(B * Hkv * p.chunks) * (double)Sk;
  const double here = 15.0 + heads * (double)Sq * (wide ? 0.0215 : 0.008) + chunk_keys * (wide ? 1.75e-4 : 1.1e-4);
  const double there = (wide ? 30.0 : 25.0) + heads * (double)((Sk + 63) / 64 + 1) * (wide ? 0.1 : 0.05);
  return here <= there;
}

size_t attention_rows_workspace(int64_t B, int64_t Hq, int64_t Sq, int64_t Hkv, int64_t Sk, int d) {
  const RowsPlan p = rows_plan(B, Hq, Sq, Hkv, Sk);
  return ((size_t)B * Hkv * p.nsplit * p.rows * (d + 2) * sizeof(float) + 255) & ~(size_t)255;
}

int attention_rows(const AttnArgs& a, int64_t B, int d, int bits, void* part_ws, cudaStream_t stream) {
  const RowsPlan p = rows_plan(B, a.Hq, a.Sq, a.Hkv, a.Sk);
  TQ_REQUIRE(B <= 65535 && a.Hkv * p.chunks <= 65535, "batch or head count too large for the few-rows kernel");
  float* part_o = static_cast<float*>(part_ws);
  float* part_ml = part_o + (size_t)B * a.Hkv * p.nsplit * p.rows * d;
  const RowsArgs x{a, part_o, part_ml, p.nsplit, p.per, p.rows, p.chunks};
  if (int st = d == 128 ? launch_bits<128>(bits, p.r, x, B, stream) : launch_bits<64>(bits, p.r, x, B, stream)) return st;
  return finish_splits(a, B, d, p.rows, p.nsplit, part_o, part_ml, stream);
}

}  // namespace tq
