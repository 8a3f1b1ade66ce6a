// Argument block and entry points shared by the fp32 (CUDA-core) and bf16 (tcgen05)
// implementations of the fused compressed attention.
#pragma once
#include <cuda_bf16.h>

#include "tq_common.cuh"

namespace tq {

// Layout of the per-compressor constants buffer that tq_prepare_constants fills once: byte offsets of its parts
// (each a multiple of 256) for head_dim d.  Everything a launch needs that depends only on the compressor pair:
// the fp32 matrices and codebooks themselves, and the operand images the tensor-core kernels bulk-copy into
// shared memory (so that no call rebuilds them).
struct ConstLayout {
  size_t header;                                                  // magic, d, bits
  size_t pi_k, s_eff, pi_v, cen_k, bnd_k, cen_v, bnd_v;           // fp32 originals
  size_t w_cat_pair, w_unrot_pair, luts, w_cat_plain, w_unrot_plain;  // attention: bf16 operand images, fp16 pair tables
  size_t pik_hi, pik_lo, se_hi, se_lo, piv_hi, piv_lo;            // compression: split-bf16 K-major operand images
  size_t pik16_hi, pik16_lo, se16_hi, se16_lo, piv16_hi, piv16_lo;  // ... and split-fp16 ones, scaled by powers of two
  size_t x_key, x_val;  // expansion: fp16 images of Pi_k^T and (S_eff Pi_k)^T, of Pi_v^T, scaled by powers of two
  size_t total;
};
// The fp16 images of a rotation hold Pi x 128 (entries of about 0.1 would put the low parts into fp16's subnormals); a matrix
// whose rows do not have norm 1 is brought there by another power of two.  The scales of Pi_k and Pi_v and the inverse of
// the first are floats at word kScaleWord of the header.  Rows of the sketch, of which only signs are read, are scaled
// each to entries of about 1.
constexpr float kPi16Scale = 128.f;
constexpr int kScaleWord = 4;
// ... and, at this word, what the accumulators of the expansion are multiplied by: of indices, of signs (sqrt(pi/2)/d
// included), of values.
constexpr int kExpandScaleWord = 8;
constexpr uint32_t kConstMagic = 0x31425154u;  // "TQB1"
inline ConstLayout const_layout(int d) {
  ConstLayout L{};
  size_t off = 0;
  auto take = [&](size_t bytes) { const size_t at = off; off += (bytes + 255) & ~(size_t)255; return at; };
  const size_t m32 = (size_t)d * d * 4, m16 = (size_t)d * d * 2;
  L.header = take(256);
  L.pi_k = take(m32); L.s_eff = take(m32); L.pi_v = take(m32);
  L.cen_k = take(64); L.bnd_k = take(64); L.cen_v = take(64); L.bnd_v = take(64);
  L.w_cat_pair = take(2 * m16); L.w_unrot_pair = take(m16); L.luts = take(2048);
  L.w_cat_plain = take(2 * m16); L.w_unrot_plain = take(m16);
  L.pik_hi = take(m16); L.pik_lo = take(m16); L.se_hi = take(m16); L.se_lo = take(m16);
  L.piv_hi = take(m16); L.piv_lo = take(m16);
  L.pik16_hi = take(m16); L.pik16_lo = take(m16); L.se16_hi = take(m16); L.se16_lo = take(m16);
  L.piv16_hi = take(m16); L.piv16_lo = take(m16);
  L.x_key = take(2 * m16); L.x_val = take(m16);
  L.total = off;
  return L;
}
int prepare_constants(const float* Pi_k, const float* S_eff, const float* cen_k, const float* bnd_k, const float* Pi_v,
                      const float* cen_v, const float* bnd_v, int bits, int d, void* constants, cudaStream_t stream);

// Summary of a mask (tq_mask.cu): visibility bits, classes of 16 rows x 128 keys, rows with a visible key.
struct MaskBits {
  const uint32_t* words;  // [batch][Sq][4 T]; NULL: no summary
  const uint32_t* rows;   // [batch][NG][NC]: bit r set when row 16 g + r has a visible key in this chunk of 16 tiles
  const uint8_t* tiles;   // [batch][NG][T]: 1 some key visible, 2 some hidden, 4 some other additive value
  int T, NG, NC;          // 128-key tiles, 16-row groups, chunks of 16 tiles
  int batch;              // 0: one mask for every batch element
};
// The pointers of a summary of `nb` masks at `base` (which may be NULL to ask for the size only).
MaskBits mask_bits_layout(int64_t nb, int64_t Sq, int64_t Sk, void* base, size_t* bytes);
int summarize_mask(const void* mask, bool boolean, int64_t nb, int64_t stride_b, int64_t stride_q, int64_t Sq, int64_t Sk,
                   int causal, const MaskBits& m, cudaStream_t stream);

struct AttnArgs {
  const void* q_cat;   // fp32 [n, 2d] (fp32 mode) or bf16 [n, 2d] (bf16 mode), row n = (b*Hq+h)*Sq+s
  int64_t Hq, Sq, Hkv, Sk;
  const uint8_t* key_idx;
  const uint8_t* key_sgn;
  const uint16_t* key_vn;
  const uint16_t* key_rn;
  const uint8_t* val_idx;
  const uint16_t* val_vn;
  const float* cen_k;
  const float* cen_v;
  const float* Pi_v;
  float sm_scale;
  int causal;
  const float* mask;
  int64_t mask_stride_b, mask_stride_q;
  void* out;
  int out_dtype;
  int64_t o_stride_b, o_stride_h, o_stride_s;
  // keys between the packed rows of consecutive (batch, KV head) pairs in every packed array: Sk for the
  // contiguous [B, Hkv, Sk] layout, the capacity of a persistent cache otherwise
  int64_t kv_stride;
  MaskBits mb;  // summary of the mask; where it exists, `mask` is read in tiles of its third class only
};

int check_attention_args(const void* q, int dtype, int64_t B, int64_t Hq, int64_t Sq, int d, int64_t sb, int64_t sh,
                         int64_t ss, int64_t Hkv, int64_t Sk, int bits, int mode);

// q_cat rows [q Pi^T | coeff (q Pi^T) S_eff^T] of few query rows (fp32 arithmetic; bf16 or fp32 result), any dtype and
// strides of q; row n = (b * Hq + h) * Sq + s.  `beside_previous`: the kernel launched last (a mask's summary) has nothing
// that this one reads, they may run side by side; this one does not finish before that one has.
int qprep_rows(const void* q, int dtype, int64_t n_q, int64_t Hq, int64_t Sq, int d, int64_t sb, int64_t sh, int64_t ss,
               const float* Pi, const float* S_eff, void* q_cat, bool bf16_out, cudaStream_t stream, bool beside_previous = false);

// fp32 mode: query preparation + CUDA-core flash kernel.  `workspace` holds q_cat fp32.
int attention_fwd_fp32(const void* q, int dtype, int64_t B, int64_t Hq, int64_t Sq, int d, int64_t sb, int64_t sh,
                       int64_t ss, const float* Pi_k, const float* S_eff, AttnArgs a, int bits, void* workspace,
                       cudaStream_t stream, bool prepared = false);

// How a bf16-mode call of the SM-pair kernel's is served: keys and values expanded first, that kernel split over the keys, or
// that kernel unsplit.  The first two take scratch; this is the choice for prepared calls that have it.
enum class PairRoute { kExpand, kSplit, kWhole };
PairRoute attention_pair_route(int64_t B, int64_t Hq, int64_t Sq, int64_t Hkv, int64_t Sk, int d);

// bf16 mode: tcgen05 query preparation, tcgen05 flash kernel, tcgen05 back-rotation.
// `prepared` (optional): a constants buffer filled by prepare_constants for the same matrices; the operand images
// are then taken from it and nothing is rebuilt.
int attention_fwd_bf16(const void* q, int dtype, int64_t B, int64_t Hq, int64_t Sq, int d, int64_t sb, int64_t sh,
                       int64_t ss, const float* Pi_k, const float* S_eff, AttnArgs a, int bits, void* workspace,
                       cudaStream_t stream, const uint8_t* prepared, PairRoute route);
// Whether a bf16-mode call is the SM-pair kernel's, on one of the routes above.
bool attention_bf16_on_sm_pairs(int64_t Hq, int64_t Sq, int64_t Hkv, int64_t Sk, int64_t kv_stride, int d);
// TQ_OK where the kernel that serves a bf16-mode call can read packed rows and norms at their addresses.
int check_packed_rows_bf16(const AttnArgs& a, int64_t Sq, int d, int bits, PairRoute route);
// scratch bytes of a bf16-mode call with a prepared constants buffer, by the kernel that will serve it
size_t workspace_bytes_bf16_prepared(int64_t B, int64_t Hq, int64_t Sq, int64_t Hkv, int64_t Sk, int64_t kv_stride,
                                     int d);

size_t workspace_bytes_bf16(int64_t BHq, int64_t Sq, int d);

// Decode-sized calls (few query rows per KV head, long keys; tq_attention_decode.cu), three launches: query
// preparation into `q_cat` (bf16 [n_q, 2d]), the split-KV kernel, then merge + back-rotation into a.out.
// `part_ws` holds decode_workspace_bytes(B * Hq).
bool decode_applies(const AttnArgs& a, int d);  // a.kv_stride != a.Sk: any key count
size_t decode_workspace_bytes(int64_t BHq);
int attention_decode(const AttnArgs& a, int64_t B, int bits, const void* q, int q_dtype, int64_t sb, int64_t sh,
                     int64_t ss, const float* Pi_k, const float* S_eff, void* q_cat, void* part_ws, cudaStream_t stream);

// Merge of partial results [B * Hkv][nsplit][rows][d] (unnormalised, rotated; maxima in log2 units) and back-rotation into
// a.out; row r of a KV head is query head kvh * G + r / Sq, position r % Sq.
int finish_splits(const AttnArgs& a, int64_t B, int d, int rows, int nsplit, const float* part_o, const float* part_ml,
                  cudaStream_t stream);

// fp32 mode, at most 16 query rows per KV head (tq_attention_rows.cu): a.q_cat holds the fp32 query rows, `part_ws`
// attention_rows_workspace bytes.
bool attention_rows_applies(int64_t B, int64_t Hq, int64_t Sq, int64_t Hkv, int64_t Sk, int d);
size_t attention_rows_workspace(int64_t B, int64_t Hq, int64_t Sq, int64_t Hkv, int64_t Sk, int d);
int attention_rows(const AttnArgs& a, int64_t B, int d, int bits, void* part_ws, cudaStream_t stream);

// Raw queries and the constant bf16 operands of the SM-pair kernel, which prepares its own query tile
// (q [Pi ; coeff S]^T) and rotates its output back (o Pi_v) on the tensor pipe.
struct PairArgs {
  const void* q;
  int q_dtype;
  int64_t q_stride_b, q_stride_h, q_stride_s;
  const __nv_bfloat16* w_cat;    // [2d, d] = [Pi ; coeff S]
  const __nv_bfloat16* w_unrot;  // [d, d]  = Pi_v^T
  const uint32_t* luts;          // pair tables: 4^(bits-1) key entries, then 4^bits value entries (bf16x2 words)
  int nsplit;                    // clusters that share the keys of a pair of query tiles; 1: no partial results
  float* part_o;                 // [B*Hq][ceil(Sq / 128)][nsplit][128][d], unnormalised, rotated
  float* part_ml;                // [B*Hq][ceil(Sq / 128)][nsplit][128][2]: running maximum (log2 units), row sum
};
// Clusters per pair of query tiles that the SM-pair kernel is split over, and the partial results' bytes (0 unsplit).
int attention_c2_splits(int64_t B, int64_t Hq, int64_t Sq, int64_t Hkv, int64_t Sk);
// Keys that the average query walks, for the estimates of either prefill kernel: calls are taken for causal, but those of more
// queries than keys cannot be.
inline double attention_walked_keys(int64_t Sq, int64_t Sk) { return Sq > Sk ? (double)Sk : (double)Sk - 0.5 * (double)Sq; }
// What that kernel is expected to take, in microseconds (the estimate behind the splits).
double attention_c2_us(int64_t B, int64_t Hq, int64_t Sq, int64_t Hkv, int64_t Sk, int d);
size_t attention_c2_part_bytes(int64_t B, int64_t Hq, int64_t Sq, int d, int nsplit);
// Merge of tiles of 128 query rows and back-rotation by Pi_v (fp32) into a.out.
int merge_split_tiles(const AttnArgs& a, int64_t B, int d, int nsplit, float* part_o, float* part_ml, cudaStream_t stream);

// SM-pair (2-CTA cluster) tensor-core kernel, head_dim 64 and 128; scratch only for the partial results of a split call.
int attention_c2(const AttnArgs& a, const PairArgs& x, int64_t B, int d, int bits, cudaStream_t stream);
int read_c2_faults(unsigned long long* out);
int trace_enable_c2(int on);
int trace_read_c2(long long* host_buf, int max_records, int* n_out);

int prepare_queries_bf16(const void* q, int dtype, int64_t B, int64_t Hq, int64_t Sq, int d, int64_t sb, int64_t sh,
                         int64_t ss, const float* Pi_k, const float* S_eff, void* w_cat_scratch, void* q_cat,
                         cudaStream_t stream, int q_cat_dtype = TQ_BF16);

}  // namespace tq
