// Attention over keys and values expanded to fp16 rows (tq_expand.cu, tq_attention_dense.cu).
#pragma once
#include "tq_attention.cuh"

namespace tq {

// Expanded tiles of 128 keys, [pairs][T][K', V'][128 x d fp16]; a pair is a (batch element, KV head).
struct ExpandArgs {
  const uint8_t *key_idx, *key_sgn;
  const uint16_t *key_vn, *key_rn;
  const uint8_t* val_idx;
  const uint16_t* val_vn;
  int64_t kv_stride, Sk;         // packed rows of a pair, of which Sk are in use
  const uint8_t *w_key, *w_val;  // operand images of the constants buffer
  const uint32_t* luts;
  const float* scales;           // of index, sign and value accumulators
  int64_t pair0;                 // first pair
  int pairs, T, key_ctas;        // pairs, tiles of a pair; CTAs of the key side (set by the launcher)
  MaskBits mb;                   // words != NULL: tiles that it hides from every query are left out
  int Sq, parts;                 // queries; threads that share a tile's classes (set by the launcher)
  int64_t Hkv;
  uint8_t* dst;
};
int expand_kv(const ExpandArgs& a, int d, int bits, cudaStream_t stream);

// Tiles of the maps that the dense kernel skips masked key tiles by; where there are more, it reads every tile.
constexpr int kMapTiles = 2048;

// Whether a bf16-mode call of the SM-pair kernel's is served by expansion and the dense kernel when it has the scratch for it,
// and that scratch.
bool attention_dense_applies(int64_t B, int64_t Hq, int64_t Sq, int64_t Hkv, int64_t Sk, int d);
size_t attention_dense_bytes(int64_t B, int64_t Hq, int64_t Sq, int64_t Hkv, int64_t Sk, int d);
int attention_dense(const AttnArgs& a, int64_t B, int d, int bits, const void* q, int q_dtype, int64_t sb, int64_t sh, int64_t ss,
                    const uint8_t* constants, void* workspace, cudaStream_t stream);

}  // namespace tq
