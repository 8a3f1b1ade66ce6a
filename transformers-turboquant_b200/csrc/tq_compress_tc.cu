// Key / value compression with the rotation and the QJL projection on the tensor cores
// (TQ_MODE_BF16, bf16 inputs).
//
// A persistent CTA walks tiles of 128 vectors with D/32 threads per vector (row r = tensor-memory lane
// r; a thread owns 32 consecutive coordinates of its row, so the per-coordinate work of the epilogues
// runs on 16 warps at head_dim 128).  Per tile:
//   1. each thread loads its 64 bytes of the row (the next tile's are prefetched into registers while the
//      current one is processed), accumulates its part of the squared norm in fp32 (parts are summed
//      through shared memory in a fixed order) and writes the raw bf16 values into the A operand tile.  bf16 inputs are EXACT operands; the fp32 rotation matrix is split
//      into bf16 hi + lo parts, so y_raw = x (Pi_hi + Pi_lo)^T carries ~16 mantissa bits;
//   2. tcgen05.mma: Y_raw = X Pi_hi^T + X Pi_lo^T (fp32 accumulation in tensor memory);
//   3. epilogue: y = y_raw / (n + 1e-8), Lloyd-Max index by boundary counting, the row's packed
//      bytes assembled in registers and stored with 16-byte stores;
//   4. keys only: residual in rotated coordinates r = y_raw - n C[idx] (fp32), its squared norm,
//      r split into bf16 hi + lo and written over the A tile; tcgen05.mma
//      proj = r_hi Se_hi^T + r_hi Se_lo^T + r_lo Se_hi^T; sign bits of proj -> 16 bytes per row.
// Follows compressors.py:98-161, :270-294 of the reference; the arithmetic differs from the fp32
// kernel only in the ~2^-17 relative rounding of the split operands.
#include "tq_compress.cuh"
#include "tq_simt.cuh"
#include "tq_tcgen05.cuh"

namespace tq {

__device__ unsigned long long g_compress_faults = 0ull;  // expired bounded waits in this file's kernels
// this device's slot of the host-visible status page (NULL until the first call on the device installs it)
__device__ unsigned long long* g_fault_mailbox_compress = nullptr;
int set_fault_mailbox_compress(unsigned long long* slot) {
  TQ_CUDA_OK(cudaMemcpyToSymbol(g_fault_mailbox_compress, &slot, sizeof(slot)));
  return TQ_OK;
}

int read_compress_faults(unsigned long long* out) {
  TQ_CUDA_OK(cudaMemcpyFromSymbol(out, g_compress_faults, sizeof(*out)));
  return TQ_OK;
}

namespace {

__device__ __forceinline__ uint32_t bf16_bits(float v) {
  return static_cast<uint32_t>(__bfloat16_as_ushort(__float2bfloat16_rn(v)));
}
__device__ __forceinline__ float bf16_value(uint32_t b) { return __uint_as_float(b << 16); }

// Copy a row-major fp32 [D, D] matrix into two canonical K-major bf16 operand tiles: hi = bf16(m),
// lo = bf16(m - hi).  Row j, 8-element chunk c at (j/8)*SBO + c*128 + (j%8)*16.
template <int D>
__device__ void load_split_matrix(const float* __restrict__ M, uint8_t* hi, uint8_t* lo, int tid, int nthreads) {
  constexpr int G = D / 8;
  constexpr uint32_t SBO = G * 128;
  for (int e = tid; e < D * G; e += nthreads) {
    const int j = e % 8 + 8 * (e / (8 * G)), c = (e / 8) % G;
    float v[8];
    load8<float>(M + j * D + c * 8, v);
    uint32_t h[4], l[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const uint32_t h0 = bf16_bits(v[2 * i]), h1 = bf16_bits(v[2 * i + 1]);
      h[i] = h0 | (h1 << 16);
      l[i] = bf16_bits(v[2 * i] - bf16_value(h0)) | (bf16_bits(v[2 * i + 1] - bf16_value(h1)) << 16);
    }
    const uint32_t off = (j / 8) * SBO + c * 128 + (j % 8) * 16;
    *reinterpret_cast<uint4*>(hi + off) = make_uint4(h[0], h[1], h[2], h[3]);
    *reinterpret_cast<uint4*>(lo + off) = make_uint4(l[0], l[1], l[2], l[3]);
  }
}

template <int D, int IB, bool IS_KEY>
__global__ void __launch_bounds__(4 * D, 1) compress_tc_kernel(const CompressArgs a) {
  constexpr int G = D / 8;
  constexpr int NP = D / 32;               // threads per row: each owns 32 consecutive coordinates
  constexpr int kThreads = 128 * NP;
  constexpr uint32_t SBO = G * 128;
  constexpr uint32_t MAT = D * D * 2;      // one bf16 matrix
  constexpr uint32_t TILE = 128 * D * 2;   // one bf16 A tile
  constexpr int NB = (1 << IB) - 1;
  constexpr int ROWB = D * IB / 8;         // packed index bytes per row (4 * IB of them per thread)
  constexpr int kCols = IS_KEY ? 2 * D : D;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* PiH = smem;
  uint8_t* PiL = PiH + MAT;
  uint8_t* SeH = PiL + MAT;                 // keys only
  uint8_t* SeL = SeH + (IS_KEY ? MAT : 0);
  uint8_t* A0 = SeL + (IS_KEY ? MAT : 0);   // X, later r_hi
  uint8_t* A1 = A0 + TILE;                  // r_lo (keys only)
  __shared__ __align__(8) uint64_t bar;
  __shared__ uint32_t tmem_slot;
  __shared__ int s_abort;
  __shared__ float cen_s[IS_KEY ? (1 << IB) : 1];
  __shared__ float ss_part[NP][128];        // partial squared norms of the row's parts
  __shared__ float rr_part[IS_KEY ? NP : 1][128];
  const int tid = threadIdx.x, warp = tid / 32, lane = tid % 32;
  const int row = (warp % 4) * 32 + lane;   // = tensor-memory lane
  const int part = warp / 4;                // coordinates [32 part, 32 part + 32)

  if (tid == 0) {
    s_abort = 0;
    tc::mbar_init(tc::smem_u32(&bar), 1);
    tc::fence_mbar_init();
  }
  if (warp == 0) tc::tmem_alloc(tc::smem_u32(&tmem_slot), kCols < 32 ? 32 : kCols);
  load_split_matrix<D>(a.Pi, PiH, PiL, tid, kThreads);
  if (IS_KEY) {
    load_split_matrix<D>(a.S_eff, SeH, SeL, tid, kThreads);
    if (tid < (1 << IB)) cen_s[tid] = a.centroids[tid];
  }
  float bnd[NB];
#pragma unroll
  for (int j = 0; j < NB; ++j) bnd[j] = __ldg(a.boundaries + j);
  tc::fence_async_smem();
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = tmem_slot;
  const uint32_t lane_base = (uint32_t)((warp % 4) * 32) << 16;
  const uint32_t bar_addr = tc::smem_u32(&bar);
  constexpr uint32_t idesc = tc::idesc_bf16(128, D, false, false);
  const uint64_t a0d = tc::smem_desc(tc::smem_u32(A0), 128, SBO), a1d = tc::smem_desc(tc::smem_u32(A1), 128, SBO);
  const uint64_t pihd = tc::smem_desc(tc::smem_u32(PiH), 128, SBO), pild = tc::smem_desc(tc::smem_u32(PiL), 128, SBO);
  const uint64_t sehd = tc::smem_desc(tc::smem_u32(SeH), 128, SBO), seld = tc::smem_desc(tc::smem_u32(SeL), 128, SBO);
  const __nv_bfloat16* src = static_cast<const __nv_bfloat16*>(a.src);
  const int64_t HS = a.H * a.S;
  uint32_t phase = 0;
  volatile int* abort_flag = &s_abort;

  uint4 rowbuf[4];  // this thread's 32 coordinates of its row of the tile about to be processed
  auto fetch = [&](int tile) {
    const int64_t n = static_cast<int64_t>(tile) * 128 + row;
    if (tile < a.num_tiles && n < a.n_vec) {
      const int64_t b = n / HS, rem = n % HS;
      const uint4* p = reinterpret_cast<const uint4*>(src + b * a.stride_b + (rem / a.S) * a.stride_h +
                                                      (rem % a.S) * a.stride_s) + 4 * part;
#pragma unroll
      for (int c = 0; c < 4; ++c) rowbuf[c] = p[c];
    } else {
#pragma unroll
      for (int c = 0; c < 4; ++c) rowbuf[c] = make_uint4(0, 0, 0, 0);
    }
  };
  fetch(blockIdx.x);

  for (int tile = blockIdx.x; tile < a.num_tiles; tile += gridDim.x) {
    const int64_t n = static_cast<int64_t>(tile) * 128 + row;
    const bool live = n < a.n_vec;
    const int64_t no = compress_out_row(a, n);  // where this vector's packed row goes
    // ---- 1. norm + A tile ------------------------------------------------------------------
    {
      float ss = 0.f;
      uint8_t* dst = A0 + (row / 8) * SBO + (row % 8) * 16 + 4 * part * 128;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const uint32_t w[4] = {rowbuf[c].x, rowbuf[c].y, rowbuf[c].z, rowbuf[c].w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float lo = __uint_as_float(w[i] << 16), hi = __uint_as_float(w[i] & 0xffff0000u);
          ss = fmaf(lo, lo, ss);
          ss = fmaf(hi, hi, ss);
        }
        *reinterpret_cast<uint4*>(dst + c * 128) = rowbuf[c];
      }
      ss_part[part][row] = ss;
    }
    tc::fence_async_smem();
    tc::fence_before_sync();
    __syncthreads();
    // ---- 2. rotate ---------------------------------------------------------------------------
    if (tid == 0) {
      tc::fence_after_sync();
#pragma unroll
      for (int ks = 0; ks < D / 16; ++ks)
        tc::mma_bf16(tmem, a0d + (uint64_t)(ks * 256 >> 4), pihd + (uint64_t)(ks * 256 >> 4), idesc, ks > 0);
#pragma unroll
      for (int ks = 0; ks < D / 16; ++ks)
        tc::mma_bf16(tmem, a0d + (uint64_t)(ks * 256 >> 4), pild + (uint64_t)(ks * 256 >> 4), idesc, 1u);
      tc::mma_commit(bar_addr);
    }
    fetch(tile + gridDim.x);  // next tile's rows travel while this one is processed
    float ss = 0.f;  // summed in a fixed order, so that every part of the row sees the same norm
#pragma unroll
    for (int q = 0; q < NP; ++q) ss += ss_part[q][row];
    const float nv = sqrtf(ss), den = nv + 1e-8f;
    // y = y_raw / den is compared with the boundaries as y_raw > b * den (den > 0): one multiply per
    // boundary and row instead of one division per coordinate
    float bden[NB];
#pragma unroll
    for (int j = 0; j < NB; ++j) bden[j] = bnd[j] * den;
    if (!tc::mbar_wait_or_abort(bar_addr, phase, abort_flag)) break;
    phase ^= 1;
    tc::fence_after_sync();
    // ---- 3. index + pack (4. residual) ----------------------------------------------------------
    float rr = 0.f;
    uint32_t packed[IB];
#pragma unroll
    for (int i = 0; i < IB; ++i) packed[i] = 0;
    {
      uint32_t raw[32];
      tc::tmem_ld32(tmem + lane_base + 32 * part, raw);
      tc::wait_ld();
#pragma unroll
      for (int g8 = 0; g8 < 4; ++g8) {
        uint64_t word = 0;
        uint32_t rh[4], rl[4];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const float yr = __uint_as_float(raw[g8 * 8 + e]);
          const int idx = count_below<NB>(yr, bden);
          word |= static_cast<uint64_t>(idx) << (e * IB);
          if (IS_KEY) {
            const float res = fmaf(-nv, cen_s[idx], yr);
            rr = fmaf(res, res, rr);
            const uint32_t hb = bf16_bits(res), lb = bf16_bits(res - bf16_value(hb));
            if (e & 1) { rh[e / 2] |= hb << 16; rl[e / 2] |= lb << 16; }
            else { rh[e / 2] = hb; rl[e / 2] = lb; }
          }
        }
        // the 8 fields of this group are IB whole bytes at byte offset g8*IB of the thread's 4*IB bytes
#pragma unroll
        for (int bt = 0; bt < IB; ++bt) {
          const int byte = g8 * IB + bt;
          packed[byte / 4] |= static_cast<uint32_t>((word >> (8 * bt)) & 0xffu) << (8 * (byte % 4));
        }
        if (IS_KEY) {
          const uint32_t off = (row / 8) * SBO + (4 * part + g8) * 128 + (row % 8) * 16;
          *reinterpret_cast<uint4*>(A0 + off) = make_uint4(rh[0], rh[1], rh[2], rh[3]);
          *reinterpret_cast<uint4*>(A1 + off) = make_uint4(rl[0], rl[1], rl[2], rl[3]);
        }
      }
    }
    if (live) {
      uint32_t* dst = reinterpret_cast<uint32_t*>(a.packed_idx + no * ROWB + 4 * IB * part);
      if constexpr (IB == 4) *reinterpret_cast<uint4*>(dst) = make_uint4(packed[0], packed[1], packed[2], packed[3]);
      else if constexpr (IB == 2) *reinterpret_cast<uint2*>(dst) = make_uint2(packed[0], packed[1]);
      else {
#pragma unroll
        for (int i = 0; i < IB; ++i) dst[i] = packed[i];
      }
      if (part == 0) a.vec_norms[no] = fp16_bits(nv);
    }
    if (IS_KEY) {
      // ---- QJL sketch of the residual --------------------------------------------------------
      rr_part[part][row] = rr;
      tc::fence_async_smem();
      tc::fence_before_sync();
      __syncthreads();
      if (tid == 0) {
        tc::fence_after_sync();
#pragma unroll
        for (int ks = 0; ks < D / 16; ++ks)
          tc::mma_bf16(tmem + D, a0d + (uint64_t)(ks * 256 >> 4), sehd + (uint64_t)(ks * 256 >> 4), idesc, ks > 0);
#pragma unroll
        for (int ks = 0; ks < D / 16; ++ks)
          tc::mma_bf16(tmem + D, a0d + (uint64_t)(ks * 256 >> 4), seld + (uint64_t)(ks * 256 >> 4), idesc, 1u);
#pragma unroll
        for (int ks = 0; ks < D / 16; ++ks)
          tc::mma_bf16(tmem + D, a1d + (uint64_t)(ks * 256 >> 4), sehd + (uint64_t)(ks * 256 >> 4), idesc, 1u);
        tc::mma_commit(bar_addr);
      }
      if (live && part == 0) {
        float rs = 0.f;
#pragma unroll
        for (int q = 0; q < NP; ++q) rs += rr_part[q][row];
        a.residual_norms[no] = fp16_bits(sqrtf(rs));
      }
      if (!tc::mbar_wait_or_abort(bar_addr, phase, abort_flag)) break;
      phase ^= 1;
      tc::fence_after_sync();
      uint32_t raw[32];
      tc::tmem_ld32(tmem + D + lane_base + 32 * part, raw);
      tc::wait_ld();
      uint32_t bits = 0;
#pragma unroll
      for (int e = 0; e < 32; ++e) bits |= (__uint_as_float(raw[e]) >= 0.f ? 1u : 0u) << e;
      if (live) *reinterpret_cast<uint32_t*>(a.packed_signs + no * (D / 8) + 4 * part) = bits;
    }
    tc::fence_before_sync();
    __syncthreads();  // the next tile overwrites the A tiles, the partial sums and the accumulators
  }
  if (s_abort) {
    if (tid == 0) {
      atomicAdd(&g_compress_faults, 1ull);
      notify_host_of_fault(g_fault_mailbox_compress);
    }
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 0) tc::tmem_dealloc(tmem, kCols < 32 ? 32 : kCols);
}

template <int D, int IB, bool IS_KEY>
int launch(const CompressArgs& a, cudaStream_t stream) {
  constexpr size_t smem_req = (size_t)(IS_KEY ? 4 : 2) * D * D * 2 + (size_t)(IS_KEY ? 2 : 1) * 128 * D * 2;
  // one CTA of 4 D threads per SM (16 warps at head_dim 128): the register file does not hold two
  constexpr int per_sm = 1;
  auto kern = compress_tc_kernel<D, IB, IS_KEY>;
  TQ_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_req));
  const int tiles = (int)((a.n_vec + 127) / 128);
  CompressArgs b = a;
  b.num_tiles = tiles;
  int grid = sm_count() * per_sm;
  if (grid > tiles) grid = tiles;
  {
    ProfScope prof(IS_KEY ? kProfCompressKeys : kProfCompressValues, stream);
    kern<<<grid, 4 * D, smem_req, stream>>>(b);
  }
  TQ_CUDA_OK(cudaGetLastError());
  return TQ_OK;
}

// ---- value decompression -------------------------------------------------------------------
//
// out = n C[idx] Pi for tiles of 128 vectors.  Centroids (x 256) are split into three fp16 parts, the rotation (x 128) into
// hi + lo (22 mantissa bits, scaled so that the low parts are normal numbers); the four products that matter run as tcgen05
// MMAs, small ones first (the accumulator is truncated at every step), and the norm and 2^-15 are applied in fp32.  Against
// fp64 the result is as close as the fp32 CUDA-core product it replaces (relative
// errors 1.2e-7 to 2.0e-7 at either head_dim, 1.5e-7 to 2.1e-7 before).  The fixed scales hold those bits for rotations whose
// columns reach 2^-7 and stay below 2^8 and for centroids that are 0 or between 2^-9 and 2^7, as every orthonormal matrix
// and codebook of its coordinates is; with other constants the CTA multiplies in fp32, coordinate by coordinate.
// A CTA converts the rotation once and walks tiles; 16384 vectors at head_dim 128 took 20 us on the CUDA cores, bound by
// the latency of shared-memory operands at 8 warps per tile; 11 us here, most of it the conversion and the launch.
template <int D, int VB>
__global__ void __launch_bounds__(256, 1) decompress_tc_kernel(const uint8_t* __restrict__ idx, const uint16_t* __restrict__ vn,
                                                               int64_t n_vec, const float* __restrict__ Pi,
                                                               const float* __restrict__ cen, float* __restrict__ out,
                                                               int num_tiles) {
  constexpr int G = D / 8;
  constexpr uint32_t MAT = D * D * 2, TILE = 128 * D * 2, SBO = G * 128;  // A: K-major, 8-row groups SBO apart
  constexpr uint32_t LBO = G * 128;                                       // B: MN-major, 8-row groups of Pi LBO apart
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t *BH = smem, *BL = BH + MAT, *AH = BL + MAT, *AL = AH + TILE, *AX = AL + TILE;
  __shared__ __align__(8) uint64_t bar;
  __shared__ uint32_t tmem_slot;
  __shared__ int s_abort;
  __shared__ float cen_s[1 << VB];
  __shared__ uint32_t s_reach[8][G];                 // per warp and eight columns: those with an entry that reaches 2^-7
  __shared__ uint32_t lut[1 << VB], lut_x[1 << VB];  // low half: fp16 hi part of the centroid, high half: lo part; what is left
  const int tid = threadIdx.x, warp = tid / 32, lane = tid % 32;
  if (tid == 0) {
    s_abort = 0;
    tc::mbar_init(tc::smem_u32(&bar), 1);
    tc::fence_mbar_init();
  }
  if (warp == 0) tc::tmem_alloc(tc::smem_u32(&tmem_slot), D);
  auto split = [](float v, uint32_t& hi, uint32_t& lo) {
    const __half h = __float2half_rn(v);
    hi = __half_as_ushort(h);
    lo = __half_as_ushort(__float2half_rn(v - __half2float(h)));
  };
  bool fits = true;  // the constants suit the fixed scales (a NaN does not)
  if (tid < (1 << VB)) {
    uint32_t hi, lo;
    cen_s[tid] = cen[tid];
    const float v = cen[tid] * 256.f;
    fits = v == 0.f || (fabsf(v) >= 0.5f && fabsf(v) <= 32768.f);
    split(v, hi, lo);
    lut[tid] = hi | (lo << 16);
    // (an error of a centroid would be that of every coordinate at its level)
    const float rest = (v - __half2float(__ushort_as_half((unsigned short)hi))) - __half2float(__ushort_as_half((unsigned short)lo));
    lut_x[tid] = __half_as_ushort(__float2half_rn(rest));
  }
  uint32_t reach = 0;  // (a thread's pieces are the same eight columns: 256 is a multiple of G)
#pragma unroll 4
  for (int e = tid; e < D * G; e += 256) {  // eight columns of a row of Pi
    const int i = e / G, c = e % G;
    const float4 p0 = ldg4(Pi + i * D + 8 * c), p1 = ldg4(Pi + i * D + 8 * c + 4);
    const float v[8] = {p0.x, p0.y, p0.z, p0.w, p1.x, p1.y, p1.z, p1.w};
    uint32_t h[8], l[8];
#pragma unroll
    for (int x = 0; x < 8; ++x) {
      split(v[x] * 128.f, h[x], l[x]);
      fits = fits && fabsf(v[x]) <= 256.f;
      reach |= fabsf(v[x]) >= 0.0078125f ? 1u << x : 0u;
    }
    const uint32_t off = (i / 8) * LBO + c * 128 + (i % 8) * 16;
    *reinterpret_cast<uint4*>(BH + off) = make_uint4(h[0] | (h[1] << 16), h[2] | (h[3] << 16), h[4] | (h[5] << 16), h[6] | (h[7] << 16));
    *reinterpret_cast<uint4*>(BL + off) = make_uint4(l[0] | (l[1] << 16), l[2] | (l[3] << 16), l[4] | (l[5] << 16), l[6] | (l[7] << 16));
  }
#pragma unroll
  for (int off = G; off < 32; off <<= 1) reach |= __shfl_xor_sync(0xffffffffu, reach, off);
  if (lane < G) s_reach[warp][lane] = reach;
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  if (tid < G) {
    uint32_t all = 0;
#pragma unroll
    for (int w = 0; w < 8; ++w) all |= s_reach[w][tid];
    fits = fits && all == 0xffu;
  }
  const bool scaled = __syncthreads_and(fits);
  const uint32_t tmem = tmem_slot, bar_addr = tc::smem_u32(&bar);
  constexpr uint32_t idesc = tc::idesc_f16(128, D, false, true);
  const uint64_t ah = tc::smem_desc(tc::smem_u32(AH), 128, SBO), al = tc::smem_desc(tc::smem_u32(AL), 128, SBO);
  const uint64_t ax = tc::smem_desc(tc::smem_u32(AX), 128, SBO);
  const uint64_t bh = tc::smem_desc(tc::smem_u32(BH), LBO, 128), bl = tc::smem_desc(tc::smem_u32(BL), LBO, 128);
  volatile int* abort_flag = &s_abort;
  uint32_t phase = 0;
  bool ok = true;
  for (int tile = blockIdx.x; tile < num_tiles; tile += gridDim.x) {
    const int64_t base = (int64_t)tile * 128;
    if (!scaled) {
#pragma unroll 1
      for (int r = tid / D; r < 128 && base + r < n_vec; r += 256 / D) {
        const uint8_t* row = idx + (base + r) * (D * VB / 8);
        float acc = 0.f;
#pragma unroll 1
        for (int c = 0; c < G; ++c) {
          const uint64_t w = load_fields8<VB>(row + c * VB);
#pragma unroll
          for (int x = 0; x < 8; ++x)
            acc = fmaf(cen_s[(uint32_t)(w >> (x * VB)) & ((1u << VB) - 1)], __ldg(Pi + (8 * c + x) * D + tid % D), acc);
        }
        out[(base + r) * D + tid % D] = acc * fp16_value(vn[base + r]);
      }
      continue;
    }
#pragma unroll 4
    for (int e = tid; e < 128 * G; e += 256) {
      const int r = e % 8 + 8 * (e / (8 * G)), c = (e / 8) % G;
      const uint64_t w = base + r < n_vec ? load_fields8<VB>(idx + (base + r) * (D * VB / 8) + c * VB) : 0ull;
      uint32_t t[8], u[8];
#pragma unroll
      for (int x = 0; x < 8; ++x) {
        const uint32_t i = (uint32_t)(w >> (x * VB)) & ((1u << VB) - 1);
        t[x] = lut[i];
        u[x] = lut_x[i];
      }
      const uint32_t off = (r / 8) * SBO + c * 128 + (r % 8) * 16;
      *reinterpret_cast<uint4*>(AH + off) = make_uint4(__byte_perm(t[0], t[1], 0x5410), __byte_perm(t[2], t[3], 0x5410),
                                                       __byte_perm(t[4], t[5], 0x5410), __byte_perm(t[6], t[7], 0x5410));
      *reinterpret_cast<uint4*>(AL + off) = make_uint4(__byte_perm(t[0], t[1], 0x7632), __byte_perm(t[2], t[3], 0x7632),
                                                       __byte_perm(t[4], t[5], 0x7632), __byte_perm(t[6], t[7], 0x7632));
      *reinterpret_cast<uint4*>(AX + off) = make_uint4(u[0] | (u[1] << 16), u[2] | (u[3] << 16), u[4] | (u[5] << 16), u[6] | (u[7] << 16));
    }
    tc::fence_async_smem();
    tc::fence_before_sync();
    __syncthreads();
    if (tid == 0) {
      tc::fence_after_sync();
      auto product = [&](uint64_t a, uint64_t b, uint32_t accumulate) {
#pragma unroll
        for (int ks = 0; ks < D / 16; ++ks)
          tc::mma_bf16(tmem, a + (uint64_t)(ks * 256 >> 4), b + (uint64_t)(ks * 2 * LBO >> 4), idesc, ks > 0 ? 1u : accumulate);
      };
      product(ax, bh, 0u);
      product(al, bh, 1u);
      product(ah, bl, 1u);
      product(ah, bh, 1u);
      tc::mma_commit(bar_addr);
    }
    if (!(ok = tc::mbar_wait_or_abort(bar_addr, phase, abort_flag))) break;
    phase ^= 1;
    tc::fence_after_sync();
    const int64_t n = base + (warp % 4) * 32 + lane;
    const float scale = n < n_vec ? fp16_value(vn[n]) * (1.f / 32768.f) : 0.f;
#pragma unroll
    for (int c0 = 0; c0 < D / 2; c0 += 32) {
      const int col = warp / 4 * (D / 2) + c0;
      uint32_t raw[32];
      tc::tmem_ld32(tmem + ((uint32_t)((warp % 4) * 32) << 16) + col, raw);
      tc::wait_ld();
      if (n < n_vec) {
        float4* dst = reinterpret_cast<float4*>(out + n * D + col);
#pragma unroll
        for (int i = 0; i < 8; ++i)
          dst[i] = make_float4(__uint_as_float(raw[4 * i]) * scale, __uint_as_float(raw[4 * i + 1]) * scale,
                               __uint_as_float(raw[4 * i + 2]) * scale, __uint_as_float(raw[4 * i + 3]) * scale);
      }
    }
    tc::fence_before_sync();
    __syncthreads();  // the next tile overwrites the operand tiles and the accumulator
    tc::fence_after_sync();
  }
  if (!ok && atomicExch(&s_abort, 2) != 2) {  // one fault per CTA
    atomicAdd(&g_compress_faults, 1ull);
    notify_host_of_fault(g_fault_mailbox_compress);
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 0) tc::tmem_dealloc(tmem, D);
}

template <int D, int VB>
int launch_decompress(const uint8_t* idx, const uint16_t* vn, int64_t n, const float* Pi, const float* cen, float* out,
                      cudaStream_t stream) {
  constexpr size_t smem = (size_t)2 * D * D * 2 + (size_t)3 * 128 * D * 2;
  auto kern = decompress_tc_kernel<D, VB>;
  TQ_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const int64_t tiles = (n + 127) / 128;
  TQ_REQUIRE(tiles < ((int64_t)1 << 31), "too many vectors");
  const int grid = (int)(tiles < sm_count() ? tiles : sm_count());
  kern<<<grid, 256, smem, stream>>>(idx, vn, n, Pi, cen, out, (int)tiles);
  TQ_CUDA_OK(cudaGetLastError());
  return TQ_OK;
}

}  // namespace

int decompress_tc(const uint8_t* idx, const uint16_t* vn, int64_t n, int d, const float* Pi, const float* cen, int bits,
                  float* out, cudaStream_t stream) {
  if (d == 128)
    return bits == 2 ? launch_decompress<128, 2>(idx, vn, n, Pi, cen, out, stream)
           : bits == 3 ? launch_decompress<128, 3>(idx, vn, n, Pi, cen, out, stream)
                       : launch_decompress<128, 4>(idx, vn, n, Pi, cen, out, stream);
  return bits == 2 ? launch_decompress<64, 2>(idx, vn, n, Pi, cen, out, stream)
         : bits == 3 ? launch_decompress<64, 3>(idx, vn, n, Pi, cen, out, stream)
                     : launch_decompress<64, 4>(idx, vn, n, Pi, cen, out, stream);
}

int compress_tc(bool is_key, int d, int ib, const CompressArgs& a, cudaStream_t stream) {
  if (is_key) {
    if (d == 128) return ib == 1 ? launch<128, 1, true>(a, stream) : ib == 2 ? launch<128, 2, true>(a, stream)
                                                                             : launch<128, 3, true>(a, stream);
    return ib == 1 ? launch<64, 1, true>(a, stream) : ib == 2 ? launch<64, 2, true>(a, stream)
                                                              : launch<64, 3, true>(a, stream);
  }
  if (d == 128) return ib == 2 ? launch<128, 2, false>(a, stream) : ib == 3 ? launch<128, 3, false>(a, stream)
                                                                            : launch<128, 4, false>(a, stream);
  return ib == 2 ? launch<64, 2, false>(a, stream) : ib == 3 ? launch<64, 3, false>(a, stream)
                                                             : launch<64, 4, false>(a, stream);
}

}  // namespace tq
