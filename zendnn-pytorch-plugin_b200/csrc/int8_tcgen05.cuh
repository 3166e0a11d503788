// int8 x int8 -> int32 GEMM on tcgen05 tensor cores with the dynamic-qlinear epilogue fused.
//
//   acc[M,N] = Q[M,K] . W[N,K]^T          (Q: per-token quantised activations, s8 or u8; W: s8)
//   Y = post_ops( (acc - zp_m * wsum_n) * (s_m * w_n) + bias_n )
//
// Both operands are K-major, so they go from global memory to shared memory with plain 2-D TMA tile
// loads (128 bytes of K per row, 128-byte swizzle; up to four such blocks of K per stage for small tiles) and are
// consumed in place by tcgen05.mma.kind::i8 (K = 32 per instruction, four per 128-byte block).  The kernel is
// persistent: one CTA per SM walks over (MH*128) x BN output tiles (MH = 2 reuses each weight
// stage for two 128-row accumulators, which halves the weight bytes pulled per MAC) (tiles that share a weight column
// block are adjacent in the order, so they run at the same time on neighbouring SMs and the weight
// block is fetched from HBM once).  The tile's width BN is a run-time argument (pick_tile in int8_tcgen05.cu).  The
// int32 accumulator lives in tensor memory and is double buffered up to 512 columns in all, so the epilogue of tile i overlaps
// the main loop of tile i+1:
//
//   warp 0      TMA producer: fills the shared-memory ring, across tile boundaries
//   warp 1      allocates tensor memory, issues the MMAs, frees tensor memory
//   warps 2..9  epilogue: tcgen05.ld the accumulator (lane == output row; two warps per 32-lane
//               quarter, each taking every other 32-column chunk), scale, bias, post-op, cast,
//               16-byte stores
//
// The producer and the issuer run as whole warps, one lane issuing, with uniform control flow (see tc05.cuh), and the
// issuer looks at the next stage's barrier while it issues: M = 1 on 8192 -> 10240 25.5 -> 22.4 us; M = 512 and larger, bound
// by operand delivery out of L2 and by power, did not change.
//
// Ring stages are recycled through full/empty mbarriers (tcgen05.commit frees a stage when the MMAs
// that read it retire); accumulator buffers through tmem_full/tmem_empty mbarriers.  Every wait is
// bounded: on expiry the role records a status code and stops, the other roles run into their own
// bounded waits, tensor memory is freed and the kernel returns.
#pragma once

#include "int8.cuh"
#include "tc05.cuh"

namespace zt {

namespace i8tc {

constexpr int kBM = 128;
constexpr int kBK = 128;  // bytes (= int8 elements) of K per stage
constexpr int kEpiWarps = 8;
constexpr int kThreads = 64 + kEpiWarps * 32;

// kEpiStatic: the static-quantisation form (per-tensor activation parameters, optional per-tensor weight scale,
// requantised or strided output); kept apart so that the dynamic form's epilogue carries none of it
enum EpiMode { kEpiS32 = 0, kEpiLinear = 1, kEpiStatic = 2 };

constexpr int kMaxBN = 256;
constexpr int kMaxStages = 24;

struct TcParams {
  int M, N, K;
  int m_tiles, n_tiles;
  // tile and ring, chosen by the host (see pick_tile): tile width (a multiple of 16), accumulator buffers, rows of an
  // activation box (MH * 128, or fewer when the call has fewer), ring stages, 128-byte blocks of K per stage, stage size,
  // bytes behind the ring that the MMAs may read
  int bn, nbuf, a_rows, stages, group, stage_bytes, ring_pad;
  // epilogue
  const float *src_scale;  // [M]
  const int32_t *src_zp;   // [M] or null
  const void *w_scale;     // [N]
  const int32_t *w_rowsum; // [N] or null
  const void *bias;        // [N] or null
  int w_scale_dtype, bias_dtype, y_dtype;
  void *y;                 // [M,N] (y_dtype) or int32 for kEpiS32
  PostOpsDev post;
  int *status;             // device status word (bounded-wait failures)
  // kEpiStatic only
  bool w_scale_per_tensor;
  int post_dtype;
  const float *out_scale;
  const int32_t *out_zp;
  int64_t ldy;
};

// Dynamic shared memory: the ring, then the vectors and the barriers.  The MMA always reads MH * 128 rows of A; with
// fewer in a stage it runs on into what follows (rows that are never stored), so the ring is padded to keep that inside:
// furthest from the last of the stage's blocks of K.
constexpr int kVecBytes = 2 * 3 * kMaxBN * 4;            // per accumulator buffer: w_scale, bias, rowsum
constexpr int kBarBytes = (2 * kMaxStages + 4) * 8 + 8;
constexpr int kSmemLimit = 227 * 1024;
// Columns of tensor memory of a 128-row accumulator.
__host__ __device__ constexpr int acc_stride(int bn) { return (bn + 31) & ~31; }
constexpr int ring_pad(int mh, int a_rows, int bn, int group) {
  const int read = ((group - 1) * a_rows + mh * kBM) * kBK, stage_bytes = group * (a_rows + bn) * kBK;
  return read > stage_bytes ? read - stage_bytes : 0;
}
static_assert(ring_pad(1, 16, 16, 4) == 48 * kBK && ring_pad(1, 48, 16, 2) == 48 * kBK && ring_pad(1, 128, 16, 1) == 0, "reads past a stage");
constexpr int smem_bytes(int stages, int stage_bytes, int pad) {
  return stages * stage_bytes + pad + kVecBytes + kBarBytes + 1024;   // + slack to align to 1024
}

// A post-op chain on `n` (up to 32) consecutive outputs of one row.  The chain's code exists once, in a loop: unrolled over
// the 32 values (and its four steps) it is some hundred kilobytes of instructions that a tile walks through once, which
// made a 384 x 4096 x 1024 call of the static form take 54 us with 3 % of the issue slots used (12.2 us without a chain now,
// 30 with an addition and 52 with a multiplication and an addition, where it took 75 and 108; the dynamic form on 512 x 4096
// x 4096 37 and 58 us for 84 and 118).
__device__ __forceinline__ void post_chain(float (&v)[32], const PostOpsDev &post, int64_t base, int n, int dtype) {
  float w[32];          // indexed by the loop, so it lives in local memory; `v` stays in registers
#pragma unroll
  for (int j = 0; j < 32; ++j) w[j] = v[j];
#pragma unroll 1
  for (int j = 0; j < n; ++j) w[j] = apply_post_ops(w[j], post, base + j, dtype);
#pragma unroll
  for (int j = 0; j < 32; ++j) v[j] = w[j];
}

__device__ __forceinline__ uint4 pack_bf16x8(const float *v) {
  __nv_bfloat162 t0 = __floats2bfloat162_rn(v[0], v[1]);
  __nv_bfloat162 t1 = __floats2bfloat162_rn(v[2], v[3]);
  __nv_bfloat162 t2 = __floats2bfloat162_rn(v[4], v[5]);
  __nv_bfloat162 t3 = __floats2bfloat162_rn(v[6], v[7]);
  return make_uint4(*reinterpret_cast<uint32_t *>(&t0), *reinterpret_cast<uint32_t *>(&t1),
                    *reinterpret_cast<uint32_t *>(&t2), *reinterpret_cast<uint32_t *>(&t3));
}
// `left` (at most 32) consecutive outputs of one row, in 16-byte stores where `vec` says that the row allows them.
__device__ __forceinline__ void store_bf16(__nv_bfloat16 *dst, const float (&v)[32], int left, bool vec) {
  if (vec && left >= 32) {
#pragma unroll
    for (int j = 0; j < 32; j += 8) *reinterpret_cast<uint4 *>(dst + j) = pack_bf16x8(v + j);
  } else if (vec && left >= 16 && (left & 7) == 0) {      // a tile whose width is an odd multiple of 16
#pragma unroll
    for (int j = 0; j < 32; j += 8)
      if (j < left) *reinterpret_cast<uint4 *>(dst + j) = pack_bf16x8(v + j);
  } else {
#pragma unroll
    for (int j = 0; j < 32; ++j)
      if (j < left) dst[j] = __float2bfloat16_rn(v[j]);
  }
}
__device__ __forceinline__ void store_f32(float *dst, const float (&v)[32], int left, bool vec) {
  if (vec && (left >= 32 || (left & 3) == 0)) {
#pragma unroll
    for (int j = 0; j < 32; j += 4)
      if (j < left) *reinterpret_cast<float4 *>(dst + j) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
  } else {
#pragma unroll
    for (int j = 0; j < 32; ++j)
      if (j < left) dst[j] = v[j];
  }
}

// Scale, bias and post-op for 32 consecutive outputs of one row, then the store.
template <int UNARY>
__device__ __forceinline__ void finish_chunk(const TcParams &p, const uint32_t (&r)[32], float s_m, int zp_m,
                                             const float *wscale, const float *bias, const int32_t *rowsum, int m,
                                             int nb, int n_end) {
  float v[32];
  // per-column vectors of the chunk, read as 16-byte shared loads (same address in every lane: broadcast)
  float wsc[32], bia[32];
#pragma unroll
  for (int j = 0; j < 32; j += 4) {
    const float4 a = *reinterpret_cast<const float4 *>(wscale + j);
    const float4 b = *reinterpret_cast<const float4 *>(bias + j);
    wsc[j] = a.x; wsc[j + 1] = a.y; wsc[j + 2] = a.z; wsc[j + 3] = a.w;
    bia[j] = b.x; bia[j + 1] = b.y; bia[j + 2] = b.z; bia[j + 3] = b.w;
  }
  if (p.src_zp) {
    // u8 activations: remove zp_m * sum_k W[n,k].  |acc|, |zp*rowsum| and their difference are all
    // bounded by 255 * 127 * K, which fits 32 bits for K <= 65536; longer rows take 64 bits.
    if (p.K <= 65536) {
#pragma unroll
      for (int j = 0; j < 32; j += 4) {
        const int4 rs = *reinterpret_cast<const int4 *>(rowsum + j);
        v[j] = (float)((int32_t)r[j] - zp_m * rs.x);
        v[j + 1] = (float)((int32_t)r[j + 1] - zp_m * rs.y);
        v[j + 2] = (float)((int32_t)r[j + 2] - zp_m * rs.z);
        v[j + 3] = (float)((int32_t)r[j + 3] - zp_m * rs.w);
      }
    } else {
#pragma unroll
      for (int j = 0; j < 32; ++j) v[j] = (float)((int64_t)(int32_t)r[j] - (int64_t)zp_m * rowsum[j]);
    }
  } else {
#pragma unroll
    for (int j = 0; j < 32; ++j) v[j] = (float)(int32_t)r[j];
  }
#pragma unroll
  for (int j = 0; j < 32; ++j) v[j] = v[j] * (s_m * wsc[j]) + bia[j];
  const int64_t base = (int64_t)m * p.N + nb;
  if (UNARY >= 0) {
#pragma unroll
    for (int j = 0; j < 32; ++j) v[j] = unary_post(v[j], UNARY);
  } else {
    post_chain(v, p.post, base, min(32, n_end - nb), p.y_dtype);
  }
  const int left = n_end - nb;             // columns of the chunk that belong to the tile
  if (p.y_dtype == ZT_BF16) {
    store_bf16(reinterpret_cast<__nv_bfloat16 *>(p.y) + base, v, left, (p.N & 7) == 0);
  } else {
    store_f32(reinterpret_cast<float *>(p.y) + base, v, left, (p.N & 3) == 0);
  }
}

// The same for the static-quantisation form: separately rounded product and sum (a requantised output sits
// on rounding boundaries of the float result), post-op operands of their own dtype, and a store that
// requantises or honours a row stride.
__device__ __forceinline__ void finish_chunk_static(const TcParams &p, const uint32_t (&r)[32], float s_x, int zp_x,
                                                    const float *wscale, const float *bias, const int32_t *rowsum,
                                                    const OutQuant &oq, int m, int nb, int n_end) {
  float v[32];
  // |acc| and |zp * rowsum| of 8-bit operands stay below 2^31 for K <= 65536 (as in the dynamic form) when the zero point
  // is one that 8 bits can hold; other zero points and longer rows take 64 bits
  const bool narrow = p.K <= 65536 && zp_x >= 0 && zp_x <= 255;
#pragma unroll
  for (int j = 0; j < 32; ++j) {
    const float af = !p.src_zp ? (float)(int32_t)r[j]
                     : narrow  ? (float)((int32_t)r[j] - zp_x * rowsum[j])
                               : (float)((int64_t)(int32_t)r[j] - (int64_t)zp_x * rowsum[j]);
    v[j] = __fadd_rn(__fmul_rn(af, s_x * wscale[j]), bias[j]);
  }
  const int64_t base = (int64_t)m * p.N + nb;
  if (p.post.n_ops > 0) post_chain(v, p.post, base, min(32, n_end - nb), p.post_dtype);
  const int64_t out = (int64_t)m * p.ldy + nb;
  const int left = n_end - nb;
  if (p.y_dtype == ZT_U8 || p.y_dtype == ZT_S8) {
    uint8_t *dst = reinterpret_cast<uint8_t *>(p.y) + out;
    const bool vec = (reinterpret_cast<uintptr_t>(dst) & 15) == 0;
#pragma unroll
    for (int j = 0; j < 32; j += 16) {
      if (vec && j + 16 <= left) {
        uint32_t w4[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          w4[q] = 0;
#pragma unroll
          for (int b = 0; b < 4; ++b) w4[q] |= ((uint32_t)requantize(v[j + 4 * q + b], oq) & 0xffu) << (8 * b);
        }
        *reinterpret_cast<uint4 *>(dst + j) = make_uint4(w4[0], w4[1], w4[2], w4[3]);
      } else {
#pragma unroll
        for (int e = 0; e < 16; ++e)
          if (j + e < left) dst[j + e] = (uint8_t)requantize(v[j + e], oq);
      }
    }
  } else if (p.y_dtype == ZT_BF16) {
    __nv_bfloat16 *dst = reinterpret_cast<__nv_bfloat16 *>(p.y) + out;
    store_bf16(dst, v, left, (reinterpret_cast<uintptr_t>(dst) & 15) == 0);
  } else {
    float *dst = reinterpret_cast<float *>(p.y) + out;
    store_f32(dst, v, left, (reinterpret_cast<uintptr_t>(dst) & 15) == 0);
  }
}

// One operand of a stage: `group` blocks of 128 bytes of K, one copy (a two-dimensional map for one block, which also takes a
// K that is no multiple of 128).
__device__ __forceinline__ void load_stage(bool leader, int group, uint32_t dst, const CUtensorMap *m, uint32_t bar, int kb, int row) {
  if (group == 1)
    tc::load_2d_if(leader, dst, m, bar, kb * kBK, row);
  else
    tc::load_3d_if(leader, dst, m, bar, 0, row, kb * group);
}

template <int MH, int EPI, bool A_SIGNED>
__global__ void __launch_bounds__(kThreads, 1) int8_tcgen05_kernel(const __grid_constant__ CUtensorMap tmap_a,
                                                                   const __grid_constant__ CUtensorMap tmap_b,
                                                                   const TcParams p) {
  extern __shared__ unsigned char smem_dyn[];
  // align on the shared-window address (what the descriptors and TMA see), not the generic one
  unsigned char *smem = smem_dyn + ((1024u - (smem_u32(smem_dyn) & 1023u)) & 1023u);
  const int BN = p.bn, STAGES = p.stages;
  const uint32_t stage_bytes = (uint32_t)p.stage_bytes, a_bytes = (uint32_t)(p.a_rows * p.group) * kBK, NBUF = (uint32_t)p.nbuf;
  unsigned char *after_ring = smem + STAGES * stage_bytes + p.ring_pad;
  float *s_vec = reinterpret_cast<float *>(after_ring);  // [2][3][kMaxBN]
  uint64_t *full_bar = reinterpret_cast<uint64_t *>(after_ring + kVecBytes);
  uint64_t *empty_bar = full_bar + kMaxStages;
  uint64_t *tmem_full = empty_bar + kMaxStages;   // [2]
  uint64_t *tmem_empty = tmem_full + 2;       // [2]
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(tmem_empty + 2);

  constexpr uint32_t kTmemCols = 512;
  const uint32_t acc_cols = (uint32_t)acc_stride(BN);
  const int warp = tc::uniform_warp(), lane = threadIdx.x & 31;
  const bool leader = lane == 0;     // the producer and the issuer run as whole warps, lane 0 issuing
  const int num_kb = (p.K + kBK * p.group - 1) / (kBK * p.group);   // stages per tile (K past the end reads as zeros)
  const int total_tiles = p.m_tiles * p.n_tiles;

  if (threadIdx.x == 0) {
    tc::prefetch_tensormap(&tmap_a);
    tc::prefetch_tensormap(&tmap_b);
    for (int s = 0; s < STAGES; ++s) {
      tc::mbar_init(&full_bar[s], 1);
      tc::mbar_init(&empty_bar[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      tc::mbar_init(&tmem_full[b], 1);
      tc::mbar_init(&tmem_empty[b], kEpiWarps);
    }
    tc::mbar_fence_init();
  }
  if (warp == 1) tc::tmem_alloc(tmem_slot, kTmemCols);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  // Programmatic dependent launch: the next kernel on the stream may start its prologue now; this one waits
  // for its predecessor (the per-token quantisation) only where it touches what that kernel writes.
  grid_launch_dependents();

  if (warp == 0) {
    // ---------------- TMA producer ----------------
    {
      const uint32_t full0 = smem_u32(full_bar), empty0 = smem_u32(empty_bar), smem0 = smem_u32(smem);
      // First pass over the ring: the weight tiles do not depend on the preceding kernel, so they are
      // requested before the dependency wait and the activation tiles of the same stages after it.
      int pre = 0;
      if ((int)blockIdx.x < total_tiles) {
        const int m0 = ((int)blockIdx.x % p.m_tiles) * (MH * kBM);
        const int n0 = ((int)blockIdx.x / p.m_tiles) * BN;
        pre = num_kb < STAGES ? num_kb : STAGES;
        for (int kb = 0; kb < pre; ++kb) {
          tc::expect_tx_if(leader, full0 + kb * 8, stage_bytes);
          load_stage(leader, p.group, smem0 + kb * stage_bytes + a_bytes, &tmap_b, full0 + kb * 8, kb, n0);
        }
        grid_dependency_wait();
        for (int kb = 0; kb < pre; ++kb)
          load_stage(leader, p.group, smem0 + kb * stage_bytes, &tmap_a, full0 + kb * 8, kb, m0);
      }
      uint32_t s = pre == STAGES ? 0u : (uint32_t)pre, ph = pre == STAGES ? 0u : 1u;   // ring slot, parity of its "free" barrier
      bool ok = true;
      for (int tile = blockIdx.x; tile < total_tiles && ok; tile += gridDim.x) {
        const int m0 = (tile % p.m_tiles) * (MH * kBM);
        const int n0 = (tile / p.m_tiles) * BN;
        for (int kb = (tile == (int)blockIdx.x ? pre : 0); kb < num_kb; ++kb) {
          ok = tc::warp_wait(empty0 + s * 8, ph);
          if (!ok) {
            tc::report_timeout(p.status, kStatusProducerTimeout);
            break;
          }
          const uint32_t a_dst = smem0 + s * stage_bytes, bar = full0 + s * 8;
          tc::expect_tx_if(leader, bar, stage_bytes);
          load_stage(leader, p.group, a_dst, &tmap_a, bar, kb, m0);
          load_stage(leader, p.group, a_dst + a_bytes, &tmap_b, bar, kb, n0);
          if (++s == (uint32_t)STAGES) {
            s = 0;
            ph ^= 1;
          }
        }
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer ----------------
    {
      const uint32_t idesc = tc::instr_desc(2u, A_SIGNED ? 1u : 0u, 1u, kBM, (uint32_t)BN);
      const uint64_t d0 = tc::smem_desc_k_sw128(0);
      const uint32_t desc_hi = (uint32_t)(d0 >> 32);
      const uint32_t field0 = (uint32_t)d0 | ((smem_u32(smem) & 0x3FFFF) >> 4);
      const uint32_t full0 = smem_u32(full_bar), empty0 = smem_u32(empty_bar);
      const uint32_t a_block = (uint32_t)p.a_rows * (kBK / 16), b_block = (uint32_t)BN * (kBK / 16);   // a 128-byte block of K
      uint32_t s = 0, ph = 0;
      bool ok = true, ready = false;
      int local = 0;
      for (int tile = blockIdx.x; tile < total_tiles; tile += gridDim.x, ++local) {
        const uint32_t buf = NBUF == 2 ? (uint32_t)local & 1u : 0u;
        const uint32_t use = NBUF == 2 ? (uint32_t)local >> 1 : (uint32_t)local;  // how many times this buffer was used before
        ok = ok && tc::warp_wait(smem_u32(&tmem_empty[buf]), (use & 1) ^ 1);
        if (!ok) tc::report_timeout(p.status, kStatusMmaTimeout);
        tc::fence_after_sync();
        const uint32_t d_tmem = tmem_base + buf * (MH * acc_cols);
        for (int kb = 0; kb < num_kb && ok; ++kb) {
          if (!ready) ok = tc::warp_wait(full0 + s * 8, ph);
          if (!ok) {
            tc::report_timeout(p.status, kStatusMmaTimeout);
            break;
          }
          tc::fence_after_sync();
          const uint32_t a_lo = field0 + s * (stage_bytes >> 4), b_lo = a_lo + (a_bytes >> 4), bar = empty0 + s * 8;
          if (++s == (uint32_t)STAGES) {
            s = 0;
            ph ^= 1;
          }
          // a look at the next stage, answered while the MMAs are being issued
          const uint32_t next = tc::mbar_test_addr(full0 + s * 8, ph);
#pragma unroll 1
          for (int g = 0; g < p.group; ++g) {
            const uint32_t a_g = a_lo + g * a_block, b_g = b_lo + g * b_block;
#pragma unroll
            for (int h = 0; h < MH; ++h) {
#pragma unroll
              for (int k = 0; k < kBK / 32; ++k) {
                // 32 bytes of K per instruction: advance both start addresses by 32 >> 4 = 2; the second
                // 128-row half of the A stage starts 128 * 128 bytes further (>> 4 = 1024)
                tc::mma_i8_if(leader, d_tmem + h * acc_cols, tc::smem_desc_from_words(a_g + h * (kBM * kBK / 16) + 2 * k, desc_hi),
                              tc::smem_desc_from_words(b_g + 2 * k, desc_hi), idesc, (kb > 0 || g > 0 || k > 0) ? 1u : 0u);
              }
            }
          }
          tc::mma_commit_if(leader, bar);
          ready = __all_sync(0xffffffffu, next);
        }
        // Arrive on the accumulator barrier in every case so that the epilogue never waits for a
        // commit that will not come; after a timeout the result is garbage but the kernel ends.
        tc::mma_commit_if(leader, smem_u32(&tmem_full[buf]));
      }
    }
  } else {
    // ---------------- epilogue warps (2..9) ----------------
    grid_dependency_wait();                    // activation scales / zero points come from the preceding kernel
    const int et = threadIdx.x - 64;           // 0..255
    const int quarter = warp & 3;              // TMEM lanes this warp may read: 32*quarter ..
    const int parity = (warp - 2) >> 2;        // which 32-column chunks this warp takes
    const int row = quarter * 32 + lane;
    // a single unary post-op is resolved once, outside the element loops
    int unary = -1;
    if (p.post.n_ops == 0) unary = ZT_POST_NONE;
    else if (p.post.n_ops == 1 && p.post.ids[0] < ZT_POST_MUL) unary = p.post.ids[0];
    OutQuant out_quant{0.f, 0.f, 0.f, 0.f};
    if (EPI == kEpiStatic) out_quant = load_out_quant(p.out_scale, p.out_zp, p.y_dtype);
    int local = 0;
    bool ok = true;
    for (int tile = blockIdx.x; tile < total_tiles; tile += gridDim.x, ++local) {
      const int m0 = (tile % p.m_tiles) * (MH * kBM);
      const int n0 = (tile / p.m_tiles) * BN;
      const uint32_t buf = NBUF == 2 ? (uint32_t)local & 1u : 0u;
      const uint32_t use = NBUF == 2 ? (uint32_t)local >> 1 : (uint32_t)local;
      float *v_wscale = s_vec + (local & 1) * 3 * kMaxBN;
      float *v_bias = v_wscale + kMaxBN;
      int32_t *v_rowsum = reinterpret_cast<int32_t *>(v_bias + kMaxBN);
      const int n_end = min(p.N, n0 + BN);               // the 32-column chunks may reach past a tile's width
      if (EPI != kEpiS32) {
        for (int j = et; j < BN; j += kEpiWarps * 32) {
          const int n = n0 + j;
          const bool in = n < p.N;
          v_wscale[j] = in ? load_as_float(p.w_scale, (EPI == kEpiStatic && p.w_scale_per_tensor) ? 0 : n, p.w_scale_dtype) : 0.f;
          v_bias[j] = (in && p.bias) ? load_as_float(p.bias, n, p.bias_dtype) : 0.f;
          v_rowsum[j] = (in && p.w_rowsum) ? p.w_rowsum[n] : 0;
        }
      }
      // All epilogue threads: the vectors of this tile are visible, and everybody has finished
      // reading the vectors of the tile two back (same buffer).
      asm volatile("bar.sync 1, %0;" ::"n"(kEpiWarps * 32) : "memory");
      ok = ok && tc::warp_wait(smem_u32(&tmem_full[buf]), use & 1);
      if (!ok && leader) tc::report_timeout(p.status, kStatusEpilogueTimeout);
      tc::fence_after_sync();
#pragma unroll 1
      for (int h = 0; h < MH; ++h) {
        const int m = m0 + h * kBM + row;
        const bool row_ok = m < p.M;
        float s_m = 0.f;
        int zp_m = 0;
        if (EPI == kEpiLinear && row_ok) {
          s_m = p.src_scale[m];
          if (p.src_zp) zp_m = p.src_zp[m];
        }
        if (EPI == kEpiStatic) {                     // one scale and zero point for the whole tensor
          s_m = p.src_scale[0];
          if (p.src_zp) zp_m = p.src_zp[0];
        }
        const uint32_t t_row = tmem_base + ((uint32_t)(quarter * 32) << 16) + (buf * MH + h) * acc_cols;
#pragma unroll 1
        for (int c = parity * 32; c < BN; c += 64) {
          uint32_t r[32];
          tc::tmem_ld_32x32b_x32(t_row + c, r);
          tc::tmem_ld_wait();
          const int nb = n0 + c;
          if (row_ok && nb < n_end) {
            if (EPI == kEpiS32) {
              int32_t *dst = reinterpret_cast<int32_t *>(p.y) + (size_t)m * p.N + nb;
#pragma unroll
              for (int j = 0; j < 32; j += 4) {
                if ((p.N & 3) == 0 && nb + j + 4 <= n_end) {
                  *reinterpret_cast<uint4 *>(dst + j) = make_uint4(r[j], r[j + 1], r[j + 2], r[j + 3]);
                } else {
#pragma unroll
                  for (int e = 0; e < 4; ++e)
                    if (nb + j + e < n_end) dst[j + e] = (int32_t)r[j + e];
                }
              }
            } else if (EPI == kEpiStatic) {
              finish_chunk_static(p, r, s_m, zp_m, v_wscale + c, v_bias + c, v_rowsum + c, out_quant, m, nb, n_end);
            } else {
              const float *ws = v_wscale + c, *bs = v_bias + c;
              const int32_t *rs = v_rowsum + c;
              switch (unary) {
                case ZT_POST_NONE: finish_chunk<ZT_POST_NONE>(p, r, s_m, zp_m, ws, bs, rs, m, nb, n_end); break;
                case ZT_POST_RELU: finish_chunk<ZT_POST_RELU>(p, r, s_m, zp_m, ws, bs, rs, m, nb, n_end); break;
                case ZT_POST_SILU: finish_chunk<ZT_POST_SILU>(p, r, s_m, zp_m, ws, bs, rs, m, nb, n_end); break;
                case ZT_POST_GELU_TANH: finish_chunk<ZT_POST_GELU_TANH>(p, r, s_m, zp_m, ws, bs, rs, m, nb, n_end); break;
                case ZT_POST_GELU_ERF: finish_chunk<ZT_POST_GELU_ERF>(p, r, s_m, zp_m, ws, bs, rs, m, nb, n_end); break;
                default: finish_chunk<-1>(p, r, s_m, zp_m, ws, bs, rs, m, nb, n_end); break;
              }
            }
          }
          __syncwarp();  // the next tcgen05.ld is warp-collective
        }
      }
      // this warp has drained its part of the accumulator buffer
      tc::fence_before_sync();
      __syncwarp();
      tc::arrive_if(leader, smem_u32(&tmem_empty[buf]));
    }
  }

  tc::fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    tc::fence_after_sync();
    tc::tmem_dealloc(tmem_base, kTmemCols);
  }
}

// CTA pairs (tcgen05.mma.cta_group::2): 512 x bn tiles, each CTA loads half of every weight block.  Linear
// epilogue only.  Own translation unit (int8_tcgen05_pair.cu).
bool int8_pair_supported(int64_t M, int bn);
int launch_pair(int bn, const Int8GemmArgs &a, const TcParams &p, bool a_signed, cudaStream_t st);

}  // namespace i8tc
}  // namespace zt
