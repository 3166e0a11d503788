// Weight-only int4 linear for M > 16 (prefill and decode batches) on tcgen05 tensor cores.
//
//   Y[M,N] = post_ops( X[M,K] . dq(Wq)[K,N] + bias ),   dq = bf16(q*s)  or  bf16((q-8)*s + z)
//
// The weight is the 128-row operand of the MMA (UMMA M = 128 output columns n) and lives in tensor memory: a
// conversion thread owns one weight row (tensor-memory lane), turns its packed nibbles into bf16 pairs in
// registers and stores them with tcgen05.st, 32 columns (64 k) at a time.  The activations are the other operand
// (UMMA N = the tile's token rows rounded up to 16, chosen at run time), staged in shared memory by TMA.
//
//   warp 0        TMA producer of the activation tiles
//   warp 1        TMEM allocation, tcgen05.mma.kind::f16 issue (A from tensor memory, B from shared memory)
//   warp 2        TMA producer of the packed weights in chunks of 256 k (128 rows x 128 B, 128-byte swizzle) with
//                 their scales / zero points, several chunks ahead, never waiting for the preceding kernel
//   warps 3..6    epilogue: tcgen05.ld (lane = output column n, register j = token), transpose through shared
//                 memory so that stores run along n, bias + post-ops, bf16 stores
//   warps 7..     conversion, teams of four warps; team t of T takes the ring positions congruent to t mod T; then,
//                 idle, they help with the epilogue of the CTA's last tile
//
// What bounds it.  Converting a 128 x 64 block costs its SM about 200 cycles of the two half-rate pipes (per packed word
// of eight weights 9 shift / permute / lop3 operations on one and 8 - 12 bf16x2 operations on the other); its MMAs take 2
// cycles per token and at least 128.  A block takes 300 - 350 cycles up to 128 tokens (650 when the converted operand
// went through shared memory and the issuing threads ran divergent code); M = 32 on 4096 -> 14336: 21.6 -> 13.7 us, M = 128
// on 8192 -> 8192: 31 -> 24 us, M = 2048 on 4096 -> 14336: 259 -> 217 us (0.70 of the bf16 peak; from 128 tokens on an
// SM pulls 35 bytes per cycle of activations and weights out of L2, which is what it can get).  What that took:
//   * The converted operand lives in tensor memory: its 32 KB per block (store, then MMA read) leave the shared-memory
//     port.
//   * The warp index comes from a shuffle, so the compiler knows every role's control flow to be uniform across the
//     warp: descriptors stay in uniform registers and waits are uniform branches.  Single-lane operations are
//     predicated instructions, not branches.  (M = 16, K = 14336 on all SMs: 53 us with divergent roles, 40 with
//     uniform ones, 85 with one polling lane per warp.)
//   * The issuer tests the next stage's barriers in the same straight line of code as the current stage's MMAs: a
//     completed wait costs about 200 cycles of latency.
//   * The conversion loop is one 16-byte piece long, so that it stays in the instruction caches next to the schedulers.
//
// Rings.  Converted stages of KS k in tensor memory (SLOTS of them; a slot always belongs to the same team, which
// therefore waits on each of its phases in order), activation slots of XK k in shared memory (one bulk copy each; they
// are requested long before use because a copy takes over a thousand cycles), packed chunks of 256 k.
//
// Work split.  The unit is a chunk (256 k of a tile).  A CTA usually takes whole tiles; where few tiles have a long K
// ("split", see dense_plan) the chunks of all tiles are dealt to the CTAs in equal contiguous ranges.  The pieces of a
// tile that spans CTAs go through fp32 partial sums in the workspace; the last warp to arrive (a ticket per 16 tokens x
// 32 columns) adds them in CTA order, so results do not depend on timing.
//
// Grouped mode (mixture-of-experts): the rows of X are sorted by expert, a device-side table lists the row tiles
// {expert, first row, valid rows}, and each tile uses its expert's slice of the stacked weight and scale tensors;
// the number of tiles is read from device memory, so no host synchronisation is needed between routing and GEMM.
//
// Accumulators are double buffered in tensor memory.  All waits are bounded (see tc05.cuh).
//
// Rounding.  q (an integer in [-8, 7]) is exact in bf16.  With bf16 scales q*s is one bf16x2 multiplication, i.e.
// exactly bf16(q*s), and (q-8)*s + z one bf16x2 fma, rounded once.  With fp32 scales s is split into s_hi + s_lo
// (both bf16) and dq = fma(q, s_hi, q*s_lo), which equals bf16(q*s) except for rare double-rounding cases one bf16
// ulp apart; the zero-point form is evaluated in fp32 and rounded once.
#include <algorithm>
#include <mutex>
#include <unordered_map>

#include "tc05.cuh"
#include "woq.cuh"

namespace zt {

namespace {

constexpr int kBN = 128;            // output columns per tile (UMMA M)
constexpr int kTeamWarps = 4;       // one warp per 32-lane quarter of tensor memory
constexpr int kEpiWarps = 4;
constexpr int kFirstTeam = 3 + kEpiWarps;   // warps 0..2: activation producer, MMA issuer, packed-weight producer
constexpr int kPackedProducer = 2;
constexpr int threads_for(int teams) { return 32 * (kFirstTeam + teams * kTeamWarps); }
constexpr int kEpiRowStride = 36;   // floats; 144 bytes keeps 16-byte alignment and spreads banks
constexpr int kEpiScratch = 16 * kEpiRowStride;   // per warp: 16 tokens x 32 columns
constexpr int kChunkK = 256;        // k per packed chunk: one 128-byte row of nibbles
constexpr int kChunkBytes = kBN * 128;
// per packed chunk: up to two groups x 128 columns of fp32 scales (1 KB), then the same for zero points
constexpr int kScaleSlotBytes = 2048;
constexpr int kZeroSlotOffset = 1024;
constexpr int kTickets = ZT_WOQ_COUNTER_BYTES / 4;   // one per tile, 16 tokens and 32 columns

// How a weight is dequantised (template parameter of the kernel).
enum DqMode { kSymF32 = 0, kSymBf16 = 1, kAsymBf16 = 2, kAsymF32 = 3 };

struct TcParams {
  int M, N, K;
  int m_tiles, n_tiles, bt;   // dense mode: row tiles of bt tokens
  int chunks;                 // per tile
  int x_box, x_box2;          // rows of the activation box: the first when the tile's rows fit, else the second
  int split;                  // chunks dealt out in equal ranges (else whole tiles)
  int gs, gs_log2;            // gs_log2 < 0: not a power of two
  const int32_t *wq;
  const void *scales;
  const void *zeros;
  const void *bias;
  int bias_dtype;
  __nv_bfloat16 *y;
  PostOpsDev post;
  int *status;
  float *partial;             // split: [2 * CTAs][4 quarters][NMAX / 16][16 x 32] fp32
  unsigned int *tickets;      // split: [tiles][NMAX / 16][4], zero between launches
  // grouped mode (g_count != nullptr)
  const int *g_count;         // number of row tiles
  const int4 *g_tiles;        // per row tile: {expert, first row, valid rows, 0}
  // Scales (and zero points) staged in shared memory with every packed chunk: groups per chunk (1 or 2; 0 = the
  // conversion threads fetch them from global memory), groups per expert.
  int staged_gpc, groups;
};

struct TileInfo {
  int m0, rows, n0, expert;
};
__device__ __forceinline__ TileInfo decode_tile(const TcParams &p, uint32_t tile, uint32_t n_mt) {
  TileInfo t;
  const uint32_t mt = tile % n_mt;
  t.n0 = (int)(tile / n_mt) * kBN;
  if (p.g_count) {
    const int4 g = p.g_tiles[mt];
    t.expert = g.x;
    t.m0 = g.y;
    t.rows = g.z;
  } else {
    t.expert = 0;
    t.m0 = (int)mt * p.bt;
    t.rows = min(p.bt, p.M - t.m0);
  }
  return t;
}

// The chunks a CTA works on, tile by tile.  `total` = tiles x chunks.
struct Work {
  uint32_t pos, end, total, chunks;
  bool split;
  uint32_t tile, c0, c1;   // current segment: chunks [c0, c1) of `tile`

  __device__ __forceinline__ Work(const TcParams &p, uint32_t n_mt) {
    chunks = (uint32_t)p.chunks;
    total = n_mt * (uint32_t)p.n_tiles * chunks;
    split = p.split != 0;
    pos = split ? first_of(blockIdx.x) : blockIdx.x * chunks;
    end = split ? first_of(blockIdx.x + 1) : total;
  }
  __device__ __forceinline__ uint32_t first_of(uint32_t cta) const {
    return (uint32_t)((uint64_t)cta * total / gridDim.x);
  }
  __device__ __forceinline__ uint32_t cta_of(uint32_t position) const {   // the CTA whose range holds it
    return (uint32_t)(((uint64_t)(position + 1) * gridDim.x - 1) / total);
  }
  __device__ __forceinline__ bool next() {
    if (pos >= end) return false;
    tile = pos / chunks;
    c0 = pos - tile * chunks;
    c1 = split ? min(chunks, c0 + (end - pos)) : chunks;
    pos += split ? c1 - c0 : gridDim.x * chunks;
    return true;
  }
  // chunks of this CTA, before the first next()
  __device__ __forceinline__ uint32_t chunks_of_cta() const {
    if (split) return end - pos;
    const uint32_t tiles = total / chunks;
    return blockIdx.x < tiles ? (tiles - blockIdx.x + gridDim.x - 1) / gridDim.x * chunks : 0u;
  }
  __device__ __forceinline__ bool last() const { return pos >= end; }     // of the segment that next() has set
  __device__ __forceinline__ bool whole() const { return c1 - c0 == chunks; }
};

template <int NMAX, int KS, int TEAMS, int SLOTS, int XK, int XSTAGES, int PSTAGES>
struct SmemLayout {
  static constexpr int kXBytes = (XK / 64) * NMAX * 128;
  static constexpr int kXRing = XSTAGES * kXBytes;
  static constexpr int kPackedBytes = PSTAGES * kChunkBytes;
  static constexpr int kScaleBytes = PSTAGES * kScaleSlotBytes;
  static constexpr int kEpiBytes = kEpiWarps * kEpiScratch * 4;
  static constexpr int kBarBytes = (2 * SLOTS + 2 * XSTAGES + 2 * PSTAGES + 5) * 8 + 8;
  static_assert(TEAMS * kTeamWarps * kEpiScratch * 4 <= kXRing, "scratch of the conversion warps");
  static constexpr int kTotal = kXRing + kPackedBytes + kScaleBytes + kEpiBytes + kBarBytes + 1024;
};

__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {
  uint32_t r;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(sel));
  return r;
}
// The low nibbles of both halves of w as bf16: 128 + (nibble ^ 8) for two's complement nibbles, 128 + nibble otherwise.
template <bool SIGNED>
__device__ __forceinline__ uint32_t nib_pair_to_bf16x2(uint32_t w) {
  uint32_t r;
  if (SIGNED) {
    asm("lop3.b32 %0, %1, %2, %3, 0x6a;" : "=r"(r) : "r"(w), "n"(0x000f000f), "n"(0x43084308));
  } else {
    asm("lop3.b32 %0, %1, %2, %3, 0xea;" : "=r"(r) : "r"(w), "n"(0x000f000f), "n"(0x43004300));
  }
  return r;
}
__device__ __forceinline__ uint32_t bf2_sub(uint32_t a, uint32_t b) {
  uint32_t r;
  asm("sub.rn.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}
__device__ __forceinline__ uint32_t bf2_mul(uint32_t a, uint32_t b) {
  uint32_t r;
  asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}
__device__ __forceinline__ uint32_t bf2_fma(uint32_t a, uint32_t b, uint32_t c) {
  uint32_t r;
  asm("fma.rn.bf16x2 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(c));
  return r;
}
__device__ __forceinline__ uint32_t bf2_pack(float lo, float hi) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t *>(&v);
}
__device__ __forceinline__ uint32_t bf16_twice(float v) { return bf2_pack(v, v); }

// Scale and zero point of a group as the conversion takes them: kSymF32 the two bf16 parts of the scale, kSymBf16
// the scale, kAsymBf16 scale and zero point (all in both halves of a register), kAsymF32 the fp32 values.
__device__ __forceinline__ uint4 lds128(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
  return v;
}
struct DqParam {
  uint32_t a, b;
};
template <int MODE>
__device__ __forceinline__ DqParam dq_param(float s, float z) {
  DqParam d;
  if (MODE == kAsymF32) {
    d.a = __float_as_uint(s);
    d.b = __float_as_uint(z);
  } else {
    d.a = bf16_twice(s);
    d.b = MODE == kSymF32 ? bf16_twice(s - __uint_as_float(d.a << 16)) : MODE == kAsymBf16 ? bf16_twice(z) : 0u;
  }
  return d;
}

// 32 k of one weight row: four packed words -> 16 registers of bf16 pairs in k order.
template <int MODE>
__device__ __forceinline__ void convert32(const uint4 &packed, const DqParam &d, uint32_t (&out)[16]) {
  const uint32_t words[4] = {packed.x, packed.y, packed.z, packed.w};
  constexpr bool kAsym = MODE == kAsymBf16 || MODE == kAsymF32;
  if (MODE == kAsymF32) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float f[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const uint32_t bits = ((words[i] >> (4 * e)) & 0xFu) | 0x4B000000u;   // 2^23 + q
        f[e] = fmaf(__uint_as_float(bits) - 8388616.0f, __uint_as_float(d.a), __uint_as_float(d.b));   // (q - 8) * s + z
      }
#pragma unroll
      for (int e = 0; e < 4; ++e) out[4 * i + e] = bf2_pack(f[2 * e], f[2 * e + 1]);
    }
    return;
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const uint32_t w = words[i], w4 = w >> 4;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      // byte e of w holds k = 2e (low nibble), byte e of w >> 4 k = 2e + 1: one per half
      uint32_t v = prmt(w, w4, (uint32_t)(e | (e << 4) | ((4 + e) << 8) | ((4 + e) << 12)));
      v = bf2_sub(nib_pair_to_bf16x2<!kAsym>(v), 0x43084308u);   // exact
      if (MODE == kSymF32)
        v = bf2_fma(v, d.a, bf2_mul(v, d.b));
      else if (MODE == kSymBf16)
        v = bf2_mul(v, d.a);
      else
        v = bf2_fma(v, d.a, d.b);
      out[4 * i + e] = v;
    }
  }
}

// One unary post-op on a thread's 16 values; the switch is outside the element loop so that its code exists once.
__device__ __forceinline__ void unary_post16(float (&v)[4][4], int id) {
#pragma unroll 1
  for (int q = 0; q < 4; ++q) {
    float w[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) w[e] = q == 0 ? v[0][e] : q == 1 ? v[1][e] : q == 2 ? v[2][e] : v[3][e];
#pragma unroll
    for (int e = 0; e < 4; ++e) w[e] = unary_post(w[e], id);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      if (q == 0) v[0][e] = w[e];
      if (q == 1) v[1][e] = w[e];
      if (q == 2) v[2][e] = w[e];
      if (q == 3) v[3][e] = w[e];
    }
  }
}

// The MMAs of one stage, 16 k each: A at consecutive columns of tensor memory, B by descriptor; then the commits that
// free the converted slot and, when `free_x`, the activation slot.  Issued by the lane whose `leader` is set.  A completed
// barrier wait takes its thread about 200 cycles, a third of a stage, so the barriers of the next stage are
// tested in the same straight line of code: their answer arrives while the MMAs are being issued.
template <int N>
struct MmaStage;
template <>
struct MmaStage<4> {
  static __device__ __forceinline__ void issue(uint32_t leader, uint32_t d, uint32_t a, const uint64_t (&b)[4], uint32_t idesc,
                                               uint32_t accumulate, uint32_t bar_a, uint32_t bar_x, uint32_t free_x,
                                               uint32_t next_a, uint32_t par_a, uint32_t next_x, uint32_t par_x,
                                               uint32_t &ready) {
    asm volatile(
        "{\n\t.reg .pred pa, px, pl, pc, pt;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 pa, [%9], %10;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 px, [%11], %12;\n\t"
        "setp.ne.b32 pl, %1, 0;\n\tsetp.ne.b32 pc, %5, 0;\n\tsetp.eq.b32 pt, 0, 0;\n\t"
        "{.reg .b32 t; add.u32 t, %3, 0; @pl tcgen05.mma.cta_group::1.kind::f16 [%2], [t], %13, %4, pc;}\n\t"
        "{.reg .b32 t; add.u32 t, %3, 8; @pl tcgen05.mma.cta_group::1.kind::f16 [%2], [t], %14, %4, pt;}\n\t"
        "{.reg .b32 t; add.u32 t, %3, 16; @pl tcgen05.mma.cta_group::1.kind::f16 [%2], [t], %15, %4, pt;}\n\t"
        "{.reg .b32 t; add.u32 t, %3, 24; @pl tcgen05.mma.cta_group::1.kind::f16 [%2], [t], %16, %4, pt;}\n\t"
        "@pl tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%6];\n\t"
        "setp.ne.and.b32 pl, %8, 0, pl;\n\t"
        "@pl tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%7];\n\t"
        "and.pred pa, pa, px;\n\tselp.u32 %0, 1, 0, pa;\n\t}"
        : "=r"(ready)
        : "r"(leader), "r"(d), "r"(a), "r"(idesc), "r"(accumulate), "r"(bar_a), "r"(bar_x), "r"(free_x), "r"(next_a),
          "r"(par_a), "r"(next_x), "r"(par_x), "l"(b[0]), "l"(b[1]), "l"(b[2]), "l"(b[3])
        : "memory");
  }
};
template <>
struct MmaStage<8> {
  static __device__ __forceinline__ void issue(uint32_t leader, uint32_t d, uint32_t a, const uint64_t (&b)[8], uint32_t idesc,
                                               uint32_t accumulate, uint32_t bar_a, uint32_t bar_x, uint32_t free_x,
                                               uint32_t next_a, uint32_t par_a, uint32_t next_x, uint32_t par_x,
                                               uint32_t &ready) {
    asm volatile(
        "{\n\t.reg .pred pa, px, pl, pc, pt;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 pa, [%9], %10;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 px, [%11], %12;\n\t"
        "setp.ne.b32 pl, %1, 0;\n\tsetp.ne.b32 pc, %5, 0;\n\tsetp.eq.b32 pt, 0, 0;\n\t"
        "{.reg .b32 t; add.u32 t, %3, 0; @pl tcgen05.mma.cta_group::1.kind::f16 [%2], [t], %13, %4, pc;}\n\t"
        "{.reg .b32 t; add.u32 t, %3, 8; @pl tcgen05.mma.cta_group::1.kind::f16 [%2], [t], %14, %4, pt;}\n\t"
        "{.reg .b32 t; add.u32 t, %3, 16; @pl tcgen05.mma.cta_group::1.kind::f16 [%2], [t], %15, %4, pt;}\n\t"
        "{.reg .b32 t; add.u32 t, %3, 24; @pl tcgen05.mma.cta_group::1.kind::f16 [%2], [t], %16, %4, pt;}\n\t"
        "{.reg .b32 t; add.u32 t, %3, 32; @pl tcgen05.mma.cta_group::1.kind::f16 [%2], [t], %17, %4, pt;}\n\t"
        "{.reg .b32 t; add.u32 t, %3, 40; @pl tcgen05.mma.cta_group::1.kind::f16 [%2], [t], %18, %4, pt;}\n\t"
        "{.reg .b32 t; add.u32 t, %3, 48; @pl tcgen05.mma.cta_group::1.kind::f16 [%2], [t], %19, %4, pt;}\n\t"
        "{.reg .b32 t; add.u32 t, %3, 56; @pl tcgen05.mma.cta_group::1.kind::f16 [%2], [t], %20, %4, pt;}\n\t"
        "@pl tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%6];\n\t"
        "setp.ne.and.b32 pl, %8, 0, pl;\n\t"
        "@pl tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%7];\n\t"
        "and.pred pa, pa, px;\n\tselp.u32 %0, 1, 0, pa;\n\t}"
        : "=r"(ready)
        : "r"(leader), "r"(d), "r"(a), "r"(idesc), "r"(accumulate), "r"(bar_a), "r"(bar_x), "r"(free_x), "r"(next_a),
          "r"(par_a), "r"(next_x), "r"(par_x), "l"(b[0]), "l"(b[1]), "l"(b[2]), "l"(b[3]), "l"(b[4]), "l"(b[5]), "l"(b[6]), "l"(b[7])
        : "memory");
  }
};

template <int NMAX, int KS, int TEAMS, int SLOTS, int XK, int XSTAGES, int PSTAGES, int MODE>
__global__ void __launch_bounds__(threads_for(TEAMS), 1) woq_tcgen05_kernel(const __grid_constant__ CUtensorMap tmap_x,
                                                                  const __grid_constant__ CUtensorMap tmap_x2,
                                                                  const __grid_constant__ CUtensorMap tmap_w,
                                                                  const __grid_constant__ CUtensorMap tmap_s,
                                                                  const __grid_constant__ CUtensorMap tmap_z,
                                                                  const __grid_constant__ TcParams p) {
  using L = SmemLayout<NMAX, KS, TEAMS, SLOTS, XK, XSTAGES, PSTAGES>;
  constexpr bool kAsym = MODE == kAsymBf16 || MODE == kAsymF32;
  constexpr int kScaleDtype = (MODE == kSymF32 || MODE == kAsymF32) ? ZT_F32 : ZT_BF16;
  constexpr int kSPC = kChunkK / KS;                     // stages per chunk
  constexpr int kSPX = XK / KS;                           // stages per activation slot
  static_assert(XK % KS == 0 && kChunkK % XK == 0, "activation slots");
  static_assert(SLOTS % TEAMS == 0, "a slot belongs to one team");
  static_assert(TEAMS % kSPC == 0, "a team takes the same stage of every chunk that it visits");
  constexpr int kTeamsPerChunk = kSPC;
  constexpr uint32_t kACols = KS / 2;                    // tensor-memory columns of a converted stage
  constexpr uint32_t kABase = 2 * NMAX;                  // after the two accumulators
  static_assert(kABase + SLOTS * kACols <= 512, "tensor memory");
  extern __shared__ unsigned char smem_dyn[];
  unsigned char *smem = smem_dyn + ((1024u - (smem_u32(smem_dyn) & 1023u)) & 1023u);
  unsigned char *packed = smem + L::kXRing;
  unsigned char *sc_ring = packed + L::kPackedBytes;
  float *epi_scratch = reinterpret_cast<float *>(sc_ring + L::kScaleBytes);
  uint64_t *full_a = reinterpret_cast<uint64_t *>(sc_ring + L::kScaleBytes + L::kEpiBytes);   // converted
  uint64_t *empty_a = full_a + SLOTS;        // multiplied
  uint64_t *full_x = empty_a + SLOTS;        // activations landed
  uint64_t *empty_x = full_x + XSTAGES;      // multiplied
  uint64_t *full_p = empty_x + XSTAGES;      // packed chunk landed
  uint64_t *empty_p = full_p + PSTAGES;      // packed chunk read by its teams
  uint64_t *tmem_full = empty_p + PSTAGES;   // [2]
  uint64_t *tmem_empty = tmem_full + 2;      // [2]
  uint64_t *last_full = tmem_empty + 2;      // accumulator of the CTA's last segment
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(last_full + 1);

  const int warp = tc::uniform_warp(), lane = threadIdx.x & 31;
  // Programmatic dependent launch: packed weights and scales are read before the wait for the preceding
  // kernel, activations, partial sums and output after it.  The grouped form reads its tile list (made by the
  // routing kernels before it) at once, so it waits first.
  if (p.g_count) grid_dependency_wait();
  const uint32_t n_mt = p.g_count ? (uint32_t)*p.g_count : (uint32_t)p.m_tiles;

  if (threadIdx.x == 0) {
    tc::prefetch_tensormap(&tmap_x);
    tc::prefetch_tensormap(&tmap_x2);
    tc::prefetch_tensormap(&tmap_w);
    if (p.staged_gpc) {
      tc::prefetch_tensormap(&tmap_s);
      if (kAsym) tc::prefetch_tensormap(&tmap_z);
    }
    for (int s = 0; s < SLOTS; ++s) {
      tc::mbar_init(&full_a[s], kTeamWarps);
      tc::mbar_init(&empty_a[s], 1);
    }
    for (int s = 0; s < XSTAGES; ++s) {
      tc::mbar_init(&full_x[s], 1);
      tc::mbar_init(&empty_x[s], 1);
    }
    for (int s = 0; s < PSTAGES; ++s) {
      tc::mbar_init(&full_p[s], 1);
      tc::mbar_init(&empty_p[s], kTeamsPerChunk * kTeamWarps);
    }
    for (int b = 0; b < 2; ++b) {
      tc::mbar_init(&tmem_full[b], 1);
      tc::mbar_init(&tmem_empty[b], kEpiWarps);
    }
    tc::mbar_init(last_full, 1);
    tc::mbar_fence_init();
  }
  if (warp == 1) tc::tmem_alloc(tmem_slot, 512);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  grid_launch_dependents();

  // Every role walks the same segments, chunks and stages.  A stage past the end of K is void: nothing is loaded,
  // converted or multiplied, its barriers complete all the same, so ring positions stay aligned with chunks.
  Work wk(p, n_mt);
  // the producers and the issuer run as whole warps, lane 0 issuing
  const bool leader = tc::elect_one();

  if (warp == kPackedProducer) {
    // ---------------- TMA producer of the packed-weight chunks (with their scales / zero points) ----------------
    {
      const uint32_t full_p0 = smem_u32(full_p), empty_p0 = smem_u32(empty_p);
      const uint32_t packed0 = smem_u32(packed), sc0 = smem_u32(sc_ring);
      const uint32_t chunk_tx = kChunkBytes + (kAsym ? 2u : 1u) * (uint32_t)p.staged_gpc * kBN * (kScaleDtype == ZT_F32 ? 4u : 2u);
      uint32_t s = 0, ph = 1;
      bool ok = true;
      while (ok && wk.next()) {
        const TileInfo t = decode_tile(p, wk.tile, n_mt);
        const int row = t.expert * p.N + t.n0;     // rows of the stacked weight: expert * N + n0
        for (uint32_t c = wk.c0; c < wk.c1; ++c) {
          ok = tc::warp_wait(empty_p0 + s * 8, ph);
          if (!ok) {
            tc::report_timeout(p.status, kStatusProducerTimeout);
            break;
          }
          const uint32_t bar = full_p0 + s * 8;
          const int g0 = t.expert * p.groups + (int)((c * kChunkK) >> (p.gs_log2 & 31));
          tc::expect_tx_if(leader, bar, chunk_tx);
          tc::load_2d_if(leader, packed0 + s * kChunkBytes, &tmap_w, bar, (int)c * (kChunkK / 8), row);
          if (p.staged_gpc) {
            tc::load_2d_if(leader, sc0 + s * kScaleSlotBytes, &tmap_s, bar, t.n0, g0);
            if (kAsym) tc::load_2d_if(leader, sc0 + s * kScaleSlotBytes + kZeroSlotOffset, &tmap_z, bar, t.n0, g0);
          }
          if (++s == PSTAGES) {
            s = 0;
            ph ^= 1;
          }
        }
      }
    }
  } else if (warp == 0) {
    // ---------------- TMA producer of the activation tiles ----------------
    {
      const uint32_t full0 = smem_u32(full_x), empty0 = smem_u32(empty_x), x0 = smem_u32(smem);
      grid_dependency_wait();
      uint32_t s = 0, ph = 1;
      bool ok = true;
      while (ok && wk.next()) {
        const TileInfo t = decode_tile(p, wk.tile, n_mt);
        const bool first = t.rows <= p.x_box;
        const CUtensorMap *map = first ? &tmap_x : &tmap_x2;
        const uint32_t bytes = (uint32_t)(first ? p.x_box : p.x_box2) * (XK / 64) * 128u;
        int k = (int)wk.c0 * kChunkK;
        for (uint32_t i = 0; i < (wk.c1 - wk.c0) * (kChunkK / XK); ++i, k += XK) {
          ok = tc::warp_wait(empty0 + s * 8, ph);
          if (!ok) {
            tc::report_timeout(p.status, kStatusProducerTimeout);
            break;
          }
          const uint32_t bar = full0 + s * 8, dst = x0 + s * L::kXBytes;
          if (k >= p.K) {                     // void
            tc::arrive_if(leader, bar);
          } else {
            tc::expect_tx_if(leader, bar, bytes);
            // 64 k x rows x (XK / 64) in one copy: k past the end of K reads as zeros and is not multiplied
            tc::load_3d_if(leader, dst, map, bar, 0, t.m0, k >> 6);
          }
          if (++s == XSTAGES) {
            s = 0;
            ph ^= 1;
          }
        }
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer ----------------
    {
      bool ok = true;
      const uint64_t d0 = tc::smem_desc_k_sw128(0);
      const uint32_t desc_hi = (uint32_t)(d0 >> 32);
      const uint32_t x_field0 = (uint32_t)d0 | ((smem_u32(smem) & 0x3FFFF) >> 4);
      const uint32_t full_a0 = smem_u32(full_a), empty_a0 = smem_u32(empty_a);
      const uint32_t full_x0 = smem_u32(full_x), empty_x0 = smem_u32(empty_x);
      uint32_t s = 0, ph = 0, xs = 0, xph = 0, local = 0;
      uint32_t ready = 0;
      while (wk.next()) {
        const TileInfo t = decode_tile(p, wk.tile, n_mt);
        const uint32_t buf = local & 1, use = local >> 1;
        ++local;
        const uint32_t idesc = tc::instr_desc(1u, 1u, 1u, kBN, (uint32_t)((t.rows + 15) & ~15));
        ok = ok && tc::warp_wait(smem_u32(&tmem_empty[buf]), (use & 1) ^ 1);
        if (!ok) tc::report_timeout(p.status, kStatusMmaTimeout);
        tc::fence_after_sync();
        const uint32_t d_tmem = tmem_base + buf * NMAX;
        uint32_t accumulate = 0;
        int k = (int)wk.c0 * kChunkK;
        const uint32_t stages = (wk.c1 - wk.c0) * kSPC;
        const uint32_t block = (uint32_t)(t.rows <= p.x_box ? p.x_box : p.x_box2) * 8u;   // 64 k of the tile, in 16 bytes
        for (uint32_t i = 0; i < stages && ok; ++i, k += KS) {
          if (!ready) {
            ok = tc::warp_wait(full_x0 + xs * 8, xph) && tc::warp_wait(full_a0 + s * 8, ph);
            if (!ok) {
              tc::report_timeout(p.status, kStatusMmaTimeout);
              break;
            }
          }
          tc::fence_after_sync();
          const uint32_t a = tmem_base + kABase + s * kACols, bar_a = empty_a0 + s * 8, bar_x = empty_x0 + xs * 8;
          const uint32_t b_lo = x_field0 + xs * (L::kXBytes >> 4) + (i % kSPX) * (KS / 64) * block;
          const int steps = (p.K - k) / 16;                   // K is a multiple of 64; <= 0: void
          const bool free_x = kSPX == 1 || i % kSPX == kSPX - 1;
          if (++s == SLOTS) {
            s = 0;
            ph ^= 1;
          }
          if (free_x && ++xs == XSTAGES) {
            xs = 0;
            xph ^= 1;
          }
          // 16 k: 8 columns of tensor memory, 32 bytes of a 128-byte row of the 64-k block
          if (steps >= KS / 16) {
            uint64_t b[KS / 16];
#pragma unroll
            for (int j = 0; j < KS / 16; ++j) b[j] = tc::smem_desc_from_words(b_lo + (j >> 2) * block + 2 * (j & 3), desc_hi);
            MmaStage<KS / 16>::issue(leader, d_tmem, a, b, idesc, accumulate, bar_a, bar_x, free_x, full_a0 + s * 8, ph,
                                     full_x0 + xs * 8, xph, ready);
          } else {
            if (leader) {
              for (int j = 0; j < steps; ++j)
                tc::mma_f16_ts(d_tmem, a + 8 * j, tc::smem_desc_from_words(b_lo + (j >> 2) * block + 2 * (j & 3), desc_hi), idesc,
                               accumulate | (uint32_t)j);
              tc::mma_commit_addr(bar_a);
              if (free_x) tc::mma_commit_addr(bar_x);
            }
            __syncwarp();
            ready = 0;
          }
          ready = __all_sync(0xffffffffu, ready);
          accumulate = 1;
        }
        if (leader) tc::mma_commit(wk.last() ? last_full : &tmem_full[buf]);
        __syncwarp();
      }
    }
  } else {
  if (warp >= kFirstTeam) {
    // ---------------- conversion teams: a thread converts one weight row of a stage ----------------
    const uint32_t team = (uint32_t)(warp - kFirstTeam) / kTeamWarps;
    const int quarter = warp & 3;                        // tensor-memory lanes this warp may write
    const int row = quarter * 32 + lane;                 // weight row (output column) within the tile
    const uint32_t row_x = row & 7;
    const uint32_t a_addr0 = tmem_base + ((uint32_t)(quarter * 32) << 16) + kABase;
    const uint32_t full_a0 = smem_u32(full_a), empty_a0 = smem_u32(empty_a);
    uint32_t slot = team;                                // of the ring of converted stages
    constexpr int kSub = KS / 32;                        // 32-k pieces of a stage, 16 bytes of packed row each
    // a team takes every kStep-th chunk of the ring order, and in it always the same stage
    constexpr uint32_t kStep = TEAMS / kSPC;
    const uint32_t j = team % kSPC;
    const uint32_t row0 = smem_u32(packed) + row * 128 + (((j * kSub) ^ row_x) << 4);   // piece u: ^ (u << 4)
    // Chunks of this CTA in ring order, and where the next of this team's stages lies in its tile
    uint32_t left = wk.chunks_of_cta();
    const uint32_t skip = team / kSPC;
    uint32_t c = wk.pos - wk.pos / wk.chunks * wk.chunks + skip;
    while (c >= wk.chunks) c -= wk.chunks;
    left = left > skip ? (left - skip + kStep - 1) / kStep : 0;              // visits of this team
    uint32_t ps = skip % PSTAGES, pph = 0;               // packed ring: slot, parity
    uint32_t e_ph = 1;                                   // parity of the slot's "free" barrier
    bool ok = true;

    // one stage: `param()` gives the dequantisation parameters of its 32-k pieces, one after the other
    auto convert_stage = [&](int quads, auto &&param) {
      // also for a void stage: its arrival below must not run ahead of the slot's previous round
      ok = ok && tc::warp_wait(empty_a0 + slot * 8, e_ph);
      tc::fence_after_sync();
      if (ok && quads > 0) {
        // One copy of the conversion code, a 16-byte piece of the row per iteration: the teams are at different
        // places in it, and with a whole stage unrolled they evict one another's instructions.
        const uint32_t src = row0 + ps * kChunkBytes, a_addr = a_addr0 + slot * kACols;
        uint4 w = lds128(src);
#pragma unroll 1
        for (int u = 0; u < quads; ++u) {
          uint32_t out[16];
          const uint4 next = lds128(src ^ (((u + 1) & (kSub - 1)) << 4));
          convert32<MODE>(w, param(), out);
          tc::tmem_st_32x32b_x16(a_addr + 16 * u, out);
          w = next;
        }
      }
      tc::tmem_st_wait();
      tc::fence_before_sync();
      __syncwarp();
      tc::arrive_if(lane == 0, full_a0 + slot * 8);
      tc::arrive_if(lane == 0, smem_u32(&empty_p[ps]));
      slot += TEAMS;
      if (slot >= SLOTS) {
        slot = team;
        e_ph ^= 1;
      }
    };
    auto next_stage = [&]() {
      c += kStep;
      while (c >= wk.chunks) c -= wk.chunks;
      ps += kStep;
      if (ps >= PSTAGES) {
        ps -= PSTAGES;
        pph ^= 1;
      }
    };
    if (p.staged_gpc) {
      // groups are at least 128 k wide: one scale per stage, in the chunk's slot
      const uint32_t sc_off = ((p.staged_gpc == 2 ? (j * KS) >> 7 : 0u) * kBN + row) * (kScaleDtype == ZT_F32 ? 4 : 2);
      for (; left > 0; --left) {
        ok = ok && tc::warp_wait(smem_u32(&full_p[ps]), pph);
        const unsigned char *slot = sc_ring + ps * kScaleSlotBytes + sc_off;
        const DqParam d = dq_param<MODE>(load_as_float(slot, 0, kScaleDtype),
                                         kAsym ? load_as_float(slot + kZeroSlotOffset, 0, kScaleDtype) : 0.f);
        convert_stage(ok ? min(kSub, (p.K - (int)(c * kChunkK + j * KS)) / 32) : 0, [&]() { return d; });
        next_stage();
      }
    } else {
      // groups of 32 or 64 k, of no power of two, or tables that TMA cannot address: scales from global memory, one
      // of this team's stages ahead
      Work fw(p, n_mt);
      int64_t f_base = 0;
      uint32_t f_i = 0, f_n = 0, f_it = 0;               // stage within the segment, stages of it, ring position
      float ns[kSub], nz[kSub];
      auto fetch = [&]() {
        for (;;) {
          if (f_i >= f_n) {
            if (!fw.next()) return;
            const TileInfo t = decode_tile(p, fw.tile, n_mt);
            f_base = (int64_t)t.expert * p.groups * p.N + min(t.n0 + row, p.N - 1);
            f_i = 0;
            f_n = (fw.c1 - fw.c0) * kSPC;
          }
          const uint32_t turn = (team + TEAMS - f_it % TEAMS) % TEAMS;   // stages until this team's turn
          if (f_i + turn < f_n) {
            f_i += turn;
            f_it += turn;
            break;
          }
          f_it += f_n - f_i;
          f_i = f_n;
        }
        const int k = (int)fw.c0 * kChunkK + (int)f_i * KS;
        if (k < p.K) {
          int last = -1;
#pragma unroll
          for (int u = 0; u < kSub; ++u) {
            const int ku = min(k + 32 * u, p.K - 32);
            const int g = p.gs_log2 >= 0 ? (ku >> p.gs_log2) : (ku / p.gs);
            if (g == last) {
              ns[u] = ns[u - (u > 0)];
              if (kAsym) nz[u] = nz[u - (u > 0)];
            } else {
              ns[u] = load_as_float(p.scales, f_base + (int64_t)g * p.N, kScaleDtype);
              if (kAsym) nz[u] = load_as_float(p.zeros, f_base + (int64_t)g * p.N, kScaleDtype);
            }
            last = g;
          }
        }
        ++f_i;
        ++f_it;
      };
      fetch();
      for (; left > 0; --left) {
        DqParam d[kSub];
#pragma unroll
        for (int u = 0; u < kSub; ++u) d[u] = dq_param<MODE>(ns[u], kAsym ? nz[u] : 0.f);
        fetch();
        ok = ok && tc::warp_wait(smem_u32(&full_p[ps]), pph);
        convert_stage(ok ? min(kSub, (p.K - (int)(c * kChunkK + j * KS)) / 32) : 0, [&]() {
          const DqParam first = d[0];
#pragma unroll
          for (int i = 0; i + 1 < kSub; ++i) d[i] = d[i + 1];
          return first;
        });
        next_stage();
      }
    }
    if (!ok && lane == 0) tc::report_timeout(p.status, kStatusConvertTimeout);
  }
  // ---------------- epilogue: the epilogue warps; for a CTA's last segment the conversion warps too ----------------
  // A job is 16 tokens x 32 columns of the accumulator.  The last segment is the part of a launch that nothing
  // overlaps, and by then the conversion teams are idle: with them a 128-token tile is drained by twenty warps
  // instead of four (their scratch lies in the activation ring, which the last MMAs have read).
  grid_dependency_wait();                // output, partial sums and post-op operands are shared with earlier work
  const bool epi_warp = warp < kFirstTeam;
  const uint32_t group = epi_warp ? 0u : 1u + (uint32_t)(warp - kFirstTeam) / kTeamWarps;
  const int quarter = warp & 3;          // tensor-memory lanes 32*quarter .. +31
  float *scratch = epi_warp ? epi_scratch + (warp - 3) * kEpiScratch
                            : reinterpret_cast<float *>(smem) + (warp - kFirstTeam) * kEpiScratch;
  const int sub_row = lane >> 3, col4 = (lane & 7) * 4;   // a lane's token row within a group of 4, its four columns
  // 8-byte accesses: rows of y start on 8-byte boundaries, and so do those of the binary post-op operands
  const bool vec = (p.N & 3) == 0 && (reinterpret_cast<uintptr_t>(p.y) & 7) == 0;
  bool vec_post = vec;
#pragma unroll
  for (int o = 0; o < ZT_MAX_POST_OPS; ++o) vec_post = vec_post && (reinterpret_cast<uintptr_t>(p.post.bufs[o]) & 7) == 0;
  uint32_t local = 0;
  bool ok = true;
  Work wd(p, n_mt);
  while (wd.next()) {
    const bool last = wd.last();
    const uint32_t buf = local & 1, use = local >> 1;
    ++local;
    if (!last && !epi_warp) continue;
    const TileInfo ti = decode_tile(p, wd.tile, n_mt);
    const int nq = ti.n0 + quarter * 32 + col4;           // first of this lane's output columns
    float bias4[4] = {0.f, 0.f, 0.f, 0.f};
    if (p.bias) {
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (nq + e < p.N) bias4[e] = load_as_float(p.bias, nq + e, p.bias_dtype);
    }
    // A tile that spans CTAs cta_first .. cta_last: a CTA's piece goes to its slot 0 when its range starts in this
    // tile, else to its slot 1; only the first CTA's range can start before the tile.
    const bool whole = wd.whole();
    uint32_t cta_first = 0, cta_last = 0, first_slot = 0;
    if (!whole) {
      cta_first = wd.cta_of(wd.tile * wd.chunks);
      cta_last = wd.cta_of(wd.tile * wd.chunks + wd.chunks - 1);
      first_slot = wd.first_of(cta_first) < wd.tile * wd.chunks ? 1u : 0u;
    }
    ok = ok && tc::warp_wait_idle(last ? smem_u32(last_full) : smem_u32(&tmem_full[buf]), last ? 0u : (use & 1));
    if (!ok && lane == 0) tc::report_timeout(p.status, kStatusEpilogueTimeout);
    tc::fence_after_sync();
    const uint32_t t_row = tmem_base + ((uint32_t)(quarter * 32) << 16) + buf * NMAX;
    const uint32_t jobs = (uint32_t)(ti.rows + 15) >> 4;
    const uint32_t job0 = last ? group : 0u, stride = last ? (uint32_t)TEAMS + 1u : 1u;
    const uint32_t mine = jobs > job0 ? (jobs - job0 + stride - 1) / stride : 0u;     // jobs of this warp
    // 16 tokens of the accumulator, transposed through scratch: v[q][e] = token r0 + 4 q, column nq + e
    auto drain = [&](uint32_t job, float (&v)[4][4]) {
      uint32_t r[16];
      tc::tmem_ld_32x32b_x16(t_row + job * 16, r);
      tc::tmem_ld_wait();
#pragma unroll
      for (int j = 0; j < 16; ++j) scratch[j * kEpiRowStride + lane] = __uint_as_float(r[j]);
      __syncwarp();
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const float4 t4 = *reinterpret_cast<const float4 *>(&scratch[(q * 4 + sub_row) * kEpiRowStride + col4]);
        v[q][0] = t4.x;
        v[q][1] = t4.y;
        v[q][2] = t4.z;
        v[q][3] = t4.w;
      }
      __syncwarp();                                      // scratch is rewritten by the next job
    };
    auto piece_of = [&](uint32_t cta, uint32_t job) {
      const uint32_t slot = 2 * cta + (cta == cta_first ? first_slot : 0u);
      return reinterpret_cast<float4 *>(p.partial) + (size_t)((slot * 4 + quarter) * (NMAX / 16) + job) * 128 + lane;
    };
    uint32_t todo = (1u << mine) - 1u;                   // jobs to finish, by position in this warp's list
    if (!whole) {
#pragma unroll 1
      for (uint32_t i = 0; i < mine; ++i) {
        float v[4][4];
        drain(job0 + i * stride, v);
        float4 *dst = piece_of(blockIdx.x, job0 + i * stride);
#pragma unroll
        for (int q = 0; q < 4; ++q) __stcg(dst + q * 32, make_float4(v[q][0], v[q][1], v[q][2], v[q][3]));
      }
      // one fence for all of them (it takes about a microsecond), then a ticket each, a lane per job
      __threadfence();
      __syncwarp();
      bool complete = false;
      if (lane < (int)mine) {
        unsigned int *ticket = p.tickets + (wd.tile * (NMAX / 16) + job0 + lane * stride) * 4 + quarter;
        complete = atomicAdd(ticket, 1u) == cta_last - cta_first;
        if (complete) *ticket = 0;                       // ready for the next launch
      }
      todo = __ballot_sync(0xffffffffu, complete);
      __threadfence();
    }
#pragma unroll 1
    for (; todo; todo &= todo - 1) {
      const uint32_t job = job0 + (uint32_t)(__ffs(todo) - 1) * stride;
      const int r0 = (int)job * 16 + sub_row;            // this lane's tokens of the tile: r0 + 4 q
      const int64_t base0 = (int64_t)(ti.m0 + r0) * p.N + nq, step = (int64_t)4 * p.N;
      // of the lane's four tokens, those that exist (rows past the valid ones belong to nobody, or to the next expert)
      const int live = nq < p.N ? (ti.rows - r0 + 3) >> 2 : 0;
      uint2 operand[2][4];                               // of the first two binary post-ops, requested early
      if (vec_post) {
#pragma unroll
        for (int o = 0; o < 2; ++o)
          if (p.post.bufs[o])
#pragma unroll
            for (int q = 0; q < 4; ++q)
              if (q < live)
                operand[o][q] = *reinterpret_cast<const uint2 *>(reinterpret_cast<const __nv_bfloat16 *>(p.post.bufs[o]) + base0 + q * step);
      }
      float v[4][4];
      if (whole) {
        drain(job, v);
      } else {
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
          for (int e = 0; e < 4; ++e) v[q][e] = 0.f;
#pragma unroll 4
        for (uint32_t cta = cta_first; cta <= cta_last; ++cta) {   // in CTA order, whoever adds
          const float4 *src = piece_of(cta, job);
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const float4 t4 = __ldcg(src + q * 32);
            v[q][0] += t4.x;
            v[q][1] += t4.y;
            v[q][2] += t4.z;
            v[q][3] += t4.w;
          }
        }
      }
#pragma unroll
      for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int e = 0; e < 4; ++e) v[q][e] += bias4[e];
      int b = 0;
#pragma unroll 1
      for (int o = 0; o < p.post.n_ops; ++o) {
        const int id = p.post.ids[o];
        if (id != ZT_POST_MUL && id != ZT_POST_ADD) {
          unary_post16(v, id);
          continue;
        }
        const __nv_bfloat16 *other = reinterpret_cast<const __nv_bfloat16 *>(p.post.bufs[b]);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          float t[4];
          if (vec_post) {
            uint2 raw = b == 0 ? operand[0][q] : operand[1][q];
            if (b >= 2 && q < live) raw = *reinterpret_cast<const uint2 *>(other + base0 + q * step);
            t[0] = __uint_as_float(raw.x << 16);
            t[1] = __uint_as_float(raw.x & 0xffff0000u);
            t[2] = __uint_as_float(raw.y << 16);
            t[3] = __uint_as_float(raw.y & 0xffff0000u);
          } else {
#pragma unroll
            for (int e = 0; e < 4; ++e) t[e] = (q < live && nq + e < p.N) ? __bfloat162float(other[base0 + q * step + e]) : 0.f;
          }
#pragma unroll
          for (int e = 0; e < 4; ++e) v[q][e] = id == ZT_POST_MUL ? v[q][e] * t[e] : v[q][e] + t[e];
        }
        ++b;
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        if (q >= live) continue;
        __nv_bfloat16 *dst = p.y + base0 + q * step;
        if (vec) {
          *reinterpret_cast<uint2 *>(dst) = make_uint2(bf2_pack(v[q][0], v[q][1]), bf2_pack(v[q][2], v[q][3]));
        } else {
#pragma unroll
          for (int e = 0; e < 4; ++e)
            if (nq + e < p.N) dst[e] = __float2bfloat16_rn(v[q][e]);
        }
      }
    }
    if (!last) {
      tc::fence_before_sync();
      __syncwarp();
      tc::arrive_if(lane == 0, smem_u32(&tmem_empty[buf]));
    }
  }
  }

  tc::fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    tc::fence_after_sync();
    tc::tmem_dealloc(tmem_base, 512);
  }
}

// ---- host ----------------------------------------------------------------------------------------
struct MapKey {
  const void *ptr;
  uint64_t inner, rows;
  uint32_t box_rows;
  bool operator==(const MapKey &o) const {
    return ptr == o.ptr && inner == o.inner && rows == o.rows && box_rows == o.box_rows;
  }
};
struct MapKeyHash {
  size_t operator()(const MapKey &k) const {
    return std::hash<const void *>()(k.ptr) ^ (k.inner * 1315423911u) ^ (k.rows << 17) ^ k.box_rows;
  }
};

// Tensor maps, memoised per process.  With `blocks` == 0 a 2-D map [rows, inner] with a (box_rows x box_inner) box;
// otherwise (activations) the same matrix as [inner / box_inner][rows][box_inner] with a (blocks x box_rows x
// box_inner) box, so that one copy brings several 128-byte wide, swizzled column blocks.
int cached_map(CUtensorMap *out, const void *ptr, CUtensorMapDataType dt, uint64_t inner, uint64_t rows,
               uint64_t pitch_bytes, uint32_t box_inner, uint32_t box_rows, bool swizzle = true, uint32_t blocks = 0) {
  static std::mutex mu;
  static std::unordered_map<MapKey, CUtensorMap, MapKeyHash> cache;
  const MapKey key{ptr, inner * 4 + (uint64_t)dt % 4, rows, ((box_rows * 1024 + box_inner) * 2 + (swizzle ? 1u : 0u)) * 8 + blocks};
  std::lock_guard<std::mutex> lock(mu);
  auto it = cache.find(key);
  if (it != cache.end()) {
    *out = it->second;
    return ZT_SUCCESS;
  }
  int rc;
  if (blocks) {
    const uint64_t dims[3] = {box_inner, rows, inner / box_inner}, strides[2] = {pitch_bytes, 128};
    const uint32_t box[3] = {box_inner, box_rows, blocks};
    rc = make_tensor_map(out, ptr, dt, 3, dims, strides, box, swizzle);
  } else {
    const uint64_t dims[2] = {inner, rows}, strides[1] = {pitch_bytes};
    const uint32_t box[2] = {box_inner, box_rows};
    rc = make_tensor_map(out, ptr, dt, 2, dims, strides, box, swizzle);
  }
  if (rc != ZT_SUCCESS) return rc;
  if (cache.size() > 4096) cache.clear();
  cache.emplace(key, *out);
  return ZT_SUCCESS;
}

template <int NMAX, int KS, int TEAMS, int SLOTS, int XK, int XSTAGES, int PSTAGES>
int launch_cfg(const TcParams &p0, int scale_dtype, const void *x, int64_t x_rows, int64_t w_rows, int max_row_tiles,
               cudaStream_t st) {
  using L = SmemLayout<NMAX, KS, TEAMS, SLOTS, XK, XSTAGES, PSTAGES>;
  static_assert(L::kTotal <= 227 * 1024, "rings exceed shared memory");
  TcParams p = p0;
  const bool asym = p.zeros != nullptr;
  CUtensorMap tx, tx2, tw;
  int rc = cached_map(&tx, x, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, (uint64_t)p.K, (uint64_t)x_rows, (uint64_t)p.K * 2, 64,
                      (uint32_t)p.x_box, true, XK / 64);
  if (rc != ZT_SUCCESS) return rc;
  rc = cached_map(&tx2, x, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, (uint64_t)p.K, (uint64_t)x_rows, (uint64_t)p.K * 2, 64,
                  (uint32_t)p.x_box2, true, XK / 64);
  if (rc != ZT_SUCCESS) return rc;
  rc = cached_map(&tw, p.wq, CU_TENSOR_MAP_DATA_TYPE_UINT32, (uint64_t)p.K / 8, (uint64_t)w_rows, (uint64_t)p.K / 2,
                  kChunkK / 8, kBN);
  if (rc != ZT_SUCCESS) return rc;
  // Scales and zero points travel with the packed chunks (one or two groups x 128 columns per chunk) when a
  // group is a power of two of at least 128 k and the tables can be addressed by TMA; otherwise the conversion
  // threads fetch them from global memory.
  CUtensorMap ts = tw, tz = tw;
  p.staged_gpc = 0;
  p.groups = p.K / p.gs;
  p.gs_log2 = -1;
  if ((p.gs & (p.gs - 1)) == 0)
    for (p.gs_log2 = 0; (1 << p.gs_log2) < p.gs;) ++p.gs_log2;
  {
    const uint64_t esz = scale_dtype == ZT_F32 ? 4 : 2;
    const bool aligned = ((uint64_t)p.N * esz) % 16 == 0 && (reinterpret_cast<uintptr_t>(p.scales) & 15) == 0 &&
                         (!asym || (reinterpret_cast<uintptr_t>(p.zeros) & 15) == 0);
    if (p.gs_log2 >= 7 && aligned) {
      p.staged_gpc = p.gs == 128 ? 2 : 1;
      const uint64_t table_rows = (uint64_t)(w_rows / p.N) * (uint64_t)p.groups;   // experts x groups
      const CUtensorMapDataType sdt = scale_dtype == ZT_F32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
      rc = cached_map(&ts, p.scales, sdt, (uint64_t)p.N, table_rows, (uint64_t)p.N * esz, kBN, (uint32_t)p.staged_gpc, false);
      if (rc != ZT_SUCCESS) return rc;
      if (asym) {
        rc = cached_map(&tz, p.zeros, sdt, (uint64_t)p.N, table_rows, (uint64_t)p.N * esz, kBN, (uint32_t)p.staged_gpc, false);
        if (rc != ZT_SUCCESS) return rc;
      }
    }
  }
  const int64_t tiles = (int64_t)(p.g_count ? max_row_tiles : p.m_tiles) * p.n_tiles;
  const int sms = sm_count();
  const dim3 grid(p.split ? (unsigned)p.split : (unsigned)(tiles < sms ? tiles : sms));
  // every instantiation needs its own once-per-device attribute set-up
  static PerDeviceOnce configured[4];
  auto launch = [&](auto kern, int which) -> int {
    if (int rc_cfg = allow_dynamic_smem(configured[which], kern, L::kTotal)) return rc_cfg;
    ZT_CUDA_OK(launch_overlapped(kern, grid, dim3(threads_for(TEAMS)), (size_t)L::kTotal, st, tx, tx2, tw, ts, tz, p));
    return launch_status("woq_tcgen05_kernel");
  };
  if (scale_dtype == ZT_F32)
    return asym ? launch(woq_tcgen05_kernel<NMAX, KS, TEAMS, SLOTS, XK, XSTAGES, PSTAGES, kAsymF32>, kAsymF32)
                : launch(woq_tcgen05_kernel<NMAX, KS, TEAMS, SLOTS, XK, XSTAGES, PSTAGES, kSymF32>, kSymF32);
  return asym ? launch(woq_tcgen05_kernel<NMAX, KS, TEAMS, SLOTS, XK, XSTAGES, PSTAGES, kAsymBf16>, kAsymBf16)
              : launch(woq_tcgen05_kernel<NMAX, KS, TEAMS, SLOTS, XK, XSTAGES, PSTAGES, kSymBf16>, kSymBf16);
}

// `cap`: the instantiation's largest token tile
int launch_any(int cap, const TcParams &p, int scale_dtype, const void *x, int64_t x_rows, int64_t w_rows,
               int max_row_tiles, cudaStream_t st) {
  switch (cap) {
    // <token tile, k per stage, conversion teams, converted slots, k per activation slot, activation slots, packed chunks>
    case 32: return launch_cfg<32, 128, 6, 6, 256, 5, 6>(p, scale_dtype, x, x_rows, w_rows, max_row_tiles, st);
    case 64: return launch_cfg<64, 128, 6, 6, 256, 3, 6>(p, scale_dtype, x, x_rows, w_rows, max_row_tiles, st);
    case 128: return launch_cfg<128, 128, 4, 4, 128, 4, 4>(p, scale_dtype, x, x_rows, w_rows, max_row_tiles, st);
    case 192: return launch_cfg<192, 64, 4, 4, 64, 5, 4>(p, scale_dtype, x, x_rows, w_rows, max_row_tiles, st);
    default: break;
  }
  set_error("zt_woq_linear: unsupported token-tile width %d for the tcgen05 kernel", cap);
  return ZT_UNSUPPORTED;
}

// Row tiling and work split of a dense call.
struct DensePlan {
  int cap;       // instantiation
  int m_tiles, bt;
  int split;     // CTAs that share the chunks of all tiles; 0 = whole tiles
};
int cap_for(int64_t rows) { return rows <= 32 ? 32 : rows <= 64 ? 64 : rows <= 128 ? 128 : 192; }

// The number of row tiles, and whether the chunks of all tiles are shared out, by estimated cycles.  A 128 x 64 block
// takes the slower of the conversion pipeline (about 300 cycles measured) and the MMAs (2 per token, and about 90
// around them).  Sharing out costs about 20,000 cycles at the end of the launch (pieces to L2, fence, tickets, the
// addition; 10,000 - 21,000 measured), so it pays for few tiles with a long K only: M = 32, 4096 -> 14336 takes 13.7 us
// with whole tiles on 112 SMs and 16.6 shared by 148; M = 64, 4096 -> 4096 12.5 and 15.7.
DensePlan dense_plan(int64_t M, int64_t N, int64_t K, int hint, bool may_split) {
  const int sms = sm_count();
  const int64_t n_tiles = ceil_div<int64_t>(N, kBN), chunks = ceil_div<int64_t>(K, kChunkK);
  const int64_t limit = hint > 0 ? std::min(hint, 192) : 192;
  const int64_t first = ceil_div<int64_t>(M, limit);
  DensePlan best{};
  double best_cost = 1e300;
  for (int64_t mt = first; mt <= first + first / 2 + (hint > 0 ? 0 : 1) && mt <= ceil_div<int64_t>(M, 16); ++mt) {
    const int64_t bt = ceil_div<int64_t>(ceil_div(M, mt), 16) * 16, tiles_m = ceil_div(M, bt);
    const int64_t tiles = tiles_m * n_tiles;
    const double chunk = 4.0 * std::max(300.0, 2.0 * (double)bt + 90.0);
    double cost = (double)ceil_div<int64_t>(tiles, sms) * chunks * chunk;
    int split = 0;
    if (may_split && tiles * (cap_for(bt) / 4) <= kTickets) {
      // at least two chunks per CTA, at most sixteen CTAs per tile
      const int64_t ctas = std::min<int64_t>({(int64_t)sms, tiles * 16, std::max<int64_t>(tiles * chunks / 2, 1)});
      const double c = (double)(tiles * chunks) / ctas * chunk + 20000.0;
      if (ctas > 1 && c < cost) {
        cost = c;
        split = (int)ctas;
      }
    }
    if (cost < best_cost) {
      best_cost = cost;
      best = {cap_for(bt), (int)tiles_m, (int)bt, split};
    }
  }
  return best;
}
size_t split_bytes(const DensePlan &d) {
  return d.split ? (size_t)d.split * 2 * kBN * d.cap * sizeof(float) : 0;
}

}  // namespace

size_t woq_tcgen05_workspace_bytes(int64_t M, int64_t N, int64_t K) { return split_bytes(dense_plan(M, N, K, 0, true)); }

bool woq_tcgen05_supported(const zt_woq_linear_args_t &a) {
  if (a.M < 1 || a.N < 1 || a.K < 64 || a.K % 64 != 0) return false;
  if (a.n_groups <= 0 || a.K % a.n_groups != 0) return false;
  const int64_t gs = a.K / a.n_groups;
  if (gs % 32 != 0) return false;
  if ((reinterpret_cast<uintptr_t>(a.x) | reinterpret_cast<uintptr_t>(a.wq)) & 15) return false;
  return a.M <= (1 << 30) && a.N <= (1 << 30) && a.K <= (1 << 30);
}

int woq_tcgen05_launch(const zt_woq_linear_args_t &a, cudaStream_t st) {
  TcParams p{};
  p.M = (int)a.M;
  p.N = (int)a.N;
  p.K = (int)a.K;
  p.gs = (int)(a.K / a.n_groups);
  p.wq = a.wq;
  p.scales = a.scales;
  p.zeros = a.zeros;
  p.bias = a.bias;
  p.bias_dtype = a.bias_dtype;
  p.y = reinterpret_cast<__nv_bfloat16 *>(a.y);
  p.post = to_dev(a.post);
  p.status = device_status_ptr();
  const int hint = (a.algo >> 8) & 0xffff;
  ZT_REQUIRE(hint == 0 || hint == 32 || hint == 64 || hint == 128 || hint == 256, ZT_UNSUPPORTED,
             "zt_woq_linear: unsupported token-tile width %d for the tcgen05 kernel", hint);
  const bool may_split = hint == 0 && !(a.algo & ZT_ALGO_SINGLE_ISSUER) && a.workspace != nullptr;
  DensePlan d = dense_plan(a.M, a.N, a.K, hint, may_split);
  if (d.split && a.workspace_bytes < ZT_WOQ_COUNTER_BYTES + split_bytes(d)) d = dense_plan(a.M, a.N, a.K, hint, false);
  p.m_tiles = d.m_tiles;
  p.n_tiles = (int)ceil_div<int64_t>(a.N, kBN);
  p.bt = d.bt;
  p.chunks = (int)ceil_div<int64_t>(a.K, kChunkK);
  p.x_box = p.x_box2 = d.m_tiles == 1 ? (int)ceil_div<int64_t>(a.M, 8) * 8 : d.bt;   // 128-byte swizzle: 8-row atoms
  p.split = d.split;
  p.tickets = reinterpret_cast<unsigned int *>(a.workspace);
  p.partial = d.split ? reinterpret_cast<float *>(reinterpret_cast<char *>(a.workspace) + ZT_WOQ_COUNTER_BYTES) : nullptr;
  return launch_any(d.cap, p, a.scale_dtype, a.x, a.M, a.N, 0, st);
}

// Grouped form for mixture-of-experts: `x` holds `total_rows` rows sorted by expert; `tiles` / `tile_count`
// (device memory) list the row tiles of at most `row_tile` rows; weights and scales are stacked per expert.
int woq_tcgen05_grouped_launch(const void *x, int64_t total_rows, int64_t N, int64_t K, const int32_t *wq,
                               const void *scales, int scale_dtype, int64_t n_groups, int num_experts, void *y,
                               const int *tile_count, const int4 *tiles, int max_row_tiles, int row_tile, cudaStream_t st) {
  TcParams p{};
  p.M = (int)total_rows;
  p.N = (int)N;
  p.K = (int)K;
  p.gs = (int)(K / n_groups);
  p.wq = wq;
  p.scales = scales;
  p.bias_dtype = ZT_BF16;
  p.y = reinterpret_cast<__nv_bfloat16 *>(y);
  p.status = device_status_ptr();
  p.n_tiles = (int)ceil_div<int64_t>(N, kBN);
  p.bt = row_tile;
  p.chunks = (int)ceil_div<int64_t>(K, kChunkK);
  p.x_box = row_tile > 64 ? 64 : row_tile;
  p.x_box2 = row_tile;
  p.g_count = tile_count;
  p.g_tiles = tiles;
  return launch_any(cap_for(row_tile), p, scale_dtype, x, total_rows, (int64_t)num_experts * N, max_row_tiles, st);
}

}  // namespace zt
