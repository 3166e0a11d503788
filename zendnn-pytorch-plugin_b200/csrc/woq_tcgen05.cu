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
//   warps 3..6    epilogue: tcgen05.ld (lane = output column n, register j = token), the sum of a tile's accumulators, bias +
//                 post-ops, bf16 stores of 64 contiguous bytes per token
//   warps 7..     conversion, teams of four warps; team t of T takes the ring positions congruent to t mod T; then,
//                 idle, they help with the epilogue of the CTA's last tile
//
// What bounds it.  Converting a 128 x 64 block costs its SM about 200 cycles of the two half-rate pipes (per packed word
// of eight weights 9 shift / permute / lop3 operations on one and 8 - 12 bf16x2 operations on the other); its MMAs take 2
// cycles per token and at least 128.  A block takes 300 - 350 cycles up to 64 tokens and 350 - 450 up to 128 (650 when the
// converted operand went through shared memory and the issuing threads ran divergent code); per call, M = 32 on 4096 -> 14336:
// 21.6 -> 14.8 us, M = 128 on 8192 -> 8192 with two operands: 39.4 -> 24.9 us, M = 2048 on 4096 -> 14336: 263 -> 217 us (0.67 of the
// bf16 peak; from 128 tokens on an SM pulls 35 bytes per cycle of activations and weights out of L2, which is what it can
// get).  What that took:
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
// Work split.  An item is a tile, or a slice of its K (whole chunks) where there are fewer tiles than SMs or a shorter sum is
// wanted (see min_sums and dense_plan).  The slices' fp32 sums are added in order, so results do not depend on timing: by a
// cluster through its shared memory, or by a second kernel through the workspace (see launch_cfg).  Without slices the layers
// of few tiles leave most SMs idle: M = 17 on 4096 -> 4096 took 12.8 us on 32 SMs and takes 7.9 in four slices.  The slices used to
// meet at the end of this kernel by tickets, which cost 5 - 10 us and so was hardly ever worth it.
//
// Sums.  The tensor core's fp32 accumulation truncates, so its error grows with the length of the sum: tiles of up to 128 rows
// are therefore summed in two accumulators, one for each parity of the 64-k blocks, which the epilogue adds.
//
// Grouped mode (mixture-of-experts): the rows of X are sorted by expert, a device-side table lists the row tiles
// {expert, first row, valid rows}, and each tile uses its expert's slice of the stacked weight and scale tensors;
// the number of tiles is read from device memory, so no host synchronisation is needed between routing and GEMM.
//
// Accumulators are double buffered in tensor memory as far as they fit (see Accumulators).  All waits are bounded (see
// tc05.cuh).
//
// Rounding.  q (an integer in [-8, 7]) is exact in bf16.  With bf16 scales q*s is one bf16x2 multiplication, i.e.
// exactly bf16(q*s), and (q-8)*s + z one bf16x2 fma, rounded once.  With fp32 scales s is split into s_hi + s_lo
// (both bf16) and dq = fma(q, s_hi, q*s_lo), which equals bf16(q*s) except for rare double-rounding cases one bf16
// ulp apart; the zero-point form is evaluated in fp32 and rounded once.
#include <algorithm>
#include <atomic>
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
constexpr int kChunkK = 256;        // k per packed chunk: one 128-byte row of nibbles
constexpr int kChunkBytes = kBN * 128;
// per packed chunk: up to eight groups x 128 columns of scales, then the same for zero points (8 KB when both are fp32; where
// the activation ring leaves no room for that, tables that need more than 4 KB are read from global memory)
__host__ __device__ constexpr int scale_slot_bytes(int nmax) { return nmax == 64 ? 4096 : 8192; }
constexpr int kMaxSlices = 32;      // K slices of a tile
constexpr int kMaxCluster = 8;      // of them added by a cluster (the portable size)

// How a weight is dequantised (template parameter of the kernel).
enum DqMode { kSymF32 = 0, kSymBf16 = 1, kAsymBf16 = 2, kAsymF32 = 3 };

struct TcParams {
  int M, N, K;
  int m_tiles, n_tiles, bt;   // dense mode: row tiles of bt tokens
  int chunks, slices;         // per tile: chunks of K, and the slices that share them
  int accs;                   // accumulators of a tile: 2 = one for each parity of the 64-k blocks, added by the epilogue
  int x_box, x_box2;          // rows of the activation box: the first when the tile's rows fit, else the second
  int gs, gs_log2;            // gs_log2 < 0: not a power of two
  const int32_t *wq;
  const void *scales;
  const void *zeros;
  const void *bias;
  int bias_dtype;
  __nv_bfloat16 *y;
  PostOpsDev post;
  int *status;
  int cluster;                // slices > 1: a tile's slices are a cluster, which adds them through shared memory ...
  float *partial;             // ... or else their sums [slices][M][N rounded up to 4], which woq_slices_kernel adds
  // grouped mode (g_count != nullptr)
  const int *g_count;         // number of row tiles
  const int4 *g_tiles;        // per row tile: {expert, first row, valid rows, 0}
  // Scales (and zero points) staged in shared memory with every packed chunk: groups per chunk (1 .. 8; 0 = the
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

// The work of a CTA: every gridDim.x-th item, an item being a slice of K of a tile.
struct Work {
  uint32_t item, items, chunks, slices;
  uint32_t tile, slice, c0, c1;   // current item: chunks [c0, c1) of `tile`

  __device__ __forceinline__ Work(const TcParams &p, uint32_t n_mt)
      : item(blockIdx.x), items(n_mt * (uint32_t)p.n_tiles * (uint32_t)p.slices), chunks((uint32_t)p.chunks), slices((uint32_t)p.slices) {}
  __device__ __forceinline__ bool next() {
    if (item >= items) return false;
    tile = item / slices;
    slice = item - tile * slices;
    c0 = slice * chunks / slices;
    c1 = (slice + 1) * chunks / slices;
    item += gridDim.x;
    return true;
  }
  __device__ __forceinline__ bool last() const { return item >= items; }     // of the item that next() has set
};

// The accumulators of consecutive tiles.  Two sets take turns, so that a tile is summed while the one before it is drained;
// a tile of two accumulators that are wider than half a set (`wide`) takes both sets.
template <int NMAX>
struct Accumulators {
  static constexpr uint32_t kCount = NMAX <= 32 ? 4 : 2, kSetCols = kCount / 2 * NMAX;
  uint32_t turn = 0, used[2] = {0, 0};
  uint32_t set, use;              // of the current tile; use: how often the set was used before
  uint32_t col, second;           // first column, distance of the second accumulator
  bool wide;
  __device__ __forceinline__ void next(bool two, int rows) {
    wide = two && (kCount == 2 && rows > NMAX / 2);
    set = wide ? 0u : turn;
    turn = wide ? 0u : turn ^ 1;
    use = set ? used[1]++ : used[0]++;
    col = set * kSetCols;
    second = !two ? 0u : kCount == 4 || wide ? (uint32_t)NMAX : (uint32_t)NMAX / 2;
  }
};

template <int NMAX, int KS, int TEAMS, int SLOTS, int XK, int XSTAGES, int PSTAGES>
struct SmemLayout {
  static constexpr int kXBytes = (XK / 64) * NMAX * 128;
  static constexpr int kXRing = XSTAGES * kXBytes;
  static constexpr int kPackedBytes = PSTAGES * kChunkBytes;
  static constexpr int kScaleBytes = PSTAGES * scale_slot_bytes(NMAX);
  static constexpr int kBarBytes = (2 * SLOTS + 2 * XSTAGES + 2 * PSTAGES + 5) * 8 + 8;
  static_assert(NMAX * kBN * 4 <= kXRing, "sums of a slice");
  static constexpr int kTotal = kXRing + kPackedBytes + kScaleBytes + kBarBytes + 1024;
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
      const uint32_t w = words[i], high = w >> 20;
      float f[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        // a nibble where it lies, as 2^23 + 16^j q; times 16^-j and without the offset it is q - 8, exactly
        const int j = e < 5 ? e : e - 5;
        const uint32_t bits = ((e < 5 ? w : high) & (0xFu << (4 * j))) | 0x4B000000u;
        const float unit = 1.0f / (float)(1 << (4 * j));
        f[e] = fmaf(fmaf(__uint_as_float(bits), unit, -8388608.0f * unit - 8.0f), __uint_as_float(d.a), __uint_as_float(d.b));
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

// One unary post-op on a thread's 16 values; the switch is outside the element loop so that its code exists once.  The two
// short ones are unrolled; the others go through four values at a time, because fetching a long straight run of code
// that is executed once takes longer than the loop.
__device__ __forceinline__ void unary_post16(float (&v)[16], int id) {
  if (id == ZT_POST_RELU) {
#pragma unroll
    for (int j = 0; j < 16; ++j) v[j] = unary_post(v[j], ZT_POST_RELU);
    return;
  }
  if (id == ZT_POST_SILU) {
#pragma unroll
    for (int j = 0; j < 16; ++j) v[j] = unary_post(v[j], ZT_POST_SILU);
    return;
  }
#pragma unroll 1
  for (int q = 0; q < 4; ++q) {
    // the first four, then rotate: after four rounds every value is back in its place
    float w[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) w[e] = unary_post(v[e], id);
#pragma unroll
    for (int e = 0; e < 12; ++e) v[e] = v[e + 4];
#pragma unroll
    for (int e = 0; e < 4; ++e) v[12 + e] = w[e];
  }
}

// The MMAs of one stage, 16 k each: A at consecutive columns of tensor memory, B by descriptor, the second 64 k into the
// accumulator `d2`; then the commits that
// free the converted slot and, when `free_x`, the activation slot.  Issued by the lane whose `leader` is set.  A completed
// barrier wait takes its thread about 200 cycles, a third of a stage, so the barriers of the next stage are
// tested in the same straight line of code: their answer arrives while the MMAs are being issued.
template <int N>
struct MmaStage;
template <>
struct MmaStage<4> {
  static __device__ __forceinline__ void issue(uint32_t leader, uint32_t d, uint32_t, uint32_t a, const uint64_t (&b)[4],
                                               uint32_t idesc, uint32_t accumulate, uint32_t, uint32_t bar_a, uint32_t bar_x, uint32_t free_x,
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
  static __device__ __forceinline__ void issue(uint32_t leader, uint32_t d, uint32_t d2, uint32_t a, const uint64_t (&b)[8],
                                               uint32_t idesc, uint32_t accumulate, uint32_t accumulate2, uint32_t bar_a, uint32_t bar_x, uint32_t free_x,
                                               uint32_t next_a, uint32_t par_a, uint32_t next_x, uint32_t par_x,
                                               uint32_t &ready) {
    asm volatile(
        "{\n\t.reg .pred pa, px, pl, pc, pt, pd;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 pa, [%9], %10;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 px, [%11], %12;\n\t"
        "setp.ne.b32 pl, %1, 0;\n\tsetp.ne.b32 pc, %5, 0;\n\tsetp.eq.b32 pt, 0, 0;\n\t"
        "setp.ne.b32 pd, %22, 0;\n\t"
        "{.reg .b32 t; add.u32 t, %3, 0; @pl tcgen05.mma.cta_group::1.kind::f16 [%2], [t], %13, %4, pc;}\n\t"
        "{.reg .b32 t; add.u32 t, %3, 8; @pl tcgen05.mma.cta_group::1.kind::f16 [%2], [t], %14, %4, pt;}\n\t"
        "{.reg .b32 t; add.u32 t, %3, 16; @pl tcgen05.mma.cta_group::1.kind::f16 [%2], [t], %15, %4, pt;}\n\t"
        "{.reg .b32 t; add.u32 t, %3, 24; @pl tcgen05.mma.cta_group::1.kind::f16 [%2], [t], %16, %4, pt;}\n\t"
        "{.reg .b32 t; add.u32 t, %3, 32; @pl tcgen05.mma.cta_group::1.kind::f16 [%21], [t], %17, %4, pd;}\n\t"
        "{.reg .b32 t; add.u32 t, %3, 40; @pl tcgen05.mma.cta_group::1.kind::f16 [%21], [t], %18, %4, pt;}\n\t"
        "{.reg .b32 t; add.u32 t, %3, 48; @pl tcgen05.mma.cta_group::1.kind::f16 [%21], [t], %19, %4, pt;}\n\t"
        "{.reg .b32 t; add.u32 t, %3, 56; @pl tcgen05.mma.cta_group::1.kind::f16 [%21], [t], %20, %4, pt;}\n\t"
        "@pl tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%6];\n\t"
        "setp.ne.and.b32 pl, %8, 0, pl;\n\t"
        "@pl tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%7];\n\t"
        "and.pred pa, pa, px;\n\tselp.u32 %0, 1, 0, pa;\n\t}"
        : "=r"(ready)
        : "r"(leader), "r"(d), "r"(a), "r"(idesc), "r"(accumulate), "r"(bar_a), "r"(bar_x), "r"(free_x), "r"(next_a),
          "r"(par_a), "r"(next_x), "r"(par_x), "l"(b[0]), "l"(b[1]), "l"(b[2]), "l"(b[3]), "l"(b[4]), "l"(b[5]), "l"(b[6]), "l"(b[7]),
          "r"(d2), "r"(accumulate2)
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
  constexpr uint32_t kScaleSlot = scale_slot_bytes(NMAX), kScaleSize = kScaleDtype == ZT_F32 ? 4 : 2;
  constexpr int kSPX = XK / KS;                           // stages per activation slot
  static_assert(XK % KS == 0 && kChunkK % XK == 0, "activation slots");
  static_assert(SLOTS % TEAMS == 0, "a slot belongs to one team");
  static_assert(TEAMS % kSPC == 0, "a team takes the same stage of every chunk that it visits");
  constexpr int kTeamsPerChunk = kSPC;
  constexpr uint32_t kACols = KS / 2;                    // tensor-memory columns of a converted stage
  constexpr bool kTwoAccs = KS == 128;                   // may sum a tile in two accumulators, a stage's halves in one each
  constexpr uint32_t kABase = Accumulators<NMAX>::kCount * NMAX;   // the converted stages follow the accumulators
  static_assert(kABase + SLOTS * kACols <= 512, "tensor memory");
  extern __shared__ unsigned char smem_dyn[];
  unsigned char *smem = smem_dyn + ((1024u - (smem_u32(smem_dyn) & 1023u)) & 1023u);
  unsigned char *packed = smem + L::kXRing;
  unsigned char *sc_ring = packed + L::kPackedBytes;
  uint64_t *full_a = reinterpret_cast<uint64_t *>(sc_ring + L::kScaleBytes);   // converted
  uint64_t *empty_a = full_a + SLOTS;        // multiplied
  uint64_t *full_x = empty_a + SLOTS;        // activations landed
  uint64_t *empty_x = full_x + XSTAGES;      // multiplied
  uint64_t *full_p = empty_x + XSTAGES;      // packed chunk landed
  uint64_t *empty_p = full_p + PSTAGES;      // packed chunk read by its teams
  uint64_t *tmem_full = empty_p + PSTAGES;   // [2]
  uint64_t *tmem_empty = tmem_full + 2;      // [2]
  uint64_t *last_full = tmem_empty + 2;      // accumulator of the CTA's last item
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

  // Every role walks the same items, chunks and stages.  A stage past the end of K is void: nothing is loaded,
  // converted or multiplied, its barriers complete all the same, so ring positions stay aligned with chunks.
  Work wk(p, n_mt);
  const bool two = kTwoAccs && p.accs == 2;
  // the producers and the issuer run as whole warps, lane 0 issuing
  const bool leader = tc::elect_one();

  if (warp == kPackedProducer) {
    // ---------------- TMA producer of the packed-weight chunks (with their scales / zero points) ----------------
    {
      const uint32_t full_p0 = smem_u32(full_p), empty_p0 = smem_u32(empty_p);
      const uint32_t packed0 = smem_u32(packed), sc0 = smem_u32(sc_ring);
      const uint32_t chunk_tx = kChunkBytes + (kAsym ? 2u : 1u) * (uint32_t)p.staged_gpc * kBN * kScaleSize;
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
            tc::load_2d_if(leader, sc0 + s * kScaleSlot, &tmap_s, bar, t.n0, g0);
            if (kAsym) tc::load_2d_if(leader, sc0 + s * kScaleSlot + (uint32_t)p.staged_gpc * kBN * kScaleSize, &tmap_z, bar, t.n0, g0);
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
      uint32_t s = 0, ph = 0, xs = 0, xph = 0;
      Accumulators<NMAX> acc;
      uint32_t ready = 0;
      while (wk.next()) {
        const TileInfo t = decode_tile(p, wk.tile, n_mt);
        acc.next(two, t.rows);
        const uint32_t idesc = tc::instr_desc(1u, 1u, 1u, kBN, (uint32_t)((t.rows + 15) & ~15));
        ok = ok && tc::warp_wait(smem_u32(&tmem_empty[acc.set]), (acc.use & 1) ^ 1);
        if (acc.wide) ok = ok && tc::warp_wait(smem_u32(&tmem_empty[1]), (acc.used[1] & 1) ^ 1);
        if (!ok) tc::report_timeout(p.status, kStatusMmaTimeout);
        tc::fence_after_sync();
        const uint32_t d_tmem = tmem_base + acc.col, d_tmem2 = d_tmem + acc.second;
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
            MmaStage<KS / 16>::issue(leader, d_tmem, d_tmem2, a, b, idesc, accumulate, two ? accumulate : 1u, bar_a, bar_x, free_x,
                                     full_a0 + s * 8, ph, full_x0 + xs * 8, xph, ready);
          } else {                            // the end of K: the first 64 k of the stage at most
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
        if (leader) tc::mma_commit(wk.last() ? last_full : &tmem_full[acc.set]);
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
    uint32_t c = team / kSPC, end = 0;                   // this team's next chunk, end of the item it is counted in
    auto next_chunk = [&]() {
      while (c >= end) {
        if (!wk.next()) return false;
        c += wk.c0 - end;
        end = wk.c1;
      }
      return true;
    };
    uint32_t ps = c % PSTAGES, pph = 0;                  // packed ring: slot, parity
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
      ps += kStep;
      if (ps >= PSTAGES) {
        ps -= PSTAGES;
        pph ^= 1;
      }
    };
    if (p.staged_gpc) {
      // the group of a 32-k piece: its k within the chunk >> log2 of the group size (one group, if that is larger)
      const uint32_t zero_off = (uint32_t)p.staged_gpc * kBN * kScaleSize, shift = p.staged_gpc == 1 ? 31u : (uint32_t)p.gs_log2;
      for (; next_chunk(); c += kStep) {
        ok = ok && tc::warp_wait(smem_u32(&full_p[ps]), pph);
        const unsigned char *slot = sc_ring + ps * kScaleSlot + row * kScaleSize;
        uint32_t k = j * KS;
        auto group_param = [&]() {
          const unsigned char *at = slot + (k >> shift) * (kBN * kScaleSize);
          return dq_param<MODE>(load_as_float(at, 0, kScaleDtype), kAsym ? load_as_float(at + zero_off, 0, kScaleDtype) : 0.f);
        };
        const int quads = ok ? min(kSub, (p.K - (int)(c * kChunkK + j * KS)) / 32) : 0;
        if (p.gs_log2 >= 7) {                            // one group per stage
          const DqParam d = group_param();
          convert_stage(quads, [&]() { return d; });
        } else {
          convert_stage(quads, [&]() {
            const DqParam d = group_param();
            k += 32;
            return d;
          });
        }
        next_stage();
      }
    } else {
      // groups of no power of two, or tables that TMA cannot address or that do not fit: scales from global memory, one of
      // this team's stages ahead
      Work fw(p, n_mt);
      int64_t f_base = 0;
      uint32_t f_i = 0, f_n = 0, f_it = 0;               // stage within the item, stages of it, ring position
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
      for (; next_chunk(); c += kStep) {
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
  // ---------------- epilogue: the epilogue warps; for a CTA's last item the conversion warps too ----------------
  // A job is 16 tokens x 32 columns of the accumulator; a lane holds one column, so that loads and stores of a token's
  // outputs are 64 contiguous bytes (as wide as a transposition through shared memory makes them, which cost 20 more
  // shared-memory accesses and two barriers per job).  The last item is the part of a launch that nothing
  // overlaps, and by then the conversion teams are idle: with them a 128-token tile is drained by twenty warps
  // instead of four.
  grid_dependency_wait();                // output, partial sums and post-op operands are shared with earlier work
  const bool epi_warp = warp < kFirstTeam;
  const uint32_t group = epi_warp ? 0u : 1u + (uint32_t)(warp - kFirstTeam) / kTeamWarps;
  const int quarter = warp & 3;          // tensor-memory lanes 32*quarter .. +31
  Accumulators<NMAX> acc;
  bool ok = true;
  Work wd(p, n_mt);
  while (wd.next()) {
    const bool last = wd.last();
    const TileInfo ti = decode_tile(p, wd.tile, n_mt);
    acc.next(two, ti.rows);
    if (!last && !epi_warp) continue;
    const int n = ti.n0 + quarter * 32 + lane;            // this lane's output column
    const bool live = n < p.N;
    const float bias = p.bias && !p.partial && live ? load_as_float(p.bias, n, p.bias_dtype) : 0.f;
    // operands of the first two binary post-ops for a job (two tokens' bf16 to a register), fetched before its sums are awaited
    uint32_t operand[2][8];
    auto request = [&](int job) {
      const int rows = live ? min(16, ti.rows - job * 16) : 0;
#pragma unroll
      for (int o = 0; o < 2; ++o) {
        const uint16_t *src = reinterpret_cast<const uint16_t *>(p.post.bufs[o]);
        if (!src) continue;
        src += (int64_t)(ti.m0 + job * 16) * p.N + n;
#pragma unroll
        for (int j = 0; j < 16; j += 2, src += 2 * (int64_t)p.N)
          operand[o][j / 2] = (j < rows ? (uint32_t)src[0] : 0u) | (j + 1 < rows ? (uint32_t)src[p.N] << 16 : 0u);
      }
    };
    const bool with_operands = p.post.bufs[0] != nullptr && !p.partial;
    // bias, post-ops and store of a job's sums
    auto finish = [&](int job, float (&v)[16]) {
      // rows past the valid ones belong to nobody, or to the next expert
      const int rows = live ? min(16, ti.rows - job * 16) : 0;
      const int64_t at = (int64_t)(ti.m0 + job * 16) * p.N + n;
#pragma unroll
      for (int j = 0; j < 16; ++j) v[j] += bias;
      int b = 0;
#pragma unroll 1
      for (int o = 0; o < p.post.n_ops; ++o) {
        const int id = p.post.ids[o];
        if (id != ZT_POST_MUL && id != ZT_POST_ADD) {
          unary_post16(v, id);
          continue;
        }
        const uint16_t *src = b < 2 ? nullptr : reinterpret_cast<const uint16_t *>(p.post.bufs[b]) + at;
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          const uint32_t pair = b == 0 ? operand[0][j / 2] : operand[1][j / 2];
          float t = __uint_as_float(j % 2 ? pair & 0xffff0000u : pair << 16);
          if (src && j < rows) t = bf16_bits_to_float(src[(int64_t)j * p.N]);
          v[j] = id == ZT_POST_MUL ? v[j] * t : v[j] + t;
        }
        ++b;
      }
      __nv_bfloat16 *dst = p.y + at;
#pragma unroll
      for (int j = 0; j < 16; ++j, dst += p.N)
        if (j < rows) *dst = __float2bfloat16_rn(v[j]);
    };
    const int jobs = (ti.rows + 15) >> 4, stride = last ? TEAMS + 1 : 1, job0 = last ? (int)group : 0;
    // of a cluster's jobs every CTA finishes its share
    const int first = p.cluster ? job0 * p.slices + (int)wd.slice : job0;
    if (with_operands && first < jobs) request(first);
    ok = ok && tc::warp_wait_idle(last ? smem_u32(last_full) : smem_u32(&tmem_full[acc.set]), last ? 0u : (acc.use & 1));
    if (!ok && lane == 0) tc::report_timeout(p.status, kStatusEpilogueTimeout);
    tc::fence_after_sync();
    const uint32_t t_row = tmem_base + ((uint32_t)(quarter * 32) << 16) + acc.col;
    // the second accumulator, unless the item has only 64 k (a tail of K)
    const bool add_second = two && min(p.K, (int)wd.c1 * kChunkK) - (int)wd.c0 * kChunkK > 64;
    const uint32_t sums = smem_u32(smem) + (uint32_t)(quarter * 32 + lane) * 4;   // cluster: [tokens][128], over the activation ring
#pragma unroll 1
    for (int job = job0; job < jobs; job += stride) {
      float v[16];
      {
        uint32_t r[16];
        tc::tmem_ld_32x32b_x16(t_row + job * 16, r);
        if (add_second) {
          uint32_t r2[16];
          tc::tmem_ld_32x32b_x16(t_row + acc.second + job * 16, r2);
          tc::tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(r[j]) + __uint_as_float(r2[j]);
        } else {
          tc::tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(r[j]);
        }
      }
      if (!last && job + stride >= jobs) {               // read: the next tile may be summed here
        tc::fence_before_sync();
        __syncwarp();
        tc::arrive_if(lane == 0, smem_u32(&tmem_empty[acc.set]));
      }
      if (p.slices == 1) {
        finish(job, v);
        if (with_operands && job + stride < jobs) request(job + stride);
      } else if (p.cluster) {
#pragma unroll
        for (int j = 0; j < 16; ++j)
          asm volatile("st.shared.f32 [%0], %1;" ::"r"(sums + (uint32_t)(job * 16 + j) * (kBN * 4)), "f"(v[j]) : "memory");
      } else {                                           // the sums of this slice; bias and post-ops come when they are added
        const int rows = live ? min(16, ti.rows - job * 16) : 0;
        const int64_t pitch = (p.N + 3) & ~3;
        float *dst = p.partial + ((int64_t)wd.slice * p.M + ti.m0 + job * 16) * pitch + n;
#pragma unroll
        for (int j = 0; j < 16; ++j, dst += pitch)
          if (j < rows) __stcg(dst, v[j]);
      }
    }
    if (p.cluster) {                                     // all slices' sums are in shared memory: add them in order
      tc::cluster_sync();
#pragma unroll 1
      for (int job = first; job < jobs; job += stride * p.slices) {
        float v[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) v[j] = 0.f;
#pragma unroll 2
        for (int s = 0; s < p.slices; ++s) {
          const uint32_t src = tc::map_to_rank(sums, (uint32_t)s) + (uint32_t)job * (16 * kBN * 4);
#pragma unroll
          for (int j = 0; j < 16; ++j) v[j] += tc::load_cluster_f32(src + j * (kBN * 4));
        }
        finish(job, v);
        if (with_operands && job + stride * p.slices < jobs) request(job + stride * p.slices);
      }
    }
  }
  }
  if (p.cluster) {
    if (warp < 3) tc::cluster_sync();      // the other warps' first
    tc::cluster_sync();                    // a peer may still read this CTA's sums
  }

  tc::fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    tc::fence_after_sync();
    tc::tmem_dealloc(tmem_base, 512);
  }
}

constexpr int kSliceThreads = 128;

// y = post_ops(sum over the slices + bias), the slices in order, four columns per thread.  Bound by latency and, for many
// rows, by L2: a launch of its own on the dependency of the one before it costs less than a meeting of the slices' CTAs at
// the end of the main kernel (pieces to L2, fence, ticket, addition by the last to arrive: 5 - 10 us).
__global__ void __launch_bounds__(kSliceThreads) woq_slices_kernel(const float *__restrict__ partial, int slices, int M, int N,
                                                                   const void *__restrict__ bias, int bias_dtype,
                                                                   const __grid_constant__ PostOpsDev post,
                                                                   __nv_bfloat16 *__restrict__ y) {
  grid_launch_dependents();
  grid_dependency_wait();
  const int quads_n = (N + 3) >> 2;
  const int64_t quad = (int64_t)blockIdx.x * kSliceThreads + threadIdx.x;
  if (quad >= (int64_t)M * quads_n) return;
  const int64_t m = quad / quads_n;
  const int n = (int)(quad - m * quads_n) * 4, live = min(4, N - n);
  const int64_t base = m * N + n, step = (int64_t)M * quads_n * 4;
  float v[4] = {0.f, 0.f, 0.f, 0.f};
  const float *src = partial + quad * 4;
#pragma unroll 4
  for (int s = 0; s < slices; ++s) {
    const float4 t = __ldcg(reinterpret_cast<const float4 *>(src + s * step));
    v[0] += t.x;
    v[1] += t.y;
    v[2] += t.z;
    v[3] += t.w;
  }
  int b = 0;
#pragma unroll
  for (int e = 0; e < 4; ++e)
    if (bias && e < live) v[e] += load_as_float(bias, n + e, bias_dtype);
#pragma unroll 1
  for (int o = 0; o < post.n_ops; ++o) {
    const int id = post.ids[o];
    const bool binary = id == ZT_POST_MUL || id == ZT_POST_ADD;
    const __nv_bfloat16 *other = binary ? reinterpret_cast<const __nv_bfloat16 *>(post.bufs[b++]) + base : nullptr;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      if (!binary) {
        v[e] = unary_post(v[e], id);
      } else if (e < live) {
        const float t = __bfloat162float(other[e]);
        v[e] = id == ZT_POST_MUL ? v[e] * t : v[e] + t;
      }
    }
  }
  if (live == 4 && (N & 3) == 0 && (reinterpret_cast<uintptr_t>(y) & 7) == 0) {
    *reinterpret_cast<uint2 *>(y + base) = make_uint2(bf2_pack(v[0], v[1]), bf2_pack(v[2], v[3]));
  } else {
#pragma unroll
    for (int e = 0; e < 4; ++e)
      if (e < live) y[base + e] = __float2bfloat16_rn(v[e]);
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

// How many clusters of a size the device can run at once, asked for once per device and size.
struct ClusterRoom {
  std::atomic<int> known[64][kMaxCluster + 1] = {};   // + 1
  template <typename Kernel>
  int clusters(Kernel kern, int threads, int smem, int size) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
    std::atomic<int> &entry = known[dev][size];
    if (const int k = entry.load(std::memory_order_relaxed)) return k - 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)size);
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = (size_t)smem;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = (unsigned)size;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) {
      cudaGetLastError();
      n = 0;
    }
    entry.store(n + 1, std::memory_order_relaxed);
    return n;
  }
};

template <int NMAX, int KS, int TEAMS, int SLOTS, int XK, int XSTAGES, int PSTAGES>
int launch_cfg(const TcParams &p0, int scale_dtype, const void *x, int64_t x_rows, int64_t w_rows, int max_row_tiles,
               bool *slices_added, cudaStream_t st) {
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
  // Scales and zero points travel with the packed chunks when the group size is a power of two, the tables can be
  // addressed by TMA and a chunk's part of them fits its slot; otherwise the conversion threads fetch them from global memory.
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
    const int gpc = p.gs >= kChunkK ? 1 : kChunkK / p.gs;
    if (p.gs_log2 >= 0 && aligned && (size_t)gpc * kBN * esz * (asym ? 2 : 1) <= (size_t)scale_slot_bytes(NMAX)) {
      p.staged_gpc = gpc;
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
  const int64_t items = (int64_t)(p.g_count ? max_row_tiles : p.m_tiles) * p.n_tiles * p.slices;
  const int sms = sm_count();
  const dim3 grid((unsigned)(items < sms ? items : sms));
  // every instantiation needs its own once-per-device attribute set-up
  static PerDeviceOnce configured[4];
  auto launch = [&](auto kern, int which) -> int {
    if (int rc_cfg = allow_dynamic_smem(configured[which], kern, L::kTotal)) return rc_cfg;
    // Slices are added by clusters where there are two of them (M = 128, 8192 -> 8192: 22.3 us with the second kernel, 19.7
    // so), and where a slice is so short that submitting a second kernel takes longer than the call (M = 100, 1024 -> 1024 called
    // in a row: 10.2 and 7.5 us, although on the device it is 6.2 and 7.2).  Larger clusters of longer slices start later than as
    // many single CTAs: M = 17, 4096 -> 4096 in four slices 7.9 us with the second kernel and 10.1 as clusters.
    static ClusterRoom room[4];
    const bool cluster = p.slices == 2 || (p.slices > 2 && p.slices <= kMaxCluster && p.chunks <= 2 * p.slices);
    if (cluster && items <= sms &&
        room[which].clusters(kern, threads_for(TEAMS), L::kTotal, p.slices) * p.slices >= items) {
      TcParams c = p;
      c.cluster = 1;
      c.partial = nullptr;
      *slices_added = true;
      ZT_CUDA_OK(launch_overlapped_cluster(kern, grid, dim3(threads_for(TEAMS)), (size_t)L::kTotal, st, dim3((unsigned)p.slices), tx, tx2,
                                           tw, ts, tz, c));
      return launch_status("woq_tcgen05_kernel");
    }
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
               int max_row_tiles, bool *slices_added, cudaStream_t st) {
  switch (cap) {
    // <token tile, k per stage, conversion teams, converted slots, k per activation slot, activation slots, packed chunks>
    case 32: return launch_cfg<32, 128, 6, 6, 256, 5, 6>(p, scale_dtype, x, x_rows, w_rows, max_row_tiles, slices_added, st);
    case 64: return launch_cfg<64, 128, 6, 6, 256, 3, 6>(p, scale_dtype, x, x_rows, w_rows, max_row_tiles, slices_added, st);
    case 128: return launch_cfg<128, 128, 4, 4, 128, 4, 4>(p, scale_dtype, x, x_rows, w_rows, max_row_tiles, slices_added, st);
    case 192: return launch_cfg<192, 64, 4, 4, 64, 5, 4>(p, scale_dtype, x, x_rows, w_rows, max_row_tiles, slices_added, st);
    default: break;
  }
  set_error("zt_woq_linear: unsupported token-tile width %d for the tcgen05 kernel", cap);
  return ZT_UNSUPPORTED;
}

// Row tiling and work split of a dense call.
struct DensePlan {
  int cap;       // instantiation
  int m_tiles, bt;
  int slices;    // of K, per tile
  int accs;      // accumulators per item
};
int cap_for(int64_t rows) { return rows <= 32 ? 32 : rows <= 64 ? 64 : rows <= 128 ? 128 : 192; }
// How many sums a tile's K is at least divided among.  The tensor core's fp32 accumulation truncates, so its error grows
// with the number of products added to one accumulator (relative to the result's root mean square 3.5e-6 for 4096 k in
// one sum, 1.6e-6 in two; 8192 k: 7.7e-6 in one, 1.6e-6 in four).  Up to 128 rows two accumulators take alternate blocks of
// 64 k, and up to 256 rows K is cut into as many equal slices of whole chunks as the SMs can work on at once.
int64_t min_sums(int64_t M, int64_t N, int64_t K) {
  if (M > 256) return 1;
  const int64_t room = std::min<int64_t>(kMaxSlices, sm_count() / ceil_div<int64_t>(N, kBN)), chunks = K / kChunkK;
  int64_t slices = 1;
  for (int64_t ks = 2; ks <= room && K % kChunkK == 0; ++ks)
    if (chunks % ks == 0) slices = ks;
  return M <= 128 ? 2 * slices : slices;
}

// The number of row tiles and of K slices by estimated cycles.  A 128 x 64 block takes the slower of the conversion
// (350 cycles, 400 where it calculates in fp32) and the MMAs (2 per token, and about 90 around them), and then waits for its
// operands out of L2 the longer, the more rows a tile has and the more SMs pull; adding slices up takes a launch of its own
// (5000 cycles; the same is charged where a cluster does it) and their way through L2.  The constants are fitted to 108 shapes of 130 - 1024 rows timed with every plan:
// the chosen one is 0.7 % above the fastest in the mean and 9 % at most.  M = 192, 14336 -> 4096: 53 us in one slice, 22.5 in
// four; M = 384: 39 as 2 x 2, 53 as three row tiles of whole K; M = 256, 2816 -> 5003: 14.0 whole, 21.6 in two slices.
DensePlan dense_plan(int64_t M, int64_t N, int64_t K, bool fp32_conversion, bool may_slice) {
  const int64_t sms = sm_count(), n_tiles = ceil_div<int64_t>(N, kBN), chunks = ceil_div<int64_t>(K, kChunkK);
  const int64_t sums = may_slice ? min_sums(M, N, K) : M <= 128 ? 2 : 1, first = ceil_div<int64_t>(M, 192);
  DensePlan best{};
  double best_cost = 1e300;
  for (int64_t mt = first; mt <= first + first / 2 + 1 && mt <= ceil_div<int64_t>(M, 16); ++mt) {
    const int64_t bt = ceil_div<int64_t>(ceil_div(M, mt), 16) * 16, tiles_m = ceil_div(M, bt), tiles = tiles_m * n_tiles;
    const int64_t accs_max = bt <= 128 ? 2 : 1;
    const double block = std::max(fp32_conversion ? 400.0 : 350.0, 2.0 * (double)bt + 90.0);
    const int64_t least = std::min(ceil_div(sums, accs_max), chunks);
    const int64_t most = may_slice ? std::max(least, std::min<int64_t>({sms / tiles, kMaxSlices, chunks})) : 1;
    for (int64_t ks = std::max<int64_t>(least, 1); ks <= most; ++ks) {
      if (ks > least && ceil_div(chunks, ks) == ceil_div(chunks, ks - 1)) continue;     // no shorter than with fewer
      const double wait = 0.4 * (double)(bt + 36) * (double)std::min(tiles * ks, sms) / (double)sms;
      double cost = (double)(ceil_div<int64_t>(tiles * ks, sms) * ceil_div(chunks, ks)) * 4.0 * (block + wait);
      if (ks > 1) cost += 5000.0 + (double)(ks * M * N) / 400.0;
      if (cost < best_cost) {
        best_cost = cost;
        best = {cap_for(bt), (int)tiles_m, (int)bt, (int)ks, ks < sums && accs_max == 2 ? 2 : 1};
      }
    }
  }
  return best;
}
size_t slices_bytes(const DensePlan &d, int64_t M, int64_t N) {
  return d.slices > 1 ? (size_t)d.slices * M * ((N + 3) & ~3) * sizeof(float) : 0;
}

}  // namespace

size_t woq_tcgen05_workspace_bytes(int64_t M, int64_t N, int64_t K) {
  return std::max(slices_bytes(dense_plan(M, N, K, false, true), M, N), slices_bytes(dense_plan(M, N, K, true, true), M, N));
}

void woq_tcgen05_plan(int64_t M, int64_t N, int64_t K, bool fp32_conversion, int32_t *plan) {
  const DensePlan d = dense_plan(M, N, K, fp32_conversion, true);
  const int values[5] = {d.cap, d.m_tiles, d.bt, d.slices, d.accs};
  std::copy(values, values + 5, plan);
}

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
  const bool one_acc = (a.algo & ZT_ALGO_ONE_ACCUMULATOR) != 0, fp32_conversion = a.zeros && a.scale_dtype == ZT_F32;
  DensePlan d = dense_plan(a.M, a.N, a.K, fp32_conversion, hint == 0 && !one_acc && a.workspace != nullptr);
  if (d.slices > 1 && a.workspace_bytes < ZT_WOQ_COUNTER_BYTES + slices_bytes(d, a.M, a.N))
    d = dense_plan(a.M, a.N, a.K, fp32_conversion, false);
  if (hint > 0) {                      // the instantiation that takes tiles of this width (the widest: 192)
    d.cap = hint == 256 ? 192 : hint;
    d.m_tiles = (int)ceil_div<int64_t>(a.M, d.cap);
    d.bt = (int)ceil_div<int64_t>(ceil_div<int64_t>(a.M, d.m_tiles), 16) * 16;
    d.m_tiles = (int)ceil_div<int64_t>(a.M, d.bt);
    d.accs = d.cap <= 128 ? 2 : 1;
  }
  if (one_acc) d.accs = 1;
  p.m_tiles = d.m_tiles;
  p.n_tiles = (int)ceil_div<int64_t>(a.N, kBN);
  p.bt = d.bt;
  p.chunks = (int)ceil_div<int64_t>(a.K, kChunkK);
  p.slices = d.slices;
  p.accs = d.accs;
  p.x_box = p.x_box2 = d.m_tiles == 1 ? (int)ceil_div<int64_t>(a.M, 8) * 8 : d.bt;   // 128-byte swizzle: 8-row atoms
  p.partial = d.slices > 1 ? reinterpret_cast<float *>(reinterpret_cast<char *>(a.workspace) + ZT_WOQ_COUNTER_BYTES) : nullptr;
  bool slices_added = d.slices == 1;
  const int rc = launch_any(d.cap, p, a.scale_dtype, a.x, a.M, a.N, 0, &slices_added, st);
  if (rc != ZT_SUCCESS || slices_added) return rc;
  const int64_t quads = a.M * ceil_div<int64_t>(a.N, 4);
  ZT_CUDA_OK(launch_overlapped(woq_slices_kernel, dim3((unsigned)ceil_div<int64_t>(quads, kSliceThreads)), dim3(kSliceThreads), (size_t)0, st,
                               (const float *)p.partial, d.slices, p.M, p.N, p.bias, p.bias_dtype, p.post, p.y));
  return launch_status("woq_slices_kernel");
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
  p.slices = 1;
  p.accs = row_tile <= 128 ? 2 : 1;
  p.x_box = row_tile > 64 ? 64 : row_tile;
  p.x_box2 = row_tile;
  p.g_count = tile_count;
  p.g_tiles = tiles;
  bool slices_added = true;
  return launch_any(cap_for(row_tile), p, scale_dtype, x, total_rows, (int64_t)num_experts * N, max_row_tiles, &slices_added, st);
}

}  // namespace zt
