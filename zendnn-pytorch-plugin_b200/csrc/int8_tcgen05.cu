// Host side of the int8 tcgen05 GEMM: tensor-map cache, tile-shape choice, dispatch to the compiled
// configurations (the kernel itself is in int8_tcgen05.cuh).
#include <algorithm>
#include <mutex>
#include <unordered_map>

#include "int8_tcgen05.cuh"

namespace zt {

using namespace i8tc;

namespace {

// ---- host ----------------------------------------------------------------------------------------
struct MapKey {
  const void *ptr;
  uint64_t inner, rows;
  uint32_t box_rows, group;
  bool operator==(const MapKey &o) const {
    return ptr == o.ptr && inner == o.inner && rows == o.rows && box_rows == o.box_rows && group == o.group;
  }
};
struct MapKeyHash {
  size_t operator()(const MapKey &k) const {
    return std::hash<const void *>()(k.ptr) ^ (k.inner * 1315423911u) ^ (k.rows << 17) ^ k.box_rows ^ (k.group << 12);
  }
};

// Tensor maps depend only on (pointer, shape, box); encoding one costs a driver call, so they are
// memoised per process.
// `group` > 1: the matrix as [K / 128][rows][128] (K a multiple of 128), a box of `group` blocks x box_rows x 128 bytes.
int cached_map(CUtensorMap *out, const void *ptr, uint64_t inner, uint64_t rows, uint32_t box_rows, uint32_t group) {
  static std::mutex mu;
  static std::unordered_map<MapKey, CUtensorMap, MapKeyHash> cache;
  const MapKey key{ptr, inner, rows, box_rows, group};
  std::lock_guard<std::mutex> lock(mu);
  auto it = cache.find(key);
  if (it != cache.end()) {
    *out = it->second;
    return ZT_SUCCESS;
  }
  int rc;
  if (group > 1) {
    const uint64_t dims[3] = {kBK, rows, inner / kBK}, strides[2] = {inner, kBK};
    const uint32_t box[3] = {kBK, box_rows, group};
    rc = make_tensor_map(out, ptr, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, dims, strides, box, true);
  } else {
    rc = make_tensor_map_2d(out, ptr, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, inner, rows, inner, kBK, box_rows);
  }
  if (rc != ZT_SUCCESS) return rc;
  if (cache.size() > 4096) cache.clear();
  cache.emplace(key, *out);
  return ZT_SUCCESS;
}

// Tile shape: the candidate (rows per CTA tile, tile width) that minimises rounds x tile time.  A tile's main loop
// costs, per byte of K, the larger of the tensor-pipe time (rows/128 * BN/64 cycles) and the operand-delivery time
// ((rows + BN) bytes at the 44 B/clk that an SM gets out of L2 when all of them pull); narrow tiles additionally pay
// shared-memory reads of the A block that every instruction repeats.  A tile whose accumulator cannot be double
// buffered, or that is the only one of its CTA, exposes its epilogue.
// The width is a run-time argument of the kernel, in steps of 16 columns, and a call with at most 112 rows loads only
// those: 16 rows x 80 columns on 128 SMs instead of 128 x 64 in two rounds for M = 1, 8192 -> 10240; 256 x 240 in 13 full
// rounds instead of 256 x 256 in 13 with the last one nearly empty for M = 4096, 8192 -> 28672.
struct TileChoice {
  int mh, bn;
};
int a_rows_of(int mh, int64_t M) { return mh == 1 && M < kBM ? (int)ceil_div<int64_t>(M, 16) * 16 : mh * kBM; }
int nbuf_of(int mh, int bn) { return 2 * mh * acc_stride(bn) <= 512 ? 2 : 1; }

TileChoice pick_tile(int64_t M, int64_t N, int64_t K) {
  const int64_t sms = sm_count();
  double best = 1e30;
  TileChoice pick{1, 128};
  for (int mh = 1; mh <= (M <= kBM ? 1 : 2); ++mh) {
    const double rows = a_rows_of(mh, M);
    for (int bn = mh == 1 ? 16 : 64; bn <= kMaxBN; bn += 16) {
      const int64_t tiles = ceil_div<int64_t>(M, (int64_t)mh * kBM) * ceil_div<int64_t>(N, bn);
      const int64_t rounds = ceil_div<int64_t>(tiles, sms);
      const double mma = mh * std::max(bn / 64.0, (32.0 + bn / 4.0) / 32.0);
      const double data = (rows + bn) / 44.0;
      const double epilogue = mh * bn * 4.0;  // cycles, when not hidden behind the next tile
      const double exposed = nbuf_of(mh, bn) == 1 ? rounds * epilogue : epilogue;
      // all tiles' operands, lightly: of two equal shapes the one that moves less draws less power (M = 1024, 14336 -> 4096 in
      // a long run: 256 x 112 76.4 us, 128 x 256 73.4)
      const double traffic = 0.05 * (double)tiles / (double)sms * data * (double)K;
      const double cost = rounds * std::max(mma, data) * (double)K + exposed + rounds * 500.0 + traffic;
      if (cost < best * (1.0 - 1e-9)) {
        best = cost;
        pick = {mh, bn};
      }
    }
  }
  return pick;
}

template <int MH, int EPI, bool A_SIGNED>
int launch_cfg(const CUtensorMap &ta, const CUtensorMap &tb, const TcParams &p, cudaStream_t st) {
  auto kern = int8_tcgen05_kernel<MH, EPI, A_SIGNED>;
  static PerDeviceOnce configured;
  if (int rc = allow_dynamic_smem(configured, kern, kSmemLimit)) return rc;
  const int tiles = p.m_tiles * p.n_tiles, sms = sm_count();
  const dim3 grid((unsigned)(tiles < sms ? tiles : sms));
  ZT_CUDA_OK(launch_overlapped(kern, grid, dim3(kThreads), (size_t)smem_bytes(p.stages, p.stage_bytes, p.ring_pad), st, ta, tb, p));
  return launch_status("int8_tcgen05_kernel");
}
template <int MH>
int launch_mh(const CUtensorMap &ta, const CUtensorMap &tb, const TcParams &p, int epi, bool a_signed, cudaStream_t st) {
  if (epi == kEpiS32) return a_signed ? launch_cfg<MH, kEpiS32, true>(ta, tb, p, st) : launch_cfg<MH, kEpiS32, false>(ta, tb, p, st);
  if (epi == kEpiStatic)
    return a_signed ? launch_cfg<MH, kEpiStatic, true>(ta, tb, p, st) : launch_cfg<MH, kEpiStatic, false>(ta, tb, p, st);
  return a_signed ? launch_cfg<MH, kEpiLinear, true>(ta, tb, p, st) : launch_cfg<MH, kEpiLinear, false>(ta, tb, p, st);
}

}  // namespace

bool int8_tcgen05_supported(int64_t M, int64_t N, int64_t K, const void *q, const void *w) {
  if (M < 1 || N < 1 || K < 16 || K % 16 != 0) return false;
  if (M > (1 << 30) || N > (1 << 30) || K > (1 << 30)) return false;
  if ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(w)) & 15) return false;
  return true;
}

int int8_tcgen05_launch(const Int8GemmArgs &a, cudaStream_t st) {
  TcParams p{};
  p.M = (int)a.M;
  p.N = (int)a.N;
  p.K = (int)a.K;
  p.src_scale = a.src_scale;
  p.src_zp = a.src_zp;
  p.w_scale = a.w_scale;
  p.w_rowsum = a.w_rowsum;
  p.bias = a.bias;
  p.w_scale_dtype = a.w_scale_dtype;
  p.bias_dtype = a.bias_dtype;
  p.y_dtype = a.y_dtype;
  p.y = a.y;
  p.post = a.post;
  p.status = device_status_ptr();
  p.w_scale_per_tensor = a.w_scale_per_tensor;
  p.post_dtype = a.post_dtype;
  p.out_scale = a.out_scale;
  p.out_zp = a.out_zp;
  p.ldy = a.ldy;
  const int epi = a.raw_s32 ? kEpiS32 : a.static_mode ? kEpiStatic : kEpiLinear;
  // force_bn: tile width, + 1000 for 256-row tiles (e.g. 1160 = 256 x 160), + 2000 for CTA pairs (512 x width)
  TileChoice tile = pick_tile(a.M, a.N, a.K);
  if (a.force_bn >= 2000) {
    ZT_REQUIRE(!a.raw_s32 && !a.static_mode && int8_pair_supported(a.M, a.force_bn % 1000), ZT_UNSUPPORTED,
               "int8_tcgen05_launch: CTA-pair tiles need the linear epilogue, M > 256 and a width of 128, 160, 192 or 256");
    return launch_pair(a.force_bn % 1000, a, p, !a.q_is_u8, st);
  }
  if (a.force_bn > 0) tile = {a.force_bn >= 1000 ? 2 : 1, a.force_bn % 1000};
  ZT_REQUIRE(tile.bn >= 16 && tile.bn <= kMaxBN && tile.bn % 16 == 0, ZT_UNSUPPORTED,
             "int8_tcgen05_launch: unsupported tile width %d", tile.bn);
  p.bn = tile.bn;
  p.nbuf = nbuf_of(tile.mh, tile.bn);
  p.a_rows = a_rows_of(tile.mh, a.M);
  p.m_tiles = ceil_div(p.M, tile.mh * kBM);
  p.n_tiles = ceil_div(p.N, tile.bn);
  // A stage costs its producer two copies, an expect and a wait, about 400 cycles whatever their size; small tiles take up to
  // four 128-byte blocks of K per stage while at least four stages fit (M = 1 on 8192 -> 10240: 22.3 -> 21.2 us; M = 16 on 4096 -> 11008 with narrower boxes 19.5 -> 12.7 us).
  const int block_bytes = (p.a_rows + tile.bn) * kBK, room = kSmemLimit - smem_bytes(0, 0, 0);
  p.group = 1;
  while (p.group < 4 && a.K % kBK == 0 && p.group * kBK < a.K && 2 * p.group * block_bytes * 4 <= room) p.group *= 2;
  p.stage_bytes = p.group * block_bytes;
  p.ring_pad = ring_pad(tile.mh, p.a_rows, tile.bn, p.group);
  p.stages = std::min(kMaxStages, (kSmemLimit - smem_bytes(0, 0, p.ring_pad)) / p.stage_bytes);
  CUtensorMap ta, tb;
  // q_rows: rows that may be addressed behind q (the caller's scratch is padded to kMinQRows rows so that the
  // activation map never has fewer; rows beyond M hold stale bytes whose products are never stored)
  const uint64_t q_rows = a.q_rows > a.M ? (uint64_t)a.q_rows : (uint64_t)a.M;
  int rc = cached_map(&ta, a.q, (uint64_t)a.K, q_rows, (uint32_t)p.a_rows, (uint32_t)p.group);
  if (rc != ZT_SUCCESS) return rc;
  rc = cached_map(&tb, a.w, (uint64_t)a.K, (uint64_t)a.N, (uint32_t)p.bn, (uint32_t)p.group);
  if (rc != ZT_SUCCESS) return rc;
  const bool sgn = !a.q_is_u8;
  return tile.mh == 2 ? launch_mh<2>(ta, tb, p, epi, sgn, st) : launch_mh<1>(ta, tb, p, epi, sgn, st);
}

}  // namespace zt
