// Grouped expert GEMM on the dispatched layout, for sm_100a tensor cores (tcgen05 + TMEM + TMA).
//
//   out[rows of expert e, :] = act(rows[rows of expert e, :] x weights[e]^T)
//
// rows    [L, K] bf16: the output of dispatch (path e starts at e * max_path_load when padded,
//                      else at sum(loads[0..e)); only the first loads[e] rows of a path count)
// weights [E, N, K] bf16 (every expert's [N, K] matrix, K contiguous)
// out     [L, N] bf16
// loads   [E] int32 ON THE DEVICE: the kernel never needs them on the host.
//
// The weights are the M operand of the MMA and the rows its N operand (the tile computed is
// out^T): out_features is a multiple of the 128-row half of a tile, while the number of rows of
// an expert is anything, and N may be any multiple of 16 up to 256.  An expert's rows are cut
// into ceil(load / 256) equal tiles, so hardly anything is computed for padding; with rows as
// the M operand every expert's last 128-row tile was computed in full.
//
// One persistent CTA pair (kPair = 2: cta_group::2, M = 256, each CTA holds 128 weight rows and
// half of the tile's rows) or, when out_features is an odd multiple of 128, one CTA (M = 128)
// walks the list of (expert, row tile, feature tile) work items that it derives from `loads`
// itself.  Roles inside a CTA (192 threads):
//   warp 0     one elected lane issues the TMA loads (cp.async.bulk.tensor, 128B swizzle, no
//              multicast) of its weight tile [128 x 64] and of its rows, in one box of 32, 64, 96
//              or 128 x 64, into a shared-memory ring; the bytes of both CTAs count on the first
//              CTA's mbarrier;
//   warp 1     allocates tensor memory (2 accumulators of 128 lanes x 256 fp32 columns); one
//              elected lane of the first CTA issues tcgen05.mma (K = 16) four times per k-block
//              for the pair, releasing ring slots and publishing accumulators in both CTAs with
//              tcgen05.commit;
//   warps 2-5  epilogue: tcgen05.ld of the 32 lanes (features) their warp id selects, optional
//              ReLU, fp32 -> bf16, transposed through 2 KB of shared memory per warp so that
//              a row is stored 64 bytes at a time, and only if it exists (row < loads[e]).
// The second accumulator lets the epilogue of tile i run under the MMAs of tile i + 1.
// Every mbarrier wait is bounded: after the limit the role records an error and leaves its
// loop, the copies in flight are given time to land, the CTAs meet, free their tensor memory
// and return.
//
// What bounds it: HBM reads of the weights for few rows per expert (32 experts of 4 rows, 1024 ->
// 4096: 48 us, 5.6 TB/s); for many, shared memory and the tensor pipe together: the MMAs of the
// 1024 -> 4096 layer over 27732 rows take 155 us without their loads, the loads and stores
// 154 us without the MMAs, both 192 us (1208 TFLOP/s).  Single CTAs with 128 x 256 tiles, rows as
// the M operand, took 211 us there and moved 2.9 instead of 2.0 GB from L2 to the SMs; 36343
// rows in 128 very uneven experts, 768 -> 3072, took 222 us and take 185.  The rows come in one
// box of the size needed: boxes of 32 rows alone cost 12 %.  An L2 prefetch of the weights of
// the next tile made every shape slower (66 -> 76 us with few rows).
#include <cuda.h>

#include "common.cuh"

namespace brt_b200 {
namespace {

constexpr int kBM = 128, kBK = 64;  // weight rows per CTA; kBK bf16 = one 128-byte swizzle row
constexpr int kBN = 256;            // rows of an expert in one tile, at most
constexpr int kBoxStep = 32;        // the row operand is fetched in one box of 32, 64, 96 or
constexpr int kBoxSizes = 4;        // 128 rows (two of them when a single CTA needs more)
constexpr int kUmmaK = 16;
constexpr int kThreads = 192;
constexpr int kMaxExperts = 1024;
constexpr uint32_t kTileBytes = kBM * kBK * 2;         // 16 KB: one CTA's weight tile
constexpr uint32_t kRowBytes = kBK * 2;                // one row of a k-block
constexpr unsigned long long kWaitLimitNs = 2000000000ull;  // of one wait
// ring slots: 32 KB each with a pair (half of the rows per CTA), 48 KB without
template <int kPair>
constexpr int kStages = kPair == 2 ? 6 : 4;

struct RowMaps {
  CUtensorMap box[kBoxSizes];  // box[i]: (i + 1) * kBoxStep rows
};

struct GemmArgs {
  const int* loads;
  __nv_bfloat16* out;
  int* error;
  int experts;
  int max_path_load;  // 0: packed
  int m_tiles;        // N / (128 * kPair)
  int k_blocks;       // K / kBK
  long long N;
  long long total_rows;
  int relu;
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
               "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ unsigned long long now_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
// Bounded wait for the phase with the given parity; false when the limit ran out.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity) {
  const uint32_t addr = smem_u32(bar);
  unsigned long long until = 0;
  for (int spin = 0;; spin++) {
    uint32_t done;
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        "selp.u32 %0, 1, 0, p;\n"
        "}\n"
        : "=r"(done)
        : "r"(addr), "r"(parity)
        : "memory");
    if (done) return true;
    if (spin > 64) {
      const unsigned long long now = now_ns();
      if (until == 0) until = now + kWaitLimitNs;
      else if (now > until) return false;
      __nanosleep(32);
    }
  }
}
// The address of `p`'s twin in the shared memory of CTA `rank` of the cluster.
__device__ __forceinline__ uint32_t map_to_cta(const void* p, uint32_t rank) {
  uint32_t addr;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(addr) : "r"(smem_u32(p)), "r"(rank));
  return addr;
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr)
               : "memory");
}
// `bar` is a cluster address: with a pair, the copies of both CTAs count on the first one's.
template <int kPair>
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, uint32_t bar,
                                            int x, int y) {
  if constexpr (kPair == 2)
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes.cta_group::2"
        " [%0], [%1, {%3, %4}], [%2];" ::"r"(smem_u32(dst)),
        "l"(map), "r"(bar), "r"(x), "r"(y)
        : "memory");
  else
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, "
        "{%3, %4}], [%2];" ::"r"(smem_u32(dst)),
        "l"(map), "r"(bar), "r"(x), "r"(y)
        : "memory");
}
template <int kPair>
__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, uint32_t bar,
                                            int x, int y, int z) {
  if constexpr (kPair == 2)
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes.cta_group::2"
        " [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(smem_u32(dst)),
        "l"(map), "r"(bar), "r"(x), "r"(y), "r"(z)
        : "memory");
  else
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, "
        "{%3, %4, %5}], [%2];" ::"r"(smem_u32(dst)),
        "l"(map), "r"(bar), "r"(x), "r"(y), "r"(z)
        : "memory");
}

// Shared-memory matrix descriptor of a K-major tile stored with the 128-byte swizzle (rows of
// 128 bytes, groups of 8 rows 1024 bytes apart): start address, leading byte offset 1 (unused
// by swizzled K-major layouts), stride byte offset 1024, descriptor version 1, layout type 2.
__device__ __forceinline__ uint64_t umma_desc(const void* tile) {
  uint64_t d = 0;
  d |= (uint64_t)((smem_u32(tile) & 0x3ffff) >> 4);
  d |= (uint64_t)1 << 16;
  d |= (uint64_t)(1024 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}
// kind::f16 instruction descriptor: fp32 accumulate, bf16 x bf16, both operands K-major.
template <int kPair>
__device__ __forceinline__ uint32_t umma_idesc(int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) |
         ((uint32_t)(kPair * kBM >> 4) << 24);
}
template <int kPair>
__device__ __forceinline__ void umma_bf16(uint32_t tmem_d, uint64_t a, uint64_t b, uint32_t idesc,
                                          uint32_t accumulate) {
  if constexpr (kPair == 2)
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n"
        "}\n" ::"r"(tmem_d),
        "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
        : "memory");
  else
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n"
        "}\n" ::"r"(tmem_d),
        "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
        : "memory");
}
// Arrive on `bar` (with a pair: on both CTAs' barriers at that offset) once every MMA issued
// before has finished.
template <int kPair>
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  if constexpr (kPair == 2)
    asm volatile(
        "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64"
        " [%0], %1;" ::"r"(smem_u32(bar)),
        "h"((uint16_t)3)
        : "memory");
  else
    asm volatile(
        "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
            smem_u32(bar))
        : "memory");
}
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// All threads of the pair (or of the CTA).
template <int kPair>
__device__ __forceinline__ void group_sync() {
  if constexpr (kPair == 2) {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  } else {
    __syncthreads();
  }
}
__device__ __forceinline__ void tmem_load_32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, "
      "%20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]),
        "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]),
        "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}

template <int kPair>
struct alignas(1024) GemmSmem {
  unsigned char a[kStages<kPair>][kTileBytes];
  unsigned char b[kStages<kPair>][kBN / kPair * kBK * 2];
  __nv_bfloat16 turn[4][2][32 * 32];  // per epilogue warp, two buffers: [row][feature]
  uint64_t full[kStages<kPair>];
  uint64_t empty[kStages<kPair>];
  uint64_t acc_full[2];
  uint64_t acc_empty[2];
  uint32_t tmem_base;
  int first_tile[kMaxExperts + 1];  // exclusive prefix of the tiles per expert
  int row_base[kMaxExperts];
  int load[kMaxExperts];
};

struct TileAt {
  int expert, m_tile;
  int row0, rows;  // within the expert
  int width;       // columns of the MMA: rows of a tile, rounded up to 16
};
template <int kPair>
__device__ __forceinline__ TileAt tile_at(const GemmSmem<kPair>& s, int experts, int m_tiles,
                                          int t) {
  int lo = 0, hi = experts - 1;  // last expert whose first tile is <= t (empty ones skipped)
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (s.first_tile[mid] <= t) lo = mid; else hi = mid - 1;
  }
  const int local = t - s.first_tile[lo];
  const int load = s.load[lo];
  const int parts = (load + kBN - 1) / kBN;
  const int each = ((load + parts - 1) / parts + 15) & ~15;
  const int part = local / m_tiles;
  TileAt at;
  at.expert = lo;
  at.m_tile = local - part * m_tiles;
  at.row0 = part * each;
  at.rows = load - at.row0 < each ? load - at.row0 : each;  // <= 0: rounding left none
  at.width = each;
  return at;
}

template <int kPair>
__global__ void __launch_bounds__(kThreads, 1)
expert_gemm_kernel(const __grid_constant__ CUtensorMap map_w,
                   const __grid_constant__ RowMaps map_r, const GemmArgs g) {
  constexpr uint32_t kTmemCols = 2 * kBN;
  constexpr int kRing = kStages<kPair>;
  extern __shared__ __align__(1024) unsigned char s_raw[];
  GemmSmem<kPair>& s = *reinterpret_cast<GemmSmem<kPair>*>(
      (reinterpret_cast<uintptr_t>(s_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  const int tid = threadIdx.x;
  const int warp = tid >> 5;
  const int lane = tid & 31;
  const uint32_t rank = kPair == 2 ? cluster_rank() : 0;
  const int group = blockIdx.x / kPair;
  const int groups = gridDim.x / kPair;

  if (warp == 0) {  // tiles per expert and the first row of every expert
    int tiles = 0, row = 0;
    for (int p = 0; p < g.experts; p += 32) {
      const int e = p + lane;
      int load = e < g.experts ? g.loads[e] : 0;
      if (load < 0) load = 0;
      if (g.max_path_load != 0 && load > g.max_path_load) load = g.max_path_load;
      const int mine = (load + kBN - 1) / kBN * g.m_tiles;
      int tiles_incl = mine, rows_incl = load;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int tn = __shfl_up_sync(0xffffffffu, tiles_incl, d);
        const int rn = __shfl_up_sync(0xffffffffu, rows_incl, d);
        if (lane >= d) { tiles_incl += tn; rows_incl += rn; }
      }
      if (e < g.experts) {
        s.first_tile[e] = tiles + tiles_incl - mine;
        s.row_base[e] = g.max_path_load != 0 ? e * g.max_path_load : row + rows_incl - load;
        s.load[e] = load;
      }
      tiles += __shfl_sync(0xffffffffu, tiles_incl, 31);
      row += __shfl_sync(0xffffffffu, rows_incl, 31);
    }
    if (lane == 0) {
      s.first_tile[g.experts] = tiles;
      for (int i = 0; i < kRing; i++) {
        mbar_init(&s.full[i], 1);
        mbar_init(&s.empty[i], 1);
      }
      for (int i = 0; i < 2; i++) {
        mbar_init(&s.acc_full[i], 1);
        mbar_init(&s.acc_empty[i], 4 * kPair);  // one arrival per epilogue warp
      }
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
  }
  if (warp == 1) {
    if constexpr (kPair == 2) {
      asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                       smem_u32(&s.tmem_base)),
                   "r"(kTmemCols)
                   : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    } else {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                       smem_u32(&s.tmem_base)),
                   "r"(kTmemCols)
                   : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  group_sync<kPair>();  // the peer's barriers exist
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = s.tmem_base;
  const int total_tiles = s.first_tile[g.experts];
  bool failed = false;

  if (warp == 0) {
    if (lane == 0) {
      int slot = 0;
      uint32_t phase = 0;
      for (int t = group; t < total_tiles && !failed; t += groups) {
        const TileAt at = tile_at(s, g.experts, g.m_tiles, t);
        const int half = at.width / kPair;  // rows this CTA stages (a multiple of 8)
        const int boxes = half > kBoxSizes * kBoxStep ? 2 : 1;
        const int size = (half / boxes + kBoxStep - 1) / kBoxStep;  // half / 2 is a multiple of 8
        const int box_rows = size * kBoxStep;
        const CUtensorMap* const map_box = &map_r.box[size - 1];
        const int row0 = s.row_base[at.expert] + at.row0 + (int)rank * half;
        const int feature0 = (at.m_tile * kPair + (int)rank) * kBM;
        const uint32_t bytes = kPair * (kTileBytes + (uint32_t)(boxes * box_rows) * kRowBytes);
        for (int kb = 0; kb < g.k_blocks; kb++) {
          if (!mbar_wait(&s.empty[slot], phase ^ 1)) { failed = true; break; }
          if (rank == 0) mbar_expect_tx(&s.full[slot], bytes);
          const uint32_t bar = kPair == 2 ? map_to_cta(&s.full[slot], 0) : smem_u32(&s.full[slot]);
          tma_load_3d<kPair>(s.a[slot], &map_w, bar, kb * kBK, feature0, at.expert);
          for (int b = 0; b < boxes; b++)
            tma_load_2d<kPair>(s.b[slot] + b * box_rows * kRowBytes, map_box, bar, kb * kBK,
                               row0 + b * box_rows);
          if (++slot == kRing) { slot = 0; phase ^= 1; }
        }
      }
      // copies still in flight land before the CTA's shared memory is given back
      if (failed)
        for (int i = 0; i < 1024; i++) __nanosleep(1000);
    }
  } else if (warp == 1) {
    if (lane == 0 && rank == 0) {
      int slot = 0;
      uint32_t phase = 0;
      int acc = 0;
      uint32_t acc_phase = 0;
      for (int t = group; t < total_tiles && !failed; t += groups) {
        const TileAt at = tile_at(s, g.experts, g.m_tiles, t);
        const uint32_t idesc = umma_idesc<kPair>(at.width);
        if (!mbar_wait(&s.acc_empty[acc], acc_phase ^ 1)) { failed = true; break; }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t d = tmem + (uint32_t)acc * kBN;
        for (int kb = 0; kb < g.k_blocks; kb++) {
          if (!mbar_wait(&s.full[slot], phase)) { failed = true; break; }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint64_t da = umma_desc(s.a[slot]);
          const uint64_t db = umma_desc(s.b[slot]);
#pragma unroll
          for (int k = 0; k < kBK / kUmmaK; k++) {
            // 16 bf16 = 32 bytes further along K inside the swizzled row: +2 in 16-byte units
            umma_bf16<kPair>(d, da + 2 * k, db + 2 * k, idesc, (kb | k) != 0);
          }
          umma_commit<kPair>(&s.empty[slot]);  // free once these MMAs have read the slot
          if (++slot == kRing) { slot = 0; phase ^= 1; }
        }
        if (failed) break;
        umma_commit<kPair>(&s.acc_full[acc]);  // complete once they have finished
        if (++acc == 2) { acc = 0; acc_phase ^= 1; }
      }
    }
  } else {
    // epilogue: this warp reads the 32 accumulator lanes (features) of quarter warp % 4
    const int quarter = warp & 3;
    int acc = 0;
    uint32_t acc_phase = 0;
    int buffer = 0;
    const int my_row = lane >> 2;         // of 8 rows stored at a time
    const int my_piece = (lane & 3) * 8;  // 16 bytes of the row's 64
    for (int t = group; t < total_tiles && !failed; t += groups) {
      const TileAt at = tile_at(s, g.experts, g.m_tiles, t);
      const long long first_row = (long long)s.row_base[at.expert] + at.row0;
      const long long left = g.total_rows - first_row;
      const int rows = at.rows < left ? at.rows : (int)(left > 0 ? left : 0);
      __nv_bfloat16* const out =
          g.out + first_row * g.N + (long long)(at.m_tile * kPair + (int)rank) * kBM +
          quarter * 32 + my_piece;
      if (!mbar_wait(&s.acc_full[acc], acc_phase)) { failed = true; break; }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll 1
      for (int c0 = 0; c0 < rows; c0 += 32) {
        uint32_t v[32];
        tmem_load_32(tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(acc * kBN + c0), v);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        // two buffers: the barrier below also says that everybody has read this one's last rows
        __nv_bfloat16* const turn = s.turn[quarter][buffer];
        buffer ^= 1;
#pragma unroll
        for (int i = 0; i < 16; i++) {
          float lo = __uint_as_float(v[2 * i]);
          float hi = __uint_as_float(v[2 * i + 1]);
          if (g.relu) { lo = fmaxf(lo, 0.f); hi = fmaxf(hi, 0.f); }
          const __nv_bfloat162 p = __floats2bfloat162_rn(lo, hi);
          turn[(2 * i) * 32 + lane] = p.x;
          turn[(2 * i + 1) * 32 + lane] = p.y;
        }
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 4; i++) {
          const int r = i * 8 + my_row;
          if (c0 + r < rows)
            *reinterpret_cast<uint4*>(out + (long long)(c0 + r) * g.N) =
                *reinterpret_cast<const uint4*>(turn + r * 32 + my_piece);
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) {
        if (rank == 0) mbar_arrive(&s.acc_empty[acc]);
        else mbar_arrive_cluster(map_to_cta(&s.acc_empty[acc], 0));
      }
      if (++acc == 2) { acc = 0; acc_phase ^= 1; }
    }
  }
  if (failed) atomicExch(g.error, BRT_ERR_TIMEOUT);
  __syncwarp();  // the single-lane roles rejoin their warps before the barrier

  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  group_sync<kPair>();  // nobody leaves while the peer may still signal its barriers
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (warp == 1) {
    if constexpr (kPair == 2)
      asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                   "r"(kTmemCols)
                   : "memory");
    else
      asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                   "r"(kTmemCols)
                   : "memory");
  }
}

}  // namespace
}  // namespace brt_b200

using namespace brt_b200;

namespace {

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                  const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// The driver's tensor-map encoder, looked up through the runtime (no link against libcuda).
EncodeTiledFn encode_tiled() {
  static EncodeTiledFn fn = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult found;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &found) !=
            cudaSuccess ||
        found != cudaDriverEntryPointSuccess)
      p = nullptr;
    return reinterpret_cast<EncodeTiledFn>(p);
  }();
  return fn;
}

template <int kPair>
int launch_expert_gemm(const CUtensorMap& map_w, const RowMaps& map_r, const GemmArgs& g,
                       cudaStream_t st) {
  const size_t smem = sizeof(GemmSmem<kPair>) + 1024;
  static thread_local int configured_device = -1;
  int dev = 0;
  BRT_CUDA_TRY(cudaGetDevice(&dev));
  if (configured_device != dev) {
    BRT_CUDA_TRY(cudaFuncSetAttribute(expert_gemm_kernel<kPair>,
                                      cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    configured_device = dev;
  }
  cudaLaunchAttribute cluster;
  cluster.id = cudaLaunchAttributeClusterDimension;
  cluster.val.clusterDim.x = kPair;
  cluster.val.clusterDim.y = 1;
  cluster.val.clusterDim.z = 1;
  cudaLaunchConfig_t config = {};
  config.gridDim = dim3((unsigned)(sm_count() / kPair * kPair));
  config.blockDim = dim3(kThreads);
  config.dynamicSmemBytes = smem;
  config.stream = st;
  config.attrs = &cluster;
  config.numAttrs = 1;
  const KernelTimer timer("expert_gemm_kernel", st);
  BRT_CUDA_TRY(cudaLaunchKernelEx(&config, expert_gemm_kernel<kPair>, map_w, map_r, g));
  note_launch();
  return BRT_OK;
}

}  // namespace

extern "C" {

BRT_API int brt_grouped_expert_gemm(const void* rows, const void* weights, void* out,
                                    const int32_t* loads, int path_num, int64_t total_rows,
                                    int32_t max_path_load, int64_t in_features,
                                    int64_t out_features, int relu, void* error_word,
                                    void* stream) {
  clear_error();
  BRT_REQUIRE(path_num > 0 && path_num <= kMaxExperts, "path_num %d outside [1, %d]", path_num,
              kMaxExperts);
  BRT_REQUIRE(total_rows >= 0 && max_path_load >= 0, "negative size");
  BRT_REQUIRE(loads != nullptr && error_word != nullptr, "loads or error_word is null");
  if (in_features <= 0 || out_features <= 0 || in_features % kBK != 0 || out_features % 128 != 0)
    return set_error(BRT_ERR_UNSUPPORTED,
                     "the tensor-core expert GEMM needs in_features %% %d == 0 and "
                     "out_features %% 128 == 0 (got %lld, %lld)",
                     kBK, (long long)in_features, (long long)out_features);
  // a pair of CTAs computes 256 features; an odd multiple of 128 leaves half a pair idle on
  // the last tile, and single CTAs do not
  const int pair = out_features % 256 == 0 ? 2 : 1;
  if (total_rows == 0) return BRT_OK;
  BRT_REQUIRE(rows != nullptr && weights != nullptr && out != nullptr, "null pointer argument");
  BRT_REQUIRE(aligned_to(rows, 16) && aligned_to(weights, 16) && aligned_to(out, 16),
              "rows, weights and out must be 16-byte aligned");
  BRT_REQUIRE(total_rows <= 0x7fffffffLL, "more than 2^31-1 rows");
  EncodeTiledFn encode = encode_tiled();
  if (encode == nullptr)
    return set_error(BRT_ERR_CUDA, "the driver does not offer cuTensorMapEncodeTiled");

  alignas(64) CUtensorMap map_w;
  alignas(64) RowMaps map_r;
  for (int i = 0; i < kBoxSizes; i++) {
    const cuuint64_t dims[2] = {(cuuint64_t)in_features, (cuuint64_t)total_rows};
    const cuuint64_t strides[1] = {(cuuint64_t)in_features * 2};
    const cuuint32_t box[2] = {kBK, (cuuint32_t)((i + 1) * kBoxStep)};
    const cuuint32_t elem[2] = {1, 1};
    const CUresult r = encode(&map_r.box[i], CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2,
                              const_cast<void*>(rows), dims, strides, box, elem,
                              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                              CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS)
      return set_error(BRT_ERR_CUDA, "cuTensorMapEncodeTiled(rows) failed with %d", (int)r);
  }
  {
    const cuuint64_t dims[3] = {(cuuint64_t)in_features, (cuuint64_t)out_features,
                                (cuuint64_t)path_num};
    const cuuint64_t strides[2] = {(cuuint64_t)in_features * 2,
                                   (cuuint64_t)in_features * out_features * 2};
    const cuuint32_t box[3] = {kBK, kBM, 1};
    const cuuint32_t elem[3] = {1, 1, 1};
    const CUresult r = encode(&map_w, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3,
                              const_cast<void*>(weights), dims, strides, box, elem,
                              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                              CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS)
      return set_error(BRT_ERR_CUDA, "cuTensorMapEncodeTiled(weights) failed with %d", (int)r);
  }
  GemmArgs g;
  g.loads = loads;
  g.out = static_cast<__nv_bfloat16*>(out);
  g.error = static_cast<int*>(error_word);
  g.experts = path_num;
  g.max_path_load = max_path_load;
  g.m_tiles = (int)(out_features / (kBM * pair));
  g.k_blocks = (int)(in_features / kBK);
  g.N = out_features;
  g.total_rows = total_rows;
  g.relu = relu != 0;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int rc = pair == 2 ? launch_expert_gemm<2>(map_w, map_r, g, st)
                           : launch_expert_gemm<1>(map_w, map_r, g, st);
  if (rc != BRT_OK) return rc;
  BRT_LAUNCH_CHECK("expert_gemm_kernel");
  return BRT_OK;
}

}  // extern "C"
