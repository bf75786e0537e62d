// scatter_add with the aten CPU kernel's summation order (bit-identical fp results).
//
// For every destination element the contributions src[p] are added one after another in
// ascending p[dim], starting from self, in fp32 (bf16/f16 tensors accumulate in fp32 and
// round once at the end) -- exactly what the sequential CPU loop does. Atomics cannot
// reproduce that order, so ordering is made structural. self is viewed as
// [outer, rows, cols] with `rows` the scatter dimension:
//
//   strip kernel (cols > 1): a CTA owns a strip of 4 output columns and keeps it as fp32
//     in shared memory (column-major, so random destination rows spread over the banks;
//     64 KB at 4096 rows, so two CTAs share an SM). Source rows stream through a cp.async
//     ring of 128-row tiles (index and value segments of the 4 columns). Two warps share
//     one column, split by the parity of the destination row, and each walks a tile 32
//     source rows at a time, lane = source row. Whether two lanes of a step hit the same
//     destination is screened with a tiny per-warp tag table (each lane drops its id at a
//     slot hashed from the destination and reads it back); only on a clash is the rank of
//     every lane among EARLIER rows with the same destination taken (one match over the
//     warp) and the additions applied rank by rank: source-row order is kept.
//   row kernel (cols == 1, i.e. the scatter dimension is the last one): a warp owns two
//     rows of `outer`, their destination rows sit in shared memory, and the 16 lanes of a
//     row read 16 consecutive source positions (coalesced) with the same screen and ranks.
//   bins (matrices too tall for a strip, or off its grid): contributions are sorted by bins of
//     destination rows, in source order, and a warp adds up a bin's in shared memory.
//   chains and buckets (neither fits): contributions are chained or grouped by destination
//     in global memory, and a thread adds up each destination's in order.
//   Destinations that do not fit in shared memory are processed in windows (each window
//     re-scans the sources); HBM traffic is the algorithmic minimum otherwise: self, index
//     and src read once, out written once.
//   line kernel (any strides / ragged shapes): one thread per "line" applies its
//     contributions sequentially in global memory on an fp32 accumulator.
#include <cuda_pipeline.h>

#include <type_traits>

#include "b200_common.cuh"
#include "tma_common.cuh"

namespace b200 {

constexpr int kStripCols = 4;
constexpr int kTileRows = 128;
constexpr int kStripThreads = 256;  // 8 warps: (column, destination parity)
constexpr int kSmemBudget = 220 * 1024;
constexpr int kStripSmemTarget = 110 * 1024;  // two strip CTAs per SM when the destination fits

// A CTA touches only a 16- or 32-byte segment of every row it reads (its 4 columns); the
// CTAs of the neighbouring strips read the neighbouring segments at about the same time.
// Asking L2 to fetch 256 bytes around each request turns those per-CTA slivers into full
// DRAM bursts: one CTA misses, its seven neighbours hit in L2.
__device__ __forceinline__ void cp_async8_wide(void* smem_dst, const void* gsrc) {
  asm volatile("cp.async.ca.shared.global.L2::256B [%0], [%1], 8;" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(smem_dst))), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void cp_async4_wide(void* smem_dst, const void* gsrc) {
  asm volatile("cp.async.ca.shared.global.L2::256B [%0], [%1], 4;" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(smem_dst))), "l"(gsrc) : "memory");
}
__device__ __forceinline__ uint4 ld_wide(const uint4* p) {
  uint4 v;
  asm volatile("ld.global.L2::256B.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ uint2 ld_wide(const uint2* p) {
  uint2 v;
  asm volatile("ld.global.L2::256B.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
  return v;
}

__device__ __forceinline__ void flag_oob(uint32_t* status) {
  if (status) atomicOr(status, B200_DEV_INDEX_OOB);
}

// Rank of this lane among the EARLIER in-order elements of its own group of adjacent lanes that carry the same destination `k`
// (negative k = nothing to apply; the rank is not used then). `pos` is the lane's position inside its group. (One match over the
// warp: with a shuffle and a comparison per earlier lane, fp16 30000 x 300 onto 64 rows took 470 us, 308 so.)
__device__ __forceinline__ int rank_among_earlier(int k, int pos) {
  const int lane = threadIdx.x & 31;
  const uint32_t same = __match_any_sync(0xffffffffu, k);
  return __popc(same & (((1u << pos) - 1u) << (lane - pos)));
}
// Same-destination lanes add one rank after the other, so the in-order sequence is kept.
__device__ __forceinline__ void apply_in_rank_order(float* col, int k, float v, int rank) {
  const int rounds = __reduce_max_sync(0xffffffffu, k >= 0 ? rank : 0);
  for (int t = 0; t <= rounds; ++t) {
    if (k >= 0 && rank == t) col[k] += v;
    __syncwarp();
  }
}

// One in-order step of a warp: GROUP adjacent lanes hold consecutive in-order elements of
// one independent unit (`unit` tells the groups of a warp apart), `col` is that unit's fp32
// destination array in shared memory. A cheap screen makes the ranking rare: every
// lane drops its lane id into a small per-warp table at a slot hashed from (destination,
// unit) and reads it back. If all lanes read their own id, no two lanes share a slot, hence
// no two lanes share a destination, and the additions are applied in one go. A clash (a
// real duplicate or a slot collision) falls back to ranking.
constexpr int kTagSlots = 2048;
template <int GROUP, int SLOTS = kTagSlots>
__device__ __forceinline__ void ordered_step(float* col, unsigned char* tags, int k, float v, int unit, int pos, int lane) {
  constexpr int kUnits = 32 / GROUP;  // groups per warp share one table: fold the unit into the slot
  const int slot = (k * kUnits + unit) & (SLOTS - 1);
  if (k >= 0) tags[slot] = static_cast<unsigned char>(lane);
  __syncwarp();
  const bool lost = k >= 0 && tags[slot] != static_cast<unsigned char>(lane);
  if (!__any_sync(0xffffffffu, lost)) {  // the vote also orders these reads before the next step's writes
    if (k >= 0) col[k] += v;
    __syncwarp();
  } else {
    apply_in_rank_order(col, k, v, rank_among_earlier(k, pos));
  }
}

// ------------------------------------------------------------------ strip kernel (cols > 1)
// Nothing is done where `only_if` points to a zero.
struct StripArgs {
  int64_t outer, rows, cols;         // self / out: [outer, rows, cols] contiguous
  int64_t idx_outer, idx_rows, idx_cols;
  int64_t idx_so, idx_sr, src_so, src_sr;  // element strides of index / src (inner stride 1)
  int win_rows;                      // destination rows held in shared memory per pass
  int stages;                        // cp.async ring depth
};

template <typename T>
__global__ void __launch_bounds__(kStripThreads, 2)
scatter_add_strip(const T* __restrict__ self, const int64_t* __restrict__ index, const T* __restrict__ src, T* __restrict__ out, StripArgs A, const int* only_if, uint32_t* status) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  after_grids_before();
  if (only_if && *only_if == 0) return;
  constexpr int kIdxTile = kTileRows * kStripCols * 8, kSrcTile = kTileRows * kStripCols * static_cast<int>(sizeof(T));
  unsigned char* ring = smem_raw;                                                                             // stages x (idx tile, src tile)
  unsigned char* tags = smem_raw + static_cast<size_t>(A.stages) * (kIdxTile + kSrcTile) + (threadIdx.x >> 5) * kTagSlots;  // one screening table per warp
  float* strip = reinterpret_cast<float*>(smem_raw + static_cast<size_t>(A.stages) * (kIdxTile + kSrcTile) + (kStripThreads / 32) * kTagSlots);  // [8][win_rows]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int mycol = warp >> 1, myparity = warp & 1;
  using RowSeg = typename std::conditional<sizeof(T) == 4, uint4, uint2>::type;  // the 4 strip columns of one row
  const int64_t nstrips = A.cols / kStripCols;
  const int64_t ntiles = (A.idx_rows + kTileRows - 1) / kTileRows;

  for (int64_t item = blockIdx.x; item < A.outer * nstrips; item += gridDim.x) {
    const int64_t o = item / nstrips, j0 = (item - o * nstrips) * kStripCols;
    const T* self_o = self + o * A.rows * A.cols;
    T* out_o = out + o * A.rows * A.cols;
    const bool active = j0 < A.idx_cols && o < A.idx_outer && A.idx_rows > 0;
    for (int64_t r0 = 0; r0 < A.rows; r0 += A.win_rows) {
      const int wrows = static_cast<int>(A.rows - r0 < A.win_rows ? A.rows - r0 : A.win_rows);
      // ---- stage self[r0 : r0 + wrows, j0 : j0 + 4] column-major as fp32 (8 loads in flight per thread)
      for (int q0 = 0; q0 < wrows; q0 += kStripThreads * 8) {
        RowSeg seg[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const int r = q0 + u * kStripThreads + tid;
          if (r < wrows) seg[u] = ld_wide(reinterpret_cast<const RowSeg*>(self_o + (r0 + r) * A.cols + j0));
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const int r = q0 + u * kStripThreads + tid;
          if (r < wrows) {
            const T* e = reinterpret_cast<const T*>(&seg[u]);
#pragma unroll
            for (int c = 0; c < kStripCols; ++c) strip[c * A.win_rows + r] = to_f32(e[c]);
          }
        }
      }
      if (active) {
        // Tiles are staged TRANSPOSED ([column][row]) with 8-byte (index) and 4-byte (value)
        // cp.async granules: four adjacent threads still read one contiguous 32-byte index
        // segment of a source row, and a warp later reads its column with unit stride (no
        // bank conflicts). 16-bit values travel as column pairs.
        constexpr int kValCols = sizeof(T) == 4 ? kStripCols : kStripCols / 2;  // 4-byte granules per row
        const int64_t* idx_g = index + o * A.idx_so + j0;
        const uint32_t* src_g = reinterpret_cast<const uint32_t*>(src + o * A.src_so + j0);
        const int64_t src_sr32 = A.src_sr * static_cast<int64_t>(sizeof(T)) / 4;  // source row pitch in 4-byte units
        auto issue_tile = [&](int tile, int slot) {
          if (tile < ntiles) {
            int64_t* idx_s = reinterpret_cast<int64_t*>(ring + static_cast<size_t>(slot) * (kIdxTile + kSrcTile));
            uint32_t* src_s = reinterpret_cast<uint32_t*>(reinterpret_cast<unsigned char*>(idx_s) + kIdxTile);
            const int64_t i0 = static_cast<int64_t>(tile) * kTileRows;
            const int c = tid & 3, rbase = tid >> 2;  // 256 threads = 64 rows x 4 columns per sweep
#pragma unroll
            for (int u = 0; u < kTileRows / 64; ++u) {
              const int r = rbase + u * 64;
              if (i0 + r < A.idx_rows) {
                cp_async8_wide(idx_s + c * kTileRows + r, idx_g + (i0 + r) * A.idx_sr + c);
                if (c < kValCols) cp_async4_wide(src_s + c * kTileRows + r, src_g + (i0 + r) * src_sr32 + c);
              }
            }
          }
          __pipeline_commit();  // one group per tile slot, empty past the end, so the wait depth stays constant
        };
        const int nt = static_cast<int>(ntiles);
        for (int sidx = 0; sidx < A.stages - 1; ++sidx) issue_tile(sidx, sidx);
        float* col = strip + static_cast<int64_t>(mycol) * A.win_rows;
        int slot = 0, fill_slot = A.stages - 1;
        for (int tile = 0; tile < nt; ++tile) {
          __pipeline_wait_prior(A.stages - 2);  // this thread's copies of tile `tile` have landed
          __syncthreads();                      // ... everyone's have; all warps are also done with tile - 1
          issue_tile(tile + A.stages - 1, fill_slot);  // refills the slot that tile - 1 used
          const int64_t* idx_s = reinterpret_cast<const int64_t*>(ring + static_cast<size_t>(slot) * (kIdxTile + kSrcTile));
          const T* src_s = reinterpret_cast<const T*>(reinterpret_cast<const unsigned char*>(idx_s) + kIdxTile);
          const int64_t i0 = static_cast<int64_t>(tile) * kTileRows;
          constexpr int kSteps = kTileRows / 32;
          int k[kSteps];
          float v[kSteps];
#pragma unroll
          for (int st = 0; st < kSteps; ++st) {
            const int r = st * 32 + lane;
            k[st] = -1 - lane;
            v[st] = 0.f;
            if (i0 + r < A.idx_rows) {
              const int64_t key = idx_s[mycol * kTileRows + r];
              if (key < 0 || key >= A.rows) flag_oob(status);
              else if (key >= r0 && key < r0 + wrows && (static_cast<int>(key) & 1) == myparity) {
                k[st] = static_cast<int>(key - r0);
                // fp32: [column][row]; 16-bit: [column pair][row][2]
                v[st] = sizeof(T) == 4 ? to_f32(src_s[mycol * kTileRows + r]) : to_f32(src_s[((mycol >> 1) * kTileRows + r) * 2 + (mycol & 1)]);
              }
            }
          }
#pragma unroll
          for (int st = 0; st < kSteps; ++st) ordered_step<32>(col, tags, k[st], v[st], 0, lane, lane);
          if (++slot == A.stages) slot = 0;
          if (++fill_slot == A.stages) fill_slot = 0;
        }
        __pipeline_wait_prior(0);
      }
      __syncthreads();
      // ---- write the window back, rounding once
      for (int r = tid; r < wrows; r += kStripThreads) {
        RowSeg seg;
        T* e = reinterpret_cast<T*>(&seg);
#pragma unroll
        for (int c = 0; c < kStripCols; ++c) e[c] = from_f32<T>(strip[c * A.win_rows + r]);
        __stcs(reinterpret_cast<RowSeg*>(out_o + (r0 + r) * A.cols + j0), seg);
      }
      __syncthreads();  // the strip is rewritten by the next window / item
    }
  }
}

// ------------------------------------------------------------------ wide strip kernel
// The strip kernel again, for destinations of at most 4096 rows, sized for the memory
// system instead of for occupancy. A CTA owns EIGHT columns (its fp32 strip is 128 KB at
// 4096 rows: one CTA per SM), so every source row contributes a 64-byte index segment and
// a 32-byte (fp32) value segment -- whole sectors.
// Source rows arrive in tiles of 128 rows through a ring filled by the copy engine: a ninth
// warp issues two tiled TMA loads per tile (index box 8 x 128 int64 with the 64-byte swizzle,
// value box 8 x 128 with the 32-byte swizzle: the 16-byte chunks of a staged row are XORed
// with the row number, so the 32 rows a warp reads of one column spread over the banks) onto
// the tile's `full` mbarrier, as soon as the eight compute warps have released the slot on its
// `empty` mbarrier. The compute warps never meet at a CTA-wide barrier inside a strip: each
// owns one column, waits for a tile, walks it 32 source rows at a time (lane = source row) and
// releases it, so a warp that met more clashes than its neighbours falls behind by a few
// tiles instead of holding all of them up, and the next strip's first tiles load while this
// strip is written back. Every wait is bounded (a wait that runs out raises
// B200_DEV_WAIT_TIMEOUT, and the CTA finishes its barriers and leaves).
// With one or two warps per scheduler the kernel runs at the speed of its dependent
// instruction chain, so the step is kept to a couple of dozen instructions: every offset
// that depends only on the lane is computed once, row-bound tests exist only for the
// ragged last tile, and the steps are software-pipelined by hand (the compiler must assume
// that the tag table and the strip alias): while step st waits for its tag read-back and
// for the strip value it read ahead, keys, values and tags of step st + 1 are under way.
constexpr int kWideCols = 8;
constexpr int kWideTileRows = 128;
constexpr int kWideComputeThreads = 256;  // eight warps: one column each
constexpr int kWideThreads = 288;         // ... and the warp that feeds the ring
constexpr int kWideTagSlots = 4096;       // one table per warp, exact up to 4096 destinations ...
constexpr int kWideDummies = 32;          // ... plus a slot (and a strip element) per lane for rows that have nothing to add
constexpr int kWideSelfRows = 256;        // rows of the destination strip per ring slot on its way in (the largest TMA box)
constexpr int kWideOutRows = 32;          // rows of the destination strip per tiled store on its way out: a warp's share of a slab
constexpr int kWideOutBlocks = 4;         // staging blocks per warp for those stores
constexpr int kWideStages = 5;            // 12 KB tiles (fp32): 48 KB of source rows in flight per SM
constexpr int kWideMaxRows = 4096;
constexpr uint64_t kWideWaitLimitNs = 2000000000ull;

__device__ __forceinline__ void compute_warps_barrier() { asm volatile("bar.sync 1, %0;" ::"n"(kWideComputeThreads) : "memory"); }

template <typename T>
__global__ void __launch_bounds__(kWideThreads, 1)
scatter_add_strip_wide(const __grid_constant__ CUtensorMap map_idx, const __grid_constant__ CUtensorMap map_src, const __grid_constant__ CUtensorMap map_self, const __grid_constant__ CUtensorMap map_out, StripArgs A, uint32_t* status) {
  extern __shared__ unsigned char smem_dyn[];
  unsigned char* smem_raw = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_dyn) + 1023) & ~static_cast<uintptr_t>(1023));  // the swizzle patterns repeat every 512 bytes
  constexpr int kIdxTile = kWideTileRows * kWideCols * 8;                            // 8 KB: [row][4 chunks of 2 indices]
  constexpr int kSrcRow = kWideCols * static_cast<int>(sizeof(T));                   // 32 or 16 bytes of values per row
  constexpr int kSrcTile = kWideTileRows * kSrcRow;
  constexpr int kSrcChunks = kSrcRow / 16;                                           // 16-byte chunks per value row: 2 or 1
  constexpr int kTile = kIdxTile + kSrcTile;                                         // 12 KB / 10 KB: every slot starts on a 1 KB boundary
  unsigned char* ring = smem_raw;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  unsigned char* tags = smem_raw + kWideStages * kTile + (warp & 7) * (kWideTagSlots + kWideDummies);
  float* strip = reinterpret_cast<float*>(smem_raw + kWideStages * kTile + 8 * (kWideTagSlots + kWideDummies));  // [8][rows + 32]
  const int rows = static_cast<int>(A.rows);
  const int cstride = rows + kWideDummies;  // a column of the strip, then one dummy element per lane
  uint64_t* bars = reinterpret_cast<uint64_t*>(reinterpret_cast<unsigned char*>(strip) + static_cast<size_t>(kWideMaxRows + kWideDummies) * kWideCols * 4);  // full[S], empty[S]
  volatile uint32_t* abort_flag = reinterpret_cast<volatile uint32_t*>(bars + 2 * kWideStages);
  const uint32_t bar_base = smem_u32(bars);
  auto full_bar = [&](int s) { return bar_base + 8u * s; };
  auto empty_bar = [&](int s) { return bar_base + 8u * (kWideStages + s); };
  const int64_t nstrips = A.cols / kWideCols;
  const int ntiles = static_cast<int>((A.idx_rows + kWideTileRows - 1) / kWideTileRows);
  constexpr int kSegsPerRow = kSrcRow / 16, kPerSeg = 16 / static_cast<int>(sizeof(T));  // 16-byte segments of a destination row
  constexpr int kSelfBytes = kWideSelfRows * kSrcRow;  // a slab of the destination strip fits a ring slot
  static_assert(kSelfBytes <= kTile, "a slab of the destination strip travels in one ring slot");
  static_assert(8 * kWideOutBlocks * kWideOutRows * 32 <= 8 * (kWideTagSlots + kWideDummies), "the blocks on their way out are staged in the tag tables");
  static_assert(kWideSelfRows == kWideComputeThreads && kWideOutRows == 32, "thread t owns row t of every slab, on the way in and on the way out");
  const int nslabs = (static_cast<int>(A.rows) + kWideSelfRows - 1) / kWideSelfRows;

  if (tid == 0) {
    for (int s = 0; s < kWideStages; ++s) {
      mbar_init(full_bar(s), 1);   // the producer's expect_tx arrival; the copies complete the bytes
      mbar_init(empty_bar(s), 8);  // one arrival per compute warp
    }
    *abort_flag = 0u;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();

  if (warp == 8) {
    // ------------------------------------------------------------ producer: the ring, tile after tile, strip after strip
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int64_t item = blockIdx.x; item < A.outer * nstrips && ok; item += gridDim.x) {
        const int64_t o = item / nstrips, j0 = (item - o * nstrips) * kWideCols;
        for (int slab = 0; slab < nslabs && ok; ++slab) {  // self[:, j0 : j0 + 8], 256 rows per slot
          if (!mbar_wait(empty_bar(stage), phase ^ 1u, abort_flag, kWideWaitLimitNs)) { ok = false; break; }
          mbar_expect_tx(full_bar(stage), kSelfBytes);
          tma_load_3d(smem_u32(ring) + stage * kTile, &map_self, full_bar(stage), static_cast<int>(j0), slab * kWideSelfRows, static_cast<int>(o));
          if (++stage == kWideStages) { stage = 0; phase ^= 1u; }
        }
        if (!(j0 < A.idx_cols && o < A.idx_outer && ntiles > 0)) continue;
        for (int tile = 0; tile < ntiles && ok; ++tile) {
          if (!mbar_wait(empty_bar(stage), phase ^ 1u, abort_flag, kWideWaitLimitNs)) { ok = false; break; }
          const uint32_t dst = smem_u32(ring) + stage * kTile;
          mbar_expect_tx(full_bar(stage), kTile);  // a box counts in full, rows past the end of the tensor arrive as zeros
          tma_load_3d(dst, &map_idx, full_bar(stage), static_cast<int>(j0), tile * kWideTileRows, static_cast<int>(o));
          tma_load_3d(dst + kIdxTile, &map_src, full_bar(stage), static_cast<int>(j0), tile * kWideTileRows, static_cast<int>(o));
          if (++stage == kWideStages) { stage = 0; phase ^= 1u; }
        }
      }
      if (!ok) {
        *abort_flag = 1u;
        if (status) atomicOr(status, B200_DEV_WAIT_TIMEOUT);
      }
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------ compute warps: lane reads row `lane` (+ 32 per step) of column `warp`
    const int c_idx_off = lane * 64 + (((warp >> 1) ^ ((lane >> 1) & 3)) << 4) + (warp & 1) * 8;
    const int c_src_off = kIdxTile + lane * kSrcRow + (kSrcChunks == 2 ? (((warp >> 2) ^ ((lane >> 2) & 1)) << 4) : 0) + (warp & (kPerSeg - 1)) * static_cast<int>(sizeof(T));
    float* col = strip + warp * cstride;
    const int dummy = rows + lane;  // where a lane with nothing to add "adds" zero: its own slot, so it never clashes
    const uint32_t ring_a = smem_u32(ring), tags_a = smem_u32(tags), col_a = smem_u32(col), strip_a = smem_u32(strip);
    const uint32_t out_stage_a = ring_a + kWideStages * kTile + warp * (kWideOutBlocks * kWideOutRows * 32);  // four blocks of 32 rows per warp inside the tag tables
    int out_parity = 0;
    // Rows r0 .. r0 + 31 of the finished strip (this warp's share of a slab) leave for
    // out[po, r0 .., pj0 : pj0 + 8], rounded once: back to rows of 8 values in one of the warp's
    // four staging blocks inside the tag tables (idle between tile loops), then one tiled store,
    // which clips at the last row. The warp only waits for the engine to have read the block it
    // staged four stores ago.
    auto store_rows = [&](int r0, int64_t pj0, int64_t po) {
      if (r0 >= rows) return;
      if (lane == 0) tma_store_wait_read_but<kWideOutBlocks - 1>();
      __syncwarp();
      const int r = r0 + lane < rows ? r0 + lane : rows - 1;  // rows past the end are clipped by the store
      const uint32_t block_a = out_stage_a + out_parity * (kWideOutRows * 32);
      float f[kWideCols];
#pragma unroll
      for (int c = 0; c < kWideCols; ++c) asm volatile("ld.shared.f32 %0, [%1];" : "=f"(f[c]) : "r"(strip_a + 4u * static_cast<uint32_t>(c * cstride + r)) : "memory");
#pragma unroll
      for (int h = 0; h < kSegsPerRow; ++h) {
        const uint4 seg = narrow<T>(f + h * kPerSeg);
        asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(block_a + lane * kSrcRow + h * 16), "r"(seg.x), "r"(seg.y), "r"(seg.z), "r"(seg.w) : "memory");
      }
      fence_async_smem();
      __syncwarp();
      if (lane == 0) {
        tma_store_3d(&map_out, block_a, static_cast<int>(pj0), r0, static_cast<int>(po));
        tma_store_commit();
      }
      out_parity = (out_parity + 1) & (kWideOutBlocks - 1);
    };
    bool have_prev = false;
    int64_t prev_j0 = 0, prev_o = 0;
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (int64_t item = blockIdx.x; item < A.outer * nstrips; item += gridDim.x) {
      const int64_t o = item / nstrips, j0 = (item - o * nstrips) * kWideCols;
      const bool active = j0 < A.idx_cols && o < A.idx_outer && ntiles > 0;

      // ---- one pass over the strip, 256 rows at a time: the previous item's result leaves, and
      // self[:, j0 : j0 + 8] of this item, which arrives through the ring (256 rows per slot),
      // takes its place column-major as fp32. Thread t owns row t of every slab in both
      // directions, so nothing orders the two but the thread's own program; the 32 lanes of a
      // warp read and write 32 adjacent rows of one column.
      for (int slab = 0; slab < nslabs && ok; ++slab) {
        if (have_prev) store_rows(slab * kWideSelfRows + warp * 32, prev_j0, prev_o);
        int got = 0;
        if (lane == 0) got = mbar_wait(full_bar(stage), phase, abort_flag, kWideWaitLimitNs) ? 1 : 0;
        got = __shfl_sync(0xffffffffu, got, 0);
        if (!got) {
          ok = false;
          if (lane == 0) {
            *abort_flag = 1u;
            if (status) atomicOr(status, B200_DEV_WAIT_TIMEOUT);
          }
          break;
        }
        const uint32_t slab_a = ring_a + stage * kTile + tid * kSrcRow;
        const int r = slab * kWideSelfRows + tid;
#pragma unroll
        for (int h = 0; h < kSegsPerRow; ++h) {
          uint4 seg;
          asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(seg.x), "=r"(seg.y), "=r"(seg.z), "=r"(seg.w) : "r"(slab_a + h * 16));
          float f[kPerSeg];
          widen<T>(seg, f);
          if (r < rows) {
#pragma unroll
            for (int c = 0; c < kPerSeg; ++c) asm volatile("st.shared.f32 [%0], %1;" ::"r"(strip_a + 4u * static_cast<uint32_t>((h * kPerSeg + c) * cstride + r)), "f"(f[c]) : "memory");
          }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(empty_bar(stage));
        if (++stage == kWideStages) { stage = 0; phase ^= 1u; }
      }
      if (lane == 0) tma_store_wait_read();  // the tag tables are free again
      compute_warps_barrier();               // the strip is staged

      if (active) {
        for (int tile = 0; tile < ntiles && ok; ++tile) {
          int got = 0;
          if (lane == 0) got = mbar_wait(full_bar(stage), phase, abort_flag, kWideWaitLimitNs) ? 1 : 0;
          got = __shfl_sync(0xffffffffu, got, 0);
          if (!got) {
            ok = false;
            if (lane == 0) {
              *abort_flag = 1u;
              if (status) atomicOr(status, B200_DEV_WAIT_TIMEOUT);
            }
            break;
          }
          // shared-memory accesses of the step by 32-bit shared addresses (the ring, the tag table
          // and the strip are carved out of one aligned buffer, which hides their address space
          // from the compiler: generic accesses would cost 64-bit address arithmetic per access)
          const uint32_t tile_a = ring_a + stage * kTile;
          const int valid_rows = static_cast<int>(A.idx_rows - static_cast<int64_t>(tile) * kWideTileRows);  // >= 128 except in the last tile
          const bool ragged = valid_rows < kWideTileRows;
          constexpr int kSteps = kWideTileRows / 32;
          unsigned oob = 0u;
          // Every lane always has a destination: a row past the end of the tensor, or an index
          // out of range (reported once per tile), adds zero to the lane's own dummy element.
          // The step below therefore has no per-lane conditions at all -- with two warps per
          // scheduler the kernel runs at the speed of its instruction chain, and every
          // `if (k >= 0)` cost a branch and its reconvergence bookkeeping.
          auto fetch = [&](int st, int& k, float& v) {
            uint32_t lo, hi;
            asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(lo), "=r"(hi) : "r"(tile_a + c_idx_off + st * (32 * 64)));
            float val;
            if (sizeof(T) == 4) {
              asm volatile("ld.shared.f32 %0, [%1];" : "=f"(val) : "r"(tile_a + c_src_off + st * (32 * kSrcRow)));
            } else {
              unsigned short raw;
              asm volatile("ld.shared.u16 %0, [%1];" : "=h"(raw) : "r"(tile_a + c_src_off + st * (32 * kSrcRow)));
              val = to_f32(*reinterpret_cast<const T*>(&raw));
            }
            const bool in_range = hi == 0u && lo < static_cast<uint32_t>(rows);
            const bool in_tensor = !ragged || st * 32 + lane < valid_rows;
            oob |= (in_tensor && !in_range) ? 1u : 0u;
            const bool use = in_tensor && in_range;
            k = use ? static_cast<int>(lo) : dummy;
            v = use ? val : 0.f;
          };
          auto tag_put = [&](int k) { asm volatile("st.shared.u8 [%0], %1;" ::"r"(tags_a + k), "r"(lane) : "memory"); };
          auto tag_get = [&](int k) {
            uint32_t w;
            asm volatile("ld.shared.u8 %0, [%1];" : "=r"(w) : "r"(tags_a + k) : "memory");
            return w;
          };
          auto col_get = [&](int k) {
            float f;
            asm volatile("ld.shared.f32 %0, [%1];" : "=f"(f) : "r"(col_a + 4 * k) : "memory");
            return f;
          };
          auto col_put = [&](int k, float f) { asm volatile("st.shared.f32 [%0], %1;" ::"r"(col_a + 4 * k), "f"(f) : "memory"); };
          int k[2];
          float v[2];
          fetch(0, k[0], v[0]);
          tag_put(k[0]);
#pragma unroll
          for (int st = 0; st < kSteps; ++st) {
            const int cur = st & 1, nxt = cur ^ 1;
            if (st + 1 < kSteps) fetch(st + 1, k[nxt], v[nxt]);
            __syncwarp();  // the tags of step st are written
            const unsigned winner = tag_get(k[cur]);
            const bool lost = winner != static_cast<unsigned>(lane);
            const float old = col_get(k[cur]);  // read ahead; used only by lanes that nothing clashes with
            if (st + 1 < kSteps) tag_put(k[nxt]);  // after this step's read-back, in program order
            const unsigned losers = __ballot_sync(0xffffffffu, lost);
            if (losers == 0u) {
              col_put(k[cur], old + v[cur]);
            } else {
              // All lanes that share a slot read the same tag: the one lane it names is not
              // lost, every other one is. So the lanes in a clash are exactly the losers and
              // the lanes they name; everybody else adds at once, and the few involved add one
              // after the other in lane order, which is source-row order.
              unsigned involved = losers | __reduce_or_sync(0xffffffffu, lost ? 1u << winner : 0u);
              if (__popc(involved) <= 8) {
                if (!((involved >> lane) & 1u)) col_put(k[cur], old + v[cur]);
                while (involved) {
                  const int l = __ffs(involved) - 1;
                  if (lane == l) col_put(k[cur], col_get(k[cur]) + v[cur]);
                  involved &= involved - 1;
                  __syncwarp();
                }
              } else {
                apply_in_rank_order(col, k[cur], v[cur], rank_among_earlier(k[cur], lane));
              }
            }
          }
          if (__any_sync(0xffffffffu, oob != 0u) && lane == 0) flag_oob(status);
          __syncwarp();                                   // every lane is done with the tile ...
          if (lane == 0) mbar_arrive(empty_bar(stage));   // ... and this warp hands its share of the slot back
          if (++stage == kWideStages) { stage = 0; phase ^= 1u; }
        }
      }
      compute_warps_barrier();  // every column of the strip is final
      have_prev = true;
      prev_j0 = j0;
      prev_o = o;
    }
    if (have_prev)  // the last strip of this CTA
      for (int slab = 0; slab < nslabs; ++slab) store_rows(slab * kWideSelfRows + warp * 32, prev_j0, prev_o);
    if (lane == 0) tma_store_wait_all();
  }
  __syncthreads();
  if (*abort_flag) {
    for (int i = 0; i < 64; ++i) __nanosleep(1000);  // copies still under way land before the shared memory is handed on
    __syncthreads();
  }
}

// ------------------------------------------------------------------ row kernel (scatter along the last dim)
struct RowArgs {
  int64_t outer, rows;               // self / out: [outer, rows] contiguous, scatter along `rows`
  int64_t idx_outer, idx_len;        // index / src: [idx_outer, idx_len], inner stride 1
  int64_t idx_so, src_so;
  int win_rows;
};

template <typename T>
__global__ void __launch_bounds__(256) scatter_add_rows(const T* __restrict__ self, const int64_t* __restrict__ index, const T* __restrict__ src, T* __restrict__ out, RowArgs A,
                                                        uint32_t* status) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  const int half = lane >> 4, p16 = lane & 15;  // lanes 0-15: first row of the pair, 16-31: second
  unsigned char* tags = smem_raw + warp * kTagSlots;  // one screening table per warp, ahead of the destination rows
  float* mine = reinterpret_cast<float*>(smem_raw + nwarps * kTagSlots) + (static_cast<int64_t>(warp) * 2 + half) * A.win_rows;
  const int64_t npairs = (A.outer + 1) / 2;
  for (int64_t pair = static_cast<int64_t>(blockIdx.x) * nwarps + warp; pair < npairs; pair += static_cast<int64_t>(gridDim.x) * nwarps) {
    const int64_t o = pair * 2 + half;
    const bool row_ok = o < A.outer;
    const bool active = row_ok && o < A.idx_outer;
    for (int64_t r0 = 0; r0 < A.rows; r0 += A.win_rows) {
      const int wrows = static_cast<int>(A.rows - r0 < A.win_rows ? A.rows - r0 : A.win_rows);
      if (row_ok)
        for (int r = p16; r < wrows; r += 16) mine[r] = to_f32(self[o * A.rows + r0 + r]);
      __syncwarp();
      for (int64_t j0 = 0; j0 < A.idx_len; j0 += 64) {  // warp-uniform trip count
        int k[4];
        float v[4];
#pragma unroll
        for (int s = 0; s < 4; ++s) {
          const int64_t j = j0 + s * 16 + p16;
          k[s] = -1 - lane;
          v[s] = 0.f;
          if (active && j < A.idx_len) {
            const int64_t key = index[o * A.idx_so + j];
            if (key < 0 || key >= A.rows) flag_oob(status);
            else if (key >= r0 && key < r0 + wrows) {
              k[s] = static_cast<int>(key - r0);
              v[s] = to_f32(src[o * A.src_so + j]);
            }
          }
        }
#pragma unroll
        for (int s = 0; s < 4; ++s) ordered_step<16>(mine, tags, k[s], v[s], half, p16, lane);
      }
      if (row_ok)
        for (int r = p16; r < wrows; r += 16) out[o * A.rows + r0 + r] = from_f32<T>(mine[r]);
      __syncwarp();
    }
  }
}

// Few rows, long ones (17 x 2051: nine warps of the kernel above would walk 2051 sources
// each, one global-memory round trip per 64): the destinations of a row are cut into
// `slices` ranges and a warp owns one range of one row. It reads ALL sources of the row (32
// per step, the next step's loads in flight while this one is applied; the other warps of the
// row read the same lines out of L1 / L2) and applies those that fall into its range, in
// source order. The order of the additions into a destination is untouched.
template <typename T>
__global__ void __launch_bounds__(256) scatter_add_rows_sliced(const T* __restrict__ self, const int64_t* __restrict__ index, const T* __restrict__ src, T* __restrict__ out, RowArgs A,
                                                               int slices, int slice_rows, uint32_t* status) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  unsigned char* tags = smem_raw + warp * kTagSlots;
  float* mine = reinterpret_cast<float*>(smem_raw + nwarps * kTagSlots) + static_cast<int64_t>(warp) * slice_rows;
  const int64_t items = A.outer * slices;
  for (int64_t item = static_cast<int64_t>(blockIdx.x) * nwarps + warp; item < items; item += static_cast<int64_t>(gridDim.x) * nwarps) {
    const int64_t o = item / slices;
    const int d = static_cast<int>(item - o * slices);
    const int64_t lo = static_cast<int64_t>(d) * slice_rows;
    const int n = static_cast<int>(A.rows - lo < slice_rows ? A.rows - lo : slice_rows);  // > 0 by the choice of slices
    for (int r = lane; r < n; r += 32) mine[r] = to_f32(self[o * A.rows + lo + r]);
    __syncwarp();
    if (o < A.idx_outer) {
      const int64_t* irow = index + o * A.idx_so;
      const T* srow = src + o * A.src_so;
      int64_t key = lane < A.idx_len ? irow[lane] : -1;
      T val = lane < A.idx_len ? srow[lane] : from_f32<T>(0.f);
      for (int64_t j0 = 0; j0 < A.idx_len; j0 += 32) {
        const int64_t jn = j0 + 32 + lane;
        const int64_t key_n = jn < A.idx_len ? irow[jn] : -1;
        const T val_n = jn < A.idx_len ? srow[jn] : from_f32<T>(0.f);
        const bool real = j0 + lane < A.idx_len;
        if (real && d == 0 && (key < 0 || key >= A.rows)) flag_oob(status);
        const bool take = real && key >= lo && key < lo + n;
        ordered_step<32>(mine, tags, take ? static_cast<int>(key - lo) : -1 - lane, take ? to_f32(val) : 0.f, 0, lane, lane);
        key = key_n;
        val = val_n;
      }
    }
    for (int r = lane; r < n; r += 32) out[o * A.rows + lo + r] = from_f32<T>(mine[r]);
    __syncwarp();
  }
}

// ------------------------------------------------------------------ generic line kernel
struct ScatterArgs {
  int ndim, dim;
  int64_t nlines, dim_len, self_dim_size;
  int64_t shape[B200_MAX_DIMS];  // index shape with shape[dim] forced to 1
  int64_t out_stride[B200_MAX_DIMS], idx_stride[B200_MAX_DIMS], src_stride[B200_MAX_DIMS];
};

template <typename T>
__global__ void __launch_bounds__(128) scatter_add_lines(float* __restrict__ out, const int64_t* __restrict__ index, const T* __restrict__ src, ScatterArgs A, uint32_t* status) {
  const int64_t line = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (line >= A.nlines) return;
  int64_t lin = line, oo = 0, io = 0, so = 0;
  for (int d = A.ndim - 1; d >= 0; --d) {
    const int64_t q = lin / A.shape[d], r = lin - q * A.shape[d];
    oo += r * A.out_stride[d];
    io += r * A.idx_stride[d];
    so += r * A.src_stride[d];
    lin = q;
  }
  const int64_t os = A.out_stride[A.dim], is = A.idx_stride[A.dim], ss = A.src_stride[A.dim];
  for (int64_t k = 0; k < A.dim_len; ++k) {
    const int64_t key = index[io + k * is];
    if (key < 0 || key >= A.self_dim_size) {
      flag_oob(status);
      continue;
    }
    out[oo + key * os] += to_f32(src[so + k * ss]);
  }
}

// ------------------------------------------------------------------ bucket path
// For shapes with little column / row parallelism (tall and narrow, ragged, strided) the
// sources are first grouped by DESTINATION: count per destination (integer atomics -- their
// order does not matter), a segment for each, then every source drops (position along the
// scatter dimension, value) into its destination's segment at an arbitrary slot. One thread
// per destination finally replays its segment in ascending position, i.e. in the aten CPU
// order. Fully parallel over sources and destinations; ~3x the algorithmic traffic.
// Destinations with more than kLightMax contributions go to a CTA-cooperative replay.
constexpr int kLightMax = 32;
constexpr int kHeavyWindow = 4096;

struct BucketArgs {
  int ndim, dim;
  int64_t n_idx, n_self, dim_len, self_dim_size;
  int64_t shape[B200_MAX_DIMS];  // index shape
  int64_t out_stride[B200_MAX_DIMS], idx_stride[B200_MAX_DIMS], src_stride[B200_MAX_DIMS];
};

__device__ __forceinline__ bool bucket_decode(const BucketArgs& A, int64_t p, const int64_t* __restrict__ index, int64_t& dest, int64_t& so, int& pos, uint32_t* status) {
  int64_t oo = 0, io = 0;
  so = 0;
  pos = 0;
  if (A.n_idx <= 0x7fffffffLL) {  // coordinates by 32-bit division (a 64-bit one costs ~5x the instructions)
    uint32_t lin = static_cast<uint32_t>(p);
    for (int d = A.ndim - 1; d >= 0; --d) {
      const uint32_t ext = static_cast<uint32_t>(A.shape[d]);
      const uint32_t q = lin / ext, r = lin - q * ext;
      io += r * A.idx_stride[d];
      so += r * A.src_stride[d];
      if (d == A.dim) pos = static_cast<int>(r);
      else oo += r * A.out_stride[d];
      lin = q;
    }
  } else {
    int64_t lin = p;
    for (int d = A.ndim - 1; d >= 0; --d) {
      const int64_t q = lin / A.shape[d], r = lin - q * A.shape[d];
      io += r * A.idx_stride[d];
      so += r * A.src_stride[d];
      if (d == A.dim) pos = static_cast<int>(r);
      else oo += r * A.out_stride[d];
      lin = q;
    }
  }
  const int64_t key = index[io];
  if (key < 0 || key >= A.self_dim_size) {
    flag_oob(status);
    return false;
  }
  dest = oo + key * A.out_stride[A.dim];
  return true;
}

__global__ void __launch_bounds__(256) bucket_count(const int64_t* __restrict__ index, int* __restrict__ cnt, BucketArgs A, uint32_t* status) {
  for (int64_t p = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; p < A.n_idx; p += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    int64_t dest, so;
    int pos;
    if (bucket_decode(A, p, index, dest, so, pos, nullptr)) atomicAdd(&cnt[dest], 1);
  }
}

// Every counter gets a segment of its size: cursor[i] = first slot. Which part of the pool a
// block of counters gets is decided by one atomic per block, since no result depends on
// where a segment lies: one pass instead of an exclusive scan's three. Counters above `light`
// are listed. The counters start at `zero`.
template <int ITEMS>
__device__ __forceinline__ void assign_segments_of(const int* cnt, int zero, int* cursor, int64_t n, int* total, int light, int* heavy_count,
                                                   int* heavy_list) {
  __shared__ int warp_sums[8];
  __shared__ int block_base;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t base = (static_cast<int64_t>(blockIdx.x) * 256 + threadIdx.x) * ITEMS;
  const bool whole = base + ITEMS <= n && ((reinterpret_cast<uintptr_t>(cnt) | reinterpret_cast<uintptr_t>(cursor)) & 15u) == 0;
  int v[ITEMS], s = 0;
  if (whole) {
#pragma unroll
    for (int q = 0; q < ITEMS / 4; ++q) {
      const int4 t = reinterpret_cast<const int4*>(cnt + base)[q];
      v[4 * q] = t.x; v[4 * q + 1] = t.y; v[4 * q + 2] = t.z; v[4 * q + 3] = t.w;
    }
  } else {
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) v[k] = base + k < n ? cnt[base + k] : zero;
  }
#pragma unroll
  for (int k = 0; k < ITEMS; ++k) {
    v[k] -= zero;
    s += v[k];
    if (v[k] > light) heavy_list[atomicAdd(heavy_count, 1)] = static_cast<int>(base + k);
  }
  int inc = s;
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += y;
  }
  if (lane == 31) warp_sums[warp] = inc;
  __syncthreads();
  int prefix = inc - s, all = 0;
#pragma unroll
  for (int w = 0; w < 8; ++w) {
    if (w < warp) prefix += warp_sums[w];
    all += warp_sums[w];
  }
  if (threadIdx.x == 0) block_base = atomicAdd(total, all);
  __syncthreads();
  prefix += block_base;
  if (whole) {
#pragma unroll
    for (int q = 0; q < ITEMS / 4; ++q) {
      int4 t;
      t.x = prefix; prefix += v[4 * q];
      t.y = prefix; prefix += v[4 * q + 1];
      t.z = prefix; prefix += v[4 * q + 2];
      t.w = prefix; prefix += v[4 * q + 3];
      reinterpret_cast<int4*>(cursor + base)[q] = t;
    }
    return;
  }
#pragma unroll
  for (int k = 0; k < ITEMS; ++k) {
    if (base + k < n) cursor[base + k] = prefix;
    prefix += v[k];
  }
}
template <int ITEMS>
__global__ void __launch_bounds__(256) assign_segments(const int* cnt, int* cursor, int64_t n, int* total, int light, int* heavy_count,
                                                       int* heavy_list) {
  after_grids_before();
  assign_segments_of<ITEMS>(cnt, 0, cursor, n, total, light, heavy_count, heavy_list);
}

template <typename T>
__global__ void __launch_bounds__(256) bucket_fill(const int64_t* __restrict__ index, const T* __restrict__ src, int* __restrict__ cursor, int2* __restrict__ seg,
                                                   BucketArgs A, uint32_t* status) {
  for (int64_t p = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; p < A.n_idx; p += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    int64_t dest, so;
    int pos;
    if (bucket_decode(A, p, index, dest, so, pos, status)) {
      const int slot = atomicAdd(&cursor[dest], 1);
      seg[slot] = make_int2(pos, __float_as_int(to_f32(src[so])));  // (position, value) in one 8-byte store
    }
  }
}

// One thread per destination: replay its segment in ascending source position. The counters start at
// `zero`; nothing is done where `only_if` points to a zero.
template <typename T>
__global__ void __launch_bounds__(256) bucket_replay(const T* __restrict__ self, T* __restrict__ out, const int* cnt, int zero, const int* cursor,
                                                     const int2* seg, int64_t n_self, const int* only_if) {
  after_grids_before();
  if (only_if && *only_if == 0) return;
  for (int64_t d = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; d < n_self; d += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int c = cnt[d] - zero;
    if (c == 0) {
      out[d] = self[d];
    } else if (c <= kLightMax) {
      const int e = cursor[d], b = e - c;
      float acc = to_f32(self[d]);
      int last = -1;
      for (int i = 0; i < c; ++i) {
        int best = 0x7fffffff;
        float bv = 0.f;
        for (int j = b; j < e; ++j) {
          const int2 pv = seg[j];
          if (pv.x > last && pv.x < best) { best = pv.x; bv = __int_as_float(pv.y); }
        }
        acc += bv;
        last = best;
      }
      out[d] = from_f32<T>(acc);
    }
  }
}

// Destinations with long segments: one CTA each. The segment is visited in windows of
// kHeavyWindow source positions; inside a window every element is parked at its position,
// the occupied slots are compacted in order with a block scan, and one thread adds them.
// The counters belong to the destinations, starting at `zero`, or, unless *grouped is set, to the entries of the list
// (`listed_cnt`, may be NULL).
struct HeavyCounters {
  const int* cnt;
  const int* cursor;
  int zero;
  const int* listed_cnt;
  const int* listed_cursor;
  const int* grouped;
};
template <typename T>
__global__ void __launch_bounds__(256) bucket_replay_heavy(const T* __restrict__ self, T* __restrict__ out, HeavyCounters H, const int2* seg, int64_t dim_len,
                                                           const int* heavy_count, const int* heavy_list) {
  __shared__ float slot_val[kHeavyWindow];
  __shared__ unsigned char slot_set[kHeavyWindow];
  __shared__ float ordered[kHeavyWindow];
  __shared__ int warp_sums[8];
  __shared__ int window_count;
  __shared__ float acc_s;
  after_grids_before();
  const int nheavy = *heavy_count;
  const bool by_list = nheavy > 0 && H.listed_cnt && *H.grouped == 0;
  constexpr int kPer = kHeavyWindow / 256;
  for (int h = blockIdx.x; h < nheavy; h += gridDim.x) {
    const int64_t d = heavy_list[h];
    const int e = by_list ? H.listed_cursor[h] : H.cursor[d], b = e - (by_list ? H.listed_cnt[h] : H.cnt[d] - H.zero);
    if (threadIdx.x == 0) acc_s = to_f32(self[d]);
    for (int64_t w0 = 0; w0 < dim_len; w0 += kHeavyWindow) {
      for (int i = threadIdx.x; i < kHeavyWindow; i += 256) slot_set[i] = 0;
      __syncthreads();
      for (int j = b + threadIdx.x; j < e; j += 256) {
        const int2 pv = seg[j];
        const int64_t pj = pv.x;
        if (pj >= w0 && pj < w0 + kHeavyWindow) {
          slot_val[pj - w0] = __int_as_float(pv.y);
          slot_set[pj - w0] = 1;
        }
      }
      __syncthreads();
      int mine = 0;
#pragma unroll
      for (int k = 0; k < kPer; ++k) mine += slot_set[threadIdx.x * kPer + k];
      int inc = mine;
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, inc, o);
        if ((threadIdx.x & 31) >= o) inc += y;
      }
      if ((threadIdx.x & 31) == 31) warp_sums[threadIdx.x >> 5] = inc;
      __syncthreads();
      int prefix = inc - mine;
      for (int w = 0; w < (threadIdx.x >> 5); ++w) prefix += warp_sums[w];
      if (threadIdx.x == 255) window_count = prefix + mine;
#pragma unroll
      for (int k = 0; k < kPer; ++k)
        if (slot_set[threadIdx.x * kPer + k]) ordered[prefix++] = slot_val[threadIdx.x * kPer + k];
      __syncthreads();
      if (threadIdx.x == 0) {
        float acc = acc_s;
        const int n = window_count;
        for (int i = 0; i < n; ++i) acc += ordered[i];
        acc_s = acc;
      }
      __syncthreads();
    }
    if (threadIdx.x == 0) out[d] = from_f32<T>(acc_s);
    __syncthreads();
  }
}

struct BucketScratch {
  int64_t cnt_bytes, cursor_bytes, seg_bytes, heavy_bytes, total;
};
static int64_t up256(int64_t b) { return (b + 255) / 256 * 256; }
static BucketScratch bucket_scratch(int64_t n_self, int64_t n_idx) {
  BucketScratch s;
  s.cnt_bytes = 256 + up256(4 * n_self);  // [0] slots handed out, [1] long segments; the counters behind them
  s.cursor_bytes = up256(4 * n_self);
  s.seg_bytes = up256(8 * n_idx);
  s.heavy_bytes = up256(4 * (n_idx / (kLightMax + 1) + 1));
  s.total = s.cnt_bytes + s.cursor_bytes + s.seg_bytes + s.heavy_bytes;
  return s;
}
static int items_grid(int64_t n, int per) {
  const int64_t g = (n + per - 1) / per, cap = 32LL * kNumSMs;
  return static_cast<int>(g < 1 ? 1 : (g > cap ? cap : g));
}

template <typename T>
static int launch_bucket(const void* self, const void* index, const void* src, void* out, const BucketArgs& A, void* scratch, uint32_t* status, cudaStream_t st) {
  const BucketScratch S = bucket_scratch(A.n_self, A.n_idx);
  char* base = static_cast<char*>(scratch);
  int* head = reinterpret_cast<int*>(base);
  int* cnt = reinterpret_cast<int*>(base + 256);
  int* cursor = reinterpret_cast<int*>(base + S.cnt_bytes);
  int2* seg = reinterpret_cast<int2*>(base + S.cnt_bytes + S.cursor_bytes);  // (source position, value bits) per contribution
  int* heavy = reinterpret_cast<int*>(base + S.cnt_bytes + S.cursor_bytes + S.seg_bytes);
  const cudaError_t e = cudaMemsetAsync(head, 0, static_cast<size_t>(S.cnt_bytes), st);
  if (e != cudaSuccess) { set_last_cuda_error(e); return B200_ELAUNCH; }
  const int64_t* pi = static_cast<const int64_t*>(index);
  bucket_count<<<items_grid(A.n_idx, 256), 256, 0, st>>>(pi, cnt, A, status);
  assign_segments<16><<<grid_for(A.n_self, 4096), 256, 0, st>>>(cnt, cursor, A.n_self, head, kLightMax, head + 1, heavy);
  bucket_fill<T><<<items_grid(A.n_idx, 256), 256, 0, st>>>(pi, static_cast<const T*>(src), cursor, seg, A, status);
  bucket_replay<T><<<items_grid(A.n_self, 256), 256, 0, st>>>(static_cast<const T*>(self), static_cast<T*>(out), cnt, 0, cursor, seg, A.n_self, nullptr);
  bucket_replay_heavy<T><<<2 * kNumSMs, 256, 0, st>>>(static_cast<const T*>(self), static_cast<T*>(out), HeavyCounters{cnt, cursor, 0, nullptr, nullptr, nullptr}, seg, A.dim_len, head + 1, heavy);
  return check_launch(5);
}

// ------------------------------------------------------------------ chain path
// The same geometries with a scatter dimension no longer than self's (features of graph nodes, a
// random half of the rows): most destinations get none or one, so grouping costs more than
// the sums. One pass hangs every contribution into its destination's chain (`head[d]`, then
// `link[p]`; any order), one pass over the destinations walks the chains and adds in ascending
// position -- for one destination the linear position p orders like the position along the
// dim. Four destinations per thread advance together, three links deep with the entries in
// registers; deeper chains collect their positions in an array. What bounds it: the random
// 4-byte exchanges, and one random 8-byte look per contribution (the value lies beside the
// link: a second look, into `src`, made the second pass 91 us instead of 61). f16
// 150134 x 63, half as many rows picked: 251 us in segments -> 133 us.
// A chain of more than kLightMax entries is not walked to its end (a dependent chain of loads):
// its destination goes on a list, and the kernels that follow group just those contributions the
// way the bucket path does. Where the indices crowd on few destinations that is two passes more
// than grouping everything at once (fp32 7000 x 333, 3500 rows into one: 224 us against 156;
// Zipf-distributed 257 against 169), so a sample of the contributions is looked at first (`chain_begin`) and
// where it is crowded the chains are left out and the same kernels group all of them.
constexpr int kChainUnroll = 4;
enum { kCtlSlots = 0, kCtlListed = 1, kCtlGrouped = 2 };  // words of the control block: slots handed out, long chains or segments, 1 = everything is grouped

// Empties the chains, while the first CTA looks at up to 1024 contributions, one to a thread, spread over all of them. How
// many pairs of them share a destination estimates how crowded the destinations are: evenly
// spread indices give about s^2 / (2 destinations); four times that, and enough pairs for the estimate
// to mean something, is crowded. Which way is taken changes no result.
constexpr int kSample = 1024, kSampleSlotBits = 11;
static_assert((1 << kSampleSlotBits) == 2 * kSample, "the table of samples");
// Pairs among the samples `key` (one per thread and trip; negative: none) that agree. `table`: 4 * kSample words of shared memory.
template <int THREADS>
__device__ __forceinline__ int equal_pairs(const int (&key)[kSample / THREADS], int* table) {
  __shared__ int pairs;
  int* cnt = table + 2 * kSample;
  for (int i = threadIdx.x; i < 2 * kSample; i += THREADS) { table[i] = -1; cnt[i] = 0; }
  if (threadIdx.x == 0) pairs = 0;
  __syncthreads();
  int mine = 0;
#pragma unroll
  for (int t = 0; t < kSample / THREADS; ++t) {
    if (key[t] < 0) continue;
    uint32_t slot = static_cast<uint32_t>(key[t]) * 2654435761u >> (32 - kSampleSlotBits);
    for (;;) {  // a free slot is found: there are twice as many as samples
      const int was = atomicCAS(&table[slot], -1, key[t]);
      if (was == -1 || was == key[t]) break;
      slot = (slot + 1) & (2 * kSample - 1);
    }
    mine += atomicAdd(&cnt[slot], 1);
  }
  if (mine) atomicAdd(&pairs, mine);
  __syncthreads();
  const int all = pairs;
  __syncthreads();
  return all;
}
// `times` as many pairs as an even index has on average
__device__ __forceinline__ bool crowded(int pairs, int s, double places, double times = 4.0) { return pairs > 16.0 + times * (static_cast<double>(s) * s / (2.0 * places)); }
// This thread's samples: their destinations, -1 where there is none.
template <int THREADS>
__device__ __forceinline__ int sample_destinations(const int64_t* __restrict__ index, const BucketArgs& A, int (&dest)[kSample / THREADS]) {
  const int s = A.n_idx < kSample ? static_cast<int>(A.n_idx) : kSample;
  const uint32_t every = static_cast<uint32_t>(A.n_idx / s);  // n_idx is below 2^31
#pragma unroll
  for (int t = 0; t < kSample / THREADS; ++t) {
    const uint32_t i = threadIdx.x + t * THREADS;
    dest[t] = -1;
    if (static_cast<int>(i) >= s) continue;
    // not an even spacing: it could keep to a few columns
    const int64_t p = static_cast<int64_t>(i) * every + (i * 2654435761u >> 4) % every;
    int64_t d, so;
    int pos;
    if (bucket_decode(A, p, index, d, so, pos, nullptr)) dest[t] = static_cast<int>(d);
  }
  return s;
}
__global__ void __launch_bounds__(kSample) chain_begin(const int64_t* __restrict__ index, int* __restrict__ head, int64_t n_self, int* __restrict__ ctl, int* __restrict__ listed_cnt, int64_t listed,
                                                   const __grid_constant__ BucketArgs A) {
  if (blockIdx.x != 0) {
    const int64_t first = static_cast<int64_t>(blockIdx.x - 1) * kSample + threadIdx.x, step = static_cast<int64_t>(gridDim.x - 1) * kSample;
    for (int64_t i = first; i < listed; i += step) listed_cnt[i] = 0;
    const int64_t words = (reinterpret_cast<uintptr_t>(head) & 15u) == 0 ? n_self / 4 : 0;
    for (int64_t i = first; i < words; i += step) reinterpret_cast<int4*>(head)[i] = make_int4(-1, -1, -1, -1);
    for (int64_t i = 4 * words + first; i < n_self; i += step) head[i] = -1;
    return;
  }
  __shared__ int table[4 * kSample];
  int dest[1] = {-1};
  const int s = listed == 0 ? 0 : sample_destinations<kSample>(index, A, dest);
  const int pairs = equal_pairs<kSample>(dest, table);
  if (threadIdx.x == 0) {
    ctl[kCtlSlots] = 0;
    ctl[kCtlListed] = 0;
    ctl[kCtlGrouped] = crowded(pairs, s, static_cast<double>(A.n_idx / A.dim_len) * static_cast<double>(A.self_dim_size)) ? 1 : 0;
  }
}

// link[p] = {the entry hung before p, or -1; the value's bits as fp32}
template <typename T>
__global__ void __launch_bounds__(256) chain_link(const int64_t* __restrict__ index, const T* __restrict__ src, int* __restrict__ head, int2* __restrict__ link, const int* __restrict__ ctl,
                                                  const __grid_constant__ BucketArgs A, uint32_t* status) {
  if (ctl[kCtlGrouped]) return;
  for (int64_t p0 = static_cast<int64_t>(blockIdx.x) * (256 * kChainUnroll) + threadIdx.x; p0 < A.n_idx; p0 += static_cast<int64_t>(gridDim.x) * (256 * kChainUnroll)) {
    int64_t dest[kChainUnroll];
    T v[kChainUnroll];
    int before[kChainUnroll];
#pragma unroll
    for (int u = 0; u < kChainUnroll; ++u) {
      const int64_t p = p0 + u * 256;
      int64_t so;
      int pos;
      if (p >= A.n_idx || !bucket_decode(A, p, index, dest[u], so, pos, status)) dest[u] = -1;
      else v[u] = src[so];
    }
#pragma unroll
    for (int u = 0; u < kChainUnroll; ++u)
      if (dest[u] >= 0) before[u] = atomicExch(&head[dest[u]], static_cast<int>(p0 + u * 256));
#pragma unroll
    for (int u = 0; u < kChainUnroll; ++u)
      if (dest[u] >= 0) link[p0 + u * 256] = make_int2(before[u], __float_as_int(to_f32(v[u])));
  }
}

// A chain of four entries or more. False: too long to walk.
__device__ __noinline__ bool chain_deep(const int2* __restrict__ link, int p, float& acc) {
  int pos[kLightMax];
  float val[kLightMax];
  int c = 0;
  while (p >= 0) {
    if (c == kLightMax) return false;
    const int2 e = link[p];
    int k = c++;
    for (; k > 0 && pos[k - 1] > p; --k) {
      pos[k] = pos[k - 1];
      val[k] = val[k - 1];
    }
    pos[k] = p;
    val[k] = __int_as_float(e.y);
    p = e.x;
  }
  for (int k = 0; k < c; ++k) acc += val[k];
  return true;
}

template <typename T>
__global__ void __launch_bounds__(256) chain_replay(const T* __restrict__ self, T* __restrict__ out, int* __restrict__ head, const int2* __restrict__ link, int64_t n_self,
                                                    int* __restrict__ ctl, int* __restrict__ heavy_list) {
  constexpr int U = kChainUnroll;
  if (ctl[kCtlGrouped]) return;
  for (int64_t d0 = static_cast<int64_t>(blockIdx.x) * (256 * U) + threadIdx.x; d0 < n_self; d0 += static_cast<int64_t>(gridDim.x) * (256 * U)) {
    int k[4][U];  // the first three entries of each chain and what follows them, -1 past its end
    T s[U];
    float v[3][U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int64_t d = d0 + u * 256;
      k[0][u] = d < n_self ? head[d] : -1;
      if (d < n_self) s[u] = self[d];
    }
#pragma unroll
    for (int l = 0; l < 3; ++l) {
#pragma unroll
      for (int u = 0; u < U; ++u) {
        int2 e = make_int2(-1, 0);
        if (k[l][u] >= 0) e = link[k[l][u]];
        k[l + 1][u] = e.x;
        v[l][u] = __int_as_float(e.y);
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int64_t d = d0 + u * 256;
      if (d >= n_self) break;
      if (k[0][u] < 0) {
        out[d] = s[u];
        continue;
      }
      float acc = to_f32(s[u]);
      if (k[3][u] < 0) {
        int a = k[0][u], b = k[1][u] < 0 ? 0x7fffffff : k[1][u], c = k[2][u] < 0 ? 0x7fffffff : k[2][u];
        float va = v[0][u], vb = v[1][u], vc = v[2][u];
        if (b < a) { int t = a; a = b; b = t; float x = va; va = vb; vb = x; }
        if (c < b) { int t = b; b = c; c = t; float x = vb; vb = vc; vc = x; }
        if (b < a) { int t = a; a = b; b = t; float x = va; va = vb; vb = x; }
        acc += va;
        if (b != 0x7fffffff) acc += vb;
        if (c != 0x7fffffff) acc += vc;
      } else if (!chain_deep(link, k[0][u], acc)) {
        const int h = atomicAdd(&ctl[kCtlListed], 1);
        heavy_list[h] = static_cast<int>(d);
        head[d] = -2 - h;
        continue;
      }
      out[d] = from_f32<T>(acc);
    }
  }
}

// The contributions of listed destinations, or all of them: counted (into the list's counters, or into
// the heads, which stand at -1), given segments, filled in.
__global__ void __launch_bounds__(256) chain_count(const int64_t* __restrict__ index, int* head, int* listed_cnt, const __grid_constant__ BucketArgs A,
                                                   const int* ctl) {
  after_grids_before();
  const bool grouped = ctl[kCtlGrouped] != 0;
  if (!grouped && ctl[kCtlListed] == 0) return;
  for (int64_t p = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; p < A.n_idx; p += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    int64_t dest, so;
    int pos;
    if (!bucket_decode(A, p, index, dest, so, pos, nullptr)) continue;
    if (grouped) {
      atomicAdd(&head[dest], 1);
    } else {
      const int h = head[dest];
      if (h <= -2) atomicAdd(&listed_cnt[-2 - h], 1);
    }
  }
}
__global__ void __launch_bounds__(256) chain_assign(const int* head, int* cursor, int64_t n_self, const int* listed_cnt, int* listed_cursor,
                                                    int64_t listed, int* ctl, int* heavy_list) {
  constexpr int ITEMS = 16;
  after_grids_before();
  const bool grouped = ctl[kCtlGrouped] != 0;
  if (!grouped && (ctl[kCtlListed] == 0 || static_cast<int64_t>(blockIdx.x) * 256 * ITEMS >= listed)) return;
  if (grouped) assign_segments_of<ITEMS>(head, -1, cursor, n_self, ctl + kCtlSlots, kLightMax, ctl + kCtlListed, heavy_list);
  else assign_segments_of<ITEMS>(listed_cnt, 0, listed_cursor, listed, ctl + kCtlSlots, 0x7fffffff, nullptr, nullptr);
}
template <typename T>
__global__ void __launch_bounds__(256) chain_fill(const int64_t* __restrict__ index, const T* __restrict__ src, const int* head, int* cursor, int* listed_cursor,
                                                  int2* seg, const __grid_constant__ BucketArgs A, const int* ctl, uint32_t* status) {
  after_grids_before();
  const bool grouped = ctl[kCtlGrouped] != 0;
  if (!grouped && ctl[kCtlListed] == 0) return;
  for (int64_t p = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; p < A.n_idx; p += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    int64_t dest, so;
    int pos;
    if (!bucket_decode(A, p, index, dest, so, pos, grouped ? status : nullptr)) continue;  // (chains: chain_link has set it)
    int* at = &cursor[dest];
    if (!grouped) {
      const int h = head[dest];
      if (h > -2) continue;
      at = &listed_cursor[-2 - h];
    }
    seg[atomicAdd(at, 1)] = make_int2(pos, __float_as_int(to_f32(src[so])));
  }
}

// As a rule these five have nothing to do. listed_cnt: NULL where there are no chains
template <typename T>
static int launch_group(const int64_t* index, const T* src, const T* self, T* out, const BucketArgs& A, int* head, int* cursor, int* ctl, int* listed_cnt, int* listed_cursor, int* list, int2* seg,
                        int64_t listed, uint32_t* status, cudaStream_t st) {
  auto capped = [](int64_t n, int per, int64_t cap) { const int64_t g = (n + per - 1) / per; return g < 1 ? 1 : (g > cap ? cap : g); };
  const int64_t walk = capped(A.n_idx, 256, 16 * kNumSMs);
  cudaError_t e = launch_after(chain_count, walk, 256, 0, st, index, head, listed_cnt, A, ctl);
  if (e == cudaSuccess) e = launch_after(chain_assign, grid_for(A.n_self, 4096), 256, 0, st, head, cursor, A.n_self, listed_cnt, listed_cursor, listed, ctl, list);
  if (e == cudaSuccess) e = launch_after(chain_fill<T>, walk, 256, 0, st, index, src, head, cursor, listed_cursor, seg, A, ctl, status);
  if (e == cudaSuccess) e = launch_after(bucket_replay<T>, capped(A.n_self, 256, 16 * kNumSMs), 256, 0, st, self, out, head, -1, cursor, seg, A.n_self, ctl + kCtlGrouped);
  if (e == cudaSuccess)
    e = launch_after(bucket_replay_heavy<T>, 2 * kNumSMs, 256, 0, st, self, out, HeavyCounters{head, cursor, -1, listed_cnt, listed_cursor, ctl + kCtlGrouped}, seg, A.dim_len, ctl + kCtlListed, list);
  if (e != cudaSuccess) { set_last_cuda_error(e); return B200_ELAUNCH; }
  return check_launch(5);
}

struct ChainScratch {
  int64_t head_bytes, link_bytes, list_bytes, seg_bytes, total;
};
static ChainScratch chain_scratch(int64_t n_self, int64_t n_idx) {
  ChainScratch s;
  s.head_bytes = up256(4 * n_self);
  s.link_bytes = up256(8 * n_idx);
  s.list_bytes = up256(4 * (n_idx / (kLightMax + 1) + 1));
  s.seg_bytes = up256(8 * n_idx);
  s.total = 2 * s.head_bytes + 256 + 3 * s.list_bytes + s.link_bytes + s.seg_bytes;
  return s;
}

template <typename T>
static int launch_chain(const void* self, const void* index, const void* src, void* out, const BucketArgs& A, void* scratch, uint32_t* status, cudaStream_t st) {
  const ChainScratch S = chain_scratch(A.n_self, A.n_idx);
  char* at = static_cast<char*>(scratch);
  auto take = [&](int64_t bytes) { char* p = at; at += bytes; return p; };
  int* head = reinterpret_cast<int*>(take(S.head_bytes));
  int* cursor = reinterpret_cast<int*>(take(S.head_bytes));
  int* ctl = reinterpret_cast<int*>(take(256));
  int* listed_cnt = reinterpret_cast<int*>(take(S.list_bytes));
  int* listed_cursor = reinterpret_cast<int*>(take(S.list_bytes));
  int* list = reinterpret_cast<int*>(take(S.list_bytes));
  int2* link = reinterpret_cast<int2*>(take(S.link_bytes));
  int2* seg = reinterpret_cast<int2*>(take(S.seg_bytes));
  const int64_t* pi = static_cast<const int64_t*>(index);
  const T* ps = static_cast<const T*>(src);
  const T* px = static_cast<const T*>(self);
  T* po = static_cast<T*>(out);
  const int64_t listed = A.n_idx / (kLightMax + 1);  // no more long chains (or segments) than this
  auto capped = [](int64_t n, int per, int64_t cap) { const int64_t g = (n + per - 1) / per; return static_cast<int>(g < 1 ? 1 : (g > cap ? cap : g)); };
  chain_begin<<<1 + capped(A.n_self, 8 * kSample, 2 * kNumSMs), kSample, 0, st>>>(pi, head, A.n_self, ctl, listed_cnt, listed, A);
  chain_link<T><<<items_grid(A.n_idx, 256 * kChainUnroll), 256, 0, st>>>(pi, ps, head, link, ctl, A, status);
  chain_replay<T><<<grid_for(A.n_self, 256 * kChainUnroll), 256, 0, st>>>(px, po, head, link, A.n_self, ctl, list);
  if (int rc = check_launch(3)) return rc;
  if (listed == 0) return B200_OK;
  return launch_group<T>(pi, ps, px, po, A, head, cursor, ctl, listed_cnt, listed_cursor, list, seg, listed, status, st);
}

// ------------------------------------------------------------------ binned path
// Matrices too tall for a strip of their columns to fit in shared memory, or off the strips'
// 16-byte grid. self is viewed as [outer, rows, cols]; its columns are dealt into groups of at most 32, and the
// rows of a group into bins of 2^shift rows whose sums fit in a warp's share of shared memory (kBinDests). Two launches:
//   binned_sort: a CTA takes a chunk of the index -- rows of one column group -- and writes its
//     contributions out grouped by bin, with a table of where each bin begins. The order is
//     stable for every destination: a thread owns ONE column of a run of rows and takes its places
//     in order from counters of its own run, and the runs follow one another; so nothing is sorted by
//     position and a record is the destination and the value alone.
//   binned_replay: a warp owns a bin. It walks the bin's records chunk after chunk, 32 to a step, and adds them to the
//     sums in shared memory; two records of a step with one destination are found with a tag
//     table, as in the strip kernels, and added in lane order, which is source order.
// Every global access is in runs of a row or of a segment; what is random stays in shared memory, where the chain path
// has its exchanges and look-ups in L2. fp16 150134 x 63, 75067 rows: 133 us in chains, 87 so (binned_sort 29, half of its
// issue slots busy counting and placing; binned_replay 45: nine warps of 4096 sums fill an SM's shared memory, and each goes
// at the speed of its chain of tag, look, sum; six more launches that begin and find nothing to do; 82 with the 4096 sums of a warp read 32 to
// a lane behind the first table, 16 before). fp32 4095 x 4095 556 -> 283,
// 160000 x 400 3640 -> 1140, 888 x 4065 99 -> 58. Tried: a CTA to a bin, its records in chains in shared memory (123 us
// for the replay, 18 instructions' worth of divergence to a destination); the records of 8 steps in registers
// (80: a step unrolled eight times does not fit the instruction cache); 256 threads with runs of 32 rows in binned_sort (44).
constexpr int kBinThreads = 512;
constexpr int kBinItems = 16;  // rows of its column per thread of binned_sort, at most
constexpr int kBinDests = 4096;
constexpr int kBinAhead = 8;  // steps whose records are on the way while those before are added
constexpr int kBinCountBytes = 40 * 1024;  // counters of binned_sort: two CTAs of it per SM

struct BinnedArgs {
  int64_t outer, rows, cols;  // self / out, contiguous
  int64_t idx_outer, idx_rows, idx_cols;
  int64_t idx_so, idx_sr, idx_sc, src_so, src_sr, src_sc;  // element strides of index / src
  int c, groups, idx_groups;   // columns of a group; groups of self's columns, of the index's
  int shift, bins;             // log2 of a bin's rows; bins of a group
  int items, runs, chunk_rows, chunks;  // rows of a run (one thread's), runs of a chunk, rows of a chunk, chunks of a group
  uint32_t c_magic;            // x / c == __umulhi(x, c_magic) for x < 2^16
};

template <typename T> struct BinRec { typedef uint32_t type; };
template <> struct BinRec<float> { typedef uint2 type; };
__device__ __forceinline__ uint32_t bin_rec(int dest, uint16_t bits) { return static_cast<uint32_t>(dest) | static_cast<uint32_t>(bits) << 16; }
__device__ __forceinline__ void bin_make(uint32_t& r, int dest, __nv_bfloat16 v) { r = bin_rec(dest, __bfloat16_as_ushort(v)); }
__device__ __forceinline__ void bin_make(uint32_t& r, int dest, __half v) { r = bin_rec(dest, __half_as_ushort(v)); }
__device__ __forceinline__ void bin_make(uint2& r, int dest, float v) { r = make_uint2(static_cast<uint32_t>(dest), __float_as_uint(v)); }
__device__ __forceinline__ int bin_dest(uint32_t r) { return static_cast<int>(r & 0xffffu); }
__device__ __forceinline__ int bin_dest(uint2 r) { return static_cast<int>(r.x); }
template <typename T> __device__ __forceinline__ float bin_value(typename BinRec<T>::type r);
template <> __device__ __forceinline__ float bin_value<float>(uint2 r) { return __uint_as_float(r.y); }
template <> __device__ __forceinline__ float bin_value<__nv_bfloat16>(uint32_t r) { return __uint_as_float(r & 0xffff0000u); }
template <> __device__ __forceinline__ float bin_value<__half>(uint32_t r) { return __half2float(__ushort_as_half(static_cast<unsigned short>(r >> 16))); }

// Exclusive prefix sums over the CTA's threads; `total` is the sum of all. `sums`: 16 words.
__device__ __forceinline__ int bin_scan(int v, int* sums, int& total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int inc = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += y;
  }
  __syncthreads();  // the sums of a call before
  if (lane == 31) sums[warp] = inc;
  __syncthreads();
  int w = lane < kBinThreads / 32 ? sums[lane] : 0;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, w, o);
    if (lane >= o) w += y;
  }
  total = __shfl_sync(0xffffffffu, w, 31);
  const int before = __shfl_sync(0xffffffffu, w, (warp + 31) & 31);
  return inc - v + (warp ? before : 0);
}

// Looks at a sample: where the destinations, or the bins, are crowded, one warp would walk most of the
// records, and everything is grouped by destination instead, as on the chain path.
__global__ void __launch_bounds__(kSample) binned_begin(const int64_t* __restrict__ index, const __grid_constant__ BinnedArgs A, const __grid_constant__ BucketArgs B, int* __restrict__ ctl, double times) {
  __shared__ int table[4 * kSample];
  next_grid_may_start();
  int dest[1];
  const int s = sample_destinations<kSample>(index, B, dest);
  const int same = equal_pairs<kSample>(dest, table);
  if (dest[0] >= 0) {
    const uint32_t d = static_cast<uint32_t>(dest[0]), cols = static_cast<uint32_t>(A.cols), rows = static_cast<uint32_t>(A.rows), row = d / cols, o = row / rows;
    dest[0] = static_cast<int>((o * A.groups + (d - row * cols) / A.c) * A.bins + ((row - o * rows) >> A.shift));
  }
  const int near = equal_pairs<kSample>(dest, table);
  if (threadIdx.x == 0) {
    ctl[kCtlSlots] = 0;
    ctl[kCtlListed] = 0;
    ctl[kCtlGrouped] = crowded(same, s, static_cast<double>(A.idx_outer) * A.idx_cols * A.rows, times) || crowded(near, s, static_cast<double>(A.idx_outer) * A.idx_groups * A.bins, times) ? 1 : 0;
  }
}

// rec: [outer][group][chunk][chunk_rows * c]; first: [outer][group][chunk][bins + 1], where each bin begins in its chunk
template <typename T>
__global__ void __launch_bounds__(kBinThreads, 2) binned_sort(const int64_t* __restrict__ index, const T* __restrict__ src, typename BinRec<T>::type* __restrict__ rec, uint16_t* __restrict__ first,
                                                              const __grid_constant__ BinnedArgs A, const int* ctl, uint32_t* status) {
  typedef typename BinRec<T>::type Rec;
  extern __shared__ __align__(16) unsigned char bin_smem[];
  __shared__ int sums[kBinThreads / 32];
  const int tid = threadIdx.x;
  const int words = (A.bins + 1) / 2;  // two 16-bit counters to a word
  Rec* stage = reinterpret_cast<Rec*>(bin_smem);
  uint32_t* count = reinterpret_cast<uint32_t*>(stage + A.chunk_rows * A.c);  // [runs][words]
  const int chunk = static_cast<int>(blockIdx.x % static_cast<uint32_t>(A.chunks));
  const int64_t og = blockIdx.x / static_cast<uint32_t>(A.chunks);
  const int64_t o = og / A.idx_groups;
  const int run = static_cast<int>(__umulhi(tid, A.c_magic)), col = tid - run * A.c;
  const int64_t j = (og - o * A.idx_groups) * A.c + col;
  const int64_t row0 = static_cast<int64_t>(chunk) * A.chunk_rows + run * A.items;
  const int64_t left = A.idx_rows - row0;
  const int mine = run < A.runs && j < A.idx_cols && left > 0 ? (left < A.items ? static_cast<int>(left) : A.items) : 0;
  for (int i = tid; i < A.runs * words; i += kBinThreads) count[i] = 0;
  __syncthreads();
  const int64_t* pi = index + o * A.idx_so + row0 * A.idx_sr + j * A.idx_sc;
  const T* ps = src + o * A.src_so + row0 * A.src_sr + j * A.src_sc;
  uint32_t* counters = count + run * words;
  constexpr uint32_t kNone = 0xffffffffu;
  constexpr int kFlight = 16;  // index elements on the way
  uint32_t key[kBinItems];
  T v[kBinItems];
  bool bad = false;
#pragma unroll
  for (int h = 0; h < kBinItems; h += kFlight) {
    int64_t raw[kFlight];
#pragma unroll
    for (int u = 0; u < kFlight; ++u) {
      raw[u] = -1;
      if (h + u < mine) {
        raw[u] = __ldcs(pi);
        v[h + u] = __ldcs(ps);
      }
      pi += A.idx_sr;
      ps += A.src_sr;
    }
#pragma unroll
    for (int u = 0; u < kFlight; ++u) {
      key[h + u] = kNone;
      if (static_cast<uint64_t>(raw[u]) < static_cast<uint64_t>(A.rows)) {
        key[h + u] = static_cast<uint32_t>(raw[u]);
        const uint32_t bin = key[h + u] >> A.shift;
        atomicAdd(&counters[bin >> 1], 1u << (16 * (bin & 1)));
      } else if (h + u < mine) {
        bad = true;
      }
    }
  }
  if (bad) flag_oob(status);
  next_grid_may_start();
  after_grids_before();  // (the index has been there all along)
  if (ctl && ctl[kCtlGrouped]) return;
  __syncthreads();
  // counters -> the first place of the run's records of that bin
  int total = 0;
  uint16_t* f = first + static_cast<int64_t>(blockIdx.x) * (A.bins + 1);
  for (int w0 = 0; w0 < words; w0 += kBinThreads) {
    const int w = w0 + tid;
    uint32_t sum = 0;
    if (w < words)
      for (int r = 0; r < A.runs; ++r) sum += count[r * words + w];
    const int low = static_cast<int>(sum & 0xffffu), both = low + static_cast<int>(sum >> 16);
    int all;
    const int at = total + bin_scan(both, sums, all);
    total += all;
    if (w < words) {
      uint32_t next = static_cast<uint32_t>(at) | static_cast<uint32_t>(at + low) << 16;
      f[2 * w] = static_cast<uint16_t>(at);
      if (2 * w + 1 <= A.bins) f[2 * w + 1] = static_cast<uint16_t>(at + low);
      if (2 * w + 2 == A.bins) f[A.bins] = static_cast<uint16_t>(at + both);
      for (int r = 0; r < A.runs; ++r) {
        const uint32_t n = count[r * words + w];
        count[r * words + w] = next;
        next += n;
      }
    }
  }
  __syncthreads();
#pragma unroll
  for (int u = 0; u < kBinItems; ++u)
    if (key[u] != kNone) {
      const uint32_t bin = key[u] >> A.shift, half = 16 * (bin & 1);
      const uint32_t at = (atomicAdd(&counters[bin >> 1], 1u << half) >> half) & 0xffffu;
      bin_make(stage[at], 4 * (static_cast<int>(key[u] & ((1u << A.shift) - 1u)) * A.c + col), v[u]);
    }
  __syncthreads();
  Rec* to = rec + static_cast<int64_t>(blockIdx.x) * (A.chunk_rows * A.c);
  for (int i = tid; i < total; i += kBinThreads) to[i] = stage[i];
}

template <typename T>
__global__ void __launch_bounds__(32) binned_replay(const T* __restrict__ self, T* __restrict__ out, const typename BinRec<T>::type* rec, const uint16_t* first,
                                                    const __grid_constant__ BinnedArgs A, const int* ctl, int* head, int64_t n_self) {
  typedef typename BinRec<T>::type Rec;
  constexpr uint32_t kAll = 0xffffffffu;
  constexpr int kMove = 32;   // elements of self on the way per lane
  extern __shared__ __align__(16) unsigned char bin_smem[];
  __shared__ uint32_t piece[32];
  __shared__ __align__(16) Rec ring[2][kBinAhead][32];
  const int dests = A.c << A.shift, lane = threadIdx.x;
  float* sum = reinterpret_cast<float*>(bin_smem);  // [dests + 32]: one to spare for each lane; behind them a byte of tag for each
  const uint32_t sum_a = static_cast<uint32_t>(__cvta_generic_to_shared(bin_smem)), tag_a = sum_a + 4 * (dests + 32);
  const int bin = static_cast<int>(blockIdx.x % static_cast<uint32_t>(A.bins));
  const int64_t og = blockIdx.x / static_cast<uint32_t>(A.bins);
  const int64_t o = og / A.groups, g = og - o * A.groups;
  const int64_t row0 = static_cast<int64_t>(bin) << A.shift;
  const int rows = static_cast<int>(A.rows - row0 < (1 << A.shift) ? A.rows - row0 : (1 << A.shift));
  const int width = static_cast<int>(A.cols - g * A.c < A.c ? A.cols - g * A.c : A.c);
  const int64_t base = (o * A.rows + row0) * A.cols + g * A.c;
  // a group is 32 columns of a row, or whole rows (c == cols < 32): in memory, too, a lane's elements lie a constant step apart
  const int used = rows * A.c;
  const int64_t step = A.c == 32 ? A.cols : 32;
  const int end = A.c < 32 || lane < width ? used : 0;
  after_grids_before();
  if (ctl && ctl[kCtlGrouped]) {  // the counters of the kernels that follow
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * 32 + lane; i < n_self; i += static_cast<int64_t>(gridDim.x) * 32) head[i] = -1;
    return;
  }
  const int chunks = g < A.idx_groups && o < A.idx_outer ? A.chunks : 0;
  const int per_chunk = A.chunk_rows * A.c;
  const int64_t chunk0 = (o * A.idx_groups + g) * A.chunks;
  const uint16_t* f = first + (chunk0 + lane) * (A.bins + 1) + bin;
  const int64_t f_step = 32LL * (A.bins + 1);
  const Rec* from = rec + chunk0 * per_chunk;
  // 32 chunks are a batch: a lane knows where its chunk's piece of this bin lies and which numbers its records have
  int b = 0, e = 0, c_next = 0;            // the next batch's table and first chunk
  int start = 0, total = 0, before = 0;    // number of the first record of the lane's piece; records of the batch; pieces that start before `pos`
  int pos = 0;                             // records of the batch asked for
  auto read_table = [&]() {
    b = e = 0;
    if (c_next + lane < chunks) { b = f[0]; e = f[1]; }
    f += f_step;
  };
  auto open = [&]() {
    int upto = e - b;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int y = __shfl_up_sync(kAll, upto, d);
      if (lane >= d) upto += y;
    }
    total = __shfl_sync(kAll, upto, 31);
    pos = before = 0;
    start = upto - (e - b);
    const uint32_t filled = __ballot_sync(kAll, e > b);
    // where record number 0 would lie, were it this piece's; the pieces that have records stand side by side
    if (e > b) piece[__popc(filled & ((1u << lane) - 1u))] = static_cast<uint32_t>(c_next + lane) * static_cast<uint32_t>(per_chunk) + static_cast<uint32_t>(b - start);
    else start = 0x40000000;
    __syncwarp();
    c_next += 32;
    read_table();
  };
  // asks for the next records, up to 32 * kBinAhead of a batch; how many there are
  auto load = [&](int buf) {
    while (pos >= total && c_next < chunks) open();
    const int n = total - pos < 32 * kBinAhead ? total - pos : 32 * kBinAhead;
#pragma unroll 1
    for (int u = 0; 32 * u < n; ++u, pos += 32) {
      const uint32_t t = static_cast<uint32_t>(start - pos);
      const uint32_t starts = __reduce_or_sync(kAll, t < 32u ? 1u << t : 0u);
      const int q = before + __popc(starts & ((2u << lane) - 1u)) - 1;
      before += __popc(starts);
      if (32 * u + lane < n) __pipeline_memcpy_async(&ring[buf][u][lane], from + (piece[q] + static_cast<uint32_t>(pos + lane)), sizeof(Rec));
    }
    __pipeline_commit();
    __syncwarp();
    return n;
  };
  auto add = [&](uint32_t off, float v) {  // off: 4 * destination
    const uint32_t tag = tag_a + (off >> 2), at = sum_a + off;
    asm volatile("st.shared.u8 [%0], %1;" ::"r"(tag), "r"(lane) : "memory");
    __syncwarp();
    uint32_t winner;
    float old;
    asm volatile("ld.shared.u8 %0, [%1];" : "=r"(winner) : "r"(tag) : "memory");
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(old) : "r"(at) : "memory");
    const bool lost = winner != static_cast<uint32_t>(lane);
    const uint32_t losers = __ballot_sync(kAll, lost);
    if (losers == 0u) {
      asm volatile("st.shared.f32 [%0], %1;" ::"r"(at), "f"(old + v) : "memory");
      __syncwarp();
      return;
    }
    // the lanes of a clash are the losers and the lanes they name; all others add at once
    uint32_t involved = losers | __reduce_or_sync(kAll, lost ? 1u << winner : 0u);
    const int k = static_cast<int>(off >> 2);
    if (__popc(involved) <= 8) {
      if (!(involved >> lane & 1u)) sum[k] = old + v;
      __syncwarp();
      while (involved) {
        if (lane == __ffs(involved) - 1) sum[k] += v;
        involved &= involved - 1;
        __syncwarp();
      }
    } else {
      apply_in_rank_order(sum, k, v, rank_among_earlier(k, lane));
    }
  };
  if (chunks > 0) read_table();  // (on its way while self is read)
  {
    const T* p = self + base + lane;
    for (int d0 = lane; d0 < end; d0 += 32 * kMove) {
      T s[kMove];
#pragma unroll
      for (int u = 0; u < kMove; ++u) {
        if (d0 + 32 * u < end) s[u] = *p;
        p += step;
      }
#pragma unroll
      for (int u = 0; u < kMove; ++u)
        if (d0 + 32 * u < end) sum[d0 + 32 * u] = to_f32(s[u]);
    }
  }
  __syncwarp();
  int n = load(0);
#pragma unroll 1
  for (int buf = 0; n > 0; buf ^= 1) {
    const int then = load(buf ^ 1);
    __pipeline_wait_prior(1);
#pragma unroll 1
    for (int u = 0; 32 * u < n; ++u) {
      uint32_t off = 4u * (dests + lane);
      float v = 0.f;
      if (32 * u + lane < n) {  // (a lane reads what it has copied itself)
        const Rec r = ring[buf][u][lane];
        off = static_cast<uint32_t>(bin_dest(r));
        v = bin_value<T>(r);
      }
      add(off, v);
    }
    n = then;
  }
  __syncwarp();
  T* p = out + base + lane;
#pragma unroll 8
  for (int d = lane; d < end; d += 32, p += step) *p = from_f32<T>(sum[d]);
}

// Fills in the geometry behind `src_sc`; false: not for this path (more bins than there is room to count in).
static bool plan_binned(BinnedArgs& A) {
  if (A.cols < 2 || A.rows >= 0x7fffffffLL || A.idx_rows >= 0x7fffffffLL) return false;
  A.c = static_cast<int>(A.cols < 32 ? A.cols : 32);
  A.groups = static_cast<int>((A.cols + A.c - 1) / A.c);
  A.idx_groups = static_cast<int>((A.idx_cols + A.c - 1) / A.c);
  A.c_magic = 0xffffffffu / static_cast<uint32_t>(A.c) + 1u;
  A.runs = kBinThreads / A.c;
  // bins: as large as a warp's share of shared memory, smaller where that leaves fewer than eight per SM
  auto bins = [&](int sh) { return (A.rows + (1LL << sh) - 1) >> sh; };
  A.shift = 0;
  while ((A.c << (A.shift + 1)) <= kBinDests) ++A.shift;
  while (A.shift > 0 && A.outer * A.groups * bins(A.shift) < 8LL * kNumSMs) --A.shift;
  if (A.runs * ((bins(A.shift) + 1) / 2) * 4 > kBinCountBytes) return false;
  A.bins = static_cast<int>(bins(A.shift));
  // chunks: all a CTA can hold, less where that leaves fewer than two per SM
  const int64_t columns = A.idx_outer * A.idx_groups;
  A.items = static_cast<int>((A.idx_rows + A.runs - 1) / A.runs < kBinItems ? (A.idx_rows + A.runs - 1) / A.runs : kBinItems);
  while (A.items > 1 && columns * ((A.idx_rows + A.items * A.runs - 1) / (A.items * A.runs)) < 2 * kNumSMs) --A.items;
  A.chunk_rows = A.items * A.runs;
  A.chunks = static_cast<int>((A.idx_rows + A.chunk_rows - 1) / A.chunk_rows);
  return A.outer * A.groups * A.bins < 0x7fffffffLL && columns * A.chunks < 0x7ffffffeLL && static_cast<int64_t>(A.chunks) * A.chunk_rows * A.c < 0x7fffffffLL;
}
// With few source rows the worst that a crowded index can do is soon done: a warp that gets all records of its columns walks
// idx_rows * c of them, 32 to a step, of which 32 / c at most have one destination. So nothing is looked at first and
// nothing waits behind.
constexpr int kBinUnseen = 128;
struct BinnedScratch {
  int64_t first_bytes, rec_bytes, head_bytes, list_bytes, seg_bytes, total;
};
static BinnedScratch binned_scratch(const BinnedArgs& A, int es, int64_t n_self, int64_t n_idx) {
  BinnedScratch s;
  const int64_t chunks = A.idx_outer * A.idx_groups * A.chunks;
  s.first_bytes = up256(2 * chunks * (A.bins + 1LL));
  s.rec_bytes = up256(chunks * A.chunk_rows * A.c * (es == 4 ? 8 : 4));
  s.head_bytes = up256(4 * n_self);
  s.list_bytes = up256(4 * (n_idx / (kLightMax + 1) + 1));
  s.seg_bytes = up256(8 * n_idx);
  // the records, or what the groups of launch_group need in their place
  const int64_t grouped = 2 * s.head_bytes + s.list_bytes + s.seg_bytes;
  s.total = 256 + (s.first_bytes + s.rec_bytes > grouped ? s.first_bytes + s.rec_bytes : grouped);
  return s;
}

template <typename T>
static int launch_strip(const void* self, const void* index, const void* src, void* out, StripArgs A, uint32_t* status, cudaStream_t st, const int* only_if = nullptr);

// `strip`: NULL, or the geometry for the strip kernel, which takes a crowded index then: its time does not depend on where the
// index points. (f16 2672 x 332, all rows into five, 111.5 us grouped by destination, 72.1 in strips behind the look at the
// sample, 67.6 in strips alone; fp32 181 x 8164, 362 skewed rows of it, 195 in bins that are not crowded enough for groups, 102, 95; fp32 829 x 156, 23 of them, skewed 285, 118, 110; bins of an even index have one launch that finds
// nothing to do behind them and not five: the first shape 31.2 -> 24.4 us.)
template <typename T>
static int launch_binned(const void* self, const void* index, const void* src, void* out, const BinnedArgs& A, const BucketArgs& B, const StripArgs* strip, void* scratch, uint32_t* status,
                         cudaStream_t st) {
  typedef typename BinRec<T>::type Rec;
  const bool unseen = A.idx_rows <= kBinUnseen;
  const int64_t n_self = strip || unseen ? 0 : B.n_self;
  const BinnedScratch S = binned_scratch(A, static_cast<int>(sizeof(T)), n_self, strip || unseen ? 0 : B.n_idx);
  int* ctl = unseen ? nullptr : static_cast<int*>(scratch);
  char* base = static_cast<char*>(scratch) + 256;
  uint16_t* first = reinterpret_cast<uint16_t*>(base);
  Rec* rec = reinterpret_cast<Rec*>(base + S.first_bytes);
  const size_t sort_smem = sizeof(Rec) * A.chunk_rows * A.c + 4 * static_cast<size_t>(A.runs) * ((A.bins + 1) / 2);
  const size_t replay_smem = 5 * (static_cast<size_t>(A.c << A.shift) + 32);
  cudaError_t e = cudaFuncSetAttribute(binned_sort<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, 108 * 1024);
  const int64_t sorts = A.idx_outer * A.idx_groups * A.chunks, replays = A.outer * A.groups * A.bins;
  const int64_t* pi = static_cast<const int64_t*>(index);
  const T* ps = static_cast<const T*>(src);
  const T* px = static_cast<const T*>(self);
  T* po = static_cast<T*>(out);
  int* head = reinterpret_cast<int*>(base);
  int* cursor = reinterpret_cast<int*>(base + S.head_bytes);
  int* list = reinterpret_cast<int*>(base + 2 * S.head_bytes);
  int2* seg = reinterpret_cast<int2*>(base + 2 * S.head_bytes + S.list_bytes);
  if (unseen) {  // (the call's first kernel is launched the ordinary way)
    if (e == cudaSuccess) binned_sort<T><<<static_cast<unsigned>(sorts), kBinThreads, sort_smem, st>>>(pi, ps, rec, first, A, ctl, status);
  } else {
    binned_begin<<<1, kSample, 0, st>>>(pi, A, B, ctl, strip ? 1.5 : 4.0);  // (strips cost little more than even bins, groups several times as much)
    if (e == cudaSuccess) e = launch_after(binned_sort<T>, sorts, kBinThreads, sort_smem, st, pi, ps, rec, first, A, ctl, status);
  }
  if (e == cudaSuccess) e = launch_after(binned_replay<T>, replays, 32, replay_smem, st, px, po, rec, first, A, ctl, head, n_self);
  if (e != cudaSuccess) { set_last_cuda_error(e); return B200_ELAUNCH; }
  if (int rc = check_launch(unseen ? 2 : 3)) return rc;
  if (unseen) return B200_OK;
  if (strip) return launch_strip<T>(self, index, src, out, *strip, status, st, ctl + kCtlGrouped);
  return launch_group<T>(pi, ps, px, po, B, head, cursor, ctl, nullptr, nullptr, list, seg, 0, status, st);
}

// ------------------------------------------------------------------ embedding_dense_backward
// out[v, :] = sum over the positions i with indices[i] == v (and v != padding_idx) of
// grad[i, :], in ascending i, fp32 accumulation, one rounding. Five launches: count per table
// row; a segment for every row (`assign_segments`); fill the segments with source positions
// in any order; sort every segment; replay.
// What bounds it: writing the table. The replay therefore walks the table in the order of its
// addresses, a CTA on whole rows (a warp to a row kept some 9,500 rows open at once and stored
// at 3.9 TB/s), and the rows of more than kEmbLight contributions are summed meanwhile by CTAs
// of their own, a warp to 32 words of a row with 32 loads in flight (one CTA to a row, a load
// at a time, took four times as long as all the rest for text-like ids, whose most frequent
// one is 6 % of the tokens). bf16 128,256 x 4,096, 16,384 such ids: replay 266 + 1,076 us -> 214
// us (1.19 GB, 5.5 TB/s; a write-only stream reaches 5.9), the whole call 1,364 -> 235 us.
constexpr int kEmbLight = 32;
constexpr int kEmbWindowBits = 1 << 17;
constexpr int kEmbWindowWords = kEmbWindowBits / 32;

__device__ __forceinline__ int64_t emb_index(const void* idx, int64_t i, int i32) { return i32 ? static_cast<const int32_t*>(idx)[i] : static_cast<const int64_t*>(idx)[i]; }

__global__ void __launch_bounds__(256) emb_count(const void* __restrict__ idx, int i32, int64_t n, int64_t V, int64_t padding_idx, int* __restrict__ cnt, uint32_t* status) {
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t v = emb_index(idx, i, i32);
    if (v == padding_idx) continue;
    if (v < 0 || v >= V) { flag_oob(status); continue; }
    atomicAdd(&cnt[v], 1);
  }
}
__global__ void __launch_bounds__(256) emb_fill(const void* __restrict__ idx, int i32, int64_t n, int64_t V, int64_t padding_idx, int* cursor, int* __restrict__ seg_pos) {
  after_grids_before();
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t v = emb_index(idx, i, i32);
    if (v == padding_idx || v < 0 || v >= V) continue;
    seg_pos[atomicAdd(&cursor[v], 1)] = static_cast<int>(i);
  }
}

// `sorted` = the segments of `seg_pos` with their positions in ascending order (all positions of
// a segment are distinct). cursor[v] is the END of row v's segment by now. A CTA takes the
// long ones: a bitmap of a window of positions, prefix sums of its words' bit counts, and
// every position finds its own rank. A warp takes the others, ranked with shuffles.
__global__ void __launch_bounds__(256) emb_sort(const int* cnt, const int* cursor, const int* seg_pos, int* __restrict__ sorted, int64_t V, int64_t n,
                                                const int* heavy_count, const int* heavy_list) {
  __shared__ uint32_t bitmap[kEmbWindowWords];
  __shared__ int before[kEmbWindowWords];
  __shared__ int warp_sums[8];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  after_grids_before();
  const int nheavy = *heavy_count;
  for (int h = blockIdx.x; h < nheavy; h += gridDim.x) {
    const int64_t v = heavy_list[h];
    const int c = cnt[v], b = cursor[v] - c;
    int done = 0;  // positions ranked in the windows before
    for (int64_t w0 = 0; w0 < n && done < c; w0 += kEmbWindowBits) {
      const int words = static_cast<int>(((n - w0 < kEmbWindowBits ? n - w0 : kEmbWindowBits) + 31) / 32);
      const int per = (words + 255) / 256;
      __syncthreads();
      for (int i = threadIdx.x; i < words; i += 256) bitmap[i] = 0u;
      __syncthreads();
      for (int j = threadIdx.x; j < c; j += 256) {
        const int64_t rel = static_cast<int64_t>(seg_pos[b + j]) - w0;
        if (rel >= 0 && rel < kEmbWindowBits) atomicOr(&bitmap[rel >> 5], 1u << (rel & 31));
      }
      __syncthreads();
      int mine = 0;
      for (int k = 0; k < per; ++k) {
        const int i = threadIdx.x * per + k;
        if (i < words) mine += __popc(bitmap[i]);
      }
      int inc = mine;
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += y;
      }
      if (lane == 31) warp_sums[warp] = inc;
      __syncthreads();
      int prefix = done + inc - mine;
#pragma unroll
      for (int w = 0; w < 8; ++w) {
        if (w < warp) prefix += warp_sums[w];
        done += warp_sums[w];
      }
      for (int k = 0; k < per; ++k) {
        const int i = threadIdx.x * per + k;
        if (i < words) {
          before[i] = prefix;
          prefix += __popc(bitmap[i]);
        }
      }
      __syncthreads();
      for (int j = threadIdx.x; j < c; j += 256) {
        const int p = seg_pos[b + j];
        const int64_t rel = static_cast<int64_t>(p) - w0;
        if (rel >= 0 && rel < kEmbWindowBits) sorted[b + before[rel >> 5] + __popc(bitmap[rel >> 5] & ((1u << (rel & 31)) - 1u))] = p;
      }
    }
  }
  // a warp looks at 32 rows and ranks the short segments among them one after another; its rows
  // lie far apart, because the rows of frequent ids stand together (16,384 text-like ids in a
  // table of 128,256 rows: 23 us with 32 neighbouring rows to a warp, 6 us so)
  const int64_t groups = (V + 31) / 32;
  for (int64_t g = static_cast<int64_t>(blockIdx.x) * 8 + warp; g < groups; g += static_cast<int64_t>(gridDim.x) * 8) {
    const int64_t row = g + lane * groups;
    const int c = row < V ? cnt[row] : 0;
    const int b = c ? cursor[row] - c : 0;
    if (c == 1) sorted[b] = seg_pos[b];
    uint32_t todo = __ballot_sync(0xffffffffu, c > 1 && c <= kEmbLight);
    while (todo) {
      const int r = __ffs(todo) - 1;
      todo &= todo - 1;
      const int cr = __shfl_sync(0xffffffffu, c, r), br = __shfl_sync(0xffffffffu, b, r);
      const int p = lane < cr ? seg_pos[br + lane] : 0x7fffffff;
      int rank = 0;
      for (int k = 0; k < cr; ++k) rank += __shfl_sync(0xffffffffu, p, k) < p ? 1 : 0;
      if (lane < cr) sorted[br + rank] = p;
    }
  }
}

// Few tokens and a short table: one CTA sorts (row, position) as one word and reads the segments off the sorted
// words, in place of a memset and the four kernels above, whose launches are most of what they take (254 tokens on 43 rows
// of 47 the call 18.8 us, 9.3 so). From some 2000 tokens on the one CTA takes longer.
constexpr int kEmbSmallTokens = 1024, kEmbSmallRows = 1 << 15;
__global__ void __launch_bounds__(kEmbSmallTokens / 2) emb_small(const void* __restrict__ idx, int i32, int n, int V, int64_t padding_idx, int* __restrict__ cnt, int* __restrict__ cursor, int* __restrict__ sorted,
                                                  int* __restrict__ heavy_count, int* __restrict__ heavy_list, int slots, uint32_t* status) {
  constexpr uint32_t kNone = 0xffffffffu;
  constexpr int kPosBits = 10;
  static_assert(kEmbSmallTokens == 1 << kPosBits, "a position in the low bits of a word");
  __shared__ uint32_t key[kEmbSmallTokens];
  __shared__ int heavy;
  const int t = threadIdx.x;
  if (t == 0) heavy = 0;
  for (int i = t; i < slots; i += blockDim.x) {
    uint32_t k = kNone;
    if (i < n) {
      const int64_t v = emb_index(idx, i, i32);
      if (v == padding_idx) k = kNone;
      else if (v < 0 || v >= V) flag_oob(status);
      else k = static_cast<uint32_t>(v) << kPosBits | static_cast<uint32_t>(i);
    }
    key[i] = k;
  }
  for (int v = t; v < V; v += blockDim.x) cnt[v] = 0;
  __syncthreads();
  for (int size = 2; size <= slots; size <<= 1) {  // bitonic; `slots` is a power of two
    for (int gap = size >> 1; gap > 0; gap >>= 1) {
      for (int i = t; i < slots / 2; i += blockDim.x) {
        const int a = 2 * i - (i & (gap - 1)), b = a + gap;
        const uint32_t x = key[a], y = key[b];
        if ((x > y) == ((a & size) == 0)) {
          key[a] = y;
          key[b] = x;
        }
      }
      __syncthreads();
    }
  }
  for (int i = t; i < n; i += blockDim.x) {
    const uint32_t k = key[i];
    if (k == kNone) continue;
    sorted[i] = static_cast<int>(k & ((1u << kPosBits) - 1u));
    const uint32_t v = k >> kPosBits;
    if (i + 1 < n && key[i + 1] >> kPosBits == v) continue;
    // the last of its row: the first one is found by bisection
    int lo = 0, hi = i;
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (key[mid] >> kPosBits < v) lo = mid + 1;
      else hi = mid;
    }
    const int c = i + 1 - lo;
    cnt[v] = c;  // (every counter was cleared before the barriers above)
    cursor[v] = i + 1;
    if (c > kEmbLight) heavy_list[atomicAdd(&heavy, 1)] = static_cast<int>(v);
  }
  __syncthreads();
  if (t == 0) *heavy_count = heavy;
}

// WORD: the type of one load of the long rows (4 bytes where row length and bases allow it)
template <typename T, typename WORD> __device__ __forceinline__ void emb_word_add(float* acc, WORD w) {
  if constexpr (sizeof(WORD) == sizeof(T)) {
    acc[0] += to_f32(*reinterpret_cast<const T*>(&w));
  } else {
    const T* e = reinterpret_cast<const T*>(&w);
    acc[0] += to_f32(e[0]);
    acc[1] += to_f32(e[1]);
  }
}

template <typename T, bool VEC, typename WORD>
__global__ void __launch_bounds__(256, 4) emb_replay(const T* __restrict__ grad, T* __restrict__ out, const int* cnt, const int* cursor, const int* sorted,
                                                     int64_t V, int64_t D, const int* heavy_count, const int* heavy_list, int heavy_blocks, int tx_log2) {
  after_grids_before();
  if (static_cast<int>(blockIdx.x) < heavy_blocks) {
    constexpr int PK = sizeof(WORD) / sizeof(T);
    const int lane = threadIdx.x & 31;
    const int64_t words = D / PK, chunks = (words + 31) / 32;
    const int64_t nunits = *heavy_count * chunks;
    const WORD* gw = reinterpret_cast<const WORD*>(grad);
    for (int64_t unit = static_cast<int64_t>(blockIdx.x) * 8 + (threadIdx.x >> 5); unit < nunits; unit += static_cast<int64_t>(heavy_blocks) * 8) {
      const int64_t h = unit / chunks;
      const int64_t w = (unit - h * chunks) * 32 + lane;
      const int64_t v = heavy_list[h];
      const int c = cnt[v];
      const int* seg = sorted + (cursor[v] - c);
      const WORD* gl = gw + (w < words ? w : words - 1);  // lanes past the row read its last word and store nothing
      float acc[PK];
#pragma unroll
      for (int q = 0; q < PK; ++q) acc[q] = 0.f;
      // 32 rows at a time. A lane works out where one of the next 32 lies, and brings its line into L2 a batch ahead;
      // the lanes hand these around. (With a product per load, and 16 at a time of 2-byte words: f16 21648 tokens on 56 rows of 3527
      // 416 us the call, 180 so; bf16 32768 tokens on 16 rows of 4096 399, 278. Half a batch on its way while the other is added: 445.)
      auto row_of = [&](int k) { return k + lane < c ? static_cast<int64_t>(seg[k + lane]) * words : 0; };
      int64_t at = row_of(0), ahead = row_of(32);
      int k0 = 0;
      for (; k0 + 32 <= c; k0 += 32) {
        WORD r[32];
#pragma unroll
        for (int k = 0; k < 32; ++k) r[k] = gl[__shfl_sync(0xffffffffu, at, k)];
        at = ahead;
        ahead = row_of(k0 + 64);
        asm volatile("prefetch.global.L2 [%0];" ::"l"(gw + (w - lane) + ahead));
#pragma unroll
        for (int k = 0; k < 32; ++k) emb_word_add<T, WORD>(acc, r[k]);
      }
      for (int k = 0; k < c - k0; ++k) emb_word_add<T, WORD>(acc, gl[__shfl_sync(0xffffffffu, at, k)]);
      if (w < words) {
        WORD o;
        T* e = reinterpret_cast<T*>(&o);
#pragma unroll
        for (int q = 0; q < PK; ++q) e[q] = from_f32<T>(acc[q]);
        reinterpret_cast<WORD*>(out)[v * words + w] = o;
      }
    }
    return;
  }
  if constexpr (!VEC) {
    if (tx_log2 < 0) {
      // rows off the 16-byte grid, most of them without a contribution: 16 bytes of the table to a thread, which meet one row
      // or two (fp32 39666 x 363, one token: element by element the call took 35 us, 20 so)
      constexpr int VE = Vec<T>::N;
      const int64_t total = V * D, step = static_cast<int64_t>(gridDim.x - heavy_blocks) * (256 * VE);
      for (int64_t p = (static_cast<int64_t>(blockIdx.x - heavy_blocks) * 256 + threadIdx.x) * VE; p < total; p += step) {
        const int64_t v = total <= 0x7fffffffLL ? static_cast<int64_t>(static_cast<uint32_t>(p) / static_cast<uint32_t>(D)) : p / D;
        const int64_t u0 = p - v * D;
        const bool crosses = u0 + VE > D && v + 1 < V;
        const int c0 = cnt[v], c1 = crosses ? cnt[v + 1] : 0;
        if ((c0 | c1) == 0 && p + VE <= total) {
          st_stream(out + p, make_uint4(0, 0, 0, 0));
          continue;
        }
        for (int e = 0; e < VE && p + e < total; ++e) {
          const bool next = u0 + e >= D;
          const int64_t row = next ? v + 1 : v, u = next ? u0 + e - D : u0 + e;
          const int c = next ? c1 : c0;
          if (c > kEmbLight) continue;  // a long row: not ours
          const int* seg = sorted + (c ? cursor[row] - c : 0);
          float acc = 0.f;
#pragma unroll 4
          for (int k = 0; k < c; ++k) acc += to_f32(grad[static_cast<int64_t>(seg[k]) * D + u]);
          out[p + e] = from_f32<T>(acc);
        }
      }
      return;
    }
  }
  constexpr int VE = VEC ? Vec<T>::N : 1;
  const int64_t units = D / VE;
  const int tx = threadIdx.x & ((1 << tx_log2) - 1), ty = threadIdx.x >> tx_log2, rows = 256 >> tx_log2;
  const int64_t step = static_cast<int64_t>(gridDim.x - heavy_blocks) * rows;
  int64_t v = static_cast<int64_t>(blockIdx.x - heavy_blocks) * rows + ty;
  int c = v < V ? cnt[v] : 0;
  while (v < V) {
    const int64_t vn = v + step;
    const int cn = vn < V ? cnt[vn] : 0;
    if (c <= kEmbLight) {
      const int* seg = sorted + (c ? cursor[v] - c : 0);
      for (int64_t u = tx; u < units; u += 1 << tx_log2) {
        if constexpr (VEC) {
          float acc[VE];
#pragma unroll
          for (int q = 0; q < VE; ++q) acc[q] = 0.f;
          int k = 0;
          for (; k + 4 <= c; k += 4) {
            uint4 raw[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) raw[q] = ld_stream(grad + static_cast<int64_t>(seg[k + q]) * D + u * VE);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              float f[VE];
              widen<T>(raw[q], f);
#pragma unroll
              for (int e = 0; e < VE; ++e) acc[e] += f[e];
            }
          }
          for (; k < c; ++k) {
            float f[VE];
            widen<T>(ld_stream(grad + static_cast<int64_t>(seg[k]) * D + u * VE), f);
#pragma unroll
            for (int e = 0; e < VE; ++e) acc[e] += f[e];
          }
          st_stream(out + v * D + u * VE, narrow<T>(acc));
        } else {
          float acc = 0.f;
#pragma unroll 4
          for (int k = 0; k < c; ++k) acc += to_f32(grad[static_cast<int64_t>(seg[k]) * D + u]);
          out[v * D + u] = from_f32<T>(acc);
        }
      }
    }
    v = vn;
    c = cn;
  }
}

struct EmbScratch {
  int64_t cnt_bytes, cursor_bytes, pos_bytes, heavy_bytes, total;
};
static EmbScratch emb_scratch(int64_t V, int64_t n) {
  EmbScratch s;
  s.cnt_bytes = 256 + up256(4 * V);  // [0] slots handed out, [1] long rows; the counters behind them
  s.cursor_bytes = up256(4 * V);
  s.pos_bytes = up256(4 * n);
  s.heavy_bytes = up256(4 * (n / (kEmbLight + 1) + 1));
  s.total = s.cnt_bytes + s.cursor_bytes + 2 * s.pos_bytes + s.heavy_bytes;
  return s;
}

template <typename T>
static int launch_embedding_backward(const void* grad, const void* idx, void* out, int64_t n, int64_t V, int64_t D, int64_t padding_idx, int i32, void* scratch, uint32_t* status, cudaStream_t st) {
  const EmbScratch S = emb_scratch(V, n);
  char* base = static_cast<char*>(scratch);
  int* head = reinterpret_cast<int*>(base);
  int* cnt = reinterpret_cast<int*>(base + 256);
  int* cursor = reinterpret_cast<int*>(base + S.cnt_bytes);
  int* seg_pos = reinterpret_cast<int*>(base + S.cnt_bytes + S.cursor_bytes);
  int* sorted = reinterpret_cast<int*>(base + S.cnt_bytes + S.cursor_bytes + S.pos_bytes);
  int* heavy = reinterpret_cast<int*>(base + S.cnt_bytes + S.cursor_bytes + 2 * S.pos_bytes);
  auto grid = [](int64_t items, int per, int64_t cap) { const int64_t g = (items + per - 1) / per; return static_cast<int>(g < 1 ? 1 : (g > cap ? cap : g)); };
  int launches = 2;
  cudaError_t e = cudaSuccess;
  if (n <= kEmbSmallTokens && V <= kEmbSmallRows) {
    int slots = 32;
    while (slots < n) slots <<= 1;
    emb_small<<<1, slots / 2 < 64 ? 64 : slots / 2, 0, st>>>(idx, i32, static_cast<int>(n), static_cast<int>(V), padding_idx, cnt, cursor, sorted, head + 1, heavy, slots, status);
  } else {
    e = cudaMemsetAsync(head, 0, static_cast<size_t>(S.cnt_bytes), st);
    if (e != cudaSuccess) { set_last_cuda_error(e); return B200_ELAUNCH; }
    emb_count<<<grid(n, 256, 32 * kNumSMs), 256, 0, st>>>(idx, i32, n, V, padding_idx, cnt, status);
    e = launch_after(assign_segments<4>, (V + 1023) / 1024, 256, 0, st, cnt, cursor, V, head, kEmbLight, head + 1, heavy);
    if (e == cudaSuccess) e = launch_after(emb_fill, grid(n, 256, 32 * kNumSMs), 256, 0, st, idx, i32, n, V, padding_idx, cursor, seg_pos);
    // a CTA to 256 rows of the table or to one long row, of which a short table under many tokens has more (fp32, 32768
    // tokens on 256 rows of 64: 88 us the call, 424 with the one CTA that the table alone asks for)
    const int64_t long_rows = n / (kEmbLight + 1) < V ? n / (kEmbLight + 1) : V, row_groups = (V + 255) / 256;
    if (e == cudaSuccess) e = launch_after(emb_sort, grid(long_rows > row_groups ? long_rows : row_groups, 1, 2 * kNumSMs), 256, 0, st, cnt, cursor, seg_pos, sorted, V, n, head + 1, heavy);
    launches = 5;
  }
  const T* g = static_cast<const T*>(grad);
  T* o = static_cast<T*>(out);
  const bool vec = (D * static_cast<int64_t>(sizeof(T))) % 16 == 0 && aligned16(grad) && aligned16(out);
  const bool words = (D * static_cast<int64_t>(sizeof(T))) % 4 == 0 && ((reinterpret_cast<uintptr_t>(grad) | reinterpret_cast<uintptr_t>(out)) & 3u) == 0;
  const int64_t units = vec ? D / Vec<T>::N : D;
  // threads of a CTA along a row: the power of two that covers it, 256 at most; for a row that one trip covers less,
  // down to 64, where that leaves fewer than one thread in eight idle (fp32 32000 x 768, 32768 tokens: 64 threads to a
  // row 70 us, 256 78 us)
  int tx_log2 = 0;
  while (tx_log2 < 8 && (1LL << tx_log2) < units) ++tx_log2;
  for (int t = tx_log2; t >= 6 && units <= 256; --t) {
    if ((units + (1LL << t) - 1) / (1LL << t) * (1LL << t) * 7 <= units * 8) { tx_log2 = t; break; }
  }
  // a table so short that a list of long rows cannot exist gets no CTAs for it
  const int heavy_blocks = n > kEmbLight ? grid(n / (kEmbLight + 1) * ((D * static_cast<int64_t>(sizeof(T)) + 127) / 128), 8, kNumSMs) : 0;
  // (flat: 16 bytes of the table to a thread, see emb_replay)
  const bool flat = !vec && n <= V && D * static_cast<int64_t>(sizeof(T)) >= 16 && aligned16(out);
  const int light_blocks = flat ? grid(V * D, 256 * Vec<T>::N, 16 * kNumSMs) : grid(V, 256 >> tx_log2, 8 * kNumSMs);
  if (flat) tx_log2 = -1;
  auto launch = [&](auto kernel) {
    if (e == cudaSuccess) e = launch_after(kernel, heavy_blocks + light_blocks, 256, 0, st, g, o, cnt, cursor, sorted, V, D, head + 1, heavy, heavy_blocks, tx_log2);
  };
  if (vec) launch(emb_replay<T, true, uint32_t>);
  else if (words) launch(emb_replay<T, false, uint32_t>);
  else if constexpr (sizeof(T) == 2) launch(emb_replay<T, false, uint16_t>);
  if (e != cudaSuccess) { set_last_cuda_error(e); return B200_ELAUNCH; }
  return check_launch(launches);
}

template <typename T>
static int launch_strip(const void* self, const void* index, const void* src, void* out, StripArgs A, uint32_t* status, cudaStream_t st, const int* only_if) {
  const int tile_bytes = kTileRows * kStripCols * (8 + static_cast<int>(sizeof(T)));
  const int tag_bytes = (kStripThreads / 32) * kTagSlots;
  // keep at least 4 stages of source tiles; the rest of the budget holds destination rows
  int64_t win = (kSmemBudget - tag_bytes - 4 * tile_bytes) / (kStripCols * 4);
  if (win > A.rows) win = A.rows;
  A.win_rows = static_cast<int>(win);
  // a destination that fits in half an SM's shared memory leaves room for a second CTA
  const int64_t budget = tag_bytes + win * kStripCols * 4 + 3 * tile_bytes <= kStripSmemTarget ? kStripSmemTarget : kSmemBudget;
  int stages = static_cast<int>((budget - tag_bytes - win * kStripCols * 4) / tile_bytes);
  if (stages > 8) stages = 8;  // the wait depth cp.async can express
  if (stages < 2) stages = 2;
  A.stages = stages;
  const size_t smem = static_cast<size_t>(stages) * tile_bytes + tag_bytes + static_cast<size_t>(win) * kStripCols * 4;
  const cudaError_t ae = cudaFuncSetAttribute(scatter_add_strip<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBudget);
  if (ae != cudaSuccess) { set_last_cuda_error(ae); return B200_ELAUNCH; }
  const int64_t items = A.outer * (A.cols / kStripCols);
  const int grid = static_cast<int>(items < 8LL * kNumSMs ? items : 8LL * kNumSMs);
  const T *px = static_cast<const T*>(self), *ps = static_cast<const T*>(src);
  const int64_t* pi = static_cast<const int64_t*>(index);
  T* po = static_cast<T*>(out);
  if (only_if) {
    const cudaError_t e = launch_after(scatter_add_strip<T>, grid, kStripThreads, smem, st, px, pi, ps, po, A, only_if, status);
    if (e != cudaSuccess) { set_last_cuda_error(e); return B200_ELAUNCH; }
  } else {
    scatter_add_strip<T><<<grid, kStripThreads, smem, st>>>(px, pi, ps, po, A, only_if, status);
  }
  return check_launch();
}

template <typename T>
static int launch_strip_wide(const void* self, const void* index, const void* src, void* out, const StripArgs& A, uint32_t* status, cudaStream_t st) {
  // tensor maps over the index and value tensors (this GPU's own memory, no multicast): boxes
  // of 8 columns x 128 rows, swizzled the way the compute warps read them
  if (!encode_fn()) return B200_EDRIVER;
  alignas(64) CUtensorMap map_idx, map_src;
  const cuuint64_t dims[3] = {static_cast<cuuint64_t>(A.idx_cols), static_cast<cuuint64_t>(A.idx_rows), static_cast<cuuint64_t>(A.idx_outer)};
  const cuuint32_t box[3] = {kWideCols, kWideTileRows, 1};
  const cuuint32_t estr[3] = {1, 1, 1};
  auto outer_stride = [&](int64_t so, int64_t sr, int64_t es) { return static_cast<cuuint64_t>((A.idx_outer > 1 && so > 0 ? so : sr * A.idx_rows) * es); };
  const cuuint64_t istr[2] = {static_cast<cuuint64_t>(A.idx_sr) * 8, outer_stride(A.idx_so, A.idx_sr, 8)};
  const int es = static_cast<int>(sizeof(T));
  const cuuint64_t sstr[2] = {static_cast<cuuint64_t>(A.src_sr) * es, outer_stride(A.src_so, A.src_sr, es)};
  if (istr[1] % 16 || sstr[1] % 16) return B200_EALIGN;
  if (encode_fn()(&map_idx, CU_TENSOR_MAP_DATA_TYPE_INT64, 3, const_cast<void*>(index), dims, istr, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
    return B200_EDRIVER;
  const CUtensorMapDataType vt = std::is_same<T, float>::value ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : std::is_same<T, __nv_bfloat16>::value ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
  const CUtensorMapSwizzle vs = sizeof(T) == 4 ? CU_TENSOR_MAP_SWIZZLE_32B : CU_TENSOR_MAP_SWIZZLE_NONE;  // 16-bit rows are one 16-byte chunk
  if (encode_fn()(&map_src, vt, 3, const_cast<void*>(src), dims, sstr, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, vs, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) !=
      CUDA_SUCCESS)
    return B200_EDRIVER;
  alignas(64) CUtensorMap map_self;  // the destination strip on its way in: 8 columns x 256 rows, rows as they lie
  {
    const cuuint64_t ddims[3] = {static_cast<cuuint64_t>(A.cols), static_cast<cuuint64_t>(A.rows), static_cast<cuuint64_t>(A.outer)};
    const cuuint64_t dstr[2] = {static_cast<cuuint64_t>(A.cols) * es, static_cast<cuuint64_t>(A.rows) * static_cast<cuuint64_t>(A.cols) * es};
    const cuuint32_t dbox[3] = {kWideCols, kWideSelfRows, 1};
    if (dstr[0] % 16 || (reinterpret_cast<uintptr_t>(self) & 15)) return B200_EALIGN;
    if (encode_fn()(&map_self, vt, 3, const_cast<void*>(self), ddims, dstr, dbox, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return B200_EDRIVER;
  }
  alignas(64) CUtensorMap map_out;  // ... and on its way out: 8 columns x 32 rows
  {
    const cuuint64_t ddims[3] = {static_cast<cuuint64_t>(A.cols), static_cast<cuuint64_t>(A.rows), static_cast<cuuint64_t>(A.outer)};
    const cuuint64_t dstr[2] = {static_cast<cuuint64_t>(A.cols) * es, static_cast<cuuint64_t>(A.rows) * static_cast<cuuint64_t>(A.cols) * es};
    const cuuint32_t dbox[3] = {kWideCols, kWideOutRows, 1};
    if (reinterpret_cast<uintptr_t>(out) & 15) return B200_EALIGN;
    if (encode_fn()(&map_out, vt, 3, out, ddims, dstr, dbox, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) !=
        CUDA_SUCCESS)
      return B200_EDRIVER;
  }
  // ring + tag tables + the strip at its largest + barriers + room to align the ring to 1 KB
  const size_t smem = static_cast<size_t>(kWideStages) * kWideTileRows * kWideCols * (8 + sizeof(T)) + 8 * (kWideTagSlots + kWideDummies) + static_cast<size_t>(kWideMaxRows + kWideDummies) * kWideCols * 4 + 128 + 1024;
  const cudaError_t ae = cudaFuncSetAttribute(scatter_add_strip_wide<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
  if (ae != cudaSuccess) { set_last_cuda_error(ae); return B200_ELAUNCH; }
  const int64_t items = A.outer * (A.cols / kWideCols);
  const int grid = static_cast<int>(items < kNumSMs ? items : kNumSMs);  // one CTA per SM: a strip leaves while the next one comes in
  scatter_add_strip_wide<T><<<grid, kWideThreads, smem, st>>>(map_idx, map_src, map_self, map_out, A, status);
  return check_launch();
}

template <typename T>
static int launch_rows(const void* self, const void* index, const void* src, void* out, RowArgs A, uint32_t* status, cudaStream_t st) {
  // few long rows: several warps per row, each with a range of the row's destinations
  if (A.outer < 2LL * kNumSMs && A.idx_len >= 256 && A.rows >= 128) {
    int64_t slices = (4LL * kNumSMs + A.outer - 1) / A.outer;
    if (slices > A.rows / 64) slices = A.rows / 64;
    if (slices > 32) slices = 32;
    if (slices >= 2) {
      const int64_t slice_rows = (A.rows + slices - 1) / slices;
      slices = (A.rows + slice_rows - 1) / slice_rows;  // no empty range at the end
      int warps = 8;
      while (warps > 1 && static_cast<int64_t>(warps) * (slice_rows * 4 + kTagSlots) > 96 * 1024) warps >>= 1;
      const size_t smem = static_cast<size_t>(warps) * (slice_rows * 4 + kTagSlots);
      if (smem <= static_cast<size_t>(kSmemBudget)) {
        const cudaError_t ae = cudaFuncSetAttribute(scatter_add_rows_sliced<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBudget);
        if (ae != cudaSuccess) { set_last_cuda_error(ae); return B200_ELAUNCH; }
        const int64_t items = A.outer * slices;
        // one item per warp where the machine has room: spread the items over the SMs first
        int per_cta = static_cast<int>((items + kNumSMs - 1) / kNumSMs);
        if (per_cta > warps) per_cta = warps;
        if (per_cta < 1) per_cta = 1;
        const int64_t blocks = (items + per_cta - 1) / per_cta;
        scatter_add_rows_sliced<T><<<static_cast<int>(blocks), per_cta * 32, static_cast<size_t>(per_cta) * (slice_rows * 4 + kTagSlots), st>>>(
            static_cast<const T*>(self), static_cast<const int64_t*>(index), static_cast<const T*>(src), static_cast<T*>(out), A, static_cast<int>(slices), static_cast<int>(slice_rows), status);
        return check_launch();
      }
    }
  }
  // two destination rows per warp; shrink the CTA before windowing the destination
  int warps = 8;
  while (warps > 1 && static_cast<int64_t>(warps) * (2 * A.rows * 4 + kTagSlots) > 96 * 1024) warps >>= 1;
  int64_t win = A.rows;
  const int64_t dest_budget = kSmemBudget - static_cast<int64_t>(warps) * kTagSlots;
  if (static_cast<int64_t>(warps) * 2 * win * 4 > dest_budget) win = dest_budget / (warps * 2 * 4);
  A.win_rows = static_cast<int>(win);
  const size_t smem = static_cast<size_t>(warps) * (2 * win * 4 + kTagSlots);
  const cudaError_t ae = cudaFuncSetAttribute(scatter_add_rows<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBudget);
  if (ae != cudaSuccess) { set_last_cuda_error(ae); return B200_ELAUNCH; }
  const int64_t pairs = (A.outer + 1) / 2;
  int64_t blocks = (pairs + warps - 1) / warps;
  if (blocks > 16LL * kNumSMs) blocks = 16LL * kNumSMs;
  scatter_add_rows<T><<<static_cast<int>(blocks), warps * 32, smem, st>>>(static_cast<const T*>(self), static_cast<const int64_t*>(index), static_cast<const T*>(src), static_cast<T*>(out), A, status);
  return check_launch();
}

}  // namespace b200

namespace b200 {

// Nanoseconds, as measured over 64 x 1024 ... 15000 x 1024 and 150134 x 63. A strip CTA takes 14.5 for a source row, whatever its
// few columns are (twice that where the destination takes two windows), and 2400 to begin and end, and there are one or two of
// them per SM; the binned path has more launches to pay for, and then time for each contribution and destination. Strips
// against bins, in the stream, as many source rows as rows: fp32 2000 x 256 31.7 / 24.8 us, 4000 x 512 59.6 / 39.7, 12000 x 512 315 / 118, f16 969 x 252
// 19.6 / 24.8, 2672 x 332 43.2 / 26.9; half as many: fp32 2446 x 168 24.7 / 25.5, bf16 1951 x 140 18.6 / 20.7.
static bool binned_beats_strip(const StripArgs& S, int64_t n_idx) {
  const int64_t bytes = S.rows * kStripCols * 4, at_once = kNumSMs * (bytes <= kStripSmemTarget - 34 * 1024 ? 2 : 1);
  const int64_t rounds = (S.outer * (S.cols / kStripCols) + at_once - 1) / at_once, windows = bytes <= kSmemBudget - 40 * 1024 ? 1 : 2;
  const double strip = static_cast<double>(rounds) * (14.5 * static_cast<double>(S.idx_rows * windows) + 2400.0) + 2000.0;
  return strip > 20000.0 + 0.009 * static_cast<double>(n_idx) + 0.003 * static_cast<double>(S.outer * S.rows * S.cols);
}

enum ScatterPath { kPathNone = 0, kPathStrip, kPathStripWide, kPathRows, kPathBinned, kPathBucket, kPathChain, kPathLines };

struct ScatterPlan {
  ScatterPath path;
  int64_t n_self, n_idx, scratch_bytes;
  bool strips;  // bins, with strips for a crowded index
  StripArgs strip;
  RowArgs rows;
  BinnedArgs binned;
};

// Decides which kernel family serves a geometry (shared by the launcher and the scratch
// query so that both always agree).
static ScatterPlan plan_scatter(const void* self, const void* index, const void* src, const void* out, int ndim, const int64_t* self_shape, const int64_t* index_shape,
                                const int64_t* index_strides, const int64_t* src_strides, int dim, int dtype) {
  ScatterPlan P{};
  P.n_self = numel_of(ndim, self_shape);
  P.n_idx = numel_of(ndim, index_shape);
  const int es = dtype_size(dtype);
  P.path = kPathLines;
  if (P.n_self == 0 || P.n_idx == 0) { P.path = kPathNone; return P; }
  const bool small = P.n_idx <= (1 << 16);  // launch-bound either way
  const bool aligned = aligned16(self) && aligned16(out) && aligned16(index) && aligned16(src);
  {
    int64_t outer = 1, cols = 1, idx_outer = 1, idx_cols = 1;
    for (int d = 0; d < dim; ++d) { outer *= self_shape[d]; idx_outer *= index_shape[d]; }
    for (int d = dim + 1; d < ndim; ++d) { cols *= self_shape[d]; idx_cols *= index_shape[d]; }
    const int64_t rows = self_shape[dim], idx_rows = index_shape[dim];
    int lead = 0, trail = 0, dl = -1, dt = -1;  // collapsible only with at most one non-trivial dim on each side
    for (int d = 0; d < dim; ++d)
      if (self_shape[d] > 1 || index_shape[d] > 1) { ++lead; dl = d; }
    for (int d = dim + 1; d < ndim; ++d)
      if (self_shape[d] > 1 || index_shape[d] > 1) { ++trail; dt = d; }
    if (lead <= 1 && trail <= 1 && rows < 0x7fffffffLL) {
      const int64_t idx_so = dl >= 0 ? index_strides[dl] : 0, src_so = dl >= 0 ? src_strides[dl] : 0;
      if (dt >= 0) {
        const bool inner_ok = index_strides[dt] == 1 && src_strides[dt] == 1;
        const bool shape_ok = cols % kStripCols == 0 && idx_cols % kStripCols == 0;
        const bool stride_ok = (src_strides[dim] * es) % 4 == 0 && (src_so * es) % 4 == 0;  // 4-byte value granules
        const int64_t strips = outer * (cols / kStripCols);
        const bool fits = rows * kStripCols * 4 <= 2 * (kSmemBudget - 64 * 1024);  // at most two destination windows
        P.binned = BinnedArgs{outer, rows, cols, idx_outer, idx_rows, idx_cols, idx_so, index_strides[dim], index_strides[dt], src_so, src_strides[dim], src_strides[dt]};
        // fp32, as many source rows as rows, lines or chains against bins: 32 x 333 21.2 / 7.1 us, 64 x 63 35.8 / 7.3, 65 x 333 21.5 / 7.5, 128 x 1023
        // 23.1 / 11.4, 200 x 63 20.8 / 15.7, 200 x 4095 39.6 / 34.1; with the look at the index 65 x 8191 30 / 35 and 100 x 4095 27 / 29. Lines that there are
        // many of: bf16 64 x 24, 267 of them, 20.3 / 29.5, f16 42 x 565, 145, 66 / 93.
        const bool bins_pay = (idx_rows >= 128 || (idx_rows > 24 && outer * cols <= 2048)) && P.n_self < 0x7fffffffLL && P.n_idx < 0x7fffffffLL && plan_binned(P.binned);
        if (aligned && inner_ok && shape_ok && stride_ok && fits && (strips >= 32 || small)) {
          P.path = kPathStrip;
          P.strip = StripArgs{outer, rows, cols, idx_outer, idx_rows, idx_cols, idx_so, index_strides[dim], src_so, src_strides[dim], 0, 0};
          // eight columns per CTA when the whole destination strip fits and every staged chunk is 16-byte aligned
          const bool wide_shape = cols % kWideCols == 0 && idx_cols % kWideCols == 0 && rows <= kWideMaxRows && idx_rows >= 256 && idx_rows < 0x7fffffffLL && outer * (cols / kWideCols) >= kNumSMs / 2;
          const bool wide_align = index_strides[dim] % 2 == 0 && idx_so % 2 == 0 && (src_strides[dim] * es) % 16 == 0 && (src_so * es) % 16 == 0;
          if (wide_shape && wide_align) P.path = kPathStripWide;
          if (P.path == kPathStripWide || !bins_pay || !binned_beats_strip(P.strip, P.n_idx)) return P;
          P.strips = true;
        }
        if (bins_pay) {
          P.path = kPathBinned;
          const bool alone = P.strips || idx_rows <= kBinUnseen;
          P.scratch_bytes = binned_scratch(P.binned, es, alone ? 0 : P.n_self, alone ? 0 : P.n_idx).total;
          return P;
        }
      } else if (aligned && index_strides[dim] == 1 && src_strides[dim] == 1) {
        const bool fits = rows * 2 * 4 <= kSmemBudget - 16 * 1024;
        if (fits && (outer >= 64 || small)) {
          P.path = kPathRows;
          P.rows = RowArgs{outer, rows, idx_outer, idx_rows, idx_so, src_so, 0};
          return P;
        }
      }
    }
  }
  // short lines are cheapest walked by one thread each; anything longer is grouped by destination
  if (P.n_self < 0x7fffffffLL && P.n_idx < 0x7fffffffLL && index_shape[dim] < 0x7fffffffLL && index_shape[dim] > 64) {
    // at most one contribution per reachable destination on average: chains (fp32 150134 x 63, as many
    // rows: 245 us, segments 530). More make chains long, and a segment's entries lie side by side
    // where a chain's do not.
    P.path = index_shape[dim] <= self_shape[dim] ? kPathChain : kPathBucket;
    P.scratch_bytes = P.path == kPathChain ? chain_scratch(P.n_self, P.n_idx).total : bucket_scratch(P.n_self, P.n_idx).total;
    return P;
  }
  P.scratch_bytes = dtype == B200_F32 ? 0 : P.n_self * 4;  // fp32 accumulator of the line kernel
  return P;
}

}  // namespace b200

using namespace b200;

extern "C" int64_t b200_scatter_add_scratch_bytes(const void* self, const void* index, const void* src, const void* out, int ndim, const int64_t* self_shape,
                                                   const int64_t* index_shape, const int64_t* index_strides, const int64_t* src_strides, int dim, int dtype) {
  if (ndim < 1 || ndim > B200_MAX_DIMS || dim < 0 || dim >= ndim || !self_shape || !index_shape || !index_strides || !src_strides || !is_float_dtype(dtype)) return 0;
  return plan_scatter(self, index, src, out, ndim, self_shape, index_shape, index_strides, src_strides, dim, dtype).scratch_bytes;
}

extern "C" int b200_scatter_add_path(const void* self, const void* index, const void* src, const void* out, int ndim, const int64_t* self_shape, const int64_t* index_shape,
                                     const int64_t* index_strides, const int64_t* src_strides, int dim, int dtype) {
  if (ndim < 1 || ndim > B200_MAX_DIMS || dim < 0 || dim >= ndim || !self_shape || !index_shape || !index_strides || !src_strides || !is_float_dtype(dtype)) return B200_EINVAL;
  const ScatterPath p = plan_scatter(self, index, src, out, ndim, self_shape, index_shape, index_strides, src_strides, dim, dtype).path;
  static_assert(kPathNone == B200_SCATTER_NONE && kPathStrip == B200_SCATTER_STRIP && kPathStripWide == B200_SCATTER_STRIP_WIDE && kPathRows == B200_SCATTER_ROWS &&
                    kPathBinned == B200_SCATTER_BINS && kPathBucket == B200_SCATTER_BUCKETS && kPathChain == B200_SCATTER_CHAINS && kPathLines == B200_SCATTER_LINES, "the header's names");
  return p;
}

extern "C" int b200_scatter_add(const void* self, const void* index, const void* src, void* out, int ndim, const int64_t* self_shape, const int64_t* index_shape,
                                const int64_t* index_strides, const int64_t* src_strides, int dim, int dtype, void* scratch, int64_t scratch_bytes, uint32_t* status, void* stream) {
  if (ndim < 1 || ndim > B200_MAX_DIMS || dim < 0 || dim >= ndim || !self_shape || !index_shape || !index_strides || !src_strides) return B200_EINVAL;
  if (!is_float_dtype(dtype)) return B200_EDTYPE;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  for (int d = 0; d < ndim; ++d)
    if (self_shape[d] < 0 || index_shape[d] < 0 || (d != dim && index_shape[d] > self_shape[d])) return B200_EINVAL;
  const int64_t n_self = numel_of(ndim, self_shape);
  const int64_t n_idx = numel_of(ndim, index_shape);
  if (n_self == 0) return B200_OK;
  if (!self || !out) return B200_EINVAL;
  if (n_idx > 0 && (!index || !src)) return B200_EINVAL;
  const int es = dtype_size(dtype);
  const ScatterPlan P = plan_scatter(self, index, src, out, ndim, self_shape, index_shape, index_strides, src_strides, dim, dtype);

  if (P.path == kPathNone) {  // nothing to add: the result is a copy of self (no scratch, whatever the dtype)
    if (out != self) {
      const cudaError_t ce = cudaMemcpyAsync(out, self, static_cast<size_t>(n_self) * es, cudaMemcpyDeviceToDevice, st);
      if (ce != cudaSuccess) { set_last_cuda_error(ce); return B200_ELAUNCH; }
    }
    return B200_OK;
  }
  if (P.path == kPathStrip) {
    switch (dtype) {
      case B200_F32: return launch_strip<float>(self, index, src, out, P.strip, status, st);
      case B200_BF16: return launch_strip<__nv_bfloat16>(self, index, src, out, P.strip, status, st);
      default: return launch_strip<__half>(self, index, src, out, P.strip, status, st);
    }
  }
  if (P.path == kPathStripWide) {
    switch (dtype) {
      case B200_F32: return launch_strip_wide<float>(self, index, src, out, P.strip, status, st);
      case B200_BF16: return launch_strip_wide<__nv_bfloat16>(self, index, src, out, P.strip, status, st);
      default: return launch_strip_wide<__half>(self, index, src, out, P.strip, status, st);
    }
  }
  if (P.path == kPathRows) {
    switch (dtype) {
      case B200_F32: return launch_rows<float>(self, index, src, out, P.rows, status, st);
      case B200_BF16: return launch_rows<__nv_bfloat16>(self, index, src, out, P.rows, status, st);
      default: return launch_rows<__half>(self, index, src, out, P.rows, status, st);
    }
  }
  if (P.path == kPathBinned || P.path == kPathBucket || P.path == kPathChain) {
    if (!scratch || scratch_bytes < P.scratch_bytes) return B200_ESCRATCH;
    BucketArgs A;
    A.ndim = ndim;
    A.dim = dim;
    A.n_idx = n_idx;
    A.n_self = n_self;
    A.dim_len = index_shape[dim];
    A.self_dim_size = self_shape[dim];
    int64_t st_out = 1;
    for (int d = ndim - 1; d >= 0; --d) {
      A.shape[d] = index_shape[d];
      A.out_stride[d] = st_out;
      st_out *= self_shape[d];
      A.idx_stride[d] = index_strides[d];
      A.src_stride[d] = src_strides[d];
    }
    if (P.path == kPathBinned) {
      switch (dtype) {
        case B200_F32: return launch_binned<float>(self, index, src, out, P.binned, A, P.strips ? &P.strip : nullptr, scratch, status, st);
        case B200_BF16: return launch_binned<__nv_bfloat16>(self, index, src, out, P.binned, A, P.strips ? &P.strip : nullptr, scratch, status, st);
        default: return launch_binned<__half>(self, index, src, out, P.binned, A, P.strips ? &P.strip : nullptr, scratch, status, st);
      }
    }
    const bool chain = P.path == kPathChain;
    switch (dtype) {
      case B200_F32: return chain ? launch_chain<float>(self, index, src, out, A, scratch, status, st) : launch_bucket<float>(self, index, src, out, A, scratch, status, st);
      case B200_BF16: return chain ? launch_chain<__nv_bfloat16>(self, index, src, out, A, scratch, status, st) : launch_bucket<__nv_bfloat16>(self, index, src, out, A, scratch, status, st);
      default: return chain ? launch_chain<__half>(self, index, src, out, A, scratch, status, st) : launch_bucket<__half>(self, index, src, out, A, scratch, status, st);
    }
  }

  // ---- line kernel: acc = fp32(self), ordered lines on acc, out = round(acc)
  const bool wide = dtype == B200_F32;
  float* acc = wide ? static_cast<float*>(out) : static_cast<float*>(scratch);
  if (!wide && (!scratch || scratch_bytes < n_self * 4)) return B200_ESCRATCH;
  if (wide) {
    if (out != self) {
      const cudaError_t ce = cudaMemcpyAsync(out, self, static_cast<size_t>(n_self) * es, cudaMemcpyDeviceToDevice, st);
      if (ce != cudaSuccess) { set_last_cuda_error(ce); return B200_ELAUNCH; }
    }
  } else {
    const int64_t one = 1;
    if (int rc = b200_copy_strided(self, acc, 1, &n_self, &one, dtype, B200_F32, stream)) return rc;
  }
  if (n_idx > 0) {
    if (!index || !src) return B200_EINVAL;
    ScatterArgs A;
    A.ndim = ndim;
    A.dim = dim;
    A.dim_len = index_shape[dim];
    A.self_dim_size = self_shape[dim];
    A.nlines = 1;
    int64_t st_out = 1;
    for (int d = ndim - 1; d >= 0; --d) {
      A.shape[d] = d == dim ? 1 : index_shape[d];
      A.nlines *= A.shape[d];
      A.out_stride[d] = st_out;
      st_out *= self_shape[d];
      A.idx_stride[d] = index_strides[d];
      A.src_stride[d] = src_strides[d];
    }
    const int g = grid_for(A.nlines, 128);
    const int64_t* pi = static_cast<const int64_t*>(index);
    switch (dtype) {
      case B200_F32: scatter_add_lines<float><<<g, 128, 0, st>>>(acc, pi, static_cast<const float*>(src), A, status); break;
      case B200_BF16: scatter_add_lines<__nv_bfloat16><<<g, 128, 0, st>>>(acc, pi, static_cast<const __nv_bfloat16*>(src), A, status); break;
      default: scatter_add_lines<__half><<<g, 128, 0, st>>>(acc, pi, static_cast<const __half*>(src), A, status); break;
    }
    if (int rc = check_launch()) return rc;
  }
  if (!wide) {
    const int64_t one = 1;
    return b200_copy_strided(acc, out, 1, &n_self, &one, B200_F32, dtype, stream);
  }
  return B200_OK;
}

extern "C" int64_t b200_embedding_backward_scratch_bytes(int64_t n_indices, int64_t num_weights) {
  if (n_indices < 0 || num_weights <= 0) return 0;
  return emb_scratch(num_weights, n_indices).total;
}

extern "C" int b200_embedding_backward(const void* grad, const void* indices, void* out, int64_t n_indices, int64_t num_weights, int64_t row_len, int64_t padding_idx, int dtype, int idx_dtype,
                                       void* scratch, int64_t scratch_bytes, uint32_t* status, void* stream) {
  if (n_indices < 0 || num_weights < 0 || row_len < 0) return B200_EINVAL;
  if (!is_float_dtype(dtype)) return B200_EDTYPE;
  if (idx_dtype != B200_I32 && idx_dtype != B200_I64) return B200_EDTYPE;
  if (num_weights == 0 || row_len == 0) return B200_OK;
  if (!out || (n_indices > 0 && (!grad || !indices))) return B200_EINVAL;
  if (n_indices >= 0x7fffffffLL || num_weights >= 0x7fffffffLL) return B200_EINVAL;
  if (!scratch || scratch_bytes < b200_embedding_backward_scratch_bytes(n_indices, num_weights)) return B200_ESCRATCH;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int i32 = idx_dtype == B200_I32;
  switch (dtype) {
    case B200_F32: return launch_embedding_backward<float>(grad, indices, out, n_indices, num_weights, row_len, padding_idx, i32, scratch, status, st);
    case B200_BF16: return launch_embedding_backward<__nv_bfloat16>(grad, indices, out, n_indices, num_weights, row_len, padding_idx, i32, scratch, status, st);
    default: return launch_embedding_backward<__half>(grad, indices, out, n_indices, num_weights, row_len, padding_idx, i32, scratch, status, st);
  }
}
