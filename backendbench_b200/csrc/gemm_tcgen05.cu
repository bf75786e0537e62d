// mm / addmm / bmm on the 5th-generation tensor cores (tcgen05) for bf16 / f16 operands.
//
//   C[b] (M x N, row-major) = alpha * A[b] (M x K) @ B[b] (K x N) + beta * bias
//
// One persistent CTA per SM walks 128 x 256 (or 128 x 128) output tiles. Roles by warp:
//   warp 0   : TMA producer -- one lane issues cp.async.bulk.tensor loads
//              of a 128 x 64 A slab and a 64 x 256 B slab per pipeline stage into
//              128-byte-swizzled shared memory, completion on an mbarrier.
//   warp 1   : owns tensor memory (allocates all 512 TMEM columns = two fp32 accumulators
//              of 128 lanes x 256 columns) and issues tcgen05.mma (kind::f16, M128 N256
//              K16, four per stage); tcgen05.commit releases the stage / publishes the
//              accumulator through mbarriers.
//   warps 2-9: epilogue -- tcgen05.ld the accumulator (a warp may read only the 32 TMEM
//              lanes of its quarter, so two warps share a quarter and split the 256
//              columns), scale / add bias in fp32, round once, 16-byte stores. While they
//              drain accumulator `a`, the MMA warp already fills accumulator `a ^ 1`.
// Tiles are walked in groups of 16 row-blocks x all column-blocks so that the CTAs running
// at the same time share A and B slabs in L2.
// Operands may be K-major or MN-major in global memory (A row- or column-major, B given
// as [K,N] or as a transposed [N,K] view): the layout goes into the shared-memory and
// instruction descriptors, nothing is copied or transposed. Ragged M / N / K edges rely on
// TMA zero fill for loads and predicated stores.
//
// CTA pairs (kPair): two CTAs of a 2-CTA cluster, on the two SMs of one TPC, share a 256 x 256
// tile. Each keeps the accumulator of ITS 128 rows in its own tensor memory and loads its own
// 128 x 64 A slab and HALF of the 64 x 256 B slab (32 KB per stage instead of 48, six stages);
// one thread of the even CTA issues tcgen05.mma.cta_group::2 (M256 N256 K16), which reads A
// from both shared memories and each half of B from its own. The odd CTA's copies complete on
// the even CTA's barrier, and tcgen05.commit.cta_group::2 hands stages and accumulators back
// to both. Per FLOP a third fewer operand bytes cross the L2-to-SM fabric, which is what the
// single-CTA kernel waits on at large shapes. No cluster multicast is used anywhere: every
// CTA fetches its own tiles.
//
// Every mbarrier wait is bounded: when a wait gives up the CTA sets an abort flag, ORs
// B200_DEV_WAIT_TIMEOUT into the caller's status word, lets outstanding copies land, frees
// its tensor memory and returns -- a protocol bug can produce a wrong result plus an error
// status, never a hung GPU.
#include <cuda.h>

#include <cstdlib>

#include "b200_common.cuh"
#include "tma_common.cuh"

namespace b200 {

constexpr int kBM = 128, kBK = 64;                      // tile: 128 x BN outputs (BN = 256 or 128), 64-deep K slabs
constexpr int kABytes = kBM * kBK * 2;                  // 16 KB
constexpr int kTmemCols = 512;                          // 512 / BN fp32 accumulators of 128 lanes x BN columns
// BN = 256: 48 KB stages x 4, two accumulators (compute-bound shapes).
// BN = 128: 32 KB stages x 6, four accumulators, for C no wider than 128 columns.
// A CTA of a pair holds half of the B slab: 32 KB stages x 6, two accumulators.
template <int BN, bool PAIR = false> struct TileCfg {
  static constexpr int kBRows = PAIR ? BN / 2 : BN;      // rows (N) of the B slab in THIS CTA's shared memory
  static constexpr int kBBytes = kBRows * kBK * 2;
  static constexpr int kStageBytes = kABytes + kBBytes;
  static constexpr int kStages = kStageBytes == 49152 ? 4 : 6;
  static constexpr int kAccs = kTmemCols / BN;
};
constexpr int kGemmThreads = 320;                       // TMA warp, MMA warp, 8 epilogue warps
constexpr int kGroupM = 16;                             // row-blocks per rasterisation group
constexpr uint64_t kWaitLimitNs = 2000000000ull;        // every mbarrier wait gives up after 2 s
constexpr int kEpiWarps = 8;
constexpr int kEpiStageBytes = 32 * 128;                // per epilogue warp: 32 rows x 64 16-bit outputs, TMA-store staging
constexpr int kRingBytes = 4 * (kABytes + 256 * kBK * 2);  // 4 x 48 KB = 6 x 32 KB
constexpr int kMaxStages = 8;                             // of 24 KB
constexpr size_t kGemmSmem = static_cast<size_t>(kRingBytes) + kEpiWarps * kEpiStageBytes + 1024 /*align*/ + 256 /*barriers*/;  // same for both tile shapes (6 x 32 KB = 4 x 48 KB)

// ------------------------------------------------------------------ PTX wrappers (mbarrier and timer helpers: tma_common.cuh)
// The same load issued by a CTA of a pair: the destination is this CTA's shared memory, the
// mbarrier (a shared::cluster address) may be the peer CTA's.
__device__ __forceinline__ void tma_load_3d_pair(uint32_t dst, const CUtensorMap* map, uint32_t bar_cluster, int c0, int c1, int c2) {
  asm volatile("cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(dst), "l"(map), "r"(bar_cluster), "r"(c0),
               "r"(c1), "r"(c2)
               : "memory");
}
// 4-D forms: the 64-wide blocks of an MN-major operand in one copy
__device__ __forceinline__ void tma_load_4d_pair(uint32_t dst, const CUtensorMap* map, uint32_t bar_cluster, int c0, int c1, int c2, int c3) {
  asm volatile("cp.async.bulk.tensor.4d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];" ::"r"(dst), "l"(map), "r"(bar_cluster), "r"(c0),
               "r"(c1), "r"(c2), "r"(c3)
               : "memory");
}
__device__ __forceinline__ void tma_load_4d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1, int c2, int c3) {
  asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];" ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(c2),
               "r"(c3)
               : "memory");
}
__device__ __forceinline__ uint32_t map_to_cta(uint32_t addr, uint32_t rank) { return map_to_cta_addr(addr, rank); }
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar_cluster) { asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar_cluster) : "memory"); }
__device__ __forceinline__ void cluster_sync_all() { cluster_barrier(); }

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_commit(uint32_t bar) { asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory"); }
__device__ __forceinline__ void tc_mma_f16(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// pair forms: the barrier address is a shared::cluster address (own or peer CTA)
__device__ __forceinline__ void tc_commit_pair(uint32_t bar_cluster) { asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar_cluster) : "memory"); }
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
  return p != 0;
}
__device__ __forceinline__ void tc_mma_f16_pair(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  const uint32_t z = 0u;  // no output lane is disabled
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, {%5, %5, %5, %5, %5, %5, %5, %5}, p;\n\t}" ::"r"(d_tmem),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(z)
      : "memory");
}
__device__ __forceinline__ void tc_ld_32x32(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]),
        "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tc_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// Shared-memory matrix descriptor (128-byte swizzle, sm_100 format): start address,
// leading-dimension byte offset and stride byte offset in 16-byte units, version 1.
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((addr >> 4) & 0x3fffu);
  d |= static_cast<uint64_t>((lbo_bytes >> 4) & 0x3fffu) << 16;
  d |= static_cast<uint64_t>((sbo_bytes >> 4) & 0x3fffu) << 32;
  d |= 1ull << 46;  // descriptor version for sm_100
  d |= 2ull << 61;  // SWIZZLE_128B
  return d;
}

struct GemmTcParams {
  int64_t M, N, K, batch;
  int64_t sbm, sbn;  // bias strides in elements (0 = broadcast)
  float alpha, beta;
  int a_mn_major, b_mn_major;  // 0: K contiguous in global memory, 1: M (resp. N) contiguous, 2: so and a multiple of 64 (see encode_operand)
  int is_bf16;
  int has_bias;
  int tma_store;    // 1 = C goes out through TMA tile stores (N % 8 == 0, aligned), 0 = plain stores
  int col_fastest;  // tile order: 1 = column-block fastest (write-bound shapes), 0 = grouped row-block fastest
  int split_slabs;  // 0, or K slabs per plane of fp32 operands split into three bf16 planes (see gemm_f32_split_dispatch)
  int range_slabs;  // fp32 results: 0, or slabs (per plane) per range of K; the ranges are what the kernel sees as batch entries
  const uint32_t* skip_if_set;  // when not NULL: the kernel returns at once if this device word is non-zero
  uint64_t wait_limit_ns;       // every mbarrier wait gives up after this long (kWaitLimitNs in ordinary calls)
  int withhold_first_slab;      // wait probe only: the producer never loads the first K slab of a CTA's first tile
  int group_m;                  // row-blocks per rasterisation group (see tile_coords)
  int bn;                       // pairs: columns of a tile, 256, 192 or 128 (see pair_tile_columns)
};

// Tile t of one batch entry -> (row-block, column-block): column-block fastest, or groups of
// kGroupM row-blocks with the row-block fastest inside a group.
__device__ __forceinline__ void tile_coords(int64_t rem, int64_t mt, int64_t nt, int& mb, int& nb, int col_fastest, int group_m = kGroupM) {
  if (col_fastest) {
    mb = static_cast<int>(rem / nt);
    nb = static_cast<int>(rem - static_cast<int64_t>(mb) * nt);
    return;
  }
  const int64_t per_group = static_cast<int64_t>(group_m) * nt;
  const int64_t g = rem / per_group, in_g = rem - g * per_group;
  const int64_t gm = (mt - g * group_m) < group_m ? (mt - g * group_m) : group_m;  // the last group may be short
  mb = static_cast<int>(g * group_m + in_g % gm);
  nb = static_cast<int>(in_g / gm);
}

// T: operand type in shared memory (bf16 / f16). TO: type of C and of the bias -- T itself,
// or float when the operands are the bf16 planes of split fp32 matrices.
template <typename T, int kBN, typename TO, bool kPair = false, bool kRows = false>
__global__ void __launch_bounds__(kGemmThreads, 1)
gemm_tcgen05_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, const __grid_constant__ CUtensorMap map_c, const TO* bias, TO* __restrict__ C, GemmTcParams p,
                    uint32_t* __restrict__ status) {
  using Cfg = TileCfg<kBN, kPair>;
  constexpr int kAccs = Cfg::kAccs;
  constexpr int kTileM = kPair ? 2 * kBM : kBM;  // rows of C one tile covers (both CTAs of a pair)
  static_assert(!kPair || kBN == 256, "CTA pairs work on 256 x 256 tiles");
  extern __shared__ unsigned char smem_raw[];
  // 1024-byte alignment: the 128B swizzle pattern repeats every 8 rows x 128 bytes
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  unsigned char* epi_stage = smem + kRingBytes;  // kEpiWarps x 4 KB, each 1024-byte aligned
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + kRingBytes + kEpiWarps * kEpiStageBytes);
  // barrier slots, S = kMaxStages: [0,S) full, [S,2S) empty, then one tmem_full and one tmem_empty per accumulator
  uint32_t* tmem_base_slot = reinterpret_cast<uint32_t*>(bars + 2 * kMaxStages + 2 * kAccs);
  volatile uint32_t* abort_flag = tmem_base_slot + 1;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t smem_base = smem_u32(smem);
  const uint32_t bar_base = smem_u32(bars);
  auto full_bar = [&](int s) { return bar_base + 8u * s; };
  auto empty_bar = [&](int s) { return bar_base + 8u * (kMaxStages + s); };
  auto tfull_bar = [&](int a) { return bar_base + 8u * (2 * kMaxStages + a); };
  auto tempty_bar = [&](int a) { return bar_base + 8u * (2 * kMaxStages + kAccs + a); };
  // a pair's stages are as large as its tile is wide, and there are as many as fit
  const int bn = kPair ? p.bn : kBN;
  const int b_rows = kPair ? bn / 2 : Cfg::kBRows;  // of the B slab, in this CTA's shared memory: one box, or as many boxes of 64 as cover them
  const uint32_t stage_bytes = kPair ? static_cast<uint32_t>(kABytes + (p.b_mn_major ? (b_rows + 63) / 64 * 64 : b_rows) * kBK * 2) : static_cast<uint32_t>(Cfg::kStageBytes);
  const int stages = kPair ? kRingBytes / static_cast<int>(stage_bytes) : Cfg::kStages;

  // pair: rank of this CTA in its 2-CTA cluster (0 = the CTA that issues the MMAs), and the
  // shared::cluster addresses of the even CTA's barriers that both CTAs signal
  const uint32_t cta_rank = kPair ? cluster_ctarank() : 0u;
  if (threadIdx.x == 64) {
    // the copy engine's descriptors are on their way while the barriers and the tensor memory are set up
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&map_a)) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&map_b)) : "memory");
    if (p.tma_store) asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&map_c)) : "memory");
  }
  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; ++s) {
      mbar_init(full_bar(s), 1);   // pair: only the even CTA's is used (its producer arms it for both CTAs' bytes)
      mbar_init(empty_bar(s), 1);  // one tcgen05.commit per use (pair: the even CTA commits to both CTAs')
    }
    for (int a = 0; a < kAccs; ++a) {
      mbar_init(tfull_bar(a), 1);
      mbar_init(tempty_bar(a), kPair ? 16 : 8);  // one arrival per epilogue warp (pair: of both CTAs, on the even CTA's)
    }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    if (kPair) {
      asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_base_slot)), "r"(kTmemCols) : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    } else {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_base_slot)), "r"(kTmemCols) : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
  }
  tc_fence_before();
  __syncthreads();
  if (kPair) cluster_sync_all();  // the peer's barriers exist before anything arrives on them
  tc_fence_after();
  const uint32_t tmem_base = *tmem_base_slot;
  after_grids_before();  // what is above needs nothing that an earlier kernel writes
  const TO* bias_w = waited(bias);
  const bool skip = p.skip_if_set && *p.skip_if_set != 0u;  // the same word for every thread of every CTA

  const int64_t mt = (p.M + kTileM - 1) / kTileM, nt = (p.N + bn - 1) / bn;
  const int64_t tiles = skip ? 0 : p.batch * mt * nt;
  const int64_t tile_first = kPair ? (blockIdx.x >> 1) : blockIdx.x, tile_step = kPair ? (gridDim.x >> 1) : gridDim.x;
  // Split operands: plane q of an operand occupies K coordinates [q * Kp, q * Kp + K) of its
  // tensor map, Kp = 64 * split_slabs. One slab of the product needs the six plane pairs
  // whose product is not below fp32 resolution: (0,0) (0,1) (1,0) (0,2) (1,1) (2,0).
  // They are walked pair by pair over all slabs (see the producer).
  const bool ranged = sizeof(TO) == 4 && p.range_slabs != 0;
  const int k_slabs = static_cast<int>((p.K + kBK - 1) / kBK), planes = p.split_slabs ? 6 : 1, num_kb_all = planes * k_slabs;
  // a range of K has the slabs [b * range_slabs, (b + 1) * range_slabs), the last one what is left
  auto slabs_of = [&](int64_t b) {
    const int left = k_slabs - static_cast<int>(b) * p.range_slabs;
    return left < p.range_slabs ? left : p.range_slabs;
  };

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int64_t t = tile_first; t < tiles && ok; t += tile_step) {
        const int64_t b = t / (mt * nt), rem = t - b * (mt * nt);
        int mb, nb;
        tile_coords(rem, mt, nt, mb, nb, p.col_fastest, p.group_m);
        // pair: this CTA's 128 rows of A and its half of the B slab's rows
        const int m0 = mb * kTileM + static_cast<int>(cta_rank) * kBM, n0 = nb * bn + static_cast<int>(cta_rank) * (kPair ? b_rows : 0);
        const int tile_slabs = ranged ? slabs_of(b) : k_slabs, slab0 = ranged ? static_cast<int>(b) * p.range_slabs : 0;
        const int num_kb = planes * tile_slabs;
        const int entry = ranged ? 0 : static_cast<int>(b);  // the planes are one batch entry whatever range is walked
        int slab = 0, pair4 = 0;  // split operands: slab of the range, plane pair (times 4)
        for (int kb = 0; kb < num_kb; ++kb) {
          if (!mbar_wait(empty_bar(stage), phase ^ 1u, abort_flag, p.wait_limit_ns)) { ok = false; break; }
          const uint32_t a_dst = smem_base + stage * stage_bytes, b_dst = a_dst + kABytes;
          if (!kPair && p.withhold_first_slab && t == blockIdx.x && kb == 0) {
            // wait probe: this stage is never armed and never filled, so the MMA warp's wait on
            // it must run into its limit; the producer carries on until it needs the stage back
            if (++stage == stages) { stage = 0; phase ^= 1u; }
            continue;
          }
          // pair: every copy of both CTAs completes on the even CTA's barrier, which its
          // producer arms for the bytes of both
          const uint32_t fbar = kPair ? map_to_cta(full_bar(stage), 0u) : full_bar(stage);
          if (!kPair) mbar_expect_tx(full_bar(stage), stage_bytes);
          else if (cta_rank == 0u) mbar_expect_tx(full_bar(stage), 2 * stage_bytes);
          auto load = [&](uint32_t dst, const CUtensorMap* map, int c0, int c1, int c2) {
            if (kPair) tma_load_3d_pair(dst, map, fbar, c0, c1, c2);
            else tma_load_3d(dst, map, fbar, c0, c1, c2);
          };
          auto load_blocks = [&](uint32_t dst, const CUtensorMap* map, int k, int block, int c2) {
            if (kPair) tma_load_4d_pair(dst, map, fbar, 0, k, block, c2);
            else tma_load_4d(dst, map, fbar, 0, k, block, c2);
          };
          int ka = (slab0 + kb) * kBK, kbb = ka;
          if (sizeof(TO) == 4 && p.split_slabs) {
            // pairs (2,0) (1,1) (0,2) (1,0) (0,1) over all slabs first, then (0,0): the tensor
            // core truncates when it adds into the accumulator, by half a unit in the last
            // place of the running sum on average, so the small products go in while the sum
            // is still small and only the K/16 steps of the leading product pay full price
            ka = (((0x001012 >> pair4) & 0xf) * p.split_slabs + slab0 + slab) * kBK;
            kbb = (((0x010210 >> pair4) & 0xf) * p.split_slabs + slab0 + slab) * kBK;
            if (++slab == tile_slabs) { slab = 0; pair4 += 4; }  // counted, not divided: one thread issues every copy
          }
          if (!p.a_mn_major) {
            load(a_dst, &map_a, ka, m0, entry);  // box [128 rows][64 k]
          } else if (p.a_mn_major == 2) {
            load_blocks(a_dst, &map_a, ka, m0 >> 6, entry);  // box [2][64 k][64 m]
          } else {
#pragma unroll
            for (int c = 0; c < kBM / 64; ++c) load(a_dst + c * 8192, &map_a, m0 + c * 64, ka, entry);  // box [64 k][64 m]
          }
          if (!p.b_mn_major) {
            load(b_dst, &map_b, kbb, n0, entry);  // box [b_rows rows][64 k]
          } else if (p.b_mn_major == 2) {
            load_blocks(b_dst, &map_b, kbb, n0 >> 6, entry);  // box [b_rows / 64][64 k][64 n]
          } else {
#pragma unroll
            for (int c = 0; c < Cfg::kBRows / 64; ++c)
              if (!kPair || c * 64 < b_rows) load(b_dst + c * 8192, &map_b, n0 + c * 64, kbb, entry);  // box [64 k][64 n]
          }
          if (++stage == stages) { stage = 0; phase ^= 1u; }
        }
      }
      if (kPair && ok) {
        // tail: the even CTA's commits arrive on THIS CTA's empty barriers from afar; wait for
        // the ones still outstanding so that none lands after this CTA's shared memory is gone
        for (int i = 0; i < stages && ok; ++i) {
          if (!mbar_wait(empty_bar(stage), phase ^ 1u, abort_flag, p.wait_limit_ns)) ok = false;
          if (++stage == stages) { stage = 0; phase ^= 1u; }
        }
      }
      if (!ok) {
        *abort_flag = 1;
        if (status) atomicOr(status, B200_DEV_WAIT_TIMEOUT);
      }
    }
    __syncwarp();  // lanes 1..31 rejoin lane 0 before the CTA-wide barrier below
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer
    if (cta_rank == 0u) {  // pair: the even CTA issues for both
      // instruction descriptor: fp32 accumulate, A/B format, majors, N >> 3, M >> 4
      const uint32_t fmt = p.is_bf16 ? 1u : 0u;
      const uint32_t idesc = (1u << 4) | (fmt << 7) | (fmt << 10) | (p.a_mn_major ? 1u << 15 : 0u) | (p.b_mn_major ? 1u << 16 : 0u) |
                             (static_cast<uint32_t>(bn >> 3) << 17) | (static_cast<uint32_t>(kTileM >> 4) << 24);
      // per-UMMA (K = 16) advance of the start address and the two byte offsets per layout
      const uint32_t a_adv = p.a_mn_major ? 2048u : 32u, b_adv = p.b_mn_major ? 2048u : 32u;
      const uint32_t a_lbo = p.a_mn_major ? 8192u : 16u, b_lbo = p.b_mn_major ? 8192u : 16u;
      const uint32_t empty0 = kPair ? map_to_cta(empty_bar(0), 0u) : 0u, empty1 = kPair ? map_to_cta(empty_bar(0), 1u) : 0u;
      // The whole warp walks the slabs and one elected lane issues: descriptors and addresses are then the same in
      // every lane, and the compiler works them out once per warp. With a single lane in the loop the issue took longer
      // than the tensor cores need for a tile of 192 or 128 columns (4096^3 in tiles of 128: 132 -> 114 us).
      auto warp_wait = [&](uint32_t bar, uint32_t parity) { return __all_sync(0xffffffffu, mbar_wait(bar, parity, abort_flag, p.wait_limit_ns)) != 0; };
      int stage = 0, acc = 0;
      uint32_t phase = 0, acc_phase = 0;
      bool ok = true;
      for (int64_t t = tile_first; t < tiles && ok; t += tile_step) {
        if (!warp_wait(tempty_bar(acc), acc_phase ^ 1u)) { ok = false; break; }
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + static_cast<uint32_t>(acc * kBN);
        const int num_kb = ranged ? planes * slabs_of(t / (mt * nt)) : num_kb_all;
        for (int kb = 0; kb < num_kb; ++kb) {
          if (!warp_wait(full_bar(stage), phase)) { ok = false; break; }
          tc_fence_after();
          const uint32_t a_addr = smem_base + stage * stage_bytes, b_addr = a_addr + kABytes;
          uint64_t da[kBK / 16], db[kBK / 16];
#pragma unroll
          for (int k = 0; k < kBK / 16; ++k) {
            da[k] = smem_desc(a_addr + k * a_adv, a_lbo, 1024u);
            db[k] = smem_desc(b_addr + k * b_adv, b_lbo, 1024u);
          }
          const uint32_t e0 = kPair ? empty0 + 8u * stage : empty_bar(stage), e1 = empty1 + 8u * stage;
          if (elect_one()) {
#pragma unroll
            for (int k = 0; k < kBK / 16; ++k) {
              if (kPair) tc_mma_f16_pair(d_tmem, da[k], db[k], idesc, (kb | k) != 0 ? 1u : 0u);
              else tc_mma_f16(d_tmem, da[k], db[k], idesc, (kb | k) != 0 ? 1u : 0u);
            }
            if (kPair) {
              tc_commit_pair(e0);
              tc_commit_pair(e1);
            } else {
              tc_commit(e0);
            }
          }
          __syncwarp();
          if (++stage == stages) { stage = 0; phase ^= 1u; }
        }
        if (!ok) break;
        // accumulator complete (pair: each CTA's epilogue waits on its own barrier)
        if (elect_one()) {
          if (kPair) {
            tc_commit_pair(map_to_cta(tfull_bar(acc), 0u));
            tc_commit_pair(map_to_cta(tfull_bar(acc), 1u));
          } else {
            tc_commit(tfull_bar(acc));
          }
        }
        __syncwarp();
        if (++acc == kAccs) { acc = 0; acc_phase ^= 1u; }
      }
      if (!ok && lane == 0) {
        *abort_flag = 1;
        if (status) atomicOr(status, B200_DEV_WAIT_TIMEOUT);
      }
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------ epilogue (warps 2..9)
    const int q = warp & 3;             // TMEM lane quarter this warp may read: lanes [32q, 32q + 32)
    const int chalf = (warp - 2) >> 2;  // which 128 of the 256 columns
    int acc = 0;
    uint32_t acc_phase = 0;
    bool ok = true;
    constexpr int kOutVec = 16 / static_cast<int>(sizeof(TO));  // outputs per 16-byte store
    const bool vec_ok = (p.N % kOutVec == 0) && ((reinterpret_cast<uintptr_t>(C) & 15u) == 0);
    const uint32_t tempty_target = kPair ? map_to_cta(tempty_bar(0), 0u) : 0u;  // the even CTA's tmem_empty[0]
    for (int64_t t = tile_first; t < tiles && ok; t += tile_step) {
      const int64_t b = t / (mt * nt), rem = t - b * (mt * nt);
      int mb, nb_blk;
      tile_coords(rem, mt, nt, mb, nb_blk, p.col_fastest, p.group_m);
      const int64_t m0 = static_cast<int64_t>(mb) * kTileM + static_cast<int64_t>(cta_rank) * kBM, n0 = static_cast<int64_t>(nb_blk) * bn + chalf * (kBN / 2);
      const int64_t tile_end = static_cast<int64_t>(nb_blk + 1) * bn, n_end = tile_end < p.N ? tile_end : p.N;  // (a chunk of 64 columns lies in the tile or behind it)
      int got = 0;
      if (lane == 0) got = mbar_wait(tfull_bar(acc), acc_phase, abort_flag, p.wait_limit_ns) ? 1 : 0;
      got = __shfl_sync(0xffffffffu, got, 0);
      if (!got) { ok = false; break; }
      tc_fence_after();
      const int64_t m = m0 + q * 32 + lane;
      const uint32_t t_base = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + static_cast<uint32_t>(acc * kBN + chalf * (kBN / 2));
      // the 64-column chunks of this warp's half are double-buffered in registers: the
      // tensor-memory load of the next chunk is in flight while this one is converted and stored
      constexpr int kChunks = kBN / 2 / 64;
      uint32_t r[kChunks > 1 ? 2 : 1][64];
      tc_ld_32x32(t_base, r[0]);
      tc_ld_32x32(t_base + 32, r[0] + 32);
      const bool plain = p.alpha == 1.f && !p.has_bias;  // C = A x B: nothing to do but round
      const bool unit_scales = p.alpha == 1.f && p.beta == 1.f;
      const bool bias_vec = sizeof(TO) == sizeof(T) && p.has_bias && p.sbn == 1 && p.sbm % 8 == 0 && (reinterpret_cast<uintptr_t>(bias) & 15u) == 0;
      // a lane's 64 values of columns nb.. of its row: scaled, bias added in fp32, where they are (apart from
      // the rounding, so that a product without either runs through none of this code)
      auto scale = [&](uint32_t* rc, int64_t nb) {
#pragma unroll
        for (int g = 0; g < 8; ++g) {
          const int64_t n = nb + g * 8;
          if (bias_vec && m < p.M && n + 8 <= p.N) {
            // unit-stride bias (a row vector, or a matrix like C): eight values in one load
            float bv[8];
            widen<T>(ld_keep_after(bias_w + m * p.sbm + n), bv);  // TO is T on this path
            if (unit_scales) {  // addmm as models call it: one add per value
#pragma unroll
              for (int e = 0; e < 8; ++e) rc[g * 8 + e] = __float_as_uint(__uint_as_float(rc[g * 8 + e]) + bv[e]);
            } else {
#pragma unroll
              for (int e = 0; e < 8; ++e) rc[g * 8 + e] = __float_as_uint(fmaf(p.beta, bv[e], p.alpha * __uint_as_float(rc[g * 8 + e])));
            }
          } else {
#pragma unroll
            for (int e = 0; e < 8; ++e) {
              float v = p.alpha * __uint_as_float(rc[g * 8 + e]);
              if (p.has_bias && m < p.M && n + e < p.N) v = fmaf(p.beta, to_f32(bias[m * p.sbm + (n + e) * p.sbn]), v);
              rc[g * 8 + e] = __float_as_uint(v);
            }
          }
        }
      };
      // rounded once, into the 128-byte-swizzle layout of `mine`
      auto park = [&](const uint32_t* rc, unsigned char* mine) {
#pragma unroll
        for (int g = 0; g < 8; ++g) {
          float v[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) v[e] = __uint_as_float(rc[g * 8 + e]);
          *reinterpret_cast<uint4*>(mine + lane * 128 + ((g ^ (lane & 7)) << 4)) = narrow<T>(v);
        }
      };
#pragma unroll
      for (int c = 0; c < kChunks; ++c) {
        tc_ld_wait();
        if (c + 1 < kChunks) {
          tc_ld_32x32(t_base + (c + 1) * 64, r[(c + 1) & 1]);
          tc_ld_32x32(t_base + (c + 1) * 64 + 32, r[(c + 1) & 1] + 32);
        } else {
          // every value of the accumulator is in registers: hand it back to the MMA warp now
          tc_fence_before();
          __syncwarp();
          if (lane == 0) {
            if (kPair) mbar_arrive_cluster(tempty_target + 8u * acc);
            else mbar_arrive(tempty_bar(acc));
          }
        }
        uint32_t* rc = r[c & 1];
        const int64_t nb = n0 + c * 64;
        if constexpr (sizeof(TO) == 2) {
          if (!plain) scale(rc, nb);
        }
        if (p.tma_store) {
          // scale / bias in fp32, round once, park the lane's 64 outputs of its row in this
          // warp's 32 x 128-byte buffer in the 128-byte-swizzle layout (16-byte chunk index
          // XOR row) -- conflict-free to write and exactly what a SWIZZLE_128B tiled store
          // reads -- then one lane hands the 32 x 64 tile to the copy engine, which writes
          // whole lines and clips at the edges of C.
          unsigned char* mine = epi_stage + (warp - 2) * kEpiStageBytes;
          if (lane == 0) tma_store_wait_read();  // the previous tile store has finished reading the buffer
          __syncwarp();
          park(rc, mine);
          fence_async_smem();
          __syncwarp();
          if (lane == 0 && nb < n_end && m0 + q * 32 < p.M) {
            tma_store_3d(&map_c, smem_u32(mine), static_cast<int>(nb), static_cast<int>(m0 + q * 32), static_cast<int>(b));
            tma_store_commit();
          }
        } else if constexpr (sizeof(TO) == 2) {
          // 16-bit C whose rows are off the 16-byte grid (N not a multiple of 8): a lane owns a
          // row, so storing from registers would put every lane of a store in another row, one
          // 32-byte sector per 2-byte element. Park the chunk in the warp's buffer as above and
          // write it out row by row, two elements to a lane; where a row starts between two 4-byte words
          // a lane's pair is its second element and its neighbour's first, and the row's first element goes out alone.
          // Element by element, with a row's address and the bias worked out for each, a tile took
          // 12 us more than through the copy engine: bf16 4096 x 4098 x 512 75 -> 30 us (4096 wide 20), 2537 x 3709 x 920 61 -> 35.
          unsigned char* mine = epi_stage + (warp - 2) * kEpiStageBytes;
          __syncwarp();  // the previous chunk has been read out of the buffer
          park(rc, mine);
          __syncwarp();
          const int64_t left = n_end - nb, mr0 = m0 + q * 32;
          const int ncols = left < 64 ? static_cast<int>(left) : 64;  // <= 0: the chunk lies right of C
          const int nrows = p.M - mr0 < 32 ? static_cast<int>(p.M - mr0) : 32;
          if (ncols > 0) {
            unsigned short* crow = reinterpret_cast<unsigned short*>(C + (b * p.M + mr0) * p.N + nb);
            const uint32_t mine_a = smem_u32(mine) + static_cast<uint32_t>(lane & 3) * 4;
#pragma unroll 1
            for (int r0 = 0; r0 < nrows; r0 += 8) {
              uint32_t w[8];  // columns 2 lane, 2 lane + 1 of eight rows
#pragma unroll
              for (int u = 0; u < 8; ++u) asm volatile("ld.shared.u32 %0, [%1];" : "=r"(w[u]) : "r"(mine_a + (r0 + u) * 128 + (((lane >> 2) ^ u) << 4)) : "memory");
#pragma unroll
              for (int u = 0; u < 8; ++u, crow += p.N) {
                const uint32_t odd = static_cast<uint32_t>(reinterpret_cast<uintptr_t>(crow) >> 1) & 1u;
                const uint32_t after = __shfl_down_sync(0xffffffffu, w[u], 1), pair = __byte_perm(w[u], after, odd ? 0x5432 : 0x3210);
                const int e0 = 2 * lane + static_cast<int>(odd), end = r0 + u < nrows ? ncols : 0;
                if (e0 + 1 < end) *reinterpret_cast<uint32_t*>(crow + e0) = pair;
                if (e0 + 1 == end) crow[e0] = static_cast<unsigned short>(pair);
                if (odd && lane == 0 && end) crow[0] = static_cast<unsigned short>(w[u]);
              }
            }
          }
        } else if constexpr (!kRows) {
          // fp32 C, a lane to a row: 16 bytes at a time where the rows are on the grid. (Going through the
          // buffer as below costs more than the wider stores give back: 8192 x 256 x 2048 91 us against 72.)
          if (m < p.M && nb < n_end) {
            TO* crow = C + (b * p.M + m) * p.N;
#pragma unroll
            for (int g = 0; g < 8; ++g) {
              const int64_t n = nb + g * 8;
              float v[8];
#pragma unroll
              for (int e = 0; e < 8; ++e) {
                v[e] = p.alpha * __uint_as_float(rc[g * 8 + e]);
                if (p.has_bias && n + e < p.N) v[e] = fmaf(p.beta, to_f32(bias[m * p.sbm + (n + e) * p.sbn]), v[e]);
              }
              if (vec_ok && n + 8 <= p.N) {
#pragma unroll
                for (int h = 0; h < 8 / kOutVec; ++h) *reinterpret_cast<uint4*>(crow + n + h * kOutVec) = narrow<TO>(v + h * kOutVec);
              } else {
#pragma unroll
                for (int e = 0; e < 8; ++e)
                  if (n + e < p.N) crow[n + e] = from_f32<TO>(v[e]);
              }
            }
          }
        } else {
          // fp32 C off the grid (kRows): the same parking, 32 columns at a time, written out row by row, 128
          // contiguous bytes per store; the bias is looked up there, where a row and a column are all
          // that is live. Stores straight from the registers put every lane in another row, a
          // sector per 4-byte element (1531 x 2050 x 1027 in fp32: 65.6 -> 59.6 us; eight rows on the way together 57.5).
          unsigned char* mine = epi_stage + (warp - 2) * kEpiStageBytes;
          const int64_t mr0 = m0 + q * 32;
          const int nrows = p.M - mr0 < 32 ? static_cast<int>(p.M - mr0) : 32;
          const bool row_bias = p.has_bias && p.sbm == 0;
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int64_t n = nb + h * 32 + lane;
            __syncwarp();  // the columns before have been read out of the buffer
#pragma unroll
            for (int g = 0; g < 8; ++g) {
              float v[4];
#pragma unroll
              for (int e = 0; e < 4; ++e) v[e] = p.alpha * __uint_as_float(rc[h * 32 + g * 4 + e]);
              *reinterpret_cast<uint4*>(mine + lane * 128 + ((g ^ (lane & 7)) << 4)) = narrow<float>(v);
            }
            __syncwarp();
            const float same = row_bias && n < p.N ? to_f32(bias[n * p.sbn]) : 0.f;  // a bias vector: one look for all rows
            TO* c = C + (b * p.M + mr0) * p.N + n;
            const uint32_t mine_a = smem_u32(mine) + static_cast<uint32_t>(lane & 3) * 4;
#pragma unroll 1
            for (int r0 = 0; r0 < nrows; r0 += 8) {
              float v[8];
#pragma unroll
              for (int u = 0; u < 8; ++u) asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v[u]) : "r"(mine_a + (r0 + u) * 128 + (((lane >> 2) ^ u) << 4)) : "memory");
#pragma unroll
              for (int u = 0; u < 8; ++u, c += p.N) {
                if (n < n_end && r0 + u < nrows) {
                  if (p.has_bias && !row_bias) v[u] = fmaf(p.beta, to_f32(bias[(mr0 + r0 + u) * p.sbm + n * p.sbn]), v[u]);
                  *c = from_f32<TO>(row_bias ? fmaf(p.beta, same, v[u]) : v[u]);
                }
              }
            }
          }
        }
      }
      if (++acc == kAccs) { acc = 0; acc_phase ^= 1u; }
    }
    if (lane == 0) tma_store_wait_read();  // the tile stores have read their shared memory: the CTA may exit (the writes complete on their own)
    if (!ok && lane == 0) {
      *abort_flag = 1;
      if (status) atomicOr(status, B200_DEV_WAIT_TIMEOUT);
    }
    __syncwarp();
  }

  // ---------------------------------------------------------------- teardown
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (*abort_flag) {
    // give copies that are still in flight time to land before the shared memory goes away
    for (int i = 0; i < 64; ++i) __nanosleep(1000);
    __syncthreads();
  }
  if (kPair) cluster_sync_all();  // neither CTA leaves while the other may still signal its barriers or read its operands
  if (warp == 1) {
    if (kPair) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kTmemCols) : "memory");
    else asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kTmemCols) : "memory");
  }
}

// ------------------------------------------------------------------ host side
struct OperandLayout {
  bool ok, mn_major;
};
// An operand [rows(MN), K] with element strides (s_mn, s_k) is TMA-loadable when one of
// the two strides is 1 and the other (and the batch stride) keeps 16-byte alignment.
static OperandLayout operand_layout(int64_t mn, int64_t k, int64_t s_mn, int64_t s_k, int64_t s_b, int64_t batch, const void* base) {
  OperandLayout r{false, false};
  if (!aligned16(base)) return r;
  if (batch > 1 && (s_b % 8 != 0 || s_b <= 0)) return r;
  if (s_k == 1 && (s_mn % 8 == 0) && s_mn >= k) { r.ok = true; r.mn_major = false; return r; }
  if (s_mn == 1 && (s_k % 8 == 0) && s_k >= mn) { r.ok = true; r.mn_major = true; return r; }
  // a single row / column is contiguous either way
  if (mn == 1 && s_k == 1) { r.ok = true; r.mn_major = false; return r; }
  return r;
}

int gemm_simt_dispatch(const void* A, const void* B, const void* bias, void* C, int64_t batch, int64_t M, int64_t N, int64_t K, int64_t sAb, int64_t sAm, int64_t sAk,
                       int64_t sBb, int64_t sBk, int64_t sBn, int64_t sbm, int64_t sbn, double alpha, double beta, int dtype, cudaStream_t st, const uint32_t* gate);

bool gemm_tc_eligible(int64_t batch, int64_t M, int64_t N, int64_t K, int64_t sAb, int64_t sAm, int64_t sAk, int64_t sBb, int64_t sBk, int64_t sBn, int dtype, const void* A,
                      const void* B, const void* C) {
  if (dtype != B200_BF16 && dtype != B200_F16) return false;
  if (batch < 1 || M < 1 || N < 1 || K < 1) return false;
  if (M > 0x7fffffffLL || N > 0x7fffffffLL || K > 0x7fffffffLL || batch > 0x7fffffffLL) return false;
  // tiny problems are launch-bound either way; the CUDA-core kernel has no TMEM / barrier set-up
  if (M * N * K < (1LL << 15)) return false;
  if (!operand_layout(M, K, sAm, sAk, sAb, batch, A).ok) return false;
  if (!operand_layout(N, K, sBn, sBk, sBb, batch, B).ok) return false;
  if (!C) return false;
  return encode_fn() != nullptr;
}

// An MN-major operand arrives as blocks of 64 columns. Where its columns are a multiple of 64 they are a dimension of
// their own (the map ends where the operand does), and a tile's blocks, two or four copies otherwise, are one: a single thread issues them, and
// with both operands MN-major that is what a slab waits for.
static bool in_blocks(bool mn_major, int64_t mn, int tile_mn) { return mn_major && mn % 64 == 0 && tile_mn % 64 == 0; }
static int mn_form(bool mn_major, int64_t mn, int tile_mn) { return mn_major ? (in_blocks(mn_major, mn, tile_mn) ? 2 : 1) : 0; }
static bool encode_operand(CUtensorMap* map, const void* base, int dtype, bool mn_major, int64_t mn, int64_t k, int64_t s_mn, int64_t s_k, int64_t s_b, int64_t batch, int tile_mn) {
  const cuuint64_t inner = mn_major ? mn : k, outer = mn_major ? k : mn;
  int64_t outer_stride = mn_major ? s_k : s_mn;  // elements
  if (outer == 1 && outer_stride % 8 != 0) outer_stride = (static_cast<int64_t>(inner) + 7) / 8 * 8;  // never dereferenced beyond row 0
  int64_t batch_stride = batch > 1 ? s_b : outer_stride * static_cast<int64_t>(outer);
  if (batch_stride % 8 != 0 || batch_stride <= 0) batch_stride = (batch_stride / 8 + 1) * 8;
  const CUtensorMapDataType dt = dtype == B200_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
  if (in_blocks(mn_major, mn, tile_mn)) {  // [batch][mn / 64][k][64]: the blocks of a tile in one copy
    cuuint64_t dims[4] = {64, outer, inner / 64, static_cast<cuuint64_t>(batch)};
    cuuint64_t strides[3] = {static_cast<cuuint64_t>(outer_stride) * 2, 128, static_cast<cuuint64_t>(batch_stride) * 2};
    cuuint32_t box[4] = {64, kBK, static_cast<cuuint32_t>(tile_mn / 64), 1};
    cuuint32_t estr[4] = {1, 1, 1, 1};
    return encode_fn()(map, dt, 4, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                       CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
  }
  cuuint64_t dims[3] = {inner, outer, static_cast<cuuint64_t>(batch)};
  cuuint64_t strides[2] = {static_cast<cuuint64_t>(outer_stride) * 2, static_cast<cuuint64_t>(batch_stride) * 2};
  cuuint32_t box[3] = {64, static_cast<cuuint32_t>(mn_major ? kBK : tile_mn), 1};
  cuuint32_t estr[3] = {1, 1, 1};
  const CUresult r = encode_fn()(map, dt, 3, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                                 CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS;
}

// Rows of C per rasterisation group: the CTAs that run together walk the column blocks of one
// group of row blocks, so the group's A panel (rows x K 16-bit values) stays in L2 while B
// streams past it once per group. The panel is sized to a fraction of the 126 MB L2; fewer
// groups mean fewer passes over B (at 8192 x 4096 x 11008 groups of 2048 rows read B four
// times: 441 MB of DRAM reads for 157 MB of operands).
#ifndef B200_GEMM_PANEL_MB
#define B200_GEMM_PANEL_MB 32
#endif
static int group_rows_for(int64_t k_elems) {
  int64_t rows = (static_cast<int64_t>(B200_GEMM_PANEL_MB) << 20) / (2 * (k_elems > 0 ? k_elems : 1));
  rows = rows / 256 * 256;
  if (rows < 2048) rows = 2048;    // never smaller than the groups the kernel always used
  if (rows > 65536) rows = 65536;
  return static_cast<int>(rows);
}

// One launch of the kernel: a plain grid, or 2-CTA clusters for the pair variant.
template <typename Kernel, typename TB, typename TC>
static int launch_tc(Kernel kernel, bool pair, int grid, cudaStream_t st, const CUtensorMap& map_a, const CUtensorMap& map_b, const CUtensorMap& map_c, const TB* bias_t, TC* c_t,
                     const GemmTcParams& p, uint32_t* status) {
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kGemmSmem));
  if (e != cudaSuccess) { set_last_cuda_error(e); return B200_ELAUNCH; }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(grid), 1, 1);
  cfg.blockDim = dim3(kGemmThreads, 1, 1);
  cfg.dynamicSmemBytes = kGemmSmem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;  // (see launch_after)
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = 2;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pair ? 2 : 1;
  const cudaError_t le = cudaLaunchKernelEx(&cfg, kernel, map_a, map_b, map_c, bias_t, c_t, p, status);
  if (le != cudaSuccess) { set_last_cuda_error(le); return B200_ELAUNCH; }
  return B200_OK;
}

// CTA pairs can be switched off with B200_GEMM_PAIR=0 in the environment (read once): the
// single-CTA kernel then serves every shape, which is how the two are compared.
static bool pair_launch_ok() {
  static const bool on = []() {
    const char* e = getenv("B200_GEMM_PAIR");
    return !(e && e[0] == '0');
  }();
  return on;
}

// Columns of a pair's tile: 256, or 192 or 128 where tiles of 256 are few rounds and leave pairs without one in the last. A
// round of narrower tiles takes 0.83 or 0.69 of the time (with B along N, whose boxes are 64 columns wide, 192 columns
// take as long as 256, and 128 0.73):
// their rows of A are loaded and their slabs handed on all the same (4096^3 in tiles of 256, 192 and 128: 4, 5
// and 7 rounds in 94, 97 and 114 us). Another width is taken where it saves a twentieth: bf16 2537 x 920 x 3712 24.7 -> 20.7
// us, 1024^3 12.2 -> 10.5; fp32 1531 x 2050 x 1027 53.6 -> 48.7.
static double tile_time(int bn, bool b_mn) { return bn == 256 ? 1.0 : bn == 192 ? (b_mn ? 1.0 : 0.83) : (b_mn ? 0.73 : 0.69); }
static int64_t pair_tiles(int64_t M, int64_t N, int bn) { return ((M + 2 * kBM - 1) / (2 * kBM)) * ((N + bn - 1) / bn); }
static double pair_rounds(int64_t entries, int64_t M, int64_t N, int bn, bool b_mn) {
  const int64_t slots = kNumSMs / 2;
  return static_cast<double>((entries * pair_tiles(M, N, bn) + slots - 1) / slots) * tile_time(bn, b_mn);
}
static int pair_tile_columns(int64_t batch, int64_t M, int64_t N, bool b_mn) {
  int best = 256;
  double least = pair_rounds(batch, M, N, 256, b_mn);
  if (least > 4.0) return best;
  least *= 0.95;
  for (int bn : {192, 128}) {
    const double t = pair_rounds(batch, M, N, bn, b_mn);
    if (t < least) { least = t; best = bn; }
  }
  return best;
}

int gemm_tc_dispatch(const void* A, const void* B, const void* bias, void* C, int64_t batch, int64_t M, int64_t N, int64_t K, int64_t sAb, int64_t sAm, int64_t sAk, int64_t sBb,
                     int64_t sBk, int64_t sBn, int64_t sbm, int64_t sbn, double alpha, double beta, int dtype, uint32_t* status, cudaStream_t st, uint64_t wait_probe_limit_ns,
                     bool allow_pair) {
  const OperandLayout la = operand_layout(M, K, sAm, sAk, sAb, batch, A);
  const OperandLayout lb = operand_layout(N, K, sBn, sBk, sBb, batch, B);
  if (!la.ok || !lb.ok || !encode_fn()) return B200_EALIGN;
  alignas(64) CUtensorMap map_a, map_b;
  if (!encode_operand(&map_a, A, dtype, la.mn_major, M, K, sAm, sAk, sAb, batch, kBM)) return B200_EDRIVER;
  // CTA pairs on 256 x 256 tiles whenever C has more than one 128-row block and is not narrow;
  // the wait probe stays on the single-CTA kernel
  // (with four K slabs or fewer the kernel is bound by writing C and the pair is slower:
  // bmm 32 x 2048 x 128 x 2048 0.087 ms against 0.061 ms)
  const bool pair = allow_pair && M > kBM && N > 128 && (K + kBK - 1) / kBK > 4 && wait_probe_limit_ns == 0 && pair_launch_ok();
  const bool narrow = N <= 128;
  const int bn = pair ? pair_tile_columns(batch, M, N, lb.mn_major) : narrow ? 128 : 256;
  const int bn_box = pair ? bn / 2 : bn;  // rows of the B box: a CTA of a pair loads half of them
  if (!encode_operand(&map_b, B, dtype, lb.mn_major, N, K, sBn, sBk, sBb, batch, bn_box)) return B200_EDRIVER;
  alignas(64) CUtensorMap map_c;
  const bool tma_store = (N % 8 == 0) && aligned16(C);
  if (tma_store) {
    cuuint64_t dims[3] = {static_cast<cuuint64_t>(N), static_cast<cuuint64_t>(M), static_cast<cuuint64_t>(batch)};
    cuuint64_t strides[2] = {static_cast<cuuint64_t>(N) * 2, static_cast<cuuint64_t>(M) * static_cast<cuuint64_t>(N) * 2};
    cuuint32_t box[3] = {64, 32, 1};
    cuuint32_t estr[3] = {1, 1, 1};
    const CUtensorMapDataType dt = dtype == B200_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
    if (encode_fn()(&map_c, dt, 3, C, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return B200_EDRIVER;
  } else {
    map_c = map_a;  // unused by the kernel in this mode
  }
  GemmTcParams p;
  p.tma_store = tma_store ? 1 : 0;
  p.M = M; p.N = N; p.K = K; p.batch = batch;
  p.sbm = sbm; p.sbn = sbn;
  p.alpha = static_cast<float>(alpha);
  p.beta = static_cast<float>(beta);
  p.a_mn_major = mn_form(la.mn_major, M, kBM);
  p.b_mn_major = mn_form(lb.mn_major, N, bn_box);
  p.is_bf16 = dtype == B200_BF16 ? 1 : 0;
  p.has_bias = (bias != nullptr && p.beta != 0.f) ? 1 : 0;
  // few K slabs per tile: the kernel is bound by writing C, so CTAs that run together should
  // write neighbouring column blocks of the same rows (whole DRAM pages); otherwise order
  // tiles for operand reuse in L2
  p.col_fastest = (K + kBK - 1) / kBK <= 4 ? 1 : 0;
  p.split_slabs = 0;
  p.range_slabs = 0;
  p.skip_if_set = nullptr;
  p.wait_limit_ns = wait_probe_limit_ns ? wait_probe_limit_ns : kWaitLimitNs;
  p.withhold_first_slab = wait_probe_limit_ns ? 1 : 0;
  p.group_m = group_rows_for(K) / (pair ? 2 * kBM : kBM);
  p.bn = bn;
  // a narrow C takes the 128-wide tile. (Write-bound shapes with few K slabs were measured
  // slower on it: 256-byte row segments instead of 512-byte ones cost more in DRAM than the
  // deeper pipeline gains -- bmm 32x2048x128x2048: 0.162 ms vs 0.116 ms.)
  const int tile_m = pair ? 2 * kBM : kBM;
  const int64_t tiles = batch * ((M + tile_m - 1) / tile_m) * ((N + bn - 1) / bn);
  const int64_t slots = pair ? kNumSMs / 2 : kNumSMs;  // persistent: one CTA (or CTA pair) per SM (or TPC)
  const int grid = static_cast<int>(tiles < slots ? tiles : slots) * (pair ? 2 : 1);
  auto launch = [&](auto kernel, auto* bias_t, auto* c_t) -> int { return launch_tc(kernel, pair, grid, st, map_a, map_b, map_c, bias_t, c_t, p, status); };
  int rc;
  if (dtype == B200_BF16) {
    const __nv_bfloat16* bt = static_cast<const __nv_bfloat16*>(bias);
    __nv_bfloat16* ct = static_cast<__nv_bfloat16*>(C);
    rc = pair ? launch(gemm_tcgen05_kernel<__nv_bfloat16, 256, __nv_bfloat16, true>, bt, ct)
              : narrow ? launch(gemm_tcgen05_kernel<__nv_bfloat16, 128, __nv_bfloat16>, bt, ct) : launch(gemm_tcgen05_kernel<__nv_bfloat16, 256, __nv_bfloat16>, bt, ct);
  } else {
    const __half* bt = static_cast<const __half*>(bias);
    __half* ct = static_cast<__half*>(C);
    rc = pair ? launch(gemm_tcgen05_kernel<__half, 256, __half, true>, bt, ct)
              : narrow ? launch(gemm_tcgen05_kernel<__half, 128, __half>, bt, ct) : launch(gemm_tcgen05_kernel<__half, 256, __half>, bt, ct);
  }
  if (rc == B200_ELAUNCH && pair) {
    // the cluster launch was refused (a device or a partition without thread-block clusters):
    // the same product on single CTAs
    (void)cudaGetLastError();
    return gemm_tc_dispatch(A, B, bias, C, batch, M, N, K, sAb, sAm, sAk, sBb, sBk, sBn, sbm, sbn, alpha, beta, dtype, status, st, wait_probe_limit_ns, false);
  }
  if (rc) return rc;
  return check_launch();
}

// ------------------------------------------------------------------ long contraction, few output tiles
// A 16-bit product whose C is a handful of tiles leaves most SMs idle while one CTA per tile
// walks all of K (5 x 4096 x 512: two CTAs, 64 K slabs each, 26 us). Here the contraction is
// cut into S ranges of whole slabs that the kernel above sees as S batch entries and writes as
// fp32 partial products [S][M][N] into caller scratch; a second kernel adds the S partials of
// every element in the order 0 .. S-1, applies alpha, beta and the bias and rounds once. No
// atomics: the result does not depend on scheduling. The ranges need not be equal, so any K can be cut (in
// equal ones on the 16-byte grid a K of 7221 could not: f16 17 x 152 x 7221 78 -> 35 us, 61 x 64 x 3966 35 -> 22, most of what is left moving the operands onto the 16-byte grid).
struct SplitKPlan {
  int splits;       // 1 = not worth it
  int range_slabs;  // K slabs per range; the last one has what is left
};
static SplitKPlan plan_splitk(int64_t batch, int64_t M, int64_t N, int64_t K) {
  SplitKPlan r{1, 0};
  if (batch != 1) return r;
  const int bn = N <= 128 ? 128 : 256;
  const int64_t tiles = ((M + kBM - 1) / kBM) * ((N + bn - 1) / bn), slabs = (K + kBK - 1) / kBK;
  // (more tiles than a quarter of the SMs: 5722 x 4096 x 256, 45 tiles, ran 30 us in two ranges against 26 us whole)
  if (tiles > kNumSMs / 4 || slabs < 24) return r;  // (16 slabs: 104 x 1024 x 1024 took 12 us either way)
  int64_t s = kNumSMs / tiles;
  if (s > slabs / 4) s = slabs / 4;  // every range keeps at least four K slabs
  if (s > 32) s = 32;
  if (s < 2) return r;
  r.range_slabs = static_cast<int>((slabs + s - 1) / s);
  r.splits = static_cast<int>((slabs + r.range_slabs - 1) / r.range_slabs);
  return r;
}

int64_t gemm_tc_splitk_scratch_bytes(int64_t batch, int64_t M, int64_t N, int64_t K) {
  const SplitKPlan pl = plan_splitk(batch, M, N, K);
  return pl.splits < 2 ? 0 : static_cast<int64_t>(pl.splits) * M * N * 4 + 256;
}

// The sum over the ranges. U elements per thread, the partial sums of all of them in flight
// together: four where that leaves every SM eight CTAs' worth of elements (1531 x 1027 in 3 ranges
// 12.3 -> 4.7 us), one below, where fewer and busier threads only wait longer, and of a small result B
// ranges at a time (20000 deep, 40 x 128 outputs: the call 12.7 us, 16 with eight in flight).
template <typename T, int U, int B>
__global__ void __launch_bounds__(256) splitk_reduce(const float* part, int splits, int64_t M, int64_t N, const T* bias, int64_t sbm, int64_t sbn, float alpha, float beta,
                                                     T* __restrict__ C, const uint32_t* skip_if_set) {
  after_grids_before();
  const float* part_w = waited(part);
  if (skip_if_set && *skip_if_set != 0u) return;  // the partial products were not computed either
  const int64_t total = M * N;
  for (int64_t i0 = static_cast<int64_t>(blockIdx.x) * (256 * U) + threadIdx.x; i0 < total; i0 += static_cast<int64_t>(gridDim.x) * (256 * U)) {
    float sum[U];
#pragma unroll
    for (int u = 0; u < U; ++u) sum[u] = 0.f;
    if constexpr (B > 1) {
      for (int s = 0; s < splits; s += B) {  // past the last one nothing is added
        float v[B];
#pragma unroll
        for (int k = 0; k < B; ++k) v[k] = s + k < splits ? part[(s + k) * total + i0] : 0.f;
#pragma unroll
        for (int k = 0; k < B; ++k) sum[0] += v[k];
      }
    } else if constexpr (U == 1) {
      for (int s = 0; s < splits; ++s) sum[0] += part[s * total + i0];
    } else {
#pragma unroll 4
      for (int s = 0; s < splits; ++s) {
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (i0 + u * 256 < total) sum[u] += ld_stream_after_f(part_w + s * total + i0 + u * 256);
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int64_t i = i0 + u * 256;
      if (i >= total) break;
      float r = alpha * sum[u];
      if (bias && beta != 0.f) {
        const int64_t m = i / N, n = i - m * N;
        r = fmaf(beta, to_f32(bias[m * sbm + n * sbn]), r);
      }
      C[i] = from_f32<T>(r);
    }
  }
}

template <typename T>
static cudaError_t launch_splitk_reduce(const float* part, int splits, int64_t M, int64_t N, const void* bias, int64_t sbm, int64_t sbn, float alpha, float beta, void* C, const uint32_t* skip_if_set,
                                 cudaStream_t st) {
  const int64_t total = M * N, cap = kNumSMs * 8;
  const bool wide = total >= cap * 1024;
  int64_t blocks = wide ? (total + 1023) / 1024 : (total + 255) / 256;
  if (blocks > cap) blocks = cap;
  auto go = [&](auto kernel) { return launch_after(kernel, blocks, 256, 0, st, part, splits, M, N, static_cast<const T*>(bias), sbm, sbn, alpha, beta, static_cast<T*>(C), skip_if_set); };
  return wide ? go(splitk_reduce<T, 4, 1>) : total >= 1 << 16 ? go(splitk_reduce<T, 1, 1>) : go(splitk_reduce<T, 1, 16>);
}

int gemm_tc_splitk_dispatch(const void* A, const void* B, const void* bias, void* C, int64_t M, int64_t N, int64_t K, int64_t sAm, int64_t sAk, int64_t sBk, int64_t sBn, int64_t sbm,
                            int64_t sbn, double alpha, double beta, int dtype, void* scratch, int64_t scratch_bytes, uint32_t* status, cudaStream_t st) {
  const SplitKPlan pl = plan_splitk(1, M, N, K);
  if (pl.splits < 2) return B200_EINVAL;
  if (!scratch || scratch_bytes < gemm_tc_splitk_scratch_bytes(1, M, N, K)) return B200_ESCRATCH;
  float* part = reinterpret_cast<float*>((reinterpret_cast<uintptr_t>(scratch) + 255) & ~static_cast<uintptr_t>(255));
  const int64_t S = pl.splits;
  const OperandLayout la = operand_layout(M, K, sAm, sAk, 0, 1, A);
  const OperandLayout lb = operand_layout(N, K, sBn, sBk, 0, 1, B);
  if (!la.ok || !lb.ok || !encode_fn()) return B200_EALIGN;
  const int bn = N <= 128 ? 128 : 256;
  alignas(64) CUtensorMap map_a, map_b;
  if (!encode_operand(&map_a, A, dtype, la.mn_major, M, K, sAm, sAk, 0, 1, kBM)) return B200_EDRIVER;
  if (!encode_operand(&map_b, B, dtype, lb.mn_major, N, K, sBn, sBk, 0, 1, bn)) return B200_EDRIVER;
  GemmTcParams p;
  p.tma_store = 0;
  p.M = M; p.N = N; p.K = K; p.batch = S;
  p.sbm = 0; p.sbn = 0;
  p.alpha = 1.f;
  p.beta = 0.f;
  p.a_mn_major = mn_form(la.mn_major, M, kBM);
  p.b_mn_major = mn_form(lb.mn_major, N, bn);
  p.is_bf16 = dtype == B200_BF16 ? 1 : 0;
  p.has_bias = 0;
  p.col_fastest = 1;
  p.split_slabs = 0;
  p.range_slabs = pl.range_slabs;
  p.skip_if_set = nullptr;
  p.wait_limit_ns = kWaitLimitNs;
  p.withhold_first_slab = 0;
  p.group_m = group_rows_for(K) / kBM;
  p.bn = bn;
  const int64_t tiles = S * ((M + kBM - 1) / kBM) * ((N + bn - 1) / bn);
  const int grid = static_cast<int>(tiles < kNumSMs ? tiles : kNumSMs);
  auto launch = [&](auto kernel) -> int { return launch_tc(kernel, false, grid, st, map_a, map_b, map_a, static_cast<const float*>(nullptr), part, p, status); };
  int rc;
  auto launch_as = [&](auto as_rows) -> int {  // (rows of partial sums off the 16-byte grid: bf16 256 x 250 x 4096 27 -> 12 us)
    constexpr bool kRows = decltype(as_rows)::value;
    if (dtype == B200_BF16) return bn == 128 ? launch(gemm_tcgen05_kernel<__nv_bfloat16, 128, float, false, kRows>) : launch(gemm_tcgen05_kernel<__nv_bfloat16, 256, float, false, kRows>);
    return bn == 128 ? launch(gemm_tcgen05_kernel<__half, 128, float, false, kRows>) : launch(gemm_tcgen05_kernel<__half, 256, float, false, kRows>);
  };
  rc = N >= 32 && N % 4 != 0 ? launch_as(std::true_type{}) : launch_as(std::false_type{});
  if (rc) return rc;
  const float al = static_cast<float>(alpha), be = static_cast<float>(beta);
  const cudaError_t re = dtype == B200_BF16 ? launch_splitk_reduce<__nv_bfloat16>(part, static_cast<int>(S), M, N, bias, sbm, sbn, al, be, C, nullptr, st)
                                            : launch_splitk_reduce<__half>(part, static_cast<int>(S), M, N, bias, sbm, sbn, al, be, C, nullptr, st);
  if (re != cudaSuccess) { set_last_cuda_error(re); return B200_ELAUNCH; }
  return check_launch(2);
}

// ------------------------------------------------------------------ fp32 operands on the tensor cores
// An fp32 value is the sum of three bf16 values to within 2^-25 of itself (x1 = bf16(x),
// x2 = bf16(x - x1), x3 = bf16(x - x1 - x2); the subtractions are exact). A product of fp32
// matrices is therefore, to fp32 accuracy, the sum of the six bf16 products
// A1B1 + A1B2 + A2B1 + A1B3 + A2B2 + A3B1 (the three left out are below 2^-25 relative) --
// every one exact in the tensor core's fp32 accumulator. The kernel above runs them as one
// contraction of depth 6 K: the operands are split once into planes laid side by side along
// K, and the producer warp walks the six plane pairs of every K slab.
//
// split_f32_planes: x [batch, mn, k] (any strides) -> bf16 planes. K-major form (src K
// stride 1, or neither stride 1): out[b][mn][q * Kp + k]; MN-major form (src MN stride 1):
// out[b][q * Kp + k][mn]. Kp = K rounded up to 64; the pad [K, Kp) is written as zero.
// Infinities and NaN stay in plane 0 alone (x - x1 would be NaN); a value whose bf16
// rounding overflows is truncated instead. An infinity still meets the residual planes of
// the other operand, whose signs are arbitrary (inf - inf = NaN where fp32 arithmetic gives
// inf), so the split raises a device flag when it meets a non-finite value: the tensor-core
// kernel returns at once when the flag is up and the CUDA-core kernel, launched behind it
// and gated the other way, computes that product in plain fp32.
struct SplitArgs {
  const float* x;
  const float* end;              // behind the last element of x
  __nv_bfloat16* out;
  int64_t batch, mn, k, kp;
  int64_t s_b, s_mn, s_k;        // source strides, elements
  int64_t o_b, o_row;            // output batch stride and row pitch, elements
  int mn_major;                  // output form
  uint32_t* any_flag;            // set when the operand holds an infinity or a NaN
};
__device__ __forceinline__ float4 ld_f4(const float* p) { return __ldg(reinterpret_cast<const float4*>(p)); }
__device__ __forceinline__ void split3(float x, __nv_bfloat16& a, __nv_bfloat16& b, __nv_bfloat16& c) {
  if (!isfinite(x)) { a = __float2bfloat16_rn(x); b = c = __float2bfloat16_rn(0.f); return; }
  float x1 = __bfloat162float(__float2bfloat16_rn(x));
  if (!isfinite(x1)) x1 = __uint_as_float(__float_as_uint(x) & 0xffff0000u);
  const float r1 = x - x1;
  const float x2 = __bfloat162float(__float2bfloat16_rn(r1));
  const float r2 = r1 - x2;
  a = __float2bfloat16_rn(x1);
  b = __float2bfloat16_rn(x2);
  c = __float2bfloat16_rn(r2);
}
// Both operands in one launch: the first `blocks0` CTAs take the one, the others the other. A thread produces 8
// consecutive elements along the contiguous dimension of the output (k in the K-major form, mn in the MN-major form) with
// three 16-byte stores. Where the source is contiguous there it is read 16 bytes at a time: two loads, or, for
// rows that start off the grid, three around the eight elements, which are then moved up by as many as
// the row is off. (Element by element a warp's load touched 32 sectors: 1531 x 1027 and 2050 x 1027
// together 12 -> 8 us.)
__global__ void __launch_bounds__(256) split_f32_planes(const __grid_constant__ SplitArgs A0, const __grid_constant__ SplitArgs A1, unsigned blocks0) {
  next_grid_may_start();  // (the product's CTAs set themselves up meanwhile)
  const bool second = blockIdx.x >= blocks0;
  const SplitArgs& A = second ? A1 : A0;
  const int64_t block = second ? blockIdx.x - blocks0 : blockIdx.x, nblocks = second ? gridDim.x - blocks0 : blocks0;
  const int64_t inner = A.mn_major ? A.mn : A.kp, outer = A.mn_major ? A.kp : A.mn;
  const int64_t groups = (inner + 7) / 8;  // kp is a multiple of 8; a ragged mn tail is a partial group
  const int64_t per_batch = groups * outer;
  const int64_t total = A.batch * per_batch;
  const int64_t s_in = A.mn_major ? A.s_mn : A.s_k, s_out = A.mn_major ? A.s_k : A.s_mn;  // source strides along inner / outer
  const int64_t lim_in = A.mn_major ? A.mn : A.k, lim_out = A.mn_major ? A.k : A.mn;      // where real data ends
  for (int64_t i = block * 256 + threadIdx.x; i < total; i += nblocks * 256) {
    int64_t b, o, g;
    if (total <= 0x7fffffffLL) {
      const uint32_t q = static_cast<uint32_t>(i) / static_cast<uint32_t>(groups), qb = A.batch == 1 ? 0u : q / static_cast<uint32_t>(outer);
      g = static_cast<uint32_t>(i) - q * static_cast<uint32_t>(groups);
      o = q - qb * static_cast<uint32_t>(outer);
      b = qb;
    } else {
      b = i / per_batch;
      const int64_t r = i - b * per_batch;
      o = r / groups;
      g = r - o * groups;
    }
    const int64_t in0 = g * 8;
    float v[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) v[e] = 0.f;
    if (o < lim_out) {
      const float* src = A.x + b * A.s_b + o * s_out + in0 * s_in;
      const int off = static_cast<int>(reinterpret_cast<uintptr_t>(src) >> 2) & 3;
      const float* p = src - off;
      if (s_in == 1 && in0 + 8 <= lim_in && p >= A.x && p + 12 <= A.end) {
        const float4 lo = ld_f4(p), mid = ld_f4(p + 4);
        float4 hi = make_float4(0.f, 0.f, 0.f, 0.f);
        if (off) hi = ld_f4(p + 8);
        float w[11] = {lo.x, lo.y, lo.z, lo.w, mid.x, mid.y, mid.z, mid.w, hi.x, hi.y, hi.z};
        if (off & 1) {
#pragma unroll
          for (int e = 0; e < 10; ++e) w[e] = w[e + 1];
        }
        if (off & 2) {
#pragma unroll
          for (int e = 0; e < 8; ++e) w[e] = w[e + 2];
        }
#pragma unroll
        for (int e = 0; e < 8; ++e) v[e] = w[e];
      } else {
#pragma unroll
        for (int e = 0; e < 8; ++e)
          if (in0 + e < lim_in) v[e] = src[e * s_in];
      }
    }
    __nv_bfloat16 q0[8], q1[8], q2[8];
    bool bad = false;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      split3(v[e], q0[e], q1[e], q2[e]);
      bad |= !isfinite(v[e]);
    }
    if (bad) *A.any_flag = 1u;
    // o_row is a multiple of 8 and so are in0 and kp: every store below is 16-byte aligned
    __nv_bfloat16* ob = A.out + b * A.o_b;
    const int64_t plane = A.mn_major ? A.kp * A.o_row : A.kp;
    __nv_bfloat16* to = ob + o * A.o_row + in0;
    *reinterpret_cast<uint4*>(to) = *reinterpret_cast<const uint4*>(q0);
    *reinterpret_cast<uint4*>(to + plane) = *reinterpret_cast<const uint4*>(q1);
    *reinterpret_cast<uint4*>(to + 2 * plane) = *reinterpret_cast<const uint4*>(q2);
  }
}

static inline int64_t round_up(int64_t v, int64_t m) { return (v + m - 1) / m * m; }

// Width of the tiles, and ranges of K for a product with fewer tiles than CTA pairs. What the product takes is the rounds of
// tiles a pair walks times the time of a tile times the slabs of a range (a slab, six plane pairs of 256 columns, takes about
// 2.4 us), and writing and adding up the ranges' fp32 sums, 8 bytes per range and element of C at
// about 5 TB/s; the cut that makes the sum least is taken where it saves an eighth or more. fp32
// 1531 x 1027 x 2050 (30 tiles on 74 pairs) 99 -> 66 us, 2050 x 1027 x 1531 (45 tiles) 81 -> 74 us.
// Shorter chains of truncating additions make the result more exact, not less.
struct F32Plan {
  int ranges, bn;
};
static F32Plan plan_f32(int64_t batch, int64_t M, int64_t N, int64_t K, bool b_mn) {
  if (M <= kBM || N <= 128 || !pair_launch_ok()) return F32Plan{1, N <= 128 ? 128 : 256};
  const int64_t slabs = (K + kBK - 1) / kBK;
  F32Plan best{1, pair_tile_columns(batch, M, N, b_mn)};
  if (batch != 1 || pair_tiles(M, N, 256) >= kNumSMs / 2) return best;
  const double sums = static_cast<double>(M) * static_cast<double>(N) * 8 / 14e6;  // slabs' worth of time per range
  double least = pair_rounds(1, M, N, best.bn, b_mn) * static_cast<double>(slabs) * 0.875;
  for (int bn : {256, 192, 128}) {
    for (int64_t s = 2; s <= 8 && slabs / s >= 4; ++s) {
      const int64_t per = (slabs + s - 1) / s, n = (slabs + per - 1) / per;
      const double cost = pair_rounds(n, M, N, bn, b_mn) * static_cast<double>(per) + sums * static_cast<double>(n);
      if (cost < least) { least = cost; best = F32Plan{static_cast<int>(n), bn}; }
    }
  }
  return best;
}

int64_t gemm_f32_split_scratch_bytes(int64_t batch, int64_t M, int64_t N, int64_t K) {
  const int64_t kp = round_up(K, kBK);
  const int along_k = plan_f32(batch, M, N, K, false).ranges, along_n = plan_f32(batch, M, N, K, true).ranges, ranges = along_k > along_n ? along_k : along_n;
  return batch * 3 * kp * (round_up(M, 64) + round_up(N, 64)) * 2 + 256 + 512 + (ranges > 1 ? ranges * M * N * 4 : 0);
}

bool gemm_f32_split_eligible(int64_t batch, int64_t M, int64_t N, int64_t K) {
  if (batch < 1 || M < 1 || N < 1 || K < 1) return false;
  if (M > 0x7fffffffLL || N > 0x7fffffffLL || 3 * round_up(K, kBK) > 0x7fffffffLL || batch > 0x7fffffffLL) return false;
  return encode_fn() != nullptr;
}

int gemm_f32_split_dispatch(const void* A, const void* B, const void* bias, void* C, int64_t batch, int64_t M, int64_t N, int64_t K, int64_t sAb, int64_t sAm, int64_t sAk, int64_t sBb,
                            int64_t sBk, int64_t sBn, int64_t sbm, int64_t sbn, double alpha, double beta, void* scratch, int64_t scratch_bytes, uint32_t* status, cudaStream_t st) {
  if (!gemm_f32_split_eligible(batch, M, N, K)) return B200_EINVAL;
  if (!scratch || scratch_bytes < gemm_f32_split_scratch_bytes(batch, M, N, K)) return B200_ESCRATCH;
  const int64_t kp = round_up(K, kBK);
  // scratch: [flag word, padded to 256 bytes] [planes of A] [planes of B]
  unsigned char* flags = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(scratch) + 255) & ~static_cast<uintptr_t>(255));
  const int64_t flag_bytes = 256;
  uint32_t* any_flag = reinterpret_cast<uint32_t*>(flags);
  const cudaError_t me = cudaMemsetAsync(flags, 0, 4, st);
  if (me != cudaSuccess) { set_last_cuda_error(me); return B200_ELAUNCH; }
  auto* pa = reinterpret_cast<__nv_bfloat16*>(flags + flag_bytes);
  const bool a_mn = sAm == 1 && sAk != 1 && M > 1, b_mn = sBn == 1 && sBk != 1 && N > 1;  // keep the contiguous dimension of each source
  // (MN-major planes have whole blocks of 64 columns, see encode_operand; what lies behind an operand's last column
  // belongs to rows or columns that C does not have)
  const int64_t a_row = a_mn ? round_up(M, 64) : 3 * kp, a_rows = a_mn ? 3 * kp : M;
  const int64_t b_row = b_mn ? round_up(N, 64) : 3 * kp, b_rows = b_mn ? 3 * kp : N;
  __nv_bfloat16* pb = pa + batch * a_rows * a_row;  // a multiple of 8 elements: stays 16-byte aligned
  const float* fa = static_cast<const float*>(A);
  const float* fb = static_cast<const float*>(B);
  const SplitArgs sa{fa, fa + (batch - 1) * sAb + (M - 1) * sAm + (K - 1) * sAk + 1, pa, batch, M, K, kp, sAb, sAm, sAk, a_rows * a_row, a_row, a_mn ? 1 : 0, any_flag};
  const SplitArgs sb{fb, fb + (batch - 1) * sBb + (N - 1) * sBn + (K - 1) * sBk + 1, pb, batch, N, K, kp, sBb, sBn, sBk, b_rows * b_row, b_row, b_mn ? 1 : 0, any_flag};
  auto blocks = [](int64_t n) { const int64_t b = (n + 255) / 256; return static_cast<int>(b < 1 ? 1 : (b > kNumSMs * 32LL ? kNumSMs * 32LL : b)); };
  const int blocks_a = blocks(batch * a_rows * a_row / 24), blocks_b = blocks(batch * b_rows * b_row / 24);
  split_f32_planes<<<blocks_a + blocks_b, 256, 0, st>>>(sa, sb, static_cast<unsigned>(blocks_a));
  const cudaError_t se = cudaGetLastError();
  if (se != cudaSuccess) { set_last_cuda_error(se); return B200_ELAUNCH; }

  // the planes as [rows, 3 Kp] (K-major) or [3 Kp, rows] (MN-major) bf16 operands
  alignas(64) CUtensorMap map_a, map_b;
  const bool pair = M > kBM && N > 128 && pair_launch_ok();  // the contraction is six planes deep: never write-bound
  const F32Plan plan = plan_f32(batch, M, N, K, b_mn);
  const int bn = plan.bn;
  if (!encode_operand(&map_a, pa, B200_BF16, a_mn, a_mn ? a_row : M, 3 * kp, a_mn ? 1 : a_row, a_mn ? a_row : 1, a_rows * a_row, batch, kBM)) return B200_EDRIVER;
  if (!encode_operand(&map_b, pb, B200_BF16, b_mn, b_mn ? b_row : N, 3 * kp, b_mn ? 1 : b_row, b_mn ? b_row : 1, b_rows * b_row, batch, pair ? bn / 2 : bn)) return B200_EDRIVER;
  GemmTcParams p;
  p.tma_store = 0;
  p.M = M; p.N = N; p.K = K; p.batch = batch;
  p.sbm = sbm; p.sbn = sbn;
  p.alpha = static_cast<float>(alpha);
  p.beta = static_cast<float>(beta);
  p.a_mn_major = mn_form(a_mn, a_row, kBM);
  p.b_mn_major = mn_form(b_mn, b_row, pair ? bn / 2 : bn);
  p.is_bf16 = 1;
  p.has_bias = (bias != nullptr && p.beta != 0.f) ? 1 : 0;
  p.split_slabs = static_cast<int>(kp / kBK);
  // fp32 partial products [ranges][M][N] behind the planes, added in the order of the ranges
  const int ranges = plan.ranges;
  float* part = reinterpret_cast<float*>(pb + batch * b_rows * b_row);
  p.range_slabs = ranges > 1 ? (p.split_slabs + ranges - 1) / ranges : 0;
  if (ranges > 1) {
    p.batch = ranges;
    p.alpha = 1.f;
    p.has_bias = 0;
  }
  p.skip_if_set = any_flag;
  p.wait_limit_ns = kWaitLimitNs;
  p.withhold_first_slab = 0;
  p.col_fastest = 6 * p.split_slabs <= 4 ? 1 : 0;
  p.group_m = group_rows_for(3 * kp) / (pair ? 2 * kBM : kBM);
  p.bn = bn;
  const int tile_m = pair ? 2 * kBM : kBM;
  const int64_t tiles = p.batch * ((M + tile_m - 1) / tile_m) * ((N + bn - 1) / bn);
  const int64_t slots = pair ? kNumSMs / 2 : kNumSMs;
  const int grid = static_cast<int>(tiles < slots ? tiles : slots) * (pair ? 2 : 1);
  auto launch = [&](auto kernel) -> int { return launch_tc(kernel, pair, grid, st, map_a, map_b, map_a, static_cast<const float*>(bias), ranges > 1 ? part : static_cast<float*>(C), p, status); };
  // rows of C off the 16-byte grid go out through the staging buffer (a handful of columns does not pay for it)
  const bool rows = N >= 32 && (N % 4 != 0 || (ranges == 1 && !aligned16(C)));
  auto launch_as = [&](auto as_rows) -> int {
    constexpr bool kRows = decltype(as_rows)::value;
    return pair ? launch(gemm_tcgen05_kernel<__nv_bfloat16, 256, float, true, kRows>)
                : bn == 128 ? launch(gemm_tcgen05_kernel<__nv_bfloat16, 128, float, false, kRows>) : launch(gemm_tcgen05_kernel<__nv_bfloat16, 256, float, false, kRows>);
  };
  const int rc = rows ? launch_as(std::true_type{}) : launch_as(std::false_type{});
  if (rc) return rc;
  if (ranges > 1) {
    const cudaError_t re = launch_splitk_reduce<float>(part, ranges, M, N, bias, sbm, sbn, static_cast<float>(alpha), static_cast<float>(beta), C, any_flag, st);
    if (re != cudaSuccess) { set_last_cuda_error(re); return B200_ELAUNCH; }
  }
  // the same product on the CUDA cores, run only when the split met an infinity or a NaN
  const int rs = gemm_simt_dispatch(A, B, bias, C, batch, M, N, K, sAb, sAm, sAk, sBb, sBk, sBn, sbm, sbn, alpha, beta, B200_F32, st, any_flag);
  if (rs) return rs;
  return check_launch(ranges > 1 ? 3 : 2);
}

}  // namespace b200
