// mm / addmm / bmm with few outputs and a long contraction, on the CUDA cores.
#include <cooperative_groups.h>

#include "b200_common.cuh"

namespace cg = cooperative_groups;

namespace b200 {

bool gemm_small_path_on();

namespace {

constexpr int kDeepWarps = 8;
constexpr int kDeepStep = 32;  // k per step of a warp: one to a lane where A (or a K-fast B) is read

struct DeepArgs {
  int64_t M, N, K;
  int64_t sAb, sAm, sAk, sBb, sBk, sBn, sbm, sbn;
  float alpha, beta;
  const uint32_t* gate;  // when not NULL: the kernel does its work only if this device word is non-zero
  int ksplit;            // CTAs per cluster sharing one output tile
  int64_t kwarp;         // k per warp, a multiple of kDeepStep
};

template <typename T, int RM, int NC, bool KFAST> struct DeepShape {
  static constexpr bool kAsync = KFAST && sizeof(T) == 4;  // copied into shared memory a step ahead
  static constexpr int kStage = kDeepStep * (RM + 4) + (KFAST ? 32 * NC * (kDeepStep + 1) : 0);  // floats of a warp's step
  static constexpr int kStages = kDeepWarps * kStage * (kAsync ? 2 : 1);
  static constexpr int kParts = (kDeepWarps + 1) * RM * 32 * NC;
  static constexpr int kFloats = kStages > kParts ? kStages : kParts;
  static constexpr int kPerSM = (kAsync ? NC > 1 : RM * NC > 16 && !KFAST) ? 1 : 2;
};

// 4 bytes from global to shared memory in the background, zero where not `valid`
__device__ __forceinline__ void copy4(float* dst, const void* src, bool valid) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(dst))), "l"(src), "r"(valid ? 4 : 0) : "memory");
}

// RM rows by 32 * NC columns of C per CTA, a lane to NC columns. What bounds such a product is the chain of global reads,
// so K is cut once per warp: ksplit CTAs of a cluster x 8 warps walk a range each, 32 k of A and B per step and all of a step's
// loads requested before the first is used. A goes through a few hundred bytes of shared memory that only its warp touches (read
// back as broadcasts); B is used from the registers it arrived in where a row of it is contiguous, else (KFAST) it is read
// along K and turned in shared memory. The partial tiles are added in the order of the ranges: warps, then CTAs.
// (The tile kernel of gemm_simt.cu gives a slice of 16 k to 256 threads at a time, 0.9 us each: 4 x 4104 x 128 fp32 34.5 us there, 6.6 here;
// the error against 64 bits is half: 4.0e-7 of the norm and 1.7e-7, the chains being shorter. fp32 along K copied into shared memory
// a step ahead, not through registers: 8 x 4096 x 32000 188 us, 267. 16 rows by 64 columns want 135 to 168 registers: at two CTAs
// to an SM they spill, 8 of 11 x 1024 x 1024 25 us against 14.)
template <typename T, int RM, int NC, bool KFAST>
__global__ void __launch_bounds__(32 * kDeepWarps, DeepShape<T, RM, NC, KFAST>::kPerSM) gemm_deep(const T* __restrict__ A, const T* __restrict__ B, const T* __restrict__ bias, T* __restrict__ C, DeepArgs g) {
  extern __shared__ __align__(16) float smem[];
  constexpr int W = 32 * NC, kPitch = RM + 4;
  constexpr bool kAsync = DeepShape<T, RM, NC, KFAST>::kAsync;
  if (g.gate && *g.gate == 0u) return;  // the same word for every CTA: whole clusters leave together
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t n0 = static_cast<int64_t>(blockIdx.x) * W, m0 = static_cast<int64_t>(blockIdx.y) * RM;
  const int64_t b = blockIdx.z / g.ksplit;
  const int rank = static_cast<int>(blockIdx.z % g.ksplit);
  const int64_t k_lo = (static_cast<int64_t>(rank) * kDeepWarps + warp) * g.kwarp;
  const int64_t k_hi = k_lo + g.kwarp < g.K ? k_lo + g.kwarp : g.K;
  const T* Ab = A + b * g.sAb + m0 * g.sAm;
  const T* Bb = B + b * g.sBb;
  float* as = smem + warp * (DeepShape<T, RM, NC, KFAST>::kStage * (kAsync ? 2 : 1));
  const int rows = g.M - m0 < RM ? static_cast<int>(g.M - m0) : RM;
  const int64_t cols = g.N - n0 < W ? g.N - n0 : W;
  float acc[RM][NC];
#pragma unroll
  for (int i = 0; i < RM; ++i)
#pragma unroll
    for (int j = 0; j < NC; ++j) acc[i][j] = 0.f;
  // fp32 along K: the copies of a step, into one of two stages (no pointer moves past the last row or column)
  auto request = [&](int64_t k0, float* st) {
    const bool live = k0 + lane < k_hi;
    const T* pa = Ab + (live ? k0 + lane : 0) * g.sAk;
    const T* pb = Bb + n0 * g.sBn + (live ? k0 + lane : 0) * g.sBk;
#pragma unroll
    for (int i = 0; i < RM; ++i, pa += i < rows ? g.sAm : 0) copy4(st + lane * kPitch + i, pa, live && i < rows);
#pragma unroll 8
    for (int q = 0; q < W; ++q, pb += q < cols ? g.sBn : 0) copy4(st + kDeepStep * kPitch + q * (kDeepStep + 1) + lane, pb, live && q < cols);
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  float* next = as + DeepShape<T, RM, NC, KFAST>::kStage;
  if (kAsync && k_lo < k_hi) request(k_lo, as);
  for (int64_t k0 = k_lo; k0 < k_hi; k0 += kDeepStep) {
    const float* bs = as + kDeepStep * kPitch;
    T rb[KFAST ? 1 : kDeepStep][NC];
    if constexpr (kAsync) {
      if (k0 + kDeepStep < k_hi) {
        request(k0 + kDeepStep, next);
        asm volatile("cp.async.wait_group 1;" ::: "memory");
      } else {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
      }
    } else {
      const int kn = k_hi - k0 < kDeepStep ? static_cast<int>(k_hi - k0) : kDeepStep;
      const T zero = from_f32<T>(0.f);
      T ra[RM];
      const T* pa = Ab + (k0 + lane) * g.sAk;
#pragma unroll
      for (int i = 0; i < RM; ++i, pa += g.sAm) ra[i] = (i < rows && lane < kn) ? *pa : zero;
      if constexpr (!KFAST) {
        const T* pb = Bb + k0 * g.sBk + n0 + lane;
#pragma unroll
        for (int q = 0; q < kDeepStep; ++q, pb += g.sBk)
#pragma unroll
          for (int j = 0; j < NC; ++j) rb[q][j] = (j * 32 + lane < cols && q < kn) ? pb[j * 32] : zero;
      }
      __syncwarp();  // the step before has been read
      if constexpr (KFAST) {
        const T* pb = Bb + n0 * g.sBn + (k0 + lane) * g.sBk;
#pragma unroll
        for (int j = 0; j < NC; ++j) {
          T r[32];
#pragma unroll
          for (int q = 0; q < 32; ++q, pb += g.sBn) r[q] = (j * 32 + q < cols && lane < kn) ? *pb : zero;
#pragma unroll
          for (int q = 0; q < 32; ++q) as[kDeepStep * kPitch + (j * 32 + q) * (kDeepStep + 1) + lane] = to_f32(r[q]);
        }
      }
#pragma unroll
      for (int i = 0; i < RM; i += 4) *reinterpret_cast<float4*>(as + lane * kPitch + i) = make_float4(to_f32(ra[i]), to_f32(ra[i + 1]), to_f32(ra[i + 2]), to_f32(ra[i + 3]));
    }
    __syncwarp();
#pragma unroll
    for (int q = 0; q < kDeepStep; ++q) {
      float a[RM], bb[NC];
#pragma unroll
      for (int i = 0; i < RM; i += 4) *reinterpret_cast<float4*>(a + i) = *reinterpret_cast<const float4*>(as + q * kPitch + i);
#pragma unroll
      for (int j = 0; j < NC; ++j) bb[j] = KFAST ? bs[(j * 32 + lane) * (kDeepStep + 1) + q] : to_f32(rb[KFAST ? 0 : q][j]);
#pragma unroll
      for (int i = 0; i < RM; ++i)
#pragma unroll
        for (int j = 0; j < NC; ++j) acc[i][j] = fmaf(a[i], bb[j], acc[i][j]);
    }
    if constexpr (kAsync) {
      __syncwarp();  // read before it is filled again
      float* t = as;
      as = next;
      next = t;
    }
  }
  __syncthreads();  // every warp is done with its stage: the partial tiles take its place
#pragma unroll
  for (int i = 0; i < RM; ++i)
#pragma unroll
    for (int j = 0; j < NC; ++j) smem[(warp * RM + i) * W + j * 32 + lane] = acc[i][j];
  __syncthreads();
  float* sums = smem + kDeepWarps * RM * W;
  for (int e = threadIdx.x; e < RM * W; e += 32 * kDeepWarps) {
    float s = 0.f;
#pragma unroll
    for (int w = 0; w < kDeepWarps; ++w) s += smem[w * RM * W + e];
    sums[e] = s;
  }
  cg::cluster_group cluster = cg::this_cluster();
  cluster.sync();  // (a cluster of one: the CTA's barrier)
  T* Cb = C + b * g.M * g.N;
  for (int e = rank * 32 * kDeepWarps + threadIdx.x; e < RM * W; e += g.ksplit * 32 * kDeepWarps) {
    const int i = e / W, n = e % W;
    if (i >= rows || n >= cols) continue;
    float s = 0.f;
    for (int r = 0; r < g.ksplit; ++r) s += cluster.map_shared_rank(sums, r)[e];
    float r = g.alpha * s;
    // beta == 0 drops the bias term entirely (a NaN bias must not leak through)
    if (bias && g.beta != 0.f) r = fmaf(g.beta, to_f32(bias[(m0 + i) * g.sbm + (n0 + n) * g.sbn]), r);
    Cb[(m0 + i) * g.N + n0 + n] = from_f32<T>(r);
  }
  cluster.sync();  // nobody leaves while its sums may still be read
}

// How many CTAs share a tile: the number with the fewest steps one after the other, over all waves of clusters, two more
// to each wave for its start and its sums. The clusters that run at once (one CTA to an SM; as the occupancy query gives them):
// eight CTAs have to lie within one GPC, which leaves SMs over.
int deep_split(int64_t tiles, int64_t K, int per_sm) {
  constexpr int kClusters[9] = {0, 148, 74, 45, 33, 26, 22, 15, 15};
  int best = 1;
  int64_t least = 0;
  for (int s = 1; s <= 8; ++s) {
    const int64_t steps = (K + s * kDeepWarps * kDeepStep - 1) / (s * kDeepWarps * kDeepStep);
    const int64_t waves = (tiles + kClusters[s] * per_sm - 1) / (kClusters[s] * per_sm);
    const int64_t cost = waves * (steps + 2);
    if (s == 1 || cost < least) { least = cost; best = s; }
    if (steps == 1) break;
  }
  return best;
}

template <typename T, int RM, int NC, bool KFAST>
int launch_deep(const T* A, const T* B, const T* bias, T* C, int64_t batch, DeepArgs g, cudaStream_t st) {
  constexpr int smem = DeepShape<T, RM, NC, KFAST>::kFloats * 4;
  if (smem > 48 * 1024) {
    const cudaError_t ae = cudaFuncSetAttribute(gemm_deep<T, RM, NC, KFAST>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (ae != cudaSuccess) { set_last_cuda_error(ae); return B200_ELAUNCH; }
  }
  const int64_t gx = (g.N + 32 * NC - 1) / (32 * NC), gy = (g.M + RM - 1) / RM;
  const int64_t tiles = batch * gx * gy;
  const int split = deep_split(tiles, g.K, DeepShape<T, RM, NC, KFAST>::kPerSM);
  const int64_t per = (g.K + split * kDeepWarps - 1) / (split * kDeepWarps);
  g.ksplit = split;
  g.kwarp = (per + kDeepStep - 1) / kDeepStep * kDeepStep;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(gx), static_cast<unsigned>(gy), static_cast<unsigned>(batch * split));
  cfg.blockDim = dim3(32 * kDeepWarps);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 1;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = static_cast<unsigned>(split);
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, gemm_deep<T, RM, NC, KFAST>, A, B, bias, C, g);
  if (e != cudaSuccess) { set_last_cuda_error(e); return B200_ELAUNCH; }
  return check_launch();
}

template <typename T, int RM>
int launch_deep_rows(const T* A, const T* B, const T* bias, T* C, int64_t batch, const DeepArgs& g, cudaStream_t st) {
  const bool narrow = g.N <= 32;
  if (g.sBn == 1) return narrow ? launch_deep<T, RM, 1, false>(A, B, bias, C, batch, g, st) : launch_deep<T, RM, 2, false>(A, B, bias, C, batch, g, st);
  return narrow ? launch_deep<T, RM, 1, true>(A, B, bias, C, batch, g, st) : launch_deep<T, RM, 2, true>(A, B, bias, C, batch, g, st);
}

template <typename T>
int launch_deep_typed(const void* A, const void* B, const void* bias, void* C, int64_t batch, const DeepArgs& g, cudaStream_t st) {
  const T *a = static_cast<const T*>(A), *b = static_cast<const T*>(B), *bs = static_cast<const T*>(bias);
  T* c = static_cast<T*>(C);
  if (g.M <= 4) return launch_deep_rows<T, 4>(a, b, bs, c, batch, g, st);
  if (g.M <= 8) return launch_deep_rows<T, 8>(a, b, bs, c, batch, g, st);
  return launch_deep_rows<T, 16>(a, b, bs, c, batch, g, st);
}

}  // namespace

// Where it is the faster one (us here / what it replaces; A and B from L2). A B with unit stride along N first:
//  - up to 40 rows: 1 x 4096 x 4096 12 / 50, 8 x 4096 x 32000 104 / 347, 16 x 1024 x 4096 9.2 / 16, 24 x 4096 x 8192 96 / 100. (A along
//    M and more than 16 rows: 37 x 2048 x 4096 42 / 56, but 32 x 4096 x 4096 64 / 50.)
//  - more rows: up to half a tile to an SM (183 x 4096 x 64 9 / 28, 128 x 4096 x 128 12 / 28, 1071 x 2048 x 64 14 / 23; beyond, 300 x 1024 x 300
//    with 95 tiles 14 / 14 and 347 x 1024 x 512 with 176 27 / 18), with a short K a quarter (16 of 64 x 256 x 64 6.5 to 8.4 / 7.2 to 8.0).
// B along K is slower to read: 16 x 4096 x 32000 238 / 428 and 183 x 4096 x 64 12 / 30, but 32 x 4096 x 4096 65 / 59 and 847 x 4096 x 64,
// 53 tiles, 35 / 31. A batch of products large enough for the bf16 planes, which cut no K there: 4 of 98 x 1024 x 512 27 to 43 / 45.
// 16-bit operands come here only when neither tensor-core kernel can load them as they are, in place of a copy and a product
// (64 of 4 x 1024 x 35 5.6 / 23, 300 x 300 x 301 9 / 14; 64 x 4097 x 1025, 68 tiles, 28 / 23; B along K, 16 x 4097 x 4097 44 / 34).
bool gemm_deep_preferred(int64_t batch, int64_t M, int64_t N, int64_t K, int64_t sAk, int64_t sBn, int dtype) {
  const int64_t rows = (M + 15) / 16, tiles = batch * rows * ((N + 63) / 64);
  if (!gemm_small_path_on() || batch < 1 || M < 1 || N < 1 || K < (M <= 8 ? 64 : 128) || batch * 8 > 65535 || rows > 65535) return false;
  const bool b_along_k = sBn != 1, a_along_m = sAk != 1;
  if (dtype != B200_F32) return tiles <= (b_along_k ? (a_along_m ? 8 : 24) : a_along_m ? 32 : M <= 16 ? 1024 : 64);
  if (batch > 1 && M > 64 && N > 64 && batch * M * N * K >= (1LL << 26) && tiles <= 224) return true;
  if (M > 40) return tiles <= (K < 512 ? 32 : !b_along_k ? kNumSMs / 2 : K <= 1024 ? 64 : 48);
  if (M <= 16 || tiles <= 64) return true;
  return b_along_k ? batch > 1 : !(a_along_m && K > 2048);
}

int gemm_deep_dispatch(const void* A, const void* B, const void* bias, void* C, int64_t batch, int64_t M, int64_t N, int64_t K, int64_t sAb, int64_t sAm, int64_t sAk, int64_t sBb,
                       int64_t sBk, int64_t sBn, int64_t sbm, int64_t sbn, double alpha, double beta, int dtype, cudaStream_t st, const uint32_t* gate) {
  const DeepArgs g{M, N, K, sAb, sAm, sAk, sBb, sBk, sBn, sbm, sbn, static_cast<float>(alpha), static_cast<float>(beta), gate, 1, 0};
  switch (dtype) {
    case B200_F32: return launch_deep_typed<float>(A, B, bias, C, batch, g, st);
    case B200_BF16: return launch_deep_typed<__nv_bfloat16>(A, B, bias, C, batch, g, st);
    case B200_F16: return launch_deep_typed<__half>(A, B, bias, C, batch, g, st);
    default: return B200_EDTYPE;
  }
}

}  // namespace b200
