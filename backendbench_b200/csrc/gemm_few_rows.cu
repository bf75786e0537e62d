// 16-bit mm / addmm with at most 16 rows of A against a large B whose rows lie along K (the weight
// matrix of a linear layer, [out, in], while a model decodes a few tokens): bound by reading B
// once. The tcgen05 kernel gives such a product 128-row tiles of which 16 are used, N / 256
// CTAs, and a handful of stages in flight in each: 16 x 4096 x 11008 ran on 43 SMs (44 us,
// 2.1 TB/s), 16 x 11008 x 4096 in 16 CTAs split over K with a second pass (29 us).
//
// Here a CTA owns 8 to 40 columns of C and its eight warps share K. A warp streams B from global
// memory straight into mma.sync operands, with no shared memory in between: in
// mma.m16n8k16 lane (q, c) holds elements 2c, 2c + 1, 2c + 8, 2c + 9 of row q of B (and of rows
// q, q + 8 of A). The order of the products in a sum over k is free, so the 32 k of
// two such steps are dealt out as the 16-byte pieces 8c .. 8c + 7 of a row: one load
// each. Three or four steps of both operands are in flight per lane; A comes from L2, where every CTA
// reads it. The warps' sums are added in warp order in fp32, then alpha, beta, the bias and
// one rounding. bf16, 16 rows: K 4096 x N 11008 44 -> 16.6 us (5.4 TB/s), K 11008 x N 4096 29 -> 17.1 us
// (5.3 TB/s; 256 CTAs, so the busiest SM has 32 columns where the mean is 27.7).
#include <type_traits>

#include "b200_common.cuh"

namespace b200 {

namespace {

constexpr int kFewRows = 16;
constexpr int kFewWarps = 8;
constexpr int kFewMaxFragments = 5;       // of eight columns each, to a CTA: see few_fragments
template <int NT> struct FewSteps { static constexpr int value = NT > 3 ? 3 : 4; };  // 32-k steps in flight per lane
// Where the kernel is the faster one; bf16 with B out of HBM, us here / the tcgen05 kernel or its ranges of K.
// The tcgen05 kernel has a CTA to 256 columns: up to 96 of them leave it SMs idle (N 20000, K 4096: 8 rows 31.1 /
// 43.5, 16 rows 33.2 / 37.2; N 24000: 16 rows 41.5 / 40.7). Beyond, this one wins by what it does not read twice, as long as the rows of A,
// which every CTA reads from L2, are few (N 32000, K 4096: 8 rows 48.9 / 59.0, 16 rows 51.7 / 49.0; K 2048: 16 rows 28.4 / 32.6; between the two the line
// could lie further out: K 3072, 12 rows 37.7 / 45.5) and K is long enough to pay for the many CTAs (N 32000: K 264 12.0 / 9.9, K 512 13.2 / 10.7, K 768
// 14.6 / 14.2, K 1024 16.8 / 18.4; N 128256, K 1024: 4 rows 49.5 / 53.8, 16 rows 54.8 / 54.5).
constexpr int64_t kFewMaxK = 16384;
constexpr int64_t kFewMaxN = 96 * 256;  // with any number of rows
constexpr int64_t kFewShortK = 256, kFewShortMaxN = 16384;  // (N 20000, K 64: 4 rows 5.3 / 5.1, 16 rows 5.7 / 5.1)
static bool few_rows_pay(int64_t M, int64_t N, int64_t K) {
  if (N > kFewShortMaxN && K < kFewShortK) return false;
  return N <= kFewMaxN || (K >= (N > 65536 && M > 4 ? 2048 : 1024) && (M <= 8 || K <= 2048));
}

struct FewRowsArgs {
  int64_t M, N, K, sAm, sBn, sbm, sbn;
  float alpha, beta;
};

template <typename T>
__device__ __forceinline__ void mma_step(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  if (std::is_same<T, __nv_bfloat16>::value) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
  } else {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
  }
}

template <typename T, int NT>
__global__ void __launch_bounds__(32 * kFewWarps, 2) gemm_few_rows(const T* A, const T* B, const T* bias, T* __restrict__ C, FewRowsArgs p) {
  constexpr int kCols = 8 * NT, kPitch = kCols + 1, kFewSteps = FewSteps<NT>::value;
  __shared__ float red[kFewWarps][kFewRows][kPitch];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, q = lane >> 2, c = lane & 3;
  const int64_t n0 = static_cast<int64_t>(blockIdx.x) * kCols;
  const bool row0 = q < p.M, row1 = q + 8 < p.M;
  const T* a0 = A + (row0 ? q : 0) * p.sAm + 8 * c;
  const T* a1 = A + (row1 ? q + 8 : 0) * p.sAm + 8 * c;
  const T* b[NT];
  bool col[NT];
#pragma unroll
  for (int t = 0; t < NT; ++t) {
    col[t] = n0 + 8 * t + q < p.N;
    b[t] = B + (col[t] ? n0 + 8 * t + q : 0) * p.sBn + 8 * c;
  }
  float acc[NT][4];
#pragma unroll
  for (int t = 0; t < NT; ++t) acc[t][0] = acc[t][1] = acc[t][2] = acc[t][3] = 0.f;
  const int K = static_cast<int>(p.K);  // a multiple of 8: a piece is inside the row or outside it
  // While the kernel before ends, the lines that the warp reads first are brought into L2 (which holds what that
  // kernel writes all the same, should it be these). A CTA that comes after the first round has nothing to wait for: there it was
  // the same lines asked for twice (bf16, 3 rows, K 3880 x N 18080 29.8 -> 27.7 us, 13 rows, K 1600 x N 44992 36.6 -> 34.8).
  next_grid_may_start();
#pragma unroll
  for (int u = 0; u < 2 * kFewSteps; ++u) {
    const int k = (warp + (u / kFewSteps) * kFewWarps) * 32 * kFewSteps + 32 * (u % kFewSteps);
#pragma unroll
    for (int t = 0; t < NT; ++t)
      if (blockIdx.x < 2 * kNumSMs && (c & 1) == 0 && k + 8 * c < K && col[t]) asm volatile("prefetch.global.L2 [%0];" ::"l"(b[t] + k));
  }
  after_grids_before();
  a0 = waited(a0);
  a1 = waited(a1);
#pragma unroll
  for (int t = 0; t < NT; ++t) b[t] = waited(b[t]);
  for (int k0 = warp * 32 * kFewSteps; k0 < K; k0 += kFewWarps * 32 * kFewSteps) {
    uint4 ra[kFewSteps], rA[kFewSteps], rb[NT][kFewSteps];
    const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
    for (int u = 0; u < kFewSteps; ++u) {
      const int k = k0 + 32 * u;
      const bool in = k + 8 * c < K;
#pragma unroll
      for (int t = 0; t < NT; ++t) rb[t][u] = in && col[t] ? ld_stream_after(b[t] + k) : zero;
      ra[u] = in && row0 ? ld_keep_after(a0 + k) : zero;
      rA[u] = in && row1 ? ld_keep_after(a1 + k) : zero;
    }
#pragma unroll
    for (int u = 0; u < kFewSteps; ++u) {
#pragma unroll
      for (int t = 0; t < NT; ++t) {
        mma_step<T>(acc[t], ra[u].x, rA[u].x, ra[u].y, rA[u].y, rb[t][u].x, rb[t][u].y);
        mma_step<T>(acc[t], ra[u].z, rA[u].z, ra[u].w, rA[u].w, rb[t][u].z, rb[t][u].w);
      }
    }
  }
#pragma unroll
  for (int t = 0; t < NT; ++t) {
    red[warp][q][8 * t + 2 * c] = acc[t][0];
    red[warp][q][8 * t + 2 * c + 1] = acc[t][1];
    red[warp][q + 8][8 * t + 2 * c] = acc[t][2];
    red[warp][q + 8][8 * t + 2 * c + 1] = acc[t][3];
  }
  __syncthreads();
  for (int i = threadIdx.x; i < kFewRows * kCols; i += 32 * kFewWarps) {
    const int m = i / kCols, j = i - m * kCols;
    const int64_t n = n0 + j;
    if (m >= p.M || n >= p.N) continue;
    float s = red[0][m][j];
#pragma unroll
    for (int w = 1; w < kFewWarps; ++w) s += red[w][m][j];
    float r = p.alpha * s;
    if (bias) r = fmaf(p.beta, to_f32(bias[m * p.sbm + n * p.sbn]), r);
    C[m * p.N + n] = from_f32<T>(r);
  }
}

}  // namespace

bool gemm_few_rows_preferred(const void* A, const void* B, int64_t batch, int64_t M, int64_t N, int64_t K, int64_t sAm, int64_t sAk, int64_t sBk, int64_t sBn, int dtype) {
  if (dtype != B200_BF16 && dtype != B200_F16) return false;
  if (batch != 1 || M < 1 || M > kFewRows || N < 1 || N > 0x7fffffffLL || K < 64 || K > kFewMaxK || K % 8 != 0) return false;
  if (!few_rows_pay(M, N, K)) return false;
  if (sAk != 1 || sBk != 1 || !aligned16(A) || !aligned16(B)) return false;
  return (M == 1 || (sAm % 8 == 0 && sAm >= 0)) && (N == 1 || (sBn % 8 == 0 && sBn >= 0));
}

// A CTA walks all of K. With few columns, so few CTAs, a long K can be cut into ranges instead, where the K-split can take the
// product. The line was drawn with 16 columns to every CTA; with as many as few_fragments gives, few rows do better here on
// its far side, too, and only 16 rows are near it (here / ranges; 4 rows, N 512: K 8192 6.2 / 10.4, K 12288 8.4 / 11.6; N 128: K 8192 5.6 / 8.0; N 64: K
// 11008 6.8 / 8.4; N 1024: K 11008 8.3 / 12.8, K 16384 11.6 / 14.5; N 1536: K 16384 12.8 / 16.6; N 2048: K 16384 14.1 / 19.1; 16 rows, N 128: K 8192 7.0 / 8.1; N 1536: K 12288
// 14.2 / 15.0, K 16384 18.3 / 16.8).
bool gemm_few_rows_leaves_to_ranges(int64_t N, int64_t K) {
  return N < 2048 && (K > (N <= 1024 ? 11264 : 14336) || (K > 8448 && N >= 16 && N <= 512) || (K > 7168 && N > 64 && N <= 128));
}

// Fragments of eight columns to a CTA. What counts is that the CTAs, two to an SM, come out even, and best that all of
// them run at once: 16 x 4096 against 11008 columns takes 21.7 us with two (688 CTAs, 2.3 rounds) and 16.6 with five (276), 8192 columns 25.9
// with two (512), 30.8 with three, 22.4 with four (256). One CTA alone on an SM has too few loads in flight (4096 columns: 22.9 with four, 128
// CTAs; 17.1 with two). Over many rounds the width matters by what a CTA reads of A and by what it keeps in flight: 32000 columns 59 / 47.5 /
// 46.6 / 48.4 / 50.5 us with one to five. The figures below are those ratios.
static int few_fragments(int64_t N) {
  constexpr int kPer[kFewMaxFragments] = {127, 102, 100, 104, 108};
  int best = 1;
  double least = 0.;
  for (int nt = 1; nt <= kFewMaxFragments; ++nt) {
    const int64_t ctas = (N + 8 * nt - 1) / (8 * nt), slots = 2 * kNumSMs;
    const double rounds = static_cast<double>(ctas) / slots, whole = static_cast<double>((ctas + slots - 1) / slots);
    const double columns = nt * (ctas <= kNumSMs ? 1.16 : ctas <= slots ? 2. * 0.85 : rounds + whole);  // ("2 *" their mean)
    if (nt == 1 || columns * kPer[nt - 1] < least) { least = columns * kPer[nt - 1]; best = nt; }
  }
  return best;
}

template <typename T>
static cudaError_t launch_few_rows(const void* A, const void* B, const void* bias, void* C, const FewRowsArgs& p, cudaStream_t st) {
  const int nt = few_fragments(p.N);
  auto launch = [&](auto kernel) {
    return launch_after(kernel, (p.N + 8 * nt - 1) / (8 * nt), 32 * kFewWarps, 0, st, static_cast<const T*>(A), static_cast<const T*>(B), static_cast<const T*>(bias), static_cast<T*>(C), p);
  };
  switch (nt) {
    case 1: return launch(gemm_few_rows<T, 1>);
    case 2: return launch(gemm_few_rows<T, 2>);
    case 3: return launch(gemm_few_rows<T, 3>);
    case 4: return launch(gemm_few_rows<T, 4>);
    default: return launch(gemm_few_rows<T, 5>);
  }
}

int gemm_few_rows_dispatch(const void* A, const void* B, const void* bias, void* C, int64_t M, int64_t N, int64_t K, int64_t sAm, int64_t sBn, int64_t sbm, int64_t sbn, double alpha,
                           double beta, int dtype, cudaStream_t st) {
  const FewRowsArgs p{M, N, K, sAm, sBn, sbm, sbn, static_cast<float>(alpha), static_cast<float>(beta)};
  const void* bs = static_cast<float>(beta) != 0.f ? bias : nullptr;  // beta = 0 ignores the bias, NaN included
  const cudaError_t e = dtype == B200_BF16 ? launch_few_rows<__nv_bfloat16>(A, B, bs, C, p, st) : launch_few_rows<__half>(A, B, bs, C, p, st);
  if (e != cudaSuccess) { set_last_cuda_error(e); return B200_ELAUNCH; }
  return check_launch();
}

}  // namespace b200
