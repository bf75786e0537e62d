// Device side of the evaluation path: one fused pass that answers both questions the
// harness asks about a (reference, result) pair -- "are they close?" (assert_close with
// equal_nan) and "how far apart?" (max abs / max rel error) -- plus the L2 flush used
// between timed repetitions. One read of each tensor, one 32-byte record back.
#include <cooperative_groups.h>
#include <math_constants.h>

#include "b200_common.cuh"

namespace cg = cooperative_groups;

namespace b200 {

struct CloseAcc {
  unsigned long long bad;
  float max_abs, max_rel;
  unsigned nan_seen;
};

// max_rel = max(max_rel, diff / den), dividing only when the quotient can raise the
// maximum. The product test is loose by 1e-6, far more than the roundings of the product
// and of the quotient, so it never hides a new maximum; after the first few elements of a
// thread almost every element fails it and costs a multiply instead of a division.
__device__ __forceinline__ void take_rel(CloseAcc& a, float diff, float den) {
  if (diff > a.max_rel * den * 0.999999f) a.max_rel = fmaxf(a.max_rel, diff / den);
}

// The rare side of one element pair: the difference is outside the band, infinite or NaN.
// Equal values (equal infinities: their difference is NaN) and NaN pairs are still close.
// Returns bit 0 = mismatch, bit 1 = the difference is NaN.
__device__ __noinline__ unsigned close_step_rare(float r, float s, float diff) {
  const bool close = (r == s) || (r != r && s != s);
  return (close ? 0u : 1u) | (diff != diff ? 2u : 0u);
}

// One element pair. The common path is kept to about ten instructions, which is what bounds
// the kernel next to its loads (an earlier form spent thirty and ran at half the issue rate
// of the SM):
//  * closeness, as torch.isclose(actual = reference output, expected = backend output) with
//    equal_nan: a finite difference inside the band atol + rtol * |expected| (NaN compares
//    false, so a NaN anywhere takes the rare path); everything else is decided there;
//  * error magnitudes follow `(ref - res).abs().max()`: fmaxf drops a NaN operand, so the
//    running maximum needs no guard.
__device__ __forceinline__ void close_step(CloseAcc& a, float r, float s, float rtol, float atol) {
  const float diff = fabsf(r - s);
  const float band = fmaf(rtol, fabsf(s), atol);
  if (!(diff <= band && diff != CUDART_INF_F)) {
    const unsigned what = close_step_rare(r, s, diff);
    a.bad += what & 1u;
    a.nan_seen |= what >> 1;
  }
  a.max_abs = fmaxf(a.max_abs, diff);
  take_rel(a, diff, fabsf(r) + 1e-10f);
}

__device__ __forceinline__ void warp_merge(CloseAcc& a) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    a.bad += __shfl_xor_sync(0xffffffffu, a.bad, o);
    a.max_abs = fmaxf(a.max_abs, __shfl_xor_sync(0xffffffffu, a.max_abs, o));
    a.max_rel = fmaxf(a.max_rel, __shfl_xor_sync(0xffffffffu, a.max_rel, o));
    a.nan_seen |= __shfl_xor_sync(0xffffffffu, a.nan_seen, o);
  }
}

// Merge the CTA's accumulators and fold them into the record with at most one
// atomic per field per CTA, and only where the CTA's value can still change the record: every
// atomic of every CTA goes to the same 32 bytes, so they queue up behind one another in L2
// (one set per WARP cost more time than reading 128 MiB of operands). Non-negative floats
// order like their bit patterns.
// `direct`: the record is to start from zero and the launch is one CTA, or (kCluster) one cluster,
// whose CTAs leave their accumulators with the first: it simply writes the record (no memset node before the
// kernel, no atomics). The first one's shared memory may be written only once that CTA is known to run: every CTA
// arrives at the cluster's barrier as it starts and waits there before it stores, by when the others have long
// arrived (their loads come in between).
constexpr int kCloseCluster = 8, kClusterThreads = 1024;
__device__ __forceinline__ void cluster_started_arrive() { asm volatile("barrier.cluster.arrive.relaxed;" ::: "memory"); }
__device__ __forceinline__ void cluster_started_wait() { asm volatile("barrier.cluster.wait;" ::: "memory"); }
__device__ __forceinline__ void write_record(const CloseAcc& a, b200_close_record* rec) {
  rec->mismatches = a.bad;
  rec->max_abs = a.max_abs;
  rec->max_rel = a.max_rel;
  rec->nan_seen = a.nan_seen;
  rec->pad[0] = rec->pad[1] = rec->pad[2] = 0u;
}
template <bool kCluster>
__device__ __forceinline__ void publish(CloseAcc a, b200_close_record* rec, int direct) {
  constexpr int kWarps = kCluster ? kClusterThreads / 32 : 8;
  __shared__ CloseAcc part[kWarps];
  warp_merge(a);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) part[warp] = a;
  __syncthreads();
  if (warp == 0) {
    a = lane < static_cast<int>(blockDim.x >> 5) ? part[lane] : CloseAcc{0ull, 0.f, 0.f, 0u};
    warp_merge(a);
  }
  if constexpr (kCluster) {
    __shared__ CloseAcc from[kCloseCluster];
    cg::cluster_group cluster = cg::this_cluster();
    cluster_started_wait();
    if (threadIdx.x == 0) *cluster.map_shared_rank(&from[cluster.block_rank()], 0) = a;
    cluster.sync();
    if (cluster.block_rank() != 0 || warp != 0) return;
    a = lane < kCloseCluster ? from[lane] : CloseAcc{0ull, 0.f, 0.f, 0u};
    warp_merge(a);
    if (lane == 0) write_record(a, rec);
    return;
  }
  if (warp != 0 || lane != 0) return;
  if (direct) {
    write_record(a, rec);
    return;
  }
  if (a.bad) atomicAdd(reinterpret_cast<unsigned long long*>(&rec->mismatches), a.bad);
  volatile unsigned* cur_abs = reinterpret_cast<volatile unsigned*>(&rec->max_abs);
  volatile unsigned* cur_rel = reinterpret_cast<volatile unsigned*>(&rec->max_rel);
  if (a.max_abs > 0.f && __float_as_uint(a.max_abs) > *cur_abs) atomicMax(reinterpret_cast<unsigned*>(&rec->max_abs), __float_as_uint(a.max_abs));
  if (a.max_rel > 0.f && __float_as_uint(a.max_rel) > *cur_rel) atomicMax(reinterpret_cast<unsigned*>(&rec->max_rel), __float_as_uint(a.max_rel));
  if (a.nan_seen && *reinterpret_cast<volatile unsigned*>(&rec->nan_seen) == 0u) atomicOr(&rec->nan_seen, 1u);
}

// exponent field of both halves of a packed pair of 16-bit floats
template <typename T> struct kExpMask16 { static constexpr uint32_t value = 0u; };
template <> struct kExpMask16<__nv_bfloat16> { static constexpr uint32_t value = 0x7f807f80u; };
template <> struct kExpMask16<__half> { static constexpr uint32_t value = 0x7c007c00u; };

template <typename T, bool kCluster>
__global__ void __launch_bounds__(kCluster ? kClusterThreads : 256, kCluster ? 1 : 4) allclose_kernel(const T* __restrict__ ref, const T* __restrict__ res, int64_t n, float rtol, float atol, b200_close_record* rec, int vec_ok, int direct) {
  constexpr int VE = Vec<T>::N;
  if constexpr (kCluster) cluster_started_arrive();  // (publish waits)
  CloseAcc a{0ull, 0.f, 0.f, 0u};
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  const int64_t t0 = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  int64_t done = 0;
  if (vec_ok) {
    const int64_t nvec = n / VE;
    // one vector pair of the record update; vectors that are bit-identical and hold no
    // infinity or NaN are close with zero error and leave at once (the update costs ten
    // instructions an element, and most vectors of a correct result are identical: the bit-exact
    // operators, and every elementwise one). 16-bit: exponent field not all ones; fp32: the sum
    // of the four magnitudes is finite (a sum that overflows only sends the vector the long way).
    auto take = [&](const uint4& vr, const uint4& vs) {
      if (((vr.x ^ vs.x) | (vr.y ^ vs.y) | (vr.z ^ vs.z) | (vr.w ^ vs.w)) == 0u) {
        if (sizeof(T) == 2) {
          const uint32_t m = kExpMask16<T>::value;
          if ((__vcmpeq2(vr.x & m, m) | __vcmpeq2(vr.y & m, m) | __vcmpeq2(vr.z & m, m) | __vcmpeq2(vr.w & m, m)) == 0u) return;
        } else {
          const float t = (fabsf(__uint_as_float(vr.x)) + fabsf(__uint_as_float(vr.y))) + (fabsf(__uint_as_float(vr.z)) + fabsf(__uint_as_float(vr.w)));
          if (t < CUDART_INF_F) return;
        }
      }
      float fr[VE], fs[VE];
      widen<T>(vr, fr);
      widen<T>(vs, fs);
#pragma unroll
      for (int e = 0; e < VE; ++e) close_step(a, fr[e], fs[e], rtol, atol);
    };
    // two vector pairs (four 16-byte loads) in flight per thread and four CTAs per SM
    constexpr int U = 2;
    int64_t j = t0;
    for (; j + (U - 1) * stride < nvec; j += U * stride) {
      uint4 vr[U], vs[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        vr[u] = ld_stream(ref + (j + u * stride) * VE);
        vs[u] = ld_stream(res + (j + u * stride) * VE);
      }
#pragma unroll
      for (int u = 0; u < U; ++u) take(vr[u], vs[u]);
    }
    for (; j < nvec; j += stride) take(ld_stream(ref + j * VE), ld_stream(res + j * VE));
    done = nvec * VE;
  }
  for (int64_t i = done + t0; i < n; i += stride) close_step(a, to_f32(ref[i]), to_f32(res[i]), rtol, atol);
  publish<kCluster>(a, rec, direct);
}

// Integer / bool tensors: the same band as for floating point, |ref - res| <= atol + rtol * |res|,
// evaluated in double (assert_close applies its tolerances to integers too: 5000 and 5001 are
// close under the harness's 1e-2); atol = rtol = 0 makes the comparison exact. Error magnitudes
// after conversion to fp32 as the host formula does.
template <typename T>
__global__ void __launch_bounds__(256) allclose_int_kernel(const T* __restrict__ ref, const T* __restrict__ res, int64_t n, double rtol, double atol, b200_close_record* rec, int direct) {
  CloseAcc a{0ull, 0.f, 0.f, 0u};
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const T r = ref[i], s = res[i];
    if (r != s) {  // zero tolerances: unequal is a mismatch, whatever double makes of the difference
      const double ds = static_cast<double>(s);
      const bool inside = (rtol > 0.0 || atol > 0.0) && fabs(static_cast<double>(r) - ds) <= atol + rtol * fabs(ds);
      if (!inside) ++a.bad;
    }
    const float fr = static_cast<float>(r), fs = static_cast<float>(s);
    const float diff = fabsf(fr - fs);
    a.max_abs = fmaxf(a.max_abs, diff);
    take_rel(a, diff, fabsf(fr) + 1e-10f);
  }
  publish<false>(a, rec, direct);
}

__global__ void __launch_bounds__(256) l2_flush_kernel(uint4* __restrict__ p, int64_t nvec) {
  const uint4 z = make_uint4(0, 0, 0, 0);
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < nvec; i += static_cast<int64_t>(gridDim.x) * blockDim.x) p[i] = z;
}

template <typename T>
static int launch_allclose(const T* ref, const T* res, int64_t n, float rtol, float atol, b200_close_record* rec, int vec_ok, int direct, int grid, cudaStream_t st) {
  if (direct != kCloseCluster) {
    allclose_kernel<T, false><<<grid, 256, 0, st>>>(ref, res, n, rtol, atol, rec, vec_ok, direct);
    return check_launch();
  }
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(kCloseCluster);
  cfg.blockDim = dim3(n <= kCloseCluster * 256 * Vec<T>::N ? 256 : kClusterThreads);  // (a vector to a thread)
  cfg.stream = st;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = kCloseCluster;
  attr.val.clusterDim.y = 1;
  attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, allclose_kernel<T, true>, ref, res, n, rtol, atol, rec, vec_ok, direct);
  if (e != cudaSuccess) { set_last_cuda_error(e); return B200_ELAUNCH; }
  return check_launch();
}

}  // namespace b200

using namespace b200;

extern "C" int b200_allclose(const void* ref, const void* res, int64_t n, int dtype, double rtol, double atol, b200_close_record* rec, int reset, void* stream) {
  if (n < 0 || !rec) return B200_EINVAL;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  // Small comparisons whose record is to be reset are one launch that writes the record itself, in place of a memset
  // and a launch (most of the sweep's cases are this small, and their cost is launches, not bytes): one CTA up to 2048
  // elements, a cluster of eight up to 65536. fp32, equal / different values: 32768 elements 6.2 / 15.2 us with
  // one CTA, 3.0 / 4.4 with a cluster; 65536 5.5 / 6.6 with a memset and 32 CTAs, 3.5 / 6.4; bf16 131072 6.1 / 6.7 and 3.8 / 8.3.
  const int direct = !reset || n == 0 ? 0 : n <= 2048 ? 1 : n <= 65536 && is_float_dtype(dtype) ? kCloseCluster : n <= 32768 ? 1 : 0;
  if (reset && !direct) {
    const cudaError_t e = cudaMemsetAsync(rec, 0, sizeof(b200_close_record), st);
    if (e != cudaSuccess) { set_last_cuda_error(e); return B200_ELAUNCH; }
  }
  if (n == 0) return B200_OK;
  if (!ref || !res) return B200_EINVAL;
  const int es = dtype_size(dtype);
  if (es == 0) return B200_EDTYPE;
  int64_t blocks = n <= 32768 ? 1 : (n + 256 * 8 - 1) / (256 * 8);
  const int64_t cap = static_cast<int64_t>(kNumSMs) * 8;  // one resident wave of 256-thread CTAs
  const int g = static_cast<int>(blocks < 1 ? 1 : (blocks > cap ? cap : blocks));
  const int vec_ok = aligned16(ref) && aligned16(res);
  const float rt = static_cast<float>(rtol), at = static_cast<float>(atol);
  switch (dtype) {
    case B200_F32: return launch_allclose(static_cast<const float*>(ref), static_cast<const float*>(res), n, rt, at, rec, vec_ok, direct, g, st);
    case B200_BF16: return launch_allclose(static_cast<const __nv_bfloat16*>(ref), static_cast<const __nv_bfloat16*>(res), n, rt, at, rec, vec_ok, direct, g, st);
    case B200_F16: return launch_allclose(static_cast<const __half*>(ref), static_cast<const __half*>(res), n, rt, at, rec, vec_ok, direct, g, st);
    case B200_I64: allclose_int_kernel<int64_t><<<g, 256, 0, st>>>(static_cast<const int64_t*>(ref), static_cast<const int64_t*>(res), n, rtol, atol, rec, direct); break;
    case B200_I32: allclose_int_kernel<int32_t><<<g, 256, 0, st>>>(static_cast<const int32_t*>(ref), static_cast<const int32_t*>(res), n, rtol, atol, rec, direct); break;
    case B200_I16: allclose_int_kernel<int16_t><<<g, 256, 0, st>>>(static_cast<const int16_t*>(ref), static_cast<const int16_t*>(res), n, rtol, atol, rec, direct); break;
    case B200_I8: allclose_int_kernel<int8_t><<<g, 256, 0, st>>>(static_cast<const int8_t*>(ref), static_cast<const int8_t*>(res), n, rtol, atol, rec, direct); break;
    case B200_BOOL: case B200_U8: allclose_int_kernel<uint8_t><<<g, 256, 0, st>>>(static_cast<const uint8_t*>(ref), static_cast<const uint8_t*>(res), n, rtol, atol, rec, direct); break;
    default: return B200_EDTYPE;
  }
  return check_launch();
}

extern "C" int b200_l2_flush(void* scratch, int64_t bytes, void* stream) {
  if (bytes < 0 || (bytes > 0 && !scratch) || !aligned16(scratch)) return B200_EINVAL;
  if (bytes < 16) return B200_OK;
  l2_flush_kernel<<<kNumSMs * 8, 256, 0, static_cast<cudaStream_t>(stream)>>>(static_cast<uint4*>(scratch), bytes / 16);
  return check_launch();
}
