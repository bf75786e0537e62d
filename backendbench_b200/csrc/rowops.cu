// _softmax / _log_softmax / native_layer_norm / sum.dim_IntList / argmax.
//
// The input is contiguous, viewed as [outer, dim, inner], the op runs along `dim`.
//   inner == 1, row fits in registers : "resident" kernels -- the row is read from HBM
//       exactly once with 16-byte streaming loads, held as fp32 in registers by one
//       warp (short rows) or one CTA (long rows), reduced with warp shuffles (+ one
//       shared-memory hop for CTA rows) and written once: 1 read + 1 write per element.
//   inner == 1, anything else        : "streaming" kernels, one CTA per row, scalar
//       accesses, re-reads served by L2.
//   inner  > 1                        : one thread per (outer, inner) column, coalesced
//       across `inner`, sequential along `dim`.
// sum and argmax are single-pass; when few outputs face a long reduction the reduction
// is split over gridDim.y CTAs and finished by a second tiny kernel from scratch memory.
#include <math_constants.h>

#include <mutex>
#include <type_traits>

#include "b200_common.cuh"

namespace b200 {

constexpr float kLog2e = 1.4426950408889634f;

template <typename T> constexpr int dtype_of();
template <> constexpr int dtype_of<float>() { return B200_F32; }
template <> constexpr int dtype_of<__nv_bfloat16>() { return B200_BF16; }
template <> constexpr int dtype_of<__half>() { return B200_F16; }

// ---- group = one warp (WARP) or the whole CTA: reductions over the threads of a row
template <bool WARP, typename F>
__device__ __forceinline__ float group_reduce(float v, F f, float identity, float* smem, int phase) {
  if (WARP) return warp_reduce(v, f);
  return block_reduce_once(v, f, identity, smem, phase);
}

// Store VE fp32 values at element offset `e0` of `out`, as T (16-byte store) or as fp32.
template <typename T>
__device__ __forceinline__ void store_row_vec(void* out, int64_t e0, const float* f, bool out_f32) {
  constexpr int VE = Vec<T>::N;
  if (sizeof(T) == 4 || out_f32) {
    float* o = static_cast<float*>(out) + e0;
#pragma unroll
    for (int q = 0; q < VE / 4; ++q) st_stream(o + 4 * q, make_uint4(__float_as_uint(f[4 * q]), __float_as_uint(f[4 * q + 1]), __float_as_uint(f[4 * q + 2]), __float_as_uint(f[4 * q + 3])));
  } else {
    st_stream(static_cast<T*>(out) + e0, narrow<T>(f));
  }
}

// Load VE weights (dtype TW) starting at element e0 as fp32; weights are re-read by
// every row, so they take the cached read-only path.
template <int VE, typename TW>
__device__ __forceinline__ void load_weights(const TW* w, int e0, float* f) {
  constexpr int PER = 16 / sizeof(TW);
#pragma unroll
  for (int q = 0; q < VE / PER; ++q) {
    widen<TW>(ld_keep(w + e0 + q * PER), f + q * PER);
  }
}

// ------------------------------------------------------------------ softmax, resident
// One row by one group of threads (a warp, or the whole CTA).
template <typename T, int VPT, bool WARP, bool IS_LOG>
__device__ __forceinline__ void softmax_row(const T* __restrict__ xr, void* __restrict__ out, int64_t out_e0, int nvec, int t, int tpr, int out_f32, float* red) {
  constexpr int VE = Vec<T>::N;
  float f[VPT][VE];
  float m = -CUDART_INF_F;
#pragma unroll
  for (int u = 0; u < VPT; ++u) {
    const int j = t + u * tpr;
    if (j < nvec) {
      widen<T>(ld_stream(xr + static_cast<int64_t>(j) * VE), f[u]);
#pragma unroll
      for (int e = 0; e < VE; ++e) m = fmaxf(m, f[u][e]);
    }
  }
  m = group_reduce<WARP>(m, MaxF{}, -CUDART_INF_F, red, 0);
  float s = 0.f;
  // softmax: 2^(x*log2(e) - c) with c = m*log2(e) rounded once; the rounding of c scales
  // every term of the row alike and cancels in the quotient. Not when c would overflow,
  // and not for log_softmax, which needs x - m itself.
  if (!IS_LOG && fabsf(m) < 1e37f) {
    const float c = m * kLog2e;
#pragma unroll
    for (int u = 0; u < VPT; ++u) {
      if (t + u * tpr < nvec) {
#pragma unroll
        for (int e = 0; e < VE; ++e) {
          f[u][e] = ex2_approx(fmaf(f[u][e], kLog2e, -c));
          s += f[u][e];
        }
      }
    }
  } else {
#pragma unroll
    for (int u = 0; u < VPT; ++u) {
      if (t + u * tpr < nvec) {
#pragma unroll
        for (int e = 0; e < VE; ++e) {
          const float d = f[u][e] - m;
          const float ex = ex2_approx(d * kLog2e);
          s += ex;
          f[u][e] = IS_LOG ? d : ex;
        }
      }
    }
  }
  s = group_reduce<WARP>(s, SumF{}, 0.f, red, 1);
  const float k = IS_LOG ? logf(s) : 1.f / s;
#pragma unroll
  for (int u = 0; u < VPT; ++u) {
    const int j = t + u * tpr;
    if (j < nvec) {
#pragma unroll
      for (int e = 0; e < VE; ++e) f[u][e] = IS_LOG ? f[u][e] - k : f[u][e] * k;
      store_row_vec<T>(out, out_e0 + static_cast<int64_t>(j) * VE, f[u], out_f32 != 0);
    }
  }
}

template <typename T, int VPT, bool WARP, bool IS_LOG>
__global__ void __launch_bounds__(WARP ? 128 : 1024)
softmax_resident(const T* __restrict__ x, void* __restrict__ out, int64_t rows, int cols, int out_f32) {
  __shared__ float red[64];
  const int tpr = WARP ? 32 : blockDim.x;
  const int t = WARP ? (threadIdx.x & 31) : threadIdx.x;
  const int64_t row = WARP ? static_cast<int64_t>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5) : blockIdx.x;
  if (WARP && row >= rows) return;
  softmax_row<T, VPT, WARP, IS_LOG>(x + row * cols, out, row * cols, cols / Vec<T>::N, t, tpr, out_f32, red);
}

// ------------------------------------------------------------------ softmax / log_softmax backward
// aten._softmax_backward_data:      gin = (g - sum(g * y)) * y
// aten._log_softmax_backward_data:  gin = g - exp(y) * sum(g)
// with y the forward output, along `dim` of [outer, dim, inner]. Resident kernel: the rows
// of g and y are read once with 16-byte loads and held in registers (one warp or one CTA
// per row), one reduction, one write -- the forward kernel's geometry with two inputs.
template <typename T, int VPT, bool WARP, bool IS_LOG>
__global__ void __launch_bounds__(WARP ? 128 : 1024)
softmax_bwd_resident(const T* __restrict__ g, const T* __restrict__ y, void* __restrict__ out, int64_t rows, int cols, int out_f32) {
  constexpr int VE = Vec<T>::N;
  __shared__ float red[64];
  const int tpr = WARP ? 32 : blockDim.x;
  const int t = WARP ? (threadIdx.x & 31) : threadIdx.x;
  const int64_t row = WARP ? static_cast<int64_t>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5) : blockIdx.x;
  if (WARP && row >= rows) return;
  const int nvec = cols / VE;
  const T* gr = g + row * cols;
  const T* yr = y + row * cols;
  float fg[VPT][VE], fy[VPT][VE];
  float s = 0.f;
#pragma unroll
  for (int u = 0; u < VPT; ++u) {
    const int j = t + u * tpr;
    if (j < nvec) {
      widen<T>(ld_stream(gr + j * VE), fg[u]);
      widen<T>(ld_stream(yr + j * VE), fy[u]);
#pragma unroll
      for (int e = 0; e < VE; ++e) s += IS_LOG ? fg[u][e] : fg[u][e] * fy[u][e];
    }
  }
  s = group_reduce<WARP>(s, SumF{}, 0.f, red, 0);
#pragma unroll
  for (int u = 0; u < VPT; ++u) {
    const int j = t + u * tpr;
    if (j < nvec) {
#pragma unroll
      for (int e = 0; e < VE; ++e) fg[u][e] = IS_LOG ? fg[u][e] - ex2_approx(fy[u][e] * kLog2e) * s : (fg[u][e] - s) * fy[u][e];
      store_row_vec<T>(out, row * cols + static_cast<int64_t>(j) * VE, fg[u], out_f32 != 0);
    }
  }
}

// Rows too long for the registers of a CTA, or off the 16-byte grid (a vocabulary of 50,257):
// one CTA per row, single elements up to the row's first 16-byte boundary and behind its
// last one, 16-byte accesses in between, four of each operand in flight per thread (ONE_TRIP: that is
// all of the row). The first
// pass needs grad alone for log_softmax (and both operands for softmax); the second reads it
// again from L2. All three rows have to lie at the same offset from the grid. Bound by HBM:
// log_softmax, bf16 4096 x 50257, 205 us (6.0 TB/s; a warp per row with element-wise accesses,
// the kernel below, 468 us).
template <typename T, bool IS_LOG, bool ONE_TRIP>
__global__ void __launch_bounds__(512) softmax_bwd_stream(const T* __restrict__ g, const T* __restrict__ y, T* __restrict__ out, int cols) {
  constexpr int VE = Vec<T>::N;
  __shared__ float red[64];
  const int64_t row = blockIdx.x;
  const T* gr = g + row * cols;
  const T* yr = y + row * cols;
  T* orow = out + row * cols;
  const int t = threadIdx.x, nth = blockDim.x;
  const int to_grid = static_cast<int>((16u - (reinterpret_cast<uintptr_t>(gr) & 15u)) & 15u) / static_cast<int>(sizeof(T));
  const int lead = to_grid < cols ? to_grid : cols;
  const int nv = (cols - lead) / VE, tail = lead + nv * VE;
  const int single = t < lead ? t : (tail + t - lead < cols ? tail + t - lead : -1);  // one of the at most 2 (VE - 1) elements off the vectors
  const T* gv = gr + lead;
  const T* yv = yr + lead;
  float s = 0.f;
  if (single >= 0) s = IS_LOG ? to_f32(gr[single]) : to_f32(gr[single]) * to_f32(yr[single]);
  auto take = [&](const uint4& rg, const uint4& ry) {  // (one trip: a vector's own sum, then the thread's, a shorter chain of additions)
    float own = ONE_TRIP ? 0.f : s;
    if (IS_LOG) {
      vec_accumulate<T>(own, rg);
    } else {
      float fg[VE], fy[VE];
      widen<T>(rg, fg);
      widen<T>(ry, fy);
#pragma unroll
      for (int e = 0; e < VE; ++e) own += fg[e] * fy[e];
    }
    s = ONE_TRIP ? s + own : own;
  };
  int j = t;
  if constexpr (ONE_TRIP) {
    uint4 rg[4], ry[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if (j + u * nth < nv) {
        rg[u] = ld_keep(gv + (j + u * nth) * VE);
        ry[u] = IS_LOG ? rg[u] : ld_keep(yv + (j + u * nth) * VE);
      }
    }
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (j + u * nth < nv) take(rg[u], ry[u]);
  } else {
    for (; j + 3 * nth < nv; j += 4 * nth) {
      uint4 rg[4], ry[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        rg[u] = ld_keep(gv + (j + u * nth) * VE);
        ry[u] = IS_LOG ? rg[u] : ld_keep(yv + (j + u * nth) * VE);
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) take(rg[u], ry[u]);
    }
    for (; j < nv; j += nth) {
      const uint4 rg = ld_keep(gv + j * VE);
      take(rg, IS_LOG ? rg : ld_keep(yv + j * VE));
    }
  }
  s = block_reduce_once(s, SumF{}, 0.f, red, 0);
  auto gradient = [&](float fg, float fy) { return IS_LOG ? fg - ex2_approx(fy * kLog2e) * s : (fg - s) * fy; };
  if (single >= 0) orow[single] = from_f32<T>(gradient(to_f32(gr[single]), to_f32(yr[single])));
  auto give = [&](int jj, const uint4& rg, const uint4& ry) {
    float fg[VE], fy[VE];
    widen<T>(rg, fg);
    widen<T>(ry, fy);
#pragma unroll
    for (int e = 0; e < VE; ++e) fg[e] = gradient(fg[e], fy[e]);
    st_stream(orow + lead + jj * VE, narrow<T>(fg));
  };
  j = t;
  if constexpr (ONE_TRIP) {
    uint4 rg[4], ry[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if (j + u * nth < nv) {
        ry[u] = ld_stream(yv + (j + u * nth) * VE);
        rg[u] = ld_stream(gv + (j + u * nth) * VE);
      }
    }
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (j + u * nth < nv) give(j + u * nth, rg[u], ry[u]);
  } else {
    for (; j + 3 * nth < nv; j += 4 * nth) {
      uint4 rg[4], ry[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        ry[u] = ld_stream(yv + (j + u * nth) * VE);
        rg[u] = ld_stream(gv + (j + u * nth) * VE);
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) give(j + u * nth, rg[u], ry[u]);
    }
    for (; j < nv; j += nth) give(j, ld_stream(gv + j * VE), ld_stream(yv + j * VE));
  }
}

// Any geometry and alignment: one warp per (outer, inner) line, elements `inner` apart,
// two passes over the line (the second from cache).
template <typename T, bool IS_LOG>
__global__ void __launch_bounds__(128) softmax_bwd_lines(const T* __restrict__ g, const T* __restrict__ y, void* __restrict__ out, int64_t outer, int64_t dim, int64_t inner, int dto) {
  const int lane = threadIdx.x & 31;
  const int64_t line = static_cast<int64_t>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (line >= outer * inner) return;
  const int64_t o = line / inner, i = line - o * inner, base = o * dim * inner + i;
  float s = 0.f;
  for (int64_t k = lane; k < dim; k += 32) s += IS_LOG ? to_f32(g[base + k * inner]) : to_f32(g[base + k * inner]) * to_f32(y[base + k * inner]);
  s = warp_reduce(s, SumF{});
  for (int64_t k = lane; k < dim; k += 32) {
    const float gv = to_f32(g[base + k * inner]), yv = to_f32(y[base + k * inner]);
    store_from_f32(out, base + k * inner, dto, IS_LOG ? gv - ex2_approx(yv * kLog2e) * s : (gv - s) * yv);
  }
}

// ------------------------------------------------------------------ softmax, streaming
// One CTA per row, three scalar passes (max, sum of exponentials, write); the second
// and third read come from L2. Any `cols`, any alignment. NaN / inf rows behave as in
// the resident kernel: the arithmetic is the same, only the data path differs.
template <typename T>
__global__ void __launch_bounds__(256) softmax_stream(const T* __restrict__ x, void* __restrict__ out, int64_t cols, int dto, int is_log) {
  __shared__ float red[33];
  const int64_t row = blockIdx.x;
  const T* xr = x + row * cols;
  float m = -CUDART_INF_F;
  for (int64_t c = threadIdx.x; c < cols; c += blockDim.x) m = fmaxf(m, to_f32(xr[c]));
  m = block_reduce(m, MaxF{}, -CUDART_INF_F, red);
  float s = 0.f;
  for (int64_t c = threadIdx.x; c < cols; c += blockDim.x) s += exp2f((to_f32(xr[c]) - m) * kLog2e);
  s = block_reduce(s, SumF{}, 0.f, red);
  const float k = is_log ? logf(s) : 1.f / s;
  for (int64_t c = threadIdx.x; c < cols; c += blockDim.x) {
    const float d = to_f32(xr[c]) - m;
    store_from_f32(out, row * cols + c, dto, is_log ? d - k : exp2f(d * kLog2e) * k);
  }
}

// Long rows (more than the registers of a CTA hold) and rows whose start is off the 16-byte
// grid, with 16-byte accesses all the same: the CTA walks the aligned span that covers its
// row -- from `head` elements before the row's first element, inside the first element's
// own 16-byte block, to the end of the last element's block -- and masks what lies outside
// the row. Pass 1 keeps a running (max, sum of exponentials relative to it) per thread and
// merges them over the CTA; pass 2 re-reads the row (from L2 for rows up to some hundreds
// of KB), writes whole 16-byte vectors inside the row and single elements in the first and
// last block. Four vectors are in flight per thread, and one look
// at the maximum (packed max.NaN) serves all four. bf16 4096 x 50257, log: 146 us (5.6 TB/s of
// 1 read + 1 write); one vector at a time in CTAs of 1024 threads took 188. Prefetching through a
// cp.async ring gained nothing, holding the row in shared memory between the passes lost. The
// output row must sit at the same offset inside its 16-byte block as the input row and have the
// input's type. max.NaN makes a NaN element the maximum, hence the
// whole row NaN, as the three-pass kernel above does through its sum.
__device__ __forceinline__ float max_nan(float a, float b) {
  float r;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}
// the largest element of a 16-byte vector, NaN if there is one: 16-bit elements two at a time
template <typename T> __device__ __forceinline__ uint32_t max_nan_pair(uint32_t a, uint32_t b) {
  uint32_t r;
  if constexpr (std::is_same<T, __nv_bfloat16>::value) asm("max.NaN.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  else asm("max.NaN.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}
template <typename T> __device__ __forceinline__ uint32_t vec_max_word(const uint4& v) { return max_nan_pair<T>(max_nan_pair<T>(v.x, v.y), max_nan_pair<T>(v.z, v.w)); }
template <typename T> __device__ __forceinline__ float pair_max_nan(uint32_t w) {
  const T* e = reinterpret_cast<const T*>(&w);
  return max_nan(to_f32(e[0]), to_f32(e[1]));
}
template <typename T> __device__ __forceinline__ float vec_max_nan(const uint4& v) {
  if constexpr (sizeof(T) == 4) return max_nan(max_nan(__uint_as_float(v.x), __uint_as_float(v.y)), max_nan(__uint_as_float(v.z), __uint_as_float(v.w)));
  else return pair_max_nan<T>(vec_max_word<T>(v));
}
// (m, s): s = sum of 2^((x - m) log2 e) over the elements seen; m = -inf means none yet (s = 0)
__device__ __forceinline__ void online_merge(float& m, float& s, float m2, float s2) {
  const float mn = max_nan(m, m2);
  const float a = m == -CUDART_INF_F ? 0.f : s * ex2_approx((m - mn) * kLog2e);
  const float b = m2 == -CUDART_INF_F ? 0.f : s2 * ex2_approx((m2 - mn) * kLog2e);
  m = mn;
  s = a + b;
}
template <typename T> __device__ __forceinline__ uint4 vec_minus_inf() {
  const uint32_t w = sizeof(T) == 4 ? 0xff800000u : std::is_same<T, __nv_bfloat16>::value ? 0xff80ff80u : 0xfc00fc00u;
  return make_uint4(w, w, w, w);
}
template <typename T, int NV> __device__ __forceinline__ float vecs_max_nan(const uint4* v) {
  if constexpr (sizeof(T) == 4) {
    float m = vec_max_nan<T>(v[0]);
#pragma unroll
    for (int u = 1; u < NV; ++u) m = max_nan(m, vec_max_nan<T>(v[u]));
    return m;
  } else {
    uint32_t w = vec_max_word<T>(v[0]);
#pragma unroll
    for (int u = 1; u < NV; ++u) w = max_nan_pair<T>(w, vec_max_word<T>(v[u]));
    return pair_max_nan<T>(w);
  }
}
// elements f[0, N), none of them above m, into a thread's running sum
template <int N>
__device__ __forceinline__ void online_add(const float* f, float m, float& s) {
  if (fabsf(m) < 1e37f) {  // 2^(x log2e - m log2e) in one fused multiply-add per element
    const float c = m * kLog2e;
#pragma unroll
    for (int e = 0; e < N; ++e) s += ex2_approx(fmaf(f[e], kLog2e, -c));
  } else if (m != -CUDART_INF_F) {
#pragma unroll
    for (int e = 0; e < N; ++e) s += ex2_approx((f[e] - m) * kLog2e);
  }
}
__device__ __forceinline__ void online_raise(float lm, float& m, float& s) {
  const float mn = max_nan(m, lm);
  if (mn != m) {  // a new maximum (or a NaN): bring the sum so far onto it; 0 * 2^-inf when there was none
    s *= ex2_approx((m - mn) * kLog2e);
    m = mn;
  }
}
// NV whole vectors at once: one look at the maximum for all of them
template <typename T, int NV>
__device__ __forceinline__ void online_take(const uint4* v, float& m, float& s) {
  online_raise(vecs_max_nan<T, NV>(v), m, s);
#pragma unroll
  for (int u = 0; u < NV; ++u) {
    float f[Vec<T>::N];
    widen<T>(v[u], f);
    online_add<Vec<T>::N>(f, m, s);
  }
}
// a vector that reaches outside the row
template <typename T>
__device__ __forceinline__ void online_take_edge(uint4 v, int j, int head, int cols, float& m, float& s) {
  constexpr int VE = Vec<T>::N;
  float f[VE];
  widen<T>(v, f);
  const int c0 = j * VE - head;
#pragma unroll
  for (int e = 0; e < VE; ++e)
    if (c0 + e < 0 || c0 + e >= cols) f[e] = -CUDART_INF_F;
  float lm = f[0];
#pragma unroll
  for (int e = 1; e < VE; ++e) lm = max_nan(lm, f[e]);
  online_raise(lm, m, s);
  online_add<VE>(f, m, s);
}
template <typename T, bool IS_LOG, bool MASKED>
__device__ __forceinline__ void online_write(uint4 v, T* __restrict__ orow, int j, int head, int cols, float m, float k, bool fused) {
  constexpr int VE = Vec<T>::N;
  float f[VE];
  widen<T>(v, f);
  if (fused) {  // |m| < 1e37: log: x - (m + log s); softmax: 2^(x log2e - m log2e) / s
    const float c = IS_LOG ? m + k : m * kLog2e;
#pragma unroll
    for (int e = 0; e < VE; ++e) f[e] = IS_LOG ? f[e] - c : ex2_approx(fmaf(f[e], kLog2e, -c)) * k;
  } else {
#pragma unroll
    for (int e = 0; e < VE; ++e) {
      const float d = f[e] - m;
      f[e] = IS_LOG ? d - k : ex2_approx(d * kLog2e) * k;
    }
  }
  const int c0 = j * VE - head;
  if (!MASKED) {
    store_row_vec<T>(orow, c0, f, false);
  } else {
#pragma unroll
    for (int e = 0; e < VE; ++e)
      if (c0 + e >= 0 && c0 + e < cols) orow[c0 + e] = from_f32<T>(f[e]);
  }
}
template <typename T, bool IS_LOG, bool ONE_TRIP>
__global__ void __launch_bounds__(512, 3) softmax_stream_vec(const T* __restrict__ x, T* __restrict__ out, int cols) {
  constexpr int VE = Vec<T>::N;
  __shared__ float red_m[32], red_s[32];
  const int64_t row = blockIdx.x;
  const T* xr = x + row * cols;
  const int head = static_cast<int>((reinterpret_cast<uintptr_t>(xr) & 15u) / sizeof(T));
  const T* xa = xr - head;
  const int nvec = (head + cols + VE - 1) / VE;
  const int tid = threadIdx.x, nth = blockDim.x;
  const int last = nvec - 1;  // interior vectors are 1 .. last - 1: they never reach outside the row
  float m = -CUDART_INF_F, s = 0.f;
  if (tid == 0) online_take_edge<T>(ld_keep(xa), 0, head, cols, m, s);
  if (tid == 32 && nvec > 1) online_take_edge<T>(ld_keep(xa + static_cast<int64_t>(last) * VE), last, head, cols, m, s);
  int j = 1 + tid;
  if constexpr (ONE_TRIP || sizeof(T) == 4) {  // what lies behind the last interior vector counts as -inf
    for (; j < last; j += 4 * nth) {
      uint4 v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) v[u] = j + u * nth < last ? ld_keep(xa + static_cast<int64_t>(j + u * nth) * VE) : vec_minus_inf<T>();
      online_take<T, 4>(v, m, s);
      if (ONE_TRIP) break;
    }
  } else {
    for (; j + 3 * nth < last; j += 4 * nth) {
      uint4 v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) v[u] = ld_keep(xa + static_cast<int64_t>(j + u * nth) * VE);
      online_take<T, 4>(v, m, s);
    }
    for (; j < last; j += nth) {
      const uint4 v = ld_keep(xa + static_cast<int64_t>(j) * VE);
      online_take<T, 1>(&v, m, s);
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) online_merge(m, s, __shfl_xor_sync(0xffffffffu, m, o), __shfl_xor_sync(0xffffffffu, s, o));
  const int lane = tid & 31, warp = tid >> 5, nwarps = nth >> 5;
  if (lane == 0) { red_m[warp] = m; red_s[warp] = s; }
  __syncthreads();
  m = lane < nwarps ? red_m[lane] : -CUDART_INF_F;
  s = lane < nwarps ? red_s[lane] : 0.f;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) online_merge(m, s, __shfl_xor_sync(0xffffffffu, m, o), __shfl_xor_sync(0xffffffffu, s, o));
  const float k = IS_LOG ? logf(s) : 1.f / s;
  const bool fused = fabsf(m) < 1e37f && (!IS_LOG || fabsf(k) < 1e37f);
  T* orow = out + row * cols;
  if (tid == 0) online_write<T, IS_LOG, true>(ld_stream(xa), orow, 0, head, cols, m, k, fused);
  if (tid == 32 && nvec > 1) online_write<T, IS_LOG, true>(ld_stream(xa + static_cast<int64_t>(last) * VE), orow, last, head, cols, m, k, fused);
  j = 1 + tid;
  if constexpr (ONE_TRIP || sizeof(T) == 4) {
    for (; j < last; j += 4 * nth) {
      uint4 v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (j + u * nth < last) v[u] = ld_stream(xa + static_cast<int64_t>(j + u * nth) * VE);
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (j + u * nth < last) online_write<T, IS_LOG, false>(v[u], orow, j + u * nth, head, cols, m, k, fused);
      if (ONE_TRIP) break;
    }
  } else {
    for (; j + 3 * nth < last; j += 4 * nth) {
      uint4 v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) v[u] = ld_stream(xa + static_cast<int64_t>(j + u * nth) * VE);
#pragma unroll
      for (int u = 0; u < 4; ++u) online_write<T, IS_LOG, false>(v[u], orow, j + u * nth, head, cols, m, k, fused);
    }
    for (; j < last; j += nth) online_write<T, IS_LOG, false>(ld_stream(xa + static_cast<int64_t>(j) * VE), orow, j, head, cols, m, k, fused);
  }
}

// ------------------------------------------------------------------ ragged rows, one warp each
// Rows of 33 ... 32 * NPL elements whose length or base is off the 16-byte grid (the vector
// kernels cannot take them, and a CTA per row would idle most of its threads): a warp reads
// its row with coalesced scalar loads, lane l holding elements l, l + 32, ..., in registers,
// and does the same arithmetic as the resident kernels.
template <typename T, int NPL, bool IS_LOG>
__global__ void __launch_bounds__(128) softmax_warp_ragged(const T* __restrict__ x, void* __restrict__ out, int64_t rows, int cols, int dto) {
  const int lane = threadIdx.x & 31;
  const int64_t row = static_cast<int64_t>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (row >= rows) return;
  const T* xr = x + row * cols;
  float f[NPL];
  float m = -CUDART_INF_F;
#pragma unroll
  for (int i = 0; i < NPL; ++i) {
    const int c = lane + 32 * i;
    f[i] = c < cols ? to_f32(xr[c]) : -CUDART_INF_F;
    m = fmaxf(m, f[i]);
  }
  m = warp_reduce(m, MaxF{});
  float s = 0.f;
#pragma unroll
  for (int i = 0; i < NPL; ++i) {
    const float d = f[i] - m;
    const float ex = lane + 32 * i < cols ? ex2_approx(d * kLog2e) : 0.f;
    s += ex;
    f[i] = IS_LOG ? d : ex;
  }
  s = warp_reduce(s, SumF{});
  const float k = IS_LOG ? logf(s) : 1.f / s;
#pragma unroll
  for (int i = 0; i < NPL; ++i) {
    const int c = lane + 32 * i;
    if (c < cols) store_from_f32(out, row * cols + c, dto, IS_LOG ? f[i] - k : f[i] * k);
  }
}

template <typename T, int NPL>
__global__ void __launch_bounds__(128) layernorm_warp_ragged(const T* __restrict__ x, const void* __restrict__ w, const void* __restrict__ b, T* __restrict__ y, void* __restrict__ mean,
                                                             void* __restrict__ rstd, int64_t rows, int cols, float eps, int dt_wb, int dt_stat) {
  const int lane = threadIdx.x & 31;
  const int64_t row = static_cast<int64_t>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (row >= rows) return;
  const T* xr = x + row * cols;
  float f[NPL];
  float s = 0.f;
#pragma unroll
  for (int i = 0; i < NPL; ++i) {
    const int c = lane + 32 * i;
    f[i] = c < cols ? to_f32(xr[c]) : 0.f;
    s += f[i];
  }
  s = warp_reduce(s, SumF{});
  float mu = s / static_cast<float>(cols);
  if (!isfinite(mu)) mu = CUDART_NAN_F;  // same non-finite rule as the resident kernel
  float q = 0.f;
#pragma unroll
  for (int i = 0; i < NPL; ++i) {
    const float d = lane + 32 * i < cols ? f[i] - mu : 0.f;
    q = fmaf(d, d, q);
  }
  q = warp_reduce(q, SumF{});
  const float rs = rsqrtf(q / static_cast<float>(cols) + eps);
  if (lane == 0) {
    store_from_f32(mean, row, dt_stat, mu);
    store_from_f32(rstd, row, dt_stat, rs);
  }
#pragma unroll
  for (int i = 0; i < NPL; ++i) {
    const int c = lane + 32 * i;
    if (c < cols) {
      float r = (f[i] - mu) * rs;
      if (w) r *= load_as_f32(w, c, dt_wb);
      if (b) r += load_as_f32(b, c, dt_wb);
      y[row * cols + c] = from_f32<T>(r);
    }
  }
}

// NPL for a ragged row of `cols` elements: 2, 4, ..., 32 elements per lane (cols <= 1024)
#define B200_DISPATCH_NPL(COLS, BODY)                       \
  if ((COLS) <= 64) { constexpr int NPL = 2; BODY; }        \
  else if ((COLS) <= 128) { constexpr int NPL = 4; BODY; }  \
  else if ((COLS) <= 256) { constexpr int NPL = 8; BODY; }  \
  else if ((COLS) <= 512) { constexpr int NPL = 16; BODY; } \
  else { constexpr int NPL = 32; BODY; }
constexpr int kRaggedMaxCols = 1024;

// ------------------------------------------------------------------ softmax backward along a non-last dim
// [outer, dim, inner] with many columns: a CTA owns 32 words of columns (a word is one element, or
// two 16-bit ones where rows and bases allow it), its warps share `dim`, four rows in flight per
// thread in two sums; the warps' sums are added eight at a time as trees, and the second pass reads again (from L2 where it
// fits). A warp per line touches a sector per element and lane: bf16 4096 x 4096 along dim 0 327 us,
// so 44 us; fp32 1000 x 50257 890 us, so 158 us.
template <typename T, typename WORD, bool IS_LOG>
__global__ void __launch_bounds__(1024) softmax_bwd_cols_tile(const T* __restrict__ g, const T* __restrict__ y, T* __restrict__ out, int64_t dim, int64_t inner) {
  constexpr int E = sizeof(WORD) / sizeof(T), U = 4;
  __shared__ float red[32][32 * E];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  const int64_t col = (static_cast<int64_t>(blockIdx.x) * 32 + lane) * E;
  const bool in = col < inner;
  const int64_t base = static_cast<int64_t>(blockIdx.y) * dim * inner + col;
  float s2[2][E], s[E];  // even and odd rows of a trip: half the chain of additions
#pragma unroll
  for (int e = 0; e < E; ++e) s2[0][e] = s2[1][e] = 0.f;
  auto fetch = [&](const T* t, int64_t k, WORD (&v)[U]) {
#pragma unroll
    for (int u = 0; u < U; ++u) {
      v[u] = WORD{};
      if (k + u * warps < dim) v[u] = *reinterpret_cast<const WORD*>(t + base + (k + u * warps) * inner);
    }
  };
  if (in) {
    for (int64_t k = warp; k < dim; k += U * warps) {
      WORD vg[U], vy[U];
      fetch(g, k, vg);
      if (!IS_LOG) fetch(y, k, vy);
#pragma unroll
      for (int e = 0; e < E; ++e) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const float fg = to_f32(reinterpret_cast<const T*>(&vg[u])[e]);
          if (IS_LOG) s2[u & 1][e] += fg;
          else s2[u & 1][e] = fmaf(fg, to_f32(reinterpret_cast<const T*>(&vy[u])[e]), s2[u & 1][e]);
        }
      }
    }
  }
#pragma unroll
  for (int e = 0; e < E; ++e) red[warp][e * 32 + lane] = s2[0][e] + s2[1][e];
  __syncthreads();
  if (!in) return;
#pragma unroll
  for (int e = 0; e < E; ++e) {
    const float* r = &red[0][e * 32 + lane];
    constexpr int P = 32 * E;
    s[e] = 0.f;
    for (int w = 0; w < warps; w += 8) {  // (a warp that is not there adds nothing)
      float f[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) f[q] = w + q < warps ? r[(w + q) * P] : 0.f;
      s[e] += tree_sum<8>(f);
    }
  }
  for (int64_t k = warp; k < dim; k += U * warps) {
    WORD vg[U], vy[U];
    fetch(g, k, vg);
    fetch(y, k, vy);
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (k + u * warps >= dim) break;
      WORD r;
#pragma unroll
      for (int e = 0; e < E; ++e) {
        const float fg = to_f32(reinterpret_cast<const T*>(&vg[u])[e]), fy = to_f32(reinterpret_cast<const T*>(&vy[u])[e]);
        reinterpret_cast<T*>(&r)[e] = from_f32<T>(IS_LOG ? fg - ex2_approx(fy * kLog2e) * s[e] : (fg - s[e]) * fy);
      }
      __stcs(reinterpret_cast<WORD*>(out + base + (k + u * warps) * inner), r);
    }
  }
}
// Two 16-bit columns per lane where every row and base is on the 4-byte grid and 32 lanes still
// find columns.
template <typename T>
static bool cols_in_pairs(int64_t inner, const void* a, const void* b, const void* c) {
  return sizeof(T) == 2 && inner % 2 == 0 && inner >= 64 && ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b) | reinterpret_cast<uintptr_t>(c)) & 3u) == 0;
}
static int cols_tile_threads(int64_t dim, int64_t ctas) {
  // four rows to a warp; with two CTAs for every SM sixteen warps to each, else all a CTA can have
  const int most = ctas >= 2 * kNumSMs ? 16 : 32;
  int warps = 1;
  while (warps < most && warps * 4 < dim) warps <<= 1;
  return 32 * warps;
}

// ------------------------------------------------------------------ softmax, inner > 1
template <typename T>
__global__ void __launch_bounds__(128) softmax_cols(const T* __restrict__ x, void* __restrict__ out, int64_t dim, int64_t inner, int dto, int is_log) {
  const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= inner) return;
  const int64_t base = static_cast<int64_t>(blockIdx.y) * dim * inner + i;
  float m = -CUDART_INF_F;
  for (int64_t k = 0; k < dim; ++k) m = fmaxf(m, to_f32(x[base + k * inner]));
  float s = 0.f;
  for (int64_t k = 0; k < dim; ++k) s += exp2f((to_f32(x[base + k * inner]) - m) * kLog2e);
  const float kk = is_log ? logf(s) : 1.f / s;
  for (int64_t k = 0; k < dim; ++k) {
    const float d = to_f32(x[base + k * inner]) - m;
    store_from_f32(out, base + k * inner, dto, is_log ? d - kk : exp2f(d * kLog2e) * kk);
  }
}

// ------------------------------------------------------------------ layer norm, resident
// HOLD: the row is widened to fp32 once and held in registers (VE floats per vector);
// otherwise it stays in its storage type (16 bytes per vector) and is widened again in
// each of the three passes, which for 16-bit rows halves the registers held across the two
// reductions. AFFINE: weight and bias are both present (the usual call), so the last pass
// is one fused multiply-add per element with no per-element tests.
template <typename T, typename TW, int VPT, bool WARP, bool HOLD, bool AFFINE>
__global__ void __launch_bounds__(WARP ? 128 : 1024)
layernorm_resident(const T* __restrict__ x, const TW* __restrict__ w, const TW* __restrict__ b, T* __restrict__ y,
                   void* __restrict__ mean, void* __restrict__ rstd, int64_t rows, int cols, float inv_cols, float eps, int dt_stat) {
  constexpr int VE = Vec<T>::N;
  __shared__ float red[64];
  const int tpr = WARP ? 32 : blockDim.x;
  const int t = WARP ? (threadIdx.x & 31) : threadIdx.x;
  const int64_t row = WARP ? static_cast<int64_t>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5) : blockIdx.x;
  if (WARP && row >= rows) return;
  const int nvec = cols / VE;
  const T* xr = x + row * cols;
  T* yr = y + row * cols;
  uint4 raw[HOLD ? 1 : VPT];
  float f[HOLD ? VPT : 1][VE];
  float s = 0.f;
  if (HOLD) {
#pragma unroll
    for (int u = 0; u < VPT; ++u) {
      const int j = t + u * tpr;
      if (j < nvec) {
        widen<T>(ld_stream(xr + j * VE), f[HOLD ? u : 0]);
#pragma unroll
        for (int e = 0; e < VE; ++e) s += f[HOLD ? u : 0][e];
      }
    }
  } else {
#pragma unroll
    for (int u = 0; u < VPT; ++u) {
      const int j = t + u * tpr;
      if (j < nvec) raw[HOLD ? 0 : u] = ld_stream(xr + j * VE);
    }
#pragma unroll
    for (int u = 0; u < VPT; ++u) {
      if (t + u * tpr < nvec) vec_accumulate<T>(s, raw[HOLD ? 0 : u]);
    }
  }
  s = group_reduce<WARP>(s, SumF{}, 0.f, red, 0);
  float mu = s * inv_cols;
  // a row holding NaN or inf has NaN statistics in aten (its running moments turn inf
  // into NaN once another element follows), not mean = inf
  if (!isfinite(mu)) mu = CUDART_NAN_F;
  float q = 0.f;
#pragma unroll
  for (int u = 0; u < VPT; ++u) {
    if (t + u * tpr < nvec) {
      float d[VE];
      if (HOLD) {
#pragma unroll
        for (int e = 0; e < VE; ++e) d[e] = f[HOLD ? u : 0][e] - mu;
      } else {
        vec_minus<T>(raw[HOLD ? 0 : u], mu, d);
      }
#pragma unroll
      for (int e = 0; e < VE; ++e) q = fmaf(d[e], d[e], q);
    }
  }
  q = group_reduce<WARP>(q, SumF{}, 0.f, red, 1);
  const float rs = rsqrtf(fmaf(q, inv_cols, eps));
  if (t == 0) {
    store_from_f32(mean, row, dt_stat, mu);
    store_from_f32(rstd, row, dt_stat, rs);
  }
#pragma unroll
  for (int u = 0; u < VPT; ++u) {
    const int j = t + u * tpr;
    if (j < nvec) {
      float o[VE], wv[VE], bv[VE], d[VE];
      if (HOLD) {
#pragma unroll
        for (int e = 0; e < VE; ++e) d[e] = f[HOLD ? u : 0][e] - mu;
      } else {
        vec_minus<T>(raw[HOLD ? 0 : u], mu, d);
      }
      if (AFFINE || w) load_weights<VE, TW>(w, j * VE, wv);
      if (AFFINE || b) load_weights<VE, TW>(b, j * VE, bv);
#pragma unroll
      for (int e = 0; e < VE; ++e) {
        float r = d[e] * rs;
        if (AFFINE) {
          r = fmaf(r, wv[e], bv[e]);
        } else {
          if (w) r *= wv[e];
          if (b) r += bv[e];
        }
        o[e] = r;
      }
      st_stream(yr + j * VE, narrow<T>(o));
    }
  }
}

// The same for many 16-bit rows with weight and bias: persistent CTAs. A thread owns the same
// columns of every row its CTA sees, so it widens its share of weight and bias ONCE (the
// per-row kernel above fetched and unpacked 16 KB of them for every 8 KB row: two of its
// eighteen instructions per element, and more L2-to-SM traffic than the rows themselves), and
// the next row's vectors are requested before this row's two reductions.
template <typename T, typename TW, int VPT>
__global__ void __launch_bounds__(256, 4)
layernorm_persistent(const T* __restrict__ x, const TW* __restrict__ w, const TW* __restrict__ b, T* __restrict__ y, void* __restrict__ mean, void* __restrict__ rstd, int64_t rows, int cols,
                     float inv_cols, float eps, int dt_stat) {
  constexpr int VE = Vec<T>::N;
  __shared__ float red[64];
  const int t = threadIdx.x, tpr = blockDim.x;
  const int nvec = cols / VE;
  float wv[VPT][VE], bv[VPT][VE];
#pragma unroll
  for (int u = 0; u < VPT; ++u) {
    const int j = t + u * tpr;
    if (j < nvec) {
      load_weights<VE, TW>(w, j * VE, wv[u]);
      load_weights<VE, TW>(b, j * VE, bv[u]);
    }
  }
  uint4 nxt[VPT];
  int64_t row = blockIdx.x;
  if (row < rows) {
#pragma unroll
    for (int u = 0; u < VPT; ++u) {
      const int j = t + u * tpr;
      if (j < nvec) nxt[u] = ld_stream(x + row * cols + j * VE);
    }
  }
  for (; row < rows; row += gridDim.x) {
    // the row stays packed (16 bytes per vector) and is widened again in each of the three
    // passes: held as fp32 it costs a CTA per SM (three instead of four) and ran 7 % slower
    uint4 raw[VPT];
#pragma unroll
    for (int u = 0; u < VPT; ++u) raw[u] = nxt[u];
    const int64_t nrow = row + gridDim.x;
    if (nrow < rows) {
#pragma unroll
      for (int u = 0; u < VPT; ++u) {
        const int j = t + u * tpr;
        if (j < nvec) nxt[u] = ld_stream(x + nrow * cols + j * VE);
      }
    }
    float s = 0.f;
#pragma unroll
    for (int u = 0; u < VPT; ++u)
      if (t + u * tpr < nvec) vec_accumulate<T>(s, raw[u]);
    s = block_reduce_once(s, SumF{}, 0.f, red, 0);
    float mu = s * inv_cols;
    if (!isfinite(mu)) mu = CUDART_NAN_F;  // as the per-row kernel: NaN statistics for a row holding NaN or inf
    float q = 0.f;
#pragma unroll
    for (int u = 0; u < VPT; ++u) {
      if (t + u * tpr < nvec) {
        float d[VE];
        vec_minus<T>(raw[u], mu, d);
#pragma unroll
        for (int e = 0; e < VE; ++e) q = fmaf(d[e], d[e], q);
      }
    }
    q = block_reduce_once(q, SumF{}, 0.f, red, 1);
    const float rs = rsqrtf(fmaf(q, inv_cols, eps));
    if (t == 0) {
      store_from_f32(mean, row, dt_stat, mu);
      store_from_f32(rstd, row, dt_stat, rs);
    }
#pragma unroll
    for (int u = 0; u < VPT; ++u) {
      const int j = t + u * tpr;
      if (j < nvec) {
        float d[VE], o[VE];
        vec_minus<T>(raw[u], mu, d);
#pragma unroll
        for (int e = 0; e < VE; ++e) o[e] = fmaf(d[e] * rs, wv[u][e], bv[u][e]);
        st_stream(y + row * cols + j * VE, narrow<T>(o));
      }
    }
  }
}

// ------------------------------------------------------------------ layer norm backward
// aten.native_layer_norm_backward: with xhat = (x - mean) * rstd and gy = dy * w per row,
//   dx = rstd * (gy - mean_j(gy) - xhat * mean_j(gy * xhat))
//   dw = sum_rows dy * xhat,  db = sum_rows dy.
// Fused kernel (row length a multiple of the 16-byte vector, everything aligned): persistent
// CTAs, one row at a time per CTA; a thread owns the same columns of every row it sees, so it
// carries its share of dw / db in registers across rows and writes one partial per CTA at
// the end (dy and x are read once for all three results). A small second kernel adds the
// per-CTA partials in order. fp32 arithmetic throughout. bf16 8192 x 4096: 53.7 -> 51.3 us with both sums behind one barrier
// and the row statistics fetched ahead; bound by its instructions (two CTAs of 512 threads on an SM, half of the issue
// slots busy, and 20 % more instructions were 20 % more time), so two elements to an instruction (P, below), a shuffle per level for both sums,
// and the partial sums stored 16 bytes at a time: 54 -> 44.6 us the call with its second kernel. Tried: a ring of four rows in shared
// memory (`cp.async`) in place of the one row in registers (52.4 for 51.3); the row before finished behind the next row's sums,
// so that nothing waits right after a barrier (64.9 for 54.3); two to eight rows to a CTA of 512 threads, fewer partial sums, behind
// barriers of their own (30000 x 768 49.7 for 38.5).
template <typename T, typename TW, int VPT, bool kAhead>
__global__ void __launch_bounds__(1024)
layernorm_bwd_fused(const T* __restrict__ dy, const T* __restrict__ x, const TW* __restrict__ w, const void* __restrict__ mean, const void* __restrict__ rstd, T* __restrict__ dx,
                    float* __restrict__ part_w, float* __restrict__ part_b, int64_t rows, int cols, int dt_stat) {
  constexpr int VE = Vec<T>::N, VP = VE / 2;
  typedef typename std::conditional<sizeof(T) == 2, F2, TwoF>::type P;  // (fp32 8192 x 4096, bound by memory: 74 us, 80 with F2)
  __shared__ float red[2][2][32];  // [row parity][sum][warp]
  const int t = threadIdx.x, tpr = blockDim.x;
  const int nvec = cols / VE;
  const float inv_cols = 1.f / static_cast<float>(cols);
  P wv[VPT][VP], aw[VPT][VP], ab[VPT][VP];  // (pairs: half the instructions of what bounds this)
#pragma unroll
  for (int u = 0; u < VPT; ++u) {
    const int j = t + u * tpr;
    float wf[VE];
#pragma unroll
    for (int e = 0; e < VE; ++e) wf[e] = 1.f;
    if (w && j < nvec) load_weights<VE, TW>(w, j * VE, wf);
#pragma unroll
    for (int e = 0; e < VP; ++e) {
      wv[u][e] = P::of(wf[2 * e], wf[2 * e + 1]);
      aw[u][e] = ab[u][e] = P::of(0.f, 0.f);
    }
  }
  // the vectors of the next row are requested before this row is worked on: twice the bytes in flight per thread
  uint4 ndy[VPT], nx[VPT];
  float nmu = 0.f, nrs = 0.f;
  if (static_cast<int64_t>(blockIdx.x) < rows) {
    if (kAhead) {
      nmu = load_as_f32(mean, blockIdx.x, dt_stat);
      nrs = load_as_f32(rstd, blockIdx.x, dt_stat);
    }
#pragma unroll
    for (int u = 0; u < VPT; ++u) {
      const int j = t + u * tpr;
      if (j < nvec) {
        ndy[u] = ld_stream(dy + static_cast<int64_t>(blockIdx.x) * cols + j * VE);
        nx[u] = ld_stream(x + static_cast<int64_t>(blockIdx.x) * cols + j * VE);
      }
    }
  }
  int phase = 0;
  for (int64_t row = blockIdx.x; row < rows; row += gridDim.x, phase ^= 1) {
    // (without kAhead: many small CTAs per SM hide these loads by themselves)
    const float mu = kAhead ? nmu : load_as_f32(mean, row, dt_stat), rs = kAhead ? nrs : load_as_f32(rstd, row, dt_stat);
    const P rs2 = P::of(rs, rs);
    P g[VPT][VP], h[VPT][VP];  // dy, then dy * w; x - mean, then xhat
#pragma unroll
    for (int u = 0; u < VPT; ++u) {
      float gf[VE], hf[VE];
      widen<T>(ndy[u], gf);
      vec_minus<T>(nx[u], mu, hf);  // (16 bits: widened inside the subtraction)
#pragma unroll
      for (int e = 0; e < VP; ++e) {
        g[u][e] = P::of(gf[2 * e], gf[2 * e + 1]);
        h[u][e] = P::of(hf[2 * e], hf[2 * e + 1]);
      }
    }
    const int64_t next = row + gridDim.x;
    if (next < rows) {
      if (kAhead) {
        nmu = load_as_f32(mean, next, dt_stat);
        nrs = load_as_f32(rstd, next, dt_stat);
      }
#pragma unroll
      for (int u = 0; u < VPT; ++u) {
        const int j = t + u * tpr;
        if (j < nvec) {
          ndy[u] = ld_stream(dy + next * cols + j * VE);
          nx[u] = ld_stream(x + next * cols + j * VE);
        }
      }
    }
    P p1 = P::of(0.f, 0.f), p2 = p1;
#pragma unroll
    for (int u = 0; u < VPT; ++u) {
      if (t + u * tpr < nvec) {
#pragma unroll
        for (int e = 0; e < VP; ++e) {
          h[u][e] = p_mul(h[u][e], rs2);
          ab[u][e] = p_add(ab[u][e], g[u][e]);
          aw[u][e] = p_fma(g[u][e], h[u][e], aw[u][e]);
          g[u][e] = p_mul(g[u][e], wv[u][e]);
          p1 = p_add(p1, g[u][e]);
          p2 = p_fma(g[u][e], h[u][e], p2);
        }
      }
    }
    float s1, s2, other;
    p_parts(p1, s1, other);
    s1 += other;
    p_parts(p2, s2, other);
    s2 += other;
    if constexpr (kAhead) {
      // both sums behind one barrier; the row after next is the first to write these slots again. The lower half
      // of a warp goes on with the first sum, the upper with the second.
      const int half = (t & 31) >> 4;
      float s = (half ? s2 : s1) + __shfl_xor_sync(0xffffffffu, half ? s1 : s2, 16);
#pragma unroll
      for (int d = 8; d > 0; d >>= 1) s += __shfl_xor_sync(0xffffffffu, s, d);
      if ((t & 15) == 0) red[phase][half][t >> 5] = s;
      __syncthreads();
      s = 0.f;
      for (int k = t & 15; k < (tpr >> 5); k += 16) s += red[phase][half][k];
#pragma unroll
      for (int d = 8; d > 0; d >>= 1) s += __shfl_xor_sync(0xffffffffu, s, d);
      other = __shfl_xor_sync(0xffffffffu, s, 16);
      s1 = half ? other : s;
      s2 = half ? s : other;
    } else {  // (one after the other where the CTAs are small and many: fp32 65536 x 1024 144 us, 153 us behind one barrier)
      s1 = block_reduce_once(s1, SumF{}, 0.f, &red[0][0][0], 0);
      s2 = block_reduce_once(s2, SumF{}, 0.f, &red[0][0][0], 1);
    }
    const P m1 = P::of(-s1 * inv_cols, -s1 * inv_cols), m2 = P::of(-s2 * inv_cols, -s2 * inv_cols);
    if (dx) {
#pragma unroll
      for (int u = 0; u < VPT; ++u) {
        const int j = t + u * tpr;
        if (j < nvec) {
          float o[VE];
#pragma unroll
          for (int e = 0; e < VP; ++e) p_parts(p_mul(rs2, p_fma(h[u][e], m2, p_add(g[u][e], m1))), o[2 * e], o[2 * e + 1]);
          st_stream(dx + row * cols + j * VE, narrow<T>(o));
        }
      }
    }
  }
  if (part_w) {
    // (16 bytes at a time: a word at a time, 32 bytes apart over a warp, bf16 1000 x 4096 took 20.5 us, 13.1 so, 8192 x 4096 51 and 45. fp32
    // sums would have to lie in registers in fours all through the loop, which spills: 8192 x 4096 73 us, 82)
#pragma unroll
    for (int u = 0; u < VPT; ++u) {
      const int j = t + u * tpr;
      if (j < nvec) {
        float pw[VE], pb[VE];
#pragma unroll
        for (int e = 0; e < VP; ++e) {
          p_parts(aw[u][e], pw[2 * e], pw[2 * e + 1]);
          p_parts(ab[u][e], pb[2 * e], pb[2 * e + 1]);
        }
        float* to_w = part_w + static_cast<int64_t>(blockIdx.x) * cols + j * VE;
        float* to_b = part_b + static_cast<int64_t>(blockIdx.x) * cols + j * VE;
        if constexpr (sizeof(T) == 2) {
#pragma unroll
          for (int e = 0; e < VE; e += 4) {
            *reinterpret_cast<float4*>(to_w + e) = make_float4(pw[e], pw[e + 1], pw[e + 2], pw[e + 3]);
            *reinterpret_cast<float4*>(to_b + e) = make_float4(pb[e], pb[e + 1], pb[e + 2], pb[e + 3]);
          }
        } else {
#pragma unroll
          for (int e = 0; e < VE; ++e) {
            to_w[e] = pw[e];
            to_b[e] = pb[e];
          }
        }
      }
    }
  }
}

// ------------------------------------------------------------------ layer norm, rows off the 16-byte grid
// A row is dealt out in chunks of E elements, the largest that every row starts on: one, two (16-bit rows
// of even length), or a whole vector.
template <typename T, int E> struct RowChunk;  // a chunk as it is loaded
template <typename T> struct RowChunk<T, 1> {
  T raw;
  __device__ __forceinline__ void load(const T* p) { raw = __ldcs(p); }
  __device__ __forceinline__ void widen_to(float* f) const { f[0] = to_f32(raw); }
  static __device__ __forceinline__ void store(T* p, const float* f) { __stcs(p, from_f32<T>(f[0])); }
};
template <typename T> struct RowChunk<T, 2> {
  uint32_t raw;
  __device__ __forceinline__ void load(const T* p) { raw = __ldcs(reinterpret_cast<const uint32_t*>(p)); }
  __device__ __forceinline__ void widen_to(float* f) const {
    const T* e = reinterpret_cast<const T*>(&raw);
    f[0] = to_f32(e[0]);
    f[1] = to_f32(e[1]);
  }
  static __device__ __forceinline__ void store(T* p, const float* f) {
    const T e[2] = {from_f32<T>(f[0]), from_f32<T>(f[1])};
    __stcs(reinterpret_cast<uint32_t*>(p), *reinterpret_cast<const uint32_t*>(e));
  }
};
template <typename T> struct RowVector {
  uint4 raw;
  __device__ __forceinline__ void load(const T* p) { raw = ld_stream(p); }
  __device__ __forceinline__ void widen_to(float* f) const { widen<T>(raw, f); }
  static __device__ __forceinline__ void store(T* p, const float* f) { st_stream(p, narrow<T>(f)); }
};
template <> struct RowChunk<float, 4> : RowVector<float> {};
template <> struct RowChunk<__nv_bfloat16, 8> : RowVector<__nv_bfloat16> {};
template <> struct RowChunk<__half, 8> : RowVector<__half> {};

// Forward, a CTA to a row, which stays in registers as fp32. Three scalar passes over it (`layernorm_stream`)
// took bf16 12544 x 2934 192 us, 56 so; fp32 8000 x 8191 356 and 138.
template <typename T, typename TW, int E, int NPT>
__global__ void __launch_bounds__(1024) layernorm_rows(const T* __restrict__ x, const TW* __restrict__ w, const TW* __restrict__ b, T* __restrict__ y, void* __restrict__ mean, void* __restrict__ rstd, int cols,
                                                       float eps, int dt_stat) {
  __shared__ float red[64];
  const int64_t row = blockIdx.x;
  const int t = threadIdx.x, tpr = blockDim.x, chunks = cols / E;
  const T* xr = x + row * cols;
  RowChunk<T, E> raw[NPT];
  float f[NPT][E], s = 0.f;
#pragma unroll
  for (int u = 0; u < NPT; ++u)
    if (t + u * tpr < chunks) raw[u].load(xr + (t + u * tpr) * E);
#pragma unroll
  for (int u = 0; u < NPT; ++u) {
#pragma unroll
    for (int e = 0; e < E; ++e) f[u][e] = 0.f;
    if (t + u * tpr < chunks) raw[u].widen_to(f[u]);
#pragma unroll
    for (int e = 0; e < E; ++e) s += f[u][e];
  }
  s = block_reduce_once(s, SumF{}, 0.f, red, 0);
  float mu = s / static_cast<float>(cols);
  if (!isfinite(mu)) mu = CUDART_NAN_F;  // same non-finite rule as the resident kernel
  float q = 0.f;
#pragma unroll
  for (int u = 0; u < NPT; ++u)
    if (t + u * tpr < chunks) {
#pragma unroll
      for (int e = 0; e < E; ++e) {
        f[u][e] -= mu;
        q = fmaf(f[u][e], f[u][e], q);
      }
    }
  q = block_reduce_once(q, SumF{}, 0.f, red, 1);
  const float rs = rsqrtf(q / static_cast<float>(cols) + eps);
  if (t == 0) {
    store_from_f32(mean, row, dt_stat, mu);
    store_from_f32(rstd, row, dt_stat, rs);
  }
#pragma unroll
  for (int u = 0; u < NPT; ++u) {
    const int c = (t + u * tpr) * E;
    if (t + u * tpr < chunks) {
      float o[E];
#pragma unroll
      for (int e = 0; e < E; ++e) {
        o[e] = f[u][e] * rs;
        if (w) o[e] *= to_f32(w[c + e]);
        if (b) o[e] += to_f32(b[c + e]);
      }
      RowChunk<T, E>::store(y + row * cols + c, o);
    }
  }
}

// Backward, as layernorm_bwd_fused: persistent, the next row on its way, dw and db in registers across rows. A row is a
// CTA's, or, up to 256 elements, a warp's: eight warps of a CTA then add up their shares of dw and db one
// after the other before they go out, so that short rows fill an SM without many partial rows (a CTA of one warp each, eight to an SM: bf16 20000 x 256
// 29.8 -> 14.3 us). Ragged rows, in three passes for dx and by columns for dw and db until now: bf16 12544 x 2934 510 -> 75, f16 29952 x 60
// 240 -> 13.4, fp32 65536 x 33 449 -> 17.6.
template <typename T, int E, int NPT, bool WARP>
__global__ void __launch_bounds__(WARP ? 256 : 1024)
layernorm_bwd_rows(const T* __restrict__ dy, const T* __restrict__ x, const void* __restrict__ w, const void* __restrict__ mean, const void* __restrict__ rstd, T* __restrict__ dx,
                   float* __restrict__ part_w, float* __restrict__ part_b, int64_t rows, int cols, int dt_wb, int dt_stat) {
  __shared__ float2 red[2][32];
  __shared__ float share[WARP ? 2 * 32 * NPT * E : 1];
  const int t = WARP ? threadIdx.x & 31 : threadIdx.x, tpr = WARP ? 32 : blockDim.x, chunks = cols / E;
  const int64_t row0 = WARP ? static_cast<int64_t>(blockIdx.x) * 8 + (threadIdx.x >> 5) : blockIdx.x, step = static_cast<int64_t>(gridDim.x) * (WARP ? 8 : 1);
  const float inv_cols = 1.f / static_cast<float>(cols);
  float wv[NPT][E], aw[NPT][E], ab[NPT][E];
#pragma unroll
  for (int u = 0; u < NPT; ++u) {
    const int j = t + u * tpr;
#pragma unroll
    for (int e = 0; e < E; ++e) {
      aw[u][e] = ab[u][e] = 0.f;
      wv[u][e] = w && j < chunks ? load_as_f32(w, j * E + e, dt_wb) : 1.f;
    }
  }
  RowChunk<T, E> ndy[NPT], nx[NPT];
  float nmu = 0.f, nrs = 0.f;
  auto request = [&](int64_t row) {
    nmu = load_as_f32(mean, row, dt_stat);
    nrs = load_as_f32(rstd, row, dt_stat);
#pragma unroll
    for (int u = 0; u < NPT; ++u) {
      const int j = t + u * tpr;
      if (j < chunks) {
        ndy[u].load(dy + row * cols + j * E);
        nx[u].load(x + row * cols + j * E);
      }
    }
  };
  if (row0 < rows) request(row0);
  int phase = 0;
  for (int64_t row = row0; row < rows; row += step, phase ^= 1) {
    const float mu = nmu, rs = nrs;
    float g[NPT][E], h[NPT][E], s1 = 0.f, s2 = 0.f;
#pragma unroll
    for (int u = 0; u < NPT; ++u) {
      ndy[u].widen_to(g[u]);
      nx[u].widen_to(h[u]);
    }
    if (row + step < rows) request(row + step);
#pragma unroll
    for (int u = 0; u < NPT; ++u)
      if (t + u * tpr < chunks) {
#pragma unroll
        for (int e = 0; e < E; ++e) {
          const float xhat = (h[u][e] - mu) * rs;
          ab[u][e] += g[u][e];
          aw[u][e] = fmaf(g[u][e], xhat, aw[u][e]);
          const float gy = g[u][e] * wv[u][e];
          s1 += gy;
          s2 = fmaf(gy, xhat, s2);
          g[u][e] = gy;
          h[u][e] = xhat;
        }
      }
    s1 = warp_reduce(s1, SumF{});
    s2 = warp_reduce(s2, SumF{});
    if constexpr (!WARP) {  // both sums behind one barrier; the row after next is the first to write these slots again
      if ((t & 31) == 0) red[phase][t >> 5] = make_float2(s1, s2);
      __syncthreads();
      const float2 part = (t & 31) < (tpr >> 5) ? red[phase][t & 31] : make_float2(0.f, 0.f);
      s1 = warp_reduce(part.x, SumF{});
      s2 = warp_reduce(part.y, SumF{});
    }
    const float c1 = s1 * inv_cols, c2 = s2 * inv_cols;
    if (dx) {
#pragma unroll
      for (int u = 0; u < NPT; ++u)
        if (t + u * tpr < chunks) {
          float o[E];
#pragma unroll
          for (int e = 0; e < E; ++e) o[e] = rs * (g[u][e] - c1 - h[u][e] * c2);
          RowChunk<T, E>::store(dx + row * cols + (t + u * tpr) * E, o);
        }
    }
  }
  if (!part_w) return;
  if constexpr (WARP) {
    constexpr int kShare = 32 * NPT * E;
    for (int k = 0; k < 8; ++k) {
      if (static_cast<int>(threadIdx.x >> 5) == k) {
#pragma unroll
        for (int u = 0; u < NPT; ++u) {
#pragma unroll
          for (int e = 0; e < E; ++e) {
            const int i = (u * E + e) * 32 + t;
            share[i] = k ? share[i] + aw[u][e] : aw[u][e];
            share[kShare + i] = k ? share[kShare + i] + ab[u][e] : ab[u][e];
          }
        }
      }
      __syncthreads();
    }
    if (threadIdx.x >= 32) return;
#pragma unroll
    for (int u = 0; u < NPT; ++u) {
#pragma unroll
      for (int e = 0; e < E; ++e) {
        aw[u][e] = share[(u * E + e) * 32 + t];
        ab[u][e] = share[kShare + (u * E + e) * 32 + t];
      }
    }
  }
#pragma unroll
  for (int u = 0; u < NPT; ++u) {
    const int j = t + u * tpr;
    if (j < chunks) {
#pragma unroll
      for (int e = 0; e < E; ++e) {
        part_w[static_cast<int64_t>(blockIdx.x) * cols + j * E + e] = aw[u][e];
        part_b[static_cast<int64_t>(blockIdx.x) * cols + j * E + e] = ab[u][e];
      }
    }
  }
}

// Any row length and alignment. dx: one CTA per row, scalar, three passes (the second and
// third from cache). dw / db partials: one thread per column walking a chunk of rows
// (coalesced across columns), one partial row per chunk.
__global__ void __launch_bounds__(256) layernorm_bwd_dx_lines(const void* __restrict__ dy, const void* __restrict__ x, const void* __restrict__ w, const void* __restrict__ mean,
                                                              const void* __restrict__ rstd, void* __restrict__ dx, int64_t rows, int64_t cols, int dt, int dt_wb, int dt_stat) {
  __shared__ float red[64];
  for (int64_t row = blockIdx.x; row < rows; row += gridDim.x) {
    const float mu = load_as_f32(mean, row, dt_stat), rs = load_as_f32(rstd, row, dt_stat);
    const int64_t base = row * cols;
    float s1 = 0.f, s2 = 0.f;
    for (int64_t c = threadIdx.x; c < cols; c += blockDim.x) {
      const float gy = load_as_f32(dy, base + c, dt) * (w ? load_as_f32(w, c, dt_wb) : 1.f);
      s1 += gy;
      s2 = fmaf(gy, (load_as_f32(x, base + c, dt) - mu) * rs, s2);
    }
    __syncthreads();  // the reduction buffers of the row before are free
    s1 = block_reduce_once(s1, SumF{}, 0.f, red, 0);
    s2 = block_reduce_once(s2, SumF{}, 0.f, red, 1);
    const float c1 = s1 / static_cast<float>(cols), c2 = s2 / static_cast<float>(cols);
    for (int64_t c = threadIdx.x; c < cols; c += blockDim.x) {
      const float gy = load_as_f32(dy, base + c, dt) * (w ? load_as_f32(w, c, dt_wb) : 1.f);
      const float xhat = (load_as_f32(x, base + c, dt) - mu) * rs;
      store_from_f32(dx, base + c, dt, rs * (gy - c1 - xhat * c2));
    }
  }
}
__global__ void __launch_bounds__(256) layernorm_bwd_wb_lines(const void* __restrict__ dy, const void* __restrict__ x, const void* __restrict__ mean, const void* __restrict__ rstd,
                                                              float* __restrict__ part_w, float* __restrict__ part_b, int64_t rows, int64_t cols, int64_t rows_per, int dt, int dt_stat) {
  const int64_t c = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (c >= cols) return;
  const int64_t r0 = static_cast<int64_t>(blockIdx.y) * rows_per, r1 = r0 + rows_per < rows ? r0 + rows_per : rows;
  float aw = 0.f, ab = 0.f;
  for (int64_t r = r0; r < r1; ++r) {
    const float g = load_as_f32(dy, r * cols + c, dt);
    ab += g;
    aw = fmaf(g, (load_as_f32(x, r * cols + c, dt) - load_as_f32(mean, r, dt_stat)) * load_as_f32(rstd, r, dt_stat), aw);
  }
  part_w[static_cast<int64_t>(blockIdx.y) * cols + c] = aw;
  part_b[static_cast<int64_t>(blockIdx.y) * cols + c] = ab;
}
// dw[c] = sum over the `parts` partial rows, same for db: a CTA takes W columns, its 1024 / W rows of threads the partial
// rows in turn; their sums are added in order. 32 columns (whole lines) where that makes enough CTAs, else 8, a sector:
// bf16 2000 x 600, 1184 partial rows, 16.9 us the call with 32 columns to a CTA, 12.2 with 8.
template <int W>
__global__ void __launch_bounds__(1024) layernorm_bwd_finalize(const float* part_w, const float* part_b, void* __restrict__ dw, void* __restrict__ db, int64_t parts,
                                                               int64_t cols, int dt_wb) {
  constexpr int R = 1024 / W;
  __shared__ float sw[R][W + 1], sb[R][W + 1];
  const int tx = threadIdx.x % W, ty = threadIdx.x / W;
  const int64_t c = static_cast<int64_t>(blockIdx.x) * W + tx;
  float aw = 0.f, ab = 0.f;
  after_grids_before();
  if (c < cols && parts <= R) {
    if (ty < parts) {
      aw = part_w[ty * cols + c];
      ab = part_b[ty * cols + c];
    }
  } else if (c < cols) {
    constexpr int U = 8;  // partial rows on the way (one after the other 1184 of 112 columns took 14.5 us)
    for (int64_t p0 = ty; p0 < parts; p0 += R * U) {
      float w[U], b[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int64_t p = p0 + R * u;
        w[u] = p < parts ? part_w[p * cols + c] : 0.f;
        b[u] = p < parts ? part_b[p * cols + c] : 0.f;
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        aw += w[u];
        ab += b[u];
      }
    }
  }
  sw[ty][tx] = aw;
  sb[ty][tx] = ab;
  __syncthreads();
  // the first 32 rows of threads add up R / 32 sums each, the first row what these leave
  if constexpr (R > 32) {
    if (ty < 32) {
#pragma unroll
      for (int k = 1; k < R / 32; ++k) {
        aw += sw[ty + 32 * k][tx];
        ab += sb[ty + 32 * k][tx];
      }
      sw[ty][tx] = aw;
      sb[ty][tx] = ab;
    }
    __syncthreads();
  }
  if (ty == 0 && c < cols) {
    float tw = 0.f, tb = 0.f;
#pragma unroll
    for (int k = 0; k < 32; ++k) {
      tw += sw[k][tx];
      tb += sb[k][tx];
    }
    if (dw) store_from_f32(dw, c, dt_wb, tw);
    if (db) store_from_f32(db, c, dt_wb, tb);
  }
}

// layer norm, streaming: one CTA per row, three scalar passes (second and third from L2).
__global__ void __launch_bounds__(256) layernorm_stream(const void* __restrict__ x, const void* __restrict__ w, const void* __restrict__ b, void* __restrict__ y,
                                                        void* __restrict__ mean, void* __restrict__ rstd, int64_t cols, float eps, int dt, int dt_wb, int dt_stat) {
  __shared__ float red[33];
  const int64_t row = blockIdx.x, base = row * cols;
  float s = 0.f;
  for (int64_t c = threadIdx.x; c < cols; c += blockDim.x) s += load_as_f32(x, base + c, dt);
  s = block_reduce(s, SumF{}, 0.f, red);
  float mu = s / static_cast<float>(cols);
  if (!isfinite(mu)) mu = CUDART_NAN_F;  // same non-finite rule as the resident kernel
  float q = 0.f;
  for (int64_t c = threadIdx.x; c < cols; c += blockDim.x) {
    const float d = load_as_f32(x, base + c, dt) - mu;
    q = fmaf(d, d, q);
  }
  q = block_reduce(q, SumF{}, 0.f, red);
  const float rs = rsqrtf(q / static_cast<float>(cols) + eps);
  if (threadIdx.x == 0) {
    store_from_f32(mean, row, dt_stat, mu);
    store_from_f32(rstd, row, dt_stat, rs);
  }
  for (int64_t c = threadIdx.x; c < cols; c += blockDim.x) {
    float r = (load_as_f32(x, base + c, dt) - mu) * rs;
    if (w) r *= load_as_f32(w, c, dt_wb);
    if (b) r += load_as_f32(b, c, dt_wb);
    store_from_f32(y, base + c, dt, r);
  }
}

// ------------------------------------------------------------------ sum / argmax
// argmax order: NaN beats everything, then larger value, then smaller index.
struct ArgPair {
  float v;
  int64_t i;
};
__device__ __forceinline__ bool arg_better(float v, int64_t i, float bv, int64_t bi) {
  const bool vn = v != v, bn = bv != bv;
  if (vn || bn) return vn && (!bn || i < bi);
  return v > bv || (v == bv && i < bi);
}
__device__ __forceinline__ void arg_take(ArgPair& a, float v, int64_t i) {
  if (a.i < 0 || arg_better(v, i, a.v, a.i)) { a.v = v; a.i = i; }
}
// Streaming form for a thread that visits its elements in ASCENDING index order: one
// compare per element on the common path. `v <= best` is false when v is larger, when v is
// NaN, or when best is already NaN; only then the slow test runs (a NaN best is final:
// the first NaN wins; otherwise v is larger or NaN and, being the earliest such, is taken).
__device__ __forceinline__ void arg_take_ascending(ArgPair& a, float v, int64_t i) {
  if (!(v <= a.v)) {
    if (a.i < 0 || a.v == a.v) { a.v = v; a.i = i; }
  }
}
__device__ __forceinline__ ArgPair arg_warp_reduce(ArgPair a) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float v = __shfl_xor_sync(0xffffffffu, a.v, o);
    const int64_t i = __shfl_xor_sync(0xffffffffu, a.i, o);
    if (i >= 0) arg_take(a, v, i);
  }
  return a;
}

// Row reduction (inner == 1). grid = (row groups, splits). A row's [c0, c1) slice of
// split blockIdx.y is consumed by one warp (WARP) or one CTA: single elements up to the first
// 16-byte boundary, 16-byte loads from there, single elements at the end. Rows off the 16-byte
// grid (a vocabulary of 50,257) so take the same path as the others: bound by HBM, argmax of
// bf16 4096 x 50257 168 us with element-wise loads -> 80 us (5.2 TB/s).
template <typename T, bool WARP, bool ARG>
__global__ void __launch_bounds__(256) reduce_rows(const T* __restrict__ x, void* __restrict__ out, float* __restrict__ part_v, int64_t* __restrict__ part_i,
                                                   int64_t rows, int64_t cols, int64_t chunk, int dto) {
  constexpr int VE = Vec<T>::N;
  __shared__ float red[33];
  __shared__ float av[32];
  __shared__ int64_t ai[32];
  const int tpr = WARP ? 32 : blockDim.x;
  const int t = WARP ? (threadIdx.x & 31) : threadIdx.x;
  const int64_t row = WARP ? static_cast<int64_t>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5) : blockIdx.x;
  if (WARP && row >= rows) return;
  const int64_t c0 = static_cast<int64_t>(blockIdx.y) * chunk;
  const int64_t c1 = c0 + chunk < cols ? c0 + chunk : cols;
  const T* xr = x + row * cols;
  float s = 0.f;
  ArgPair a{0.f, -1};
  // a0: the slice's first element on the grid
  const int64_t to_grid = static_cast<int64_t>((16u - (reinterpret_cast<uintptr_t>(xr + c0) & 15u)) & 15u) / static_cast<int64_t>(sizeof(T));
  const int64_t a0 = c0 + to_grid < c1 ? c0 + to_grid : c1;
  const T* xa = xr + a0;
  const int nv = static_cast<int>((c1 - a0) / VE);
  // the at most 2 (VE - 1) elements off the vectors, one to a thread: a sum asks for them before the first
  // vector, argmax, which is short of registers, before and behind the vectors
  float sv = 0.f;
  if constexpr (ARG) {
    if (c0 + t < a0) arg_take(a, to_f32(xr[c0 + t]), c0 + t);
  } else {
    const int64_t c = c0 + t < a0 ? c0 + t : a0 + static_cast<int64_t>(nv) * VE + t - (a0 - c0);
    if (c < c1) sv = to_f32(xr[c]);
  }
  // argmax keeps the largest element of whole vectors and the first vector that holds it (a
  // NaN beats everything, the first one stays); which element it was is asked once per row
  float best = -CUDART_INF_F;
  int best_j = -1;
  auto take = [&](const uint4& raw, int j) {
    if (ARG) {
      const float m = vec_max_nan<T>(raw);
      if (!(m <= best) && best == best) {
        best = m;
        best_j = j;
      }
    } else {
      vec_accumulate<T>(s, raw);  // 16-bit elements are widened inside the add
    }
  };
  int j = t;
  for (; j + 3 * tpr < nv; j += 4 * tpr) {
    uint4 v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) v[u] = ld_stream(xa + static_cast<int64_t>(j + u * tpr) * VE);
#pragma unroll
    for (int u = 0; u < 4; ++u) take(v[u], j + u * tpr);
  }
  if constexpr (ARG) {
    for (; j < nv; j += tpr) take(ld_stream(xa + static_cast<int64_t>(j) * VE), j);
  } else if (j < nv) {  // up to three more
    uint4 v[3];
#pragma unroll
    for (int u = 0; u < 3; ++u)
      if (j + u * tpr < nv) v[u] = ld_stream(xa + static_cast<int64_t>(j + u * tpr) * VE);
#pragma unroll
    for (int u = 0; u < 3; ++u)
      if (j + u * tpr < nv) take(v[u], j + u * tpr);
  }
  if (ARG && t < nv) {
    if (best_j < 0) best_j = t;  // nothing but -inf so far: the first element is the answer
    arg_take(a, best, a0 + static_cast<int64_t>(best_j) * VE);  // the vector's place stands for its element's until the row is decided
  }
  if constexpr (ARG) {
    if (const int64_t c = a0 + static_cast<int64_t>(nv) * VE + t; c < c1) arg_take(a, to_f32(xr[c]), c);
  } else {
    s += sv;
  }
  const bool split = gridDim.y > 1;
  const int64_t slot = static_cast<int64_t>(blockIdx.y) * rows + row;
  if (!ARG) {
    s = WARP ? warp_reduce(s, SumF{}) : block_reduce(s, SumF{}, 0.f, red);
    if (t == 0) {
      if (split) part_v[slot] = s;
      else store_from_f32(out, row, dto, s);
    }
  } else {
    a = arg_warp_reduce(a);
    if (!WARP) {
      const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
      if (lane == 0) { av[warp] = a.v; ai[warp] = a.i; }
      __syncthreads();
      if (warp == 0) {
        a.v = lane < (blockDim.x >> 5) ? av[lane] : 0.f;
        a.i = lane < (blockDim.x >> 5) ? ai[lane] : -1;
        a = arg_warp_reduce(a);
      }
    }
    if (threadIdx.x == 0 || (WARP && t == 0)) {
      if (a.i >= a0 && a.i < a0 + static_cast<int64_t>(nv) * VE) {  // a vector won: its first element of that value
        float f[VE];
        widen<T>(ld_stream(xr + a.i), f);
        int first = 0;
#pragma unroll
        for (int e = VE - 1; e >= 0; --e)
          if (a.v == a.v ? f[e] == a.v : f[e] != f[e]) first = e;
        a.i += first;
      }
      if (split) { part_v[slot] = a.v; part_i[slot] = a.i; }
      else static_cast<int64_t*>(out)[row] = a.i;
    }
  }
}

// The same for short rows, a warp to each and single elements throughout (see rows_one_by_one).
template <typename T, bool ARG>
__global__ void __launch_bounds__(256) reduce_rows_single(const T* __restrict__ x, void* __restrict__ out, int64_t rows, int64_t cols, int dto) {
  const int lane = threadIdx.x & 31;
  const int64_t row = static_cast<int64_t>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (row >= rows) return;
  const T* xr = x + row * cols;
  float s = 0.f;
  ArgPair a{CUDART_NAN_F, -1};  // NaN start: the first element fails `v <= NaN` and is taken through a.i < 0
  for (int64_t c = lane; c < cols; c += 32) {
    const float v = to_f32(xr[c]);
    if (ARG) arg_take_ascending(a, v, c);
    else s += v;
  }
  if (ARG) {
    a = arg_warp_reduce(a);
    if (lane == 0) static_cast<int64_t*>(out)[row] = a.i;
  } else {
    s = warp_reduce(s, SumF{});
    if (lane == 0) store_from_f32(out, row, dto, s);
  }
}

// argmax over columns (inner > 1): thread per inner element, grid = (inner tiles, outer, splits).
template <typename T>
__global__ void __launch_bounds__(256) argmax_cols(const T* __restrict__ x, int64_t* __restrict__ out, float* __restrict__ part_v, int64_t* __restrict__ part_i,
                                                   int64_t outer, int64_t dim, int64_t inner, int64_t chunk) {
  const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= inner) return;
  const int64_t o = blockIdx.y;
  const int64_t k0 = static_cast<int64_t>(blockIdx.z) * chunk;
  const int64_t k1 = k0 + chunk < dim ? k0 + chunk : dim;
  const T* p = x + o * dim * inner + i;
  ArgPair a{0.f, -1};
  int64_t k = k0;
  for (; k + 7 < k1; k += 8) {  // eight rows requested before the first comparison
    T f[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) f[u] = p[(k + u) * inner];
#pragma unroll
    for (int u = 0; u < 8; ++u) arg_take(a, to_f32(f[u]), k + u);
  }
  for (; k < k1; ++k) arg_take(a, to_f32(p[k * inner]), k);
  const int64_t oi = o * inner + i;
  if (gridDim.z > 1) {
    const int64_t slot = static_cast<int64_t>(blockIdx.z) * outer * inner + oi;
    part_v[slot] = a.v;
    part_i[slot] = a.i;
  } else {
    out[oi] = a.i;
  }
}

// Sum over columns (inner > 1; the bias gradient of a linear layer). grid = (inner tiles, outer,
// splits). A lane owns the columns of G WORDs that lie 32 words apart (a word as wide as the rows' length and
// base allow), a warp 32 G such words of every blockDim / 32 -th row of the slice, eight rows in
// flight; the eight are added as a tree before they go into the accumulator, and so are the warps'
// sums: the chain of additions behind a result is a 128th of the slice long. Bound by HBM: bf16 8192 x 11008
// (180 MB) 93 -> 32 us (5.6 TB/s) and fp32 8192 x 11007, off the grid, 94 -> 62 us against a thread
// per column with four loads in flight (the kernel below); root mean square error there 3.2e-7 -> 1.2e-7.
template <typename T, typename WORD, int G>
__global__ void __launch_bounds__(512, 2) sum_cols(const T* __restrict__ x, void* __restrict__ out, float* __restrict__ part_v, int64_t outer, int64_t dim, int64_t inner, int64_t chunk, int dto) {
  constexpr int E = sizeof(WORD) / sizeof(T), U = 8;
  __shared__ float red[16][32 * E * G];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  const int64_t o = blockIdx.y, first = static_cast<int64_t>(blockIdx.x) * (32 * E * G);
  const int64_t k0 = static_cast<int64_t>(blockIdx.z) * chunk;
  const int64_t k1 = k0 + chunk < dim ? k0 + chunk : dim;
  float acc[G][E];
  bool in[G];
#pragma unroll
  for (int g = 0; g < G; ++g) {
    in[g] = first + (g * 32 + lane) * E < inner;
#pragma unroll
    for (int e = 0; e < E; ++e) acc[g][e] = 0.f;
  }
  const T* p = x + (o * dim + k0 + warp) * inner + first + lane * E;
  for (int64_t k = k0 + warp; k < k1; k += U * warps, p += U * warps * inner) {
    WORD v[U][G];
#pragma unroll
    for (int u = 0; u < U; ++u) {
#pragma unroll
      for (int g = 0; g < G; ++g) {
        v[u][g] = WORD{};
        if (k + u * warps < k1 && in[g]) v[u][g] = __ldcs(reinterpret_cast<const WORD*>(p + u * warps * inner + g * 32 * E));
      }
    }
#pragma unroll
    for (int g = 0; g < G; ++g) {
#pragma unroll
      for (int e = 0; e < E; ++e) {
        float f[U];
#pragma unroll
        for (int u = 0; u < U; ++u) f[u] = to_f32(reinterpret_cast<const T*>(&v[u][g])[e]);
        acc[g][e] += tree_sum<U>(f);
      }
    }
  }
#pragma unroll
  for (int g = 0; g < G; ++g) {
#pragma unroll
    for (int e = 0; e < E; ++e) red[warp][(g * E + e) * 32 + lane] = acc[g][e];
  }
  __syncthreads();
  for (int j = threadIdx.x; j < 32 * E * G; j += blockDim.x) {
    const int64_t i = first + ((j / (32 * E)) * 32 + (j & 31)) * E + (j >> 5) % E;
    if (i >= inner) continue;
    float f[16];
#pragma unroll
    for (int w = 0; w < 16; ++w) f[w] = w < warps ? red[w][j] : 0.f;
    const float sum = tree_sum<16>(f);
    const int64_t oi = o * inner + i;
    if (gridDim.z > 1) part_v[static_cast<int64_t>(blockIdx.z) * outer * inner + oi] = sum;
    else store_from_f32(out, oi, dto, sum);
  }
}

// The same with a thread to a column: few rows, or columns that would leave the tiles above mostly empty.
template <typename T>
__global__ void __launch_bounds__(256) sum_cols_thread(const T* __restrict__ x, void* __restrict__ out, float* __restrict__ part_v, int64_t outer, int64_t dim, int64_t inner, int64_t chunk, int dto) {
  const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= inner) return;
  const int64_t o = blockIdx.y;
  const int64_t k0 = static_cast<int64_t>(blockIdx.z) * chunk;
  const int64_t k1 = k0 + chunk < dim ? k0 + chunk : dim;
  const T* p = x + o * dim * inner + i;
  float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
  int64_t k = k0;
  for (; k + 3 < k1; k += 4) {
    s0 += to_f32(p[k * inner]);
    s1 += to_f32(p[(k + 1) * inner]);
    s2 += to_f32(p[(k + 2) * inner]);
    s3 += to_f32(p[(k + 3) * inner]);
  }
  for (; k < k1; ++k) s0 += to_f32(p[k * inner]);
  const float s = (s0 + s1) + (s2 + s3);
  const int64_t oi = o * inner + i;
  if (gridDim.z > 1) part_v[static_cast<int64_t>(blockIdx.z) * outer * inner + oi] = s;
  else store_from_f32(out, oi, dto, s);
}

// Column reduction with at most 32 columns (the bias-gradient shape: many rows, few columns):
// a thread per column would leave most lanes of a warp without work, so the lanes of a warp
// tile rows x columns instead -- W = the next power of two above `inner` columns, 32 / W rows
// per warp and trip, i.e. a warp reads 32 consecutive elements when inner == W -- and the
// row-lanes are folded by shuffles, the CTA's 8 warps through shared memory, in a fixed order.
template <typename T, bool ARG>
__global__ void __launch_bounds__(256) reduce_cols_narrow(const T* __restrict__ x, void* __restrict__ out, float* __restrict__ part_v, int64_t* __restrict__ part_i,
                                                          int64_t outer, int64_t dim, int inner, int W, int64_t chunk, int dto) {
  __shared__ float sh_v[8][32];
  __shared__ int64_t sh_i[ARG ? 8 : 1][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int col = lane & (W - 1), rsub = lane / W, rpw = 32 / W;
  const int64_t o = blockIdx.y;
  const int64_t k0 = static_cast<int64_t>(blockIdx.z) * chunk;
  const int64_t k1 = k0 + chunk < dim ? k0 + chunk : dim;
  const T* p = x + o * dim * inner + col;
  const int64_t step = 8 * rpw;
  float s0 = 0.f, s1 = 0.f;
  ArgPair a{0.f, -1};
  if (col < inner) {
    int64_t k = k0 + warp * rpw + rsub;
    if (!ARG) {
      for (; k + step < k1; k += 2 * step) {
        s0 += to_f32(p[k * inner]);
        s1 += to_f32(p[(k + step) * inner]);
      }
    }
    for (; k < k1; k += step) {
      const float fv = to_f32(p[k * inner]);
      if (ARG) arg_take(a, fv, k);
      else s0 += fv;
    }
  }
  float s = s0 + s1;
  for (int off = W; off < 32; off <<= 1) {  // fold the row-lanes of the warp onto lanes 0 .. W-1
    if (ARG) {
      const float v = __shfl_xor_sync(0xffffffffu, a.v, off);
      const int64_t i = __shfl_xor_sync(0xffffffffu, a.i, off);
      if (i >= 0) arg_take(a, v, i);
    } else {
      s += __shfl_xor_sync(0xffffffffu, s, off);
    }
  }
  if (lane < W) {
    sh_v[warp][lane] = ARG ? a.v : s;
    if (ARG) sh_i[warp][lane] = a.i;
  }
  __syncthreads();
  if (warp == 0 && lane < inner) {
    float t = 0.f;
    ArgPair b{0.f, -1};
    for (int w = 0; w < 8; ++w) {
      if (ARG) { if (sh_i[w][lane] >= 0) arg_take(b, sh_v[w][lane], sh_i[w][lane]); }
      else t += sh_v[w][lane];
    }
    const int64_t oi = o * inner + lane;
    if (gridDim.z > 1) {
      const int64_t slot = static_cast<int64_t>(blockIdx.z) * outer * inner + oi;
      if (ARG) { part_v[slot] = b.v; part_i[slot] = b.i; }
      else part_v[slot] = t;
    } else {
      if (ARG) static_cast<int64_t*>(out)[oi] = b.i;
      else store_from_f32(out, oi, dto, t);
    }
  }
}

// Second stage of a split reduction: n outputs, `splits` partials each, ascending split
// order (so the earliest index wins argmax ties and sums are run-to-run identical).
template <bool ARG>
__global__ void __launch_bounds__(256) reduce_finalize(const float* __restrict__ part_v, const int64_t* __restrict__ part_i, void* __restrict__ out, int64_t n, int splits, int dto) {
  const int64_t o = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (o >= n) return;
  // eight partials are requested before the first one is combined: a thread that waited for
  // each in turn spent a round trip to L2 per partial (1059 x 3072 argmax over dim 0: 12 us)
  if (ARG) {
    ArgPair a{0.f, -1};
    for (int s0 = 0; s0 < splits; s0 += 8) {
      int64_t i[8];
      float v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const bool in = s0 + u < splits;
        i[u] = in ? part_i[(s0 + u) * n + o] : -1;
        v[u] = in ? part_v[(s0 + u) * n + o] : 0.f;
      }
#pragma unroll
      for (int u = 0; u < 8; ++u)
        if (i[u] >= 0) arg_take(a, v[u], i[u]);
    }
    static_cast<int64_t*>(out)[o] = a.i;
  } else {
    float s = 0.f;
    for (int k0 = 0; k0 < splits; k0 += 8) {
      float v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) v[u] = k0 + u < splits ? part_v[(k0 + u) * n + o] : 0.f;
#pragma unroll
      for (int u = 0; u < 8; ++u)
        if (k0 + u < splits) s += v[u];  // the same order of additions as one by one
    }
    store_from_f32(out, o, dto, s);
  }
}

// The same with one warp per output, for many partials of few outputs (a whole-tensor
// reduction): lanes take partials s = lane, lane + 32, ... and combine by shuffles. The
// order of the additions is fixed by (lane, shuffle tree), so sums stay run-to-run
// identical; argmax combines by (NaN, value, index), which is order-free.
template <bool ARG>
__global__ void __launch_bounds__(256) reduce_finalize_warp(const float* __restrict__ part_v, const int64_t* __restrict__ part_i, void* __restrict__ out, int64_t n, int splits, int dto) {
  const int64_t o = static_cast<int64_t>(blockIdx.x) * 8 + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (o >= n) return;
  if (ARG) {
    ArgPair a{0.f, -1};
    for (int s = lane; s < splits; s += 32) {
      const int64_t i = part_i[s * n + o];
      if (i >= 0) arg_take(a, part_v[s * n + o], i);
    }
    a = arg_warp_reduce(a);
    if (lane == 0) static_cast<int64_t*>(out)[o] = a.i;
  } else {
    float s = 0.f;
    for (int k = lane; k < splits; k += 32) s += part_v[k * n + o];
    s = warp_reduce(s, SumF());
    if (lane == 0) store_from_f32(out, o, dto, s);
  }
}

__global__ void fill_zero_typed(void* out, int64_t n, int dto) {
  const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i < n) store_from_f32(out, i, dto, 0.f);
}

// ------------------------------------------------------------------ very short rows (dim <= 32, inner == 1)
// Millions of rows of a handful of elements: one THREAD per row, the row in registers (NC
// slots, the next multiple of 8 above the row length). A CTA owns 256 consecutive rows, one
// contiguous span of memory, and reaches it in one of three ways.
//   direct: each thread loads and stores its own row element by element. A warp-wide access
//     then touches one 32-byte sector per lane, and the load/store unit spends a cycle per
//     sector: the cost is ~2 x 32 x cols cycles per warp, far above the bytes moved. Kept
//     for bases off the 16-byte grid and outputs of another element size.
//   vector: rows that are whole 16-byte vectors are loaded and stored as such.
//   staged: any other row length. The CTA copies its span into shared memory with 16-byte
//     accesses, threads read and overwrite their rows there (the stride is not a multiple of
//     16 bytes, so at most two lanes of a quarter-warp meet in a bank), and the span goes
//     back out the same way.
constexpr int kSmallRow = 32;
constexpr int kSmallRows = 256;  // rows (threads) per CTA
enum { SMALL_SOFTMAX = 0, SMALL_LOGSOFTMAX = 1, SMALL_SUM = 2, SMALL_ARGMAX = 3, SMALL_LAYERNORM = 4 };
enum { SMALL_DIRECT = 0, SMALL_STAGED = 1, SMALL_VECTOR = 2 };

template <typename T, int OP, int NC, int MODE>
__global__ void __launch_bounds__(kSmallRows) rows_small(const T* __restrict__ x, void* __restrict__ out, int64_t rows, int cols, int dto, const void* __restrict__ w,
                                                         const void* __restrict__ b, int dt_wb, void* __restrict__ mean, void* __restrict__ rstd, int dt_stat, float eps) {
  extern __shared__ __align__(16) unsigned char small_smem[];
  constexpr bool WRITES_ROWS = OP == SMALL_SOFTMAX || OP == SMALL_LOGSOFTMAX || OP == SMALL_LAYERNORM;
  constexpr bool STAGED = MODE == SMALL_STAGED, VECTOR = MODE == SMALL_VECTOR;
  constexpr int VE = 16 / static_cast<int>(sizeof(T));
  const int tid = threadIdx.x;
  const int64_t row0 = static_cast<int64_t>(blockIdx.x) * kSmallRows;
  const int64_t row = row0 + tid;
  const bool live = row < rows;
  T* sm = reinterpret_cast<T*>(small_smem);
  __shared__ float wb[2 * kSmallRow];  // layer norm: weight and bias as fp32 (1 and 0 when absent)
  if (OP == SMALL_LAYERNORM) {
    if (tid < cols) {
      wb[tid] = w ? load_as_f32(w, tid, dt_wb) : 1.f;
      wb[kSmallRow + tid] = b ? load_as_f32(b, tid, dt_wb) : 0.f;
    }
    if (!STAGED) __syncthreads();
  }
  int span = 0;
  if (STAGED) {
    const int64_t left = rows - row0;
    span = static_cast<int>(left < kSmallRows ? left : kSmallRows) * cols;  // elements this CTA owns
    const T* src = x + row0 * cols;
    const int nv = span / VE;
    for (int j = tid; j < nv; j += kSmallRows) reinterpret_cast<uint4*>(sm)[j] = ld_stream(src + static_cast<int64_t>(j) * VE);
    for (int j = nv * VE + tid; j < span; j += kSmallRows) sm[j] = src[j];
    __syncthreads();
  }
  const T* xr = STAGED ? sm + tid * cols : x + row * cols;
  T* orow = sm + tid * cols;  // staged results overwrite the row in shared memory
  float f[NC];
  auto put = [&](int c, float v) {
    if (STAGED) orow[c] = from_f32<T>(v);
    else if (VECTOR) f[c] = v;  // in place: slot c has been consumed; stored as vectors below
    else store_from_f32(out, row * cols + c, dto, v);
  };
  if (live) {
    if (VECTOR) {
#pragma unroll
      for (int v = 0; v < NC / VE; ++v) {
        if (v * VE < cols) {
          widen<T>(ld_stream(xr + v * VE), f + v * VE);
        } else {
#pragma unroll
          for (int e = 0; e < VE; ++e) f[v * VE + e] = 0.f;
        }
      }
    } else {
#pragma unroll
      for (int c = 0; c < NC; ++c) f[c] = c < cols ? to_f32(xr[c]) : 0.f;
    }
    if (OP == SMALL_SUM) {
      float s = 0.f;
#pragma unroll
      for (int c = 0; c < NC; ++c) s += c < cols ? f[c] : 0.f;
      store_from_f32(out, row, dto, s);
    } else if (OP == SMALL_ARGMAX) {
      ArgPair a{CUDART_NAN_F, -1};
#pragma unroll
      for (int c = 0; c < NC; ++c)
        if (c < cols) arg_take_ascending(a, f[c], c);
      static_cast<int64_t*>(out)[row] = a.i;
    } else if (OP == SMALL_LAYERNORM) {
      float s = 0.f;
#pragma unroll
      for (int c = 0; c < NC; ++c) s += c < cols ? f[c] : 0.f;
      float mu = s / static_cast<float>(cols);
      if (!isfinite(mu)) mu = CUDART_NAN_F;
      float q = 0.f;
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        const float d = f[c] - mu;
        q = c < cols ? fmaf(d, d, q) : q;
      }
      const float rs = rsqrtf(q / static_cast<float>(cols) + eps);
      store_from_f32(mean, row, dt_stat, mu);
      store_from_f32(rstd, row, dt_stat, rs);
#pragma unroll
      for (int c = 0; c < NC; ++c)
        if (c < cols) put(c, (f[c] - mu) * rs * wb[c] + wb[kSmallRow + c]);
    } else {
      float m = -CUDART_INF_F;
#pragma unroll
      for (int c = 0; c < NC; ++c) m = c < cols ? fmaxf(m, f[c]) : m;
      float s = 0.f;
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        const float d = f[c] - m;
        const float ex = ex2_approx(d * kLog2e);
        s += c < cols ? ex : 0.f;
        f[c] = OP == SMALL_LOGSOFTMAX ? d : ex;
      }
      const float k = OP == SMALL_LOGSOFTMAX ? logf(s) : 1.f / s;
#pragma unroll
      for (int c = 0; c < NC; ++c)
        if (c < cols) put(c, OP == SMALL_LOGSOFTMAX ? f[c] - k : f[c] * k);
    }
    if (VECTOR && WRITES_ROWS) {
#pragma unroll
      for (int v = 0; v < NC / VE; ++v)
        if (v * VE < cols) store_row_vec<T>(out, row * cols + v * VE, f + v * VE, false);
    }
  }
  if (STAGED && WRITES_ROWS) {
    __syncthreads();
    T* dst = static_cast<T*>(out) + row0 * cols;
    const int nv = span / VE;
    for (int j = tid; j < nv; j += kSmallRows) st_stream(dst + static_cast<int64_t>(j) * VE, reinterpret_cast<const uint4*>(sm)[j]);
    for (int j = nv * VE + tid; j < span; j += kSmallRows) dst[j] = sm[j];
  }
}

template <typename T, int OP, int NC>
static void launch_rows_small_nc(const void* x, void* out, int64_t rows, int cols, int dti, int dto, const void* w, const void* b, int dt_wb, void* mean, void* rstd, int dt_stat, float eps,
                                 cudaStream_t st) {
  constexpr bool WRITES_ROWS = OP == SMALL_SOFTMAX || OP == SMALL_LOGSOFTMAX || OP == SMALL_LAYERNORM;
  const int g = grid_for(rows, kSmallRows);
  // 16-byte accesses need 16-byte aligned bases and, for row results, an output of the input's type
  const bool wide = aligned16(x) && (!WRITES_ROWS || (dto == dti && aligned16(out)));
  const T* px = static_cast<const T*>(x);
  if (wide && (cols * sizeof(T)) % 16 == 0) {
    rows_small<T, OP, NC, SMALL_VECTOR><<<g, kSmallRows, 0, st>>>(px, out, rows, cols, dto, w, b, dt_wb, mean, rstd, dt_stat, eps);
  } else if (wide) {
    const size_t smem = (static_cast<size_t>(kSmallRows) * cols * sizeof(T) + 15) / 16 * 16;
    rows_small<T, OP, NC, SMALL_STAGED><<<g, kSmallRows, smem, st>>>(px, out, rows, cols, dto, w, b, dt_wb, mean, rstd, dt_stat, eps);
  } else {
    rows_small<T, OP, NC, SMALL_DIRECT><<<g, kSmallRows, 0, st>>>(px, out, rows, cols, dto, w, b, dt_wb, mean, rstd, dt_stat, eps);
  }
}

template <typename T, int OP>
static void launch_rows_small_T(const void* x, void* out, int64_t rows, int cols, int dti, int dto, const void* w, const void* b, int dt_wb, void* mean, void* rstd, int dt_stat, float eps,
                                cudaStream_t st) {
  if (cols <= 8) launch_rows_small_nc<T, OP, 8>(x, out, rows, cols, dti, dto, w, b, dt_wb, mean, rstd, dt_stat, eps, st);
  else if (cols <= 16) launch_rows_small_nc<T, OP, 16>(x, out, rows, cols, dti, dto, w, b, dt_wb, mean, rstd, dt_stat, eps, st);
  else if (cols <= 24) launch_rows_small_nc<T, OP, 24>(x, out, rows, cols, dti, dto, w, b, dt_wb, mean, rstd, dt_stat, eps, st);
  else launch_rows_small_nc<T, OP, 32>(x, out, rows, cols, dti, dto, w, b, dt_wb, mean, rstd, dt_stat, eps, st);
}

template <int OP>
static int launch_rows_small(const void* x, void* out, int64_t rows, int cols, int dti, int dto, const void* w, const void* b, int dt_wb, void* mean, void* rstd, int dt_stat, float eps,
                             cudaStream_t st) {
  switch (dti) {
    case B200_F32: launch_rows_small_T<float, OP>(x, out, rows, cols, dti, dto, w, b, dt_wb, mean, rstd, dt_stat, eps, st); break;
    case B200_BF16: launch_rows_small_T<__nv_bfloat16, OP>(x, out, rows, cols, dti, dto, w, b, dt_wb, mean, rstd, dt_stat, eps, st); break;
    default: launch_rows_small_T<__half, OP>(x, out, rows, cols, dti, dto, w, b, dt_wb, mean, rstd, dt_stat, eps, st); break;
  }
  return check_launch();
}

// ------------------------------------------------------------------ host-side planning
struct ReducePlan {
  int splits;
  int64_t chunk;  // elements of `dim` per split (a multiple of 64 for rows, of 16 for columns)
};

static ReducePlan plan_reduce(int64_t outer, int64_t dim, int64_t inner) {
  // CTAs available without splitting
  int64_t ctas = inner == 1 ? outer : outer * ((inner + 255) / 256);
  ReducePlan p{1, dim};
  const int64_t want = 2LL * kNumSMs;
  // A row reduction (inner == 1) is worth splitting from 4096 elements, 1024 per split. A
  // column reduction walks `dim` one row per iteration, every row a coalesced read, and with
  // few columns it has few threads: split it from 64 rows, 16 per split (argmax over 112
  // rows of 6144 columns: 24 CTAs unsplit).
  const int64_t min_dim = inner == 1 ? 4096 : 64, min_chunk = inner == 1 ? 1024 : 16;
  if (ctas >= want || dim < min_dim) return p;
  int64_t s = (want + ctas - 1) / ctas;
  const int64_t max_s = dim / min_chunk;
  if (s > max_s) s = max_s;
  if (s > 1024) s = 1024;
  if (s <= 1) return p;
  int64_t chunk = (dim + s - 1) / s;
  const int64_t gran = inner == 1 ? 64 : 16;  // row chunks stay on the 16-byte grid of any element type
  chunk = (chunk + gran - 1) / gran * gran;
  p.splits = static_cast<int>((dim + chunk - 1) / chunk);
  p.chunk = chunk;
  return p;
}

// Bytes of the words `sum_cols` reads: the widest that every row starts on and ends with, and
// that still gives 32 lanes columns.
static int sum_cols_word(const void* x, int64_t inner, int esize) {
  int bytes = 16;
  while (bytes > esize && (((inner * esize) | static_cast<int64_t>(reinterpret_cast<uintptr_t>(x))) % bytes || inner * esize < 32 * bytes)) bytes >>= 1;
  return bytes;
}
struct SumColsPlan {
  bool by_thread;  // sum_cols_thread, as `plan_reduce` cuts it
  int word, groups, warps, splits;
  int64_t chunk;
};
// How a column sum is cut up; `p`: what `plan_reduce` says (its scratch holds four fp32 partials per slice and output). All times in
// us, fp32, with the other way behind the bar.
static SumColsPlan plan_sum_cols(const void* x, int64_t outer, int64_t dim, int64_t inner, int esize, const ReducePlan& p) {
  SumColsPlan s{false, sum_cols_word(x, inner, esize), 1, 16, 1, dim};
  s.groups = s.word == esize ? 2 : 1;
  auto tile = [&] { return static_cast<int64_t>(32) * (s.word / esize) * s.groups; };
  auto tiles = [&] { return (inner + tile() - 1) / tile(); };
  // 8 x 100 2.5 | 3.7; 7000 times 33 x 5 7.1 | 8.5; 16384 x 130 5.4 | 6.4, whose last tile is nearly empty
  s.by_thread = dim < 16 || inner <= 16 || (tiles() > 1 && tiles() * tile() * 10 > inner * 13 && outer * dim * inner * esize <= (16LL << 20));
  if (s.by_thread) {
    s.splits = p.splits;
    s.chunk = p.chunk;
    return s;
  }
  constexpr int64_t kSlots = 2 * kNumSMs;  // CTAs of sixteen warps resident at once
  if (dim <= 384 || (dim <= 512 && outer * tiles() >= kNumSMs)) {
    // a CTA walks these rows in three or four trips, a second launch costs as much: no slices (100 x 4099 3.3 | 4.9),
    // narrower tiles if that is what gives every SM one
    while (outer * tiles() < kNumSMs && (s.groups > 1 || s.word > esize)) {
      if (s.groups > 1) s.groups = 1;
      else s.word >>= 1;
    }
  } else {
    // the fewest slices that fill the rounds of CTAs to six sevenths (bf16 8192 x 11008, 43 tiles: 6 slices, one
    // round, 32 us; 7, a round and a bit, 49), not below 32 rows each
    const int64_t most = p.splits > 1 ? (4LL * p.splits < dim / 32 ? 4LL * p.splits : dim / 32) : 1;
    int64_t best = 1;
    double best_full = 0.;
    for (int64_t n = 1; n <= most && best_full < 6. / 7; ++n) {
      const int64_t ctas = outer * tiles() * n, rounds = (ctas + kSlots - 1) / kSlots;
      const double full = static_cast<double>(ctas) / static_cast<double>(rounds * kSlots);
      if (full > best_full) { best = n; best_full = full; }
    }
    s.chunk = (dim + best - 1) / best;
    s.splits = static_cast<int>((dim + s.chunk - 1) / s.chunk);
  }
  // eight rows to a warp; more, smaller CTAs where sixteen warps each would make two rounds (64 x 50257 4.7 | 5.6)
  while (s.warps > 1 && s.warps * 4 >= s.chunk) s.warps >>= 1;
  while (s.warps > 4 && s.splits == 1 && outer * tiles() > kSlots * 16 / s.warps) s.warps >>= 1;
  return s;
}
template <typename T, typename WORD, int G>
static void launch_sum_cols_as(const T* x, void* out, float* pv, int64_t outer, int64_t dim, int64_t inner, const SumColsPlan& s, int dto, cudaStream_t st) {
  const dim3 g(grid_for(inner, 32 * (sizeof(WORD) / sizeof(T)) * G), static_cast<unsigned>(outer), static_cast<unsigned>(s.splits));
  sum_cols<T, WORD, G><<<g, 32 * s.warps, 0, st>>>(x, out, pv, outer, dim, inner, s.chunk, dto);
}
template <typename T>
static void launch_sum_cols(const T* x, void* out, float* pv, int64_t outer, int64_t dim, int64_t inner, const SumColsPlan& s, int dto, cudaStream_t st) {
  typedef typename std::conditional<sizeof(T) == 2, uint16_t, uint32_t>::type One;
  if (s.by_thread) {
    const dim3 g(grid_for(inner, 256), static_cast<unsigned>(outer), static_cast<unsigned>(s.splits));
    sum_cols_thread<T><<<g, 256, 0, st>>>(x, out, pv, outer, dim, inner, s.chunk, dto);
  } else if (s.word == 16) {
    launch_sum_cols_as<T, uint4, 1>(x, out, pv, outer, dim, inner, s, dto, st);
  } else if (s.word == 8) {
    launch_sum_cols_as<T, uint2, 1>(x, out, pv, outer, dim, inner, s, dto, st);
  } else if (sizeof(T) == 2 && s.word == 4) {
    launch_sum_cols_as<T, uint32_t, 1>(x, out, pv, outer, dim, inner, s, dto, st);
  } else if (s.groups == 2) {
    launch_sum_cols_as<T, One, 2>(x, out, pv, outer, dim, inner, s, dto, st);
  } else {
    launch_sum_cols_as<T, One, 1>(x, out, pv, outer, dim, inner, s, dto, st);
  }
}

// Whether rows of a warp each go one element at a time. Off the 16-byte grid a vector costs the look at both ends of
// the row, and argmax a second look at the vector that won. Measured with vectors / one by one, us: argmax f32
// 65536 x 333 41 / 29, 16384 x 2047 32.8 / 29.2 (longer rows are a CTA's); bf16 65536 x 777 51 / 40, 32768 x 1001 26.6 / 29.4; on the grid f32
// 65536 x 128 26 / 22, 65536 x 512 31 / 35; sum bf16 100000 x 131 22 / 18, 65536 x 333 16 / 18; f32 100000 x 33 18.4 / 16.9,
// 100000 x 65 19 / 21.
template <bool ARG>
static bool rows_one_by_one(const void* x, int64_t dim, int esize) {
  const bool on_grid = aligned16(x) && (dim * esize) % 16 == 0;
  if (ARG) return on_grid ? dim * esize <= 512 : dim <= (esize == 4 ? 2048 : 896);
  return !on_grid && dim <= (esize == 4 ? 48 : 160);
}

template <typename T, bool ARG>
static int launch_reduce_T(const void* x, void* out, int64_t outer, int64_t dim, int64_t inner, int dto, void* scratch, int64_t scratch_bytes, cudaStream_t st) {
  ReducePlan p = plan_reduce(outer, dim, inner);
  const int64_t nout = outer * inner;
  float* pv = nullptr;
  int64_t* pi = nullptr;
  if (p.splits > 1) {
    const int64_t need = static_cast<int64_t>(p.splits) * nout * 16;
    if (!scratch || scratch_bytes < need) return B200_ESCRATCH;
    pi = static_cast<int64_t*>(scratch);  // int64 block first keeps it 8-byte aligned
    pv = reinterpret_cast<float*>(pi + static_cast<int64_t>(p.splits) * nout);
  }
  const T* px = static_cast<const T*>(x);
  if (inner == 1) {
    // a warp to a row; a few longer rows are sooner done by a CTA each (sum f32 300 x 2047: 6.3 us by warps)
    const int64_t row_bytes = dim * static_cast<int64_t>(sizeof(T));
    const bool warp = p.splits == 1 && row_bytes <= 8192 && (ARG || row_bytes <= 2048 || outer >= 4 * kNumSMs);
    if (!warp && outer > 0x7fffffffLL) return B200_EINVAL;
    if (warp) {
      dim3 g(grid_for(outer, 8), 1);
      if (rows_one_by_one<ARG>(x, dim, sizeof(T))) reduce_rows_single<T, ARG><<<g, 256, 0, st>>>(px, out, outer, dim, dto);
      else reduce_rows<T, true, ARG><<<g, 256, 0, st>>>(px, out, pv, pi, outer, dim, p.chunk, dto);
    } else {
      dim3 g(static_cast<unsigned>(outer), p.splits);
      reduce_rows<T, false, ARG><<<g, 256, 0, st>>>(px, out, pv, pi, outer, dim, p.chunk, dto);
    }
  } else {
    if (outer > 65535) {
      // grid.y limit: fold by launching per slab of 65535 outer rows
      for (int64_t o0 = 0; o0 < outer; o0 += 65535) {
        const int64_t on = outer - o0 < 65535 ? outer - o0 : 65535;
        if (ARG) argmax_cols<T><<<dim3(grid_for(inner, 256), static_cast<unsigned>(on), 1), 256, 0, st>>>(px + o0 * dim * inner, static_cast<int64_t*>(out) + o0 * inner, nullptr, nullptr, on, dim, inner, dim);
        else launch_sum_cols<T>(px + o0 * dim * inner, static_cast<char*>(out) + o0 * inner * dtype_size(dto), nullptr, on, dim, inner, plan_sum_cols(px + o0 * dim * inner, on, dim, inner, sizeof(T), ReducePlan{1, dim}), dto, st);
      }
      return check_launch();
    }
    if (inner <= 32 && dim >= 64) {
      int W = 1;
      while (W < inner) W <<= 1;
      dim3 g(1, static_cast<unsigned>(outer), p.splits);
      reduce_cols_narrow<T, ARG><<<g, 256, 0, st>>>(px, out, pv, pi, outer, dim, static_cast<int>(inner), W, p.chunk, dto);
    } else if (ARG) {
      dim3 g(grid_for(inner, 256), static_cast<unsigned>(outer), p.splits);
      argmax_cols<T><<<g, 256, 0, st>>>(px, static_cast<int64_t*>(out), pv, pi, outer, dim, inner, p.chunk);
    } else {
      const SumColsPlan sp = plan_sum_cols(px, outer, dim, inner, sizeof(T), p);
      if (p.splits > 1) pv = static_cast<float*>(scratch);  // (no indices to keep: all of it is for sums)
      launch_sum_cols<T>(px, out, pv, outer, dim, inner, sp, dto, st);
      p.splits = sp.splits;
    }
  }
  // few outputs of many slices: a warp to an output (2048 x 514 in 32 slices: 4.7 us the call, 6.0 with a thread to each)
  if (p.splits >= (ARG ? 64 : 16) && nout <= 8LL * kNumSMs * 8) reduce_finalize_warp<ARG><<<grid_for(nout, 8), 256, 0, st>>>(pv, pi, out, nout, p.splits, dto);
  else if (p.splits > 1) reduce_finalize<ARG><<<grid_for(nout, 256), 256, 0, st>>>(pv, pi, out, nout, p.splits, dto);
  return check_launch(p.splits > 1 ? 2 : 1);
}

// Resident-kernel geometry for `nvec` 16-byte vectors per row.
struct ResidentCfg {
  bool ok, warp;
  int vpt, threads;
};
static ResidentCfg resident_cfg(int64_t nvec, int max_vpt, int target_vpt = 2) {
  ResidentCfg c{false, false, 1, 128};
  if (nvec <= 0) return c;
  auto pow2_at_least = [](int64_t v) { int64_t p = 1; while (p < v) p <<= 1; return p; };
  if (nvec <= 32LL * max_vpt && nvec <= 256) {
    c.ok = true; c.warp = true; c.threads = 128;
    c.vpt = static_cast<int>(pow2_at_least((nvec + 31) / 32));
    return c;
  }
  // two 16-byte vectors per thread (fewer registers, more resident warps), except fp32
  // layer norm: four (its two CTA-wide reductions cost more with many warps)
  int64_t th = pow2_at_least((nvec + target_vpt - 1) / target_vpt);
  if (th < 128) th = 128;
  if (th > 1024) th = 1024;
  const int64_t vpt = pow2_at_least((nvec + th - 1) / th);
  if (vpt > max_vpt) return c;
  c.ok = true; c.warp = false; c.threads = static_cast<int>(th); c.vpt = static_cast<int>(vpt);
  return c;
}

#define B200_DISPATCH_VPT(VPT_VALUE, MAXV, BODY)                     \
  switch (VPT_VALUE) {                                               \
    case 1: { constexpr int VPT = 1; BODY; } break;                  \
    case 2: { constexpr int VPT = 2; BODY; } break;                  \
    case 4: { constexpr int VPT = 4; BODY; } break;                  \
    default: { constexpr int VPT = (MAXV) >= 8 ? 8 : 4; BODY; } break; \
  }

template <typename T, int VPT, bool WARP>
static void softmax_launch(unsigned grid, int threads, cudaStream_t st, int is_log, const T* x, void* out, int64_t rows, int cols, int out_f32) {
  if (is_log) softmax_resident<T, VPT, WARP, true><<<grid, threads, 0, st>>>(x, out, rows, cols, out_f32);
  else softmax_resident<T, VPT, WARP, false><<<grid, threads, 0, st>>>(x, out, rows, cols, out_f32);
}
// Threads of a CTA that streams a row of `nvec` vectors: four vectors to each, which is what a thread has in flight, so that rows
// of up to 2048 vectors are one trip (ONE_TRIP; fp32 30000 x 1030: 46 us, with a vector to each of four times as many
// threads 138; 8192 x 4097 49 / 90). Rows that do not give every SM one are done sooner by more threads.
static int stream_threads(int64_t rows, int64_t nvec, int least) {
  const int64_t th = (nvec / (rows >= kNumSMs ? 4 : 1) + 31) / 32 * 32;
  return static_cast<int>(th < least ? least : (th > 512 ? 512 : th));
}

template <typename T>
static int softmax_T(const void* x, void* out, int64_t outer, int64_t dim, int64_t inner, int dto, int is_log, cudaStream_t st) {
  constexpr int VE = Vec<T>::N;
  constexpr int MAXV = 32 / VE;  // at most 32 fp32 registers of row data per thread
  const T* px = static_cast<const T*>(x);
  const int out_f32 = dto == B200_F32;
  if (inner == 1) {
    const ResidentCfg c = (dim % VE == 0 && aligned16(x) && aligned16(out) && dim < (1LL << 30)) ? resident_cfg(dim / VE, MAXV) : ResidentCfg{false, false, 1, 128};
    // 16-bit rows past 16384 elements leave a 1024-thread CTA with 3-4 vectors per thread and
    // one CTA per SM; the two-pass streaming kernel (two CTAs per SM, the second read from L2)
    // measured faster there: 3.6-4.1 TB/s against 3.1-3.5 at 24576 and 32768 bf16 columns
    const bool same_phase = dto == dtype_of<T>() && ((reinterpret_cast<uintptr_t>(x) ^ reinterpret_cast<uintptr_t>(out)) & 15u) == 0;
    const bool prefer_stream = sizeof(T) == 2 && dim / VE > 2048 && same_phase;
    if (c.ok && outer <= 0x7fffffffLL && !prefer_stream) {
      if (c.warp) {
        B200_DISPATCH_VPT(c.vpt, MAXV, (softmax_launch<T, VPT, true>(grid_for(outer, 4), 128, st, is_log, px, out, outer, static_cast<int>(dim), out_f32)))
      } else {
        B200_DISPATCH_VPT(c.vpt, MAXV, (softmax_launch<T, VPT, false>(static_cast<unsigned>(outer), c.threads, st, is_log, px, out, outer, static_cast<int>(dim), out_f32)))
      }
    } else if (dim <= kRaggedMaxCols && outer >= 64) {
      const unsigned g = grid_for(outer, 4);
      if (is_log) { B200_DISPATCH_NPL(dim, (softmax_warp_ragged<T, NPL, true><<<g, 128, 0, st>>>(px, out, outer, static_cast<int>(dim), dto))) }
      else { B200_DISPATCH_NPL(dim, (softmax_warp_ragged<T, NPL, false><<<g, 128, 0, st>>>(px, out, outer, static_cast<int>(dim), dto))) }
    } else {
      if (outer > 0x7fffffffLL) return B200_EINVAL;
      if (same_phase && dim < (1LL << 30)) {  // same type out, and rows of x and out at the same offset inside their 16-byte blocks
        const int th = stream_threads(outer, dim / VE, 64);  // (the second warp takes the last block)
        auto go = [&](auto kernel) { kernel<<<static_cast<unsigned>(outer), th, 0, st>>>(px, static_cast<T*>(out), static_cast<int>(dim)); };
        if (dim / VE <= 4 * th) {
          if (is_log) go(softmax_stream_vec<T, true, true>);
          else go(softmax_stream_vec<T, false, true>);
        } else {
          if (is_log) go(softmax_stream_vec<T, true, false>);
          else go(softmax_stream_vec<T, false, false>);
        }
      } else {
        softmax_stream<T><<<static_cast<unsigned>(outer), 256, 0, st>>>(px, out, dim, dto, is_log);
      }
    }
  } else {
    for (int64_t o0 = 0; o0 < outer; o0 += 65535) {
      const int64_t on = outer - o0 < 65535 ? outer - o0 : 65535;
      dim3 g(grid_for(inner, 128), static_cast<unsigned>(on));
      softmax_cols<T><<<g, 128, 0, st>>>(px + o0 * dim * inner, static_cast<char*>(out) + o0 * dim * inner * dtype_size(dto), dim, inner, dto, is_log);
    }
  }
  return check_launch();
}

template <typename T>
static int softmax_bwd_T(const void* g, const void* y, void* out, int64_t outer, int64_t dim, int64_t inner, int dti, int dto, int is_log, cudaStream_t st) {
  constexpr int VE = Vec<T>::N;
  constexpr int MAXV = 16 / VE;  // two rows are held: at most 16 fp32 registers of each per thread
  const T* pg = static_cast<const T*>(g);
  const T* py = static_cast<const T*>(y);
  const int out_f32 = dto == B200_F32;
  const bool out_ok = dto == B200_F32 || dto == dti;  // the vector store writes T or fp32
  if (inner == 1 && out_ok && dim % VE == 0 && aligned16(g) && aligned16(y) && aligned16(out) && dim < (1LL << 30) && outer <= 0x7fffffffLL) {
    const ResidentCfg c = resident_cfg(dim / VE, MAXV);
    if (c.ok) {
      const int cols = static_cast<int>(dim);
      if (c.warp) {
        const unsigned gr = grid_for(outer, 4);
        if (is_log) { B200_DISPATCH_VPT(c.vpt, MAXV, (softmax_bwd_resident<T, VPT, true, true><<<gr, 128, 0, st>>>(pg, py, out, outer, cols, out_f32))) }
        else { B200_DISPATCH_VPT(c.vpt, MAXV, (softmax_bwd_resident<T, VPT, true, false><<<gr, 128, 0, st>>>(pg, py, out, outer, cols, out_f32))) }
      } else {
        const unsigned gr = static_cast<unsigned>(outer);
        if (is_log) { B200_DISPATCH_VPT(c.vpt, MAXV, (softmax_bwd_resident<T, VPT, false, true><<<gr, c.threads, 0, st>>>(pg, py, out, outer, cols, out_f32))) }
        else { B200_DISPATCH_VPT(c.vpt, MAXV, (softmax_bwd_resident<T, VPT, false, false><<<gr, c.threads, 0, st>>>(pg, py, out, outer, cols, out_f32))) }
      }
      return check_launch();
    }
  }
  const bool same_phase = (((reinterpret_cast<uintptr_t>(g) ^ reinterpret_cast<uintptr_t>(y)) | (reinterpret_cast<uintptr_t>(g) ^ reinterpret_cast<uintptr_t>(out))) & 15u) == 0;
  // shorter rows are a warp's work (the kernel below); a CTA for each would idle most of its threads
  if (inner == 1 && dto == dti && same_phase && dim > kRaggedMaxCols && dim < (1LL << 30) && outer <= 0x7fffffffLL) {
    const int th = stream_threads(outer, dim / VE, 32);
    auto go = [&](auto kernel) { kernel<<<static_cast<unsigned>(outer), th, 0, st>>>(pg, py, static_cast<T*>(out), static_cast<int>(dim)); };
    if (dim / VE <= 4 * th) {
      if (is_log) go(softmax_bwd_stream<T, true, true>);
      else go(softmax_bwd_stream<T, false, true>);
    } else {
      if (is_log) go(softmax_bwd_stream<T, true, false>);
      else go(softmax_bwd_stream<T, false, false>);
    }
    return check_launch();
  }
  // (fewer columns: 32 of them to a CTA leave too few CTAs -- fp32 2000 x 333 took 23 us so, 15 us with
  // a warp per line)
  if (inner >= 64 && outer * inner >= 1024 && dto == dti && outer <= 65535) {
    T* po = static_cast<T*>(out);
    auto go = [&](auto word) {
      typedef decltype(word) W;
      const dim3 gr(grid_for(inner, 32 * (sizeof(W) / sizeof(T))), static_cast<unsigned>(outer));
      const int threads = cols_tile_threads(dim, static_cast<int64_t>(gr.x) * gr.y);
      if (is_log) softmax_bwd_cols_tile<T, W, true><<<gr, threads, 0, st>>>(pg, py, po, dim, inner);
      else softmax_bwd_cols_tile<T, W, false><<<gr, threads, 0, st>>>(pg, py, po, dim, inner);
    };
    if (cols_in_pairs<T>(inner, g, y, out)) go(uint32_t{});
    else go(typename std::conditional<sizeof(T) == 2, uint16_t, uint32_t>::type{});
    return check_launch();
  }
  const int64_t lines = outer * inner;
  if ((lines + 3) / 4 > 0x7fffffffLL) return B200_EINVAL;
  if (is_log) softmax_bwd_lines<T, true><<<grid_for(lines, 4), 128, 0, st>>>(pg, py, out, outer, dim, inner, dto);
  else softmax_bwd_lines<T, false><<<grid_for(lines, 4), 128, 0, st>>>(pg, py, out, outer, dim, inner, dto);
  return check_launch();
}

template <typename T, typename TW, bool HOLD, bool AFFINE>
static int layernorm_launch(const T* px, const TW* pw, const TW* pb, T* py, void* mean, void* rstd, int64_t rows, int64_t cols, float eps, int dt_stat, const ResidentCfg& c, cudaStream_t st) {
  constexpr int VE = Vec<T>::N;
  constexpr int MAXV = 32 / VE;
  const float inv_cols = 1.f / static_cast<float>(cols);
  if (c.warp) {
    B200_DISPATCH_VPT(c.vpt, MAXV, (layernorm_resident<T, TW, VPT, true, HOLD, AFFINE><<<grid_for(rows, 4), 128, 0, st>>>(px, pw, pb, py, mean, rstd, rows, static_cast<int>(cols), inv_cols, eps, dt_stat)))
  } else if (AFFINE && !HOLD && c.vpt <= 2 && c.threads <= 256 && rows >= 8LL * kNumSMs) {
    // many 16-bit rows: persistent CTAs that keep weight and bias in registers (four CTAs per SM)
    const unsigned grid = static_cast<unsigned>(4 * kNumSMs);
    if (c.vpt == 1) layernorm_persistent<T, TW, 1><<<grid, c.threads, 0, st>>>(px, pw, pb, py, mean, rstd, rows, static_cast<int>(cols), inv_cols, eps, dt_stat);
    else layernorm_persistent<T, TW, 2><<<grid, c.threads, 0, st>>>(px, pw, pb, py, mean, rstd, rows, static_cast<int>(cols), inv_cols, eps, dt_stat);
  } else {
    B200_DISPATCH_VPT(c.vpt, MAXV, (layernorm_resident<T, TW, VPT, false, HOLD, AFFINE><<<static_cast<unsigned>(rows), c.threads, 0, st>>>(px, pw, pb, py, mean, rstd, rows, static_cast<int>(cols), inv_cols, eps, dt_stat)))
  }
  return check_launch();
}

template <typename T, typename TW>
static int layernorm_T(const void* x, const void* w, const void* b, void* y, void* mean, void* rstd, int64_t rows, int64_t cols, float eps, int dt_stat, const ResidentCfg& c, cudaStream_t st) {
  const T* px = static_cast<const T*>(x);
  const TW* pw = static_cast<const TW*>(w);
  const TW* pb = static_cast<const TW*>(b);
  T* py = static_cast<T*>(y);
  constexpr bool hold = sizeof(T) == 4;  // 16-bit rows stay packed: fewer registers, more resident warps
  const bool affine = w && b;
  return affine ? layernorm_launch<T, TW, hold, true>(px, pw, pb, py, mean, rstd, rows, cols, eps, dt_stat, c, st) : layernorm_launch<T, TW, hold, false>(px, pw, pb, py, mean, rstd, rows, cols, eps, dt_stat, c, st);
}

}  // namespace b200

using namespace b200;

extern "C" int b200_softmax(const void* x, void* out, int64_t outer, int64_t dim, int64_t inner, int dti, int dto, int is_log, void* stream) {
  if (outer < 0 || dim < 0 || inner < 0) return B200_EINVAL;
  if (!is_float_dtype(dti) || !(dto == dti || dto == B200_F32)) return B200_EDTYPE;
  if (outer == 0 || dim == 0 || inner == 0) return B200_OK;
  if (!x || !out) return B200_EINVAL;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (inner == 1 && dim <= kSmallRow && outer >= 4096)
    return is_log ? launch_rows_small<SMALL_LOGSOFTMAX>(x, out, outer, static_cast<int>(dim), dti, dto, nullptr, nullptr, 0, nullptr, nullptr, 0, 0.f, st)
                  : launch_rows_small<SMALL_SOFTMAX>(x, out, outer, static_cast<int>(dim), dti, dto, nullptr, nullptr, 0, nullptr, nullptr, 0, 0.f, st);
  switch (dti) {
    case B200_F32: return softmax_T<float>(x, out, outer, dim, inner, dto, is_log, st);
    case B200_BF16: return softmax_T<__nv_bfloat16>(x, out, outer, dim, inner, dto, is_log, st);
    default: return softmax_T<__half>(x, out, outer, dim, inner, dto, is_log, st);
  }
}

extern "C" int b200_softmax_backward(const void* grad, const void* output, void* grad_input, int64_t outer, int64_t dim, int64_t inner, int dti, int dto, int is_log, void* stream) {
  if (outer < 0 || dim < 0 || inner < 0) return B200_EINVAL;
  if (!is_float_dtype(dti) || !is_float_dtype(dto)) return B200_EDTYPE;
  if (outer == 0 || dim == 0 || inner == 0) return B200_OK;
  if (!grad || !output || !grad_input) return B200_EINVAL;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  switch (dti) {
    case B200_F32: return softmax_bwd_T<float>(grad, output, grad_input, outer, dim, inner, dti, dto, is_log, st);
    case B200_BF16: return softmax_bwd_T<__nv_bfloat16>(grad, output, grad_input, outer, dim, inner, dti, dto, is_log, st);
    default: return softmax_bwd_T<__half>(grad, output, grad_input, outer, dim, inner, dti, dto, is_log, st);
  }
}

extern "C" int64_t b200_reduce_scratch_bytes(int64_t outer, int64_t dim, int64_t inner) {
  if (outer <= 0 || dim <= 0 || inner <= 0) return 0;
  const ReducePlan p = plan_reduce(outer, dim, inner);
  return p.splits > 1 ? static_cast<int64_t>(p.splits) * outer * inner * 16 : 0;
}

extern "C" int b200_sum(const void* x, void* out, int64_t outer, int64_t dim, int64_t inner, int dti, int dto, void* scratch, int64_t scratch_bytes, void* stream) {
  if (outer < 0 || dim < 0 || inner < 0) return B200_EINVAL;
  if (!is_float_dtype(dti) || !is_float_dtype(dto)) return B200_EDTYPE;
  if (outer == 0 || inner == 0) return B200_OK;
  if (!out) return B200_EINVAL;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (dim == 0) {  // empty reduction: the sum is 0
    fill_zero_typed<<<grid_for(outer * inner, 256), 256, 0, st>>>(out, outer * inner, dto);
    return check_launch();
  }
  if (!x) return B200_EINVAL;
  if (inner == 1 && dim <= kSmallRow && outer >= 4096) return launch_rows_small<SMALL_SUM>(x, out, outer, static_cast<int>(dim), dti, dto, nullptr, nullptr, 0, nullptr, nullptr, 0, 0.f, st);
  switch (dti) {
    case B200_F32: return launch_reduce_T<float, false>(x, out, outer, dim, inner, dto, scratch, scratch_bytes, st);
    case B200_BF16: return launch_reduce_T<__nv_bfloat16, false>(x, out, outer, dim, inner, dto, scratch, scratch_bytes, st);
    default: return launch_reduce_T<__half, false>(x, out, outer, dim, inner, dto, scratch, scratch_bytes, st);
  }
}

extern "C" int b200_argmax(const void* x, int64_t* out, int64_t outer, int64_t dim, int64_t inner, int dt, void* scratch, int64_t scratch_bytes, void* stream) {
  if (outer < 0 || dim <= 0 || inner < 0) return B200_EINVAL;
  if (!is_float_dtype(dt)) return B200_EDTYPE;
  if (outer == 0 || inner == 0) return B200_OK;
  if (!x || !out) return B200_EINVAL;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (inner == 1 && dim <= kSmallRow && outer >= 4096) return launch_rows_small<SMALL_ARGMAX>(x, out, outer, static_cast<int>(dim), dt, B200_I64, nullptr, nullptr, 0, nullptr, nullptr, 0, 0.f, st);
  switch (dt) {
    case B200_F32: return launch_reduce_T<float, true>(x, out, outer, dim, inner, B200_I64, scratch, scratch_bytes, st);
    case B200_BF16: return launch_reduce_T<__nv_bfloat16, true>(x, out, outer, dim, inner, B200_I64, scratch, scratch_bytes, st);
    default: return launch_reduce_T<__half, true>(x, out, outer, dim, inner, B200_I64, scratch, scratch_bytes, st);
  }
}

// Rows off the 16-byte grid, a CTA each: eight elements per thread, or as many as 128 threads leave
constexpr int64_t kLnRowsMax = 8192;
static int ln_rows_threads(int64_t cols, int e, int npt) { return static_cast<int>(((cols / e + npt - 1) / npt + 31) / 32 * 32); }
// go(elements of a chunk, chunks of a thread): 8 elements per thread from 1024 columns on, 4 and 2 below
template <typename T, typename Go>
static void with_ln_chunks(bool pairs, int64_t cols, int64_t per_thread8, Go go) {
  const int elems = cols > per_thread8 / 2 ? 8 : cols > per_thread8 / 4 ? 4 : 2;
  if constexpr (sizeof(T) == 2) {
    if (pairs) {
      if (elems == 8) go(std::integral_constant<int, 2>{}, std::integral_constant<int, 4>{});
      else if (elems == 4) go(std::integral_constant<int, 2>{}, std::integral_constant<int, 2>{});
      else go(std::integral_constant<int, 2>{}, std::integral_constant<int, 1>{});
      return;
    }
  }
  if (elems == 8) go(std::integral_constant<int, 1>{}, std::integral_constant<int, 8>{});
  else if (elems == 4) go(std::integral_constant<int, 1>{}, std::integral_constant<int, 4>{});
  else go(std::integral_constant<int, 1>{}, std::integral_constant<int, 2>{});
}
static bool ln_pairs(int64_t cols, std::initializer_list<const void*> ps) {
  uintptr_t m = static_cast<uintptr_t>(cols) * 2;
  for (const void* p : ps) m |= reinterpret_cast<uintptr_t>(p);
  return (m & 3u) == 0;
}
template <typename T, typename TW>
static void layernorm_rows_launch(const void* x, const void* w, const void* b, void* y, void* mean, void* rstd, int64_t rows, int cols, float eps, int dt_stat, cudaStream_t st) {
  with_ln_chunks<T>(ln_pairs(cols, {x, y}), cols, 1024, [&](auto e, auto npt) {
    constexpr int E = decltype(e)::value, NPT = decltype(npt)::value;
    layernorm_rows<T, TW, E, NPT><<<static_cast<unsigned>(rows), ln_rows_threads(cols, E, NPT), 0, st>>>(static_cast<const T*>(x), static_cast<const TW*>(w), static_cast<const TW*>(b), static_cast<T*>(y), mean,
                                                                                                         rstd, cols, eps, dt_stat);
  });
}

extern "C" int b200_layer_norm(const void* x, const void* w, const void* b, void* y, void* mean, void* rstd, int64_t rows, int64_t cols, double eps, int dt, int dt_wb, int dt_stat, void* stream) {
  if (rows < 0 || cols < 0) return B200_EINVAL;
  if (!is_float_dtype(dt) || !is_float_dtype(dt_stat) || ((w || b) && !is_float_dtype(dt_wb))) return B200_EDTYPE;
  if (rows == 0) return B200_OK;
  if (!mean || !rstd) return B200_EINVAL;
  if (cols > 0 && (!x || !y)) return B200_EINVAL;
  if (rows > 0x7fffffffLL) return B200_EINVAL;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const float e = static_cast<float>(eps);
  if (cols > 0 && cols <= kSmallRow && rows >= 4096) return launch_rows_small<SMALL_LAYERNORM>(x, y, rows, static_cast<int>(cols), dt, dt, w, b, dt_wb, mean, rstd, dt_stat, e, st);
  const int ve = 16 / dtype_size(dt);
  const bool wb_ok = (!w && !b) || dt_wb == dt || dt_wb == B200_F32;
  const bool al = aligned16(x) && aligned16(y) && (!w || aligned16(w)) && (!b || aligned16(b));
  ResidentCfg c{false, false, 1, 128};
  if (cols > 0 && cols % ve == 0 && (dt_wb != B200_F32 || cols % 4 == 0) && al && wb_ok && cols < (1LL << 30)) c = resident_cfg(cols / ve, 32 / ve, ve == 4 ? 4 : 2);
  // ragged rows: a warp each where they are short and many, a CTA each elsewhere (bf16 20000 x 70 8.4 us against 12.7, 20000 x 301 26.4 / 18.4,
  // 300 x 70 4.1 / 2.8). The shorter they are, the fewer it takes: 2760 x 1 2.6 / 3.4, 3264 x 2 2.5 / 3.4, 2333 x 23 2.4 / 3.0, 952 x 4 2.2 / 2.5, 414 x 19 2.2 / 2.3;
  // 1762 x 37 2.9 / 3.0, 652 x 44 2.8 / 2.6; 3632 x 95 3.9 / 4.1, 2392 x 71 3.8 / 3.3.
  if (!c.ok && cols > 0 && cols <= 256 && rows >= (cols <= 32 ? 768 : cols <= 64 ? 2048 : 4096)) {
    const unsigned g = grid_for(rows, 4);
    const int ci = static_cast<int>(cols);
    auto go = [&](auto npl) {
      constexpr int NPL = decltype(npl)::value;
      switch (dt) {
        case B200_F32: layernorm_warp_ragged<float, NPL><<<g, 128, 0, st>>>(static_cast<const float*>(x), w, b, static_cast<float*>(y), mean, rstd, rows, ci, e, dt_wb, dt_stat); break;
        case B200_BF16: layernorm_warp_ragged<__nv_bfloat16, NPL><<<g, 128, 0, st>>>(static_cast<const __nv_bfloat16*>(x), w, b, static_cast<__nv_bfloat16*>(y), mean, rstd, rows, ci, e, dt_wb, dt_stat); break;
        default: layernorm_warp_ragged<__half, NPL><<<g, 128, 0, st>>>(static_cast<const __half*>(x), w, b, static_cast<__half*>(y), mean, rstd, rows, ci, e, dt_wb, dt_stat); break;
      }
    };
    if (cols <= 64) go(std::integral_constant<int, 2>{});
    else if (cols <= 128) go(std::integral_constant<int, 4>{});
    else go(std::integral_constant<int, 8>{});
    return check_launch();
  }
  if (!c.ok && cols > 0 && cols <= kLnRowsMax && wb_ok) {
    const bool f32 = (w || b) && dt_wb == B200_F32;
    switch (dt) {
      case B200_F32: layernorm_rows_launch<float, float>(x, w, b, y, mean, rstd, rows, static_cast<int>(cols), e, dt_stat, st); break;
      case B200_BF16:
        if (f32) layernorm_rows_launch<__nv_bfloat16, float>(x, w, b, y, mean, rstd, rows, static_cast<int>(cols), e, dt_stat, st);
        else layernorm_rows_launch<__nv_bfloat16, __nv_bfloat16>(x, w, b, y, mean, rstd, rows, static_cast<int>(cols), e, dt_stat, st);
        break;
      default:
        if (f32) layernorm_rows_launch<__half, float>(x, w, b, y, mean, rstd, rows, static_cast<int>(cols), e, dt_stat, st);
        else layernorm_rows_launch<__half, __half>(x, w, b, y, mean, rstd, rows, static_cast<int>(cols), e, dt_stat, st);
        break;
    }
    return check_launch();
  }
  if (!c.ok) {
    layernorm_stream<<<static_cast<unsigned>(rows), 256, 0, st>>>(x, w, b, y, mean, rstd, cols, e, dt, dt_wb, dt_stat);
    return check_launch();
  }
  const bool wf32 = (w || b) && dt_wb == B200_F32;
  switch (dt) {
    case B200_F32: return layernorm_T<float, float>(x, w, b, y, mean, rstd, rows, cols, e, dt_stat, c, st);
    case B200_BF16:
      return wf32 ? layernorm_T<__nv_bfloat16, float>(x, w, b, y, mean, rstd, rows, cols, e, dt_stat, c, st)
                  : layernorm_T<__nv_bfloat16, __nv_bfloat16>(x, w, b, y, mean, rstd, rows, cols, e, dt_stat, c, st);
    default:
      return wf32 ? layernorm_T<__half, float>(x, w, b, y, mean, rstd, rows, cols, e, dt_stat, c, st)
                  : layernorm_T<__half, __half>(x, w, b, y, mean, rstd, rows, cols, e, dt_stat, c, st);
  }
}

// ---- layer norm backward: host side
static const int64_t kLnBwdMaxParts = 8LL * kNumSMs;  // partial rows of dw / db in scratch

extern "C" int64_t b200_layer_norm_backward_scratch_bytes(int64_t rows, int64_t cols) {
  if (rows <= 0 || cols <= 0) return 0;
  const int64_t parts = rows < kLnBwdMaxParts ? rows : kLnBwdMaxParts;
  return parts * cols * 2 * 4;
}

// The fused kernel for a row of `threads` threads: a 16-bit row always is one vector per thread.
// 16-bit rows of more than one warp: the sums behind one barrier and the statistics a row ahead (bf16 8192 x
// 4096 53.7 -> 51.3 us, 60000 x 768 84.3 -> 82.0). One warp to a row (20000 x 256: 32.5 us so, 31.0 one sum after the other)
// and fp32 rows (65536 x 1024 153, 144) have no barrier worth saving, or many small CTAs to hide it.
template <typename T, typename TW, typename Go>
static void with_layernorm_bwd_fused(int threads, int vpt, Go go) {
  if constexpr (sizeof(T) == 2) {
    if (threads > 32) go(layernorm_bwd_fused<T, TW, 1, true>);
    else go(layernorm_bwd_fused<T, TW, 1, false>);
  } else {
    if (vpt == 1) go(layernorm_bwd_fused<T, TW, 1, false>);
    else go(layernorm_bwd_fused<T, TW, 2, false>);
  }
}
template <typename T, typename TW>
static void layernorm_bwd_fused_launch(const void* dy, const void* x, const void* w, const void* mean, const void* rstd, void* dx, float* pw, float* pb, int64_t rows, int64_t cols, int dt_stat,
                                       int threads, int vpt, int grid, cudaStream_t st) {
  with_layernorm_bwd_fused<T, TW>(threads, vpt, [&](auto kernel) {
    kernel<<<grid, threads, 0, st>>>(static_cast<const T*>(dy), static_cast<const T*>(x), static_cast<const TW*>(w), mean, rstd, static_cast<T*>(dx), pw, pb, rows, static_cast<int>(cols), dt_stat);
  });
}
// CTAs of the fused kernel one SM holds at this block size (registers decide).
template <typename T, typename TW>
static int layernorm_bwd_fused_per_sm(int threads, int vpt) {
  int n = 0;
  cudaError_t e = cudaErrorUnknown;
  with_layernorm_bwd_fused<T, TW>(threads, vpt, [&](auto kernel) { e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, threads, 0); });
  return e == cudaSuccess && n > 0 ? n : 1;
}

// Launches layernorm_bwd_rows; the number of partial rows.
template <typename T, int E, int NPT, bool WARP>
static int64_t layernorm_bwd_rows_go(const void* dy, const void* x, const void* w, const void* mean, const void* rstd, void* dx, float* pw, float* pb, int64_t rows, int cols, int dt_wb, int dt_stat,
                                     int64_t parts_max, cudaStream_t st) {
  auto kernel = layernorm_bwd_rows<T, E, NPT, WARP>;
  const int threads = WARP ? 256 : ln_rows_threads(cols, E, NPT);
  int per_sm = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, 0) != cudaSuccess || per_sm < 1) per_sm = 1;
  int64_t grid = static_cast<int64_t>(per_sm > 8 ? 8 : per_sm) * kNumSMs;
  const int64_t need = WARP ? (rows + 7) / 8 : rows;
  if (grid > need) grid = need;
  if (grid > parts_max) grid = parts_max;
  kernel<<<static_cast<unsigned>(grid), threads, 0, st>>>(static_cast<const T*>(dy), static_cast<const T*>(x), w, mean, rstd, static_cast<T*>(dx), pw, pb, rows, cols, dt_wb, dt_stat);
  return grid;
}
template <typename T>
static int64_t layernorm_bwd_rows_launch(const void* dy, const void* x, const void* w, const void* mean, const void* rstd, void* dx, float* pw, float* pb, int64_t rows, int cols, int dt_wb, int dt_stat,
                                         bool vectors, int64_t parts_max, cudaStream_t st) {
  constexpr int VE = Vec<T>::N;
  int64_t parts = 0;
  auto go = [&](auto e, auto npt, auto warp) {
    parts = layernorm_bwd_rows_go<T, decltype(e)::value, decltype(npt)::value, decltype(warp)::value>(dy, x, w, mean, rstd, dx, pw, pb, rows, cols, dt_wb, dt_stat, parts_max, st);
  };
  if (vectors) {  // at most 256 columns
    if (cols <= 32 * VE) go(std::integral_constant<int, VE>{}, std::integral_constant<int, 1>{}, std::true_type{});
    else if constexpr (VE == 4) go(std::integral_constant<int, VE>{}, std::integral_constant<int, 2>{}, std::true_type{});
  } else if (cols <= 256) {
    with_ln_chunks<T>(ln_pairs(cols, {dy, x, dx}), cols, 256, [&](auto e, auto npt) { go(e, npt, std::true_type{}); });
  } else {
    with_ln_chunks<T>(ln_pairs(cols, {dy, x, dx}), cols, 1024, [&](auto e, auto npt) { go(e, npt, std::false_type{}); });
  }
  return parts;
}

extern "C" int b200_layer_norm_backward(const void* dy, const void* x, const void* mean, const void* rstd, const void* w, void* dx, void* dw, void* db, int64_t rows, int64_t cols, int dt,
                                        int dt_wb, int dt_stat, void* scratch, int64_t scratch_bytes, void* stream) {
  if (rows < 0 || cols < 0) return B200_EINVAL;
  if (!is_float_dtype(dt) || !is_float_dtype(dt_stat) || ((w || dw || db) && !is_float_dtype(dt_wb))) return B200_EDTYPE;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (cols == 0) return B200_OK;
  if (rows == 0) {  // nothing to sum: the parameter gradients are zero
    if (dw) fill_zero_typed<<<grid_for(cols, 256), 256, 0, st>>>(dw, cols, dt_wb);
    if (db) fill_zero_typed<<<grid_for(cols, 256), 256, 0, st>>>(db, cols, dt_wb);
    return check_launch();
  }
  if (!dy || !x || !mean || !rstd) return B200_EINVAL;
  const bool need_wb = dw || db;
  const int64_t parts_max = rows < kLnBwdMaxParts ? rows : kLnBwdMaxParts;
  float* pw = nullptr;
  float* pb = nullptr;
  if (need_wb) {
    if (!scratch || scratch_bytes < b200_layer_norm_backward_scratch_bytes(rows, cols)) return B200_ESCRATCH;
    pw = static_cast<float*>(scratch);
    pb = pw + parts_max * cols;
  }
  const int ve = 16 / dtype_size(dt);
  const bool wb_ok = !w || dt_wb == dt || dt_wb == B200_F32;
  const bool al = aligned16(dy) && aligned16(x) && (!dx || aligned16(dx)) && (!w || aligned16(w));
  int64_t parts = 0;
  // a thread keeps five values per owned column in registers (dy, xhat, w, and its share of dw
  // and db): one 16-byte vector of a 16-bit row, two of an fp32 row -- rows of up to 8192
  // elements; longer ones would spill
  const int target = ve == 4 ? 2 : 1;
  const bool vectors = cols % ve == 0 && al;
  if (vectors ? cols <= 256 && rows >= 64 : cols <= kLnRowsMax) {
    const int ci = static_cast<int>(cols);
    switch (dt) {
      case B200_F32: parts = layernorm_bwd_rows_launch<float>(dy, x, w, mean, rstd, dx, pw, pb, rows, ci, dt_wb, dt_stat, vectors, parts_max, st); break;
      case B200_BF16: parts = layernorm_bwd_rows_launch<__nv_bfloat16>(dy, x, w, mean, rstd, dx, pw, pb, rows, ci, dt_wb, dt_stat, vectors, parts_max, st); break;
      default: parts = layernorm_bwd_rows_launch<__half>(dy, x, w, mean, rstd, dx, pw, pb, rows, ci, dt_wb, dt_stat, vectors, parts_max, st); break;
    }
  } else if (vectors && (dt_wb != B200_F32 || !w || cols % 4 == 0) && wb_ok && cols / ve <= 1024 * target) {
    const int64_t nvec = cols / ve;
    int threads = 32;
    while (threads < 1024 && threads * target < nvec) threads <<= 1;
    const int vpt = static_cast<int>((nvec + threads - 1) / threads);
    const bool wf32 = w && dt_wb == B200_F32;
    int per_sm = 1;
    switch (dt) {
      case B200_F32: per_sm = layernorm_bwd_fused_per_sm<float, float>(threads, vpt); break;
      case B200_BF16: per_sm = wf32 ? layernorm_bwd_fused_per_sm<__nv_bfloat16, float>(threads, vpt) : layernorm_bwd_fused_per_sm<__nv_bfloat16, __nv_bfloat16>(threads, vpt); break;
      default: per_sm = wf32 ? layernorm_bwd_fused_per_sm<__half, float>(threads, vpt) : layernorm_bwd_fused_per_sm<__half, __half>(threads, vpt); break;
    }
    if (per_sm > 8) per_sm = 8;
    parts = static_cast<int64_t>(per_sm) * kNumSMs;  // a persistent grid: exactly what the device holds at once
    if (parts > parts_max) parts = parts_max;
    const int grid = static_cast<int>(parts);
    switch (dt) {
      case B200_F32: layernorm_bwd_fused_launch<float, float>(dy, x, w, mean, rstd, dx, pw, pb, rows, cols, dt_stat, threads, vpt, grid, st); break;
      case B200_BF16:
        if (wf32) layernorm_bwd_fused_launch<__nv_bfloat16, float>(dy, x, w, mean, rstd, dx, pw, pb, rows, cols, dt_stat, threads, vpt, grid, st);
        else layernorm_bwd_fused_launch<__nv_bfloat16, __nv_bfloat16>(dy, x, w, mean, rstd, dx, pw, pb, rows, cols, dt_stat, threads, vpt, grid, st);
        break;
      default:
        if (wf32) layernorm_bwd_fused_launch<__half, float>(dy, x, w, mean, rstd, dx, pw, pb, rows, cols, dt_stat, threads, vpt, grid, st);
        else layernorm_bwd_fused_launch<__half, __half>(dy, x, w, mean, rstd, dx, pw, pb, rows, cols, dt_stat, threads, vpt, grid, st);
        break;
    }
  } else {
    if (dx) {
      const int64_t g = rows < 8LL * kNumSMs ? rows : 8LL * kNumSMs;
      layernorm_bwd_dx_lines<<<static_cast<int>(g), 256, 0, st>>>(dy, x, w, mean, rstd, dx, rows, cols, dt, dt_wb, dt_stat);
    }
    if (need_wb) {
      parts = parts_max < 64 ? parts_max : 64;
      const int64_t rows_per = (rows + parts - 1) / parts;
      parts = (rows + rows_per - 1) / rows_per;
      const int64_t gx = (cols + 255) / 256;
      if (gx > 0x7fffffffLL) return B200_EINVAL;
      layernorm_bwd_wb_lines<<<dim3(static_cast<unsigned>(gx), static_cast<unsigned>(parts)), 256, 0, st>>>(dy, x, mean, rstd, pw, pb, rows, cols, rows_per, dt, dt_stat);
    }
  }
  if (need_wb) {
    auto finalize = [&](auto kernel, int w) -> cudaError_t {
      if (parts > 32) return launch_after(kernel, grid_for(cols, w), 1024, 0, st, pw, pb, dw, db, parts, cols, dt_wb);
      kernel<<<grid_for(cols, w), 1024, 0, st>>>(pw, pb, dw, db, parts, cols, dt_wb);
      return cudaSuccess;
    };
    const cudaError_t e = parts > 32 && cols < 32 * (kNumSMs / 2) ? finalize(layernorm_bwd_finalize<8>, 8) : finalize(layernorm_bwd_finalize<32>, 32);
    if (e != cudaSuccess) { set_last_cuda_error(e); return B200_ELAUNCH; }
  }
  return check_launch(need_wb ? 2 : 1);
}

// ------------------------------------------------------------------ sum without any allocation
// Scratch for the split-reduction partials of b200_sum_static. It lives in the library
// image: every GPU that loads the library holds these bytes until the process exits.
static __device__ __align__(256) unsigned char g_sum_static_scratch[B200_STATIC_SCRATCH_BYTES];

// Device address of the array above on the CURRENT device. In host code the array's name
// is only a handle, not something a kernel can dereference, so the address is asked for
// once per device (cudaGetSymbolAddress, return code checked) and remembered.
static void* sum_static_scratch_address(void) {
  static std::mutex mu;
  static void* per_device[64] = {};
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess || dev < 0 || dev >= 64) {
    set_last_cuda_error(e != cudaSuccess ? e : cudaErrorInvalidDevice);
    return nullptr;
  }
  std::lock_guard<std::mutex> lock(mu);
  if (!per_device[dev]) {
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, g_sum_static_scratch);
    if (e != cudaSuccess || !p) {
      set_last_cuda_error(e);
      return nullptr;
    }
    per_device[dev] = p;
  }
  return per_device[dev];
}

extern "C" int b200_sum_static(const void* x, void* out, int64_t outer, int64_t dim, int64_t inner, int dti, int dto, void* stream) {
  const int64_t need = b200_reduce_scratch_bytes(outer, dim, inner);
  if (need > B200_STATIC_SCRATCH_BYTES) return B200_ESCRATCH;
  void* scratch = nullptr;
  if (need > 0) {
    scratch = sum_static_scratch_address();
    if (!scratch) return B200_ELAUNCH;
  }
  // every partial slot is written by the first stage before the second stage reads it, so
  // whatever an earlier call left in the array never needs clearing
  return b200_sum(x, out, outer, dim, inner, dti, dto, scratch, need > 0 ? B200_STATIC_SCRATCH_BYTES : 0, stream);
}
