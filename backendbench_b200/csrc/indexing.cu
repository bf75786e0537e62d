// embedding / index_select / gather: bit-exact data movement driven by integer indices.
//
// Rows (embedding, index_select dim 0) are copied with 16-byte accesses, one CTA per
// output row when rows are wide (>= 1 KB) and a flattened (row, vector) space when they
// are narrow, so loads within a row and all stores are coalesced. gather moves single
// elements: index reads and output writes are coalesced, source reads hit one 32-byte
// sector each and are served by L2 when the source fits there.
// An index outside [0, size) never faults: the element/row is written as zero and
// B200_DEV_INDEX_OOB is OR-ed into the caller's status word. Negative indices are out of
// range here, as they are for the aten CPU kernels.
#include <cstdlib>

#include "b200_common.cuh"
#include "tma_common.cuh"

namespace b200 {

__device__ __forceinline__ int64_t load_index(const void* idx, int64_t i, int idx_i32) {
  return idx_i32 ? static_cast<int64_t>(static_cast<const int32_t*>(idx)[i]) : static_cast<const int64_t*>(idx)[i];
}
__device__ __forceinline__ void flag_oob(uint32_t* status) {
  if (status) atomicOr(status, B200_DEV_INDEX_OOB);
}
// The gathered-from tensor is re-read at random while index and output stream through once:
// pin the former in L2 (evict_last) so the streams do not push it out.
__device__ __forceinline__ uint64_t l2_keep_policy() {
  uint64_t pol;
  asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(pol));
  return pol;
}
__device__ __forceinline__ uint32_t ld_keep_l2(const uint32_t* p, uint64_t pol) {
  uint32_t v;
  asm volatile("ld.global.nc.L2::cache_hint.u32 %0, [%1], %2;" : "=r"(v) : "l"(p), "l"(pol));
  return v;
}
__device__ __forceinline__ uint16_t ld_keep_l2(const uint16_t* p, uint64_t pol) {
  uint16_t v;
  asm volatile("ld.global.nc.L2::cache_hint.u16 %0, [%1], %2;" : "=h"(v) : "l"(p), "l"(pol));
  return v;
}
template <typename U> __device__ __forceinline__ U zero_of() { U z; memset(&z, 0, sizeof(U)); return z; }

// One CTA (128 threads) per output row; rows are `nvec` 16-byte vectors.
__global__ void __launch_bounds__(128) gather_rows_wide(const uint4* __restrict__ table, const void* __restrict__ idx, uint4* __restrict__ out,
                                                        int64_t table_rows, int64_t nvec, int64_t n_idx, int idx_i32, uint32_t* status) {
  for (int64_t r = blockIdx.x; r < n_idx; r += gridDim.x) {
    const int64_t src = load_index(idx, r, idx_i32);
    const bool ok = src >= 0 && src < table_rows;
    if (!ok && threadIdx.x == 0) flag_oob(status);
    const uint4* s = table + (ok ? src : 0) * nvec;
    uint4* d = out + r * nvec;
    int64_t j = threadIdx.x;
    for (; j + 3 * 128 < nvec; j += 4 * 128) {
      uint4 v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) v[u] = ok ? __ldcs(s + j + u * 128) : make_uint4(0, 0, 0, 0);
#pragma unroll
      for (int u = 0; u < 4; ++u) __stcs(d + j + u * 128, v[u]);
    }
    for (; j < nvec; j += 128) __stcs(d + j, ok ? __ldcs(s + j) : make_uint4(0, 0, 0, 0));
  }
}

// Flattened index_select: x is [outer, dim_size, inner] in units of U, out is
// [outer, n_idx, inner]. A thread has W units in flight, the index of each before any of
// the units, and 32-bit coordinates wherever they suffice (two 64-bit divisions per unit were most
// of the time: f16 150134 x 63, 75067 rows picked, 22.7 -> 17.5 us).
// W = 4 from 2^18 units on; with fewer, the SMs are not full and a thread's four units only take
// longer than four threads' (fp32 5000 x 16, 5000 rows: 2.3 us with one, 3.2 with four; 64 x 300 x 33,
// 150 picked, 4.1 with one, 3.6 with four).
constexpr int kFlatUnroll = 4;
constexpr int64_t kFlatUnrollMin = 1 << 18;
template <typename U, int W>
__global__ void __launch_bounds__(256) index_select_flat(const U* __restrict__ x, const void* __restrict__ idx, U* __restrict__ out, int64_t outer, int64_t dim_size,
                                                         int64_t inner, int64_t n_idx, int idx_i32, uint32_t* status) {
  const int64_t total = outer * n_idx * inner;
  const bool small = total <= 0x7fffffffLL;
  for (int64_t p0 = static_cast<int64_t>(blockIdx.x) * (256 * W) + threadIdx.x; p0 < total; p0 += static_cast<int64_t>(gridDim.x) * (256 * W)) {
    int64_t src[W], at[W];
    U v[W];
#pragma unroll
    for (int u = 0; u < W; ++u) {
      const int64_t p = p0 + u * 256;
      src[u] = -2;  // past the end
      if (p < total) {
        int64_t o, k, i;
        if (small) {
          const uint32_t q = static_cast<uint32_t>(p) / static_cast<uint32_t>(inner);
          const uint32_t qo = outer == 1 ? 0u : q / static_cast<uint32_t>(n_idx);
          i = static_cast<uint32_t>(p) - q * static_cast<uint32_t>(inner);
          k = q - qo * static_cast<uint32_t>(n_idx);
          o = qo;
        } else {
          const int64_t q = p / inner;
          o = q / n_idx;
          k = q - o * n_idx;
          i = p - q * inner;
        }
        src[u] = load_index(idx, k, idx_i32);
        at[u] = o * dim_size * inner + i;
        if (src[u] < 0 || src[u] >= dim_size) {
          flag_oob(status);
          src[u] = -1;
        }
      }
    }
#pragma unroll
    for (int u = 0; u < W; ++u) v[u] = src[u] >= 0 ? x[at[u] + src[u] * inner] : zero_of<U>();
#pragma unroll
    for (int u = 0; u < W; ++u)
      if (src[u] > -2) out[p0 + u * 256] = v[u];
  }
}

// Rows off the 16-byte grid (126 bytes, say): a thread produces 16 bytes of the result, wherever they lie in it. They come
// from one row, or from the end of one and the beginning of the next, and each part from the one or two aligned
// 16-byte blocks around it, moved by as many bytes as source and result differ; only blocks that hold
// a byte of the part are read. Element by element the kernel above is bound by its instructions: f16
// 150134 x 63, 75067 rows 14.9 us, 9.0 so; 56 x 3527, 21648 rows 198 and 64. From 2^20 units on: with fewer, a thread's
// chain of index, blocks and shifts takes longer than a thread for each unit (fp32 5000 x 130 3.6 us, 4.5 so).
struct Block32 {
  uint32_t w[8];
};
// bytes [sh, sh + 16) of two blocks, the words of which are in w[0..7]
__device__ __forceinline__ uint4 bytes_from(Block32 b, uint32_t sh) {
  if (sh & 4u) {
#pragma unroll
    for (int i = 0; i < 7; ++i) b.w[i] = b.w[i + 1];
  }
  if (sh & 8u) {
#pragma unroll
    for (int i = 0; i < 5; ++i) b.w[i] = b.w[i + 2];
  }
  const uint32_t bits = (sh & 3u) * 8;
  return make_uint4(__funnelshift_r(b.w[0], b.w[1], bits), __funnelshift_r(b.w[1], b.w[2], bits), __funnelshift_r(b.w[2], b.w[3], bits), __funnelshift_r(b.w[3], b.w[4], bits));
}
// The 16 bytes at `at`, of which [lo, hi) count
__device__ __forceinline__ uint4 bytes_at(const unsigned char* at, int lo, int hi) {
  const uint32_t sh = static_cast<uint32_t>(reinterpret_cast<uintptr_t>(at)) & 15u;
  const uint4* block = reinterpret_cast<const uint4*>(at - sh);
  uint4 a = make_uint4(0, 0, 0, 0), b = a;
  if (static_cast<int>(sh) + lo < 16) a = __ldg(block);
  if (static_cast<int>(sh) + hi > 16) b = __ldg(block + 1);
  return bytes_from(Block32{{a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w}}, sh);
}
constexpr int kRaggedUnroll = 2;
constexpr int64_t kRaggedMinUnits = 1 << 20;
__global__ void __launch_bounds__(256) select_rows_ragged(const unsigned char* __restrict__ x, const void* __restrict__ idx, unsigned char* __restrict__ out, int64_t outer, int64_t dim_size,
                                                          int64_t row_bytes, int64_t n_idx, int idx_i32, uint32_t* status) {
  const int64_t total = outer * n_idx * row_bytes, vecs = (total + 15) / 16, step = static_cast<int64_t>(gridDim.x) * 256;
  const bool small = total <= 0x7fffffffLL;
  // the row `q` of the result: where it lies in x, NULL: an index out of range
  auto source = [&](int64_t q) -> const unsigned char* {
    const int64_t o = outer == 1 ? 0 : q / n_idx, k = load_index(idx, q - o * n_idx, idx_i32);
    if (k < 0 || k >= dim_size) {
      flag_oob(status);
      return nullptr;
    }
    return x + (o * dim_size + k) * row_bytes;
  };
  for (int64_t v0 = static_cast<int64_t>(blockIdx.x) * 256 + threadIdx.x; v0 < vecs; v0 += kRaggedUnroll * step) {
    const unsigned char *one[kRaggedUnroll], *two[kRaggedUnroll];
    int first[kRaggedUnroll];  // bytes of the vector that lie in the first row
    uint4 r[kRaggedUnroll];
#pragma unroll
    for (int u = 0; u < kRaggedUnroll; ++u) {
      const int64_t v = v0 + u * step;
      one[u] = two[u] = nullptr;
      first[u] = 16;
      if (v < vecs) {
        const int64_t p = v * 16, q = small ? static_cast<int64_t>(static_cast<uint32_t>(p) / static_cast<uint32_t>(row_bytes)) : p / row_bytes;
        const int64_t in_row = p - q * row_bytes;
        one[u] = source(q);
        if (one[u]) one[u] += in_row;
        if (row_bytes - in_row < 16) {
          first[u] = static_cast<int>(row_bytes - in_row);
          if (p + first[u] < total) two[u] = source(q + 1);
        }
      }
    }
#pragma unroll
    for (int u = 0; u < kRaggedUnroll; ++u) {
      r[u] = make_uint4(0, 0, 0, 0);
      if (one[u]) r[u] = bytes_at(one[u], 0, first[u]);
      if (first[u] < 16) {
        uint4 s = make_uint4(0, 0, 0, 0);
        if (two[u]) s = bytes_at(two[u] - first[u], first[u], 16);
        // byte i is the first row's for i < first
        auto merge = [&](uint32_t a, uint32_t b, int at) {
          const int keep = first[u] - at;
          const uint32_t mask = keep >= 4 ? 0xffffffffu : keep <= 0 ? 0u : (1u << (8 * keep)) - 1u;
          return (a & mask) | (b & ~mask);
        };
        r[u] = make_uint4(merge(r[u].x, s.x, 0), merge(r[u].y, s.y, 4), merge(r[u].z, s.z, 8), merge(r[u].w, s.w, 12));
      }
    }
#pragma unroll
    for (int u = 0; u < kRaggedUnroll; ++u) {
      const int64_t v = v0 + u * step, p = v * 16;
      if (v >= vecs) break;
      if (p + 16 <= total) {
        __stcs(reinterpret_cast<uint4*>(out + p), r[u]);
      } else {  // the result ends inside the last vector
        const uint32_t w[4] = {r[u].x, r[u].y, r[u].z, r[u].w};
#pragma unroll
        for (int i = 0; i < 16; ++i)
          if (p + i < total) out[p + i] = static_cast<unsigned char>(w[i >> 2] >> (8 * (i & 3)));
      }
    }
  }
}

struct GatherArgs {
  int ndim, dim;
  int64_t n;
  int64_t shape[B200_MAX_DIMS], self_stride[B200_MAX_DIMS], idx_stride[B200_MAX_DIMS];
  int64_t self_dim_size;
};

// Any layout: a thread has W elements in flight (W indices, then W elements of self). Four where
// there are enough of them (as above; 300 x 333 2.7 us with one, 3.7 with four): f16 150134 x 63 along dim
// 0, 75067 rows of indices, 38.1 -> 32.9 us. Where the index is not read along its rows,
// threads of different CTAs share its sectors and four at a time make them meet later: only for results of 16 MB or
// more (transposed views in fp32: 40000 x 100, 20000 rows, 22 us with one, 25 with four; 150134 x 63, 75067 rows, 57 / 52).
template <typename U, int W>
__global__ void __launch_bounds__(256) gather_generic(const U* __restrict__ self, const int64_t* __restrict__ index, U* __restrict__ out, const __grid_constant__ GatherArgs A, uint32_t* status) {
  for (int64_t p0 = static_cast<int64_t>(blockIdx.x) * (256 * W) + threadIdx.x; p0 < A.n; p0 += static_cast<int64_t>(gridDim.x) * (256 * W)) {
    int64_t io[W], so[W], k[W];
    U v[W];
#pragma unroll
    for (int u = 0; u < W; ++u) {
      const int64_t p = p0 + u * 256;
      io[u] = so[u] = 0;
      if (A.n <= 0x7fffffffLL) {  // coordinates by 32-bit division (a 64-bit one costs ~5x the instructions)
        uint32_t lin = static_cast<uint32_t>(p);
        for (int d = A.ndim - 1; d >= 0; --d) {
          const uint32_t ext = static_cast<uint32_t>(A.shape[d]);
          const uint32_t q = lin / ext, r = lin - q * ext;
          io[u] += r * A.idx_stride[d];
          if (d != A.dim) so[u] += r * A.self_stride[d];
          lin = q;
        }
      } else {
        int64_t lin = p;
        for (int d = A.ndim - 1; d >= 0; --d) {
          const int64_t q = lin / A.shape[d], r = lin - q * A.shape[d];
          io[u] += r * A.idx_stride[d];
          if (d != A.dim) so[u] += r * A.self_stride[d];
          lin = q;
        }
      }
    }
#pragma unroll
    for (int u = 0; u < W; ++u) k[u] = p0 + u * 256 < A.n ? index[io[u]] : 0;
#pragma unroll
    for (int u = 0; u < W; ++u) {
      v[u] = zero_of<U>();
      if (p0 + u * 256 < A.n) {
        if (k[u] < 0 || k[u] >= A.self_dim_size) flag_oob(status);
        else v[u] = self[so[u] + k[u] * A.self_stride[A.dim]];
      }
    }
#pragma unroll
    for (int u = 0; u < W; ++u)
      if (p0 + u * 256 < A.n) out[p0 + u * 256] = v[u];
  }
}

// 2-D, dim 0, contiguous index [R, C] and unit column stride in self (row pitch
// `self_pitch`): each thread produces the 16 bytes of adjacent outputs (4 or 8 elements) --
// 16-byte index loads, one sector read per element, one 16-byte store. The columns are
// walked in blocks of `wcols` (blockIdx.y), chosen so that the slice of `self` a block of
// columns can touch (self_rows x wcols) stays L2-resident while index and output stream past
// it: every source sector then comes from DRAM once instead of once per eviction.
template <typename U>
__global__ void __launch_bounds__(256) gather_dim0_vec(const U* __restrict__ self, const int64_t* __restrict__ index, U* __restrict__ out, int64_t rows, int64_t cols,
                                                       int64_t self_pitch, int64_t self_rows, int64_t wcols, uint32_t* status) {
  constexpr int VE = 16 / static_cast<int>(sizeof(U));
  const int64_t j0 = static_cast<int64_t>(blockIdx.y) * wcols;
  const int64_t wb = cols - j0 < wcols ? cols - j0 : wcols;
  const int64_t gpr = wb / VE;  // 16-byte groups per row inside this column block
  const int64_t ngroup = rows * gpr;
  const uint64_t keep = l2_keep_policy();
  for (int64_t q = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; q < ngroup; q += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t i = q / gpr, col = j0 + (q - i * gpr) * VE;
    const int64_t p = i * cols + col;
    int64_t k[VE];
#pragma unroll
    for (int h = 0; h < VE / 2; ++h) {
      const longlong2 t = __ldcs(reinterpret_cast<const longlong2*>(index + p) + h);
      k[2 * h] = t.x;
      k[2 * h + 1] = t.y;
    }
    __align__(16) U v[VE];
#pragma unroll
    for (int e = 0; e < VE; ++e) {
      if (k[e] < 0 || k[e] >= self_rows) {
        flag_oob(status);
        v[e] = zero_of<U>();
      } else {
        v[e] = ld_keep_l2(self + k[e] * self_pitch + col + e, keep);
      }
    }
    __stcs(reinterpret_cast<uint4*>(out + p), *reinterpret_cast<const uint4*>(v));
  }
}

// 2-D, along the LAST dim (out[i][j] = self[i][index[i][j]]), contiguous index and unit element
// stride in self: each thread produces the 16 bytes of adjacent outputs of one row -- 16-byte
// index loads, look-ups that stay inside the row (its lines are in L1 / L2 after the first
// touch), one 16-byte store, one 32-bit division per thread instead of a coordinate
// decomposition per element.
template <typename U>
__global__ void __launch_bounds__(256) gather_lastdim_vec(const U* __restrict__ self, const int64_t* __restrict__ index, U* __restrict__ out, int64_t rows, int64_t cols, int64_t self_pitch,
                                                          int64_t self_cols, uint32_t* status) {
  constexpr int VE = 16 / static_cast<int>(sizeof(U));
  const int64_t gpr = cols / VE, ngroup = rows * gpr;
  for (int64_t q = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; q < ngroup; q += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t i = ngroup <= 0x7fffffffLL ? static_cast<int64_t>(static_cast<uint32_t>(q) / static_cast<uint32_t>(gpr)) : q / gpr;
    const int64_t p = q * VE;  // = i * cols + first column of the group
    int64_t k[VE];
#pragma unroll
    for (int h = 0; h < VE / 2; ++h) {
      const longlong2 t = __ldcs(reinterpret_cast<const longlong2*>(index + p) + h);
      k[2 * h] = t.x;
      k[2 * h + 1] = t.y;
    }
    const U* row = self + i * self_pitch;
    __align__(16) U v[VE];
#pragma unroll
    for (int e = 0; e < VE; ++e) {
      if (k[e] < 0 || k[e] >= self_cols) {
        flag_oob(status);
        v[e] = zero_of<U>();
      } else {
        v[e] = row[k[e]];
      }
    }
    __stcs(reinterpret_cast<uint4*>(out + p), *reinterpret_cast<const uint4*>(v));
  }
}

// 2-D, along either dim, with rows of any length: a thread produces 16 bytes of the contiguous result -- VE adjacent outputs,
// which may go on in the next row -- with 16-byte index loads, one division and one store. (An element to a thread decodes
// its coordinates with one division per dimension and moves two or four bytes per store: f16 150134 x 63, 75067
// rows of indices, 27.3 us along the rows and 25.0 along the columns, 22.6 and 9.6 so; fp32 4095 x 4095 127 and 103, 79 and 51. With fewer
// than 2^17 outputs the two are on a par.)
constexpr int64_t kGather2dMin = 1 << 17;
template <typename U, int DIM>
__global__ void __launch_bounds__(256) gather_2d_vec(const U* __restrict__ self, const int64_t* __restrict__ index, U* __restrict__ out, uint32_t total, uint32_t cols, int64_t s_row, int64_t s_col,
                                                     int64_t self_dim_size, uint32_t* status) {
  constexpr int VE = 16 / static_cast<int>(sizeof(U));
  const uint32_t groups = (total + VE - 1) / VE;
  for (uint32_t q = blockIdx.x * 256 + threadIdx.x; q < groups; q += gridDim.x * 256) {
    const uint32_t p = q * VE;
    const bool whole = p + VE <= total;
    int64_t k[VE];
#pragma unroll
    for (int h = 0; h < VE / 2; ++h) {
      if (whole) {
        const longlong2 t = __ldcs(reinterpret_cast<const longlong2*>(index + p) + h);
        k[2 * h] = t.x;
        k[2 * h + 1] = t.y;
      } else {
        k[2 * h] = p + 2 * h < total ? index[p + 2 * h] : 0;
        k[2 * h + 1] = p + 2 * h + 1 < total ? index[p + 2 * h + 1] : 0;
      }
    }
    const uint32_t row = p / cols;
    uint32_t col = p - row * cols;
    const U* at = self + (DIM == 0 ? col * s_col : row * s_row);  // of the coordinate that is kept
    __align__(16) U v[VE];
    bool bad = false;
#pragma unroll
    for (int e = 0; e < VE; ++e) {
      const bool in = p + e < total, ok = k[e] >= 0 && k[e] < self_dim_size;
      v[e] = in && ok ? at[k[e] * (DIM == 0 ? s_row : s_col)] : zero_of<U>();
      bad |= in && !ok;
      ++col;
      if (DIM == 0) at += s_col;
      if (col == cols) {
        col = 0;
        if (DIM == 0) at = self;
        else at += s_row;
      }
    }
    if (bad) flag_oob(status);
    if (whole) {
      __stcs(reinterpret_cast<uint4*>(out + p), *reinterpret_cast<const uint4*>(v));
    } else {
#pragma unroll
      for (int e = 0; e < VE; ++e)
        if (p + e < total) out[p + e] = v[e];
    }
  }
}

// The same gather when a strip of `self` -- all its rows, kStripW columns -- fits in shared
// memory: a CTA copies the strip in once (32-byte segments, each source sector read once)
// and then streams index rows past it, looking every element up in shared memory. Index
// and output move as 64- and 32-byte row segments; neighbouring CTAs work on neighbouring
// strips, so the segments of one row meet again in L2 / DRAM pages. What the L2-resident
// walk above pays per element -- a 32-byte sector crossing the L2-to-SM fabric for 4
// useful bytes -- is paid here once per source element.
// One CTA per strip, one CTA per SM at a time, so the strips go by in waves of as many
// CTAs as there are SMs. The strips of the last, partial wave are cut into `tail_split`
// row ranges each (blockIdx.x >= whole_strips), so that the wave's work spreads over all
// SMs instead of leaving most of them idle.
constexpr int kStripW = 8;
constexpr int kStripThreads = 1024;
constexpr int64_t kStripMaxSelfBytes = 200 * 1024;
// Which strip and which rows this CTA works on (the strips of the last partial wave are cut
// into `tail_split` row ranges).
struct StripWork {
  int64_t c0, r_begin, r_end;
};
__device__ __forceinline__ StripWork strip_work(int64_t rows, int whole_strips, int tail_split) {
  int64_t s = blockIdx.x, r_begin = 0, r_end = rows;
  if (static_cast<int>(blockIdx.x) >= whole_strips) {
    const int q = (blockIdx.x - whole_strips) / tail_split, piece = (blockIdx.x - whole_strips) % tail_split;
    const int64_t per = (rows + tail_split - 1) / tail_split;
    s = whole_strips + q;
    r_begin = piece * per;
    r_end = r_begin + per < rows ? r_begin + per : rows;
  }
  return StripWork{s * kStripW, r_begin, r_end};
}

// Four index segments in flight per thread and no more: keeping the next trip's segments
// in flight as well (with 1024, 768 or 512 threads) was measured 12-19 % SLOWER (62 -> 70-74
// us at 4096 x 4096) -- the 64-byte segments of different rows lie in different DRAM pages,
// and more of them outstanding at once cost more in page misses than the latency they hid.
// Holding neighbouring strips in lockstep (clusters of 2 / 4 / 8 CTAs, a cluster barrier per
// trip) did not help either: 68 -> 76 / 84 / 90 us on the same box.
constexpr int kStripU = 4;
constexpr int64_t kStripTrip = static_cast<int64_t>(kStripThreads / 32) * (8 * kStripU);  // rows one trip of the CTA covers

__device__ __forceinline__ void strip_fetch(const int64_t* __restrict__ index, int64_t cols, const StripWork& w, int64_t r0, int rsub, int cp, longlong2 (&k)[kStripU]) {
#pragma unroll
  for (int u = 0; u < kStripU; ++u) {
    const int64_t row = r0 + u * 8 + rsub;
    if (row < w.r_end) k[u] = __ldcs(reinterpret_cast<const longlong2*>(index + row * cols + w.c0 + cp));
  }
}
__device__ __forceinline__ void strip_emit(const uint32_t* strip, uint32_t* __restrict__ out, int64_t cols, const StripWork& w, int64_t r0, int rsub, int cp, int self_rows,
                                           const longlong2 (&k)[kStripU], uint32_t* status) {
#pragma unroll
  for (int u = 0; u < kStripU; ++u) {
    const int64_t row = r0 + u * 8 + rsub;
    if (row < w.r_end) {
      uint2 v = make_uint2(0u, 0u);
      if (k[u].x < 0 || k[u].x >= self_rows) flag_oob(status);
      else v.x = strip[static_cast<int>(k[u].x) * kStripW + cp];
      if (k[u].y < 0 || k[u].y >= self_rows) flag_oob(status);
      else v.y = strip[static_cast<int>(k[u].y) * kStripW + cp + 1];
      __stcs(reinterpret_cast<uint2*>(out + row * cols + w.c0 + cp), v);
    }
  }
}

__global__ void __launch_bounds__(kStripThreads, 1) gather_dim0_strip(const uint32_t* __restrict__ self, const int64_t* __restrict__ index, uint32_t* __restrict__ out,
                                                                      int64_t rows, int64_t cols, int64_t self_pitch, int self_rows, int whole_strips, int tail_split, uint32_t* status) {
  extern __shared__ __align__(128) uint32_t strip[];  // [self_rows][kStripW]
  const StripWork w = strip_work(rows, whole_strips, tail_split);
  for (int h = threadIdx.x; h < self_rows * 2; h += kStripThreads)  // half-rows: 16 bytes each
    reinterpret_cast<uint4*>(strip)[h] = ld_keep(self + static_cast<int64_t>(h >> 1) * self_pitch + w.c0 + (h & 1) * 4);
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int rsub = lane >> 2, cp = (lane & 3) * 2;  // a warp covers 8 rows x 8 columns per load
  for (int64_t r0 = w.r_begin + warp * (8 * kStripU); r0 < w.r_end; r0 += kStripTrip) {
    longlong2 k[kStripU];
    strip_fetch(index, cols, w, r0, rsub, cp, k);
    strip_emit(strip, out, cols, w, r0, rsub, cp, self_rows, k, status);
  }
}

// The same kernel with the strip brought in by the copy engine: one thread issues a tiled TMA
// load per 256 source rows (box 8 columns x 256 rows = 8 KB, rows beyond the source read as
// zero), all of them completing on one mbarrier, and every thread requests the index
// segments of its first trip BEFORE it waits for the strip -- the strip load costs the 1024
// threads no issue slots and overlaps the first index loads instead of preceding them. The
// wait is bounded: when it runs out the CTA raises B200_DEV_WAIT_TIMEOUT and leaves.
constexpr int kStripBoxRows = 256;
constexpr int kStripBoxBytes = kStripBoxRows * kStripW * 4;
__global__ void __launch_bounds__(kStripThreads, 1) gather_dim0_strip_tma(const __grid_constant__ CUtensorMap map_self, const int64_t* __restrict__ index, uint32_t* __restrict__ out, int64_t rows,
                                                                          int64_t cols, int self_rows, int whole_strips, int tail_split, uint32_t* status) {
  extern __shared__ __align__(128) uint32_t strip[];  // [boxes * 256][kStripW]
  __shared__ __align__(8) uint64_t bar;
  __shared__ uint32_t gave_up;
  const StripWork w = strip_work(rows, whole_strips, tail_split);
  const int boxes = (self_rows + kStripBoxRows - 1) / kStripBoxRows;
  if (threadIdx.x == 0) {
    gave_up = 0u;
    mbar_init(smem_u32(&bar), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    mbar_expect_tx(smem_u32(&bar), static_cast<uint32_t>(boxes) * kStripBoxBytes);
    for (int b = 0; b < boxes; ++b) tma_load_2d(smem_u32(strip) + b * kStripBoxBytes, &map_self, smem_u32(&bar), static_cast<int>(w.c0), b * kStripBoxRows);
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int rsub = lane >> 2, cp = (lane & 3) * 2;
  int64_t r0 = w.r_begin + warp * (8 * kStripU);
  longlong2 k[kStripU];
  if (r0 < w.r_end) strip_fetch(index, cols, w, r0, rsub, cp, k);  // in flight while the strip lands
  __syncthreads();                                                  // the barrier is initialised for everybody
  if (!mbar_wait(smem_u32(&bar), 0u, &gave_up, 2000000000ull)) {
    gave_up = 1u;
    if (status) atomicOr(status, B200_DEV_WAIT_TIMEOUT);
    for (int i = 0; i < 64; ++i) __nanosleep(1000);  // copies still under way may land before this CTA's shared memory is handed on
    return;
  }
  while (r0 < w.r_end) {
    strip_emit(strip, out, cols, w, r0, rsub, cp, self_rows, k, status);
    r0 += kStripTrip;
    if (r0 < w.r_end) strip_fetch(index, cols, w, r0, rsub, cp, k);
  }
}

static int capped_grid(int64_t items, int per_block, int waves) {
  int64_t g = (items + per_block - 1) / per_block;
  const int64_t cap = static_cast<int64_t>(kNumSMs) * waves;
  return static_cast<int>(g < 1 ? 1 : (g > cap ? cap : g));
}

// Largest power-of-two unit (<= 16 bytes) dividing `bytes` and every pointer's address.
static int common_unit(int64_t bytes, const void* a, const void* b) {
  uintptr_t m = static_cast<uintptr_t>(bytes) | reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b);
  int u = 16;
  while (u > 1 && (m & (u - 1))) u >>= 1;
  return u;
}

template <typename U>
static void launch_flat(const void* x, const void* idx, void* out, int64_t outer, int64_t dim_size, int64_t inner_units, int64_t n_idx, int idx_i32, uint32_t* status, cudaStream_t st) {
  const int64_t total = outer * n_idx * inner_units;
  auto go = [&](auto kernel, int w) { kernel<<<capped_grid(total, 256 * w, 16), 256, 0, st>>>(static_cast<const U*>(x), idx, static_cast<U*>(out), outer, dim_size, inner_units, n_idx, idx_i32, status); };
  if (total >= kFlatUnrollMin) go(index_select_flat<U, kFlatUnroll>, kFlatUnroll);
  else go(index_select_flat<U, 1>, 1);
}

// index_select along the LAST dim (inner == 1): every output row is a permutation-with-
// repeats of one input row of at most 8 KB. A warp copies its input row to shared memory
// with coalesced loads and builds the output row from there with coalesced stores; the
// index list is narrowed to int32 once per CTA (-1 = out of range, reported and written as
// zero). Picking single elements straight from global memory, as the flat kernel does,
// fetches a 32-byte sector per element.
constexpr int kLastDimWarps = 8;
template <typename U>
__global__ void __launch_bounds__(kLastDimWarps * 32) index_select_lastdim(const U* __restrict__ x, const void* __restrict__ idx, U* __restrict__ out, int64_t outer, int dim, int n_idx, int row_pitch_bytes,
                                                                           int i32, int vec, uint32_t* status) {
  extern __shared__ __align__(16) unsigned char sm[];
  int* sidx = reinterpret_cast<int*>(sm);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  unsigned char* mine = sm + ((n_idx * 4 + 15) & ~15) + warp * row_pitch_bytes;
  for (int k = tid; k < n_idx; k += blockDim.x) {
    const int64_t v = load_index(idx, k, i32);
    const bool ok = v >= 0 && v < dim;
    if (!ok) flag_oob(status);
    sidx[k] = ok ? static_cast<int>(v) : -1;
  }
  __syncthreads();
  const U* row_s = reinterpret_cast<const U*>(mine);
  for (int64_t row = static_cast<int64_t>(blockIdx.x) * kLastDimWarps + warp; row < outer; row += static_cast<int64_t>(gridDim.x) * kLastDimWarps) {
    const U* xr = x + row * dim;
    if (vec) {
      const int nv = dim * static_cast<int>(sizeof(U)) / 16;
#pragma unroll 4
      for (int v = lane; v < nv; v += 32) reinterpret_cast<uint4*>(mine)[v] = ld_stream(reinterpret_cast<const uint4*>(xr) + v);
    } else {
      for (int c = lane; c < dim; c += 32) reinterpret_cast<U*>(mine)[c] = xr[c];
    }
    __syncwarp();
    U* orow = out + row * n_idx;
    for (int k = lane; k < n_idx; k += 32) {
      const int j = sidx[k];
      orow[k] = j >= 0 ? row_s[j] : zero_of<U>();
    }
    __syncwarp();  // the row buffer is rewritten in the next round
  }
}

template <typename U>
static void launch_lastdim(const void* x, const void* idx, void* out, int64_t outer, int64_t dim, int64_t n_idx, int i32, uint32_t* status, cudaStream_t st) {
  const int pitch = static_cast<int>((dim * sizeof(U) + 15) / 16 * 16);
  const size_t smem = ((n_idx * 4 + 15) & ~static_cast<size_t>(15)) + static_cast<size_t>(kLastDimWarps) * pitch;
  const int vec = (dim * sizeof(U)) % 16 == 0 && aligned16(x);
  cudaFuncSetAttribute(index_select_lastdim<U>, cudaFuncAttributeMaxDynamicSharedMemorySize, 100 * 1024);
  index_select_lastdim<U><<<capped_grid(outer, kLastDimWarps, 8), kLastDimWarps * 32, smem, st>>>(static_cast<const U*>(x), idx, static_cast<U*>(out), outer, static_cast<int>(dim), static_cast<int>(n_idx), pitch,
                                                                                                 i32, vec, status);
}

static int index_select_bytes(const void* x, const void* idx, void* out, int64_t outer, int64_t dim_size, int64_t inner_bytes, int64_t n_idx, int idx_dtype, uint32_t* status, cudaStream_t st) {
  if (idx_dtype != B200_I32 && idx_dtype != B200_I64) return B200_EDTYPE;
  const int i32 = idx_dtype == B200_I32;
  const int unit = common_unit(inner_bytes, x, out);
  const int64_t units = inner_bytes / unit;
  if (outer == 1 && unit == 16 && units >= 64) {
    gather_rows_wide<<<capped_grid(n_idx, 1, 64), 128, 0, st>>>(static_cast<const uint4*>(x), idx, static_cast<uint4*>(out), dim_size, units, n_idx, i32, status);
    return check_launch();
  }
  if (units == 1 && unit <= 8 && dim_size * unit <= 8192 && dim_size >= 32 && n_idx >= 16 && n_idx <= 8192 && outer >= 256) {
    switch (unit) {
      case 8: launch_lastdim<uint64_t>(x, idx, out, outer, dim_size, n_idx, i32, status, st); break;
      case 4: launch_lastdim<uint32_t>(x, idx, out, outer, dim_size, n_idx, i32, status, st); break;
      case 2: launch_lastdim<uint16_t>(x, idx, out, outer, dim_size, n_idx, i32, status, st); break;
      default: launch_lastdim<uint8_t>(x, idx, out, outer, dim_size, n_idx, i32, status, st); break;
    }
    return check_launch();
  }
  // (16-byte vectors of the result meet at most two rows. Rows on the 8-byte grid go a unit to a thread at every size: fp32 38 wide, 480810
  // rows of the result, 37.0 us, 51.2 in ragged vectors, f16 164 wide, 127940 rows 17.9 and 27.1, fp32 4174 wide, 719 rows 5.8 and 7.1)
  const int64_t total = outer * n_idx * inner_bytes;
  if (unit < 8 && inner_bytes >= 16 && aligned16(out) && total / unit >= kRaggedMinUnits) {
    select_rows_ragged<<<capped_grid((total + 15) / 16, 256 * kRaggedUnroll, 16), 256, 0, st>>>(static_cast<const unsigned char*>(x), idx, static_cast<unsigned char*>(out), outer, dim_size, inner_bytes, n_idx, i32,
                                                                                                status);
    return check_launch();
  }
  switch (unit) {
    case 16: launch_flat<uint4>(x, idx, out, outer, dim_size, units, n_idx, i32, status, st); break;
    case 8: launch_flat<uint64_t>(x, idx, out, outer, dim_size, units, n_idx, i32, status, st); break;
    case 4: launch_flat<uint32_t>(x, idx, out, outer, dim_size, units, n_idx, i32, status, st); break;
    case 2: launch_flat<uint16_t>(x, idx, out, outer, dim_size, units, n_idx, i32, status, st); break;
    default: launch_flat<uint8_t>(x, idx, out, outer, dim_size, units, n_idx, i32, status, st); break;
  }
  return check_launch();
}

}  // namespace b200

using namespace b200;

extern "C" int b200_gather_rows(const void* table, const void* idx, void* out, int64_t table_rows, int64_t row_bytes, int64_t n_idx, int idx_dtype, uint32_t* status, void* stream) {
  if (table_rows < 0 || row_bytes < 0 || n_idx < 0) return B200_EINVAL;
  if (n_idx == 0 || row_bytes == 0) return B200_OK;
  if (!idx || !out || (!table && table_rows > 0)) return B200_EINVAL;
  return index_select_bytes(table, idx, out, 1, table_rows, row_bytes, n_idx, idx_dtype, status, static_cast<cudaStream_t>(stream));
}

extern "C" int b200_index_select(const void* x, const void* idx, void* out, int64_t outer, int64_t dim_size, int64_t inner, int64_t n_idx, int elem_size, int idx_dtype, uint32_t* status, void* stream) {
  if (outer < 0 || dim_size < 0 || inner < 0 || n_idx < 0 || elem_size <= 0) return B200_EINVAL;
  if (outer == 0 || inner == 0 || n_idx == 0) return B200_OK;
  if (!idx || !out || (!x && dim_size > 0)) return B200_EINVAL;
  return index_select_bytes(x, idx, out, outer, dim_size, inner * elem_size, n_idx, idx_dtype, status, static_cast<cudaStream_t>(stream));
}

// B200_GATHER_TMA=0 in the environment (read once) keeps the strip on plain loads: how the two are compared.
static bool strip_tma_enabled() {
  static const bool on = []() {
    const char* e = getenv("B200_GATHER_TMA");
    return !(e && e[0] == '0');
  }();
  return on;
}

extern "C" int b200_gather(const void* self, const void* index, void* out, int ndim, const int64_t* index_shape, const int64_t* self_strides, const int64_t* index_strides, int64_t self_dim_size, int dim, int elem_size, uint32_t* status, void* stream) {
  if (ndim < 1 || ndim > B200_MAX_DIMS || dim < 0 || dim >= ndim || !index_shape || !self_strides || !index_strides) return B200_EINVAL;
  GatherArgs A;
  A.ndim = ndim;
  A.dim = dim;
  A.n = 1;
  A.self_dim_size = self_dim_size;
  for (int d = 0; d < ndim; ++d) {
    if (index_shape[d] < 0) return B200_EINVAL;
    A.shape[d] = index_shape[d];
    A.self_stride[d] = self_strides[d];
    A.idx_stride[d] = index_strides[d];
    A.n *= index_shape[d];
  }
  if (A.n == 0) return B200_OK;
  if (!self || !index || !out) return B200_EINVAL;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const bool idx_contig = is_contiguous(ndim, index_shape, index_strides);
  if (ndim == 2 && dim == 0 && elem_size == 4 && idx_contig && self_strides[1] == 1 && index_shape[1] % kStripW == 0 && self_strides[0] % 4 == 0 && aligned16(self) && aligned16(index) &&
      aligned16(out) && self_dim_size > 0 && self_dim_size * kStripW * 4 <= kStripMaxSelfBytes && index_shape[0] >= 512 && index_shape[0] * 2 >= self_dim_size && index_shape[1] / kStripW >= kNumSMs) {
    const size_t smem = static_cast<size_t>(self_dim_size) * kStripW * 4;
    {  // the attribute belongs to the current device: set it on every launch, as the other large-shared-memory kernels do
      const cudaError_t e = cudaFuncSetAttribute(gather_dim0_strip, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kStripMaxSelfBytes));
      if (e != cudaSuccess) { set_last_cuda_error(e); return B200_ELAUNCH; }
    }
    const int64_t strips = index_shape[1] / kStripW;
    const int64_t tail = strips % kNumSMs;
    int64_t tail_split = tail > 0 ? kNumSMs / tail : 1;
    if (tail_split > 8) tail_split = 8;  // every piece reloads the strip
    if (tail_split * 256 > index_shape[0]) tail_split = 1;
    const int64_t whole = tail_split > 1 ? strips - tail : strips;
    const int64_t grid = whole + (strips - whole) * tail_split;
    if (grid > 0x7fffffffLL) return B200_EINVAL;
    // the strip through the copy engine when a tensor map over `self` can be built (this GPU's own memory, no multicast)
    alignas(64) CUtensorMap map_self;
    bool tma = encode_fn() != nullptr && strip_tma_enabled();
    if (tma) {
      cuuint64_t dims[2] = {static_cast<cuuint64_t>(index_shape[1]), static_cast<cuuint64_t>(self_dim_size)};  // the columns this launch may touch x all source rows
      cuuint64_t strides[1] = {static_cast<cuuint64_t>(self_strides[0]) * 4};
      cuuint32_t box[2] = {kStripW, kStripBoxRows};
      cuuint32_t estr[2] = {1, 1};
      tma = encode_fn()(&map_self, CU_TENSOR_MAP_DATA_TYPE_UINT32, 2, const_cast<void*>(self), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                        CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
    }
    if (tma) {
      const size_t smem_tma = static_cast<size_t>((self_dim_size + kStripBoxRows - 1) / kStripBoxRows) * kStripBoxBytes;
      const cudaError_t e2 = cudaFuncSetAttribute(gather_dim0_strip_tma, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kStripMaxSelfBytes));
      if (e2 != cudaSuccess) { set_last_cuda_error(e2); return B200_ELAUNCH; }
      gather_dim0_strip_tma<<<static_cast<unsigned>(grid), kStripThreads, smem_tma, st>>>(map_self, static_cast<const int64_t*>(index), static_cast<uint32_t*>(out), index_shape[0], index_shape[1],
                                                                                        static_cast<int>(self_dim_size), static_cast<int>(whole), static_cast<int>(tail_split), status);
      return check_launch();
    }
    gather_dim0_strip<<<static_cast<unsigned>(grid), kStripThreads, smem, st>>>(static_cast<const uint32_t*>(self), static_cast<const int64_t*>(index), static_cast<uint32_t*>(out), index_shape[0],
                                                                              index_shape[1], self_strides[0], static_cast<int>(self_dim_size), static_cast<int>(whole), static_cast<int>(tail_split), status);
    return check_launch();
  }
  const int ve = elem_size == 4 ? 4 : 8;  // outputs per 16 bytes
  if (ndim == 2 && dim == 0 && (elem_size == 4 || elem_size == 2) && idx_contig && self_strides[1] == 1 && index_shape[1] % ve == 0 && aligned16(index) && aligned16(out)) {
    // column block: about 16 MB of `self` (self_rows x wcols elements), a multiple of the group width
    int64_t wcols = (16LL << 20) / (elem_size * (self_dim_size > 0 ? self_dim_size : 1));
    wcols = wcols / ve * ve;
    if (wcols < 64) wcols = 64;
    if (wcols > index_shape[1]) wcols = index_shape[1];
    const int64_t nblocks = (index_shape[1] + wcols - 1) / wcols;
    if (nblocks <= 65535) {
      dim3 grid(capped_grid(index_shape[0] * wcols / ve, 256, 32), static_cast<unsigned>(nblocks));
      if (elem_size == 4)
        gather_dim0_vec<uint32_t><<<grid, 256, 0, st>>>(static_cast<const uint32_t*>(self), static_cast<const int64_t*>(index), static_cast<uint32_t*>(out), index_shape[0], index_shape[1], self_strides[0], self_dim_size, wcols, status);
      else
        gather_dim0_vec<uint16_t><<<grid, 256, 0, st>>>(static_cast<const uint16_t*>(self), static_cast<const int64_t*>(index), static_cast<uint16_t*>(out), index_shape[0], index_shape[1], self_strides[0], self_dim_size, wcols, status);
      return check_launch();
    }
  }
  if (ndim == 2 && dim == 1 && (elem_size == 4 || elem_size == 2) && idx_contig && self_strides[1] == 1 && index_shape[1] % ve == 0 && aligned16(index) && aligned16(out)) {
    const int g2 = capped_grid(A.n / ve, 256, 32);
    if (elem_size == 4)
      gather_lastdim_vec<uint32_t><<<g2, 256, 0, st>>>(static_cast<const uint32_t*>(self), static_cast<const int64_t*>(index), static_cast<uint32_t*>(out), index_shape[0], index_shape[1], self_strides[0], self_dim_size, status);
    else
      gather_lastdim_vec<uint16_t><<<g2, 256, 0, st>>>(static_cast<const uint16_t*>(self), static_cast<const int64_t*>(index), static_cast<uint16_t*>(out), index_shape[0], index_shape[1], self_strides[0], self_dim_size, status);
    return check_launch();
  }
  if (ndim == 2 && (elem_size == 4 || elem_size == 2) && idx_contig && aligned16(index) && aligned16(out) && A.n >= kGather2dMin && A.n <= 0x7fffffffLL) {
    const int g2 = capped_grid((A.n + ve - 1) / ve, 256, 32);
    auto launch = [&](auto kernel, auto unit) {
      typedef decltype(unit) U;
      kernel<<<g2, 256, 0, st>>>(static_cast<const U*>(self), static_cast<const int64_t*>(index), static_cast<U*>(out), static_cast<uint32_t>(A.n), static_cast<uint32_t>(index_shape[1]), self_strides[0],
                                 self_strides[1], self_dim_size, status);
    };
    if (elem_size == 4) dim == 0 ? launch(gather_2d_vec<uint32_t, 0>, uint32_t{}) : launch(gather_2d_vec<uint32_t, 1>, uint32_t{});
    else dim == 0 ? launch(gather_2d_vec<uint16_t, 0>, uint16_t{}) : launch(gather_2d_vec<uint16_t, 1>, uint16_t{});
    return check_launch();
  }
  const bool along_rows = ndim == 0 || index_shape[ndim - 1] == 1 || index_strides[ndim - 1] == 1;
  const int w = along_rows ? (A.n >= kFlatUnrollMin ? kFlatUnroll : 1) : (A.n * elem_size >= (16LL << 20) ? kFlatUnroll : 1);
  const int g = capped_grid(A.n, 256 * w, 32);
  auto go = [&](auto unit) {
    typedef decltype(unit) U;
    auto launch = [&](auto kernel) { kernel<<<g, 256, 0, st>>>(static_cast<const U*>(self), static_cast<const int64_t*>(index), static_cast<U*>(out), A, status); };
    if (w == 1) launch(gather_generic<U, 1>);
    else launch(gather_generic<U, kFlatUnroll>);
  };
  switch (elem_size) {
    case 1: go(uint8_t{}); break;
    case 2: go(uint16_t{}); break;
    case 4: go(uint32_t{}); break;
    case 8: go(uint64_t{}); break;
    default: return B200_EDTYPE;
  }
  return check_launch();
}
