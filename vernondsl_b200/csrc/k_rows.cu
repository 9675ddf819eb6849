// Row reductions, softmax and column sums of a row-major [rows][cols] float matrix, sm_100a.
//
// HBM-bound: every kernel reads a row from HBM once, holds what it needs of it in registers and keeps many 16-byte loads in
// flight.  Rows whose length is no multiple of 4 start at any 4-byte boundary; their kernels (EDGE) split a row into
// up to three elements in front of the first 16-byte boundary, float4 groups, and up to three elements behind them, so
// every length runs at the speed of the round ones.  By row length:
//   up to 64               a few lanes per row, single elements (row_narrow_kernel)
//   sums and maxima        a warp, four warps or a block per row, streaming (row_reduce_kernel)
//   softmax up to 10240    one to 16 warps per row, the row in registers (row_group_kernel)
//   softmax up to 32768    a block per row, the next row already on its way (row_stream_kernel)
//   softmax beyond         a block per row, which reads it a second time out of L2 (row_two_pass_kernel)
// Summation order depends on the shape only, so results are bit-reproducible.
// The reference project has no counterpart for these operators.
#include <atomic>
#include <cstring>

#include "vrhi_internal.h"

namespace vrhi {

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ float sum4(float4 v) { return (v.x + v.y) + (v.z + v.w); }
__device__ __forceinline__ float max4(float4 v) { return fmaxf(fmaxf(v.x, v.y), fmaxf(v.z, v.w)); }
__device__ __forceinline__ float4 splat4(float v) { return make_float4(v, v, v, v); }

enum { ROW_SUM = 1, ROW_MAX = 2, ROW_SOFTMAX = 4 };

// Where the float4 groups of a row lie.  `first` is the index of the row's first element in an array that starts on a
// 16-byte boundary.  Thread t < head + tail holds the single element edge(t).  Thread t of T takes the groups
// t - shift, t - shift + T, ...: `shift` counts the groups between the row's first one and the 128-byte boundary before
// it, so that a warp's accesses start on a line whatever the row's start.  With shift = 0 every warp of an odd
// row writes two half sectors (softmax of [4099,10007]: 66 us, and 52 us with the shift).
template <bool EDGE>
struct RowParts {
  uint32_t head, n4, tail, shift;
  __device__ __forceinline__ RowParts(uint64_t first, uint32_t cols) {
    head = EDGE ? min((4u - (uint32_t)(first & 3u)) & 3u, cols) : 0u;
    n4 = (cols - head) >> 2;
    tail = EDGE ? cols - head - 4u * n4 : 0u;
    shift = EDGE ? ((uint32_t)(first + head) >> 2) & 7u : 0u;
  }
  __device__ __forceinline__ bool has_edge(uint32_t t) const { return EDGE && t < head + tail; }
  __device__ __forceinline__ uint32_t edge(uint32_t t) const { return t < head ? t : 4u * n4 + t; }
};

// Partial results of a row's warps: red[0..warps) -> every thread, in warp order (up to 8) or as a tree.
template <int WARPS, bool MAX>
__device__ __forceinline__ float combine_warps(const float *red) {
  if (WARPS <= 8) {
    float r = red[0];
#pragma unroll
    for (int j = 1; j < WARPS; ++j) r = MAX ? fmaxf(r, red[j]) : r + red[j];
    return r;
  }
  const uint32_t lane = threadIdx.x & 31u;
  const float r = lane < (uint32_t)WARPS ? red[lane] : (MAX ? -INFINITY : 0.f);
  return MAX ? warp_max(r) : warp_sum(r);
}

// ---------------------------------------------------------------------------------------------
// Sums or maxima: TPR threads per row, ROWS rows per group of threads at a time, U float4 in flight per thread and row.
// Against a block of 256 threads per row with single-element loads and a barrier per row (the path of every odd
// length before) and a warp per row that held up to 4096 elements in registers.
template <int TPR, int ROWS, int U, bool MAX, bool EDGE>
__global__ void __launch_bounds__(TPR > 256 ? TPR : 256) row_reduce_kernel(const float *__restrict__ in, float *__restrict__ out,
                                                                           uint64_t rows, uint64_t cols) {
  constexpr int THREADS = TPR > 256 ? TPR : 256, GROUPS = THREADS / TPR, WARPS = TPR / 32;
  constexpr float ID = MAX ? -INFINITY : 0.f;
  __shared__ float red[THREADS / 32];
  pdl_begin();
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, group = threadIdx.x / TPR, t = threadIdx.x % TPR;
  const uint64_t most4 = cols >> 2, per_block = (uint64_t)GROUPS * ROWS;
  for (uint64_t base = (uint64_t)blockIdx.x * per_block; base < rows; base += (uint64_t)gridDim.x * per_block) {
    const uint64_t r0 = base + (uint64_t)group * ROWS;
    float acc[ROWS];
    const float4 *src4[ROWS];
    uint64_t n4[ROWS];
#pragma unroll
    for (int q = 0; q < ROWS; ++q) {
      const bool active = r0 + q < rows;
      const uint64_t first = (r0 + q) * cols;
      const uint32_t head = EDGE ? (4u - (uint32_t)(first & 3u)) & 3u : 0u;  // cols > 64 here
      n4[q] = active ? (cols - head) >> 2 : 0;
      src4[q] = reinterpret_cast<const float4 *>(in + first + head);
      acc[q] = ID;
      if constexpr (EDGE) {
        const uint32_t tail = (uint32_t)((cols - head) & 3u);
        if (active && t < head + tail) acc[q] = __ldcs(in + first + (t < head ? t : 4u * n4[q] + t));
      }
    }
    for (uint64_t c0 = 0; c0 < most4; c0 += (uint64_t)TPR * U) {
      float4 v[ROWS][U];
#pragma unroll
      for (int q = 0; q < ROWS; ++q)
#pragma unroll
        for (int k = 0; k < U; ++k) {
          const uint64_t c = c0 + t + (uint32_t)(TPR * k);
          v[q][k] = c < n4[q] ? __ldcs(src4[q] + c) : splat4(ID);
        }
#pragma unroll
      for (int q = 0; q < ROWS; ++q) {
        float p[U];
#pragma unroll
        for (int k = 0; k < U; ++k) p[k] = MAX ? max4(v[q][k]) : sum4(v[q][k]);
#pragma unroll
        for (int n = U / 2; n > 0; n >>= 1)
#pragma unroll
          for (int k = 0; k < n; ++k) p[k] = MAX ? fmaxf(p[k], p[k + n]) : p[k] + p[k + n];
        acc[q] = MAX ? fmaxf(acc[q], p[0]) : acc[q] + p[0];
      }
    }
#pragma unroll
    for (int q = 0; q < ROWS; ++q) {
      float r = MAX ? warp_max(acc[q]) : warp_sum(acc[q]);
      if (WARPS > 1) {  // ROWS is 1 here
        if (lane == 0) red[warp] = r;
        __syncthreads();
        r = combine_warps<WARPS, MAX>(red + group * WARPS);
        __syncthreads();
      }
      if (t == 0 && r0 + q < rows) out[r0 + q] = r;
    }
  }
}

// ---------------------------------------------------------------------------------------------
// Rows of at most L * V elements: L lanes per row, V elements per lane, lane j those at j, j + L, ...  A warp's rows are
// adjacent, so its loads cover one contiguous range.  One warp per row would leave most lanes without an element.
template <int L, int V, int WHAT>
__global__ void __launch_bounds__(256) row_narrow_kernel(const float *__restrict__ in, float *__restrict__ out_sum,
                                                         float *__restrict__ out_max, float *__restrict__ out_soft,
                                                         uint64_t rows, uint32_t cols) {
  constexpr uint32_t FULL = 0xffffffffu;
  pdl_begin();
  const uint32_t j = threadIdx.x % L;
  constexpr uint64_t per_block = 256 / L;
  for (uint64_t base = (uint64_t)blockIdx.x * per_block; base < rows; base += (uint64_t)gridDim.x * per_block) {
    const uint64_t r = base + threadIdx.x / L;
    const bool active = r < rows;
    const float *src = in + r * cols;
    float x[V];
#pragma unroll
    for (int k = 0; k < V; ++k) x[k] = active && j + L * k < cols ? __ldg(src + j + L * k) : 0.f;
    if (WHAT & ROW_SUM) {
      float s[V];
#pragma unroll
      for (int k = 0; k < V; ++k) s[k] = x[k];
#pragma unroll
      for (int n = V / 2; n > 0; n >>= 1)
#pragma unroll
        for (int k = 0; k < n; ++k) s[k] += s[k + n];
#pragma unroll
      for (int o = L / 2; o > 0; o >>= 1) s[0] += __shfl_xor_sync(FULL, s[0], o);
      if (active && j == 0) out_sum[r] = s[0];
    }
    if (WHAT & (ROW_MAX | ROW_SOFTMAX)) {
      float m = -INFINITY;
#pragma unroll
      for (int k = 0; k < V; ++k)
        if (j + L * k < cols) m = fmaxf(m, x[k]);
#pragma unroll
      for (int o = L / 2; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(FULL, m, o));
      if ((WHAT & ROW_MAX) && active && j == 0) out_max[r] = m;
      if (WHAT & ROW_SOFTMAX) {
        float z[V];
#pragma unroll
        for (int k = 0; k < V; ++k) {
          x[k] = j + L * k < cols ? expf(x[k] - m) : 0.f;
          z[k] = x[k];
        }
#pragma unroll
        for (int n = V / 2; n > 0; n >>= 1)
#pragma unroll
          for (int k = 0; k < n; ++k) z[k] += z[k + n];
#pragma unroll
        for (int o = L / 2; o > 0; o >>= 1) z[0] += __shfl_xor_sync(FULL, z[0], o);
        const float inv = 1.0f / z[0];
#pragma unroll
        for (int k = 0; k < V; ++k)
          if (active && j + L * k < cols) out_soft[r * cols + j + L * k] = x[k] * inv;
      }
    }
  }
}

// exp(x - m) as 2^(x*log2e - m*log2e): one fused multiply-add and one MUFU.EX2 per element.
// ml = m*log2e is rounded once per row; that rounding is a common factor of every element of the
// row and cancels in the normalisation.  Relative error per element stays below 2e-6 for
// |x - m| < 60 (fma rounding of the exponent plus the 2^-22 of ex2.approx).
__device__ __forceinline__ float exp2_approx(float t) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(t));
  return r;
}
// Rows of an odd length and of more than 8192 elements take expf: HBM-bound all the same, and more accurate for elements
// far below the maximum.
template <bool EXPF>
struct RowExp {
  float m, ml;
  __device__ __forceinline__ explicit RowExp(float max) : m(max), ml(-max * 1.4426950408889634f) {}
  __device__ __forceinline__ float operator()(float x) const {
    return EXPF ? expf(x - m) : exp2_approx(fmaf(x, 1.4426950408889634f, ml));
  }
  __device__ __forceinline__ float4 operator()(float4 v) const { return make_float4((*this)(v.x), (*this)(v.y), (*this)(v.z), (*this)(v.w)); }
};

// Softmax rows: WPR warps share one row (8 float4 per thread at most), so a 256-thread CTA works
// on 8/WPR rows at a time with ~64 registers per thread and 32 resident warps per SM: enough
// independent warps to keep loads in flight while others are in their exp phase.  The row still
// makes exactly one trip from HBM and one back.  Cross-warp reductions go through three separate
// shared arrays (sum, max, normaliser), one CTA barrier each; partials are combined in a fixed
// order, so results do not depend on scheduling.
template <int NV, int WPR, int WHAT, bool EDGE>
__global__ void __launch_bounds__(WPR > 8 ? 32 * WPR : 256, WPR > 8 ? 3 : WPR > 4 && NV <= 5 ? 5 : 4) row_group_kernel(const float *__restrict__ in, float *__restrict__ out_sum,
                                                                           float *__restrict__ out_max, float *__restrict__ out_soft,
                                                                           uint64_t rows, uint32_t cols) {
  constexpr int GROUPS = WPR > 8 ? 1 : 8 / WPR;
  constexpr uint32_t TPR = 32u * WPR;  // threads per row
  __shared__ float red_sum[GROUPS * WPR], red_max[GROUPS * WPR], red_z[GROUPS * WPR];
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  pdl_begin();
  const uint32_t group = warp / WPR, t = threadIdx.x % TPR;
  for (uint64_t base = (uint64_t)blockIdx.x * GROUPS; base < rows; base += (uint64_t)gridDim.x * GROUPS) {
    const uint64_t r = base + group, first = r * cols;
    const bool active = r < rows;
    const RowParts<EDGE> parts(first, cols);
    const float4 *src = reinterpret_cast<const float4 *>(in + first + parts.head);
    const uint32_t n4 = parts.n4;
    const bool has_edge = active && parts.has_edge(t);
    float4 v[NV];
    float e = 0.f;
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      const uint32_t c = t + TPR * k - parts.shift;  // below the row: wraps above n4
      v[k] = (active && c < n4) ? __ldcs(src + c) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    if (EDGE && has_edge) e = __ldcs(in + first + parts.edge(t));
    float s = e, mm = EDGE && has_edge ? e : -INFINITY;
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      const uint32_t c = t + TPR * k - parts.shift;  // below the row: wraps above n4
      if (WHAT & ROW_SUM) s += sum4(v[k]);
      if (c < n4) mm = fmaxf(mm, max4(v[k]));
    }
    if (WHAT & ROW_SUM) s = warp_sum(s);
    mm = warp_max(mm);
    if (WPR > 1) {
      if (lane == 0) {
        if (WHAT & ROW_SUM) red_sum[warp] = s;
        red_max[warp] = mm;
      }
      __syncthreads();
      if (WPR <= 8) {
        s = 0.f; mm = -INFINITY;
#pragma unroll
        for (int j = 0; j < WPR; ++j) {
          if (WHAT & ROW_SUM) s += red_sum[group * WPR + j];
          mm = fmaxf(mm, red_max[group * WPR + j]);
        }
      } else
      {
      if (WHAT & ROW_SUM) s = combine_warps<WPR, false>(red_sum + group * WPR);
      mm = combine_warps<WPR, true>(red_max + group * WPR);
      }
    }
    if (active && t == 0) {
      if (WHAT & ROW_SUM) out_sum[r] = s;
      if (WHAT & ROW_MAX) out_max[r] = mm;
    }
    const RowExp<(EDGE || WPR > 8)> ex(mm);
    float z = 0.f;
    if (EDGE && has_edge) { e = ex(e); z = e; }
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      const uint32_t c = t + TPR * k - parts.shift;  // below the row: wraps above n4
      if (c < n4) {
        v[k] = ex(v[k]);
        z += sum4(v[k]);
      }
    }
    z = warp_sum(z);
    if (WPR > 1) {
      if (lane == 0) red_z[warp] = z;
      __syncthreads();
      if (WPR <= 8) {
        z = 0.f;
#pragma unroll
        for (int j = 0; j < WPR; ++j) z += red_z[group * WPR + j];
      } else
      z = combine_warps<WPR, false>(red_z + group * WPR);
    }
    const float inv = 1.0f / z;
    float4 *dst = reinterpret_cast<float4 *>(out_soft + first + parts.head);
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      const uint32_t c = t + TPR * k - parts.shift;  // below the row: wraps above n4
      if (active && c < n4) __stcs(dst + c, make_float4(v[k].x * inv, v[k].y * inv, v[k].z * inv, v[k].w * inv));
    }
    if (EDGE && has_edge) __stcs(out_soft + first + parts.edge(t), e * inv);
  }
}

// Softmax of longer rows: a resident grid whose blocks go from row to row, the next row on its way into shared memory
// (cp.async, each thread its own 16-byte slots) while this one is in registers.  A block per row as above needs three
// or more blocks per SM that happen to be in different phases; a row of 64 KiB leaves room for two, and they wait for
// their loads together: [4000,16384] 116 us, 135 us for [2048,32768], where the row is all of the SM's registers.
__device__ __forceinline__ void cp_async_16(void *smem_dst, const void *gmem_src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(smem_dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(gmem_src) : "memory");
}

template <int T, int NV, int WHAT, bool EDGE>
__global__ void __launch_bounds__(T, 1024 / T) row_stream_kernel(const float *__restrict__ in, float *__restrict__ out_sum,
                                                                 float *__restrict__ out_max, float *__restrict__ out_soft,
                                                                 uint64_t rows, uint32_t cols) {
  constexpr int WARPS = T / 32;
  extern __shared__ float4 stage[];  // [NV][T]: slot k of thread t is stage[k * T + t], written and read by that thread only
  // A row's uses of each array lie between two barriers that the next row's uses are behind, so one copy is enough.
  __shared__ float red_sum[WARPS], red_max[WARPS], red_z[WARPS];
  const uint32_t t = threadIdx.x, lane = t & 31u, warp = t >> 5;
  float e_next = 0.f;
  auto fetch = [&](uint64_t r) {
    if (r < rows) {
      const uint64_t first = r * cols;
      const RowParts<EDGE> parts(first, cols);
      const float4 *src = reinterpret_cast<const float4 *>(in + first + parts.head);
      const uint32_t c0 = t - parts.shift;  // groups in front of the row wrap above n4
#pragma unroll
      for (int k = 0; k < NV; ++k)
        if (c0 + T * k < parts.n4) cp_async_16(stage + k * T + t, src + (c0 + T * k));
      if (parts.has_edge(t)) e_next = __ldcs(in + first + parts.edge(t));
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  pdl_begin();
  uint64_t r = blockIdx.x;
  fetch(r);
  for (; r < rows; r += gridDim.x) {
    const uint64_t first = r * cols;
    const RowParts<EDGE> parts(first, cols);
    const uint32_t c0 = t - parts.shift, n4 = parts.n4;
    const bool has_edge = parts.has_edge(t);
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    float4 v[NV];
    float e = has_edge ? e_next : 0.f;
    float s = e, mm = has_edge ? e : -INFINITY;
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      v[k] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (c0 + T * k < n4) {
        v[k] = stage[k * T + t];
        mm = fmaxf(mm, max4(v[k]));
        if (WHAT & ROW_SUM) s += sum4(v[k]);
      }
    }
    if (WHAT & ROW_SUM) s = warp_sum(s);
    mm = warp_max(mm);
    if (lane == 0) {
      if (WHAT & ROW_SUM) red_sum[warp] = s;
      red_max[warp] = mm;
    }
    __syncthreads();
    fetch(r + gridDim.x);  // behind the barrier: the slots have been read
    if (WHAT & ROW_SUM) s = combine_warps<WARPS, false>(red_sum);
    mm = combine_warps<WARPS, true>(red_max);
    if (t == 0) {
      if (WHAT & ROW_SUM) out_sum[r] = s;
      if (WHAT & ROW_MAX) out_max[r] = mm;
    }
    const RowExp<(EDGE || T > 256)> ex(mm);
    float z = 0.f;
    if (has_edge) { e = ex(e); z = e; }
#pragma unroll
    for (int k = 0; k < NV; ++k)
      if (c0 + T * k < n4) {
        v[k] = ex(v[k]);
        z += sum4(v[k]);
      }
    z = warp_sum(z);
    if (lane == 0) red_z[warp] = z;
    __syncthreads();
    z = combine_warps<WARPS, false>(red_z);
    const float inv = 1.0f / z;
    float4 *dst = reinterpret_cast<float4 *>(out_soft + first + parts.head);
#pragma unroll
    for (int k = 0; k < NV; ++k)
      if (c0 + T * k < n4) __stcs(dst + (c0 + T * k), make_float4(v[k].x * inv, v[k].y * inv, v[k].z * inv, v[k].w * inv));
    if (has_edge) __stcs(out_soft + first + parts.edge(t), e * inv);
  }
}

// Softmax of rows that a block's registers do not hold: two passes, the second one out of L2 (two rows per SM under way:
// 296 rows of 65536 elements are 78 MB of the 126).  The first pass keeps a running maximum per thread and the sum of the
// exponentials relative to it, so the row is read twice and not three times.
template <int WHAT, bool EDGE>
__global__ void __launch_bounds__(512, 3) row_two_pass_kernel(const float *__restrict__ in, float *__restrict__ out_sum,
                                                              float *__restrict__ out_max, float *__restrict__ out_soft,
                                                              uint64_t rows, uint64_t cols) {
  constexpr uint32_t T = 512, U = 4, WARPS = T / 32;
  __shared__ float red_sum[WARPS], red_max[WARPS], red_z[WARPS];
  pdl_begin();
  const uint32_t t = threadIdx.x, lane = t & 31u, warp = t >> 5;
  for (uint64_t r = blockIdx.x; r < rows; r += gridDim.x) {
    const uint64_t first = r * cols;
    const uint32_t head = EDGE ? (4u - (uint32_t)(first & 3u)) & 3u : 0u;
    const uint64_t n4 = (cols - head) >> 2, edges = EDGE ? head + ((cols - head) & 3u) : 0u, shift = EDGE ? ((first + head) >> 2) & 7u : 0u;
    const bool has_edge = EDGE && t < edges;
    const uint64_t at = first + (t < head ? t : 4u * n4 + t);
    const float4 *src = reinterpret_cast<const float4 *>(in + first + head);
    float e = has_edge ? __ldg(in + at) : 0.f;
    // the edge enters like any other element: a NaN is no maximum, and NaN and +inf make the sum NaN
    float s = e, m = has_edge ? fmaxf(e, -INFINITY) : -INFINITY;
    float z = has_edge ? expf(e - (m == -INFINITY ? 0.f : m)) : 0.f;
    for (uint64_t c0 = 0; c0 < n4 + shift; c0 += T * U) {
      float4 v[U];
      float chunk = -INFINITY;
#pragma unroll
      for (uint32_t k = 0; k < U; ++k) {
        const uint64_t c = c0 + t + T * k - shift;
        v[k] = splat4(-INFINITY);
        if (c < n4) v[k] = __ldg(src + c);
      }
#pragma unroll
      for (uint32_t k = 0; k < U; ++k) {
        chunk = fmaxf(chunk, max4(v[k]));
        if (WHAT & ROW_SUM) s += c0 + t + T * k - shift < n4 ? sum4(v[k]) : 0.f;
      }
      const float next = fmaxf(m, chunk);
      // next = -inf: nothing but -inf (and NaN) so far; such a row's results are NaN through the second pass unless more follows
      if (next > m) { z *= expf(m - next); m = next; }
      const float ref = m == -INFINITY ? 0.f : m;
      float p[U];
#pragma unroll
      for (uint32_t k = 0; k < U; ++k) p[k] = sum4(make_float4(expf(v[k].x - ref), expf(v[k].y - ref), expf(v[k].z - ref), expf(v[k].w - ref)));
#pragma unroll
      for (uint32_t n = U / 2; n > 0; n >>= 1)
#pragma unroll
        for (uint32_t k = 0; k < n; ++k) p[k] += p[k + n];
      z += p[0];
    }
    if (WHAT & ROW_SUM) s = warp_sum(s);
    float mm = warp_max(m);
    if (lane == 0) {
      if (WHAT & ROW_SUM) red_sum[warp] = s;
      red_max[warp] = mm;
    }
    __syncthreads();
    if (WHAT & ROW_SUM) s = combine_warps<WARPS, false>(red_sum);
    mm = combine_warps<WARPS, true>(red_max);
    if (t == 0) {
      if (WHAT & ROW_SUM) out_sum[r] = s;
      if (WHAT & ROW_MAX) out_max[r] = mm;
    }
    z = m == mm ? z : z * expf(m - mm);  // (m = mm = +inf would be inf - inf)
    z = warp_sum(z);
    if (lane == 0) red_z[warp] = z;
    __syncthreads();
    z = combine_warps<WARPS, false>(red_z);
    const float inv = 1.0f / z;
    const RowExp<true> ex(mm);
    float4 *dst = reinterpret_cast<float4 *>(out_soft + first + head);
    for (uint64_t c0 = 0; c0 < n4 + shift; c0 += T * U) {
      float4 v[U];
#pragma unroll
      for (uint32_t k = 0; k < U; ++k) {
        const uint64_t c = c0 + t + T * k - shift;
        if (c < n4) v[k] = __ldcs(src + c);
      }
#pragma unroll
      for (uint32_t k = 0; k < U; ++k) {
        const uint64_t c = c0 + t + T * k - shift;
        if (c >= n4) continue;
        const float4 y = ex(v[k]);
        __stcs(dst + c, make_float4(y.x * inv, y.y * inv, y.z * inv, y.w * inv));
      }
    }
    if (has_edge) __stcs(out_soft + at, ex(e) * inv);
  }
}

static unsigned row_grid(uint64_t rows, uint64_t per_block) {
  const uint64_t want = (rows + per_block - 1) / per_block;
  return (unsigned)(want < 0x7fffffffull ? want : 0x7fffffffull);
}

template <bool MAX, bool EDGE>
static cudaError_t launch_reduce(vrhi_stream_t *st, const float *in, float *out, uint64_t rows, uint64_t cols) {
  if (cols <= 256) return launch_chained(chains(st), row_reduce_kernel<32, 4, 2, MAX, EDGE>, dim3(row_grid(rows, 32)), 256, 0, st->s, in, out, rows, cols);
  if (cols <= 1024) return launch_chained(chains(st), row_reduce_kernel<32, 1, 8, MAX, EDGE>, dim3(row_grid(rows, 8)), 256, 0, st->s, in, out, rows, cols);
  if (cols <= 4096) return launch_chained(chains(st), row_reduce_kernel<128, 1, 8, MAX, EDGE>, dim3(row_grid(rows, 2)), 256, 0, st->s, in, out, rows, cols);
  if (cols <= 16384) return launch_chained(chains(st), row_reduce_kernel<256, 1, 8, MAX, EDGE>, dim3(row_grid(rows, 1)), 256, 0, st->s, in, out, rows, cols);
  return launch_chained(chains(st), row_reduce_kernel<1024, 1, 8, MAX, EDGE>, dim3(row_grid(rows, 1)), 1024, 0, st->s, in, out, rows, cols);
}

template <int T, int NV, int WHAT, bool EDGE>
static cudaError_t launch_stream_nv(vrhi_stream_t *st, const float *in, float *osum, float *omax, float *osoft, uint64_t rows, uint32_t cols) {
  auto kern = row_stream_kernel<T, NV, WHAT, EDGE>;
  constexpr int smem = NV * T * (int)sizeof(float4);
  static std::atomic<uint64_t> raised{0};  // devices on which the kernel's shared memory limit has been raised (always to the same value)
  const uint64_t bit = 1ull << (st->dev->ordinal & 63);
  if (!(raised.load(std::memory_order_acquire) & bit)) {
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    raised.fetch_or(bit, std::memory_order_release);
  }
  const uint64_t resident = (uint64_t)st->dev->prop.multiProcessorCount * (1024 / T);
  return launch_chained(chains(st), kern, dim3((unsigned)(rows < resident ? rows : resident)), T, smem, st->s, in, osum, omax, osoft, rows, cols);
}

template <int T, int WHAT, bool EDGE>
static cudaError_t launch_stream(vrhi_stream_t *st, const float *in, float *osum, float *omax, float *osoft, uint64_t rows, uint32_t cols, uint64_t most4) {
  const uint64_t nv = (most4 + T - 1) / T;  // 512 threads: 2561 groups or more
  if constexpr (T > 512)
    if (nv <= 5) return launch_stream_nv<T, 5, WHAT, EDGE>(st, in, osum, omax, osoft, rows, cols);
  if (nv <= 6) return launch_stream_nv<T, 6, WHAT, EDGE>(st, in, osum, omax, osoft, rows, cols);
  if (nv <= 7) return launch_stream_nv<T, 7, WHAT, EDGE>(st, in, osum, omax, osoft, rows, cols);
  return launch_stream_nv<T, 8, WHAT, EDGE>(st, in, osum, omax, osoft, rows, cols);
}

template <int WHAT, bool EDGE>
static cudaError_t launch_softmax(vrhi_stream_t *st, const float *in, float *osum, float *omax, float *osoft, uint64_t rows, uint64_t cols) {
  cudaStream_t s = st->s;
  const uint64_t most4 = cols / 4 + (EDGE ? 7 : 0);  // with the groups in front of a row (RowParts::shift)
  if (most4 > 8192) {
    const uint64_t resident = (uint64_t)st->dev->prop.multiProcessorCount * 3;
    return launch_chained(chains(st), row_two_pass_kernel<WHAT, EDGE>, dim3((unsigned)(rows < resident ? rows : resident)), 512, 0, s, in, osum, omax, osoft, rows, cols);
  }
  if (most4 > 4096) return launch_stream<1024, WHAT, EDGE>(st, in, osum, omax, osoft, rows, (uint32_t)cols, most4);
  if (most4 > 2560) return launch_stream<512, WHAT, EDGE>(st, in, osum, omax, osoft, rows, (uint32_t)cols, most4);
  // Registers for a row of the block's: 64 per thread with 8 float4 (four blocks of 256 threads per SM), 40 with 5 (three of 512,
  // six of 256).  One more block per SM in another phase is worth more than any other choice here: [4096,10000] 50.7 us
  // with three blocks of 512 threads per SM, 60 us with two.
  // (8 warps with 8 float4, whole groups only: [4790,7004] 49.5 us, 16 warps with 4 float4 53)
  const uint32_t wpr = most4 <= 256 ? 1 : most4 <= 512 ? 2 : most4 <= 1024 ? 4 : most4 <= (EDGE ? 1280 : 1792) ? 8 : 16;
  const uint32_t nv = (uint32_t)((most4 + 32u * wpr - 1) / (32u * wpr));
  // one CTA per group of rows, not a persistent grid: measured on B200, letting the hardware
  // scheduler stream CTAs (each loads, reduces, writes and leaves) beats a resident grid whose
  // CTAs fall into lock step, all loading and then all storing (0.314 ms against 0.36 ms on [65536,4096])
  const unsigned grid = row_grid(rows, wpr > 8 ? 1 : 8 / wpr), block = wpr > 8 ? 32 * wpr : 256;
#define GROUP_LAUNCH(NV, WPR) return launch_chained(chains(st), row_group_kernel<NV, WPR, WHAT, EDGE>, dim3(grid), block, 0, s, in, osum, omax, osoft, rows, (uint32_t)cols)
#define GROUP_NV(WPR)                     \
  do {                                    \
    if (nv <= 5) GROUP_LAUNCH(5, WPR);    \
    if constexpr (EDGE) { /* whole groups with 6: [22369,1500] 57 us, with 8 43 */ \
      if (nv <= 6) GROUP_LAUNCH(6, WPR);  \
    }                                     \
    GROUP_LAUNCH(8, WPR);                 \
  } while (0)
  if (wpr == 1) {
    if (nv <= 1) GROUP_LAUNCH(1, 1);
    if (nv <= 2) GROUP_LAUNCH(2, 1);
    if (nv <= 4) GROUP_LAUNCH(4, 1);
    GROUP_LAUNCH(8, 1);
  }
  if (wpr == 2) GROUP_NV(2);
  if (wpr == 4) GROUP_NV(4);
  // 8 warps have up to 1280 groups with edges (5 per thread) and up to 1792 without (7), 16 warps what is above
  if (wpr == 8) {
    if constexpr (!EDGE)
      if (nv > 5) GROUP_LAUNCH(8, 8);
    GROUP_LAUNCH(5, 8);
  }
  if constexpr (EDGE)
    if (nv <= 3) GROUP_LAUNCH(3, 16);
  if (nv <= 4) GROUP_LAUNCH(4, 16);
  GROUP_LAUNCH(5, 16);
#undef GROUP_NV
#undef GROUP_LAUNCH
}

template <int WHAT>
static int launch_rows(vrhi_stream_t *st, const float *in, float *osum, float *omax, float *osoft, uint64_t rows, uint64_t cols,
                       const char *name) {
  if (cols <= 16) VRHI_CUDA(launch_chained(chains(st), row_narrow_kernel<4, 4, WHAT>, dim3(row_grid(rows, 64)), 256, 0, st->s, in, osum, omax, osoft, rows, (uint32_t)cols));
  else if (cols <= 64) VRHI_CUDA(launch_chained(chains(st), row_narrow_kernel<8, 8, WHAT>, dim3(row_grid(rows, 32)), 256, 0, st->s, in, osum, omax, osoft, rows, (uint32_t)cols));
  else if constexpr ((WHAT & ROW_SOFTMAX) != 0) {
    // EDGE: rows that start off a 16-byte boundary, and long ones that start inside a 32-byte sector.  Short rows of 4, 12, 20,
    // ... elements lose more to its bookkeeping than half sectors cost ([133152,252] 42 us without, 54 with).
    const bool edge = cols % 4 != 0 || (cols % 8 != 0 && cols > 8192);
    VRHI_CUDA((edge ? launch_softmax<WHAT, true>(st, in, osum, omax, osoft, rows, cols) : launch_softmax<WHAT, false>(st, in, osum, omax, osoft, rows, cols)));
  } else {
    constexpr bool MAX = WHAT == ROW_MAX;
    float *out = MAX ? omax : osum;
    VRHI_CUDA((cols % 4 != 0 ? launch_reduce<MAX, true>(st, in, out, rows, cols) : launch_reduce<MAX, false>(st, in, out, rows, cols)));
  }
  return post_launch(st, name);
}

static int rows_common(const ArgView *args, int n_args, int want_args, const void *params, size_t params_size,
                       vrhi_rows_params *q, const char *name) {
  VRHI_TRY(read_params(params, params_size, q));
  if (n_args != want_args) return fail(VRHI_ERR_INVALID, "%s takes %d arguments, got %d", name, want_args, n_args);
  if (q->cols == 0 && q->rows != 0) return fail(VRHI_ERR_SIZE, "%s: rows of zero length", name);
  if (q->rows > (1ull << 40) || q->cols > (1ull << 32)) return fail(VRHI_ERR_SIZE, "%s: shape out of range", name);
  uint64_t elements = 0;
  VRHI_TRY(element_count(q->rows, q->cols, name, &elements));
  if (args[0].bytes < elements * 4) return fail(VRHI_ERR_SIZE, "%s: input holds %llu bytes, %llu needed", name, (unsigned long long)args[0].bytes, (unsigned long long)(q->rows * q->cols * 4));
  for (int k = 1; k < n_args; ++k)
    if (!writable(args[k])) return fail(VRHI_ERR_INVALID, "%s: argument %d is read-only (class %s)", name, k, vrhi_arg_class_name(args[k].buf_cls));
  return VRHI_OK;
}

static int need(const ArgView &a, uint64_t bytes, const char *name, int k) {
  if (a.bytes < bytes) return fail(VRHI_ERR_SIZE, "%s: argument %d holds %llu bytes, %llu needed", name, k, (unsigned long long)a.bytes, (unsigned long long)bytes);
  return VRHI_OK;
}

int launch_row_sum(vrhi_stream_t *st, const ArgView *args, int n_args, const void *params, size_t params_size) {
  vrhi_rows_params q;
  VRHI_TRY(rows_common(args, n_args, 2, params, params_size, &q, "row_sum"));
  if (q.rows == 0) return VRHI_OK;
  VRHI_TRY(need(args[1], q.rows * 4, "row_sum", 1));
  return launch_rows<ROW_SUM>(st, (const float *)args[0].ptr, (float *)args[1].ptr, nullptr, nullptr, q.rows, q.cols, "row_sum");
}

int launch_row_max(vrhi_stream_t *st, const ArgView *args, int n_args, const void *params, size_t params_size) {
  vrhi_rows_params q;
  VRHI_TRY(rows_common(args, n_args, 2, params, params_size, &q, "row_max"));
  if (q.rows == 0) return VRHI_OK;
  VRHI_TRY(need(args[1], q.rows * 4, "row_max", 1));
  return launch_rows<ROW_MAX>(st, (const float *)args[0].ptr, nullptr, (float *)args[1].ptr, nullptr, q.rows, q.cols, "row_max");
}

int launch_row_softmax(vrhi_stream_t *st, const ArgView *args, int n_args, const void *params, size_t params_size) {
  vrhi_rows_params q;
  VRHI_TRY(rows_common(args, n_args, 2, params, params_size, &q, "row_softmax"));
  if (q.rows == 0) return VRHI_OK;
  VRHI_TRY(need(args[1], q.rows * q.cols * 4, "row_softmax", 1));
  return launch_rows<ROW_SOFTMAX>(st, (const float *)args[0].ptr, nullptr, nullptr, (float *)args[1].ptr, q.rows, q.cols, "row_softmax");
}

int launch_row_stats_softmax(vrhi_stream_t *st, const ArgView *args, int n_args, const void *params, size_t params_size) {
  vrhi_rows_params q;
  VRHI_TRY(rows_common(args, n_args, 4, params, params_size, &q, "row_stats_softmax"));
  if (q.rows == 0) return VRHI_OK;
  VRHI_TRY(need(args[1], q.rows * 4, "row_stats_softmax", 1));
  VRHI_TRY(need(args[2], q.rows * 4, "row_stats_softmax", 2));
  VRHI_TRY(need(args[3], q.rows * q.cols * 4, "row_stats_softmax", 3));
  return launch_rows<ROW_SUM | ROW_MAX | ROW_SOFTMAX>(st, (const float *)args[0].ptr, (float *)args[1].ptr, (float *)args[2].ptr,
                                                       (float *)args[3].ptr, q.rows, q.cols, "row_stats_softmax");
}

// ---------------------------------------------------------------------------------------------
// Column sums, HBM-bound.  Stage 1: a block owns a tile of W adjacent column groups (a group is a float4 where the
// row length allows it, else one column) and walks down the rows R at a time: thread t holds group t % W of
// the rows t / W, t / W + R, ... so a narrow matrix keeps the whole block busy and neighbouring threads always
// read neighbouring addresses (with one thread per column whatever the width, [2^20, 33] used 33 of 256 threads).
// Eight rows are in flight per thread, and the R rows of a block are added up in shared memory, so one
// partial row per block is all that stage 2 has to read.  Stage 2 adds the partial rows.  No atomics, and
// the order of every addition depends on the shape only.
// Measured on B200 against one thread per column group and a block per row: [65536,4096] 166 -> 153 us
// (7.0 TB/s), [4096,16385] 69 -> 48 us, [1000000,33] 463 -> 28 us, [1000,1001] 20.7 -> 5.0 us.
constexpr int kColRowsInFlight = 8;
template <bool VEC> constexpr int kColBlocksPerSm = VEC ? 5 : 8;  // 48 and 32 registers per thread

template <bool VEC> struct ColValue { typedef float type; };
template <> struct ColValue<true> { typedef float4 type; };
__device__ __forceinline__ void col_add(float &a, float v) { a += v; }
__device__ __forceinline__ void col_add(float4 &a, float4 v) { a.x += v.x; a.y += v.y; a.z += v.z; a.w += v.w; }
__device__ __forceinline__ void col_zero(float &a) { a = 0.f; }
__device__ __forceinline__ void col_zero(float4 &a) { a = make_float4(0.f, 0.f, 0.f, 0.f); }

// groups: column groups of a row; dst: one row of `groups` per blockIdx.y
template <bool VEC>
__global__ void __launch_bounds__(256, kColBlocksPerSm<VEC>) col_partial_kernel(const void *__restrict__ in_raw, void *__restrict__ partial_raw, uint64_t rows,
                                                          uint64_t groups, uint32_t W, uint32_t R, uint32_t *tickets, float *out) {
  typedef typename ColValue<VEC>::type V;
  __shared__ V red[256];
  __shared__ double fin[256];
  __shared__ bool last;
  pdl_begin();
  const V *__restrict__ in = static_cast<const V *>(in_raw);
  const uint32_t sub = threadIdx.x / W, w = threadIdx.x - sub * W;
  const uint64_t g = (uint64_t)blockIdx.x * W + w;
  const bool active = sub < R && g < groups;
  V acc, sums[4];
  col_zero(acc);
#pragma unroll
  for (int k = 0; k < 4; ++k) col_zero(sums[k]);
  if (active) {
    const uint64_t step = (uint64_t)gridDim.y * R;
    uint64_t r = (uint64_t)blockIdx.y * R + sub;
    const V *p = in + r * groups + g;
    const uint64_t pstep = step * groups;
    for (; r + (kColRowsInFlight - 1) * step < rows; r += kColRowsInFlight * step, p += kColRowsInFlight * pstep) {
      V v[kColRowsInFlight];
#pragma unroll
      for (int k = 0; k < kColRowsInFlight; ++k) v[k] = __ldcs(p + k * pstep);
      // A wide matrix leaves few threads per column (four in [1024,65535]): rows added one by one would be a chain of 256
      // roundings.  Groups of four columns are added as a tree per eight rows (32 + 3 roundings), single columns into four
      // running sums (64 + 2), because their tree costs time ([4096,16385] 50.2 us, one by one and so 48.6; the running
      // sums cost [1024,65535] 54.3 -> 55.9).  Relative error of that sum, values of mean 1: 1.2e-7 -> 5.1e-8.
      if constexpr (VEC) {
#pragma unroll
        for (int n = 1; n < kColRowsInFlight; n *= 2)
#pragma unroll
          for (int k = 0; k < kColRowsInFlight; k += 2 * n) col_add(v[k], v[k + n]);
        col_add(acc, v[0]);
      } else {
#pragma unroll
        for (int k = 0; k < kColRowsInFlight; ++k) col_add(sums[k & 3], v[k]);
      }
    }
    for (; r < rows; r += step, p += pstep) col_add(acc, __ldcs(p));
    if constexpr (!VEC) {
      col_add(sums[0], sums[1]);
      col_add(sums[2], sums[3]);
      col_add(sums[0], sums[2]);
      col_add(acc, sums[0]);
    }
  }
  if (R > 1) {
    red[threadIdx.x] = acc;
    // tree over the R rows of the block; R need not be a power of two
    for (uint32_t n = R; n > 1;) {
      const uint32_t half = (n + 1) >> 1;
      __syncthreads();
      if (active && sub < n - half) {
        acc = red[threadIdx.x];
        col_add(acc, red[threadIdx.x + half * W]);
        red[threadIdx.x] = acc;
      }
      n = half;
    }
  }
  if (active && sub == 0) static_cast<V *>(partial_raw)[(uint64_t)blockIdx.y * groups + g] = acc;
  if (!tickets) return;
  // Few partial rows: the last block to finish a tile adds them up, in binary64 and in an order that depends on the shape
  // only, and saves the second launch (2.5 us of host time and 2 of the GPU's).  The ticket wraps to 0 behind it.
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicInc(tickets + blockIdx.x, gridDim.y - 1u) == gridDim.y - 1u;
  __syncthreads();
  if (!last) return;
  __threadfence();
  constexpr uint32_t PER = VEC ? 4u : 1u;
  const uint64_t cols = groups * PER, c0 = (uint64_t)blockIdx.x * W * PER;
  const uint32_t n = (uint32_t)(cols - c0 < W * PER ? cols - c0 : W * PER), T = 256u / n, part = threadIdx.x / n, c = threadIdx.x - part * n;
  const float *p = static_cast<const float *>(partial_raw) + c0 + c;
  double s = 0.0;
  if (part < T) {
    uint32_t k = part;
    for (; k + 3 * T < gridDim.y; k += 4 * T) {
      const double a = __ldcg(p + k * cols), b = __ldcg(p + (k + T) * cols), d = __ldcg(p + (k + 2 * T) * cols), e = __ldcg(p + (k + 3 * T) * cols);
      s += (a + b) + (d + e);
    }
    for (; k < gridDim.y; k += T) s += (double)__ldcg(p + k * cols);
  }
  fin[threadIdx.x] = s;
  for (uint32_t m = T; m > 1;) {
    const uint32_t half = (m + 1) >> 1;
    __syncthreads();
    if (part < m - half) {
      s = fin[threadIdx.x] + fin[threadIdx.x + half * n];
      fin[threadIdx.x] = s;
    }
    m = half;
  }
  if (part == 0) out[c0 + c] = (float)s;
}

// Stage 2: a block of 1024 threads owns min(cols, 32) adjacent columns of one job; its threads take the partial rows in
// turn (coalesced, four independent loads each) and are combined in a tree, in binary64.  It is latency-bound, so the
// rows are spread over many threads (with eight warps per 32 columns, 1000 partial rows took 30 us), every sum that a
// kernel left behind is finished by one launch, and that launch is a dependent of stage 1.
__global__ void __launch_bounds__(1024) finish_partials_kernel(const __grid_constant__ FinishJobs jobs) {
  __shared__ double red[1024];
  int j = 0;
  while (j + 1 < jobs.n && blockIdx.x >= jobs.job[j].last_block) ++j;
  const FinishJobs::Job &J = jobs.job[j];
  const uint32_t block = blockIdx.x - (j ? jobs.job[j - 1].last_block : 0u), W = J.W, R = 1024u / W, groups = J.groups;
  const uint64_t cols = J.cols;
  const uint32_t sub = threadIdx.x / W, w = threadIdx.x - sub * W;
  const uint64_t c = (uint64_t)block * W + w;
  const bool active = sub < R && c < cols;
  pdl_begin();
  double s = 0.0;
  if (active) {
    uint32_t g = sub;
    const float *p = J.partial + (uint64_t)sub * cols + c;
    const uint64_t pstep = (uint64_t)R * cols;
    for (; g + 3 * R < groups; g += 4 * R, p += 4 * pstep) {
      const double a = p[0], b = p[pstep], d = p[2 * pstep], e = p[3 * pstep];
      s += (a + b) + (d + e);
    }
    for (; g < groups; g += R, p += pstep) s += (double)*p;
  }
  red[threadIdx.x] = s;
  for (uint32_t n = R < groups ? R : groups; n > 1;) {
    const uint32_t half = (n + 1) >> 1;
    __syncthreads();
    if (active && sub < n - half) {
      s = red[threadIdx.x] + red[threadIdx.x + half * W];
      red[threadIdx.x] = s;
    }
    n = half;
  }
  if (active && sub == 0) J.out[c] = (float)(s * J.scale);
}

void add_finish_job(FinishJobs *jobs, const float *partial, float *out, uint32_t groups, uint64_t cols, double scale) {
  FinishJobs::Job &J = jobs->job[jobs->n];
  J.partial = partial; J.out = out; J.scale = scale; J.cols = cols; J.groups = groups;
  J.W = (uint32_t)(cols < 32 ? cols : 32);
  J.last_block = (uint32_t)((cols + J.W - 1) / J.W) + (jobs->n ? jobs->job[jobs->n - 1].last_block : 0u);
  ++jobs->n;
}

cudaError_t finish_partials(cudaStream_t s, const FinishJobs &jobs) {
  return launch_dependent(finish_partials_kernel, dim3(jobs.job[jobs.n - 1].last_block), 1024, 0, s, jobs);
}

// Tile and grid of stage 1.  Tiles of at most 64 float4 (1 KiB of a row) or 128 columns: several rows per block even
// in a wide matrix.  At most one wave of blocks (rounded up, [4096,16385] had 1290 blocks for 1184 places), and at
// least kColRowsInFlight rows for every thread, so that a small matrix is not spread over more partial rows than it
// has rows to give.
struct ColPlan {
  bool vec;
  uint64_t groups;
  uint32_t W, R;
  unsigned gx, gy;
};
static ColPlan plan_col_sum(uint64_t rows, uint64_t cols, int sms, uint64_t most_gy) {
  ColPlan p{};
  p.vec = cols % 4 == 0;
  p.groups = p.vec ? cols / 4 : cols;
  const uint64_t most_w = p.vec ? 64 : 128;
  const uint64_t gx = (p.groups + most_w - 1) / most_w;
  p.W = (uint32_t)((p.groups + gx - 1) / gx);
  p.R = 256u / p.W;
  uint64_t gy = (uint64_t)sms * (p.vec ? kColBlocksPerSm<true> : kColBlocksPerSm<false>) / gx;
  const uint64_t by_rows = (rows + (uint64_t)p.R * kColRowsInFlight - 1) / ((uint64_t)p.R * kColRowsInFlight);
  if (gy > by_rows) gy = by_rows;
  if (gy > 4096) gy = 4096;
  if (gy > most_gy) gy = most_gy;
  p.gx = (unsigned)gx;
  p.gy = (unsigned)(gy ? gy : 1);
  return p;
}

// dst: p.gy partial rows, or, where the plan has one block row, the result itself
// tickets, out: not null where the last block of a tile is to finish the sums (launch_col_sum)
static cudaError_t launch_col_partial(bool chain, cudaStream_t s, const ColPlan &p, const float *in, float *dst, uint64_t rows,
                                      uint32_t *tickets = nullptr, float *out = nullptr) {
  const dim3 grid(p.gx, p.gy);
  return launch_chained(chain, p.vec ? col_partial_kernel<true> : col_partial_kernel<false>, grid, 256, 0, s, (const void *)in, (void *)dst, rows, p.groups, p.W, p.R, tickets, out);
}

int launch_col_sum(vrhi_stream_t *st, const ArgView *args, int n_args, const void *params, size_t params_size) {
  vrhi_rows_params q;
  VRHI_TRY(rows_common(args, n_args, 2, params, params_size, &q, "col_sum"));
  if (q.cols == 0) return VRHI_OK;
  VRHI_TRY(need(args[1], q.cols * 4, "col_sum", 1));
  if (q.rows == 0) {
    VRHI_CUDA(cudaMemsetAsync(args[1].ptr, 0, q.cols * 4, st->s));
    return VRHI_OK;
  }
  const ColPlan p = plan_col_sum(q.rows, q.cols, st->dev->prop.multiProcessorCount, ~0ull);
  float *out = (float *)args[1].ptr, *dst = out;
  uint32_t *ctrl = nullptr, *tickets = nullptr;
  if (p.gy > 1) {
    char *payload = nullptr;
    VRHI_TRY(stream_arena(st, p.gy * q.cols * 4, &ctrl, &payload));
    dst = (float *)payload;
    // at most 64 values per thread of the block that finishes a tile; beyond, 1024 threads per 32 columns are faster
    const uint64_t values = (uint64_t)p.gy * p.W * (p.vec ? 4 : 1);
    if (p.gx <= kColTickets && values <= 256 * 64) tickets = ctrl + CTRL_COL_TICKETS;
  }
  VRHI_CUDA(launch_col_partial(chains(st), st->s, p, (const float *)args[0].ptr, dst, q.rows, tickets, out));
  VRHI_TRY(post_launch(st, "col_sum"));
  if (p.gy == 1 || tickets) return VRHI_OK;
  FinishJobs jobs{};
  add_finish_job(&jobs, dst, out, p.gy, q.cols, 1.0);
  VRHI_CUDA(finish_partials(st->s, jobs));
  return post_launch(st, "col_sum (second stage)");
}

}  // namespace vrhi

// ---------------------------------------------------------------------------------------------
// Column sums for callers that must not allocate.
//
// Some users of this library sit where an allocation is not an option: a frame or control loop
// with a hard latency budget (cudaMalloc can take milliseconds and serialises the device), a
// process whose HBM was carved up front between tenants so that nothing may grow later, or code
// running between other people's kernels that may not disturb the allocator's state.  Every
// other operator here takes its scratch from a per-stream arena that is allocated on first use
// and may grow; this entry point instead keeps the per-row-group partial sums in a fixed array
// that is part of the library image.  Cost: each GPU that loads the library holds the array
// (kStaticPartialFloats * 4 bytes = 1 MiB) until the process exits.
//
// Use: the first call on a device asks CUDA for the array's device address (a lookup, not an
// allocation); let that first call happen before any stream capture is begun.  The array is
// shared by every call on the device and keeps whatever the last call left in it, so two calls
// whose kernels could run at the same time (different streams with no ordering between them)
// race; calls on one stream, or ordered by events, are safe.  No call here reaches cudaMalloc,
// cudaFree or any allocating library routine.
#include <mutex>

namespace {

constexpr uint64_t kStaticPartialFloats = 262144;  // 1 MiB: e.g. 64 row groups of 4096 columns
static __device__ __align__(256) float g_static_col_partials[kStaticPartialFloats];

constexpr int kMaxDevices = 64;
std::mutex g_static_mu;
float *g_static_partials_ptr[kMaxDevices] = {};  // device address of the array, per device ordinal
int g_static_sm_count[kMaxDevices] = {};

// The array's name is only a host-side stand-in: the device address has to be asked for, once
// per device, with that device current.
int static_scratch_for_current_device(float **out_ptr, int *out_sms) {
  int dev = -1;
  VRHI_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kMaxDevices) return vrhi::fail(VRHI_ERR_UNSUPPORTED, "device ordinal %d is beyond the %d this entry point tracks", dev, kMaxDevices);
  std::lock_guard<std::mutex> lock(g_static_mu);
  if (!g_static_partials_ptr[dev]) {
    void *p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_static_col_partials);
    if (e != cudaSuccess || !p) return vrhi::fail(VRHI_ERR_CUDA, "cudaGetSymbolAddress(static column partials) failed: %s", cudaGetErrorString(e));
    int sms = 0;
    VRHI_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    g_static_sm_count[dev] = sms;
    g_static_partials_ptr[dev] = static_cast<float *>(p);
  }
  *out_ptr = g_static_partials_ptr[dev];
  *out_sms = g_static_sm_count[dev];
  return VRHI_OK;
}

}  // namespace

extern "C" int vrhi_col_sum_static_scratch(const float *in_device, float *out_device, uint64_t rows, uint64_t cols,
                                           void *cuda_stream) {
  using namespace vrhi;
  if (!in_device || !out_device) return fail(VRHI_ERR_INVALID, "col_sum_static_scratch: NULL pointer");
  if (cols == 0) return VRHI_OK;
  if (cols > kStaticPartialFloats)
    return fail(VRHI_ERR_SIZE, "col_sum_static_scratch: %llu columns exceed the fixed scratch (%llu floats); use the col_sum operator", (unsigned long long)cols, (unsigned long long)kStaticPartialFloats);
  if (rows > (1ull << 40)) return fail(VRHI_ERR_SIZE, "col_sum_static_scratch: row count out of range");
  if (reinterpret_cast<uintptr_t>(in_device) % 16 || reinterpret_cast<uintptr_t>(out_device) % 4)
    return fail(VRHI_ERR_SIZE, "col_sum_static_scratch: input must be 16-byte aligned and output 4-byte aligned");
  cudaStream_t s = static_cast<cudaStream_t>(cuda_stream);
  if (rows == 0) {
    VRHI_CUDA(cudaMemsetAsync(out_device, 0, cols * 4, s));
    return VRHI_OK;
  }
  float *partials = nullptr;
  int sms = 0;
  VRHI_TRY(static_scratch_for_current_device(&partials, &sms));
  const ColPlan p = plan_col_sum(rows, cols, sms, kStaticPartialFloats / cols);  // at least one partial row by the check above
  // Stage 1 writes every partial that stage 2 reads (gy rows of `cols` floats), so nothing in the
  // array has to be cleared and whatever an earlier call left behind is never read.
  // (float4 stores: an output that is only 4-byte aligned goes through the array even where one partial row is enough.)
  const bool direct = p.gy == 1 && (!p.vec || reinterpret_cast<uintptr_t>(out_device) % 16 == 0);
  cudaError_t e = launch_col_partial(false, s, p, in_device, direct ? out_device : partials, rows);
  if (e != cudaSuccess) return fail(VRHI_ERR_CUDA, "launch of col_sum_static_scratch (partials) failed: %s", cudaGetErrorString(e));
  if (!direct) {
    FinishJobs jobs{};
    add_finish_job(&jobs, partials, out_device, p.gy, cols, 1.0);
    e = finish_partials(s, jobs);
  }
  if (e != cudaSuccess) return fail(VRHI_ERR_CUDA, "launch of col_sum_static_scratch (finalize) failed: %s", cudaGetErrorString(e));
  return VRHI_OK;
}
