// Per-element shader-style maps: the arithmetic of the reference's shader input file
// (source/tests/integration/color.mlir) as plain CUDA kernels over arrays.
//
//   vertex stage (color.mlir:4-39): extend each position (p0,p1,p2) to (p0,p1,p2,1), apply the
//     model, view and projection matrices one after the other (the three linalg.matvec steps the
//     file sketches at :29-36), emit gl_Position and pass the position through as the varying;
//   fragment stage (color.mlir:43-59): extend the uniform colour (c0,c1,c2) to (c0,c1,c2,1) for
//     every fragment of a pixel buffer.
//
// No graphics API is involved: inputs and outputs are device arrays, the "pixel buffer" is a
// headless [n][4] float array.  Both kernels are HBM-bound (28 + 12 bytes per vertex, 16 bytes per
// fragment).  Each matrix row is applied as one multiply and three fused multiply-adds, left to
// right.
#include <cstring>

#include "vrhi_internal.h"

namespace vrhi {

struct __align__(16) Mat4 {
  float m[16];  // row-major
};

__device__ __forceinline__ float4 matvec4(const Mat4 &M, float4 v) {
  float4 r;
  r.x = fmaf(M.m[3], v.w, fmaf(M.m[2], v.z, fmaf(M.m[1], v.y, M.m[0] * v.x)));
  r.y = fmaf(M.m[7], v.w, fmaf(M.m[6], v.z, fmaf(M.m[5], v.y, M.m[4] * v.x)));
  r.z = fmaf(M.m[11], v.w, fmaf(M.m[10], v.z, fmaf(M.m[9], v.y, M.m[8] * v.x)));
  r.w = fmaf(M.m[15], v.w, fmaf(M.m[14], v.z, fmaf(M.m[13], v.y, M.m[12] * v.x)));
  return r;
}

// A block takes 1024 vertices: their positions, one contiguous range, come in as float4s, go out again as the varying
// in the same registers, and lie in shared memory while every thread transforms four vertices (stride 3 words: no bank
// conflicts).  All global accesses are 16 bytes per thread and contiguous per warp.  Measured on B200, 1000003 vertices:
// 7.9 us with a thread per vertex (4-byte accesses, 12 bytes apart; a last wave of a third of the blocks), 6.4 us so; 2^24: 161 and 109 us.
constexpr int kVerts = 1024;
__global__ void __launch_bounds__(256, 4) vertex_transform_kernel(const float *__restrict__ pos, const float *__restrict__ model,
                                                               const float *__restrict__ view, const float *__restrict__ proj,
                                                               float4 *__restrict__ out_pos, float *__restrict__ out_varying,
                                                               uint64_t n) {
  __shared__ __align__(16) float tile[3 * kVerts];
  __shared__ Mat4 sm[3];
  pdl_begin();
  const uint32_t t = threadIdx.x;
  if (t < 48) {
    const float *src = t < 16 ? model : (t < 32 ? view : proj);
    sm[t / 16].m[t % 16] = src[t % 16];
  }
  for (uint64_t base = (uint64_t)blockIdx.x * kVerts; base < n; base += (uint64_t)gridDim.x * kVerts) {
    const uint32_t here = (uint32_t)(n - base < kVerts ? n - base : kVerts), floats = 3 * here;
    const float4 *src4 = reinterpret_cast<const float4 *>(pos + 3 * base);
    float4 *var4 = reinterpret_cast<float4 *>(out_varying + 3 * base);
    float4 v[3];
#pragma unroll
    for (int k = 0; k < 3; ++k)
      if (4 * (t + 256 * k) + 3 < floats) v[k] = __ldcs(src4 + t + 256 * k);
    const uint32_t left = floats & ~3u;  // the up to three floats behind the last float4
    const float edge = t < (floats & 3u) ? pos[3 * base + left + t] : 0.f;
#pragma unroll
    for (int k = 0; k < 3; ++k)
      if (4 * (t + 256 * k) + 3 < floats) {
        __stcs(var4 + t + 256 * k, v[k]);
        reinterpret_cast<float4 *>(tile)[t + 256 * k] = v[k];
      }
    if (t < (floats & 3u)) {
      out_varying[3 * base + left + t] = edge;
      tile[left + t] = edge;
    }
    __syncthreads();
    float4 p[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const uint32_t k = t + 256 * q;
      p[q] = k < here ? make_float4(tile[3 * k], tile[3 * k + 1], tile[3 * k + 2], 1.0f) : make_float4(0.f, 0.f, 0.f, 1.0f);
    }
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      const Mat4 M = sm[m];
#pragma unroll
      for (int q = 0; q < 4; ++q) p[q] = matvec4(M, p[q]);
    }
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (t + 256 * q < here) __stcs(out_pos + base + t + 256 * q, p[q]);
    __syncthreads();  // the tile may be filled again
  }
}

__global__ void __launch_bounds__(256) flat_color_kernel(const float *__restrict__ color, float4 *__restrict__ out, uint64_t n) {
  pdl_begin();
  const float4 c = make_float4(color[0], color[1], color[2], 1.0f);
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += stride) __stcs(out + k, c);
}

static unsigned grid_for(vrhi_stream_t *st, uint64_t n) {
  const uint64_t cap = (uint64_t)st->dev->prop.multiProcessorCount * 8;
  uint64_t want = (n + 255) / 256;
  return (unsigned)(want < cap ? (want ? want : 1) : cap);
}

int launch_vertex_transform(vrhi_stream_t *st, const ArgView *args, int n_args, const void *params, size_t params_size) {
  vrhi_map_params q;
  VRHI_TRY(read_params(params, params_size, &q));
  if (n_args != 6) return fail(VRHI_ERR_INVALID, "vertex_transform takes 6 arguments (pos, model, view, proj, gl_position, varying), got %d", n_args);
  if (q.n == 0) return VRHI_OK;
  const uint64_t need[6] = {q.n * 12, 64, 64, 64, q.n * 16, q.n * 12};
  for (int k = 0; k < 6; ++k)
    if (args[k].bytes < need[k]) return fail(VRHI_ERR_SIZE, "vertex_transform: argument %d holds %llu bytes, %llu needed", k, (unsigned long long)args[k].bytes, (unsigned long long)need[k]);
  if (!writable(args[4]) || !writable(args[5])) return fail(VRHI_ERR_INVALID, "vertex_transform: an output buffer is read-only");
  VRHI_CUDA(launch_chained(chains(st), vertex_transform_kernel, dim3(grid_for(st, (q.n + 3) / 4)), 256, 0, st->s, (const float *)args[0].ptr, (const float *)args[1].ptr, (const float *)args[2].ptr,
                                                                (const float *)args[3].ptr, (float4 *)args[4].ptr, (float *)args[5].ptr, q.n));
  return post_launch(st, "vertex_transform");
}

int launch_flat_color(vrhi_stream_t *st, const ArgView *args, int n_args, const void *params, size_t params_size) {
  vrhi_map_params q;
  VRHI_TRY(read_params(params, params_size, &q));
  if (n_args != 2) return fail(VRHI_ERR_INVALID, "flat_color takes 2 arguments (color, fragments), got %d", n_args);
  if (q.n == 0) return VRHI_OK;
  if (args[0].bytes < 12) return fail(VRHI_ERR_SIZE, "flat_color: the colour needs 12 bytes");
  if (args[1].bytes < q.n * 16) return fail(VRHI_ERR_SIZE, "flat_color: the fragment buffer holds %llu bytes, %llu needed", (unsigned long long)args[1].bytes, (unsigned long long)q.n * 16);
  if (!writable(args[1])) return fail(VRHI_ERR_INVALID, "flat_color: the fragment buffer is read-only");
  VRHI_CUDA(launch_chained(chains(st), flat_color_kernel, dim3(grid_for(st, q.n)), 256, 0, st->s, (const float *)args[0].ptr, (float4 *)args[1].ptr, q.n));
  return post_launch(st, "flat_color");
}

}  // namespace vrhi
