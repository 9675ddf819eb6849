// loss = mean((tanh(W*x + b) - t)^2) over a row-major [rows][cols] problem with b a [cols] row
// vector, and its hand-fused reverse-mode gradient, sm_100a.  HBM-bound.
//
// Backward recomputes the forward instead of reading a saved activation, which is the algorithmic
// minimum of traffic: read W, x, t once, write dW, dx once (20 bytes per element).  A thread owns
// four adjacent columns and walks down a fixed set of rows, so b is loaded once per thread and the
// column sums for db accumulate in registers in a fixed order; one partial row per row group is
// then added up by a second tiny kernel.  No float atomics anywhere: reruns are bit-identical.
// The reference project has no counterpart for these operators.
//
// Numerics: with E = exp(-2|u|), tanh(u) = sign(u)*(1-E)/(1+E) and 1 - tanh(u)^2 = 4E/(1+E)^2.
// The second form has no cancellation, so the gradient keeps its relative accuracy where tanh
// saturates (1 - y*y evaluated from a rounded y loses it).
#include <cstring>

#include <cstdlib>

#include "vrhi_internal.h"

namespace vrhi {

struct TanhPair {
  float y;      // tanh(u)
  float sech2;  // 1 - tanh(u)^2
};

__device__ __forceinline__ TanhPair tanh_pair(float u) {
  const float e = expf(-2.0f * fabsf(u));
  const float r = 1.0f / (1.0f + e);
  TanhPair p;
  p.y = copysignf((1.0f - e) * r, u);
  p.sech2 = 4.0f * e * r * r;
  return p;
}

__device__ __forceinline__ float block_sum_256(float v, float *smem) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) smem[w] = v;
  __syncthreads();
  float r = (l < 8) ? smem[l] : 0.f;
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) r += __shfl_xor_sync(0xffffffffu, r, o);
  return r;  // valid in warp 0
}

// One element of the backward.  inv = 2/denom.
__device__ __forceinline__ void bwd_one(float w, float x, float b, float t, float inv, float &dw, float &dx, float &gsum,
                                        float &lsum) {
  const TanhPair p = tanh_pair(fmaf(w, x, b));
  const float d = p.y - t;
  const float g = d * p.sech2 * inv;
  dw = g * x;
  dx = g * w;
  gsum += g;
  lsum = fmaf(d, d, lsum);
}

// The arrays are walked as rows of float4 groups whatever the row length: P = 4 / gcd(4, cols) rows together are a "super row"
// of P * cols elements, which is a multiple of 4 and starts on a 16-byte boundary.  The group g of a super row holds the
// elements 4g .. 4g+3, of the columns (4g + j) mod cols, so a thread that stays on one group down the super rows needs
// four values of b, once; and a partial row of the column sums, one super row long, is P partial rows of cols columns.
// The rows % P rows behind the last super row are a partial one: `rem` elements, done by the thread that comes to it.
// A block owns a tile of W adjacent groups and walks down the super rows R = 256 / W at a time, as the column sums of
// k_rows.cu do, so a narrow problem keeps the whole block busy.
// Measured on B200 against four adjacent columns per thread with single-element loads (row lengths that are no multiple
// of 4) and a block per row (narrow ones), gradients / loss in us: [4095,4095] 109 -> 60 / 58 -> 33,
// [65536,1023] 428 -> 220 / 250 -> 118, [65536,16] 65 -> 8 / 36 -> 5.
struct MseShape {
  uint64_t rows;    // super rows
  uint64_t groups;  // float4 groups of a super row
  uint64_t rem;     // elements of the partial super row
  uint32_t cols, W, R;
  uint32_t fold;    // P where one block holds a whole super row of several rows: it adds those up itself; else 1
};
__device__ __forceinline__ float4 load_b(const float *B, uint64_t g, uint32_t cols) {
  if ((cols & 3u) == 0) return reinterpret_cast<const float4 *>(B)[g];
  uint64_t k = 4 * g;  // below P * cols <= 4 * cols
  uint32_t c = (uint32_t)(k - ((k >= cols) + (k >= 2ull * cols) + (k >= 3ull * cols)) * (uint64_t)cols);
  float4 b;
  b.x = B[c]; c = c + 1 == cols ? 0u : c + 1;
  b.y = B[c]; c = c + 1 == cols ? 0u : c + 1;
  b.z = B[c]; c = c + 1 == cols ? 0u : c + 1;
  b.w = B[c];
  return b;
}
__device__ __forceinline__ float &component(float4 &v, int j) { return j == 0 ? v.x : j == 1 ? v.y : v.z; }

__global__ void __launch_bounds__(256, 5) mse_bwd_kernel(const float *__restrict__ W_, const float *__restrict__ X_,
                                                      const float *__restrict__ B, const float *__restrict__ T_,
                                                      float *__restrict__ dW, float *__restrict__ dX,
                                                      float *__restrict__ db_partial, float *__restrict__ loss_partial,
                                                      const MseShape q, float inv) {
  __shared__ float4 red[256];
  __shared__ float smem[8];
  pdl_begin();
  const float4 *__restrict__ w4 = reinterpret_cast<const float4 *>(W_), *__restrict__ x4 = reinterpret_cast<const float4 *>(X_), *__restrict__ t4 = reinterpret_cast<const float4 *>(T_);
  const uint32_t sub = threadIdx.x / q.W, lane = threadIdx.x - sub * q.W;
  const uint64_t gi = (uint64_t)blockIdx.x * q.W + lane;
  const bool active = sub < q.R && gi < q.groups;
  float4 g = make_float4(0.f, 0.f, 0.f, 0.f);
  float lsum = 0.f;
  if (active) {
    float4 b = load_b(B, gi, q.cols);
    const uint64_t step = (uint64_t)gridDim.y * q.R, istep = step * q.groups;
    uint64_t r = (uint64_t)blockIdx.y * q.R + sub, i = r * q.groups + gi;
    // one super row per trip: 47 registers; two (63 registers) measured slower, 0.464 ms against 0.419 ms on [32768,4096], and so
    // did the 55 registers that the compiler takes unless it is told to leave room for five blocks (0.424 ms against 0.413)
    for (; r < q.rows; r += step, i += istep) {
      const float4 wa = __ldcs(w4 + i), xa = __ldcs(x4 + i), ta = __ldcs(t4 + i);
      float4 ow, ox;
      bwd_one(wa.x, xa.x, b.x, ta.x, inv, ow.x, ox.x, g.x, lsum);
      bwd_one(wa.y, xa.y, b.y, ta.y, inv, ow.y, ox.y, g.y, lsum);
      bwd_one(wa.z, xa.z, b.z, ta.z, inv, ow.z, ox.z, g.z, lsum);
      bwd_one(wa.w, xa.w, b.w, ta.w, inv, ow.w, ox.w, g.w, lsum);
      __stcs(reinterpret_cast<float4 *>(dW) + i, ow);
      __stcs(reinterpret_cast<float4 *>(dX) + i, ox);
    }
    if (r == q.rows && 4 * gi < q.rem) {  // the partial super row
      const int n = q.rem - 4 * gi < 4 ? (int)(q.rem - 4 * gi) : 4;
      for (int j = 0; j < n; ++j) {
        const uint64_t e = 4 * i + j;
        bwd_one(W_[e], X_[e], j == 3 ? b.w : component(b, j), T_[e], inv, dW[e], dX[e], j == 3 ? g.w : component(g, j), lsum);
      }
    }
  }
  if (q.R > 1) {  // tree over the R super rows of the block; R need not be a power of two
    red[threadIdx.x] = g;
    for (uint32_t n = q.R; n > 1;) {
      const uint32_t half = (n + 1) >> 1;
      __syncthreads();
      if (active && sub < n - half) {
        const float4 o = red[threadIdx.x + half * q.W];
        g.x += o.x; g.y += o.y; g.z += o.z; g.w += o.w;
        red[threadIdx.x] = g;
      }
      n = half;
    }
  }
  if (q.fold > 1) {
    __syncthreads();
    if (active && sub == 0) red[lane] = g;
    __syncthreads();
    const float *row = reinterpret_cast<const float *>(red);
    for (uint32_t c = threadIdx.x; c < q.cols; c += 256) {
      float v = row[c];
      for (uint32_t k = 1; k < q.fold; ++k) v += row[c + k * q.cols];
      db_partial[(uint64_t)blockIdx.y * q.cols + c] = v;
    }
  } else if (active && sub == 0) {
    reinterpret_cast<float4 *>(db_partial)[(uint64_t)blockIdx.y * q.groups + gi] = g;
  }
  const float bl = block_sum_256(lsum, smem);
  if (threadIdx.x == 0) loss_partial[(uint64_t)blockIdx.y * gridDim.x + blockIdx.x] = bl;
}

__device__ __forceinline__ void fwd_one(float w, float x, float b, float t, float &lsum) {
  const float d = tanhf(fmaf(w, x, b)) - t;
  lsum = fmaf(d, d, lsum);
}
__device__ __forceinline__ void fwd_four(float4 w, float4 x, float4 b, float4 t, float &lsum) {
  fwd_one(w.x, x.x, b.x, t.x, lsum);
  fwd_one(w.y, x.y, b.y, t.y, lsum);
  fwd_one(w.z, x.z, b.z, t.z, lsum);
  fwd_one(w.w, x.w, b.w, t.w, lsum);
}

__global__ void __launch_bounds__(256) mse_fwd_kernel(const float *__restrict__ W_, const float *__restrict__ X_,
                                                      const float *__restrict__ B, const float *__restrict__ T_,
                                                      float *__restrict__ loss_partial, const MseShape q) {
  __shared__ float smem[8];
  pdl_begin();
  const float4 *__restrict__ w4 = reinterpret_cast<const float4 *>(W_), *__restrict__ x4 = reinterpret_cast<const float4 *>(X_), *__restrict__ t4 = reinterpret_cast<const float4 *>(T_);
  const uint32_t sub = threadIdx.x / q.W, lane = threadIdx.x - sub * q.W;
  const uint64_t gi = (uint64_t)blockIdx.x * q.W + lane;
  float lsum = 0.f;
  if (sub < q.R && gi < q.groups) {
    float4 b = load_b(B, gi, q.cols);
    const uint64_t step = (uint64_t)gridDim.y * q.R, istep = step * q.groups;
    uint64_t r = (uint64_t)blockIdx.y * q.R + sub, i = r * q.groups + gi;
    for (; r + step < q.rows; r += 2 * step, i += 2 * istep) {
      const float4 wa = __ldcs(w4 + i), xa = __ldcs(x4 + i), ta = __ldcs(t4 + i);
      const float4 wb = __ldcs(w4 + i + istep), xb = __ldcs(x4 + i + istep), tb = __ldcs(t4 + i + istep);
      fwd_four(wa, xa, b, ta, lsum);
      fwd_four(wb, xb, b, tb, lsum);
    }
    for (; r < q.rows; r += step, i += istep) fwd_four(__ldcs(w4 + i), __ldcs(x4 + i), b, __ldcs(t4 + i), lsum);
    if (r == q.rows && 4 * gi < q.rem) {  // the partial super row
      const int n = q.rem - 4 * gi < 4 ? (int)(q.rem - 4 * gi) : 4;
      for (int j = 0; j < n; ++j) fwd_one(W_[4 * i + j], X_[4 * i + j], j == 3 ? b.w : component(b, j), T_[4 * i + j], lsum);
    }
  }
  const float bl = block_sum_256(lsum, smem);
  if (threadIdx.x == 0) loss_partial[(uint64_t)blockIdx.y * gridDim.x + blockIdx.x] = bl;
}

struct MsePlan {
  uint64_t rows, cols;
  double denom;
  MseShape shape;
  uint32_t P;  // rows of a super row
  unsigned gx, gy;
};

static int mse_plan(vrhi_stream_t *st, const ArgView *args, int n_in_out, const vrhi_mse_params &q, const char *name, MsePlan *pl) {
  if (q.cols == 0 || q.rows == 0) return fail(VRHI_ERR_SIZE, "%s: empty problem", name);
  if (q.rows > (1ull << 40) || q.cols > (1ull << 31)) return fail(VRHI_ERR_SIZE, "%s: shape out of range", name);
  uint64_t elements = 0;
  VRHI_TRY(element_count(q.rows, q.cols, name, &elements));
  const uint64_t full = elements * 4;
  const uint64_t want[8] = {full, full, q.cols * 4, full, 0, 0, 0, 0};
  for (int k = 0; k < 4; ++k)
    if (args[k].bytes < want[k]) return fail(VRHI_ERR_SIZE, "%s: argument %d holds %llu bytes, %llu needed", name, k, (unsigned long long)args[k].bytes, (unsigned long long)want[k]);
  for (int k = 4; k < n_in_out; ++k)
    if (!writable(args[k])) return fail(VRHI_ERR_INVALID, "%s: argument %d is read-only (class %s)", name, k, vrhi_arg_class_name(args[k].buf_cls));
  pl->rows = q.rows; pl->cols = q.cols;
  pl->denom = q.denom > 0.0 ? q.denom : (double)q.rows * (double)q.cols;
  const int sms = st->dev->prop.multiProcessorCount;
  pl->P = q.cols % 4 == 0 ? 1 : q.cols % 2 == 0 ? 2 : 4;
  MseShape &S = pl->shape;
  S.cols = (uint32_t)q.cols;
  S.groups = pl->P * q.cols / 4;
  S.rows = q.rows / pl->P;
  S.rem = q.rows % pl->P * q.cols;
  // Four 256-thread blocks per SM, one wave: with a few blocks more, some SMs get five ([4097,16381], gradients: 299 us with
  // 640 blocks).  Tiles of 4 KiB of a super row; the gradients take 1 KiB tiles, which leave a quarter of the partial rows
  // for the second stage, where those would be more than a sixteenth of the rows ([1000,1001] 9.7 -> 7.3 us), and where
  // rows start on 16 bytes anyway ([32768,4096] 415.6 -> 413.2 us; [4095,4095] 60.4 us, but 78.9 with the smaller tile).
  static const int env_blocks = env_int("VRHI_MSE_BLOCKS_PER_SM", 1, 8, 4);  // tuning aid
  const uint64_t target = (uint64_t)sms * (uint64_t)env_blocks;
  auto tiles = [&](uint64_t most) { return (S.groups + most - 1) / most; };
  const bool small = n_in_out > 5 && (pl->P == 1 || target / tiles(256) * pl->P * 16 > q.rows);
  const uint64_t gx = tiles(small ? 64 : 256);
  if (gx > 0x7fffffffull) return fail(VRHI_ERR_UNSUPPORTED, "%s: too many columns", name);
  S.W = (uint32_t)((S.groups + gx - 1) / gx);
  S.R = 256u / S.W;
  S.fold = gx == 1 ? pl->P : 1;
  uint64_t gy = target / gx;
  const uint64_t by_rows = (S.rows + (S.rem != 0) + S.R - 1) / S.R;
  if (gy > by_rows) gy = by_rows;
  if (gy > 4096) gy = 4096;
  if (gy == 0) gy = 1;
  pl->gx = (unsigned)gx; pl->gy = (unsigned)gy;
  return VRHI_OK;
}

int launch_mse_tanh_fwd(vrhi_stream_t *st, const ArgView *args, int n_args, const void *params, size_t params_size) {
  vrhi_mse_params q;
  VRHI_TRY(read_params(params, params_size, &q));
  if (n_args != 5) return fail(VRHI_ERR_INVALID, "mse_tanh_fwd takes 5 arguments (W, x, b, t, loss), got %d", n_args);
  MsePlan pl;
  VRHI_TRY(mse_plan(st, args, 5, q, "mse_tanh_fwd", &pl));
  if (args[4].bytes < 4) return fail(VRHI_ERR_SIZE, "mse_tanh_fwd: loss output needs 4 bytes");
  char *payload = nullptr;
  const size_t n_part = (size_t)pl.gx * pl.gy;
  VRHI_TRY(stream_arena(st, n_part * 4, nullptr, &payload));
  dim3 grid(pl.gx, pl.gy);
  const float *W = (const float *)args[0].ptr, *X = (const float *)args[1].ptr, *B = (const float *)args[2].ptr, *T = (const float *)args[3].ptr;
  VRHI_CUDA(launch_chained(chains(st), mse_fwd_kernel, grid, 256, 0, st->s, W, X, B, T, (float *)payload, pl.shape));
  VRHI_TRY(post_launch(st, "mse_tanh_fwd"));
  FinishJobs jobs{};
  add_finish_job(&jobs, (const float *)payload, (float *)args[4].ptr, (uint32_t)n_part, 1, 1.0 / pl.denom);
  VRHI_CUDA(finish_partials(st->s, jobs));
  return post_launch(st, "mse_tanh_fwd (second stage)");
}

int launch_mse_tanh_bwd(vrhi_stream_t *st, const ArgView *args, int n_args, const void *params, size_t params_size) {
  vrhi_mse_params q;
  VRHI_TRY(read_params(params, params_size, &q));
  if (n_args != 7 && n_args != 8) return fail(VRHI_ERR_INVALID, "mse_tanh_bwd takes 7 or 8 arguments (W, x, b, t, dW, dx, db[, loss]), got %d", n_args);
  MsePlan pl;
  VRHI_TRY(mse_plan(st, args, n_args, q, "mse_tanh_bwd", &pl));
  const uint64_t full = pl.rows * pl.cols * 4;
  if (args[4].bytes < full || args[5].bytes < full) return fail(VRHI_ERR_SIZE, "mse_tanh_bwd: dW/dx outputs need %llu bytes each", (unsigned long long)full);
  if (args[6].bytes < pl.cols * 4) return fail(VRHI_ERR_SIZE, "mse_tanh_bwd: db output needs %llu bytes", (unsigned long long)pl.cols * 4);
  if (n_args == 8 && args[7].bytes < 4) return fail(VRHI_ERR_SIZE, "mse_tanh_bwd: loss output needs 4 bytes");
  char *payload = nullptr;
  const size_t n_part = (size_t)pl.gx * pl.gy;
  const uint32_t db_rows = pl.gy * pl.P / pl.shape.fold;  // partial rows of the column sums
  const size_t db_bytes = ((size_t)db_rows * pl.cols * 4 + 15) & ~size_t(15);
  VRHI_TRY(stream_arena(st, db_bytes + n_part * 4, nullptr, &payload));
  float *db_partial = (float *)payload;
  float *loss_partial = (float *)(payload + db_bytes);
  dim3 grid(pl.gx, pl.gy);
  const float *W = (const float *)args[0].ptr, *X = (const float *)args[1].ptr, *B = (const float *)args[2].ptr, *T = (const float *)args[3].ptr;
  const float inv = (float)(2.0 / pl.denom);
  VRHI_CUDA(launch_chained(chains(st), mse_bwd_kernel, grid, 256, 0, st->s, W, X, B, T, (float *)args[4].ptr, (float *)args[5].ptr, db_partial, loss_partial, pl.shape, inv));
  VRHI_TRY(post_launch(st, "mse_tanh_bwd"));
  FinishJobs jobs{};
  add_finish_job(&jobs, db_partial, (float *)args[6].ptr, db_rows, pl.cols, 1.0);
  if (n_args == 8) add_finish_job(&jobs, loss_partial, (float *)args[7].ptr, (uint32_t)n_part, 1, 1.0 / pl.denom);
  VRHI_CUDA(finish_partials(st->s, jobs));
  return post_launch(st, "mse_tanh_bwd (second stage)");
}

}  // namespace vrhi
