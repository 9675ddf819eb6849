// Escape-time map kernels (Mandelbrot / Julia), sm_100a.
//
// Loop rules follow fractal.py:18-25: every pixel is independent, the escape test comes before
// the update, the result counts the updates performed; the square is (z0*z0 - z1*z1, (z1*z0)*2)
// (fractal.py:11-13); coordinates come from the integer index at the pixel corner
// (fractal.py:20).
//
// EXACT mode reproduces these binary32 roundings and no others:
//     a = zr*zr; b = zi*zi; s = a+b; t = zr*zi; zi' = (t+t)+ci; zr' = (a-b)+cr
// (t+t)+ci is issued as fma(2, t, ci): 2*t is exact in binary32, so the fused form rounds the
// same real number once and gives the same bits with one instruction fewer.  Everything else uses
// __fmul_rn / __fadd_rn, which the compiler never contracts.
//
// This file holds the operator's launcher and the fully checked kernel: one pixel per lane, a test
// on every step.  That kernel accepts every parameter combination and is the path of record for
// parameters the kernels with unchecked blocks (k_escape_pair.cu, k_escape_block.cu) cannot take.
#include <cfloat>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <type_traits>
#include <unordered_map>

#include "escape_common.cuh"

namespace vrhi {

template <int KIND, int MODE, int OUT>
__global__ void __launch_bounds__(256) escape_checked_kernel(EscapeDev p, void *image, uint32_t *work_counter, uint16_t *wire) {
  const uint32_t lane = threadIdx.x & 31u;
  begin_launch(p);
  // work_counter == nullptr: batches are dealt to warps round-robin (small frames, where the
  // counter's reset would cost as much as the frame); otherwise warps pull batches from the counter
  uint32_t next = blockIdx.x * 8u + (threadIdx.x >> 5);
  for (;;) {
    uint32_t batch = next;
    if (work_counter) {
      if (lane == 0) batch = next_batch(work_counter, p.n_batches);
      batch = __shfl_sync(0xffffffffu, batch, 0);
    } else {
      next += gridDim.x * 8u;
    }
    if (batch >= p.n_batches) break;
    const uint32_t r = batch / p.batches_per_row;
    const uint32_t tile0 = (batch - r * p.batches_per_row) * p.batch_tiles;
    const uint32_t tile1 = min(tile0 + p.batch_tiles, p.tiles_per_row);
    const uint32_t j = owned_row_to_image_row(p, r);
    const float y = __fadd_rn(p.y0, __fmul_rn((float)j, p.dy));
    const size_t row_base = (size_t)j * p.width;
    for (uint32_t tile = tile0; tile < tile1; ++tile) {
      const uint32_t i = tile * 32u + lane;
      if (i >= p.width) continue;
      const float x = __fadd_rn(p.x0, __fmul_rn((float)i, p.dx));
      float zr, zi, cr, ci;
      if (KIND == VRHI_ESCAPE_MANDELBROT) {
        zr = 0.f; zi = 0.f; cr = p.transposed ? y : x; ci = p.transposed ? x : y;
      } else {
        zr = p.transposed ? y : x; zi = p.transposed ? x : y; cr = p.cr; ci = p.ci;
      }
      const uint32_t count = escape_count<MODE>(zr, zi, cr, ci, p.limit, 0u, p.max_iter);
      store_count<OUT>(image, row_base + i, count, p.color_scale);
      if (wire) store_wire(wire, p.bytes, row_base + i, count);
    }
  }
  end_launch();
}

template <int KIND, int MODE>
static void launch_checked(int out, int grid, cudaStream_t s, const EscapeDev &p, void *image, uint32_t *ctr, uint16_t *wire) {
  uint16_t *const none = nullptr;
  switch (out) {
    case VRHI_OUT_COUNT_U32: launch_chained(p.chained, escape_checked_kernel<KIND, MODE, VRHI_OUT_COUNT_U32>, dim3((unsigned)grid), 256, 0, s, p, image, ctr, wire); break;
    case VRHI_OUT_COUNT_U16: launch_chained(p.chained, escape_checked_kernel<KIND, MODE, VRHI_OUT_COUNT_U16>, dim3((unsigned)grid), 256, 0, s, p, image, ctr, none); break;
    default: launch_chained(p.chained, escape_checked_kernel<KIND, MODE, VRHI_OUT_COLOR_F32>, dim3((unsigned)grid), 256, 0, s, p, image, ctr, none); break;
  }
}

// The largest binary32 s with sqrt(s) < bound (square root rounded to nearest, as the device's __fsqrt_rn and the
// host's sqrtf both do): rounding is monotonic, so sqrt(s) < bound exactly when s <= this value, and the test
// VRHI_TEST_NORM_GE needs no square root per step.  -1 where no s >= 0 passes (bound <= 0 or NaN).
// Measured on B200 against a square root per step: 9.6 -> 4.7 us for a 640 x 320 frame of at most 50 steps, and the
// regrouping kernel takes the test too: 171 -> 50 us for a 1080p Mandelbrot frame of 256.
static float escape_limit(uint32_t test, float bound) {
  if (test == VRHI_TEST_NORM2_GT) return bound;
  if (!(bound > 0.0f)) return -1.0f;
  float s = bound * bound;
  if (!(s <= FLT_MAX)) s = FLT_MAX;
  while (s > 0.0f && !(sqrtf(s) < bound)) s = nextafterf(s, 0.0f);
  while (s < FLT_MAX && sqrtf(nextafterf(s, INFINITY)) < bound) s = nextafterf(s, INFINITY);
  return s;
}

// Steps from which the regrouping kernel is taken.  It pays about 2 us per tile and warp for intake and pool; the block
// kernel runs a warp as long as its slowest pixel, and an image as long as the SM that drew the most such warps.  Which
// costs more depends on how many tiles of 64 pixels a resident warp gets, hence on the pixels, and on the view.
// Measured on B200, regrouping vs blocks in us, two or three views of each set (Julia: -0.8+0.156i, whose pixels all escape;
// -0.123+0.745i, a fifth of whose pixels run to max_iter.  Mandelbrot: the whole set; -0.75+0.1i, 0.04 wide):
//   Julia        256 steps               512                     1024                    2048
//   128 x  64    7.3/7.1    7.3/7.0      10.9/12.5  11.2/12.4    15.7/19.6  19.4/23.2    15.5/19.6  35.3/44.7
//   256 x 256    7.6/7.3    7.8/7.2      11.4/12.7  11.4/12.5    17.2/20.4  19.6/23.2    20.4/29.1  35.5/44.7
//   360 x 360    11.9/7.5   12.0/7.6     18.5/12.7  19.0/12.7    26.0/22.4  34.5/23.5    26.3/29.3  64.0/45.0
//   480 x 480    13.4/11.9  13.4/11.6    20.1/19.8  20.3/19.9    29.9/33.2  35.9/37.2    32.1/36.1  66.3/71.8
//   560 x 560    14.1/13.7  14.8/13.8    20.8/21.1  23.6/24.7    31.1/32.4  42.3/46.3    34.2/34.7  79.0/89.7
//   640 x 700    15.4/14.6  17.5/18.4    22.4/25.4  27.9/32.8    33.1/36.6  50.1/62.1    37.3/38.3  94.8/120.9
//   720 x 720    17.0/18.4  19.2/16.8    24.0/32.0  30.4/29.5    34.3/47.9  55.9/55.6    37.7/48.4  104/107
//   1920 x 1080  36.2/36.9  37.9/38.5    43.1/62.1  55.1/66.3    54.5/87.9  98.4/123.7   61.6/92.1  185/235  (192: 34.0/30.0 33.7/31.2)
//   Mandelbrot
//   128 x  64    8.1/7.1    8.1/6.3      11.9/12.7  12.2/10.8    21.1/23.7  20.9/19.8    38.6/46.2  38.0/37.5
//   256 x 192    12.2/6.5   8.5/6.5      21.2/10.9  12.7/10.9    39.8/19.9  21.6/19.9    75.6/37.8  39.2/37.8
//   400 x 400    13.6/11.1  19.0/14.9    22.8/19.1  30.7/27.0    42.4/35.6  55.7/48.9    82.1/68.2  101.7/89.8
//   448 x 448    14.1/14.5  20.5/15.0    23.6/26.0  33.3/27.3    42.1/49.1  56.1/51.6    81.2/95.0  103.7/100.2
//   640 x 320    13.9/12.5  20.0/15.1    23.0/21.4  31.8/27.1    43.0/38.8  55.5/51.5    79.9/73.7  99.3/100.4
//   512 x 512    15.4/18.5  23.9/19.1    24.6/33.9  38.6/35.2    43.8/64.7  67.7/67.2    81.4/126   123/131
//   720 x 720    20.5/19.3  35.5/29.3    30.6/35.2  55.4/52.3    50.5/63.7  95.5/96.8    93.0/120   171/178
//   1024 x 768   23.7/26.5  46.0/39.7    35.1/46.5  72.4/69.4    58.7/87.2  126/127      104/166    220/234  (192: 20.6/21.6 38.9/31.9)
// and 4096 x 4096, -0.8+0.156i / the whole set: 64 steps 107 vs 106 / 141 vs 127, 128 steps 130 vs 154 / 167 vs 188.
// Where the views disagree the regrouping kernel is preferred: its time follows the number of steps, the block kernel's also
// where in the image the long pixels lie.
static uint32_t regroup_from(uint32_t kind, uint64_t pixels) {
  constexpr uint32_t NEVER = 0xffffffffu;
  constexpr uint64_t Ki = 1024;
  if (pixels >= 4096 * Ki) return 96;
  if (kind == VRHI_ESCAPE_MANDELBROT) return pixels < 24 * Ki ? 512 : pixels < 176 * Ki ? NEVER : pixels < 240 * Ki ? 1024 : pixels < 512 * Ki ? 512 : 192;
  return pixels < 88 * Ki ? 512 : pixels < 144 * Ki ? NEVER : pixels < 288 * Ki ? 1024 : pixels < 448 * Ki ? 512 : 256;
}

int launch_escape_time(vrhi_stream_t *st, const ArgView *args, int n_args, const void *params, size_t params_size) {
  vrhi_escape_params q;
  VRHI_TRY(read_params(params, params_size, &q));
  if (n_args < 1 || n_args > 3) return fail(VRHI_ERR_INVALID, "escape_time takes the image and, optionally, a uint16 wire copy and a byte plane; got %d arguments", n_args);
  if (!writable(args[0])) return fail(VRHI_ERR_INVALID, "escape_time: the image buffer is read-only (class %s)", vrhi_arg_class_name(args[0].buf_cls));
  uint16_t *wire = nullptr;
  uint8_t *byte_plane = nullptr;
  if (n_args >= 2) {
    if (q.output != VRHI_OUT_COUNT_U32) return fail(VRHI_ERR_INVALID, "escape_time: the uint16 wire copy goes with uint32 counts only");
    if (q.max_iter > 65535u) return fail(VRHI_ERR_UNSUPPORTED, "escape_time: a uint16 wire copy needs max_iter <= 65535");
    if (!writable(args[1])) return fail(VRHI_ERR_INVALID, "escape_time: the wire buffer is read-only (class %s)", vrhi_arg_class_name(args[1].buf_cls));
    if (args[1].bytes < (uint64_t)q.width * q.height * 2) return fail(VRHI_ERR_SIZE, "escape_time: the wire view holds %llu bytes, %llu needed", (unsigned long long)args[1].bytes, (unsigned long long)q.width * q.height * 2);
    wire = reinterpret_cast<uint16_t *>(args[1].ptr);
    if (n_args == 3) {
      if (!writable(args[2])) return fail(VRHI_ERR_INVALID, "escape_time: the byte plane is read-only (class %s)", vrhi_arg_class_name(args[2].buf_cls));
      if (args[2].bytes < (uint64_t)q.width * q.height) return fail(VRHI_ERR_SIZE, "escape_time: the byte plane holds %llu bytes, %llu needed", (unsigned long long)args[2].bytes, (unsigned long long)q.width * q.height);
      byte_plane = reinterpret_cast<uint8_t *>(args[2].ptr);
    }
  }
  if (q.kind > VRHI_ESCAPE_JULIA || q.mode > VRHI_ESCAPE_FAST || q.test > VRHI_TEST_NORM_GE || q.output > VRHI_OUT_COLOR_F32)
    return fail(VRHI_ERR_INVALID, "escape_time: kind/mode/test/output out of range");
  if (q.width == 0 || q.height == 0) return fail(VRHI_ERR_SIZE, "escape_time: empty image");
  if (q.output == VRHI_OUT_COUNT_U16 && q.max_iter > 65535u) return fail(VRHI_ERR_UNSUPPORTED, "escape_time: uint16 counts need max_iter <= 65535");
  if (q.max_iter > (1u << 24) && q.output == VRHI_OUT_COLOR_F32) return fail(VRHI_ERR_UNSUPPORTED, "escape_time: colour output needs max_iter <= 2^24");
  const size_t elem = q.output == VRHI_OUT_COUNT_U16 ? 2 : 4;
  const uint64_t need = (uint64_t)q.width * q.height * elem;
  if (args[0].bytes < need) return fail(VRHI_ERR_SIZE, "escape_time: image view holds %llu bytes, %llu needed", (unsigned long long)args[0].bytes, (unsigned long long)need);

  EscapeDev p{};
  p.width = q.width; p.height = q.height; p.max_iter = q.max_iter;
  p.x0 = q.x0; p.y0 = q.y0; p.dx = q.dx; p.dy = q.dy; p.cr = q.cr; p.ci = q.ci;
  p.limit = escape_limit(q.test, q.bound); p.color_scale = q.color_scale;
  p.transposed = (q.flags & VRHI_ESCAPE_FLAG_TRANSPOSED) ? 1u : 0u;
  if (q.chunk_rows == 0) {
    p.chunk_rows = q.height; p.chunk_first = 0; p.chunk_step = 1; p.rows_owned = q.height;
  } else {
    if (q.chunk_step == 0) return fail(VRHI_ERR_INVALID, "escape_time: chunk_step must be >= 1");
    p.chunk_rows = q.chunk_rows; p.chunk_first = q.chunk_first; p.chunk_step = q.chunk_step;
    uint64_t rows = 0;
    for (uint32_t k = 0; k < q.chunk_count; ++k) {
      uint64_t c = (uint64_t)q.chunk_first + (uint64_t)k * q.chunk_step;
      uint64_t r0 = c * q.chunk_rows;
      if (r0 >= q.height) return fail(VRHI_ERR_SIZE, "escape_time: chunk %llu starts beyond the image", (unsigned long long)c);
      uint64_t r1 = r0 + q.chunk_rows;
      if (r1 > q.height) {
        if (k + 1 != q.chunk_count) return fail(VRHI_ERR_SIZE, "escape_time: only the last chunk may be short");
        r1 = q.height;
      }
      rows += r1 - r0;
    }
    p.rows_owned = (uint32_t)rows;
  }
  if (p.rows_owned == 0) return VRHI_OK;  // an empty band is not an error
  p.neg_zero = -0.0f;
  p.bytes = byte_plane;
  // tuning aids, read once per process
  static const int env_batch = [] { const char *e = getenv("VRHI_ESCAPE_BATCH"); return e ? atoi(e) : 0; }();
  static const int env_per_sm = [] { const char *e = getenv("VRHI_ESCAPE_CTAS_PER_SM"); return e ? atoi(e) : 0; }();
  const int sms = st->dev->prop.multiProcessorCount;
  // The kernels with unchecked blocks take what their exactness argument covers (EscapeDev::c2_unsafe_lo); everything
  // else, and callers that ask for it, runs the step-by-step kernel.
  const double root = sqrt((double)p.limit), cmax = fmin(p.limit - 1.005 * root, 0.5 * p.limit);
  const double c2 = (double)q.cr * q.cr + (double)q.ci * q.ci;
  p.c2_unsafe_lo = (float)(cmax * cmax * (1.0 - 1e-6));
  p.c2_unsafe_hi = 4.05f;
  const bool blocks_ok = p.limit >= 4.0f && p.limit < 3.0e38f && q.max_iter <= (1u << 30) &&
                         (q.kind == VRHI_ESCAPE_MANDELBROT || sqrt(c2) <= cmax) && !(q.flags & VRHI_ESCAPE_FLAG_CHECKED_ONLY);
  // Two kernels with unchecked blocks: the regrouping one (k_escape_pair.cu) loses nothing to pixels that outlive their
  // neighbours, the block kernel (k_escape_block.cu) is cheaper per step and has no intake (see regroup_from).
  const uint64_t pixels = (uint64_t)q.width * p.rows_owned;
  bool regroup_ok = blocks_ok && q.max_iter >= regroup_from(q.kind, pixels) && (uint64_t)q.width * q.height <= 0xffffffffull;
  // The regrouping kernel's work counter lives in the stream's scratch.  A recording cannot allocate it, so on a stream that
  // has none yet the block kernel is recorded.
  if (regroup_ok && !st->arena) {
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    VRHI_CUDA(cudaStreamIsCapturing(st->s, &cap));
    regroup_ok = cap == cudaStreamCaptureStatusNone;
  }
  // A launch declared independent of the k launches before it (flags, bits 8-10) may begin before they end.
  // Such launches form runs: the first of a run is ordered behind everything earlier on the stream, each
  // further one is started with the overlap attribute, and a run ends where a launch is no longer independent
  // of the run's first (run length > k) or anything else happens on the stream.  Launch i of a run therefore
  // only ever runs beside launches it was declared independent of.  The launches of a run take their work from
  // counters of their own; every launch leaves its counter at 0 (next_batch).
  const uint32_t independent_of = (q.flags & VRHI_ESCAPE_FLAG_INDEPENDENT_MASK) >> VRHI_ESCAPE_FLAG_INDEPENDENT_SHIFT;
  const int run = st->escape_chain;  // launches of the current run so far
  const bool overlap = independent_of != 0 && run >= 1 && (uint32_t)run <= independent_of && run < 8;
  p.ordered = overlap ? 0u : 1u;
  p.chained = overlap || chains(st) ? 1u : 0u;
  const int run_after = independent_of == 0 ? 0 : overlap ? run + 1 : 1;
  if (blocks_ok && !regroup_ok && p.rows_owned <= 1u << 31) {
    VRHI_TRY(launch_escape_block(st, q, p, args[0].ptr, wire));
    VRHI_TRY(post_launch(st, "escape_time (blocks)"));
    st->escape_chain = run_after;
    return VRHI_OK;
  }
  const bool pair = regroup_ok;               // two pixels per lane (k_escape_pair.cu)
  const uint32_t tile_px = pair ? 64u : 32u;  // pixels a warp takes in per intake trip
  p.tiles_per_row = (q.width + tile_px - 1) / tile_px;
  {
    // batch = unit of work stealing: 1536 pixels of one row for large images (with the rows visited from the
    // middle outwards the last batches are the cheapest, so large batches cost no tail; on the 16384^2 image
    // with 3 blocks per SM: 2.170 ms with 512 pixels, 2.144 with 768, 2.133 with 1024, 2.121 with 1536, 2.127
    // with 2048); small images get smaller batches so that every resident warp still sees several of them
    const uint64_t resident_warps = (uint64_t)sms * 48;
    const uint64_t tiles = (uint64_t)p.tiles_per_row * p.rows_owned;
    const uint64_t most = 1536 / tile_px;
    uint64_t bt = tiles / (resident_warps * 8);
    const uint64_t least = pair ? 1 : 2;
    p.batch_tiles = (uint32_t)(bt < least ? least : bt > most ? most : bt);
    if (env_batch >= 1 && env_batch <= 64) p.batch_tiles = (uint32_t)env_batch;
  }
  p.batches_per_row = (p.tiles_per_row + p.batch_tiles - 1) / p.batch_tiles;
  uint64_t nb = (uint64_t)p.batches_per_row * p.rows_owned;
  if (nb > 0xfffffff0ull) return fail(VRHI_ERR_UNSUPPORTED, "escape_time: image too large for 32-bit batch indices");
  p.n_batches = (uint32_t)nb;

  uint64_t warps_needed = nb;
  int grid = (int)((warps_needed + 7) / 8 < (uint64_t)sms * 8 ? (warps_needed + 7) / 8 : (uint64_t)sms * 8);
  // a small image's batches are dealt out: fetching them from the counter would be most of the work
  const bool dealt = !regroup_ok && nb <= (uint64_t)grid * 8 * 4;
  uint32_t *counter = nullptr;
  if (!dealt) {
    uint32_t *ctrl = nullptr;
    VRHI_TRY(stream_arena(st, 0, &ctrl, nullptr));
    counter = independent_of == 0 ? ctrl + CTRL_WORK0 : ctrl + CTRL_ESCAPE_RING + (overlap ? run : 0);
  }
  // a grid whose failing fetches would carry the counter past 32 bits (see next_batch) is made smaller
  const uint64_t most_grid = (0xffffffffull - nb) / 8;
  if ((uint64_t)grid > most_grid) grid = (int)most_grid;
  if (regroup_ok) {
    // Measured on B200: 3-4 CTAs of 256 threads per SM are as fast as more (the kernels are bound by
    // issue or by the binary32 pipe, not by latency); small images run faster still with 2, because
    // each warp then owns enough tiles to keep its pool busy and the drain at the end is shorter.
    uint64_t ctas = (nb + 7) / 8;
    const uint64_t px_total = (uint64_t)p.tiles_per_row * tile_px * p.rows_owned;
    // Launches of less than 64 Mi pixels are usually one of several per step (a rank's rows
    // computed group by group, frames of a sequence): with 2 blocks per SM and no pinning the blocks of the next
    // launch move in beside the draining ones (measured, four launches of 1/32 of that image each on two streams:
    // 0.39 ms against 0.45 ms with 4 pinned blocks per SM).
    // Larger launches: 3 blocks per SM, pinned (measured on the 16384^2 image with 1024-pixel batches: 2.133 ms
    // against 2.145 ms with 4; with 512-pixel batches 3, 4 and 5 gave 2.170, 2.164 and 2.165 ms).
    // Between 16 and 64 Mi pixels the third block pays on one stream while the steps are few, and always costs launches on
    // two streams.  2 blocks / 3 pinned ones, us per launch on one stream and on two: 4096 x 4096, Julia, 256 steps 142/137
    // and 123/134, 1024 steps 173/175 and 149/164; Mandelbrot, 256 steps 214/212 and 192/198, 6000 x 6000, 512 steps 560/566
    // and 508/520.
    const bool few_steps = px_total >= (16ull << 20) && q.max_iter < 512u;
    uint64_t per_sm = px_total >= (64ull << 20) || few_steps ? 3 : 2;
    if (env_per_sm >= 1 && env_per_sm <= 6) per_sm = (uint64_t)env_per_sm;
    const uint64_t cap = (uint64_t)sms * per_sm;
    grid = (int)(ctas < cap ? ctas : cap);
    if ((uint64_t)grid > most_grid) grid = (int)most_grid;
    // Small images (2 blocks per SM) are short launches, usually frames of a sequence: there the next
    // frame's blocks should move in while this frame's last ones drain (65 -> 41 us per 1080p frame
    // with two alternating streams), and a few tens of microseconds cannot go far out of balance.
    const bool pin = per_sm >= 3;
    VRHI_TRY(launch_escape_pair(st, q, p, grid, (int)per_sm, pin, args[0].ptr, counter, wire));
    VRHI_TRY(post_launch(st, "escape_time (two pixels per lane)"));
    st->escape_chain = run_after;
    return VRHI_OK;
  }
  if (q.kind == VRHI_ESCAPE_MANDELBROT) {
    if (q.mode == VRHI_ESCAPE_EXACT) launch_checked<VRHI_ESCAPE_MANDELBROT, VRHI_ESCAPE_EXACT>(q.output, grid, st->s, p, args[0].ptr, counter, wire);
    else launch_checked<VRHI_ESCAPE_MANDELBROT, VRHI_ESCAPE_FAST>(q.output, grid, st->s, p, args[0].ptr, counter, wire);
  } else {
    if (q.mode == VRHI_ESCAPE_EXACT) launch_checked<VRHI_ESCAPE_JULIA, VRHI_ESCAPE_EXACT>(q.output, grid, st->s, p, args[0].ptr, counter, wire);
    else launch_checked<VRHI_ESCAPE_JULIA, VRHI_ESCAPE_FAST>(q.output, grid, st->s, p, args[0].ptr, counter, wire);
  }
  VRHI_TRY(post_launch(st, "escape_time"));
  st->escape_chain = run_after;
  return VRHI_OK;
}

// ---------------------------------------------------------------------------------------------
// FP32 issue-rate probe: independent FFMA chains, 8 per thread, nothing else in the loop body.
// Variants (vrhi_probe_params.variant) measure what the two-pixels-per-lane kernel relies on:
//   0  scalar fma.rn.f32                       the denominator of the escape-time roofline
//   1  packed fma.rn.f32x2                     the same lane-FMA rate from half the instructions
//   2  packed, one integer add per packed fma  the integer adds issue in the gaps: same time as 1
//   3  scalar, one integer add per fma         every integer add costs an issue slot: slower than 0
template <int VARIANT>
__global__ void __launch_bounds__(256) fp32_probe_kernel(float *out, uint64_t iters, float seed, uint32_t step) {
  constexpr bool PACKED = VARIANT == 1 || VARIANT == 2, WITH_INT = VARIANT >= 2;
  float v[8], w[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) { v[i] = seed + threadIdx.x + i; w[i] = v[i] * 0.5f; }
  uint32_t x[4] = {threadIdx.x, threadIdx.x + 1u, threadIdx.x + 2u, threadIdx.x + 3u};
  const float m = 0.999f, c = 0.001f;
  for (uint64_t k = 0; k < iters; ++k) {
#pragma unroll
    for (int u = 0; u < 8; ++u) {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        if (PACKED) {
          // one instruction for the pair (v[i], w[i])
          unsigned long long p, pm, pc;
          asm("mov.b64 %0, {%1, %2};" : "=l"(p) : "f"(v[i]), "f"(w[i]));
          asm("mov.b64 %0, {%1, %1};" : "=l"(pm) : "f"(m));
          asm("mov.b64 %0, {%1, %1};" : "=l"(pc) : "f"(c));
          asm volatile("fma.rn.f32x2 %0, %0, %1, %2;" : "+l"(p) : "l"(pm), "l"(pc));
          asm("mov.b64 {%0, %1}, %2;" : "=f"(v[i]), "=f"(w[i]) : "l"(p));
        } else {
          v[i] = fmaf(v[i], m, c);
        }
        if (WITH_INT) asm volatile("add.u32 %0, %0, %1;" : "+r"(x[i & 3]) : "r"(step));
      }
    }
  }
  float r = 0.f;
#pragma unroll
  for (int i = 0; i < 8; ++i) r += v[i] + (PACKED ? w[i] : 0.f);
  if (r == 12345.678f || (x[0] ^ x[1] ^ x[2] ^ x[3]) == 0x12345u) out[0] = r;  // keeps the chains alive without memory traffic
}

int launch_fp32_probe(vrhi_stream_t *st, const ArgView *args, int n_args, const void *params, size_t params_size) {
  vrhi_probe_params q;
  VRHI_TRY(read_params(params, params_size, &q));
  if (n_args != 1 || args[0].bytes < 4 || !writable(args[0])) return fail(VRHI_ERR_INVALID, "fp32_probe takes one writable argument of at least 4 bytes");
  if (q.variant > 3) return fail(VRHI_ERR_INVALID, "fp32_probe: variant %u out of range", q.variant);
  const int sms = st->dev->prop.multiProcessorCount;
  uint64_t threads = q.threads ? q.threads : (uint64_t)sms * 2048;
  uint64_t blocks = (threads + 255) / 256;
  if (blocks == 0 || blocks > 0x7fffffffull) return fail(VRHI_ERR_SIZE, "fp32_probe: thread count out of range");
  uint64_t iters = q.ffma_per_thread / 64;  // 64 fma instructions per loop trip (128 lane-FMAs when packed)
  float *o = reinterpret_cast<float *>(args[0].ptr);
  switch (q.variant) {
    case 0: fp32_probe_kernel<0><<<(unsigned)blocks, 256, 0, st->s>>>(o, iters, 1.0f, 7u); break;
    case 1: fp32_probe_kernel<1><<<(unsigned)blocks, 256, 0, st->s>>>(o, iters, 1.0f, 7u); break;
    case 2: fp32_probe_kernel<2><<<(unsigned)blocks, 256, 0, st->s>>>(o, iters, 1.0f, 7u); break;
    default: fp32_probe_kernel<3><<<(unsigned)blocks, 256, 0, st->s>>>(o, iters, 1.0f, 7u); break;
  }
  return post_launch(st, "fp32_probe");
}

}  // namespace vrhi
