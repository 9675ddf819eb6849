// Escape-time map, block kernel: one tile of 8 x 8 pixels per warp, two pixels per lane, no work stealing (sm_100a).
//
// For launches in which the regrouping kernel (k_escape_pair.cu) has too little to regroup: few steps per pixel, or too
// few tiles per resident warp to keep its pool fed.  Loop rules as in k_escape.cu (fractal.py:11-25).
//
// All pixels of a tile start together, so a running pixel's count is the number of blocks done: a block is U updates
// without a test or a counter, then one test says whether it was valid (escape is final, see EscapeDev::c2_unsafe_lo).
// A pixel whose block failed stays on the block's first state; once none is running, or fewer than U steps are left, one
// block of U steps with the test on each finds every count.  That is 6.5 packed instructions per step and pair of
// pixels where the step-by-step kernel spends 22 on the same two.  A square tile because neighbours in both directions
// escape at like counts: the warp runs as long as its slowest pixel.
#include "escape_common.cuh"

namespace vrhi {

constexpr uint32_t kTileW = 8, kTileH = 8;

template <int KIND, int OUT, int MODE, bool WIRE, int U>
__global__ void __launch_bounds__(256) escape_block_kernel(EscapeDev p, void *image, uint16_t *wire) {
  begin_launch(p);
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t FULL = 0xffffffffu;
  const uint32_t batch = blockIdx.x * 8u + (threadIdx.x >> 5);
  if (batch < p.n_batches) {
    const uint32_t ty = batch / p.batches_per_row;
    uint32_t tx = (batch - ty * p.batches_per_row) * p.batch_tiles;
    const uint32_t tx_end = min(tx + p.batch_tiles, p.tiles_per_row);
    const uint32_t r0 = middle_out(ty, p.rows_owned / kTileH + (p.rows_owned % kTileH != 0)) * kTileH + (lane >> 3), r1 = r0 + 4u;
    const bool row0 = r0 < p.rows_owned, row1 = r1 < p.rows_owned;
    const uint32_t j0 = owned_row_to_image_row(p, r0), j1 = owned_row_to_image_row(p, r1);
    const size_t pix0 = (size_t)j0 * p.width, pix1 = (size_t)j1 * p.width;
    const f32x2 NZ = pack2(p.neg_zero, p.neg_zero), TWO = pack2(2.0f, 2.0f);
    const f32x2 Y = pack2(__fadd_rn(p.y0, __fmul_rn((float)j0, p.dy)), __fadd_rn(p.y0, __fmul_rn((float)j1, p.dy)));
    const float limit = p.limit;
    for (; tx < tx_end; ++tx) {
      const uint32_t i = tx * kTileW + (lane & 7u);
      const bool valid0 = row0 && i < p.width, valid1 = row1 && i < p.width;
      const float x = __fadd_rn(p.x0, __fmul_rn((float)i, p.dx));
      const f32x2 X = pack2(x, x);
      const f32x2 RE = p.transposed ? Y : X, IM = p.transposed ? X : Y;
      f32x2 ZR, ZI, CR, CI, A = 0, B = 0;
      bool run0 = valid0, run1 = valid1;
      bool tested_only = false;  // the tile holds a constant for which escape is not provably final
      if (KIND == VRHI_ESCAPE_MANDELBROT) {
        ZR = 0; ZI = 0; CR = RE; CI = IM;
        if (p.c2_unsafe_lo < p.c2_unsafe_hi) {
          float c0r, c1r, c0i, c1i;
          unpack2(CR, c0r, c1r);
          unpack2(CI, c0i, c1i);
          tested_only = __any_sync(FULL, unsafe_constant(p, c0r, c0i) || unsafe_constant(p, c1r, c1i));
        }
      } else {
        ZR = RE; ZI = IM; CR = pack2(p.cr, p.cr); CI = pack2(p.ci, p.ci);
      }
      uint32_t cnt0 = 0, cnt1 = 0;
      bool running = true;  // some pixel has not failed a block
      if (!tested_only) {
        pair_squares<MODE>(ZR, ZI, NZ, A, B);
        for (uint32_t steps = (uint32_t)U; steps <= p.max_iter; steps += (uint32_t)U) {
          const f32x2 CKR = ZR, CKI = ZI;
#pragma unroll
          for (int k = 0; k < U; ++k) pair_advance<MODE>(ZR, ZI, A, B, CR, CI, NZ, TWO);
          float s0, s1;
          unpack2(pair_norm2<MODE>(ZR, ZI, A, B, NZ), s0, s1);
          run0 = run0 && (s0 <= limit);
          run1 = run1 && (s1 <= limit);
          // the squares of a pixel that stopped are left wrong: nothing reads them before the tested block
          ZR = select2(run0, run1, ZR, CKR);
          ZI = select2(run0, run1, ZI, CKI);
          cnt0 = run0 ? steps : cnt0;
          cnt1 = run1 ? steps : cnt1;
          running = __any_sync(FULL, run0 || run1);
          if (!running) break;
        }
      }
      bool live0 = valid0, live1 = valid1;
      pair_squares<MODE>(ZR, ZI, NZ, A, B);
      if (!running) {  // every pixel failed a block that ends at max_iter or before: no cap to watch, and each ends in here
#pragma unroll
        for (int k = 0; k < U; ++k) {
          float s0, s1;
          unpack2(pair_norm2<MODE>(ZR, ZI, A, B, NZ), s0, s1);
          live0 = live0 && (s0 <= limit);
          live1 = live1 && (s1 <= limit);
          if (k == U - 1) break;
          pair_advance<MODE>(ZR, ZI, A, B, CR, CI, NZ, TWO);
          cnt0 += live0 ? 1u : 0u;
          cnt1 += live1 ? 1u : 0u;
        }
        cnt0 += live0 ? 1u : 0u;  // the state behind the block's last update is the one that failed
        cnt1 += live1 ? 1u : 0u;
      } else {
        do {  // one trip, except for a tile that may not take unchecked blocks
#pragma unroll
          for (int k = 0; k <= U; ++k) {  // U updates and the test of the state behind the last one
            float s0, s1;
            unpack2(pair_norm2<MODE>(ZR, ZI, A, B, NZ), s0, s1);
            live0 = live0 && (s0 <= limit) && cnt0 < p.max_iter;
            live1 = live1 && (s1 <= limit) && cnt1 < p.max_iter;
            if (k == U) break;
            pair_advance<MODE>(ZR, ZI, A, B, CR, CI, NZ, TWO);
            cnt0 += live0 ? 1u : 0u;
            cnt1 += live1 ? 1u : 0u;
          }
        } while (__any_sync(FULL, live0 || live1));
      }
      if (valid0) {
        store_count<OUT>(image, pix0 + i, cnt0, p.color_scale);
        if (WIRE) store_wire(wire, p.bytes, pix0 + i, cnt0);
      }
      if (valid1) {
        store_count<OUT>(image, pix1 + i, cnt1, p.color_scale);
        if (WIRE) store_wire(wire, p.bytes, pix1 + i, cnt1);
      }
    }
  }
  end_launch();
}

template <int KIND, int OUT, bool WIRE, int U>
static cudaError_t launch_mode(uint32_t mode, int grid, cudaStream_t s, const EscapeDev &p, void *image, uint16_t *wire) {
  if (mode == VRHI_ESCAPE_EXACT) return launch_chained(p.chained, escape_block_kernel<KIND, OUT, VRHI_ESCAPE_EXACT, WIRE, U>, dim3((unsigned)grid), 256, 0, s, p, image, wire);
  return launch_chained(p.chained, escape_block_kernel<KIND, OUT, VRHI_ESCAPE_FAST, WIRE, U>, dim3((unsigned)grid), 256, 0, s, p, image, wire);
}

template <int KIND, int U>
static cudaError_t launch_out(const vrhi_escape_params &q, int grid, cudaStream_t s, const EscapeDev &p, void *image, uint16_t *wire) {
  if (wire) return launch_mode<KIND, VRHI_OUT_COUNT_U32, true, U>(q.mode, grid, s, p, image, wire);
  switch (q.output) {
    case VRHI_OUT_COUNT_U32: return launch_mode<KIND, VRHI_OUT_COUNT_U32, false, U>(q.mode, grid, s, p, image, nullptr);
    case VRHI_OUT_COUNT_U16: return launch_mode<KIND, VRHI_OUT_COUNT_U16, false, U>(q.mode, grid, s, p, image, nullptr);
    default: return launch_mode<KIND, VRHI_OUT_COLOR_F32, false, U>(q.mode, grid, s, p, image, nullptr);
  }
}

int launch_escape_block(vrhi_stream_t *st, const vrhi_escape_params &q, EscapeDev p, void *image, uint16_t *wire) {
  p.tiles_per_row = (p.width + kTileW - 1) / kTileW;
  const uint64_t tile_rows = ((uint64_t)p.rows_owned + kTileH - 1) / kTileH, tiles = p.tiles_per_row * tile_rows;
  // Adjacent tiles of a row of tiles per warp, so that a tile's share of the row's index arithmetic is small, as long as
  // every warp place of the GPU sees eight warps (measured, 4096 x 4096 Julia of 50 steps: one tile per warp 111 us,
  // four waves of warps 93, eight 95, two 101; at 256 steps 249, 275, 253, 337).
  const uint64_t bt = tiles / ((uint64_t)st->dev->prop.multiProcessorCount * 64 * 8);
  p.batch_tiles = (uint32_t)(bt < 1 ? 1 : bt > 16 ? 16 : bt);
  p.batches_per_row = (p.tiles_per_row + p.batch_tiles - 1) / p.batch_tiles;
  const uint64_t batches = p.batches_per_row * tile_rows;
  if (batches > 0xfffffff0ull) return fail(VRHI_ERR_UNSUPPORTED, "escape_time: image too large for 32-bit batch indices");
  p.n_batches = (uint32_t)batches;
  const int grid = (int)((batches + 7) / 8);
  // Updates per block: a tile spends one tested block of that length whatever its counts, so few where few steps are
  // allowed (1080p Julia, 50 steps: 16.2 us with 4, 18.3 with 8), more where the test between blocks counts (256 steps:
  // 45.2 and 43.3 us; Mandelbrot 50.2 and 47.4).
  const bool shallow = q.max_iter < 128u;
  if (q.kind == VRHI_ESCAPE_MANDELBROT) {
    if (shallow) VRHI_CUDA((launch_out<VRHI_ESCAPE_MANDELBROT, 4>(q, grid, st->s, p, image, wire)));
    else VRHI_CUDA((launch_out<VRHI_ESCAPE_MANDELBROT, 8>(q, grid, st->s, p, image, wire)));
  } else {
    if (shallow) VRHI_CUDA((launch_out<VRHI_ESCAPE_JULIA, 4>(q, grid, st->s, p, image, wire)));
    else VRHI_CUDA((launch_out<VRHI_ESCAPE_JULIA, 8>(q, grid, st->s, p, image, wire)));
  }
  return VRHI_OK;
}

}  // namespace vrhi
