// Shared pieces of the escape-time kernels (k_escape.cu: one pixel per lane; k_escape_pair.cu: two
// pixels per lane in packed binary32 pairs): the device-side parameter block, the step primitives
// of the two arithmetic modes, and the store helpers.  Loop rules follow fractal.py:11-25.
#pragma once

#include <cstdlib>
#include <mutex>
#include <unordered_map>

#include "vrhi_internal.h"

namespace vrhi {

struct EscapeDev {
  uint32_t width, height, max_iter;
  float x0, y0, dx, dy, cr, ci;
  float limit;               // a pixel has escaped once !(a+b <= limit), whichever test the caller asked for (escape_limit)
  // A pixel goes through blocks of updates without a test only where escape is final: once a+b > limit, every later
  // a+b is larger still (or Inf/NaN).  |z'| >= |z|^2 - |c|, so with L = limit >= 4 that holds for
  // |c| <= cmax = min(L - 1.005 sqrt(L), L / 2): each step grows |z| by half a percent at least, and the roundings
  // of a step by at most 24 units of 2^-24.  In the Mandelbrot iteration z = c after one step, so it also holds for
  // |c| >= 2.01, escaped or not: |z| >= |c| there and |z'| >= |z| (|z| - 1).  What is left are the constants with
  // c2_unsafe_lo < |c|^2 < c2_unsafe_hi (none for L >= 4.05, a ring of 0.02 around |c| = 2 for L = 4).
  float c2_unsafe_lo, c2_unsafe_hi;
  float color_scale;
  uint32_t chunk_rows, chunk_first, chunk_step;
  uint32_t rows_owned;       // rows this launch computes
  uint32_t tiles_per_row;    // ceil(width / tile), tile = 32 pixels (one per lane) or 64 (two per lane)
  uint32_t batch_tiles;      // tiles per stolen batch (a batch never straddles a row)
  uint32_t batches_per_row;
  uint32_t n_batches;
  uint32_t transposed;       // 1: the row coordinate is the real part and the column coordinate the imaginary part
  float neg_zero;            // -0.0f, set by the host: an addend the assembler cannot fold (k_escape_pair.cu)
  uint32_t ordered;          // 1: everything before the launch has to have finished when it begins (begin_launch)
  uint32_t chained;          // host: the launch carries the programmatic-serialization attribute
  uint8_t *bytes;            // optional third copy of every count, min(count, 255), at the same pixel index (nullptr: none)
};

__device__ __forceinline__ bool unsafe_constant(const EscapeDev &p, float cr, float ci) {
  const float c2 = __fmaf_rn(cr, cr, __fmul_rn(ci, ci));
  return c2 > p.c2_unsafe_lo && c2 < p.c2_unsafe_hi;
}

// Step primitives.  EXACT keeps a = zr*zr and b = zi*zi alongside z so that one update costs six
// instructions; FAST lets multiply-adds fuse (four instructions per update) and is a different,
// equally well-defined rounding sequence:
//     test  s = fma(zi, zi, zr*zr)        update  zi' = fma(zr+zr, zi, ci);  zr' = fma(zr, zr, fma(-zi, zi, cr))
template <int MODE>
__device__ __forceinline__ void z_squares(float zr, float zi, float &a, float &b) {
  if (MODE == VRHI_ESCAPE_EXACT) { a = __fmul_rn(zr, zr); b = __fmul_rn(zi, zi); }
}
template <int MODE>
__device__ __forceinline__ float z_norm2(float zr, float zi, float a, float b) {
  if (MODE == VRHI_ESCAPE_EXACT) return __fadd_rn(a, b);
  return __fmaf_rn(zi, zi, __fmul_rn(zr, zr));
}
template <int MODE>
__device__ __forceinline__ void z_advance(float &zr, float &zi, float &a, float &b, float cr, float ci) {
  if (MODE == VRHI_ESCAPE_EXACT) {
    const float t = __fmul_rn(zr, zi);
    zi = __fmaf_rn(2.0f, t, ci);
    zr = __fadd_rn(__fsub_rn(a, b), cr);
    a = __fmul_rn(zr, zr);
    b = __fmul_rn(zi, zi);
  } else {
    const float nzi = __fmaf_rn(__fadd_rn(zr, zr), zi, ci);
    zr = __fmaf_rn(zr, zr, __fmaf_rn(-zi, zi, cr));
    zi = nzi;
  }
}

// s = a+b against EscapeDev::limit.  NaN counts as escaped; s > limit otherwise.
__device__ __forceinline__ bool escaped(float s, float limit) { return !(s <= limit); }

// TWO PIXELS IN ONE REGISTER PAIR.  A packed operation rounds each half exactly like the scalar operation, so the counts
// are the same bits as the one-pixel-per-lane kernel and the CPU statement.  One trap: the
// assembler contracts mul.rn.f32x2 followed by add/sub.rn.f32x2 into a fused multiply-add (it does
// so even through fma(x, y, -0.0) with a literal -0.0), which changes the rounding of
// (zr*zr - zi*zi).  Every product here is therefore fma(x, y, nz) with nz = -0.0 read from the
// kernel parameters, a value the assembler cannot see: x*y + (-0.0) is x*y rounded once, sign of
// zero included, and an fma feeding an add is never contracted further.
typedef unsigned long long f32x2;  // two binary32 values in one 64-bit register; "lo" is slot 0

__device__ __forceinline__ f32x2 pack2(float lo, float hi) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpack2(f32x2 v, float &lo, float &hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
  f32x2 d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ f32x2 sub2(f32x2 a, f32x2 b) {
  f32x2 d;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ f32x2 neg2(f32x2 a) { return a ^ 0x8000000080000000ull; }
// lo half from `n` where c0 holds, else from `o`; hi half likewise with c1
__device__ __forceinline__ f32x2 select2(bool c0, bool c1, f32x2 n, f32x2 o) {
  float nl, nh, ol, oh;
  unpack2(n, nl, nh);
  unpack2(o, ol, oh);
  return pack2(c0 ? nl : ol, c1 ? nh : oh);
}

// The step primitives of escape_common.cuh on pairs; `nz` is the invisible -0.0 (see the top).
template <int MODE>
__device__ __forceinline__ void pair_squares(f32x2 zr, f32x2 zi, f32x2 nz, f32x2 &a, f32x2 &b) {
  if (MODE == VRHI_ESCAPE_EXACT) { a = fma2(zr, zr, nz); b = fma2(zi, zi, nz); }
}
template <int MODE>
__device__ __forceinline__ f32x2 pair_norm2(f32x2 zr, f32x2 zi, f32x2 a, f32x2 b, f32x2 nz) {
  if (MODE == VRHI_ESCAPE_EXACT) return add2(a, b);
  return fma2(zi, zi, fma2(zr, zr, nz));
}
template <int MODE>
__device__ __forceinline__ void pair_advance(f32x2 &zr, f32x2 &zi, f32x2 &a, f32x2 &b, f32x2 cr, f32x2 ci, f32x2 nz, f32x2 two) {
  if (MODE == VRHI_ESCAPE_EXACT) {
    const f32x2 t = fma2(zr, zi, nz);
    zi = fma2(two, t, ci);
    zr = add2(sub2(a, b), cr);
    a = fma2(zr, zr, nz);
    b = fma2(zi, zi, nz);
  } else {
    const f32x2 nzi = fma2(add2(zr, zr), zi, ci);
    zr = fma2(zr, zr, fma2(neg2(zi), zi, cr));
    zi = nzi;
  }
}

template <int OUT>
__device__ __forceinline__ void store_count(void *image, size_t pix, uint32_t count, float color_scale) {
  if (OUT == VRHI_OUT_COUNT_U32)
    static_cast<uint32_t *>(image)[pix] = count;
  else if (OUT == VRHI_OUT_COUNT_U16)
    static_cast<uint16_t *>(image)[pix] = (uint16_t)count;
  else
    static_cast<float *>(image)[pix] = __fsub_rn(1.0f, __fmul_rn((float)count, color_scale));
}

// Second copy of a count as uint16 at the same pixel index (the compact form a rank sends to its
// peers when the image is gathered; counts up to 65535 lose nothing).
// With `bytes` also min(count, 255) as one byte: the plane that crosses NVLink where the counts are squeezed
// (a byte of 255 tells the receiving side to fetch the uint16 count).
__device__ __forceinline__ void store_wire(uint16_t *wire, uint8_t *bytes, size_t pix, uint32_t count) {
  wire[pix] = (uint16_t)count;
  if (bytes) bytes[pix] = (uint8_t)min(count, 255u);
}

// From `count` steps done: the step-by-step loop to the end.
template <int MODE>
__device__ __forceinline__ uint32_t escape_count(float zr, float zi, float cr, float ci, float limit, uint32_t count, uint32_t max_iter) {
  float a = 0.f, b = 0.f;
  z_squares<MODE>(zr, zi, a, b);
  while (!escaped(z_norm2<MODE>(zr, zi, a, b), limit) && count < max_iter) {
    z_advance<MODE>(zr, zi, a, b, cr, ci);
    ++count;
  }
  return count;
}

// The blocks of a launch that carries the programmatic-serialization attribute (EscapeDev::chained) may become resident
// as soon as every block of the launch before it has executed launch_dependents.  An ordinary launch waits in
// begin_launch() until everything before it has finished, and only then lets the next one come.  A launch that its caller
// declared independent of the launches before it does not wait there and runs beside them; every block ends with
// end_launch(), so its grid cannot complete before the grid before it has, and whatever follows on the stream still
// finds everything earlier finished.  (Were the next launch let in before the wait, one that is independent of this
// launch, but not of what came before it, could start too early.)  All of it is a no-op without the attribute.
__device__ __forceinline__ void begin_launch(const EscapeDev &p) {
  if (p.ordered) asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;");
}
__device__ __forceinline__ void end_launch() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Work stealing: the next batch for this warp, n_batches or more when none is left.  A launch makes exactly n_batches
// fetches that succeed and one that fails per warp, so the wrapping increment leaves the counter at 0 behind the
// last one and the next launch needs no memset in front of it (a node of its own in a recorded sequence, and the
// gap before the kernel: measured on B200, a 1080p Mandelbrot frame of 256 steps, 52.8 us with, 50.0 us without).
// The host keeps n_batches + warps within 32 bits.
__device__ __forceinline__ uint32_t next_batch(uint32_t *counter, uint32_t n_batches) {
  return atomicInc(counter, n_batches + gridDim.x * (blockDim.x >> 5) - 1u);
}

// Order in which a launch visits its rows: from the middle outwards (k = 0 is the middle row).  The
// expensive rows of these images lie around the middle and hold the pixels that run for thousands
// of steps; a pixel started late is a tail nothing else covers (one warp, one dependent chain, tens
// of microseconds), so those rows go first and the cheap outer rows, whose pixels end within a few
// steps, go last.
__device__ __forceinline__ uint32_t middle_out(uint32_t k, uint32_t rows) {
  const uint32_t mid = rows >> 1, h = (k + 1u) >> 1;
  // k odd: rows below the middle (mid-1, mid-2, ...); k even: the middle and above; past the shorter side the rest follows in order
  if (k & 1u) return h <= mid ? mid - h : k;
  return mid + h < rows ? mid + h : rows - 1u - k;
}

// Row of the image that owned row r maps to (rows are owned in chunks dealt round-robin).
__device__ __forceinline__ uint32_t owned_row_to_image_row(const EscapeDev &p, uint32_t r) {
  uint32_t k = r / p.chunk_rows;
  return (p.chunk_first + k * p.chunk_step) * p.chunk_rows + (r - k * p.chunk_rows);
}

// Launch of a work-stealing escape-time kernel with its residency pinned.  Such a kernel is a
// persistent grid of `per_sm` blocks per SM; that only balances if the blocks really sit per_sm to
// an SM.  On an idle GPU they do, but when blocks of another stream's kernel are resident at launch
// time the hardware packs the grid onto whichever SMs have room, and the SMs that got more than
// their share then finish late (measured: 3.7 ms instead of 2.5 ms for the 16384^2 image).  Unused
// dynamic shared memory sized so that exactly per_sm blocks fit makes the surplus blocks wait for
// their own SM instead.  `pin` false launches without the padding.
// The opt-in limit of a kernel is only ever raised, under the lock and per device, so concurrent
// launches from several host threads never see a limit below what they ask for.
template <class Kern>
int launch_pinned(Kern kern, int grid, int per_sm, vrhi_stream_t *st, const EscapeDev &p, void *image, uint32_t *counter,
                  uint16_t *wire, bool pin = true) {
  struct Entry { size_t fixed; size_t limit; };
  static std::mutex mu;
  static std::unordered_map<uint64_t, Entry> cache;  // key: kernel address mixed with the device ordinal
  static const int pin_env = [] { const char *e = getenv("VRHI_ESCAPE_PIN"); return e ? atoi(e) : 1; }();  // tuning aid: 0 = no padding
  const uint64_t key = (uint64_t)reinterpret_cast<uintptr_t>(reinterpret_cast<const void *>(kern)) * 64u + (uint64_t)st->dev->ordinal;
  size_t dyn = 0;
  {
    std::lock_guard<std::mutex> lock(mu);
    auto it = cache.find(key);
    if (it == cache.end()) {
      cudaFuncAttributes fa{};
      VRHI_CUDA(cudaFuncGetAttributes(&fa, kern));
      it = cache.emplace(key, Entry{fa.sharedSizeBytes, 0}).first;
    }
    if (pin && pin_env != 0 && per_sm >= 1) {
      const size_t per_sm_bytes = st->dev->prop.sharedMemPerMultiprocessor;  // each resident block also reserves 1 KB
      size_t total = ((size_t)((double)per_sm_bytes / (per_sm + 0.5)) - 1024) & ~size_t(127);
      const size_t optin = st->dev->prop.sharedMemPerBlockOptin;
      if (total > optin) total = optin;
      dyn = total > it->second.fixed ? total - it->second.fixed : 0;
    }
    if (dyn > it->second.limit) {
      VRHI_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn));
      it->second.limit = dyn;
    }
  }
  VRHI_CUDA(launch_chained(p.chained, kern, dim3((unsigned)grid), 256, dyn, st->s, p, image, counter, wire));
  return VRHI_OK;
}

// the regrouping kernel (k_escape_pair.cu); it needs max_iter >= 12, the length of its blocks and of its intake
int launch_escape_pair(vrhi_stream_t *st, const vrhi_escape_params &q, const EscapeDev &p, int grid, int per_sm, bool pin,
                       void *image, uint32_t *counter, uint16_t *wire);

// the kernel for launches with little to regroup (k_escape_block.cu)
int launch_escape_block(vrhi_stream_t *st, const vrhi_escape_params &q, EscapeDev p, void *image, uint16_t *wire);

}  // namespace vrhi
