// NCHW <-> [n][ceil(c/CB)][h][w][CB] for 1-, 2- and 4-byte elements and CB = 4 or 16: one kernel per direction
// for every image size, odd ones included.
//
// What bounds it: HBM.  The work of one image's channel block ("unit": CB channels x h*w pixels) is a transpose of a
// contiguous run of the NCHW tensor into a contiguous run of the blocked one, and consecutive units are consecutive
// runs on both sides.  A thread block takes about 16 KB of it: whole units where they are small, a span of pixels of
// one unit (CB rows) where they are large.  Both sides of global memory are touched in aligned 16-byte vectors
// (cp.async in, vector stores out) whatever the row length; the transpose itself happens on elements in shared memory,
// with consecutive lanes on consecutive pixels, so an odd row pitch costs no bank conflicts.  Eight blocks per SM keep
// some 128 KB per SM in flight.
// Measured with L2 flushed, us (before -> now): fp16 (64, 256, 35, 35) to blocks 114 -> 20.5, back 95 -> 24.4 (80 MB of
// traffic each: 12.3 us at the copy rate); u8 56 -> 14.3 and 93 -> 16.3; u8 (64, 3, 299, 299) 42 -> 15 and 83 -> 21;
// int32 (64, 256, 56, 56), 411 MB, 69 -> 67.6.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "igemm_sm100.cuh"  // FastDiv, cp_async16

namespace unit {

constexpr int kLayoutThreads = 256;
constexpr int kLayoutTileBytes = 16384;

struct LayoutParams {
  const uint8_t *src;
  uint8_t *dst;
  long long src_bytes, dst_bytes;  // whole tensors
  int units;                       // n * channel blocks
  int c, cc;                       // channels, channel blocks per image
  long long hw;                    // pixels
  int group;                       // > 0: units per tile; 0: tiles are spans of one unit
  int span, spans;                 // pixels per span (a multiple of 16), spans per unit
  FastDiv div_cc, div_hw, div_spans;
};

// Byte offset of unit u in the NCHW tensor, and how many of its channels exist.
template <int EB, int CB>
__device__ __forceinline__ long long nchw_offset(const LayoutParams &p, int u, int &channels) {
  const int img = (int)fast_div((uint32_t)u, p.div_cc);
  const int chunk = u - img * p.cc;
  channels = min(CB, p.c - chunk * CB);
  return ((long long)img * p.c + (long long)chunk * CB) * p.hw * EB;
}

// Copies global bytes [from, from + bytes) into shared memory, keeping their position modulo 16: byte `from` lands at
// smem + (from & 15).  Vectors that reach outside [lo, hi) (the tensor) are copied byte by byte.
__device__ __forceinline__ void load_run(uint32_t smem, uint8_t *smem_ptr, uintptr_t from, long long bytes, uintptr_t lo, uintptr_t hi,
                                         int first, int step) {
  const uintptr_t base = from & ~(uintptr_t)15;
  const int vectors = (int)((from + (uintptr_t)bytes - base + 15) >> 4);
  for (int i = first; i < vectors; i += step) {
    const uintptr_t at = base + (uintptr_t)i * 16;
    if (at >= lo && at + 16 <= hi) {
      cp_async16(smem + (uint32_t)i * 16u, reinterpret_cast<const void *>(at), 16u);
    } else {
      for (int b = 0; b < 16; ++b)
        if (at + b >= lo && at + b < hi) smem_ptr[i * 16 + b] = *reinterpret_cast<const uint8_t *>(at + b);
    }
  }
}
// The inverse: shared bytes at smem + (to & 15) go to global [to, to + bytes), whole vectors where they fit.
__device__ __forceinline__ void store_run(const uint8_t *smem, uintptr_t to, long long bytes, int first, int step) {
  const uintptr_t base = to & ~(uintptr_t)15, end = to + (uintptr_t)bytes;
  const int vectors = (int)((end - base + 15) >> 4);
  for (int i = first; i < vectors; i += step) {
    const uintptr_t at = base + (uintptr_t)i * 16;
    if (at >= to && at + 16 <= end) {
      *reinterpret_cast<uint4 *>(at) = *reinterpret_cast<const uint4 *>(smem + i * 16);
    } else {
      for (int b = 0; b < 16; ++b)
        if (at + b >= to && at + b < end) *reinterpret_cast<uint8_t *>(at + b) = smem[i * 16 + b];
    }
  }
}

template <int EB> struct ElementOf;
template <> struct ElementOf<1> { using T = uint8_t; };
template <> struct ElementOf<2> { using T = uint16_t; };
template <> struct ElementOf<4> { using T = uint32_t; };

// A tile: units [u0, u0 + nu), pixels [px0, px0 + npx) of each (all of them when group > 0).
struct LayoutTile {
  int u0, nu;
  long long px0;
  int npx;
};
__device__ __forceinline__ LayoutTile layout_tile(const LayoutParams &p) {
  LayoutTile t;
  if (p.group > 0) {
    t.u0 = (int)blockIdx.x * p.group;
    t.nu = min(p.group, p.units - t.u0);
    t.px0 = 0;
    t.npx = (int)p.hw;
  } else {
    t.u0 = (int)fast_div(blockIdx.x, p.div_spans);
    t.nu = 1;
    t.px0 = (long long)((int)blockIdx.x - t.u0 * p.spans) * p.span;
    t.npx = (int)min((long long)p.span, p.hw - t.px0);
  }
  return t;
}

// Vectors of the blocked side: a pixel is CB * EB bytes, moved 16 bytes at a time (4 or 8 where a pixel is smaller).
template <int EB, int CB>
struct Blocked {
  static constexpr int kPixel = CB * EB;
  static constexpr int kVec = kPixel < 16 ? kPixel : 16;
  static constexpr int kParts = kPixel / kVec;   // vectors per pixel
  static constexpr int kElems = kVec / EB;       // elements per vector
};

// Where a thread finds its elements among the staged rows.  Element (channel k, pixel px) of a unit lies at
// row(k) + px * EB: whole units keep their rows one behind the other; a span's row k starts at k * pitch plus its own
// position modulo 16 in global memory.  A thread meets the same channels in every vector (the block's threads are a
// multiple of the parts of a pixel), so its row offsets are worked out once: the inner loop is one addition and one
// access per element, which matters because the element work, not memory, is what bounds 1- and 2-byte elements.
template <int EB, int CB>
struct StagedRows {
  uint32_t row[Blocked<EB, CB>::kElems];
  __device__ __forceinline__ void init(const LayoutParams &p, uint32_t first, uint32_t span_first, int part) {
    const uint32_t row_bytes = (uint32_t)p.hw * EB, pitch = (uint32_t)p.span * EB + 16u;
#pragma unroll
    for (int e = 0; e < Blocked<EB, CB>::kElems; ++e) {
      const uint32_t k = (uint32_t)(part * Blocked<EB, CB>::kElems + e);
      row[e] = p.group > 0 ? first + k * row_bytes : k * pitch + ((span_first + k * row_bytes) & 15u);
    }
  }
};
// Pixel q of the tile: its offset into the staged rows, and how many channels its unit has.
template <int EB, int CB>
__device__ __forceinline__ uint32_t staged_pixel(const LayoutParams &p, const LayoutTile &t, long long off0, int q, int &ch) {
  if (p.group <= 1) return (uint32_t)q * EB;
  const int ul = (int)fast_div((uint32_t)q, p.div_hw), px = q - ul * (int)p.hw;
  return (uint32_t)(nchw_offset<EB, CB>(p, t.u0 + ul, ch) - off0) + (uint32_t)px * EB;
}

template <int EB, int CB>
__global__ void __launch_bounds__(kLayoutThreads) nchw_to_nchwc_kernel(const LayoutParams p) {
  using T = typename ElementOf<EB>::T;
  using B = Blocked<EB, CB>;
  extern __shared__ __align__(16) uint8_t layout_smem[];
  const LayoutTile t = layout_tile(p);
  const uintptr_t src = reinterpret_cast<uintptr_t>(p.src), hi = src + (uintptr_t)p.src_bytes;
  const uint32_t smem = smem_u32(layout_smem);
  int channels;
  const long long off0 = nchw_offset<EB, CB>(p, t.u0, channels);
  const uint32_t pitch = (uint32_t)p.span * EB + 16u;  // spans: bytes between the staged rows
  if (p.group > 0) {
    int dummy;
    const long long off1 = t.u0 + t.nu < p.units ? nchw_offset<EB, CB>(p, t.u0 + t.nu, dummy) : p.src_bytes;
    load_run(smem, layout_smem, src + (uintptr_t)off0, off1 - off0, src, hi, threadIdx.x, kLayoutThreads);
  } else {
    // sixteen (or four) rows at once: 16 threads per row
    const int lanes = kLayoutThreads / CB, k = (int)threadIdx.x / lanes;
    if (k < channels)
      load_run(smem + (uint32_t)k * pitch, layout_smem + k * pitch, src + (uintptr_t)(off0 + (k * p.hw + t.px0) * EB),
               (long long)t.npx * EB, src, hi, (int)threadIdx.x % lanes, lanes);
  }
  cp_async_commit();
  cp_async_wait<0>();
  __syncthreads();
  uint8_t *to = p.dst + ((long long)t.u0 * p.hw + t.px0) * B::kPixel;
  const bool whole = (reinterpret_cast<uintptr_t>(p.dst) & (B::kVec - 1)) == 0;  // (always so for tensors of an allocator)
  const int count = t.nu * t.npx * B::kParts;
  StagedRows<EB, CB> at;
  at.init(p, (uint32_t)(src + (uintptr_t)off0) & 15u, (uint32_t)(src + (uintptr_t)(off0 + t.px0 * EB)) & 15u, threadIdx.x % B::kParts);
  for (int v = threadIdx.x; v < count; v += kLayoutThreads) {
    const int part = v % B::kParts, q = v / B::kParts;
    int ch = channels;
    const uint32_t px = staged_pixel<EB, CB>(p, t, off0, q, ch);
    uint32_t w[4] = {0u, 0u, 0u, 0u};
    if (ch == CB) {
#pragma unroll
      for (int e = 0; e < B::kElems; ++e)
        w[e * EB / 4] |= (uint32_t)*reinterpret_cast<const T *>(layout_smem + (at.row[e] + px)) << (8 * (e * EB % 4));
    } else {
#pragma unroll
      for (int e = 0; e < B::kElems; ++e)
        if (part * B::kElems + e < ch)
          w[e * EB / 4] |= (uint32_t)*reinterpret_cast<const T *>(layout_smem + (at.row[e] + px)) << (8 * (e * EB % 4));
    }
    uint8_t *d = to + (long long)v * B::kVec;
    if (whole) {
      if constexpr (B::kVec == 16) *reinterpret_cast<uint4 *>(d) = make_uint4(w[0], w[1], w[2], w[3]);
      else if constexpr (B::kVec == 8) *reinterpret_cast<uint2 *>(d) = make_uint2(w[0], w[1]);
      else *reinterpret_cast<uint32_t *>(d) = w[0];
    } else {
      for (int b = 0; b < B::kVec; ++b) d[b] = (uint8_t)(w[b >> 2] >> (8 * (b & 3)));
    }
  }
}

template <int EB, int CB>
__global__ void __launch_bounds__(kLayoutThreads) nchwc_to_nchw_kernel(const LayoutParams p) {
  using T = typename ElementOf<EB>::T;
  using B = Blocked<EB, CB>;
  extern __shared__ __align__(16) uint8_t rows[];
  const LayoutTile t = layout_tile(p);
  const uint32_t pitch = (uint32_t)p.span * EB + 16u;
  const uint8_t *from = p.src + ((long long)t.u0 * p.hw + t.px0) * B::kPixel;
  const uintptr_t dst = reinterpret_cast<uintptr_t>(p.dst);
  int channels;
  const long long off0 = nchw_offset<EB, CB>(p, t.u0, channels);
  const bool whole = (reinterpret_cast<uintptr_t>(p.src) & (B::kVec - 1)) == 0;
  const int count = t.nu * t.npx * B::kParts;
  StagedRows<EB, CB> at;
  at.init(p, (uint32_t)(dst + (uintptr_t)off0) & 15u, (uint32_t)(dst + (uintptr_t)(off0 + t.px0 * EB)) & 15u, threadIdx.x % B::kParts);
  // consecutive lanes read consecutive vectors of the blocked tensor, four of them per thread in flight, and
  // scatter their elements over the staged rows
  constexpr int kFlight = 4;
  for (int v0 = threadIdx.x; v0 < count; v0 += kFlight * kLayoutThreads) {
    uint32_t w[kFlight][4];
#pragma unroll
    for (int i = 0; i < kFlight; ++i) {
      const int v = v0 + i * kLayoutThreads;
      w[i][0] = w[i][1] = w[i][2] = w[i][3] = 0u;
      if (v >= count) continue;
      const uint8_t *s = from + (long long)v * B::kVec;
      if (whole) {
        if constexpr (B::kVec == 16) {
          const uint4 x = __ldg(reinterpret_cast<const uint4 *>(s));
          w[i][0] = x.x; w[i][1] = x.y; w[i][2] = x.z; w[i][3] = x.w;
        } else if constexpr (B::kVec == 8) {
          const uint2 x = __ldg(reinterpret_cast<const uint2 *>(s));
          w[i][0] = x.x; w[i][1] = x.y;
        } else {
          w[i][0] = __ldg(reinterpret_cast<const uint32_t *>(s));
        }
      } else {
#pragma unroll
        for (int b = 0; b < B::kVec; ++b) w[i][b >> 2] |= (uint32_t)s[b] << (8 * (b & 3));
      }
    }
#pragma unroll
    for (int i = 0; i < kFlight; ++i) {
      const int v = v0 + i * kLayoutThreads;
      if (v >= count) continue;
      const int part = v % B::kParts, q = v / B::kParts;
      int ch = channels;
      const uint32_t px = staged_pixel<EB, CB>(p, t, off0, q, ch);
      if (ch == CB) {
#pragma unroll
        for (int e = 0; e < B::kElems; ++e)
          *reinterpret_cast<T *>(rows + (at.row[e] + px)) = (T)(w[i][e * EB / 4] >> (8 * (e * EB % 4)));
      } else {
#pragma unroll
        for (int e = 0; e < B::kElems; ++e)
          if (part * B::kElems + e < ch) *reinterpret_cast<T *>(rows + (at.row[e] + px)) = (T)(w[i][e * EB / 4] >> (8 * (e * EB % 4)));
      }
    }
  }
  __syncthreads();
  if (p.group > 0) {
    int dummy;
    const long long off1 = t.u0 + t.nu < p.units ? nchw_offset<EB, CB>(p, t.u0 + t.nu, dummy) : p.dst_bytes;
    store_run(rows, dst + (uintptr_t)off0, off1 - off0, threadIdx.x, kLayoutThreads);
  } else {
    const int lanes = kLayoutThreads / CB, k = (int)threadIdx.x / lanes;
    if (k < channels)
      store_run(rows + k * pitch, dst + (uintptr_t)(off0 + (k * p.hw + t.px0) * EB), (long long)t.npx * EB,
                (int)threadIdx.x % lanes, lanes);
  }
}

// The blocked -> NCHW direction where the rows are whole 4-byte words (hw * EB a multiple of 4): a thread owns one word
// position (P = 4 / EB pixels) of one unit.  Its P pixels are 4 CB contiguous bytes on the blocked side (CB / 4
// 16-byte reads), its result one word per channel, and consecutive lanes write consecutive words of a row (128 bytes a
// warp instruction), so nothing goes through shared memory.  u8 (64, 256, 56, 56) 23 us against 30 through the staged
// rows, fp16 38 against 45, u8 (64, 3, 224, 224) with CB = 4 13.2 against 14.7; fp16 and 32-bit elements with CB = 4 are faster
// through the staged rows (16.4 against 17.3, 20.6 against 25.6 on that shape).
template <int EB, int CB>
__global__ void __launch_bounds__(kLayoutThreads) nchwc_to_nchw_words_kernel(const LayoutParams p, long long words) {
  const uint32_t *src = reinterpret_cast<const uint32_t *>(p.src);
  uint32_t *dst = reinterpret_cast<uint32_t *>(p.dst);
  const long long total = (long long)p.units * words;
  for (long long idx = blockIdx.x * (long long)kLayoutThreads + threadIdx.x; idx < total; idx += (long long)gridDim.x * kLayoutThreads) {
    const int u = (int)(idx / words);
    const long long wpos = idx - (long long)u * words;
    int channels;
    const long long row = nchw_offset<EB, CB>(p, u, channels) / 4 + wpos;
    uint32_t in[CB];
    const uint4 *s4 = reinterpret_cast<const uint4 *>(src + idx * CB);
#pragma unroll
    for (int q = 0; q < CB / 4; ++q) {
      const uint4 v = __ldg(s4 + q);
      in[4 * q] = v.x; in[4 * q + 1] = v.y; in[4 * q + 2] = v.z; in[4 * q + 3] = v.w;
    }
    // in: pixel-major words; out word k = the P pixels of channel k
#pragma unroll
    for (int k = 0; k < CB; ++k) {
      uint32_t out;
      if constexpr (EB == 4) {
        out = in[k];
      } else if constexpr (EB == 2) {
        out = __byte_perm(in[k / 2], in[CB / 2 + k / 2], (k & 1) ? 0x7632 : 0x5410);
      } else {
        const uint32_t sel = (uint32_t)((4 + (k & 3)) << 4 | (k & 3));
        out = __byte_perm(__byte_perm(in[k / 4], in[CB / 4 + k / 4], sel), __byte_perm(in[CB / 2 + k / 4], in[3 * CB / 4 + k / 4], sel), 0x5410);
      }
      if (k < channels) dst[row + k * words] = out;
    }
  }
}

}  // namespace unit
