// Device-side walk over the neighbour lists of one item (the lists of
// nhood.hpp), shared by the hand-written schemes and by schemes generated
// from the scheme language.
#pragma once

#include "nhood.hpp"

namespace prtcl_gpu {

// neighbour entries a sweep thread holds at a time (16 or 8) where the sweep
// does not choose
constexpr uint32_t kNbrBatchDefault = 16;

struct NbrList {
  unsigned char const *chunks; // units of 96-byte chunks (16 offsets + 16 factors), at chunk_unit(c, n, i, u)
  uint32_t const *idx32;       // [i * cap + k]: j (read for wide items only)
  uint2 const *cb;             // per item: (count | kWide, base)
  uint32_t cap;                // row length in entries, a multiple of 16
  uint32_t n;                  // rows
};

// One unit (32 bytes, 32-byte aligned) in one 256-bit load: streaming
// (neither kept in L1 nor, for long, in L2: the lists are read once per
// sweep, the gathered particle records should stay in both), or cached where
// the row is walked again right after.
template <bool KEEP> __device__ __forceinline__ void load_unit(unsigned char const *p, uint32_t (&w)[8]) {
  if (KEEP)
    asm("ld.global.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]), "=r"(w[4]), "=r"(w[5]), "=r"(w[6]), "=r"(w[7])
                 : "l"(p));
  else
    asm("ld.global.L1::no_allocate.L2::evict_first.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]), "=r"(w[4]), "=r"(w[5]), "=r"(w[6]), "=r"(w[7])
                 : "l"(p));
}

// Calls f(j, factor) for the neighbours of item i, in list order.  Entries
// are taken kNbrBatch at a time (16: a whole chunk; 8: half a chunk, fewer
// registers held per thread), so that as many gathers can be in flight
// together.  Measured per sweep on the 1M dam break (see the shape lists in
// schemes.cu).  KEEP: the row's units stay cached.
template <uint32_t kNbrBatch = kNbrBatchDefault, bool KEEP = false, class F>
__device__ __forceinline__ void for_each_nbr(NbrList const &L, uint32_t i, bool with_gf, F &&f) {
  uint2 cb = __ldg(L.cb + i);
  uint32_t c = min(cb.x & ~kWide, L.cap);
  bool wide = (cb.x & kWide) != 0;
  unsigned char const *ch = L.chunks + chunk_unit(0, L.n, i, 0);
  size_t plane = chunk_plane(L.n);
  constexpr int kHalves = int(kChunk / kNbrBatch), kUnits = int(kNbrBatch / 8);
  for (uint32_t k0 = 0; k0 < c; k0 += kChunk, ch += plane) {
#pragma unroll
    for (int h = 0; h < kHalves; ++h) {
      uint32_t kb = k0 + uint32_t(h) * kNbrBatch;
      if (h > 0 && kb >= c) break;
      uint32_t j[kNbrBatch];
      if (wide) {
        uint4 const *w32 = reinterpret_cast<uint4 const *>(L.idx32 + size_t(i) * L.cap + kb);
#pragma unroll
        for (int v = 0; v < int(kNbrBatch / 4); ++v) {
          uint4 a = __ldcs(w32 + v);
          j[4 * v] = a.x;
          j[4 * v + 1] = a.y;
          j[4 * v + 2] = a.z;
          j[4 * v + 3] = a.w;
        }
      } else {
        uint32_t w[8];
        if (kHalves == 1) {
          load_unit<KEEP>(ch, w);
        } else {
          // half a unit; its sector stays in L1 for the other half
          uint4 a = __ldg(reinterpret_cast<uint4 const *>(ch) + h);
          w[0] = a.x;
          w[1] = a.y;
          w[2] = a.z;
          w[3] = a.w;
        }
#pragma unroll
        for (int t = 0; t < int(kNbrBatch / 2); ++t) {
          // signed 16-bit offsets from the row's base
          j[2 * t] = cb.y + uint32_t(int32_t(int16_t(w[t] & 0xFFFFu)));
          j[2 * t + 1] = cb.y + uint32_t(int32_t(w[t]) >> 16);
        }
      }
      float g[kNbrBatch];
      if (with_gf) {
#pragma unroll
        for (int u = 0; u < kUnits; ++u) {
          uint32_t q[8];
          load_unit<KEEP>(ch + (1 + h * kUnits + u) * int(kUnitSpan), q);
#pragma unroll
          for (int t = 0; t < 8; ++t) g[8 * u + t] = __uint_as_float(q[t]);
        }
      } else {
#pragma unroll
        for (int t = 0; t < int(kNbrBatch); ++t) g[t] = 0.0f;
      }
#pragma unroll
      for (int t = 0; t < int(kNbrBatch); ++t)
        if (kb + t < c) f(j[t], g[t]);
    }
  }
}

// Calls f(slot, factor) for the neighbours of item i, in list order, from
// staged lists (nhood.hpp): slot is the neighbour's place among the staged
// items of the item's tile, which the caller has copied to shared memory.
// The slots of chunk c of item i are the 16 halves at (c * n + i) * 16 of
// `slots`; the factors are those of the chunks.
template <uint32_t kNbrBatch = kNbrBatchDefault, class F>
__device__ __forceinline__ void for_each_staged(NbrList const &L, uint16_t const *slots, uint32_t i, F &&f) {
  uint2 cb = __ldg(L.cb + i);
  uint32_t c = min(cb.x & ~kWide, L.cap);
  for (uint32_t kb = 0; kb < c; kb += kNbrBatch) {
    uint32_t h = (kb % kChunk) / kNbrBatch;
    unsigned char const *ch = L.chunks + chunk_unit(kb / kChunk, L.n, i, 1 + h * (kNbrBatch / 8));
    uint4 const *sp = reinterpret_cast<uint4 const *>(slots + (size_t(kb / kChunk) * L.n + i) * kChunk);
    uint32_t sl[kNbrBatch];
#pragma unroll
    for (int v = 0; v < int(kNbrBatch / 8); ++v) {
      uint4 a = __ldcs(sp + h * (kNbrBatch / 8) + v);
      uint32_t w[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        sl[8 * v + 2 * t] = w[t] & 0xFFFFu;
        sl[8 * v + 2 * t + 1] = w[t] >> 16;
      }
    }
    float g[kNbrBatch];
#pragma unroll
    for (int u = 0; u < int(kNbrBatch / 8); ++u) {
      uint32_t q[8];
      load_unit<false>(ch + u * int(kUnitSpan), q);
#pragma unroll
      for (int t = 0; t < 8; ++t) g[8 * u + t] = __uint_as_float(q[t]);
    }
#pragma unroll
    for (int t = 0; t < int(kNbrBatch); ++t)
      if (kb + t < c) f(sl[t], g[t]);
  }
}

} // namespace prtcl_gpu
