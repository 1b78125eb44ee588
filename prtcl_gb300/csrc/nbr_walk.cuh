// Device-side walk over the neighbour lists of one item (the lists of
// nhood.hpp), shared by the hand-written schemes and by schemes generated
// from the scheme language.
#pragma once

#include "nhood.hpp"

#include <type_traits>

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

// Calls use(load(j), factor, true) for the neighbours of item i, in list
// order, and use(some record, some factor, false), which must change nothing,
// up to the end of the last batch.
//
// Entries are taken kNbrHeld at a time: their offsets and factors are loaded
// together, then their records, as many at a time as FORM says.  Nothing
// branches between the entries of a batch, so that their gathers are in flight
// together and their arithmetic overlaps.  for_each_nbr, with a branch around
// every entry, computes a thread's pairs one after the other.  That suits
// sweeps whose many warps keep L1 busy (1M items, 60 to 70 % of its
// wavefronts): a lane past its row's end then loads nothing.  It does not suit
// the sweeps of small scenes, which last as long as one thread's chain of
// pairs, nor those bound by their arithmetic.  Per launch, for_each_nbr / this
// walk: 27k items density 20.7 / 12.7 us, set-up 24.7 / 14.6, acceleration
// 16.4 / 10.9, pressure 19.4 / 14.4, PCG product 23.3 / 17.0; 1M items density
// 100 / 87, set-up 233 / 193, diagonal 115 / 112, but acceleration 96 / 102,
// pressure 141 / 150, PCG product 154 / 158.
//
// FORM is the number of records gathered together and
//   kAhead: the next kNbrHeld entries are loaded before these are worked on
//     (27k items, set-up 16.6 -> 14.6 us; at 1M items the registers it takes
//     cost warps: 193 -> 221);
//   kFill: a record past the row's end is the row's first neighbour's, else
//     its load is predicated off.  Which is faster depends on the sweep's
//     registers (1M items, filled / not: diagonal 113 / 116 us, set-up 199 /
//     193);
//   kAlone: for_each_nbr (walk_nbrs_cached only).
constexpr uint32_t kAhead = 0x100, kFill = 0x200, kAlone = 0x400;
constexpr uint32_t kNbrHeld = 8;

struct NbrHeld {
  uint32_t w[4];
  float g[kNbrHeld];
};
template <bool GF, bool KEEP>
__device__ __forceinline__ void load_held(NbrHeld &H, unsigned char const *ch, uint32_t k) {
  // half a unit of offsets (its sector stays in L1 for the other half), a unit of factors
  uint32_t h = (k / kNbrHeld) % 2;
  uint4 a = __ldg(reinterpret_cast<uint4 const *>(ch) + h);
  H.w[0] = a.x;
  H.w[1] = a.y;
  H.w[2] = a.z;
  H.w[3] = a.w;
  if constexpr (GF) {
    uint32_t q[8];
    load_unit<KEEP>(ch + (1 + h) * kUnitSpan, q);
#pragma unroll
    for (int t = 0; t < 8; ++t) H.g[t] = __uint_as_float(q[t]);
  } else {
#pragma unroll
    for (int t = 0; t < 8; ++t) H.g[t] = 0.0f;
  }
}

template <uint32_t FORM, bool GF, bool KEEP = false, class Load, class Use>
__device__ __forceinline__ void walk_nbrs(NbrList const &L, uint32_t i, Load &&load, Use &&use) {
  constexpr uint32_t GATHER = FORM & 0xFFu;
  constexpr bool AHEAD = (FORM & kAhead) != 0u, FILL = (FORM & kFill) != 0u;
  static_assert(kNbrHeld % GATHER == 0 && GATHER % 2 == 0, "whole batches");
  uint2 cb = __ldg(L.cb + i);
  uint32_t c = min(cb.x & ~kWide, L.cap);
  if (c == 0) return;
  bool wide = (cb.x & kWide) != 0;
  unsigned char const *ch = L.chunks + chunk_unit(0, L.n, i, 0);
  size_t plane = chunk_plane(L.n);
  NbrHeld H, N;
  if (AHEAD) load_held<GF, KEEP>(N, ch, 0);
  for (uint32_t k = 0; k < c; k += kNbrHeld) {
    unsigned char const *next = (k / kNbrHeld) % 2 ? ch + plane : ch;
    if (AHEAD) {
      H = N;
      if (k + kNbrHeld < c) load_held<GF, KEEP>(N, next, k + kNbrHeld);
    } else {
      load_held<GF, KEEP>(H, ch, k);
    }
    ch = next;
#pragma unroll
    for (uint32_t u = 0; u < kNbrHeld; u += GATHER) {
      uint32_t j[GATHER];
      if (wide) {
        uint32_t const *w32 = L.idx32 + size_t(i) * L.cap + k + u;
#pragma unroll
        for (uint32_t t = 0; t < GATHER; ++t) j[t] = __ldcs(w32 + t);
      } else {
#pragma unroll
        for (uint32_t t = 0; t < GATHER; t += 2) {
          // signed 16-bit offsets from the row's base
          uint32_t w = H.w[(u + t) / 2];
          j[t] = cb.y + uint32_t(int32_t(int16_t(w & 0xFFFFu)));
          j[t + 1] = cb.y + uint32_t(int32_t(w) >> 16);
        }
      }
      decltype(load(0u)) r[GATHER];
#pragma unroll
      for (uint32_t t = 0; t < GATHER; ++t) {
        bool in = k + u + t < c;
        if (FILL) {
          r[t] = load(in ? j[t] : cb.y);
        } else {
          r[t] = {};
          if (in) r[t] = load(j[t]);
        }
      }
#pragma unroll
      for (uint32_t t = 0; t < GATHER; ++t) use(r[t], H.g[u + t], k + u + t < c);
    }
  }
}

// The same walk one entry at a time, without factors: use(load(j), 0, true)
template <class Load, class Use>
__device__ __forceinline__ void walk_nbrs_singly(NbrList const &L, uint32_t i, Load &&load, Use &&use) {
  uint2 cb = __ldg(L.cb + i);
  uint32_t c = min(cb.x & ~kWide, L.cap);
#pragma unroll 1
  for (uint32_t k = 0; k < c; ++k) {
    uint32_t j;
    if (cb.x & kWide) {
      j = __ldg(L.idx32 + size_t(i) * L.cap + k);
    } else {
      unsigned char const *ch = L.chunks + chunk_unit(k / kChunk, L.n, i, 0);
      j = cb.y + uint32_t(int32_t(__ldg(reinterpret_cast<int16_t const *>(ch) + k % kChunk)));
    }
    use(load(j), 0.0f, true);
  }
}

// use(record, factor, in, cached).  Where `flat` (which implies cached) by
// walk_nbrs, with the lists' factors; `cached` then comes as std::true_type.
// Else, and where the form is kAlone, by for_each_nbr, and it comes as a bool:
// whether the lists' factors hold (they do not once the smoothing scale has
// changed since the lists were built).
template <uint32_t FORM, class Load, class Use>
__device__ __forceinline__ void walk_nbrs_flat(NbrList const &L, uint32_t i, bool flat, bool cached, Load &&load,
                                               Use &&use) {
  constexpr bool kAlways = (FORM & kAlone) != 0u;
  if (!kAlways && flat)
    walk_nbrs<kAlways ? kNbrHeld : FORM, true>(
        L, i, load, [&](auto const &r, float g, bool in) { use(r, g, in, std::true_type{}); });
  else
    for_each_nbr<kAlways ? (FORM & 0xFFu) : kNbrHeld>(
        L, i, cached, [&](uint32_t j, float g) { use(load(j), g, true, cached); });
}
// The same where flat and cached are one, for the sweeps whose registers do not
// stand for_each_nbr beside the branch-free walk: the other walk takes one entry
// at a time, without the lists' factors (`cached` comes as std::false_type).
// After a change of the scale, this / for_each_nbr: 1M items set-up 352 / 415 us,
// diagonal 191 / 200, correction 272 / 324, 27k items 49 / 43, 27 / 25, 28 / 27; PCG
// with its divisions 338 / 325, but 48 scenes 36.2 / 36.4 ms throughout.
template <uint32_t FORM, bool KEEP = false, class Load, class Use>
__device__ __forceinline__ void walk_nbrs_cached(NbrList const &L, uint32_t i, bool cached, Load &&load, Use &&use) {
  if constexpr ((FORM & kAlone) != 0u) {
    walk_nbrs_flat<FORM>(L, i, cached, cached, load, use);
  } else {
    if (cached)
      walk_nbrs<FORM, true, KEEP>(L, i, load, [&](auto const &r, float g, bool in) { use(r, g, in, std::true_type{}); });
    else
      walk_nbrs_singly(L, i, load, [&](auto const &r, float g, bool in) { use(r, g, in, std::false_type{}); });
  }
}
__device__ __forceinline__ bool is_cached(bool c) { return c; }
template <bool C> __device__ __forceinline__ constexpr bool is_cached(std::bool_constant<C>) { return C; }

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
