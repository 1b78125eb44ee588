// Device implementations of the generated prtcl procedures on the hot path.
//
// Every procedure is one thread per particle: the thread walks its fluid
// neighbour list(s) and then its boundary neighbour list(s) sequentially, in
// the grid's traversal order, accumulating in FP32 in exactly the operation
// order of the generated C++ (the file:line cited at each kernel).  With FMA
// contraction off this reproduces the reference arithmetic per particle.
//
// Neighbour data is gathered from packed 16-byte records (position + mass,
// position + volume, position + m/rho) and the kernel gradient of a pair is
// rebuilt from the factor cached in the neighbour list; both hold values
// computed with the same operations as the on-the-fly expressions, so the
// results stay bit-identical (kernels fall back to the full kernel-gradient
// evaluation if the smoothing scale changed after the lists were built).
//
// Reductions that decide convergence (IISPH density error, PCG dot products)
// are FP64 with a fixed, batch-independent order: per-block tree sums, then
// the last block of the launch sums the block partials.  The relaxed-Jacobi
// loop (iisph.solve_pressure) and the PCG loop run on the device as CUDA
// graphs with a conditional while node: no host round trip per iteration.
#include "mat3.cuh"
#include "nbr_walk.cuh"
#include "schemes.hpp"

#include <algorithm>
#include <cstring>
#include <tuple>

namespace prtcl_gpu {

// kernels executed by device-side loops (graph bodies); read by the host
// through launch_count()
__device__ unsigned long long g_loop_kernels = 0;

namespace {

constexpr int kNT = 128;            // threads per block for particle kernels
// resident blocks per SM the neighbour sweeps are compiled for (caps their
// registers at 64): the sweeps wait on gathers, and more resident warps hide
// more of that latency
constexpr int kMinBlocks = 8;
constexpr int kMaxRedBlocks = 4096; // block partials per reduced value

// model scratch layout
constexpr int kSPcg = 0;     // scalars[0..7]: PCG
constexpr int kSJacobi = 16; // scalars[16]: FP64 density error
constexpr int kStPcgIter = 0, kStPcgActive = 1, kStPcgBody = 2;
constexpr int kStJacIter = 4, kStJacDone = 5;
// The relaxed-Jacobi loop starts from the pressure that setup has just set to
// zero, so its first iteration needs no neighbours: with p = 0 every term of
// the pressure acceleration is a zero, hence a = +0, hence every term of
// iteration_pressure's sum is a zero, hence the sum is +0 (sums that start at
// +0 and add or subtract zeros of either sign stay +0).  That holds while all
// masses, volumes, densities and kernel gradients of the pairs, and the products
// of rest density and volume, are finite; setup's helper sum c walks the same
// pairs with the same factors, and is not finite where one of them is not (every
// item in the grid is its own neighbour, so its own mass and density count too),
// nor is its diagonal sum where one of the products is not.  Setup notes what it
// found (kStSetupBad, and in scalars[kSSetup..] the smoothing scale and rest
// densities it used), the host checks that no field, list or pressure has
// changed since, and k_jacobi_begin (k_jacobi_loop) takes them where both agree.  Of
// the 4 to 5 iterations a step takes, this takes out one pair of sweeps (95 +
// 138 us at 1M items; 11 us are left of them): set-up and solve of the 1M dam
// break 1.54 -> 1.31 ms, of the 27k one 222 -> 204 us.
constexpr int kStJacFirst = 6, kStSetupBad = 7; // kStSetupBad: 0 after a clean setup, until a solve takes it
constexpr int kSSetup = 32; // scalars[32]: smoothing scale, then one rest density per fluid group

// ---------------------------------------------------------------------------
// argument structs
// ---------------------------------------------------------------------------

// the pair's kernel gradient: from the cached factor (bit-identical to
// kgradW) when the lists were built with the current smoothing scale
__device__ __forceinline__ f3 pgrad(bool cached, float factor, KernelParams const &K, f3 xij) {
  return cached ? kgrad_from(factor, xij) : kgradW(K, xij);
}

// the sum with the pair's term where the pair counts
__device__ __forceinline__ float add_if(bool in, float a, float t) { return in ? a + t : a; }
__device__ __forceinline__ f3 add_if(bool in, f3 a, f3 t) {
  f3 s = add3(a, t);
  return {in ? s.x : a.x, in ? s.y : a.y, in ? s.z : a.z};
}
__device__ __forceinline__ f3 sub_if(bool in, f3 a, f3 t) {
  f3 s = sub3(a, t);
  return {in ? s.x : a.x, in ? s.y : a.y, in ? s.z : a.z};
}

struct FluidN {
  NbrList L;
  float4 const *xm; // (x, y, z, m)
  float4 const *v;  // velocity
  float4 const *a;  // acceleration
  float const *pr;  // p / (rho rho)
};

// a / b in a walk: without a branch where FLAT, noting in `off` operands that
// this does not divide exactly (the row is then walked again, dividing)
template <bool FLAT> __device__ __forceinline__ float divide_noting(float a, float b, bool &off) {
  if (!FLAT) return a / b;
  float q = divide_flat(a, b);
  off = off || !divides_flat(a, b, q);
  return q;
}
template <bool FLAT> __device__ __forceinline__ float divide_noting(float a, Divisor const &b, bool &off) {
  if (!FLAT) return a / b.d;
  off = off || !quotient_exact(a, b);
  return quotient(a, b);
}

// a neighbour's record and a second value of it
template <class T> struct WithRec {
  float4 x;
  T v;
};

struct BoundN {
  NbrList L;
  float4 const *xV; // (x, y, z, V)
  float const *mu;  // uniform dynamic_viscosity (wkbb18)
};

template <int NF, int NB> struct Nbrs {
  FluidN f[NF > 0 ? NF : 1];
  BoundN b[NB > 0 ? NB : 1];
  float const *hcache; // smoothing scale of the cached gradient factors
};
template <class N> __device__ __forceinline__ bool use_cache(N const &nb, KernelParams const &K) {
  return *nb.hcache == K.h;
}

struct Globals {
  float const *h;
  float const *dt;
  float const *t;
  float const *fade;
  float const *omega;
  float *aprde;
  int *nprde;
  float const *gravity; // 3 floats
  float *max_speed;
  int const *jac_max;   // iisph_maximum_iterations
  float const *jac_eta; // iisph_maximum_density_error
  int *jac_iters;       // iisph_iterations
  unsigned const *turn; // of the solver loops' barriers (Meet)
};
// whether a solver loop gave up and the host has not seen it yet: what it was
// for is left alone then.  (Only an earlier launch writes it: an ordinary load,
// which L1 serves.  One past L1 by every warp to the one word took the velocity
// integration of 1M items from 10.8 to 16.6 us.)
constexpr unsigned kGaveUp = 0x80000000u;
__device__ __forceinline__ bool gave_up(Globals const &G) { return (*G.turn & kGaveUp) != 0u; }

struct Red {
  double *partials; // [3][kMaxRedBlocks]
  unsigned *ticket;
  double *scalars;
  int *status;
  double *stats; // device-loop statistics (Model::stats_d)
};

__device__ __forceinline__ uint32_t grid_tid() { return blockIdx.x * blockDim.x + threadIdx.x; }


// NV block sums, two at a time; valid in thread 0
template <int NV> __device__ __forceinline__ void block_sums(double const (&v)[NV], double *sh, double (&out)[NV]) {
#pragma unroll
  for (int k = 0; k + 1 < NV; k += 2) block_sum2(v[k], v[k + 1], sh, out[k], out[k + 1]);
  if constexpr (NV % 2 != 0) out[NV - 1] = block_sum(v[NV - 1], sh);
}

// FP64 block sums of NV values, committed by the last block of the launch.
// Returns true in the last block; out[] is valid in its thread 0.
template <int NV>
__device__ bool reduce_commit(double const (&v)[NV], Red const &R, double (&out)[NV]) {
  __shared__ double sh[32];
  __shared__ int last;
  double sum[NV];
  block_sums<NV>(v, sh, sum);
  if (threadIdx.x == 0)
    for (int k = 0; k < NV; ++k) R.partials[k * kMaxRedBlocks + blockIdx.x] = sum[k];
  __threadfence();
  if (threadIdx.x == 0) last = (atomicAdd(R.ticket, 1u) == gridDim.x - 1) ? 1 : 0;
  __syncthreads();
  if (!last) return false;
  __threadfence();
  double acc[NV];
  for (int k = 0; k < NV; ++k) {
    acc[k] = 0.0;
    for (unsigned b = threadIdx.x; b < gridDim.x; b += blockDim.x)
      acc[k] += __ldcg(&R.partials[k * kMaxRedBlocks + b]);
  }
  block_sums<NV>(acc, sh, out);
  if (threadIdx.x == 0) *R.ticket = 0u;
  return true;
}

unsigned red_grid(size_t n) { return unsigned(std::min<size_t>(div_up(n, kNT), kMaxRedBlocks)); }

// Launch shapes of the tuned sweeps (Model::tune): threads per block,
// blocks resident per SM (which caps the registers) and the neighbour-walk
// batch.  Entry 0 is the default.  Every entry computes the same bits: the
// per-item arithmetic does not depend on the shape, and the sweeps with an
// FP64 reduction keep 128 threads per block and their grid, so the shape of
// the reduction tree does not change.
// The defaults are the fastest forms of the walk (nbr_walk.cuh, which has the
// times) at 1M items; where the second one is the other number of records,
// density 87 (4) / 88 us (8), set-up 193 (8) / 199 (4), diagonal 113 (4) / 118
// (8).  The tiled sweeps of a batch have rows of other lengths side by side and
// fewer warps once scenes have converged: 48 scenes, 8 steps, second form /
// default, acceleration 7.8 / 6.7 ms, pressure 10.0 / 9.7, PCG product 3.0 / 2.8.
template <int NT_, int MINB_, int BT_> struct Shape {
  static constexpr int nt = NT_, minb = MINB_, bt = BT_;
};
// sweeps without a reduction: the block size may change too
template <int B0, int B1>
using FreeShapes = std::tuple<Shape<kNT, kMinBlocks, B0>, Shape<kNT, kMinBlocks, B1>, Shape<256, 4, B0>,
                              Shape<512, 2, B0>>;
// sweeps with an FP64 reduction, and the tiled sweeps of a batched model
template <int B0, int B1>
using RedShapes = std::tuple<Shape<kNT, kMinBlocks, B0>, Shape<kNT, kMinBlocks, B1>, Shape<kNT, 6, B0>,
                             Shape<kNT, 12, B0>>;
// Up to kSmallItems every block of a sweep is resident at once at four blocks
// per SM, so warps are few anyway and a thread may have the registers to load
// its entries ahead: where the knob has its default, the set-up, Jacobi and PCG
// sweeps take this shape.  At 27k items set-up 17.6 -> 14.6 us, acceleration
// 16.4 -> 10.7, pressure 19.4 -> 14.4, PCG product 23.3 -> 17.0; at 150k items
// pressure 29.4 -> 32.6.
constexpr uint32_t kSmallItems = 152 * 4 * kNT;
using SmallShape = Shape<kNT, 4, 8 | kAhead>;
// f(shape) with the knob's shape where the layout is tuned, else the default
template <class Shapes, bool Tuned, class F> void with_shape(int v, F &&f) {
  if constexpr (Tuned) {
    switch (v) {
    case 1: f(std::tuple_element_t<1, Shapes>{}); return;
    case 2: f(std::tuple_element_t<2, Shapes>{}); return;
    case 3: f(std::tuple_element_t<3, Shapes>{}); return;
    default: break;
    }
  }
  f(std::tuple_element_t<0, Shapes>{});
}
// Many items that were not permuted into cell order: the records of a warp's
// gathers lie far apart, and L1 holds few of them until they are read again, so
// the more loads in flight the better.  The walk with a branch per entry takes 16
// entries together (8 in the diagonal) where the branch-free one gathers 4:
// where the knob has its default, density and diagonal take it.  Branch-free /
// branching, us: density of a lattice in its own order, 422k items 37 / 41, 636k
// 91 / 65, 1M 144 / 95; in random order 85 / 72, 122 / 98, 189 / 143; diagonal 51 /
// 61, 113 / 100, 177 / 154 and 99 / 83, 160 / 128, 237 / 193.  In cell order 1M is a
// draw (78 / 78, 112 / 115) and fewer items are faster branch-free (636k 50 / 53,
// 72 / 74).  Explicit viscosity gains nothing by it (181 / 181, 279 / 287).
constexpr uint32_t kSpreadItems = 500'000;
bool spread(uint32_t n, NbrView const &v) { return !v.ordered && n >= kSpreadItems; }
template <class Shapes, class Spread, bool Tuned, class F> void with_shape_spread(bool spread, int v, F &&f) {
  if (spread && v == 0) f(Spread{});
  else with_shape<Shapes, Tuned>(v, f);
}
// the same for a plain launch over n items of a sweep that takes SmallShape
template <class Shapes, bool Tuned, bool Small, class F> void with_shape_for(uint32_t n, int v, F &&f) {
  if constexpr (Small) {
    if (v == 0 && n <= kSmallItems) {
      f(SmallShape{});
      return;
    }
  }
  with_shape<Shapes, Tuned>(v, f);
}
template <class Sh> std::string shape_text() {
  uint32_t f = uint32_t(Sh::bt);
  return std::to_string(Sh::nt) + "x" + std::to_string(Sh::minb) + "/" + std::to_string(f & 0xFFu) +
         ((f & kAlone) ? "b" : (f & kFill) ? "f" : (f & kAhead) ? "a" : "p");
}
template <class Shapes> std::string shapes_text() {
  return "0=" + shape_text<std::tuple_element_t<0, Shapes>>() + " 1=" + shape_text<std::tuple_element_t<1, Shapes>>() +
         " 2=" + shape_text<std::tuple_element_t<2, Shapes>>() + " 3=" + shape_text<std::tuple_element_t<3, Shapes>>();
}
using DensityShapes = FreeShapes<4 | kFill, 8 | kFill>;
using DensitySpread = Shape<kNT, kMinBlocks, 16 | kAlone>;
using SetupShapes = FreeShapes<8, 4>;
using AccelShapes = FreeShapes<8 | kAlone, 8 | kFill>;
using AccelSegShapes = RedShapes<8 | kFill, 8 | kAlone>;
using PressureShapes = RedShapes<8 | kAlone, 8 | kFill>;
using DiagShapes = FreeShapes<4 | kFill, 8 | kFill>;
using DiagSpread = Shape<kNT, kMinBlocks, 8 | kAlone>;
using PcgShapes = RedShapes<8 | kAlone, 8>;
using PcgSegShapes = RedShapes<8, 8 | kAlone>;

// Staged sweeps (the `staging` knob; lists built staged, nhood.hpp): a
// block's items are the tiles of kStageTile consecutive items the list build
// staged; per tile the block copies the tile's staged items' records to
// shared memory (two float4 per item, in slot order) and the threads read
// their neighbours from there by the lists' slots.  A tile that did not fit
// takes the global gathers.  The records and the order of the terms are
// those of the unstaged sweeps, so the results are bit-identical.
static_assert(kNT == int(kStageTile), "a staged sweep's block is one tile");
struct StageArgs {
  uint16_t const *fslots, *bslots; // slots of the fluid group's lists towards itself and the boundary group
  uint2 const *tile_info, *tile_cells;
  uint32_t const *sorted;          // sorted handles (group << 28 | index)
  int fg, bg;                      // the two groups' indices
};
constexpr size_t kStageSmem = 2 * kStageCap * sizeof(float4);

// copies tile `tile`'s staged records (rec(handle, x, y) per item) to sx, sy;
// false (block-uniform) for a tile that was not staged
// asynchronous global -> shared copies (cp.async): 16 bytes (L2 only), or
// 4 bytes; the records of a tile are all in flight at once
__device__ __forceinline__ void cp_async16(float4 *dst, void const *src) {
  uint32_t d = static_cast<uint32_t>(__cvta_generic_to_shared(dst));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async4(float *dst, void const *src) {
  uint32_t d = static_cast<uint32_t>(__cvta_generic_to_shared(dst));
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// copies tile `tile`'s staged records to sx, sy: rec(handle, sx + p, sy + p)
// issues the copies of slot p (only the parts its sweep reads); false
// (block-uniform) for a tile that was not staged
template <class Rec>
__device__ bool stage_copy(StageArgs const &SA, uint32_t tile, float4 *sx, float4 *sy, Rec &&rec) {
  __shared__ uint32_t s_src[kStageCap]; // sorted index of each staged slot
  __shared__ uint2 s_info;
  if (threadIdx.x == 0) s_info = SA.tile_info[tile];
  __syncthreads();
  uint2 info = s_info;
  if (info.y == kNoStage) return false;
  // each staged cell's slots name its sorted range
  for (uint32_t u = threadIdx.x; u < info.x; u += blockDim.x) {
    uint2 e = SA.tile_cells[size_t(tile) * kStageCells + u];
    uint32_t end = u + 1 < info.x ? SA.tile_cells[size_t(tile) * kStageCells + u + 1].y : info.y;
    for (uint32_t q = e.y; q < end; ++q) s_src[q] = e.x + (q - e.y);
  }
  __syncthreads();
  constexpr int kU = 4; // handles loaded together
  for (uint32_t p0 = threadIdx.x; p0 < info.y; p0 += kU * blockDim.x) {
    uint32_t h[kU];
#pragma unroll
    for (int k = 0; k < kU; ++k) {
      uint32_t p = p0 + k * blockDim.x;
      h[k] = p < info.y ? __ldg(SA.sorted + s_src[p]) : 0u;
    }
#pragma unroll
    for (int k = 0; k < kU; ++k) {
      uint32_t p = p0 + k * blockDim.x;
      if (p < info.y) rec(h[k], sx + p, sy + p);
    }
  }
  cp_async_wait_all();
  __syncthreads();
  return true;
}

// Batched (segmented) models: block b of a tiled launch handles tile b, up to
// kSegTile consecutive items of one slot (scene).  Reductions are per slot:
// each tile stores its FP64 block sum; the last tile of the slot to finish
// sums the slot's tile partials in tile order (one warp, fixed order), so a
// slot's sums depend only on its own items.
static_assert(kNT == int(kSegTile), "tiled kernels run one tile per block");
struct SegArgs {
  uint4 const *tiles;         // (slot, begin, end, 0)
  uint32_t const *slot_tiles; // [slots + 1]
  uint16_t const *seg;        // slot of each item
  uint32_t ntiles, slots;
  double *partials;           // [3][pcap]
  size_t pcap;
  unsigned *tickets;          // [slots]
  double *scal;               // [slots][16]
  int *stat;                  // [slots][8]
  double *stats;              // [slots][8]
  int const *nprde;           // [slots]
  int *iters;                 // [slots]
  uint32_t *active;           // tiles of the slots still iterating ([nactive[0]])
  uint32_t *nactive;          // [0] their count, [1] / [2] work counters (acceleration / pressure)
};
constexpr int kSegScal = 16, kSegStat = 8, kSegStats = 8;
// blocks of the kernels that walk the active tiles (a multiple of the SM
// count times the blocks resident per SM)
constexpr uint32_t kActiveBlocks = 152 * 8;
constexpr int kSsAprde = 8;        // scal: density error of the iteration
constexpr int kSegUpdateNT = 32;   // threads of a tiled PCG update block
constexpr int kStPcgEnded = 3;     // stat: the slot's PCG loop has ended

template <int NV>
__device__ bool seg_commit(double const (&v)[NV], SegArgs const &S, uint32_t slot, double (&out)[NV],
                           uint32_t tile) {
  __shared__ double sh[32];
  __shared__ int last;
  double sum[NV];
  block_sums<NV>(v, sh, sum);
  if (threadIdx.x == 0)
    for (int k = 0; k < NV; ++k) S.partials[k * S.pcap + tile] = sum[k];
  __threadfence();
  uint32_t t0 = S.slot_tiles[slot], t1 = S.slot_tiles[slot + 1];
  if (threadIdx.x == 0) last = (atomicAdd(&S.tickets[slot], 1u) == t1 - t0 - 1) ? 1 : 0;
  __syncthreads();
  if (!last) return false;
  __threadfence();
  if (threadIdx.x < 32) {
    for (int k = 0; k < NV; ++k) {
      double acc = 0.0;
      for (uint32_t t = t0 + threadIdx.x; t < t1; t += 32) acc += __ldcg(&S.partials[k * S.pcap + t]);
      out[k] = warp_sum(acc);
    }
  }
  if (threadIdx.x == 0) S.tickets[slot] = 0u;
  return true;
}

// The tiles of the slots whose Jacobi loop still iterates, in slot order
// (one block, all threads): the Jacobi sweeps of a batched model walk this
// list, so that the slots that have converged cost nothing in the
// iterations that follow.
__device__ void seg_list_active(SegArgs const &S) {
  __shared__ uint32_t warp_tot[32];
  __shared__ uint32_t base;
  if (threadIdx.x == 0) base = 0;
  __syncthreads();
  int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (uint32_t s0 = 0; s0 < S.slots; s0 += blockDim.x) {
    uint32_t sl = s0 + threadIdx.x;
    uint32_t t0 = 0, cnt = 0;
    if (sl < S.slots && !S.stat[sl * kSegStat + kStJacDone]) {
      t0 = S.slot_tiles[sl];
      cnt = S.slot_tiles[sl + 1] - t0;
    }
    // block-exclusive prefix of the counts
    uint32_t incl = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    if (lane == 31) warp_tot[w] = incl;
    __syncthreads();
    uint32_t wbase = 0, total = 0;
    for (int k = 0; k < nw; ++k) {
      if (k < w) wbase += warp_tot[k];
      total += warp_tot[k];
    }
    uint32_t off = base + wbase + incl - cnt;
    for (uint32_t j = 0; j < cnt; ++j) S.active[off + j] = t0 + j;
    __syncthreads();
    if (threadIdx.x == 0) base += total;
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    S.nactive[0] = base;
    S.nactive[1] = 0u; // the persistent sweeps of the next iteration start at tile 0
    S.nactive[2] = 0u;
  }
}
__global__ void k_seg_active(SegArgs S) { seg_list_active(S); }

// ---------------------------------------------------------------------------
// density.compute_density (schemes/density.hpp:160-220)
//   rho_i = sum_f m_j W(x_ij) + sum_b (V_j rho0) W(x_ij)
// ---------------------------------------------------------------------------

// use(record, in, kernel parameters): the walk of the sweeps that evaluate the
// kernel per pair
template <uint32_t FORM, class Load, class Use>
__device__ __forceinline__ void walk_kernel(NbrList const &L, uint32_t i, QuickKernel const &K, Load &&load, Use &&use) {
  if constexpr ((FORM & kAlone) != 0u) {
    if (K.quick) {
      for_each_nbr<FORM & 0xFFu>(L, i, false, [&](uint32_t j, float) { use(load(j), true, K); });
      return;
    }
  } else if (K.quick) {
    walk_nbrs<FORM, false>(L, i, load, [&](float4 x, float, bool in) { use(x, in, K); });
    return;
  }
  for_each_nbr<16>(L, i, false, [&](uint32_t j, float) { use(load(j), true, K.k); });
}

template <int NF, int NB, int NT = kNT, int MINB = kMinBlocks, int BT = 4 | kFill>
__global__ void __launch_bounds__(NT, MINB) k_density(uint32_t n, float4 const *__restrict__ x, float *__restrict__ rho,
                                                 float const *rho0p, Globals G, Nbrs<NF, NB> N) {
  uint32_t i = grid_tid();
  if (i >= n) return;
  QuickKernel K = quick_kernel(kparams(*G.h));
  float rho0 = *rho0p;
  f3 xi = mk3(x[i]);
  float acc = 0.0f;
#pragma unroll
  for (int q = 0; q < NF; ++q) {
    FluidN const &F = N.f[q];
    walk_kernel<BT>(F.L, i, K, [&](uint32_t j) { return __ldg(F.xm + j); }, [&](float4 xm, bool in, auto const &k) {
      acc = add_if(in, acc, xm.w * kW(k, sub3(xi, mk3(xm))));
    });
  }
#pragma unroll
  for (int q = 0; q < NB; ++q) {
    BoundN const &B = N.b[q];
    walk_kernel<BT>(B.L, i, K, [&](uint32_t j) { return __ldg(B.xV + j); }, [&](float4 xv, bool in, auto const &k) {
      acc = add_if(in, acc, (xv.w * rho0) * kW(k, sub3(xi, mk3(xv))));
    });
  }
  rho[i] = acc;
}

// aiast12.compute_volume (schemes/aiast12.hpp:125-175): V_i = 1 / sum_b W
template <int NB>
__global__ void __launch_bounds__(kNT, kMinBlocks) k_volume(uint32_t n, float4 const *__restrict__ x, float *__restrict__ V,
                                                Globals G, Nbrs<0, NB> N) {
  uint32_t i = grid_tid();
  if (i >= n) return;
  QuickKernel K = quick_kernel(kparams(*G.h));
  f3 xi = mk3(x[i]);
  float acc = 0.0f;
#pragma unroll
  for (int q = 0; q < NB; ++q) {
    BoundN const &B = N.b[q];
    walk_kernel<4 | kFill>(B.L, i, K, [&](uint32_t j) { return __ldg(B.xV + j); }, [&](float4 xv, bool in, auto const &k) {
      acc = add_if(in, acc, kW(k, sub3(xi, mk3(xv))));
    });
  }
  V[i] = 1.0f / acc;
}

// gravity.initialize_acceleration (schemes/gravity.hpp:133-158): a = g
__global__ void k_gravity(uint32_t n, float4 *__restrict__ a, Globals G) {
  uint32_t i = grid_tid();
  if (i < n) a[i] = make_float4(G.gravity[0], G.gravity[1], G.gravity[2], 0.0f);
}

// symplectic_euler.integrate_velocity_with_hard_fade
// (schemes/symplectic_euler.hpp:172-201): v += (dt a) * [0 < (t - t_b) - fade]
__global__ void k_integrate_velocity(uint32_t n, float4 *__restrict__ v, float4 const *__restrict__ a,
                                     float const *__restrict__ tb, Globals G) {
  uint32_t i = grid_tid();
  if (i >= n) return;
  bool keep = gave_up(G);
  float dt = *G.dt, t = *G.t, fade = *G.fade;
  float u = ustep(0.0f, (t - tb[i]) - fade);
  float4 vi = v[i], ai = a[i];
  vi.x = vi.x + (dt * ai.x) * u;
  vi.y = vi.y + (dt * ai.y) * u;
  vi.z = vi.z + (dt * ai.z) * u;
  if (!keep) v[i] = vi;
}

// symplectic_euler.integrate_position (schemes/symplectic_euler.hpp:236-270):
// x += dt v; max_speed = max(max_speed, |v|) over all dynamic particles
//
// A speed is never negative, and the bits of non-negative floats, and of a
// negative or NaN maximum beside them, compare as integers like the floats'
// maximum: one atomic per warp that raises it, on the global itself.  xm, where
// given: the packed records (x, m) of the next sweeps.  (The maximum's two
// conversions and the records each had a launch of their own, 2 to 4 us of a
// small scene's step of 220.)
__global__ void k_integrate_position(uint32_t n, float4 *__restrict__ x, float4 const *__restrict__ v, Globals G,
                                     float4 *__restrict__ xm, float const *__restrict__ m) {
  uint32_t i = grid_tid();
  int top = *reinterpret_cast<volatile int const *>(G.max_speed);
  bool keep = gave_up(G);
  float sp = -INFINITY;
  if (i < n) {
    float dt = *G.dt;
    float4 xi = x[i], vi = v[i];
    xi.x = xi.x + dt * vi.x;
    xi.y = xi.y + dt * vi.y;
    xi.z = xi.z + dt * vi.z;
    float mi = xm ? m[i] : 0.0f;
    if (!keep) {
      x[i] = xi;
      if (xm) xm[i] = make_float4(xi.x, xi.y, xi.z, mi);
      sp = sqrtf(nsq3(mk3(vi)));
    }
  }
  for (int o = 16; o > 0; o >>= 1) sp = fmaxf(sp, __shfl_down_sync(0xffffffffu, sp, o));
  if ((threadIdx.x & 31) == 0 && sp > -INFINITY && __float_as_int(sp) > top)
    atomicMax(reinterpret_cast<int *>(G.max_speed), __float_as_int(sp));
}

// ---------------------------------------------------------------------------
// iisph.setup (schemes/iisph.hpp:188-354)
//   pass 1: c_i = -sum_f (m_j / rho_i^2) gradW - sum_b ((0.7*2) rho0 (V_j / rho_i^2)) gradW
//   pass 2: p = 0, source term s and diagonal element AA; also p / rho^2
//           (= 0) for the pressure acceleration
// ---------------------------------------------------------------------------

// Passes 1 and 2 in one sweep: pass 2 reads only the item's own c, so each
// thread computes c over its neighbours, stores it, then walks the same (now
// cached) neighbour rows again for s and AA, with the operations of the
// generated passes.
template <int NF, int NB, int NT = kNT, int MINB = kMinBlocks, int BT = 8>
__global__ void __launch_bounds__(NT, MINB) k_iisph_setup(uint32_t n, float4 const *__restrict__ x,
                                                                 float4 const *__restrict__ v,
                                                                 float4 *__restrict__ cout, float const *__restrict__ m,
                                                                 float const *__restrict__ rho, float *__restrict__ p,
                                                                 float *__restrict__ pr, float *__restrict__ s,
                                                                 float *__restrict__ AA, float const *rho0p, Globals G,
                                                                 Nbrs<NF, NB> N, int *bad) {
  uint32_t i = grid_tid();
  if (i >= n) return;
  KernelParams K = kparams(*G.h);
  bool uc = use_cache(N, K);
  float rho0 = *rho0p, dt = *G.dt;
  f3 xi = mk3(x[i]);
  float ri = rho[i];
  Divisor rr = divisor(ri * ri);
  f3 c;
  bool flat = uc, off;
  do {
    c = {0.0f, 0.0f, 0.0f};
    off = false;
#pragma unroll
    for (int q = 0; q < NF; ++q) {
      FluidN const &F = N.f[q];
      walk_nbrs_cached<BT, true>(F.L, i, flat, [&](uint32_t j) { return __ldg(F.xm + j); },
                                 [&](float4 xm, float gf, bool in, auto cached) {
        constexpr bool kFlat = std::is_same_v<decltype(cached), std::true_type>;
        c = sub_if(in, c, scl3(divide_noting<kFlat>(xm.w, rr, off), pgrad(is_cached(cached), gf, K, sub3(xi, mk3(xm)))));
      });
    }
#pragma unroll
    for (int q = 0; q < NB; ++q) {
      BoundN const &B = N.b[q];
      walk_nbrs_cached<BT, true>(B.L, i, flat, [&](uint32_t j) { return __ldg(B.xV + j); },
                                 [&](float4 xv, float gf, bool in, auto cached) {
        constexpr bool kFlat = std::is_same_v<decltype(cached), std::true_type>;
        c = sub_if(in, c, scl3(((0.7f * 2.0f) * rho0) * divide_noting<kFlat>(xv.w, rr, off),
                               pgrad(is_cached(cached), gf, K, sub3(xi, mk3(xv)))));
      });
    }
    if (!off) break;
    flat = false;
  } while (true);
  cout[i] = make_float4(c.x, c.y, c.z, 0.0f);
  bool finite = isfinite(c.x) && isfinite(c.y) && isfinite(c.z);
  f3 vi = mk3(v[i]), ci = c;
  float mi = m[i];
  float sa = 0.0f, aa = 0.0f;
#pragma unroll
  for (int q = 0; q < NF; ++q) {
    FluidN const &F = N.f[q];
    walk_nbrs_cached<BT>(F.L, i, uc, [&](uint32_t j) { return WithRec<f3>{__ldg(F.xm + j), mk3(__ldg(F.v + j))}; },
                         [&](WithRec<f3> const &r, float gf, bool in, auto cached) {
      f3 g = pgrad(is_cached(cached), gf, K, sub3(xi, mk3(r.x)));
      float mj = r.x.w;
      sa = add_if(in, sa, mj * dot3(sub3(vi, r.v), g));
      aa = add_if(in, aa, mj * dot3(ci, g));
      aa = add_if(in, aa, -((mj * (mi / (ri * ri))) * nsq3(g)));
    });
  }
#pragma unroll
  for (int q = 0; q < NB; ++q) {
    BoundN const &B = N.b[q];
    walk_nbrs_cached<BT>(B.L, i, uc, [&](uint32_t j) { return __ldg(B.xV + j); },
                         [&](float4 xv, float gf, bool in, auto cached) {
      f3 g = pgrad(is_cached(cached), gf, K, sub3(xi, mk3(xv)));
      float w = rho0 * xv.w;
      sa = add_if(in, sa, w * dot3(sub3(vi, f3{0.0f, 0.0f, 0.0f}), g));
      aa = add_if(in, aa, w * dot3(ci, g));
    });
  }
  if (!(finite && isfinite(aa))) *bad = 1;
  p[i] = 0.0f;
  pr[i] = 0.0f / (ri * ri);
  s[i] = (rho0 - ri) - ((dt * (rho0 / ri)) * sa);
  AA[i] = aa * ((dt * dt) * (rho0 / ri));
}

struct RestDensities {
  float const *p[kMaxNbrGroups];
  int n;
};
// before the set-up sweeps
__global__ void k_setup_begin(int *status, int *nprde, int total, Globals G, RestDensities D, double *scalars) {
  status[kStSetupBad] = 0;
  *nprde = total;
  scalars[kSSetup] = double(*G.h);
  for (int k = 0; k < D.n; ++k) scalars[kSSetup + 1 + k] = double(*D.p[k]);
}
// whether the loop's first iteration may take zero sums (see kStJacFirst):
// `same` is the host's part
__device__ __forceinline__ bool zero_sums_hold(Globals const &G, RestDensities const &D, int const *status,
                                               double const *scalars, int same) {
  bool ok = same && !status[kStSetupBad] && scalars[kSSetup] == double(*G.h);
  for (int k = 0; k < D.n; ++k) ok = ok && scalars[kSSetup + 1 + k] == double(*D.p[k]) && isfinite(*D.p[k]);
  return ok;
}
__device__ __forceinline__ int jacobi_first(Globals const &G, RestDensities const &D, int *status,
                                            double const *scalars, int same) {
  bool ok = zero_sums_hold(G, D, status, scalars, same);
  status[kStSetupBad] = 1; // the solve changes the pressure
  return ok ? 1 : 0;
}

// iisph.iteration_pressure_acceleration (schemes/iisph.hpp:358-423).
// `done` (device-loop mode) skips the work once the loop has converged.
template <int NF, int NB, int BT = 8 | kAlone>
__device__ __forceinline__ void iisph_accel_item(uint32_t i, float4 const *__restrict__ x, float const *__restrict__ p,
                                                 float const *__restrict__ rho, float4 *__restrict__ a,
                                                 KernelParams const &K, bool uc, float rho0, Nbrs<NF, NB> const &N) {
  f3 xi = mk3(x[i]);
  float pi = p[i], ri = rho[i];
  float pri = pi / (ri * ri);
  f3 acc = {0.0f, 0.0f, 0.0f};
#pragma unroll
  for (int q = 0; q < NF; ++q) {
    FluidN const &F = N.f[q];
    walk_nbrs_flat<BT>(F.L, i, uc, uc, [&](uint32_t j) { return WithRec<float>{__ldg(F.xm + j), __ldg(F.pr + j)}; },
                         [&](WithRec<float> const &r, float gf, bool in, auto cached) {
      float coef = r.x.w * (pri + r.v);
      acc = sub_if(in, acc, scl3(coef, pgrad(is_cached(cached), gf, K, sub3(xi, mk3(r.x)))));
    });
  }
  float bterm = (2.0f * pi) / (ri * ri);
#pragma unroll
  for (int q = 0; q < NB; ++q) {
    BoundN const &B = N.b[q];
    walk_nbrs_flat<BT>(B.L, i, uc, uc, [&](uint32_t j) { return __ldg(B.xV + j); },
                         [&](float4 xv, float gf, bool in, auto cached) {
      float coef = ((0.7f * rho0) * xv.w) * bterm;
      acc = sub_if(in, acc, scl3(coef, pgrad(is_cached(cached), gf, K, sub3(xi, mk3(xv)))));
    });
  }
  a[i] = make_float4(acc.x, acc.y, acc.z, 0.0f);
}
template <int NF, int NB, int NT = kNT, int MINB = kMinBlocks, int BT = 8 | kAlone>
__global__ void __launch_bounds__(NT, MINB) k_iisph_accel(uint32_t n, float4 const *__restrict__ x, float const *__restrict__ p,
                                                     float const *__restrict__ rho, float4 *__restrict__ a,
                                                     float const *rho0p, Globals G, Nbrs<NF, NB> N, int const *done) {
  // (the two words are loaded together)
  int ended = done ? *(volatile int const *)done : 0, first = done ? *(volatile int const *)(done + 1) : 0;
  if (ended) return;
  uint32_t i = grid_tid();
  if (i >= n) return;
  if (first) {
    a[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    return;
  }
  KernelParams K = kparams(*G.h);
  iisph_accel_item<NF, NB, BT>(i, x, p, rho, a, K, use_cache(N, K), *rho0p, N);
}
// batched models: the tiles of the slots still iterating
// (DYN: each block takes the next tile from a work counter instead of a
// static share of the tiles; the tiles' items and arithmetic are the same)
template <int NF, int NB, int MINB = kMinBlocks, int BT = 8 | kAlone, bool DYN = false>
__global__ void __launch_bounds__(kNT, MINB) k_iisph_accel_seg(float4 const *__restrict__ x, float const *__restrict__ p,
                                                         float const *__restrict__ rho, float4 *__restrict__ a,
                                                         float const *rho0p, Globals G, Nbrs<NF, NB> N, SegArgs S,
                                                         int const *first) {
  bool zero = *(volatile int const *)first != 0;
  KernelParams K = kparams(*G.h);
  bool uc = use_cache(N, K);
  float rho0 = *rho0p;
  uint32_t na = S.nactive[0];
  __shared__ uint32_t next;
  for (uint32_t t = blockIdx.x;;) {
    if (DYN) {
      if (threadIdx.x == 0) next = atomicAdd(&S.nactive[1], 1u);
      __syncthreads();
      t = next;
      __syncthreads();
    }
    if (t >= na) break;
    uint4 T = S.tiles[S.active[t]];
    uint32_t i = T.y + threadIdx.x;
    if (i < T.z) {
      if (zero) a[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      else iisph_accel_item<NF, NB, BT>(i, x, p, rho, a, K, uc, rho0, N);
    }
    if (!DYN) t += gridDim.x;
  }
}

// iisph.iteration_pressure (schemes/iisph.hpp:426-516) with the FP64
// density-error reduction.  scalars[kSJacobi] accumulates aprde across the
// fluid groups of one call: `first` starts it from the global aprde (or
// from 0 in device-loop mode, where aprde := 0 precedes every iteration),
// `last_group` stores it.  Also writes p / rho^2 for the next acceleration.
struct PressureArgs {
  float4 const *x, *a;
  float const *rho, *s, *AA;
  float *p, *pr, *Ap;
  float const *rho0;
};

// the end of iteration_pressure for one item, from its neighbour sum ap:
// Ap, the new pressure (and p / rho^2); returns the density-error term
__device__ __forceinline__ double pressure_finish(uint32_t i, PressureArgs const &A, float ap, float rho0, float dt,
                                                  float omega) {
  float ri = A.rho[i];
  ap *= (dt * dt) * (rho0 / ri);
  A.Ap[i] = ap;
  float si = A.s[i], aai = A.AA[i];
  float t = A.p[i] + ((omega * (si - ap)) * rcp0(aai, 1e-9f));
  // std::max({0, t}) returns the first largest element: t only if 0 < t
  float pn = ((0.0f < t) ? t : 0.0f) * ustep(1e-9f, fabsf(aai));
  A.p[i] = pn;
  A.pr[i] = pn / (ri * ri);
  return f2d(((ap - si) / rho0) * ustep(1e-9f, pn));
}

// one item of iteration_pressure; returns its density-error term
template <int NF, int NB, int BT = 8 | kAlone>
__device__ __forceinline__ double iisph_pressure_item(uint32_t i, PressureArgs const &A, KernelParams const &K, bool uc,
                                                      float rho0, float dt, float omega, Nbrs<NF, NB> const &N) {
  f3 xi = mk3(A.x[i]), ai = mk3(A.a[i]);
  float ap = 0.0f;
#pragma unroll
  for (int q = 0; q < NF; ++q) {
    FluidN const &F = N.f[q];
    walk_nbrs_flat<BT>(F.L, i, uc, uc, [&](uint32_t j) { return WithRec<f3>{__ldg(F.xm + j), mk3(__ldg(F.a + j))}; },
                         [&](WithRec<f3> const &r, float gf, bool in, auto cached) {
      ap = add_if(in, ap, r.x.w * dot3(sub3(ai, r.v), pgrad(is_cached(cached), gf, K, sub3(xi, mk3(r.x)))));
    });
  }
#pragma unroll
  for (int q = 0; q < NB; ++q) {
    BoundN const &B = N.b[q];
    walk_nbrs_flat<BT>(B.L, i, uc, uc, [&](uint32_t j) { return __ldg(B.xV + j); },
                         [&](float4 xv, float gf, bool in, auto cached) {
      ap = add_if(in, ap, (rho0 * xv.w) * dot3(sub3(ai, f3{0.0f, 0.0f, 0.0f}), pgrad(is_cached(cached), gf, K, sub3(xi, mk3(xv)))));
    });
  }
  return pressure_finish(i, A, ap, rho0, dt, omega);
}

template <int NF, int NB, int MINB = kMinBlocks, int BT = 8 | kAlone>
__global__ void __launch_bounds__(kNT, MINB) k_iisph_pressure(uint32_t n, PressureArgs A, Globals G, Nbrs<NF, NB> N, Red R,
                                                        int first, int last_group, int const *done) {
  int ended = done ? *(volatile int const *)done : 0, zero = done ? *(volatile int const *)(done + 1) : 0;
  if (ended) return;
  KernelParams K = kparams(*G.h);
  bool uc = use_cache(N, K);
  float rho0 = *A.rho0, dt = *G.dt, omega = *G.omega;
  double part = 0.0;
  if (zero) {
    for (uint32_t i = grid_tid(); i < n; i += gridDim.x * blockDim.x)
      part += pressure_finish(i, A, 0.0f, rho0, dt, omega);
  } else {
    for (uint32_t i = grid_tid(); i < n; i += gridDim.x * blockDim.x)
      part += iisph_pressure_item<NF, NB, BT>(i, A, K, uc, rho0, dt, omega, N);
  }
  double v[1] = {part}, out[1];
  if (reduce_commit<1>(v, R, out) && threadIdx.x == 0) {
    double start = first ? (done ? 0.0 : double(*G.aprde)) : R.scalars[kSJacobi];
    double acc = start + out[0];
    R.scalars[kSJacobi] = acc;
    if (last_group) *G.aprde = float(acc);
    // (also where a captured graph runs it unseen by the host: the pressure is
    // not set-up's any more)
    if (!done) R.status[kStSetupBad] = 1;
  }
}

// iteration_pressure over the tiles of a batched model: the density error of
// each slot's iteration goes to scal[slot][kSsAprde]
// (DYN: a persistent grid whose blocks take tiles from a work counter; the
// per-tile partial sums and their per-slot commit are unchanged)
template <int NF, int NB, int MINB = kMinBlocks, int BT = 8 | kAlone, bool DYN = false>
__global__ void __launch_bounds__(kNT, MINB) k_iisph_pressure_seg(PressureArgs A, Globals G, Nbrs<NF, NB> N, SegArgs S,
                                                                  int const *first) {
  bool zero = *(volatile int const *)first != 0;
  // one active tile per block (the hardware's block scheduling balances the
  // tiles' uneven costs); the blocks past the active tiles exit at once
  uint32_t na = S.nactive[0];
  if (!DYN && blockIdx.x >= na) return;
  KernelParams K = kparams(*G.h);
  bool uc = use_cache(N, K);
  float rho0 = *A.rho0, dt = *G.dt, omega = *G.omega;
  __shared__ uint32_t next;
  for (uint32_t k = blockIdx.x;;) {
    if (DYN) {
      if (threadIdx.x == 0) next = atomicAdd(&S.nactive[2], 1u);
      __syncthreads();
      k = next;
      __syncthreads();
      if (k >= na) break;
    }
    uint32_t t = S.active[k];
    uint4 T = S.tiles[t];
    uint32_t slot = T.x;
    uint32_t i = T.y + threadIdx.x;
    double part = 0.0;
    if (i < T.z)
      part = zero ? pressure_finish(i, A, 0.0f, rho0, dt, omega)
                  : iisph_pressure_item<NF, NB, BT>(i, A, K, uc, rho0, dt, omega, N);
    double v[1] = {part}, out[1];
    if (seg_commit<1>(v, S, slot, out, t) && threadIdx.x == 0) S.scal[slot * kSegScal + kSsAprde] = out[0];
    if (!DYN) break;
  }
}

// staged relaxed-Jacobi sweeps (one fluid and one boundary group; the
// `staging` knob).  Per tile, the staged records: a fluid item's (x, m) and
// p / rho^2 (acceleration) or acceleration (pressure); a boundary item's
// (x, V).
template <int BT = 8>
__global__ void __launch_bounds__(kNT, 4) k_iisph_accel_staged(uint32_t n, float4 const *__restrict__ x,
                                                               float const *__restrict__ p,
                                                               float const *__restrict__ rho, float4 *__restrict__ a,
                                                               float const *rho0p, Globals G, Nbrs<1, 1> N,
                                                               int const *done, StageArgs SA) {
  if (done && *(volatile int const *)done) return;
  extern __shared__ float4 sm[];
  float4 *sx = sm, *sy = sm + kStageCap;
  KernelParams K = kparams(*G.h);
  bool uc = use_cache(N, K);
  float rho0 = *rho0p;
  FluidN const &F = N.f[0];
  BoundN const &B = N.b[0];
  for (uint32_t tile = blockIdx.x; size_t(tile) * kNT < n; tile += gridDim.x) {
    uint32_t i = tile * kNT + threadIdx.x;
    // fluid: (x, m) and p / rho^2 (in .x); boundary: (x, V)
    bool st = stage_copy(SA, tile, sx, sy, [&](uint32_t h, float4 *dx, float4 *dy) {
      uint32_t j = h & 0x0FFFFFFFu;
      if (int(h >> 28) == SA.fg) {
        cp_async16(dx, F.xm + j);
        cp_async4(&dy->x, F.pr + j);
      } else if (int(h >> 28) == SA.bg) {
        cp_async16(dx, B.xV + j);
      }
    });
    if (i < n) {
      if (st) {
        f3 xi = mk3(x[i]);
        float pi = p[i], ri = rho[i];
        float pri = pi / (ri * ri);
        f3 acc = {0.0f, 0.0f, 0.0f};
        for_each_staged<BT>(F.L, SA.fslots, i, [&](uint32_t sl, float gf_) {
          float4 xm = sx[sl];
          float coef = xm.w * (pri + sy[sl].x);
          acc = sub3(acc, scl3(coef, pgrad(uc, gf_, K, sub3(xi, mk3(xm)))));
        });
        float bterm = (2.0f * pi) / (ri * ri);
        for_each_staged<BT>(B.L, SA.bslots, i, [&](uint32_t sl, float gf_) {
          float4 xv = sx[sl];
          float coef = ((0.7f * rho0) * xv.w) * bterm;
          acc = sub3(acc, scl3(coef, pgrad(uc, gf_, K, sub3(xi, mk3(xv)))));
        });
        a[i] = make_float4(acc.x, acc.y, acc.z, 0.0f);
      } else {
        iisph_accel_item<1, 1, 8 | kAlone>(i, x, p, rho, a, K, uc, rho0, N);
      }
    }
    __syncthreads(); // the next tile reuses the shared memory
  }
}

// the tiles of a block are those of k_iisph_pressure's grid-stride items,
// so the FP64 partial sums are the same
template <int BT = 8>
__global__ void __launch_bounds__(kNT, 4) k_iisph_pressure_staged(uint32_t n, PressureArgs A, Globals G,
                                                                  Nbrs<1, 1> N, Red R, int first, int last_group,
                                                                  int const *done, StageArgs SA) {
  if (done && *(volatile int const *)done) return;
  extern __shared__ float4 sm[];
  float4 *sx = sm, *sy = sm + kStageCap;
  KernelParams K = kparams(*G.h);
  bool uc = use_cache(N, K);
  float rho0 = *A.rho0, dt = *G.dt, omega = *G.omega;
  FluidN const &F = N.f[0];
  BoundN const &B = N.b[0];
  double part = 0.0;
  for (uint32_t tile = blockIdx.x; size_t(tile) * kNT < n; tile += gridDim.x) {
    uint32_t i = tile * kNT + threadIdx.x;
    // fluid: (x, m) and the acceleration; boundary: (x, V)
    bool st = stage_copy(SA, tile, sx, sy, [&](uint32_t h, float4 *dx, float4 *dy) {
      uint32_t j = h & 0x0FFFFFFFu;
      if (int(h >> 28) == SA.fg) {
        cp_async16(dx, F.xm + j);
        cp_async16(dy, F.a + j);
      } else if (int(h >> 28) == SA.bg) {
        cp_async16(dx, B.xV + j);
      }
    });
    if (i < n) {
      if (st) {
        f3 xi = mk3(A.x[i]), ai = mk3(A.a[i]);
        float ap = 0.0f;
        for_each_staged<BT>(F.L, SA.fslots, i, [&](uint32_t sl, float gf_) {
          float4 xm = sx[sl];
          ap += xm.w * dot3(sub3(ai, mk3(sy[sl])), pgrad(uc, gf_, K, sub3(xi, mk3(xm))));
        });
        for_each_staged<BT>(B.L, SA.bslots, i, [&](uint32_t sl, float gf_) {
          float4 xv = sx[sl];
          ap += (rho0 * xv.w) * dot3(sub3(ai, f3{0.0f, 0.0f, 0.0f}), pgrad(uc, gf_, K, sub3(xi, mk3(xv))));
        });
        part += pressure_finish(i, A, ap, rho0, dt, omega);
      } else {
        part += iisph_pressure_item<1, 1, 8 | kAlone>(i, A, K, uc, rho0, dt, omega, N);
      }
    }
    __syncthreads();
  }
  double v[1] = {part}, out[1];
  if (reduce_commit<1>(v, R, out) && threadIdx.x == 0) {
    double start = first ? (done ? 0.0 : double(*G.aprde)) : R.scalars[kSJacobi];
    double acc = start + out[0];
    R.scalars[kSJacobi] = acc;
    if (last_group) *G.aprde = float(acc);
  }
}

// per-slot loop start: a slot without fluid items does not iterate
__global__ void k_seg_jacobi_begin(SegArgs S, Globals G, Red R, RestDensities D, int same) {
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    R.status[kStJacDone] = 0;
    R.status[kStJacFirst] = jacobi_first(G, D, R.status, R.scalars, same);
  }
  for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < S.slots; k += gridDim.x * blockDim.x) {
    S.stat[k * kSegStat + kStJacIter] = 0;
    S.stat[k * kSegStat + kStJacDone] = (S.nprde[k] >= 1) ? 0 : 1;
  }
}

// per-slot relaxed-Jacobi control (the rule of k_jacobi_control, per slot);
// one block; the loop continues while any slot iterates.  stats per slot:
// 0 solves, 1 iterations, 2 solves stopped at the cap, 3 largest final
// aprde / nprde, 7 final aprde / nprde of the last solve
__global__ void k_seg_jacobi_control(Globals G, SegArgs S, cudaGraphConditionalHandle h, int use_handle,
                                     int kernels, int *all_done, int *first) {
  int any = 0;
  int maxit = *G.jac_max > 0 ? *G.jac_max : 100;
  float eta = *G.jac_eta > 0.0f ? *G.jac_eta : 1e-3f;
  for (uint32_t k = threadIdx.x; k < S.slots; k += blockDim.x) {
    int *st = S.stat + k * kSegStat;
    int done = st[kStJacDone];
    if (!done) {
      int it = st[kStJacIter] + 1;
      st[kStJacIter] = it;
      double rel = S.scal[k * kSegScal + kSsAprde] / double(S.nprde[k]);
      bool converged = it >= 2 && rel < double(eta);
      if (converged || it >= maxit || it >= 100000) done = 1;
      st[kStJacDone] = done;
      if (done) {
        double *sv = S.stats + k * kSegStats;
        sv[0] += 1.0;
        sv[1] += double(it);
        if (!converged) sv[2] += 1.0;
        if (rel > sv[3]) sv[3] = rel;
        sv[7] = rel;
      }
    }
    any |= !done;
  }
  any = __syncthreads_or(any);
  if (any) seg_list_active(S);
  else if (threadIdx.x == 0) {
    // repeats of the loop body after the end sweep nothing
    S.nactive[0] = 0u;
    S.nactive[1] = 0u;
    S.nactive[2] = 0u;
  }
  if (threadIdx.x == 0) {
    *all_done = any ? 0 : 1;
    *first = 0;
    if (kernels) atomicAdd(&g_loop_kernels, (unsigned long long)kernels);
    if (use_handle) cudaGraphSetConditional(h, any ? 1u : 0u);
  }
}

// relaxed-Jacobi loop control (share/scripts/prtcl-lua.example.lua:409-420):
// at least two iterations; stop when aprde / nprde < eta or at the cap
__global__ void k_jacobi_begin(Globals G, Red R, RestDensities D, int same) {
  R.status[kStJacFirst] = jacobi_first(G, D, R.status, R.scalars, same);
  R.status[kStJacIter] = 0;
  R.status[kStJacDone] = (*G.nprde >= 1) ? 0 : 1;
  *G.jac_iters = 0;
}
// (one thread; returns whether the loop has ended)
__device__ int jacobi_control(Globals const &G, Red const &R) {
  int done = R.status[kStJacDone];
  if (!done) {
    int it = R.status[kStJacIter] + 1;
    R.status[kStJacIter] = it;
    int maxit = *G.jac_max > 0 ? *G.jac_max : 100;
    float eta = *G.jac_eta > 0.0f ? *G.jac_eta : 1e-3f;
    double rel = R.scalars[kSJacobi] / double(*G.nprde);
    bool converged = it >= 2 && rel < double(eta);
    if (converged || it >= maxit || it >= 100000) done = 1;
    R.status[kStJacDone] = done;
    R.status[kStJacFirst] = 0;
    *G.jac_iters = it;
    if (done) {
      R.stats[0] += 1.0;
      R.stats[1] += double(it);
      if (!converged) R.stats[2] += 1.0;
      if (rel > R.stats[3]) R.stats[3] = rel;
    }
  }
  return done;
}
__global__ void k_jacobi_control(Globals G, Red R, cudaGraphConditionalHandle h, int use_handle, int kernels) {
  int done = jacobi_control(G, R);
  // the body's kernels ran (those of a repeat after the end return at once)
  if (kernels) atomicAdd(&g_loop_kernels, (unsigned long long)kernels);
  if (use_handle) cudaGraphSetConditional(h, done ? 0u : 1u);
}

// The whole relaxed-Jacobi loop of a small scene in one cooperative launch: the
// blocks are all resident (one item a thread), so they meet at barriers where
// the graph's loop has two launches, a control's launch and a turn of the loop.  A thread keeps its item's values in
// registers; the fields that its neighbours read (acceleration, p / rho^2) go
// through memory, with ordinary loads, which the barriers order for compiler and
// device alike (a read-only or cache-hinted load need not be).
// Values, sums and their order are those of the separate sweeps.  Set-up and
// solve of the 27k dam break 159 -> 144 us, an 8-step run of 2k particles 1.71
// -> 1.54 ms, of 27k 2.00 -> 1.84.
//
// A barrier gives up after `polls` polls.  That marks the turn (kGaveUp) and
// notes the launch where the host sees it (Model::check_solver, which raises an
// error and zeroes the words again).  Until then every barrier gives up at once,
// loops that begin return, and the fields that the solve was for stay as they
// are: velocities, positions and PCG's results are not written (gave_up).
struct Meet {
  unsigned *arrived, *turn; // arrivals at the running barrier (zero between launches); barriers passed, modulo 2^31
  int *host, launch;
  unsigned polls;
};
// The turn to wait for, read where the launch begins: it moves on only after
// this block's first arrival, which a fence follows the read before.  Later ones
// are counted.  (Read beside each arrival, with nothing between the two, the
// load could take effect after the arrival and find the next turn: the block
// would wait for one that does not come.)
// (thread 0 reads it before the launch's other first loads, the block shares
// it after them)
__device__ __forceinline__ unsigned meet_read(Meet const &M) {
  return threadIdx.x == 0 ? *(volatile unsigned *)M.turn : 0u;
}
__device__ __forceinline__ unsigned meet_share(unsigned turn) {
  __shared__ unsigned s_turn;
  if (threadIdx.x == 0) s_turn = turn;
  __syncthreads();
  return s_turn;
}
// last(): run by the block that arrives last, in all its threads, before the
// others go on.  False where the barrier gave up.
template <class F> __device__ bool meet(Meet const &M, unsigned &turn, F &&last) {
  __shared__ int s_last, s_ok;
  unsigned next = (turn + 1u) & (kGaveUp - 1u);
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    bool all = atomicAdd(M.arrived, 1u) == gridDim.x - 1;
    s_ok = !all || *(volatile unsigned *)M.turn == turn ? 1 : 0;
    s_last = all && s_ok ? 1 : 0;
  }
  __syncthreads();
  if (s_last) {
    __threadfence();
    last();
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
      *M.arrived = 0u;
      __threadfence();
      atomicAdd(M.turn, next - turn);
    }
  } else if (threadIdx.x == 0 && s_ok) {
    unsigned now, polls = 0;
    while ((now = *(volatile unsigned *)M.turn) == turn && polls++ < M.polls) __nanosleep(64);
    if (now == turn) {
      atomicOr(M.turn, kGaveUp);
      *(volatile int *)M.host = M.launch;
      __threadfence_system();
    }
    if (now != next) s_ok = 0;
    __threadfence();
  }
  turn = next;
  __syncthreads();
  return s_ok != 0;
}

__global__ void __launch_bounds__(kNT, 4) k_jacobi_loop(uint32_t n, PressureArgs A, float4 *a, Globals G, Nbrs<1, 1> N,
                                                        Red R, Meet M, const __grid_constant__ RestDensities D,
                                                        int same) {
  constexpr uint32_t kForm = 8 | kAhead;
  uint32_t i = grid_tid();
  unsigned turn = meet_read(M);
  bool mine = i < n;
  KernelParams K = kparams(*G.h);
  bool uc = use_cache(N, K);
  float rho0 = *A.rho0, dt = *G.dt, omega = *G.omega;
  FluidN const &F = N.f[0];
  BoundN const &B = N.b[0];
  f3 xi = {0.0f, 0.0f, 0.0f};
  float ri = 1.0f, pi = 0.0f;
  if (mine) {
    xi = mk3(A.x[i]);
    ri = A.rho[i];
    pi = A.p[i];
  }
  // what k_jacobi_begin does, by every block for itself; the flags are written
  // once every block has read them
  bool zero = zero_sums_hold(G, D, R.status, R.scalars, same);
  int ended = *G.nprde >= 1 ? 0 : 1;
  turn = meet_share(turn);
  if (turn & kGaveUp) return;
  if (ended && i == 0) {
    R.status[kStSetupBad] = 1;
    R.status[kStJacIter] = 0;
    R.status[kStJacDone] = 1;
    *G.jac_iters = 0;
  }
  bool begun = false;
  __shared__ double sh[32];
  __shared__ int s_ended;
  while (!ended) {
    f3 ai = {0.0f, 0.0f, 0.0f};
    float ap = 0.0f;
    if (mine && !zero) {
      float pri = pi / (ri * ri), bterm = (2.0f * pi) / (ri * ri);
      walk_nbrs_cached<kForm>(F.L, i, uc, [&](uint32_t j) { return WithRec<float>{__ldg(F.xm + j), F.pr[j]}; },
                              [&](WithRec<float> const &r, float gf, bool in, auto cached) {
        ai = sub_if(in, ai, scl3(r.x.w * (pri + r.v), pgrad(is_cached(cached), gf, K, sub3(xi, mk3(r.x)))));
      });
      walk_nbrs_cached<kForm>(B.L, i, uc, [&](uint32_t j) { return __ldg(B.xV + j); },
                              [&](float4 xv, float gf, bool in, auto cached) {
        ai = sub_if(in, ai, scl3(((0.7f * rho0) * xv.w) * bterm, pgrad(is_cached(cached), gf, K, sub3(xi, mk3(xv)))));
      });
    }
    if (mine) a[i] = make_float4(ai.x, ai.y, ai.z, 0.0f);
    // (with zero sums nobody reads an acceleration)
    if (!zero && !meet(M, turn, [] {})) break;
    double part = 0.0;
    if (mine) {
      if (!zero) {
        walk_nbrs_cached<kForm>(F.L, i, uc, [&](uint32_t j) { return WithRec<f3>{__ldg(F.xm + j), mk3(F.a[j])}; },
                                [&](WithRec<f3> const &r, float gf, bool in, auto cached) {
          ap = add_if(in, ap, r.x.w * dot3(sub3(ai, r.v), pgrad(is_cached(cached), gf, K, sub3(xi, mk3(r.x)))));
        });
        walk_nbrs_cached<kForm>(B.L, i, uc, [&](uint32_t j) { return __ldg(B.xV + j); },
                                [&](float4 xv, float gf, bool in, auto cached) {
          ap = add_if(in, ap, (rho0 * xv.w) * dot3(sub3(ai, f3{0.0f, 0.0f, 0.0f}),
                                                   pgrad(is_cached(cached), gf, K, sub3(xi, mk3(xv)))));
        });
      }
      part += pressure_finish(i, A, ap, rho0, dt, omega);
      pi = A.p[i];
    }
    // the density error, as reduce_commit sums it, and the loop's control
    double sum = block_sum(part, sh);
    if (threadIdx.x == 0) R.partials[blockIdx.x] = sum;
    bool ok = meet(M, turn, [&] {
      double acc = 0.0;
      for (unsigned b = threadIdx.x; b < gridDim.x; b += blockDim.x) acc += R.partials[b];
      acc = block_sum(acc, sh);
      if (threadIdx.x == 0) {
        acc = 0.0 + acc;
        R.scalars[kSJacobi] = acc;
        *G.aprde = float(acc);
        if (!begun) {
          R.status[kStSetupBad] = 1;
          R.status[kStJacIter] = 0;
          R.status[kStJacDone] = 0;
        }
        jacobi_control(G, R);
      }
    });
    begun = true;
    if (!ok) break;
    if (threadIdx.x == 0) s_ended = *(volatile int const *)&R.status[kStJacDone];
    __syncthreads();
    ended = s_ended;
    zero = false;
  }
}

// ---------------------------------------------------------------------------
// viscosity.accumulate_acceleration (share/schemes/viscosity.prtcl:31-66,
// generated schemes/viscosity.hpp:171-240): explicit viscosity added to a.
//   a_i += ((10 (mu_i / rho_i)) (m_j / rho_j) (v_i - v_j).x_ij / (|x_ij|^2 + 0.01 h^2)) gradW
//   a_i += ((10 (mu_b / rho_i)) (rho0 V_b / rho_i) v_i.x_ib / (|x_ib|^2 + 0.01 h^2)) gradW
// over the neighbours of every fluid group, then of every boundary group.
// The fluid records are (x, m / rho) (the packed xmr records: m_j / rho_j is
// the generated code's division).
// ---------------------------------------------------------------------------

template <int NF, int NB>
__global__ void __launch_bounds__(kNT, kMinBlocks) k_viscosity(uint32_t n, float4 const *__restrict__ x,
                                                               float4 const *__restrict__ v,
                                                               float const *__restrict__ rho, float4 *__restrict__ a,
                                                               float const *rho0p, float const *mup, Globals G,
                                                               Nbrs<NF, NB> N) {
  uint32_t i = grid_tid();
  if (i >= n) return;
  KernelParams K = kparams(*G.h);
  bool uc = use_cache(N, K);
  float h = K.h, rho0 = *rho0p, mu = *mup;
  float hh = (0.01f * h) * h;
  f3 xi = mk3(x[i]), vi = mk3(v[i]);
  float ri = rho[i];
  f3 ai, a0 = mk3(a[i]);
  Divisor rdiv = divisor(ri);
  bool flat = uc && hh >= 0x1p-40f && hh <= 0x1p40f, off; // (an item is its own neighbour, and divides by hh)
  do {
    ai = a0;
    off = false;
#pragma unroll
    for (int q = 0; q < NF; ++q) {
      FluidN const &F = N.f[q];
      walk_nbrs_flat<8>(F.L, i, flat, uc, [&](uint32_t j) { return WithRec<f3>{__ldg(F.xm + j), mk3(__ldg(F.v + j))}; },
                          [&](WithRec<f3> const &r, float gf, bool in, auto cached) {
        constexpr bool kFlat = std::is_same_v<decltype(cached), std::true_type>;
        f3 xij = sub3(xi, mk3(r.x));
        float coef = divide_noting<kFlat>(((10.0f * (mu / ri)) * r.x.w) * dot3(sub3(vi, r.v), xij), nsq3(xij) + hh, off);
        ai = add_if(in, ai, scl3(coef, pgrad(is_cached(cached), gf, K, xij)));
      });
    }
#pragma unroll
    for (int q = 0; q < NB; ++q) {
      BoundN const &B = N.b[q];
      float bmu = *B.mu;
      walk_nbrs_flat<8>(B.L, i, flat, uc, [&](uint32_t j) { return __ldg(B.xV + j); },
                          [&](float4 xv, float gf, bool in, auto cached) {
        constexpr bool kFlat = std::is_same_v<decltype(cached), std::true_type>;
        f3 xij = sub3(xi, mk3(xv));
        float vr = divide_noting<kFlat>(rho0 * xv.w, rdiv, off);
        float coef = divide_noting<kFlat>(((10.0f * (bmu / ri)) * vr) * dot3(sub3(vi, f3{0.0f, 0.0f, 0.0f}), xij),
                                          nsq3(xij) + hh, off);
        ai = add_if(in, ai, scl3(coef, pgrad(is_cached(cached), gf, K, xij)));
      });
    }
    if (!off) break;
    flat = false;
  } while (true);
  a[i] = make_float4(ai.x, ai.y, ai.z, 0.0f);
}

// ---------------------------------------------------------------------------
// WKBB18 (schemes/wkbb18.hpp)
// ---------------------------------------------------------------------------

// correction.compute_gradient_correction (share/schemes/correction.prtcl:
// 25-43, schemes/correction.hpp:162-230):
//   L_f = invert_pm(sum_{fluid neighbours} (m_j / rho_i) gradW(x_ij) (x_j - x_i)^T)
template <int NF, int NB>
__global__ void __launch_bounds__(kNT, kMinBlocks) k_correction(uint32_t n, uint32_t cap, float4 const *__restrict__ x,
                                                                float const *__restrict__ rho, float *__restrict__ L,
                                                                Globals G, Nbrs<NF, NB> N) {
  uint32_t i = grid_tid();
  if (i >= n) return;
  KernelParams K = kparams(*G.h);
  bool uc = use_cache(N, K);
  f3 xi = mk3(x[i]);
  float ri = rho[i];
  M3 A;
  Divisor rdiv = divisor(ri);
  bool flat = uc, off;
  do {
#pragma unroll
    for (int e = 0; e < 9; ++e) A.m[e] = 0.0f;
    off = false;
#pragma unroll
    for (int q = 0; q < NF; ++q) {
      FluidN const &F = N.f[q];
      walk_nbrs_cached<8>(F.L, i, flat, [&](uint32_t j) { return __ldg(F.xm + j); },
                          [&](float4 xm, float gf, bool in, auto cached) {
        constexpr bool kFlat = std::is_same_v<decltype(cached), std::true_type>;
        f3 xj = mk3(xm);
        f3 g = pgrad(is_cached(cached), gf, K, sub3(xi, xj));
        f3 d = sub3(xj, xi);
        float sc = divide_noting<kFlat>(xm.w, rdiv, off);
        float gv[3] = {g.x, g.y, g.z}, dv[3] = {d.x, d.y, d.z};
#pragma unroll
        for (int c = 0; c < 3; ++c)
#pragma unroll
          for (int r = 0; r < 3; ++r) A.m[3 * c + r] = add_if(in, A.m[3 * c + r], sc * (gv[r] * dv[c]));
      });
    }
    if (!off) break;
    flat = false;
  } while (true);
  M3 R = pinv3(A);
#pragma unroll
  for (int e = 0; e < 9; ++e) L[size_t(e) * cap + i] = R.m[e];
}

__global__ void k_identity9(uint32_t n, uint32_t cap, float *L) {
  uint32_t i = grid_tid();
  if (i < n)
#pragma unroll
    for (int e = 0; e < 9; ++e) L[size_t(e) * cap + i] = (e % 4 == 0) ? 1.0f : 0.0f;
}

// wkbb18.compute_diagonal (schemes/wkbb18.hpp:194-270): block-Jacobi
// preconditioner sp_i = (I - dt S_i)^-1, stored as 9 planes.  The fluid sum
// runs over the particle's own group (`foreach _ neighbor`); xmr holds
// (x, m / rho).
// GC (wkbb18_gc, share/schemes/wkbb18_gc.prtcl): every kernel gradient
// premultiplied by the item's gradient correction L_i (planar, capacity lcap)
template <int NB, bool GC = false, int NT = kNT, int MINB = kMinBlocks, int BT = 4 | kFill>
__global__ void __launch_bounds__(NT, MINB) k_wkbb18_diag(uint32_t n, uint32_t cap, float4 const *__restrict__ xmr,
                                                     float const *__restrict__ rho, float *__restrict__ sp,
                                                     float const *rho0p, float const *mup, Globals G, NbrList self,
                                                     Nbrs<0, NB> N, float const *__restrict__ Lc, uint32_t lcap) {
  uint32_t i = grid_tid();
  if (i >= n) return;
  KernelParams K = kparams(*G.h);
  bool uc = use_cache(N, K);
  float Li[9];
  if (GC)
#pragma unroll
    for (int e = 0; e < 9; ++e) Li[e] = Lc[size_t(e) * lcap + i];
  float h = K.h, dt = *G.dt, rho0 = *rho0p, mu = *mup;
  f3 xi = mk3(xmr[i]);
  float ri = rho[i];
  float S[9];
#pragma unroll
  for (int k = 0; k < 9; ++k) S[k] = 0.0f;
  float hh = (0.01f * h) * h;
  float cmu = 10.0f * (mu / ri);
  // (bound by its arithmetic: 113 us with divisions, 119 without their branches)
  walk_nbrs_cached<BT>(self, i, uc, [&](uint32_t j) { return __ldg(xmr + j); },
                       [&](float4 xj, float gf, bool in, auto cached) {
    f3 xij = sub3(xi, mk3(xj));
    float coef = (cmu * xj.w) / (nsq3(xij) + hh);
    f3 g = pgrad(is_cached(cached), gf, K, xij);
    if (GC) g = mv3(Li, g);
    float gv[3] = {g.x, g.y, g.z}, xv[3] = {xij.x, xij.y, xij.z};
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
      for (int r = 0; r < 3; ++r) S[3 * c + r] = add_if(in, S[3 * c + r], coef * (gv[r] * xv[c]));
  });
#pragma unroll
  for (int q = 0; q < NB; ++q) {
    BoundN const &B = N.b[q];
    float bmu = *B.mu;
    walk_nbrs_cached<BT>(B.L, i, uc, [&](uint32_t j) { return __ldg(B.xV + j); },
                         [&](float4 xv, float gf, bool in, auto cached) {
      f3 xij = sub3(xi, mk3(xv));
      float coef = ((10.0f * (bmu / ri)) * ((rho0 * xv.w) / ri)) / (nsq3(xij) + hh);
      f3 g = pgrad(is_cached(cached), gf, K, xij);
      if (GC) g = mv3(Li, g);
      float gv[3] = {g.x, g.y, g.z}, xw[3] = {xij.x, xij.y, xij.z};
#pragma unroll
      for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int r = 0; r < 3; ++r) S[3 * c + r] = add_if(in, S[3 * c + r], coef * (gv[r] * xw[c]));
    });
  }
  M3 A;
#pragma unroll
  for (int c = 0; c < 3; ++c)
#pragma unroll
    for (int r = 0; r < 3; ++r) A.m[3 * c + r] = (r == c ? 1.0f : 0.0f) - dt * S[3 * c + r];
  M3 inv = minv3(A);
#pragma unroll
  for (int k = 0; k < 9; ++k) sp[size_t(k) * cap + i] = inv.m[k];
}

// y = sp * r  (row . vector, a0 + (a1 + a2))
__device__ __forceinline__ f3 precond(float const *__restrict__ sp, uint32_t cap, uint32_t i, f3 r) {
  float s[9];
#pragma unroll
  for (int k = 0; k < 9; ++k) s[k] = sp[size_t(k) * cap + i];
  return {s[0] * r.x + (s[3] * r.y + s[6] * r.z), s[1] * r.x + (s[4] * r.y + s[7] * r.z),
          s[2] * r.x + (s[5] * r.y + s[8] * r.z)};
}

struct PcgArgs {
  uint32_t n, cap;
  float4 const *xmr; // (x, m / rho)
  float4 const *v;
  float const *rho;
  float const *sp;
  float const *tb;
  float4 *vd;
  float4 *a;
  float4 *X, *Y, *Rr, *P, *Q;
  float const *rho0, *mu, *tol;
  int const *max_k;
  int *iterations; // uniform wkbb18_iterations
  NbrList self;
  float const *L;  // gradient correction (wkbb18_gc), planar with capacity lcap
  uint32_t lcap;
};

// system product of wkbb18.accumulate_acceleration (schemes/wkbb18.hpp:
// 339-396): (A w)_i = w_i - dt * a_f(w)_i
// LOOP: w changes during the launch (its loads are ordered by the barriers)
template <int NB, bool GC, int BT = 8 | kAlone, bool LOOP = false>
__device__ __forceinline__ f3 wkbb18_system(PcgArgs const &P, KernelParams const &K, bool uc, float dt, float rho0,
                                            float mu, Nbrs<0, NB> const &N, float4 const *w, uint32_t i) {
  float Li[9];
  if (GC)
#pragma unroll
    for (int e = 0; e < 9; ++e) Li[e] = P.L[size_t(e) * P.lcap + i];
  float h = K.h;
  float hh = (0.01f * h) * h;
  f3 xi = mk3(P.xmr[i]), wi = mk3(w[i]);
  float ri = P.rho[i];
  float cmu = 10.0f * (mu / ri);
  Divisor rdiv = divisor(ri);
  f3 af;
  bool flat = uc, off;
  do {
    af = {0.0f, 0.0f, 0.0f};
    off = false;
    walk_nbrs_cached<BT>(P.self, i, flat, [&](uint32_t j) { return WithRec<f3>{__ldg(P.xmr + j), mk3(LOOP ? w[j] : __ldg(w + j))}; },
                         [&](WithRec<f3> const &r, float gf, bool in, auto cached) {
      constexpr bool kFlat = std::is_same_v<decltype(cached), std::true_type>;
      f3 xij = sub3(xi, mk3(r.x));
      float coef = divide_noting<kFlat>((cmu * r.x.w) * dot3(sub3(wi, r.v), xij), nsq3(xij) + hh, off);
      f3 g = pgrad(is_cached(cached), gf, K, xij);
      if (GC) g = mv3(Li, g);
      af = add_if(in, af, scl3(coef, g));
    });
#pragma unroll
    for (int q = 0; q < NB; ++q) {
      BoundN const &B = N.b[q];
      float bmu = *B.mu;
      float cb_mu = 10.0f * (bmu / ri);
      walk_nbrs_cached<BT>(B.L, i, flat, [&](uint32_t j) { return __ldg(B.xV + j); },
                           [&](float4 xv, float gf, bool in, auto cached) {
        constexpr bool kFlat = std::is_same_v<decltype(cached), std::true_type>;
        f3 xij = sub3(xi, mk3(xv));
        float vr = divide_noting<kFlat>(rho0 * xv.w, rdiv, off);
        float coef = divide_noting<kFlat>((cb_mu * vr) * dot3(wi, xij), nsq3(xij) + hh, off);
        f3 g = pgrad(is_cached(cached), gf, K, xij);
        if (GC) g = mv3(Li, g);
        af = add_if(in, af, scl3(coef, g));
      });
    }
    if (!off) break;
    flat = false;
  } while (true);
  return sub3(wi, scl3(dt, af));
}

// scalars: 0 b_nsq, 1 thr, 2 r_nsq, 3 next_rdy, 4 prev_rdy, 5 pdq,
// 6 alpha, 7 beta (f32 values held in double slots)
__global__ void k_pcg_guess(PcgArgs P) {
  uint32_t i = grid_tid();
  if (i < P.n) P.X[i] = P.v[i];
}

__device__ __forceinline__ void pcg_init_finish(PcgArgs const &P, uint32_t i, f3 ax, double &bb, double &rr,
                                                double &ry);
// the rest of pcg_q_item from q = A p: stores q, returns p . q
__device__ __forceinline__ double pcg_q_finish(PcgArgs const &P, uint32_t i, f3 q) {
  P.Q[i] = make_float4(q.x, q.y, q.z, 0.0f);
  return f2d(dot3(mk3(P.P[i]), q));
}

// r = A x - b (b = v: the right-hand side's boundary term has v_b = 0),
// y = M r, p = -y; dots b.b, r.r, r.y (solver/cg_openmp.hpp:48-96)
// per-item parts of the PCG kernels (shared by the plain and the tiled
// launches, so both compute the same values)
template <int NB, bool GC, int BT = 8 | kAlone>
__device__ __forceinline__ void pcg_init_item(PcgArgs const &P, KernelParams const &K, bool uc, float dt, float rho0,
                                              float mu, Nbrs<0, NB> const &N, uint32_t i, double &bb, double &rr,
                                              double &ry) {
  pcg_init_finish(P, i, wkbb18_system<NB, GC, BT>(P, K, uc, dt, rho0, mu, N, P.X, i), bb, rr, ry);
}
// the rest of pcg_init_item from A x
__device__ __forceinline__ void pcg_init_finish(PcgArgs const &P, uint32_t i, f3 ax, double &bb, double &rr,
                                                double &ry) {
  f3 b = mk3(P.v[i]);
  f3 r = sub3(ax, b);
  f3 y = precond(P.sp, P.cap, i, r);
  P.Rr[i] = make_float4(r.x, r.y, r.z, 0.0f);
  P.Y[i] = make_float4(y.x, y.y, y.z, 0.0f);
  P.P[i] = make_float4(-y.x, -y.y, -y.z, 0.0f);
  bb += f2d(dot3(b, b));
  rr += f2d(dot3(r, r));
  ry += f2d(dot3(r, y));
}
template <int NB, bool GC, int BT = 8 | kAlone, bool LOOP = false>
__device__ __forceinline__ double pcg_q_item(PcgArgs const &P, KernelParams const &K, bool uc, float dt, float rho0,
                                             float mu, Nbrs<0, NB> const &N, uint32_t i) {
  return pcg_q_finish(P, i, wkbb18_system<NB, GC, BT, LOOP>(P, K, uc, dt, rho0, mu, N, P.P, i));
}
__device__ __forceinline__ void pcg_update_item(PcgArgs const &P, float alpha, uint32_t i, double &rr, double &ry) {
  f3 x = mk3(P.X[i]), p = mk3(P.P[i]), r = mk3(P.Rr[i]), q = mk3(P.Q[i]);
  x = add3(x, scl3(alpha, p));
  r = add3(r, scl3(alpha, q));
  f3 y = precond(P.sp, P.cap, i, r);
  P.X[i] = make_float4(x.x, x.y, x.z, 0.0f);
  P.Rr[i] = make_float4(r.x, r.y, r.z, 0.0f);
  P.Y[i] = make_float4(y.x, y.y, y.z, 0.0f);
  rr += f2d(dot3(r, r));
  ry += f2d(dot3(r, y));
}
__device__ __forceinline__ void pcg_p_item(PcgArgs const &P, float beta, uint32_t i) {
  f3 y = mk3(P.Y[i]), p = mk3(P.P[i]);
  f3 r = add3(f3{-y.x, -y.y, -y.z}, scl3(beta, p));
  P.P[i] = make_float4(r.x, r.y, r.z, 0.0f);
}
// solver scalars after the initial residual (thr = max(tol^2 |b|^2, FLT_MIN))
__device__ __forceinline__ void pcg_init_scalars(double *sc, int *st, double const (&out)[3], float tol_f) {
  double tol = double(tol_f);
  sc[0] = out[0];
  double thr = tol * tol * out[0], fmin_ = double(1.17549435082228750797e-38f);
  sc[1] = (thr < fmin_) ? fmin_ : thr;
  sc[2] = out[1];
  sc[3] = out[2];
  st[kStPcgIter] = 0;
  st[kStPcgActive] = 1; // iteration 0 always runs (min_k = 1)
  st[kStPcgBody] = 0;
}
// after p.q: alpha, or stop on |p.q| < tol
__device__ __forceinline__ void pcg_q_scalars(double *sc, int *st, double pq, float tol) {
  double prev = sc[3];
  sc[4] = prev;
  sc[5] = pq;
  if (fabs(pq) < double(tol)) st[kStPcgActive] = 0;
  else sc[6] = double(float(prev / pq));
}
// after the update: stop on |r.y| < tol, else beta, k + 1 and the loop test
__device__ __forceinline__ void pcg_update_scalars(double *sc, int *st, double rr, double ry, float tol, int max_k) {
  double prev = sc[4];
  sc[2] = rr;
  sc[3] = ry;
  if (fabs(prev) < double(tol)) {
    st[kStPcgActive] = 0;
  } else {
    sc[7] = double(float(ry / prev));
    int k = st[kStPcgIter] + 1;
    st[kStPcgIter] = k;
    // loop condition ok(k, r_nsq): k < 1 -> run; k > max_k -> stop;
    // r_nsq < thr -> stop
    bool ok = (k < 1) || (!(k > max_k) && !(rr < sc[1]));
    st[kStPcgActive] = ok ? 1 : 0;
  }
}

template <int NB, bool GC = false, int MINB = kMinBlocks, int BT = 8 | kAlone>
__global__ void __launch_bounds__(kNT, MINB) k_pcg_init(PcgArgs P, Globals G, Nbrs<0, NB> N, Red R) {
  KernelParams K = kparams(*G.h);
  bool uc = use_cache(N, K);
  float dt = *G.dt, rho0 = *P.rho0, mu = *P.mu;
  double bb = 0.0, rr = 0.0, ry = 0.0;
  for (uint32_t i = grid_tid(); i < P.n; i += gridDim.x * blockDim.x)
    pcg_init_item<NB, GC, BT>(P, K, uc, dt, rho0, mu, N, i, bb, rr, ry);
  double v[3] = {bb, rr, ry}, out[3];
  if (reduce_commit<3>(v, R, out) && threadIdx.x == 0) pcg_init_scalars(R.scalars + kSPcg, R.status, out, *P.tol);
}

// q = A p; p.q; alpha or break (solver/cg_openmp.hpp:121-151)
template <int NB, bool GC = false, int MINB = kMinBlocks, int BT = 8 | kAlone>
__global__ void __launch_bounds__(kNT, MINB) k_pcg_q(PcgArgs P, Globals G, Nbrs<0, NB> N, Red R) {
  if (!*(volatile int *)&R.status[kStPcgActive]) return;
  KernelParams K = kparams(*G.h);
  bool uc = use_cache(N, K);
  float dt = *G.dt, rho0 = *P.rho0, mu = *P.mu;
  double pq = 0.0;
  for (uint32_t i = grid_tid(); i < P.n; i += gridDim.x * blockDim.x)
    pq += pcg_q_item<NB, GC, BT>(P, K, uc, dt, rho0, mu, N, i);
  double v[1] = {pq}, out[1];
  if (reduce_commit<1>(v, R, out) && threadIdx.x == 0) pcg_q_scalars(R.scalars + kSPcg, R.status, out[0], *P.tol);
}

// the system product from staged lists (one boundary group, no gradient
// correction): the staged records are a fluid item's (x, m / rho) and w, a
// boundary item's (x, V); terms and order those of wkbb18_system
template <int BT = 8>
__device__ __forceinline__ f3 wkbb18_system_staged(PcgArgs const &P, KernelParams const &K, bool uc, float dt,
                                                   float rho0, float mu, float bmu, StageArgs const &SA,
                                                   BoundN const &B, float4 const *sx, float4 const *sy,
                                                   float4 const *__restrict__ w, uint32_t i) {
  float h = K.h;
  float hh = (0.01f * h) * h;
  f3 xi = mk3(P.xmr[i]), wi = mk3(w[i]);
  float ri = P.rho[i];
  float cmu = 10.0f * (mu / ri);
  f3 af = {0.0f, 0.0f, 0.0f};
  for_each_staged<BT>(P.self, SA.fslots, i, [&](uint32_t sl, float gf_) {
    float4 xj = sx[sl];
    f3 xij = sub3(xi, mk3(xj));
    float coef = ((cmu * xj.w) * dot3(sub3(wi, mk3(sy[sl])), xij)) / (nsq3(xij) + hh);
    af = add3(af, scl3(coef, pgrad(uc, gf_, K, xij)));
  });
  float cb_mu = 10.0f * (bmu / ri);
  for_each_staged<BT>(B.L, SA.bslots, i, [&](uint32_t sl, float gf_) {
    float4 xv = sx[sl];
    f3 xij = sub3(xi, mk3(xv));
    float coef = ((cb_mu * ((rho0 * xv.w) / ri)) * dot3(wi, xij)) / (nsq3(xij) + hh);
    af = add3(af, scl3(coef, pgrad(uc, gf_, K, xij)));
  });
  return sub3(wi, scl3(dt, af));
}

// stages tile `tile` for the system product with vector w
__device__ __forceinline__ bool stage_system(StageArgs const &SA, uint32_t tile, float4 *sx, float4 *sy,
                                             PcgArgs const &P, BoundN const &B, float4 const *w) {
  // fluid: (x, m / rho) and w; boundary: (x, V)
  return stage_copy(SA, tile, sx, sy, [&](uint32_t h, float4 *dx, float4 *dy) {
    uint32_t j = h & 0x0FFFFFFFu;
    if (int(h >> 28) == SA.fg) {
      cp_async16(dx, P.xmr + j);
      cp_async16(dy, w + j);
    } else if (int(h >> 28) == SA.bg) {
      cp_async16(dx, B.xV + j);
    }
  });
}

// staged k_pcg_init / k_pcg_q (the `staging` knob): a block's tiles are the
// items of the plain kernels' grid-stride loop, so the FP64 sums are the same
template <int BT = 8>
__global__ void __launch_bounds__(kNT, 4) k_pcg_init_staged(PcgArgs P, Globals G, Nbrs<0, 1> N, Red R, StageArgs SA) {
  extern __shared__ float4 sm[];
  float4 *sx = sm, *sy = sm + kStageCap;
  KernelParams K = kparams(*G.h);
  bool uc = use_cache(N, K);
  float dt = *G.dt, rho0 = *P.rho0, mu = *P.mu;
  BoundN const &B = N.b[0];
  float bmu = *B.mu;
  double bb = 0.0, rr = 0.0, ry = 0.0;
  for (uint32_t tile = blockIdx.x; size_t(tile) * kNT < P.n; tile += gridDim.x) {
    uint32_t i = tile * kNT + threadIdx.x;
    bool st = stage_system(SA, tile, sx, sy, P, B, P.X);
    if (i < P.n) {
      if (st)
        pcg_init_finish(P, i, wkbb18_system_staged<BT>(P, K, uc, dt, rho0, mu, bmu, SA, B, sx, sy, P.X, i), bb, rr,
                        ry);
      else
        pcg_init_item<1, false, 8 | kAlone>(P, K, uc, dt, rho0, mu, N, i, bb, rr, ry);
    }
    __syncthreads();
  }
  double v[3] = {bb, rr, ry}, out[3];
  if (reduce_commit<3>(v, R, out) && threadIdx.x == 0) pcg_init_scalars(R.scalars + kSPcg, R.status, out, *P.tol);
}

template <int BT = 8>
__global__ void __launch_bounds__(kNT, 4) k_pcg_q_staged(PcgArgs P, Globals G, Nbrs<0, 1> N, Red R, StageArgs SA) {
  if (!*(volatile int *)&R.status[kStPcgActive]) return;
  extern __shared__ float4 sm[];
  float4 *sx = sm, *sy = sm + kStageCap;
  KernelParams K = kparams(*G.h);
  bool uc = use_cache(N, K);
  float dt = *G.dt, rho0 = *P.rho0, mu = *P.mu;
  BoundN const &B = N.b[0];
  float bmu = *B.mu;
  double pq = 0.0;
  for (uint32_t tile = blockIdx.x; size_t(tile) * kNT < P.n; tile += gridDim.x) {
    uint32_t i = tile * kNT + threadIdx.x;
    bool st = stage_system(SA, tile, sx, sy, P, B, P.P);
    if (i < P.n)
      pq += st ? pcg_q_finish(P, i, wkbb18_system_staged<BT>(P, K, uc, dt, rho0, mu, bmu, SA, B, sx, sy, P.P, i))
               : pcg_q_item<1, false, 8 | kAlone>(P, K, uc, dt, rho0, mu, N, i);
    __syncthreads();
  }
  double v[1] = {pq}, out[1];
  if (reduce_commit<1>(v, R, out) && threadIdx.x == 0) pcg_q_scalars(R.scalars + kSPcg, R.status, out[0], *P.tol);
}

// q = A p as a cell-tile sweep (the pcg_q knob's shape 4): no neighbour
// lists.  A block stages, per tile of 128 consecutive fluid items, the
// packed records of every cell adjacent to the tile's cells in shared
// memory (position and handle; the search direction and m / rho for a fluid
// item, the volume for a boundary item), and each thread walks its 27 cells
// in the lists' traversal order (own cell, adjacency slots 0..25, sorted
// order within a cell), fluid items first, then boundary items, testing
// every candidate with the exact d^2 < T of the list build and computing the
// gradient factor with the same operations.  The terms and their order are
// those of wkbb18_system, so q is bit-identical; the grid and the
// item-to-thread mapping are those of k_pcg_q, so the FP64 sum of p . q is
// too.  A tile whose cells hold more than kTileStage items (or more than
// kTileHash cells) takes the list walk instead.
constexpr int kTileStage = 1536; // staged items per tile (2 x 16 bytes each)
constexpr int kTileHash = 512;   // cells per tile (open-addressing table)

__device__ __forceinline__ uint32_t tile_hash(int c) { return (uint32_t(c) * 2654435761u) >> 23; } // 9 bits

// slot of cell c in the tile's table (the cell is present)
__device__ __forceinline__ int tile_find(int const *hkey, int c) {
  uint32_t h = tile_hash(c);
  for (int probe = 0; probe < kTileHash; ++probe) {
    int slot = int((h + uint32_t(probe)) & (kTileHash - 1));
    if (hkey[slot] == c) return slot;
  }
  return -1;
}

template <int NB>
__global__ void __launch_bounds__(kNT, 4) k_pcg_q_tiles(PcgArgs P, Globals G, Nbrs<0, NB> N, Red R, GridView gv,
                                                         float4 const *__restrict__ xs, int fg, int bg) {
  static_assert(NB == 1, "the cell-tile sweep handles one boundary group");
  if (!*(volatile int *)&R.status[kStPcgActive]) return;
  extern __shared__ float4 stage[]; // [kTileStage] records, then [kTileStage] payloads
  __shared__ int hkey[kTileHash];
  __shared__ uint32_t hval[kTileHash]; // base << 16 | count
  __shared__ int homes[kNT];
  __shared__ uint32_t wsum[kNT / 32], wocc[kNT / 32];
  __shared__ int ccell[kTileHash];     // occupied slots' cells, compacted
  __shared__ uint32_t cbase[kTileHash]; // and their staged bases (ascending)
  __shared__ int s_over, s_cells;
  float4 *pay = stage + kTileStage;
  KernelParams K = kparams(*G.h);
  bool uc = use_cache(N, K);
  float dt = *G.dt, rho0 = *P.rho0, mu = *P.mu;
  float hh = (0.01f * K.h) * K.h;
  BoundN const &B = N.b[0];
  float bmu = *B.mu;
  double pq = 0.0;
  for (uint32_t tile = blockIdx.x; size_t(tile) * kNT < P.n; tile += gridDim.x) {
    uint32_t i = tile * kNT + threadIdx.x;
    bool has = i < P.n;
    for (int sl = threadIdx.x; sl < kTileHash; sl += kNT) {
      hkey[sl] = -1;
      hval[sl] = 0u;
    }
    if (threadIdx.x == 0) s_over = 0;
    int home = has ? gv.s2c[gv.r2s[gv.goff[fg] + i]] : -1;
    homes[threadIdx.x] = home;
    __syncthreads();
    // the first item of each run of equal home cells enters the run's 27 cells
    if (has && (threadIdx.x == 0 || homes[threadIdx.x - 1] != home)) {
      for (int k = -1; k < 26; ++k) {
        int c = k < 0 ? home : gv.cell_adj[size_t(home) * 26 + k];
        if (c < 0) continue;
        uint32_t h = tile_hash(c);
        bool placed = false;
        for (int probe = 0; probe < kTileHash && !placed; ++probe) {
          int slot = int((h + uint32_t(probe)) & (kTileHash - 1));
          int old = atomicCAS(&hkey[slot], -1, c);
          placed = old == -1 || old == c;
        }
        if (!placed) s_over = 1;
      }
    }
    __syncthreads();
    // staged ranges: each thread owns table slots tid, tid + 128, ...
    uint32_t cnt[kTileHash / kNT], mine = 0;
#pragma unroll
    for (int m = 0; m < kTileHash / kNT; ++m) {
      int c = hkey[threadIdx.x + m * kNT];
      cnt[m] = c >= 0 ? uint32_t(gv.cell_start[c + 1] - gv.cell_start[c]) : 0u;
      mine += cnt[m];
    }
    // block-exclusive prefix of the per-thread counts
    uint32_t incl = mine;
    int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    if (lane == 31) wsum[w] = incl;
    __syncthreads();
    uint32_t off = incl - mine, total = 0;
    for (int k = 0; k < kNT / 32; ++k) {
      if (k < w) off += wsum[k];
      total += wsum[k];
    }
    if (total > uint32_t(kTileStage)) s_over = 1;
    __syncthreads();
    bool over = s_over != 0;
    if (!over) {
      // bases in (thread, m) order, and the occupied slots compacted in the
      // same order, so that the compacted bases ascend
      uint32_t occ = 0;
#pragma unroll
      for (int m = 0; m < kTileHash / kNT; ++m) occ += hkey[threadIdx.x + m * kNT] >= 0 ? 1u : 0u;
      uint32_t oincl = occ;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        uint32_t v = __shfl_up_sync(0xffffffffu, oincl, o);
        if (lane >= o) oincl += v;
      }
      if (lane == 31) wocc[w] = oincl;
      __syncthreads();
      uint32_t u = oincl - occ;
      for (int k = 0; k < w; ++k) u += wocc[k];
#pragma unroll
      for (int m = 0; m < kTileHash / kNT; ++m) {
        int sl = threadIdx.x + m * kNT;
        int c = hkey[sl];
        if (c >= 0) {
          hval[sl] = (off << 16) | cnt[m];
          ccell[u] = c;
          cbase[u] = off;
          off += cnt[m];
          ++u;
        }
      }
      if (threadIdx.x == kNT - 1) s_cells = u;
    }
    __syncthreads();
    if (!over) {
      // every thread copies staged items p = tid, tid + 128, ...: the cell of
      // p is the last compacted cell whose base is <= p
      int ncel = s_cells;
      for (uint32_t pidx = threadIdx.x; pidx < total; pidx += kNT) {
        int lo = 0, hi = ncel - 1;
        while (lo < hi) {
          int mid = (lo + hi + 1) >> 1;
          if (cbase[mid] <= pidx) lo = mid;
          else hi = mid - 1;
        }
        int c = ccell[lo];
        uint32_t e = pidx - cbase[lo];
        float4 X = xs[gv.cell_start[c] + int(e)];
        uint32_t hd = __float_as_uint(X.w);
        int g = int(hd >> 28);
        uint32_t j = hd & 0x0FFFFFFFu;
        float4 W = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (g == fg) {
          float4 pj = P.P[j];
          W = make_float4(pj.x, pj.y, pj.z, P.xmr[j].w);
        } else if (g == bg) {
          W.w = B.xV[j].w;
        }
        stage[pidx] = X;
        pay[pidx] = W;
      }
    }
    __syncthreads();
    if (has) {
      f3 q;
      if (over) {
        q = wkbb18_system<NB, false, 8 | kAlone>(P, K, uc, dt, rho0, mu, N, P.P, i);
      } else {
        f3 xi = mk3(P.xmr[i]), wi = mk3(P.P[i]);
        float ri = P.rho[i];
        float cmu = 10.0f * (mu / ri);
        float cb_mu = 10.0f * (bmu / ri);
        f3 af = {0.0f, 0.0f, 0.0f};
        // fluid neighbours (the group's own lists), then boundary neighbours
        for (int pass = 0; pass < 2; ++pass) {
          int want = pass == 0 ? fg : bg;
          for (int k = -1; k < 26; ++k) {
            int c = k < 0 ? home : gv.cell_adj[size_t(home) * 26 + k];
            if (c < 0) continue;
            int sl = tile_find(hkey, c); // present: the run's first item entered it
            uint32_t hv = sl >= 0 ? hval[sl] : 0u;
            uint32_t b0 = hv >> 16, b1 = b0 + (hv & 0xFFFFu);
            for (uint32_t e = b0; e < b1; ++e) {
              float4 X = stage[e];
              if (int(__float_as_uint(X.w) >> 28) != want) continue;
              f3 xij = sub3(xi, mk3(X));
              float d2 = nsq3(xij);
              if (!(d2 < gv.r2lt)) continue;
              float4 W = pay[e];
              f3 g = kgrad_from(kgrad_factor(K, d2), xij);
              float coef;
              if (pass == 0) coef = ((cmu * W.w) * dot3(sub3(wi, mk3(W)), xij)) / (nsq3(xij) + hh);
              else coef = ((cb_mu * ((rho0 * W.w) / ri)) * dot3(wi, xij)) / (nsq3(xij) + hh);
              af = add3(af, scl3(coef, g));
            }
          }
        }
        q = sub3(wi, scl3(dt, af));
      }
      P.Q[i] = make_float4(q.x, q.y, q.z, 0.0f);
      pq += f2d(dot3(mk3(P.P[i]), q));
    }
    __syncthreads(); // the next tile reuses the shared memory
  }
  double v[1] = {pq}, out[1];
  if (reduce_commit<1>(v, R, out) && threadIdx.x == 0) pcg_q_scalars(R.scalars + kSPcg, R.status, out[0], *P.tol);
}

// x += alpha p; r += alpha q; y = M r; r.r; r.y; break / beta
// (solver/cg_openmp.hpp:153-191)
__global__ void __launch_bounds__(kNT, kMinBlocks) k_pcg_update(PcgArgs P, Red R) {
  if (!*(volatile int *)&R.status[kStPcgActive]) return;
  float alpha = float(R.scalars[kSPcg + 6]);
  double rr = 0.0, ry = 0.0;
  // (two items' loads in flight together, 34.6 -> 32.4 us at 1M items; with the
  // two sums in one tree, the 1M diagonal and solve 1196 -> 1167 us)
#pragma unroll 2
  for (uint32_t i = grid_tid(); i < P.n; i += gridDim.x * blockDim.x) pcg_update_item(P, alpha, i, rr, ry);
  double v[2] = {rr, ry}, out[2];
  if (reduce_commit<2>(v, R, out) && threadIdx.x == 0)
    pcg_update_scalars(R.scalars + kSPcg, R.status, out[0], out[1], *P.tol, *P.max_k);
}

// p = -y + beta p (only when the loop continues)
__global__ void k_pcg_p(PcgArgs P, Red R) {
  if (!*(volatile int *)&R.status[kStPcgActive]) return;
  float beta = float(R.scalars[kSPcg + 7]);
  for (uint32_t i = grid_tid(); i < P.n; i += gridDim.x * blockDim.x) pcg_p_item(P, beta, i);
}

// loop control of the device PCG loop: continue while active, and never run
// more than max_k + 1 bodies
// (one thread; returns whether the loop goes on)
__device__ bool pcg_control(PcgArgs const &P, Red const &R) {
  int body = R.status[kStPcgBody] + 1;
  R.status[kStPcgBody] = body;
  int maxk = *P.max_k;
  bool cont = R.status[kStPcgActive] && body < (maxk < 0 ? 0 : maxk) + 1 && body < 1000000;
  if (!cont) {
    R.stats[4] += 1.0;
    R.stats[5] += double(R.status[kStPcgIter]);
    if (R.status[kStPcgActive]) R.stats[6] += 1.0;
    R.status[kStPcgActive] = 0;
  }
  return cont;
}
__global__ void k_pcg_control(PcgArgs P, Red R, cudaGraphConditionalHandle h, int use_handle, int kernels) {
  bool cont = pcg_control(P, R);
  if (kernels) atomicAdd(&g_loop_kernels, (unsigned long long)kernels);
  if (use_handle) cudaGraphSetConditional(h, cont ? 1u : 0u);
}

// The PCG loop of a small scene in one cooperative launch, as k_jacobi_loop is
// of the Jacobi loop: three barriers where the graph's loop has four launches
// and a turn.  Diagonal and solve 89 -> 77 us at 2k items, 124 -> 110 at 27k, 146
// -> 136 at 60k (with gradient correction 239 -> 230).
template <bool GC>
__global__ void __launch_bounds__(kNT, 4) k_pcg_loop(PcgArgs P, Globals G, Nbrs<0, 1> N, Red R, Meet M) {
  uint32_t i = grid_tid();
  unsigned turn = meet_read(M);
  bool mine = i < P.n;
  KernelParams K = kparams(*G.h);
  bool uc = use_cache(N, K);
  float dt = *G.dt, rho0 = *P.rho0, mu = *P.mu;
  double volatile const *sc = R.scalars + kSPcg;
  int volatile const *active = &R.status[kStPcgActive];
  turn = meet_share(turn);
  if (turn & kGaveUp) return;
  __shared__ double sh[32];
  // the sums of the block that arrives last, as reduce_commit forms them
  auto total = [&](int k) {
    double acc = 0.0;
    for (unsigned b = threadIdx.x; b < gridDim.x; b += blockDim.x) acc += R.partials[k * kMaxRedBlocks + b];
    return block_sum(acc, sh);
  };
  auto partial = [&](int k, double v) {
    double t = block_sum(v, sh);
    if (threadIdx.x == 0) R.partials[k * kMaxRedBlocks + blockIdx.x] = t;
  };
  bool ok = true;
  while (ok && *active) {
    partial(0, mine ? 0.0 + pcg_q_item<1, GC, 8 | kAhead, true>(P, K, uc, dt, rho0, mu, N, i) : 0.0);
    ok = meet(M, turn, [&] {
      double pq = total(0);
      if (threadIdx.x == 0) {
        pcg_q_scalars(R.scalars + kSPcg, R.status, pq, *P.tol);
        if (!R.status[kStPcgActive]) pcg_control(P, R);
      }
    });
    if (!ok || !*active) break;
    double rr = 0.0, ry = 0.0;
    if (mine) pcg_update_item(P, float(sc[6]), i, rr, ry);
    partial(0, rr);
    partial(1, ry);
    ok = meet(M, turn, [&] {
      double t0 = total(0), t1 = total(1);
      if (threadIdx.x == 0) {
        pcg_update_scalars(R.scalars + kSPcg, R.status, t0, t1, *P.tol, *P.max_k);
        pcg_control(P, R);
      }
    });
    if (!ok || !*active) break;
    if (mine) pcg_p_item(P, float(sc[7]), i);
    ok = meet(M, turn, [] {});
  }
}

// --- the PCG loop over the tiles of a batched model, per slot -------------

template <int NB, bool GC = false, int MINB = kMinBlocks, int BT = 8 | kAlone>
__global__ void __launch_bounds__(kNT, MINB) k_pcg_init_seg(PcgArgs P, Globals G, Nbrs<0, NB> N, SegArgs S) {
  uint4 T = S.tiles[blockIdx.x];
  uint32_t slot = T.x;
  KernelParams K = kparams(*G.h);
  bool uc = use_cache(N, K);
  float dt = *G.dt, rho0 = *P.rho0, mu = *P.mu;
  double bb = 0.0, rr = 0.0, ry = 0.0;
  uint32_t i = T.y + threadIdx.x;
  if (i < T.z) pcg_init_item<NB, GC, BT>(P, K, uc, dt, rho0, mu, N, i, bb, rr, ry);
  double v[3] = {bb, rr, ry}, out[3];
  if (seg_commit<3>(v, S, slot, out, blockIdx.x) && threadIdx.x == 0) {
    int *st = S.stat + slot * kSegStat;
    pcg_init_scalars(S.scal + slot * kSegScal, st, out, *P.tol);
    st[kStPcgEnded] = 0;
  }
}

template <int NB, bool GC = false, int MINB = kMinBlocks, int BT = 8 | kAlone>
__global__ void __launch_bounds__(kNT, MINB) k_pcg_q_seg(PcgArgs P, Globals G, Nbrs<0, NB> N, SegArgs S) {
  uint4 T = S.tiles[blockIdx.x];
  uint32_t slot = T.x;
  if (!S.stat[slot * kSegStat + kStPcgActive]) return;
  KernelParams K = kparams(*G.h);
  bool uc = use_cache(N, K);
  float dt = *G.dt, rho0 = *P.rho0, mu = *P.mu;
  uint32_t i = T.y + threadIdx.x;
  double v[1] = {(i < T.z) ? pcg_q_item<NB, GC, BT>(P, K, uc, dt, rho0, mu, N, i) : 0.0}, out[1];
  if (seg_commit<1>(v, S, slot, out, blockIdx.x) && threadIdx.x == 0)
    pcg_q_scalars(S.scal + slot * kSegScal, S.stat + slot * kSegStat, out[0], *P.tol);
}

__global__ void __launch_bounds__(kNT, kMinBlocks) k_pcg_update_seg(PcgArgs P, SegArgs S) {
  uint4 T = S.tiles[blockIdx.x];
  uint32_t slot = T.x;
  if (!S.stat[slot * kSegStat + kStPcgActive]) return;
  float alpha = float(S.scal[slot * kSegScal + 6]);
  double rr = 0.0, ry = 0.0;
  // one warp per tile (kSegUpdateNT): each lane folds four items before the
  // FP64 tree, which this GPU's narrow FP64 pipe makes the costly part
  for (uint32_t i = T.y + threadIdx.x; i < T.z; i += blockDim.x) pcg_update_item(P, alpha, i, rr, ry);
  double v[2] = {rr, ry}, out[2];
  if (seg_commit<2>(v, S, slot, out, blockIdx.x) && threadIdx.x == 0)
    pcg_update_scalars(S.scal + slot * kSegScal, S.stat + slot * kSegStat, out[0], out[1], *P.tol, *P.max_k);
}

__global__ void k_pcg_p_seg(PcgArgs P, SegArgs S) {
  uint32_t i = grid_tid();
  if (i >= P.n) return;
  uint32_t slot = S.seg[i];
  if (!S.stat[slot * kSegStat + kStPcgActive]) return;
  pcg_p_item(P, float(S.scal[slot * kSegScal + 7]), i);
}

// per-slot PCG loop control (the rule of k_pcg_control, per slot); one
// block.  stats per slot: 4 solves, 5 iterations, 6 solves stopped by the
// iteration limit
__global__ void k_seg_pcg_control(PcgArgs P, SegArgs S, cudaGraphConditionalHandle h, int use_handle, int kernels,
                                  int *any_active) {
  int any = 0;
  int maxk = *P.max_k;
  for (uint32_t k = threadIdx.x; k < S.slots; k += blockDim.x) {
    int *st = S.stat + k * kSegStat;
    if (st[kStPcgEnded]) continue;
    int body = st[kStPcgBody] + 1;
    st[kStPcgBody] = body;
    bool cont = st[kStPcgActive] && body < (maxk < 0 ? 0 : maxk) + 1 && body < 1000000;
    if (!cont) {
      double *sv = S.stats + k * kSegStats;
      sv[4] += 1.0;
      sv[5] += double(st[kStPcgIter]);
      if (st[kStPcgActive]) sv[6] += 1.0;
      st[kStPcgActive] = 0;
      st[kStPcgEnded] = 1;
      S.iters[k] = st[kStPcgIter];
    }
    any |= cont ? 1 : 0;
  }
  any = __syncthreads_or(any);
  if (threadIdx.x == 0) {
    *any_active = any;
    if (kernels) atomicAdd(&g_loop_kernels, (unsigned long long)kernels);
    if (use_handle) cudaGraphSetConditional(h, any ? 1u : 0u);
  }
}

// slots without fluid items take no part in the loop
__global__ void k_seg_pcg_begin(SegArgs S) {
  for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < S.slots; k += gridDim.x * blockDim.x) {
    int *st = S.stat + k * kSegStat;
    if (S.slot_tiles[k] == S.slot_tiles[k + 1]) {
      st[kStPcgActive] = 0;
      st[kStPcgEnded] = 1;
      st[kStPcgIter] = 0;
      S.iters[k] = 0;
    }
  }
}

// apply (schemes/wkbb18.hpp:401-413): vd = (x - v) [0 < (t - t_b) - fade];
// a = vd / dt
__global__ void k_pcg_apply(PcgArgs P, Globals G, Red R) {
  uint32_t i = grid_tid();
  bool keep = gave_up(G);
  if (i == 0 && R.status && !keep) *P.iterations = R.status[kStPcgIter];
  if (i >= P.n) return;
  float dt = *G.dt, t = *G.t, fade = *G.fade;
  float u = ustep(0.0f, (t - P.tb[i]) - fade);
  f3 d = scl3(u, sub3(mk3(P.X[i]), mk3(P.v[i])));
  if (keep) return;
  P.vd[i] = make_float4(d.x, d.y, d.z, 0.0f);
  P.a[i] = make_float4(d.x / dt, d.y / dt, d.z / dt, 0.0f);
}

// ---------------------------------------------------------------------------
// host helpers
// ---------------------------------------------------------------------------

FieldType ft_real() { return FieldType{}; }
FieldType ft_vec3() {
  FieldType t;
  t.rank = 1;
  t.ext[0] = 3;
  return t;
}
FieldType ft_mat3() {
  FieldType t;
  t.rank = 2;
  t.ext[0] = 3;
  t.ext[1] = 3;
  return t;
}
FieldType ft_int() {
  FieldType t;
  t.ctype = CType::I32;
  return t;
}

template <class T> T *dptr(VaryingField *f) { return static_cast<T *>(f->d); }

// dispatch on the number of fluid (1..2) and boundary (0..2) neighbour groups
template <template <int, int> class F, class... A> void dispatch_fb(int nf, int nb, A &&...a) {
  if (nf == 1 && nb == 1) return F<1, 1>::go(a...);
  if (nf == 1 && nb == 0) return F<1, 0>::go(a...);
  if (nf == 1 && nb == 2) return F<1, 2>::go(a...);
  if (nf == 2 && nb == 1) return F<2, 1>::go(a...);
  if (nf == 2 && nb == 0) return F<2, 0>::go(a...);
  if (nf == 2 && nb == 2) return F<2, 2>::go(a...);
  throw Error("unsupported group configuration: " + std::to_string(nf) + " fluid and " + std::to_string(nb) +
              " boundary groups (1..2 and 0..2 are supported)");
}

// A CUDA graph holding one conditional while node; the body is captured from
// the launches `body(stream, handle)` queues.  Rebuilt when the signature
// (the bytes of every kernel argument of the body) changes.
class WhileLoop {
public:
  ~WhileLoop() { reset(); }
  void reset() {
    if (exec_) cudaGraphExecDestroy(exec_);
    if (graph_) cudaGraphDestroy(graph_);
    exec_ = nullptr;
    graph_ = nullptr;
    sig_.clear();
  }
  template <class Body> void run(cudaStream_t s, std::string const &sig, Body &&body) {
    if (!exec_ || sig != sig_) {
      reset();
      PG_CUDA(cudaGraphCreate(&graph_, 0));
      cudaGraphConditionalHandle h;
      PG_CUDA(cudaGraphConditionalHandleCreate(&h, graph_, 1, cudaGraphCondAssignDefault));
      cudaGraphNodeParams p{};
      p.type = cudaGraphNodeTypeConditional;
      p.conditional.handle = h;
      p.conditional.type = cudaGraphCondTypeWhile;
      p.conditional.size = 1;
      cudaGraphNode_t node;
      PG_CUDA(cudaGraphAddNode(&node, graph_, nullptr, nullptr, 0, &p));
      cudaGraph_t bodyg = p.conditional.phGraph_out[0];
      cudaStream_t cs;
      PG_CUDA(cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking));
      PG_CUDA(cudaStreamBeginCaptureToGraph(cs, bodyg, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal));
      uint64_t counted = launch_count();
      try {
        body(cs, h);
      } catch (...) {
        cudaGraph_t dummy;
        cudaStreamEndCapture(cs, &dummy);
        cudaStreamDestroy(cs);
        reset();
        throw;
      }
      uncount_launches(launch_count() - counted); // captured, not launched
      cudaGraph_t out;
      cudaError_t err = cudaStreamEndCapture(cs, &out);
      cudaStreamDestroy(cs);
      PG_CUDA(err);
      PG_CUDA(cudaGraphInstantiate(&exec_, graph_, 0));
      sig_ = sig;
      builds++;
    }
    PG_CUDA(cudaGraphLaunch(exec_, s));
  }
  int builds = 0;

private:
  cudaGraph_t graph_ = nullptr;
  cudaGraphExec_t exec_ = nullptr;
  std::string sig_;
};

template <class T> void sig_add(std::string &s, T const &v) { s.append(reinterpret_cast<char const *>(&v), sizeof(T)); }

} // namespace

// ===========================================================================
// Tuning knobs
// ===========================================================================

char const *tune_knob_name(int k) {
  static char const *names[kTuneKnobs] = {"density", "iisph_setup", "iisph_accel", "iisph_pressure",
                                          "wkbb18_diag", "pcg_init", "pcg_q", "jacobi_unroll", "staging",
                                          "grid_sort", "list_split"};
  return (k >= 0 && k < kTuneKnobs) ? names[k] : "";
}
int tune_knob_find(std::string const &name) {
  for (int k = 0; k < kTuneKnobs; ++k)
    if (name == tune_knob_name(k)) return k;
  return -1;
}
bool tune_value_ok(int k, int v) {
  if (k == kTuneJacobiUnroll) return v == 1 || v == 2 || v == 4;
  if (k == kTuneStaging || k == kTuneGridSort || k == kTuneListSplit) return v == 0 || v == 1;
  if (k == kTunePcgQ) return v >= 0 && v <= 4; // 4: the cell-tile sweep
  // 4: the persistent tiled sweeps of a batched model (work counter)
  if (k == kTuneAccel || k == kTunePressure) return v >= 0 && v <= 4;
  return k >= 0 && k < kTuneKnobs && v >= 0 && v <= 3;
}
std::string tune_knob_table() {
  // shapes as threads-per-block x blocks-per-SM / walk batch, form of the walk
  // (b: a branch per entry; without: f records filled in past a row's end, p
  // predicated off, a entries loaded ahead), and what stands for value 0 at
  // some sizes
  std::string t, small = " small: " + shape_text<SmallShape>() + " to " + std::to_string(kSmallItems);
  std::string from = " from " + std::to_string(kSpreadItems);
  t += "density 0 " + shapes_text<DensityShapes>() + " unordered: " + shape_text<DensitySpread>() + from + "\n";
  t += "iisph_setup 0 " + shapes_text<SetupShapes>() + small + "\n";
  t += "iisph_accel 0 " + shapes_text<AccelShapes>() + small + " batched: " + shapes_text<AccelSegShapes>() +
       " 4=persistent tiles (batched; 0 otherwise)\n";
  t += "iisph_pressure 0 " + shapes_text<PressureShapes>() + small + " 4=persistent tiles (batched; 0 otherwise)\n";
  t += "wkbb18_diag 0 " + shapes_text<DiagShapes>() + " unordered: " + shape_text<DiagSpread>() + from + "\n";
  t += "pcg_init 0 " + shapes_text<PcgShapes>() + small + " batched: " + shapes_text<PcgSegShapes>() + "\n";
  t += "pcg_q 0 " + shapes_text<PcgShapes>() + small + " batched: " + shapes_text<PcgSegShapes>() +
       " 4=cell-tiles (no lists; plain models)\n";
  t += "jacobi_unroll 1 1=1 (one launch to " + std::to_string(kSmallItems) + " items) 2=2 4=4\n";
  t += "staging 0 0=off 1=staged lists and sweeps (unbatched models)\n";
  t += "grid_sort 1 0=tiled radix sort 1=counting where the keys are short, else one cluster launch up to 128k items\n";
  t += "list_split 1 0=one thread per query 1=one warp per run of queries of a cell\n";
  return t;
}

// ===========================================================================
// Scheme base
// ===========================================================================

void Scheme::run(std::string const &procedure, Nhood &nh, cudaStream_t s) {
  auto it = procs_.find(procedure);
  if (it == procs_.end()) throw Error("procedure does not exist");
  if (!model_) throw Error("scheme has not been loaded");
  model_->check_solver(s);
  if (!capturing(s)) {
    it->second(nh, s);
    return;
  }
  std::vector<uint64_t> before = model_->field_versions();
  try {
    it->second(nh, s);
  } catch (...) {
    model_->note_captured(before);
    throw;
  }
  model_->note_captured(before);
}

std::vector<std::string> Scheme::procedure_names() const {
  std::vector<std::string> r;
  for (auto &kv : procs_) r.push_back(kv.first);
  return r;
}

uint64_t device_loop_kernels() {
  unsigned long long v = 0;
  if (cudaMemcpyFromSymbol(&v, g_loop_kernels, sizeof(v)) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return uint64_t(v);
}

namespace {

// groups of a model selected by type / tag, with their fields
struct FluidG {
  Group *g;
  VaryingField *x, *v, *a, *rho, *p, *m, *c, *s, *AA, *Ap, *tb, *vd, *sp, *L;
  SmallField *rho0, *mu, *tol, *max_k, *iters;
};
struct BoundG {
  Group *g;
  VaryingField *x, *V;
  SmallField *mu;
};

class SchemeCommon : public Scheme {
protected:
  Globals globals(Model &m) {
    Globals G{};
    auto gp = [&](char const *n) -> void * {
      SmallField *f = m.find_global(n);
      return f ? m.small_ptr(*f) : nullptr;
    };
    G.h = static_cast<float const *>(gp("smoothing_scale"));
    G.dt = static_cast<float const *>(gp("time_step"));
    G.t = static_cast<float const *>(gp("current_time"));
    G.fade = static_cast<float const *>(gp("fade_duration"));
    G.omega = static_cast<float const *>(gp("iisph_relaxation"));
    G.aprde = static_cast<float *>(gp("iisph_aprde"));
    G.nprde = static_cast<int *>(gp("iisph_nprde"));
    G.gravity = static_cast<float const *>(gp("gravity"));
    G.max_speed = static_cast<float *>(gp("maximum_speed"));
    G.jac_max = static_cast<int const *>(gp("iisph_maximum_iterations"));
    G.jac_eta = static_cast<float const *>(gp("iisph_maximum_density_error"));
    G.jac_iters = static_cast<int *>(gp("iisph_iterations"));
    G.turn = m.red_count_d + Model::kMeetSlot + 1;
    return G;
  }
  Meet meeting(Model &m) {
    return Meet{m.red_count_d + Model::kMeetSlot, m.red_count_d + Model::kMeetSlot + 1, m.solver_gave_up_d,
                ++m.solver_launches, m.solver_polls};
  }
  Red red(Model &m, int slot) {
    Red R;
    R.partials = m.red_d;
    R.ticket = m.red_count_d + slot;
    R.scalars = m.scalars_d;
    R.status = m.status_d;
    R.stats = m.stats_d;
    return R;
  }
  std::vector<FluidG> fluid_;
  std::vector<BoundG> bound_;

  // the per-slot view of a segmented group (batched models), or nullptr
  bool segmented(Group const *g) const { return model_->seg && model_->seg->find(g); }
  SegArgs seg_args(Group const *g) {
    Segments &S = *model_->seg;
    SegGroup const *G = S.find(g);
    if (!G) throw Error("group '" + g->name + "' has no segments");
    SegArgs a{};
    a.tiles = G->tiles;
    a.slot_tiles = G->slot_tiles;
    a.seg = G->seg;
    a.ntiles = G->ntiles;
    a.slots = S.slots;
    a.partials = S.partials;
    a.pcap = S.partial_cap;
    a.tickets = S.tickets;
    a.scal = S.scal;
    a.stat = S.stat;
    a.stats = S.stats;
    a.nprde = S.nprde;
    a.iters = S.iters;
    a.active = G->active;
    a.nactive = G->nactive;
    return a;
  }

  static NbrList nl(NbrView const &v, int g) { return NbrList{v.chunks[g], v.idx32[g], v.cb[g], v.cap[g], v.n}; }
  // packed neighbour records of the fluid / boundary groups (made current
  // here: may launch a pack kernel on `s`)
  FluidN fn(FluidG const &F, NbrView const &v, cudaStream_t s) {
    FluidN r{};
    r.L = nl(v, F.g->index);
    r.xm = model_->packed_xs(F.g, F.x, F.m, "xm", s);
    r.v = F.v ? dptr<float4>(F.v) : nullptr;
    r.a = F.a ? dptr<float4>(F.a) : nullptr;
    r.pr = nullptr;
    return r;
  }
  BoundN bn(BoundG const &B, NbrView const &v, cudaStream_t s) {
    BoundN r{};
    r.L = nl(v, B.g->index);
    r.xV = model_->packed_xs(B.g, B.x, B.V, "xV", s);
    r.mu = B.mu ? static_cast<float const *>(model_->small_ptr(*B.mu)) : nullptr;
    return r;
  }
  template <int NF, int NB> Nbrs<NF, NB> nbrs(NbrView const &v, cudaStream_t s) {
    Nbrs<NF, NB> N{};
    for (int q = 0; q < NF; ++q) N.f[q] = fn(fluid_[q], v, s);
    for (int q = 0; q < NB; ++q) N.b[q] = bn(bound_[q], v, s);
    N.hcache = v.hcache;
    return N;
  }
  template <int NB> Nbrs<0, NB> bnbrs(NbrView const &v, cudaStream_t s) {
    Nbrs<0, NB> N{};
    for (int q = 0; q < NB; ++q) N.b[q] = bn(bound_[q], v, s);
    N.hcache = v.hcache;
    return N;
  }
  // staged lists when the model's staging knob is on (fluid groups of an
  // unbatched model; the neighbourhood builds them only for the layouts the
  // staged sweeps handle)
  NbrView const &lists(Nhood &nh, Group *g, Globals const &G, cudaStream_t s) {
    bool stage = model_->tune.v[kTuneStaging] != 0 && g->type == "fluid" && !segmented(g);
    return nh.lists(g->index, s, G.h, stage);
  }
  // the staged sweeps' arguments for fluid group F (one fluid and one
  // boundary group, unbatched); false where the lists are not staged
  bool stage_args(Nhood &nh, NbrView const &v, FluidG const &F, StageArgs &SA) {
    if (!model_->tune.v[kTuneStaging] || fluid_.size() != 1 || bound_.size() != 1 || segmented(F.g)) return false;
    int fg = F.g->index, bg = bound_[0].g->index;
    if (!v.tile_info || !v.tile_cells || !v.slots[fg] || !v.slots[bg]) return false;
    SA = StageArgs{v.slots[fg], v.slots[bg], v.tile_info, v.tile_cells, nh.view().sorted, fg, bg};
    // per device and cheap: set on every solve (never inside a capture)
    static_assert(kStageSmem <= 64 * 1024, "staged records fit four blocks per SM");
    PG_CUDA(cudaFuncSetAttribute(k_iisph_accel_staged<8>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kStageSmem)));
    PG_CUDA(cudaFuncSetAttribute(k_iisph_pressure_staged<16>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 int(kStageSmem)));
    PG_CUDA(cudaFuncSetAttribute(k_pcg_init_staged<8>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kStageSmem)));
    PG_CUDA(cudaFuncSetAttribute(k_pcg_q_staged<8>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kStageSmem)));
    return true;
  }
  // blocks of a cooperative kernel of kNT threads that the device holds at once
  // (asked for once per scheme: `known` starts at -1)
  template <class Kernel> static int resident_blocks(Kernel *kernel, int &known) {
    if (known < 0) {
      int dev = 0, sms = 0, coop = 0, per = 0;
      PG_CUDA(cudaGetDevice(&dev));
      PG_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
      PG_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev));
      PG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, kNT, 0));
      known = coop ? sms * per : 0;
    }
    return known;
  }
  // a cooperative launch; false, and no further ones, where the context at hand
  // holds fewer blocks than the device
  template <class Kernel>
  static bool launch_resident(Kernel *kernel, unsigned blocks, void **args, cudaStream_t s, int &known) {
    cudaError_t e = cudaLaunchCooperativeKernel(reinterpret_cast<void const *>(kernel), dim3(blocks), dim3(kNT), args, 0, s);
    if (e == cudaErrorCooperativeLaunchTooLarge || e == cudaErrorNotSupported) {
      cudaGetLastError();
      known = 0;
      return false;
    }
    PG_CUDA(e);
    count_launch();
    return true;
  }
  float const *u(SmallField *f) { return static_cast<float const *>(model_->small_ptr(*f)); }
  void need(std::initializer_list<std::pair<void const *, char const *>> l) {
    for (auto &p : l)
      if (!p.first) throw Error(std::string("global field missing: ") + p.second);
  }
  void collect(Model &m, bool fluid_fields, bool boundary_fields) {
    fluid_.clear();
    bound_.clear();
    for (Group *g : m.groups_by_index()) {
      if (g->type == "fluid" && fluid_fields) fluid_.push_back(FluidG{g});
      if (g->type == "boundary" && boundary_fields) bound_.push_back(BoundG{g});
    }
  }
};

// ---------------------------------------------------------------------------
// density
// ---------------------------------------------------------------------------

class Density : public SchemeCommon {
public:
  Density() { reg("compute_density", [this](Nhood &nh, cudaStream_t s) { compute_density(nh, s); }); }
  std::string name() const override { return "density"; }
  std::string source() const override {
    return "procedure compute_density: rho_f = sum_fluid m W(x_ff) + sum_boundary V rho0 W(x_fb)";
  }
  void load(Model &m) override {
    m.add_global("smoothing_scale", ft_real());
    collect(m, true, true);
    for (auto &F : fluid_) {
      F.rho0 = &F.g->add_uniform("rest_density", ft_real());
      F.x = &F.g->add_varying("position", ft_vec3());
      F.rho = &F.g->add_varying("density", ft_real());
      F.m = &F.g->add_varying("mass", ft_real());
    }
    for (auto &B : bound_) {
      B.x = &B.g->add_varying("position", ft_vec3());
      B.V = &B.g->add_varying("volume", ft_real());
    }
    bind(m);
  }
  template <int NF, int NB> struct L {
    static void go(Density *S, FluidG &F, NbrView const &v, Globals G, cudaStream_t s) {
      uint32_t n = uint32_t(F.g->count);
      auto N = S->nbrs<NF, NB>(v, s);
      ProfScope ps(S->model_->prof, "density", s);
      with_shape_spread<DensityShapes, DensitySpread, NF == 1 && NB == 1>(spread(n, v), S->model_->tune.v[kTuneDensity],
                                                                         [&](auto sh) {
        using Sh = decltype(sh);
        k_density<NF, NB, Sh::nt, Sh::minb, Sh::bt><<<div_up(n, Sh::nt), Sh::nt, 0, s>>>(
            n, dptr<float4>(F.x), dptr<float>(F.rho), S->u(F.rho0), G, N);
      });
      count_launch();
    }
  };
  void compute_density(Nhood &nh, cudaStream_t s) {
    Globals G = globals(*model_);
    for (auto &F : fluid_) {
      if (F.g->count == 0) continue;
      NbrView const &v = lists(nh, F.g, G, s);
      dispatch_fb<L>(int(fluid_.size()), int(bound_.size()), this, F, v, G, s);
      PG_LAUNCH_CHECK();
      F.rho->version++;
    }
  }
};

// ---------------------------------------------------------------------------
// aiast12
// ---------------------------------------------------------------------------

class Aiast12 : public SchemeCommon {
public:
  Aiast12() { reg("compute_volume", [this](Nhood &nh, cudaStream_t s) { compute_volume(nh, s); }); }
  std::string name() const override { return "aiast12"; }
  std::string source() const override { return "procedure compute_volume: V_b = 1 / sum_boundary W(x_bb)"; }
  void load(Model &m) override {
    m.add_global("smoothing_scale", ft_real());
    collect(m, false, true);
    for (auto &B : bound_) {
      B.x = &B.g->add_varying("position", ft_vec3());
      B.V = &B.g->add_varying("volume", ft_real());
    }
    bind(m);
  }
  void compute_volume(Nhood &nh, cudaStream_t s) {
    Globals G = globals(*model_);
    int nb = int(bound_.size());
    if (nb > 2) throw Error("unsupported group configuration: at most 2 boundary groups");
    // every group's sums read the positions before any volume is written
    std::vector<std::pair<BoundG *, NbrView const *>> todo;
    for (auto &B : bound_)
      if (B.g->count) todo.push_back({&B, &lists(nh, B.g, G, s)});
    for (auto &t : todo) {
      BoundG &B = *t.first;
      uint32_t n = uint32_t(B.g->count);
      NbrView const &v = *t.second;
      ProfScope ps(model_->prof, "aiast12_volume", s);
      if (nb == 1) {
        k_volume<1><<<div_up(n, kNT), kNT, 0, s>>>(n, dptr<float4>(B.x), dptr<float>(B.V), G, bnbrs<1>(v, s));
        count_launch();
      } else {
        k_volume<2><<<div_up(n, kNT), kNT, 0, s>>>(n, dptr<float4>(B.x), dptr<float>(B.V), G, bnbrs<2>(v, s));
        count_launch();
      }
      PG_LAUNCH_CHECK();
    }
    for (auto &t : todo) t.first->V->version++;
  }
};

// ---------------------------------------------------------------------------
// gravity / symplectic_euler (groups selected by the tag "dynamic")
// ---------------------------------------------------------------------------

class Gravity : public SchemeCommon {
public:
  Gravity() {
    reg("initialize_acceleration", [this](Nhood &, cudaStream_t s) {
      Globals G = globals(*model_);
      for (Group *g : dyn_) {
        uint32_t n = uint32_t(g->count);
        if (!n) continue;
        VaryingField *a = g->find_varying("acceleration");
        ProfScope ps(model_->prof, "gravity", s);
        k_gravity<<<div_up(n, 256), 256, 0, s>>>(n, dptr<float4>(a), G); count_launch();
        PG_LAUNCH_CHECK();
        a->version++;
      }
    });
  }
  std::string name() const override { return "gravity"; }
  std::string source() const override { return "procedure initialize_acceleration: a = g"; }
  void load(Model &m) override {
    m.add_global("gravity", ft_vec3());
    m.add_global("gravity_center", ft_vec3());
    dyn_.clear();
    for (Group *g : m.groups_by_index())
      if (g->has_tag("dynamic")) {
        g->add_varying("position", ft_vec3());
        g->add_varying("acceleration", ft_vec3());
        dyn_.push_back(g);
      }
    bind(m);
  }

private:
  std::vector<Group *> dyn_;
};

class SymplecticEuler : public SchemeCommon {
public:
  SymplecticEuler() {
    reg("integrate_velocity_with_hard_fade", [this](Nhood &, cudaStream_t s) {
      Globals G = globals(*model_);
      for (Group *g : dyn_) {
        uint32_t n = uint32_t(g->count);
        if (!n) continue;
        VaryingField *v = g->find_varying("velocity");
        ProfScope ps(model_->prof, "integrate_velocity", s);
        k_integrate_velocity<<<div_up(n, 256), 256, 0, s>>>(n, dptr<float4>(v),
                                                            dptr<float4>(g->find_varying("acceleration")),
                                                            dptr<float>(g->find_varying("time_of_birth")), G);
        count_launch();
        PG_LAUNCH_CHECK();
        v->version++;
      }
    });
    reg("integrate_position", [this](Nhood &, cudaStream_t s) {
      Globals G = globals(*model_);
      for (Group *g : dyn_) {
        uint32_t n = uint32_t(g->count);
        if (!n) continue;
        VaryingField *x = g->find_varying("position"), *m = g->find_varying("mass");
        if (m && m->type != ft_real()) m = nullptr;
        // the sweeps' records of the group, where they are current
        float4 *xm = m ? model_->current_xs(g, x, m, "xm") : nullptr;
        ProfScope ps(model_->prof, "integrate_position", s);
        k_integrate_position<<<div_up(n, 256), 256, 0, s>>>(n, dptr<float4>(x),
                                                            dptr<float4>(g->find_varying("velocity")), G, xm,
                                                            xm ? dptr<float>(m) : nullptr);
        count_launch();
        PG_LAUNCH_CHECK();
        x->version++;
        if (xm) model_->xs_written(g, x, m, "xm");
      }
    });
  }
  std::string name() const override { return "symplectic_euler"; }
  std::string source() const override {
    return "procedures integrate_velocity_with_hard_fade: v += dt a [0 < t - t_birth - dt_fade]; "
           "integrate_position: x += dt v, max_speed max= |v|";
  }
  void load(Model &m) override {
    m.add_global("time_step", ft_real());
    m.add_global("current_time", ft_real());
    m.add_global("fade_duration", ft_real());
    m.add_global("maximum_speed", ft_real());
    dyn_.clear();
    for (Group *g : m.groups_by_index())
      if (g->has_tag("dynamic")) {
        g->add_varying("position", ft_vec3());
        g->add_varying("velocity", ft_vec3());
        g->add_varying("acceleration", ft_vec3());
        g->add_varying("time_of_birth", ft_real());
        dyn_.push_back(g);
      }
    bind(m);
  }

private:
  std::vector<Group *> dyn_;
};

// ---------------------------------------------------------------------------
// iisph
// ---------------------------------------------------------------------------

class Iisph : public SchemeCommon {
public:
  Iisph() {
    reg("setup", [this](Nhood &nh, cudaStream_t s) { setup(nh, s); });
    reg("iteration_pressure_acceleration", [this](Nhood &nh, cudaStream_t s) { accel(nh, s); });
    reg("iteration_pressure", [this](Nhood &nh, cudaStream_t s) { pressure(nh, s); });
    // the whole relaxed-Jacobi loop of the driver script on the device
    reg("solve_pressure", [this](Nhood &nh, cudaStream_t s) { solve(nh, s); });
  }
  std::string name() const override { return "iisph"; }
  std::string source() const override {
    return "procedures setup (c, p = 0, s, AA, nprde), iteration_pressure_acceleration (a), "
           "iteration_pressure (Ap, relaxed Jacobi p, aprde += (Ap - s) / rho0 [p > 1e-9]), "
           "solve_pressure (repeat aprde := 0, acceleration, pressure while the iteration count is < 2 or "
           "aprde / nprde >= iisph_maximum_density_error, at most iisph_maximum_iterations times)";
  }
  void load(Model &m) override {
    m.add_global("gravity", ft_vec3());
    m.add_global("smoothing_scale", ft_real());
    m.add_global("time_step", ft_real());
    m.add_global("iisph_relaxation", ft_real());
    m.add_global("iisph_aprde", ft_real());
    m.add_global("iisph_nprde", ft_int());
    m.add_global("iisph_maximum_iterations", ft_int());
    m.add_global("iisph_maximum_density_error", ft_real());
    m.add_global("iisph_iterations", ft_int());
    collect(m, true, true);
    for (auto &F : fluid_) {
      F.rho0 = &F.g->add_uniform("rest_density", ft_real());
      F.x = &F.g->add_varying("position", ft_vec3());
      F.v = &F.g->add_varying("velocity", ft_vec3());
      F.a = &F.g->add_varying("acceleration", ft_vec3());
      F.rho = &F.g->add_varying("density", ft_real());
      F.p = &F.g->add_varying("pressure", ft_real());
      F.m = &F.g->add_varying("mass", ft_real());
      F.c = &F.g->add_varying("iisph_helper_c", ft_vec3());
      F.s = &F.g->add_varying("iisph_source_term", ft_real());
      F.AA = &F.g->add_varying("iisph_diagonal_element", ft_real());
      F.Ap = &F.g->add_varying("iisph_right_hand_side", ft_real());
    }
    for (auto &B : bound_) {
      B.x = &B.g->add_varying("position", ft_vec3());
      B.V = &B.g->add_varying("volume", ft_real());
    }
    bind(m);
    loop_.reset();
  }
  template <int NF, int NB> struct SETUP {
    static void go(Iisph *S, FluidG &F, NbrView const &v, Globals G, cudaStream_t s) {
      uint32_t n = uint32_t(F.g->count);
      auto N = S->nbrs<NF, NB>(v, s);
      float *pr = S->model_->pr_buffer(F.g, s);
      ProfScope ps(S->model_->prof, "iisph_setup", s);
      with_shape_for<SetupShapes, NF == 1 && NB == 1, NF == 1 && NB == 1>(n, S->model_->tune.v[kTuneSetup], [&](auto sh) {
        using Sh = decltype(sh);
        k_iisph_setup<NF, NB, Sh::nt, Sh::minb, Sh::bt><<<div_up(n, Sh::nt), Sh::nt, 0, s>>>(
            n, dptr<float4>(F.x), dptr<float4>(F.v), dptr<float4>(F.c), dptr<float>(F.m), dptr<float>(F.rho),
            dptr<float>(F.p), pr, dptr<float>(F.s), dptr<float>(F.AA), S->u(F.rho0), G, N,
            S->model_->status_d + kStSetupBad);
      });
      count_launch();
    }
  };
  // Pressure-acceleration / pressure launches of one group.  With `sig`
  // non-null nothing is launched: the kernel arguments are appended to the
  // signature of the device loop instead.  `done` is the loop flag
  // (nullptr outside the device loop); `prof` brackets the launch with
  // timing events (never on a capture stream).
  template <int NF, int NB> struct A {
    static void go(Iisph *S, FluidG &F, NbrView const &v, Globals G, cudaStream_t s, int const *done, bool prof,
                   std::string *sig, SegArgs const *SA = nullptr, StageArgs const *ST = nullptr) {
      uint32_t n = uint32_t(F.g->count);
      auto N = S->nbrs<NF, NB>(v, s);
      for (int q = 0; q < NF; ++q) N.f[q].pr = S->model_->packed_pr(S->fluid_[q].g, S->fluid_[q].p, S->fluid_[q].rho, s);
      float4 const *x = dptr<float4>(F.x);
      float const *p = dptr<float>(F.p), *rho = dptr<float>(F.rho);
      float4 *a = dptr<float4>(F.a);
      float const *rho0 = S->u(F.rho0);
      if (sig) {
        sig_add(*sig, n);
        sig_add(*sig, N);
        sig_add(*sig, x);
        sig_add(*sig, p);
        sig_add(*sig, rho);
        sig_add(*sig, a);
        sig_add(*sig, rho0);
        if (SA) sig_add(*sig, *SA);
        if (ST) sig_add(*sig, *ST);
        return;
      }
      if (prof) S->model_->prof.begin("iisph_accel", s);
      int tv = S->model_->tune.v[kTuneAccel];
      bool staged = false;
      if constexpr (NF == 1 && NB == 1) {
        if (ST && !SA) {
          k_iisph_accel_staged<8><<<div_up(n, kNT), kNT, kStageSmem, s>>>(n, x, p, rho, a, rho0, G, N, done, *ST);
          staged = true;
        }
      }
      if (staged) {
      } else if (SA) {
        if (SA->ntiles) {
          if (NF == 1 && NB == 1 && tv == 4)
            k_iisph_accel_seg<NF, NB, kMinBlocks, 8 | kAlone, true><<<std::min(SA->ntiles, kActiveBlocks), kNT, 0, s>>>(
                x, p, rho, a, rho0, G, N, *SA, S->model_->status_d + kStJacFirst);
          else
            with_shape<AccelSegShapes, NF == 1 && NB == 1>(tv, [&](auto sh) {
              using Sh = decltype(sh);
              k_iisph_accel_seg<NF, NB, Sh::minb, Sh::bt><<<std::min(SA->ntiles, kActiveBlocks), kNT, 0, s>>>(
                  x, p, rho, a, rho0, G, N, *SA, S->model_->status_d + kStJacFirst);
            });
        }
      } else {
        with_shape_for<AccelShapes, NF == 1 && NB == 1, NF == 1 && NB == 1>(n, tv, [&](auto sh) {
          using Sh = decltype(sh);
          k_iisph_accel<NF, NB, Sh::nt, Sh::minb, Sh::bt><<<div_up(n, Sh::nt), Sh::nt, 0, s>>>(n, x, p, rho, a, rho0,
                                                                                            G, N, done);
        });
      }
      count_launch();
      if (prof) S->model_->prof.end(s);
    }
  };
  template <int NF, int NB> struct P {
    static void go(Iisph *S, FluidG &F, NbrView const &v, Globals G, cudaStream_t s, int first, int last,
                   int const *done, bool prof, std::string *sig, SegArgs const *SA = nullptr,
                   StageArgs const *ST = nullptr) {
      uint32_t n = uint32_t(F.g->count);
      auto N = S->nbrs<NF, NB>(v, s);
      float *pr = S->model_->pr_buffer(F.g, s);
      Red R = S->red(*S->model_, 0);
      PressureArgs PA{dptr<float4>(F.x), dptr<float4>(F.a), dptr<float>(F.rho), dptr<float>(F.s), dptr<float>(F.AA),
                      dptr<float>(F.p), pr, dptr<float>(F.Ap), S->u(F.rho0)};
      if (sig) {
        sig_add(*sig, n);
        sig_add(*sig, N);
        sig_add(*sig, R);
        sig_add(*sig, PA);
        sig_add(*sig, first);
        sig_add(*sig, last);
        if (SA) sig_add(*sig, *SA);
        if (ST) sig_add(*sig, *ST);
        return;
      }
      if (prof) S->model_->prof.begin("iisph_pressure", s);
      int tvp = S->model_->tune.v[kTunePressure];
      bool staged = false;
      if constexpr (NF == 1 && NB == 1) {
        if (ST && !SA) {
          k_iisph_pressure_staged<16><<<red_grid(n), kNT, kStageSmem, s>>>(n, PA, G, N, R, first, last, done, *ST);
          staged = true;
        }
      }
      if (staged) {
      } else if (SA && NF == 1 && NB == 1 && tvp == 4) {
        if (SA->ntiles)
          k_iisph_pressure_seg<NF, NB, kMinBlocks, 8 | kAlone, true><<<std::min(SA->ntiles, kActiveBlocks), kNT, 0, s>>>(
              PA, G, N, *SA, S->model_->status_d + kStJacFirst);
      } else
      with_shape_for<PressureShapes, NF == 1 && NB == 1, NF == 1 && NB == 1>(SA ? ~0u : n, tvp, [&](auto sh) {
        using Sh = decltype(sh);
        if (SA) {
          if (SA->ntiles)
            k_iisph_pressure_seg<NF, NB, Sh::minb, Sh::bt><<<SA->ntiles, kNT, 0, s>>>(
                PA, G, N, *SA, S->model_->status_d + kStJacFirst);
        } else {
          k_iisph_pressure<NF, NB, Sh::minb, Sh::bt><<<red_grid(n), kNT, 0, s>>>(n, PA, G, N, R, first, last, done);
        }
      });
      count_launch();
      if (prof) S->model_->prof.end(s);
    }
  };
  Globals checked_globals() {
    Globals G = globals(*model_);
    need({{G.h, "smoothing_scale"}, {G.dt, "time_step"}, {G.omega, "iisph_relaxation"}, {G.aprde, "iisph_aprde"},
          {G.nprde, "iisph_nprde"}, {G.jac_max, "iisph_maximum_iterations"}});
    return G;
  }
  std::vector<FluidG *> active() {
    std::vector<FluidG *> act;
    for (auto &F : fluid_)
      if (F.g->count) act.push_back(&F);
    return act;
  }
  // p and p / rho^2 were written together by a kernel
  void wrote_pressure(FluidG &F) {
    F.p->version++;
    model_->pack_commit(F.g, "pr", {uint64_t(F.g->count), reinterpret_cast<uint64_t>(F.p->d), F.p->version,
                                    reinterpret_cast<uint64_t>(F.rho->d), F.rho->version});
  }
  void setup(Nhood &nh, cudaStream_t s) {
    Globals G = checked_globals();
    int nf = int(fluid_.size()), nb = int(bound_.size());
    // one fused sweep per group (pass 2 of a group reads only its own c)
    long long total = 0;
    for (auto *F : active()) total += (long long)F->g->count;
    // nprde = number of fluid particles (the generated reduction adds 1 per particle)
    k_setup_begin<<<1, 1, 0, s>>>(model_->status_d, G.nprde, int(total), G, rest_densities(), model_->scalars_d);
    count_launch();
    for (auto *F : active()) {
      dispatch_fb<SETUP>(nf, nb, this, *F, lists(nh, F->g, G, s), G, s);
      PG_LAUNCH_CHECK();
      F->c->version++;
      F->s->version++;
      F->AA->version++;
      wrote_pressure(*F);
    }
    PG_LAUNCH_CHECK();
    if (capturing(s)) zero_key_.clear(); // queued for later, possibly more than once
    else zero_key_ = zero_key(nh, s);
  }
  RestDensities rest_densities() {
    RestDensities D{};
    for (auto &F : fluid_)
      if (D.n < kMaxNbrGroups) D.p[D.n++] = u(F.rho0);
    return D;
  }
  // What the first iteration's zero sums rest on (kStJacFirst): the fields
  // that setup read, the pressure it wrote, the grid of its lists and the
  // stream it ran on; empty where captured work writes one of the fields.  A
  // solve takes them only where the key is still the same; it is cleared by the
  // solve, which changes the pressure.
  std::vector<uint64_t> zero_key(Nhood &nh, cudaStream_t s) {
    std::vector<uint64_t> k{reinterpret_cast<uint64_t>(&nh), nh.epoch(), reinterpret_cast<uint64_t>(s)};
    bool seen = true; // (else a replayed graph may have changed them)
    auto add = [&](Group *g, std::initializer_list<VaryingField const *> fs) {
      k.push_back(uint64_t(g->count));
      for (auto *f : fs) {
        k.push_back(reinterpret_cast<uint64_t>(f->d));
        k.push_back(f->version);
        seen = seen && !f->unseen;
      }
    };
    for (auto &F : fluid_) add(F.g, {F.x, F.m, F.rho, F.p});
    for (auto &B : bound_) add(B.g, {B.x, B.V});
    if (!seen) k.clear();
    return k;
  }
  void no_segments(char const *what) {
    for (auto &F : fluid_)
      if (segmented(F.g))
        throw Error(std::string(what) + " sums the density error over the whole group; on a batched (segmented) "
                    "model use solve_pressure, which decides convergence per scene");
  }
  void accel(Nhood &nh, cudaStream_t s) {
    no_segments("iteration_pressure_acceleration");
    Globals G = checked_globals();
    int nf = int(fluid_.size()), nb = int(bound_.size());
    for (auto *F : active()) {
      dispatch_fb<A>(nf, nb, this, *F, lists(nh, F->g, G, s), G, s, static_cast<int const *>(nullptr), true,
                     static_cast<std::string *>(nullptr));
      PG_LAUNCH_CHECK();
      F->a->version++;
    }
  }
  void pressure(Nhood &nh, cudaStream_t s) {
    no_segments("iteration_pressure");
    Globals G = checked_globals();
    int nf = int(fluid_.size()), nb = int(bound_.size());
    auto act = active();
    for (size_t k = 0; k < act.size(); ++k) {
      dispatch_fb<P>(nf, nb, this, *act[k], lists(nh, act[k]->g, G, s), G, s, k == 0 ? 1 : 0,
                     k + 1 == act.size() ? 1 : 0, static_cast<int const *>(nullptr), true,
                     static_cast<std::string *>(nullptr));
      PG_LAUNCH_CHECK();
      act[k]->Ap->version++;
      wrote_pressure(*act[k]);
    }
  }
  // The relaxed-Jacobi loop on the device: a CUDA graph whose conditional
  // while node repeats [acceleration, pressure, control] until the control
  // kernel clears the condition.  With profiling enabled the same kernels
  // are driven from the host, one iteration at a time, so that each launch
  // can be timed.
  void solve(Nhood &nh, cudaStream_t s) {
    Globals G = checked_globals();
    need({{G.jac_eta, "iisph_maximum_density_error"}, {G.jac_iters, "iisph_iterations"}});
    int nf = int(fluid_.size()), nb = int(bound_.size());
    auto act = active();
    Red R = red(*model_, 0);
    int const *done = R.status + kStJacDone;
    // batched model: one segmented fluid group, convergence per slot
    bool seg = false;
    for (auto &F : fluid_)
      if (segmented(F.g)) seg = true;
    SegArgs SA{};
    if (seg) {
      if (fluid_.size() != 1) throw Error("a batched model has exactly one fluid group");
      SA = seg_args(fluid_[0].g);
    }
    SegArgs const *sa = seg ? &SA : nullptr;
    // lists and packed records are made current before the loop, so that
    // building the loop launches nothing else
    std::vector<NbrView const *> views;
    for (auto *F : act) {
      views.push_back(&lists(nh, F->g, G, s));
      model_->packed_xs(F->g, F->x, F->m, "xm", s);
      model_->packed_pr(F->g, F->p, F->rho, s);
    }
    for (auto &B : bound_)
      if (B.g->count) model_->packed_xs(B.g, B.x, B.V, "xV", s);
    // staged sweeps (the staging knob): one fluid group, staged lists
    StageArgs st{};
    bool staged = !seg && act.size() == 1 && stage_args(nh, *views[0], *act[0], st);
    StageArgs const *stp = staged ? &st : nullptr;
    // (the staged sweeps take every iteration in full)
    int same = !staged && !zero_key_.empty() && !capturing(s) && zero_key_ == zero_key(nh, s) ? 1 : 0;
    zero_key_.clear();
    bool one_launch = !seg && !staged && act.size() == 1 && !model_->prof.enabled &&
                      loop_in_one_launch(*act[0], nf, nb, s) && jacobi_loop(*act[0], *views[0], G, R, same, s);
    if (one_launch) {
    } else if (seg) {
      k_seg_jacobi_begin<<<div_up(std::max<uint32_t>(SA.slots, 1), 256), 256, 0, s>>>(SA, G, R, rest_densities(), same);
      count_launch();
      k_seg_active<<<1, 1024, 0, s>>>(SA); count_launch();
    } else {
      k_jacobi_begin<<<1, 1, 0, s>>>(G, R, rest_densities(), same); count_launch();
    }
    PG_LAUNCH_CHECK();
    int kernels = 2 * int(act.size()) + 1;
    // iterations per graph iteration (the jacobi_unroll knob): the kernels of
    // the repeats after the control has ended the loop return at once, and
    // the last control of the body decides whether the body runs again
    int unroll = model_->tune.v[kTuneJacobiUnroll];
    auto body = [&](cudaStream_t cs, cudaGraphConditionalHandle h, bool use_handle, bool prof, std::string *sig) {
      int reps = (sig || prof) ? 1 : unroll;
      for (int rep = 0; rep < reps; ++rep) {
        for (size_t k = 0; k < act.size(); ++k)
          dispatch_fb<A>(nf, nb, this, *act[k], *views[k], G, cs, done, prof, sig, sa, stp);
        for (size_t k = 0; k < act.size(); ++k)
          dispatch_fb<P>(nf, nb, this, *act[k], *views[k], G, cs, k == 0 ? 1 : 0, k + 1 == act.size() ? 1 : 0, done,
                         prof, sig, sa, stp);
        if (sig) return;
        if (seg) {
          k_seg_jacobi_control<<<1, 1024, 0, cs>>>(G, SA, h, use_handle ? 1 : 0, use_handle ? kernels : 0,
                                                   R.status + kStJacDone, R.status + kStJacFirst);
        } else {
          k_jacobi_control<<<1, 1, 0, cs>>>(G, R, h, use_handle ? 1 : 0, use_handle ? kernels : 0);
        }
        count_launch();
      }
    };
    if (one_launch) {
    } else if (model_->prof.enabled) {
      // host-driven: one iteration per round trip
      for (int it = 0; it < 100000; ++it) {
        body(s, cudaGraphConditionalHandle{}, false, true, nullptr);
        PG_LAUNCH_CHECK();
        int d = 0;
        PG_CUDA(cudaMemcpyAsync(&d, done, sizeof(int), cudaMemcpyDeviceToHost, s));
        PG_CUDA(cudaStreamSynchronize(s));
        if (d) break;
      }
    } else {
      std::string sig;
      body(s, cudaGraphConditionalHandle{}, true, false, &sig);
      sig_add(sig, G);
      sig_add(sig, R);
      sig_add(sig, model_->tune); // a changed shape or repeat count rebuilds the graph
      loop_.run(s, sig, [&](cudaStream_t cs, cudaGraphConditionalHandle h) { body(cs, h, true, false, nullptr); });
      PG_LAUNCH_CHECK();
    }
    for (auto *F : act) {
      F->a->version++;
      F->Ap->version++;
      wrote_pressure(*F);
    }
  }

private:
  // one cooperative launch takes the loop of a small scene of the tuned layout
  // where every block is resident, whatever the sweeps' shapes (which the tuner
  // times in launches of their own) unless iterations are repeated in a graph
  bool loop_in_one_launch(FluidG const &F, int nf, int nb, cudaStream_t s) {
    auto const &t = model_->tune.v;
    if (nf != 1 || nb != 1 || t[kTuneJacobiUnroll] != 1) return false;
    if (F.g->count == 0 || F.g->count > kSmallItems || capturing(s)) return false;
    return div_up(F.g->count, kNT) <= unsigned(resident_blocks(k_jacobi_loop, resident_));
  }
  bool jacobi_loop(FluidG &F, NbrView const &v, Globals G, Red R, int same, cudaStream_t s) {
    uint32_t n = uint32_t(F.g->count);
    auto N = nbrs<1, 1>(v, s);
    N.f[0].pr = model_->packed_pr(F.g, F.p, F.rho, s);
    PressureArgs PA{dptr<float4>(F.x), dptr<float4>(F.a), dptr<float>(F.rho), dptr<float>(F.s), dptr<float>(F.AA),
                    dptr<float>(F.p), model_->pr_buffer(F.g, s), dptr<float>(F.Ap), u(F.rho0)};
    float4 *a = dptr<float4>(F.a);
    Meet M = meeting(*model_);
    RestDensities D = rest_densities();
    void *args[] = {&n, &PA, &a, &G, &N, &R, &M, &D, &same};
    return launch_resident(k_jacobi_loop, div_up(n, kNT), args, s, resident_);
  }
  WhileLoop loop_;
  std::vector<uint64_t> zero_key_;
  int resident_ = -1; // blocks of k_jacobi_loop that fit the device
};

// ---------------------------------------------------------------------------
// wkbb18
// ---------------------------------------------------------------------------

// gc: wkbb18_gc (share/schemes/wkbb18_gc.prtcl), the same procedures with
// every kernel gradient premultiplied by the item's gradient correction
class Wkbb18 : public SchemeCommon {
public:
  explicit Wkbb18(bool gc = false) : gc_(gc) {
    reg("compute_diagonal", [this](Nhood &nh, cudaStream_t s) { diag(nh, s); });
    reg("accumulate_acceleration", [this](Nhood &nh, cudaStream_t s) { pcg(nh, s); });
  }
  ~Wkbb18() override { free_vectors(); }
  std::string name() const override { return gc_ ? "wkbb18_gc" : "wkbb18"; }
  std::string source() const override {
    return std::string("procedures compute_diagonal (sp = (I - dt S)^-1), accumulate_acceleration (PCG over fluid "
                       "velocities with the implicit viscosity system, Jacobi block preconditioner sp, apply vd and "
                       "a = vd / dt)") +
           (gc_ ? "; every kernel gradient premultiplied by gradient_correction" : "");
  }
  void load(Model &m) override {
    m.add_global("smoothing_scale", ft_real());
    m.add_global("time_step", ft_real());
    m.add_global("current_time", ft_real());
    m.add_global("fade_duration", ft_real());
    collect(m, true, true);
    for (auto &F : fluid_) {
      F.rho0 = &F.g->add_uniform("rest_density", ft_real());
      F.mu = &F.g->add_uniform("dynamic_viscosity", ft_real());
      F.tol = &F.g->add_uniform("wkbb18_maximum_error", ft_real());
      F.max_k = &F.g->add_uniform("wkbb18_maximum_iterations", ft_int());
      F.iters = &F.g->add_uniform("wkbb18_iterations", ft_int());
      F.x = &F.g->add_varying("position", ft_vec3());
      F.v = &F.g->add_varying("velocity", ft_vec3());
      F.a = &F.g->add_varying("acceleration", ft_vec3());
      F.rho = &F.g->add_varying("density", ft_real());
      F.m = &F.g->add_varying("mass", ft_real());
      F.vd = &F.g->add_varying("wkbb18_velocity_delta", ft_vec3());
      F.sp = &F.g->add_varying("wkbb18_system_diagonal", ft_mat3());
      F.tb = &F.g->add_varying("time_of_birth", ft_real());
      F.L = gc_ ? &F.g->add_varying("gradient_correction", ft_mat3()) : nullptr;
    }
    for (auto &B : bound_) {
      B.mu = &B.g->add_uniform("dynamic_viscosity", ft_real());
      B.x = &B.g->add_varying("position", ft_vec3());
      B.V = &B.g->add_varying("volume", ft_real());
    }
    bind(m);
    loops_.clear();
  }
  template <int NB> void diag_launch(FluidG &F, NbrView const &v, Globals G, cudaStream_t s) {
    uint32_t n = uint32_t(F.g->count);
    auto N = bnbrs<NB>(v, s);
    float4 const *xmr = model_->packed_xmr(F.g, F.x, F.m, F.rho, s);
    ProfScope ps(model_->prof, "wkbb18_diag", s);
    bool sp = spread(n, v);
    if (gc_)
      with_shape_spread<DiagShapes, DiagSpread, false>(sp, 0, [&](auto sh) {
        using Sh = decltype(sh);
        k_wkbb18_diag<NB, true, Sh::nt, Sh::minb, Sh::bt><<<div_up(n, kNT), kNT, 0, s>>>(
            n, uint32_t(F.sp->cap), xmr, dptr<float>(F.rho), dptr<float>(F.sp), u(F.rho0), u(F.mu), G,
            nl(v, F.g->index), N, dptr<float>(F.L), uint32_t(F.L->cap));
      });
    else
      with_shape_spread<DiagShapes, DiagSpread, NB == 1>(sp, fluid_.size() == 1 ? model_->tune.v[kTuneDiag] : 0, [&](auto sh) {
        using Sh = decltype(sh);
        k_wkbb18_diag<NB, false, Sh::nt, Sh::minb, Sh::bt><<<div_up(n, Sh::nt), Sh::nt, 0, s>>>(
            n, uint32_t(F.sp->cap), xmr, dptr<float>(F.rho), dptr<float>(F.sp), u(F.rho0), u(F.mu), G,
            nl(v, F.g->index), N, nullptr, 0u);
      });
    count_launch();
  }
  void diag(Nhood &nh, cudaStream_t s) {
    Globals G = globals(*model_);
    int nb = int(bound_.size());
    for (auto &F : fluid_) {
      if (!F.g->count) continue;
      NbrView const &v = lists(nh, F.g, G, s);
      if (nb == 0) diag_launch<0>(F, v, G, s);
      else if (nb == 1) diag_launch<1>(F, v, G, s);
      else if (nb == 2) diag_launch<2>(F, v, G, s);
      else throw Error("unsupported group configuration: at most 2 boundary groups");
      PG_LAUNCH_CHECK();
      F.sp->version++;
    }
  }

  // solver/cg_openmp.hpp:35-215 on the device: guess and initial residual,
  // then a device loop of [q = A p, update, p update, control], then apply
  template <int NB> void pcg_group(FluidG &F, NbrView const &v, Globals G, cudaStream_t s, Nhood &nh) {
    if (gc_) pcg_group_t<NB, true>(F, v, G, s, nh);
    else pcg_group_t<NB, false>(F, v, G, s, nh);
  }
  template <int NB, bool GC> void pcg_group_t(FluidG &F, NbrView const &v, Globals G, cudaStream_t s, Nhood &nh) {
    uint32_t n = uint32_t(F.g->count);
    ensure_vectors(n);
    PcgArgs P{};
    P.n = n;
    P.cap = uint32_t(F.sp->cap);
    P.xmr = model_->packed_xmr(F.g, F.x, F.m, F.rho, s);
    P.v = dptr<float4>(F.v);
    P.rho = dptr<float>(F.rho);
    P.sp = dptr<float>(F.sp);
    P.tb = dptr<float>(F.tb);
    P.vd = dptr<float4>(F.vd);
    P.a = dptr<float4>(F.a);
    P.X = vec_[0];
    P.Y = vec_[1];
    P.Rr = vec_[2];
    P.P = vec_[3];
    P.Q = vec_[4];
    P.rho0 = u(F.rho0);
    P.mu = u(F.mu);
    P.tol = u(F.tol);
    P.max_k = static_cast<int const *>(model_->small_ptr(*F.max_k));
    P.iterations = static_cast<int *>(model_->small_ptr(*F.iters));
    P.self = nl(v, F.g->index);
    P.L = GC ? dptr<float>(F.L) : nullptr;
    P.lcap = GC ? uint32_t(F.L->cap) : 0u;
    auto N = bnbrs<NB>(v, s);
    Red R = red(*model_, 1);
    unsigned rg = red_grid(n), eg = div_up(n, 256);
    // batched model: one PCG per slot
    bool seg = segmented(F.g);
    SegArgs SA = seg ? seg_args(F.g) : SegArgs{};
    unsigned tg = SA.ntiles;
    k_pcg_guess<<<eg, 256, 0, s>>>(P); count_launch();
    constexpr bool kTuned = NB == 1 && !GC;
    int tv_init = fluid_.size() == 1 ? model_->tune.v[kTunePcgInit] : 0;
    int tv_q = fluid_.size() == 1 ? model_->tune.v[kTunePcgQ] : 0;
    // staged sweeps (the staging knob) for the tuned layout, except with the
    // cell-tile sweep
    StageArgs st{};
    bool staged = false;
    if constexpr (kTuned) staged = !seg && tv_q != 4 && stage_args(nh, v, F, st);
    {
      ProfScope ps(model_->prof, "pcg_init", s);
      if (seg) {
        k_seg_pcg_begin<<<div_up(std::max<uint32_t>(SA.slots, 1), 256), 256, 0, s>>>(SA); count_launch();
      }
      if constexpr (kTuned)
        if (staged) k_pcg_init_staged<8><<<rg, kNT, kStageSmem, s>>>(P, G, N, R, st);
      if (staged) {
      } else if (seg) {
        with_shape<PcgSegShapes, kTuned>(tv_init, [&](auto sh) {
          using Sh = decltype(sh);
          if (tg) k_pcg_init_seg<NB, GC, Sh::minb, Sh::bt><<<tg, kNT, 0, s>>>(P, G, N, SA);
        });
      } else {
        with_shape_for<PcgShapes, kTuned, NB == 1>(P.n, tv_init, [&](auto sh) {
          using Sh = decltype(sh);
          k_pcg_init<NB, GC, Sh::minb, Sh::bt><<<rg, kNT, 0, s>>>(P, G, N, R);
        });
      }
      count_launch();
    }
    PG_LAUNCH_CHECK();
    // shape 4 of pcg_q: the cell-tile sweep (plain models of the tuned layout)
    bool tiles = false;
    GridView gv{};
    float4 const *xs = nullptr;
    int fg = F.g->index, bg = bound_.empty() ? -1 : bound_[0].g->index;
    if constexpr (kTuned) {
      if (!seg && tv_q == 4) nh.need_r2s(s);
      gv = nh.view();
      // the tiles walk the grid's cells: the fluid group must be in the grid
      if (!seg && tv_q == 4 && gv.in_grid[fg]) {
        tiles = true;
        xs = nh.sorted_positions();
        // per device and cheap: set on every solve (never inside a capture)
        PG_CUDA(cudaFuncSetAttribute(k_pcg_q_tiles<NB>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     int(2 * kTileStage * sizeof(float4))));
      }
    }
    auto body = [&](cudaStream_t cs, cudaGraphConditionalHandle h, bool use_handle, bool prof) {
      if (prof) model_->prof.begin("pcg_q", cs);
      if constexpr (kTuned) {
        if (tiles)
          k_pcg_q_tiles<NB><<<rg, kNT, 2 * kTileStage * sizeof(float4), cs>>>(P, G, N, R, gv, xs, fg, bg);
        else if (staged)
          k_pcg_q_staged<8><<<rg, kNT, kStageSmem, cs>>>(P, G, N, R, st);
      }
      if (tiles || staged) {
      } else if (seg) {
        with_shape<PcgSegShapes, kTuned>(tv_q, [&](auto sh) {
          using Sh = decltype(sh);
          if (tg) k_pcg_q_seg<NB, GC, Sh::minb, Sh::bt><<<tg, kNT, 0, cs>>>(P, G, N, SA);
        });
      } else {
        with_shape_for<PcgShapes, kTuned, NB == 1>(P.n, tv_q, [&](auto sh) {
          using Sh = decltype(sh);
          k_pcg_q<NB, GC, Sh::minb, Sh::bt><<<rg, kNT, 0, cs>>>(P, G, N, R);
        });
      }
      count_launch();
      if (prof) model_->prof.end(cs);
      if (prof) model_->prof.begin("pcg_update", cs);
      if (seg) {
        if (tg) k_pcg_update_seg<<<tg, kSegUpdateNT, 0, cs>>>(P, SA);
      } else {
        // one resident wave: each thread folds several items before the
        // block's FP64 tree (the FP64 pipe is narrow on this GPU)
        k_pcg_update<<<std::min(rg, unsigned(152 * kMinBlocks)), kNT, 0, cs>>>(P, R);
      }
      count_launch();
      if (prof) model_->prof.end(cs);
      if (prof) model_->prof.begin("pcg_p", cs);
      if (seg) k_pcg_p_seg<<<eg, 256, 0, cs>>>(P, SA);
      else k_pcg_p<<<rg, kNT, 0, cs>>>(P, R);
      count_launch();
      if (prof) model_->prof.end(cs);
      if (seg)
        k_seg_pcg_control<<<1, 1024, 0, cs>>>(P, SA, h, use_handle ? 1 : 0, use_handle ? 4 : 0,
                                              R.status + kStPcgActive);
      else
        k_pcg_control<<<1, 1, 0, cs>>>(P, R, h, use_handle ? 1 : 0, use_handle ? 4 : 0);
      count_launch();
    };
    bool one_launch = false;
    if constexpr (NB == 1) {
      Meet M = meeting(*model_);
      void *args[] = {&P, &G, &N, &R, &M};
      one_launch = !seg && !staged && !tiles && fluid_.size() == 1 && !model_->prof.enabled && n <= kSmallItems &&
                   !capturing(s) && rg <= unsigned(resident_blocks(k_pcg_loop<GC>, resident_)) &&
                   launch_resident(k_pcg_loop<GC>, rg, args, s, resident_);
    }
    if (one_launch) {
    } else if (model_->prof.enabled) {
      // host-driven (timed launches): one iteration per round trip
      for (int it = 0; it < 1000000; ++it) {
        body(s, cudaGraphConditionalHandle{}, false, true);
        PG_LAUNCH_CHECK();
        int active = 0;
        PG_CUDA(cudaMemcpyAsync(&active, R.status + kStPcgActive, sizeof(int), cudaMemcpyDeviceToHost, s));
        PG_CUDA(cudaStreamSynchronize(s));
        if (!active) break;
      }
    } else {
      std::string sig;
      sig_add(sig, P);
      sig_add(sig, N);
      sig_add(sig, R);
      sig_add(sig, G);
      sig_add(sig, rg);
      sig_add(sig, SA);
      sig_add(sig, model_->tune); // a changed shape rebuilds the graph
      if (tiles) {
        sig_add(sig, gv);
        sig_add(sig, xs);
      }
      if (staged) sig_add(sig, st);
      loops_[F.g].run(s, sig, [&](cudaStream_t cs, cudaGraphConditionalHandle h) { body(cs, h, true, false); });
      PG_LAUNCH_CHECK();
    }
    Red RA = R;
    if (seg) RA.status = nullptr; // per-slot iteration counts are in the segments' state
    k_pcg_apply<<<eg, 256, 0, s>>>(P, G, RA); count_launch();
    PG_LAUNCH_CHECK();
    F.vd->version++;
    F.a->version++;
  }
  void pcg(Nhood &nh, cudaStream_t s) {
    Globals G = globals(*model_);
    int nb = int(bound_.size());
    for (auto &F : fluid_) {
      if (!F.g->count) {
        int zero = 0;
        model_->small_set(*F.iters, &zero, s);
        continue;
      }
      NbrView const &v = lists(nh, F.g, G, s);
      if (nb == 0) pcg_group<0>(F, v, G, s, nh);
      else if (nb == 1) pcg_group<1>(F, v, G, s, nh);
      else if (nb == 2) pcg_group<2>(F, v, G, s, nh);
      else throw Error("unsupported group configuration: at most 2 boundary groups");
    }
  }

private:
  bool gc_;
  float4 *vec_[5] = {};
  size_t vec_cap_ = 0;
  std::map<Group *, WhileLoop> loops_;
  int resident_ = -1; // blocks of k_pcg_loop that fit the device
  void free_vectors() {
    for (auto &p : vec_)
      if (p) {
        cudaFree(p);
        p = nullptr;
      }
    vec_cap_ = 0;
  }
  void ensure_vectors(size_t n) {
    if (n <= vec_cap_) return;
    loops_.clear(); // the captured loops hold the old vectors
    free_vectors();
    for (auto &p : vec_) PG_CUDA(cudaMalloc(&p, n * 16));
    vec_cap_ = n;
  }
};

// ---------------------------------------------------------------------------
// viscosity (explicit)
// ---------------------------------------------------------------------------

class Viscosity : public SchemeCommon {
public:
  Viscosity() {
    reg("accumulate_acceleration", [this](Nhood &nh, cudaStream_t s) { accumulate(nh, s); });
  }
  std::string name() const override { return "viscosity"; }
  std::string source() const override {
    return "procedure accumulate_acceleration: a_f += 10 (mu_f / rho_f) (m_f' / rho_f') (v_f - v_f').x_ff' / "
           "(|x_ff'|^2 + 0.01 h^2) gradW + boundary term with v_b = 0";
  }
  void load(Model &m) override {
    m.add_global("smoothing_scale", ft_real());
    collect(m, true, true);
    for (auto &F : fluid_) {
      F.rho0 = &F.g->add_uniform("rest_density", ft_real());
      F.mu = &F.g->add_uniform("dynamic_viscosity", ft_real());
      F.x = &F.g->add_varying("position", ft_vec3());
      F.v = &F.g->add_varying("velocity", ft_vec3());
      F.a = &F.g->add_varying("acceleration", ft_vec3());
      F.rho = &F.g->add_varying("density", ft_real());
      F.m = &F.g->add_varying("mass", ft_real());
    }
    for (auto &B : bound_) {
      B.mu = &B.g->add_uniform("dynamic_viscosity", ft_real());
      B.x = &B.g->add_varying("position", ft_vec3());
      B.V = &B.g->add_varying("volume", ft_real());
    }
    bind(m);
  }
  template <int NF, int NB> struct L {
    static void go(Viscosity *S, FluidG &F, NbrView const &v, Globals G, cudaStream_t s) {
      uint32_t n = uint32_t(F.g->count);
      auto N = S->nbrs<NF, NB>(v, s);
      // fluid neighbour records (x, m / rho)
      for (int q = 0; q < NF; ++q) {
        FluidG &Q = S->fluid_[q];
        N.f[q].xm = S->model_->packed_xmr(Q.g, Q.x, Q.m, Q.rho, s);
      }
      ProfScope ps(S->model_->prof, "viscosity", s);
      k_viscosity<NF, NB><<<div_up(n, kNT), kNT, 0, s>>>(n, dptr<float4>(F.x), dptr<float4>(F.v), dptr<float>(F.rho),
                                                          dptr<float4>(F.a), S->u(F.rho0), S->u(F.mu), G, N);
      count_launch();
    }
  };
  void accumulate(Nhood &nh, cudaStream_t s) {
    Globals G = globals(*model_);
    need({{G.h, "smoothing_scale"}});
    // every group's sums read the accelerations of no neighbour: groups in turn
    for (auto &F : fluid_) {
      if (!F.g->count) continue;
      NbrView const &v = lists(nh, F.g, G, s);
      dispatch_fb<L>(int(fluid_.size()), int(bound_.size()), this, F, v, G, s);
      PG_LAUNCH_CHECK();
      F.a->version++;
    }
  }
};

// ---------------------------------------------------------------------------
// correction (gradient correction for wkbb18_gc)
// ---------------------------------------------------------------------------

class Correction : public SchemeCommon {
public:
  Correction() {
    reg("identity_gradient_correction", [this](Nhood &, cudaStream_t s) {
      for (auto &F : fluid_) {
        uint32_t n = uint32_t(F.g->count);
        if (!n) continue;
        k_identity9<<<div_up(n, 256), 256, 0, s>>>(n, uint32_t(F.L->cap), dptr<float>(F.L));
        count_launch();
        PG_LAUNCH_CHECK();
        F.L->version++;
      }
    });
    reg("compute_gradient_correction", [this](Nhood &nh, cudaStream_t s) { compute(nh, s); });
  }
  std::string name() const override { return "correction"; }
  std::string source() const override {
    return "procedures identity_gradient_correction (L = I), compute_gradient_correction (L_f = invert_pm(sum_fluid "
           "(m_f' / rho_f) gradW(x_ff') (x_f' - x_f)^T))";
  }
  void load(Model &m) override {
    m.add_global("smoothing_scale", ft_real());
    collect(m, true, false);
    for (auto &F : fluid_) {
      F.x = &F.g->add_varying("position", ft_vec3());
      F.rho = &F.g->add_varying("density", ft_real());
      F.m = &F.g->add_varying("mass", ft_real());
      F.L = &F.g->add_varying("gradient_correction", ft_mat3());
    }
    bind(m);
  }
  template <int NF, int NB> struct L {
    static void go(Correction *S, FluidG &F, NbrView const &v, Globals G, cudaStream_t s) {
      uint32_t n = uint32_t(F.g->count);
      auto N = S->nbrs<NF, 0>(v, s);
      ProfScope ps(S->model_->prof, "correction", s);
      k_correction<NF, 0><<<div_up(n, kNT), kNT, 0, s>>>(n, uint32_t(F.L->cap), dptr<float4>(F.x), dptr<float>(F.rho),
                                                          dptr<float>(F.L), G, N);
      count_launch();
    }
  };
  void compute(Nhood &nh, cudaStream_t s) {
    Globals G = globals(*model_);
    need({{G.h, "smoothing_scale"}});
    // every group's sums read positions, masses and densities only
    for (auto &F : fluid_) {
      if (!F.g->count) continue;
      NbrView const &v = lists(nh, F.g, G, s);
      dispatch_fb<L>(int(fluid_.size()), 0, this, F, v, G, s);
      PG_LAUNCH_CHECK();
      F.L->version++;
    }
  }
};

using Factory = std::unique_ptr<Scheme> (*)();

std::unique_ptr<Scheme> make_wkbb18_gc() { return std::unique_ptr<Scheme>(new Wkbb18(true)); }

template <class S> std::unique_ptr<Scheme> make() { return std::unique_ptr<Scheme>(new S()); }

std::map<std::string, Factory> const &registry() {
  static std::map<std::string, Factory> r = [] {
    std::map<std::string, Factory> m;
    auto add = [&](Factory f) { m[f()->full_name()] = f; };
    add(&make<Aiast12>);
    add(&make<Density>);
    add(&make<Gravity>);
    add(&make<Iisph>);
    add(&make<SymplecticEuler>);
    add(&make<Wkbb18>);
    add(&make<Viscosity>);
    add(&make<Correction>);
    add(&make_wkbb18_gc);
    return m;
  }();
  return r;
}

} // namespace

namespace {
std::map<std::string, SchemeFactory> &added() {
  static std::map<std::string, SchemeFactory> m;
  return m;
}
} // namespace

void register_scheme(std::string const &full_name, SchemeFactory f) {
  if (registry().count(full_name) || added().count(full_name))
    throw Error("scheme is already registered: " + full_name);
  added()[full_name] = std::move(f);
}

std::unique_ptr<Scheme> new_scheme(std::string const &full_name) {
  auto const &r = registry();
  auto it = r.find(full_name);
  if (it != r.end()) return it->second();
  auto jt = added().find(full_name);
  if (jt != added().end()) return jt->second();
  throw Error("scheme is not registered");
}

std::vector<std::string> scheme_names() {
  std::vector<std::string> v;
  for (auto &kv : registry()) v.push_back(kv.first);
  for (auto &kv : added()) v.push_back(kv.first);
  return v;
}

} // namespace prtcl_gpu
