// Sweeps: several time steps in one launch, in place.
//
// A step kernel streams the whole lattice through HBM. A sweep runs two (or
// more) consecutive steps over the x planes as a wavefront, step s + 1 a few
// planes behind step s, so a plane's populations are read from HBM once, stay
// in the L2 between the steps, and are written back once: half of the HBM
// traffic of two steps (ncu, 128 x 256 x 256, FP64, compact: 1.06 GB read and
// 1.06 GB written for two steps, against 2.0 GB each).
//
// In place for every pattern. A pair of AA steps (local even, shifted odd)
// takes a natural state to a natural state in one lattice. The push state is
// natural too, so two push steps are that pair. The pull state keeps f_d(x)
// at (d, x - c_d) and, behind a wall, at (inv d, x): these are the slots the
// AA odd step gathers with d and inv d exchanged, so two pull steps are a
// shifted and then a local step with every plane index inverted (FLIP). The
// second lattice of push and pull is not touched, and each cell goes through
// the same operations in the same order as in the single-step kernels: the
// states are bit-identical.
//
// Order and dependencies (lbm_sweep_plan.h). A cell of step s reads and
// writes slots of its own and its neighbours' cells, all of which step s - 1
// must have finished: planes x - 1, x, x + 1. Each block of a step that has a
// successor raises its plane's counter when its stores are done, and a block
// of the next step waits for the counters it needs. Everything a block waits
// for has a lower block index, and blocks are dispatched in index order (as
// chained-scan kernels assume), so it is running or done; taking the order
// from an atomic ticket instead cost 5.7% (0.553 against 0.522 ms a step at
// 256^3). Every wait has an iteration limit all the same, after which the
// kernel sets the solver's error word and goes on (its accesses are in range
// whatever the order); the host then reports it and keeps to single steps.
//   fronts (lattice larger than the L2): two steps, the second `lag` planes
//     behind the first.
//   step-major (lattice in the L2): all planes of a step, then the next
//     step's, up to 32 steps a launch: no launch gaps, and no end of a step
//     at which the chip runs empty.
// What was measured and left out: one signal and one wait per warp (0.72 ms;
// the counter's line serialises them), both steps of a front in one block
// (0.74 ms), persistent blocks with the next ticket fetched ahead (0.62 ms),
// two items per block (0.61 ms), unspaced counters (0.57 ms).
#pragma once

#include "lbm_step_cp.cuh"
#include "lbm_sweep_plan.h"

namespace lbm {

static_assert(kSweepThreads == kStepThreads, "block size");

__device__ __forceinline__ uint32_t ld_acquire(const uint32_t *p)
{
  uint32_t v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// One warp waits until step s - 1 has finished what the item needs of it.
__device__ __forceinline__ void sweep_wait(const SweepPlan &p, int nx, const SweepItem &it,
    int lane)
{
  int j = 0, x = 0;
  const bool need = lane < 9 && sweep_needs(it, nx, lane, j, x);
  const uint32_t *c = p.done + sweep_counter(p, nx, it.s - 1, need ? j : 0, x);
  const uint32_t target = p.nb[(it.s - 1) & 1];
  for (uint32_t n = 0;; ++n) {
    if (__all_sync(0xFFFFFFFFu, !need || ld_acquire(c) >= target))
      break;
    // the error word ends the wait early: an error, or polls counted as made
    // (a limit in the arguments cost registers: dense pull 1.8% slower)
    if (n >= kSweepSpin || ((n & 15u) == 15u && ld_acquire(p.err) > kSweepSpin - n)) {
      if (lane == 0)
        atomicOr(p.err, kErrSweepWait);
      break;
    }
    __nanosleep(64);
  }
}

// STREAM: stores of the second step of fronts, whose lines are not read again
// before they leave the L2, are marked evict-first (0.554 -> 0.522 ms).
template <bool STREAM, typename S> __device__ __forceinline__ void sweep_store(S *p, S v)
{
  if constexpr (STREAM)
    __stcs(p, v);
  else
    *p = v;
}

// The same value, unknown to the compiler: the scatter of an in-place step
// computes its offsets again (a multiply-add each) instead of keeping the
// gather's, which are the same set, live across the collision (spills).
__device__ __forceinline__ uint32_t recompute(uint32_t v)
{
  asm volatile("" : "+r"(v));
  return v;
}

// BODY: local(a, item, tid, wait) and shifted(a, item, tid, wait) update one
// block's share of an item. They look up indices and masks, which no step
// changes, then call wait() (block-wide: one warp polls) and only then touch
// populations, with plain loads: the acquire in wait() orders them after the
// previous step's stores. kLocalFirst: even steps of the sweep are local.
template <class BODY>
__global__ void __launch_bounds__(kStepThreads, BODY::kMinBlocks)
    sweep_kernel(const __grid_constant__ typename BODY::Args a)
{
  const SweepPlan &p = a.p;
  SweepItem it;
  if (!sweep_item(p, a.g.nx, a.g.ny, blockIdx.x, it))
    return;
  const int tid = threadIdx.x;
  auto wait = [&] {
    if (it.s > 0) {
      if (tid < 32)
        sweep_wait(p, a.g.nx, it, tid);
      __syncthreads();
    }
  };
  if (((it.s & 1) == 0) == BODY::kLocalFirst)
    BODY::local(a, it, tid, wait);
  else
    BODY::shifted(a, it, tid, wait);
  if (it.s + 1 < p.steps) {
    __syncthreads();
    if (tid == 0)
      asm volatile("red.release.gpu.global.add.u32 [%0], 1;"
                   :: "l"(p.done + sweep_counter(p, a.g.nx, it.s, it.j, it.x)) : "memory");
  }
}

// Row and unit of warp `warp` of an item's block; false past its rows.
__device__ __forceinline__ bool sweep_unit(const SweepPlan &p, int ny, const SweepItem &it,
    int warp, int &y, uint32_t &unit)
{
  const uint32_t u = it.b * kSweepWarps + (uint32_t)warp;
  const uint32_t q = p.units == 1 ? u : __umulhi(u, p.umagic);
  unit = u - q * p.units;
  y = it.r0 + (int)q;
  const bool ok = y < it.r1;
  y += it.rot;
  if (y >= ny)
    y -= ny;
  return ok;
}

// Compact layout: the stored cells of an item's rows as up to two ranges of
// storage numbers (the second one: rows that wrap past the last).
struct SweepCells {
  uint32_t c0, n0, c1, n1;
};
__device__ __forceinline__ uint32_t row_start(const Grid &g, int x, int y)
{
  return __ldg(&g.wb[((uint32_t)x * (uint32_t)g.ny + (uint32_t)y) * (uint32_t)g.W].y);
}
__device__ __forceinline__ SweepCells sweep_cells(const Grid &g, const SweepItem &it)
{
  const int a = it.r0 + it.rot, e = it.r1 + it.rot;
  SweepCells c;
  c.c0 = row_start(g, it.x, a);
  c.n0 = row_start(g, it.x, min(e, g.ny)) - c.c0; // row ny: the next plane's first
  c.c1 = c.n1 = 0;
  if (e > g.ny) {
    c.c1 = row_start(g, it.x, 0);
    c.n1 = row_start(g, it.x, e - g.ny) - c.c1;
  }
  return c;
}

// Asks the L2 for what the same block of the next plane will read in a local
// first step: its populations come from HBM (0.522 -> 0.512 ms; two planes
// ahead 0.524).
template <int CELLS, typename S>
__device__ __forceinline__ void sweep_prefetch(const Grid &g, const S *src,
    const uint32_t *mask, const SweepItem &it, int tid)
{
  if (tid > Q || it.x + 1 >= g.nx)
    return;
  const uint32_t lo = row_start(g, it.x + 1, it.r0) + it.b * CELLS;
  const uint32_t hi = min(lo + CELLS, row_start(g, it.x + 1, it.r1));
  if (lo >= hi)
    return;
  if (tid < Q)
    l2_prefetch_bytes(src + (long long)tid * g.plane, (unsigned long long)lo * sizeof(S),
        (unsigned long long)hi * sizeof(S));
  else
    l2_prefetch_bytes(mask, lo * 4ull, hi * 4ull);
}

// RowTab for a sweep's shifted step. Where z wraps, RowTab::at looks each of the
// ten neighbours above and below up when it is asked, one after the other, and
// a sweep asks twice, behind its wait: sweeps of z-periodic boxes were slower
// than single steps (256^3 without walls, us a step, single / lookups / this
// table: FP64 pull 803 / 909 / 612, AA 852 / 709 / 630, FP32 pull 461 / 523 /
// 312; FP64 AA 32^3 5.1 / 5.8 / 3.3). Here they are six more entries of the table:
// the first cell of a row is stored at the row's start and the last one before
// the next row's start, and those words are loaded together before the wait.
template <bool ZPER> struct SweepTab : RowTab<ZPER> {
  using T = RowTab<ZPER>;
  static constexpr int kRows = kTabRows + (ZPER ? 6 : 0);

  // entry of row q's z - 1 (the index is one less); 4, the own row
  __device__ __forceinline__ static int below(int q)
  {
    return kTabRows + (q == 1 ? 0 : q == 3 ? 1 : q == 5 ? 2 : q == 7 ? 3 : 4);
  }
  static constexpr int kOwnAbove = kTabRows + 5;

  __device__ __forceinline__ void build(const Grid &g, int x, int y, int z, uint32_t cell,
      uint32_t wi, uint32_t lt, int lane, uint32_t k0)
  {
    T::template build<true>(g, x, y, z, cell, wi, lt, lane, k0);
    if constexpr (ZPER) {
      const bool first = z == 0, last = z == g.nz - 1;
#pragma unroll
      for (int i = 0; i < 5; ++i) {
        const int q = i < 4 ? 2 * i + 1 : 4;
        int xr = x + q / 3 - 1, yr = y + q % 3 - 1;
        xr = xr < 0 ? g.nx - 1 : xr >= g.nx ? 0 : xr;
        yr = yr < 0 ? g.ny - 1 : yr >= g.ny ? 0 : yr;
        const uint32_t row = (uint32_t)xr * (uint32_t)g.ny + (uint32_t)yr;
        const int up = q == 4 ? kOwnAbove : T::axis_slot(q);
        uint32_t lo = T::B[q], hi = q == 4 ? cell + 1u : T::B[up];
        if (first)
          lo = __ldg(&g.wb[(row + 1u) * (uint32_t)g.W].y);
        if (last)
          hi = __ldg(&g.wb[row * (uint32_t)g.W].y);
        T::sB[below(q) * kStepThreads] = lo;
        T::sB[up * kStepThreads] = hi;
        if (q != 4)
          T::B[up] = hi;
      }
    }
  }

  __device__ __forceinline__ uint32_t at(const Grid &g, int d, bool regs = false) const
  {
    if constexpr (ZPER) {
      const int q = (cx(d) + 1) * 3 + (cy(d) + 1);
      if (cz(d) < 0)
        return T::sB[below(q) * kStepThreads] - 1u;
      if (cz(d) > 0)
        return q == 4 ? T::sB[kOwnAbove * kStepThreads] : T::entry(T::axis_slot(q), regs);
      return T::entry(q, regs);
    } else {
      return T::at(g, d, regs);
    }
  }
};

template <class ST> struct SweepArgs {
  Grid g;
  const typename ST::S *src; // the lattice, twice: with one pointer the compiler keeps
  typename ST::S *dst;       // the 19 load addresses for the stores (spills)
  const uint32_t *mask;
  Consts<typename ST::V> c;
  SweepPlan p;
};

// 64 registers: 8 blocks per SM (7: 0.528 ms, 6: 0.584, 8: 0.522).
#ifndef LBM_MINB_SWEEP_F64
#define LBM_MINB_SWEEP_F64 8
#endif

// FP64, compact layout, one cell per thread. OFF as in step_kernel_cp.
template <class ST, bool FORCE, bool FLIP, bool ZPER, bool FRONTS, typename OFF>
struct SweepCp {
  using Args = SweepArgs<ST>;
  using V = typename ST::V;
  static constexpr int kMinBlocks = LBM_MINB_SWEEP_F64;
  static constexpr bool kLocalFirst = !FLIP;

  __device__ static OFF el(const Args &a, int plane, uint32_t i)
  {
    return (OFF)(FLIP ? inv(plane) : plane) * (OFF)a.g.plane + (OFF)i;
  }

  // AA even: slot d of x -> slot inv d of x
  template <class WAIT>
  __device__ __forceinline__ static void local(const Args &a, const SweepItem &it, int tid,
      WAIT &&wait)
  {
    const SweepCells sc = sweep_cells(a.g, it);
    const uint32_t i = it.b * kStepThreads + (uint32_t)tid;
    uint32_t cell = i < sc.n0 ? sc.c0 + i : sc.c1 + (i - sc.n0);
    if (FRONTS && kLocalFirst)
      sweep_prefetch<kStepThreads>(a.g, a.src, a.mask, it, tid);
    wait();
    if (i >= sc.n0 + sc.n1)
      return;
    V v[Q];
    const uint32_t mask = __ldg(a.mask + cell);
#pragma unroll
    for (int d = 0; d < Q; ++d)
      v[d] = ST::decode(a.src[el(a, d, cell)], a.c.inv_scale);
    V o[Q];
    collide<V, false>(v, o, a.c, V(0));
    cell = recompute(cell);
#pragma unroll
    for (int d = 0; d < Q; ++d) {
      const bool bb = (mask >> d) & 1u;
      const V w = FORCE ? o[d] + force_term(a.c.force, d, bb) : o[d];
      sweep_store<FRONTS && !kLocalFirst>(a.dst + el(a, inv(d), cell), ST::encode(w, a.c.scale));
    }
  }

  // AA odd: slot inv d of x - c_d -> slot d of x + c_d (step_kernel_cp)
  template <class WAIT>
  __device__ __forceinline__ static void shifted(const Args &a, const SweepItem &it, int tid,
      WAIT &&wait)
  {
    __shared__ uint32_t tab[SweepTab<ZPER>::kRows * kStepThreads];
    const Grid &g = a.g;
    const int lane = tid & 31;
    int y;
    uint32_t wi;
    SweepTab<ZPER> t;
    t.sB = tab + tid;
    bool fluid = false;
    uint32_t cell = 0, mask = 0;
    if (sweep_unit(a.p, g.ny, it, tid >> 5, y, wi)) {
      const uint32_t lt = (1u << lane) - 1u;
      const uint32_t k0 = ((uint32_t)it.x * (uint32_t)g.ny + (uint32_t)y) * (uint32_t)g.W + wi;
      const uint2 wb0 = __ldg(g.wb + k0);
      fluid = (wb0.x >> lane) & 1u;
      cell = wb0.y + (uint32_t)__popc(wb0.x & lt);
      mask = __ldg(a.mask + (fluid ? cell : 0u));
      t.build(g, it.x, y, (int)(32u * wi) + lane, cell, wi, lt, lane, k0);
    }
    wait();
    if (!fluid)
      return;
    V v[Q];
    if (!__any_sync(__activemask(), (mask & 0x7FFFFu) != 0u)) {
#pragma unroll
      for (int d = 0; d < Q; ++d)
        v[d] = ST::decode(a.src[el(a, inv(d), t.at(g, inv(d), true))], a.c.inv_scale);
    } else {
#pragma unroll
      for (int d = 0; d < Q; ++d) {
        const bool back = (mask >> inv(d)) & 1u;
        const OFF o = back ? el(a, d, cell) : el(a, inv(d), t.at(g, inv(d), true));
        v[d] = ST::decode(a.src[o], a.c.inv_scale);
      }
    }
    V o[Q];
    collide<V, false>(v, o, a.c, V(0));
    cell = recompute(cell);
#pragma unroll
    for (int d = 0; d < Q; ++d) {
      const bool bb = (mask >> d) & 1u;
      const V w = FORCE ? o[d] + force_term(a.c.force, d, bb) : o[d];
      sweep_store<FRONTS && kLocalFirst>(a.dst + (bb ? el(a, inv(d), cell) : el(a, d, t.at(g, d))),
          ST::encode(w, a.c.scale));
    }
  }
};

// Blocks per SM, from AA and push / pull at 256^3: 8 0.564 / 0.585 ms, 7 0.529 /
// 0.601, 6 0.542 / 0.638.
#ifndef LBM_MINB_SWEEP_DENSE
#define LBM_MINB_SWEEP_DENSE 7
#endif
#ifndef LBM_MINB_SWEEP_DENSE_PULL
#define LBM_MINB_SWEEP_DENSE_PULL 8
#endif

// FP64, dense layout, one cell per thread (step_kernel). BRINK adds the
// Brinkman term of a.porosity, and saves each step's momentum (3 planes a step,
// u_save from the sweep's first step on) when u_save is set. Offsets of the 19 planes fit 32 bits (checked
// at planning).
template <class ST> struct SweepArgsD : SweepArgs<ST> {
  const float *porosity;
  typename ST::V *u_save;
};

template <class ST, bool FORCE, bool FLIP, bool BRINK, bool FRONTS> struct SweepDense {
  using Args = SweepArgsD<ST>;
  using V = typename ST::V;
  static constexpr int kMinBlocks = FLIP ? LBM_MINB_SWEEP_DENSE_PULL : LBM_MINB_SWEEP_DENSE;
  static constexpr bool kLocalFirst = !FLIP;

  __device__ static uint32_t el(const Args &a, int plane, uint32_t i)
  {
    return (uint32_t)(FLIP ? inv(plane) : plane) * (uint32_t)a.g.plane + i;
  }

  template <bool SHIFTED, class WAIT>
  __device__ __forceinline__ static void step(const Args &a, const SweepItem &it, int tid,
      WAIT &&wait)
  {
    constexpr bool kLast = SHIFTED == kLocalFirst;
    const Grid &g = a.g;
    int y;
    uint32_t unit;
    uint32_t cell = 0, mask = kSolidBit;
    const bool row_ok = sweep_unit(a.p, g.ny, it, tid >> 5, y, unit);
    const int z = (int)(32u * unit) + (tid & 31);
    if (row_ok && z < g.nz) {
      cell = cell_index(g, it.x, y, z);
      mask = __ldg(a.mask + cell);
    }
    if (FRONTS && !kLast && !SHIFTED && tid <= Q && it.x + 1 < g.nx) {
      // what this block's share of the next plane's rows will read
      const uint32_t lo = cell_index(g, it.x + 1, it.r0, 0) + it.b * kStepThreads;
      const uint32_t hi = min(lo + kStepThreads, cell_index(g, it.x + 1, it.r1, 0));
      if (lo < hi) {
        if (tid < Q)
          l2_prefetch_bytes(a.src + tid * g.plane, (unsigned long long)lo * sizeof(V),
              (unsigned long long)hi * sizeof(V));
        else
          l2_prefetch_bytes(a.mask, lo * 4ull, hi * 4ull);
      }
    }
    wait();
    if (mask & kSolidBit)
      return;
    const Offs of = make_offs(g, it.x, y, z);
    V v[Q];
    if (!SHIFTED) {
#pragma unroll
      for (int d = 0; d < Q; ++d)
        v[d] = ST::decode(a.src[el(a, d, cell)], a.c.inv_scale);
    } else if (!__any_sync(__activemask(), (mask & 0x7FFFFu) != 0u)) {
#pragma unroll
      for (int d = 0; d < Q; ++d)
        v[d] = ST::decode(a.src[el(a, inv(d), cell + of.at(inv(d)))],
            a.c.inv_scale);
    } else {
#pragma unroll
      for (int d = 0; d < Q; ++d) {
        const bool back = (mask >> inv(d)) & 1u;
        const uint32_t o = back ? el(a, d, cell) : el(a, inv(d), cell + of.at(inv(d)));
        v[d] = ST::decode(a.src[o], a.c.inv_scale);
      }
    }
    V kappa = V(0);
    if (BRINK)
      kappa = a.c.alpha * (V(1.0) - V(a.porosity[cell]));
    V o[Q];
    V u3[3];
    collide<V, BRINK>(v, o, a.c, kappa, BRINK ? u3 : nullptr);
    cell = recompute(cell);
    if (BRINK && a.u_save) {
      V *u = a.u_save + 3 * (long long)it.s * g.plane + cell;
      u[0] = u3[0];
      u[g.plane] = u3[1];
      u[2 * g.plane] = u3[2];
    }
#pragma unroll
    for (int d = 0; d < Q; ++d) {
      const bool bb = (mask >> d) & 1u;
      const V w = FORCE ? o[d] + (bb ? a.c.force[inv(d)] : a.c.force[d]) : o[d];
      const uint32_t o = !SHIFTED || bb ? el(a, inv(d), cell) : el(a, d, cell + of.at(d));
      sweep_store<FRONTS && kLast>(a.dst + o, ST::encode(w, a.c.scale));
    }
  }
  template <class WAIT>
  __device__ __forceinline__ static void local(const Args &a, const SweepItem &it, int tid,
      WAIT &&wait)
  {
    step<false>(a, it, tid, wait);
  }
  template <class WAIT>
  __device__ __forceinline__ static void shifted(const Args &a, const SweepItem &it, int tid,
      WAIT &&wait)
  {
    step<true>(a, it, tid, wait);
  }
};

} // namespace lbm
