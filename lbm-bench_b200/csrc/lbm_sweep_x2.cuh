// Sweeps (lbm_sweep.cuh) of the reduced-precision storage modes in the
// compact layout: two cells per thread with the pair arithmetic, operation for
// operation that of the single-step kernels (lbm_step_cp2.cuh).
//
// FP32 at 256^3 (20% solid): 0.310 ms a step (AA, push) and 0.314 (pull)
// against 0.357, 0.439 and 0.388 in single steps. HBM is then at 48% of its
// peak; what bounds it is the L1's request rate to the L2 (66% busy: a warp's
// store is 128 bytes, half of an FP64 one) and instruction issue (61%).
// FP16 halves the bytes but not the requests and takes the same 0.310 ms, so
// its AA steps (0.274 ms) sweep only where the launch gaps count.
#pragma once

#include "lbm_step_cp2.cuh"
#include "lbm_sweep.cuh"

namespace lbm {

template <class ST> struct SweepArgs2 {
  Grid g;
  const typename ST::S *src;
  typename ST::S *dst;
  const uint32_t *mask;
  Consts2 c;
  SweepPlan p;
};

// 64 registers: 8 blocks per SM (9: 0.330 ms, 7: 0.313, 6: 0.327; 8: 0.310).
#ifndef LBM_MINB_SWEEP_CP2
#define LBM_MINB_SWEEP_CP2 8
#endif

// Compact layout. Local step: two consecutive stored cells per thread.
// Shifted step: cells z and z + 32 of one row per thread.
template <class ST, bool FORCE, bool FLIP, bool ZPER, bool FRONTS, typename OFF>
struct SweepCp2 {
  using Args = SweepArgs2<ST>;
  using PT = PairOf<ST>;
  using S = typename PT::S;
  using P = typename PT::P;
  static constexpr int kMinBlocks = LBM_MINB_SWEEP_CP2;
  static constexpr bool kLocalFirst = !FLIP;

  __device__ static OFF el(const Args &a, int plane, uint32_t i)
  {
    return (OFF)(FLIP ? inv(plane) : plane) * (OFF)a.g.plane + (OFF)i;
  }

  // The pair (cell, cell + 1), cell even.
  __device__ __forceinline__ static void local_pair(const Args &a, uint32_t cell)
  {
    const uint2 m = *reinterpret_cast<const uint2 *>(a.mask + cell);
    float2 f[Q];
#pragma unroll
    for (int d = 0; d < Q; ++d)
      f[d] = PT::dec(*reinterpret_cast<const P *>(a.src + el(a, d, cell)));
    float2 o[Q];
    collide2<false>(f, o, a.c, f2(0.f), nullptr);
#pragma unroll
    for (int d = 0; d < Q; ++d) {
      const float2 v = FORCE ? add_force2(o[d], d, m.x, m.y, a.c.force) : o[d];
      sweep_store<FRONTS && !kLocalFirst>(reinterpret_cast<P *>(a.dst + el(a, inv(d), cell)),
          PT::enc(v));
    }
  }

  // One cell whose pair partner belongs to another item (collide1 repeats
  // collide2's operations).
  __device__ __forceinline__ static void local_one(const Args &a, uint32_t cell)
  {
    const uint32_t m = a.mask[cell];
    float f[Q], o[Q];
#pragma unroll
    for (int d = 0; d < Q; ++d)
      f[d] = PT::dec1(a.src[el(a, d, cell)]);
    collide1(f, o, a.c);
#pragma unroll
    for (int d = 0; d < Q; ++d)
      a.dst[el(a, inv(d), cell)] =
          PT::enc1(FORCE ? __fadd_rn(o[d], force_term(a.c.force, d, (m >> d) & 1u)) : o[d]);
  }

  template <class WAIT>
  __device__ __forceinline__ static void local(const Args &a, const SweepItem &it, int tid,
      WAIT &&wait)
  {
    const SweepCells sc = sweep_cells(a.g, it);
    // pairs start at even cells: the first and last of a range may be partial
    uint32_t i = it.b * kStepThreads + (uint32_t)tid;
    uint32_t lo = sc.c0, hi = sc.c0 + sc.n0;
    uint32_t cell = (lo & ~1u) + 2u * i;
    if (cell >= hi && sc.n1) {
      i -= (hi - (lo & ~1u) + 1u) / 2u;
      lo = sc.c1;
      hi = sc.c1 + sc.n1;
      cell = (lo & ~1u) + 2u * i;
    }
    if (FRONTS && kLocalFirst)
      sweep_prefetch<2 * kStepThreads>(a.g, a.src, a.mask, it, tid);
    wait();
    if (cell >= hi)
      return;
    if (cell >= lo && cell + 1u < hi)
      local_pair(a, cell);
    else if (cell >= lo)
      local_one(a, cell);
    else if (cell + 1u < hi)
      local_one(a, cell + 1u);
  }

  template <class WAIT>
  __device__ __forceinline__ static void shifted(const Args &a, const SweepItem &it, int tid,
      WAIT &&wait)
  {
    __shared__ uint32_t tab[2 * kTabRows * kStepThreads];
    const Grid &g = a.g;
    const int lane = tid & 31;
    int y;
    uint32_t unit;
    RowTab<ZPER> t0, t1;
    t0.sB = tab + tid;
    t1.sB = tab + kTabRows * kStepThreads + tid;
    bool fl0 = false, fl1 = false;
    uint32_t cell0 = 0, cell1 = 0, m0 = 0, m1 = 0;
    if (sweep_unit(a.p, g.ny, it, tid >> 5, y, unit)) {
      const uint32_t wi0 = 2u * unit;
      const bool has1 = wi0 + 1u < (uint32_t)g.W;
      const uint32_t lt = (1u << lane) - 1u;
      const uint32_t k0 = ((uint32_t)it.x * (uint32_t)g.ny + (uint32_t)y) * (uint32_t)g.W + wi0;
      const uint2 wb0 = __ldg(g.wb + k0);
      const uint2 wb1 = has1 ? __ldg(g.wb + k0 + 1u) : make_uint2(0u, 0u);
      fl0 = (wb0.x >> lane) & 1u;
      fl1 = (wb1.x >> lane) & 1u;
      cell0 = wb0.y + (uint32_t)__popc(wb0.x & lt);
      cell1 = wb1.y + (uint32_t)__popc(wb1.x & lt);
      m0 = fl0 ? __ldg(a.mask + cell0) : 0u;
      m1 = fl1 ? __ldg(a.mask + cell1) : 0u;
      const int z0 = 32 * (int)wi0 + lane;
      t0.template build<true>(g, it.x, y, z0, cell0, wi0, lt, lane, k0);
      if (has1)
        t1.template build<true>(g, it.x, y, z0 + 32, cell1, wi0 + 1u, lt, lane, k0 + 1u);
    }
    wait();
    if (!fl0 && !fl1)
      return;
    auto ld = [&](bool fl, OFF o) { return fl ? PT::dec1(a.src[o]) : 0.0f; };
    float2 f[Q];
    if (!__any_sync(__activemask(), ((m0 | m1) & 0x7FFFFu) != 0u)) {
#pragma unroll
      for (int d = 0; d < Q; ++d)
        f[d] = make_float2(ld(fl0, el(a, inv(d), t0.at(g, inv(d), true))),
                           ld(fl1, el(a, inv(d), t1.at(g, inv(d), true))));
    } else {
#pragma unroll
      for (int d = 0; d < Q; ++d) {
        const bool b0 = (m0 >> inv(d)) & 1u, b1 = (m1 >> inv(d)) & 1u;
        const OFF o0 = b0 ? el(a, d, cell0) : el(a, inv(d), t0.at(g, inv(d), true));
        const OFF o1 = b1 ? el(a, d, cell1) : el(a, inv(d), t1.at(g, inv(d), true));
        f[d] = make_float2(ld(fl0, o0), ld(fl1, o1));
      }
    }
    float2 o[Q];
    collide2<false>(f, o, a.c, make_float2(0.0f, 0.0f), nullptr);
#pragma unroll
    for (int d = 0; d < Q; ++d) {
      const float2 v = FORCE ? add_force2(o[d], d, m0, m1, a.c.force) : o[d];
      S *q0 = a.dst + (((m0 >> d) & 1u) ? el(a, inv(d), cell0) : el(a, d, t0.at(g, d)));
      S *q1 = a.dst + (((m1 >> d) & 1u) ? el(a, inv(d), cell1) : el(a, d, t1.at(g, d)));
      if (fl0)
        sweep_store<FRONTS && kLocalFirst>(q0, PT::enc1(v.x));
      if (fl1)
        sweep_store<FRONTS && kLocalFirst>(q1, PT::enc1(v.y));
    }
  }
};

} // namespace lbm
