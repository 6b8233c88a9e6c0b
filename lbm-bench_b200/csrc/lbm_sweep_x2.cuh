// Sweeps (lbm_sweep.cuh) of the reduced-precision storage modes, two cells per
// thread with the pair arithmetic, operation for operation that of the
// single-step kernels (lbm_step_x2.cuh, lbm_step_cp2.cuh).
//
// At 256^3 (20% solid), ms a step, sweeps / single steps:
//   compact FP32  AA 0.303 / 0.357   pull 0.305 / 0.388   push 0.303 / 0.439
//   dense FP32    AA 0.310 / 0.487   pull 0.330 / 0.406   push 0.310 / 0.619
//   dense FP16    AA 0.310 / 0.353   push 0.309 / 0.417
// HBM is then at 48% of its peak; what bounds a sweep is the L1's request rate
// to the L2 (66% busy: a warp's store is 128 bytes, half of an FP64 one) and
// instruction issue (61%). FP16 halves the bytes but not the requests and
// takes the same time, so compact FP16 AA (0.274 in single steps) sweeps only
// where the launch gaps count.
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

// 64 registers: 8 blocks per SM (FP32 AA 9: 0.330 ms, 8: 0.310, 7: 0.313, 6: 0.327).
#ifndef LBM_MINB_SWEEP_CP2
#define LBM_MINB_SWEEP_CP2 8
#endif

// Compact layout. Local step: two consecutive stored cells per thread.
// Shifted step: cells z and z + 32 of one row per thread. Offsets of the 19
// planes fit 32 bits (checked at planning).
template <class ST, bool FORCE, bool FLIP, bool ZPER, bool FRONTS> struct SweepCp2 {
  using Args = SweepArgs2<ST>;
  using PT = PairOf<ST>;
  using S = typename PT::S;
  using P = typename PT::P;
  static constexpr int kMinBlocks = LBM_MINB_SWEEP_CP2;
  static constexpr bool kLocalFirst = !FLIP;

  __device__ static uint32_t el(const Args &a, int plane, uint32_t i)
  {
    return (uint32_t)(FLIP ? inv(plane) : plane) * (uint32_t)a.g.plane + i;
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
    cell = recompute(cell);
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
    __shared__ uint32_t tab[2 * SweepTab<ZPER>::kRows * kStepThreads];
    const Grid &g = a.g;
    const int lane = tid & 31;
    int y;
    uint32_t unit;
    SweepTab<ZPER> t0, t1;
    t0.sB = tab + tid;
    t1.sB = tab + SweepTab<ZPER>::kRows * kStepThreads + tid;
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
      t0.build(g, it.x, y, z0, cell0, wi0, lt, lane, k0);
      if (has1)
        t1.build(g, it.x, y, z0 + 32, cell1, wi0 + 1u, lt, lane, k0 + 1u);
    }
    wait();
    if (!fl0 && !fl1)
      return;
    auto ld = [&](bool fl, uint32_t o) { return fl ? PT::dec1(a.src[o]) : 0.0f; };
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
        const uint32_t o0 = b0 ? el(a, d, cell0) : el(a, inv(d), t0.at(g, inv(d), true));
        const uint32_t o1 = b1 ? el(a, d, cell1) : el(a, inv(d), t1.at(g, inv(d), true));
        f[d] = make_float2(ld(fl0, o0), ld(fl1, o1));
      }
    }
    float2 o[Q];
    collide2<false>(f, o, a.c, make_float2(0.0f, 0.0f), nullptr);
    cell0 = recompute(cell0);
    cell1 = recompute(cell1);
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

// Blocks per SM, from AA / pull at 256^3: FP32 8 0.316 / 0.355 ms, 7 0.310 /
// 0.330, 6 0.324 / 0.360; FP16 0.310 / 0.321, 0.313 / 0.325, 0.325 / 0.330.
#ifndef LBM_MINB_SWEEP_X2
#define LBM_MINB_SWEEP_X2 7
#endif
#ifndef LBM_MINB_SWEEP_X2_F16
#define LBM_MINB_SWEEP_X2_F16 8
#endif

// Dense layout. Local step: cells z and z + 1 of one row per thread, one
// aligned pair access per plane. Shifted step: cells z and z + 32, so that
// every access of a warp is 32 consecutive elements and, away from walls and
// row ends, the second cell's is the first's address plus a constant (as
// z-adjacent pairs it needs twice the addresses, and 250-500 bytes of spills).
// BRINK adds the Brinkman term of a.porosity. Offsets of the 19 planes fit 32
// bits (checked at planning).
template <class ST> struct SweepArgsD2 : SweepArgs2<ST> {
  const float *porosity;
  float *u_save; // as in SweepArgsD
};

template <class ST, bool FORCE, bool FLIP, bool BRINK, bool FRONTS> struct SweepDense2 {
  using Args = SweepArgsD2<ST>;
  using PT = PairOf<ST>;
  using S = typename PT::S;
  using P = typename PT::P;
  static constexpr int kMinBlocks = sizeof(S) == 2 ? LBM_MINB_SWEEP_X2_F16 : LBM_MINB_SWEEP_X2;
  static constexpr bool kLocalFirst = !FLIP;

  __device__ static uint32_t el(const Args &a, int plane, uint32_t i)
  {
    return (uint32_t)(FLIP ? inv(plane) : plane) * (uint32_t)a.g.plane + i;
  }

  template <class WAIT>
  __device__ __forceinline__ static void local(const Args &a, const SweepItem &it, int tid,
      WAIT &&wait)
  {
    const Grid &g = a.g;
    int y;
    uint32_t unit;
    uint32_t cell = 0;
    uint2 m = make_uint2(kSolidBit, kSolidBit);
    const bool row_ok = sweep_unit(a.p, g.ny, it, tid >> 5, y, unit);
    const int z = (int)(64u * unit) + 2 * (tid & 31);
    if (row_ok && z < g.nz) {
      // the pair starts at an even element; a cell z + 1 = nz is padding and
      // carries the wall bit
      cell = cell_index(g, it.x, y, z);
      m = *reinterpret_cast<const uint2 *>(a.mask + cell);
    }
    if (FRONTS && kLocalFirst && tid <= Q && it.x + 1 < g.nx) {
      const uint32_t lo = cell_index(g, it.x + 1, it.r0, 0) + it.b * 2 * kStepThreads;
      const uint32_t hi = min(lo + 2 * kStepThreads, cell_index(g, it.x + 1, it.r1, 0));
      if (lo < hi) {
        if (tid < Q)
          l2_prefetch_bytes(a.src + tid * g.plane, (unsigned long long)lo * sizeof(S),
              (unsigned long long)hi * sizeof(S));
        else
          l2_prefetch_bytes(a.mask, lo * 4ull, hi * 4ull);
      }
    }
    wait();
    if (m.x & m.y & kSolidBit)
      return;
    float2 f[Q];
#pragma unroll
    for (int d = 0; d < Q; ++d)
      f[d] = PT::dec(*reinterpret_cast<const P *>(a.src + el(a, d, cell)));
    float2 kappa = f2(0.f);
    if (BRINK) {
      const float2 por = *reinterpret_cast<const float2 *>(a.porosity + cell);
      kappa = make_float2(a.c.alpha * (1.f - por.x), a.c.alpha * (1.f - por.y));
    }
    float2 o[Q], u3[3];
    collide2<BRINK>(f, o, a.c, kappa, BRINK ? u3 : nullptr);
    cell = recompute(cell);
    if (BRINK && a.u_save) {
      float *u = a.u_save + 3 * (long long)it.s * g.plane + cell;
#pragma unroll
      for (int k = 0; k < 3; ++k)
        *reinterpret_cast<float2 *>(u + k * g.plane) = u3[k];
    }
#pragma unroll
    for (int d = 0; d < Q; ++d) {
      // a wall cell's own slot is never read: both cells are written
      const float2 v = FORCE ? add_force2(o[d], d, m.x, m.y, a.c.force) : o[d];
      sweep_store<FRONTS && !kLocalFirst>(reinterpret_cast<P *>(a.dst + el(a, inv(d), cell)),
          PT::enc(v));
    }
  }

  template <class WAIT>
  __device__ __forceinline__ static void shifted(const Args &a, const SweepItem &it, int tid,
      WAIT &&wait)
  {
    constexpr bool kStream = FRONTS && kLocalFirst;
    const Grid &g = a.g;
    int y;
    uint32_t unit;
    uint32_t cell = 0, m0 = kSolidBit, m1 = kSolidBit;
    const bool row_ok = sweep_unit(a.p, g.ny, it, tid >> 5, y, unit);
    const int z = (int)(64u * unit) + (tid & 31);
    if (row_ok && z < g.nz) {
      cell = cell_index(g, it.x, y, z);
      m0 = __ldg(a.mask + cell);
      if (z + 32 < g.nz)
        m1 = __ldg(a.mask + cell + 32u);
    }
    wait();
    const bool fl0 = !(m0 & kSolidBit), fl1 = !(m1 & kSolidBit);
    if (!fl0 && !fl1)
      return;
    const Offs of = make_offs(g, it.x, y, z);
    // z neighbours of the second cell: it can only wrap at the row's end,
    // the first one only at its start (a row that ends in the first 32 cells
    // has no second cell)
    Offs of1 = of;
    of1.zm = 0u - 1u;
    of1.zp = ((g.per >> 2) & 1) && z + 32 == g.nz - 1 ? 0u - (uint32_t)(g.nz - 1) : 1u;
    auto ld = [&](bool fl, uint32_t o) { return fl ? PT::dec1(a.src[o]) : 0.0f; };
    const bool links = __any_sync(__activemask(), ((m0 | m1) & 0x7FFFFu) != 0u);
    float2 f[Q];
#pragma unroll
    for (int d = 0; d < Q; ++d) {
      const int e = inv(d); // x - c_d = x + c_e
      uint32_t p0 = el(a, inv(d), cell + of.at(e));
      uint32_t p1 = cz(e) == 0 ? p0 + 32u : el(a, inv(d), cell + 32u + of1.at(e));
      if (links) {
        p0 = ((m0 >> e) & 1u) ? el(a, d, cell) : p0;
        p1 = ((m1 >> e) & 1u) ? el(a, d, cell + 32u) : p1;
      }
      f[d] = make_float2(ld(fl0, p0), ld(fl1, p1));
    }
    float2 kappa = f2(0.f);
    if (BRINK)
      kappa = make_float2(fl0 ? a.c.alpha * (1.f - a.porosity[cell]) : 0.f,
          fl1 ? a.c.alpha * (1.f - a.porosity[cell + 32u]) : 0.f);
    float2 o[Q], u3[3];
    collide2<BRINK>(f, o, a.c, kappa, BRINK ? u3 : nullptr);
    cell = recompute(cell);
    if (BRINK && a.u_save) {
      float *u = a.u_save + 3 * (long long)it.s * g.plane + cell;
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        if (fl0)
          u[k * g.plane] = u3[k].x;
        if (fl1)
          u[k * g.plane + 32] = u3[k].y;
      }
    }
#pragma unroll
    for (int d = 0; d < Q; ++d) {
      const float2 v = FORCE ? add_force2(o[d], d, m0, m1, a.c.force) : o[d];
      uint32_t q0 = el(a, d, cell + of.at(d));
      uint32_t q1 = cz(d) == 0 ? q0 + 32u : el(a, d, cell + 32u + of1.at(d));
      q0 = ((m0 >> d) & 1u) ? el(a, inv(d), cell) : q0;
      q1 = ((m1 >> d) & 1u) ? el(a, inv(d), cell + 32u) : q1;
      if (fl0)
        sweep_store<kStream>(a.dst + q0, PT::enc1(v.x));
      if (fl1)
        sweep_store<kStream>(a.dst + q1, PT::enc1(v.y));
    }
  }
};

} // namespace lbm
