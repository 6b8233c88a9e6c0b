// Plan of a sweep (lbm_sweep.cuh): which block of the launch updates which
// cells in which step. Plain C++ (no CUDA), shared by the kernel, the host
// that sizes the launch, and a CPU test that replays the order.
#pragma once

#include <stdint.h>

#ifdef __CUDACC__
#define LBM_HD __host__ __device__
#else
#define LBM_HD
#endif

namespace lbm {

constexpr int kSweepThreads = 128;         // threads of a block
constexpr int kSweepWarps = kSweepThreads / 32;
constexpr int kSweepPad = 32;              // words between counters: a 128-byte line each
constexpr int kSweepMaxSteps = 32;         // steps of one step-major launch
constexpr uint32_t kSweepSpin = 1u << 20;  // polls of one wait (about a second)

struct SweepPlan {
  uint32_t *done = nullptr;     // [steps - 1][slabs][nx] counters, kSweepPad words apart
  unsigned int *err = nullptr;  // the solver's error word
  uint32_t nb[2] = { 0, 0 };    // blocks of a plane (and slab) in even / odd steps
  uint32_t front = 0;           // nb[0] + nb[1]
  uint32_t slab_blocks = 0;     // fronts: blocks of a slab
  uint32_t lag = 0;             // fronts: planes between the two steps; 0: step-major
  uint32_t slabs = 1, rows = 0; // y slabs and their rows
  uint32_t units = 0;           // warp units per row of a step that maps warps to rows
  uint32_t umagic = 0;          // ceil(2^32 / units), for units > 1
  uint32_t blocks = 0;          // grid size
  int steps = 2;
};

// What a block does: block b of the row positions [r0, r1) of plane x and
// slab j in step s; row = position + rot, wrapped.
struct SweepItem {
  int s, j, x, r0, r1, rot;
  uint32_t b;
};

// Row positions [r0, r1) of slab j in step s. The second step's slabs lie two
// rows before the first's: its rows, shifted up by rot = 1, then need the
// first step's rows up to the end of the same slab only. Slabs near ny may be
// empty.
LBM_HD inline void sweep_rows(const SweepPlan &p, int ny, int s, int j, int &r0, int &r1)
{
  if (p.slabs == 1) {
    r0 = 0;
    r1 = ny;
    return;
  }
  const int a = j * (int)p.rows - 2 * s, e = (j + 1) * (int)p.rows - 2 * s;
  r0 = j == 0 ? 0 : a < ny ? a : ny;
  r1 = j == (int)p.slabs - 1 || e > ny ? ny : e;
}

// The item of block t; false if the block has none (ends of the wavefront).
LBM_HD inline bool sweep_item(const SweepPlan &p, int nx, int ny, uint32_t t, SweepItem &it)
{
  int pos;
  if (p.lag) { // front w: plane w of the first step, plane w - lag of the second
    it.j = (int)(t / p.slab_blocks);
    const uint32_t r = t - (uint32_t)it.j * p.slab_blocks;
    const uint32_t w = r / p.front;
    it.b = r - w * p.front;
    it.s = it.b >= p.nb[0];
    if (it.s)
      it.b -= p.nb[0];
    pos = (int)w - (it.s ? (int)p.lag : 0);
    if (pos < 0 || pos >= nx)
      return false;
    it.x = pos + it.s;
  } else { // all planes of a step, then the next step's
    const uint32_t pair = p.front * (uint32_t)nx, first = p.nb[0] * (uint32_t)nx;
    const uint32_t u = t / pair;
    uint32_t r = t - u * pair;
    it.s = (int)(2 * u) + (r >= first);
    if (r >= first)
      r -= first;
    const uint32_t n = p.nb[it.s & 1];
    pos = (int)(r / n);
    it.b = r - (uint32_t)pos * n;
    it.j = 0;
    it.x = pos + it.s % nx;
  }
  if (it.x >= nx) // step s takes the planes in the order s, s + 1, ..., wrapped
    it.x -= nx;
  it.rot = p.slabs > 1 ? it.s : 0;
  sweep_rows(p, ny, it.s, it.j, it.r0, it.r1);
  return true;
}

// Counters that a block of step s >= 1 waits for: k = 0 .. 8, planes x - 1,
// x, x + 1 of the slabs j, j - 1 and 0 (rows that wrap). False if there is
// no such slab.
LBM_HD inline bool sweep_needs(const SweepItem &it, int nx, int k, int &j, int &x)
{
  const int q = k / 3;
  j = q == 2 ? 0 : it.j - q;
  x = it.x + k % 3 - 1;
  x = x < 0 ? nx - 1 : x >= nx ? 0 : x;
  return j >= 0;
}

LBM_HD inline uint32_t sweep_counter(const SweepPlan &p, int nx, int s, int j, int x)
{
  return (uint32_t)((s * (int)p.slabs + j) * nx + x) * kSweepPad;
}

// Sizes of a lattice for sweep_plan.
struct SweepShape {
  int nx, ny;
  uint32_t units;            // warp units per row
  const uint32_t *row_start; // compact layout: first storage number of each row (x * ny + y),
                             // with the total behind the last; NULL: local steps map rows too
  bool pair;                 // two cells per thread
  bool local_first;          // even steps of the sweep are local ones
  double plane_bytes;        // stored bytes of an x plane
  uint32_t resident;         // blocks that run at a time
};

// Blocks of an item of step parity `odd`, over all planes and slabs.
inline uint32_t sweep_blocks_per_item(const SweepShape &h, const SweepPlan &p, int odd)
{
  const bool cells = h.row_start && (odd == 0) == h.local_first;
  uint64_t most = 1;
  for (int j = 0; j < (int)p.slabs; ++j) {
    int r0, r1;
    sweep_rows(p, h.ny, odd, j, r0, r1);
    if (!cells) {
      const uint64_t n = ((uint64_t)(r1 - r0) * h.units + kSweepWarps - 1) / kSweepWarps;
      most = n > most ? n : most;
      continue;
    }
    const int rot = p.slabs > 1 ? odd : 0;
    const int a = r0 + rot, e = r1 + rot < h.ny ? r1 + rot : h.ny;
    const int wrapped = r1 + rot > h.ny ? r1 + rot - h.ny : 0;
    for (int x = 0; x < h.nx; ++x) {
      const uint32_t *row = h.row_start + (long long)x * h.ny;
      // a pair may start one cell before a range and end one cell after it
      uint64_t n = row[e] - row[a];
      n = h.pair ? (n + 2) / 2 : n;
      if (wrapped) {
        const uint64_t m = row[wrapped] - row[0];
        n += h.pair ? (m + 2) / 2 : m;
      }
      n = (n + kSweepThreads - 1) / kSweepThreads;
      most = n > most ? n : most;
    }
  }
  return (uint32_t)most;
}

// Plan of fronts (two steps) or of step-major sweeps of up to kSweepMaxSteps
// steps; false if the box is outside the index arithmetic's range.
//   Slabs: the planes between the two steps (lag + 1, and those in work) have
//   to stay in the L2. At about 9 MB per plane and slab (256^2 cells of 19
//   FP64 populations, 20% solid) that is 45 MB; 4 MB to 16 MB measured alike
//   within 3% except the dense layout's 10 MB planes, 4% better in two slabs.
//   Lag: blocks that run at a time, in planes, and the two planes a step
//   needs ahead; smaller and the second step waits (256^3: 3 planes 0.526 ms a
//   step, 4 0.517), larger and the window leaves the L2 (5 0.534, 7 0.594).
//   With two cells per thread the shifted step in front takes longer than the
//   local one behind it and wants twice the distance (FP32 pull 0.347 ms at
//   4, 0.328 at 5, 0.314 at 7), which its half-size cells leave room for.
inline bool sweep_plan(const SweepShape &h, bool fronts, SweepPlan &p)
{
  p = SweepPlan();
  p.rows = (uint32_t)h.ny;
  if (fronts) {
    const double target = 9e6;
    const int want = (int)(h.plane_bytes / target) + 1;
    const int rows = (h.ny + 2 + want - 1) / want < 8 ? 8 : (h.ny + 2 + want - 1) / want;
    const int slabs = (h.ny + 2 + rows - 1) / rows;
    if (slabs > 1) {
      p.slabs = (uint32_t)slabs;
      p.rows = (uint32_t)rows;
    }
  }
  p.units = h.units;
  p.umagic = (uint32_t)(((1ull << 32) + h.units - 1) / h.units);
  p.nb[0] = sweep_blocks_per_item(h, p, 0);
  p.nb[1] = sweep_blocks_per_item(h, p, 1);
  p.front = p.nb[0] + p.nb[1];
  uint64_t total;
  if (fronts) {
    const uint32_t ahead = (h.pair && !h.local_first ? 2u : 1u) * h.resident;
    p.lag = 2 + (ahead + p.front - 1) / p.front;
    p.slab_blocks = p.front * ((uint32_t)h.nx + p.lag);
    total = (uint64_t)p.front * ((uint64_t)h.nx + p.lag) * p.slabs;
  } else {
    total = (uint64_t)p.front * (uint64_t)h.nx * (kSweepMaxSteps / 2);
  }
  p.blocks = (uint32_t)total;
  // grid size; unit / row split by a 32-bit multiplication
  return total < (1ull << 31) &&
      ((uint64_t)h.ny * h.units + kSweepWarps) * h.units < (1ull << 32);
}

// Where a sweep is faster than single steps. A block of a sweep costs a wait
// and a release besides its cells; single steps pack cells of several planes
// into a block and have kernels for special cases that sweeps do not have
// (rows without links, rows of whole 64-cell segments).
struct SweepUse {
  int bytes;     // of a stored population
  bool aa, pull; // else push
  bool compact, zper;
  int nx, nz;
  double mb;     // lattice
  double fluid;  // fluid share of the box
  double plane_cells; // fluid cells of a plane, on average
  double fill;   // fluid cells per cell that the blocks of a step could take
  double waves;  // blocks of a step, in blocks that run at a time
};

inline SweepUse sweep_use(const SweepShape &h, const SweepPlan &p, double cells)
{
  SweepUse u = SweepUse();
  const double blocks = 0.5 * p.front * p.slabs * h.nx;
  u.nx = h.nx;
  u.compact = h.row_start != nullptr;
  u.pull = !h.local_first;
  u.mb = h.plane_bytes * h.nx / 1e6;
  u.plane_cells = cells / h.nx;
  u.fill = cells / (blocks * kSweepThreads * (h.pair ? 2 : 1));
  u.waves = blocks / h.resident;
  return u;
}

// Measured on a B200 at about 250 boxes (fully periodic, channels, pipes,
// blocks and spheres; 1 to 65535 planes) in every pattern, precision and
// layout; us per step, single steps / sweep, (fill).
inline bool sweep_pays(const SweepUse &u, bool fronts)
{
  const bool pair = u.bytes < 8, push = !u.aa && !u.pull;
  // few planes: each waits for nearly the whole step before
  if (u.nx < 4 && u.waves > 0.2) {
    if (u.compact) { // channel 2 x 300^2, FP64 AA 9.2 / 11.1; periodic 1 x 512^2, push 18.4 / 11.9,
      if (!u.zper || (u.pull && (fronts || !pair))) // pull 2 x 1000^2 102 / 109
        return false;
    } else if (!pair ? u.waves > 0.5 : u.bytes == 4 ? fronts && !u.aa : u.pull || u.waves > 3.1) {
      return false; // FP64 pull 2 x 300^2 9.3 / 11.9; FP32 pull 2 x 1000^2 51.7 / 56.7, AA 64.6 /
    }               // 52.4; FP16 pull 1 x 512^2 6.2 / 8.6
  }
  // thin planes and mostly solid boxes: blocks with few cells
  if (u.compact && u.zper) // FP32 push 16384 x 3^2 51.2 / 68.3, 4096 x 4^2 19.5 / 15.8; FP64 AA
    // 16384 x 3^2 44.1 / 49.8, 4096 x 8^2 30.7 / 22.7; pull in a fifth of 256 x 128^2 57.4 / 71.9
    return u.waves <= (pair ? 2.0 : 3.0) || (u.fluid >= 0.25 && u.plane_cells >= 16);
  if (u.compact) {
    if (u.waves <= (pair ? 2.0 : 3.0)) // 64^3 channel, FP64 AA 11.3 / 8.3, FP16 push 9.2 / 5.2
      return true;
    if (push) // FP16 channels: 2048 x 32^2 50.1 / 58.8 (half of each pair of words is
      return pair ? u.nz > 32 && u.fill >= 0.25 : u.fill >= 0.1; // missing), 1024 x 40^2 57.4 / 41.5
    if (u.pull) // FP64 pull pipe in 369 x 287 x 32 28.2 / 28.9 (0.14), 71^2 x 297 22.6 / 19.8 (0.28)
      return u.fill >= (u.bytes == 2 ? 0.15 : 0.2);
    if (u.bytes == 2) // 300^2 x 8 59.5 / 65.0 (0.17), pipe in 184 x 73 x 98 25.0 / 24.7 (0.58)
      return u.fill >= 0.4;
    if (pair && fronts) // 1024 x 40^2 (100 MB) 45.0 / 46.6 (0.62), 128^3 52.6 / 42.4,
      return u.nx >= 8 && (u.fill >= 0.75 || u.mb > 130); // 517 x 75 x 92 (164 MB) 78.5 / 73.2
    return u.fill >= 0.3; // FP64 AA 8192 x 10^2 45.1 / 57.2 (0.25), 300^2 x 8 55.0 / 53.7 (0.31)
  }
  // FP16 single pull steps of rows of whole segments: 128^3 36.9 / 41.7, channel
  // 41.4 / 43.0; periodic 64-cell rows 300 x 64^2 21.0 / 22.4
  const bool segments = u.bytes == 2 && u.pull &&
      (u.nz % 128 == 0 || (u.zper && u.nz % 64 == 0));
  if (u.waves <= (!segments ? 3.1 : u.nx >= 8 ? 2.0 : 0.2)) // 64^3 channel, FP64 AA 11.3 / 8.0,
    return true;                                            // FP32 push 10.2 / 5.0
  // a mostly solid box touches less than the L2 holds (pipe in 369 x 287 x 32:
  // FP64 AA 23.8 / 55.4, FP32 pull 24.6 / 40.5)
  if (fronts && u.fluid < 0.25)
    return false;
  if (push) // periodic 16384 x 3^2 FP64 41.0 / 49.3 (0.07); 65535 x 2^2 FP32 163 / 204 (0.02)
    return u.fill >= (!u.zper ? 0.015 : pair ? 0.03 : 0.15);
  if (u.pull) {
    if (!pair) // periodic 16384 x 3^2 38.9 / 45.6 (0.07)
      return u.fill >= (u.zper ? 0.15 : 0.05);
    if (u.bytes == 2 && (segments || u.nx < 8)) // 4 x 1000^2 76.3 / 84.2
      return false;
    // FP32 channel 248 x 329 x 24 82.0 / 85.5 (0.34); pipe in 93 x 378 x 162 82.5 / 68.1 (0.28)
    return u.fill >= (u.nz > 32 ? 0.25 : u.bytes == 4 || !u.zper ? 0.4 : 0.55);
  }
  if (!pair) // 8192 x 8^2 52.7 / 59.1 (0.25); channel 1024 x 24^2 (90 MB) 23.4 / 26.1 (0.63)
    return u.fill >= (!fronts ? 0.3 : u.mb <= 100 ? 0.7 : 0.26);
  if (u.bytes == 4) // periodic 8192 x 8^2 62.6 / 65.1 (0.12); channel 8192 x 10^2 118 / 85.7 (0.08)
    return u.fill >= (u.zper ? 0.2 : 0.015);
  // FP16 128-cell rows without walls 256^3 272 / 297, with 20% spheres 355 / 310
  return u.fill >= (u.zper ? 0.03 : 0.015) && !(u.nz % 128 == 0 && u.fluid > 0.9);
}

// Steps from which a sweep pays: a step-major launch of two steps still has the
// clearing of its counters and one full wait for two launches. Calls of lbm_run
// back to back, us a step, single steps / sweep, channels: 20^3 FP64 AA dense 4.1
// / 5.0 in calls of two steps, 4.1 / 3.7 of four; 32^3 FP32 push compact 4.2 / 5.2,
// 4.1 / 4.1; 200 x 64^2 FP16 AA compact 16.8 / 19.1; but 64^3 FP64 push dense
// 12.7 / 11.8, 20^3 FP32 push dense 6.2 / 5.2, periodic 20^2 x 40 FP16 pull
// compact 10.3 / 5.2.
inline int sweep_least(const SweepUse &u, bool fronts)
{
  if (fronts || (u.compact && u.zper))
    return 2;
  if (u.bytes == 2 && (u.compact ? u.aa : u.pull))
    return 4;
  return u.waves < 0.5 && (u.compact || u.pull || u.bytes == 8) ? 4 : 2;
}

} // namespace lbm
