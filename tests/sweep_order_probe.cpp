// Replays the block order of the sweep plans (csrc/lbm_sweep_plan.h) on random
// boxes: every cell row of every step is covered exactly once, by blocks whose
// neighbour rows in the step before are complete at lower block indices and
// among the counters the block waits for. Prints "ok <plans>".
#include <cstdio>
#include <cstdlib>
#include <set>
#include <tuple>
#include <vector>

#include "lbm_sweep_plan.h"

using namespace lbm;

static int bad(const char *what, int nx, int ny, const SweepPlan &p)
{
  std::printf("%s: nx %d ny %d slabs %u rows %u lag %u nb %u %u steps %d\n", what, nx, ny, p.slabs,
      p.rows, p.lag, p.nb[0], p.nb[1], p.steps);
  return 1;
}

int main()
{
  std::srand(7);
  int plans = 0;
  for (int n = 0; n < 1500; ++n) {
    const int nx = 1 + std::rand() % 12, ny = 1 + std::rand() % 60;
    const bool fronts = std::rand() % 2, compact = std::rand() % 2;
    SweepShape h;
    h.nx = nx;
    h.ny = ny;
    h.units = 1 + std::rand() % 3;
    h.pair = std::rand() % 2;
    h.local_first = std::rand() % 2;
    h.plane_bytes = (std::rand() % 45) * 1e6;
    h.resident = 1 + std::rand() % 40;
    std::vector<uint32_t> rows((size_t)nx * ny + 1, 0u);
    for (size_t r = 0; r + 1 < rows.size(); ++r)
      rows[r + 1] = rows[r] + std::rand() % (64 * h.units + 1);
    h.row_start = compact ? rows.data() : nullptr;
    SweepPlan p;
    if (!sweep_plan(h, fronts, p))
      return bad("refused", nx, ny, p);
    p.steps = fronts ? 2 : 2 * (1 + std::rand() % 4);
    if (!fronts)
      p.blocks = p.front * nx * (p.steps / 2);
    ++plans;
    std::vector<uint32_t> done(sweep_counter(p, nx, p.steps, 0, 0) / kSweepPad, 0u);
    auto count = [&](int s, int j, int x) -> uint32_t & {
      return done[sweep_counter(p, nx, s, j, x) / kSweepPad];
    };
    std::set<std::tuple<int, int, int>> seen;
    for (uint32_t t = 0; t < p.blocks; ++t) {
      SweepItem it;
      if (!sweep_item(p, nx, ny, t, it))
        continue;
      if (it.s >= p.steps || it.x < 0 || it.x >= nx || it.j < 0 || it.j >= (int)p.slabs ||
          it.b >= p.nb[it.s & 1] || it.r0 < 0 || it.r1 > ny || it.r1 < it.r0)
        return bad("out of range", nx, ny, p);
      std::set<std::pair<int, int>> waits;
      for (int k = 0; k < 9 && it.s > 0; ++k) {
        int j, x;
        if (!sweep_needs(it, nx, k, j, x))
          continue;
        if (count(it.s - 1, j, x) != p.nb[(it.s - 1) & 1])
          return bad("waits for a later block", nx, ny, p);
        waits.insert({ j, x });
      }
      for (int r = it.r0; r < it.r1; ++r) {
        const int y = (r + it.rot) % ny;
        for (int k = 0; k < 9 && it.s > 0; ++k) {
          const int x = (it.x + k / 3 - 1 + nx) % nx, yy = (y + k % 3 - 1 + ny) % ny;
          const int pos = (yy - (p.slabs > 1 ? it.s - 1 : 0) + ny) % ny;
          int slab = -1;
          for (int j = 0; j < (int)p.slabs; ++j) {
            int a, e;
            sweep_rows(p, ny, it.s - 1, j, a, e);
            slab = pos >= a && pos < e ? j : slab;
          }
          if (!waits.count({ slab, x }))
            return bad("a neighbour row is not waited for", nx, ny, p);
        }
        if (it.b == 0 && !seen.insert(std::make_tuple(it.s, it.x, y)).second)
          return bad("a row is taken twice", nx, ny, p);
      }
      // enough blocks for the item
      const bool cells = compact && ((it.s & 1) == 0) == h.local_first;
      if (!cells && (uint64_t)(it.r1 - it.r0) * h.units > (uint64_t)p.nb[it.s & 1] * kSweepWarps)
        return bad("too few blocks", nx, ny, p);
      if (cells) {
        uint64_t m = 0;
        for (int part = 0; part < 2; ++part) { // rows before and after the wrap
          int a = part ? 0 : it.r0 + it.rot;
          int e = part ? it.r1 + it.rot - ny : it.r1 + it.rot;
          e = !part && e > ny ? ny : e;
          if (e <= a)
            continue;
          const uint32_t c0 = rows[(size_t)it.x * ny + a], c1 = rows[(size_t)it.x * ny + e];
          m += h.pair ? (c1 - (c0 & ~1u) + 1) / 2 : c1 - c0;
        }
        if (m > (uint64_t)p.nb[it.s & 1] * kSweepThreads)
          return bad("too few blocks", nx, ny, p);
      }
      // the split of a unit number into row and unit
      for (uint32_t u = it.b * kSweepWarps; u < (it.b + 1) * kSweepWarps; ++u) {
        const uint32_t q = p.units == 1 ? u : (uint32_t)(((uint64_t)u * p.umagic) >> 32);
        if (q != u / p.units)
          return bad("unit split", nx, ny, p);
      }
      ++count(it.s, it.j, it.x);
    }
    if ((int)seen.size() != p.steps * nx * ny)
      return bad("rows missing", nx, ny, p);
  }
  std::printf("ok %d\n", plans);
  return 0;
}
