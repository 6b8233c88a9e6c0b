// Discrete adjoint of the Brinkman TRT step (no counterpart in the
// reference; the forward step is the reference's, src/kernel_pull_soa.c:
// 118-198, plus the Brinkman resistance of collide() in lbm_device.cuh).
//
// Forward step in the receiver view: out(x) = C(f(x); u(x), phi(x)) is the
// collision of cell x, and population d of it goes to r(x, d) =
// (d, x + c_d), or to (inv d, x) if x + c_d is a wall; the body force is a
// constant. For an objective J of the final state, with
// lambda_d(x) = dJ / df_d(x) kept in the natural layout (plane d, cell x):
//   mu_d(x)       = lambda^{t+1}[r(x, d)]
//   lambda^t_k(x) = sum_d mu_d(x) d out_d / d f_k (x)
//   dJ/dphi(x)   += sum_d mu_d(x) d out_d / d phi (x)
// The collision Jacobian depends only on the momentum u(x, t) of the
// populations the cell collided at step t, which the forward kernels save
// during the segment recomputation. With oE = omega, oO = omegaOdd,
// kappa = alpha (1 - phi), D = rho - 1.5 |u|^2, pairs (a, b = inv a) with
// weight w and ui = c_a . u:
//   out_a = f_a - oE (f_a+f_b)/2 - oO (f_a-f_b)/2 + oE w (4.5 ui^2 + D)
//           + 3 w (oO - kappa) ui            (out_b: signs of the odd terms flip)
//   out_C = f_C - oE (f_C - w0 D)
// so that
//   lambda_a = (1 - (oE+oO)/2) mu_a + ((oO-oE)/2) mu_b + sD + g . c_a
//   lambda_C = (1 - oE) mu_C + sD
//   sD = oE (w0 mu_C + sum_pairs w (mu_a + mu_b))
//   g  = sum_pairs [oE 9 w ui (mu_a + mu_b) + 3 w (oO - kappa)(mu_a - mu_b)] c_a - 3 u sD
//   dJ/dphi += sum_pairs 3 w alpha ui (mu_a - mu_b).
#pragma once

#include "lbm_device.cuh"
#include "lbm_sweep.cuh"

namespace lbm {

template <typename V> struct AdjArgs {
  Grid g;
  const V *lam_next; // lambda^{t+1}, natural layout
  V *lam;            // lambda^t
  const V *u;        // momentum at step t, 3 planes (x, y, z)
  const uint32_t *mask;
  const float *porosity;
  double *grad;      // dJ/dphi accumulator per cell
  V oE, oO, w0, w1, w2, alpha;
};

// a * b + c. In FP64 rounded once by its own word: the FP64 kernels are compiled
// without contraction, so that steps and sweeps agree bit for bit, which had made
// single reverse steps 10-15% slower. 60 steps with their recomputation, ms,
// contracted / not / with these: 60000 x 5 x 5 26.5 / 30.6 / 27.9, pipe in 200 x
// 100 x 33 1.92 / 2.11 / 2.00. (The sums of `pair` as well: 27.3 and 1.99, but
// sweeps spill 120 bytes for 80: 128^3 17.5 for 17.3.) FP32 leaves it to the
// compiler.
__device__ __forceinline__ double mul_add(double a, double b, double c) { return fma(a, b, c); }
__device__ __forceinline__ float mul_add(float a, float b, float c) { return a * b + c; }

// One cell's reverse step: mu and the momentum u of the step to lambda^t
// (store(k, value)) and this step's dJ/dphi (returned).
template <typename V, class STORE>
__device__ __forceinline__ V adjoint_cell(const AdjArgs<V> &a, const V (&mu)[Q], V ux, V uy, V uz,
    V kappa, STORE &&store)
{
  const V oE = a.oE, oO = a.oO;
  const V cdir = V(1) - V(0.5) * oE - V(0.5) * oO, ccross = V(0.5) * oO - V(0.5) * oE;

  // first the sums every output needs (sD, g, the porosity gradient), then
  // each output from mu directly, stored at once: no array of partial
  // results stays live next to mu
  V sD = oE * a.w0 * mu[dC];
  V gx = 0, gy = 0, gz = 0, gphi = 0;
  auto pair = [&](int pa, int pb, V w) {
    const V ui = V(cx(pa)) * ux + V(cy(pa)) * uy + V(cz(pa)) * uz;
    const V ms = mu[pa] + mu[pb], md = mu[pa] - mu[pb];
    sD += oE * w * ms;
    const V sp = oE * V(9) * w * ui * ms + V(3) * w * (oO - kappa) * md;
    gx += sp * V(cx(pa));
    gy += sp * V(cy(pa));
    gz += sp * V(cz(pa));
    gphi += V(3) * w * a.alpha * ui * md;
  };
  pair(dN, dS, a.w1);
  pair(dE, dW, a.w1);
  pair(dT, dB, a.w1);
  pair(dNW, dSE, a.w2);
  pair(dNE, dSW, a.w2);
  pair(dTW, dBE, a.w2);
  pair(dTE, dBW, a.w2);
  pair(dTS, dBN, a.w2);
  pair(dTN, dBS, a.w2);
  gx = mul_add(V(-3) * ux, sD, gx);
  gy = mul_add(V(-3) * uy, sD, gy);
  gz = mul_add(V(-3) * uz, sD, gz);
#pragma unroll
  for (int k = 0; k < Q; ++k) {
    const V part = (k == dC) ? (V(1) - oE) * mu[dC] : mul_add(cdir, mu[k], ccross * mu[inv(k)]);
    store(k, part + sD + gx * V(cx(k)) + gy * V(cy(k)) + gz * V(cz(k)));
  }
  return gphi;
}

// 6 CTAs of 128 per SM (80 registers): fastest in a sweep at 128^3 (B200)
#ifndef LBM_MINB_ADJ
#define LBM_MINB_ADJ 6
#endif
template <typename V>
__global__ void __launch_bounds__(128, LBM_MINB_ADJ) adjoint_step_kernel(AdjArgs<V> a)
{
  const Grid &g = a.g;
  const int z = blockIdx.x * blockDim.x + threadIdx.x;
  const int y = blockIdx.y * blockDim.y + threadIdx.y;
  const int x = blockIdx.z;
  if (z >= g.nz || y >= g.ny)
    return;
  const uint32_t cell = cell_index(g, x, y, z);
  const uint32_t mask = a.mask[cell];
  // The step writes lambda into a lattice it has not read. The solid cells
  // of 32-byte sectors that also hold fluid cells store their own lambda
  // (0, as the seed sets it; no step reads a wall's slots), so that such
  // sectors are written whole and the L2 does not fetch them from DRAM to
  // merge a partial write. Lane l holds z = l mod (32 / sizeof(V)) of its
  // sector: rows start on 32-byte boundaries and blockDim.x % 32 == 0.
  const unsigned fluid = __ballot_sync(__activemask(), !(mask & kSolidBit));
  if (mask & kSolidBit) {
    constexpr int kSectorLanes = 32 / (int)sizeof(V);
    const int lane = threadIdx.x & 31;
    if ((fluid >> (lane & ~(kSectorLanes - 1))) & ((1u << kSectorLanes) - 1u)) {
#pragma unroll
      for (int k = 0; k < Q; ++k)
        a.lam[k * g.plane + cell] = V(0);
    }
    return;
  }
  const Offs of = make_offs(g, x, y, z);
  const long long P = g.plane;

  V mu[Q];
#pragma unroll
  for (int d = 0; d < Q; ++d) {
    const bool bb = (mask >> d) & 1u;
    mu[d] = bb ? a.lam_next[inv(d) * P + cell] : a.lam_next[d * P + (uint32_t)(cell + of.at(d))];
  }
  const V ux = a.u[cell], uy = a.u[P + cell], uz = a.u[2 * P + cell];
  const V kappa = a.alpha * (V(1) - V(a.porosity[cell]));
  const V gphi = adjoint_cell(a, mu, ux, uy, uz, kappa,
      [&](int k, V v) { a.lam[k * P + cell] = v; });
  a.grad[cell] += (double)gphi;
}

// Sweeps of FP64 reverse steps (lbm_sweep.cuh), in place: a step streams the
// adjoint lattice through HBM, a pair of them in a sweep once (96^3, 100 steps:
// reverse sweep with its recomputation 9.8 -> 8.0 ms). A shifted step gathers
// lambda^{t+1} from the slots r(x, d) and leaves lambda_k(x) where the receiver
// that needs it next looks in its own slots: in (inv k, x - c_k), or behind a
// wall in (k, x). The local step then finds mu_d(x) in (inv d, x) for every d
// and restores the natural layout. A cell's slots are its own in both.
template <typename V> struct SweepAdjArgs : AdjArgs<V> {
  const V *src; // the lattice, twice (as in SweepArgs)
  V *dst;
  SweepPlan p;
};

// 80 registers (figures at plan_adjoint_sweep)
#ifndef LBM_MINB_SWEEP_ADJ
#define LBM_MINB_SWEEP_ADJ 6
#endif

template <typename V, bool FRONTS> struct SweepAdjoint {
  using Args = SweepAdjArgs<V>;
  static constexpr int kMinBlocks = LBM_MINB_SWEEP_ADJ;
  static constexpr bool kLocalFirst = false;

  __device__ static uint32_t el(const Args &a, int plane, uint32_t i)
  {
    return (uint32_t)plane * (uint32_t)a.g.plane + i;
  }

  template <bool SHIFTED, class WAIT>
  __device__ __forceinline__ static void step(const Args &a, const SweepItem &it, int tid,
      WAIT &&wait)
  {
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
    wait();
    if (mask & kSolidBit)
      return;
    const Offs of = make_offs(g, it.x, y, z);
    V mu[Q];
#pragma unroll
    for (int d = 0; d < Q; ++d) {
      const bool bb = (mask >> d) & 1u;
      mu[d] = a.src[!SHIFTED || bb ? el(a, inv(d), cell) : el(a, d, cell + of.at(d))];
    }
    // the sweep's first step is the latest one: earlier momenta lie before it
    const V *u = a.u - 3 * (long long)it.s * g.plane + cell;
    const V ux = u[0], uy = u[g.plane], uz = u[2 * g.plane];
    const V kappa = a.alpha * (V(1) - V(a.porosity[cell]));
    const uint32_t own = recompute(cell);
    const V gphi = adjoint_cell(a, mu, ux, uy, uz, kappa, [&](int k, V v) {
      const bool wall = (mask >> inv(k)) & 1u; // x - c_k
      sweep_store<FRONTS && !SHIFTED>(
          a.dst + (!SHIFTED || wall ? el(a, k, own) : el(a, inv(k), own + of.at(inv(k)))), v);
    });
    a.grad[cell] += (double)gphi;
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

// lambda^N = dJ/df^N for J = mean over the fluid cells of device plane
// x = xo of sum_k c_kx f_k: c_kx / count there, 0 elsewhere.
template <typename V>
__global__ void adjoint_seed_kernel(Grid g, int xo, double inv_count, V *lam,
    const uint32_t *__restrict__ mask)
{
  const int z = blockIdx.x * blockDim.x + threadIdx.x;
  const int y = blockIdx.y * blockDim.y + threadIdx.y;
  const int x = blockIdx.z;
  if (z >= g.nz || y >= g.ny)
    return;
  const uint32_t cell = cell_index(g, x, y, z);
  const bool on = x == xo && !(mask[cell] & kSolidBit);
#pragma unroll
  for (int k = 0; k < Q; ++k)
    lam[k * g.plane + cell] = on ? V(cx(k) * inv_count) : V(0);
}

} // namespace lbm
