"""Performance cases of the D3Q19 TRT step: what a user of this framework has
it do, through its public entry points (lbmb200.Solver and lbmb200.DropIn).

A case is a dict of plain values:
  path      "solver"  Solver.run(steps), then the result read to the host
            "dropin"  kd->Kernel of a registered kernel: host arrays in, host
                      arrays out, as LBM-Bench's driver calls it
            "adjoint" Solver.adjoint_gradient: forward and reverse sweep
  geometry  LBM-Bench's box / channel / pipe / blocks / fluid, or the porous
            channel of the benchmark (spheres of radius rmin..rmax until the
            fraction `solid` is solid)
  nx ny nz, steps, and per path: pattern (push / pull / aa), precision
  (fp64 / fp32 / fp16 storage), compact (fluid-only layout or the default
  dense one), force (Luo body force or not), read ("state": all populations,
  into a page-locked buffer the caller keeps; "moments": density and momentum)
"""
import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(_ROOT, "lbm-bench_b200"))
import lbmb200  # noqa: E402

# Relaxation rate, magic parameter, body force and initial perturbation of the
# repository's benchmark and of its 64^3 channel.
OMEGA, LAMBDA, XFORCE, AMPLITUDE = 1.25, 3.0 / 16.0, 1e-6, 1e-4
ALPHA = 0.1  # Brinkman scale of the adjoint cases
FLOPS_PER_UPDATE = 190  # additions and multiplications of one cell's collision
BYTES = {"fp64": 8, "fp32": 4, "fp16": 2}


def _case(name, path, geometry, dims, steps, pattern="aa", precision="fp64", compact=True,
          force=True, read="state", solid=0.2, rmin=4.0, rmax=8.0):
    nx, ny, nz = dims
    c = {"path": path, "geometry": geometry, "nx": nx, "ny": ny, "nz": nz, "steps": steps,
         "pattern": pattern, "precision": precision, "compact": compact, "force": force,
         "read": read, "solid": solid, "rmin": rmin, "rmax": rmax}
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # The reference driver's default run (20^3 box, 10 iterations, push):
        # the smallest call, where launches and transfers are everything.
        _case("dropin-box20-push", "dropin", "box", (20, 20, 20), 10, "push"),
        # A short exchange with a control loop on a small ragged pipe.
        _case("pipe-ragged-push-fp64", "solver", "pipe", (67, 45, 51), 50, "push",
              compact=False),
        # The 64^3 channel of the accuracy configuration, 1000 steps, default
        # layout: the lattice sits in the L2 cache.
        _case("channel64-aa-fp64", "solver", "channel", (64, 64, 64), 1000, compact=False),
        # Flow around obstacles watched through its density and velocity
        # fields, as the reference's statistics do every 100 iterations.
        _case("porous128-pull-moments", "solver", "porous", (128, 128, 128), 100, "pull",
              read="moments"),
        # Fully periodic box (periodic z wraps inside a row), FP32 storage.
        _case("periodic-push-fp32", "solver", "fluid", (128, 120, 100), 201, "push", "fp32",
              compact=False, force=False),
        # The benchmark's headline: 256^3 porous channel, FP64 AA, compact.
        _case("porous256-aa-fp64", "solver", "porous", (256, 256, 256), 500),
        # The same domain on the default (dense) layout, two lattices.
        _case("porous256-pull-fp64-dense", "solver", "porous", (256, 256, 256), 200, "pull",
              compact=False),
        # Reduced storage on the headline domain.
        _case("porous256-aa-fp32", "solver", "porous", (256, 256, 256), 500, "aa", "fp32"),
        _case("porous256-aa-fp16", "solver", "porous", (256, 256, 256), 500, "aa", "fp16"),
        # Odd extents in every direction and larger obstacles, FP16 pull.
        _case("porous-ragged-pull-fp16", "solver", "porous", (231, 177, 205), 301, "pull",
              "fp16", solid=0.3, rmin=6.0, rmax=12.0),
        # The benchmark's end-to-end call: upload, steps, download.
        _case("dropin-porous160-aa", "dropin", "porous", (160, 160, 160), 100, "aa"),
        # Forward and reverse sweep of the Brinkman channel.
        _case("adjoint96-fp64", "adjoint", "channel", (96, 96, 96), 100, compact=False),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choice(["solver"] * 6 + ["dropin", "adjoint"])
    cells_most = {"solver": 256 ** 3, "dropin": 160 ** 3, "adjoint": 96 ** 3}[path]
    while True:
        dims = tuple(_log_int(rng, 16, 400) for _ in range(3))
        cells = dims[0] * dims[1] * dims[2]
        if cells <= cells_most:
            break
    if path == "adjoint":
        return _case(None, path, "channel", dims, _log_int(rng, 10, 100),
                     precision=rng.choice(["fp64", "fp32"]), compact=False)
    geometry = rng.choice(["porous", "porous", "porous", "channel", "pipe", "box", "blocks",
                           "fluid"])
    solid, rmin, rmax = rng.choice([(0.2, 4.0, 8.0), (0.3, 6.0, 12.0), (0.15, 2.0, 5.0)])
    # walls alone can be a larger share of a thin channel
    walls = 1.0 - (dims[1] - 2) * (dims[2] - 2) / (dims[1] * dims[2])
    solid = round(max(solid, walls + 0.02), 3)
    if path == "dropin":
        # whole pairs of steps: the result is in the first host array
        return _case(None, path, geometry, dims, 2 * _log_int(rng, 5, 50),
                     rng.choice(["aa", "push"]), solid=solid, rmin=rmin, rmax=rmax)
    most = max(2, min(1000, 256 ** 3 * 500 // cells))
    return _case(None, path, geometry, dims, _log_int(rng, 2, most),
                 rng.choice(["aa", "pull", "push"]), rng.choice(["fp64", "fp32", "fp16"]),
                 rng.choice([True, False]), rng.choice([True, True, False]),
                 rng.choice(["state", "state", "moments"]), solid, rmin, rmax)


# ---------------------------------------------------------------------------
# inputs, made from the seed
# ---------------------------------------------------------------------------

def _fluid(case, seed):
    """bool[nx, ny, nz]: the fluid cells of the case's geometry (the rules of
    src/lbm.c:52-187), and the periodic axes."""
    nx, ny, nz = n = (case["nx"], case["ny"], case["nz"])
    kind = case["geometry"]
    periodic = {"box": (0, 0, 0), "fluid": (1, 1, 1)}.get(kind, (1, 0, 0))
    f = np.ones(n, dtype=bool)
    for a in range(3):
        if not periodic[a]:
            face = [slice(None)] * 3
            for i in (0, n[a] - 1):
                face[a] = i
                f[tuple(face)] = False
    if kind == "pipe":
        y = np.arange(ny)[:, None] - (ny / 2.0 - 0.5)
        z = np.arange(nz)[None, :] - (nz / 2.0 - 0.5)
        r = min(ny, nz) / 2.0 - 1
        f &= (y * y + z * z < r * r)[None]
    elif kind == "blocks":
        b = 8
        x, y, z = ((np.arange(m) % (2 * b)) >= b for m in n)
        f &= ~(x[:, None, None] & y[None, :, None] & z[None, None, :])
    elif kind == "porous":
        rng = np.random.default_rng(seed)
        want, solid = case["solid"] * f.size, int(f.size - f.sum())
        while solid < want:
            c = rng.random(3) * n
            r = case["rmin"] + (case["rmax"] - case["rmin"]) * rng.random()
            lo = np.floor(c - r).astype(int)
            hi = np.ceil(c + r).astype(int) + 1
            xs = np.arange(lo[0], hi[0])
            ys = np.arange(max(lo[1], 0), min(hi[1], ny))
            zs = np.arange(max(lo[2], 0), min(hi[2], nz))
            ball = ((xs - c[0]) ** 2)[:, None, None] + ((ys - c[1]) ** 2)[None, :, None] + \
                ((zs - c[2]) ** 2)[None, None, :] <= r * r
            xw = xs % nx  # spheres wrap around the periodic x axis
            if len(xw) > nx:
                continue
            part = f[np.ix_(xw, ys, zs)]
            solid += int((part & ball).sum())
            f[np.ix_(xw, ys, zs)] = part & ~ball
    return f, periodic


_C = [(0, 1, 0), (0, -1, 0), (1, 0, 0), (-1, 0, 0), (1, 1, 0), (1, -1, 0), (-1, 1, 0),
      (-1, -1, 0), (0, 0, 1), (0, 1, 1), (1, 0, 1), (-1, 0, 1), (0, -1, 1), (0, 0, -1),
      (0, -1, -1), (0, 1, -1), (-1, 0, -1), (1, 0, -1), (0, 0, 0)]
_W = [(1 / 3, 1 / 18, 1 / 36)[sum(abs(k) for k in c)] for c in _C]
_INV = [_C.index((-a, -b, -c)) for a, b, c in _C]


def _initial(fluid, seed):
    """float64[19, nx, ny, nz] on the GPU: equilibrium at density 1 with a
    velocity uniform in +-AMPLITUDE per fluid cell, 0 on obstacles."""
    dev = torch.device("cuda")
    g = torch.Generator(dev).manual_seed(seed)
    m = torch.from_numpy(fluid).to(dev)
    u = (torch.rand((3,) + fluid.shape, generator=g, device=dev, dtype=torch.float64) * 2 - 1) \
        * AMPLITUDE
    usq = 1.0 - 1.5 * (u[0] * u[0] + u[1] * u[1] + u[2] * u[2])
    f = torch.empty((19,) + fluid.shape, device=dev, dtype=torch.float64)
    for d, c in enumerate(_C):
        cu = c[0] * u[0] + c[1] * u[1] + c[2] * u[2]
        f[d] = torch.where(m, _W[d] * (usq + 3.0 * cu + 4.5 * cu * cu), 0.0)
    return f


def _porosity(case, seed):
    rng = np.random.default_rng(seed)
    return rng.uniform(0.0, 1.0, (case["nx"], case["ny"], case["nz"])).astype(np.float32)


def _flags(fluid):
    return np.ascontiguousarray(np.transpose(fluid, (2, 1, 0)), dtype=np.int32)


class _Pdfs(np.ndarray):
    """A view of kd->Pdfs, which lives as long as its kernel: keeps it."""

    kernel = None


class _Run:
    """What the user's program keeps between calls."""

    def __init__(self, case):
        self.case, self.solver, self.kernel, self.out = case, None, None, None


class _Kernel(lbmb200.DropIn):
    """A drop-in kernel that is deinitialised with its last reference."""

    def __del__(self):
        self.close()


def prepare(case, seed):
    s = _Run(case)
    fluid, periodic = _fluid(case, seed)
    f0 = _initial(fluid, seed)
    if case["path"] == "dropin":
        k = s.kernel = _Kernel("cuda-%s-soa" % case["pattern"], _flags(fluid), periodic,
                               omega=OMEGA, xforce=XFORCE, iterations=case["steps"],
                               force_on=True, lam=LAMBDA)
        k.pdfs(0)[:, 1:-1, 1:-1, 1:-1] = f0.cpu().numpy()
        return s
    sol = s.solver = lbmb200.Solver(_flags(fluid), periodic, case["pattern"], case["precision"],
                                    compact=case["compact"])
    sol.set_params(OMEGA, LAMBDA, XFORCE, case["force"])
    if case["path"] == "adjoint":
        sol.set_porosity(_porosity(case, seed), ALPHA)
    s.out = torch.empty(f0.shape, dtype=torch.float64, pin_memory=True)
    s.out.copy_(f0)
    torch.cuda.synchronize()
    sol.set_state(s.out.numpy())
    return s


def run(s):
    case = s.case
    if case["path"] == "dropin":
        s.kernel.run(case["steps"])
        out = s.kernel.pdfs(0).view(_Pdfs)
        out.kernel = s.kernel
        return out
    if case["path"] == "adjoint":
        j, grad, _ = s.solver.adjoint_gradient(case["steps"], 0)
        return j, grad
    s.solver.run(case["steps"])
    if case["read"] == "moments":
        return s.solver.moments()
    s.solver.get_state(s.out.numpy())
    return s.out


def work(case):
    """What one pass cannot do without: the initial populations read once and
    the result written once, and the collisions of all its steps. (Keeping a
    large lattice on chip between steps is not possible in whole; a step that
    streams it through memory moves 2 x 19 populations per cell more each.)"""
    cells = case["nx"] * case["ny"] * case["nz"]
    fluid = float(_fluid(case, 1)[0].sum()) if cells < 100_000 else _expected_fluid(case)
    size = BYTES[case["precision"]]
    flops = FLOPS_PER_UPDATE * fluid * case["steps"]
    if case["path"] == "adjoint":
        # forward and reverse sweep; porosity read, gradient written
        return {"bytes": fluid * (19 * size + 4 + 8), "flops": 2.0 * flops}
    if case["path"] == "dropin":
        return {"bytes": 2.0 * 19 * 8 * fluid, "flops": flops}
    written = 4 * 8 if case["read"] == "moments" else 19 * 8
    return {"bytes": fluid * (19 * size + written), "flops": flops}


def _expected_fluid(case):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    if case["geometry"] == "porous":
        return (1.0 - case["solid"]) * nx * ny * nz
    return float(_fluid(case, 1)[0].sum())


# ---------------------------------------------------------------------------
# the same results in plain torch, 64 bits
# ---------------------------------------------------------------------------

def _collide(f, force, kappa=None):
    """TRT collision of f[19, ...]; `force` is added when populations stream."""
    odd = 1.0 / (0.5 + LAMBDA / (1.0 / OMEGA - 0.5))
    rho = f.sum(0)
    u = []
    for a in range(3):
        p = [d for d in range(19) if _C[d][a] > 0]
        q = [d for d in range(19) if _C[d][a] < 0]
        u.append(sum(f[d] for d in p) - sum(f[d] for d in q))
    base = rho - 1.5 * (u[0] * u[0] + u[1] * u[1] + u[2] * u[2])
    out = [None] * 19
    out[18] = f[18] - OMEGA * (f[18] - _W[18] * base)
    for a in range(18):
        b = _INV[a]
        if a > b:
            continue
        cu = sum(k * v for k, v in zip(_C[a], u) if k)
        even = OMEGA * (0.5 * (f[a] + f[b]) - _W[a] * (base + 4.5 * cu * cu))
        odd_part = odd * (0.5 * (f[a] - f[b]) - 3.0 * _W[a] * cu)
        if kappa is not None:
            odd_part = odd_part + 3.0 * _W[a] * kappa * cu
        out[a] = f[a] - even - odd_part
        out[b] = f[b] - even + odd_part
    return out, u


def _walls(fluid):
    """Per direction: where the population arriving along d comes from a wall
    (the geometry puts walls on every face of an axis that is not periodic)."""
    return [fluid & ~torch.roll(fluid, c, (0, 1, 2)) for c in _C]


def _stream(out, back, force):
    new = []
    for d, c in enumerate(_C):
        v = torch.roll(out[d], c, (0, 1, 2)) if any(c) else out[d]
        if any(c):
            v = torch.where(back[d], out[_INV[d]], v)
        new.append(v + force * 3.0 * _W[d] * c[0] if force and c[0] else v)
    return new


def exact(case, seed):
    fluid_np, _ = _fluid(case, seed)
    f = _initial(fluid_np, seed)
    fluid = torch.from_numpy(fluid_np).cuda()
    back = _walls(fluid)
    if case["path"] == "adjoint":
        return _exact_adjoint(case, seed, f, fluid, back)
    force = XFORCE if case["force"] else 0.0
    for _ in range(case["steps"]):
        out, _ = _collide(f, force)
        new = _stream(out, back, force)
        del out
        for d in range(19):
            f[d] = torch.where(fluid, new[d], 0.0)
        del new
    if case["path"] == "dropin":
        pad = torch.zeros((19,) + tuple(n + 2 for n in fluid.shape), dtype=torch.float64)
        pad[:, 1:-1, 1:-1, 1:-1] = f.cpu()
        return pad
    if case["read"] == "moments":
        q = [f.sum(0)]
        for a in range(3):
            q.append(sum(_C[d][a] * f[d] for d in range(19) if _C[d][a]))
        return [v.cpu() for v in q]
    return f.cpu()


def _exact_adjoint(case, seed, f0, fluid, back):
    """Gradient by automatic differentiation, steps recomputed in segments."""
    from torch.utils.checkpoint import checkpoint

    por = torch.from_numpy(_porosity(case, seed)).cuda().double().requires_grad_()

    def steps(f, phi, n):
        kappa = ALPHA * (1.0 - phi)
        for _ in range(n):
            out, _ = _collide(f, XFORCE, kappa)
            f = torch.stack([torch.where(fluid, v, 0.0) for v in _stream(out, back, XFORCE)])
        return f

    f, left = f0, case["steps"]
    while left:
        n = min(left, 10)
        f = checkpoint(steps, f, por, n, use_reentrant=False)
        left -= n
    ux = sum(_C[d][0] * f[d, -1] for d in range(19) if _C[d][0])
    j = ux.sum() / fluid[-1].sum()
    j.backward()
    grad = torch.where(fluid, por.grad, 0.0)
    return float(j.detach()), grad.cpu().numpy()
