"""Measured work of the homogenization engine, as programs call it.

Every case goes through ``fem_b200.femh.Engine``:

* ``solve`` -- the optimizer's step: six periodic load cases of one cell,
  C^H, and dL/drho of L = ||C^H - C_t||_F^2 (density on the device, gradient
  left there);
* ``batch`` -- the sample generator's call: many cells of uneven size from
  host memory, C^H and dL/drho of each;
* ``table`` -- the sensitivities of a solved cell: the 21 fields dC^H/drho and
  the gradient of a loss from the resident displacement fields.

A program keeps its engine (levels, tuned tile shapes, workspaces) between
cells of the same shape, so ``prepare`` makes the engine and lays it out on
another, easy cell (mild contrast: a few iterations).
"""
from __future__ import annotations

import math

import numpy as np
import torch

from fem_b200 import femh

_PRECISION = {"fp64": femh.FP64, "mixed": femh.MIXED, "mixed_pc": femh.MIXED_PC}
_SOLVER = {"jacobi": femh.JACOBI_PCG, "multigrid": femh.GMG_PCG}
_INTERP = {"simp": femh.INTERP_SIMP, "ramp3": femh.INTERP_RAMP3}

_BATCH_SIZES = (16, 24, 32, 48, 64)
_BATCH_PROBS = (0.30, 0.25, 0.25, 0.15, 0.05)


def _solve(name, nx, ny, nz, field, precision, solver="multigrid", interp="simp", p=0.5, sigma=4.0,
           tol=1e-10):
    case = {"kind": "solve", "nx": nx, "ny": ny, "nz": nz, "field": field, "precision": precision,
            "solver": solver, "interp": interp, "p": p, "sigma": sigma, "tol": tol}
    return {"name": name, **case} if name else case


def listed():
    return [
        # the smallest cells of the sample generator: a solve is a few dozen
        # iterations of very small launches, so launch latency is all there is
        _solve("cell16_binary", 16, 16, 16, "binary", "mixed_pc"),
        # the reference's plain method at the parity size: one Jacobi-PCG per
        # load case, everything FP64 (a digit more than the default tolerance: the
        # point-wise gradient converges late without a multigrid)
        _solve("cell32_plain_jacobi", 32, 32, 32, "binary", "fp64", solver="jacobi", tol=1e-11),
        # an ordinary cell with the engine's default options (FP64 multigrid)
        _solve("cell48_binary_fp64", 48, 48, 48, "binary", "fp64"),
        # the topology optimizer's cell: smooth densities, the adjoint each
        # step, fast_fem's material law
        _solve("cell64_smooth_ramp", 64, 64, 64, "smooth", "mixed_pc", interp="ramp3"),
        # the same work with FP32 inner solves in FP64 defect correction
        _solve("cell64_defect", 64, 64, 64, "smooth", "mixed", interp="ramp3"),
        # a brick whose extents halve to odd numbers (5 x 7 x 3 at the coarsest level)
        _solve("brick40x56x24", 40, 56, 24, "smooth", "mixed_pc", sigma=3.0, tol=1e-11),
        # extents that do not halve at all: only the Jacobi solver takes them
        _solve("odd33x45x37_jacobi", 33, 45, 37, "smooth", "fp64", solver="jacobi", interp="ramp3", sigma=3.0,
               tol=1e-11),
        # the benchmark cell in both precisions that a program picks for it (as
        # above, a digit more for the gradient where SIMP leaves soft voxels)
        _solve("cell128_smooth", 128, 128, 128, "smooth", "mixed_pc", tol=1e-11),
        _solve("cell128_smooth_fp64", 128, 128, 128, "smooth", "fp64", tol=1e-11),
        # the largest: a fine optimizer cell beyond the z extents with kernels of their own
        _solve("cell192_smooth_ramp", 192, 192, 192, "smooth", "mixed_pc", interp="ramp3", sigma=6.0),
        # the sample generator's batch of uneven cells
        {"name": "batch64_uneven", "kind": "batch", "cells": 64, "precision": "mixed_pc", "sizes": 7},
        # sensitivities of a (tightly) solved cell: one pass over its displacement fields
        {"name": "table96", "kind": "table", "nx": 96, "ny": 96, "nz": 96, "field": "smooth",
         "precision": "mixed_pc", "solver": "multigrid", "interp": "ramp3", "p": 0.5, "sigma": 4.0, "tol": 1e-11},
    ]


def _coarse_nodes(dims):
    """Nodes of the coarsest multigrid level of a cell."""
    x, y, z = dims
    while x * y * z > 64 and x % 2 == y % 2 == z % 2 == 0 and min(x, y, z) >= 4:
        x, y, z = x // 2, y // 2, z // 2
    return x * y * z


def _extent(rng, lo, hi, step):
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(lo, min(hi, int(round(v / step)) * step))


def draw(rng):
    kind = rng.choice(["cube", "cube", "cube", "brick", "brick", "odd", "batch", "table"])
    field = rng.choice(["smooth", "smooth", "binary", "median"])
    precision = rng.choice(["mixed_pc", "mixed_pc", "fp64"])
    interp = rng.choice(["simp", "simp", "ramp3"])   # SIMP: stiffness contrast 1e6; ramp3: 3e3
    if field == "median":   # thresholded designs come from the optimizer, with its law and clamp
        interp = "ramp3"
    tol = 1e-11 if (field, interp) == ("smooth", "simp") else 1e-10
    sigma = rng.choice([2.0, 3.0, 4.0, 6.0])
    p = round(rng.uniform(0.4, 0.6), 3)
    if kind == "batch":
        return {"kind": "batch", "cells": _extent(rng, 8, 96, 1), "precision": precision,
                "sizes": rng.randrange(1, 1 << 20)}
    if kind == "odd":
        dims = [_extent(rng, 9, 45, 2) | 1 for _ in range(3)]
        return _solve(None, *dims, rng.choice(["smooth", "binary"]), "fp64", "jacobi", interp, p, sigma, 1e-11)
    if kind == "brick":
        while True:
            dims = [_extent(rng, 12, 96, 4) for _ in range(3)]
            if _coarse_nodes(dims) <= 216:
                break
        if rng.random() < 0.25:
            return _solve(None, *dims, "smooth", "mixed", "multigrid", "ramp3", p, sigma)
        return _solve(None, *dims, field, precision, "multigrid", interp, p, sigma, tol)
    while True:
        n = _extent(rng, 12, 160, 4)
        if _coarse_nodes((n, n, n)) <= 216:
            break
    if n > 64 and field == "median":
        field = "smooth"
    case = _solve(None, n, n, n, field, precision, "multigrid", interp, p, sigma, tol)
    if kind == "table":
        case.update(kind="table", interp="ramp3", tol=1e-11)
    return case


def _density(case, seed):
    """The cell's density on the device: what optimizers (smooth) and sample
    generators (binary, thresholded) meet."""
    shape = (case["nx"], case["ny"], case["nz"])
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    if case["field"] == "binary":
        r = torch.rand(shape, generator=g, device="cuda", dtype=torch.float64)
        return (r < case["p"]).double().contiguous()
    z = torch.randn(shape, generator=g, device="cuda", dtype=torch.float64)
    k = [torch.fft.fftfreq(n, device="cuda", dtype=torch.float64) * (2 * math.pi) for n in shape]
    k2 = k[0][:, None, None] ** 2 + k[1][None, :, None] ** 2 + k[2][None, None, :] ** 2
    f = torch.fft.ifftn(torch.fft.fftn(z) * torch.exp(-0.5 * case["sigma"] ** 2 * k2)).real
    f = (f - f.mean()) / f.std()
    if case["field"] == "median":
        return (f > f.median()).double().contiguous()
    return (1e-3 + (1.0 - 1e-3) * torch.sigmoid(4.0 * f)).contiguous()


def _target(seed):
    """C_t of the loss: an isotropic tensor softer than the solid."""
    r = np.random.Generator(np.random.PCG64(int(seed)))
    e, nu = r.uniform(0.05, 0.4), r.uniform(0.1, 0.35)
    lam, mu = e * nu / ((1 + nu) * (1 - 2 * nu)), e / (2 * (1 + nu))
    c = np.zeros((6, 6))
    c[:3, :3] = lam
    c[range(6), range(6)] += [2 * mu] * 3 + [mu] * 3
    return c


def _batch_shapes(case):
    r = np.random.Generator(np.random.PCG64(int(case["sizes"])))
    return [int(n) for n in r.choice(_BATCH_SIZES, size=case["cells"], p=_BATCH_PROBS)]


def _batch_cells(case, seed):
    r = np.random.Generator(np.random.PCG64(int(seed)))
    return [(r.random((n, n, n)) < r.uniform(0.35, 0.6)).astype(np.float64) for n in _batch_shapes(case)]


def _weights(case, seed):
    """dL/dC of each cell of a batch."""
    r = np.random.Generator(np.random.PCG64(int(seed) + 1))
    w = r.standard_normal((case["cells"], 6, 6))
    return w + w.transpose(0, 2, 1)


def _options(case):
    opt = {"precision": _PRECISION[case["precision"]]}
    if case["kind"] != "batch":
        opt["tol"] = case["tol"]
        opt["solver"] = _SOLVER[case["solver"]]
        opt["interp"] = _INTERP[case["interp"]]
        opt["rho_min"] = 1e-3 if case["interp"] == "ramp3" else 0.0   # fast_fem's clamp
    return opt


def prepare(case, seed):
    engine = femh.Engine(**_options(case))
    if case["kind"] == "batch":
        rhos = _batch_cells(case, seed)
        engine.batch([0.5 + 0.5 * r for r in rhos], dLdC=_weights(case, seed), allow_unconverged=True)
        return {"kind": "batch", "engine": engine, "rhos": rhos, "dLdC": _weights(case, seed)}
    stream = torch.cuda.Stream()   # the program's own stream: engine and tensors share it
    engine.set_stream(stream.cuda_stream)
    rho = _density(case, seed)
    state = {"kind": case["kind"], "engine": engine, "stream": stream, "rho": rho, "target": _target(seed),
             "grad": torch.empty_like(rho)}
    torch.cuda.synchronize()
    if case["kind"] == "table":
        C, _ = engine.homogenize(rho, allow_unconverged=True)
        state["dLdC"] = 2.0 * (C - state["target"])
        state["table"] = torch.empty((21,) + tuple(rho.shape), dtype=torch.float64, device="cuda")
    else:
        engine.homogenize(0.5 + 0.5 * rho.flip(0).contiguous(), allow_unconverged=True)
        engine.grad(state["target"], out=state["grad"])
    torch.cuda.synchronize()
    return state


def run(state):
    engine = state["engine"]
    if state["kind"] == "batch":
        C, _, grads = engine.batch(state["rhos"], dLdC=state["dLdC"], allow_unconverged=True)
        return {"C": C, "grad": np.concatenate([g.ravel() for g in grads])}
    if state["kind"] == "table":
        return {"table": engine.dCdrho(out=state["table"]), "grad": engine.grad(state["dLdC"], out=state["grad"])}
    C, _ = engine.homogenize(state["rho"], allow_unconverged=True)
    return {"C": C, "grad": engine.grad(2.0 * (C - state["target"]), out=state["grad"])}


def _voxels(case):
    if case["kind"] == "batch":
        return sum(n ** 3 for n in _batch_shapes(case))
    return case["nx"] * case["ny"] * case["nz"]


def work(case):
    """A solve cannot do without reading the densities, and for each iteration
    of a preconditioned Krylov method reading and writing the six load cases'
    iterate, residual and direction once and applying the operator once; the
    count below asks for 12 such iterations (far fewer than any cell here
    takes).  A table reads the fields once and writes its 21 + 1 values."""
    n = _voxels(case)
    if case["kind"] == "table":
        return {"bytes": 8.0 * n * (2 * (18 + 1) + 22), "flops": n * (18 * 24 + 6 * 100 + 21 * 2 * 21)}
    iterations = 12
    return {"bytes": n * (8.0 * 2 + iterations * 18 * 8.0 * 6), "flops": float(n) * iterations * 6 * 500}


# ------------------------------------------------------------------ exact --
def _element():
    """24x24 stiffness of a unit voxel (E = 1, nu = 0.3), nodes 4x + 2y + z, and
    the six unit macro strains' nodal displacements (Voigt, engineering shear)."""
    nu, g = 0.3, 1.0 / math.sqrt(3.0)
    lam, mu = nu / ((1 + nu) * (1 - 2 * nu)), 0.5 / (1 + nu)
    D = np.zeros((6, 6))
    D[:3, :3] = lam
    D[range(6), range(6)] += [2 * mu] * 3 + [mu] * 3
    corner = np.array([[a >> 2 & 1, a >> 1 & 1, a & 1] for a in range(8)], dtype=float)
    K = np.zeros((24, 24))
    for q in 2 * corner - 1:
        N = np.ones((8, 3))
        for a in range(8):
            s = 2 * corner[a] - 1
            f = 1 + s * q * g
            for d in range(3):
                N[a, d] = s[d] / 4 * np.prod(np.delete(f, d))
        B = np.zeros((6, 24))
        for a in range(8):
            x, y, z = N[a]
            B[0, 3 * a], B[1, 3 * a + 1], B[2, 3 * a + 2] = x, y, z
            B[3, 3 * a + 1], B[3, 3 * a + 2] = z, y
            B[4, 3 * a], B[4, 3 * a + 2] = z, x
            B[5, 3 * a], B[5, 3 * a + 1] = y, x
        K += B.T @ D @ B / 8
    U = np.zeros((6, 24))
    for i, (r, c) in enumerate([(0, 0), (1, 1), (2, 2), (1, 2), (0, 2), (0, 1)]):
        eps = np.zeros((3, 3))
        eps[r, c] += 0.5
        eps[c, r] += 0.5
        U[i] = (corner @ eps).reshape(24)
    return K, U


def _gather(v):
    """[6, x, y, z, 3] nodal values -> [6, x, y, z, 24] element values."""
    parts = []
    for a in range(8):
        parts.append(torch.roll(v, shifts=(-(a >> 2 & 1), -(a >> 1 & 1), -(a & 1)), dims=(1, 2, 3)))
    return torch.cat(parts, dim=-1)


def _scatter(f):
    out = f[..., 0:3].clone()
    for a in range(1, 8):
        out += torch.roll(f[..., 3 * a:3 * a + 3], shifts=(a >> 2 & 1, a >> 1 & 1, a & 1), dims=(1, 2, 3))
    return out


def _modulus(rho, interp):
    if interp == "ramp3":
        r = rho.clamp(1e-3, 1.0)
        return r / (3 - 2 * r), 3 / (3 - 2 * r) ** 2
    r = rho.clamp(0.0, 1.0)
    return 1e-6 + r ** 3 * (1 - 1e-6), 3 * r ** 2 * (1 - 1e-6)


def _solve_exact(rho, interp):
    """Element displacements of the six load cases by Jacobi-PCG far below the
    engine's tolerance (unit cell scaled to voxel edge 1: C^H and the pair
    energies do not depend on the edge)."""
    K, U = (torch.from_numpy(m).to(rho.device) for m in _element())
    E, dE = _modulus(rho, interp)
    e = E[None, ..., None]
    u0 = U[:, None, None, None, :]
    b = -_scatter(e * (u0 @ K))
    dinv = 1.0 / (_scatter(e.expand(1, *E.shape, 24)) * K[0, 0])
    x, r = torch.zeros_like(b), b.clone()
    p = dinv * r
    rz, bb = (r * p).sum((1, 2, 3, 4)), (b * b).sum((1, 2, 3, 4)).clamp_min(1e-300)
    for it in range(40000):
        q = _scatter(e * (_gather(p) @ K))
        a = rz / (p * q).sum((1, 2, 3, 4)).clamp_min(1e-300)
        x += a[:, None, None, None, None] * p
        r -= a[:, None, None, None, None] * q
        if it % 20 == 0 and float(((r * r).sum((1, 2, 3, 4)) / bb).max()) < 1e-26:
            break
        z = dinv * r
        new = (r * z).sum((1, 2, 3, 4))
        p = z + (new / rz.clamp_min(1e-300))[:, None, None, None, None] * p
        rz = new
    u = _gather(x) + u0
    return u, u @ K, E, dE


def _exact_cell(rho, interp):
    u, ku, E, dE = _solve_exact(rho, interp)
    s = torch.einsum("ixyzk,jxyzk->ijxyz", u, ku)
    n = rho.numel()
    return (s * E).sum((2, 3, 4)) / n, s * dE / n


def exact(case, seed):
    n = _voxels(case)
    if case["kind"] == "batch" or n > 64 ** 3:   # 64-bit Jacobi solves of these take minutes
        return None
    rho = _density(case, seed)
    C, dC = _exact_cell(rho, case["interp"])
    dLdC = 2.0 * (C - torch.from_numpy(_target(seed)).to(C.device))
    grad = (dLdC[:, :, None, None, None] * dC).sum((0, 1))
    if case["kind"] == "table":
        return {"table": torch.stack([dC[i, j] for i in range(6) for j in range(i + 1)]), "grad": grad}
    return {"C": C.cpu().numpy(), "grad": grad}
