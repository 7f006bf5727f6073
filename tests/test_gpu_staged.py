"""The bulk-copy staged stencil kernels on z extents between their compile-time
row pitches (row-by-row copies, idle lanes), on the pitches themselves, and on
cells whose rows wrap around y more than once in a tile: the operator against
the scalar kernel (variant 1), and whole solves (sweeps, residuals, fused dot
products) against the Jacobi solver."""
import numpy as np
import pytest

from fem_b200 import femh

pytestmark = pytest.mark.gpu

SHAPES = [(5, 7, 36), (3, 2, 40), (4, 3, 48), (6, 16, 52), (4, 33, 60), (2, 9, 68), (3, 14, 96), (4, 8, 100),
          (3, 5, 128), (2, 4, 132), (4, 7, 160), (3, 3, 192), (2, 5, 196), (2, 2, 252), (3, 4, 256)]


def _field(shape):
    rng = np.random.default_rng(sum(shape))
    return rng.uniform(0.1, 1.0, shape), rng.standard_normal((6, *shape, 3))


@pytest.mark.parametrize("shape", SHAPES)
def test_fp64_operator(shape):
    rho, u = _field(shape)
    ref = femh.Engine(stencil_variant=1, solver=femh.JACOBI_PCG).apply_operator(rho, u, h=0.1)
    y = femh.Engine(stencil_variant=6, solver=femh.JACOBI_PCG).apply_operator(rho, u, h=0.1)
    assert np.abs(y - ref).max() <= 1e-14 * np.abs(ref).max()   # sums of 24 x 8 terms in another order


@pytest.mark.parametrize("variant", [5, 7])
@pytest.mark.parametrize("shape", SHAPES)
def test_fp32_operator(shape, variant):
    rho, u = _field(shape)
    ref = femh.Engine(stencil_variant=1, solver=femh.JACOBI_PCG).apply_operator(rho, u, h=0.1)
    y = femh.Engine(stencil_variant=variant, solver=femh.JACOBI_PCG, precision=femh.MIXED).apply_operator(rho, u, h=0.1)
    assert np.abs(y - ref).max() <= 4e-6 * np.abs(ref).max()    # FP32: 24 x 8 terms of 6e-8 each, signs mixed


@pytest.mark.parametrize("shape", [(8, 12, 40), (12, 8, 72), (4, 16, 144), (8, 8, 96), (4, 4, 192)])
@pytest.mark.parametrize("kw", [dict(stencil_variant=5, precision=femh.MIXED_PC),
                                dict(stencil_variant=7, precision=femh.MIXED_PC),
                                dict(stencil_variant=7, precision=femh.MIXED),
                                dict(stencil_variant=7, precision=femh.MIXED_PC, block_jacobi=0),
                                dict(stencil_variant=6), dict(stencil_variant=6, block_cg=0),
                                dict(stencil_variant=6, block_jacobi=0),
                                dict(stencil_variant=6, precision=femh.MIXED_PC)])
def test_solves(shape, kw):
    rho, _ = _field(shape)
    Cj, _ = femh.Engine(solver=femh.JACOBI_PCG, stencil_variant=1).homogenize(rho, h=0.1)
    C, _ = femh.Engine(**kw).homogenize(rho, h=0.1)
    assert np.abs(C - Cj).max() <= 1e-8 * np.abs(Cj).max()
