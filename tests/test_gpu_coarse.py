"""The dense coarse solve of the multigrid preconditioner at the sizes where
its block inversion can go wrong: one partial block, exact multiples of the
32-wide blocks, odd and even numbers of block steps, and large ragged levels.

The solution does not depend on the preconditioner, so C^H is compared with
the Jacobi solver's at the engine's 1e-8 bar; a wrong or unsymmetric inverse
shows in the iteration count (these cells take 15-30 iterations; a V-cycle
without its coarse correction takes hundreds)."""
import numpy as np
import pytest

from fem_b200 import femh, fields

pytestmark = pytest.mark.gpu

# extents -> nodes of the coarsest level (unknowns = 3 x nodes)
SHAPES = [
    (4, 4, 4),      # 64 nodes at once: the cell is its own coarsest level (6 block steps)
    (6, 4, 2),      # 48 nodes, 144 unknowns: 4.5 blocks
    (12, 12, 12),   # 3^3 = 27: 81 unknowns
    (20, 20, 20),   # 5^3 = 125: 375
    (10, 14, 18),   # 5 x 7 x 9 = 315: 945
    (28, 28, 28),   # 7^3 = 343: 1029
]


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("prec", [femh.FP64, femh.MIXED_PC])
def test_ragged_coarse_levels(shape, prec):
    n = max(shape)
    rho = np.ascontiguousarray(fields.smooth_cell(n, sigma=1.5, seed=11)[: shape[0], : shape[1], : shape[2]])
    Cj, _ = femh.Engine(solver=femh.JACOBI_PCG).homogenize(rho)
    C, info = femh.Engine(precision=prec).homogenize(rho)
    assert np.abs(C - Cj).max() <= 1e-8 * np.abs(Cj).max()
    assert max(info["iterations"]) <= 60


def test_too_large_coarse_level_is_refused():
    # 22 x 11 x 11 = 2662 nodes
    with pytest.raises(femh.FemhError):
        femh.Engine().homogenize(np.full((44, 22, 22), 0.5))


def test_batch_of_different_coarse_sizes():
    """Cells with odd and even numbers of block steps in one launch."""
    rhos = [fields.binary_cell(n, 0.55, seed=30 + n) for n in (4, 8, 12, 20, 24, 20)]
    C, infos, _ = femh.Engine(precision=femh.MIXED_PC).batch(rhos)
    for r, c, i in zip(rhos, C, infos):
        Cj, _ = femh.Engine(solver=femh.JACOBI_PCG).homogenize(r)
        assert np.abs(c - Cj).max() <= 1e-8 * np.abs(Cj).max()
        assert max(i["iterations"]) <= 80
