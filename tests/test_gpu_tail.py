"""The fused coarse end of the V-cycle and the block PCG's products on the
shapes where they can go wrong: levels at the shared-memory limit, extents of
two nodes, several fused levels, other sweep counts, odd plane strides and odd
cell offsets.  C^H against the Jacobi solver at the engine's 1e-8 bar; a wrong
V-cycle or product shows in the iteration count."""
import numpy as np
import pytest

from fem_b200 import femh, fields

pytestmark = pytest.mark.gpu


def _cell(shape):
    n = max(shape)
    return np.ascontiguousarray(fields.smooth_cell(n, sigma=1.5, seed=5)[: shape[0], : shape[1], : shape[2]])


SHAPES = [(24, 24, 24),    # 12^3 below level 0: the FP32 limit (FP64 starts at 6^3)
          (20, 20, 20),    # 10^3: the FP64 limit, odd 5^3 below
          (32, 32, 32), (4, 8, 32), (16, 4, 4), (48, 8, 24), (56, 40, 24)]
CONFIGS = [dict(precision=femh.MIXED_PC), dict(precision=femh.FP64), dict(precision=femh.MIXED),
           dict(precision=femh.MIXED_PC, block_jacobi=0), dict(precision=femh.FP64, pre_smooth=1, post_smooth=1),
           dict(precision=femh.MIXED_PC, pre_smooth=4, post_smooth=4),
           dict(precision=femh.MIXED_PC, pre_smooth=9, post_smooth=9)]   # beyond the fused kernel's table


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("kw", CONFIGS)
def test_solves(shape, kw):
    rho = _cell(shape)
    Cj, _ = femh.Engine(solver=femh.JACOBI_PCG).homogenize(rho)
    C, info = femh.Engine(**kw).homogenize(rho)
    assert np.abs(C - Cj).max() <= 1e-8 * np.abs(Cj).max()
    if kw["precision"] != femh.MIXED:
        assert max(info["iterations"]) <= 100


def test_fused_and_level_kernels_agree():
    """200 cells are past the fused kernel's limit: the level kernels run the
    same V-cycle, up to rounding."""
    rhos = [fields.binary_cell(16, 0.55, seed=s) for s in range(4)] * 50
    C, infos, _ = femh.Engine(precision=femh.MIXED_PC).batch(rhos)
    e = femh.Engine(precision=femh.MIXED_PC)
    for s in range(4):
        Cs, i = e.homogenize(rhos[s])
        assert np.abs(C[s] - Cs).max() <= 1e-10 * np.abs(Cs).max()
        assert abs(max(infos[s]["iterations"]) - max(i["iterations"])) <= 1


@pytest.mark.parametrize("prec", [femh.FP64, femh.MIXED_PC])
def test_odd_strides_and_offsets(prec):
    """Cells small enough to be their own coarsest level: 45, 27 and 64 nodes,
    alone (an odd plane stride) and one after another (odd offsets)."""
    rhos = [np.random.default_rng(n).uniform(0.2, 1.0, s) for n, s in enumerate([(5, 3, 3), (3, 3, 3), (4, 4, 4)])]
    ref = [femh.Engine(solver=femh.JACOBI_PCG).homogenize(r)[0] for r in rhos]
    C, infos, _ = femh.Engine(precision=prec).batch(rhos)
    for r, Cr, Cb, i in zip(rhos, ref, C, infos):
        Cs, info = femh.Engine(precision=prec).homogenize(r)
        for X, n in ((Cb, i), (Cs, info)):
            assert np.abs(X - Cr).max() <= 1e-8 * np.abs(Cr).max()
            assert max(n["iterations"]) <= 8   # the dense solve is exact up to the storage type
