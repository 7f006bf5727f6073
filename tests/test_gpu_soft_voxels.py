"""Voxels without stiffness, or almost: cells that are their own coarsest level,
so that the V-cycle is the dense inverse and a solve takes a step or two.  It
must leave out the unknowns that nothing holds (node 0 among them, where it lies
in the void) and keep the digits of the soft ones.

The multigrid's C^H at E_min against the Jacobi solver's at the same E_min, or,
where E_min = 0 leaves that solver no diagonal, against its C^H at 1e-9: void of
relative stiffness e adds at most O(e) to C^H.  The bars are the engine's 1e-8
of the largest entry."""
import numpy as np
import pytest

from fem_b200 import femh

pytestmark = pytest.mark.gpu


def _cell(name):
    if name == "cavity":            # node 0 in the solid
        r = np.ones((5, 7, 9))
        r[1:4, 2:5, 3:7] = 0
    elif name == "cavity 4^3":
        r = np.ones((4, 4, 4))
        r[1:3, 1:3, 1:3] = 0
    elif name == "slab":
        r = np.zeros((5, 7, 9))
        r[:2] = 1
    else:                           # a frame, node 0 in the void
        r = np.zeros((5, 5, 5))
        r[:, 1:3, 1:3] = r[1:3, :, 1:3] = r[1:3, 1:3, :] = 1
    return r


@pytest.mark.parametrize("kw", [dict(), dict(precision=femh.MIXED_PC), dict(block_cg=0)])
@pytest.mark.parametrize("e_min", [0.0, 1e-12, 1e-9])
@pytest.mark.parametrize("name", ["cavity", "cavity 4^3", "slab", "frame"])
def test_dense_solve_takes_a_step_or_two(name, e_min, kw):
    rho = _cell(name)
    Cj, _ = femh.Engine(solver=femh.JACOBI_PCG, E_min=e_min or 1e-9, autotune=0).homogenize(rho)
    C, info = femh.Engine(E_min=e_min, autotune=0, **kw).homogenize(rho)
    assert info["status"] == 0
    assert max(info["iterations"]) <= 3
    assert np.abs(C - Cj).max() <= 1e-8 * np.abs(Cj).max()


@pytest.mark.parametrize("kw", [dict(), dict(precision=femh.MIXED_PC), dict(block_cg=0)])
def test_load_of_soft_layers(kw):
    """Layers of 1 and 1e-12 in series: C_11 in closed form.  It is the soft
    layers' alone, so a net force of rounding size (1e-17) left on their nodes
    shows at 2e-9 of it; the direct solve and the energy sum round at 1e-13."""
    e = 1e-12
    rho = np.zeros((5, 7, 9))
    rho[:2] = 1
    C, info = femh.Engine(E_min=e, autotune=0, **kw).homogenize(rho)
    m = 0.7 / (1.3 * 0.4)   # (1 - nu) / ((1 + nu) (1 - 2 nu)), nu = 0.3
    exact = 1.0 / (0.4 / m + 0.6 / (e * m))
    assert info["status"] == 0 and abs(C[0, 0] / exact - 1) <= 1e-10
