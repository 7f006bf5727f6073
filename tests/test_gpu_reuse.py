"""A handle keeps its captured CG loops between solves: every solve on a used
handle gives the bits of a fresh one -- other densities, other shapes in
between, batches whose unit lists were compacted, profiling in between, and
the one-case loop that follows a failed block."""
import numpy as np
import pytest

from fem_b200 import femh, fields

pytestmark = pytest.mark.gpu

CONFIGS = [dict(precision=femh.FP64), dict(precision=femh.MIXED_PC), dict(precision=femh.MIXED),
           dict(solver=femh.JACOBI_PCG), dict(precision=femh.MIXED_PC, graph_chunk=3),
           dict(omega=1.9, cheb_ratio=0.0)]   # an indefinite V-cycle: block, then one case at a time


def _fresh(kw, rho):
    C, info = femh.Engine(autotune=0, **kw).homogenize(rho, allow_unconverged=True)
    return C, info["iterations"]


@pytest.mark.parametrize("kw", CONFIGS)
def test_used_handle_gives_the_same_bits(kw):
    a, b = fields.smooth_cell(16, 2.0, seed=1), fields.binary_cell(16, 0.6, seed=2)
    c = fields.smooth_cell(24, 2.0, seed=3)
    e = femh.Engine(autotune=0, **kw)
    for rho in (a, b, a, c, b):
        C, info = e.homogenize(rho, allow_unconverged=True)
        Cf, itf = _fresh(kw, rho)
        assert info["iterations"] == itf
        assert (C == Cf).all()
    e.profile(True)
    e.homogenize(b, allow_unconverged=True)
    e.profile(False)
    assert (e.homogenize(b, allow_unconverged=True)[0] == C).all()


def test_batches_on_a_used_handle():
    rhos = [fields.binary_cell(n, 0.35 + 0.03 * i, seed=70 + i) for i, n in enumerate((8, 16, 12, 24, 16, 8, 16, 24))]
    e = femh.Engine(autotune=0, precision=femh.MIXED_PC)
    C1 = e.batch(rhos)[0]
    C2 = e.batch(rhos)[0]
    C3 = e.batch(rhos[::-1])[0][::-1]
    assert (C1 == C2).all()
    assert np.abs(C1 - C3).max() <= 1e-12 * np.abs(C1).max()
