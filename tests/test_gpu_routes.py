"""Routes that other tests rely on, and one that none of them takes: the fused
coarse end of the V-cycle runs for a few cells and not for many, the staged
kernels run in a batch whose cells share a z extent between two pitches, and
SIMP's exponent 3 gives what the general power gives."""
import numpy as np
import pytest

from fem_b200 import femh, fields

pytestmark = pytest.mark.gpu


def _kernels(e, solve):
    e.profile(True)
    solve()
    names = {k["name"] for k in e.profile_read()}
    e.profile(False)
    return names


def test_fused_end_for_few_cells_level_kernels_for_many():
    import torch
    rho = fields.binary_cell(16, 0.55, seed=0)
    e = femh.Engine(precision=femh.MIXED_PC, autotune=0)
    one = _kernels(e, lambda: e.homogenize(rho))
    assert "k_tail" in one and "k_coarse_solve" not in one
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    few, many = sms * 8 // 6, sms * 8 // 6 + 1   # six CTAs a cell, eight waves
    assert "k_tail" in _kernels(e, lambda: e.batch([rho] * few))
    assert "k_tail" not in _kernels(e, lambda: e.batch([rho] * many))


@pytest.mark.parametrize("prec", [femh.FP64, femh.MIXED_PC])
def test_fused_end_with_an_unknown_per_thread(prec):
    """7 x 7 x 3 = 147 coarsest nodes, 441 unknowns for its 512 threads, and
    5 x 5 x 7 = 175 nodes, 525 unknowns: two passes over the dense inverse."""
    for shape, fused in [((28, 28, 12), True), ((20, 20, 28), False)]:
        e = femh.Engine(precision=prec, autotune=0)
        rho = np.random.default_rng(2).uniform(0.2, 1.0, shape)
        assert ("k_tail" in _kernels(e, lambda: e.homogenize(rho))) == fused


@pytest.mark.parametrize("kw", [dict(stencil_variant=5, precision=femh.MIXED_PC),
                                dict(stencil_variant=6), dict(stencil_variant=7, precision=femh.MIXED)])
def test_batch_on_one_z_extent_between_pitches(kw):
    """40 and 20 on the levels: rows of 40 in a pitch of 48, cells at offsets
    that are not multiples of it."""
    rng = np.random.default_rng(1)
    rhos = [rng.uniform(0.1, 1.0, s) for s in [(8, 12, 40), (4, 8, 40), (12, 4, 40)]]
    C, infos, _ = femh.Engine(**kw).batch(rhos)
    for r, c, i in zip(rhos, C, infos):
        Cj, _ = femh.Engine(solver=femh.JACOBI_PCG, stencil_variant=1).homogenize(r)
        assert i["status"] == 0 and np.abs(c - Cj).max() <= 1e-8 * np.abs(Cj).max()


@pytest.mark.parametrize("p", [np.nextafter(3.0, 0.0), np.nextafter(3.0, 4.0)])
def test_exponent_three_is_the_general_power(p):
    """rho^3 and rho^2 by products against pow at the next exponents: rho >= 0.05,
    so the exponent's ulp moves the power by 3 x 4.4e-16 and its rounding by a
    few ulp; C^H and dC^H/drho are as smooth in the coefficients, and their sums
    and the solve (residual 1e-12) add rounding below 1e-10 of the largest value."""
    rho = 0.05 + 0.95 * fields.smooth_cell(16, 2.0, seed=3)
    out = []
    for q in (3.0, p):
        e = femh.Engine(penal=float(q), tol=1e-12, autotune=0)
        C, _ = e.homogenize(rho)
        out.append((C, e.dCdrho()))
    for a, b in zip(*out):
        assert np.abs(a - b).max() <= 1e-10 * np.abs(b).max()
