"""A call that is refused while the handle lays out its cells -- bad extents, a
bad voxel edge, a cell that does not halve, no memory -- leaves the handle
without a set-up: the solve before it can be repeated, with the same bits, and
until then what needs a solved cell is refused as out of order."""
import numpy as np
import pytest

from fem_b200 import femh, fields

pytestmark = pytest.mark.gpu

REFUSED = [((1, 16, 16), 1.0, femh.FEMH_E_ARG), ((16, 16, 260), 1.0, femh.FEMH_E_ARG),
           ((16, 16, 16), 0.0, femh.FEMH_E_ARG), ((44, 22, 22), 1.0, femh.FEMH_E_ARG),
           ((64, 64, 64), 1.0, femh.FEMH_E_OOM)]


@pytest.mark.parametrize("shape,h,code", REFUSED)
@pytest.mark.parametrize("prec", [femh.FP64, femh.MIXED_PC])
def test_the_cell_before_a_refused_call(shape, h, code, prec, monkeypatch):
    monkeypatch.setenv("FEMH_ARENA_LIMIT_BYTES", str(64 << 20))   # 16^3 fits, 64^3 does not
    e = femh.Engine(precision=prec, autotune=0)
    rho = fields.binary_cell(16, 0.5, seed=4)
    C, info = e.homogenize(rho, h=1.0)
    with pytest.raises(femh.FemhError) as ex:
        e.homogenize(np.full(shape, 0.5), h=h)
    assert ex.value.code == code
    with pytest.raises(femh.FemhError) as ex:
        e.grad(np.eye(6), out=np.zeros(rho.shape))
    assert ex.value.code == femh.FEMH_E_STATE
    C2, info2 = e.homogenize(rho, h=1.0)
    assert (C2 == C).all() and info2["iterations"] == info["iterations"]


def test_operator_after_a_refused_call():
    e = femh.Engine(autotune=0)
    rho = fields.binary_cell(16, 0.5, seed=4)
    u = np.random.default_rng(0).standard_normal((6, 16, 16, 16, 3))
    y = e.apply_operator(rho, u)
    with pytest.raises(femh.FemhError):
        e.apply_operator(np.full((16, 16, 260), 0.5), np.zeros((6, 16, 16, 260, 3)))
    assert (e.apply_operator(rho, u) == y).all()
