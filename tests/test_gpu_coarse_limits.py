"""The dense coarse matrix's assembly keeps three rows of it in dynamic shared
memory, 72 B per coarse node: coarsest levels on both sides of the 48 KB that a
launch gets without asking (static shared memory included), and up to the
largest that the multigrid accepts.  The limit belongs to the function, not to
the handle, so every cell is solved first in a process of its own, and handles
of different sizes run side by side."""
import os
import subprocess
import sys
import threading

import numpy as np
import pytest

from fem_b200 import femh

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CHILD = """
import sys
import numpy as np
from fem_b200 import femh
shape = tuple(int(v) for v in sys.argv[1].split("x"))
prec = int(sys.argv[2])
rho = np.random.default_rng(3).uniform(0.2, 1.0, shape)
C, info = femh.Engine(precision=prec, autotune=0).homogenize(rho)
Cj, _ = femh.Engine(solver=femh.JACOBI_PCG, autotune=0).homogenize(rho)
assert abs(C - Cj).max() <= 1e-8 * abs(Cj).max()
assert max(info["iterations"]) <= 60, info
"""


# nodes of the coarsest level: 680 (48,960 B, above 48 KB only with the static
# part), 682, 684 (above by itself), 1331, 1530 and 1536, the largest
@pytest.mark.parametrize("shape", ["17x10x4", "34x20x8", "31x11x2", "19x9x4", "22x22x22", "17x15x6", "2x24x32"])
@pytest.mark.parametrize("prec", [femh.FP64, femh.MIXED_PC])
def test_first_cell_of_a_process(shape, prec):
    res = subprocess.run([sys.executable, "-c", CHILD, shape, str(prec)], cwd=ROOT, capture_output=True, text=True,
                         timeout=300)
    assert res.returncode == 0, res.stderr[-2000:]


def test_handles_side_by_side():
    """Two handles in two threads whose assembly needs 49,248 and 52,488 B."""
    rhos = [np.random.default_rng(n).uniform(0.2, 1.0, s) for n, s in enumerate([(19, 9, 4), (9, 9, 9)])]
    cfg = dict(tol=1e-3, autotune=0)
    alone = [femh.Engine(**cfg).homogenize(r)[0] for r in rhos]
    start, errors = threading.Barrier(2), []

    def work(q):
        try:
            e = femh.Engine(**cfg)
            start.wait()
            for _ in range(200):
                C, info = e.homogenize(rhos[q])
                assert info["status"] == 0 and (C == alone[q]).all()
        except Exception as ex:
            errors.append(ex)

    threads = [threading.Thread(target=work, args=(q,)) for q in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
