"""2x2-block solvers whose level 1 lies on either side of the largest one that the
small-level launch takes (33,000 nodes; on a tall grid it fits): 32,896 and
33,152 nodes.  Both converge by the oracle's residual, whose FP64 sums round
at a few units of the solution."""
import numpy as np
import pytest

from oracle import tgmg_oracle as O
from test_gpu_tgmg import _block_operator

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n", [(256, 512), (256, 516)])
def test_either_side_of_the_limit(m, n):
    import stz_gb300.tgmg as tg
    table, cls = _block_operator(m, n, 1, 0, lt=0.2)
    b = np.random.default_rng(9).standard_normal((n, m, 2))
    q = tg.Problem(m, n, table, cls, 1e-20, x_prd=1, y_prd=0, block=2)
    q.b[...] = b
    g = tg.Tgmg(q)
    assert (g.levels()[1][0] * g.levels()[1][1] <= 33000) == (n == 512)
    assert g.solve_v_cycle(tg.Predict())
    A = O.operator(m, n, 1, 0, table, cls, 2)
    assert O.l2_error(A, q.z, b, 2) <= 1.01e-20 + (64 * 2.0 ** -53 * np.abs(q.z).max()) ** 2
    g.close()
