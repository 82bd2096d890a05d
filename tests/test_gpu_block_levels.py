"""The general multigrid's small levels of 2x2-block operators in one launch
(x periodic): the solution against the CPU oracle's at sizes where the levels
it takes change, with walls and with y periodic (even and odd coarse lines,
odd rows, the largest level just inside and outside its limit)."""
import numpy as np
import pytest

from oracle import tgmg_oracle as O
from test_gpu_tgmg import _block_operator

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,yp", [(16, 9, 0), (31, 30, 0), (48, 40, 1), (64, 64, 1), (90, 50, 1), (97, 65, 0),
                                    (128, 33, 0), (200, 131, 0)])
def test_solution_matches_oracle(m, n, yp):
    import stz_gb300.tgmg as tg
    table, cls = _block_operator(m, n, 1, yp, lt=0.2, seed=m)
    ops, _ = O.hierarchy(m, n, 1, yp, table, cls, 2)
    b = np.random.default_rng(m + n).standard_normal((n, m, 2))
    if yp:
        b -= b.mean(axis=(0, 1))
    q = tg.Problem(m, n, table, cls, 1e-26, x_prd=1, y_prd=yp, block=2)
    q.b[...] = b
    g = tg.Tgmg(q)
    assert g.solve_v_cycle(tg.Predict())
    # the solver's threshold on the mean squared residual, seen by the oracle
    assert O.l2_error(ops[0], q.z, b, 2) <= 1.01e-26 + (64 * 2.0 ** -53 * np.abs(q.z).max()) ** 2
    if not yp:
        z = O.solve(ops[0], b)
        assert np.abs(q.z - z).max() <= 1e-10 * np.abs(z).max()
    g.close()


@pytest.mark.parametrize("m,n", [(510, 257), (512, 257), (514, 259)])
def test_largest_level_in_and_out(m, n):
    """Level 1 at 32895, 33024 and 33410 points around the 33000 the launch
    takes: both sides converge, by the oracle's residual too, whose FP64 sums
    round at a few units of the solution."""
    import stz_gb300.tgmg as tg
    table, cls = _block_operator(m, n, 1, 0, lt=0.2)
    A = O.operator(m, n, 1, 0, table, cls, 2)
    b = np.random.default_rng(9).standard_normal((n, m, 2))
    q = tg.Problem(m, n, table, cls, 1e-20, x_prd=1, y_prd=0, block=2)
    q.b[...] = b
    g = tg.Tgmg(q)
    assert g.solve_v_cycle(tg.Predict())
    assert O.l2_error(A, q.z, b, 2) <= 1.01e-20 + (64 * 2.0 ** -53 * np.abs(q.z).max()) ** 2
    g.close()
