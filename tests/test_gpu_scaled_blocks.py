"""FP64 solves of 2x2-block operators over FP64's range: a power of two on the
right-hand side or on the operator is exact in every operation, so iterates
and counts have to be the same up to that power, bit for bit."""
import numpy as np
import pytest

from test_gpu_tgmg import _block_operator

pytestmark = pytest.mark.gpu

POWERS = [-400, -150, -100, 100, 150, 400]


def _solved(m, n, yp, b, table, cls, acc, iterate=False):
    import stz_gb300.tgmg as tg
    q = tg.Problem(m, n, table, cls, acc, x_prd=1, y_prd=yp, block=2)
    q.b[...] = b
    g = tg.Tgmg(q)
    if iterate:
        for _ in range(2):
            g.v_cycle()
    else:
        assert g.solve_v_cycle(tg.Predict())
    g.close()
    return q.z.copy(), None if iterate else g.iterations


@pytest.mark.parametrize("iterate", [False, True])
@pytest.mark.parametrize("m,n,yp", [(64, 33, 0), (48, 40, 1), (31, 30, 0)])
@pytest.mark.parametrize("k", POWERS)
def test_right_hand_side_and_operator(m, n, yp, k, iterate):
    table, cls = _block_operator(m, n, 1, yp, lt=0.2, seed=m)
    b = np.random.default_rng(m + n).standard_normal((n, m, 2))
    if yp:
        b -= b.mean(axis=(0, 1))
    s = 2.0 ** k
    z, it = _solved(m, n, yp, b, table, cls, 1e-20, iterate)
    zk, itk = _solved(m, n, yp, b * s, table, cls, 1e-20 * s * s, iterate)
    assert itk == it
    np.testing.assert_array_equal(zk, z * s)
    zk, itk = _solved(m, n, yp, b, table * s, cls, 1e-20, iterate)
    assert itk == it
    np.testing.assert_array_equal(zk, z / s)
