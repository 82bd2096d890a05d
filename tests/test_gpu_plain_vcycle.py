"""V-cycles asked for by themselves, whose result no residual is tested on, are
FP64 V-cycles: the same bits as the kernels that run one colour at a time."""
import numpy as np
import pytest

from stz_gb300 import _lib
from stz_gb300.batch import Batch
from stz_gb300.params import simple_shear
from stz_gb300.shear_sim import ShearSim
from test_gpu_tgmg import _block_operator

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n", [(30, 31), (64, 64), (128, 100)])
def test_quasi_static(m, n):
    """Against a batch instance tuned to fuse = 0, whose FP64 cycles are those
    kernels."""
    P = simple_shear(m, n, viscosity=0.02)
    rng = np.random.default_rng(m)
    b, z = rng.standard_normal((2, n + 1, m, 2))
    batch = Batch([P], precision=_lib.FP64)
    batch.set_tuning(m, n, 1, -1, 0)
    batch.run(0.01, 1)
    with ShearSim(P, precision=_lib.FP64) as sim:
        for g in (0 * z, z):
            np.testing.assert_array_equal(sim.mg_vcycle(0.01, b, g), batch.sim(0).mg_vcycle(0.01, b, g))
    batch.close()


@pytest.mark.parametrize("m,n,yp", [(64, 33, 0), (128, 65, 0), (31, 30, 0)])
def test_blocks(m, n, yp):
    """An exactly solved coarsest level does not depend on the number of its
    sweeps; 11 of them run every level by itself."""
    import stz_gb300.tgmg as tg
    table, cls = _block_operator(m, n, 1, yp, lt=0.2)
    rng = np.random.default_rng(m)
    b, z = rng.standard_normal((2, n, m, 2))
    out = []
    for sweeps in (10, 11):
        q = tg.Problem(m, n, table, cls, 1e-20, x_prd=1, y_prd=yp, block=2)
        q.b[...], q.z[...] = b, z
        g = tg.Tgmg(q)
        g.v_cycle(hcyc_bottom=sweeps)
        out.append(q.z.copy())
        g.close()
    np.testing.assert_array_equal(*out)
