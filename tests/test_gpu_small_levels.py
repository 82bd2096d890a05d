"""The V-cycle's small-level kernel (bands over a cluster of blocks, the
coarsest levels as one matrix) and the float-pair tiles of FP64 handles, at
the sizes where their cuts and halos change: one block and many, odd coarse
lines, levels just inside and outside each limit, thin grids.  The converged
velocity of one solve against the CPU oracle's."""
import numpy as np
import pytest

from oracle.bind import OracleSim
from stz_gb300 import _lib
from stz_gb300.params import simple_shear
from stz_gb300.shear_sim import ShearSim

pytestmark = pytest.mark.gpu

SIZES = [(4, 6), (6, 5), (8, 40), (12, 29), (20, 20), (30, 31), (42, 40), (42, 43), (64, 64), (66, 130), (80, 15),
         (128, 128), (130, 130), (164, 163), (190, 142), (256, 64), (300, 128), (354, 98), (64, 500)]


@pytest.mark.parametrize("m,n", SIZES)
def test_solve_matches_oracle(m, n):
    P = simple_shear(m, n, viscosity=0.02)
    rng = np.random.default_rng(m * 1000 + n)
    src = rng.standard_normal((n + 1, m, 2)) * (m / (P.bx - P.ax)) ** 2
    o = OracleSim(P, np.full((n, m), 600.0 / P.TZ))
    o.set_tolerance(1, 1e-13)
    ref, _, ok = o.mg_solve(0.01, src, np.zeros_like(src))
    assert ok
    scale = np.abs(ref).max()
    # the repository's gates: FP64 1e-10, mixed 1e-8 of the field's scale
    for prec, tol, gate in ((_lib.FP64, 1e-13, 1e-10), (_lib.MIXED, 1e-12, 1e-8)):
        g = ShearSim(P, precision=prec, tol_mode=_lib.TOL_RELATIVE, tol=tol)
        vel, cycles, _ = g.mg_solve(0.01, src, np.zeros_like(src))
        assert np.abs(vel.reshape(ref.shape) - ref).max() < gate * scale, (prec, cycles)
        g.close()
    o.close()
