"""A batch's handle that is stepped by itself after the batch ran has the chip to
itself again: its V-cycle takes as long as that of a handle outside of any
batch (the batch's own schedule, for cycles that share the chip, takes twice
as long at this size)."""
import pytest

from stz_gb300 import _lib
from stz_gb300.batch import Batch
from stz_gb300.params import simple_shear
from stz_gb300.shear_sim import ShearSim

pytestmark = pytest.mark.gpu


def _cycle(sim, kernel):
    sim.time_kernel(0.01, kernel, 20)
    return min(sim.time_kernel(0.01, kernel, 50) for _ in range(5))


@pytest.mark.parametrize("prec,kernel", [(_lib.FP64, 3), (_lib.MIXED, 4)])
def test_schedule_after_a_batch(prec, kernel):
    P = simple_shear(256)
    batch = Batch([P] + [simple_shear(32)] * 23, precision=prec)
    batch.run(0.01, 1)
    with ShearSim(P, precision=prec) as sim:
        alone, after = _cycle(sim, kernel), _cycle(batch.sim(0), kernel)
    batch.close()
    assert after <= 1.1 * alone, (alone, after)
