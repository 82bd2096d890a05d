"""Device memory of a handle: a mixed-precision one, whose solves run FP32
V-cycles, holds nothing that only FP64 V-cycles use."""
import gc

import pytest

from stz_gb300 import _lib
from stz_gb300.params import simple_shear
from stz_gb300.shear_sim import ShearSim

pytestmark = pytest.mark.gpu


def _bytes(P, prec):
    import torch
    gc.collect()
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    sim = ShearSim(P, precision=prec)
    used = before - torch.cuda.mem_get_info()[0]
    sim.close()
    return used


def test_mixed_handle_has_no_fp64_cycle_buffers():
    """Over an FP64 handle a mixed one has the pairs of iterate and right-hand
    side (32 bytes a node) and the FP32 levels (24 bytes, times 4/3 with the
    coarse ones): 64 bytes; without the FP64 cycles' correction (16 bytes) 48.
    Half the correction is left for the allocator's granularity."""
    m, n = 2048, 1023
    P = simple_shear(m, n)
    _bytes(P, _lib.FP64)  # the context and the modules
    extra = _bytes(P, _lib.MIXED) - _bytes(P, _lib.FP64)
    assert extra <= 56 * m * (n + 1)
