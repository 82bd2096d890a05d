"""The small levels' tables and matrices of a 2x2-block solver are made by the
first FP64 V-cycle that takes them, not by every handle and operator."""
import gc

import numpy as np
import pytest

from test_gpu_tgmg import _block_operator

pytestmark = pytest.mark.gpu


def _free():
    import torch
    gc.collect()
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def test_laid_out_on_first_use():
    import stz_gb300.tgmg as tg
    m, n = 448, 226  # the levels from 28 x 16 on are matrices
    table, cls = _block_operator(m, n, 1, 0, lt=0.2)
    b = np.random.default_rng(1).standard_normal((n, m, 2))
    solvers = []
    for _ in range(8):
        q = tg.Problem(m, n, table, cls, 1e-16, x_prd=1, y_prd=0, block=2)
        q.b[...] = b
        g = tg.Tgmg(q)
        g.set_precision(True)
        assert g.solve_v_cycle(tg.Predict())
        g.set_operator(table, keep_classes=True)
        assert g.solve_v_cycle(tg.Predict())
        solvers.append((g, q))
    before = _free()
    for g, q in solvers:
        z = q.z.copy()
        g.set_precision(False)
        q.z[...] = 0
        assert g.solve_v_cycle(tg.Predict())
        assert np.abs(q.z - z).max() <= 1e-6 * np.abs(z).max()
    # the matrices, as far as the allocator does not have the room left over
    assert before - _free() >= 4 * (2 * 28 * 16) ** 2 * 8
    for g, _ in solvers:
        g.close()


def test_new_operators_and_class_maps():
    """After operators and class maps that it solved, skipped (no FP64 solve in
    between) or kept, a solver solves bit for bit like a new one."""
    import stz_gb300.tgmg as tg
    m, n = 64, 48
    t0, c0 = _block_operator(m, n, 1, 0, lt=0.1)
    t1, _ = _block_operator(m, n, 1, 0, lt=0.4)
    c1 = c0.copy()
    c1[n // 2, :] = 1
    c2 = c0.copy()
    c2[n // 3, m // 4] = 1  # classes per point
    b = np.random.default_rng(2).standard_normal((n, m, 2))

    def solve(g, q):
        q.b[...], q.z[...] = b, 0
        assert g.solve_v_cycle(tg.Predict())
        return q.z.copy()

    q = tg.Problem(m, n, t0, c0, 1e-22, x_prd=1, y_prd=0, block=2)
    g = tg.Tgmg(q)
    solve(g, q)
    for t, c, use in ((t1, c1, True), (t0, c2, False), (t1, c2, True), (t0, None, False), (t1, c0, False),
                      (t0, None, True), (t0, c2, True), (t1, c1, True)):
        g.set_operator(t, c, keep_classes=c is None)
        if use:
            qf = tg.Problem(m, n, t, q.cls, 1e-22, x_prd=1, y_prd=0, block=2)
            gf = tg.Tgmg(qf)
            np.testing.assert_array_equal(solve(g, q), solve(gf, qf))
            gf.close()
    g.close()
