"""Step ends (one launch: pieces, instances, stop tests, the next step's start) at the edges of a reduction
piece: one full piece of 256 cells, a piece and a remainder, less than one, hundreds of pieces, the most
(592, 151,552 cells), several cells a thread (above that); instances of a batch that stop at different
steps."""

import numpy as np
import pytest

import teal_b200 as tb
from tests.cases import vortex

pytestmark = pytest.mark.gpu

LO, HI = (0, 0, 0), (10, 10, 0.625)


def problem(n):
    e = tb.Equations.euler(tb.Mesh.create(LO, HI, n, (1, 1, 1)))
    e.set_initial_condition("domain", vortex)
    return e


@pytest.mark.parametrize("n", [(16, 16, 2), (13, 11, 3), (5, 5, 3), (16, 8, 2), (150, 127, 4), (37, 64, 64), (53, 52, 55),
                               (90, 83, 61)])
def test_residual_norm_and_resident_steps(n):
    e = problem(n)
    ctx = e.context()
    C = e.mesh.num_inner_cells
    vol = e.mesh.cell_volume[:C]
    rng = np.random.default_rng(1)
    d = rng.standard_normal((C, 5)) * 10.0 ** rng.integers(-3, 3, (C, 5))
    # sums of C non-negative terms in trees: (log2 C + cells a thread) ulps at most
    want = np.sqrt((vol[:, None] * d**2).sum(axis=0) / e.mesh.sum_volume)
    assert np.allclose(ctx.residual(d), want, rtol=1e-14 * np.log2(C))
    # run(k) starts each next step in the launch that ends the last one; k Advance calls start their own
    ctx.set_primitive(e.primitive)
    t = 0.0
    for _ in range(4):
        t, step0, res = ctx.advance(tb.TG_ADVANCE_LSERK, 0.5, t)
    want = ctx.get_primitive().copy()
    ctx.set_primitive(e.primitive)
    t_run, it, res_run = ctx.run(tb.TG_ADVANCE_LSERK, 0.5, 4)
    assert (t_run, it) == (t, 4)
    assert ctx.last_step0() == step0
    assert np.array_equal(res_run, res)
    assert np.array_equal(ctx.get_primitive(), want)


def test_instances_stop_on_their_own():
    sizes, steps = [(16, 16, 2), (13, 11, 3), (20, 14, 4)], [2, 5, 3]
    alone = []
    for n, k in zip(sizes, steps):
        e = problem(n)
        ctx = e.context()
        t, it, res = ctx.run(tb.TG_ADVANCE_LSERK, 0.5, k)
        alone.append((t, it, res, ctx.get_primitive().copy(), e))
    b = tb.Batch([a[4] for a in alone])
    t, it, res = b.run(tb.TG_ADVANCE_LSERK, 0.5, steps)
    for i, a in enumerate(alone):
        assert (t[i], it[i]) == a[:2]
        assert np.array_equal(res[i], a[2])
        assert np.array_equal(b.get_primitive(i), a[3])
