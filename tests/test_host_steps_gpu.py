"""Steps from host state to host state on both sides of the chunk rule (two chunks from 262,144 cells on, below
that the replayed step with the copy behind it), against the three calls, and after a run loop that left
an end time behind."""

import numpy as np
import pytest
import torch

import teal_b200 as tb
from tests.cases import vortex

pytestmark = pytest.mark.gpu


def pinned(rows):
    return torch.empty((rows, 5), dtype=torch.float64, pin_memory=True).numpy()


@pytest.mark.parametrize("cells", [(30, 31, 29), (64, 64, 63), (64, 64, 65), (67, 63, 66)])
def test_host_step_equals_the_three_calls(cells):
    m = tb.Mesh.create((0, 0, 0), (10, 10, 10), cells, (1, 1, 1))
    e = tb.Equations.euler(m)
    e.set_initial_condition("domain", vortex)
    ctx = e.context()
    out, state = pinned(m.num_cells), e.primitive.copy()
    t = t_want = 0.0
    for _ in range(2):
        ctx.set_primitive(state)
        t_want, s_want, r_want = ctx.advance(tb.TG_ADVANCE_LSERK, 0.8, t)
        want = ctx.get_primitive()
        t, s, r = ctx.advance_host(tb.TG_ADVANCE_LSERK, 0.8, t, state, out)
        assert (t, s) == (t_want, s_want)
        assert np.array_equal(r, r_want)
        assert np.array_equal(out, want)
        state = want


@pytest.mark.parametrize("cells", [(20, 20, 4), (64, 64, 65)])
def test_host_step_after_a_run_with_an_end_time(cells):
    m = tb.Mesh.create((0, 0, 0), (10, 10, 10), cells, (1, 1, 1))
    e = tb.Equations.euler(m)
    e.set_initial_condition("domain", vortex)
    ctx = e.context()
    out = pinned(m.num_cells)
    _, step, _ = ctx.advance_host(tb.TG_ADVANCE_LSERK, 0.8, 0.0, e.primitive, out)
    ctx.set_primitive(e.primitive)
    ctx.run(tb.TG_ADVANCE_LSERK, 0.8, 5, max_time=0.5 * step)
    t, again, _ = ctx.advance_host(tb.TG_ADVANCE_LSERK, 0.8, 0.0, e.primitive, out)
    assert (t, again) == (step, step)
