"""Steps from host state to host state on both sides of the chunk rule (two chunks from 262,144 cells on, below
that the replayed step with the copy behind it), against the three calls, and after a run loop that left
an end time behind; steps whose time order changes at the same number of stages; read-backs into
pageable memory."""

import threading
import time

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


def test_host_steps_of_changing_courant_numbers():
    """A kind of step is launched plainly the first time and replayed after that: the same bits either way,
    and as the three calls."""
    m = tb.Mesh.create((0, 0, 0), (10, 10, 10), (20, 18, 4), (1, 1, 1))
    e = tb.Equations.euler(m)
    e.set_initial_condition("domain", vortex)
    ctx, three = tb.Context(m, e), tb.Context(m, e)
    out, state = pinned(m.num_cells), e.primitive.copy()
    t = 0.0
    for courant in (0.4, 0.4, 0.4, 0.6, 0.4, 0.4, 0.8, 0.8, 0.6):
        three.set_primitive(state)
        want = three.advance(tb.TG_ADVANCE_LSERK, courant, t)
        got = ctx.advance_host(tb.TG_ADVANCE_LSERK, courant, t, state, out)
        assert got[:2] == want[:2]
        assert np.array_equal(got[2], want[2])
        assert np.array_equal(out, three.get_primitive())
        state, t = out.copy(), got[0]


@pytest.mark.parametrize("how", ["advance", "advance_host", "run"])
def test_time_order_changes_at_a_fixed_stage_count(how):
    m = tb.Mesh.create((0, 0, 0), (10, 10, 10), (20, 18, 4), (1, 1, 1))
    e = tb.Equations.euler(m)
    e.set_initial_condition("domain", vortex)
    out = pinned(m.num_cells)

    def state(ctx, rk):
        if how == "advance_host":
            ctx.advance_host(tb.TG_ADVANCE_LSERK, 0.8, 0.0, e.primitive, out, context=rk)
            return out.copy()
        ctx.set_primitive(e.primitive)
        if how == "advance":
            ctx.advance(tb.TG_ADVANCE_LSERK, 0.8, 0.0, context=rk)
        else:
            ctx.run(tb.TG_ADVANCE_LSERK, 0.8, 2, context=rk)
        return ctx.get_primitive()

    orders = [(3, 3), (2, 3), (1, 3), (3, 3)]
    want = [state(tb.Context(m, e), rk) for rk in orders]  # a context each
    ctx = e.context()
    for rk, w in zip(orders, want):
        assert np.array_equal(state(ctx, rk), w), rk
    assert not np.array_equal(want[0], want[1])


# one chunk of 1 MiB and a little, several, with helpers (16 MiB), and more than 64 chunks (which then grow)
@pytest.mark.parametrize("cells", [(31, 29, 30), (64, 64, 65), (76, 75, 78), (120, 121, 122)])
def test_pageable_read_back(cells):
    m = tb.Mesh.create((0, 0, 0), (10, 10, 10), cells, (1, 1, 1))
    e = tb.Equations.euler(m)
    rng = np.random.default_rng(1)
    e.primitive[:] = 1 + rng.random((m.num_cells, 5))
    ctx = tb.Context(m, e)
    ctx.set_primitive(e.primitive)
    want = pinned(m.num_cells)
    ctx.get_primitive(want)
    stream = torch.cuda.Stream()
    ctx.set_stream(stream.cuda_stream)
    got = np.empty((m.num_cells, 5))
    ctx.get_primitive(got)
    assert np.array_equal(got, want)
    # while the device still computes, the threads that will copy sleep
    got[:] = 0
    with torch.cuda.stream(stream):
        torch.cuda._sleep(600_000_000)  # about 0.3 s
    wall, cpu = time.perf_counter(), time.process_time()
    ctx.get_primitive(got)
    wall, cpu = time.perf_counter() - wall, time.process_time() - cpu
    assert np.array_equal(got, want)
    assert wall > 0.1
    assert cpu < 1.8 * wall  # this thread and the copies; three spinning threads more would be near four
    ctx.close()


def test_pageable_read_backs_of_several_threads():
    """Each context's helpers serve its own calls: contexts read back by several threads at once, many times, into
    arrays that change, one of them destroyed and made anew in between."""
    wrong = []

    def work(seed, cells):
        m = tb.Mesh.create((0, 0, 0), (10, 10, 10), cells, (1, 1, 1))
        e = tb.Equations.euler(m)
        rng = np.random.default_rng(seed)
        for _ in range(3):
            ctx = tb.Context(m, e)
            for _ in range(20):
                e.primitive[: m.num_inner_cells] = 1 + rng.random((m.num_inner_cells, 5))
                ctx.set_primitive(e.primitive)
                got = np.zeros((m.num_cells, 5))
                ctx.get_primitive(got)
                if not np.array_equal(got[: m.num_inner_cells], e.primitive[: m.num_inner_cells]):
                    wrong.append(seed)
            ctx.close()

    threads = [threading.Thread(target=work, args=a) for a in ((1, (31, 29, 31)), (2, (76, 75, 78)), (3, (77, 74, 79)))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
