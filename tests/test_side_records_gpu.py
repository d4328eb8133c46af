"""Residuals through the side records (second order without a viscous flux) where they can go wrong: cell
counts that are no multiple of a 32-cell tile, periodic axes two and three cells thick (the periodic
faces have no slot in their right cell), boundaries, mixed cells whose tiles hold fewer slots. Against the
CPU restatement (oracle/port.py), the gradient entry point beside them, and the states the fluxes may read.

Bars: 1e-12 in FP64, the residual bar of the plain form. The FP32-flux residual rounds states of order one
to 2^-24 at h of about 1/10, where a residual component is a sum of six face fluxes over h: about
6 x 6e-8 x 10 = 4e-6 of the state, on residuals of order one."""

import numpy as np
import pytest

import teal_b200 as tb
from oracle import port
from teal_b200 import meshes
from teal_b200 import partition as pt
from tests.cases import rel_l2

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not port.available(), reason="CPU restatement not built")]

FREE = (1.0, 1.1, 0.2, 0.1, 1.0 / 1.4)


def problem(shape):
    if shape == "ramp":
        m = tb.Mesh.from_cells(meshes.ramp_mesh(n=(10, 9, 8), block=4, seed=3))
        periodic = False
    else:
        n, per = shape
        m = tb.Mesh.create((0, 0, 0), tuple(0.1 * x for x in n), n, per)
        periodic = all(per)
    e = tb.Equations.euler(m)
    if not periodic:
        s = m.struct
        for i in range(s.num_inner_entities, s.off_boundary_entities):
            side = m.entities[i][0]
            e.set_boundary_condition(side, "slipwall" if side in ("bottom", "back") else "farfield",
                                     None if side in ("bottom", "back") else FREE)
    rng = np.random.default_rng(5)
    prim = np.tile(np.array(FREE), (m.num_cells, 1)) * (1 + 0.1 * rng.random((m.num_cells, 5)))
    return m, e, prim


@pytest.mark.parametrize("limiter", [None, "minmod", "venkatakrishnan"])
@pytest.mark.parametrize("shape", [((3, 3, 2), (1, 1, 1)), ((7, 5, 3), (1, 1, 1)), ((8, 4, 2), (1, 0, 1)),
                                   ((11, 3, 2), (0, 0, 1)), ((16, 2, 3), (0, 1, 0)), "ramp"])
def test_residual_matches_the_restatement(shape, limiter):
    m, e, prim = problem(shape)
    e.set_limiter(limiter, 1.0)
    e.set_convective_flux("hllc")
    p = port.Port(m, e)
    want = p.derivative(prim)
    ctx = e.context()
    got = ctx.derivative(prim)
    assert rel_l2(got, want).max() <= 1e-12
    # gradients asked for between two residuals do not disturb them
    ctx.set_primitive(prim)
    g = ctx.gradient(limited=limiter is not None)
    g_want = p.gradient(prim, limited=limiter is not None)[: m.num_inner_cells]
    assert np.abs(g - g_want).max() <= 1e-12 * np.abs(g_want).max()
    assert np.array_equal(ctx.derivative(), got)
    if shape == "ramp":
        # jittered faces do not close a cell exactly, so the FP32-flux form's reference pressure shows there
        return
    f = e.context(tb.TG_PRECISION_FP32_FLUX)
    f.set_primitive(prim)
    assert np.linalg.norm(f.derivative() - want) <= 2e-5 * np.linalg.norm(want)


@pytest.mark.parametrize("precision", [tb.TG_PRECISION_FP64, tb.TG_PRECISION_FP32_FLUX])
@pytest.mark.parametrize("n,periodic", [((7, 5, 3), (1, 1, 1)), ((8, 4, 2), (1, 0, 1)), ((33, 2, 3), (0, 1, 0))])
def test_fluxes_read_no_inner_state(n, periodic, precision):
    """The fluxes of a stage come from the records alone: the fused face and cell kernel writes the state
    while other blocks form theirs. A partition's phases let the state change between the two."""
    m, e, prim = problem((n, periodic))
    part = pt.partition(m, np.zeros(m.num_inner_cells, int))[0]
    other = prim * 1.5
    other[0, 4] = prim[0, 4]  # the FP32-flux form's reference pressure
    got = []
    for change in (False, True):
        r = pt.Rank(part, e, precision)
        r.set_state(prim)
        r.set_step(0.5 * r.step_begin(), 0.0)
        r.phase(0)
        r.phase(1)
        if change:
            r.set_state(other)
        r.phase(2, 1.0, 1)
        got.append(r.state().copy())
        r.close()
    assert np.array_equal(got[0], got[1])
    assert not np.array_equal(got[0], prim[: m.num_inner_cells])
