"""Limited gradients where the limiter's minimum over faces is decided at an edge: constant states (every
delta2 below 1e-8), a single spike (cells at an extremum: delta1 zero), a step, a linear field, on
hexahedra and on mixed cells. Against the CPU restatement, whose candidates are taken face by face.

Bar: 1e-12 of the largest gradient, the plain form's gradient bar."""

import numpy as np
import pytest

import teal_b200 as tb
from oracle import port
from teal_b200 import meshes

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not port.available(), reason="CPU restatement not built")]

BASE = np.array([1.0, 0.4, 0.1, 0.05, 0.8])


def states(x, seed):
    rng = np.random.default_rng(seed)
    n = x.shape[0]
    flat = np.tile(BASE, (n, 1))
    spike = flat.copy()
    spike[rng.integers(n)] *= 1.3
    step = flat * np.where(x[:, :1] > np.median(x[:, 0]), 1.2, 1.0)
    return {"constant": flat, "spike": spike, "step": step, "linear": flat * (1 + 0.1 * x[:, :1]),
            "tiny": flat * (1 + 1e-9 * rng.random((n, 5)))}


@pytest.mark.parametrize("limiter", ["minmod", "venkatakrishnan"])
@pytest.mark.parametrize("mesh", ["box", "ramp"])
def test_limited_gradients_match_the_restatement(mesh, limiter):
    m = tb.Mesh.from_cells(meshes.ramp_mesh(n=(9, 8, 8), block=4, seed=3)) if mesh == "ramp" else \
        tb.Mesh.create((0, 0, 0), (1.1, 0.7, 0.5), (11, 7, 5), (1, 1, 1))
    e = tb.Equations.euler(m)
    e.set_limiter(limiter, 1.0)
    s = m.struct
    for i in range(s.num_inner_entities, s.off_boundary_entities):
        e.set_boundary_condition(m.entities[i][0], "slipwall")
    p, ctx = port.Port(m, e), e.context()
    C = m.num_inner_cells
    for name, prim in states(m.cell_center[: m.num_cells], 2).items():
        ctx.set_primitive(prim)
        got, want = ctx.gradient(limited=True), p.gradient(prim, limited=True)[:C]
        assert np.abs(got - want).max() <= 1e-12 * max(np.abs(want).max(), 1.0), name
