"""Face fluxes and cell update in one launch (arenas of at most TG_FUSED_CELLS cells) against the two
launches of larger arenas: a mesh alone takes the first, packed beside a larger one the second, and its
bits are the same. Sizes around a 32-cell tile, mixed cells, boundaries, both precisions, explicit and
implicit steps, instances that stop early; fully periodic boxes of up to the most cells that one launch
takes, whose tiles do not all start together, over many steps."""

import numpy as np
import pytest

import teal_b200 as tb
from teal_b200 import meshes

pytestmark = pytest.mark.gpu

FREE = (1.0, 1.3, 0.1, 0.0, 1.0 / 1.4)


def problem(mesh, flux, seed):
    e = tb.Equations.euler(mesh)
    e.set_convective_flux(flux)
    e.set_limiter("venkatakrishnan", 1.0)
    s = mesh.struct
    for i in range(s.num_inner_entities, s.off_boundary_entities):
        side = mesh.entities[i][0]
        far = side in ("left", "right", "top")
        e.set_boundary_condition(side, "farfield" if far else "slipwall", FREE if far else None)
    rng = np.random.default_rng(seed)
    e.primitive[:] = np.tile(np.array(FREE), (mesh.num_cells, 1)) * (1 + 0.02 * rng.random((mesh.num_cells, 5)))
    return e


def box(n, periodic=(0, 0, 1)):
    return tb.Mesh.create((0, 0, 0), tuple(0.1 * x for x in n), n, periodic)


@pytest.fixture(scope="module")
def large():
    return box((40, 40, 27))  # 43,200 cells


@pytest.mark.parametrize("precision", [tb.TG_PRECISION_FP64, tb.TG_PRECISION_FP32_FLUX])
@pytest.mark.parametrize("method", [(tb.TG_ADVANCE_LSERK, 0.5, (3, 3)), (tb.TG_ADVANCE_IMPLICIT_EULER, 10.0, (0.1, 0.3, 30))])
@pytest.mark.parametrize("shape,flux", [((4, 4, 2), "roe"), ((5, 3, 3), "hllc"), ((13, 11, 3), "ausmd"), ("ramp", "hllc"),
                                        ("ramp", "hll"), ("ramp", "hlle"), ("ramp", "ausmdv"), ("ramp", "lxf"),
                                        ((6, 5, 4), "central")])
def test_alone_equals_packed(large, shape, flux, method, precision):
    mesh = tb.Mesh.from_cells(meshes.ramp_mesh(n=(9, 8, 8), block=4, seed=3)) if shape == "ramp" else box(shape)
    how, cfl, context = method
    small = problem(mesh, flux, 1)
    ctx = small.context(precision)
    t, it, res = ctx.run(how, cfl, 3, context=context)
    b = tb.Batch([small, problem(large, flux, 2)], precision)
    t_b, it_b, res_b = b.run(how, cfl, [3, 1], context=context)
    assert (t_b[0], it_b[0], it_b[1]) == (t, it, 1)
    assert np.array_equal(res_b[0], res)
    assert np.array_equal(b.get_primitive(0), ctx.get_primitive())


@pytest.mark.parametrize("precision", [tb.TG_PRECISION_FP64, tb.TG_PRECISION_FP32_FLUX])
@pytest.mark.parametrize("shape", [(5, 4, 3), (27, 23, 11), (64, 64, 4), (37, 32, 16), (33, 31, 18), (37, 16, 33)])
def test_periodic_alone_equals_packed(large, shape, precision):
    # up to 592 tiles (18,944 cells); 37 x 16 x 33 = 19,536 cells are past the limit
    mesh = box(shape, (1, 1, 1))
    small = problem(mesh, "hllc", 1)
    ctx = small.context(precision)
    b = tb.Batch([small, problem(large, "hllc", 2)], precision)
    want = b.run(tb.TG_ADVANCE_LSERK, 0.5, [40, 1])
    for _ in range(3):
        ctx.set_primitive(small.primitive)
        t, it, res = ctx.run(tb.TG_ADVANCE_LSERK, 0.5, 40)
        assert (t, it) == (want[0][0], want[1][0])
        assert np.array_equal(res, want[2][0])
        assert np.array_equal(ctx.get_primitive(), b.get_primitive(0))
