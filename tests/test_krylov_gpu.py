"""The Krylov vector passes of the implicit step at the sizes where they can go wrong: cell counts around
a piece (PIECE_CELLS = 256 cells, one a thread), pieces of several cells a thread (above PIECE_COUNT = 592 of
them, 151,552 cells), bases that are no multiple of the four vectors loaded together, that fill the
Krylov dimension, and that are longer than one accumulator tile (64), with one cell a thread and with
two. Against the CPU restatement (oracle/port.py).

Bar: the implicit bar without a limiter. The restatement's own step moves by 3e-9..9e-9 when its input
is perturbed by 1e-16 (test_parity_gpu.py states the measurement); 1e-7 is about ten times that."""

import numpy as np
import pytest

import teal_b200 as tb
from oracle import port
from tests.cases import rel_l2

pytestmark = pytest.mark.gpu

FREE = (1.0, 0.6, 0.1, 0.0, 1.0 / 1.4)


@pytest.mark.skipif(not port.available(), reason="CPU restatement not built")
@pytest.mark.parametrize("cells,krylov_tol,dim", [
    ((16, 16, 1), 0.3, 30),      # one full piece
    ((33, 8, 1), 0.3, 30),       # a piece and 8 cells
    ((7, 5, 3), 1e-3, 5),        # less than a piece, the Krylov dimension filled
    ((10, 9, 4), 1e-10, 100),    # more columns than an accumulator tile holds
    ((44, 42, 41), 0.05, 30),    # 75,768 cells: 296 pieces, the last one short
    ((44, 42, 43), 0.05, 30),    # 79,464 cells: 311 pieces
    ((37, 64, 64), 0.1, 30),     # 151,552 cells: 592 full pieces, the most of one cell a thread
    ((53, 52, 55), 0.05, 30),    # 151,580 cells: two cells a thread, 297 pieces, 28 cells in the last
    ((53, 52, 55), 1e-10, 70),   # the same with more columns than an accumulator tile holds
])
def test_implicit_step_matches_the_restatement(cells, krylov_tol, dim):
    n = np.array(cells)
    m = tb.Mesh.create((0, 0, 0), tuple(n / n.max()), cells, (0, 0, 1))
    e = tb.Equations.euler(m)
    e.set_limiter(None)
    for side in ("left", "right", "bottom", "top"):
        e.set_boundary_condition(side, "farfield", FREE)
    rng = np.random.default_rng(7)
    prim = np.tile(np.array(FREE), (m.num_cells, 1))
    wave = np.sin(m.cell_center[: m.num_cells] @ rng.uniform(2, 5, (3, 5)))
    prim *= 1 + 0.05 * wave
    prim[:, 3] = 0.05 * wave[:, 3]
    nk = (0.1, krylov_tol, dim)
    want, t_want, _, res_want = port.Port(m, e).advance(prim, "implicit", 30.0, 1, nk=nk)
    ctx = e.context()
    ctx.set_primitive(prim)
    t, _, res = ctx.advance(tb.TG_ADVANCE_IMPLICIT_EULER, 30.0, 0.0, context=nk)
    C = m.num_inner_cells
    assert abs(t - t_want) <= 1e-13 * t_want
    assert rel_l2(ctx.get_primitive()[:C], want[:C]).max() <= 1e-7
    assert np.allclose(res, res_want, rtol=1e-5)
