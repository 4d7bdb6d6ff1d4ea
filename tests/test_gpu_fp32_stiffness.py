"""FP32 element stiffness of C3D20 meshes away from the origin: its error against the FP64 matrix.

Bound: the coordinates (up to 32 element lengths) cancel in the Jacobian, so FP32 shape derivatives alone
leave an error of a few units of 6e-8 times that ratio. 1.4e-6 and 0.45e-6 in the norm are what a summation by trees
of FP32 warp reductions leaves on these meshes (1.3e-6, 0.4e-6); 20 FP32 terms in sequence leave 1.9e-6 and 0.7e-6."""
import numpy as np
import pytest

import ferrix_b200 as fx
from ferrix_b200 import decks

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells,jitter,bound", [((8, 8, 32), 0.1, 1.4e-6), ((3, 2, 9), 0.0, 0.45e-6)])
def test_error(cells, jitter, bound):
    mesh = decks.hex20_box(*cells, *(float(c) for c in cells), jitter=jitter, seed=2)
    ctx = fx.Context(0)
    p = fx.Project.from_arrays(**decks.deck_arrays(decks.DeckSpec(mesh, [(2.0e5, 0.3, None)])), ctx=ctx)
    fx.SolutionState(p.num_dofs, p.num_nodes).initialize(p)
    a, b = (p.assemble_csr(None, prec)[2] for prec in (fx.PREC_FP64, fx.PREC_MIXED))
    p.close()
    ctx.close()
    assert np.linalg.norm(a - b) <= bound * np.linalg.norm(a)
