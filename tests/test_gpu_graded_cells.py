"""A strongly graded C3D20 box, whose constrained layer is over 100 times thinner than the last: it is not singular, whatever a
coarse operator below its corners or by smoothed transfers looks like, and is solved; the same box with one node held
is, and is refused.

The solve's own FP64 residual, as the statistics report it, is what is tested, at the target."""
import numpy as np
import pytest

import ferrix_b200 as fx
from ferrix_b200 import decks

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def arrays():
    lengths = (11.40388579, 32.87523111, 52.70647)
    mesh = decks.hex20_box(27, 10, 7, *lengths, jitter=0.1, seed=235)
    mesh.xyz[:, 0] = lengths[0] * (mesh.xyz[:, 0] / lengths[0]) ** 2.2881865908883756
    return decks.deck_arrays(decks.DeckSpec(mesh, [(2.0e5, 0.45, None)], clamp_axis=0, load_total=(-128.0, 72.3, 99.7)))


@pytest.mark.parametrize("prec", [fx.PREC_FP64, fx.PREC_MIXED])
@pytest.mark.parametrize("held", [True, False])
def test_graded(arrays, prec, held):
    a = dict(arrays)
    if not held:
        a["steps"] = [dict(a["steps"][0], bcs=a["steps"][0]["bcs"][:3])]
    ctx = fx.Context(0)
    p = fx.Project.from_arrays(**a, ctx=ctx)
    st = fx.SolutionState(p.num_dofs, p.num_nodes)
    st.initialize(p)
    opts = fx.solve_opts(precision=prec, rtol=1e-8, max_iter=3000)
    try:
        if held:
            s = p.steps[0].solve(1, p, st, None, fx.SolverTime(), opts)
            assert s["last_linear_relres"] <= 1e-8 and np.all(np.isfinite(st.displacements))
        else:
            with pytest.raises(fx.FerrixError, match="rigid body modes"):
                p.steps[0].solve(1, p, st, None, fx.SolverTime(), opts)
    finally:
        p.close()
        ctx.close()
