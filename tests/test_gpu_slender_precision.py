"""Mixed precision on slender C3D20 cantilevers, whose cycle FP16 smoothing spoils: by default it is given up within 64
iterations, so that the mixed solve takes at most those and about the FP64 solve's iterations (a third more and four,
the spread that FP32 smoothing leaves), and its displacements are those of FP64 to 1e-6 (the residual target of
1e-9 times the conditioning that these decks show, ~1e3)."""
import numpy as np
import pytest

import ferrix_b200 as fx
from ferrix_b200 import decks

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells", [(7, 5, 35), (4, 3, 40)])
@pytest.mark.parametrize("kw", [dict(), dict(amg_cycle=1), dict(amg_fused_coarse=1), dict(use_graphs=0)])
def test_slender(cells, kw):
    mesh = decks.hex20_box(*cells, 0.25 * cells[0], 0.038 * cells[1], 0.4 * cells[2])
    spec = decks.DeckSpec(mesh, [(2.0e5, 0.3, None)], load_total=(10.0, -20.0, 30.0), clamp_axis=2)
    ctx = fx.Context(0)
    p = fx.Project.from_arrays(**decks.deck_arrays(spec), ctx=ctx)
    st = fx.SolutionState(p.num_dofs, p.num_nodes)
    u, its = [], []
    for prec in (fx.PREC_FP64, fx.PREC_MIXED):
        st.initialize(p)
        its.append(p.steps[0].solve(1, p, st, None, fx.SolverTime(), fx.solve_opts(precision=prec, rtol=1e-9, **kw))
                   ["pcg_iterations"])
        u.append(st.displacements)
    p.close()
    ctx.close()
    assert its[1] <= its[0] + its[0] // 3 + 4 + 64, its
    assert float(np.linalg.norm(u[1] - u[0]) / np.linalg.norm(u[0])) <= 1e-6
