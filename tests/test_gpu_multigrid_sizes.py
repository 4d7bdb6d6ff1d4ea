"""The multigrid's coarsest-level inverse at the sizes where its panels and tiles end: one
aggregate (6 DOF, a partial panel), just below and above one 32-pivot panel, partial last
panels, sizes on both sides of a 64-row tile, up to the largest dense level. The size follows
from the aggregate size asked for; the solve must meet the oracle's FP64 direct solution.

Tolerance: the FP64 solver's bound of the other parity tests, 1e-10 relative in the 2-norm, with the
residual target tightened to 1e-11 so that the bound does not depend on the stopping point."""
import numpy as np
import pytest

import ferrix_b200 as fx
from ferrix_b200 import decks
from oracle import inp, static_step

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = fx.Context(0)
    yield c
    c.close()


@pytest.fixture(scope="module")
def deck():
    text = decks.c3d4_cantilever(4, 5, 9)  # 300 nodes
    return text, static_step.Runner(inp.parse_inp_text(text)).run().displacements


@pytest.mark.parametrize("nodes", [2, 3, 4, 6, 9, 14, 20, 33, 50, 75, 120, 300, 5000])
def test_coarsest_inverse_sizes(ctx, deck, nodes):
    text, ref = deck
    p = fx.Project.from_inp_text(text, ctx)
    st = fx.SolutionState(p.num_dofs, p.num_nodes)
    st.initialize(p)
    p.steps[0].solve(1, p, st, opts=fx.solve_opts(precision=fx.PREC_FP64, rtol=1e-11, amg_aggregate_nodes=nodes,
                                                  amg_persistent_max_dof=-1))
    err = float(np.linalg.norm(st.displacements - ref) / np.linalg.norm(ref))
    p.close()
    assert err <= 1e-10, err
