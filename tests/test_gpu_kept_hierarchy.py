"""A Newton solve that fails on the hierarchy kept from its increment's first tangent is done over on one of its
own. The failure is a cap on the CG iterations that the first solve of an increment meets (four on a small
beam, whose hierarchy is the exact inverse) and later ones on the kept hierarchy do not.

Tolerance: the NLGEOM bound of the other parity tests, 1e-8 against the oracle."""
import numpy as np
import pytest

import ferrix_b200 as fx
from ferrix_b200 import decks
from oracle import inp, static_step

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("max_iter", [4, 6])
def test_iteration_cap(max_iter):
    ctx = fx.Context(0)
    text = decks.write_deck(decks.c3d4_nlgeom_beam_spec(12, 3, 3, tip_load=3.0e4, increments=2))
    ref = static_step.Runner(inp.parse_inp_text(text)).run().displacements
    p = fx.Project.from_inp_text(text, ctx)
    st = fx.SolutionState(p.num_dofs, p.num_nodes)
    st.initialize(p)
    free = p.steps[0].solve(1, p, st, opts=fx.solve_opts(rtol=1e-10))
    assert free["pcg_iterations"] > max_iter * free["linear_solves"]  # the kept hierarchy needs more
    st.initialize(p)
    p.steps[0].solve(1, p, st, opts=fx.solve_opts(rtol=1e-10, max_iter=max_iter))
    err = float(np.linalg.norm(st.displacements - ref) / np.linalg.norm(ref))
    p.close()
    ctx.close()
    assert err <= 1e-8
