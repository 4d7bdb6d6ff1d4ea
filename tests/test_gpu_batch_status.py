"""A deck that cannot be solved among good ones in a batch: its status says so, and every other deck of
the batch is solved, whichever worker it shares.

Nine decks on four workers, the second one without constraints: it shares its worker with the sixth. Sizes on both
sides of the dense inverse's (400 nodes, C3D20: 400 corners) and of the persistent launch's.

Tolerance: displacements against the oracle's FP64 direct solution, 1e-8 (the mixed solver's bound)."""
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


def _without_constraints(text):
    out, skip = [], False
    for line in text.split("\n"):
        skip = line.upper().startswith("*BOUNDARY") or (skip and not line.startswith("*"))
        if not skip:
            out.append(line)
    return "\n".join(out)


def _text(npe, cells):
    lengths = tuple(float(c) for c in cells)
    mesh = decks.tet_box(*cells, *lengths) if npe == 4 else decks.hex20_box(*cells, *lengths)
    return decks.write_deck(decks.DeckSpec(mesh, [(2.1e5, 0.3, None)], load_total=(100.0, 50.0, -30.0)))


@pytest.mark.parametrize("npe,cells", [(4, (3, 3, 6)), (4, (6, 6, 14)), (20, (1, 1, 3)), (20, (3, 3, 9)), (20, (5, 6, 11))])
def test_one_unconstrained_deck(ctx, npe, cells):
    good = _text(npe, cells)
    ref = static_step.Runner(inp.parse_inp_text(good)).run().displacements
    texts = [good] * 9
    texts[1] = _without_constraints(good)
    projects, states = [], []
    for text in texts:
        p = fx.Project.from_inp_text(text, ctx)
        states.append(fx.SolutionState(p.num_dofs, p.num_nodes))
        states[-1].initialize(p)
        projects.append(p)
    status, _ = fx.batch_solve(ctx, projects)
    u = [st.displacements for st in states]
    for p in projects:
        p.close()
    assert status.tolist() == [0, 11] + [0] * 7  # FX_NUMERICAL
    for k, v in enumerate(u):
        if k != 1:
            assert float(np.linalg.norm(v - ref) / np.linalg.norm(ref)) <= 1e-8, k
