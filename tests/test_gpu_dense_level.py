"""The dense inverse of a small planar level (a C3D4 system of up to 400 nodes, or the corner level of a
C3D20 mesh of up to 400 corners), where it is the whole coarse solve or the whole preconditioner.

Two materials in one column, on both sides of the dense size: the inverse must cover the DOFs of the soft
one, however stiff the other and the constraints are. Against the oracle's FP64 direct solution.

Tolerance: 1e-8, the mixed solver's bound; the residual target is 1e-10 and the stiff end is clamped, so that the
conditioning of the system does not enter."""
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


def _ids(a):
    return "\n".join(", ".join(str(int(v) + 1) for v in a[i:i + 12]) for i in range(0, len(a), 12))


def two_materials(npe, cells, lengths, stiff, soft, jitter=0.05):
    """A column clamped at z = 0 whose lower and upper half have Young's moduli stiff and soft."""
    mesh = decks.tet_box(*cells, *lengths) if npe == 4 else decks.hex20_box(*cells, *lengths, jitter=jitter, seed=1)
    text = decks.write_deck(decks.DeckSpec(mesh, [(stiff, 0.3, None)], load_total=(1.0, 2.0, -1.0)))
    is_soft = mesh.xyz[mesh.conn].mean(axis=1)[:, 2] > lengths[2] / 2
    text = text.replace("*Elset, Elset=Vol\nSolid\n", "*Elset, Elset=Vol\n" + _ids(np.nonzero(~is_soft)[0]) +
                        "\n*Elset, Elset=Soft\n" + _ids(np.nonzero(is_soft)[0]) + "\n")
    return text.replace("*Solid section, Elset=Vol, Material=Mat\n", "*Material, Name=Mat2\n*Density\n7.8E-09\n"
                        f"*Elastic\n{soft!r}, 0.3\n*Solid section, Elset=Vol, Material=Mat\n"
                        "*Solid section, Elset=Soft, Material=Mat2\n")


def solve(ctx, text, **kw):
    p = fx.Project.from_inp_text(text, ctx)
    st = fx.SolutionState(p.num_dofs, p.num_nodes)
    st.initialize(p)
    try:
        stats = p.steps[0].solve(1, p, st, opts=fx.solve_opts(rtol=1e-10, max_iter=3000, **kw))
        return st.displacements, stats
    finally:
        p.close()


def error(text, u):
    ref = static_step.Runner(inp.parse_inp_text(text)).run().displacements
    return float(np.linalg.norm(u - ref) / np.linalg.norm(ref))


SIZES = [(4, (3, 3, 10), (3.0, 3.0, 10.0)), (4, (3, 3, 10), (3.0, 3.0, 2.0)), (4, (3, 3, 24), (3.0, 3.0, 24.0)),
         (4, (3, 3, 25), (3.0, 3.0, 25.0)), (20, (2, 2, 10), (2.0, 2.0, 10.0)), (20, (3, 3, 26), (3.0, 3.0, 26.0))]


@pytest.mark.parametrize("prec", [fx.PREC_FP64, fx.PREC_MIXED])
@pytest.mark.parametrize("contrast", [1e4, 1e5, 4e6, 1e8])
@pytest.mark.parametrize("npe,cells,lengths", SIZES)
def test_soft_on_stiff(ctx, npe, cells, lengths, contrast, prec):
    text = two_materials(npe, cells, lengths, 2.0e5, 2.0e5 / contrast)
    u, stats = solve(ctx, text, precision=prec)
    assert error(text, u) <= 1e-8, stats


@pytest.mark.parametrize("prec", [fx.PREC_FP64, fx.PREC_MIXED])
@pytest.mark.parametrize("contrast", [1e4, 1e5])
def test_coarse_operator_below_the_corners(ctx, contrast, prec):
    """A stiff plate on cells eight times wider than high and much softer: the coarse operator below the corner
    level has pivots as of a singular one, that below the nodes has not, and the system is solved.

    Tolerance: mean displacement of the loaded face, 1e-6: contrast x unit round-off = 1e-11, and at most 1e2 by the
    plate's lever on the pad."""
    text = two_materials(20, (6, 6, 24), (6.0, 6.0, 3.0), 2.0e5 / contrast, 2.0e5, jitter=0.0)
    u, _ = solve(ctx, text, precision=prec)
    ref = static_step.Runner(inp.parse_inp_text(text)).run().displacements
    mesh = decks.hex20_box(6, 6, 24, 6.0, 6.0, 3.0)
    top = decks.face_nodes(mesh, 2, 1)
    a, b = (v.reshape(-1, 3)[top].mean(axis=0) for v in (u, ref))
    assert np.linalg.norm(a - b) <= 1e-6 * np.linalg.norm(b)
