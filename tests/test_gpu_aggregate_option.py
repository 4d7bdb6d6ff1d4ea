"""An aggregate size that the caller asks for is used, also where the dense inverse would cover the system,
and counts the mesh's nodes: the level count shows the aggregated level, and the coarsest level's inverse is tested at the sizes
around its 32-pivot panels and 64-row tiles on a system above the dense size.

Tolerance: 1e-10 against the oracle's FP64 direct solution at a residual target of 1e-11, as the other
tests of the multigrid's sizes."""
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
def solved():
    out = {}
    for name, text in (("small", decks.c3d4_cantilever(4, 5, 9)),   # 300 nodes
                       ("large", decks.c3d4_cantilever(5, 6, 11)),  # 504 nodes
                       ("corners", decks.c3d20_box(2, 2, 6, lengths=(2.0, 2.0, 6.0)))):  # 63 corners
        out[name] = text, static_step.Runner(inp.parse_inp_text(text)).run().displacements
    return out


def _solve(ctx, solved, name, **kw):
    text, ref = solved[name]
    p = fx.Project.from_inp_text(text, ctx)
    st = fx.SolutionState(p.num_dofs, p.num_nodes)
    st.initialize(p)
    stats = p.steps[0].solve(1, p, st, opts=fx.solve_opts(precision=fx.PREC_FP64, rtol=1e-11, **kw))
    err = float(np.linalg.norm(st.displacements - ref) / np.linalg.norm(ref))
    p.close()
    assert err <= 1e-10, (err, stats)
    return stats["amg_levels"]


@pytest.mark.parametrize("persistent", [0, -1])
def test_small_systems(ctx, solved, persistent):
    for name, dense in (("small", 1), ("corners", 2)):
        assert _solve(ctx, solved, name, amg_persistent_max_dof=persistent) == dense
        assert _solve(ctx, solved, name, amg_aggregate_nodes=12, amg_persistent_max_dof=persistent) == dense + 1


@pytest.mark.parametrize("nodes", [3, 4, 5, 8, 12, 20, 33, 45, 47, 50, 75, 120, 300, 5000])
def test_coarsest_inverse_sizes(ctx, solved, nodes):
    assert _solve(ctx, solved, "large", amg_aggregate_nodes=nodes, amg_persistent_max_dof=-1) == 2


@pytest.mark.parametrize("nodes", [4, 8, 16, 24])
def test_unsmoothed_transfers(ctx, nodes):
    """Above 5,000 rows small aggregates take the tentative transfer itself (24: the smoothed one)."""
    text = decks.c3d4_cantilever(13, 13, 28)  # 5,684 nodes
    ref = static_step.Runner(inp.parse_inp_text(text)).run().displacements
    p = fx.Project.from_inp_text(text, ctx)
    st = fx.SolutionState(p.num_dofs, p.num_nodes)
    for prec, tol in ((fx.PREC_FP64, 1e-10), (fx.PREC_MIXED, 1e-8)):
        st.initialize(p)
        p.steps[0].solve(1, p, st, opts=fx.solve_opts(precision=prec, rtol=1e-11, amg_aggregate_nodes=nodes))
        assert float(np.linalg.norm(st.displacements - ref) / np.linalg.norm(ref)) <= tol
    p.close()


def test_unsmoothed_transfers_below_the_corners(ctx):
    """The same on a corner level of 5,400 corners, whose lower levels are smoothed: against the default hierarchy, 1e-8."""
    text = decks.c3d20_box(14, 14, 23, lengths=(14.0, 14.0, 23.0))
    p = fx.Project.from_inp_text(text, ctx)
    st = fx.SolutionState(p.num_dofs, p.num_nodes)
    u = []
    for nodes in (0, 16, 40):
        st.initialize(p)
        p.steps[0].solve(1, p, st, opts=fx.solve_opts(rtol=1e-11, amg_aggregate_nodes=nodes))
        u.append(st.displacements)
    p.close()
    for v in u[1:]:
        assert float(np.linalg.norm(v - u[0]) / np.linalg.norm(u[0])) <= 1e-8


def test_counts_mesh_nodes(ctx):
    """1,820 corners among 6,768 nodes: 16 nodes of the mesh per aggregate leave 408 aggregates, more than the dense
    inverse's 200 (one more level); 16 corners, or 64 nodes, leave 132."""
    text = decks.c3d20_box(6, 9, 25, lengths=(6.0, 9.0, 25.0))
    levels = []
    for nodes in (16, 64):
        p = fx.Project.from_inp_text(text, ctx)
        assert p.num_nodes == 6768
        st = fx.SolutionState(p.num_dofs, p.num_nodes)
        st.initialize(p)
        levels.append(p.steps[0].solve(1, p, st, opts=fx.solve_opts(amg_aggregate_nodes=nodes))["amg_levels"])
        p.close()
    assert levels == [4, 3]


def test_correction_scale(ctx):
    """Smoothed transfers take their corrections unscaled by default: asked for as 1.0 it is the same cycle."""
    text = decks.c3d4_cantilever(8, 8, 30)
    its = []
    for kw in ({}, dict(amg_overcorrect=1.0)):
        p = fx.Project.from_inp_text(text, ctx)
        st = fx.SolutionState(p.num_dofs, p.num_nodes)
        st.initialize(p)
        its.append(p.steps[0].solve(1, p, st, opts=fx.solve_opts(rtol=1e-10, **kw))["pcg_iterations"])
        p.close()
    assert its[0] == its[1]
