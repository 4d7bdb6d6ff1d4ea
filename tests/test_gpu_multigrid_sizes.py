"""The multigrid's kernels at the sizes where they can go wrong.

Coarsest-level inverse, transfers and aggregate factorisation: the aggregate size asked for sets
the coarsest size (one aggregate: 6 DOF, a partial panel; both sides of a 32-pivot panel and of
a 64-row tile; up to the largest dense level), the entries per transfer row and the rows per
aggregate (beyond 256 its factorisation leaves shared memory). Corner level: C3D20 decks down to
one element, with distorted mid nodes, beside C3D4 elements on the same corners, and with
a C3D4 element on a mid node (where the hierarchy does without the corner level).
Every solve must meet the oracle's FP64 direct solution.

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


def _solve(ctx, text, **kw):
    p = fx.Project.from_inp_text(text, ctx)
    st = fx.SolutionState(p.num_dofs, p.num_nodes)
    st.initialize(p)
    stats = p.steps[0].solve(1, p, st, opts=fx.solve_opts(rtol=1e-11, **kw))
    u = st.displacements
    p.close()
    return u, stats


def _with_tets(nodes_of_face):
    """A C3D20 box with C3D4 elements on its top: apex nodes above triples of its nodes."""
    spec = decks.c3d20_box_spec(2, 2, 4, lengths=(2.0, 2.0, 4.0))
    m = spec.mesh
    lines, extra, nid, eid = decks.write_deck(spec).split("\n"), [], len(m.xyz) + 1, len(m.conn) + 1
    nodes = []
    for tri in nodes_of_face(m):
        c = m.xyz[list(tri)].mean(axis=0) + [0.0, 0.0, 0.6]
        nodes.append(f"{nid}, {c[0]!r}, {c[1]!r}, {c[2]!r}".replace("np.float64(", "").replace(")", ""))
        extra.append(f"{eid}, " + ", ".join(str(int(i) + 1) for i in tri) + f", {nid}")
        nid, eid = nid + 1, eid + 1
    at = next(i for i, line in enumerate(lines) if line.startswith("*Element"))
    lines[at:at] = nodes
    at = next(i for i, line in enumerate(lines) if line.startswith("*Nset"))
    return "\n".join(lines[:at] + ["*Element, Type=C3D4, Elset=Solid"] + extra + lines[at:])


def _corner_tris(m):  # two triangles of the top face's first quad, corners only
    c = m.conn[-1]
    return [(c[4], c[5], c[6]), (c[4], c[6], c[7])]


def _mid_tri(m):  # a triangle with a mid-edge node of the top face
    c = m.conn[-1]
    return [(c[4], c[5], c[14])]


CORNER = {
    "one_element": lambda: decks.c3d20_box(1, 1, 1, lengths=(1.0, 1.0, 1.0)),
    "column": lambda: decks.c3d20_box(1, 1, 9, lengths=(1.0, 1.0, 9.0)),
    "slender": lambda: decks.c3d20_box(2, 3, 33, lengths=(2.0, 3.0, 33.0)),
    "block": lambda: decks.c3d20_box(5, 6, 7, lengths=(5.0, 6.0, 7.0)),
    "with_tets": lambda: _with_tets(_corner_tris),
    "tet_on_mid_node": lambda: _with_tets(_mid_tri),
}


@pytest.mark.parametrize("prec", [fx.PREC_FP64, fx.PREC_MIXED])
@pytest.mark.parametrize("case", list(CORNER))
def test_corner_level(ctx, case, prec):
    text = CORNER[case]()
    ref = static_step.Runner(inp.parse_inp_text(text)).run().displacements
    per_step, s1 = _solve(ctx, text, precision=prec, amg_persistent_max_dof=-1)
    cluster, s2 = _solve(ctx, text, precision=prec, amg_persistent_max_dof=100000)
    for u in (per_step, cluster):
        assert float(np.linalg.norm(u - ref) / np.linalg.norm(ref)) <= 1e-10, (s1, s2)


@pytest.mark.parametrize("persistent", [-1, 100000])
@pytest.mark.parametrize("npe", [4, 20])
def test_kept_hierarchy_over_newton_iterations(ctx, npe, persistent):
    """An NLGEOM step with displacements of up to a seventh of the beam's length (the C3D20 beam, which
    is softer, at a load for which the reference's Newton iteration converges): the hierarchy kept from
    an increment's first tangent preconditions ever different ones; the increments must end where the
    oracle's do (the NLGEOM bound of the other parity tests, 1e-8)."""
    spec = decks.c3d4_nlgeom_beam_spec(10, 2, 2, tip_load=6.0e4 if npe == 4 else 1.5e4, increments=3)
    if npe == 20:
        spec.mesh = decks.hex20_box(6, 1, 1, 50.0, 10.0, 10.0, jitter=0.05, seed=3)
        spec.init_temp = 20.0 + 200.0 * spec.mesh.xyz[:, 0] / 50.0
    text = decks.write_deck(spec)
    ref = static_step.Runner(inp.parse_inp_text(text)).run().displacements
    u, stats = _solve(ctx, text, amg_persistent_max_dof=persistent)
    assert stats["linear_solves"] > 2 * stats["increments"]
    assert float(np.linalg.norm(u - ref) / np.linalg.norm(ref)) <= 1e-8, stats


@pytest.mark.parametrize("prec", [fx.PREC_FP64, fx.PREC_MIXED])
@pytest.mark.parametrize("npe,cells", [(4, (1, 1, 1)), (4, (2, 1, 3)), (4, (3, 3, 23)), (4, (3, 3, 24)), (4, (3, 3, 25)),
                                       (20, (3, 3, 24)), (20, (3, 3, 25))])
def test_dense_planar_level(ctx, npe, cells, prec):
    """Small systems whose fine level (C3D4) or corner level (C3D20) takes the dense inverse itself, up to
    its largest size (400 nodes or corners) and just beyond."""
    lengths = tuple(float(c) for c in cells)
    spec = decks.c3d20_box_spec(*cells, lengths=lengths)
    if npe == 4:
        spec.mesh = decks.tet_box(*cells, *lengths)
    text = decks.write_deck(spec)
    ref = static_step.Runner(inp.parse_inp_text(text)).run().displacements
    u, stats = _solve(ctx, text, precision=prec)
    # FP64: 1e-10 as elsewhere; these slender columns leave up to 1e-9 at the mixed solver's residual
    assert float(np.linalg.norm(u - ref) / np.linalg.norm(ref)) <= (1e-10 if prec == fx.PREC_FP64 else 1e-8), stats


@pytest.mark.parametrize("nodes", [0, 2])
def test_hub_node(ctx, nodes):
    """A ball of C3D4 elements around one node: with two nodes per aggregate, that node's row reaches more
    aggregates than the row-wise products hold, which then go by sorted operand pairs."""
    k = np.arange(1500)
    z = 1.0 - (2.0 * k + 1.0) / len(k)
    phi = k * np.pi * (3.0 - np.sqrt(5.0))
    r = np.sqrt(1.0 - z * z)
    sphere = np.stack([r * np.cos(phi), r * np.sin(phi), z], axis=1)
    from scipy.spatial import ConvexHull
    tri = ConvexHull(sphere).simplices
    xyz = np.concatenate([[[0.0, 0.0, 0.0]], sphere])
    conn = np.concatenate([np.zeros((len(tri), 1), dtype=np.int64), tri + 1], axis=1)
    v = np.einsum("ij,ij->i", np.cross(xyz[conn[:, 1]], xyz[conn[:, 2]]), xyz[conn[:, 3]])
    conn[v < 0, 1], conn[v < 0, 2] = conn[v < 0, 2].copy(), conn[v < 0, 1].copy()
    lattice = np.ones((len(xyz), 3), dtype=np.int64)
    lattice[xyz[:, 2] < -0.7] = 0  # clamped cap
    lattice[xyz[:, 2] > 0.7] = 2   # loaded cap
    mesh = decks.BoxMesh(xyz, conn, 4, lattice, (2, 2, 2), (2.0, 2.0, 2.0))
    text = decks.write_deck(decks.DeckSpec(mesh, [(2.0e5, 0.3, None)], load_total=(100.0, 50.0, -200.0)))
    ref = static_step.Runner(inp.parse_inp_text(text)).run().displacements
    u, stats = _solve(ctx, text, precision=fx.PREC_FP64, amg_aggregate_nodes=nodes, amg_persistent_max_dof=-1)
    assert float(np.linalg.norm(u - ref) / np.linalg.norm(ref)) <= 1e-10, stats


@pytest.mark.parametrize("prec", [fx.PREC_FP64, fx.PREC_MIXED])
@pytest.mark.parametrize("cycle", [0, 1])
@pytest.mark.parametrize("npe,cells,nodes", [(4, (4, 5, 9), 0), (4, (6, 6, 14), 4), (4, (6, 6, 14), 40),
                                             (20, (2, 2, 6), 0), (20, (5, 5, 12), 4)])
def test_chained_launches(ctx, npe, cells, nodes, cycle, prec):
    """Each kernel of the iteration may begin before the one ahead has ended: replayed from graphs and
    launched one by one, with one, two and more levels under the cycle, the solve gives the same bits."""
    spec = decks.c3d20_box_spec(*cells, lengths=tuple(float(c) for c in cells))
    if npe == 4:
        spec.mesh = decks.tet_box(*cells, *(float(c) for c in cells))
    text = decks.write_deck(spec)
    ref = static_step.Runner(inp.parse_inp_text(text)).run().displacements
    runs = [_solve(ctx, text, precision=prec, amg_cycle=cycle, amg_aggregate_nodes=nodes, use_graphs=g,
                   amg_persistent_max_dof=-1) for g in (1, 0, 1, 1)]
    for u, stats in runs:
        assert np.array_equal(u, runs[0][0]) and stats["pcg_iterations"] == runs[0][1]["pcg_iterations"]
        assert float(np.linalg.norm(u - ref) / np.linalg.norm(ref)) <= (1e-10 if prec == fx.PREC_FP64 else 1e-8), stats
