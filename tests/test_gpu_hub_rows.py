"""Row-wise transfer products around the longest row they hold: a ball of C3D4 elements about one node whose row
meets from some 100 to over 384 aggregates, the last by the sorted pair lists.

Tolerance: 1e-10 against the oracle's FP64 direct solution at a residual target of 1e-11, as the other tests
of the multigrid's sizes."""
import numpy as np
import pytest

import ferrix_b200 as fx
from ferrix_b200 import decks
from oracle import inp, static_step

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ball():
    from scipy.spatial import ConvexHull
    k = np.arange(1500)
    z = 1.0 - (2.0 * k + 1.0) / len(k)
    phi = k * np.pi * (3.0 - np.sqrt(5.0))
    r = np.sqrt(1.0 - z * z)
    sphere = np.stack([r * np.cos(phi), r * np.sin(phi), z], axis=1)
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
    return text, static_step.Runner(inp.parse_inp_text(text)).run().displacements


@pytest.mark.parametrize("nodes", [1, 3, 4, 5, 7, 10, 15])
def test_hub_rows(ball, nodes):
    text, ref = ball
    ctx = fx.Context(0)
    p = fx.Project.from_inp_text(text, ctx)
    st = fx.SolutionState(p.num_dofs, p.num_nodes)
    st.initialize(p)
    stats = p.steps[0].solve(1, p, st, opts=fx.solve_opts(precision=fx.PREC_FP64, rtol=1e-11, amg_aggregate_nodes=nodes,
                                                          amg_persistent_max_dof=-1))
    err = float(np.linalg.norm(st.displacements - ref) / np.linalg.norm(ref))
    p.close()
    ctx.close()
    assert err <= 1e-10, stats


def test_setup_beside_a_hub():
    """A node whose row reaches some 350 aggregates must not fill the coarse matrix between them: the set-up of a box with a
    ball of 1,800 nodes about one node beside it takes at most 12 times the box's own (some 40 times
    with that row smoothed). The least of four solves each."""
    from scipy.spatial import ConvexHull

    def setup_ms(mesh):
        ctx = fx.Context(0)
        p = fx.Project.from_arrays(**decks.deck_arrays(decks.DeckSpec(mesh, [(2.0e5, 0.3, None)],
                                                                      load_total=(100.0, 50.0, -200.0))), ctx=ctx)
        st = fx.SolutionState(p.num_dofs, p.num_nodes)
        ms = []
        for _ in range(4):
            st.initialize(p)
            ms.append(p.steps[0].solve(1, p, st)["amg_setup_ms"])
        p.close()
        ctx.close()
        return min(ms)

    box = decks.tet_box(16, 16, 40, 16.0, 16.0, 40.0)
    k = np.arange(1800)
    z = 1.0 - (2.0 * k + 1.0) / len(k)
    phi = k * np.pi * (3.0 - np.sqrt(5.0))
    r = np.sqrt(1.0 - z * z)
    sphere = np.stack([r * np.cos(phi), r * np.sin(phi), z], axis=1)
    tri = ConvexHull(sphere).simplices
    xyz = 12.0 * np.concatenate([[[0.0, 0.0, 0.0]], sphere])
    conn = np.concatenate([np.zeros((len(tri), 1), dtype=np.int64), tri + 1], axis=1)
    v = np.einsum("ij,ij->i", np.cross(xyz[conn[:, 1]], xyz[conn[:, 2]]), xyz[conn[:, 3]])
    conn[v < 0, 1], conn[v < 0, 2] = conn[v < 0, 2].copy(), conn[v < 0, 1].copy()
    lattice = np.ones((len(xyz), 3), dtype=np.int64)
    lattice[xyz[:, 2] < -8.4] = 0  # clamped cap
    mesh = decks.BoxMesh(np.concatenate([box.xyz, xyz + [50.0, 8.0, 20.0]]), np.concatenate([box.conn, conn + len(box.xyz)]),
                         4, np.concatenate([box.lattice, lattice]), box.dims, box.lengths)
    assert setup_ms(mesh) <= 12.0 * setup_ms(box)
