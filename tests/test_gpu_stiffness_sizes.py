"""Element stiffness at the element counts where the kernels' work splits end (C3D4: 64 elements to a CTA,
written out together; C3D20: a warp per element, four to a CTA), constant and temperature-dependent
constants, against the oracle's assembly.

Tolerance: 1e-12 relative to the largest entry in FP64, 2e-6 in FP32, as the other stiffness parity tests."""
import dataclasses

import numpy as np
import pytest

import ferrix_b200 as fx
from ferrix_b200 import decks
from oracle import elem, inp

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = fx.Context(0)
    yield c
    c.close()


def _spec(npe, n):
    if npe == 20:
        return decks.c3d20_box_spec(1, 1, n, lengths=(1.0, 1.1, 0.9 * n))
    spec = decks.c3d4_cantilever_spec(1, 2, (n + 11) // 12)  # 12 tets per layer
    spec.mesh.conn = spec.mesh.conn[:n]
    used = np.unique(spec.mesh.conn)
    index = -np.ones(len(spec.mesh.xyz), dtype=np.int64)
    index[used] = np.arange(len(used))
    return dataclasses.replace(spec, mesh=dataclasses.replace(
        spec.mesh, xyz=spec.mesh.xyz[used], conn=index[spec.mesh.conn], lattice=spec.mesh.lattice[used]))


@pytest.mark.parametrize("tdep", [False, True])
@pytest.mark.parametrize("npe,n", [(4, 1), (4, 63), (4, 64), (4, 65), (4, 130), (20, 1), (20, 3), (20, 4), (20, 5)])
def test_stiffness(ctx, npe, n, tdep):
    spec = _spec(npe, n)
    if tdep:
        spec = dataclasses.replace(spec, materials=[(2.1e5, 0.3, 20.0), (1.9e5, 0.32, 220.0)],
                                   init_temp=20.0 + 150.0 * spec.mesh.xyz[:, 2] / spec.mesh.xyz[:, 2].max())
    text = decks.write_deck(spec)
    m = inp.model_arrays(inp.parse_inp_text(text))
    tc = np.zeros(len(spec.mesh.xyz)) if spec.init_temp is None else spec.init_temp
    u = 1e-3 * np.random.default_rng(n).normal(size=3 * len(spec.mesh.xyz))
    K, md = elem.assemble(m, u, tc)
    K = K.toarray()
    p = fx.Project.from_inp_text(text, ctx)
    st = fx.SolutionState(p.num_dofs, p.num_nodes)
    st.initialize(p)
    for prec, tol in ((fx.PREC_FP64, 1e-12), (fx.PREC_MIXED, 2e-6)):
        ip, ind, dat, maxdiag = p.assemble_csr(u, prec)
        A = np.zeros_like(K)
        A[np.repeat(np.arange(len(ip) - 1), np.diff(ip)), ind] = dat
        assert np.abs(A - K).max() <= tol * np.abs(K).max()
        assert abs(maxdiag - md) <= tol * md
    p.close()
