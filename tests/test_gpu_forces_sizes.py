"""C3D20 internal and thermal force at the element counts where the kernel's work split ends (one warp
per element, eight to a CTA), with constant and temperature-dependent constants and with a
separate configuration, against the oracle's element loops.

Tolerance: 1e-11 relative to the largest entry, as the other force parity tests."""
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


@pytest.mark.parametrize("tdep", [False, True])
@pytest.mark.parametrize("n", [1, 7, 8, 9, 17])
def test_c3d20_forces(ctx, n, tdep):
    spec = decks.c3d20_box_spec(1, 1, n, lengths=(1.0, 1.2, 0.9 * n))
    if tdep:
        spec = dataclasses.replace(spec, materials=[(2.1e5, 0.3, 20.0), (1.9e5, 0.32, 220.0)], expansion=(1.2e-5, 20.0),
                                   init_temp=20.0 + 150.0 * spec.mesh.xyz[:, 2] / spec.mesh.xyz[:, 2].max())
    text = decks.write_deck(spec)
    m = inp.model_arrays(inp.parse_inp_text(text))
    rng = np.random.default_rng(n)
    u, uc = (1e-3 * rng.normal(size=3 * len(spec.mesh.xyz)) for _ in range(2))
    ti = np.zeros(len(spec.mesh.xyz)) if spec.init_temp is None else spec.init_temp
    tc = ti + 40.0
    p = fx.Project.from_inp_text(text, ctx)
    st = fx.SolutionState(p.num_dofs, p.num_nodes)
    st.initialize(p)
    st.set_temperatures(t_cur=tc)
    for got, want in ((p.internal_force(u), elem.internal_force(m, u, None, ti, tc)),
                      (p.internal_force(u, uc), elem.internal_force(m, u, uc, ti, tc)),
                      (p.thermal_force(), elem.thermal_force(m, ti, tc))):
        assert np.abs(got - want).max() <= 1e-11 * max(np.abs(want).max(), 1e-300)
    p.close()
