"""The error of an element that is wrong in two ways: missing elastic constants are reported before a singular
Jacobian, as the element's material is looked up first."""
import pytest

import ferrix_b200 as fx
from ferrix_b200 import decks

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("elastic,kind", [(False, "InvalidModelState"), (True, "NumericalError")])
def test_flat_element(elastic, kind):
    text = decks.c3d4_cantilever(1, 1, 2)
    out, node = [], False
    for line in text.split("\n"):  # every node moved into one plane
        if line.startswith("*"):
            node = line.strip() == "*Node"
        elif node:
            n, x, y, z = line.split(",")
            line = f"{n},{x},{y}, 0.0"
        out.append(line)
    text = "\n".join(out)
    if not elastic:
        a = text.index("*Elastic")
        text = text[:a] + text[text.index("*", a + 1):]
    ctx = fx.Context(0)
    p = fx.Project.from_inp_text(text, ctx)
    st = fx.SolutionState(p.num_dofs, p.num_nodes)
    st.initialize(p)
    with pytest.raises(fx.FerrixError) as e:
        p.assemble_csr()
    p.close()
    ctx.close()
    assert e.value.kind == kind
