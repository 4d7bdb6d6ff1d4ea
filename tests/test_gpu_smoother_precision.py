"""Mixed precision on systems where a stiff part hangs on a soft one: by default its fine-level smoother keeps
enough digits, so that the mixed solve takes about the FP64 solve's iterations (a third more and four, the
spread that FP32 smoothing leaves) and is not given up."""
import pytest

import ferrix_b200 as fx
from test_gpu_dense_level import solve, two_materials

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = fx.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("soft", [2.0, 20.0, 200.0])
@pytest.mark.parametrize("npe,cells", [(20, (2, 2, 10)), (20, (6, 6, 24)), (4, (10, 10, 24))])
def test_stiff_on_soft(ctx, npe, cells, soft):
    text = two_materials(npe, cells, tuple(float(c) for c in cells), soft, 2.0e5)  # the soft half is clamped
    its = [solve(ctx, text, precision=prec)[1]["pcg_iterations"] for prec in (fx.PREC_FP64, fx.PREC_MIXED)]
    assert its[1] <= its[0] + its[0] // 3 + 4, its
