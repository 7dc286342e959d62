"""FP32 line-owner element kernel (orders 7 and 8) against the compact layout: the same arithmetic in the same order,
so the same bits, at ragged element counts (less than a tile, one over a grid's worth of tiles)."""
import numpy as np
import pytest

from montjoie_gb300 import mesh as M
from montjoie_gb300.problem import AcousticProblem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", [7, 8])
@pytest.mark.parametrize("cells", [1, 2, 3, 11])
def test_bitwise_the_compact_layout(order, cells):
    m = M.perturbed_cube(cells, seed=cells, amplitude=0.05, kind="random", c_mode="element")
    pb = AcousticProblem(m, M.AcousticSetup(order=order, src_radius=0.4), defer_time=True)
    op = pb.operator("fp32")
    x = np.random.default_rng(order).uniform(-1, 1, pb.n_dof)
    x[::97] = 0.0
    assert op.tuning()["layout"] == "line_owner"
    a, b = np.zeros(pb.n_dof), np.zeros(pb.n_dof)
    op.MltVector(x, a)
    op.set_variant(2, 0)
    op.MltVector(x, b)
    assert np.array_equal(a, b)
    op.close()
