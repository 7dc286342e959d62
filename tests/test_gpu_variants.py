"""Every compiled tile size of the fixed-point (FP64, both forms of the derivative matrix) and line-owner (FP32) element
kernels, forced, on ragged meshes that give each CTA several tiles: the same bits whatever the tile."""
import numpy as np
import pytest

from montjoie_gb300 import _lib, mesh as M
from montjoie_gb300.operator import FemMatrixFreeOperator
from montjoie_gb300.problem import AcousticProblem, derivative_matrix, gauss_lobatto

pytestmark = pytest.mark.gpu

TILES = {1: (30, 60), 2: (12, 24), 3: (8, 16), 4: (4, 5, 8, 10), 5: (3, 4, 6), 6: (2, 3, 4, 5), 7: (2, 3, 4), 8: (1, 2, 3)}
CELLS = {1: 57, 2: 37, 3: 29, 4: 23, 5: 17, 6: 15, 7: 13, 8: 11}
# both kernels within 24 roundings of absolute sums below 20 times the result (random field), as for one FP64 product
TOL = 2 * 24 * 2.0 ** -53 * 20


def _problem(order):
    m = M.perturbed_cube(CELLS[order], seed=order, amplitude=0.05, kind="random", c_mode="element")
    return AcousticProblem(m, M.AcousticSetup(order=order, src_radius=0.4), defer_time=True)


def _product(op, x):
    y = np.zeros(x.size)
    op.MltVector(x, y)
    return y


@pytest.mark.parametrize("order", range(1, 9))
@pytest.mark.parametrize("form", ["mirror", "general"])
def test_fixed_point_tiles(order, form):
    pb = _problem(order)
    G = derivative_matrix(gauss_lobatto(order)[0])
    G = 0.5 * (G - G[::-1, ::-1])
    if form == "general":
        G[0, -1] = np.nextafter(G[0, -1], 9.0)
    op = FemMatrixFreeOperator(order, pb.nodle, pb.factors, pb.n_dof, "fp64", gradphi=np.ascontiguousarray(G))
    rng = np.random.default_rng(order)
    x = np.sin(np.arange(pb.n_dof) * 0.1) + 0.2 * rng.uniform(-1, 1, pb.n_dof)
    x[rng.choice(pb.n_dof, 40)] *= 1e6  # elements in FP64 among the others
    t = op.tuning()
    assert t["layout"] == "fixed_point" and t["tile_elems"] in TILES[order]
    want = _product(op, x)
    for E in TILES[order]:
        op.set_variant(E, 5)
        assert op.tuning()["layout"] == "fixed_point" and op.tuning()["tile_elems"] == E
        assert np.array_equal(_product(op, x), want), E
    op.set_variant(TILES[order][0], 0)
    pipe = _product(op, x)
    assert np.linalg.norm(want - pipe) <= TOL * np.linalg.norm(pipe)
    op.set_variant(t["tile_elems"], 5)  # back to the default kernel
    assert np.array_equal(_product(op, x), want)
    op.close()


@pytest.mark.parametrize("order", [7, 8])
def test_line_owner_tiles(order):
    pb = _problem(order)
    op = pb.operator("fp32")
    x = np.random.default_rng(order).uniform(-1, 1, pb.n_dof)
    op.set_variant(2, 0)
    want = _product(op, x)
    for E in (1, 2):
        op.set_variant(E, 6)
        assert op.tuning()["layout"] == "line_owner" and op.tuning()["tile_elems"] == E
        assert np.array_equal(_product(op, x), want), E
    op.close()


def test_layouts_that_an_operator_does_not_have():
    pb = _problem(8)
    for precision, layout, tile in (("fp32", 5, 1), ("fp64", 6, 1), ("fp32", 6, 3), ("fp32", 7, 1), ("fp64", 5, 7)):
        op = pb.operator(precision)
        with pytest.raises(_lib.MontjoieError) as e:
            op.set_variant(tile, layout)
        assert e.value.code == _lib.MJ_ERR_ARG
        op.close()
        pb._op = None
