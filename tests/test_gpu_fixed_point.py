"""Fixed-point form of the FP64 element kernel (layout "fixed_point", the default of FP64 operators) against the
FP64-pipe kernel (``set_variant(E, 0)``), the oracle's element loop and its own scaling invariance."""
import numpy as np
import pytest

from montjoie_gb300 import mesh as M
from montjoie_gb300.operator import FemMatrixFreeOperator
from montjoie_gb300.problem import AcousticProblem, derivative_matrix, gauss_lobatto

pytestmark = pytest.mark.gpu

FP64_PIPE_TILE = {1: 30, 2: 12, 3: 8, 4: 4, 5: 3, 6: 2, 7: 2, 8: 1}
# A product of n terms in FP64 rounds by at most (n + 1) u of its absolute sum (u = 2^-53); two contractions and the
# factor row are 2 (n + 1) + 4 <= 24 roundings per direction, and for a random field the absolute sums are below 20
# times the result (in norm): 24 u x 20 = 5.3e-14.  Either kernel may be that far off.
TOL = 2 * 5.3e-14


def build(order, cells, gradphi=None, seed=1):
    m = M.perturbed_cube(cells, seed=seed, amplitude=0.05, kind="random", c_mode="element")
    pb = AcousticProblem(m, M.AcousticSetup(order=order, src_radius=0.4), defer_time=True)
    op = FemMatrixFreeOperator(order, pb.nodle, pb.factors, pb.n_dof, "fp64", gradphi=gradphi)
    return pb, op


def product(op, x):
    y = np.zeros(op.n_dof)
    op.MltVector(x, y)
    return y


def both(op, order, x):
    """(fixed point, FP64 pipe) products; the operator is left in the FP64-pipe form."""
    assert op.tuning()["layout"] == "fixed_point"
    a = product(op, x)
    op.set_variant(FP64_PIPE_TILE[order], 0)
    return a, product(op, x)


@pytest.mark.parametrize("order", range(1, 9))
@pytest.mark.parametrize("cells", [1, 2, 5])
def test_random_field(order, cells):
    pb, op = build(order, cells)
    x = np.random.default_rng(order).uniform(-1, 1, pb.n_dof)
    a, b = both(op, order, x)
    assert np.linalg.norm(a - b) <= TOL * np.linalg.norm(b)


@pytest.mark.parametrize("order", [1, 4, 7, 8])
def test_matrix_that_is_not_antisymmetric(order):
    G = derivative_matrix(gauss_lobatto(order)[0])
    G = G + 1e-3 * np.random.default_rng(0).uniform(-1, 1, G.shape)
    pb, op = build(order, 3, gradphi=np.ascontiguousarray(G))
    x = np.random.default_rng(order).uniform(-1, 1, pb.n_dof)
    a, b = both(op, order, x)
    assert np.linalg.norm(a - b) <= TOL * np.linalg.norm(b)


@pytest.mark.parametrize("order", [2, 4, 8])
def test_scaling_by_powers_of_two_is_exact(order):
    pb, op = build(order, 3)
    x = np.random.default_rng(order).uniform(-1, 1, pb.n_dof)
    y = product(op, x)
    for k in (-700, -40, 1, 30, 700):
        assert np.array_equal(product(op, np.ldexp(x, k)), np.ldexp(y, k))
    assert np.array_equal(product(op, np.zeros(pb.n_dof)), np.zeros(pb.n_dof))


@pytest.mark.parametrize("order", [1, 4, 8])
@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf, 1e-310, 1e-290, 1e300])
def test_values_out_of_range(order, value):
    """One such value (the rest of the field scaled with a finite one): the same non-finite entries as the FP64-pipe
    kernel, and its values elsewhere."""
    pb, op = build(order, 3)
    rng = np.random.default_rng(order)
    x = rng.uniform(-1, 1, pb.n_dof)
    if np.isfinite(value):
        x *= value
    x[int(rng.integers(pb.n_dof))] = value
    with np.errstate(all="ignore"):
        a, b = both(op, order, x)
    assert np.array_equal(np.isnan(a), np.isnan(b)) and np.array_equal(np.isinf(a), np.isinf(b))
    f = np.isfinite(b)
    s = np.abs(b[f]).max()  # scaled first: sums of squares would leave the range
    assert np.linalg.norm((a[f] - b[f]) / s) <= TOL * np.linalg.norm(b[f] / s)


@pytest.mark.parametrize("order", [3, 4])
def test_element_scale_reaches_the_fixed_point_factors(order):
    pb, op = build(order, 3)
    rng = np.random.default_rng(order)
    x, sc = rng.uniform(-1, 1, pb.n_dof), rng.uniform(0, 4, op.n_elt)
    sc[::5] = 0.0
    before = product(op, x)
    op.set_element_scale(sc)
    a, b = both(op, order, x)
    assert np.linalg.norm(a - before) > 0.1 * np.linalg.norm(before)
    assert np.linalg.norm(a - b) <= TOL * np.linalg.norm(b)
