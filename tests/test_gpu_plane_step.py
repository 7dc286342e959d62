"""Plane form of the one-kernel many-source step against the two-kernel step: the same arithmetic in the same order, so
the same bits, for every variant, with sources at interior dofs (whose elements update them) and elsewhere, on ragged
element counts, and for numberings whose interior dofs are scattered or shared between elements."""
import numpy as np
import pytest

from adjoint_case import build_case
from conftest import load_golden
from montjoie_gb300 import mesh as M
from montjoie_gb300.leapfrog import BatchLeapFrog
from montjoie_gb300.operator import FemMatrixFreeOperator
from montjoie_gb300.problem import AcousticProblem

pytestmark = pytest.mark.gpu

# order, elements per tile, lanes, sources per thread, sources (whole passes, the last two several)
VARIANTS = [(2, 16, 2, 4, 8), (2, 8, 4, 4, 32), (2, 4, 8, 4, 32), (3, 4, 8, 2, 16),
            (3, 2, 16, 2, 64), (3, 1, 32, 2, 64), (4, 4, 8, 1, 24), (4, 4, 8, 2, 16), (4, 2, 16, 2, 96),
            (4, 1, 32, 2, 64), (5, 2, 16, 1, 16), (5, 1, 32, 1, 32), (6, 4, 8, 1, 8), (6, 2, 16, 1, 48),
            (6, 1, 32, 1, 32)]


def _sources(rng, n_dof, S):
    idx = np.concatenate([rng.choice(n_dof, size=min(n_dof, 40), replace=False) for _ in range(S)])
    rhs = np.repeat(np.arange(S), min(n_dof, 40))
    return idx, rhs, rng.uniform(-1, 1, idx.size)


def _equal_to_two_kernels(make, variant):
    a, b = make(), make()
    a.set_step_variant(*variant)
    b.set_fused(False)
    for k, graph in ((3, False), (40, True), (2, False)):
        a.advance(k, graph=graph)
        b.advance(k, graph=graph)
        for x, y in zip(a.state(), b.state()):
            assert np.array_equal(x, y)
    assert np.abs(a.state()[0]).max() > 0
    a.close()
    b.close()


@pytest.mark.parametrize("order,E,LB,V,S", VARIANTS)
@pytest.mark.parametrize("cells", [1, 3, 7])
def test_every_plane_variant_equals_two_kernel_step(order, E, LB, V, S, cells):
    m = M.perturbed_cube(cells, seed=cells, amplitude=0.05, kind="random", c_mode="element")
    pb = AcousticProblem(m, M.AcousticSetup(order=order, src_radius=0.4), defer_time=True)
    op = pb.operator("fp32")
    rng = np.random.default_rng(order + S)
    src = _sources(rng, pb.n_dof, S)
    u0 = rng.uniform(-1, 1, (pb.n_dof, S))

    def make():
        b = BatchLeapFrog(op, 1e-3 / cells, S, pb.mass, None, *src, np.linspace(-1, 1, 30))
        b.init(u0)
        return b

    _equal_to_two_kernels(make, (E, LB, V))
    op.close()


@pytest.mark.parametrize("numbering", ["scattered", "shared"])
def test_numberings_without_interior_blocks(numbering):
    g = load_golden("cube3_q4")
    n_dof, S = g["massD"].size, 16
    nodle, mass = np.array(g["nodle"]), np.array(g["massD"])
    rng = np.random.default_rng(3)
    if numbering == "scattered":
        perm = rng.permutation(n_dof)
        nodle = perm[nodle]
        mass[perm] = g["massD"]
    else:  # one interior point of the second element on the first one's dof: that dof has two contributions
        el, q = nodle.reshape(-1, 125), 2 * 25 + 2 * 5 + 2
        gone = el[1, q]
        el[1, q] = el[0, q]
        nodle, mass, n_dof = el - (el > gone), np.delete(mass, gone), n_dof - 1  # no dof without an element
    op = FemMatrixFreeOperator(4, nodle.astype(np.int32), g["bh"], n_dof, "fp32", gradphi=g["gradphi"])
    src = _sources(rng, n_dof, S)
    u0 = rng.uniform(-1, 1, (n_dof, S))

    def make():
        b = BatchLeapFrog(op, float(g["dt"]), S, mass, None, *src, g["pulse"])
        b.init(u0)
        return b

    _equal_to_two_kernels(make, (4, 8, 2))
    op.close()


@pytest.mark.parametrize("variant,S", [((4, 8, 1), 8), ((4, 8, 2), 16), ((2, 16, 2), 32), ((1, 32, 2), 64)])
def test_gradient_term_equals_two_kernel_form(variant, S):
    from test_gpu_adjoint import make_model
    case = build_case(S=S, nsteps=40)
    ref = make_model(case, checkpoint_every=7)
    ref.batch.set_fused(False)
    J0, g0 = ref.loss_and_grad(case["c0"], case["data"])
    ref.close()
    for kw in (dict(checkpoint_every=7), dict(snapshots=3)):
        m = make_model(case, **kw)
        m.batch.set_step_variant(*variant)
        J, grad = m.loss_and_grad(case["c0"], case["data"])
        m.close()
        assert J == J0 and np.array_equal(grad, g0), kw
