"""Bulk-copy waits of the fixed-point and line-owner element kernels, the FP64 streaming gather and the plane form of the
many-source step, made to run out (instances compiled with a wait limit of 0): the call returns an error status after the
kernel's copies have landed, and the next call gives the same result as before."""
import numpy as np
import pytest

from conftest import load_golden
from montjoie_gb300 import _lib, mesh as M
from montjoie_gb300.leapfrog import BatchLeapFrog
from montjoie_gb300.operator import FemMatrixFreeOperator
from montjoie_gb300.problem import AcousticProblem, cfl_time_step

pytestmark = pytest.mark.gpu


@pytest.fixture
def waits():
    L = _lib.load()

    def limits(*v):
        _lib.check(L.mj_debug_set_wait_limits(*v))

    yield limits
    limits(-1, -1, -1)


def _problem(order, cells):
    m = M.perturbed_cube(cells, seed=3, amplitude=0.05, kind="random", c_mode="element")
    pb = AcousticProblem(m, M.AcousticSetup(order=order, dt=1.0, nsteps=60, src_radius=2.0 / cells), defer_time=True)
    pb.set_time_step(cfl_time_step(pb, safety=0.5), 60)
    return pb


@pytest.mark.parametrize("precision,order,variant", [("fp64", 4, (5, 5)), ("fp32", 7, (2, 6))])
def test_element_kernels(waits, precision, order, variant):
    pb = _problem(order, 9)
    op = pb.operator(precision)
    op.set_variant(*variant)
    x = np.random.default_rng(0).uniform(-1, 1, pb.n_dof)
    want, y = np.zeros(pb.n_dof), np.zeros(pb.n_dof)
    op.MltVector(x, want)
    waits(0, -1, -1)
    with pytest.raises(_lib.MontjoieError) as e:
        op.MltVector(x, y)
    assert e.value.code == _lib.MJ_ERR_CUDA and "bounded wait" in str(e.value)
    waits(-1, -1, -1)
    op.MltVector(x, y)
    assert np.array_equal(y, want)
    op.close()


@pytest.mark.parametrize("diagnostics", [False, True])
def test_streaming_gather_fp64(waits, diagnostics):
    pb = _problem(4, 9)
    op = pb.operator("fp64")
    op.set_variant(4, 5)  # the element kernel's own waits hold
    lf = pb.integrator(op, diagnostics=diagnostics)
    lf.set_graph(False)

    def run():
        lf.SetInitialConditionS(np.zeros(pb.n_dof))
        return lf.Advance(12), lf.GetState()

    want = run()
    waits(0, -1, -1)
    with pytest.raises(_lib.MontjoieError) as e:
        run()
    assert e.value.code == _lib.MJ_ERR_CUDA and "bounded wait" in str(e.value)
    waits(-1, -1, -1)
    got = run()
    assert all(np.array_equal(a, b) for a, b in zip(got[1], want[1]))
    if diagnostics:
        assert np.array_equal(got[0][0], want[0][0])
    lf.close()
    op.close()


def test_plane_step(waits):
    g = load_golden("cube3_q4")
    op = FemMatrixFreeOperator(4, g["nodle"], g["bh"], g["massD"].size, "fp32", gradphi=g["gradphi"])
    S = 8
    idx = np.concatenate([g["src_idx"]] * S)
    rhs = np.repeat(np.arange(S), g["src_idx"].size)
    b = BatchLeapFrog(op, float(g["dt"]), S, g["massD"], g["invD"], idx, rhs, np.tile(g["src_val"], S), g["pulse"])
    b.set_step_variant(4, 8, 1)

    def run():
        b.init()
        b.advance(15, graph=False)
        return b.state()

    want = run()
    waits(0, 0, 0)  # CTAs without a tile go straight to the grid barrier, where nobody comes
    with pytest.raises(_lib.MontjoieError) as e:
        run()
    assert e.value.code == _lib.MJ_ERR_STATE and "timed out" in str(e.value)
    waits(-1, -1, -1)
    for a, c in zip(run(), want):
        assert np.array_equal(a, c)
    b.close()
    op.close()
