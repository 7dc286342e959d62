"""FP64 operators and runs where the device has no room for what only makes them faster: the factors' second copy of the
fixed-point kernel, the streaming gather's arrays.  They fall back to the kernels that need neither."""
import numpy as np
import pytest

from conftest import rel_l2
from montjoie_gb300 import _lib, mesh as M
from montjoie_gb300.leapfrog import LeapFrogIterator
from montjoie_gb300.operator import FemMatrixFreeOperator
from montjoie_gb300.problem import AcousticProblem

pytestmark = pytest.mark.gpu


@pytest.fixture
def memory_limit():
    L = _lib.load()
    yield lambda more: _lib.check(L.mj_debug_set_memory_limit(int(more)))
    _lib.check(L.mj_debug_set_memory_limit(-1))


@pytest.fixture(scope="module")
def problem():
    m = M.perturbed_cube(6, seed=1, amplitude=0.05, kind="random", c_mode="element")
    return AcousticProblem(m, M.AcousticSetup(order=4, src_radius=0.3), defer_time=True)


def _operator(pb):
    return FemMatrixFreeOperator(4, pb.nodle, pb.factors, pb.n_dof, "fp64")


def _integrator(pb, op):
    src = np.arange(5, dtype=np.int32) * 100
    return LeapFrogIterator(op, 1e-3, pb.mass, None, src, np.ones(5), np.linspace(-1, 1, 30), pb.norm_weight)


def test_operator_without_room_for_the_second_factors(problem, memory_limit):
    pb = problem
    full = _operator(pb)
    limbs = 240 * 125 // 4 * 4 * 6 * 8  # 216 elements padded to 240
    x = np.random.default_rng(0).uniform(-1, 1, pb.n_dof)
    y0, y1 = np.zeros(pb.n_dof), np.zeros(pb.n_dof)
    full.MltVector(x, y0)
    memory_limit(full.device_bytes() - limbs // 2)
    op = _operator(pb)
    memory_limit(-1)
    assert full.tuning()["layout"] == "fixed_point" and op.tuning()["layout"] == "compact"
    assert op.device_bytes() < full.device_bytes() - limbs
    op.MltVector(x, y1)
    assert rel_l2(y1, y0) < 1e-13
    op.set_element_scale(np.full(op.n_elt, 2.0))
    op.MltVector(x, y1)
    assert rel_l2(y1, 2.0 * y0) < 1e-13
    for o in (op, full):
        o.close()


def test_run_without_room_for_the_streaming_gather(problem, memory_limit):
    pb = problem
    op = _operator(pb)
    u0 = np.random.default_rng(1).uniform(-1, 1, pb.n_dof)
    states, launches = [], []
    for more in (-1, 44 * pb.n_dof):  # a run's own arrays are 40 bytes per dof, the streaming gather's 8 more
        memory_limit(more)
        lf = _integrator(pb, op)
        memory_limit(-1)
        u, norms, _ = lf.Run(u0, None, 40)
        before = _lib.load().mj_kernel_launches()
        lf.Advance(1)
        launches.append(_lib.load().mj_kernel_launches() - before)
        states.append((u, norms))
        lf.close()
    assert launches[1] > launches[0]  # gather and source kernels
    assert rel_l2(states[1][0], states[0][0]) < 1e-12 and rel_l2(states[1][1], states[0][1]) < 1e-12
    op.close()
