"""FP64 order-2 step with the streaming gather (the default) against the gather, source and diagnostics kernels of
their own (``set_stream_gather(False)``), at chunk edges: fewer dofs than a chunk, ragged counts, orders whose dofs
have up to 8 contributions."""
import numpy as np
import pytest

from montjoie_gb300 import mesh as M
from montjoie_gb300._lib import MontjoieError
from montjoie_gb300.leapfrog import LeapFrogIterator
from montjoie_gb300.problem import AcousticProblem

pytestmark = pytest.mark.gpu

# The two forms round alike up to the contraction of one multiply-add per dof and step (and the order of the norm's
# sums): at most one ulp (1.1e-16) per dof and step, growing at most linearly in the 27 steps of a stable run.
TOL = 27 * 27 * 1.2e-16


@pytest.mark.parametrize("order,cells", [(1, 1), (1, 9), (2, 3), (3, 5), (4, 1), (4, 6), (8, 2)])
@pytest.mark.parametrize("norm", ["mass", "other", None])
def test_streaming_gather_matches_the_separate_kernels(order, cells, norm):
    m = M.perturbed_cube(cells, seed=order, amplitude=0.05, kind="random", c_mode="element")
    pb = AcousticProblem(m, M.AcousticSetup(order=order, src_radius=0.5, dt=0.1 / (cells * order * order), nsteps=20),
                         receivers=np.array([[0.3, 0.4, 0.6], [0.9, 0.1, 0.2], [0.5, 0.5, 0.5]]))
    op = pb.operator("fp64")
    w = {"mass": pb.mass, "other": pb.mass * np.linspace(0.5, 2.0, pb.n_dof), None: None}[norm]
    u0 = np.random.default_rng(order).uniform(-1, 1, pb.n_dof)
    out = []
    for stream in (True, False):
        lf = LeapFrogIterator(op, pb.setup.dt, pb.mass, None, pb.src_idx, pb.src_val, pb.pulse, w, pb.rec_idx, pb.rec_w)
        if not stream:
            lf.set_stream_gather(False)
        lf.SetInitialConditionS(u0, 0.1 * u0)
        a = lf.Advance(1)
        b = lf.Advance(25)  # a replayed graph and plain steps
        c = lf.Run(u0, None, 3)
        lf.SetInitialConditionS(u0)
        lf.Advance(27)
        out.append([x for x in (*a, *b, *c, *lf.GetState()) if x is not None])
        lf.close()
    assert len(out[0]) == len(out[1])
    for x, y in zip(*out):
        assert np.linalg.norm(x - y) <= TOL * np.linalg.norm(y)


def test_fp64_refuses_to_switch_it_on():
    m = M.perturbed_cube(2, seed=1)
    pb = AcousticProblem(m, M.AcousticSetup(order=2, src_radius=0.5))
    lf = pb.integrator(pb.operator("fp64"))
    with pytest.raises(MontjoieError):
        lf.set_stream_gather(True)
