"""Integrators used from several host threads: each reads its own error word and stages its own copies."""
import threading

import numpy as np
import pytest

from conftest import load_golden
from montjoie_gb300 import _lib
from montjoie_gb300.leapfrog import BatchLeapFrog, LeapFrogIterator
from montjoie_gb300.operator import FemMatrixFreeOperator

pytestmark = pytest.mark.gpu


def _in_threads(*work):
    errors, go = [], threading.Barrier(len(work))

    def run(f):
        try:
            go.wait()
            f()
        except BaseException as e:  # handed to the test's own thread
            errors.append(e)

    threads = [threading.Thread(target=run, args=(f,)) for f in work]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors


def test_a_failing_batch_beside_a_good_one():
    """Two batches on one operator, one whose every step times out at its grid barrier (limits lowered, which the
    two-kernel form of the other has none of): every call of the first is an error, every call of the other is not."""
    g = load_golden("cube3_q4")
    op = FemMatrixFreeOperator(4, g["nodle"], g["bh"], g["massD"].size, "fp32", gradphi=g["gradphi"])
    S = 8
    bad, good = (BatchLeapFrog(op, float(g["dt"]), S, g["massD"], g["invD"], np.zeros(0, np.int32),
                               np.zeros(0, np.int32), np.zeros(0), g["pulse"]) for _ in range(2))
    good.set_fused(False)
    for b in (bad, good):
        b.init()
    L = _lib.load()
    _lib.check(L.mj_debug_set_wait_limits(-1, 0, 0))
    try:
        def fail():
            for _ in range(400):
                with pytest.raises(_lib.MontjoieError) as e:
                    bad.advance(1)
                assert e.value.code == _lib.MJ_ERR_STATE

        def succeed():
            for _ in range(400):
                good.advance(1)

        _in_threads(fail, succeed)
    finally:
        _lib.check(L.mj_debug_set_wait_limits(-1, -1, -1))
        bad.close()
        good.close()
        op.close()


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_state_read_by_several_threads(precision):
    g = load_golden("cube4_q4")
    n = g["massD"].size
    op = FemMatrixFreeOperator(4, g["nodle"], g["bh"], n, precision, gradphi=g["gradphi"])
    lf = LeapFrogIterator(op, float(g["dt"]), g["massD"])
    lf.SetInitialConditionS(np.random.default_rng(0).uniform(-1, 1, n))
    lf.Advance(7)
    want = lf.GetState()
    assert not np.array_equal(*want)

    def read():
        for _ in range(200):
            for a, b in zip(lf.GetState(), want):
                assert np.array_equal(a, b)

    _in_threads(read, read, read)
    lf.close()
    op.close()
