"""FP64 gathers that sum a block's dofs in the order of their degree: every degree from 1 to far beyond the sort's 16
bins, block ends (256 threads x 4 dofs) and an empty last block, against the oracle's element loop."""
import numpy as np
import pytest

from montjoie_gb300.operator import FemMatrixFreeOperator

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_dof", [9, 1023, 1024, 1025, 3001])
@pytest.mark.parametrize("hubs", [0, 3])
def test_mltadd_sums_every_degree(n_dof, hubs):
    from oracle import oracle as oc
    r = 2
    rng = np.random.default_rng(n_dof + hubs)
    n_elt = max(2, n_dof // 9)
    nodle = rng.integers(0, n_dof, size=(n_elt, 27))
    nodle.reshape(-1)[:n_dof] = rng.permutation(n_dof)[:min(n_dof, nodle.size)]  # every dof belongs to an element
    for h in range(hubs):  # dofs with a contribution of every element: n_elt of them
        nodle[:, 26 - h] = np.where(np.arange(n_elt) * 27 + 26 - h < n_dof, nodle[:, 26 - h], h)
    nodle = nodle.astype(np.int32)
    bh = rng.uniform(0.5, 1.5, size=(n_elt, 27, 6))
    op = FemMatrixFreeOperator(r, nodle, bh, n_dof, "fp64")
    x, y0 = rng.uniform(-1, 1, n_dof), rng.uniform(-1, 1, n_dof)
    y = y0.copy()
    op.MltAddVector(-0.7, x, 0.5, y)
    ref = oc.stiffness_mltadd(r, nodle, bh, -0.7, x, 0.5, y0.copy())
    degree = np.bincount(nodle.reshape(-1), minlength=n_dof).max()
    # absolute sum of one contribution: 3 directions x 8 (row sum of |G|, order 2) x 3 factors of 1.5 x 8 = 864; it rounds
    # by at most about 24 u of that (two contractions and a factor row), a sum of `degree` of them by as many u more
    tol = (24 + degree) * 2.0 ** -53 * 864 * degree
    assert np.abs(y - ref).max() <= tol
    op.close()
