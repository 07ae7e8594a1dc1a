"""The one-block V-cycle (FP32, grids up to 64^2) against the launch-by-launch
one (FP64) on wide grids without equatorial symmetry, where no multigrid
correction reduces the residual and neither solver gets anywhere."""
import numpy as np
import pytest

from parity_util import params
from test_gpu_elliptic import MIXED_2LEV

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nr, nz", [(66, 34), (128, 96)])
def test_wide_grids_without_equator_stop_both_solvers_alike(nr, nz):
    from ollin.gpu import Evolution
    h = {}
    for solver in ("mixed", "fp64mg"):
        e = Evolution(params(dict(MIXED_2LEV, nl0=0, nrtotal=nr, nztotal=nz, eqsym=0, dr0=9.6 / max(nr, nz),
                                  dz0=9.6 / max(nr, nz), ell_solver=solver)))
        e.initial_data()
        h[solver] = e.ell_history(0)
        assert np.all(np.isfinite(h[solver])), solver
        assert np.all(np.isfinite(e.download(0, "chi"))), solver
        e.close()
    # the residual before any correction is the same system's, in FP64
    assert abs(h["mixed"][0] - h["fp64mg"][0]) <= 1e-12 * h["fp64mg"][0]
    # and the best that either reaches; an FP32 cycle may be refused a little
    # earlier or later than an FP64 one, but not reach another residual
    assert abs(h["mixed"].min() - h["fp64mg"].min()) <= 1e-3 * h["fp64mg"][0]
