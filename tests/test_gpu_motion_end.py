"""lbm_get_markers reports the solve residual of the last step. A call that
ends because the motion does checks its last step too, as a batch does, on
each of the routes a step can take."""
import numpy as np
import pytest

from fortran_loadfile_mitiwing_b200 import Batch, Lbm, cases

pytestmark = pytest.mark.gpu
LBM_TIMING_KERNELS = 1

SMALL = dict()
LARGE = dict(nx=1301, ny=655, chord=290, pivot=(511, 329), markers=580, pitch_deg=25.0)


@pytest.mark.parametrize("kw", [SMALL, LARGE], ids=["small", "large"])
@pytest.mark.parametrize("staged", [False, True], ids=["", "staged"])
@pytest.mark.parametrize("n", [18, 19, 20, 21, 34])
def test_residual_of_the_last_step(gpu_lib, kw, staged, n):
    h, member = (Lbm.from_case(cases.small_case(n_steps=n, **kw), gpu_lib) for _ in range(2))
    if staged:
        assert gpu_lib.lbm_set_timing(h.h, LBM_TIMING_KERNELS) == 0
    rows = h.run(60)
    assert n - 2 <= rows.shape[0] < 60
    with Batch([member]) as b:
        b.set_graphs(False)
        np.testing.assert_array_equal(b.run(60)[0], rows)
    x, y, residual, width = h.solver_info()
    xm, ym, rm, wm = member.solver_info()
    assert 0.0 < residual < 1e-10 and residual == rm and width == wm
    np.testing.assert_array_equal(x, xm)
    np.testing.assert_array_equal(y, ym)
