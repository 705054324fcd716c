"""Starting over discards steps that were factorized ahead and not run, and
with them the errors of their factorization: here the body would leave the
lattice at step 61, the run stops at step 52, and the repeated run from the
first step must not meet that error in the slot that step 61 used."""
import numpy as np
import pytest

from fortran_loadfile_mitiwing_b200 import Batch, Lbm, cases
from fortran_loadfile_mitiwing_b200.solver import LbmError

pytestmark = pytest.mark.gpu


def make(lib, precision="fp32"):
    case = cases.small_case(precision=precision, n_steps=80)
    case.table[60:, 1 + 6] = 2.0   # the pivot two chords up, past the upper edge
    return case, Lbm.from_case(case, lib)


@pytest.mark.parametrize("batched", [False, True], ids=["alone", "batch"])
def test_errors_of_discarded_steps(gpu_lib, batched, tmp_path):
    case, h = make(gpu_lib)

    def run(k):
        if not batched:
            return h.run(k)
        with Batch([h]) as b:
            return b.run(k)[0]

    first = run(10)
    h.save_checkpoint(str(tmp_path / "c"))
    first = np.concatenate([first, run(42)])
    h.init(case.du, case.dv)
    np.testing.assert_array_equal(run(52), first)
    h.load_checkpoint(str(tmp_path / "c"))
    np.testing.assert_array_equal(run(42), first[10:])
    with pytest.raises(LbmError, match="LBM_ERR_RANGE"):
        run(20)
