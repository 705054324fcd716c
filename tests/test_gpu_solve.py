"""The marker solve of single steps (ib_solve, and the tiles' last level of the
back-substitution) at the block counts where its form changes: one block, an
odd and an even number, a level with more even blocks than warps, and the
counts where the resident levels begin at 4 instead of 2 (more than 69 blocks).

Each step's system is solved in FP64 by both sides, in another order of
summation; with the marker system's condition below 1e4 the differences stay
below 1e-12 a step. The bars are those of the FP64 parity tests: 1e-11 on
populations of order 0.1, 1e-8 relative on the forces, and a residual of the
solve below 1e-10."""
import numpy as np
import pytest

from fortran_loadfile_mitiwing_b200 import Batch, Lbm, cases

pytestmark = pytest.mark.gpu

STEPS = 6   # the residual of the fourth is checked


@pytest.mark.parametrize("markers", [8, 16, 18, 32, 34, 256, 512, 530, 1104, 1106])
def test_single_steps(gpu_lib, oracle_mod, markers):
    chord, ny = max(8, markers // 2), markers // 8 + 80
    case = cases.small_case(nx=2 * chord + 80, ny=ny, chord=chord, pivot=(chord + 40, ny // 2), markers=markers,
                            n_steps=STEPS + 4, precision="fp64", heave=0.02, pitch_deg=0.0)
    g, member, o = Lbm.from_case(case, gpu_lib), Lbm.from_case(case, gpu_lib), oracle_mod.Oracle.from_case(case)
    rg = np.array([g.evolution() for _ in range(STEPS)])
    ro = o.run(STEPS)
    assert np.abs(g.populations() - o.populations()).max() < 1e-11
    floor = np.sqrt(np.mean(ro[:, 1:4] ** 2, axis=0))
    assert np.max(np.abs(rg[:, 1:4] - ro[:, 1:4]) / np.maximum(np.abs(ro[:, 1:4]), floor)) < 1e-8
    assert g.solver_info()[2] < 1e-10
    with Batch([member]) as b:
        np.testing.assert_array_equal(b.run(STEPS)[0], rg)
    np.testing.assert_array_equal(member.populations(), g.populations())
