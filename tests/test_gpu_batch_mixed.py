"""Batches whose cases need solves of different forms: up to 68 blocks of 16
markers the solve keeps the factor blocks of every level above the first in
shared memory, from 69 blocks on those of every second one, so that a case of
fewer markers may need more shared memory than the batch's largest. Each case
gives in the batch, bit for bit, what it gives alone."""
import numpy as np
import pytest

from fortran_loadfile_mitiwing_b200 import Batch, Lbm, cases

pytestmark = pytest.mark.gpu

STEPS = 6


def case_of(markers):
    chord, ny = max(8, markers // 2), markers // 8 + 80
    return cases.small_case(nx=2 * chord + 80, ny=ny, chord=chord, pivot=(chord + 40, ny // 2), markers=markers,
                            n_steps=STEPS + 4, precision="fp64", heave=0.02, pitch_deg=0.0)


def make(markers, lib):
    return Lbm.from_case(case_of(markers), lib)


@pytest.mark.parametrize("markers", [1088, 1090])
def test_either_side_of_the_change(gpu_lib, oracle_mod, markers):
    """68 and 69 blocks, one case alone against the oracle (the bars are those
    of the other FP64 solves of six steps: 1e-11 on populations, 1e-8 relative
    on the forces)."""
    g, o = make(markers, gpu_lib), oracle_mod.Oracle.from_case(case_of(markers))
    rg, ro = np.array([g.evolution() for _ in range(STEPS)]), o.run(STEPS)
    assert np.abs(g.populations() - o.populations()).max() < 1e-11
    floor = np.sqrt(np.mean(ro[:, 1:4] ** 2, axis=0))
    assert np.max(np.abs(rg[:, 1:4] - ro[:, 1:4]) / np.maximum(np.abs(ro[:, 1:4]), floor)) < 1e-8
    assert g.solver_info()[2] < 1e-10


@pytest.mark.parametrize("markers", [(1104, 800), (1104, 1024), (1088, 1090), (640, 1600, 40), (1984, 1088, 610)], ids=str)
def test_mixed_marker_counts(gpu_lib, markers):
    alone, member = ([make(m, gpu_lib) for m in markers] for _ in range(2))
    with Batch(member) as b:
        rows = b.run(STEPS)
    for a, m, r in zip(alone, member, rows):
        np.testing.assert_array_equal(a.run(STEPS), r)
        np.testing.assert_array_equal(a.populations(), m.populations())
        assert a.solver_info()[2] == m.solver_info()[2] < 1e-10
