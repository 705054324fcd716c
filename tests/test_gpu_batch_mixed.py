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


def make(markers, lib):
    chord, ny = max(8, markers // 2), markers // 8 + 80
    return Lbm.from_case(cases.small_case(nx=2 * chord + 80, ny=ny, chord=chord, pivot=(chord + 40, ny // 2), markers=markers,
                                          n_steps=STEPS + 4, precision="fp64", heave=0.02, pitch_deg=0.0), lib)


@pytest.mark.parametrize("markers", [(1104, 800), (1104, 1024), (1088, 1090), (640, 1600, 40), (1984, 1088, 610)], ids=str)
def test_mixed_marker_counts(gpu_lib, markers):
    alone, member = ([make(m, gpu_lib) for m in markers] for _ in range(2))
    with Batch(member) as b:
        rows = b.run(STEPS)
    for a, m, r in zip(alone, member, rows):
        np.testing.assert_array_equal(a.run(STEPS), r)
        np.testing.assert_array_equal(a.populations(), m.populations())
        assert a.solver_info()[2] == m.solver_info()[2] < 1e-10
