"""Batches of small cases whose factorization batches are shorter than the
default (LBM_IB_BATCH): a graph segment of 16 steps then holds several
step_loop launches, from one to sixteen, and up to two factorization launches
beside each. Every case gives what it gives alone, bit for bit, whatever phase
of a factorization batch a run begins at."""
import numpy as np
import pytest

from fortran_loadfile_mitiwing_b200 import Batch, Lbm, cases

pytestmark = pytest.mark.gpu

SHAPES = [
    # nx, ny, chord, pivot, markers
    (96, 64, 24, (33, 33), 40),
    (127, 66, 20, (41, 33), 34),
    (240, 121, 40, (80, 61), 80),
]


def make(lib, n):
    return [Lbm.from_case(cases.small_case(nx=nx, ny=ny, chord=c, pivot=p, markers=m, n_steps=n), lib) for nx, ny, c, p, m in SHAPES]


@pytest.mark.parametrize("steps", [1, 2, 3, 4, 5, 6, 7, 8, 11, 15])
def test_short_factorization_batches(gpu_lib, monkeypatch, steps):
    alone = make(gpu_lib, 400)                # (sixteen steps)
    monkeypatch.setenv("LBM_IB_BATCH", str(steps))
    member = make(gpu_lib, 400)
    monkeypatch.delenv("LBM_IB_BATCH")
    with Batch(member) as b:
        for k in (3, 40, 21, 1, 90, 22, 23):
            rows = b.run(k)
            for a, r in zip(alone, rows):
                np.testing.assert_array_equal(a.run(k), r)
        assert b.graph_stats()[0] > 0
    for a, m in zip(alone, member):
        np.testing.assert_array_equal(a.populations(), m.populations())
        for x, y in zip(a.fields(), m.fields()):
            np.testing.assert_array_equal(x, y)
