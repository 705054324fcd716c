"""A case that moves from batch to batch: each batch numbers the
factorization launches that its graph segments wait for by itself, and must
not take another's numbers for its own."""
import numpy as np
import pytest

from fortran_loadfile_mitiwing_b200 import Batch, Lbm, cases

pytestmark = pytest.mark.gpu

SMALL = dict(n_steps=400)
LARGE = dict(nx=1301, ny=655, chord=290, pivot=(511, 329), markers=580, n_steps=400, pitch_deg=25.0)


@pytest.mark.parametrize("kw", [SMALL, LARGE], ids=["loop", "stages"])
@pytest.mark.parametrize("chunks", [(10, 42), (42, 42), (100, 3, 60), (7, 90, 26, 51)], ids=str)
def test_new_batch_each_run(gpu_lib, kw, chunks):
    alone, moved = (Lbm.from_case(cases.small_case(**kw), gpu_lib) for _ in range(2))
    rows = []
    for k in chunks:
        with Batch([moved]) as b:
            rows.append(b.run(k)[0])
    np.testing.assert_array_equal(alone.run(sum(chunks)), np.concatenate(rows))
    np.testing.assert_array_equal(alone.populations(), moved.populations())


def test_two_batches_in_turn(gpu_lib):
    alone, h, other = (Lbm.from_case(cases.small_case(**SMALL), gpu_lib) for _ in range(3))
    with Batch([h]) as a, Batch([other]) as b:
        b.run(90)
        b.remove(other)
        b.add(h)
        rows = [x.run(k)[0] for x, k in ((a, 50), (b, 40), (a, 41), (b, 60))]
    np.testing.assert_array_equal(alone.run(191), np.concatenate(rows))
    np.testing.assert_array_equal(alone.populations(), h.populations())
