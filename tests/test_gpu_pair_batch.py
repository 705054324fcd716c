"""A large lattice that moves between a batch and calls of its own. A batch
factorizes the marker system without the list of cells near the body that the
handle's own two-step launches (csrc/kf_pair.cu) work from; the handle makes
it when it needs it. Whatever the order of the calls, the result is that of
the handle run alone, bit for bit."""
import numpy as np
import pytest

from fortran_loadfile_mitiwing_b200 import Batch, Lbm, cases
from fortran_loadfile_mitiwing_b200._abi import LBM_DELTA_SMOOTH

pytestmark = pytest.mark.gpu

SHAPES = {
    # nx, ny, chord, pivot, markers per wing, wings, kwargs
    "odd": (1301, 655, 290, (511, 329), 580, 1, dict(pitch_deg=25.0)),
    "strip": (1274, 701, 300, (499, 350), 600, 1, dict(heave=0.3, delta=LBM_DELTA_SMOOTH)),
    "wings": (1403, 603, 160, (400, 301), 310, 2, {}),
    "wide": (2051, 1031, 300, (700, 515), 590, 1, dict(pitch_deg=20.0)),
}


def make(name, precision, lib):
    nx, ny, chord, pivot, markers, wings, kw = SHAPES[name]
    return Lbm.from_case(cases.small_case(nx=nx, ny=ny, chord=chord, pivot=pivot, markers=markers, wings=wings,
                                          precision=precision, n_steps=140, **kw), lib)


# steps in a batch (b) and alone (a), in turn; factorization batches hold 16
# steps, two of them at a time, so that a call finds the cells of its steps
# missing, made, or those of 32 steps before
ORDERS = ["b5 a16", "a10 b30 a25", "b17 a3 b20 a40", "a21 b1 a20 b40 a30", "b40 a1 a1 a30", "a40 b60 a20"]


@pytest.mark.parametrize("name,precision", [("odd", "fp32"), ("strip", "fp64"), ("wings", "fp32"), ("wide", "fp16")])
@pytest.mark.parametrize("order", ORDERS)
def test_batch_then_alone(gpu_lib, order, name, precision):
    alone, mixed = make(name, precision, gpu_lib), make(name, precision, gpu_lib)
    rows, total = [], 0
    for part in order.split():
        k = int(part[1:])
        total += k
        if part[0] == "a":
            rows.append(mixed.run(k))
        else:
            with Batch([mixed]) as b:
                rows.append(b.run(k)[0])
    np.testing.assert_array_equal(alone.run(total), np.concatenate(rows))
    np.testing.assert_array_equal(alone.populations(), mixed.populations())
    for x, y in zip(alone.fields(), mixed.fields()):
        np.testing.assert_array_equal(x, y)
