"""Small lattices run several steps per launch (csrc/step_loop.cu); batches
run one launch per stage. Both call the same node, marker and tile functions
in the same order, so a case alone must give exactly what it gives in a batch
of one: force rows, populations and fields, bit for bit. The cases are where
the loop's work division can go wrong: odd sizes (a last row pair or column
pair with one node), sizes at and beside a warp's and a row pair's width, one
and two wings, marker counts around the 16-marker blocks and at the largest
count one launch's solver holds (576; the next one runs kernel by kernel),
and step counts around the 8 steps of a launch."""
import numpy as np
import pytest

from fortran_loadfile_mitiwing_b200 import Batch, Lbm, cases
from fortran_loadfile_mitiwing_b200._abi import LBM_DELTA_SMOOTH

pytestmark = pytest.mark.gpu

SHAPES = [
    # nx, ny, chord, pivot, markers, wings, kwargs
    (96, 64, 24, (33, 33), 40, 1, {}),
    (97, 65, 24, (33, 33), 32, 1, {}),
    (127, 66, 20, (41, 33), 34, 1, dict(pitch_deg=25.0)),
    (129, 67, 16, (41, 34), 26, 1, dict(heave=0.3)),
    (241, 121, 24, (50, 61), 48, 2, dict(delta=LBM_DELTA_SMOOTH)),
    (400, 200, 80, (100, 100), 160, 1, dict(pitch_deg=0.0)),
    (705, 353, 88, (177, 177), 204, 1, dict(delta=LBM_DELTA_SMOOTH)),
    (1280, 641, 280, (500, 321), 576, 1, {}),
    (1280, 641, 280, (500, 321), 578, 1, {}),
]


def make(shape, precision, lib, n_steps=64):
    nx, ny, chord, pivot, markers, wings, kw = shape
    return Lbm.from_case(cases.small_case(nx=nx, ny=ny, chord=chord, pivot=pivot, markers=markers, wings=wings,
                                          precision=precision, n_steps=n_steps, **kw), lib)


def same(alone, member, rows_a, rows_b, fields=True):
    np.testing.assert_array_equal(rows_a, rows_b)
    np.testing.assert_array_equal(alone.populations(), member.populations())
    if fields:
        for x, y in zip(alone.fields(), member.fields()):
            np.testing.assert_array_equal(x, y)


@pytest.mark.parametrize("precision", ["fp32", "fp64", "fp16", "bf16"])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: f"{s[0]}x{s[1]}-{s[4]}x{s[5]}")
def test_loop_equals_kernel_by_kernel(gpu_lib, shape, precision):
    alone, member = make(shape, precision, gpu_lib), make(shape, precision, gpu_lib)
    with Batch([member]) as b:
        b.set_graphs(False)
        rows_b = b.run(21)[0]
    same(alone, member, alone.run(21), rows_b)


@pytest.mark.parametrize("chunks", [(1, 1, 1), (7, 8, 9), (2, 16, 3), (8, 8, 5)], ids=str)
def test_call_lengths(gpu_lib, chunks):
    alone, member = make(SHAPES[1], "fp32", gpu_lib), make(SHAPES[1], "fp32", gpu_lib)
    rows = np.concatenate([alone.run(k) for k in chunks] + [alone.evolution()[None]])
    assert np.isfinite(alone.erranalysis())       # the fields of the last two steps are kept
    with Batch([member]) as b:
        rows_b = b.run(sum(chunks) + 1)[0]
    same(alone, member, rows, rows_b)
    assert alone.solver_info()[2] == member.solver_info()[2] < 1e-10


def test_motion_end_inside_a_launch(gpu_lib):
    alone, member = make(SHAPES[0], "fp32", gpu_lib, n_steps=19), make(SHAPES[0], "fp32", gpu_lib, n_steps=19)
    with Batch([member]) as b:
        rows_b = b.run(40)[0]
    rows = alone.run(40)
    assert 8 < rows.shape[0] < 40
    same(alone, member, rows, rows_b, fields=False)


def test_dense_solve(gpu_lib):
    c = cases.small_case(precision="fp64", n_steps=40)
    c.params.flags = 1                            # LBM_FLAG_DENSE_SOLVE
    alone, member = Lbm.from_case(c, gpu_lib), Lbm.from_case(c, gpu_lib)
    with Batch([member]) as b:
        rows_b = b.run(11)[0]
    same(alone, member, alone.run(11), rows_b)
