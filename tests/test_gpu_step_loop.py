"""Small lattices run several steps per launch (csrc/step_loop.cu), alone and in
batches; with per-kernel timing on, a case runs one launch per stage. All call
the same node, marker and tile functions in the same order, so they must give
the same force rows, populations and fields, bit for bit. The cases are where
the loop's work division can go wrong: odd sizes (a last row pair or column
pair with one node), sizes at and beside a warp's and a row pair's width, one
and two wings, marker counts around the 16-marker blocks and at the largest
count one launch's solver holds (576; the next one runs kernel by kernel),
and step counts around the 16 steps of a launch."""
import numpy as np
import pytest

from fortran_loadfile_mitiwing_b200 import Batch, Lbm, cases
from fortran_loadfile_mitiwing_b200._abi import LBM_DELTA_SMOOTH

pytestmark = pytest.mark.gpu
LBM_TIMING_KERNELS = 1

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
    alone, member, staged = (make(shape, precision, gpu_lib) for _ in range(3))
    with Batch([member]) as b:
        b.set_graphs(False)
        rows_b = b.run(21)[0]
    assert gpu_lib.lbm_set_timing(staged.h, LBM_TIMING_KERNELS) == 0
    rows = alone.run(21)
    same(alone, member, rows, rows_b)
    same(alone, staged, rows, staged.run(21))


@pytest.mark.parametrize("chunks", [(1, 1, 1), (7, 8, 9), (2, 16, 3), (8, 8, 5), (15, 16, 17), (33, 14)], ids=str)
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


@pytest.mark.parametrize("graphs", [True, False], ids=["graphs", "stream"])
@pytest.mark.parametrize("precision", ["fp32", "fp64", "fp16"])
def test_batch_of_small_cases(gpu_lib, precision, graphs):
    """Cases of different sizes at one phase share step_loop launches, from the
    host and inside graph segments; each gives what it gives alone, over runs
    that begin at every phase of a factorization batch, and with a case that
    ends inside a run."""
    shapes = SHAPES[:5] + [SHAPES[6]]
    steps = (3, 40, 21, 1, 30)
    ends = [200, 200, 60, 200, 200, 200]
    alone = [make(s, precision, gpu_lib, n) for s, n in zip(shapes, ends)]
    member = [make(s, precision, gpu_lib, n) for s, n in zip(shapes, ends)]
    with Batch(member) as b:
        b.set_graphs(graphs)
        for k in steps:
            rows = b.run(k)
            for a, r in zip(alone, rows):
                np.testing.assert_array_equal(a.run(k), r)
        assert b.graph_stats()[0] > 0 or not graphs
    for a, m, n in zip(alone, member, ends):
        same(a, m, np.zeros(0), np.zeros(0), fields=n == 200)


def test_batch_of_many_tiny_cases(gpu_lib):
    """As many cases as one launch takes (two CTAs each), and more."""
    for count in (66, 70):
        kw = [dict(seed=c, heave=0.1 + 0.002 * c) for c in range(count)]
        alone = [Lbm.from_case(cases.small_case(n_steps=60, **k), gpu_lib) for k in kw]
        member = [Lbm.from_case(cases.small_case(n_steps=60, **k), gpu_lib) for k in kw]
        with Batch(member) as b:
            rows = b.run(27)
        for a, m, r in zip(alone, member, rows):
            same(a, m, a.run(27), r)
        for h in alone + member:
            h.close()
