"""Large lattices run two steps in one pass (csrc/kf_pair.cu), with the nodes
near the bodies and at the edge taken step by step; batches of them run one
launch per stage and step. Both must give the same bits. The cases (more
markers than step_loop takes, so that lattices of a few hundred thousand nodes
run this way) have odd sizes, strips and row chunks with remainders, one and
two wings, and bodies that move through cell borders; the runs begin and end
at odd and even steps."""
import numpy as np
import pytest

from fortran_loadfile_mitiwing_b200 import Batch, Lbm, cases
from fortran_loadfile_mitiwing_b200._abi import LBM_DELTA_SMOOTH

pytestmark = pytest.mark.gpu

SHAPES = {
    # nx, ny, chord, pivot, markers per wing, wings, kwargs
    "even": (1280, 640, 290, (500, 321), 580, 1, {}),
    "odd": (1301, 655, 290, (511, 329), 580, 1, dict(pitch_deg=25.0)),
    "strip": (1274, 701, 300, (499, 350), 600, 1, dict(heave=0.3, delta=LBM_DELTA_SMOOTH)),
    "wings": (1403, 603, 160, (400, 301), 310, 2, {}),
    "full": (1204, 640, 290, (500, 321), 580, 1, {}),   # strips of 240 (480) columns without a remainder, with one of a column
    "one": (1205, 641, 290, (500, 321), 580, 1, {}),
    "full2": (1924, 640, 290, (500, 321), 580, 1, {}),
    "one2": (1925, 641, 290, (500, 321), 580, 1, {}),
    "wide": (2051, 1031, 300, (700, 515), 590, 1, dict(pitch_deg=20.0)),
    "edge": (1283, 641, 290, (82, 28), 580, 1, dict(heave=0.005, pitch_deg=0.0)),   # cells at the left and lower edge
}


def make(name, precision, lib, n_steps=64):
    nx, ny, chord, pivot, markers, wings, kw = SHAPES[name]
    return Lbm.from_case(cases.small_case(nx=nx, ny=ny, chord=chord, pivot=pivot, markers=markers, wings=wings,
                                          precision=precision, n_steps=n_steps, **kw), lib)


def same(alone, member, rows_a, rows_b):
    np.testing.assert_array_equal(rows_a, rows_b)
    np.testing.assert_array_equal(alone.populations(), member.populations())
    for x, y in zip(alone.fields(), member.fields()):
        np.testing.assert_array_equal(x, y)


@pytest.mark.parametrize("name,precision", [("even", "fp32"), ("odd", "fp32"), ("strip", "fp32"), ("wings", "fp32"),
                                            ("edge", "fp32"), ("odd", "fp64"), ("strip", "fp64"), ("wide", "fp16"),
                                            ("wide", "bf16"), ("full", "fp32"), ("one", "fp32"), ("one", "fp64"),
                                            ("full2", "fp16"), ("one2", "bf16")])
def test_pairs_equal_single_steps(gpu_lib, name, precision):
    alone, member = make(name, precision, gpu_lib), make(name, precision, gpu_lib)
    held = alone.device_bytes()
    rows = alone.run(21)
    p = alone.params
    assert alone.device_bytes() - held > 9 * p.nx * p.ny * {"fp64": 8, "fp32": 4}.get(precision, 2)   # the state between
    with Batch([member]) as b:
        rows_b = b.run(21)[0]
    same(alone, member, rows, rows_b)


@pytest.mark.parametrize("chunks", [(1, 4, 3, 5), (2, 6, 9), (16, 1, 4)], ids=str)
def test_call_lengths(gpu_lib, chunks):
    alone, member = make("odd", "fp32", gpu_lib), make("odd", "fp32", gpu_lib)
    rows = np.concatenate([alone.run(k) for k in chunks] + [alone.evolution()[None]])
    with Batch([member]) as b:
        rows_b = b.run(sum(chunks) + 1)[0]
    same(alone, member, rows, rows_b)
    assert alone.solver_info()[2] == member.solver_info()[2] < 1e-10


def test_motion_end(gpu_lib):
    for n in (18, 19):
        alone, member = make("even", "fp32", gpu_lib, n), make("even", "fp32", gpu_lib, n)
        with Batch([member]) as b:
            rows_b = b.run(40)[0]
        rows = alone.run(40)
        np.testing.assert_array_equal(rows, rows_b)
        np.testing.assert_array_equal(alone.populations(), member.populations())
