"""The dense factor of the marker system, 8 n^2 bytes a step slot, is held only
by the cases that may need it: those that ask for it, and those whose markers
lie so close, or whose bodies come so near one another, that a coupling of more
than 16 places in the solve order cannot be ruled out."""
import numpy as np
import pytest

from fortran_loadfile_mitiwing_b200 import Batch, Lbm, cases
from fortran_loadfile_mitiwing_b200._abi import LBM_DELTA_SMOOTH, LBM_FLAG_DENSE_SOLVE
from fortran_loadfile_mitiwing_b200.serve import estimate_device_bytes

SLOTS = 32


def one(chord, markers, precision="fp64", angle=0.0, flags=0, **kw):
    """A wing that holds `angle` (degrees) and moves by a tenth of it."""
    n = 2 * chord + 40
    c = cases.small_case(nx=n, ny=n, chord=chord, pivot=(n // 2, n // 2), markers=markers, precision=precision, n_steps=60,
                         heave=0.0, pitch_deg=0.1 * angle, **kw)
    c.table[:, 1] += np.radians(angle)
    c.params.flags = flags
    return c


def two(dx, dy, chord=60, markers=120, **kw):
    c = cases.small_case(nx=320, ny=320, chord=chord, pivot=(100, 140), markers=markers, wings=2, n_steps=60, heave=0.0, **kw)
    c.table[:, 1 + 9 + 3], c.table[:, 1 + 9 + 6] = dx, dy
    return c


def dense_bytes(case):
    p = case.params
    n = p.wing_count * (p.points_per_wing - 1)
    return SLOTS * 8 * n * n


def test_estimate():
    plain = estimate_device_bytes(one(64, 128))
    assert estimate_device_bytes(one(64, 128, flags=LBM_FLAG_DENSE_SOLVE)) == plain + dense_bytes(one(64, 128))
    # 512 markers on the same chord: the rest of the scratch grows with n only
    fine = one(64, 512)
    assert dense_bytes(fine) < estimate_device_bytes(fine) - plain < 1.2 * dense_bytes(fine)
    big = one(512, 1024)
    assert dense_bytes(big) > 250e6
    with_flag = one(512, 1024, flags=LBM_FLAG_DENSE_SOLVE)
    assert estimate_device_bytes(with_flag) - estimate_device_bytes(big) == dense_bytes(big)


@pytest.mark.gpu
@pytest.mark.parametrize("make,dense", [
    (lambda: one(24, 40), False), (lambda: one(128, 256), False), (lambda: one(512, 1024, "fp32"), False),
    (lambda: one(100, 204, delta=LBM_DELTA_SMOOTH), False), (lambda: one(24, 120), True),
    (lambda: one(64, 128, flags=LBM_FLAG_DENSE_SOLVE), True), (lambda: one(24, 10, flags=LBM_FLAG_DENSE_SOLVE), True),
    (lambda: two(1.5, 0.0), False), (lambda: two(0.0, 2.0, pitch_deg=5.0), True),
], ids=["40", "256", "1024", "204", "fine", "flag", "flag10", "tandem", "stacked"])
def test_held(gpu_lib, make, dense):
    case = make()
    with Lbm.from_case(case, gpu_lib) as h:
        h.run(1)
        rest = estimate_device_bytes(case) - (dense_bytes(case) if dense or case.params.wing_count > 1 else 0)
        held = h.device_bytes() - (dense_bytes(case) if dense else 0)
        assert 0.97 * rest <= held <= rest


# contours from far apart markers to two a lattice unit, at angles to the
# lattice, and pairs of wings in line, side by side and across: whatever
# coupling the steps meet, they have the factor they need
@pytest.mark.gpu
@pytest.mark.parametrize("make", [lambda m=m, a=a: one(40, m, angle=a) for m in range(40, 180, 12) for a in (0.0, 30.0, 45.0)] +
                         [lambda m=m, a=a: one(40, m, angle=a, delta=LBM_DELTA_SMOOTH) for m in range(84, 108, 4) for a in (20.0, 45.0, 90.0)] +
                         [lambda dx=dx, dy=dy: two(dx, dy, pitch_deg=20.0) for dx, dy in
                          [(1.5, 0.0), (1.2, 0.4), (1.05, 0.0), (0.5, 0.5), (0.0, 1.0), (0.1, 2.2), (1.3, 1.3)]])
def test_every_step_has_its_factor(gpu_lib, make):
    case = make()
    with Lbm.from_case(case, gpu_lib) as h, Lbm.from_case(case, gpu_lib) as m:
        widest = 0
        rows = []
        for _ in range(40):
            rows.append(h.evolution())
            *_, residual, w = h.solver_info()
            widest = max(widest, w)
            assert residual < 1e-8
        n = case.params.wing_count * (case.params.points_per_wing - 1)
        if widest > 16:
            assert h.device_bytes() > dense_bytes(case)
        with Batch([m]) as b:
            np.testing.assert_array_equal(b.run(40)[0], np.array(rows))
        assert widest < n
