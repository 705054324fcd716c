"""Kernels launched (lbm_get_device_launches) beside the kernels of the steps'
stages (lbm_get_launch_count), counted here by what each route is made of."""
import ctypes as C

import pytest

from fortran_loadfile_mitiwing_b200 import Batch, Lbm, cases

pytestmark = pytest.mark.gpu
LBM_TIMING_KERNELS = 1

SMALL = dict(n_steps=200)                                                     # step_loop launches
LARGE = dict(nx=1301, ny=655, chord=290, pivot=(511, 329), markers=580, n_steps=200, pitch_deg=25.0)   # two steps at a time


def counts(lib, h):
    a, b = C.c_longlong(), C.c_longlong()
    assert lib.lbm_get_launch_count(h.h, C.byref(a)) == 0 and lib.lbm_get_device_launches(h.h, C.byref(b)) == 0
    return a.value, b.value


def during(lib, h, call):
    s0, d0 = counts(lib, h)
    call()
    s1, d1 = counts(lib, h)
    return s1 - s0, d1 - d0


def test_stages_do_not_depend_on_the_route(gpu_lib):
    loop, staged = (Lbm.from_case(cases.small_case(**SMALL), gpu_lib) for _ in range(2))
    assert gpu_lib.lbm_set_timing(staged.h, LBM_TIMING_KERNELS) == 0
    a, b = (during(gpu_lib, h, lambda h=h: h.run(48)) for h in (loop, staged))
    assert a[0] == b[0]
    assert a[1] < b[1]
    # steps 1 .. 48: a launch and its checks for 1-15, 16-31, 32-47 and 48, the
    # mass check, and the factorization (6 kernels) of those four batches
    assert a[1] == 4 * 2 + 1 + 4 * 6
    # every stage of a step and its force row and check, the mass check, the factorization
    assert b[1] == 48 * (4 + 1) + 1 + 4 * 6


def test_pairs(gpu_lib):
    h = Lbm.from_case(cases.small_case(**LARGE), gpu_lib)
    h.run(3)
    s, d = during(gpu_lib, h, lambda: h.run(12))
    # steps 4 .. 15: five pairs (two steps of 3 kernels of the flow, 2 of the
    # near nodes, one lattice launch for both, 2 of force rows and checks), then
    # two single steps of 5, the mass check, the next 16 steps' factorization (6
    # kernels and the near cells), unless the first call began it
    assert d in (5 * (6 + 2 + 1 + 2) + 2 * 5 + 1 + extra for extra in (0, 7))
    checks = sum(1 for n in range(4, 16) if (n + 1) % 4 == 0)
    assert s in (12 * 5 + checks + 1 + extra for extra in (0, 6))


def test_batch_counts_each_case(gpu_lib):
    hs = [Lbm.from_case(cases.small_case(**SMALL), gpu_lib) for _ in range(3)]
    with Batch(hs) as b:
        b.run(16)
        got = [during(gpu_lib, h, lambda: None) for h in hs]
        before = [counts(gpu_lib, h) for h in hs]
        b.run(80)
        after = [counts(gpu_lib, h) for h in hs]
    assert all(g == (0, 0) for g in got)
    diff = {(x[0] - y[0], x[1] - y[1]) for x, y in zip(after, before)}
    assert len(diff) == 1
    stages, launched = diff.pop()
    assert stages > 80 * 5 and launched < 80
