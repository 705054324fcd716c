"""Which batches share step_loop launches: where every case gets CTAs enough
for its lattice. With too many cases the launches per stage are faster, and a
batch runs as those; either way each case gives what it gives alone."""
import ctypes as C

import numpy as np
import pytest

from fortran_loadfile_mitiwing_b200 import Batch, Lbm, cases

pytestmark = pytest.mark.gpu

STEPS = 48


def make(nx, ny, chord, markers, lib, seed=7):
    return Lbm.from_case(cases.small_case(nx=nx, ny=ny, chord=chord, pivot=(2 * chord + 1, ny // 2 + 1), markers=markers,
                                          n_steps=200, seed=seed), lib)


def launches(lib, h):
    v = C.c_longlong()
    assert lib.lbm_get_device_launches(h.h, C.byref(v)) == 0
    return v.value


@pytest.mark.parametrize("shape,count,shared", [
    ((256, 128, 32, 64), 24, True), ((256, 128, 32, 64), 32, True), ((256, 128, 32, 64), 36, False),
    ((256, 128, 32, 64), 48, False), ((160, 96, 32, 64), 36, True), ((160, 96, 32, 64), 48, False),
    ((96, 64, 24, 40), 60, True), ((384, 192, 48, 96), 20, True), ((384, 192, 48, 96), 28, False),
], ids=str)
def test_route(gpu_lib, shape, count, shared):
    members = [make(*shape, gpu_lib, seed=c) for c in range(count)]
    with Batch(members) as b:
        n0 = launches(gpu_lib, members[0])
        rows = b.run(STEPS)
        made = launches(gpu_lib, members[0]) - n0
    # a launch and its checks for up to 16 steps, or four kernels a step and more
    assert (made < STEPS) == shared, made
    for c in (0, count - 1):
        alone = make(*shape, gpu_lib, seed=c)
        np.testing.assert_array_equal(alone.run(STEPS), rows[c])
        np.testing.assert_array_equal(alone.populations(), members[c].populations())
    for h in members:
        h.close()
