"""Handles driven from several host threads at once. The cases' step_loop
launches need different amounts of shared memory (576 markers more than 40),
and the launches' limit belongs to the process, so one thread's setting must
not refuse another's launch; nor may the results depend on what else runs."""
import threading

import numpy as np
import pytest

from fortran_loadfile_mitiwing_b200 import Batch, Lbm, cases

pytestmark = pytest.mark.gpu

SHAPES = [
    # nx, ny, chord, pivot, markers
    (1280, 641, 280, (500, 321), 576),
    (96, 64, 24, (33, 33), 40),
    (1280, 641, 280, (500, 321), 576),
    (127, 66, 20, (41, 33), 34),
]
CALLS = 150


def make(shape, lib):
    nx, ny, c, p, m = shape
    return Lbm.from_case(cases.small_case(nx=nx, ny=ny, chord=c, pivot=p, markers=m, n_steps=2 * CALLS + 10), lib)


@pytest.mark.parametrize("batched", [False, True], ids=["alone", "batch"])
def test_threads(gpu_lib, batched):
    ref = [make(s, gpu_lib) for s in SHAPES]
    got, errors, start = [None] * len(SHAPES), [], threading.Barrier(len(SHAPES))

    def work(t):
        try:
            h = make(SHAPES[t], gpu_lib)
            b = Batch([h]) if batched else None
            start.wait(60)
            rows = [b.run(2)[0] if batched else h.run(2) for _ in range(CALLS)]
            if b:
                b.close()
            got[t] = np.concatenate(rows), h.populations()
        except Exception as e:   # pylint: disable=broad-except
            errors.append((t, e))

    threads = [threading.Thread(target=work, args=(t,)) for t in range(len(SHAPES))]
    for t in threads:
        t.start()
    for t in threads:
        t.join(120)
    assert not errors and all(g is not None for g in got), errors
    for h, g in zip(ref, got):
        np.testing.assert_array_equal(np.concatenate([h.run(2) for _ in range(CALLS)]), g[0])
        np.testing.assert_array_equal(h.populations(), g[1])
