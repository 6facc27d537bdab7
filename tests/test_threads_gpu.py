"""Handles of different sizes driven from two host threads at once: each call
succeeds and gives what it gives alone.  The sizes of a pair share the kernels
they launch, with different amounts of shared memory."""
import threading

import numpy as np
import pytest

from ixchel2d_b200 import Simple2D, cases

pytestmark = pytest.mark.gpu


def _loop(s):
    for _ in range(250):
        s.iterations(1)


def _passes(s):
    for _ in range(300):
        s.energy_iterations(4)


def _gradients(s):
    for _ in range(25):
        s.adjoint_energy(12, 2, 10)
        s.adjoint_simple(2, 1, 2, 10)


# 256x256 and 300x200 run the loop's 384-thread form, 701x301 and 520x30 its 768-thread form; the passes' kernel is one
# for all sizes; x-lines of 800 and 1500 rows the gradients' 256-thread form with chunks of 4 and 6
@pytest.mark.parametrize("work, sizes", [(_loop, [(300, 200), (256, 256)]), (_loop, [(701, 301), (520, 30)]),
                                         (_passes, [(256, 256), (40, 36)]), (_gradients, [(800, 20), (1500, 24)])])
def test_two_threads(has_gpu, work, sizes):
    if not has_gpu:
        pytest.skip("no CUDA device")

    def run(mi, nj):
        with Simple2D.from_case(cases.natural_cavity(mi, nj, Ra=1e4)) as s:
            s.iterations(2)
            ready.wait(60)
            work(s)
            return s.download()

    def guarded(k, size):
        try:
            got[k] = run(*size)
        except Exception as e:  # noqa: BLE001
            got[k] = e

    got, alone = [None, None], []
    for size in sizes:
        ready = threading.Barrier(1)
        alone.append(run(*size))
    ready = threading.Barrier(2)
    threads = [threading.Thread(target=guarded, args=(k, size)) for k, size in enumerate(sizes)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for g, a in zip(got, alone):
        assert isinstance(g, dict), g
        for k in ("u", "v", "p", "T"):
            assert np.array_equal(g[k], a[k]), k
