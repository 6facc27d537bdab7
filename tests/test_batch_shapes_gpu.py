"""Batched iterations with the default launch shapes against the same
instances with explicit assembly and line-solve launches: sizes whose chunks
cover every rows-per-thread case of the register y-lines (3 to 8) and the one
beyond them, and the shape rules' line lengths.

With the same 64 threads per line the two paths run the same operations in
the same order per line, up to contraction: 1e-13 relative of the largest
value after 6 iterations in binary64; the refined form's binary32 solves
round at 6e-8 of a correction that the first iterations keep within 1e-2 of
the fields' size: 1e-8."""
import numpy as np
import pytest

from ixchel2d_b200 import Batch, cases
from ixchel2d_b200 import _ffi as F

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _need_gpu(has_gpu):
    if not has_gpu:
        pytest.skip("no CUDA device")


GROUPS = [[(5, 6), (64, 191), (193, 192), (255, 257), (40, 321)],
          [(321, 33), (384, 385), (30, 449), (449, 30)],
          [(513, 20), (20, 513), (600, 70)]]


@pytest.mark.parametrize("prec, tol", [(F.PREC_FP64, 1e-13), (F.PREC_FP32_REFINED, 1e-8)])
@pytest.mark.parametrize("sizes", GROUPS)
def test_default_shapes_match_separate_launches(sizes, prec, tol):
    flows = [cases.natural_cavity(mi, nj, Ra=1e4, T0=0.5) for mi, nj in sizes]
    out = []
    for explicit in (False, True):
        bt = Batch.from_cases(flows, prec=prec, conv_paso=0.0)
        if explicit:
            for k in range(8):
                bt.set_sweep_shape(k, 2, 64)
        bt.iterate(6)
        out.append([inst.download() for inst in bt.instances])
        bt.close()
    for size, a, b in zip(sizes, *out):
        for k in ("u", "v", "p", "T"):
            assert np.max(np.abs(a[k] - b[k])) <= tol * max(np.max(np.abs(b[k])), 1.0), (size, k)
