"""A bounded copy wait that expires in the interleaved line solve's clusters
(see test_failure_gpu.py): every CTA records it, the cluster's CTAs stop
sending, their copies in flight land, nothing is written, and the next call
is clean.  Every wait ends: after a failure each CTA also waits, at the default
bound of about two seconds each, for rows and solutions that will not come."""
import numpy as np
import pytest

from ixchel2d_b200 import _ffi as F
from oracle import oracle as O
from tests.conftest import relerr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nsys", [(1024, 4800), (3000, 800)])  # both cluster configurations, several groups each
def test_expired_tile_wait_is_reported_and_the_next_call_is_clean(has_gpu, n, nsys):
    if not has_gpu:
        pytest.skip("no CUDA device")
    import torch
    rng = np.random.default_rng(n)
    a, c, d = (-rng.uniform(0, 1, (nsys, n)) for _ in range(3))
    b = np.abs(a) + np.abs(c) + rng.uniform(0.1, 1, (nsys, n))
    dev = [torch.tensor(np.ascontiguousarray(v.T), device="cuda") for v in (a, b, c, d, np.full_like(d, np.nan))]
    stream = torch.cuda.current_stream().cuda_stream

    def solve():
        assert F.lib.ixb_tridiag_f64(*[t.data_ptr() for t in dev], n, nsys, 1, F.SOLVER_HYBRID, stream) == F.OK
        return F.lib.ixb_tridiag_status()

    F.lib.ixb_tridiag_status()
    try:
        assert F.lib.ixb_tridiag_set_first_wait_limit(0) == F.OK
        assert solve() == F.ETIMEOUT
        assert torch.isnan(dev[4]).all().item()
    finally:
        assert F.lib.ixb_tridiag_set_first_wait_limit(-1) == F.OK
    assert solve() == F.OK
    assert relerr(dev[4].cpu().numpy().T, O.tridiagonal_batch(a, b, c, d)) < 1e-12
