"""Which host arrays the state transfers may hand to a kernel: only those that
lie in one page-locked allocation or registration from end to end.  Nothing is
transferred here."""
import mmap

import numpy as np
import pytest

from ixchel2d_b200 import _ffi as F

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _need_gpu(has_gpu):
    if not has_gpu:
        pytest.skip("no CUDA device")
    import torch
    torch.zeros(1, device="cuda")


def test_allocations():
    import torch
    t = torch.empty(1 << 20, dtype=torch.uint8).pin_memory()
    p = t.data_ptr()
    assert F.lib.ixb_host_reachable(p, 1 << 20) == 1
    assert F.lib.ixb_host_reachable(p + 4096, (1 << 20) - 4096) == 1
    assert F.lib.ixb_host_reachable(p + (1 << 20) - 8, 8) == 1
    assert F.lib.ixb_host_reachable(p, 1 << 40) == 0
    assert F.lib.ixb_host_reachable(None, 8) == 0 and F.lib.ixb_host_reachable(p, 0) == 0
    a = np.empty(1000)
    assert F.lib.ixb_host_reachable(a.ctypes.data, a.nbytes) == 0


def test_registrations_with_a_gap():
    import torch
    rt = torch.cuda.cudart()
    page = 4096
    mem = mmap.mmap(-1, 6 * page)
    a = np.frombuffer(mem, dtype=np.uint8)
    p = a.ctypes.data
    assert p % page == 0
    reach = lambda first, pages: F.lib.ixb_host_reachable(p + first * page, pages * page)  # noqa: E731
    assert int(rt.cudaHostRegister(p, 2 * page, 0)) == 0
    assert int(rt.cudaHostRegister(p + 4 * page, 2 * page, 0)) == 0
    try:
        assert reach(0, 2) == 1 and reach(4, 2) == 1 and reach(5, 1) == 1
        assert reach(0, 6) == 0  # first and last byte are reachable, the middle is not
        assert reach(1, 2) == 0 and reach(2, 2) == 0
    finally:
        rt.cudaHostUnregister(p)
        rt.cudaHostUnregister(p + 4 * page)
    assert int(rt.cudaHostRegister(p, 6 * page, 0)) == 0
    try:
        assert reach(0, 6) == 1 and reach(1, 5) == 1
    finally:
        rt.cudaHostUnregister(p)
    assert reach(0, 6) == 0
