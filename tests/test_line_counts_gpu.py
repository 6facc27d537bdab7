"""The largest number of systems a line solve takes, 2^31 - 1, of one row each."""
import pytest

from ixchel2d_b200 import _ffi as F

pytestmark = pytest.mark.gpu


def test_contiguous_lines_up_to_the_last_count(has_gpu):
    if not has_gpu:
        pytest.skip("no CUDA device")
    import torch
    nsys = (1 << 31) - 1
    rows = torch.full((nsys,), 2.0, dtype=torch.float32, device="cuda")  # a, b and c: the first and the last are not read
    x = torch.full((nsys,), 3.0, dtype=torch.float32, device="cuda")
    x[-1] = 5.0
    p = rows.data_ptr()
    st = F.lib.ixb_tridiag_f32(p, p, p, x.data_ptr(), x.data_ptr(), 1, nsys, 0, F.SOLVER_HYBRID,
                               torch.cuda.current_stream().cuda_stream)
    assert st == F.OK
    torch.cuda.synchronize()
    assert F.lib.ixb_tridiag_status() == F.OK
    assert x[-1].item() == 2.5
    assert all(bool((part == 1.5).all()) for part in x[:-1].split(1 << 28))
    assert bool((rows[-1000:] == 2.0).all())
