"""Device memory that stays mapped between calls: at most 32 MB after line
solves, nothing of a handle's gradients once it is destroyed, and nothing
after ixb_release_scratch.  (4 MB are left for what the driver itself
allocates meanwhile, beyond what the first calls make it load.)"""
import pytest

from ixchel2d_b200 import Simple2D, cases
from ixchel2d_b200 import _ffi as F

pytestmark = pytest.mark.gpu
MB = 1 << 20


@pytest.fixture(autouse=True)
def _need_gpu(has_gpu):
    if not has_gpu:
        pytest.skip("no CUDA device")


def _free():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def _solve(arrs, n, nsys, solver):
    import torch
    fn = F.lib.ixb_tridiag_f64
    st = fn(*[t.data_ptr() for t in arrs], n, nsys, 1, solver, torch.cuda.current_stream().cuda_stream)
    assert st == F.OK
    torch.cuda.synchronize()


@pytest.mark.parametrize("n,nsys,solver", [(4096, 4096, F.SOLVER_EXACT), (1500, 2700, F.SOLVER_EXACT),
                                           (4095, 4095, F.SOLVER_HYBRID), (30000, 900, F.SOLVER_HYBRID)])
def test_line_solves(n, nsys, solver):
    import torch
    arrs = [torch.ones(n * nsys, dtype=torch.float64, device="cuda") for _ in range(5)]
    arrs[1].fill_(4.0)
    _solve(arrs, 1100, 7, solver)  # loads the kernel
    assert F.lib.ixb_release_scratch() == F.OK
    before = _free()
    for _ in range(3):
        _solve(arrs, n, nsys, solver)
    assert before - _free() <= 36 * MB
    assert F.lib.ixb_release_scratch() == F.OK
    assert before - _free() <= 4 * MB


def test_gradients():
    def grads(n):
        with Simple2D.from_case(cases.natural_cavity(n, n, Ra=1e4)) as s:
            s.energy_iterations(8)
            s.adjoint_simple(6, 3, 2, 20)
            s.adjoint_energy(12, 2, 20)

    grads(128)  # loads the kernels
    assert F.lib.ixb_release_scratch() == F.OK
    before = _free()
    grads(256)
    assert before - _free() <= 4 * MB
