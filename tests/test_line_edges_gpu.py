"""Line solves of the sweeps at the edges of their partition: line lengths
just below, at and above a full set of three-row chunks (64, 128 and 256
threads per line), the first lengths with longer chunks, and the smallest
grids.  Binary64 against the CPU oracle with the tolerance of
test_parity_gpu.py (1e-10 of the field's largest value); the refined form
against the same oracle with its documented distance before convergence
(1e-4 relative L2, test_parity_headline_gpu.py)."""
import numpy as np
import pytest

from ixchel2d_b200 import Simple2D, cases
from ixchel2d_b200 import _ffi as F
from oracle import oracle as O
from tests.conftest import relerr

pytestmark = pytest.mark.gpu

# (mi, nj): x-lines have mi or mi+1 rows, y-lines nj or nj+1
SIZES = [(4, 4), (5, 4), (4, 7), (33, 31), (95, 6), (96, 5), (191, 6), (192, 9), (193, 7), (6, 159), (7, 160),
         (5, 192), (383, 5), (384, 6), (386, 7), (6, 383), (5, 386), (767, 6), (768, 5), (770, 7), (13, 770)]


@pytest.mark.parametrize("mi,nj", SIZES)
@pytest.mark.parametrize("prec", [F.PREC_FP64, F.PREC_FP32_REFINED])
def test_partition_edges(has_gpu, mi, nj, prec):
    if not has_gpu:
        pytest.skip("no CUDA device")
    case = cases.lid_driven_mixed(mi, nj, Re=100.0, Ri=0.5)
    o = O.OracleCase(case)
    o.iterations(8)
    with Simple2D.from_case(case, prec=prec) as g:
        g.iterations(8)
        gs = g.download()
    os_ = o.get_state()
    for k in ("u", "v", "p", "T"):
        if prec == F.PREC_FP64:
            assert relerr(gs[k], os_[k]) < 1e-10, (k, relerr(gs[k], os_[k]))
        elif k != "p":
            d = np.linalg.norm(gs[k] - os_[k]) / max(np.linalg.norm(os_[k]), 1e-300)
            assert d < 1e-4, (k, d)


# lines beyond the resident loop's: chunks of 4 to 9 rows, and grids whose y-lines come 4, 5, 6 or 8 per CTA
LONG = [(1023, 6), (1025, 5), (1280, 7), (1281, 6), (1536, 5), (1537, 6), (1700, 4), (6, 512), (7, 513), (6, 641),
        (5, 768), (6, 896), (7, 1024), (6, 1025), (700, 400), (820, 500), (900, 390), (1250, 400)]


@pytest.mark.parametrize("mi,nj", LONG)
@pytest.mark.parametrize("prec", [F.PREC_FP64, F.PREC_FP32_REFINED])
def test_longer_lines(has_gpu, mi, nj, prec):
    test_partition_edges(has_gpu, mi, nj, prec)


# batched line solves (device pointers): unaligned starts and ends (odd n, arrays that begin inside a
# 16-byte granule), the edges of the chunk sizes and of the 128-row blocks, ragged system groups, one
# system; x must be written everywhere and nothing beside it
LINES = [(1, 3), (2, 1), (31, 7), (96, 5), (97, 300), (160, 2), (161, 33), (320, 3), (321, 17), (641, 9), (701, 302),
         (1281, 5), (4863, 2), (4865, 3), (512, 37), (513, 37), (256, 4800), (257, 2411), (512, 2500), (1024, 15),
         (1025, 15), (1025, 1), (1150, 2500), (1152, 33), (2049, 31), (4096, 17), (4097, 70), (9000, 3)]


@pytest.mark.parametrize("dtype", ["f64", "f32"])
@pytest.mark.parametrize("layout", [0, 1])
@pytest.mark.parametrize("n,nsys", LINES)
def test_batched_lines_any_alignment(has_gpu, n, nsys, layout, dtype):
    if not has_gpu:
        pytest.skip("no CUDA device")
    import torch
    tdt = torch.float64 if dtype == "f64" else torch.float32
    fn = F.lib.ixb_tridiag_f64 if dtype == "f64" else F.lib.ixb_tridiag_f32
    rng = np.random.default_rng(n + 31 * nsys + layout)
    a = rng.uniform(-1, 0, (nsys, n)); c = rng.uniform(-1, 0, (nsys, n))
    b = np.abs(a) + np.abs(c) + rng.uniform(0.1, 1, (nsys, n)); d = rng.uniform(-1, 1, (nsys, n))
    ref = O.tridiagonal_batch(a, b, c, d)
    stream = torch.cuda.current_stream().cuda_stream
    for shift in ((0, 0, 0, 0, 0), (1, 0, 2, 3, 1)):  # elements each array starts past an aligned address
        dev = []
        for v, s in zip((a, b, c, d, np.full_like(d, np.nan)), shift):
            flat = torch.full((n * nsys + 8,), -7.0, dtype=tdt, device="cuda")
            flat[s:s + n * nsys] = torch.tensor(np.ascontiguousarray(v if layout == 0 else v.T).ravel(), dtype=tdt)
            dev.append(flat)
        ptr = [t.data_ptr() + s * t.element_size() for t, s in zip(dev, shift)]
        if shift[0]:
            ptr[4] = ptr[3]  # in place: x may alias d
        st = fn(*ptr, n, nsys, layout, F.SOLVER_HYBRID, stream)
        if n == 9000 and layout == 0 and dtype == "f64":  # a contiguous line must fit one CTA's shared memory
            assert st == F.EINVAL
            return
        assert st == F.OK
        out, s = (dev[3], shift[3]) if shift[0] else (dev[4], shift[4])
        torch.cuda.synchronize()
        assert F.lib.ixb_tridiag_status() == F.OK
        got = out.cpu().numpy().astype(np.float64)
        assert np.all(got[:s] == -7.0) and np.all(got[s + n * nsys:] == -7.0)
        x = got[s:s + n * nsys].reshape((nsys, n) if layout == 0 else (n, nsys))
        x = x if layout == 0 else x.T
        assert relerr(x, ref) < (1e-12 if dtype == "f64" else 2e-5), relerr(x, ref)


# interleaved systems in thread-block clusters: the row limits of the two configurations and of their cluster
# sizes, a last group that is not full, several groups per cluster
@pytest.mark.parametrize("dtype", ["f64", "f32"])
@pytest.mark.parametrize("n,nsys", [(513, 36), (1024, 2052), (1025, 64), (2048, 2500), (2049, 16), (3000, 8),
                                    (4096, 40), (4096, 1036)])
def test_interleaved_lines_in_clusters(has_gpu, n, nsys, dtype):
    test_batched_lines_any_alignment(has_gpu, n, nsys, 1, dtype)
