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
