"""Energy adjoint on grids whose lines fall on either side of the reversed
sweeps' chunk rules, against central differences of the forward passes.

With the flow fixed the objective is affine in the wall values, so
differences of step h = 1 are exact up to the rounding of an objective of
order 10 (1e-14) against a derivative of order 1 / (number of wall values):
1e-9 relative plus 1e-12 absolute."""
import numpy as np
import pytest

from ixchel2d_b200 import _ffi as F
from ixchel2d_b200 import cases
from ixchel2d_b200.simple import Simple2D

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mi, nj", [(4, 6), (191, 12), (192, 192), (383, 14), (384, 385), (767, 8), (768, 10),
                                    (1024, 6), (1536, 7), (1537, 6), (2048, 6), (8, 512), (9, 513), (6, 768),
                                    (7, 1023), (6, 1024), (5, 3071), (3072, 6)])
def test_gradient_matches_differences(has_gpu, mi, nj):
    if not has_gpu:
        pytest.skip("no CUDA device")
    case = cases.natural_cavity(mi, nj, Ra=1e4, T0=0.5)
    j1 = nj - 2 if nj % 2 == 0 else nj - 3
    vals = 1.0 + 0.05 * np.sin(0.7 * np.arange(nj + 1))
    K = 11  # a first pass, the loop graph, and what is left
    sim = Simple2D.from_case(case)
    sim.iterations(3)
    state = sim.download()
    sim.set_bc_values(F.VAR_T, 0, vals)
    g = sim.adjoint_energy(K, 2, j1)
    for L in (3, nj // 2):
        nu = []
        for h in (1.0, -1.0):
            v = vals.copy()
            v[L - 1] += h
            sim.upload(state)
            sim.set_bc_values(F.VAR_T, 0, v)
            sim.energy_iterations(K)
            nu.append(sim.nusselt_x(2, j1)[0])
        fd = 0.5 * (nu[0] - nu[1])
        assert abs(g[L - 1] - fd) <= 1e-9 * abs(fd) + 1e-12, (L, g[L - 1], fd)
    sim.close()
