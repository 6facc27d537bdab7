"""Gradient of the coupled iteration on grids whose lines fall on either side
of the reversed sweeps' chunk rules (rows per thread, threads per line, lines
per CTA), with and without linearised sources, against central differences of
the forward run.

Three outer iterations; the difference step h = 1e-4 carries a truncation
error of order h^2 = 1e-8 and a rounding error of order 1e-14 / h = 1e-10 on
an objective of order one, whose derivative by one of up to 1100 wall values
is of order 1e-3: 1e-5 relative covers both."""
import numpy as np
import pytest

from ixchel2d_b200 import _ffi as F
from ixchel2d_b200 import cases
from ixchel2d_b200.simple import Simple2D

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _need_gpu(has_gpu):
    if not has_gpu:
        pytest.skip("no CUDA device")


def _sim(case, mi, nj, vals, sources):
    sim = Simple2D.from_case(case)
    sim.set_bc_values(F.VAR_T, 0, vals)
    if sources:
        for var, shape in ((F.VAR_U, (nj + 1, mi)), (F.VAR_V, (nj, mi + 1)), (F.VAR_T, (nj + 1, mi + 1))):
            y, x = np.mgrid[0:shape[0], 0:shape[1]]
            sim.set_sources(var, 0.01 * np.cos(0.3 * x + y), -0.2 - 0.1 * np.sin(0.2 * x - 0.5 * y))
    return sim


@pytest.mark.parametrize("mi, nj, sources", [(5, 6, False), (191, 10, True), (192, 192, False), (383, 14, True),
                                             (384, 12, False), (767, 8, False), (768, 10, True), (10, 384, False),
                                             (9, 1024, True), (8, 1030, False), (1100, 6, False)])
def test_gradient_matches_central_differences(mi, nj, sources):
    case = cases.natural_cavity(mi, nj, Ra=1e4, T0=0.5)
    j1 = nj - 2 if nj % 2 == 0 else nj - 3
    vals = 1.0 + 0.05 * np.sin(0.9 * np.arange(nj + 1))
    K = 3
    sim = _sim(case, mi, nj, vals, sources)
    g, _ = sim.adjoint_simple(K, 2, 2, j1)
    sim.close()
    assert np.all(np.isfinite(g))
    h = 1e-4
    for L in (3, nj // 2):
        nu = []
        for s in (h, -h):
            v = vals.copy()
            v[L - 1] += s
            f = _sim(case, mi, nj, v, sources)
            nu.append(f.adjoint_simple(K, 2, 2, j1, gradient=False)[1])
            f.close()
        fd = (nu[0] - nu[1]) / (2 * h)
        assert abs(g[L - 1] - fd) <= 1e-5 * abs(fd), (L, g[L - 1], fd)
