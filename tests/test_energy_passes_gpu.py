"""The resident energy passes against the same passes as single sweeps (a
launch shape set by the caller keeps them): the chunk edges of both
directions, one to three lines per CTA, sources, and wall types.  Both run in
binary64 and differ in the order of operations only: 1e-12 of the largest
temperature after nine passes."""
import numpy as np
import pytest

from ixchel2d_b200 import _ffi as F
from ixchel2d_b200 import cases
from ixchel2d_b200.simple import Simple2D

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("flow", [cases.natural_cavity, cases.lid_driven_mixed])
@pytest.mark.parametrize("mi, nj", [(4, 4), (5, 9), (95, 96), (96, 97), (149, 150), (150, 148), (298, 299), (444, 444),
                                    (767, 12), (12, 767), (700, 60)])
def test_resident_passes_match_single_sweeps(has_gpu, flow, mi, nj):
    if not has_gpu:
        pytest.skip("no CUDA device")
    out = []
    for single in (False, True):
        with Simple2D.from_case(flow(mi, nj)) as s:
            s.iterations(4)
            y, x = np.mgrid[0:nj + 1, 0:mi + 1]
            s.set_sources(F.VAR_T, 0.01 * np.cos(0.3 * x + y), -0.2 - 0.1 * np.sin(0.2 * x - 0.5 * y))
            s.set_bc_values(F.VAR_T, 0, 1.0 + 0.1 * np.sin(0.4 * np.arange(nj + 1)))
            if single:
                s.set_sweep_shape(6, 2, 64)
                s.set_sweep_shape(7, 2, 64)
            s.energy_iterations(9)
            s.energy_iterations(1)
            out.append(s.download())
    for k in ("u", "v", "p"):
        assert np.array_equal(out[0][k], out[1][k])
    assert np.max(np.abs(out[0]["T"] - out[1]["T"])) <= 1e-12 * np.max(np.abs(out[1]["T"]))
