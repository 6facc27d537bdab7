"""Solutions that decay along a line keep their small components, and a value
that is not a number reaches the whole line.

The rows are those of a diagonally dominant M-matrix with a right-hand side of
one sign, so neither the sequential elimination nor the partitioned solve with
cyclic reduction subtracts anything: every component of either is right to
rounding of itself.  Per row of decay each does a handful of operations, so a
component some r rows from the source differs by at most about 8 r roundings
between the two: r <= 1600 rows reach the end of binary64's range at the
slower decay used here (0.64 per row), 8 * 1600 * 1.1e-16 = 1.4e-12; in
binary32 r <= 160 rows reach 1e-30, 8 * 160 * 6e-8 = 8e-5.  The sweeps'
coefficients carry roundings of the velocities besides: 1e-9 and 1e-3
there.  A tail that is lost has an error of one."""
import numpy as np
import pytest

from ixchel2d_b200 import Batch, Simple2D, cases
from ixchel2d_b200 import _ffi as F
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _need_gpu(has_gpu):
    if not has_gpu:
        pytest.skip("no CUDA device")


def _worst(x, ref, floor):
    """Largest error of a component relative to itself, where |ref| > floor."""
    big = np.abs(ref) > floor
    assert big.any()
    return float(np.max(np.abs(x[big] - ref[big]) / np.abs(ref[big])))


def _solve(a, b, c, d, layout, dtype):
    import torch
    tdt = torch.float64 if dtype == "f64" else torch.float32
    fn = F.lib.ixb_tridiag_f64 if dtype == "f64" else F.lib.ixb_tridiag_f32
    nsys, n = d.shape
    dev = [torch.tensor(np.ascontiguousarray(v if layout == 0 else v.T), dtype=tdt, device="cuda")
           for v in (a, b, c, d, np.full_like(d, np.nan))]
    st = fn(*[t.data_ptr() for t in dev], n, nsys, layout, F.SOLVER_HYBRID, torch.cuda.current_stream().cuda_stream)
    assert st == F.OK
    torch.cuda.synchronize()
    assert F.lib.ixb_tridiag_status() == F.OK
    x = dev[4].cpu().numpy().astype(np.float64)
    return x if layout == 0 else x.T


# every kernel of the two layouts: streamed lines (aligned, ragged), one staged line per CTA, whole systems in
# registers, both cluster configurations, blocks of rows
LINES = [(0, 96, 8), (0, 301, 9), (0, 701, 8), (0, 1024, 6), (0, 4096, 4), (0, 4863, 3), (0, 6001, 2), (1, 63, 8),
         (1, 302, 33), (1, 512, 4800), (1, 1000, 9), (1, 1024, 4800), (1, 520, 9600), (1, 2048, 16), (1, 1153, 7), (1, 4100, 8)]


@pytest.mark.parametrize("dtype", ["f64", "f32"])
@pytest.mark.parametrize("layout,n,nsys", LINES)
def test_decaying_lines_componentwise(layout, n, nsys, dtype):
    a = np.full((nsys, n), -1.0)
    c = a.copy()
    b = np.full((nsys, n), 2.2)
    b[1::2] = 4.0
    d = np.zeros((nsys, n))
    for s in range(nsys):  # one row is the source: the first, the last, one in between
        d[s, (0, n - 1, n // 3)[s % 3]] = 1.0
    if dtype == "f32":
        b = b.astype(np.float32).astype(np.float64)  # the rows the solve is given
    x, ref = _solve(a, b, c, d, layout, dtype), O.tridiagonal_batch(a, b, c, d)
    floor, tol = (1e-290, 1.4e-12) if dtype == "f64" else (1e-30, 8e-5)
    assert _worst(x, ref, floor) < tol


@pytest.mark.parametrize("dtype", ["f64", "f32"])
@pytest.mark.parametrize("layout,n,nsys", LINES)
def test_nan_reaches_the_whole_line(layout, n, nsys, dtype):
    a = np.full((nsys, n), -1.0)
    b = np.full((nsys, n), 4.0)
    d = np.ones((nsys, n))
    d[1, n // 2] = np.nan
    x = _solve(a, b, a, d, layout, dtype)
    assert np.isnan(x[1]).all()
    assert np.isfinite(np.delete(x, 1, axis=0)).all()


def _cold(mi, nj):
    # a cavity at rest and cold, its hot wall switched on: T falls by a factor of about three per column
    return cases.natural_cavity(mi, nj, Ra=1e4, T0=0.0, dt=0.4 / max(mi, nj))


@pytest.mark.parametrize("prec", [F.PREC_FP64, F.PREC_FP32_REFINED])
@pytest.mark.parametrize("route", ["default", "shapes", "batch"])
@pytest.mark.parametrize("mi,nj", [(64, 40), (192, 30), (380, 24), (700, 12), (900, 20)])
def test_decaying_sweeps_componentwise(mi, nj, route, prec):
    case = _cold(mi, nj)
    o = O.OracleCase(case)
    o.iterations(1)
    ref = o.get_state()["T"]
    if route == "batch":
        with Batch.from_cases([case, _cold(24, 24)], prec=prec, conv_paso=0.0) as bt:
            bt.iterate(1)
            T = bt[0].download()["T"]
    else:
        with Simple2D.from_case(case, prec=prec) as g:
            if route == "shapes":  # the graph of single sweeps, assembly and solve apart
                for k in range(8):
                    g.set_sweep_shape(k, 2, 64)
            g.iterations(1)
            T = g.download()["T"]
    floor, tol = (1e-280, 1e-9) if prec == F.PREC_FP64 else (1e-30, 1e-3)
    assert _worst(T, ref, floor) < tol


@pytest.mark.parametrize("n", [64, 200, 300, 500])
@pytest.mark.parametrize("passes", [1, 6])
def test_decaying_energy_passes_componentwise(n, passes):
    case = _cold(n, n)
    o = O.OracleCase(case)
    o.energy_passes(passes)
    ref = o.get_state()["T"]
    with Simple2D.from_case(case) as g:
        g.energy_iterations(passes)
        T = g.download()["T"]
    assert _worst(T, ref, 1e-280) < 1e-9


@pytest.mark.parametrize("passes", [1, 6])
@pytest.mark.parametrize("n", [64, 300, 500])
def test_decaying_gradient_componentwise(n, passes):
    # the passes are affine in the wall values, so from a cold cavity d Nu / d value(jj) is Nu with the wall
    # value 1 at jj and 0 elsewhere; the panels are at the foot of the wall, the values further and further up
    case = _cold(n, n)
    with Simple2D.from_case(case) as g:
        grad = g.adjoint_energy(passes, 2, 4)
    far = [1, 5, 20, n // 4, n // 2]
    ref = []
    for j in far:
        o = O.OracleCase(case)
        e = np.zeros(n + 1)
        e[j] = 1.0
        o.set_bc_values(F.VAR_T, 0, e)
        o.energy_passes(passes)
        ref.append(o.nusselt_x(2, 4)[0])
    assert _worst(grad[far], np.array(ref), 1e-280) < 1e-9
