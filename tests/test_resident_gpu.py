"""The resident loop over more launches than one, its Nusselt monitor, and the
tuned shapes of the per-sweep kernels, which grids it serves run only when a
caller sets them.

Runs that are cut differently into launches, and the host-driven loop, which
runs the same kernel part by part, agree bit for bit; oracle comparisons use
the tolerance of test_parity_gpu.py (1e-10 of a field's largest value)."""
import numpy as np
import pytest

from ixchel2d_b200 import IxbError, Simple2D, cases
from ixchel2d_b200 import _ffi as F
from oracle import oracle as O
from tests.conftest import relerr
from tests.test_monitor_gpu import _oracle_monitor

pytestmark = pytest.mark.gpu
STATE = ("u", "v", "p", "T")
ONE_PASS = dict(iter_ecuaci_max=0, conv_u=1e30, conv_p=1e30, conv_t=1e30)


@pytest.fixture(autouse=True)
def _need_gpu(has_gpu):
    if not has_gpu:
        pytest.skip("no CUDA device")


def _equal(a, b):
    for k in STATE:
        assert np.array_equal(a[k], b[k]), k


# a launch runs 2048 outer iterations; up to eight are queued at a time
@pytest.mark.parametrize("total", [2047, 2048, 2049, 4100, 16384, 16390])
def test_fixed_counts_over_launches(total):
    case = cases.natural_cavity(8, 7, Ra=1e4)
    with Simple2D.from_case(case, **ONE_PASS) as a, Simple2D.from_case(case, **ONE_PASS) as b:
        rep = a.iterations(total)
        assert [rep[k] for k in ("n_simple", "n_momen", "n_pres", "n_ener")] == [total] * 4
        left = total
        while left > 0:
            last = b.iterations(min(left, 1000))
            left -= 1000
        _equal(a.download(), b.download())
        assert rep["residuo"] == last["residuo"] and rep["maxbo"] == last["maxbo"]


@pytest.mark.parametrize("every,blocks", [(2048, 3), (2100, 4), (4097, 2)])
def test_monitor_blocks_over_launches(every, blocks):
    case = cases.natural_cavity(12, 10, Ra=1e4)
    with Simple2D.from_case(case, **ONE_PASS) as a, Simple2D.from_case(case, **ONE_PASS) as b:
        r = a.converge(k0=2, k1=8, every=every, tol_dnu=0.0, max_iters=every * blocks)
        assert r["exit_code"] == 5 and r["n_simple"] == every * blocks
        nus = []
        for _ in range(blocks):
            b.iterations(every)
            nus.append(b.nusselt_x(2, 8))
        _equal(a.download(), b.download())
        assert r["nu"] == nus[-1] and r["dnu"] == abs(nus[-1][0] - nus[-2][0])


def test_loop_over_launches():
    # to the exit test at its iteration limit, beyond one launch
    case = cases.natural_cavity(8, 7, Ra=1e4)
    over = dict(ONE_PASS, iter_simple_max=3000, conv_paso=0.0, conv_resi=0.0)
    with Simple2D.from_case(case, **over) as a, Simple2D.from_case(case, **over) as b:
        r = a.loop()
        assert r["exit_code"] == 2 and r["n_simple"] == 3002
        b.iterations(3002)
        _equal(a.download(), b.download())


def test_energy_passes_over_launches():
    # a launch runs 4096 passes
    case = cases.natural_cavity(20, 16, Ra=1e4)
    with Simple2D.from_case(case) as a, Simple2D.from_case(case) as b:
        for s in (a, b):
            s.iterations(30)
        a.energy_iterations(4100)
        b.energy_iterations(4096)
        b.energy_iterations(4)
        _equal(a.download(), b.download())


def test_gradient_over_launches():
    case = cases.natural_cavity(20, 16, Ra=1e4)
    with Simple2D.from_case(case) as s:
        s.iterations(30)
        g = s.adjoint_energy(4200, 2, 14)
        assert F.lib.ixb_expire_grid_wait(s.h, 1, 0) == F.OK  # the same passes as single kernels
        h = s.adjoint_energy(4200, 2, 14)
    assert relerr(g, h) < 1e-9


MONITORS = [(dict(k0=2, k1=30, vertical=True, wall=0, every=50, tol_dnu=1e-6, tol_maxbo=0.0), 3),
            (dict(k0=2, k1=30, vertical=True, wall=1, every=36, tol_dnu=1e-6, tol_maxbo=0.0), 3),
            (dict(k0=3, k1=29, vertical=False, wall=1, every=40, tol_dnu=0.0, tol_maxbo=1e-3), 4)]


@pytest.mark.parametrize("kw,code", MONITORS)
def test_hybrid_monitor_exits(kw, code, monkeypatch):
    case = cases.natural_cavity(32, 32, Ra=1e4, T0=0.5) if code == 3 else cases.lid_driven_mixed(32, 29, Re=100.0, Ri=1.0)
    with Simple2D.from_case(case) as g:
        assert g.iteration_launches() == 0  # the resident kernel
        r = g.converge(max_iters=40000, **kw)
        end = g.download()
        assert r["exit_code"] == code
        assert (g.nusselt_x if kw["vertical"] else g.nusselt_y)(kw["k0"], kw["k1"]) == r["nu"]
    # the host-driven loop: the same rule on the host, between parts of the same kernel
    monkeypatch.setenv("IXB_NO_GRAPH", "1")
    with Simple2D.from_case(case) as h:
        q = h.converge(max_iters=40000, **kw)
        _equal(end, h.download())
    for k in ("exit_code", "n_simple", "n_momen", "n_pres", "n_ener", "nu", "dnu", "maxbo"):
        assert r[k] == q[k], k
    # and the oracle stops where it does, with its fields
    o = O.OracleCase(case)
    its, ocode, nu, _ = _oracle_monitor(o, **dict(kw, max_iters=40000))
    assert (its, ocode) == (r["n_simple"], code) and relerr(r["nu"], nu) < 1e-9
    os_ = o.get_state()
    for k in STATE:
        assert relerr(end[k], os_[k]) < 1e-9, k


@pytest.mark.parametrize("prec", [F.PREC_FP64, F.PREC_FP32_REFINED])
def test_tuned_shapes_run_when_set(prec):
    case = cases.natural_cavity(40, 36, Ra=1e5)
    with Simple2D.from_case(case, prec=prec) as g:
        assert g.iteration_launches() == 0
        names = list(g.autotune(reps=2).values())
        for k, chosen in enumerate(names):
            g.set_sweep_shape(k, chosen[0], chosen[1])
        assert g.iteration_launches() > 0  # single sweeps from here on
        g.iterations(80)
        gs = g.download()
    o = O.OracleCase(case)
    o.iterations(80)
    os_ = o.get_state()
    for k in STATE:
        if prec == F.PREC_FP64:
            assert relerr(gs[k], os_[k]) < 1e-10, k
        elif k != "p":
            assert np.linalg.norm(gs[k] - os_[k]) < 1e-4 * np.linalg.norm(os_[k]), k


@pytest.mark.parametrize("nan", [np.nan, -np.nan])
@pytest.mark.parametrize("field", ["u", "v", "T"])
@pytest.mark.parametrize("route", ["resident", "sweeps"])
def test_not_a_number_of_either_sign_ends_the_run(route, field, nan):
    case = cases.natural_cavity(24, 20, Ra=1e4)
    with Simple2D.from_case(case) as s:
        s.iterations(3)
        state = s.download()
        state[field][11, 9] = nan
        assert np.signbit(state[field][11, 9]) == np.signbit(nan)
        s.upload(state)
        if route == "sweeps":
            s.set_sweep_shape(0, 4, 64)
        with pytest.raises(IxbError) as ei:
            s.iterations(5)
        assert ei.value.status == F.ENONFINITE
