"""The waits of the resident kernels' CTAs for one another, made to run out by
ixb_expire_grid_wait (each launch then expects one CTA more than it has, and
gives up at once; nothing faults or hangs).

CTAs that do not all start (which = 1): nothing has been written, and the call
goes on with the per-sweep kernels from where the last whole launch ended, so
its fields, counts and exits are those of an undisturbed call up to the
order of operations (1e-10 of a field's largest value, as test_parity_gpu.py
allows between solvers).

A wait between phases (which = 2): IXB_ETIMEOUT, no later launch of the call
runs, and the next call on a state uploaded again is bit for bit the
undisturbed one."""
import numpy as np
import pytest

from ixchel2d_b200 import IxbError, Simple2D, cases
from ixchel2d_b200 import _ffi as F
from tests.conftest import relerr

pytestmark = pytest.mark.gpu
COUNTS = ("n_simple", "n_momen", "n_pres", "n_ener", "exit_code")


@pytest.fixture(autouse=True)
def _need_gpu(has_gpu):
    if not has_gpu:
        pytest.skip("no CUDA device")


def _expire(s, which, start=0):
    assert F.lib.ixb_expire_grid_wait(s.h, which, start) == F.OK


CALLS = {
    "iterations": lambda s: s.iterations(30),
    "one": lambda s: s.iterations(1),
    "loop": lambda s: s.loop(),
    "steps": lambda s: [s.step() for _ in range(2)][-1],
    "converge": lambda s: s.converge(k0=2, k1=30, every=20, tol_dnu=0.0, max_iters=60),
    "energy": lambda s: s.energy_iterations(9) or {},
    "gradient": lambda s: {"grad": s.adjoint_energy(40, 2, 20)},
    "simple_gradient": lambda s: {"grad": s.adjoint_simple(6, 3, 2, 20)[0]},
}
INNER = dict(conv_u=2e-3, conv_p=5e-3, conv_t=1e-3, iter_ecuaci_max=3, iter_simple_max=12, conv_paso=0.0,
             conv_resi=0.0, dt=0.5)


def _run(call, which=0, start=0, over=INNER, mi=40, nj=36):
    with Simple2D.from_case(cases.natural_cavity(mi, nj, Ra=1e5), **over) as s:
        s.iterations(5)
        _expire(s, which, start)
        rep = call(s)
        return rep, s.download()


def _same(a, b):
    for k in COUNTS:
        assert a[0].get(k) == b[0].get(k), k
    for k in ("nu", "grad"):
        if k in a[0]:
            assert relerr(a[0][k], b[0][k]) < 1e-9, k
    for k in ("u", "v", "p", "T"):
        assert relerr(a[1][k], b[1][k]) < 1e-10, k


@pytest.mark.parametrize("host_driven", [False, True])
@pytest.mark.parametrize("name", CALLS)
def test_a_grid_that_does_not_start_is_done_by_sweeps(name, host_driven, monkeypatch):
    if host_driven:
        monkeypatch.setenv("IXB_NO_GRAPH", "1")
    _same(_run(CALLS[name]), _run(CALLS[name], which=1))


# launches of 2048 outer iterations (4096 energy passes): the first ones run, the rest is done by sweeps
@pytest.mark.parametrize("start", [1, 2, 3])
def test_the_rest_of_a_call_is_done_by_sweeps(start):
    over = dict(iter_ecuaci_max=0, conv_u=1e30, conv_p=1e30, conv_t=1e30)
    small = dict(over=over, mi=12, nj=10)
    _same(_run(lambda s: s.iterations(4500), **small), _run(lambda s: s.iterations(4500), 1, start, **small))
    watch = lambda s: s.converge(k0=2, k1=8, every=2100, tol_dnu=0.0, max_iters=4200)  # noqa: E731
    _same(_run(watch, **small), _run(watch, 1, start, **small))
    if start == 1:
        _same(_run(lambda s: s.energy_iterations(4100) or {}, **small),
              _run(lambda s: s.energy_iterations(4100) or {}, 1, start, **small))


@pytest.mark.parametrize("name", [k for k in CALLS if k != "one"])
def test_an_expired_wait_is_reported_and_the_next_call_is_clean(name):
    clean = _run(CALLS[name])
    with Simple2D.from_case(cases.natural_cavity(40, 36, Ra=1e5), **INNER) as s:
        s.iterations(5)
        state = s.download()
        _expire(s, 2)
        with pytest.raises(IxbError) as ei:
            CALLS[name](s)
        assert ei.value.status == F.ETIMEOUT
        _expire(s, 0)
        s.upload(state)
        s.set_params(**dict(cases.natural_cavity(40, 36, Ra=1e5).params, **INNER))
        rep = CALLS[name](s)
        end = s.download()
    for k in COUNTS:
        assert rep.get(k) == clean[0].get(k), k
    for k in ("u", "v", "p", "T"):
        assert np.array_equal(end[k], clean[1][k]), k


def test_no_launch_runs_behind_one_that_gave_up():
    # three launches are queued; the second gives up at its first wait, so the third must leave the fields alone:
    # what is left is the first 2048 iterations' p and T (the wait comes before anything but u is swept)
    over = dict(iter_ecuaci_max=0, conv_u=1e30, conv_p=1e30, conv_t=1e30)
    with Simple2D.from_case(cases.natural_cavity(12, 10, Ra=1e5), **over) as a:
        a.iterations(2048)
        want = a.download()
    with Simple2D.from_case(cases.natural_cavity(12, 10, Ra=1e5), **over) as s:
        _expire(s, 2, 1)
        with pytest.raises(IxbError) as ei:
            s.iterations(6000)
        assert ei.value.status == F.ETIMEOUT
        got = s.download()
    for k in ("u", "v", "p", "T"):
        assert np.array_equal(got[k], want[k]), k


def test_bad_arguments():
    with Simple2D.from_case(cases.natural_cavity(8, 8)) as s:
        for which, start in ((-1, 0), (3, 0), (1, -1)):
            assert F.lib.ixb_expire_grid_wait(s.h, which, start) == F.EINVAL
    assert F.lib.ixb_expire_grid_wait(None, 0, 0) == F.EINVAL
