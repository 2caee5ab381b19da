"""Bounded waits of the coarse-level kernels that run out (a wait bound of zero
polls: no wait is ever long): what the caller gets to see.  Nothing is
compared within a tolerance except solves that have to work again afterwards.
"""
import ctypes

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import lsmf  # noqa: E402
from test_gpu_coarse_solver import WAIT_TRIES, _setup, _vcycle  # noqa: E402

TIMEOUT = 8


def _problem(precision="fp64"):
    gm, g, mu, u, b = _setup(2, (8, 8, 8), 1, "tensor4", 1, precision)
    g.setup(u)
    op = lsmf.NeoHookOperator(gm, "tensor4", 1, "fp64")
    op.set_material(mu, 0.3)
    op.cache(u)
    return g, op, u, b


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_vcycle_of_a_run_out_wait_is_no_solution(precision):
    g, op, u, b = _problem(precision)
    good = _vcycle(g, b)
    g.level_option(0, WAIT_TRIES, 0)
    assert not torch.isfinite(_vcycle(g, b)).all()  # not the coarse solution of the call before
    g.level_option(0, WAIT_TRIES, -1)
    again = _vcycle(g, b)
    assert float((again - good).abs().max() / good.abs().max()) < (1e-10 if precision == "fp64" else 1e-4)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_solve_ends_with_the_first_run_out_wait(precision):
    g, op, u, b = _problem(precision)
    x, info = torch.zeros_like(b), lsmf.SolveInfo()
    g.level_option(0, WAIT_TRIES, 0)
    st = lsmf.lib().lsmf_cg_solve(op.h, 2, 1.0, g.h, lsmf._dptr(x), lsmf._dptr(b), 1e-8 * float(b.norm()), 50,
                                  ctypes.byref(info))
    assert st == TIMEOUT and info.iterations <= 1 and not info.converged
    g.level_option(0, WAIT_TRIES, -1)
    x.zero_()
    assert lsmf.cg_solve(op, x, b, 1e-8 * float(b.norm()), 100, "gmg", g)["converged"]


def test_sync_reports_a_vcycle_once():
    g, op, u, b = _problem()
    g.sync()
    g.level_option(0, WAIT_TRIES, 0)
    _vcycle(g, b)
    with pytest.raises(lsmf.LsmfError) as e:
        g.sync()
    assert e.value.status == TIMEOUT
    g.sync()


def test_setup_reports_the_vcycle_before_it():
    g, op, u, b = _problem()
    good = _vcycle(g, b)
    g.level_option(0, WAIT_TRIES, 0)
    _vcycle(g, b)
    g.level_option(0, WAIT_TRIES, -1)
    with pytest.raises(lsmf.LsmfError) as e:
        g.setup(u)
    assert e.value.status == TIMEOUT and "before this set-up" in str(e.value)
    again = _vcycle(g, b)  # the set-up was complete
    assert float((again - good).abs().max() / good.abs().max()) < 1e-10
    g.setup(u)
    g.sync()


def test_solve_tells_an_earlier_vcycle_from_its_own():
    g, op, u, b = _problem()
    g.level_option(0, WAIT_TRIES, 0)
    _vcycle(g, b)
    g.level_option(0, WAIT_TRIES, -1)
    x, info, tol = torch.zeros_like(b), lsmf.SolveInfo(), 1e-8 * float(b.norm())
    st = lsmf.lib().lsmf_cg_solve(op.h, 2, 1.0, g.h, lsmf._dptr(x), lsmf._dptr(b), tol, 100, ctypes.byref(info))
    assert st == TIMEOUT and b"before this solve" in lsmf.lib().lsmf_last_error()
    assert info.converged and info.residual <= tol
    r = torch.empty_like(b)
    op.vmult(r, x)
    assert float((r - b).norm()) <= 1.01 * tol
    x.zero_()
    assert lsmf.cg_solve(op, x, b, tol, 100, "gmg", g)["converged"]


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_estimate_of_a_run_out_wait_fails_the_setup(precision):
    gm, g, mu, u, b = _setup(2, (8, 8, 8), 0, "tensor4", 1, precision)
    for _ in range(5):
        g.level_option(0, WAIT_TRIES, 0)
        with pytest.raises(lsmf.LsmfError) as e:
            g.setup(u)
        assert e.value.status == TIMEOUT
    g.level_option(0, WAIT_TRIES, -1)
    g.setup(u)
    assert torch.isfinite(_vcycle(g, b)).all()
