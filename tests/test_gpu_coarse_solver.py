"""The coarse-level Chebyshev iteration as one cooperative kernel (cells and
nodes of a level spread over the CTAs, sums of shared nodes exchanged every
step) against the launch-per-step form, which a level operator with the basic
kernel keeps: V-cycles of every variant, degrees 1-3, one and many CTAs,
ragged sizes and voids.  Tolerances: those of the V-cycle parity tests, 1e-10
(FP64 levels) and 1e-4 (FP32 levels).
"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import lsmf  # noqa: E402
import oracle as O  # noqa: E402
from test_gpu_operator import VARIANTS  # noqa: E402

BASIC, WAIT_TRIES = 2, 4


def _setup(p, coarse, level, caching, formulation, precision, voids=False, seed=3):
    act = O.void_mask(coarse, 3, 0.2, 5) if voids else None
    gm = lsmf.Mesh("box", coarse, level, degree=p, coarse_active=act)
    gm.set_dirichlet([(4, 7), (1, 2)])
    nc, _, nd = gm.info()
    X = gm.arrays()[0]
    rng = np.random.default_rng(seed)
    mu = np.exp(0.3 * rng.normal(size=nc))
    u = torch.tensor((0.002 * np.sin(np.pi * X[:, [1, 2, 0]])).reshape(-1), device="cuda")
    b = torch.tensor(np.where(gm.constraint_mask() == 1, 0.0, rng.uniform(-1, 1, nd)), device="cuda")
    g = lsmf.GMG(gm, caching, formulation, precision)
    g.set_material(mu, 0.3)
    return gm, g, mu, u, b


def _vcycle(g, b):
    x = torch.full_like(b, float("nan"))
    g.vmult(x, b)
    torch.cuda.synchronize()
    return x


def _compare(args, precision):
    gm, g, mu, u, b = args
    g.setup(u)
    one = _vcycle(g, b)
    g.level_option(0, BASIC, 1)
    steps = _vcycle(g, b)
    err = (torch.max(torch.abs(one - steps)) / torch.max(torch.abs(steps))).item()
    assert err < (1e-10 if precision == "fp64" else 1e-4), err
    assert g.level_info(0)[2] >= 4  # the coarse degree: both forms iterated


@pytest.mark.parametrize("caching,formulation", VARIANTS)
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_variants(caching, formulation, precision):
    _compare(_setup(2, (5, 4, 3), 1, caching, formulation, precision), precision)


@pytest.mark.parametrize("p,coarse", [(1, (3, 2, 2)), (1, (13, 11, 7)), (2, (1, 1, 1)), (2, (7, 1, 1)), (2, (15, 15, 15)),
                                      (3, (3, 3, 2)), (3, (7, 6, 5)), (4, (3, 2, 2))])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_sizes(p, coarse, precision):
    _compare(_setup(p, coarse, 1 if coarse != (15, 15, 15) else 0, "tensor4", 1, precision), precision)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_voids(precision):
    _compare(_setup(2, (6, 6, 6), 1, "tensor4", 1, precision, voids=True), precision)


def test_one_level_solve_is_reproducible():
    gm, g, mu, u, b = _setup(2, (6, 5, 4), 0, "tensor4", 1, "fp32")
    g.set_scatter("colour8")
    g.setup(u)
    assert torch.equal(_vcycle(g, b), _vcycle(g, b))


def test_run_out_wait_is_reported_and_recovers():
    gm, g, mu, u, b = _setup(2, (8, 8, 8), 0, "tensor4", 1, "fp64")
    op = lsmf.NeoHookOperator(gm, "tensor4", 1, "fp64")
    op.set_material(mu, 0.3)
    op.cache(u)
    g.setup(u)
    x = torch.zeros_like(b)
    g.level_option(0, WAIT_TRIES, 0)
    with pytest.raises(lsmf.LsmfError) as e:
        lsmf.cg_solve(op, x, b, 1e-8 * float(b.norm()), 3, "gmg", g)
    assert e.value.status == 8
    g.level_option(0, WAIT_TRIES, -1)
    x.zero_()
    assert lsmf.cg_solve(op, x, b, 1e-8 * float(b.norm()), 100, "gmg", g)["converged"]


@pytest.mark.parametrize("caching,formulation", VARIANTS)
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_eigenvalue_estimate(caching, formulation, precision):
    # the estimate's CG as one kernel against the launch-per-iteration form:
    # the tolerances of the estimates' parity tests (1e-9 / 2e-3), equal degrees
    gm, g, mu, u, b = _setup(2, (5, 4, 3), 0, caching, formulation, precision)
    g.setup(u)
    one = g.level_info(0)
    g.level_option(0, BASIC, 1)
    g.setup(u)
    steps = g.level_info(0)
    tol = 1e-9 if precision == "fp64" else 2e-3
    assert np.allclose(one[:2], steps[:2], rtol=tol, atol=0), (one, steps)
    assert one[2] == steps[2]
    assert abs(one[5] - steps[5]) <= 0.05 * steps[5]
