"""Box meshes, where the cache tables and the internal force take one reference
Jacobian per cell from four of its corners: cells of three different side
lengths (an exchange of axes shows), degrees 1 to 4, against the oracle, which
evaluates the coordinates at every quadrature point.  Tolerances: 1e-13 for
the metric table, as in test_gpu_line_kernels.py, and 1e-12 for the residual,
as in test_gpu_residual.py (relative, max norm).
"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import lsmf  # noqa: E402
import oracle as O  # noqa: E402
from prm_util import prm_text  # noqa: E402
from test_gpu_operator import VARIANTS, _rel  # noqa: E402

CELLS = (2, 3, 5)


def _state(om, rng):
    return rng.uniform(-0.002, 0.002, om.n_dofs), rng.choice([1.0, 10.0], om.n_cells)


@pytest.mark.parametrize("caching,formulation", VARIANTS)
@pytest.mark.parametrize("p", [1, 2, 3, 4])
def test_tables(caching, formulation, p):
    gm = lsmf.Mesh("box", CELLS, 0, hi=(1.0, 0.6, 2.5), degree=p)
    om = O.Mesh(O.GEOM_BOX, CELLS, 0, (0, 0, 0), (1.0, 0.6, 2.5), 1.0, p, p + 1)
    u, mu = _state(om, np.random.default_rng(3))
    ref = O.Operator(om, caching, formulation)
    ref.set_material(mu, 0.3)
    ref.set_constraints(np.zeros(om.n_dofs, dtype=np.uint8))
    assert ref.cache(u) == 0
    op = lsmf.NeoHookOperator(gm, caching, formulation, "fp64")
    op.set_material(mu, 0.3)
    op.cache(torch.tensor(u, device="cuda"))
    assert _rel(op.table(4), ref.table(4)) < 1e-13
    src = np.random.default_rng(4).uniform(-1, 1, om.n_dofs)
    dst = torch.empty(om.n_dofs, dtype=torch.float64, device="cuda")
    op.vmult(dst, torch.tensor(src, device="cuda"))
    assert _rel(dst.cpu().numpy(), ref.vmult(src)) < 1e-10


@pytest.mark.parametrize("formulation", [0, 1])
@pytest.mark.parametrize("p", [1, 2, 3, 4])
def test_internal_force(formulation, p):
    pb = lsmf.Problem(prm_text({
        "Polynomial degree": p, "Quadrature order": p + 1, "Dimension": 3, "Type": "Box",
        "Box cells": "%d, %d, %d" % CELLS, "Poisson's ratio": 0.3, "Shear modulus": 1.0, "Formulation": formulation,
        "Solver type": "MF_CG", "Preconditioner type": "jacobi", "MF caching": "scalar",
        "Dirichlet IDs and expressions": "4:0,0,0", "Dirichlet IDs and component mask": "4:true,true,true",
        "Neumann IDs and expressions": "5:0,0,t"}))
    om = O.Mesh(O.GEOM_BOX, CELLS, 0, (0, 0, 0), (1, 1, 1), 1.0, p, p + 1)
    u, mu = _state(om, np.random.default_rng(5))
    cmask = om.constraints([(4, 7)])
    pb.set_mu(mu)
    want, norm = O.residual(om, mu, 0.3, formulation, u, [(5, (0, 0, 0), (0, 0, 1))], 0.05, cmask)
    R = torch.full((om.n_dofs,), 3.0, dtype=torch.float64, device="cuda")
    got_norm = pb.residual(torch.tensor(u, device="cuda"), 0.05, R)
    assert np.max(np.abs(R.cpu().numpy() - want)) <= 1e-12 * np.max(np.abs(want))
    assert abs(got_norm - norm) <= 1e-12 * norm
