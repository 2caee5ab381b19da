"""Diagonal and internal force over the lattice colours, whose lanes add a whole
line of nodes with plain loads and stores: against the atomic scatter of the
same kernels, constrained rows, and bit for bit from call to call, on boxes of
one cell, of rows that end inside a warp's cells, and a few hundred cells.  Both
sum the same at most 8 contributions of a node in another order: 8 roundings of
the largest entry, 1e-15 and 5e-7 a piece at most, so 1e-14 and 4e-6.
"""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import numpy as np  # noqa: E402

import lsmf  # noqa: E402
from test_gpu_operator import VARIANTS  # noqa: E402

BOXES = [(1, 1, 1), (1, 2, 5), (7, 5, 3), (8, 8, 8)]


@pytest.mark.parametrize("caching,formulation", VARIANTS)
@pytest.mark.parametrize("p", [1, 2, 3, 4])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_diagonal(caching, formulation, p, precision):
    rng = np.random.default_rng(5)
    for cells in BOXES:
        mesh = lsmf.Mesh("box", cells, 0, degree=p)
        mesh.set_dirichlet([(4, 7), (1, 2)])
        nc, _, nd = mesh.info()
        op = lsmf.NeoHookOperator(mesh, caching, formulation, precision)
        op.set_material(rng.choice([1.0, 10.0], nc), 0.3)
        op.cache(torch.tensor(rng.uniform(-0.001, 0.001, nd), device="cuda").to(op.dtype))
        got = {}
        for mode in ("atomic", "colour8", "nodesum", "colour8"):
            op.set_scatter(mode)
            op.compute_diagonal()
            d = op.get_matrix_diagonal()
            assert mode not in got or torch.equal(d, got[mode])
            got[mode] = d
        assert torch.equal(got["colour8"], got["nodesum"])
        con = torch.tensor(mesh.constraint_mask(), device="cuda") != 0
        assert (got["colour8"][con] == 1).all()
        err = float((got["colour8"] - got["atomic"]).abs().max() / got["atomic"].abs().max())
        assert err < (1e-14 if precision == "fp64" else 4e-6), (cells, err)


def _prm(cells, p, formulation, scatter):
    return "\n".join([
        "subsection Finite element system", "set Polynomial degree = %d" % p, "set Quadrature order = %d" % (p + 1), "end",
        "subsection Geometry", "set Dimension = 3", "set Type = Box", "set Box cells = %d, %d, %d" % cells,
        "set Global refinement = 0", "end",
        "subsection Material properties", "set Shear modulus = 1.0", "set Poisson's ratio = 0.3",
        "set Formulation = %d" % formulation, "end",
        "subsection Linear solver", "set Solver type = MF_CG", "set Preconditioner type = jacobi",
        "set MF caching = scalar", "set MF scatter = " + scatter, "end",
        "subsection Boundary conditions", "set Dirichlet IDs and expressions = 4:0,0,0",
        "set Dirichlet IDs and component mask = 4:true,true,true",
        "set Neumann IDs and expressions = 5:0.02*t,0,-0.05*t", "end",
        "subsection Time", "set End time = 1", "set Time step size = 1", "end"]) + "\n"


@pytest.mark.parametrize("formulation", [0, 1])
@pytest.mark.parametrize("p", [1, 2, 3, 4])
def test_internal_force(p, formulation):
    rng = np.random.default_rng(6)
    for cells in BOXES:
        mu = u = None
        R = {}
        for mode in ("atomic", "colour8", "colour8"):
            pb = lsmf.Problem(_prm(cells, p, formulation, mode))
            if mu is None:
                mu = rng.choice([1.0, 10.0], pb.n_cells)
                u = torch.tensor(rng.uniform(-0.001, 0.001, pb.n_dofs), device="cuda")
            pb.set_mu(mu)
            r = torch.full_like(u, float("nan"))
            pb.residual(u, 1.0, r)
            assert mode not in R or torch.equal(r, R[mode])
            R[mode] = r
        err = float((R["colour8"] - R["atomic"]).abs().max() / R["atomic"].abs().max())
        # entries are differences of contributions up to some 10 times their size
        assert err < 1e-13, (cells, err)
