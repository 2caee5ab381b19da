"""The surface load of the residual, formed on the device (expressions of
(x, y, z, t) evaluated at the face quadrature points, contributions summed per
node in face order), against a NumPy integration of the same expressions: two
conditions on three sides of a box, one of them on two sides, degrees 1 to 4.
At u = 0 the residual is the load.  Tolerance 1e-12 relative (max norm), as
for the residual's parity with the oracle; two calls agree bit for bit.
"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import lsmf  # noqa: E402
from prm_util import prm_text  # noqa: E402

TOP = ("sin(3*x)*y+t^2", "-exp(z)/(1+x)", "abs(x-0.5)*t-sqrt(1+y)")
SIDE = ("0.25*t", "tanh(y-z)", "-(x+2)^-1+pi*cos(z)")


def _top(x, y, z, t):
    return np.array([np.sin(3 * x) * y + t * t, -np.exp(z) / (1 + x), np.abs(x - 0.5) * t - np.sqrt(1 + y)])


def _side(x, y, z, t):
    return np.array([0.25 * t, np.tanh(y - z), -1 / (x + 2) + np.pi * np.cos(z)])


def _load(p, n, t):
    """Load vector of the unit box with n cells a side direction, lattice node order."""
    g, w = np.polynomial.legendre.leggauss(p + 1)
    g, w = 0.5 * (g + 1), 0.5 * w
    inner = {1: [], 2: [0.0], 3: [-np.sqrt(0.2), np.sqrt(0.2)], 4: [-np.sqrt(3 / 7), 0.0, np.sqrt(3 / 7)]}[p]
    nodes = np.array([0.0] + [0.5 * (1 + v) for v in inner] + [1.0])
    N = np.array([[np.prod([(q - nodes[j]) / (nodes[i] - nodes[j]) for j in range(p + 1) if j != i])
                   for i in range(p + 1)] for q in g])
    nn = [p * m + 1 for m in n]
    R = np.zeros((nn[2], nn[1], nn[0], 3))
    for axis, end, fun in ((2, 1, _top), (0, 1, _side), (1, 0, _side)):
        a, b = [d for d in range(3) if d != axis]
        for i in range(n[a]):
            for j in range(n[b]):
                for qa in range(p + 1):
                    for qb in range(p + 1):
                        x = [0.0, 0.0, 0.0]
                        x[axis], x[a], x[b] = float(end), (i + g[qa]) / n[a], (j + g[qb]) / n[b]
                        T = fun(*x, t) * w[qa] * w[qb] / (n[a] * n[b])
                        for ia in range(p + 1):
                            for ib in range(p + 1):
                                k = [0, 0, 0]
                                k[axis], k[a], k[b] = end * p * n[axis], p * i + ia, p * j + ib
                                R[k[2], k[1], k[0]] += N[qa, ia] * N[qb, ib] * T
    return R.reshape(-1)


@pytest.mark.parametrize("p", [1, 2, 3, 4])
def test_load_of_expressions(p):
    n = (2, 3, 2)
    pb = lsmf.Problem(prm_text({
        "Polynomial degree": p, "Quadrature order": p + 1, "Dimension": 3, "Type": "Box",
        "Box cells": "%d, %d, %d" % n, "Poisson's ratio": 0.3, "Shear modulus": 1.0, "Formulation": 1,
        "Solver type": "MF_CG", "Preconditioner type": "jacobi", "MF caching": "tensor2",
        "Dirichlet IDs and expressions": "4:0,0,0", "Dirichlet IDs and component mask": "4:true,true,true",
        "Neumann IDs and expressions": "5:%s,%s,%s;1:%s,%s,%s;2:%s,%s,%s" % (TOP + SIDE + SIDE)}))
    t = 0.7
    want = _load(p, n, t)
    nodes = [p * m + 1 for m in n]
    want[:3 * nodes[0] * nodes[1]] = 0.0  # the clamped bottom
    u = torch.zeros(pb.n_dofs, dtype=torch.float64, device="cuda")
    R, again = torch.full_like(u, float("nan")), torch.empty_like(u)
    norm = pb.residual(u, t, R)
    got = R.cpu().numpy()
    assert np.max(np.abs(got - want)) <= 1e-12 * np.max(np.abs(want))
    assert abs(norm - np.linalg.norm(want)) <= 1e-12 * np.linalg.norm(want)
    pb.residual(u, t, again)
    assert np.max(np.abs((again - R).cpu().numpy())) <= 1e-15  # internal force of u = 0 added by atomics
