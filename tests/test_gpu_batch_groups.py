"""The colour8 vmult of the production kernel: whole batches of cells in groups
that share no node, the cells of a batch added one after the other.  Boxes whose
rows end inside a batch (batches of 8 / 3 / 2 / 1 cells at degree 1 / 2 / 3 /
4, twice that in FP32), against the basic kernel over the lattice colours, and
bit for bit from call to call.  The two sum at most 8 cells' contributions to a
node, of a few hundred operations each, in another order: 1e-12 (FP64) and
2e-5 (FP32), relative to the largest entry.
"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import lsmf  # noqa: E402
from test_gpu_operator import VARIANTS  # noqa: E402


@pytest.mark.parametrize("caching,formulation", VARIANTS)
@pytest.mark.parametrize("p", [1, 2, 3, 4])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_groups_of_batches(caching, formulation, p, precision):
    rng = np.random.default_rng(11)
    for cells in ((1, 1, 1), (1, 2, 5), (4, 3, 2), (7, 5, 3)):
        mesh = lsmf.Mesh("box", cells, 0, degree=p)
        mesh.set_dirichlet([(4, 7), (1, 2)])
        nc, _, nd = mesh.info()
        op = lsmf.NeoHookOperator(mesh, caching, formulation, precision)
        op.set_material(rng.choice([1.0, 10.0], nc), 0.3)
        u, src = (torch.tensor(rng.uniform(-a, a, nd), device="cuda").to(op.dtype) for a in (0.001, 1.0))
        op.cache(u)
        op.set_scatter("colour8")
        first, again, want = (torch.full_like(src, float("nan")) for _ in range(3))
        for ring in (-1, 0, 1, 3):
            op.set_pipeline(ring)
            op.vmult(first, src)
            op.vmult(again, src)
            assert torch.equal(first, again), (cells, ring)
        op.set_basic_kernel(True)
        op.vmult(want, src)
        err = (first - want).abs().max() / want.abs().max()
        assert float(err) < (1e-12 if precision == "fp64" else 2e-5), cells
