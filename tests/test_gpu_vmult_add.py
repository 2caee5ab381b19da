"""vmult_add and the vmult without zeroing: dst + A src whatever dst held, the
identity rows among it, over the scatters and both kernels, with constrained
dofs (whose rows are a launch of their own before the cell loop) and without.
A node sums its at most 8 contributions onto dst in another order than onto
zero: relative to the largest entry 16 roundings, 2e-15 and 1e-6; 1e-14, 4e-6.
"""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import numpy as np  # noqa: E402

import lsmf  # noqa: E402

NO_ZERO = lsmf.MASK_DEFAULT & ~lsmf.MASK_ZERO


@pytest.mark.parametrize("cells", [(1, 1, 1), (7, 5, 3), (12, 12, 12)])
@pytest.mark.parametrize("dirichlet", [[], [(4, 7), (1, 2)]])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("caching", ["tensor4", "scalar"])
def test_adds_to_what_dst_holds(cells, dirichlet, precision, caching):
    rng = np.random.default_rng(3)
    mesh = lsmf.Mesh("box", cells, 0, degree=2)
    if dirichlet:
        mesh.set_dirichlet(dirichlet)
    nc, _, nd = mesh.info()
    op = lsmf.NeoHookOperator(mesh, caching, 1, precision)
    op.set_material(rng.choice([1.0, 10.0], nc), 0.3)
    u, src, old = (torch.tensor(rng.uniform(-a, a, nd), device="cuda").to(op.dtype) for a in (0.001, 1.0, 1.0))
    op.cache(u)
    con = torch.tensor(mesh.constraint_mask(), device="cuda") != 0
    for basic in (False, True):
        op.set_basic_kernel(basic)
        op.set_scatter("atomic")
        product = torch.empty_like(src)
        op.vmult(product, src)
        assert torch.equal(product[con], src[con])
        for scatter in ("atomic", "colour8", "nodesum"):
            op.set_scatter(scatter)
            for call in (lambda d: op.vmult_add(d, src), lambda d: op.vmult(d, src, NO_ZERO)):
                dst = old.clone()
                for _ in range(3):  # launches of one call behind those of another
                    call(dst)
                assert torch.equal(dst[con], ((old + src) + src)[con] + src[con])
                want = old.double() + 3 * product.double()
                err = float((dst.double() - want).abs().max() / want.abs().max())
                assert err < (1e-14 if precision == "fp64" else 4e-6), (scatter, basic, err)
