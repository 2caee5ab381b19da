"""The launches of a colour8 vmult's groups overlap: a group's cells are loaded
and computed while the group before it adds its results.  Many calls in a row,
directly and replayed from a graph, give the bits of one call with a wait
behind it, and the basic kernel's lattice colours to rounding (at most 8
contributions a node of a few hundred operations each, in another order: 1e-12
and 2e-5 of the largest entry, as for the groups on small boxes).
"""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import numpy as np  # noqa: E402

import lsmf  # noqa: E402


@pytest.mark.parametrize("p,n", [(1, 16), (2, 12), (2, 24), (3, 8), (4, 6)])
@pytest.mark.parametrize("caching", ["tensor4", "tensor2", "scalar"])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_bits_of_one_call(p, n, caching, precision):
    rng = np.random.default_rng(13)
    mesh = lsmf.Mesh("box", (n, n, n + 1), 0, degree=p)
    mesh.set_dirichlet([(4, 7)])
    nc, _, nd = mesh.info()
    op = lsmf.NeoHookOperator(mesh, caching, 1, precision)
    op.set_material(rng.choice([1.0, 10.0], nc), 0.3)
    u = torch.tensor(rng.uniform(-0.0005, 0.0005, nd), device="cuda").to(op.dtype)
    srcs = [torch.tensor(rng.uniform(-1, 1, nd), device="cuda").to(op.dtype) for _ in range(3)]
    op.cache(u)
    op.set_scatter("colour8")
    alone = []
    for s in srcs:
        d = torch.full_like(s, float("nan"))
        op.vmult(d, s)
        op.sync()
        alone.append(d)
    row = [torch.full_like(s, float("nan")) for s in srcs]
    for _ in range(20):  # no wait between them
        for d, s in zip(row, srcs):
            op.vmult(d, s)
    for d, want in zip(row, alone):
        assert torch.equal(d, want)
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    op.set_stream(stream)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        for d, s in zip(row, srcs):
            op.vmult(d, s)
            op.vmult_add(d, s)
    graph.replay()
    graph.replay()
    torch.cuda.synchronize()
    op.set_basic_kernel(True)
    for d, s, want in zip(row, srcs, alone):
        twice = want.clone()
        op.set_basic_kernel(False)
        op.vmult_add(twice, s)
        op.sync()
        assert torch.equal(d, twice)
        op.set_basic_kernel(True)
        basic = torch.empty_like(s)
        op.vmult(basic, s)
        op.sync()
        assert float((want - basic).abs().max() / basic.abs().max()) < (1e-12 if precision == "fp64" else 2e-5)
