"""Cell loops with whole lines per lane, several cells per warp and records
interleaved over a batch of cells (8 / 3 / 2 / 1 cells at degree 1 / 2 / 3 /
4, twice that in FP32): cell counts below, at and just past a batch, so that
warps with idle cell slots and unpaired FP32 cells are met, for the vmult with
and without the record ring, the cache tables and the diagonal, against the
oracle.  Tolerances as in test_gpu_operator.py: 1e-10 (FP64), 2e-5 (FP32).
"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import lsmf  # noqa: E402
import oracle as O  # noqa: E402
from test_gpu_operator import VARIANTS, _rel  # noqa: E402

BATCH = {1: 8, 2: 3, 3: 2, 4: 1}


@pytest.mark.parametrize("caching,formulation", VARIANTS)
@pytest.mark.parametrize("p", [1, 2, 3, 4])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_cell_counts_around_a_batch(caching, formulation, p, precision):
    B = BATCH[p] * (2 if precision == "fp32" else 1)
    tol = 1e-10 if precision == "fp64" else 2e-5
    dt = torch.float64 if precision == "fp64" else torch.float32
    rng = np.random.default_rng(7)
    for n in sorted({1, B, B + 1, 2 * B - 1}):
        gm = lsmf.Mesh("box", (n, 1, 1), 0, degree=p)
        gm.set_dirichlet([(4, 7), (1, 2)])
        om = O.Mesh(O.GEOM_BOX, (n, 1, 1), 0, (0, 0, 0), (1, 1, 1), 1.0, p, p + 1)
        mu = rng.choice([1.0, 10.0], size=n)
        u = rng.uniform(-0.01 / n, 0.01 / n, size=om.n_dofs).astype(np.float32).astype(np.float64)
        src = rng.uniform(-1, 1, size=om.n_dofs).astype(np.float32).astype(np.float64)
        ref = O.Operator(om, caching, formulation)
        ref.set_material(mu, 0.3)
        cmask = om.constraints([(4, 7), (1, 2)])
        ref.set_constraints(cmask)
        assert ref.cache(u) == 0
        op = lsmf.NeoHookOperator(gm, caching, formulation, precision)
        op.set_material(mu, 0.3)
        du, dsrc = (torch.tensor(x, device="cuda", dtype=dt) for x in (u, src))
        op.cache(du)
        want = ref.vmult(src)
        for depth in (0, 1, 3):
            op.set_pipeline(depth)
            dst = torch.full_like(dsrc, float("nan"))
            op.vmult(dst, dsrc)
            got = dst.cpu().numpy().astype(np.float64)
            assert _rel(got, want) < tol, (n, depth)
            assert np.array_equal(got[cmask == 1], src[cmask == 1])
        op.set_scatter("colour8")
        op.vmult(dst, dsrc)
        assert _rel(dst.cpu().numpy().astype(np.float64), want) < tol, n
        op.set_scatter("atomic")
        op.compute_diagonal()
        # the oracle's diagonal entry by entry (constrained rows are 1)
        d = np.array([ref.vmult(np.eye(1, om.n_dofs, i)[0])[i] for i in range(0, om.n_dofs, 7)])
        assert _rel(op.get_matrix_diagonal().cpu().numpy().astype(np.float64)[::7], d) < tol, n
        # metric table of every cell (FP32: rounded)
        assert _rel(op.table(4), ref.table(4)) < (1e-13 if precision == "fp64" else 1e-6), n
