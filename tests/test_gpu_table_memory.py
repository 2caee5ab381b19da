"""Device memory of an operator: the stored records (36 / 17 / 54 values per point
and cell of tensor4 / tensor2 / tensor4_ns in FP64), two diagonals, the shear
moduli, and nothing of the size of the full tensors that memory_consumption
counts (51 / 17 / 90).  cudaMalloc rounds each of the few buffers up to 2 MiB.
"""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import lsmf  # noqa: E402

MIB = 1 << 20


@pytest.mark.parametrize("caching,values", [("tensor4", 36), ("tensor2", 17), ("tensor4_ns", 54)])
def test_operator_holds_its_records_only(caching, values):
    mesh = lsmf.Mesh("box", (24, 24, 24), 0, degree=2)
    nc, _, nd = mesh.info()
    lsmf.NeoHookOperator(mesh, "tensor2", 1, "fp64").clear()  # what the first operator sets up once
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    op = lsmf.NeoHookOperator(mesh, caching, 1, "fp64")
    torch.cuda.synchronize()
    held = free - torch.cuda.mem_get_info()[0]
    need = 8 * (nc * values * 27 + 2 * nd + nc)
    assert need <= held <= need + 12 * MIB, (held / MIB, need / MIB)
    assert op.memory_consumption() >= 8 * nc * values * 27
