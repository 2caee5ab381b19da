"""Selecting the node-sum scatter does not build the batch groups that only the
colour8 scatter uses: of the two selected in turn on a level that has neither,
colour8 is the one that pays for the groups (a pass over all cell nodes, tens
of ms at this size), though node sums came first.
"""
import time

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import lsmf  # noqa: E402


def _select(mesh, mode):
    op = lsmf.NeoHookOperator(mesh, "tensor2", 1, "fp32")  # FP32 batches: groups of their own
    torch.cuda.synchronize()
    t = time.perf_counter()
    op.set_scatter(mode)
    torch.cuda.synchronize()
    return time.perf_counter() - t


def test_groups_are_built_for_colour8():
    mesh = lsmf.Mesh("box", (64, 64, 64), 0, degree=2)
    lsmf.NeoHookOperator(mesh, "tensor2", 1, "fp64").set_scatter("nodesum")  # the level's node lists
    # of several operators the quickest: each allocates its per-cell buffer
    took = {"nodesum": min(_select(mesh, "nodesum") for _ in range(4))}
    took["colour8"] = _select(mesh, "colour8")
    assert took["nodesum"] < took["colour8"], took
