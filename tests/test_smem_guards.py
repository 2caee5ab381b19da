"""Kernels whose shared-memory layout depends on run-time values compare it with
the dynamic shared memory of the launch before they touch any (a launch that
was given less must set the operator's error word, which the host reports).
Such a launch cannot be made through the library, so this reads the sources.
"""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "large-strain-matrix-free_b200", "csrc")


def _body(name):
    for f in ("op_kernels.cuh", "coarse_kernels.cuh"):
        src = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, f)).read())
        m = re.search(r"__global__[^{;]*\b%s\([^{]*\{" % name, src)
        if m:
            depth, i = 1, m.end()
            while depth:
                depth += {"{": 1, "}": -1}.get(src[i], 0)
                i += 1
            return src[m.end():i]
    raise AssertionError("no kernel " + name)


@pytest.mark.parametrize("kernel,guard,first_use", [("apply_line_kernel", "smem_short(", "wbase"),
                                                    ("coarse_cheb_kernel", "coarse_smem_short<", "CoarseCells<"),
                                                    ("coarse_eig_kernel", "coarse_smem_short<", "CoarseCells<")])
def test_guard_comes_before_the_first_use(kernel, guard, first_use):
    body = _body(kernel)
    assert "extern __shared__" in body
    assert 0 <= body.find(guard) < body.index(first_use), kernel


def test_short_launch_sets_the_error_word():
    src = open(os.path.join(CSRC, "op_kernels.cuh")).read()
    fn = src[src.index("bool smem_short("):]
    fn = fn[:fn.index("\n}\n")]
    assert "%%dynamic_smem_size" in fn and "atomicOr(flag, FLAG_SMEM)" in fn
