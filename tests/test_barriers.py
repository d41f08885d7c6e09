"""A block-wide barrier must be reached by every thread of the block, so no call of one may stand behind a
short-circuit or a conditional operator of its own expression: lanes that skip it leave the others' wait, and
the value that a reducing barrier returns, undefined.  The scan covers every kernel source; the GPU test the FP32
digit kernel's row scales, which one such barrier decides, with every kind of row in one warp."""
import glob
import os
import re

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "oocdag_gb300", "csrc")


def _conditional_barriers(text):
    text = re.sub(r"//[^\n]*|/\*.*?\*/", "", text, flags=re.S)
    found = []
    for m in re.finditer(r"__syncthreads\w*\s*\(", text):
        head = re.split(r"[;{}]", text[: m.start()])[-1]  # the statement up to the call
        if re.search(r"&&|\|\||\?", head):
            found.append(" ".join((head + m.group()).split()))
    return found


def test_the_scan_sees_a_barrier_behind_a_short_circuit():
    assert _conditional_barriers("void f() { bool z = a == 0 && !__syncthreads_or(b); }")
    assert not _conditional_barriers("void f() { bool s = __syncthreads_or(b && c); __syncthreads(); }")


@pytest.mark.parametrize("path", sorted(glob.glob(os.path.join(CSRC, "*.cu*"))), ids=os.path.basename)
def test_no_barrier_behind_a_condition_of_its_expression(path):
    assert _conditional_barriers(open(path).read()) == []


def test_kernels_of_several_roles_read_the_status_word_once_for_the_block():
    """A kernel whose warps wait for one another on mbarriers must not have some of them leave, or see no work, because the
    status word was raised (by the diagonal tile on another stream) between two of its threads' reads."""
    kernels = 0
    for path in glob.glob(os.path.join(CSRC, "*.cu")):
        for body in open(path).read().split("__global__")[1:]:
            if "tcgen05.alloc" not in body:
                continue
            kernels += 1
            lines = [line for line in body.split("// ---- teardown")[0].split("\n") if re.search(r"\*\(volatile (const )?int\*\)status", line)]
            assert lines
            for line in lines:  # directly in the block-wide OR, or through a variable
                name = re.match(r"\s*const int (\w+) = ", line)
                assert "__syncthreads_or(" in line or (name and f"__syncthreads_or({name.group(1)})" in body), (path, line)
    assert kernels >= 6


@pytest.mark.gpu
@pytest.mark.parametrize("n", [130, 161, 300])
def test_zero_subnormal_and_normal_rows_in_one_warp(handle, n):
    """Below a 64-column identity block the rows are, in turn, normal, zero and subnormal, so L's are A's own
    and the trailing update's product of two of them is known: of two subnormal rows it is 0 in FP32.  The rest of the
    matrix is 16 I, and an element of the updated block is rounded at most twice per 32 columns."""
    import torch

    nb = 64
    rng = np.random.default_rng(n)
    A = np.zeros((n, n))
    A[:nb, :nb] = np.eye(nb)
    m = n - nb
    V = rng.uniform(-0.125, 0.125, (m, nb))
    V[1::3] = 0.0
    V[2::3] *= 2.0**-127
    A[nb:, :nb] = V
    A[nb:, nb:] = 16 * np.eye(m)
    A = A.astype(np.float32)
    T = torch.from_numpy(np.ascontiguousarray(A.T)).cuda()
    assert handle.spotrf_L(T, n, n, nb).info == 0
    L = np.tril(T.cpu().numpy().T).astype(np.float64)
    # (the block's inverse is 1 to two units of rsqrtf; subnormals to theirs)
    np.testing.assert_allclose(L[nb:, :nb], A[nb:, :nb].astype(np.float64), rtol=2.0**-20, atol=2.0**-147)
    want = np.linalg.cholesky(16 * np.eye(m) - A[nb:, :nb].astype(np.float64) @ A[nb:, :nb].astype(np.float64).T)
    assert np.abs(L[nb:, nb:] - want).max() <= 4 * (n + 2) * 2.0**-24 * 4  # rows of L have norm 4
    z = np.arange(m) % 3 != 0  # zero and subnormal rows leave the identity's as they were
    np.testing.assert_allclose(L[nb:, nb:][np.ix_(z, z)], 4 * np.eye(m)[np.ix_(z, z)], rtol=2.0**-20, atol=0)
