"""Refinement of several right-hand sides whose solutions are graded differently inside one run of 128 rows.

A couples rows of the same parity only (each half 2 sqrt(n) I + a symmetric uniform part, as in test_gpu_symm_digits.py);
the even rows of even columns of X are integers, the odd ones integers times 2^-60, and the other way round in odd columns.
The two halves of a column are separate systems, so an FP64 residual finds each to its own size: the bar of that test
(8 * 21 * 2^-54), half by half.  In digits relative to a column's largest element in a run the small half would be 0.
A control with the same grading in every column, and columns of zeros and unit vectors beside ordinary ones.
"""
import pytest

pytestmark = pytest.mark.gpu

TOL = 8 * 21 * 2.0**-54


def _matrix(n, g):
    import torch

    A = torch.rand(n, n, generator=g, dtype=torch.float64) * 2 - 1
    A = torch.tril(A) + torch.tril(A, -1).T
    A[::2, 1::2] = 0.0
    A[1::2, ::2] = 0.0
    A.diagonal().copy_(torch.full((n,), 2.0 * n**0.5, dtype=torch.float64))
    return A.cuda()


@pytest.mark.parametrize("n,r", [(2048, 3), (3072, 2), (4097, 16), (4100, 4)])
@pytest.mark.parametrize("kind", ["opposite", "same", "special"])
def test_each_half_to_its_own_size(handle, kind, n, r):
    import torch

    g = torch.Generator().manual_seed(n + r)
    A = _matrix(n, g)
    X = torch.randint(1, 1 << 20, (r, n), generator=g).double().cuda()  # one row per right-hand side
    for q in range(r):
        if kind == "special" and q == 0:
            X[q] = 0.0
        elif kind == "special" and q == 1:
            X[q] = 0.0
            X[q, 5] = 1.0
        else:
            X[q, (q if kind == "opposite" else 0) % 2 :: 2] *= 2.0**-60
    B = (X @ A).contiguous()
    out = torch.empty_like(B)
    with handle.factor(A.clone(), n, n, 256, "fp32") as F:
        assert F.info == 0
        F.refine(A, n, B, n, out, n, r, 0.0, 6)
    for q in range(r):
        for p in (0, 1):
            scale = X[q, p::2].abs().max().item()
            assert (out - X)[q, p::2].abs().max().item() <= TOL * scale, (q, p)


@pytest.mark.parametrize("n,r", [(2048, 3), (3072, 2), (4097, 16)])
def test_a_quarter_of_the_rows(handle, n, r):
    """The same with four separate systems, one of them 2^-60 the size of the others in every other column: most elements of a
    run are of a kind, and the small ones would round to 0 beside them."""
    import torch

    g = torch.Generator().manual_seed(n * r)
    A = torch.rand(n, n, generator=g, dtype=torch.float64) * 2 - 1
    A = torch.tril(A) + torch.tril(A, -1).T
    k = torch.arange(n)
    A *= (k[:, None] - k[None, :]) % 4 == 0
    A.diagonal().copy_(torch.full((n,), 2.0 * n**0.5, dtype=torch.float64))
    A = A.cuda()
    X = torch.randint(1, 1 << 20, (r, n), generator=g).double().cuda()
    X[::2, 1::4] *= 2.0**-60
    B = (X @ A).contiguous()
    out = torch.empty_like(B)
    with handle.factor(A.clone(), n, n, 256, "fp32") as F:
        assert F.info == 0
        F.refine(A, n, B, n, out, n, r, 0.0, 6)
    for q in range(r):
        for p in range(4):
            scale = X[q, p::4].abs().max().item()
            assert (out - X)[q, p::4].abs().max().item() <= TOL * scale, (q, p)
