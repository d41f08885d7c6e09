"""Refinement of several right-hand sides on a stored matrix (2 <= nrhs <= 16, n >= 2048): its
residual is formed by digit products on the tensor cores.

A = 2 sqrt(n) I + a symmetric uniform part, X of integers, so that B = A X to rounding; graded: D A D,
D^-1 X, D B with D a power of two per row.  A term of the residual is rounded at 2^-54 of the largest
|a(i, k)| |x(k)| of its row and run of 128 columns.  The run with the diagonal dominates: sqrt(128) terms' worth
of 2^-54 * 2 sqrt(n) max|x|, divided by A's smallest eigenvalue (over 1.1 sqrt(n)): about 21 * 2^-54, which the
converged solution may be off by, and B's own rounding of sqrt(n) * 2^-53 max|x| adds less.  TOL is eight times
that; without the grading's exponents the error is 2^10 times larger and more.
"""
import pytest

pytestmark = pytest.mark.gpu

TOL = 8 * 21 * 2.0**-54


def _system(n, r, graded):
    import torch

    g = torch.Generator().manual_seed(n + r)
    A = torch.rand(n, n, generator=g, dtype=torch.float64) * 2 - 1
    A = (torch.tril(A) + torch.tril(A, -1).T + torch.diag(torch.full((n,), 2.0 * n**0.5, dtype=torch.float64))).cuda()
    X = torch.randint(1, 1 << 20, (r, n), generator=g).double().cuda()  # one row per right-hand side
    B = X @ A
    d = torch.ones(n, dtype=torch.float64).cuda()
    if graded:
        d = torch.pow(2.0, torch.randint(-20, 21, (n,), generator=g).double()).cuda()
    return A * d[:, None] * d[None, :], (X / d).contiguous(), (B * d).contiguous(), d


@pytest.mark.parametrize("n,r", [(2048, 3), (3072, 2), (4096, 5), (4097, 16), (4351, 8), (4500, 13)])
@pytest.mark.parametrize("graded", [False, True])
def test_refined_solution(handle, n, r, graded):
    import torch

    A, X, B, d = _system(n, r, graded)
    out = torch.empty_like(B)
    with handle.factor(A.clone(), n, n, 256, "fp32") as F:
        assert F.info == 0
        F.refine(A, n, B, n, out, n, r, 0.0, 8)
    err = ((out - X) * d).abs().max().item() / (X * d).abs().max().item()
    assert err <= TOL, err


def test_non_finite_column_stays_alone(handle):
    import torch

    n, r = 4200, 16
    A, X, B, d = _system(n, r, False)
    B[3, 17] = float("inf")
    out = torch.empty_like(B)
    with handle.factor(A.clone(), n, n, 256, "fp32") as F:
        F.refine(A, n, B, n, out, n, r, 0.0, 6)
    keep = [q for q in range(r) if q != 3]
    err = (out - X)[keep].abs().max().item() / X.abs().max().item()
    assert err <= TOL, err
    assert not torch.isfinite(out[3]).all()
