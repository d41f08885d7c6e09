"""GPU tests of the one-launch triangular solves at the edges of their blocks (128 rows in FP32,
64 in FP64), of the panels they follow (also ragged and narrow ones) and of the right-hand
side groups (FP32: 1, 2, 4, 8 per task; FP64: one per task).

Bars: FP64 normwise backward error <= 1e-14 (|| b - A x || / (||A|| ||x|| + ||b||), infinity norms);
FP32 factors solve to n * 2^-23 of the same measure, and refinement reaches 1e-14.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _system(n, r, seed=5):
    rng = np.random.default_rng(seed)
    R = rng.uniform(-0.5, 0.5, (n, n))
    A = (R + R.T) / 2 + np.sqrt(n) * np.eye(n)
    return A, rng.standard_normal((n, r))


def _dev(M):
    import torch

    return torch.from_numpy(np.ascontiguousarray(M.T)).cuda()


def _berr(A, X, B):
    nA = np.abs(A).sum(axis=1).max()
    return max(np.abs(B[:, q] - A @ X[:, q]).max() / (nA * np.abs(X[:, q]).max() + np.abs(B[:, q]).max())
               for q in range(B.shape[1]))


@pytest.mark.parametrize("prec,bar", [("fp64", 1e-14), ("fp32", None)])
@pytest.mark.parametrize("n,nb,r", [(1, 64, 1), (63, 64, 3), (64, 64, 2), (65, 64, 1), (127, 128, 4), (129, 128, 5),
                                    (300, 100, 8), (513, 256, 9), (700, 200, 16), (1100, 512, 1), (1000, 33, 2)])
def test_factor_solve(handle, prec, bar, n, nb, r):
    A, B = _system(n, r)
    with handle.factor(_dev(A), n, n, nb, prec) as F:
        assert F.info == 0
        for _ in range(2):  # the second launch on the same exchange buffer
            X = _dev(B)
            F.solve(X, n, r)
            assert _berr(A, X.cpu().numpy().T, B) <= (bar or n * 2.0**-23 + 2.0**-20)


@pytest.mark.parametrize("n,nb,tail,r", [(1300, 256, 600, 1), (1300, 256, 600, 16), (900, 512, 24576, 3)])
def test_mixed_panel_widths(handle, ooc, n, nb, tail, r):
    import torch

    A, B = _system(n, r)
    handle.set_option(ooc.OPT_TAIL_ORDER, tail)
    try:
        Ad, Bd = _dev(A), _dev(B)
        with handle.factor(Ad, n, n, nb, "bf16x3") as F:
            X = torch.empty_like(Bd)
            _, be = F.refine(Ad, n, Bd, n, X, n, r, 1e-14)
    finally:
        handle.set_option(ooc.OPT_TAIL_ORDER, 24576)
    assert be <= 1e-14 and _berr(A, X.cpu().numpy().T, B) <= 1e-14


@pytest.mark.parametrize("where,n,nb,r,budget", [("device", 500, 96, 2, 0), ("device", 500, 96, 16, 96 * 96 * 8 + 96 * 128 + 256),
                                                ("device", 131, 16, 1, 0), ("host", 500, 96, 5, 0), ("host", 131, 16, 16, 0)])
def test_dpotrs(handle, where, n, nb, r, budget):
    A, B = _system(n, r)
    L = np.asfortranarray(np.linalg.cholesky(A) + np.triu(np.full((n, n), np.nan), 1))  # the upper part is not read
    if where == "device":
        X = _dev(B)
        handle.dpotrs_L(_dev(L), n, n, nb, X, n, r, budget=budget)
        X = X.cpu().numpy().T
    else:
        X = B.copy(order="F")
        handle.dpotrs_L(L, n, n, nb, X, n, r, budget=budget)
    assert _berr(A, X, B) <= 1e-14


@pytest.mark.parametrize("n,r", [(2300, 8), (2500, 9), (3100, 16), (5000, 3), (19600, 16), (19700, 10)])
def test_right_hand_sides_per_task(handle, n, r):
    # FP32: 1, 2, 4 or 8 right-hand sides per task by the number of tasks; orders where that changes
    import torch

    g = torch.Generator(device="cuda").manual_seed(n)
    A = torch.empty(n, n, dtype=torch.float64, device="cuda").uniform_(-0.5, 0.5, generator=g)
    A = torch.tril(A) + torch.tril(A, -1).T
    A.diagonal().add_(n**0.5)
    B = torch.randn(r, n, dtype=torch.float64, device="cuda", generator=g)
    with handle.factor(A, n, n, 256, "fp32") as F:
        assert F.info == 0
        X = B.clone()
        F.solve(X, n, r)
    R, nA = B - X @ A, A.abs().sum(dim=1).max()
    be = (R.abs().amax(dim=1) / (nA * X.abs().amax(dim=1) + B.abs().amax(dim=1))).max().item()
    assert be <= n * 2.0**-23 + 2.0**-20
