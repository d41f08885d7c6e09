"""FP64 triangular solves at the edges of their blocks (64 rows, halves of 32, slices of 16 and 8 columns), alone and with
several right-hand sides, with inverses per 64 rows (dpotrs) and inside wider tiles (factor objects).

Bar, element by element: |L L^T x - b| <= 8 n 2^-53 (|L| |L^T| |x| + |b|), a multiple of substitution's bound that covers the
explicit inverses of the well-conditioned 64-row diagonal blocks (condition below 4).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _check(L, B, X):
    n = L.shape[0]
    bound = 8 * n * 2.0**-53 * (np.abs(L) @ (np.abs(L).T @ np.abs(X)) + np.abs(B))
    assert (np.abs(L @ (L.T @ X) - B) <= bound).all()


def _dev(M):
    import torch

    return torch.from_numpy(np.ascontiguousarray(M.T)).cuda()  # column-major


@pytest.mark.parametrize("n", [1, 7, 31, 32, 33, 47, 63, 64, 65, 96, 97, 128, 129, 300, 449, 705])
@pytest.mark.parametrize("r", [1, 3, 16])
def test_dpotrs(handle, n, r):
    rng = np.random.default_rng(n)
    L = np.tril(rng.uniform(-0.5, 0.5, (n, n)) / np.sqrt(n)) + 2 * np.eye(n)
    B = rng.standard_normal((n, r))
    X = _dev(B)
    handle.dpotrs_L(_dev(L + np.triu(np.full((n, n), np.nan), 1)), n, n, 512, X, n, r)
    _check(L, B, X.cpu().numpy().T)


@pytest.mark.parametrize("n,nb", [(65, 64), (100, 48), (257, 96), (520, 100), (700, 512), (1100, 320)])
@pytest.mark.parametrize("r", [1, 5])
def test_factor_objects(handle, n, nb, r):
    rng = np.random.default_rng(n + nb)
    R = rng.uniform(-0.5, 0.5, (n, n))
    A = (R + R.T) / 2 + np.sqrt(n) * np.eye(n)
    B = rng.standard_normal((n, r))
    L, X = np.asfortranarray(np.empty((n, n))), _dev(B)
    with handle.factor(_dev(A), n, n, nb, "fp64") as F:
        assert F.info == 0
        F.copy_L(L, n)
        F.solve(X, n, r)
        Y = _dev(B)
        F.solve(Y, n, r)
    _check(np.tril(L), B, X.cpu().numpy().T)
    assert (X == Y).all()  # the same sums whatever the schedule


def test_non_finite_values_stay_in_their_column(handle):
    n, r = 200, 4
    rng = np.random.default_rng(1)
    L = np.tril(rng.uniform(-0.5, 0.5, (n, n)) / np.sqrt(n)) + 2 * np.eye(n)
    B = rng.standard_normal((n, r))
    B[70, 1], B[3, 2] = np.inf, np.nan
    X = _dev(B)
    handle.dpotrs_L(_dev(L), n, n, 64, X, n, r)
    X = X.cpu().numpy().T
    _check(L, B[:, [0, 3]], X[:, [0, 3]])
    assert not np.isfinite(X[:, 1]).all() and not np.isfinite(X[:, 2]).all()
