"""FP64 batched factor + solve: the trailing updates by digit products on the tensor cores.

|A - L L^T|(i, j) <= (n + 1) eps (|L| |L^T|)(i, j) <= (n + 1) eps sqrt(a_ii a_jj) for a factorization that
rounds once per operation (eps = 2^-53).  Here a panel's element is multiplied by a rounded reciprocal
(two more roundings) and a step's products are rounded at 2^-56 of their row scales, of which
the bound holds at most 32 per step: (2 n + 16) eps covers all of it, whatever the grading by rows.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = 2.0**-53


def _run(handle, mats, rhs, blk):
    import torch

    ns = [m.shape[0] for m in mats]
    ao = np.concatenate([[0], np.cumsum([n * n for n in ns])[:-1]])
    bo = np.concatenate([[0], np.cumsum(ns)[:-1]])
    A = torch.from_numpy(np.concatenate([m.T.ravel() for m in mats])).cuda()
    B = torch.from_numpy(np.concatenate(rhs)).cuda()
    info, _ = handle.batched_posv("fp64", ns, ao, bo, A, B, blk_table=None if blk is None else [blk] * 16)
    A, B = A.cpu().numpy(), B.cpu().numpy()
    L = [A[o : o + n * n].reshape(n, n).T for n, o in zip(ns, ao)]
    return info, L, [B[o : o + n] for n, o in zip(ns, bo)]


def _spd(n, rng):
    M = rng.standard_normal((n, n))
    return M @ M.T / n + np.eye(n)


@pytest.mark.parametrize("blk", [None, 8, 16])
@pytest.mark.parametrize("graded", [False, True])
def test_factor_and_solution(handle, blk, graded):
    rng = np.random.default_rng(3)
    orders = [1, 7, 8, 9, 15, 16, 17, 31, 32, 33, 47, 48, 49, 63, 64, 65, 95, 97, 127, 128, 129, 200, 256, 257, 303, 384, 385, 511, 512]
    mats, sols = [], []
    for n in orders:
        A = _spd(n, rng)
        x = rng.standard_normal(n)
        if graded:  # powers of two: exact
            d = 2.0 ** rng.integers(-150, 151, n)
            A, x = A * d[:, None] * d[None, :], x / d
        mats.append(A)
        sols.append(x)
    info, L, X = _run(handle, mats, [A @ x for A, x in zip(mats, sols)], blk)
    assert info == [0] * len(orders)
    for n, A, Lf, x, xs in zip(orders, mats, L, X, sols):
        Lt = np.tril(Lf)
        s = np.sqrt(np.diag(A))
        Ls = (Lt / s[:, None]).astype(np.longdouble)
        As = (A / s[:, None] / s[None, :]).astype(np.longdouble)
        err = np.abs(np.tril(As - Ls @ Ls.T)).max()
        assert err <= (2 * n + 16) * EPS, (n, float(err))
        assert np.array_equal(np.triu(Lf, 1), np.triu(A, 1))  # the strict upper triangle is not touched
        # residual of the solution: three such factors of n eps, and cond < 16 for the forward error
        e = np.abs((x - xs) * s).max() / np.abs(xs * s).max()
        assert e <= 16 * 3 * (2 * n + 16) * EPS, (n, e)


@pytest.mark.parametrize("n,bad", [(40, 0), (64, 31), (100, 32), (300, 47), (512, 255), (512, 511)])
def test_info_and_neighbours(handle, n, bad):
    rng = np.random.default_rng(5)
    A, good = _spd(n, rng), _spd(n, rng)
    A[bad, bad] = -1.0
    info, _, X = _run(handle, [good, A, good], [good @ np.ones(n)] * 3, None)
    assert info == [0, bad + 1, 0]
    for q in (0, 2):
        assert np.abs(X[q] - 1.0).max() <= 16 * 3 * (2 * n + 16) * EPS


def test_not_finite_and_tiny(handle):
    """A NaN far from the first step: the rows above it are the finite system's; a matrix whose products
    are subnormal (entries of 2^-1000) has a factor of 2^-500 with the usual bound."""
    rng = np.random.default_rng(6)
    n = 150
    A = _spd(n, rng)
    N = A.copy()
    N[140, 10] = N[10, 140] = np.nan
    T = _spd(n, rng)
    info, L, X = _run(handle, [A, N, T * 2.0**-1000], [np.ones(n)] * 3, None)
    assert info[0] == 0 and info[1] == 141 and info[2] == 0
    assert np.array_equal(np.tril(L[1])[:140], np.tril(L[0])[:140])
    Ls = np.tril(L[2]).astype(np.longdouble) * np.longdouble(2.0) ** 500
    assert np.abs(np.tril(T - Ls @ Ls.T)).max() <= (2 * n + 16) * EPS * np.diag(T).max()
