"""GPU tests of the FP32 path's tensor-core products (exact digit products) at the edges of
their blocks (128 x 128, K in stages of 32 and runs of 256): the trailing update, through
the FP32 factorization.

Bar, element by element: |A - L L^T| <= 4 (n + 2) 2^-24 sqrt(a_ii a_jj), a small multiple of the
componentwise bound of an FP32 Cholesky; a matrix scaled by 4^k gives the factor scaled by 2^k
to the same bar.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _spd(n, seed=2, graded=False):
    rng = np.random.default_rng(seed)
    R = rng.uniform(-0.5, 0.5, (n, n))
    A = (R + R.T) / 2 + np.sqrt(n) * np.eye(n)
    if graded:
        d = 2.0 ** rng.integers(-25, 25, n)
        A = A * d[:, None] * d[None, :]
    return A.astype(np.float32)


def _check(A, L):
    n = A.shape[0]
    A, L = A.astype(np.float64), np.tril(L.astype(np.float64))
    d = np.sqrt(np.diag(A))
    err = np.abs(np.tril(A - L @ L.T)) / (d[:, None] * d[None, :])
    assert err.max() <= 4 * (n + 2) * 2.0**-24, err.max()


def _factor(handle, A, nb, pad=0):
    import torch

    n = A.shape[0]
    T = torch.full((n, n + pad), 7.0, dtype=torch.float32, device="cuda")
    T[:, :n] = torch.from_numpy(np.ascontiguousarray(A.T)).cuda()
    r = handle.spotrf_L(T, n, n + pad, nb, 0)
    assert (T[:, n:] == 7.0).all()
    return r.info, T[:, :n].cpu().numpy().T


@pytest.mark.parametrize("n,nb,pad", [(79, 15, 0), (80, 16, 1), (128, 64, 0), (191, 128, 3), (257, 128, 0), (385, 128, 2),
                                      (300, 31, 0), (520, 256, 0), (777, 257, 5), (1100, 512, 0), (1000, 100, 1)])
def test_factor_residual(handle, n, nb, pad):
    A = _spd(n)
    info, L = _factor(handle, A, nb, pad)
    assert info == 0
    _check(A, L)
    np.testing.assert_array_equal(np.triu(L, 1), np.triu(A, 1))


@pytest.mark.parametrize("k", [-60, 0, 60])
def test_scales(handle, k):
    A = _spd(400, graded=k == 0)
    S = A * np.float32(2.0**k)
    info, L = _factor(handle, S, 128)
    assert info == 0
    _check(S, L)


def test_out_of_core(handle):
    n, nb = 900, 128
    A = _spd(n)
    H = np.asfortranarray(A.copy())
    r = handle.spotrf_L(H, n, n, nb, 3 * n * 256 * 4 + 1024)
    assert r.info == 0 and r.stats["npanels"] >= 3
    _check(A, H)


@pytest.mark.parametrize("bad", [5, 200, 399])
@pytest.mark.parametrize("value", [-1.0, np.inf, np.nan])
def test_bad_pivots(handle, bad, value):
    """A negative or NaN pivot is reported; an infinity off the diagonal makes its row's pivot fail."""
    A = _spd(400)
    if np.isinf(value):
        A[bad, 0] = A[0, bad] = value
    else:
        A[bad, bad] = value
    info, _ = _factor(handle, A, 128)
    assert info == bad + 1
