"""GPU tests of the FP64 update on the tensor cores (exact digit products) against extended
precision, at the edges of its tiles (128 rows, 64 columns, K in stages of 32 and runs of 128).

Bar, element by element: with |x(i, k)| < 2^e(i) the inputs are rounded to 2^(e(i) - 56) (K products,
two roundings each), orders 5..7 and their sum to two units of 2^-54, and the value and the
subtraction once to FP64:
    |err| <= 2^-52 (|C| + |v|) + 2^(e(i) + e(j)) (K 2^-55 + 2^-52) + 2^-1073.
Its root mean square is also at most that of the host's FP64 product.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _run(handle, A, C):
    import torch

    n, k = A.shape
    Ad = torch.from_numpy(np.ascontiguousarray(A.T)).cuda()
    Cd = torch.from_numpy(np.ascontiguousarray(C.T)).cuda()
    handle.dsyrk_ln("fp64", n, k, Ad, n, Cd, n)
    return Cd.cpu().numpy().T


def _check(A, C, got):
    k = A.shape[1]
    Aq = A.astype(np.longdouble)
    v = Aq @ Aq.T
    want = C.astype(np.longdouble) - v
    e = np.frexp(np.abs(A).max(axis=1))[1].astype(np.longdouble)
    scale = np.exp2(e[:, None] + e[None, :])
    bound = np.longdouble(2) ** -52 * (np.abs(C) + np.abs(v)) + scale * (k * np.longdouble(2) ** -55 + np.longdouble(2) ** -52)
    bound += np.longdouble(2) ** -1073
    lo = np.tril(np.ones(got.shape, dtype=bool))
    bad = lo & ~(np.abs(got - want) <= bound)
    assert not bad.any(), (np.argwhere(bad)[:4], float((np.abs(got - want) / bound)[lo].max()))
    np.testing.assert_array_equal(got[~lo], C[~lo])
    return np.abs(got - want)[lo]


@pytest.mark.parametrize("n,k", [(65, 16), (127, 31), (128, 32), (129, 33), (191, 64), (192, 127), (193, 128), (300, 129), (130, 300)])
def test_update_error_bound(handle, n, k):
    rng = np.random.default_rng(n + k)
    A, C = rng.standard_normal((n, k)), rng.standard_normal((n, n))
    _check(A, C, _run(handle, A, C))
    err = _check(A, 0 * C, _run(handle, A, 0 * C))
    host = np.abs(-(A @ A.T) - (-(A.astype(np.longdouble) @ A.T.astype(np.longdouble))))[np.tril(np.ones((n, n), dtype=bool))]
    assert np.sqrt(np.mean(err**2)) <= np.sqrt(np.mean(host**2)) + 1e-17 * k


@pytest.mark.parametrize("kind", ["equal", "signs", "rows_scaled", "graded", "tiny", "zeros"])
def test_update_error_bound_on_extreme_values(handle, kind):
    rng = np.random.default_rng(7)
    n, k = 200, 128
    A, C = rng.uniform(-1, 1, (n, k)), rng.uniform(-1, 1, (n, n))
    if kind == "equal":  # every digit product of an order has the same sign
        A[:] = 0.5019607843137255
    elif kind == "signs":
        A = np.where(rng.random((n, k)) < 0.5, -1.0, 1.0) * (1 - 2.0**-53)
    elif kind == "rows_scaled":
        s = 2.0 ** rng.integers(-300, 300, n)
        A, C = A * s[:, None], C * s[:, None] * s[None, :]
    elif kind == "graded":
        A *= 2.0 ** -rng.integers(0, 120, (n, k))
    elif kind == "tiny":  # subnormal elements, products and results
        A *= 2.0 ** -rng.integers(480, 1060, n)[:, None]
        C *= 2.0**-1020
    elif kind == "zeros":
        A[::3] = 0.0
        A[:, ::2] = 0.0
    _check(A, C, _run(handle, A, C))


def test_non_finite_rows_follow_ieee_sums(handle):
    rng = np.random.default_rng(9)
    n, k = 200, 100
    A, C = rng.uniform(-1, 1, (n, k)), rng.uniform(-1, 1, (n, n))
    A[3, 5], A[70, 0], A[130, 99] = np.inf, -np.inf, np.nan
    with np.errstate(invalid="ignore"):
        want = C - A @ A.T
    got = _run(handle, A, C)
    lo = np.tril(np.ones((n, n), dtype=bool))
    np.testing.assert_array_equal(np.isnan(got)[lo], np.isnan(want)[lo])
    np.testing.assert_array_equal(np.isinf(got)[lo], np.isinf(want)[lo])
    f = lo & np.isfinite(want)
    np.testing.assert_allclose(got[f], want[f], rtol=0, atol=1e-13)


@pytest.mark.parametrize("n,nb,tiles", [(700, 64, 60), (1000, 192, 20), (2600, 192, 90), (1300, 320, 14)])
def test_factor_is_schedule_invariant(oracle_mod, handle, n, nb, tiles):
    import torch

    A = oracle_mod.gen_uniform(n, 100, float(n))
    T = torch.from_numpy(np.ascontiguousarray(A.T)).cuda()
    assert handle.dpotrf_L(T, n, n, nb, 0).info == 0
    L = T.cpu().numpy().T
    H = A.copy(order="F")
    r = handle.dpotrf_L(H, n, n, nb, tiles * nb * nb * 8)
    assert r.info == 0 and r.stats["npanels"] >= 2
    np.testing.assert_array_equal(H, L)
    Lo = np.linalg.cholesky(A)
    np.testing.assert_allclose(np.tril(L), Lo, rtol=0, atol=1e-12 * np.abs(Lo).max())


@pytest.mark.parametrize("n,nb", [(65, 64), (129, 64), (500, 192), (1000, 128), (1300, 1088), (1201, 576), (700, 100)])
def test_factor_object(handle, n, nb):
    # factor objects in FP64: panels of up to 512 columns per update, tiles wider than that in several, and one
    # that 64 does not divide (FP64 MMAs).  |A - L L^T| <= 4 n eps sqrt(a_ii a_jj): the column solve multiplies by the
    # explicit inverse of a diagonal tile whose condition number is below 3.
    rng = np.random.default_rng(n)
    R = rng.uniform(-0.5, 0.5, (n, n))
    A = (R + R.T) / 2 + np.sqrt(n) * np.eye(n)
    import torch

    L = np.asfortranarray(np.empty((n, n)))
    with handle.factor(torch.from_numpy(np.ascontiguousarray(A)).cuda(), n, n, nb, "fp64") as F:
        assert F.info == 0
        F.copy_L(L, n)
    L, s = np.tril(L).astype(np.longdouble), np.sqrt(np.diag(A))
    err = np.abs(np.tril(A - L @ L.T) / s[:, None] / s[None, :]).max()
    assert err <= 4 * n * 2.0**-53, float(err)
