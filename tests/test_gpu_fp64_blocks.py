"""GPU tests of the FP64 diagonal block and row solve at the sizes where their tiling can go
wrong: edges of the 16-column blocks and the 64-column block, and row counts on both sides
of each rows-per-CTA choice (4, 8, 16 and 32 rows per CTA on a 152-SM part).

Bar: entrywise 1e-12 of max|L| against LAPACK, as the other FP64 factor tests; a matrix scaled
by a power of four must give the factor scaled by the power of two (relative 1e-12), also
where pivots leave the range of FP32 or come near the end of FP64's.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ATOL_REL = 1e-12


def _spd(n, seed=3):
    R = np.random.default_rng(seed).uniform(-0.5, 0.5, (n, n))
    return np.asfortranarray((R + R.T) / 2 + np.sqrt(n) * np.eye(n))


def _factor(handle, A, nb):
    import torch

    n = A.shape[0]
    T = torch.from_numpy(np.ascontiguousarray(A.T)).cuda()
    r = handle.dpotrf_L(T, n, n, nb, 0)
    return r.info, np.tril(T.cpu().numpy().T)


@pytest.mark.parametrize("n,nb", [(1, 64), (15, 64), (16, 64), (17, 64), (48, 48), (63, 64), (64, 64), (65, 72), (130, 72),
                                  (600, 40), (680, 40), (1300, 40), (2500, 40)])
def test_blocks_match_lapack(handle, n, nb):
    A = _spd(n)
    info, L = _factor(handle, A, nb)
    Lo = np.linalg.cholesky(A)
    assert info == 0
    np.testing.assert_allclose(L, Lo, rtol=0, atol=ATOL_REL * np.abs(Lo).max())


@pytest.mark.parametrize("k", [-500, -250, 250, 500])
def test_scaling_by_powers_of_two(handle, k):
    A = _spd(100)
    Lo = np.linalg.cholesky(A)
    info, L = _factor(handle, A * 2.0**k * 2.0**k, 64)
    assert info == 0
    np.testing.assert_allclose(L / 2.0**k, Lo, rtol=0, atol=ATOL_REL * np.abs(Lo).max())


@pytest.mark.parametrize("bad", [0, 15, 16, 31, 63, 64, 99])
@pytest.mark.parametrize("value", [-1.0, 0.0, np.nan])
def test_first_bad_pivot_is_reported(handle, bad, value):
    A = _spd(100)
    A[bad, bad] = value
    A[bad, :bad] = A[:bad, bad] = 0.0
    assert _factor(handle, A, 64)[0] == bad + 1
