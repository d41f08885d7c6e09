"""FP64 products of arbitrary caller matrices (tile dgemm and dsyrk, ooc_dsyrk_ln) above the size from which the tensor cores
take them: whatever the operands' range, each element stays within the bound of an FP64 sum of k products,
    |err| <= (k + 2) 2^-53 sum |a| |b|  (+ 2^-1074 per product, and for C - sum the rounding of |C|).
The tensor cores' digits are relative to a row's largest element, which does not imply it: operands graded along k,
rows with a few large elements, rows of a short last run that are larger than those before, and sparse ones.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LD = np.longdouble


def _bound(A, B, extra=0.0):
    k = A.shape[1]
    return (k + 2) * LD(2) ** -53 * (np.abs(A).astype(LD) @ np.abs(B).astype(LD).T + extra) + k * LD(2) ** -1074


def _operands(kind, m, n, k, rng):
    """A (m x k) and B (n x k); the product is A B^T."""
    A, B = rng.uniform(-1, 1, (m, k)), rng.uniform(-1, 1, (n, k))
    if kind == "normal":
        A, B = rng.standard_normal((m, k)), rng.standard_normal((n, k))
    elif kind == "alternating":  # 2^-60 against 1 throughout
        s = np.where(np.arange(k) % 2 == 0, 1.0, 2.0**-60)
        A, B = np.tile(s, (m, 1)), np.tile(2.0**-60 / s, (n, 1))
    elif kind == "graded":  # (A D)(D^-1 B)
        d = 2.0 ** rng.integers(-60, 61, k)
        A, B = A * d, B / d
    elif kind == "mildly graded":
        d = 2.0 ** rng.integers(-14, 15, k)
        A, B = A * d, B / d
    elif kind == "few large":  # one element of a row is 2^45 times the others, elsewhere in each operand
        A[np.arange(m), rng.integers(0, k // 2, m)] *= 2.0**45
        B[np.arange(n), k // 2 + rng.integers(0, k // 2, n)] *= 2.0**45
    elif kind == "sparse":
        A *= rng.random((m, k)) < 0.1
        B *= rng.random((n, k)) < 0.1
    elif kind == "one bad row":
        d = 2.0 ** rng.integers(-60, 61, k)
        A[m - 1] *= d
        B[0] /= d
    elif kind == "tail":  # the last two columns: large against (large, tiny)
        A[:, -2:] = [0.0, 2.0**40]
        B[:, -2:] = [1.0, 2.0**-60]
        A[:, :-2] *= 2.0**-40
    elif kind == "tail after zeros":  # a last run whose predecessor has eight columns, one of them 2^5 times the others
        A[:, : k - k % 128 - 8 if k > 128 else 0] = 0.0
        B[:, : k - k % 128 - 8 if k > 128 else 0] = 0.0
        A, B = A * 2.0**-5, B * 2.0**-5
        if k > 128:
            A[:, k - k % 128 - 8] = 1.0
            B[:, k - k % 128 - 7] = 1.0
    elif kind == "subnormal":
        A, B = A * 2.0**-1040, B * 2.0**1000
    elif kind == "zero rows":
        A[::2] = 0.0
        B[1::2] = 0.0
    return A, B


KINDS = ["uniform", "normal", "alternating", "graded", "mildly graded", "few large", "sparse", "one bad row", "tail", "tail after zeros", "subnormal", "zero rows"]
SHAPES = [(128, 128, 128), (72, 130, 257), (150, 100, 160), (129, 140, 130), (64, 65, 517), (300, 8, 1040)]


def _put(M):
    import torch

    return torch.from_numpy(np.ascontiguousarray(M.T)).cuda()  # column-major


@pytest.mark.parametrize("m,n,k", SHAPES)
@pytest.mark.parametrize("kind", KINDS)
def test_dgemm(ooc, handle, kind, m, n, k):
    import torch

    from oocdag_gb300 import offload as off

    assert off.init(0) == 0
    rng = np.random.default_rng(m + n + k)
    A, B = _operands(kind, m, n, k, rng)
    want, bound = A.astype(LD) @ B.astype(LD).T, _bound(A, B)
    for ta, tb in (("N", "T"), ("T", "N")):
        Ad, Bd = _put(A if ta == "N" else A.T), _put(B if tb == "T" else B.T)
        Cd = torch.full((n, m), float("nan"), dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        off.dgemm(ta, tb, m, n, k, 1.0, Ad, m if ta == "N" else k, Bd, n if tb == "T" else k, 0.0, Cd, m)
        assert off.last_error() == 0
        err = np.abs(Cd.cpu().numpy().T - want)
        assert (err <= bound).all(), float((err / bound).max())


def _graded_rows(kind, n, k, rng):
    A, B = _operands(kind, n, n, k, rng)
    return np.where(np.arange(n)[:, None] % 2 == 0, A, B)  # rows graded against one another


@pytest.mark.parametrize("n,k", [(128, 128), (190, 70), (130, 257), (72, 642)])
@pytest.mark.parametrize("kind", KINDS)
def test_symmetric_products(ooc, handle, kind, n, k):
    import torch

    from oocdag_gb300 import offload as off

    assert off.init(0) == 0
    rng = np.random.default_rng(n + k)
    A = _graded_rows(kind, n, k, rng)
    C = rng.uniform(-1, 1, (n, n)) * (0.0 if kind == "alternating" else 1.0)
    Ad, C1 = _put(A), _put(C)
    C2 = C1.clone()
    torch.cuda.synchronize()
    handle.dsyrk_ln("fp64", n, k, Ad, n, C1, n)
    off.dsyrk("L", "N", n, k, -1.0, Ad, n, 1.0, C2, n)
    assert off.last_error() == 0
    want = C.astype(LD) - A.astype(LD) @ A.astype(LD).T
    lo = np.tril(np.ones((n, n), dtype=bool))
    for got in (C1, C2):
        G = got.cpu().numpy().T
        over = np.abs(want) > np.finfo(np.float64).max  # (two rows of 2^1000)
        assert not np.isfinite(G[lo & over]).any()
        err, bound = np.where(over, 0, np.abs(np.where(over, 0, G) - want * ~over)), _bound(A, A, np.abs(C))
        assert (err <= bound)[lo].all(), float((err / bound)[lo].max())
        np.testing.assert_array_equal(G[~lo], C[~lo])
