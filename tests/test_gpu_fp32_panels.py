"""FP32 factorizations in panels narrower than the caller's tiles (256 columns, or 128 where 256 does not divide it).

|A - L L^T|(i, j) <= c n eps sqrt(a_ii a_jj) with eps = 2^-24 and c = 2 (the column solve multiplies by an
explicit inverse of a well-conditioned 128- or 256-column diagonal tile, so its rounding errors grow by that
tile's condition number, below 4 here)."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nb,pad", [(256, 256, 0), (257, 256, 1), (300, 512, 0), (512, 384, 3), (640, 512, 0), (1025, 256, 0),
                                      (6144, 512, 0), (6145, 512, 0), (6200, 384, 0)])
def test_spotrf_and_factor(handle, n, nb, pad):
    import torch

    g = torch.Generator(device="cuda").manual_seed(n)
    A = torch.empty(n, n + pad, device="cuda").uniform_(-0.5, 0.5, generator=g)
    A[:, :n].diagonal().add_(n**0.5)  # row j is column j of the matrix: the upper half of A here is its lower triangle
    W = A.clone()
    r = handle.spotrf_L(W, n, n + pad, nb)
    assert r.info == 0
    L = W[:, :n].double().triu()
    S = A[:, :n].double().triu()
    s = S.diagonal().sqrt()
    err = ((L.T @ L - S).triu() / s[:, None] / s[None, :]).abs().max().item()
    assert err <= 4 * 2 * n * 2.0**-24, err
    if pad == 0:  # the same through a factor object: solves with its panels' inverses, refined
        Sd = (S + S.triu(1).T).contiguous()
        B = torch.randn(3, n, dtype=torch.float64, device="cuda", generator=g)
        X = torch.empty_like(B)
        with handle.factor(Sd, n, n, nb, "fp32") as F:
            it, be = F.refine(Sd, n, B, n, X, n, 3, 1e-14)
        assert be <= 1e-14 and it <= 5
