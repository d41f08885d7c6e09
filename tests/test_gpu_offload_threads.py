"""Tile calls of one worker rank from two threads: a product keeps its own status word, so that neither a factorization's
info is cleared before it is read nor a product skipped because the matrix beside it was not definite."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_products_beside_a_failing_factorization(ooc, handle):
    import torch

    from oocdag_gb300 import offload as off

    assert off.init(0) == 0
    nb, bad, rounds = 128, 77, 300
    A = torch.eye(nb, dtype=torch.float64, device="cuda") * 4
    A[bad, bad] = -1.0
    rng = np.random.default_rng(0)
    # integers: products and sums of them are exact
    X = torch.from_numpy(rng.integers(-8, 9, (nb, nb)).astype(np.float64)).cuda()
    want = X.T @ X
    W = [torch.empty_like(A) for _ in range(rounds)]
    C = [torch.zeros_like(A) for _ in range(rounds)]
    for w in W:
        w.copy_(A)
    torch.cuda.synchronize()
    infos, errors = [], []

    def factor():
        for w in W:
            infos.append(off.dpotrf("L", nb, w, nb))

    def product():
        for c in C:
            off.dgemm("N", "T", nb, nb, nb, 1.0, X, nb, X, nb, 0.0, c, nb)
            errors.append(off.last_error())

    threads = [threading.Thread(target=f) for f in (factor, product)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert infos == [bad + 1] * rounds
    assert errors == [0] * rounds
    for c in C:
        assert torch.equal(c, want)
