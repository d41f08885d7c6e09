"""Device memory that calls hold beside what their callers gave them."""
import pytest

pytestmark = pytest.mark.gpu


def _free():
    import torch

    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def test_dpotrf_keeps_at_most_256_mib_of_planes(ooc):
    """The digit planes of n = 20000, nb = 512 take 28 * 512 bytes a row, 287 MB: more than a handle keeps."""
    import torch

    n, nb = 20000, 512
    A = torch.zeros(n, n, dtype=torch.float64, device="cuda")
    A.diagonal().fill_(4.0)
    with ooc.Handle(0) as h:
        W = torch.eye(3000, dtype=torch.float64, device="cuda")
        assert h.dpotrf_L(W, 3000, 3000, nb, 0).info == 0  # (modules loaded; 43 MB of planes, kept)
        before = _free()
        assert h.dpotrf_L(A, n, n, nb, 0).info == 0
        assert before - _free() <= 0
    assert torch.equal(A.diagonal(), torch.full((n,), 2.0, dtype=torch.float64, device="cuda"))


def _spd32(n, lda):
    import numpy as np

    rng = np.random.default_rng(n)
    A = np.full((lda, n), 5.0, dtype=np.float32, order="F")
    R = rng.uniform(-0.5, 0.5, (n, n)).astype(np.float32)
    A[:n] = np.tril(R) + np.tril(R, -1).T + np.float32(n**0.5) * np.eye(n, dtype=np.float32)
    return A


def _check32(A, L, n):
    """|A - L L^T| <= 4 (n + 2) 2^-24 sqrt(a_ii a_jj), the bar of test_gpu_fp32_digits.py."""
    import torch

    A, L = (torch.from_numpy(M[:n].copy()).cuda().double().tril() for M in (A, L))
    d = A.diagonal().sqrt()
    err = ((A - (L @ L.T).tril()).abs() / d[:, None] / d[None, :]).max().item()
    assert err <= 4 * (n + 2) * 2.0**-24, err


@pytest.mark.parametrize("n,nb,extra", [(6000, 512, 0), (6000, 512, 30 << 20), (5001, 256, 4096), (4000, 512, 1 << 20)])
def test_spotrf_out_of_core_stays_within_its_budget(ooc, n, nb, extra):
    """Buffers (kept by the handle after the call, so what is free tells) within the budget, two tiles and the allocator's
    2 MiB a buffer."""
    A = _spd32(n, n)
    L = A.copy(order="F")
    budget = 12 * n * nb + extra
    with ooc.Handle(0) as h:
        assert h.spotrf_L(_spd32(600, 600), 600, 600, nb).info == 0  # modules loaded
        before = _free()
        r = h.spotrf_L(L, n, n, nb, budget)
        assert r.info == 0 and r.stats["npanels"] >= 2
        copies = 4 * n * 512 if n % 4 else 0  # (an aligned copy of an odd-order panel for the FP32 pipe)
        assert before - _free() <= budget + copies + 8 * nb * nb + (5 << 21)
    _check32(A, L, n)


@pytest.mark.parametrize("n,lda,nb", [(777, 777, 512), (1100, 1101, 512), (1000, 1000, 256), (701, 703, 128), (300, 300, 100)])
def test_spotrf_in_core_budget_without_room_for_planes(ooc, handle, n, lda, nb):
    """The matrix fits the budget exactly: the FP32 pipe makes the updates, in both calls of a split one."""
    A = _spd32(n, lda)
    L = A.copy(order="F")
    assert handle.spotrf_L(L, n, lda, nb, 4 * n * n).info == 0
    _check32(A, L, n)


@pytest.mark.parametrize("kind", ["fp32", "fp64", "out of core"])
def test_server_admits_by_what_a_request_holds(ooc, kind):
    """A budget with room for all of a request but its digit planes: admitted, factored without them; one byte less is
    refused.  The planes: FP32 8 bytes a row for each of nb columns and 8 bytes of exponents, FP64 14 bytes
    for each of 512 columns and 16 of exponents, which factor_bytes counts; out of core twice that, per job."""
    from oocdag_gb300.server import Server

    n, nb = 4096, 512
    prec = "fp32" if kind == "fp32" else "fp64"
    planes = n * (8 * nb + 8) if kind == "fp32" else n * (14 * 512 + 16)
    assert ooc.factor_bytes(n, nb, prec) >= (4 if kind == "fp32" else 8) * n * n + planes
    if kind == "out of core":
        opts = dict(ooc_min_n=n, ooc_budget=96 << 20)
        least = (96 << 20) + 16 * n * nb + 64 * n + (64 << 20)
    else:
        opts, least = {}, ooc.factor_bytes(n, nb, prec) - planes + 64 * n + (64 << 20)
    for budget, status in ((least + 2 * planes, 0), (least, 0), (least - 1, ooc.OOC_ERR_BUDGET)):
        with Server(workers=1, nb=nb, prec=prec, hbm_budget=budget, **opts) as S:
            i = S.submit(n=n, matrix_seed=1, rhs_seed=2, key=1)
            done = []
            for _ in range(120):
                done = S.poll(wait_ms=1000)
                if done:
                    break
            assert [d["id"] for d in done] == [i] and done[0]["status"] == status, (budget, done, S.last_error())
            assert status or done[0]["backward_error"] <= 1e-14
