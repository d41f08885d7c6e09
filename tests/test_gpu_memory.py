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
