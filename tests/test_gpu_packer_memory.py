"""The packer and the sieve where there is no memory for what makes them faster: the forms without it, the same results."""
import pytest
import torch

from libortho_b200 import _C_ops

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture
def small_allocations_only(monkeypatch):
    real, refused = torch.empty, []

    def empty(*size, **kw):
        n = torch.Size(size if isinstance(size[0], int) else size[0]).numel()
        if kw.get("dtype") in (torch.uint8, torch.int32) and n >= limit[0]:
            refused.append(n)
            raise torch.OutOfMemoryError("no room")
        return real(*size, **kw)
    limit = [1 << 62]
    monkeypatch.setattr(torch, "empty", empty)
    return limit, refused


def test_csr_without_room_for_marks(small_allocations_only):
    limit, refused = small_allocations_only
    w = torch.where(torch.rand(300, 4096, device=DEV) < 0.01, torch.randn(300, 4096, device=DEV), torch.zeros((), device=DEV))
    want = _C_ops.pack_ortho_csr(w)
    limit[0] = 300 * 4096 // 32                        # the marks are the first to reach it
    got = _C_ops.pack_ortho_csr(w)
    assert len(refused) == 1 and all(torch.equal(a, b) for a, b in zip(got, want))


def test_sieve_without_room_for_candidates(small_allocations_only):
    limit, refused = small_allocations_only
    N, K = 2500, 4096
    w, h = torch.randn(N, K, device=DEV) * 0.02, torch.rand(K, device=DEV) + 0.05
    want = _C_ops.hessian_sieve(w, h, keep_top_k=N * K // 100)
    limit[0] = N * K // 2
    got = _C_ops.hessian_sieve(w, h, keep_top_k=N * K // 100)
    assert len(refused) == 1 and all(torch.equal(a, b) for a, b in zip(got, want))
