"""The one-pass form of the device-side sieve and the packer's two-call form: bit for bit the torch chain (and the forms that read W
more often), where the sample brackets the threshold well, badly or not at all, and where the list of candidates overflows."""
import pytest
import torch

from libortho_b200 import _C_ops, _lib, sieve

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def bits(t):
    return t.contiguous().view(torch.int32)


def weights(kind, N, K):
    g = torch.Generator().manual_seed(N + K)
    w = torch.randn(N, K, generator=g) * 0.02
    h = torch.rand(K, generator=g) * 2.0 + 0.05
    if kind == "rows":                                # every other row, which the sample may miss, is ten times larger
        w[1::2] *= 10.0
    elif kind == "ties":                              # seven values: thousands of equal scores, more than the list holds
        w = torch.randint(-3, 4, (N, K), generator=g) * 0.013
        h = torch.ones(K)
    elif kind == "zeros":                             # rows of zeros and of tiny weights, negative curvature
        w[::3] = 0.0
        w[1] *= 1e-30
        h[5::17] = -0.3
    elif kind == "outlier":                           # a few weights hold all of the large scores
        w[:, 3] = 2.0 * torch.rand(N, generator=g)
    return w, h


@pytest.mark.parametrize("kind", ["gauss", "rows", "ties", "zeros", "outlier"])
@pytest.mark.parametrize("N,K,target", [(300, 1024, 0.001), (5000, 2052, 0.01), (5000, 2048, 0.04), (10000, 1024, 0.02), (1300, 8200, 0.003), (2500, 4096, 0.001)])
def test_sieve_by_one_pass(kind, N, K, target):
    w, h = weights(kind, N, K)
    base_ref, ortho_ref = sieve.hessian_sieve(w, h, sparsity_target=target)
    base, ortho = sieve.hessian_sieve(w.to(DEV), h.to(DEV), sparsity_target=target)
    assert torch.equal(bits(base.cpu()), bits(base_ref)) and torch.equal(bits(ortho.cpu()), bits(ortho_ref))
    # the form with the smaller scratch
    L, ww, hh = _lib.lib(), w.to(DEV), h.to(DEV)
    scratch = torch.empty(int(L.ortho_b200_sieve_scratch_bytes(N)), dtype=torch.uint8, device=DEV)
    b2, o2 = torch.empty_like(ww), torch.empty_like(ww)
    assert L.ortho_b200_sieve(ww.data_ptr(), hh.data_ptr(), N, K, 0.0, int(target * N * K), b2.data_ptr(), o2.data_ptr(),
                              scratch.data_ptr(), scratch.numel(), torch.cuda.current_stream().cuda_stream) == 0
    assert torch.equal(bits(b2), bits(base)) and torch.equal(bits(o2), bits(ortho))


@pytest.mark.parametrize("kind", ["gauss", "zeros"])
@pytest.mark.parametrize("over", ["none", "base", "residual"])
@pytest.mark.parametrize("keep", [-1, 0])
def test_sieve_with_a_given_threshold(kind, over, keep):
    N, K = 320, 4104
    w, h = weights(kind, N, K)
    base_ref, ortho_ref = sieve.hessian_sieve(w, h, curvature_thresh=2e-5, sparsity_target=None if keep < 0 else 0.0)
    L, ww, hh = _lib.lib(), w.to(DEV), h.to(DEV)
    scratch = torch.empty(int(L.ortho_b200_sieve_scratch_bytes(N)), dtype=torch.uint8, device=DEV)
    b = ww if over == "base" else torch.empty_like(ww)
    o = ww if over == "residual" else torch.empty_like(ww)
    assert L.ortho_b200_sieve(ww.data_ptr(), hh.data_ptr(), N, K, 2e-5, keep, b.data_ptr(), o.data_ptr(),
                              scratch.data_ptr(), scratch.numel(), torch.cuda.current_stream().cuda_stream) == 0
    assert torch.equal(bits(b.cpu()), bits(base_ref)) and torch.equal(bits(o.cpu()), bits(ortho_ref))


@pytest.mark.parametrize("N,K", [(1, 8), (9, 136), (70, 4096), (33, 8320)])
@pytest.mark.parametrize("density", [0.0, 0.01, 0.05, 0.5, 1.0])
def test_csr_from_marks(N, K, density):
    g = torch.Generator().manual_seed(N * K)
    w = torch.where(torch.rand(N, K, generator=g) < density, torch.randn(N, K, generator=g), torch.zeros(()))
    if N > 8:
        w[2], w[5] = 1.5, 0.0                         # a full and an empty row
        w[7, -1], w[8, 0] = float("inf"), -0.0
    row_ptr, col, val = sieve.pack_ortho_sparse(w)
    r, c, v = _C_ops.pack_ortho_csr(w.to(DEV))
    assert torch.equal(r.cpu(), row_ptr) and torch.equal(c.cpu(), col)
    assert torch.equal(v.cpu().view(torch.int16), val.to(torch.float16).view(torch.int16))
    L, ww, nnz = _lib.lib(), w.to(DEV), int(row_ptr[-1])
    marks = torch.empty(int(L.ortho_b200_csr_marks_bytes(N, K)), dtype=torch.uint8, device=DEV)
    r2, c2, v2 = torch.empty_like(r), torch.empty(nnz, dtype=torch.int32, device=DEV), torch.empty(nnz, dtype=torch.float16, device=DEV)
    st = torch.cuda.current_stream().cuda_stream
    assert L.ortho_b200_csr_count_marks(ww.data_ptr(), N, K, r2.data_ptr(), marks.data_ptr(), st) == 0
    assert L.ortho_b200_csr_fill_marks(ww.data_ptr(), N, K, r2.data_ptr(), marks.data_ptr(), c2.data_ptr(), v2.data_ptr(), st) == 0
    assert torch.equal(r2, r) and torch.equal(c2, c) and torch.equal(v2.view(torch.int16), v.view(torch.int16))


@pytest.mark.parametrize("K", [8, 4088, 4096, 4104, 8192, 8200, 17000])
@pytest.mark.parametrize("given", [False, True])
def test_packed_base_of_rows_held_and_read_again(K, given):
    N = 13
    g = torch.Generator().manual_seed(K)
    w = torch.randn(N, K, generator=g) * 0.02
    s = torch.rand(N, generator=g) * 0.01 + 1e-3 if given else None
    q, qs = _C_ops.pack_base(w.to(DEV), s.to(DEV) if given else None)
    scales = s if given else (w.abs().max(dim=1)[0] / 7.0).clamp(min=1e-6)
    w_int = (w / scales.unsqueeze(1)).round().clamp(-8, 7).to(torch.int8).flatten()
    packed = ((w_int[0::2] & 0x0F) | ((w_int[1::2] & 0x0F) << 4)).to(torch.uint8).view(N, -1)
    assert torch.equal(q.cpu(), packed) and torch.equal(qs.cpu().view(torch.int16), scales.to(torch.float16).view(torch.int16))
