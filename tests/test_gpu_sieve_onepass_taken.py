"""Whether the sieve's one-pass form has produced the result: the passes behind it would write the same bits, so the outputs alone do
not tell."""
import pytest
import torch

from libortho_b200 import _lib

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
BINS = 4096


def one_pass_was_used(w, h, k):
    L, (N, K) = _lib.lib(), w.shape
    small = int(L.ortho_b200_sieve_scratch_bytes(N))
    scratch = torch.zeros(int(L.ortho_b200_sieve_onepass_scratch_bytes(N, K)), dtype=torch.uint8, device=DEV)
    base, ortho = torch.empty_like(w), torch.empty_like(w)
    assert L.ortho_b200_sieve(w.data_ptr(), h.data_ptr(), N, K, 0.0, k, base.data_ptr(), ortho.data_ptr(), scratch.data_ptr(), scratch.numel(),
                              torch.cuda.current_stream().cuda_stream) == 0
    # the state lies behind the other form's scratch: three histograms, ten words, then the flag (a static assertion beside the struct)
    at = (small + 255) // 256 * 256 + 3 * BINS * 4 + 40
    # the residual keeps every score above the k-th largest
    assert int((ortho != 0).sum()) < k
    return int(scratch[at:at + 4].view(torch.int32).item())


@pytest.mark.parametrize("N,K,share", [(5000, 2052, 0.01), (5000, 2048, 0.04), (1300, 8200, 0.003), (2500, 4096, 0.001)])
def test_one_pass_is_taken_on_ordinary_weights(N, K, share):
    g = torch.Generator().manual_seed(N)
    w, h = torch.randn(N, K, generator=g) * 0.02, torch.rand(K, generator=g) * 2.0 + 0.05
    assert one_pass_was_used(w.to(DEV), h.to(DEV), int(share * N * K)) == 1


def test_the_passes_follow_where_the_list_overflows():
    N, K = 2500, 4096
    g = torch.Generator().manual_seed(1)
    w = torch.randint(-3, 4, (N, K), generator=g) * 0.013                     # seven values: more equal scores than it holds
    assert one_pass_was_used(w.to(DEV), torch.ones(K, device=DEV), N * K // 100) == 0
