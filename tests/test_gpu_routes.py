"""Layers of short rows at 9 to 16 tokens run the tensor-core kernel by themselves: the bits are those of the call that is made to."""
import pytest
import torch

import workloads as wl
from libortho_b200 import _lib

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("K,N", [(512, 33200), (1024, 16592), (2048, 8288), (3072, 5520)])
@pytest.mark.parametrize("M", [9, 16])
def test_short_rows(K, N, M):
    layer = wl.make_layer(K, N, 0.003, seed=3, device=DEV)
    x = wl.make_input(M, K, seed=M, device=DEV)
    own, made, streamed = layer.to_module(), layer.to_module(), layer.to_module()
    y = own(x)
    L = _lib.lib()
    try:
        assert L.ortho_b200_set_decode_config(-4, 0, 0, 128) == 0
        want = made(x)
        assert L.ortho_b200_set_decode_config(-4, 0, 128, 128) == 0
        other = streamed(x)
    finally:
        assert L.ortho_b200_set_decode_config(-4, 0, 0, 0) == 0
    assert torch.equal(y, want)
    assert not torch.equal(y, other)                          # (the sums' order shows in some last places)
    assert torch.allclose(y.float(), other.float(), rtol=2.0 ** -9, atol=2.0 ** -12 * other.float().abs().max().item())
