"""A bias of another type than FP32, which torch adds to the FP16 output: natively and by the Python code the same bits and gradients."""
import pytest
import torch

import workloads as wl
from libortho_b200 import OrthoLinear

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def bits(t):
    return t.detach().contiguous().view(torch.int16 if t.element_size() == 2 else torch.int32)


def reference(m, x):
    """What the Python code does, step by step, on the base of a forward without bias."""
    bias, m.bias = m.bias, None
    y = m(x.to(torch.float16))
    m.bias = bias
    y = y.clone()
    y += bias
    return y.to(x.dtype)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.float32])
@pytest.mark.parametrize("bias_dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("M", [1, 24, 200])
def test_bias_that_torch_adds(M, bias_dtype, dtype, monkeypatch):
    K, N = 1024, 384
    m = wl.make_layer(K, N, 0.01, seed=3, device=DEV).to_module()
    g = torch.Generator().manual_seed(M)
    m.bias = torch.nn.Parameter((torch.randn(N, generator=g) * 3).to(bias_dtype).to(DEV))
    x = wl.make_input(M, K, seed=M, device=DEV).to(dtype)
    want = reference(m, x)
    for _ in range(3):
        assert torch.equal(bits(m(x)), bits(want))
    with monkeypatch.context() as patch:                   # the Python code compares versions on each call
        patch.setattr(OrthoLinear, "_versions", None)
        y = m(x.view(1, M, K))
        assert y.shape == (1, M, N) and torch.equal(bits(y[0]), bits(want)) and y.requires_grad
        y.float().sum().backward()
        assert torch.equal(m.bias.grad.float(), torch.full((N,), float(M), device=DEV))
        with torch.no_grad():
            assert not m(x).requires_grad
        with torch.no_grad():                              # its contents are read anew on each forward
            m.bias.mul_(2)
        y = m(x)
    assert torch.equal(bits(y), bits(reference(m, x))) and not torch.equal(bits(y), bits(want))
    m.bias = torch.nn.Parameter(torch.ones(N, device=DEV))   # FP32 now: the kernel adds it
    assert torch.equal(bits(m(x)), bits(m(x.to(torch.float16)).to(dtype)))
    m.bias = None
    assert not m(x).requires_grad
