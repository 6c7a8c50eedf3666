"""Calls that the native host path serves by itself: activations of a type that their kernel does not take, converted around the FP16
forward, and function-level calls that need scratch."""
import pytest
import torch

import workloads as wl
from libortho_b200 import OrthoLinear, _C_ops, _lib

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def bits(t):
    return t.contiguous().view(torch.int16 if t.element_size() == 2 else torch.int32)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("K,N,M", [(544, 256, 4), (8032, 470, 7), (2912, 1003, 16)])
def test_a_type_that_the_kernel_does_not_take(K, N, M, dtype, monkeypatch):
    m = wl.make_layer(K, N, 0.01, seed=3, device=DEV).to_module()
    xs = [wl.make_input(M, K, seed=s, device=DEV).to(dtype) for s in (1, 2)]
    for alpha in (1.0, 0.0, 0.5):
        m.set_alpha(alpha)
        want = [m(x.to(torch.float16)).to(dtype) for x in xs]
        for _ in range(2):
            for x, y in zip(xs, want):
                assert torch.equal(bits(m(x)), bits(y))
        shaped = m(xs[0].view(1, M, K))
        assert shaped.shape == (1, M, N) and shaped.dtype == dtype and torch.equal(bits(shaped[0]), bits(want[0]))
        with monkeypatch.context() as patch:               # the Python code compares versions on each call
            patch.setattr(OrthoLinear, "_versions", None)
            for x, y in zip(xs, want):
                assert torch.equal(bits(m(x)), bits(y))
    # other buffers are noticed
    other = wl.make_layer(K, N, 0.01, seed=4, device=DEV)
    m.base_weight = other.base_weight
    assert torch.equal(bits(m(xs[0])), bits(m(xs[0].to(torch.float16)).to(dtype)))
    m.ortho_values.mul_(2)
    assert torch.equal(bits(m(xs[0])), bits(m(xs[0].to(torch.float16)).to(dtype)))
    # and a capture replays on new activations
    graph, x = torch.cuda.CUDAGraph(), xs[0].clone()
    want = m(xs[1])
    with torch.cuda.graph(graph):
        y = m(x)
    x.copy_(xs[1])
    graph.replay()
    assert torch.equal(bits(y), bits(want))


@pytest.mark.parametrize("density", [0.0, 0.01])
@pytest.mark.parametrize("M", [24, 100, 300])
def test_function_level_calls_with_scratch(M, density, monkeypatch):
    K, N = 1024, 384
    layer = wl.make_layer(K, N, density, seed=3, device=DEV)
    plan = _C_ops.Plan(layer.row_ptr, layer.col, layer.vals, K, N) if density else None
    args = (layer.base_weight, layer.base_scales, layer.vals, layer.col, layer.row_ptr)
    x = wl.make_input(M, K, seed=M, device=DEV)
    need = _C_ops.workspace_bytes(M, K, N, plan)
    assert need > 0
    want = layer.to_module()(x)
    room, little = (torch.empty(n, dtype=torch.uint8, device=DEV) for n in (need, need // 2))
    with monkeypatch.context() as patch:                   # the Python code goes through the loaded library
        patch.setattr(_lib, "lib", None)
        for ws in (None, room, little, room.view(-1, 2)):
            y = torch.zeros(M, N, dtype=torch.float16, device=DEV)
            _C_ops.forward(*args, x, y, 1.0, plan=plan, workspace=ws)
            assert torch.equal(y, want)
            ys = [torch.zeros_like(y) for _ in range(2)]
            _C_ops.forward_multi([args, args], x, ys, plans=[plan, plan], workspace=ws)
            assert torch.equal(ys[0], want) and torch.equal(ys[1], want)
    assert _lib.lib().ortho_b200_query_kernel_status() == 0
