"""Weights written in place directly before a forward, on its stream: the forward reads its weights ahead of the end of the kernel in
front of it where that kernel lets it (programmatic dependent launch), which an ordinary writer does not."""
import pytest
import torch

import workloads as wl
from libortho_b200 import _lib

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def write(src, weight, scales):
    """By kernels (a copy of a contiguous tensor would be a memory copy, behind which every kernel waits)."""
    torch.mul(src.base_scales, 1, out=scales)
    torch.bitwise_or(src.base_weight, 0, out=weight)


@pytest.mark.parametrize("density", [0.0, 0.005])
@pytest.mark.parametrize("M", [1, 12, 16, 24, 100, 200])
def test_weights_written_directly_before_a_forward(M, density):
    K, N = 4096, 8192
    a = wl.make_layer(K, N, density, seed=1, device=DEV)
    m = a.to_module()
    x = wl.make_input(M, K, seed=M, device=DEV)
    sources = [(wl.make_layer(K, N, 0.0, seed=s, device=DEV)) for s in (2, 3)]
    weight, scales = m.base_weight.clone(), m.base_scales.clone()
    m.base_weight, m.base_scales = weight, scales
    want = []
    for s in sources:
        write(s, weight, scales)
        torch.cuda.synchronize()
        want.append(m(x))
    torch.cuda.synchronize()
    got = []
    for i in range(16):
        write(sources[i & 1], weight, scales)
        got.append(m(x))
    for i, y in enumerate(got):
        assert torch.equal(y, want[i & 1]), i
    # the same as nodes of a graph
    graph, stage = torch.cuda.CUDAGraph(), wl.make_layer(K, N, 0.0, seed=4, device=DEV)
    with torch.cuda.graph(graph):
        write(stage, weight, scales)
        y = m(x)
    for i in range(4):
        stage.base_scales.copy_(sources[i & 1].base_scales)
        stage.base_weight.copy_(sources[i & 1].base_weight)
        graph.replay()
        assert torch.equal(y, want[i & 1]), i
    assert _lib.lib().ortho_b200_query_kernel_status() == 0
