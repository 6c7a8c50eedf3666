"""Layers over one input, up to 16 tokens: one streaming launch or a launch of the tensor-core kernel per layer, whichever is faster
for the group; on either side of that line the outputs are those of each layer's own forward."""
import pytest
import torch

import workloads as wl
from libortho_b200 import _C_ops, _lib

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("K,Ns,M,density,launches", [
    (8192, (2048, 2048), 12, 0.003, 1), (8192, (2048, 2048), 16, 0.003, 2), (8192, (2048, 2048), 16, 0.0, 2),
    (4096, (8192, 8192), 12, 0.003, 1), (4096, (11008, 11008), 16, 0.0, 2), (4096, (11008, 11008), 9, 0.0, 1),
    (8192, (8192, 1024, 1024), 12, 0.0, 1), (8192, (8192, 1024, 1024), 16, 0.0, 3), (8192, (28672, 28672), 3, 0.0, 1),
])
def test_group_of_layers_in_one_launch_or_apart(K, Ns, M, density, launches):
    made = {N: wl.make_layer(K, N, density, seed=N, device=DEV) for N in set(Ns)}
    plans = [_C_ops.Plan(made[N].row_ptr, made[N].col, made[N].vals, K, N) if density else None for N in Ns]
    layers = [(made[N].base_weight, made[N].base_scales, made[N].vals, made[N].col, made[N].row_ptr) for N in Ns]
    x = wl.make_input(M, K, seed=M, device=DEV)
    outs = [torch.empty(M, N, dtype=torch.float16, device=DEV) for N in Ns]
    n0 = _lib.lib().ortho_b200_launch_count()
    _C_ops.forward_multi(layers, x, outs, plans=plans)
    assert _lib.lib().ortho_b200_launch_count() - n0 == launches
    for layer, plan, N, y in zip(layers, plans, Ns, outs):
        own = torch.empty_like(y)
        _C_ops.forward(*layer, x, own, 1.0, plan=plan)
        # both sum in FP32, in other orders, and round once to FP16: a unit in the last place apart at most
        assert torch.allclose(y.float(), own.float(), rtol=2.0 ** -9, atol=2.0 ** -12 * own.float().abs().max().item())
    assert _lib.lib().ortho_b200_query_kernel_status() == 0
