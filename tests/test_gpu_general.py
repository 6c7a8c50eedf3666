"""The tensor-core kernel that serves gathered sparse terms and the peer exchange above 128 tokens, in all of its forms on one
GPU: sparse term inactive, folded into the weight tile and gathered, long rows from their pre-pass in each, rows whose scale
the weight tile cannot fold, unordered columns.  Against the operator in 64 bits; bounds as in test_gpu_tiles."""
import pytest
import torch

import workloads as wl
from libortho_b200 import _C_ops, _lib
from test_gpu_tiles import DEV, check, dense, forward

pytestmark = pytest.mark.gpu


@pytest.fixture
def general():
    assert _lib.lib().ortho_b200_set_decode_config(-8, 0, 0, 0) == 0
    yield
    assert _lib.lib().ortho_b200_set_decode_config(-8, 0, 0, 1) == 0
    assert _lib.lib().ortho_b200_set_decode_config(-6, 0, 0, 1) == 0


def backwards(layer):
    rows = torch.repeat_interleave(torch.arange(layer.N, device=DEV), (layer.row_ptr[1:] - layer.row_ptr[:-1]).long())
    order = torch.argsort(rows * layer.K + (layer.K - 1 - layer.col.long()))
    return wl.Layer(layer.K, layer.N, layer.base_weight, layer.base_scales, layer.row_ptr, layer.col[order].contiguous(),
                    layer.vals[order].contiguous(), 1.0)


@pytest.mark.parametrize("K,N,d,kind", [(96, 130, 0.05, "gauss"), (1184, 300, 0.02, "gauss"), (4096, 1100, 0.01, "zipf"),
                                        (2048, 260, 0.02, "zipf"), (512, 4736, 0.005, "gauss")])
def test_every_form_of_the_general_kernel(general, K, N, d, kind):
    layer = wl.make_layer(K, N, d, seed=K + N, device=DEV, ortho=kind)
    layer.base_scales[3::41] = 0.0                          # some of them long rows where the layer has any
    layer.base_scales[7::67] = 6e-8
    w, s = dense(layer)
    counts = layer.row_ptr[1:] - layer.row_ptr[:-1]
    limit = max(64, 4 * -(-layer.nnz // N))
    assert (int(counts.max()) > limit) == (kind == "zipf") and bool((counts[3::41] > 0).any())
    rev = backwards(layer)
    for M in (129, 256, 257, 513):
        x = wl.make_input(M, K, seed=M, device=DEV)
        ref = x.double() @ (w + 0.75 * s).T
        check(forward(layer, x, 0.0, None), x.double() @ w.T, f"base only M={M}")
        plan = _C_ops.Plan(layer.row_ptr, layer.col, layer.vals, K, N)
        assert plan.rows_ordered
        before = _lib.lib().ortho_b200_launch_count()
        y = forward(layer, x, 0.75, plan)
        pre = _lib.lib().ortho_b200_launch_count() - before - 1
        assert (pre > 0) == (kind == "zipf")                # the long rows' GEMM (and the sum of its shares)
        check(y, ref, f"folded M={M}")
        assert torch.equal(y, forward(layer, x, 0.75, plan))
        _lib.lib().ortho_b200_set_decode_config(-6, 0, 0, 0)
        check(forward(layer, x, 0.75, plan), ref, f"gathered M={M}")
        _lib.lib().ortho_b200_set_decode_config(-6, 0, 0, 1)
        check(forward(layer, x, 0.75, None), ref, f"raw CSR M={M}")
        back = _C_ops.Plan(rev.row_ptr, rev.col, rev.vals, K, N)
        assert not back.rows_ordered
        check(forward(rev, x, 0.75, back), ref, f"unordered M={M}")
    assert _lib.lib().ortho_b200_query_kernel_status() == 0
