"""Activations of other types than FP16: the same bits as converting around the FP16 forward, on every kernel that takes them (and the
calls it leaves to the general code), and the native host path against the general one."""
import pytest
import torch

import workloads as wl
from libortho_b200 import _C_ops, _lib
from libortho_b200.ortho_linear import _SharedWorkspace

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def bits(t):
    return t.contiguous().view(torch.int16 if t.element_size() == 2 else torch.int32)


@pytest.mark.parametrize("K,N,d,kind", [(512, 200, 0.02, "gauss"), (4096, 1100, 0.01, "zipf"), (8192, 2048, 0.003, "gauss"), (1184, 96, 0.05, "gauss")])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("bias", [False, True])
def test_other_types_have_the_bits_of_converting_around(K, N, d, kind, dtype, bias):
    layer = wl.make_layer(K, N, d, seed=K + N, device=DEV, ortho=kind)
    m = layer.to_module()
    if bias:
        m.bias = torch.nn.Parameter(torch.randn(N, generator=torch.Generator().manual_seed(N)).to(DEV), requires_grad=False)
    for M in (1, 2, 7, 16, 17, 64, 100, 128, 129, 400):
        x = torch.randn(M, K, generator=torch.Generator().manual_seed(M)).to(DEV).to(dtype)
        x[0, 3], x[M // 2, 5] = 1e5, 3e-6                     # beyond FP16's range: infinite; below its normal range
        for alpha in (0.0, 0.75):
            m.set_alpha(alpha)
            want = m(x.to(torch.float16)).to(dtype)
            for _ in range(2):
                y = m(x)
                assert y.dtype == dtype and y.shape == (M, N)
                ok = bits(y) == bits(want)
                assert bool((ok | (y.isnan() & want.isnan())).all()), (M, alpha)
            assert torch.equal(bits(m(x.view(1, M, K)).nan_to_num()), bits(want.view(1, M, N).nan_to_num()))
            strided = torch.empty(M, K + 32, dtype=dtype, device=DEV)[:, :K]
            strided.copy_(x)
            assert torch.equal(bits(m(strided).nan_to_num()), bits(want.nan_to_num()))
    assert _lib.lib().ortho_b200_query_kernel_status() == 0


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("M", [1, 16, 24, 200])
def test_activations_that_are_not_16_byte_aligned(M, dtype):
    K, N = 1024, 256
    m = wl.make_layer(K, N, 0.01, seed=3, device=DEV).to_module()
    x = wl.make_input(M, K, seed=M, device=DEV).to(dtype)
    want = m(x.to(torch.float16)).to(dtype)
    buf = torch.zeros(M * K + 8, dtype=dtype, device=DEV)
    for call in range(2):                                     # with no record of that type yet, and with one
        for offset in (1, 2, 3):
            odd = buf[offset:offset + M * K].view(M, K).copy_(x)
            assert odd.data_ptr() % 16 and torch.equal(bits(m(odd)), bits(want)), (call, offset)
        assert torch.equal(bits(m(x)), bits(want))


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.float32])
@pytest.mark.parametrize("M", [1, 40])
def test_activations_with_a_negation_pending(M, dtype):
    K, N = 1024, 256
    m = wl.make_layer(K, N, 0.01, seed=3, device=DEV).to_module()
    x = wl.make_input(M, K, seed=M, device=DEV).to(dtype)
    want = m(-x)
    assert torch.equal(bits(m(torch._neg_view(x))), bits(want))
    m(x)
    assert torch.equal(bits(m(torch._neg_view(x))), bits(want))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_a_route_that_changed_since_the_record_was_made(dtype):
    K, N = 4096, 4096
    m = wl.make_layer(K, N, 0.002, seed=4, device=DEV).to_module()
    L = _lib.lib()
    for M, hook, builtin in ((200, (-8, 0, 0, 0), (-8, 0, 0, 1)), (12, (-4, 0, 8, 128), (-4, 0, 0, 0))):
        x = wl.make_input(M, K, seed=M, device=DEV).to(dtype)
        m(x)
        assert L.ortho_b200_set_decode_config(*hook) == 0
        try:
            want = m(x.to(torch.float16)).to(dtype)
            for _ in range(2):
                assert torch.equal(bits(m(x)), bits(want)), (M, hook)
        finally:
            assert L.ortho_b200_set_decode_config(*builtin) == 0
    # alpha > 0 in Python and 0 as a float: the base alone, which from 12 tokens on another kernel computes
    x = wl.make_input(12, K, seed=5, device=DEV).to(dtype)
    m(x)
    m.set_alpha(1e-60)
    y = m(x)
    m.set_alpha(0.0)
    assert torch.allclose(y.float(), m(x).float(), rtol=2e-3 if dtype == torch.float32 else 1.6e-2, atol=1e-2)


@pytest.mark.parametrize("M", [1, 24, 200])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_buffers_replaced_or_edited_between_calls(M, dtype):
    K, N = 1024, 256
    a, b = (wl.make_layer(K, N, 0.01, seed=s, device=DEV) for s in (1, 2))
    m, other = a.to_module(), b.to_module()
    x = wl.make_input(M, K, seed=M, device=DEV).to(dtype)
    y0, want = m(x), other(x)
    m(x)
    m.base_weight.data, m.base_scales.data = b.base_weight.clone(), b.base_scales.clone()
    m._buffers["ortho_values"], m._buffers["ortho_col_indices"], m._buffers["ortho_row_ptr"] = b.vals.clone(), b.col.clone(), b.row_ptr.clone()
    assert torch.equal(m(x), want)
    m.ortho_values.mul_(0.0)                                  # in place: the version counter says so
    m.set_alpha(0.0)
    base = m(x)
    m.set_alpha(1.0)
    assert torch.equal(m(x), base)
    c = wl.make_layer(K, N, 0.01, seed=1, device=DEV)         # (a's tensors hold b's data by now)
    m.base_weight, m.base_scales = c.base_weight, c.base_scales
    m.ortho_values, m.ortho_col_indices, m.ortho_row_ptr = c.vals, c.col, c.row_ptr
    assert torch.equal(m(x), y0)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        y1 = m(x)
    side.synchronize()
    assert torch.equal(y1, y0)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_a_sparse_component_that_goes_and_comes_back(dtype):
    """By `.data =`, which changes neither the buffers' identity nor their versions: no record of the first plan is left when
    it returns."""
    K, N = 1024, 256
    a, b = (wl.make_layer(K, N, 0.01, seed=s, device=DEV) for s in (1, 2))
    m = a.to_module()
    xs = [wl.make_input(M, K, seed=M, device=DEV).to(dtype) for M in (1, 24, 200)]
    want = [m(x) for x in xs]
    own = [t.data for t in (m.ortho_values, m.ortho_col_indices, m.ortho_row_ptr)]

    def put(vals, col, row_ptr):
        m.ortho_values.data, m.ortho_col_indices.data, m.ortho_row_ptr.data = vals, col, row_ptr
    put(b.vals, b.col, b.row_ptr)
    changed = m(xs[0])
    assert len(m._bound) == 1 and not torch.equal(changed, want[0])
    put(*own)
    for x, y in zip(xs, want):
        assert torch.equal(m(x), y)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_the_converted_activations_are_a_temporary_of_the_call(dtype):
    K, N = 4096, 256
    m = wl.make_layer(K, N, 0.01, seed=3, device=DEV).to_module()
    side = torch.cuda.Stream()                                # with a scratch buffer of its own
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        for M in (24, 400):
            x = wl.make_input(M, K, seed=M, device=DEV).to(dtype)
            want = m(x.to(torch.float16)).to(dtype)
            held = [w.tensor.numel() for (_, stream), w in _SharedWorkspace._by_stream.items() if stream == side.cuda_stream]
            before = torch.cuda.memory_allocated()
            y = m(x)
            assert held == [w.tensor.numel() for (_, stream), w in _SharedWorkspace._by_stream.items() if stream == side.cuda_stream]
            assert torch.cuda.memory_allocated() - before <= (y.numel() * y.element_size() + 511) // 512 * 512
            assert torch.equal(bits(y), bits(want)) and torch.equal(bits(m(x)), bits(want))
    side.synchronize()


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.float32])
@pytest.mark.parametrize("M", [1, 40, 300])
def test_capture_replays_on_new_activations(M, dtype):
    K, N = 2048, 512
    m = wl.make_layer(K, N, 0.01, seed=3, device=DEV).to_module()
    x = wl.make_input(M, K, seed=1, device=DEV).to(dtype)
    m(x)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        y = m(x)
    for seed in (2, 3):
        x.copy_(wl.make_input(M, K, seed=seed, device=DEV))
        g.replay()
        assert torch.equal(y, m(x))


def test_what_the_native_path_leaves_to_the_general_code():
    K, N = 512, 128
    layer = wl.make_layer(K, N, 0.02, seed=1, device=DEV)
    m = layer.to_module()
    x = wl.make_input(3, K, seed=1, device=DEV)
    y = m(x)
    with pytest.raises(RuntimeError):
        m(x[:, :-32])
    assert torch.equal(m(x.double()), y.double()) and m(x[:0]).shape == (0, N)
    assert torch.equal(m(x[0]), y[0])
    m.bias = torch.nn.Parameter(torch.ones(N, dtype=torch.float16, device=DEV), requires_grad=False)      # added by torch
    assert torch.equal(m(x), y + 1)
    assert torch.equal(m(x.float()), (y + 1).float())
    out = torch.empty(3, N, dtype=torch.float16, device=DEV)
    with pytest.raises(ValueError):
        _C_ops.forward(layer.base_weight, layer.base_scales, layer.vals, layer.col, layer.row_ptr[:-1], x, out, 1.0)
    with pytest.raises(TypeError):
        _C_ops.forward(layer.base_weight, layer.base_scales, layer.vals, layer.col, layer.row_ptr, x.float(), out, 1.0)
    _C_ops.forward(layer.base_weight, layer.base_scales, layer.vals, layer.col, layer.row_ptr, x, out, 1)
    ref = x.double() @ (torch.zeros(N, K, dtype=torch.float64, device=DEV)).T
    assert out.shape == ref.shape and torch.allclose(out.float(), y.float(), atol=2e-2, rtol=2e-3)
