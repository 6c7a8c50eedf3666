"""Calls at the edge of what the entry points accept: infinite activations, buffers that overlap, empty plans, very tall
layers.  The reference is the CPU oracle or the same call made another way."""
import numpy as np
import pytest
import torch

import workloads as wl
from conftest import MAX_ABS_TOL, REL_FRO_TOL, layer_oracle
from libortho_b200 import _C_ops, _lib

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def multi(layer, x, alpha, plan):
    """A forward with the workspace that the sizing rule asks for."""
    y = torch.empty(x.shape[0], layer.N, dtype=torch.float16, device=DEV)
    _C_ops.forward_multi([(layer.base_weight, layer.base_scales, layer.vals, layer.col, layer.row_ptr)], x, [y], alphas=[alpha], plans=[plan])
    return y


def kinds(a):
    """0 finite, 1 +Inf, 2 -Inf, 3 NaN"""
    return np.isposinf(a) * 1 + np.isneginf(a) * 2 + np.isnan(a) * 3


@pytest.mark.parametrize("M", [1, 4, 16, 32, 100, 200])
@pytest.mark.parametrize("K,N,kind", [(512, 300, "gauss"), (256, 300, "zipf"), (4096, 200, "zipf"), (8192, 5300, "gauss")])
def test_infinite_activations_reach_the_outputs_as_the_operator_defines_them(oracle_mod, K, N, kind, M):
    """One token each with +Inf, -Inf and NaN.  Which outputs are infinite and which NaN depends on the signs of the weights in
    that column alone, and the other tokens are not touched.  (More than 128 tokens: an entry is added to the weight before
    the contraction, so rows with an entry in the infinite column are left out there.)"""
    layer = wl.make_layer(K, N, 0.01, seed=K + N, device=DEV, ortho=kind)
    plan = _C_ops.Plan(layer.row_ptr, layer.col, layer.vals, K, N)
    x = wl.make_input(M, K, seed=M, device=DEV)
    at = {0: (int(layer.col[0]), float("inf")), M // 2: (K - 3, float("-inf")), M - 1: (130, float("inf"))}
    if M >= 4:
        at[1] = (7, float("nan"))
    for m, (k, v) in at.items():
        x[m, k] = v
    y = multi(layer, x, 0.75, plan).float().cpu().numpy()
    with np.errstate(all="ignore"):
        ref = layer_oracle(oracle_mod, layer, x, 0.75)
    rows = np.repeat(np.arange(N), np.diff(layer.row_ptr.cpu().numpy()))
    cols = layer.col.cpu().numpy()
    for m in range(M):
        ok = np.ones(N, bool)
        if m in at and M > 128:
            ok[rows[cols == at[m][0]]] = False
        assert np.array_equal(kinds(y[m])[ok], kinds(ref[m])[ok]), f"token {m}"
        if m not in at:
            err = y[m] - ref[m]
            assert np.linalg.norm(err) <= REL_FRO_TOL * np.linalg.norm(ref[m]) * 2 and np.abs(err).max() <= MAX_ABS_TOL, f"token {m}"
    assert _lib.lib().ortho_b200_query_kernel_status() == 0


def test_bfloat16_activations_beyond_fp16_become_infinite_not_nan():
    """The module rounds activations to FP16: one above 65504 is infinite, and every row with a weight there says so."""
    layer = wl.make_layer(8192, 5300, 0.003, seed=4, device=DEV)
    m = layer.to_module()
    x = wl.make_input(12, 8192, seed=5, device=DEV).to(torch.bfloat16)
    x[3, 77] = 1e6
    y = m(x)
    nib = layer.base_weight[:, 77 // 2] >> 4
    entry = torch.zeros(layer.N, dtype=torch.bool, device=DEV)
    rows = torch.repeat_interleave(torch.arange(layer.N, device=DEV), (layer.row_ptr[1:] - layer.row_ptr[:-1]).long())
    entry[rows[layer.col == 77]] = True
    plain = (nib != 0) & ~entry
    assert bool(plain.any()) and torch.isinf(y[3][plain]).all()
    assert torch.isfinite(y[torch.arange(12) != 3]).all()


@pytest.mark.parametrize("over", ["residual", "base", "both"])
@pytest.mark.parametrize("N,K,keep", [(96, 512, 0.01), (40, 4096, 0.3), (7, 64, 1.0)])
def test_sieve_outputs_may_overwrite_the_weights(N, K, keep, over):
    """An output that is W itself: every element is read before it is written."""
    g = torch.Generator().manual_seed(N + K)
    w, h = (torch.randn(N, K, generator=g) * 0.02).to(DEV), (torch.rand(K, generator=g) * 2 + 0.01).to(DEV)
    scratch = torch.empty(int(_lib.lib().ortho_b200_sieve_scratch_bytes(N)), dtype=torch.uint8, device=DEV)

    def sieve(src, base, res):
        st = _lib.lib().ortho_b200_sieve(src.data_ptr(), h.data_ptr(), N, K, 0.0, int(keep * N * K), base.data_ptr(), res.data_ptr(),
                                         scratch.data_ptr(), scratch.numel(), torch.cuda.current_stream().cuda_stream)
        assert st == 0
        return base, res

    base, res = sieve(w, torch.empty_like(w), torch.empty_like(w))
    own = w.clone()
    b2, r2 = sieve(own, own if over != "residual" else torch.empty_like(w), own if over != "base" else torch.empty_like(w))
    if over != "both":                                      # (then the residual, written last, is what stays)
        assert torch.equal(b2.view(torch.int32), base.view(torch.int32))
    assert torch.equal(r2.view(torch.int32), res.view(torch.int32))


@pytest.mark.parametrize("M", [4, 8, 20, 64, 300])
def test_an_empty_plan_runs_like_no_plan(M):
    """A plan without entries asks for the workspace of a call without one and gets the same kernels and bits."""
    K, N = 28672, 1536
    layer = wl.make_layer(K, N, 0.0, seed=6, device=DEV)
    plan = _C_ops.Plan(layer.row_ptr, layer.col, layer.vals, K, N)
    x = wl.make_input(M, K, seed=M, device=DEV)
    assert _C_ops.workspace_bytes(M, K, N, plan) == _C_ops.workspace_bytes(M, K, N)
    ys, launches = [], []
    for p in (None, plan):
        before = _lib.lib().ortho_b200_launch_count()
        ys.append(multi(layer, x, 1.0, p))
        launches.append(_lib.lib().ortho_b200_launch_count() - before)
    assert torch.equal(ys[0], ys[1]) and launches[0] == launches[1]


def test_more_long_rows_than_a_grid_dimension_holds():
    """70 000 long rows of a tall, narrow layer at more than 128 tokens."""
    K, N, M, per = 64, 400000, 130, 32
    g = torch.Generator().manual_seed(9)
    layer = wl.make_layer(K, N, 0.0, seed=9, device=DEV)
    long_rows = torch.arange(0, N, 4)[:70000]
    counts = torch.zeros(N, dtype=torch.int64)
    counts[long_rows] = per
    ptr = torch.zeros(N + 1, dtype=torch.int32)
    ptr[1:] = counts.cumsum(0).to(torch.int32)
    col = torch.rand(long_rows.numel(), K, generator=g).argsort(1)[:, :per].sort(1).values.reshape(-1).to(torch.int32)
    val = (torch.randn(col.numel(), generator=g) * 0.05).to(torch.float16)
    ptr, col, val = ptr.to(DEV), col.to(DEV), val.to(DEV)
    layer = wl.Layer(K, N, layer.base_weight, layer.base_scales, ptr, col, val, 1.0)
    assert _lib.lib().ortho_b200_set_decode_config(-5, 0, 0, 8) == 0
    try:
        plan = _C_ops.Plan(ptr, col, val, K, N)            # mean row 6 entries: rows of more than 24 are long
    finally:
        _lib.lib().ortho_b200_set_decode_config(-5, 0, 0, 0)
    x = wl.make_input(M, K, seed=1, device=DEV)
    before = _lib.lib().ortho_b200_launch_count()
    y = multi(layer, x, 1.0, plan)
    assert _lib.lib().ortho_b200_launch_count() - before == 4      # the long rows' GEMM, the main kernel, the long rows' finish twice
    q = layer.base_weight.to(torch.int16)
    w = torch.stack((q & 15, q >> 4), dim=2).view(N, K)
    w = (w - ((w & 8) << 1)).double() * layer.base_scales.double().unsqueeze(1)
    rows = torch.repeat_interleave(torch.arange(N, device=DEV), counts.to(DEV))
    w[rows, col.long()] += val.double()
    ref = x.double() @ w.T
    assert float((y.double() - ref).norm() / ref.norm()) <= REL_FRO_TOL
    assert _lib.lib().ortho_b200_query_kernel_status() == 0


@pytest.mark.parametrize("N,K", [(1, 4100), (3, 65536), (100, 20480), (295, 8196)])
def test_sieve_of_few_long_rows(N, K):
    """Rows cut into pieces (fewer rows than two per SM): bit for bit the torch chain on the CPU, with a list and without."""
    from libortho_b200 import sieve
    g = torch.Generator().manual_seed(N + K)
    w, h = torch.randn(N, K, generator=g) * 0.02, torch.rand(K, generator=g) * 2 + 0.01
    for target in (None, 0.01, 0.3, 1.0):
        base_ref, ortho_ref = sieve.hessian_sieve(w, h, curvature_thresh=1e-5, sparsity_target=target)
        base, ortho = sieve.hessian_sieve(w.to(DEV), h.to(DEV), curvature_thresh=1e-5, sparsity_target=target)
        assert torch.equal(base.cpu().view(torch.int32), base_ref.view(torch.int32))
        assert torch.equal(ortho.cpu().view(torch.int32), ortho_ref.view(torch.int32))
        own, scratch = w.to(DEV), torch.empty(int(_lib.lib().ortho_b200_sieve_scratch_bytes(N)), dtype=torch.uint8, device=DEV)
        st = _lib.lib().ortho_b200_sieve(own.data_ptr(), h.to(DEV).data_ptr(), N, K, 1e-5, -1 if target is None else int(target * N * K),
                                         own.data_ptr(), own.data_ptr(), scratch.data_ptr(), scratch.numel(),
                                         torch.cuda.current_stream().cuda_stream)
        assert st == 0 and torch.equal(own.view(torch.int32), ortho.view(torch.int32))


def test_a_captured_forward_owns_its_scratch():
    """A graph of a small batch, then a larger eager forward on the capture's stream (its scratch grows), then tensors in the
    memory that became free: a replay writes none of them and still gives the result."""
    layer = wl.make_layer(8192, 5300, 0.003, seed=11, device=DEV)
    m = layer.to_module()
    x, big = wl.make_input(12, 8192, seed=1, device=DEV), wl.make_input(600, 8192, seed=2, device=DEV)
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        m(x)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            y = m(x)
        ref = m(x)
        m(big)
        fill = [torch.full((1 << 20,), 7, dtype=torch.int32, device=DEV) for _ in range(24)]
        for i in range(3):
            y.zero_()
            graph.replay()
            torch.cuda.synchronize()
            assert torch.equal(y, ref)
            assert all(bool((f == 7).all()) for f in fill)
    assert _lib.lib().ortho_b200_query_kernel_status() == 0


def test_graphs_of_one_capture_stream_replay_side_by_side():
    """Two graphs captured on the same stream, replayed on two streams at once, beside eager forwards on a third."""
    K, N, M = 8192, 5300, 16
    a, b = (wl.make_layer(K, N, 0.003, seed=s, device=DEV).to_module() for s in (1, 2))
    xs = [wl.make_input(M, K, seed=s, device=DEV) for s in (1, 2)]
    refs = [a(xs[0]).clone(), b(xs[1]).clone()]
    torch.cuda.synchronize()
    graphs, outs = [], []
    for m, x in zip((a, b), xs):
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            for _ in range(8):
                y = m(x)
        graphs.append(g)
        outs.append(y)
    streams = [torch.cuda.Stream() for _ in range(3)]
    torch.cuda.synchronize()
    for _ in range(10):
        for g, s in zip(graphs, streams):
            with torch.cuda.stream(s):
                g.replay()
        with torch.cuda.stream(streams[2]):
            eager = a(xs[0])
    torch.cuda.synchronize()
    assert torch.equal(outs[0], refs[0]) and torch.equal(outs[1], refs[1]) and torch.equal(eager, refs[0])
    assert _lib.lib().ortho_b200_query_kernel_status() == 0


def test_scratch_is_bounded_and_given_back():
    from libortho_b200.ortho_linear import _SharedWorkspace
    layer = wl.make_layer(8192, 5300, 0.003, seed=3, device=DEV)
    m = layer.to_module()
    x = wl.make_input(12, 8192, seed=1, device=DEV)
    ref = m(x)
    torch.cuda.synchronize()
    handles = set()
    for s in [torch.cuda.Stream() for _ in range(20)] + [torch.cuda.Stream(priority=-1) for _ in range(20)]:
        with torch.cuda.stream(s):
            y = m(x)
            s.synchronize()
            assert torch.equal(y, ref)
            handles.add(s.cuda_stream)
        assert len(_SharedWorkspace._by_stream) <= _SharedWorkspace.MAX_STREAMS
    assert len(handles) > _SharedWorkspace.MAX_STREAMS
    assert torch.equal(m(x), ref)                           # the first stream's buffer had been given back
    held = set(map(id, _SharedWorkspace._by_stream.values()))
    before = torch.cuda.memory_allocated()
    del m
    assert len(_SharedWorkspace._by_stream) == 0 or not held & set(map(id, _SharedWorkspace._by_stream.values()))
    assert torch.cuda.memory_allocated() < before - (16 << 20)


def test_a_small_batch_on_raw_csr_brings_no_workspace():
    """Up to 16 tokens the streaming kernels serve the CSR arrays: the binding allocates nothing on the way, and the size query
    for such calls says so; the same layer with a plan or without a sparse term asks for room."""
    lib, K, N = _lib.lib(), 8192, 5300
    layer = wl.make_layer(K, N, 0.003, seed=3, device=DEV)
    for M in (12, 16):
        assert lib.ortho_b200_csr_workspace_bytes(M, K, N) == 0 < lib.ortho_b200_workspace_bytes(M, K, N)
        x, y = wl.make_input(M, K, seed=1, device=DEV), torch.empty(M, N, dtype=torch.float16, device=DEV)
        count = torch.cuda.memory_stats()["allocation.all.allocated"]
        _C_ops.forward(layer.base_weight, layer.base_scales, layer.vals, layer.col, layer.row_ptr, x, y, 1.0)
        _C_ops.forward_multi([(layer.base_weight, layer.base_scales, layer.vals, layer.col, layer.row_ptr)], x, [y])
        assert torch.cuda.memory_stats()["allocation.all.allocated"] == count
    for M in (17, 300):
        assert lib.ortho_b200_csr_workspace_bytes(M, K, N) == lib.ortho_b200_workspace_bytes(M, K, N) > 0


@pytest.mark.parametrize("M,K,Ns,launches", [(8, 8192, (8192, 1024, 1024), 1), (12, 8192, (8192, 1024, 1024), 1), (16, 8192, (8192, 1024, 1024), 3),
                                             (9, 4096, (11008, 11008), 1), (16, 4096, (11008, 11008), 2), (3, 8192, (4096, 264), 1)])
def test_layers_of_one_input_whose_own_routes_differ(M, K, Ns, launches):
    """One streaming launch or a launch per layer, whichever is faster for the group; the same values either way."""
    layers = [wl.make_layer(K, n, 0.003, seed=n, device=DEV) for n in Ns]
    plans = [_C_ops.Plan(t.row_ptr, t.col, t.vals, K, t.N) for t in layers]
    x = wl.make_input(M, K, seed=M, device=DEV)
    ys = [torch.empty(M, n, dtype=torch.float16, device=DEV) for n in Ns]
    before = _lib.lib().ortho_b200_launch_count()
    _C_ops.forward_multi([(t.base_weight, t.base_scales, t.vals, t.col, t.row_ptr) for t in layers], x, ys, alphas=[1.0, 0.5, 0.0][:len(Ns)], plans=plans)
    assert _lib.lib().ortho_b200_launch_count() - before == launches
    for t, p, y, alpha in zip(layers, plans, ys, (1.0, 0.5, 0.0)):
        ref = multi(t, x, alpha, p).double()
        assert float((y.double() - ref).norm() / ref.norm()) <= REL_FRO_TOL


def test_a_plan_is_refused_under_capture_and_the_capture_goes_on():
    layer = wl.make_layer(512, 96, 0.02, seed=1, device=DEV)
    y = torch.zeros(4, device=DEV)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        with pytest.raises(_lib.OrthoB200Error):
            _C_ops.Plan(layer.row_ptr, layer.col, layer.vals, layer.K, layer.N)
        y.add_(1)
    graph.replay()
    assert bool((y == 1).all())


@pytest.mark.parametrize("M", [129, 176, 177, 352, 353, 705])
def test_rows_that_cannot_be_folded_at_the_edges_of_token_tiles(M):
    """More than 128 tokens: rows with a zero or tiny scale are gathered by the epilogue, chunk by chunk of a token tile."""
    K, N = 1184, 300
    layer = wl.make_layer(K, N, 0.02, seed=12, device=DEV)
    layer.base_scales[::37], layer.base_scales[5::61] = 0.0, 6e-8
    plan = _C_ops.Plan(layer.row_ptr, layer.col, layer.vals, K, N)
    x = wl.make_input(M, K, seed=M, device=DEV)
    y = multi(layer, x, 0.75, plan)
    q = layer.base_weight.to(torch.int16)
    w = torch.stack((q & 15, q >> 4), dim=2).view(N, K)
    w = (w - ((w & 8) << 1)).double() * layer.base_scales.double().unsqueeze(1)
    rows = torch.repeat_interleave(torch.arange(N, device=DEV), (layer.row_ptr[1:] - layer.row_ptr[:-1]).long())
    w[rows, layer.col.long()] += 0.75 * layer.vals.double()
    ref = x.double() @ w.T
    err = y.double() - ref
    assert float(err.norm() / ref.norm()) <= REL_FRO_TOL and float(err.abs().max()) <= MAX_ABS_TOL
    alone = ref[:, ::37]                                    # the gathered rows by themselves: one FP16 rounding, 2^-11 of a value
    assert float((y[:, ::37].double() - alone).norm() / alone.norm()) <= 4.9e-4
    assert _lib.lib().ortho_b200_query_kernel_status() == 0


def test_a_plan_may_go_while_its_forward_runs():
    """Destroying a plan waits for the kernels that read it: plans made at once in the same memory do not disturb them."""
    K, N, M = 8192, 4096, 64
    layer = wl.make_layer(K, N, 0.01, seed=2, device=DEV)
    other = wl.Layer(K, N, layer.base_weight, layer.base_scales, layer.row_ptr, layer.col, -layer.vals, 1.0)
    x = wl.make_input(M, K, seed=2, device=DEV)
    args = (layer.base_weight, layer.base_scales, layer.vals, layer.col, layer.row_ptr)
    ref = multi(layer, x, 1.0, _C_ops.Plan(layer.row_ptr, layer.col, layer.vals, K, N))
    ys = [torch.empty(M, N, dtype=torch.float16, device=DEV) for _ in range(8)]
    ws = torch.empty(_C_ops.workspace_bytes(M, K, N), dtype=torch.uint8, device=DEV)
    for y in ys:
        plan = _C_ops.Plan(layer.row_ptr, layer.col, layer.vals, K, N)
        for _ in range(20):
            _C_ops.forward(*args, x, y, 1.0, plan=plan, workspace=ws)
        plan.close()
        _C_ops.Plan(other.row_ptr, other.col, other.vals, K, N)
    assert all(torch.equal(y, ref) for y in ys)
