"""The two tensor-memory kernels (up to 128 tokens, more than 128) and the select of the device-side sieve at the sizes
where they can go wrong: edges of token tiles, of k pairs and boxes and of row tiles, layers cut into many pieces, windows
with none, one and more entries than a warp takes at once, long rows, and replays of a captured graph.

The reference is the operator in 64 bits by plain torch (dequantised base plus the CSR entries).  Outputs are FP16: one
rounding is at most 2^-11 of a value, so 4.9e-4 in the relative 2-norm; with entries rounded to FP16 against the row's scale
(more than 128 tokens) another 2^-11 of the sparse part: 1e-3 bounds the sum."""
import pytest
import torch

import workloads as wl
from conftest import MAX_ABS_TOL, REL_FRO_TOL
from libortho_b200 import _C_ops, _lib, sieve

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def dense(layer):
    """(base, sparse) weights in 64 bits."""
    q = layer.base_weight.to(torch.int16)
    w = torch.stack((q & 15, q >> 4), dim=2).view(layer.N, layer.K)
    w = (w - ((w & 8) << 1)).double() * layer.base_scales.double().unsqueeze(1)
    rows = torch.repeat_interleave(torch.arange(layer.N, device=w.device), (layer.row_ptr[1:] - layer.row_ptr[:-1]).long())
    s = torch.zeros_like(w)
    s[rows, layer.col.long()] = layer.vals.double()
    return w, s


def forward(layer, x, alpha, plan, bias=None, force=False):
    ws = torch.full((max(256, _C_ops.workspace_bytes(max(x.shape[0], 17), layer.K, layer.N, plan)),), 0xFF, dtype=torch.uint8, device=DEV)
    y = torch.full((x.shape[0], layer.N), float("nan"), dtype=torch.float16, device=DEV)
    try:
        if force:
            assert _lib.lib().ortho_b200_set_decode_config(-4, 0, 0, 128) == 0
        _C_ops.forward_multi([(layer.base_weight, layer.base_scales, layer.vals, layer.col, layer.row_ptr)], x, [y], alphas=[alpha],
                             biases=[bias], plans=[plan], workspace=ws)
    finally:
        _lib.lib().ortho_b200_set_decode_config(-4, 0, 0, 0)
    return y


def check(y, ref, what):
    err = y.double() - ref
    rel = float(err.norm() / ref.norm())
    assert rel <= REL_FRO_TOL and float(err.abs().max()) <= MAX_ABS_TOL, (what, rel, float(err.abs().max()))


@pytest.mark.parametrize("K,N,d,kind", [(64, 40, 0.1, "gauss"), (1120, 300, 0.02, "gauss"), (2080, 130, 0.25, "gauss"),
                                        (4096, 1100, 0.01, "zipf"), (28672, 136, 0.003, "gauss"), (512, 4736, 0.005, "gauss")])
def test_up_to_128_tokens(K, N, d, kind):
    layer = wl.make_layer(K, N, d, seed=K + N, device=DEV, ortho=kind)
    plan = _C_ops.Plan(layer.row_ptr, layer.col, layer.vals, K, N)
    bias = torch.randn(N, generator=torch.Generator().manual_seed(N)).to(DEV)
    w, s = dense(layer)
    for M in (1, 9, 16, 17, 32, 33, 49, 64, 65, 81, 96, 97, 112, 113, 128):
        x = wl.make_input(M, K, seed=M, device=DEV)
        for alpha in (0.0, 0.75):
            ref = x.double() @ (w + alpha * s).T
            y = forward(layer, x, alpha, plan, force=True)
            check(y, ref, f"M={M} {K}->{N} alpha={alpha}")
            check(forward(layer, x, alpha, plan, bias, force=True), ref + bias.double(), f"bias M={M} {K}->{N} alpha={alpha}")
            assert torch.equal(y, forward(layer, x, alpha, plan, force=True))
    assert _lib.lib().ortho_b200_query_kernel_status() == 0


@pytest.mark.parametrize("K,N,d,kind", [(96, 130, 0.05, "gauss"), (1184, 300, 0.02, "gauss"), (2080, 200, 0.25, "gauss"),
                                        (4096, 1100, 0.01, "zipf"), (8192, 520, 0.003, "gauss"), (512, 9600, 0.005, "gauss")])
def test_more_than_128_tokens(K, N, d, kind):
    layer = wl.make_layer(K, N, d, seed=K + N, device=DEV, ortho=kind)
    plan = _C_ops.Plan(layer.row_ptr, layer.col, layer.vals, K, N)
    w, s = dense(layer)
    for M in (129, 176, 177, 192, 193, 352, 353, 385, 705):
        x = wl.make_input(M, K, seed=M, device=DEV)
        for alpha in (0.0, 0.75):
            ref = x.double() @ (w + alpha * s).T
            y = forward(layer, x, alpha, plan)
            check(y, ref, f"M={M} {K}->{N} alpha={alpha}")
            assert torch.equal(y, forward(layer, x, alpha, plan))
        if kind != "zipf":                                  # no long rows: the workspace is optional
            y = torch.empty(M, N, dtype=torch.float16, device=DEV)
            st = _lib.lib().ortho_b200_forward(layer.base_weight.data_ptr(), layer.base_scales.data_ptr(), None, None, None, layer.nnz,
                                               x.data_ptr(), y.data_ptr(), M, K, N, 0.75, plan.handle, None, 0,
                                               torch.cuda.current_stream().cuda_stream)
            assert st == 0
            check(y, ref, f"no workspace M={M} {K}->{N}")
    assert _lib.lib().ortho_b200_query_kernel_status() == 0


@pytest.mark.parametrize("M", [32, 100, 200])
def test_replays_of_a_captured_forward_whose_tiles_are_cut(M):
    """A replay brings the launch tag of the capture again: the collecting CTAs must have cleared the flags."""
    K, N = 4096, 300
    layer = wl.make_layer(K, N, 0.01, seed=3, device=DEV)
    plan = _C_ops.Plan(layer.row_ptr, layer.col, layer.vals, K, N)
    w, s = dense(layer)
    x = wl.make_input(M, K, seed=1, device=DEV)
    y = torch.empty(M, N, dtype=torch.float16, device=DEV)
    ws = torch.empty(_C_ops.workspace_bytes(M, K, N, plan), dtype=torch.uint8, device=DEV)

    def run():
        _C_ops.forward(layer.base_weight, layer.base_scales, layer.vals, layer.col, layer.row_ptr, x, y, 1.0, plan=plan, workspace=ws)

    run()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        run()
        run()
    for i in range(6):
        x.copy_(wl.make_input(M, K, seed=50 + i, device=DEV))
        graph.replay()
        check(y, x.double() @ (w + s).T, f"replay {i}")
    assert _lib.lib().ortho_b200_query_kernel_status() == 0


def test_rows_without_order_or_lists_agree():
    """The same entries listed backwards (no window lists: gather form) give the same result within FP16 rounding."""
    K, N = 1024, 260
    layer = wl.make_layer(K, N, 0.02, seed=8, device=DEV)
    rows = torch.repeat_interleave(torch.arange(N, device=DEV), (layer.row_ptr[1:] - layer.row_ptr[:-1]).long())
    order = torch.argsort(rows * K + (K - 1 - layer.col.long()))
    rev = wl.Layer(K, N, layer.base_weight, layer.base_scales, layer.row_ptr, layer.col[order].contiguous(), layer.vals[order].contiguous(), 1.0)
    plan = _C_ops.Plan(rev.row_ptr, rev.col, rev.vals, K, N)
    assert not plan.rows_ordered
    w, s = dense(layer)
    for M in (24, 100, 300):
        x = wl.make_input(M, K, seed=M, device=DEV)
        check(forward(rev, x, 0.5, plan), x.double() @ (w + 0.5 * s).T, f"backwards M={M}")


@pytest.mark.parametrize("kind", ["ties", "spread", "equal", "nan"])
@pytest.mark.parametrize("N,K", [(64, 8), (333, 264), (40, 4096)])
def test_sieve_where_quotients_are_close(kind, N, K):
    """Quotients on rounding ties, scores over hundreds of binades, all scores equal, NaN: the approximate quotients of the
    sieve and the packer may never decide.  Bit for bit the torch chain on the CPU."""
    g = torch.Generator().manual_seed(N + K)
    w, h = torch.randn(N, K, generator=g) * 0.02, torch.rand(K, generator=g) * 2 + 0.01
    if kind == "ties":
        w = torch.randint(-14, 15, (N, K), generator=g).float() * 0.015
    if kind == "spread":
        w, h = torch.exp(torch.randn(N, K, generator=g) * 4) * torch.sign(w), torch.exp(torch.randn(K, generator=g) * 4)
    if kind == "equal":
        w.fill_(0.25)
    if kind == "nan":
        w[3, 5] = float("nan")
    for thresh, target in ((1e-5, None), (10.0, 0.01), (10.0, 0.3), (10.0, 1.0)):
        if kind == "nan" and target:
            continue
        base_ref, ortho_ref = sieve.hessian_sieve(w, h, curvature_thresh=thresh, sparsity_target=target)
        base, ortho = sieve.hessian_sieve(w.to(DEV), h.to(DEV), curvature_thresh=thresh, sparsity_target=target)
        keep = ~torch.isnan(w).any(dim=1)                   # a NaN's payload is not specified
        assert torch.equal(base.cpu()[keep].view(torch.int32), base_ref[keep].view(torch.int32))
        assert torch.equal(ortho.cpu()[keep].view(torch.int32), ortho_ref[keep].view(torch.int32))
