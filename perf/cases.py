"""The work a program gives this operator, as cases that can be timed and checked.

One pass is one call through a public entry point: the ``OrthoLinear`` module (decode, small batches, prefill),
the function-level binding on raw CSR arrays, several projections of one input in a single call, or the
device-side sieve and packer that produce a layer.  Sizes are those of the Llama-7B-style and Llama-2-70B-style
projections that the benchmark uses, and generic ragged ones.

A forward case holds ``K`` (in features), ``N`` (out features; ``N2`` is the width of each of two more layers of a
multi-projection call, 0 otherwise), ``M`` (tokens), ``density`` and ``rows`` (share of the weights in the sparse
component, spread evenly or by a power law over the rows), ``alpha``, ``bias``, ``x`` (type of the activations) and
``api``.
"""
import math

import torch

from libortho_b200 import OrthoLinear, _C_ops
from libortho_b200.sieve import hessian_sieve

DEV = "cuda"
F16, F32, F64 = torch.float16, torch.float32, torch.float64
TYPES = {"float16": torch.float16, "bfloat16": torch.bfloat16, "float32": torch.float32}
MAX_WEIGHTS = 8192 * 57344                 # the widest layer in use
MAX_COST = 4096 * 8192 * 57344             # its prefill


def _forward(name, K, N, M, density, *, N2=0, rows="uniform", alpha=1.0, bias=False, x="float16", api="module"):
    return {"name": name, "op": "forward", "api": api, "K": K, "N": N, "N2": N2, "M": M, "density": density, "rows": rows,
            "alpha": alpha, "bias": bias, "x": x}


def listed():
    return [
        # one token through a small attention projection: the smallest call a decoder makes, latency and launches
        _forward("decode_o_proj_m1", 4096, 4096, 1, 0.005),
        # one token through the widest projection (gate + up of a 70B-style MLP): the base streams from memory
        _forward("decode_gate_up_m1", 8192, 57344, 1, 0.003),
        # four decoding sequences through Q, K and V kept as separate layers over one input (8 KV heads of 128)
        _forward("decode_qkv_m4", 8192, 8192, 4, 0.003, N2=1024, api="multi"),
        # the function-level binding on the raw CSR arrays, a layer of odd sizes and an odd batch
        _forward("decode_binding_ragged_m7", 2912, 1003, 7, 0.01, api="binding"),
        # sixteen decoding sequences through gate + up of a 7B-style MLP
        _forward("decode_gate_up_m16", 4096, 22016, 16, 0.005),
        # thirty-two decoding sequences through a fused QKV projection
        _forward("batch_qkv_m32", 8192, 10240, 32, 0.003),
        # a large decoding batch (or a short prompt) of no particular size through a long-K down projection
        _forward("batch_down_m100", 28672, 8192, 100, 0.003),
        # prompt chunks: a power-law layer, half strength
        _forward("prefill_powerlaw_m512", 8192, 8192, 512, 0.001, rows="powerlaw", alpha=0.5),
        # a bfloat16 model's prompt with the kill switch off: the base alone, a token count of no particular size
        _forward("prefill_killed_bf16_m777", 11008, 4096, 777, 0.005, alpha=0.0, x="bfloat16"),
        # a layer whose sieve kept one weight in a hundred, with a bias
        _forward("prefill_top1pct_bias_m2048", 4096, 4096, 2048, 0.01, bias=True),
        # a long prompt through the widest projection: the largest call
        _forward("prefill_gate_up_m4096", 8192, 57344, 4096, 0.003),
        # producing a layer on the GPU: sieve FP32 weights, keep the top 1 %, quantise, pack and build the CSR arrays
        {"name": "pack_top1pct", "op": "pack", "K": 4096, "N": 11008, "density": 0.01},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    if rng.random() < 0.1:
        return {"op": "pack", "K": 32 * _log_int(rng, 16, 256), "N": _log_int(rng, 256, 11008), "density": rng.choice([0.001, 0.005, 0.01])}
    api = rng.choice(["module", "module", "module", "module", "binding", "multi"])
    K = 32 * _log_int(rng, 16, 896) if rng.random() < 0.5 else 256 * _log_int(rng, 2, 112)
    N = min(_log_int(rng, 256, 57344), MAX_WEIGHTS // K)
    N2 = max(64, N // 8) if api == "multi" else 0
    M = _log_int(rng, 1, 4096)
    # raw CSR calls gather the sparse term: keep them to a smaller share of the largest case's work
    M = max(1, min(M, MAX_COST // (K * (N + 2 * N2)) // (16 if api != "module" else 1)))
    c = _forward("", K, N, M, rng.choice([0.0, 0.001, 0.003, 0.005, 0.01]), N2=N2, rows=rng.choice(["uniform", "uniform", "powerlaw"]),
                 alpha=rng.choice([0.0, 0.5, 1.0, 1.0]), bias=api != "binding" and rng.random() < 0.3,
                 x=rng.choice(["float16", "float16", "bfloat16", "float32"]) if api == "module" else "float16", api=api)
    del c["name"]
    return c


def _widths(case):
    return [case["N"]] + [case["N2"]] * 2 if case["N2"] else [case["N"]]


def _row_density(case, N, g):
    """Expected share of each row's weights in the sparse component."""
    K, d = case["K"], case["density"]
    if case["rows"] == "uniform":
        return torch.full((N, 1), d, device=DEV)
    p = torch.arange(1, N + 1, device=DEV, dtype=F32).pow(-1.2)             # Zipf over the rows, shuffled row order
    p = p / p.sum() * (d * N * K)
    return (p[torch.randperm(N, generator=g, device=DEV)] / K).clamp(max=1.0).unsqueeze(1)


def _layer(case, N, g):
    """Packed INT4 base of W ~ N(0, 0.02^2) with a scale per row, sparse values ~ N(0, 0.05^2) as CSR."""
    K = case["K"]
    weight = torch.empty(N, K // 2, dtype=torch.uint8, device=DEV)
    scales = torch.empty(N, dtype=F16, device=DEV)
    share = _row_density(case, N, g)
    counts, cols = torch.zeros(N, dtype=torch.int64, device=DEV), []
    step = max(1, (1 << 27) // K)
    for a in range(0, N, step):
        b = min(N, a + step)
        w = torch.randn(b - a, K, generator=g, device=DEV).mul_(0.02)
        s = (w.abs().amax(dim=1) / 7.0).clamp(min=1e-6)
        q = torch.round(w / s.unsqueeze(1)).clamp_(-8, 7).to(torch.int8)
        weight[a:b] = ((q[:, 0::2] & 15) | ((q[:, 1::2] & 15) << 4)).to(torch.uint8)
        scales[a:b] = s.to(F16)
        if case["density"] > 0:
            at = torch.rand(b - a, K, generator=g, device=DEV) < share[a:b]
            counts[a:b] = at.sum(dim=1)
            cols.append(at.nonzero()[:, 1].to(torch.int32))
    col = torch.cat(cols) if cols else torch.zeros(0, dtype=torch.int32, device=DEV)
    ptr = torch.zeros(N + 1, dtype=torch.int32, device=DEV)
    ptr[1:] = counts.cumsum(0).to(torch.int32)
    val = torch.randn(col.numel(), generator=g, device=DEV).mul_(0.05).to(F16)
    bias = torch.randn(N, generator=g, device=DEV).mul_(0.1) if case["bias"] else None
    return weight, scales, val, col, ptr, bias


def _inputs(case, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    if case["op"] == "pack":
        w = torch.randn(case["N"], case["K"], generator=g, device=DEV).mul_(0.02)
        h = torch.rand(case["K"], generator=g, device=DEV).mul_(2.0).add_(0.05)          # diagonal of the inverse Hessian
        return w, h
    x = torch.randn(case["M"], case["K"], generator=g, device=DEV).to(TYPES[case["x"]])
    return x, [_layer(case, n, g) for n in _widths(case)]


def prepare(case, seed):
    if case["op"] == "pack":
        w, h = _inputs(case, seed)
        return {"case": case, "w": w, "h": h}
    x, layers = _inputs(case, seed)
    if case["api"] == "module":
        weight, scales, val, col, ptr, bias = layers[0]
        m = OrthoLinear(case["K"], case["N"], bias=bias is not None, device=DEV)
        m.base_weight, m.base_scales = weight, scales
        m.ortho_values, m.ortho_col_indices, m.ortho_row_ptr = val, col, ptr
        if bias is not None:
            m.bias.data = bias
            m.bias.requires_grad_(False)
        m.set_alpha(case["alpha"])
        return {"case": case, "x": x, "module": m}
    state = {"case": case, "x": x, "layers": [t[:5] for t in layers],
             "out": [torch.empty(case["M"], n, dtype=F16, device=DEV) for n in _widths(case)]}
    if case["api"] == "multi":
        state["plans"] = [_C_ops.Plan(t[4], t[3], t[2], case["K"], n) for t, n in zip(layers, _widths(case))]
        state["biases"] = [t[5] for t in layers]
        state["alphas"] = [case["alpha"]] * len(layers)
    return state


def run(state):
    case = state["case"]
    if case["op"] == "pack":
        base, ortho = hessian_sieve(state["w"], state["h"], sparsity_target=case["density"])
        m = OrthoLinear(case["K"], case["N"], device=DEV)
        m.load_from_weights(base, ortho)
        return [m.base_weight, m.base_scales, m.ortho_row_ptr, m.ortho_col_indices, m.ortho_values]
    if case["api"] == "module":
        return state["module"](state["x"])
    if case["api"] == "binding":
        _C_ops.forward(*state["layers"][0], state["x"], state["out"][0], case["alpha"])
        return state["out"][0]
    _C_ops.forward_multi(state["layers"], state["x"], state["out"], alphas=state["alphas"], biases=state["biases"], plans=state["plans"])
    return state["out"]


def work(case):
    K = case["K"]
    if case["op"] == "pack":
        nnz = int(case["density"] * case["N"] * K)
        return {"bytes": 4 * case["N"] * K + 4 * K + case["N"] * K // 2 + 6 * case["N"] + 6 * nnz, "flops": 0}
    n, M = sum(_widths(case)), case["M"]
    size = TYPES[case["x"]].itemsize
    nbytes, flops = n * K // 2 + 2 * n + size * M * (K + n) + (4 * n if case["bias"] else 0), 2 * M * n * K
    if case["alpha"] > 0 and case["density"] > 0:
        nnz = int(case["density"] * n * K)
        nbytes, flops = nbytes + 6 * nnz + 4 * (n + 1), flops + 2 * M * nnz
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    """The packer's results are whole numbers and FP16 roundings of given values: the same bits.  A forward rounds its
    FP32 sums to FP16 once, and the tensor-core kernels also round the sparse weights to FP16 against the row's scale:
    2.1e-4 to 2.2e-4 in the 2-norm against sums in 64 bits, 1.7e-3 with bfloat16 outputs (all measured).  Two correct
    forwards can differ by one unit in the last place of a value, 9.8e-4 of it (7.8e-3 for bfloat16)."""
    if case["op"] == "pack":
        return "exact"
    if case["x"] == "bfloat16":
        return {"rel": 7e-3, "max": 1.6e-2}
    return {"rel": 1e-3, "max": 6e-3}


def exact(case, seed):
    if case["op"] == "pack":
        return None
    x, layers = _inputs(case, seed)
    x = x.to(F16).to(F64)
    outs = []
    for weight, scales, val, col, ptr, bias in layers:
        N, K = weight.shape[0], case["K"]
        y = torch.empty(case["M"], N, dtype=F64, device=DEV)
        step = max(1, (1 << 26) // K)
        ptr_h = ptr.tolist() if step < N else [0] * N + [col.numel()]
        for a in range(0, N, step):
            b = min(N, a + step)
            q = weight[a:b].to(torch.int16)
            w = torch.stack((q & 15, q >> 4), dim=2).view(b - a, K)
            w = (w - ((w & 8) << 1)).to(F64) * scales[a:b].to(F64).unsqueeze(1)
            if case["alpha"] > 0 and col.numel():
                e0, e1 = ptr_h[a], ptr_h[b]
                row = torch.repeat_interleave(torch.arange(b - a, device=DEV), (ptr[a + 1:b + 1] - ptr[a:b]).long())
                w.index_put_((row, col[e0:e1].long()), val[e0:e1].to(F64) * case["alpha"], accumulate=True)
            y[:, a:b] = x @ w.T
            if bias is not None:
                y[:, a:b] += bias[a:b].to(F64)
        outs.append(y)
    return outs if case["api"] == "multi" else outs[0]
