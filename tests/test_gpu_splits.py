"""Up to 128 tokens: shares that leave pieces of a single unit (128 k) at either turn of the two MMA issuers, against plain torch
in 64 bits.  Outputs are FP16, one rounding of an FP32 sum: at most 2^-11 of a value, so 4.9e-4 in the relative 2-norm; REL_FRO_TOL
(1e-3) and MAX_ABS_TOL leave room for the FP32 sums."""
import pytest
import torch

import workloads as wl
from libortho_b200 import _C_ops, _lib
from test_gpu_tiles import check, dense, forward

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("K,N", [(1152, 1024),      # 9 units a tile, 9 shares of 8: pieces of one unit first and last in a share
                                 (1280, 1024)])     # 10 units a tile, 10 shares of 8: pieces of two
@pytest.mark.parametrize("M", [1, 16, 32, 33, 64, 65])
def test_pieces_of_one_unit(K, N, M):
    layer = wl.make_layer(K, N, 0.02, seed=K, device=DEV)
    plan = _C_ops.Plan(layer.row_ptr, layer.col, layer.vals, K, N)
    w, s = dense(layer)
    x = wl.make_input(M, K, seed=M, device=DEV)
    for alpha in (0.0, 0.75):
        y = forward(layer, x, alpha, plan, force=True)
        check(y, x.double() @ (w + alpha * s).T, f"M={M} {K}->{N} alpha={alpha}")
        assert torch.equal(y, forward(layer, x, alpha, plan, force=True))
    assert _lib.lib().ortho_b200_query_kernel_status() == 0
