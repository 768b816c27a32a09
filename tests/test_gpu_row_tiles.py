"""The grouped GEMM's row tiles at their edges: experts whose row counts sit around the 32-row quarters of a 128-row tile
(an epilogue warp without a row of its own only hands buffers back), an empty expert, K lengths around the scale ring."""
import pytest
import torch

from oracle import moe_oracle as orc

pytestmark = pytest.mark.gpu
DEV = "cuda"
ROWS = [1, 31, 32, 33, 0, 64, 65, 96, 97, 127, 128, 129, 160, 161]


@pytest.mark.parametrize("H,I", [(128, 256), (64, 144), (640, 1152), (1344, 192)])
@pytest.mark.parametrize("mode", [0, 256, 512, 1024])
def test_ragged_row_counts_match_oracle(mode, H, I):
    from dqmoe_b200 import ops
    E, T = len(ROWS), sum(ROWS)
    g = torch.Generator().manual_seed(H + I)
    a = torch.randn(T, H, generator=g).to(torch.bfloat16)
    b = (torch.randn(E, 2 * I, H, generator=g) * 0.05).to(torch.bfloat16)
    b1 = (torch.randn(E, H, I, generator=g) * 0.05).to(torch.bfloat16)
    ids = torch.repeat_interleave(torch.arange(E), torch.tensor(ROWS))[torch.randperm(T, generator=g)]
    ids = ids.to(torch.int32).view(T, 1)
    ws = torch.empty(ops.moe_workspace_bytes(T, H, I, E, 1, mode), dtype=torch.uint8, device=DEV)
    d = torch.zeros(T, 1, H, dtype=torch.bfloat16, device=DEV)
    if mode == 0:
        ref = orc.moe_layer_bf16(a, b, b1, ids, E)
        ops.moe_forward(a.to(DEV), None, b.to(DEV), None, b1.to(DEV), None, d, ids.to(DEV), ws, mode)
    else:
        qs = orc.quantize_inputs(a, b, b1, mode)
        ref = orc.moe_layer_fp8(*qs, ids, E, mode)
        q = [t.to(DEV).contiguous() for t in qs]
        ops.moe_forward(*q, d, ids.to(DEV), ws, mode)
    assert ops.device_status() == 0
    # the layer tolerance: a rounding of the intermediate that flips moves one e4m3 step (2^-3 relative) of one of I terms
    assert orc.cosine(d.cpu(), ref) >= 0.999 and orc.max_rel_err(d.cpu(), ref) <= 2e-2
