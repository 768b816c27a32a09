"""Tiles with the rows on M load the rows that an expert has in boxes of 32: experts around their edges, and what a tile's unused rows
held before does not show."""
import pytest
import torch

from oracle import moe_oracle as orc

pytestmark = pytest.mark.gpu
DEV = "cuda"
ROWS = [1, 31, 32, 33, 63, 64, 65, 95, 96, 97, 127, 128, 129, 0, 161]


@pytest.mark.parametrize("H,I", [(256, 384), (640, 128), (4096, 1280)])  # one tile per block at most in both GEMMs; in fc2; in none
@pytest.mark.parametrize("mode", [1024, 2048])
def test_partly_filled_row_tiles(mode, H, I):
    from dqmoe_b200 import ops
    E, T = len(ROWS), sum(ROWS)
    g = torch.Generator().manual_seed(H + mode)
    a = torch.randn(T, H, generator=g).to(torch.bfloat16)
    b = (torch.randn(E, 2 * I, H, generator=g) * 0.05).to(torch.bfloat16)
    b1 = (torch.randn(E, H, I, generator=g) * 0.05).to(torch.bfloat16)
    ids = torch.repeat_interleave(torch.arange(E), torch.tensor(ROWS))[torch.randperm(T, generator=g)].to(torch.int32).view(T, 1)
    qs = orc.quantize_inputs(a, b, b1, mode)
    ref = orc.moe_layer_fp8(*qs, ids, E, mode)
    q = [t.to(DEV).contiguous() for t in qs]
    if mode == 2048:
        q[3], q[5] = ops.mx_tile_scales(q[3], H), ops.mx_tile_scales(q[5], I)
    ws = torch.empty(ops.moe_workspace_bytes(T, H, I, E, 1, mode), dtype=torch.uint8, device=DEV)

    def run(rows, ids_):
        d = torch.zeros(T, 1, H, dtype=torch.bfloat16, device=DEV)
        ops.moe_forward(rows, *q[1:], d, ids_.to(DEV), ws, mode)
        assert ops.device_status() == 0
        return d

    first = run(q[0], ids)
    nan = torch.full_like(q[0].view(torch.uint8), 0x7F).view(q[0].dtype)
    run(nan, (torch.arange(T, dtype=torch.int32) % 2).view(T, 1))  # full tiles of NaN leave their rows in shared memory
    assert torch.equal(run(q[0], ids), first)
    # the layer tolerance: a rounding of the intermediate that flips moves one e4m3 step (2^-3 relative) of one of I terms
    assert orc.cosine(first.cpu(), ref) >= 0.999 and orc.max_rel_err(first.cpu(), ref) <= 2e-2
