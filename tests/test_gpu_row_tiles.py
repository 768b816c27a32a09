"""The grouped GEMM's row tiles at their edges: experts whose row counts sit around the 32-row quarters of a 128-row tile
(an epilogue warp without a row of its own only hands buffers back), an empty expert, K lengths around the scale ring."""
import pytest
import torch

from helpers import kernels_of
from oracle import moe_oracle as orc
from test_gpu_weights_on_m import by_row_tiles

pytestmark = pytest.mark.gpu
DEV = "cuda"
ROWS = [1, 31, 32, 33, 0, 64, 65, 96, 97, 127, 128, 129, 160, 161]


@pytest.mark.parametrize("H,I", [(128, 256), (64, 144), (640, 1152), (1344, 192)])
@pytest.mark.parametrize("mode", [0, 256, 512, 1024])
def test_ragged_row_counts_match_oracle(mode, H, I):
    """The layer: row tiles in block mode, the weights on M in the others, whose row tiles the next test has."""
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


@pytest.mark.parametrize("H,I", [(128, 256), (640, 1152)])
@pytest.mark.parametrize("mode", [0, 256, 512])
def test_ragged_row_counts_of_the_stand_alone_operators(mode, H, I):
    """The stand-alone grouped GEMM has its row tiles in every mode."""
    from dqmoe_b200 import ops
    E, T = len(ROWS), sum(ROWS)
    g = torch.Generator().manual_seed(H + I)
    a = torch.randn(T, H, generator=g).to(torch.bfloat16)
    b = (torch.randn(E, 2 * I, H, generator=g) * 0.05).to(torch.bfloat16)
    b1 = (torch.randn(E, H, I, generator=g) * 0.05).to(torch.bfloat16)
    ids = torch.repeat_interleave(torch.arange(E), torch.tensor(ROWS))[torch.randperm(T, generator=g)]
    ids = ids.to(torch.int32).view(T, 1)
    if mode == 0:
        ref = orc.moe_layer_bf16(a, b, b1, ids, E)
        w = (b.to(DEV), None), (b1.to(DEV), None)
    else:
        qs = orc.quantize_inputs(a, b, b1, mode)
        ref = orc.moe_layer_fp8(*qs, ids, E, mode)
        w = [tuple(t.to(DEV).contiguous() for t in pair) for pair in (qs[2:4], qs[4:6])]
    _, _, d = by_row_tiles(ops, mode, a.to(DEV), *w, ids.to(DEV), E)
    assert ops.device_status() == 0
    # the layer tolerance (see above)
    assert orc.cosine(d.cpu(), ref) >= 0.999 and orc.max_rel_err(d.cpu(), ref) <= 2e-2


@pytest.mark.parametrize("drop", [False, True])
def test_quarters_without_rows_over_long_reductions(drop):
    """Block mode with the scales by tile, last row tiles of 1 to 128 rows and K loops of 33 and 23 blocks: warps without rows,
    and the lanes of the scale loader without a copy, go round the same barriers as the others. With dropped slots the kept
    tiles are fewer than the layout's bound. Rows are bit-identical to the same rows in a small call."""
    from dqmoe_b200 import ops
    H, I = 4112, 2832
    rows = [r + 128 * (1 + i % 3) for i, r in enumerate(ROWS)]
    E, T = len(rows), sum(rows)
    g = torch.Generator(device=DEV).manual_seed(H)
    a = torch.randn(T, H, generator=g, device=DEV).to(torch.bfloat16)
    b = ops.per_block_cast_to_fp8((torch.randn(E, 2 * I, H, generator=g, device=DEV) * 0.05).to(torch.bfloat16))
    b1 = ops.per_block_cast_to_fp8((torch.randn(E, H, I, generator=g, device=DEV) * 0.05).to(torch.bfloat16))
    q, s = ops.per_token_block_cast_to_fp8(a)
    ids = torch.repeat_interleave(torch.arange(E), torch.tensor(rows))[torch.randperm(T, generator=torch.Generator().manual_seed(H))]
    ids = ids.to(torch.int32)
    if drop:
        ids[::3] = -1
        ids[1::7] = E
    ids = ids.view(T, 1)

    def run(sel, tiled):
        n = len(sel)
        ws = torch.empty(ops.moe_workspace_bytes(n, H, I, E, 1, 1024), dtype=torch.uint8, device=DEV)
        d = torch.zeros(n, 1, H, dtype=torch.bfloat16, device=DEV)
        qd = q.view(torch.uint8)[sel.to(DEV)].contiguous().view(q.dtype)
        sd, idd = s[sel.to(DEV)].contiguous(), ids[sel].contiguous().to(DEV)
        ops.moe_forward(qd, sd, *b, *b1, d, idd, ws, 1024)
        assert ops.device_status() == 0
        names = kernels_of(lambda: ops.moe_forward(qd, sd, *b, *b1, d, idd, ws, 1024))
        assert any("scale_tiles" in k for k in names) == tiled, names
        return d.cpu()

    sample = torch.arange(0, T, 23)
    full, small = run(torch.arange(T), True), run(sample, False)
    assert torch.equal(full[sample], small)
    kept = (ids[:, 0] >= 0) & (ids[:, 0] < E)
    assert not full[~kept].any()
    sample = sample[kept[sample]]
    ref = orc.moe_layer_fp8(q.cpu()[sample], s.cpu()[sample], *[t.cpu() for t in b], *[t.cpu() for t in b1], ids[sample], E, 1024)
    # the layer tolerance (see above)
    assert orc.cosine(full[sample], ref) >= 0.999 and orc.max_rel_err(full[sample], ref) <= 2e-2
