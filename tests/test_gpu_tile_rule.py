"""CTA pairs against single CTAs: row counts on both sides of the lines of the rule that chooses them, checked against the
oracle, and a small batch bit-identical to its rows of the full one (the choice must not show in the results)."""
import pytest
import torch

from helpers import kernels_of
from oracle import moe_oracle as orc

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("mode", [0, 256, 512])
@pytest.mark.parametrize("rows", [128, 129, 200, 240, 241, 385, 560])
def test_layer_on_both_sides_of_the_pair_rule(mode, rows):
    from dqmoe_b200 import ops
    E, H, I = 3, 128, 8192 if rows < 300 else 6144
    T = E * rows
    g = torch.Generator(device=DEV).manual_seed(rows)
    a = torch.randn(T, H, generator=g, device=DEV).to(torch.bfloat16)
    b = (torch.randn(E, 2 * I, H, generator=g, device=DEV) * 0.05).to(torch.bfloat16)
    b1 = (torch.randn(E, H, I, generator=g, device=DEV) * 0.05).to(torch.bfloat16)
    ids = (torch.arange(T, dtype=torch.int32) % E).view(T, 1)
    ids[:40] = 0  # ragged experts
    qs = (a, None, b, None, b1, None)
    if mode == 256:
        qs = (*ops.per_tensor_cast_to_fp8(a), *ops.per_tensor_cast_to_fp8(b, per_expert=True), *ops.per_tensor_cast_to_fp8(b1, per_expert=True))
    elif mode == 512:
        qs = (*ops.per_token_cast_to_fp8(a), *ops.per_channel_cast_to_fp8(b), *ops.per_channel_cast_to_fp8(b1))

    def run(x, xs, idx):
        n = idx.shape[0]
        d = torch.zeros(n, 1, H, dtype=torch.bfloat16, device=DEV)
        ws = torch.empty(ops.moe_workspace_bytes(n, H, I, E, 1, mode), dtype=torch.uint8, device=DEV)
        ops.moe_forward(x, xs, *qs[2:], d, idx.to(DEV), ws, mode)
        assert ops.device_status() == 0
        return d.cpu()

    full = run(qs[0], qs[1], ids)
    sample = torch.arange(0, T, max(1, T // 48))
    xs = qs[1] if qs[1] is None or qs[1].numel() == 1 else qs[1].reshape(T, -1)[sample.to(DEV)].contiguous()
    small = run(qs[0].view(torch.uint8).reshape(T, -1)[sample.to(DEV)].contiguous().view(qs[0].dtype).view(len(sample), H), xs, ids[sample])
    if mode != 256:  # the intermediate's per-tensor scale depends on the batch
        assert torch.equal(full[sample], small)
    ws8 = [t.cpu() if t is not None else None for t in qs]
    if mode == 0:
        ref = orc.moe_layer_bf16(ws8[0][sample], ws8[2], ws8[4], ids[sample], E)
    elif mode == 512:
        ref = orc.moe_layer_fp8(ws8[0][sample], ws8[1].reshape(T, -1)[sample], *ws8[2:], ids[sample], E, mode)
    else:
        ref = orc.moe_layer_fp8(ws8[0][sample], ws8[1], *ws8[2:], ids[sample], E, mode)
    # the layer tolerance; per-tensor mode: the sample's own intermediate scale, so the small batch is the one compared
    got = small if mode == 256 else full[sample]
    assert orc.cosine(got, ref) >= 0.999 and orc.max_rel_err(got, ref) <= 2e-2


@pytest.mark.parametrize("T,k,E,H,I", [(8192, 2, 24, 2064, 2064), (7000, 1, 5, 2048, 4368)])
def test_block_scales_by_tile(T, k, E, H, I):
    """In calls of many K blocks the activation scales are also laid out by row tile: rows of the large batch are bit-identical
    to the same rows in a small one, which reads them row-major."""
    from dqmoe_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(T)
    x = torch.randn(T, H, generator=g, device=DEV).to(torch.bfloat16)
    b = ops.per_block_cast_to_fp8((torch.randn(E, 2 * I, H, generator=g, device=DEV) * 0.05).to(torch.bfloat16))
    b1 = ops.per_block_cast_to_fp8((torch.randn(E, H, I, generator=g, device=DEV) * 0.05).to(torch.bfloat16))
    score = torch.rand(T, E, generator=torch.Generator().manual_seed(T))
    score[:, 1] = score[:, E - 1] = -1.0  # experts without rows, the last among them
    score[:, 0] += 0.5
    ids = torch.topk(score, k, dim=1).indices.to(torch.int32)
    q, s = ops.per_token_block_cast_to_fp8(x)

    def run(rows, tiled):
        n = len(rows)
        d = torch.zeros(n, k, H, dtype=torch.bfloat16, device=DEV)
        ws = torch.empty(ops.moe_workspace_bytes(n, H, I, E, k, 1024), dtype=torch.uint8, device=DEV)
        qr = q.view(torch.uint8)[rows.to(DEV)].contiguous().view(q.dtype)
        sr, idr = s[rows.to(DEV)].contiguous(), ids[rows].contiguous().to(DEV)
        names = kernels_of(lambda: ops.moe_forward(qr, sr, *b, *b1, d, idr, ws, 1024))
        assert ops.device_status() == 0
        assert any("scale_tiles" in n for n in names) == tiled, names
        return d.cpu()

    sample = torch.arange(0, T, 29)
    full, small = run(torch.arange(T), True), run(sample, False)
    assert torch.equal(full[sample], small)
    ref = orc.moe_layer_fp8(q.cpu()[sample], s.cpu()[sample], *[t.cpu() for t in b], *[t.cpu() for t in b1], ids[sample], E, 1024)
    assert orc.cosine(small, ref) >= 0.999 and orc.max_rel_err(small, ref) <= 2e-2


@pytest.mark.parametrize("n,H,I,E,tiled", [
    (14592, 2048, 2048, 2, True), (14464, 2048, 2048, 2, False),  # K blocks over all tiles
    (16384, 2048, 1920, 2, False), (16384, 1920, 2048, 2, False),  # short reductions
    (19200, 2048, 2048, 100, True), (19072, 2048, 2048, 100, False)])  # rows per expert
def test_scales_are_laid_out_by_tile_where_it_pays(n, H, I, E, tiled):
    from dqmoe_b200 import ops
    z = lambda *shape: torch.zeros(*shape, dtype=torch.uint8, device=DEV).view(ops.FP8)
    one = lambda *shape: torch.ones(*shape, device=DEV)
    g = lambda v: -(-v // 128)
    d = torch.empty(n, 1, H, dtype=torch.bfloat16, device=DEV)
    ids = (torch.arange(n, device=DEV, dtype=torch.int32) % E).view(n, 1)
    ws = torch.empty(ops.moe_workspace_bytes(n, H, I, E, 1, 1024), dtype=torch.uint8, device=DEV)
    args = (z(n, H), one(n, g(H)), z(E, 2 * I, H), one(E, g(2 * I), g(H)), z(E, H, I), one(E, g(H), g(I)), d, ids, ws, 1024)
    names = kernels_of(lambda: ops.moe_forward(*args))
    assert ops.device_status() == 0 and not d.any()
    assert any("scale_tiles" in k for k in names) == tiled, names
