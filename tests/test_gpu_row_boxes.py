"""Tiles with the rows on M load the rows that an expert has in boxes of 32: experts around their edges, and what a tile's unused rows
held before does not show."""
import pytest
import torch

from oracle import moe_oracle as orc

pytestmark = pytest.mark.gpu
DEV = "cuda"
ROWS = [1, 31, 32, 33, 63, 64, 65, 95, 96, 97, 127, 128, 129, 0, 161]


@pytest.mark.parametrize("H,I", [(256, 384), (640, 128), (4096, 1280)])  # the first two: at most one tile per block, whole copies
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


@pytest.mark.parametrize("mode", [256, 512])
def test_unused_rows_stay_out_of_the_amax(mode):
    """The stand-alone gated GEMM of the two-pass modes, which also gives the largest |output| per tensor or per row: NaN left in a
    tile's unused rows by a launch of full tiles reaches neither."""
    from dqmoe_b200 import ops
    E, n, K, N = len(ROWS), sum(ROWS), 384, 1280  # 17 row tiles x 10: more than one per block, so that rows come in boxes
    g = torch.Generator(device=DEV).manual_seed(mode)
    x = torch.randn(n, K, generator=g, device=DEV).to(torch.bfloat16)
    w = (torch.randn(E, 2 * N, K, generator=g, device=DEV) * 0.05).to(torch.bfloat16)
    (q, s), (wq, ws) = ((ops.per_tensor_cast_to_fp8(x), ops.per_tensor_cast_to_fp8(w, per_expert=True)) if mode == 256 else
                        (ops.per_token_cast_to_fp8(x), ops.per_channel_cast_to_fp8(w)))

    def run(rows, counts):
        offsets = torch.tensor([0] + counts, dtype=torch.int32, device=DEV).cumsum(0, dtype=torch.int32)
        out, amax = torch.zeros(n, N, dtype=torch.bfloat16, device=DEV), torch.zeros(n if mode == 512 else 1, device=DEV)
        ops.grouped_gemm(rows, s, wq, ws, offsets, ops.mtile_prefix(offsets), N, mode, True, out, amax=amax)
        assert ops.device_status() == 0
        return out, amax

    out, amax = run(q, ROWS)
    assert torch.equal(amax, out.float().abs().amax(1) if mode == 512 else out.float().abs().amax().reshape(1))
    run(torch.full_like(q.view(torch.uint8), 0x7F).view(q.dtype), [n - n // 2, n // 2] + [0] * (E - 2))
    again, amax_again = run(q, ROWS)
    assert torch.equal(again, out) and torch.equal(amax_again, amax)


@pytest.mark.parametrize("kind", ["f16", "f32", "nvfp4"])
def test_unused_rows_in_the_other_layers(kind):
    """fp16 and fp32 operands, and NVFP4, whose e2m1 values know no NaN but whose scale bytes do."""
    from dqmoe_b200 import ops
    E, T, H, I = len(ROWS), sum(ROWS), 256, 1280
    g = torch.Generator(device=DEV).manual_seed(5)
    x = torch.randn(T, H, generator=g, device=DEV)
    w, w1 = torch.randn(E, 2 * I, H, generator=g, device=DEV) * 0.05, torch.randn(E, H, I, generator=g, device=DEV) * 0.05
    ids = torch.repeat_interleave(torch.arange(E), torch.tensor(ROWS))[torch.randperm(T, generator=torch.Generator().manual_seed(5))]
    ids = ids.to(torch.int32).view(T, 1)
    if kind == "nvfp4":
        act_g = torch.full((1,), 16.0 / 2688.0, device=DEV)
        x_g = ops.nvfp4_global_scale(x.to(torch.bfloat16))
        b, b1 = ops.nvfp4_cast_weights(w.to(torch.bfloat16)), ops.nvfp4_cast_weights(w1.to(torch.bfloat16))
        q, sf = ops.nvfp4_cast(x.to(torch.bfloat16), x_g)
        inputs, nan = (q, sf), (q, torch.full_like(sf, 0x7F))
        ws = torch.empty(ops.moe_workspace_bytes(T, H, I, E, 1, 4096), dtype=torch.uint8, device=DEV)
        layer = lambda a, d, i: ops.moe_forward_nvfp4(*a, x_g, *b, *b1, act_g, d, i, ws)
        out_type = torch.bfloat16
    else:
        out_type = torch.float16 if kind == "f16" else torch.float32
        b, b1, inputs = w.to(out_type), w1.to(out_type), x.to(out_type)
        nan = torch.full_like(inputs, float("nan"))
        need = ops.moe_workspace_bytes(T, H, I, E, 1, 0) if kind == "f16" else ops.moe_workspace_bytes_f32(T, H, I, E, 1)
        ws = torch.empty(need, dtype=torch.uint8, device=DEV)
        layer = lambda a, d, i: (ops.moe_forward_f16 if kind == "f16" else ops.moe_forward_f32)(a, b, b1, d, i, ws)

    def run(a, i):
        d = torch.zeros(T, 1, H, dtype=out_type, device=DEV)
        layer(a, d, i.to(DEV))
        assert ops.device_status() == 0
        return d

    first = run(inputs, ids)
    assert torch.isfinite(first).all() and first.any()
    run(nan, (torch.arange(T, dtype=torch.int32) % 2).view(T, 1))
    assert torch.equal(run(inputs, ids), first)
