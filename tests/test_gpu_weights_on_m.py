"""The layer's grouped GEMM with the weights on M at the edges of its tiles: units of 16 rows (32 on CTA pairs), tiles of 64 rows in
block mode and 256 otherwise, two or four K blocks per accumulator buffer, value rows that change weight-scale block inside a tile,
output columns that end inside one. Also the router and the sort of a small block call in one launch."""
import re

import numpy as np
import pytest
import torch

from helpers import kernels_of

pytestmark = pytest.mark.gpu
DEV = "cuda"

# rows per expert: around the units and tiles of single CTAs (below 30 rows on average, block mode below 40) and of pairs
FEW = [1, 15, 16, 17, 31, 32, 33, 0, 48, 63, 64, 65, 3, 97, 2, 30, 1, 0]
FEWEST = [1, 0, 5, 16, 2, 13, 1, 4]
MANY = [255, 256, 257, 288, 0, 289, 31, 33, 511, 513, 780, 1, 64, 1030]


def by_row_tiles(ops, mode, x, b, b1, ids, E):
    """The same layer step by step through the stand-alone operators, whose grouped GEMM has the rows on M."""
    counts, offsets, dest_to_src, _ = ops.route_sort(ids, E)
    kept = int(offsets[-1])
    T, k = ids.shape
    I, H = b1[0].shape[2], b1[0].shape[1]
    if mode == 0:
        q, s = x, None
    else:
        q, s = {256: ops.per_tensor_cast_to_fp8, 512: ops.per_token_cast_to_fp8, 1024: ops.per_token_block_cast_to_fp8}[mode](x)
    src = dest_to_src[:kept].long()
    rows = q.view(torch.uint8).view(T, -1)[src // k].contiguous().view(q.dtype)
    rs = s if mode in (0, 256) else s.view(T, -1)[src // k].contiguous()
    mt = ops.mtile_prefix(offsets)
    d = torch.zeros(T * k, H, dtype=torch.bfloat16, device=DEV)
    scale = (lambda w: None) if mode == 0 else (lambda w: w[1])
    act = torch.zeros(kept, I, dtype=ops.FP8 if mode == 1024 else torch.bfloat16, device=DEV)
    act_s = None
    if mode == 1024:
        act_s = torch.zeros(kept, (I + 127) // 128, device=DEV)
        ops.grouped_gemm(rows, rs, b[0], scale(b), offsets, mt, I, mode, True, act, out_scale=act_s)
    elif mode == 0:
        ops.grouped_gemm(rows, None, b[0], None, offsets, mt, I, mode, True, act)
    else:
        amax = torch.zeros(kept if mode == 512 else 1, device=DEV)
        ops.grouped_gemm(rows, rs, b[0], scale(b), offsets, mt, I, mode, True, act, amax=amax)
        act, act_s = ops.requant_from_amax(act, amax, mode == 512)
    ops.grouped_gemm(act, act_s, b1[0], scale(b1), offsets, mt, H, mode, False, d, dest_to_src=dest_to_src[:kept].contiguous())
    return q, s, d.view(T, k, H)


@pytest.mark.parametrize("mode", [0, 256, 512, 1024])
@pytest.mark.parametrize("rows,H,I", [
    (FEW, 640, 144), (FEW, 1152, 400), (FEW, 144, 1040),  # K loops of 1 to 9 blocks in groups of two and four; split scale blocks
    (FEWEST, 2064, 272), (FEWEST, 512, 1936),              # H and I that end inside a tile of columns
    (MANY, 400, 208)])
def test_rows_equal_those_of_row_tiles(mode, rows, H, I):
    """Bit-identical: both forms add the products of a K step and the K blocks in the same order, and round at the same points."""
    from dqmoe_b200 import ops
    E, n = len(rows), sum(rows)
    g = torch.Generator(device=DEV).manual_seed(n + H + mode)
    k = 2 if n % 2 == 0 else 1
    T = n // k
    x = torch.randn(T, H, generator=g, device=DEV).to(torch.bfloat16)
    ids = torch.repeat_interleave(torch.arange(E), torch.tensor(rows))[torch.randperm(n, generator=torch.Generator().manual_seed(n))]
    ids = ids.to(torch.int32).view(T, k)
    ids[3, 0] = -1  # dropped rows
    ids[T - 1, k - 1] = E
    ids = ids.to(DEV)
    w = (torch.randn(E, 2 * I, H, generator=g, device=DEV) * 0.05).to(torch.bfloat16)
    w1 = (torch.randn(E, H, I, generator=g, device=DEV) * 0.05).to(torch.bfloat16)
    cast = {0: lambda t: (t, None), 256: lambda t: ops.per_tensor_cast_to_fp8(t, per_expert=True), 512: ops.per_channel_cast_to_fp8,
            1024: ops.per_block_cast_to_fp8}[mode]
    b, b1 = cast(w), cast(w1)
    q, s, want = by_row_tiles(ops, mode, x, b, b1, ids, E)
    d = torch.zeros(T, k, H, dtype=torch.bfloat16, device=DEV)
    ws = torch.empty(ops.moe_workspace_bytes(T, H, I, E, k, mode), dtype=torch.uint8, device=DEV)
    bs, b1s = (b[1].reshape(-1), b1[1].reshape(-1)) if mode == 512 else (b[1], b1[1])
    args = (q, s, b[0], bs, b1[0], b1s, d, ids, ws, mode)
    ops.moe_forward(*args)
    assert ops.device_status() == 0
    assert torch.equal(d, want)
    on_m = any("tcgen05_wm" in name for name in kernels_of(lambda: ops.moe_forward(*args)))
    assert on_m == (mode != 1024 or n < 40 * E)


@pytest.mark.parametrize("rows,E,H,I,pairs", [(29, 37, 256, 192, [False, False]), (30, 37, 256, 192, [True, False]),
                                              (30, 38, 512, 256, [True, True]), (47, 9, 512, 256, [False, False]),
                                              (48, 9, 512, 256, [True, True])])
@pytest.mark.parametrize("mode", [0, 256, 512])
def test_lines_between_single_ctas_and_pairs(mode, rows, E, H, I, pairs):
    """fc1 and fc2 run on CTA pairs from 30 rows per expert on if a tile of 128 or 256 columns per expert fills the 74 pairs (fc1: I /
    128 tiles, fc2: H / 256), otherwise from 48."""
    from dqmoe_b200 import ops
    T = rows * E
    z = lambda *shape: torch.zeros(*shape, dtype=torch.bfloat16 if mode == 0 else torch.uint8, device=DEV).view(torch.bfloat16 if mode == 0 else ops.FP8)
    one = lambda n: torch.ones(n, device=DEV) if mode else None
    ids = (torch.arange(T, dtype=torch.int32, device=DEV) % E).view(T, 1)
    ws = torch.empty(ops.moe_workspace_bytes(T, H, I, E, 1, mode), dtype=torch.uint8, device=DEV)
    d = torch.ones(T, 1, H, dtype=torch.bfloat16, device=DEV)
    args = (z(T, H), one(1 if mode == 256 else T), z(E, 2 * I, H), one(E if mode == 256 else E * 2 * I), z(E, H, I),
            one(E if mode == 256 else E * H), d, ids, ws, mode)
    ops.moe_forward(*args)
    assert ops.device_status() == 0 and not d.any()
    forms = [m.group(1) == "1" for m in (re.search(r"tcgen05_wmILb\dELi\dELb\dELb(\d)E", name) for name in kernels_of(lambda: ops.moe_forward(*args))) if m]
    assert forms == pairs


LONG, SHORT, TINY = (4112, 2832), (6160, 1936), (640, 144)  # both reductions from 2048 on; one below; by their many experts


@pytest.mark.parametrize("rows,shapes", [
    ([30] * 8, {LONG: True, SHORT: True}),
    ([10, 20, 30, 64, 65], {LONG: True, SHORT: True}),   # 6 tiles of 64 rows against 5 of 128
    ([10, 20, 30, 65], {LONG: False, SHORT: True}),      # 5 against 4
    ([10, 65, 0, 0], {LONG: False, SHORT: True}),        # 3 against 2
    ([0, 300] + [0] * 8, {LONG: False, SHORT: False}),   # 5 against 3
    ([300] + [3] * 20, {LONG: True, SHORT: True}),
    ([128, 0, 0, 0], {LONG: False, SHORT: False}), ([129, 0, 0, 64, 0], {LONG: False, SHORT: True}), ([64, 64, 0, 0], {LONG: True, SHORT: True}),
    ([1] * 700 + [65] * 170 + [0] * 40, {TINY: True}), ([65] * 300 + [1] * 350 + [0] * 10, {TINY: True}),
    ([65] * 300 + [1] * 200 + [0] * 30, {TINY: False}),
    ([300] + [0] * 9, {TINY: None})])                    # weights that stay in L2: on M without a count
def test_row_counts_choose_the_form_of_block_calls(rows, shapes):
    for (H, I), on_m in shapes.items():
        check_block_form(rows, H, I, on_m)


def check_block_form(rows, H, I, on_m):
    """Block mode with more than 64 tokens and fewer than 40 rows per expert: the kernel takes row tiles where there are more than 1.2
    (short reductions: 1.5) times as many tiles of 64 rows as of 128. Either way the result is that of calls of up to 64 tokens, which
    have the weights on M, bit for bit, with biases too. The form shows in the intermediate's scales by column, which end the workspace
    and only one writes."""
    from dqmoe_b200 import ops
    E, T = len(rows), sum(rows)
    g = torch.Generator(device=DEV).manual_seed(T + H)
    x = torch.randn(T, H, generator=g, device=DEV).to(torch.bfloat16)
    b = ops.per_block_cast_to_fp8((torch.randn(E, 2 * I, H, generator=g, device=DEV) * 0.05).to(torch.bfloat16))
    b1 = ops.per_block_cast_to_fp8((torch.randn(E, H, I, generator=g, device=DEV) * 0.05).to(torch.bfloat16))
    bias1, bias2 = torch.randn(E, 2 * I, generator=g, device=DEV) * 0.1, torch.randn(E, H, generator=g, device=DEV) * 0.1
    ids = torch.repeat_interleave(torch.arange(E), torch.tensor(rows))[torch.randperm(T, generator=torch.Generator().manual_seed(T))]
    ids = ids.to(torch.int32).view(T, 1).to(DEV)
    q, s = ops.per_token_block_cast_to_fp8(x)

    def run(first, last):
        n = last - first
        ws = torch.full((ops.moe_workspace_bytes(n, H, I, E, 1, 1024),), 0xAB, dtype=torch.uint8, device=DEV)
        d = torch.zeros(n, 1, H, dtype=torch.bfloat16, device=DEV)
        part = lambda t: t[first:last].contiguous()
        args = (part(q.view(torch.uint8)).view(q.dtype), part(s), *b, *b1, d, part(ids), ws, 1024)
        ops.moe_forward(*args, bias1=bias1, bias2=bias2)
        assert ops.device_status() == 0
        names = kernels_of(lambda: ops.moe_forward(*args, bias1=bias1, bias2=bias2))
        assert sum("by_counts" in name for name in names) == (2 if n > 64 and on_m is not None else 0), names
        by_column = (n + 16 + 3) // 4 * 4 * ((I + 127) // 128) * 4
        return d, bool((ws[-(-(-by_column // 256) * 256):] != 0xAB).any())

    d, used = run(0, T)
    assert used == (on_m is not False)
    for first in range(0, min(T, 512), 64):
        small, used = run(first, min(T, first + 64))
        assert used and torch.equal(d[first:first + 64], small)


@pytest.mark.parametrize("T,E,k,H,I,on_m", [
    (23, 1, 1, 2048, 512, True), (24, 1, 1, 2048, 512, False), (200, 1, 1, 2048, 512, False),  # rows per expert
    (200, 3, 1, 1408, 512, False), (200, 3, 1, 1536, 512, True),                               # 33 and 36 tiles
    (300, 2, 2, 2048, 10912, False), (300, 2, 2, 2048, 10928, None)])                          # weights of 128 MiB in FP8; in bf16 beyond
@pytest.mark.parametrize("mode", [0, 256, 512])
def test_layers_of_small_models_have_row_tiles(mode, T, E, k, H, I, on_m):
    """On both sides of the lines the results are those of the row tiles, bit for bit, with biases as without (of zero)."""
    from dqmoe_b200 import ops
    if I > 10000:
        on_m = mode == 0 or on_m is None
    g = torch.Generator(device=DEV).manual_seed(T + H + mode)
    x = torch.randn(T, H, generator=g, device=DEV).to(torch.bfloat16)
    ids = torch.stack([torch.randperm(E, generator=torch.Generator().manual_seed(t))[:k] for t in range(T)]).to(torch.int32).to(DEV)
    w = (torch.randn(E, 2 * I, H, generator=g, device=DEV) * 0.05).to(torch.bfloat16)
    w1 = (torch.randn(E, H, I, generator=g, device=DEV) * 0.05).to(torch.bfloat16)
    cast = {0: lambda t: (t, None), 256: lambda t: ops.per_tensor_cast_to_fp8(t, per_expert=True), 512: ops.per_channel_cast_to_fp8}[mode]
    b, b1 = cast(w), cast(w1)
    q, s, want = by_row_tiles(ops, mode, x, b, b1, ids, E)
    bs, b1s = (b[1].reshape(-1), b1[1].reshape(-1)) if mode == 512 else (b[1], b1[1])
    ws = torch.empty(ops.moe_workspace_bytes(T, H, I, E, k, mode), dtype=torch.uint8, device=DEV)
    for bias in ({}, dict(bias1=torch.zeros(E, 2 * I, device=DEV), bias2=torch.zeros(E, H, device=DEV))):
        d = torch.zeros(T, k, H, dtype=torch.bfloat16, device=DEV)
        call = lambda: ops.moe_forward(q, s, b[0], bs, b1[0], b1s, d, ids, ws, mode, **bias)
        call()
        assert ops.device_status() == 0 and torch.equal(d, want)
        assert any("tcgen05_wm" in name for name in kernels_of(call)) == on_m


@pytest.mark.parametrize("T,E,k,n_shared", [(1, 3, 1, 0), (5, 8, 2, 0), (31, 33, 8, 1), (32, 32, 8, 1), (33, 32, 8, 1), (85, 20, 3, 2),
                                            (256, 70, 1, 5), (257, 70, 1, 5), (16, 256, 4, 0), (64, 9, 3, 0),
                                            (64, 9, 4, 0), (65, 9, 1, 0), (32, 40, 6, 2)])
@pytest.mark.parametrize("scoring", ["softmax", "sigmoid"])
def test_router_and_sort_of_a_small_block_call(T, E, k, n_shared, scoring):
    """The block's router and sort, in one launch up to 64 tokens and 192 choices, name the same experts, weights and order as the two operators:
    the block's result is that of the layer on the operators' routing, weighted."""
    from dqmoe_b200 import ops
    H, I = 128, 64
    g = torch.Generator(device=DEV).manual_seed(T * E)
    x = torch.randn(T, H, generator=g, device=DEV).to(torch.bfloat16)
    logits = torch.randn(T, E, generator=g, device=DEV)
    logits[0, : E // 2] = logits[0, 0].item()  # ties
    if T > 3:
        logits[1] = float("-inf")
        logits[2, 0] = float("inf") if scoring == "sigmoid" else 3.0e38
        logits[3] = float("nan")  # no choice: the token's rows are dropped
    E_all, slots = E + n_shared, k + n_shared
    w = (torch.randn(E_all, 2 * I, H, generator=g, device=DEV) * 0.05).to(torch.bfloat16)
    w1 = (torch.randn(E_all, H, I, generator=g, device=DEV) * 0.05).to(torch.bfloat16)
    b, b1 = ops.per_block_cast_to_fp8(w), ops.per_block_cast_to_fp8(w1)
    ws = torch.zeros(1 << 24, dtype=torch.uint8, device=DEV)  # a dropped row's result is what the workspace held
    block = lambda: ops.moe_block(x, logits, *b, *b1, k, scoring, 1024, workspace=ws, n_shared=n_shared)
    out = block()
    names = kernels_of(block)
    assert any("route_sort_small" in nm for nm in names) == (T <= 64 and T * k <= 192), names
    idx, wt = ops.route_topk(logits, k, scoring)
    shared = torch.arange(E, E_all, dtype=torch.int32, device=DEV).expand(T, n_shared)
    idx = torch.cat([idx, shared], 1).contiguous()
    wt = torch.cat([wt, torch.ones(T, n_shared, device=DEV)], 1).contiguous()
    q, s = ops.per_token_block_cast_to_fp8(x)
    d = torch.zeros(T, slots, H, dtype=torch.bfloat16, device=DEV)
    lws = torch.empty(ops.moe_workspace_bytes(T, H, I, E_all, slots, 1024), dtype=torch.uint8, device=DEV)
    ops.moe_forward(q, s, *b, *b1, d, idx, lws, 1024)
    assert ops.device_status() == 0
    want = ops.finalize_weighted(d, wt)
    assert np.array_equal(torch.isnan(want).cpu().numpy(), torch.isnan(out).cpu().numpy())
    assert torch.equal(torch.nan_to_num(want), torch.nan_to_num(out))
