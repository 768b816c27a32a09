"""Which tile form the grouped GEMM runs on - single CTAs, CTA pairs, chosen on the host or from the experts' row counts on the
device - and that the choice does not show in the results; block scales by tile likewise."""
import ctypes

import numpy as np
import pytest
import torch

from helpers import kernels_of, run_kernels, tile_form, tile_forms
from oracle import moe_oracle as orc

pytestmark = pytest.mark.gpu
DEV = "cuda"

# rows of eight experts (128 to 800 on average), the form that suits them: 2 x 256-row tiles against 1.16 x 128-row tiles
COUNTS = {
    "even-two-tiles": ([200] * 8, "pairs"),  # 16 against 16
    "ragged-two-tiles": ([129, 255, 256, 130, 200, 0, 240, 129], "pairs"),
    "odd-three-tiles": ([300] * 8, "wide"),  # 32 against 24
    "skewed": ([1400, 20, 10, 0, 130, 64, 1, 33], "wide"),  # 24 against 18, 207 rows on average
    "one-for-all": ([800, 90, 100, 120, 80, 70, 128, 60], "wide"),  # 22 against 14
    "below-the-line": ([300, 400, 600, 0, 200, 700, 10, 640], "pairs"),  # 30 against 26
    "above-the-line": ([300, 400, 600, 0, 300, 700, 10, 640], "wide"),  # 32 against 27
}


@pytest.mark.parametrize("case", list(COUNTS))
@pytest.mark.parametrize("mode,gated", [(0, True), (0, False), (256, True), (256, False), (512, True), (512, False)])
def test_row_counts_choose_the_tile_form(mode, gated, case):
    """The form that works is the one that suits the counts; every row is bit-identical to the same row in a launch of a few
    rows per expert, which takes single CTAs, and four rows of every expert agree with fp64 sums."""
    from dqmoe_b200 import _lib, ops
    counts, form = COUNTS[case]
    E, n = len(counts), sum(counts)
    K, N = (2048 if mode == 0 else 4096), (8192 if gated else 16384)  # 32 K blocks, 64 column tiles: 30000 from 15 row tiles on
    g = torch.Generator(device=DEV).manual_seed(n + mode)
    a = torch.randn(n, K, generator=g, device=DEV).to(torch.bfloat16)
    w = (torch.randn(E, (2 if gated else 1) * N, K, generator=g, device=DEV) * 0.05).to(torch.bfloat16)
    if mode == 256:
        (a, sa), (w, sw) = ops.per_tensor_cast_to_fp8(a), ops.per_tensor_cast_to_fp8(w, per_expert=True)
    elif mode == 512:
        (a, sa), (w, sw) = ops.per_token_cast_to_fp8(a), ops.per_channel_cast_to_fp8(w)
    else:
        sa = sw = None

    def run(rows_of):  # rows_of[e]: rows of expert e, as indices into the full batch
        rows = torch.cat(rows_of).to(DEV)
        off = torch.tensor(np.concatenate([[0], np.cumsum([len(r) for r in rows_of])]), dtype=torch.int32, device=DEV)
        ar = a.view(torch.uint8).view(n, -1)[rows].contiguous().view(a.dtype).view(len(rows), K)
        sr = sa if mode != 512 else sa.view(n, 1)[rows].contiguous()
        out = torch.zeros(len(rows), N, dtype=torch.bfloat16, device=DEV)
        amax = torch.zeros(len(rows) if mode == 512 else 1, device=DEV) if gated and mode else None
        mt = ops.mtile_prefix(off)
        call = lambda o, m: ops.grouped_gemm(ar, sr, w, sw, off, mt, N, mode, gated, o, amax=m)
        call(out, amax)
        # of the launched forms those that write something when they run alone
        working = []
        for f in tile_forms(lambda: call(out, amax)):
            alone, spare = torch.zeros_like(out), None if amax is None else torch.zeros_like(amax)
            run_kernels(lambda: call(alone, spare), lambda name: tile_form(name) == f)
            if alone.any():
                working.append(f)
                assert torch.equal(alone, out)
        assert ops.device_status() == 0
        return out, amax, working

    first = np.concatenate([[0], np.cumsum(counts)])
    every = [torch.arange(first[e], first[e + 1]) for e in range(E)]
    out, amax, forms = run(every)
    assert forms == [form], forms
    few = [r[torch.linspace(0, len(r) - 1, min(len(r), 60)).long()] if len(r) else r for r in every]
    small, amax_small, forms = run(few)
    assert forms == ["wide"], forms
    picked = torch.cat(few).to(DEV)
    assert torch.equal(out[picked], small)
    if not gated:  # the same rows to explicit addresses, as an expert-parallel rank stores them
        perm = torch.randperm(n, generator=g, device=DEV)
        spread = torch.zeros_like(out)
        row_dst = spread.data_ptr() + perm * (N * 2)
        off = torch.tensor(first, dtype=torch.int32, device=DEV)
        ptr = lambda t: None if t is None else ctypes.c_void_p(t.data_ptr())
        mt = ops.mtile_prefix(off)
        _lib.check(_lib.load().dqmoe_grouped_gemm_rows(ptr(a), ptr(sa), ptr(w), ptr(sw), ptr(off), ptr(mt), n, N, K, E, mode,
                                                       ptr(row_dst), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
        assert ops.device_status() == 0
        assert torch.equal(spread[perm], out)
    if mode == 512 and gated:
        assert torch.equal(amax[picked], amax_small)
        assert torch.equal(amax, out.float().abs().amax(1))
    if mode == 256 and gated:
        assert amax.item() == out.float().abs().max().item()
    for e in range(E):
        r = few[e][:: max(1, len(few[e]) // 4)].to(DEV)
        if not len(r):
            continue
        x, y = a[r].double(), w[e].double()
        if mode == 256:
            x, y = x * sa.double(), y * sw[e].double()
        elif mode == 512:
            x, y = x * sa.view(n, 1)[r].double(), y * sw[e].double()
        ref = x @ y.t()
        if gated:
            gate, val = ref.float().to(torch.bfloat16).chunk(2, dim=-1)
            ref = (torch.nn.functional.silu(gate) * val).double()
        # A flipped rounding of value, silu or product is 2^-8 of the result each, one of the gate |g| + 1 times as much (d ln
        # silu / d ln g = 1 + g (1 - sigmoid)): 2^-5 in all up to |g| = 5, beyond which silu is below 0.034 of a typical gate
        assert ((out[r].double() - ref).abs() <= 2.0 ** -5 * ref.abs() + 2.0 ** -6 * ref.abs().mean()).all()


@pytest.mark.parametrize("counts,N,K,launched,form", [
    ([127] * 8, 16384, 4096, "one", "wide"), ([256, 0] * 4, 16384, 4096, "both", "pairs"),  # from 128 rows on average: by counts
    ([200] * 8, 4096, 4096, "one", "wide"), ([511] * 8, 1024, 512, "one", "wide"), ([512] * 8, 1024, 512, "one", "pairs"),  # small
    ([896] * 4 + [640] * 4, 16384, 2048, "both", "wide"),  # 56 against 48
    ([800] * 8, 16384, 2048, "one", "pairs"), ([2000] * 4 + [1] * 4 + [0], 16384, 2048, "one", "pairs")])  # from 800 on
def test_lines_of_the_host_rule(counts, N, K, launched, form):
    """Average row counts and sizes on both sides of the lines between which the device chooses."""
    from dqmoe_b200 import ops
    E = len(counts)
    n = sum(counts)
    a = torch.zeros(n, K, dtype=torch.uint8, device=DEV).view(ops.FP8)
    w = torch.zeros(E, N, K, dtype=torch.uint8, device=DEV).view(ops.FP8)
    off = torch.tensor(np.concatenate([[0], np.cumsum(counts)]), dtype=torch.int32, device=DEV)
    out = torch.ones(n, N, dtype=torch.bfloat16, device=DEV)
    sa, sw, mt = torch.ones(1, device=DEV), torch.ones(E, device=DEV), ops.mtile_prefix(off)
    call = lambda: ops.grouped_gemm(a, sa, w, sw, off, mt, N, 256, False, out)
    forms = tile_forms(call)
    if launched == "both":
        assert forms == ["wide", "pairs"], forms
        run_kernels(call, lambda name: tile_form(name) == form)
    else:
        assert forms == [form], forms
        call()
    assert ops.device_status() == 0 and not out.any()


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
        ops.moe_forward(qr, sr, *b, *b1, d, idr, ws, 1024)
        assert ops.device_status() == 0
        names = kernels_of(lambda: ops.moe_forward(qr, sr, *b, *b1, d, idr, ws, 1024))
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
    ops.moe_forward(*args)
    assert ops.device_status() == 0 and not d.any()
    names = kernels_of(lambda: ops.moe_forward(*args))
    assert any("scale_tiles" in k for k in names) == tiled, names


@pytest.mark.parametrize("n_shared", [0, 1])
def test_block_entry_point_with_scales_by_tile(n_shared):
    """The whole MoE block lays its own workspace out and quantises on the way into expert order: with enough K blocks its scales
    go by tile too. Sampled tokens are bit-identical to a small call and agree with the oracle."""
    from dqmoe_b200 import ops
    T, k, E, H, I = 8200, 2, 7, 2048, 2064
    g = torch.Generator(device=DEV).manual_seed(3)
    x = torch.randn(T, H, generator=g, device=DEV).to(torch.bfloat16)
    b = ops.per_block_cast_to_fp8((torch.randn(E + n_shared, 2 * I, H, generator=g, device=DEV) * 0.05).to(torch.bfloat16))
    b1 = ops.per_block_cast_to_fp8((torch.randn(E + n_shared, H, I, generator=g, device=DEV) * 0.05).to(torch.bfloat16))
    logits = torch.randn(T, E, generator=g, device=DEV)
    logits[:, 1] += 3.0  # skewed, and one expert without rows
    logits[:, 4] = -100.0

    def run(rows, tiled):
        args = (x[rows].contiguous(), logits[rows].contiguous(), *b, *b1, k, "sigmoid", 1024)
        out = ops.moe_block(*args, n_shared=n_shared)
        assert ops.device_status() == 0
        names = kernels_of(lambda: ops.moe_block(*args, n_shared=n_shared))
        assert any("scale_tiles" in n for n in names) == tiled, names
        return out.cpu()

    sample = torch.arange(0, T, 173)
    full, small = run(torch.arange(T, device=DEV), True), run(sample.to(DEV), False)
    assert torch.equal(full[sample], small)
    xs = x.cpu()[sample]
    ref = orc.moe_block(xs, logits.cpu()[sample], b[0].cpu(), b1[0].cpu(), k, "sigmoid", 1024, n_shared=n_shared,
                        quantized=(*orc.quant_block_1x128(xs), *[t.cpu() for t in b], *[t.cpu() for t in b1]))
    assert orc.cosine(small, ref) >= 0.999 and orc.max_rel_err(small, ref) <= 2e-2
