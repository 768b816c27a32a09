"""The streaming kernels around the grouped GEMM at the edges of their strips and batches: scatter into expert order with
dropped slots, odd slot counts and rows that end inside a strip; weighted combine; quantisers."""
import numpy as np
import pytest
import torch

from helpers import bits, kernels_of
from oracle import moe_oracle as orc

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.fixture(scope="module")
def ops():
    from dqmoe_b200 import ops as _ops
    return _ops


@pytest.mark.parametrize("k", [1, 2, 3, 4, 5, 9, 17])
@pytest.mark.parametrize("T,H", [(1, 8), (7, 264), (300, 1032)])
def test_weighted_combine(ops, T, H, k):
    g = torch.Generator().manual_seed(T + k)
    d = torch.randn(T, k, H, generator=g).to(torch.bfloat16)
    w = torch.rand(T, k, generator=g)
    w[0, k // 2] = 0.0
    clean = d.double().clone()
    d[0, k // 2] = float("nan")  # a slot of weight zero was never written
    clean[0, k // 2] = 0.0
    ref = (clean * w.double()[:, :, None]).sum(1)
    out = ops.finalize_weighted(d.to(DEV), w.to(DEV)).cpu().double()
    # k fp32 roundings of partial sums, then one to bf16 (half an ulp = 2^-9)
    bound = (clean.abs() * w.double()[:, :, None]).sum(1) * k * 2.0 ** -24 + ref.abs() * 2.0 ** -8 + 1e-30
    assert bool(((out - ref).abs() <= bound).all())


@pytest.mark.parametrize("mode", [0, 512, 1024])
@pytest.mark.parametrize("T,H,k", [(9, 16, 1), (65, 528, 5), (40, 1040, 3), (9, 2064, 2)])
def test_expert_order_with_dropped_slots(ops, mode, T, H, k):
    import ctypes
    from dqmoe_b200 import _lib
    E, I = 6, 64
    g = torch.Generator().manual_seed(T * k)
    x = torch.randn(T, H, generator=g).to(torch.bfloat16)
    ids = torch.randint(-1, E + 1, (T, k), generator=g, dtype=torch.int32)  # -1 and E drop the slot
    b = torch.randn(E, 2 * I, H, generator=g).to(torch.bfloat16)
    b1 = torch.randn(E, H, I, generator=g).to(torch.bfloat16)
    ws = torch.empty(ops.moe_workspace_bytes(T, H, I, E, k, mode), dtype=torch.uint8, device=DEV)
    d = torch.zeros(T, k, H, dtype=torch.bfloat16, device=DEV)
    if mode == 0:
        q, s = x, None
        ops.moe_forward(x.to(DEV), None, b.to(DEV), None, b1.to(DEV), None, d, ids.to(DEV), ws, mode)
    else:
        qs = orc.quantize_inputs(x, b, b1, mode)
        q, s = qs[0], qs[1].reshape(T, -1)
        ops.moe_forward(*[t.to(DEV).contiguous() for t in qs], d, ids.to(DEV), ws, mode)
    torch.cuda.synchronize()
    assert ops.device_status() == 0
    flat = ids.reshape(-1)
    order = [i for e in range(E) for i in range(T * k) if int(flat[i]) == e]
    lib = _lib.load()

    def view(which, nbytes):
        off = lib.dqmoe_moe_workspace_ptr(ctypes.c_void_p(ws.data_ptr()), which, T, H, I, E, k, mode) - ws.data_ptr()
        return ws[off:off + nbytes].cpu()

    tok = torch.tensor([i // k for i in order], dtype=torch.long)
    rows = q.contiguous().view(torch.uint8).reshape(T, -1)[tok]
    assert torch.equal(view(2, rows.numel()).view(rows.shape), rows)
    if s is not None:
        want = s[tok].contiguous()
        assert torch.equal(view(3, want.numel() * 4).view(torch.float32).view(want.shape), want)
    for i in range(T * k):
        if not 0 <= int(flat[i]) < E:
            assert not d[i // k, i % k].any()


@pytest.mark.parametrize("rows,cols", [(1, 8), (33, 2048), (5, 2056), (257, 120)])
def test_rowwise_quantiser_bit_exact(ops, rows, cols):
    g = torch.Generator().manual_seed(cols)
    x = torch.randn(rows, cols, generator=g).to(torch.bfloat16)
    x[0] = 0
    amax = x.float().abs().amax(1, keepdim=True).clamp(1e-4)
    sf = amax / 448.0
    ref = (x.float() * (1.0 / sf)).to(torch.float8_e4m3fn)
    q, s = ops.per_token_cast_to_fp8(x.to(DEV))
    assert np.array_equal(bits(s.reshape(-1)), bits(sf.reshape(-1))) and np.array_equal(bits(q), bits(ref))


@pytest.mark.parametrize("rows,cols", [(1, 16), (3, 1040), (130, 528), (2, 136)])
def test_1x128_quantiser_bit_exact(ops, rows, cols):
    g = torch.Generator().manual_seed(cols)
    x = torch.randn(rows, cols, generator=g).to(torch.bfloat16)
    pad = torch.nn.functional.pad(x.float(), (0, -cols % 128)).view(rows, -1, 128)
    sf = pad.abs().amax(2).clamp(1e-4) / 448.0
    ref = (pad * (1.0 / sf)[:, :, None]).view(rows, -1)[:, :cols].to(torch.float8_e4m3fn)
    q, s = ops.per_token_block_cast_to_fp8(x.to(DEV))
    assert np.array_equal(bits(s), bits(sf)) and np.array_equal(bits(q), bits(ref))


@pytest.mark.parametrize("E,rows,cols", [(1, 1, 8), (2, 130, 264), (5, 900, 1000)])
def test_128x128_quantiser_bit_exact(ops, E, rows, cols):
    g = torch.Generator().manual_seed(rows)
    w = (torch.randn(E, rows, cols, generator=g) * 0.02).to(torch.bfloat16)
    R, Cb = -(-rows // 128), -(-cols // 128)
    pad = torch.zeros(E, R * 128, Cb * 128)
    pad[:, :rows, :cols] = w.float()
    blk = pad.view(E, R, 128, Cb, 128)
    sf = blk.abs().amax((2, 4)).clamp(1e-4) / 448.0
    ref = (blk * (1.0 / sf)[:, :, None, :, None]).view(E, R * 128, Cb * 128)[:, :rows, :cols].contiguous().to(torch.float8_e4m3fn)
    q, s = ops.per_block_cast_to_fp8(w.to(DEV))
    assert np.array_equal(bits(s), bits(sf)) and np.array_equal(bits(q), bits(ref))


@pytest.mark.parametrize("rows,cols,strips", [(3, 512, False), (1000, 128, False), (3, 528, True), (700, 1040, True), (5, 1032, False)])
def test_1x128_quantiser_takes_strips_for_rows_that_fill_them(ops, rows, cols, strips):
    g = torch.Generator().manual_seed(cols)
    x = torch.randn(rows, cols, generator=g).to(torch.bfloat16)
    xd = x.to(DEV)
    names = kernels_of(lambda: ops.per_token_block_cast_to_fp8(xd))
    assert any("scatter_quant" in n for n in names) == strips, names
    q, s = orc.quant_block_1x128(x)
    qd, sd = ops.per_token_block_cast_to_fp8(xd)
    assert np.array_equal(bits(sd), bits(s)) and np.array_equal(bits(qd), bits(q))


@pytest.mark.parametrize("k", [1, 3, 5, 6, 7, 8, 9])
def test_combine_batches_as_many_slots_as_there_are(ops, k):
    d, w = torch.randn(33, k, 264, device=DEV).to(torch.bfloat16), torch.rand(33, k, device=DEV)
    names = kernels_of(lambda: ops.finalize_weighted(d, w))
    assert any(f"finalize_weighted_kernelILi{4 if k == 3 else min(k, 8)}E" in n for n in names), names
