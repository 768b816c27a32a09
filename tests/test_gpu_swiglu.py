"""SwiGLU of the grouped GEMM's epilogue for every bf16 gate - subnormal, huge, infinite, NaN - and the amax that the
re-quantising modes take over its results."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def every_bf16():
    return torch.arange(-32768, 32768, dtype=torch.int32).to(torch.int16).view(torch.bfloat16)


def agrees(got, gate, value):
    """got = bf16(bf16(silu(gate)) * value) up to one flipped rounding of the silu (2^-8) and of the product (2^-8); below
    gate = -87.3 the silu, less than 1e-36, may be flushed."""
    silu = gate.double() / (1.0 + torch.exp(-gate.double()))
    silu[gate == -float("inf")] = float("nan")  # -inf / inf
    ref = (silu * value.double()).to(torch.bfloat16).double()
    got = got.double()
    assert torch.equal(torch.isnan(got), torch.isnan(ref))
    assert torch.equal(torch.isinf(got), torch.isinf(ref)) and torch.equal(got[torch.isinf(ref)], ref[torch.isinf(ref)])
    ok = torch.isfinite(ref)
    assert ((got - ref).abs()[ok] <= (2.0 ** -7 * ref.abs() + 1e-36 * value.double().abs())[ok]).all()


@pytest.mark.parametrize("value", [1.0, -3.0])
def test_every_gate_unquantised(value):
    from dqmoe_b200 import ops
    gate = every_bf16()
    N, K = gate.numel(), 8
    w = torch.zeros(1, 2 * N, K, dtype=torch.bfloat16)
    w[0, :N, 0] = gate
    w[0, N:, 0] = value
    a = torch.zeros(3, K, dtype=torch.bfloat16)
    a[:, 0] = 1.0
    off = torch.tensor([0, 3], dtype=torch.int32, device=DEV)
    out = torch.zeros(3, N, dtype=torch.bfloat16, device=DEV)
    ops.grouped_gemm(a.to(DEV), None, w.to(DEV), None, off, ops.mtile_prefix(off), N, 0, True, out)
    assert ops.device_status() == 0
    for r in range(3):
        agrees(out[r].cpu(), gate, torch.full((N,), value, dtype=torch.bfloat16))


@pytest.mark.parametrize("mode", [512, 256])
@pytest.mark.parametrize("limit", [float("inf"), 3e38, 1e4, 1e-30])
def test_amax_over_every_gate(mode, limit):
    """The gates enter as weight scales (one per column, or the tensor's) of products that are 1. NaN counts for nothing in the
    amax, infinities do."""
    from dqmoe_b200 import ops
    gate = every_bf16()
    gate = gate[(gate.float().abs() <= limit) | torch.isnan(gate.float())] if limit != float("inf") else gate
    gate = gate[: gate.numel() // 16 * 16]
    one = torch.ones(1, dtype=torch.float32)
    K = 16
    off = torch.tensor([0, 2], dtype=torch.int32, device=DEV)
    a = torch.zeros(2, K)
    a[:, 0] = 1.0
    if mode == 512:
        N = gate.numel()
        w = torch.zeros(1, 2 * N, K)
        w[0, :, 0] = 1.0
        sw = torch.cat([gate.float(), torch.ones(N)])
        sa = torch.ones(2)
        columns = gate
    else:  # one scale for gate and value: powers of two in e4m3 reach the smallest and largest products
        N = 64
        w = torch.zeros(1, 2 * N, K)
        w[0, :, 0] = torch.exp2(torch.arange(2 * N) % 16 - 7.0) * (1 - 2 * (torch.arange(2 * N) // 16 % 2))
        sw, sa = torch.tensor([min(limit, 1e36)]), one
        columns = (w[0, :N, 0] * sw).to(torch.bfloat16)
    out = torch.zeros(2, N, dtype=torch.bfloat16, device=DEV)
    amax = torch.zeros(2 if mode == 512 else 1, device=DEV)
    ops.grouped_gemm(a.to(ops.FP8).to(DEV), sa.to(DEV), w.to(ops.FP8).to(DEV), sw.to(DEV), off, ops.mtile_prefix(off), N, mode,
                     True, out, amax=amax)
    assert ops.device_status() == 0
    got = out.cpu()
    agrees(got[0], columns, torch.ones(N, dtype=torch.bfloat16) if mode == 512 else (w[0, N:, 0] * sw).to(torch.bfloat16))
    assert torch.equal(got[0].view(torch.int16), got[1].view(torch.int16))
    finite = got.float().abs().nan_to_num(nan=0.0, posinf=float("inf"))
    want = finite.amax(1) if mode == 512 else finite.amax().view(1)
    assert torch.equal(amax.cpu(), want)
