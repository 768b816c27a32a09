"""Per-tensor FP8 quantiser on both sides of the size its single-launch cluster form holds (524288 elements per slice)."""
import numpy as np
import pytest
import torch

from helpers import bits, kernels_of

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("e,numel", [(1, 8), (1, 8 * 8191), (3, 8 * 8193), (2, 524288), (1, 524288 + 8)])
def test_per_tensor_quantiser_bit_exact(e, numel):
    from dqmoe_b200 import ops
    g = torch.Generator().manual_seed(numel % 1000)
    x = (torch.randn(e, 1, numel, generator=g) * 3).to(torch.bfloat16)
    x[0, 0, -1] = 77.0  # the amax in the last element: every block and thread counts
    sf = x.float().abs().amax((1, 2)).clamp(1e-4) / 448.0
    ref = (x.float() * (1.0 / sf)[:, None, None]).to(torch.float8_e4m3fn)
    q, s = ops.per_tensor_cast_to_fp8(x.to("cuda"), per_expert=True)
    assert np.array_equal(bits(s.reshape(-1)), bits(sf)) and np.array_equal(bits(q.view(e, 1, numel)), bits(ref))


@pytest.mark.parametrize("numel", [64, 131072])
def test_cluster_form_only_while_all_slices_run_at_once(numel):
    """A slice takes eight SMs in the cluster form: more slices than that go through the general one, however short they are."""
    from dqmoe_b200 import ops
    most = torch.cuda.get_device_properties(0).multi_processor_count // 8
    for e in (most, most + 1, 8 * most):
        x = torch.randn(e, 1, numel, generator=torch.Generator().manual_seed(e)).to(torch.bfloat16)
        sf = x.float().abs().amax((1, 2)).clamp(1e-4) / 448.0
        ref = (x.float() * (1.0 / sf)[:, None, None]).to(torch.float8_e4m3fn)
        xd = x.to("cuda")
        q, s = ops.per_tensor_cast_to_fp8(xd, per_expert=True)
        names = kernels_of(lambda: ops.per_tensor_cast_to_fp8(xd, per_expert=True))
        assert np.array_equal(bits(s.reshape(-1)), bits(sf)) and np.array_equal(bits(q), bits(ref))
        assert any("tensor_small" in n for n in names) == (e <= most), (e, names)


@pytest.mark.parametrize("e,numel", [(3, 1024), (40, 1024), (1, 524288 + 8)])
def test_scratch_receives_the_largest_values(e, numel):
    """Whichever form runs, the scratch holds each slice's largest absolute value afterwards."""
    import ctypes
    from dqmoe_b200 import _lib
    x = torch.randn(e, numel, generator=torch.Generator().manual_seed(e)).to(torch.bfloat16)
    xd = x.to("cuda")
    q = torch.empty(e, numel, dtype=torch.uint8, device="cuda")
    s, scratch = torch.empty(e, device="cuda"), torch.full((e,), 1e30, device="cuda")
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    _lib.check(_lib.load().dqmoe_quant_fp8_tensor(p(xd), e, numel, p(q), p(s), p(scratch),
                                                  ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    assert torch.equal(scratch.cpu(), x.float().abs().amax(1))
