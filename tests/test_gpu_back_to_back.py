"""Calls enqueued back to back on one workspace, every one with new inputs and none waited for: kernels start before their
predecessors have ended, so each must still see only its own call's data."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"
E, H, I, K = 8, 512, 384, 2
SIZES = [3, 200, 1, 33, 1100, 4, 600, 2, 90, 1500, 64]  # decode, one and several sort blocks, in turn


@pytest.fixture(scope="module")
def ops():
    from dqmoe_b200 import ops as _ops
    return _ops


def weights(ops, kind):
    g = torch.Generator(device=DEV).manual_seed(7)
    b = (torch.randn(E, 2 * I, H, generator=g, device=DEV) * 0.05).to(torch.bfloat16)
    b1 = (torch.randn(E, H, I, generator=g, device=DEV) * 0.05).to(torch.bfloat16)
    if kind == "bf16":
        return (b, None), (b1, None)
    cast = {"tensor": lambda w: ops.per_tensor_cast_to_fp8(w, per_expert=True), "block": ops.per_block_cast_to_fp8,
            "channel": ops.per_channel_cast_to_fp8, "mx": ops.mx_cast_weights_to_fp8, "nvfp4": ops.nvfp4_cast_weights}[kind]
    out = []
    for w in (b, b1):
        c = cast(w)
        out.append((c[0], c[1].reshape(-1)) if kind == "channel" else c)
    return out


MODE = {"bf16": 0, "tensor": 256, "channel": 512, "block": 1024, "mx": 2048, "nvfp4": 4096}


def layer_call(ops, kind, w, x, ids, d, ws):
    """Quantisation and layer, as a program that has new activations calls them."""
    if kind == "nvfp4":
        one = torch.full((1,), 6.0 / 2688.0, device=DEV)
        ops.moe_forward_nvfp4(*ops.nvfp4_cast(x, one), one, *w[0], *w[1], torch.full((1,), 16.0 / 2688.0, device=DEV), d, ids, ws)
        return
    q = {"bf16": lambda: (x, None), "tensor": lambda: ops.per_tensor_cast_to_fp8(x), "channel": lambda: ops.per_token_cast_to_fp8(x),
         "block": lambda: ops.per_token_block_cast_to_fp8(x), "mx": lambda: ops.mx_cast_to_fp8(x)}[kind]()
    ops.moe_forward(*q, *w[0], *w[1], d, ids, ws, MODE[kind])


def inputs(seed, T):
    g = torch.Generator(device=DEV).manual_seed(seed)
    x = torch.randn(T, H, generator=g, device=DEV).to(torch.bfloat16)
    logits = torch.randn(T, E, generator=g, device=DEV)
    return x, logits, torch.topk(logits, K, dim=1).indices.to(torch.int32)


@pytest.mark.parametrize("kind", ["bf16", "tensor", "channel", "block", "mx"])
def test_layers_and_blocks_share_a_workspace(ops, kind):
    w = weights(ops, kind)
    lib = ops._lib.load()
    need = max(lib.dqmoe_moe_block_workspace_bytes(T, H, I, E, K, MODE[kind]) for T in SIZES)
    ws = torch.empty(need, dtype=torch.uint8, device=DEV)
    calls = [(*inputs(100 + i, T), i % 3 == 2) for i, T in enumerate(SIZES * 3)]

    def run(x, logits, ids, block, out):
        if block:
            return ops.moe_block(x, logits, w[0][0], w[0][1], w[1][0], w[1][1], K, "softmax", MODE[kind], ws)
        layer_call(ops, kind, w, x, ids, out, ws)
        return out

    outs = [torch.zeros(x.shape[0], K, H, dtype=torch.bfloat16, device=DEV) for x, *_ in calls]
    alone = []
    for c, o in zip(calls, outs):
        ws.fill_(0xff)  # NaN in every format: what a call reads before it is written shows
        torch.cuda.synchronize()
        alone.append(run(*c, o).clone())
        torch.cuda.synchronize()
    for o in outs:
        o.zero_()
    torch.cuda.synchronize()
    together = [run(*c, o) for c, o in zip(calls, outs)]
    torch.cuda.synchronize()
    assert ops.device_status() == 0
    for c, a, t in zip(calls, alone, together):
        assert torch.equal(a, t), (c[0].shape, c[3])


@pytest.mark.parametrize("kind", ["bf16", "tensor", "channel", "block", "mx", "nvfp4"])
def test_a_graph_of_layers_replayed_without_waiting(ops, kind):
    """Two layers of different sizes in one captured graph, replayed in a row; between replays new inputs are copied in on the
    same stream. Nothing is waited for until the end."""
    w = weights(ops, kind) if kind != "nvfp4" else weights_nvfp4(ops)
    hidden = H
    sizes = [700, 40]
    ws = torch.empty(max(ops.moe_workspace_bytes(T, hidden, 512 if kind == "nvfp4" else I, E, K, MODE[kind]) for T in sizes),
                     dtype=torch.uint8, device=DEV)
    rounds = [[inputs(1000 * r + T, T) for T in sizes] for r in range(6)]
    alone = []
    for rd in rounds:
        for x, _, ids in rd:
            d = torch.zeros(x.shape[0], K, H, dtype=torch.bfloat16, device=DEV)
            layer_call(ops, kind, w, x, ids, d, ws)
            torch.cuda.synchronize()
            alone.append(d)
    stream = torch.cuda.Stream()
    xs = [torch.empty_like(x) for x, _, _ in rounds[0]]
    idx = [torch.zeros_like(i) for _, _, i in rounds[0]]
    ds = [torch.zeros(T, K, H, dtype=torch.bfloat16, device=DEV) for T in sizes]
    kept = []
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            for x, i, d in zip(xs, idx, ds):
                layer_call(ops, kind, w, x, i, d, ws)
        for rd in rounds:
            for j, (x, _, ids) in enumerate(rd):
                xs[j].copy_(x)
                idx[j].copy_(ids)
            graph.replay()
            kept += [d.clone() for d in ds]
    torch.cuda.synchronize()
    assert ops.device_status() == 0
    for a, t in zip(alone, kept):
        assert torch.equal(a, t)


def weights_nvfp4(ops):
    g = torch.Generator(device=DEV).manual_seed(9)
    return [ops.nvfp4_cast_weights((torch.randn(E, r, c, generator=g, device=DEV) * 0.05).to(torch.bfloat16))
            for r, c in ((1024, H), (H, 512))]


@pytest.mark.parametrize("captured", [False, True])
@pytest.mark.parametrize("kind", ["bf16", "tensor", "channel", "block", "mx"])
def test_two_streams_with_a_workspace_each(ops, kind, captured):
    """A program that forks: one stream quantises and runs a layer, another waits for an event and runs its own, both join and
    the results are added; eagerly and as a captured graph whose launches cross streams."""
    w = weights(ops, kind)
    side, main = torch.cuda.Stream(), torch.cuda.Stream()
    (x0, _, i0), (x1, _, i1) = inputs(11, 300), inputs(12, 300)
    ws = [torch.empty(ops.moe_workspace_bytes(300, H, I, E, K, MODE[kind]), dtype=torch.uint8, device=DEV) for _ in range(2)]
    want = []
    for x, i in ((x0, i0), (x1, i1)):
        d = torch.zeros(300, K, H, dtype=torch.bfloat16, device=DEV)
        layer_call(ops, kind, w, x, i, d, ws[0])
        torch.cuda.synchronize()
        want.append(d)
    d0, d1 = torch.zeros_like(want[0]), torch.zeros_like(want[0])
    keep = []

    def step():
        scaled = x1 * 2.0  # work in front of the fork that the other stream must wait for
        halved = scaled * 0.5
        side.wait_stream(main)
        with torch.cuda.stream(side):
            layer_call(ops, kind, w, halved, i1, d1, ws[1])
        layer_call(ops, kind, w, x0, i0, d0, ws[0])
        main.wait_stream(side)
        keep.append((scaled, halved))
        return d0 + d1

    torch.cuda.synchronize()
    with torch.cuda.stream(main):
        if captured:
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=main):
                total = step()
            for _ in range(5):
                d0.zero_()
                d1.zero_()
                graph.replay()
        else:
            for _ in range(5):
                d0.zero_()
                d1.zero_()
                total = step()
    torch.cuda.synchronize()
    assert ops.device_status() == 0
    assert torch.equal(d0, want[0]) and torch.equal(d1, want[1])
    assert torch.equal(total, want[0] + want[1])
