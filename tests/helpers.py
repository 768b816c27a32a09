"""Shared helpers of the tests: seeded inputs, golden-file access, bit views."""
from __future__ import annotations

import os
import re

import numpy as np
import torch

GOLDEN = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden")


def make_inputs(seed, T, H, I, E, k, act_std=1.0, w_std=0.02):
    """Same generator as tests/golden/make_golden.py:make_inputs (CPU tensors)."""
    g = torch.Generator().manual_seed(seed)
    a = (torch.randn(T, H, generator=g) * act_std).to(torch.bfloat16)
    b = (torch.randn(E, 2 * I, H, generator=g) * w_std).to(torch.bfloat16)
    b1 = (torch.randn(E, H, I, generator=g) * w_std).to(torch.bfloat16)
    scores = torch.randn(T, E, generator=g)
    m_indices = torch.topk(scores, k, dim=1).indices.to(torch.int32)
    return a, b, b1, scores, m_indices


def golden(name: str):
    return np.load(os.path.join(GOLDEN, name))


def bf16_from_bits(arr: np.ndarray) -> torch.Tensor:
    return torch.from_numpy(np.ascontiguousarray(arr).view(np.int16)).view(torch.bfloat16)


def fp8_from_bits(arr: np.ndarray) -> torch.Tensor:
    return torch.from_numpy(np.ascontiguousarray(arr)).view(torch.float8_e4m3fn)


def bits(t: torch.Tensor) -> np.ndarray:
    t = t.detach().cpu().contiguous()
    if t.dtype == torch.bfloat16:
        return t.view(torch.int16).numpy().view(np.uint16)
    if t.dtype == torch.float8_e4m3fn:
        return t.view(torch.uint8).numpy()
    return t.numpy()


def _drv(result):
    err, rest = result[0], result[1:]
    assert int(err) == 0, err
    return rest[0] if len(rest) == 1 else rest


def _captured(fn):
    """(graph, [(node, kernel name)]) of what fn() launches on the current stream; nothing is executed."""
    from cuda.bindings import driver as drv
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        _drv(drv.cuStreamBeginCapture(stream.cuda_stream, drv.CUstreamCaptureMode.CU_STREAM_CAPTURE_MODE_RELAXED))
        try:
            fn()
        finally:
            graph = _drv(drv.cuStreamEndCapture(stream.cuda_stream))
    count = _drv(drv.cuGraphGetNodes(graph))[1]
    kernels = []
    for node in _drv(drv.cuGraphGetNodes(graph, count))[0]:
        if _drv(drv.cuGraphNodeGetType(node)) == drv.CUgraphNodeType.CU_GRAPH_NODE_TYPE_KERNEL:
            par = _drv(drv.cuGraphKernelNodeGetParams(node))
            name = _drv(drv.cuFuncGetName(par.func)) if int(par.func) else _drv(drv.cuKernelGetName(par.kern))
            kernels.append((node, name.decode()))
    return graph, kernels


def kernels_of(fn):
    """Mangled names of the CUDA kernels that fn() launches on the current stream, by capturing them; nothing is executed."""
    from cuda.bindings import driver as drv
    graph, kernels = _captured(fn)
    _drv(drv.cuGraphDestroy(graph))
    return [name for _, name in kernels]


def run_kernels(fn, keep):
    """Executes those of fn()'s kernels whose name keep() accepts, and nothing else of fn()."""
    from cuda.bindings import driver as drv
    graph, kernels = _captured(fn)
    for node, name in kernels:
        if not keep(name):
            _drv(drv.cuGraphDestroyNode(node))
    runnable = _drv(drv.cuGraphInstantiate(graph, 0))
    _drv(drv.cuGraphLaunch(runnable, torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    _drv(drv.cuGraphExecDestroy(runnable))
    _drv(drv.cuGraphDestroy(graph))


def tile_form(kernel_name):
    """"pairs", "wide" or "narrow" for a grouped GEMM of gemm_sm100.cu, by the template arguments in its mangled name <fp8, mode,
    gated, pair, rows per weight box, element>; None for any other kernel."""
    m = re.search(r"GemmUniversal_tcgen05ILb\dELi\dELb\dELb(\d)ELi(\d+)ELi\dE", kernel_name)
    if m is None:
        return None
    return "pairs" if m.group(1) == "1" else {"128": "wide", "64": "narrow"}[m.group(2)]


def tile_forms(fn):
    """Tile forms of the grouped GEMMs that fn() launches, in order."""
    return [f for f in map(tile_form, kernels_of(fn)) if f is not None]
