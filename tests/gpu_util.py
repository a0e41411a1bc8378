"""Shared helpers of the GPU parity tests (torch = device memory only)."""
from __future__ import annotations

import ctypes

import numpy as np
import torch

from cut_b200 import _lib as L
from cut_b200 import ops


def dev(a: np.ndarray) -> torch.Tensor:
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def rel_l2(got: np.ndarray, ref: np.ndarray) -> float:
    got = got.astype(np.float64)
    ref = ref.astype(np.float64)
    return float(np.linalg.norm(got - ref) / max(np.linalg.norm(ref), 1e-30))


def run_blocks(fmt, A_np, W_np, N, *, variant=L.VARIANT_AUTO, D_np=None, fusion_type=0, fusion_op=0, with_status=True, flags=0):
    """C-ABI quantized matmul over GGUF blocks on numpy inputs; returns (C, variant used, status word)."""
    A = dev(A_np)
    W = dev(W_np)
    D = dev(D_np) if D_np is not None else None
    status = torch.zeros(1, dtype=torch.int32, device="cuda") if with_status else None
    d, C_out, keep = ops.make_desc(A, W, fmt, N, D=D, fusion_type=fusion_type, fusion_op=fusion_op, variant=variant,
                                   status=status, flags=flags)
    used = ops.select_variant(d)
    need = ops.workspace_bytes(d)
    ws = None
    if need:
        ws = torch.empty(need, dtype=torch.uint8, device="cuda")
        d.workspace, d.workspace_bytes = ws.data_ptr(), need
    ops.launch(d)
    torch.cuda.synchronize()
    st = int(status.item()) if with_status else 0
    return C_out.cpu().numpy(), used, st


class _KernelNode(ctypes.Structure):  # CUDA_KERNEL_NODE_PARAMS
    _fields_ = [("func", ctypes.c_void_p), ("grid", ctypes.c_uint * 3), ("block", ctypes.c_uint * 3), ("shared", ctypes.c_uint),
                ("params", ctypes.c_void_p), ("extra", ctypes.c_void_p), ("kern", ctypes.c_void_p), ("ctx", ctypes.c_void_p)]


def kernels_of(run) -> list[str]:
    """(Mangled) names of the kernels that `run` launches, from a recording of it that is not executed."""
    cu = ctypes.CDLL("libcuda.so.1")

    def ok(rc):
        assert rc == 0, rc

    recording = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(recording):
        run()
    graph, n = ctypes.c_void_p(recording.raw_cuda_graph()), ctypes.c_size_t(0)
    ok(cu.cuGraphGetNodes(graph, None, ctypes.byref(n)))
    nodes = (ctypes.c_void_p * n.value)()
    ok(cu.cuGraphGetNodes(graph, nodes, ctypes.byref(n)))
    names = []
    for node in nodes:
        kind, p, name = ctypes.c_int(-1), _KernelNode(), ctypes.c_char_p()
        ok(cu.cuGraphNodeGetType(ctypes.c_void_p(node), ctypes.byref(kind)))
        if kind.value != 0:  # not a kernel
            continue
        ok(cu.cuGraphKernelNodeGetParams_v2(ctypes.c_void_p(node), ctypes.byref(p)))
        ok(cu.cuKernelGetName(ctypes.byref(name), ctypes.c_void_p(p.kern)) if p.kern else cu.cuFuncGetName(ctypes.byref(name), ctypes.c_void_p(p.func)))
        names.append(name.value.decode())
    return names
