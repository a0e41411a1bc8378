"""Tiles of the dense bf16 GEMM at their edges: widths of 64 to 256, single CTAs and pairs, ragged rows, columns and k.

bf16 operands are exact; fp32 sums of at most 2100 products: 1e-5; a bf16 result: 2^-9 at most, 2.5e-3."""
import ctypes

import pytest

from cut_b200 import _lib as L
from cut_b200 import ops

pytestmark = pytest.mark.gpu


def _rel(got, ref):
    return float((got.double() - ref).norm() / ref.norm())


@pytest.mark.parametrize("M,K,N,bf16,unary", [(129, 1024, 20000, True, 0), (256, 2048, 16600, False, 0), (257, 1024, 9001, True, 133), (1000, 2056, 5136, False, L.UNARY_RELU_SQUARE),
                                             (2048, 1024, 6144, True, 0), (2100, 136, 4104, False, 133), (511, 1200, 14337, True, 0), (3000, 64, 1000, False, 0)])
def test_dense_widths(M, K, N, bf16, unary):
    import torch

    g = torch.Generator(device="cuda").manual_seed(M + N)
    A = torch.randn((M, K), device="cuda", generator=g).bfloat16()
    W = torch.randn((N, K), device="cuda", generator=g).mul_(K ** -0.5).bfloat16()
    bias = torch.randn(N, device="cuda", generator=g)
    ld = (N + 7) // 8 * 8
    out = torch.full((M, ld), float("nan"), device="cuda", dtype=torch.bfloat16 if bf16 else torch.float32)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    d = ops.dense_desc(A, W, K, out, bias=bias, unary=unary, variant=L.DENSE_TC, status=status, N=N)
    ops.dense_matmul(d)
    ref = A.double() @ W.double().T + bias.double()
    ref = torch.nn.functional.silu(ref) if unary == 133 else ref.clamp(min=0).square() if unary else ref
    assert int(status.item()) == 0
    assert _rel(out[:, :N], ref) <= (2.5e-3 if bf16 else 1e-5)
    assert bool(out[:, N:].isnan().all())  # nothing past the last column


@pytest.mark.parametrize("counts,K,N,glu", [((700, 0, 1, 255, 256, 257, 31, 500), 1024, 2048, 0), ((3, 900, 130), 2056, 4128, 1), ((2048, 2048), 512, 4096, 0)])
def test_grouped_widths(counts, K, N, glu):
    import torch

    g = torch.Generator(device="cuda").manual_seed(K + N)
    E, R = len(counts), sum(counts)
    A = torch.randn((R, K), device="cuda", generator=g).bfloat16()
    W = torch.randn((E * N, K), device="cuda", generator=g).mul_(K ** -0.5).bfloat16()
    ends = torch.tensor((0,) + counts, device="cuda").cumsum(0)
    out = torch.full((R, N // 2 if glu else N), float("nan"), device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    d = ops.moe_matmul_desc(A, W, K, ends.int(), E, R, 1, out, glu=L.GLU_CLAMPED if glu else L.GLU_NONE, alpha=1.702, beta=1.0, limit=7.0,
                            variant=L.DENSE_TC, status=status)
    L.check(L.lib().cutb_moe_matmul(ctypes.byref(d), torch.cuda.current_stream().cuda_stream))
    ref = torch.cat([A[ends[e]: ends[e + 1]].double() @ W[e * N: (e + 1) * N].double().T for e in range(E)])
    if glu:
        a, u = ref[:, 0::2].clamp(max=7.0), ref[:, 1::2].clamp(-7.0, 7.0)
        ref = a * torch.sigmoid(1.702 * a) * (u + 1.0)
    assert int(status.item()) == 0
    assert _rel(out, ref) <= 1e-5


def _launched(run, tmp_path):
    """(kernel name, number of blocks) of the GEMM that `run` launches"""
    import json

    import torch
    from torch.profiler import ProfilerActivity, profile

    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        run()
        torch.cuda.synchronize()
    path = str(tmp_path / "trace.json")
    prof.export_chrome_trace(path)
    with open(path) as f:
        events = [e for e in json.load(f)["traceEvents"] if e.get("cat") == "kernel" and "dense_gemm_tc_kernel" in e["name"]]
    assert len(events) == 1
    return events[0]["name"], events[0]["args"]["grid"][0]


@pytest.mark.parametrize("M,K,N,width,pair", [(100, 256, 9000, 64, False), (100, 256, 12288, 128, False), (100, 256, 20000, 192, False),
                                              (100, 256, 30000, 208, False), (100, 256, 32000, 224, False), (100, 256, 34000, 240, False),
                                              (100, 256, 37000, 256, False), (256, 4608, 9000, 128, True), (256, 4608, 11500, 160, True),
                                              (200, 4608, 14000, 192, True), (129, 4608, 16500, 224, True), (256, 4608, 18900, 256, True)])
def test_every_width_and_pair_is_reached(M, K, N, width, pair, tmp_path):
    """Shapes whose tiles fill one wave just so: which tile runs is read from the launch.  bf16 results: 2^-9, 2.5e-3."""
    import torch

    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the shapes are chosen for 148 multiprocessors")
    g = torch.Generator(device="cuda").manual_seed(N)
    A = torch.randn((M, K), device="cuda", generator=g).bfloat16()
    W = torch.randn((N, K), device="cuda", generator=g).mul_(K ** -0.5).bfloat16()
    out = torch.full((M, N), float("nan"), device="cuda", dtype=torch.bfloat16)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    d = ops.dense_desc(A, W, K, out, variant=L.DENSE_TC, status=status, N=N)
    name, blocks = _launched(lambda: ops.dense_matmul(d), tmp_path)
    assert ("<false, true" in name or "<(bool)0, (bool)1" in name) == pair, name
    assert blocks == -(-M // (256 if pair else 128)) * -(-N // width) * (2 if pair else 1)
    assert int(status.item()) == 0
    assert _rel(out, A.double() @ W.double().T) <= 2.5e-3


@pytest.mark.parametrize("E,T,top,K,N,pair", [(16, 200, 4, 4096, 4096, False), (8, 700, 2, 1024, 2048, False), (16, 64, 4, 1024, 3072, False),
                                              (8, 2000, 4, 2560, 4096, True), (16, 700, 4, 4096, 4096, True)])
def test_pairs_only_where_experts_fill_them(E, T, top, K, N, pair, tmp_path):
    """Evenly used experts: pairs of CTAs (256 rows) from some 170 rows per expert on wide weights; with fewer they would copy and multiply
    for rows that are not there."""
    import torch

    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the shapes are chosen for 148 multiprocessors")
    R = T * top
    g = torch.Generator(device="cuda").manual_seed(T)
    A = torch.randn((R, K), device="cuda", generator=g).bfloat16()
    W = torch.randn((E * N, K), device="cuda", generator=g).mul_(K ** -0.5).bfloat16()
    ends = (torch.arange(E + 1, device="cuda") * R // E).int()
    out = torch.empty((R, N), device="cuda", dtype=torch.bfloat16)
    d = ops.moe_matmul_desc(A, W, K, ends, E, R, 1, out, variant=L.DENSE_TC)
    name, _ = _launched(lambda: L.check(L.lib().cutb_moe_matmul(ctypes.byref(d), torch.cuda.current_stream().cuda_stream)), tmp_path)
    assert ("<true, true" in name or "<(bool)1, (bool)1" in name) == pair, name
    e = E // 2
    rows = slice(int(ends[e]), int(ends[e + 1]))
    assert _rel(out[rows], A[rows].double() @ W[e * N: (e + 1) * N].double().T) <= 2.5e-3
