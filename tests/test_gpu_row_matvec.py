"""The mat-vecs of one row and of two fp16 rows (qgemv_row.cu), and of three to eight fp16 rows (qgemv_few.cu), at the edges of their tiles,
stages, groups and loads, against the checker's dequantised weights in 64 bits.

Tolerances: a 16-bit level leaves an error of at most max|x of a block| / 65024 per element, uniform, so relative to a block of normal
values (maximum about 2.5 sigma) 2.5 / 65024 / sqrt(3) = 2.2e-5 of the norm: four times that.  Two levels leave the fp32 sums: 2^-24 times
the square root of some thousand terms at worst, 2e-6."""
import re

import numpy as np
import pytest

from cut_b200 import _lib as L
from cut_b200 import synth
from oracle import oracle as O

pytestmark = pytest.mark.gpu
FMTS = [synth.Q8_0, synth.Q4_0, synth.Q4_K]
TOL = {16: 9e-5, 32: 2e-6}


def _run(fmt, A, W, N, *, shift=0, flags=0, norm=None, fusion=(0, 0), D=None):
    import torch

    from cut_b200 import ops

    M, K = A.shape
    wide = torch.zeros(M, K + 8, dtype=torch.float16 if A.dtype == np.float16 else torch.float32, device="cuda")
    a = wide[:, shift: shift + K]  # rows that start `shift` elements past an aligned address, K + 8 apart
    a.copy_(torch.from_numpy(A))
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    d, C, keep = ops.make_desc(a, torch.from_numpy(W).cuda(), fmt, N, fusion_type=fusion[0], fusion_op=fusion[1], status=status, flags=flags,
                               D=None if D is None else torch.from_numpy(D).cuda())
    if norm is not None:
        norm = torch.from_numpy(norm).cuda()
        d.flags |= L.FLAG_A_RMSNORM
        d.a_norm_weight, d.a_norm_eps = norm.data_ptr(), 1e-5
    ws = torch.empty(max(ops.workspace_bytes(d), 16), dtype=torch.uint8, device="cuda")
    d.workspace, d.workspace_bytes = ws.data_ptr(), ws.numel()
    ops.launch(d)
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    return C.cpu().numpy().astype(np.float64)


def _case(fmt, M, K, N, dtype, seed):
    W = synth.make_weights(fmt, N, K, seed)
    return synth.make_activations(M, K, seed + 1, dtype), W, O.dequant_rows(fmt, W, N, K).astype(np.float64)


def _err(got, want):
    return float(np.linalg.norm(got - want) / np.linalg.norm(want))


@pytest.mark.parametrize("fmt", FMTS)
@pytest.mark.parametrize("M,dtype,flags", [(1, np.float16, 0), (2, np.float16, 0), (1, np.float32, 0), (2, np.float32, L.FLAG_ACT_16BIT)])
@pytest.mark.parametrize("K,N", [(256, 1), (512, 17), (1280, 2400), (2048, 1500), (4096, 1201), (4352, 1300), (8192, 1250), (14336, 1216), (256, 19100)])
def test_tiles_stages_and_groups(fmt, M, dtype, flags, K, N):
    """One row to a tile, ragged tiles, stages that part of the warps share, granules beyond the last stage, more tiles than a block sums up
    at a time, K split and whole."""
    A, W, dense = _case(fmt, M, K, N, dtype, K + N + fmt)
    levels = 32 if dtype == np.float32 and not flags else 16
    assert _err(_run(fmt, A, W, N, flags=flags), A.astype(np.float64) @ dense.T) <= TOL[levels]


@pytest.mark.parametrize("fmt", FMTS)
@pytest.mark.parametrize("M,dtype,flags", [(1, np.float16, 0), (2, np.float16, 0), (1, np.float32, 0), (1, np.float32, L.FLAG_NO_OVERLAP)])
@pytest.mark.parametrize("K,N", [(3072, 4900), (3584, 2400), (768, 700), (4096, 2300), (4096, 4800), (13312, 1300), (2048, 2368), (2304, 2368)])
def test_rings_and_granules(fmt, M, dtype, flags, K, N):
    """Tiles of whole stages whose last granules are missing (a warp reads what it staged itself), of an odd number of stages (it does not),
    splits of fewer granules than a stage has, rings that hold all of a block's stages and a part of them, a launch that starts early and not;
    two rows on both sides of the line between the kernels (eight granules to a block)."""
    A, W, dense = _case(fmt, M, K, N, dtype, K + N + fmt)
    assert _err(_run(fmt, A, W, N, flags=flags), A.astype(np.float64) @ dense.T) <= TOL[32 if dtype == np.float32 else 16]


@pytest.mark.parametrize("fmt", FMTS)
@pytest.mark.parametrize("dtype,shift", [(np.float16, 1), (np.float16, 4), (np.float32, 1), (np.float32, 2)])
def test_rows_at_any_element(fmt, dtype, shift):
    K, N = 4096, 1300
    A, W, dense = _case(fmt, 1, K, N, dtype, shift + fmt)
    want = A.astype(np.float64) @ dense.T
    assert _err(_run(fmt, A, W, N, shift=shift), want) <= TOL[32 if dtype == np.float32 else 16]


@pytest.mark.parametrize("fmt", FMTS)
@pytest.mark.parametrize("K,N", [(2304, 1300), (4096, 1184), (4096, 200)])  # (the last one splits K: the squares of the whole row)
def test_rms_meets_the_sums(fmt, K, N):
    A, W, dense = _case(fmt, 1, K, N, np.float32, K + fmt)
    w = (1.0 + 0.1 * np.random.default_rng(3).normal(size=K)).astype(np.float32)
    x = A.astype(np.float64)
    want = (x / np.sqrt((x * x).mean() + 1e-5) * w) @ dense.T + 0.5
    got = _run(fmt, A, W, N, norm=w, fusion=(L.FUSION_BINARY, 0), D=np.full((1, N), 0.5, np.float32))
    assert _err(got, want) <= TOL[32]


@pytest.mark.parametrize("fmt", FMTS)
def test_values_at_the_ends_of_the_range(fmt):
    """Values so small that the inverse of a block's scale leaves the range of fp32 (as precise as subnormal scales are), one block 1e35 times
    the others, and one NaN, which every output shows."""
    K, N = 4096, 1200
    A, W, dense = _case(fmt, 1, K, N, np.float32, 9 + fmt)
    small = (A * np.float32(1e-36)).astype(np.float32)
    assert _err(_run(fmt, small, W, N), small.astype(np.float64) @ dense.T) <= 0.05  # steps of 3e-39 beside values of 1e-36: 1 %, and fp32's own
    large = A.copy()
    large[0, 32:64] *= np.float32(1e35)
    assert _err(_run(fmt, large, W, N), large.astype(np.float64) @ dense.T) <= TOL[32]
    A[0, 777] = np.nan
    assert np.isnan(_run(fmt, A, W, N)).all()


def _near_halves(rng, rows, K):
    """fp32 rows whose values lie close to halfway between two steps of their block's 16-bit scale (maximum / 32512), in blocks whose maximum
    times that scale's inverse is as far from 32512 as rounding leaves it: the residuals that the second level holds are the largest there are."""
    q = np.float32(32512)
    most = (1 + rng.random(1 << 18)).astype(np.float32)
    off = (q / most).astype(np.float64) * (most * (np.float32(1) / q)).astype(np.float64) - 1
    most = most[np.argsort(-np.abs(off))[: rows * K // 32]]
    step = (most * (np.float32(1) / q)).astype(np.float64)[:, None]
    at = rng.integers(24000, 32400, (most.size, 32)) + 0.5 + rng.uniform(-0.012, 0.012, (most.size, 32))
    x = (at * step * rng.choice([-1.0, 1.0], at.shape)).astype(np.float32)
    x[:, 0] = most
    return x.reshape(rows, K)


@pytest.mark.parametrize("fmt", FMTS)
@pytest.mark.parametrize("M,K,N", [(1, 4096, 1200), (1, 1280, 300), (2, 4096, 1200), (4, 2048, 600), (8, 1024, 600)])
def test_residuals_that_fill_the_second_level(fmt, M, K, N):
    """The second level of fp32 rows holds the residual of the first in two int8 digits, which wrap above 32639."""
    W, A = synth.make_weights(fmt, N, K, M), _near_halves(np.random.default_rng(K + M), M, K)
    want = A.astype(np.float64) @ O.dequant_rows(fmt, W, N, K).astype(np.float64).T
    got = _run(fmt, A, W, N)
    for m in range(M):
        assert _err(got[m], want[m]) <= TOL[32], m


@pytest.mark.parametrize("fmt", FMTS)
@pytest.mark.parametrize("M", [2, 4, 8])
@pytest.mark.parametrize("size,tol", [(1e-29, TOL[32]), (1e-31, TOL[16]), (1e-36, 0.05)])
def test_rows_of_small_values(fmt, M, size, tol):
    """Several fp32 rows, one of them so small that the inverse of a block's scale leaves the range of fp32: first the second level's (its steps
    are then left out: 16 bits), then the first's (steps of 3e-39 beside values of 1e-36: 1 %, and fp32's own subnormal values)."""
    K, N = 2048, 600
    A, W, dense = _case(fmt, M, K, N, np.float32, 9 + fmt)
    A[M - 1] *= np.float32(size)
    want, got = A.astype(np.float64) @ dense.T, _run(fmt, A, W, N)
    for m in range(M):
        assert _err(got[m], want[m]) <= (tol if m == M - 1 else TOL[32]), m


@pytest.mark.parametrize("fmt", [synth.Q4_0, synth.Q4_K])
@pytest.mark.parametrize("M", [3, 4, 5, 8])
@pytest.mark.parametrize("K,N", [(256, 2), (512, 1200), (1280, 2401), (2048, 9500), (4096, 200), (4096, 5000), (3072, 19100), (5120, 9600)])
def test_a_few_rows(fmt, M, K, N):
    """One tile and several per group of warps, a group without one, granules beyond the last stage, K split and whole, a longer K; rows
    that start on 16 bytes and not.  Products of fp16 and 4-bit values are exact, sums have fp32's error, some 1e-6 of the largest partial
    sum: up to sixteen times the result's where minima or offsets cancel."""
    A, W, dense = _case(fmt, M, K, N, np.float16, M + K + N + fmt)
    want = A.astype(np.float64) @ dense.T
    tol = TOL[16] if M <= 4 and K > 3072 else 2e-5  # (some of these stay with the digits)
    assert _err(_run(fmt, A, W, N), want) <= tol
    assert _err(_run(fmt, A, W, N, shift=3), want) <= tol


@pytest.mark.parametrize("fmt", [synth.Q4_0, synth.Q4_K])
@pytest.mark.parametrize("M", [3, 7])
def test_a_few_rows_in_pairs(fmt, M):
    """Gate and up rows side by side, the last tile of the matrix a part of one; a tiny and a large row beside ordinary ones."""
    K, N = 1024, 2 * 1189
    A, W, dense = _case(fmt, M, K, N, np.float16, M + fmt)
    A[0] = (A[0].astype(np.float32) * 1e-3).astype(np.float16)
    A[1] = (A[1].astype(np.float32) * 1e3).astype(np.float16)
    import torch

    from cut_b200 import ops

    out = torch.zeros(M, N // 2, device="cuda")
    d, _, keep = ops.make_desc(torch.from_numpy(A).cuda(), torch.from_numpy(W).cuda(), fmt, N, C_out=out, fusion_type=L.FUSION_UNARY, fusion_op=130,
                               flags=L.FLAG_GLU_PAIRS)
    ws = torch.empty(max(ops.workspace_bytes(d), 16), dtype=torch.uint8, device="cuda")
    d.workspace, d.workspace_bytes = ws.data_ptr(), ws.numel()
    ops.launch(d)
    torch.cuda.synchronize()
    y = A.astype(np.float64) @ dense.T
    want, got = np.maximum(y[:, 0::2], 0.0) * y[:, 1::2], out.cpu().numpy().astype(np.float64)
    for m in range(M):
        assert _err(got[m], want[m]) <= 4e-5, m


@pytest.mark.parametrize("fmt", [synth.Q4_0, synth.Q4_K])
@pytest.mark.parametrize("M,shift", [(3, 0), (5, 0), (7, 0), (8, 0), (3, 1), (8, 2)])
def test_what_is_not_finite_stays_in_its_row(fmt, M, shift):
    """An infinity, a NaN and fp16 subnormals (6e-8 to 2e-6) beside an ordinary row and the idle columns of an odd number of rows."""
    K, N = 1280, 2401
    A, W, dense = _case(fmt, M, K, N, np.float16, M + fmt)
    A[0, 700], A[M - 1, K - 1] = np.inf, np.nan
    small = (np.arange(K) % 64 - 31).astype(np.float16) * np.float16(6e-8)
    if M > 3:
        A[2] = small
    with np.errstate(invalid="ignore"):
        want = A.astype(np.float64) @ dense.T
    got = _run(fmt, A, W, N, shift=shift)
    assert not np.isfinite(got[0]).any() and np.isnan(got[M - 1]).all()
    for m in range(1, M - 1):
        assert _err(got[m], want[m]) <= 2e-5, m
    A[0] = 0
    assert (_run(fmt, A, W, N, shift=shift)[0] == 0).all()


@pytest.mark.parametrize("fmt,M,dtype,flags,K,N,kernel", [
    (synth.Q8_0, 1, np.float16, 0, 4096, 4096, "qgemv_row_kernel"), (synth.Q4_K, 1, np.float32, 0, 14336, 4096, "qgemv_row_kernel"),
    (synth.Q4_0, 1, np.float32, L.FLAG_ACT_16BIT, 512, 500, "qgemv_row_kernel"), (synth.Q4_0, 2, np.float16, 0, 2304, 2368, "qgemv_row_kernel"),
    (synth.Q4_0, 2, np.float16, 0, 2048, 2368, "qgemv_blocks_kernel"), (synth.Q8_0, 2, np.float32, L.FLAG_ACT_16BIT, 4096, 500, "qgemv_blocks_kernel"),
    (synth.Q8_0, 2, np.float32, L.FLAG_ACT_16BIT, 512, 4096, "qgemv_row_kernel"), (synth.Q4_K, 2, np.float32, 0, 4096, 4096, "qgemv_blocks_kernel"),
    (synth.Q4_0, 3, np.float16, 0, 4096, 11008, "qgemv_few_kernel"), (synth.Q8_0, 3, np.float16, 0, 4096, 11008, "qgemv_blocks_kernel"),
    (synth.Q4_K, 4, np.float16, 0, 3072, 11008, "qgemv_few_kernel"), (synth.Q4_0, 4, np.float16, 0, 4096, 5000, "qgemv_few_kernel"),
    (synth.Q4_0, 4, np.float16, 0, 4096, 2368, "qgemv_blocks_kernel"), (synth.Q4_0, 4, np.float16, 0, 4096, 14336, "qgemv_blocks_kernel"),
    (synth.Q4_K, 5, np.float16, 0, 5120, 9600, "qgemv_few_kernel"), (synth.Q4_K, 6, np.float16, 0, 5120, 5000, "qgemv_blocks_kernel"),
    (synth.Q4_0, 8, np.float16, 0, 4096, 200, "qgemv_few_kernel"), (synth.Q4_0, 4, np.float16, 0, 8192, 5000, "qgemv_blocks_kernel")])
def test_the_kernel_that_runs(fmt, M, dtype, flags, K, N, kernel):
    """Both sides of the lines between the mat-vecs: the launched kernel, by its name."""
    import torch

    from cut_b200 import ops
    from gpu_util import kernels_of

    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the lines are drawn for 148 multiprocessors")
    A = torch.zeros((M, K), dtype=torch.float16 if dtype == np.float16 else torch.float32, device="cuda")
    d, out, keep = ops.make_desc(A, torch.zeros(N * synth.row_bytes(fmt, K), dtype=torch.uint8, device="cuda"), fmt, N, flags=flags)
    ws = torch.empty(max(ops.workspace_bytes(d), 16), dtype=torch.uint8, device="cuda")
    d.workspace, d.workspace_bytes = ws.data_ptr(), ws.numel()
    ops.launch(d)
    names = kernels_of(lambda: ops.launch(d))
    assert re.findall(r"\d(qgemv_[a-z]+_kernel)", " ".join(names)) == [kernel], names


@pytest.mark.parametrize("fmt,M,dtype,K,N", [(synth.Q4_0, 1, np.float16, 4096, 2401), (synth.Q8_0, 1, np.float32, 2304, 1200), (synth.Q4_K, 2, np.float16, 4096, 2500),
                                             (synth.Q4_0, 3, np.float16, 4096, 1300), (synth.Q4_K, 8, np.float16, 1024, 2401), (synth.Q4_0, 5, np.float16, 4096, 300)])
def test_scatter_into_two_outputs(fmt, M, dtype, K, N):
    """The epilogue that stores its slice into every rank's output, with two buffers of this GPU as the ranks' (the exchange between ranks is not
    launched): the plain launch's bits, and nothing beside the slice."""
    import ctypes as C

    import torch

    from cut_b200 import ops

    A, W, _ = _case(fmt, M, K, N, dtype, M + K)
    a, w, at, total = torch.from_numpy(A).cuda(), torch.from_numpy(W).cuda(), 37, N + 100
    d, plain, keep = ops.make_desc(a, w, fmt, N, variant=L.VARIANT_GEMV_MMA)
    ws = torch.empty(max(ops.workspace_bytes(d), 16), dtype=torch.uint8, device="cuda")
    d.workspace, d.workspace_bytes = ws.data_ptr(), ws.numel()
    ops.launch(d)
    outs, flags = torch.full((2, M, total), 5.0, device="cuda"), torch.zeros(64, dtype=torch.int64, device="cuda")
    ps = L.PeerScatter()
    ps.world, ps.rank, ps.ldc_total, ps.n_offset = 2, 0, total, at
    for r in range(2):
        ps.C_peers[r], ps.flag_peers[r] = outs[r].data_ptr(), flags.data_ptr() + 256 * r
    L.check(L.lib().cutb_qmatmul_scatter(C.byref(d), C.byref(ps), None))
    torch.cuda.synchronize()
    for o in outs:
        assert torch.equal(o[:, at: at + N], plain) and bool((o[:, :at] == 5.0).all()) and bool((o[:, at + N:] == 5.0).all())
