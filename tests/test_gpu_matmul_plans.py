"""GPU parity of the matmul's plans at their edges: shares of K, token blocks, ragged columns, scratch that holds no partial sums.

Tolerance: operands are rounded to fp16 (half an ulp, 2^-11, each: at most 2^-10 of a product), sums are fp32: 1e-3 rel-L2 as in
test_gpu_qmatmul.py; Q4_K rounds its scale and its minimum as well: 2.5e-3."""
import numpy as np
import pytest

from cut_b200 import _lib as L
from cut_b200 import ops, synth
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _asked(fmt, M, K, N, act, variant=L.VARIANT_AUTO):
    """(scratch that the query asks for, the choice of a caller without scratch)"""
    import torch

    t = torch.float16 if act == np.float16 else torch.float32
    W = torch.empty(N * synth.row_bytes(fmt, K), dtype=torch.uint8, device="cuda")
    d, _, keep = ops.make_desc(torch.empty((M, K), dtype=t, device="cuda"), W, fmt, N, variant=variant)
    return ops.workspace_bytes(d), ops.select_variant(d)


def _tol(fmt):
    return 2.5e-3 if fmt == synth.Q4_K else 1e-3


def _run(fmt, A, W, N, workspace=None, ran=None, **kw):
    """workspace: its bytes (None: what the query asks for); ran: the variant that has to be the one that runs."""
    import torch

    from gpu_util import dev

    D = dev(kw.pop("D")) if "D" in kw else None
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    a, w = dev(A), dev(W)
    d, out, keep = ops.make_desc(a, w, fmt, N, D=D, status=status, **kw)
    need = ops.workspace_bytes(d) if workspace is None else workspace
    ws = torch.full((max(need, 16),), 0xFF, dtype=torch.uint8, device="cuda")  # (NaNs: nothing may be read before it is written)
    d.workspace, d.workspace_bytes = ws.data_ptr(), need
    assert ran is None or ops.select_variant(d) == ran
    ops.launch(d)
    ops.launch(d)
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    return out.cpu().numpy()


@pytest.mark.parametrize("fmt", [synth.Q8_0, synth.Q4_0, synth.Q4_K])
@pytest.mark.parametrize("M,K,N,act,op", [(129, 2048, 390, np.float16, None), (333, 2816, 256, np.float32, 0), (512, 2048, 130, np.float16, 2),
                                          (257, 4096, 384, np.float32, None), (520, 768, 129, np.float16, 0), (200, 6144, 3000, np.float16, None)])
def test_shares_of_k(fmt, M, K, N, act, op):
    from gpu_util import rel_l2

    W, A = synth.make_weights(fmt, N, K, M), synth.make_activations(M, K, 7, act)
    fuse = {} if op is None else {"fusion_type": L.FUSION_BINARY, "fusion_op": op, "D": np.random.default_rng(3).standard_normal((M, N)).astype(np.float32)}
    ref = O.qmatmul_blocks(fmt, A.astype(np.float32), W, M, K, N, **fuse)
    cast = (M * K * 2 + 15) // 16 * 16 if act == np.float32 else 0
    assert _asked(fmt, M, K, N, act)[0] >= cast + 2 * M * N * 4  # (two shares at least)
    for workspace in (None, cast):  # with and without room for partial sums
        assert rel_l2(_run(fmt, A, W, N, workspace, **fuse), ref) <= _tol(fmt), workspace


@pytest.mark.parametrize("fmt", [synth.Q8_0, synth.Q4_0, synth.Q4_K])
@pytest.mark.parametrize("M,K,N,act,op", [(9, 256, 1, np.float32, None), (16, 4096, 8600, np.float16, 0), (17, 8192, 2178, np.float16, None),
                                          (32, 1024, 20000, np.float16, 2), (13, 512, 130, np.float16, None), (24, 4096, 4098, np.float32, 0)])
def test_rows_as_fp16_mmas(fmt, M, K, N, act, op):
    """9 to 32 rows: whole tiles and shares of tiles, ragged columns, the general path where the scratch is too small.  Up to 16 rows
    weights are exact (fp32 sums of 24-bit products): 1e-5 with fp16 activations."""
    from gpu_util import rel_l2

    W, A = synth.make_weights(fmt, N, K, M), synth.make_activations(M, K, 7, act)
    fuse = {} if op is None else {"fusion_type": L.FUSION_BINARY, "fusion_op": op, "D": np.random.default_rng(3).standard_normal((M, N)).astype(np.float32)}
    ref = O.qmatmul_blocks(fmt, A.astype(np.float32), W, M, K, N, **fuse)
    exact = act == np.float16 and M <= 16 and fmt != synth.Q4_K
    got = _run(fmt, A, W, N, None, **fuse)
    assert rel_l2(got, ref) <= (1e-5 if exact else _tol(fmt))
    need, former = _asked(fmt, M, K, N, act)
    least = _asked(fmt, M, K, N, act, L.VARIANT_ROWS_MMA)[0]
    named = _run(fmt, A, W, N, least, variant=L.VARIANT_ROWS_MMA, ran=L.VARIANT_ROWS_MMA, **fuse)
    assert rel_l2(named, ref) <= (1e-5 if exact else _tol(fmt))
    # scratch that holds what the former kernel needs and not what this one does
    kept = min(_asked(fmt, M, K, N, act, former)[0], least - 16)
    assert former != L.VARIANT_ROWS_MMA
    assert rel_l2(_run(fmt, A, W, N, kept, ran=former, **fuse), ref) <= _tol(fmt)


@pytest.mark.parametrize("M", [24, 100, 300])
def test_status_of_activations_beyond_fp16(M):
    """A finite fp32 activation that rounds to infinity is reported, also beside an infinity in the same sixteen bytes; an infinity or a
    NaN of the caller's own is not."""
    import torch

    K, N = 1024, 256
    W = torch.from_numpy(synth.make_weights(synth.Q8_0, N, K, 1)).cuda()
    inf, nan = float("inf"), float("nan")
    for odd, want in (((inf, 7e4), L.ERR_RANGE), ((-7e4, nan), L.ERR_RANGE), ((inf, 1.0), 0), ((nan, -inf), 0), ((65504.0, 1.0), 0)):
        A = torch.ones((M, K), device="cuda")
        A[M - 1, 517], A[M - 1, 518] = odd
        status = torch.zeros(1, dtype=torch.int32, device="cuda")
        d, out, keep = ops.make_desc(A, W, synth.Q8_0, N, status=status)
        ws = torch.empty(max(ops.workspace_bytes(d), 16), dtype=torch.uint8, device="cuda")
        d.workspace, d.workspace_bytes = ws.data_ptr(), ws.numel()
        ops.launch(d)
        assert int(status.item()) == want, odd
        assert bool(out[: M - 1].isfinite().all())
