"""The tensor-core GEMM of up to 64 rows (qgemm_few.cu) at the edges of its tiles, units and shares, against the checker's dequantised weights
in 64 bits.

Tolerances: a Q8_0 or Q4_0 weight is rounded once, by 2^-11 of itself at most, an fp32 activation as well: 5e-4 and 1e-3 of the norm.
Q4_K rounds scale and minimum too, whose terms are up to twice the weight: 2e-3."""
import numpy as np
import pytest

from cut_b200 import _lib as L
from cut_b200 import synth
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _run(fmt, A, W, N, *, variant=L.VARIANT_GEMM_TC, scratch=None, stride=0, glu=False, kernel="qgemm_few_kernel"):
    """scratch: its bytes (None: what the query asks for); kernel: the one that has to run."""
    import torch

    from cut_b200 import ops

    M, K = A.shape
    wide = torch.zeros(M, K + 8 + stride, dtype=torch.float16 if A.dtype == np.float16 else torch.float32, device="cuda")
    a = wide[:, :K]
    a.copy_(torch.from_numpy(A))
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    fuse = {"fusion_type": 1, "fusion_op": 133, "flags": L.FLAG_GLU_PAIRS} if glu else {}
    d, out, keep = ops.make_desc(a, torch.from_numpy(W).cuda(), fmt, N, status=status, variant=variant, **fuse)
    if glu:
        out = torch.full((M, N // 2), float("nan"), device="cuda")
        d.C, d.ldc = out.data_ptr(), N // 2
    need = ops.workspace_bytes(d) if scratch is None else scratch
    ws = torch.full((need + 4096,), 0xFF, dtype=torch.uint8, device="cuda")  # (NaNs: nothing may be read before it is written)
    ws[need:] = 0xA5
    d.workspace, d.workspace_bytes = ws.data_ptr(), need
    ops.launch(d)
    first = out.cpu().numpy().copy()
    ops.launch(d)
    torch.cuda.synchronize()
    assert int(status.item()) == 0 and np.array_equal(first, out.cpu().numpy(), equal_nan=True)
    from gpu_util import kernels_of

    names = kernels_of(lambda: ops.launch(d))
    assert any(kernel in n for n in names), names
    assert bool((ws[need:] == 0xA5).all())  # nothing behind the scratch was written
    return first.astype(np.float64)


def _shares(M, K, N):
    """Rows that are read in place ask for scratch where several blocks share a tile."""
    import torch

    tiles, nk = -(-N // 128), K // 256
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    per = -(-tiles * nk // min(tiles * nk, sms))
    whole = -(-per // nk) * nk
    return (whole if whole <= per + 6 else per) % nk != 0


@pytest.mark.parametrize("fmt", [synth.Q8_0, synth.Q4_0, synth.Q4_K])
@pytest.mark.parametrize("M,K,N,act", [(1, 256, 1, np.float16), (17, 512, 130, np.float16), (32, 4096, 8600, np.float16), (33, 2048, 2178, np.float16),
                                       (64, 14336, 390, np.float16), (57, 1024, 20000, np.float16), (24, 2816, 1250, np.float32),
                                       (40, 768, 4098, np.float32), (64, 256, 38000, np.float32)])
def test_tiles_units_and_shares(fmt, M, K, N, act):
    """One unit to a CTA and many, tiles that are shared by two CTAs, by many and by none, ragged rows of both operands; activations read
    in place and staged; a scratch too small for it."""
    W, A = synth.make_weights(fmt, N, K, M), synth.make_activations(M, K, 7, act)
    want = A.astype(np.float64) @ O.dequant_rows(fmt, W, N, K).astype(np.float64).T
    tol = 2e-3 if fmt == synth.Q4_K else (1e-3 if act == np.float32 else 5e-4)
    err = lambda got: float(np.linalg.norm(got - want) / np.linalg.norm(want))
    assert err(_run(fmt, A, W, N)) <= tol
    if act == np.float16:
        shared = K > 256 and _shares(M, K, N)
        assert err(_run(fmt, A, W, N, scratch=0, kernel="qgemm_skinny_kernel" if shared else "qgemm_few_kernel")) <= tol
        if 17 <= M <= 32:  # rows that do not start on 16 bytes
            assert err(_run(fmt, A, W, N, variant=L.VARIANT_ROWS_MMA, stride=1)) <= tol
    else:  # room for the rows as fp16 and for nothing else
        assert err(_run(fmt, A, W, N, scratch=(M * K * 2 + 15) // 16 * 16, kernel="qgemm_skinny_kernel")) <= tol


@pytest.mark.parametrize("M,K,N", [(20, 4096, 2816), (64, 256, 38000), (48, 1024, 258)])
def test_paired_rows(M, K, N):
    W, A = synth.make_weights(synth.Q4_0, N, K, M), synth.make_activations(M, K, 7, np.float16)
    both = A.astype(np.float64) @ O.dequant_rows(synth.Q4_0, W, N, K).astype(np.float64).T
    gate, up = both[:, 0::2], both[:, 1::2]
    want = gate / (1 + np.exp(-gate)) * up
    got = _run(synth.Q4_0, A, W, N, glu=True)
    # (both factors carry the weights' rounding, silu's slope is at most 1.1)
    assert np.linalg.norm(got - want) <= 2.1 * 5e-4 * np.linalg.norm(np.abs(gate * up)) + 1e-6


@pytest.mark.parametrize("fmt", [synth.Q8_0, synth.Q4_0, synth.Q4_K])
@pytest.mark.parametrize("M,K,N", [(18, 512, 700), (61, 2048, 2178)])
def test_what_is_not_finite_stays_in_its_row(fmt, M, K, N):
    """An infinity, a NaN, fp16 subnormals and zeros beside ordinary rows."""
    W, A = synth.make_weights(fmt, N, K, M), synth.make_activations(M, K, 7, np.float16)
    A[3, 100], A[M - 1, K - 1], A[5] = np.inf, np.nan, 0
    A[6] = (np.arange(K) % 64 - 31).astype(np.float16) * np.float16(6e-8)
    with np.errstate(invalid="ignore"):
        prod = A.astype(np.float64) @ O.dequant_rows(fmt, W, N, K).astype(np.float64).T
    got = _run(fmt, A, W, N)
    assert not np.isfinite(got[3]).any() and np.isnan(got[M - 1]).all() and (got[5] == 0).all()
    tol = 2e-3 if fmt == synth.Q4_K else 5e-4
    for rows in ([6], [m for m in range(M - 1) if m not in (3, 5, 6)]):
        assert np.linalg.norm(got[rows] - prod[rows]) <= tol * np.linalg.norm(prod[rows])
