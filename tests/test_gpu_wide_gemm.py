"""The prompt GEMM by pairs of CTAs (qgemm_wide.cu) at the edges of its tiles, waves and accumulators, against the checker's dequantised weights
in 64 bits.

Tolerances: a Q8_0 or Q4_0 weight is rounded once, by 2^-11 of itself at most, an fp32 activation as well: 5e-4 and 1e-3 of the norm.
Q4_K rounds scale and minimum too, whose terms are up to twice the weight: 2e-3."""
import numpy as np
import pytest

from cut_b200 import _lib as L
from cut_b200 import synth
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _run(fmt, A, W, N, *, D=None, glu=False):
    import torch

    from cut_b200 import ops

    M, K = A.shape
    wide = torch.zeros(M, K + 8, dtype=torch.float16 if A.dtype == np.float16 else torch.float32, device="cuda")
    a = wide[:, :K]
    a.copy_(torch.from_numpy(A))
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    fuse = {"fusion_type": 1, "fusion_op": 133, "flags": L.FLAG_GLU_PAIRS} if glu else {}
    if D is not None:
        fuse = {"fusion_type": L.FUSION_BINARY, "fusion_op": 0, "D": torch.from_numpy(D).cuda()}
    d, out, keep = ops.make_desc(a, torch.from_numpy(W).cuda(), fmt, N, status=status, **fuse)
    if glu:
        out = torch.full((M, N // 2), float("nan"), device="cuda")
        d.C, d.ldc = out.data_ptr(), N // 2
    ws = torch.full((max(ops.workspace_bytes(d), 16),), 0xFF, dtype=torch.uint8, device="cuda")
    d.workspace, d.workspace_bytes = ws.data_ptr(), ws.numel()
    ops.launch(d)
    first = out.cpu().numpy().copy()
    ops.launch(d)
    torch.cuda.synchronize()
    assert int(status.item()) == 0 and np.array_equal(first, out.cpu().numpy(), equal_nan=True)
    from gpu_util import kernels_of

    names = kernels_of(lambda: ops.launch(d))
    assert any("qgemm_wide_kernel" in n for n in names), names
    return first.astype(np.float64)


@pytest.mark.parametrize("fmt", [synth.Q8_0, synth.Q4_0, synth.Q4_K])
@pytest.mark.parametrize("M,K,N,act,add", [(65, 256, 19300, np.float16, False), (100, 768, 19968, np.float16, True), (129, 512, 9000, np.float16, False),
                                           (250, 1024, 6145, np.float32, False), (300, 256, 20001, np.float16, False), (512, 2048, 3000, np.float16, True),
                                           (1500, 512, 2049, np.float16, False)])
def test_tiles_and_waves(fmt, M, K, N, act, add):
    """One unit of K to a tile and many, one tile to a pair and several, one accumulator and two, ragged rows of both operands."""
    W, A = synth.make_weights(fmt, N, K, M), synth.make_activations(M, K, 7, act)
    D = np.random.default_rng(3).standard_normal((M, N)).astype(np.float32) if add else None
    prod = A.astype(np.float64) @ O.dequant_rows(fmt, W, N, K).astype(np.float64).T
    got = _run(fmt, A, W, N, D=D) - (0 if D is None else D)
    tol = 2e-3 if fmt == synth.Q4_K else (1e-3 if act == np.float32 else 5e-4)
    assert np.linalg.norm(got - prod) <= tol * np.linalg.norm(prod)


@pytest.mark.parametrize("M,K,N", [(90, 512, 20000), (300, 1024, 5634)])
def test_paired_rows(M, K, N):
    W, A = synth.make_weights(synth.Q4_0, N, K, M), synth.make_activations(M, K, 7, np.float16)
    both = A.astype(np.float64) @ O.dequant_rows(synth.Q4_0, W, N, K).astype(np.float64).T
    gate, up = both[:, 0::2], both[:, 1::2]
    want = gate / (1 + np.exp(-gate)) * up
    got = _run(synth.Q4_0, A, W, N, glu=True)
    # (both factors carry the weights' rounding, silu's slope is at most 1.1)
    assert np.linalg.norm(got - want) <= 2.1 * 5e-4 * np.linalg.norm(np.abs(gate * up)) + 1e-6


@pytest.mark.parametrize("fmt", [synth.Q8_0, synth.Q4_0, synth.Q4_K])
@pytest.mark.parametrize("M,K,N", [(70, 512, 20000), (290, 1024, 6000)])
def test_what_is_not_finite_stays_in_its_row(fmt, M, K, N):
    """An infinity, a NaN, fp16 subnormals and zeros beside ordinary rows, in the last rows of a tile among them."""
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
