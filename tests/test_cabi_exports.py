"""CPU tests of the C-ABI library itself: it loads, exports every symbol the
header declares, and its argument validation answers without a GPU."""
import ctypes as C
import os
import re

import pytest

from cut_b200 import _lib as L

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _declared_symbols():
    text = open(os.path.join(ROOT, "include", "cutb.h")).read()
    return re.findall(r"CUTB_API\s+[\w\s\*]+?\b(cutb_\w+)\s*\(", text)


def test_library_exports_every_declared_symbol():
    lib = L.lib()
    names = _declared_symbols()
    assert len(names) >= 10
    assert sorted(names) == sorted(L.EXPORTS)
    for n in names:
        assert hasattr(lib, n), n
    assert lib.cutb_version() == 100


def test_descriptor_layout_matches_header():
    # field order and types of cutb_qmatmul_desc as declared in include/cutb.h
    text = open(os.path.join(ROOT, "include", "cutb.h")).read()
    body = re.search(r"typedef struct cutb_qmatmul_desc \{(.*?)\} cutb_qmatmul_desc;", text, re.S).group(1)
    body = re.sub(r"/\*.*?\*/", "", body, flags=re.S)
    fields = []
    for decl in body.split(";"):
        decl = decl.strip()
        if not decl:
            continue
        names = [n.strip().lstrip("*") for n in decl.split(",")]
        first = names[0].split()[-1].lstrip("*")
        fields += [first] + names[1:]
    assert fields == [f[0] for f in L.QMatmulDesc._fields_]
    assert C.sizeof(L.QMatmulDesc) == 168
    assert C.sizeof(L.PeerScatter) == 16 + 2 * 8 * L.MAX_PEERS


def test_validation_needs_no_device():
    lib = L.lib()
    d = L.QMatmulDesc()
    assert lib.cutb_qmatmul(C.byref(d), None) == L.ERR_INVALID
    assert b"empty shape" in lib.cutb_last_error()
    assert lib.cutb_qmatmul(None, None) == L.ERR_INVALID
    assert lib.cutb_qmatmul_select_variant(C.byref(d)) < 0
    assert lib.cutb_qmatmul_workspace_bytes(C.byref(d)) == 0
    assert lib.cutb_dequant(9, None, 0, None, 1, 32, 32, None) == L.ERR_INVALID
    assert lib.cutb_dequant(L.Q4_K, None, 0, None, 1, 100, 100, None) == L.ERR_INVALID
    assert lib.cutb_dequant(L.Q4_K, None, 0, None, 0, 0, 0, None) == L.OK  # empty tensor: nothing to do
    assert lib.cutb_transpose_q4(None, None, 3, 32, 16, 2, None) == L.ERR_INVALID
    assert b"N must be even" in lib.cutb_last_error()
    assert lib.cutb_transpose_q4(None, None, 4, 24, 12, 2, None) == L.ERR_INVALID
    assert lib.cutb_transpose_q4(None, None, 0, 0, 0, 0, None) == L.OK
    assert lib.cutb_status_string(L.ERR_TIMEOUT) == b"device-side wait timed out"
    assert lib.cutb_variant_name(L.VARIANT_GEMV_MMA) == b"QGemvBulkMma"


def test_select_variant_and_workspace_plan_without_device():
    """Variant choice and the split-K workspace size are host logic."""
    lib = L.lib()

    def desc(fmt, M, K, N, dtype=L.F16, layout=L.LAYOUT_GGUF_BLOCKS):
        d = L.QMatmulDesc()
        d.format, d.layout, d.a_dtype = fmt, layout, dtype
        d.M, d.K, d.N, d.lda, d.ldc = M, K, N, K, N
        d.A = d.W = d.C = 256  # never dereferenced here
        d.W_bytes = 1 << 40
        d.variant = L.VARIANT_AUTO
        if layout == L.LAYOUT_KN_PLANES:
            d.scales, d.ldb, d.lds = 256, N, N
        return d

    assert lib.cutb_qmatmul_select_variant(C.byref(desc(L.Q4_0, 1, 4096, 11008))) == L.VARIANT_GEMV_MMA
    assert lib.cutb_qmatmul_select_variant(C.byref(desc(L.Q4_0, 12, 4096, 11008))) == L.VARIANT_GEMV_MMA
    assert lib.cutb_qmatmul_select_variant(C.byref(desc(L.Q4_0, 16, 2048, 2048))) == L.VARIANT_GEMV_MMA
    # 13 to 16 fp16 rows on 16 M weights and more: the tensor-core GEMM for few tokens (paired rows included), unless the
    # fused RMSNorm, which only the mat-vec has, is asked for
    assert lib.cutb_qmatmul_select_variant(C.byref(desc(L.Q4_0, 16, 4096, 11008))) == L.VARIANT_GEMM_TC
    flagged = desc(L.Q4_0, 16, 4096, 11008)
    flagged.flags, flagged.fusion_type, flagged.fusion_op = L.FLAG_GLU_PAIRS, L.FUSION_UNARY, 133
    assert lib.cutb_qmatmul_select_variant(C.byref(flagged)) == L.VARIANT_GEMM_TC
    flagged.flags, flagged.a_norm_weight = L.FLAG_A_RMSNORM, 256
    assert lib.cutb_qmatmul_select_variant(C.byref(flagged)) == L.VARIANT_GEMV_MMA
    assert lib.cutb_qmatmul_select_variant(C.byref(desc(L.Q8_0, 8, 4096, 11008, L.F32))) == L.VARIANT_GEMV_MMA
    assert lib.cutb_qmatmul_select_variant(C.byref(desc(L.Q4_0, 17, 4096, 11008))) != L.VARIANT_GEMV_MMA
    assert lib.cutb_qmatmul_select_variant(C.byref(desc(L.Q8_0, 1, 4096, 4096, L.F32))) == L.VARIANT_GEMV_MMA
    assert lib.cutb_qmatmul_select_variant(C.byref(desc(L.Q8_0, 9, 4096, 4096, L.F32))) != L.VARIANT_GEMV_MMA
    assert lib.cutb_qmatmul_select_variant(C.byref(desc(L.Q4_0, 1, 96, 8))) == L.VARIANT_GENERIC
    # the reference's [K, N] planes: the coalesced mat-vec up to four rows, strides padded to 4; else the any-shape kernel
    assert lib.cutb_qmatmul_select_variant(C.byref(desc(L.Q8_0, 1, 64, 4, L.F32, L.LAYOUT_KN_PLANES))) == L.VARIANT_GEMV_PLANES
    assert lib.cutb_qmatmul_select_variant(C.byref(desc(L.Q4_0, 4, 4096, 11008, L.F32, L.LAYOUT_KN_PLANES))) == L.VARIANT_GEMV_PLANES
    assert lib.cutb_qmatmul_select_variant(C.byref(desc(L.Q8_0, 5, 64, 4, L.F32, L.LAYOUT_KN_PLANES))) == L.VARIANT_GENERIC
    assert lib.cutb_qmatmul_select_variant(C.byref(desc(L.Q8_0, 1, 64, 6, L.F32, L.LAYOUT_KN_PLANES))) == L.VARIANT_GENERIC  # ldb = 6
    assert lib.cutb_qmatmul_workspace_bytes(C.byref(desc(L.Q8_0, 1, 4096, 4096, L.F32, L.LAYOUT_KN_PLANES))) > 0  # K split over blocks
    assert lib.cutb_variant_name(L.VARIANT_GEMV_PLANES) == b"QGemvPlanes"
    assert lib.cutb_qmatmul_workspace_bytes(C.byref(desc(L.Q4_0, 1, 4096, 11008))) == 0
    # few rows, long K: split over K, partial sums staged in the workspace
    d = desc(L.Q4_0, 8, 28672, 1024)
    d.flags = L.FLAG_STAGE_PER_CTA
    ws = lib.cutb_qmatmul_workspace_bytes(C.byref(d))
    assert ws > 0 and ws % (8 * 1024 * 4) == 0
    # the tensor-core GEMM for few tokens: head / tail slots of every CTA of its K split (43 tiles of 256 rows x 16 units
    # of 256 k over 148 SMs -> runs of 5 units, 138 CTAs), [2 x CTAs][tokens rounded to 8][256] floats
    g = desc(L.Q4_0, 32, 4096, 11008)
    g.variant = L.VARIANT_GEMM_TC
    assert lib.cutb_qmatmul_workspace_bytes(C.byref(g)) == 2 * 138 * 32 * 256 * 4
    g = desc(L.Q4_0, 30, 4096, 11008, L.F32)   # fp32 rows: their fp16 copy comes first
    g.variant = L.VARIANT_GEMM_TC
    assert lib.cutb_qmatmul_workspace_bytes(C.byref(g)) == 30 * 4096 * 2 + 2 * 138 * 32 * 256 * 4
    g = desc(L.Q4_0, 32, 256, 38400)           # more tiles than SMs: no split, no slots
    g.variant = L.VARIANT_GEMM_TC
    assert lib.cutb_qmatmul_workspace_bytes(C.byref(g)) == 0
    # three rows and more: the activations are quantised once per call into the workspace as well
    d.flags = 0
    assert lib.cutb_qmatmul_workspace_bytes(C.byref(d)) > ws
    assert lib.cutb_qmatmul_workspace_bytes(C.byref(desc(L.Q4_0, 2, 4096, 11008))) == 0


def test_rows_kernel_has_a_name_and_is_named_where_it_runs():
    """9 to 32 rows over blocks: with the scratch that the query asks for the choice is QGemvRowsMma, without it the former kernel, and a
    caller may name any of them; shapes that the kernel does not take are refused."""
    lib = L.lib()

    def desc(M, variant=L.VARIANT_AUTO, flags=0, fmt=L.Q4_0, dtype=L.F16, scratch=True):
        d = L.QMatmulDesc()
        d.format, d.layout, d.a_dtype, d.variant, d.flags = fmt, L.LAYOUT_GGUF_BLOCKS, dtype, variant, flags
        d.M, d.K, d.N, d.lda, d.ldc = M, 4096, 11008, 4096, 11008
        d.A = d.W = d.C = 256  # never dereferenced here
        d.W_bytes = 1 << 40
        if scratch:
            d.workspace, d.workspace_bytes = 256, lib.cutb_qmatmul_workspace_bytes(C.byref(d))
        return d

    chosen = lambda d: lib.cutb_qmatmul_select_variant(C.byref(d))
    assert lib.cutb_variant_name(L.VARIANT_ROWS_MMA) == b"QGemvRowsMma"
    for M, dtype, former in ((9, L.F16, L.VARIANT_GEMV_MMA), (16, L.F16, L.VARIANT_GEMM_TC), (32, L.F16, L.VARIANT_GEMM_TC), (9, L.F32, L.VARIANT_GEMM_TC)):
        assert chosen(desc(M, dtype=dtype)) == L.VARIANT_ROWS_MMA
        assert chosen(desc(M, dtype=dtype, scratch=False)) == former
        assert chosen(desc(M, former, dtype=dtype)) == former
        d = desc(M, dtype=dtype)
        d.workspace_bytes -= 1
        assert chosen(d) in (former, L.VARIANT_ROWS_MMA) and chosen(d) == (former if lib.cutb_qmatmul_workspace_bytes(C.byref(desc(M, L.VARIANT_ROWS_MMA, dtype=dtype))) > d.workspace_bytes else L.VARIANT_ROWS_MMA)
    assert chosen(desc(8)) == L.VARIANT_GEMV_MMA and chosen(desc(33)) == L.VARIANT_GEMM_TC and chosen(desc(12, fmt=L.Q4_K)) == L.VARIANT_GEMV_MMA
    assert chosen(desc(12, dtype=L.F32, flags=L.FLAG_ACT_16BIT)) == L.VARIANT_GEMV_MMA  # (the mat-vec keeps their range)
    assert chosen(desc(12, L.VARIANT_ROWS_MMA)) == L.VARIANT_ROWS_MMA
    for d in (desc(8, L.VARIANT_ROWS_MMA), desc(33, L.VARIANT_ROWS_MMA), desc(12, L.VARIANT_ROWS_MMA, L.FLAG_STAGE_PER_CTA)):
        assert lib.cutb_qmatmul(C.byref(d), None) == L.ERR_UNSUPPORTED
    assert lib.cutb_qmatmul(C.byref(desc(12, L.VARIANT_ROWS_MMA, scratch=False)), None) == L.ERR_WORKSPACE
    assert chosen(desc(12, L.VARIANT_ROWS_MMA + 1)) < 0


def test_rows_kernel_runs_where_it_measured_faster():
    """The line between the row kernel and the former ones, at shapes on both of its sides."""
    lib = L.lib()

    def rows(fmt, M, K, N, dtype=L.F16):
        d = L.QMatmulDesc()
        d.format, d.layout, d.a_dtype, d.variant = fmt, L.LAYOUT_GGUF_BLOCKS, dtype, L.VARIANT_AUTO
        d.M, d.K, d.N, d.lda, d.ldc = M, K, N, K, N
        d.A = d.W = d.C = d.workspace = 256  # never dereferenced here
        d.W_bytes, d.workspace_bytes = 1 << 40, 1 << 40
        return lib.cutb_qmatmul_select_variant(C.byref(d)) == L.VARIANT_ROWS_MMA

    for M in (9, 16):  # the int8 mat-vec was up to 1.5 times as fast on these
        assert not any(rows(f, M, K, N) for f in (L.Q8_0, L.Q4_0) for K, N in ((2048, 2048), (512, 2048), (1536, 1536), (8192, 512), (4096, 1024), (28672, 512)))
        assert all(rows(f, M, K, N) for f in (L.Q8_0, L.Q4_0) for K, N in ((1024, 1000), (512, 8192), (2560, 2560), (6144, 2048), (8192, 8192), (28672, 1024)))
        assert rows(L.Q8_0, M, 3072, 2048) and not rows(L.Q4_0, M, 3072, 2048) and not rows(L.Q4_0, M, 4608, 2048)
    for M in (17, 32):
        assert not any(rows(L.Q8_0, M, K, N) for K, N in ((4096, 2048), (8192, 1536), (2048, 2048)))
        assert all(rows(L.Q8_0, M, K, N) for K, N in ((3072, 4096), (14336, 1024), (8192, 8192)))
        assert not any(rows(L.Q4_0, M, K, N) for K, N in ((8192, 4096), (8192, 2048), (14336, 4096), (16384, 2048), (2048, 4096)))
        assert all(rows(L.Q4_0, M, K, N) for K, N in ((4096, 4096), (4096, 6144), (8192, 8192), (14336, 8192)))
    assert not any(rows(L.Q4_K, M, 8192, 8192) for M in (9, 16, 17, 32))
    assert all(rows(f, M, K, N, L.F32) for f in (L.Q8_0, L.Q4_0, L.Q4_K) for M in (9, 32) for K, N in ((512, 512), (2048, 2048), (14336, 4096)))


def test_prompt_gemm_shares_k_where_it_measured_faster():
    """Planes of partial sums that the prompt GEMM asks for: the shares of K of the plan that was the fastest of all on 148
    multiprocessors."""
    lib = L.lib()
    for fmt, M, K, N, shares in ((L.Q8_0, 333, 11008, 4096, 4), (L.Q8_0, 256, 8192, 8192, 2), (L.Q8_0, 150, 4096, 4096, 4), (L.Q8_0, 700, 2048, 6144, 1),
                                 (L.Q4_K, 512, 4096, 4096, 2), (L.Q4_K, 512, 14336, 4096, 4), (L.Q4_K, 1500, 4096, 4096, 1), (L.Q4_0, 200, 4096, 4096, 4),
                                 (L.Q4_0, 1092, 11008, 1024, 6), (L.Q4_0, 235, 5120, 11008, 1), (L.Q4_0, 400, 4096, 11008, 1)):
        d = L.QMatmulDesc()
        d.format, d.layout, d.a_dtype, d.variant = fmt, L.LAYOUT_GGUF_BLOCKS, L.F16, L.VARIANT_AUTO
        d.M, d.K, d.N, d.lda, d.ldc = M, K, N, K, N
        d.A = d.W = d.C = 256  # never dereferenced here
        d.W_bytes = 1 << 40
        assert lib.cutb_qmatmul_workspace_bytes(C.byref(d)) == (shares * M * N * 4 if shares > 1 else 0), (fmt, M, K, N)
