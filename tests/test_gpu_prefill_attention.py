"""Prompt attention on the tensor cores at the edges of its tiles (128 tokens, 128 keys, boxes of 64 rows), against 64 bits.

Without rotation the kernel's queries are the test's (rounded beforehand): what is left are fp32 scores and sums, exponentials of a
few ulp and bf16 weights in two terms (2^-17) or fp16 weights (2^-11): rel-L2 1e-4 and 1e-3.  With rotation a query element may
round the other way, one ulp (2^-8 in bf16) of a part of a score: 4e-3."""
import numpy as np
import pytest

from cut_b200 import _lib as L
from cut_b200 import ops

pytestmark = pytest.mark.gpu


def _rel(got, ref):
    return float((got.double() - ref).norm() / ref.norm())


def _reference(q, k, v, scale, pos, window, sink):
    """q [T, H, d]; k, v [positions, G, .] in 64 bits; sink: a logit per head, or None."""
    import torch

    out = torch.empty((q.shape[0], q.shape[1], v.shape[2]), dtype=torch.float64, device=q.device)
    keys, rep = torch.arange(k.shape[0], device=q.device), q.shape[1] // k.shape[1]
    hidden = (keys[None, :] > pos[:, None]) | (pos[:, None] - keys[None, :] >= window)
    for h in range(q.shape[1]):
        s = (q[:, h] @ k[:, h // rep].T * scale).masked_fill(hidden, float("-inf"))
        if sink is not None:
            s = torch.cat([s, sink[h].expand(len(s), 1)], dim=1)
        out[:, h] = s.softmax(-1)[:, : k.shape[0]] @ v[:, h // rep]
    return out


def _turned(x, cos, sin, neighbours):
    import torch

    n = cos.shape[1]
    a, b = (x[..., 0: 2 * n: 2], x[..., 1: 2 * n: 2]) if neighbours else (x[..., :n], x[..., n: 2 * n])
    c, s = cos[:, None], sin[:, None]
    y = (a * c - b * s, b * c + a * s)
    y = torch.stack(y, -1).flatten(-2) if neighbours else torch.cat(y, -1)
    return torch.cat([y, x[..., 2 * n:]], -1)


@pytest.mark.parametrize("T,pos,window,dim,vdim,rot,near,scale,sink", [
    (16, 0, 1000, 128, 128, 0, True, 0.1, True), (127, 0, 64, 96, 128, 0, True, 0.1, False), (129, 63, 130, 128, 64, 128, True, 0.1, True),
    (256, 1, 128, 128, 128, 128, False, -0.1, False), (257, 500, 333, 72, 40, 24, False, 0.1, True), (300, 0, 1, 128, 128, 0, True, 0.0, False),
    (384, 200, 512, 64, 64, 64, True, 0.1, True), (2100, 0, 600, 128, 128, 32, True, 0.1, True)])
def test_window(T, pos, window, dim, vdim, rot, near, scale, sink):
    import torch

    g = torch.Generator(device="cuda").manual_seed(T + dim)
    rand = lambda *s: torch.randn(s, device="cuda", generator=g)
    H, G, end = 4, 2, pos + T
    kh, vh = (dim + 7) // 8 * 8, (vdim + 7) // 8 * 8
    ring = (min(window, end) + T + 63) // 64 * 64
    k, v = rand(end, G, dim).bfloat16(), rand(end, G, vdim).bfloat16()
    kc, vc = torch.full((ring, G, kh), float("nan"), device="cuda").bfloat16(), torch.full((ring, G, vh), float("nan"), device="cuda").bfloat16()
    kept = torch.arange(max(0, pos + 1 - window), end, device="cuda")  # (everything else is NaN)
    kc[kept % ring], vc[kept % ring] = 0, 0
    kc[kept % ring, :, :dim], vc[kept % ring, :, :vdim] = k[kept], v[kept]
    qkv = torch.empty((T, (H + G) * dim + G * vdim), device="cuda")
    q = rand(T, H, dim).bfloat16().float()
    qkv[:, : H * dim] = q.reshape(T, -1)
    cos, sin = (torch.cos(rand(end, rot // 2)), torch.sin(rand(end, rot // 2))) if rot else (None, None)
    at = torch.arange(pos, end, device="cuda")
    if rot:
        q = _turned(q, cos[at], sin[at], near).bfloat16()
    out, status = torch.full((T, H * vdim), float("nan"), device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    d = ops.window_desc(qkv, H, G, dim, vdim, kc.view(ring, -1), vc.view(ring, -1), window=window, scale=scale, out=out, cos_t=cos, sin_t=sin, rot_dims=rot,
                        pairing=L.ROT_NEIGHBOURS if near else L.ROT_HALVES, max_pos=end, sink=sink, pos=pos, status=status)
    ops.window_attention(d)
    zero = torch.zeros(H, dtype=torch.float64, device="cuda")
    ref = _reference(q.double(), k.double(), v.double(), scale, at, window, zero if sink else None)
    assert int(status.item()) == 0
    assert _rel(out.view(T, H, vdim), ref) <= (4e-3 if rot else 1e-4)


@pytest.mark.parametrize("T,heads,past,max_pos", [(300, 4, 1, 400), (300, 4, 150, 400), (500, 74, 90, 600), (130, 4, 129, 200)])
def test_window_tokens_without_table_rows(T, heads, past, max_pos):
    """The last `past` tokens lie beyond the tables: they stay unwritten and the status says so; every other token is served, wherever
    the blocks of 128 and (500 tokens x 74 heads) 256 tokens end."""
    import torch

    g = torch.Generator(device="cuda").manual_seed(T + past)
    rand = lambda *s: torch.randn(s, device="cuda", generator=g)
    pos, window, hd, n = max_pos - (T - past), 200, 128, T - past
    ring = (window + T + 63) // 64 * 64
    k, v, q = rand(max_pos, 2, hd).bfloat16(), rand(max_pos, 2, hd).bfloat16(), rand(T, heads, hd).bfloat16().float()
    kc, vc = torch.full((ring, 2, hd), float("nan"), device="cuda").bfloat16(), torch.full((ring, 2, hd), float("nan"), device="cuda").bfloat16()
    kept = torch.arange(max(0, pos + 1 - window), max_pos, device="cuda")
    kc[kept % ring], vc[kept % ring] = k[kept], v[kept]
    qkv = torch.zeros((T, (heads + 4) * hd), device="cuda")
    qkv[:, : heads * hd] = q.reshape(T, -1)
    out, status = torch.full((T, heads * hd), float("nan"), device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    ops.window_attention(ops.window_desc(qkv, heads, 2, hd, hd, kc.view(ring, -1), vc.view(ring, -1), window=window, scale=0.1, out=out, max_pos=max_pos,
                                         sink=True, pos=pos, status=status))
    zero = torch.zeros(heads, dtype=torch.float64, device="cuda")
    ref = _reference(q[:n].double(), k.double(), v.double(), 0.1, torch.arange(pos, max_pos, device="cuda"), window, zero)
    assert int(status.item()) == L.ERR_INVALID
    assert bool(out[n:].isnan().all())
    assert _rel(out[:n].view(n, heads, hd), ref) <= 1e-4


@pytest.mark.parametrize("T,pos,dim,rot,vdim,scale", [(40, 0, 128, 64, 128, 0.1), (128, 5, 64, 32, 64, 0.1), (257, 127, 128, 32, 128, -0.1),
                                                     (300, 0, 24, 8, 40, 0.1), (1100, 64, 64, 64, 128, 0.1), (130, 0, 128, 0, 72, 0.1)])
@pytest.mark.parametrize("on_device", [False, True])
def test_latent(T, pos, dim, rot, vdim, scale, on_device):
    import torch

    g = torch.Generator(device="cuda").manual_seed(T + dim + rot)
    rand = lambda *s: torch.randn(s, device="cuda", generator=g)
    H, end, rank = 3, pos + T, 64
    k, v, r = rand(end, H, dim).bfloat16(), rand(end, H, vdim).bfloat16(), rand(end, max(rot, 1)).bfloat16()[:, :rot]
    cache = torch.zeros((end + 50, rank + max(rot, 8)), device="cuda").bfloat16()
    cache[:end, rank: rank + rot], cache[end:] = r, float("nan")
    cos, sin = torch.cos(rand(end + 50, rot // 2)), torch.sin(rand(end + 50, rot // 2))
    q = rand(T, H, dim + rot).bfloat16().float()
    out, status = torch.full((T, H * vdim), float("nan"), device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    sink, where = rand(H), torch.tensor([pos], dtype=torch.int32, device="cuda")
    d = ops.latent_desc(cache, H, dim, rot, vdim, rank, scale=scale, eps=1e-6, max_pos=end + 50, n_tokens=T, cos_t=cos, sin_t=sin, sink=sink,
                        pos=0 if on_device else pos, pos_ptr=where.data_ptr() if on_device else None, q=q.view(T, -1), k_exp=k.view(end, -1),
                        v_exp=v.view(end, -1), out=out, status=status)
    import ctypes

    L.check(L.lib().cutb_latent_prefill(ctypes.byref(d), torch.cuda.current_stream().cuda_stream))
    at = torch.arange(pos, end, device="cuda")
    qt = torch.cat([q[..., :dim], _turned(q[..., dim:], cos[at], sin[at], True)], -1).bfloat16() if rot else q
    kk = torch.cat([k, r[:, None].expand(-1, H, -1)], -1)
    ref = _reference(qt.double(), kk.double(), v.double(), scale, at, 1 << 30, sink.double())
    assert int(status.item()) == 0
    assert _rel(out.view(T, H, vdim), ref) <= (4e-3 if rot else 1e-4)


@pytest.mark.parametrize("T,hd,order", [(16, 64, "up"), (129, 128, "up"), (256, 128, "down"), (300, 64, "mixed"), (1030, 128, "up")])
def test_llama(T, hd, order):
    import torch

    g = torch.Generator(device="cuda").manual_seed(T + hd)
    rand = lambda *s: torch.randn(s, device="cuda", generator=g)
    H, G, rows = 4, 2, T + 37
    at = torch.arange(20, 20 + T, device="cuda")
    at = at.flip(0) if order == "down" else at[torch.randperm(T, device="cuda", generator=g)] if order == "mixed" else at
    kc, vc = rand(rows, G, hd).half(), rand(rows, G, hd).half()
    kc[20 + T:], vc[20 + T:] = float("nan"), float("nan")
    cos, sin = torch.cos(rand(rows, hd // 2)), torch.sin(rand(rows, hd // 2))
    q = rand(T, H, hd)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    out = ops.batched_attention(q.view(T, -1), kc.view(rows, -1), vc.view(rows, -1), at.int(), cos, sin, H, G, hd, status=status)
    seen = slice(0, 20 + T)
    ref = _reference(_turned(q, cos[at], sin[at], False).half().double(), kc[seen].double(), vc[seen].double(), hd ** -0.5, at, 1 << 30, None)
    assert int(status.item()) == 0
    assert _rel(out.view(T, H, hd), ref) <= 1e-3


def _attend(mode, q, k, v, pos, window, scale, status, sink=None, order=None):
    """Unrotated attention of queries [T, H, d] at pos, pos + 1, ... (or at positions `order`) over k, v [positions, G, .], through the entry
    point of `mode`; sink: a logit per head (llama: none, window: zeros)."""
    import ctypes

    import torch

    T, H, hd = q.shape
    end, G = k.shape[0], k.shape[1]
    ones, zeros = torch.ones((end, hd // 2), device="cuda"), torch.zeros((end, hd // 2), device="cuda")
    out = torch.full((T, H * hd), float("nan"), device="cuda")
    if mode == "llama":
        at = torch.arange(pos, end, device="cuda", dtype=torch.int32) if order is None else order.int()
        ops.batched_attention(q.view(T, -1), k.view(end, -1), v.view(end, -1), at, ones, zeros, H, G, hd, out=out, scale=scale, status=status)
    elif mode == "window":
        ring = (min(window, end) + T + 63) // 64 * 64
        kc, vc = torch.full((ring, G, hd), float("nan"), device="cuda").bfloat16(), torch.full((ring, G, hd), float("nan"), device="cuda").bfloat16()
        kept = torch.arange(max(0, pos + 1 - window), end, device="cuda")
        kc[kept % ring], vc[kept % ring] = k[kept], v[kept]
        qkv = torch.zeros((T, (H + 2 * G) * hd), device="cuda")
        qkv[:, : H * hd] = q.view(T, -1)
        ops.window_attention(ops.window_desc(qkv, H, G, hd, hd, kc.view(ring, -1), vc.view(ring, -1), window=window, scale=scale, out=out, max_pos=end,
                                             sink=sink is not None, pos=pos, status=status))
    else:  # a third of the head as the shared turned part: equal in all heads
        rot = 64
        cache = torch.zeros((end, 64 + rot), device="cuda").bfloat16()
        cache[:, 64:] = k[:, 0, hd - rot:]
        d = ops.latent_desc(cache, H, hd - rot, rot, v.shape[2], 64, scale=scale, eps=1e-6, max_pos=end, n_tokens=T, cos_t=ones, sin_t=zeros, sink=sink, pos=pos,
                            q=q.view(T, -1), k_exp=k[:, :, : hd - rot].reshape(end, -1), v_exp=v.reshape(end, -1), out=out[:, : H * v.shape[2]], status=status)
        L.check(L.lib().cutb_latent_prefill(ctypes.byref(d), torch.cuda.current_stream().cuda_stream))
        out = out[:, : H * v.shape[2]]
    return out.view(T, H, -1)


def _inputs(mode, T, pos, seed):
    """q, k, v and a head count that gives blocks of 256 tokens (128 while the launch would leave multiprocessors idle) if T > 600."""
    import torch

    g = torch.Generator(device="cuda").manual_seed(seed)
    big = T > 600
    H = 50 if big else 6
    assert (-(-T // 256) * H >= torch.cuda.get_device_properties(0).multi_processor_count) == big
    G, hd, vd = (H, 192, 128) if mode == "latent" else (10 if big else 2, 128, 128)
    t = torch.float16 if mode == "llama" else torch.bfloat16
    rand = lambda *s: torch.randn(s, device="cuda", generator=g).to(t)
    q, k, v = rand(T, H, hd), rand(pos + T, G, hd), rand(pos + T, G, vd)
    if mode == "latent":
        k[:, :, 128:] = k[:, :1, 128:]
    return q.float(), k, v


@pytest.mark.parametrize("mode", ["llama", "window", "latent"])
@pytest.mark.parametrize("T,pos,window", [(300, 0, 1 << 20), (300, 77, 90), (641, 0, 1 << 20), (700, 60, 200)])
def test_values_that_are_not_finite(mode, T, pos, window):
    """An infinity or a NaN among the values reaches the tokens that see its key, in its column, and no other."""
    import torch

    if mode != "window":
        window = 1 << 20
    q, k, v = _inputs(mode, T, pos, T + pos)
    H, G, at = q.shape[1], k.shape[1], torch.arange(pos, pos + T, device="cuda")
    strays = [(3, 0, 5, float("inf")), (pos + 130, G - 1, 0, float("nan")), (pos + 255, 0, 77, float("-inf")), (pos + T - 1, G - 1, 127, float("nan"))]
    clean = v.clone()
    for key, g, col, x in strays:
        v[key, g, col], clean[key, g, col] = x, 0.0
    ref = _reference(q.double(), k.double(), clean.double(), 0.1, at, window, None)
    for key, g, col, x in strays:
        seen = (at >= key) & (at - key < window)
        ref[seen, g * (H // G): (g + 1) * (H // G), col] = x
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    got = _attend(mode, q, k, v, pos, window, 0.1, status)
    finite = ref.isfinite()
    assert int(status.item()) == 0
    assert bool((got.isfinite() == finite).all()) and bool((got.isnan() == ref.isnan()).all()) and bool((got == ref)[ref.isinf()].all())
    assert _rel(got[finite], ref[finite]) <= (1e-3 if mode == "llama" else 1e-4)


@pytest.mark.parametrize("mode", ["llama", "window", "latent"])
@pytest.mark.parametrize("T,pos,sink", [(140, 200, None), (700, 130, None), (140, 200, 0.0)])
def test_the_largest_weight_is_exact(mode, T, pos, sink):
    """One key, behind the first key tile, has a value; its logit stands 0.5 to 8 (in powers of two) above the others', another height for
    every token.  Its weight is 1 relative to the maximum, without rounding to 16 bits, so the output is that value times a quotient of
    fp32 sums: exponentials to 2^-22 and their arguments (up to 8) to 2^-21, 1e-6 in all.  (Weights relative to an older maximum carry
    2^-12 in fp16 and 2^-18 in two bf16 terms.)"""
    import torch

    if mode == "llama" and sink is not None:
        pytest.skip("no sink on the llama path")
    q, k, v = _inputs(mode, T, pos, T)
    H, at, d = q.shape[1], torch.arange(pos, pos + T, device="cuda"), q.shape[2] - (64 if mode == "latent" else 0)
    key = pos - 1
    height = torch.linspace(0.5, 8.0, T, device="cuda").to(k.dtype).float()
    q.zero_()
    q[:, :, 0] = height[:, None]
    k.zero_()
    k[key, :, 0] = 1.0
    v[:key], v[key + 1:] = 0.0, 0.0
    scale = 0.6931472
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    sinks = None if sink is None else torch.full((H,), sink, device="cuda")
    got = _attend(mode, q, k, v, pos, 1 << 20, scale, status, sinks)
    ref = _reference(q.double(), k.double(), v.double(), float(torch.tensor(scale)), at, 1 << 30, None if sink is None else sinks.double())
    assert int(status.item()) == 0
    worst = ((got.double() - ref).norm(dim=2) / ref.norm(dim=2)).max()
    assert float(worst) <= 1e-6


@pytest.mark.parametrize("mode", ["llama", "window", "latent"])
@pytest.mark.parametrize("T,pos,window", [(128, 600, 1 << 20), (257, 511, 700), (700, 60, 1 << 20), (897, 0, 640)])
def test_scores_that_jump(mode, T, pos, window):
    """Every third token meets keys whose logits stand 20 and then 40 (in powers of two) above the others', in later key tiles: the maximum
    is followed and what was summed is scaled down, several times in a row, while the other tokens of the warp stay as they are.  (700 and
    897 tokens: two token tiles to a block, the second of the last block ragged, and of one token.)"""
    import torch

    if mode != "window":
        window = 1 << 20
    q, k, v = _inputs(mode, T, pos, T + pos)
    H, at = q.shape[1], torch.arange(pos, pos + T, device="cuda")
    d = q.shape[2] - (64 if mode == "latent" else 0)
    scale = 0.1
    unit = torch.zeros(d, device="cuda")
    unit[: d // 2] = 1.0  # (exact in 16 bits)
    q[::3, :, :d] += 4.0 * unit
    for key, jump in ((140, 20.0), (139, 21.0), (300, 30.0), (420, 40.0), (421, 40.5), (pos + T - 2, 50.0)):
        k[key, :, :d] = (jump / (4.0 * (d // 2) * scale * 1.4427) * unit).to(k.dtype)
    sink = None if mode == "llama" else torch.zeros(H, device="cuda") if mode == "window" else torch.full((H,), 15.0, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    got = _attend(mode, q.to(k.dtype).float(), k, v, pos, window, scale, status, sink)
    ref = _reference(q.to(k.dtype).double(), k.double(), v.double(), scale, at, window, None if sink is None else sink.double())
    assert int(status.item()) == 0
    assert _rel(got, ref) <= (1e-3 if mode == "llama" else 1e-4)
    worst = (got.double() - ref).norm(dim=2) / ref.norm(dim=2)
    assert float(worst.max()) <= (4e-3 if mode == "llama" else 4e-4)  # (a token: rounding of few weights, not averaged over many)


@pytest.mark.parametrize("mode", ["llama", "window", "latent"])
@pytest.mark.parametrize("T,pos,window", [(769, 0, 300), (640, 33, 257), (1153, 100, 640)])
def test_two_token_tiles_to_a_block(mode, T, pos, window):
    """Blocks of 256 tokens: both tiles over shared key and value slots, a last block of one tile, of one token, and of 129 tokens; windows
    that begin and end inside a key tile; positions in no order on the llama path."""
    import torch

    if mode != "window":
        window = 1 << 20
    q, k, v = _inputs(mode, T, pos, T + pos)
    at = torch.arange(pos, pos + T, device="cuda")
    if mode == "llama":
        at = at[torch.randperm(T, device="cuda", generator=torch.Generator(device="cuda").manual_seed(T))]
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    got = _attend(mode, q, k, v, pos, window, 0.1, status, order=at)
    ref = _reference(q.double(), k.double(), v.double(), 0.1, at, window, None)
    assert int(status.item()) == 0
    assert _rel(got, ref) <= (1e-3 if mode == "llama" else 1e-4)


@pytest.mark.parametrize("T,pos", [(300, 0), (700, 60)])
def test_a_sink_of_minus_infinity_is_none(T, pos):
    import torch

    q, k, v = _inputs("latent", T, pos, T)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    one = _attend("latent", q, k, v, pos, 1 << 20, 0.1, status, torch.full((q.shape[1],), float("-inf"), device="cuda"))
    assert torch.equal(one, _attend("latent", q, k, v, pos, 1 << 20, 0.1, status)) and bool(one.isfinite().all())
    assert int(status.item()) == 0
