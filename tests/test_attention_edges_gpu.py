"""Attention kernels at the edges of their tiles and splits, against fp64 attention of the same bf16 inputs."""
import random

import pytest
import torch

from mlx_sharding_b200.ops import get_backend
from mlx_sharding_b200.ops.meta import BatchMeta

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def B():
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    return get_backend("b200")


def paged(q_lens, ctx0, Hk, dk, dv, page, seed=0):
    """Ragged batch over pools of random rows with shuffled pages."""
    need = [(a + b + page - 1) // page for a, b in zip(q_lens, ctx0)]
    order = list(range(1, 1 + sum(need)))
    random.Random(seed).shuffle(order)
    tables = [[order.pop() for _ in range(n)] for n in need]
    g = torch.Generator(device="cuda").manual_seed(seed)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda").to(torch.bfloat16)
    meta = BatchMeta.build(q_lens, ctx0, tables, page, device="cuda")
    return meta, tables, rnd(1 + sum(need), Hk, page, dk), rnd(1 + sum(need), Hk, page, dv), rnd


def exact(q, kpool, vpool, tables, q_lens, ctx0, scale, cap=0.0, one_term=False):
    """(attention, the same with |v|: what a relative error of the probabilities can move); ``one_term``: probabilities rounded to bf16 before the second product"""
    page, rep = kpool.shape[2], q.shape[1] // kpool.shape[1]
    out, at = [], 0
    for n, c, pages in zip(q_lens, ctx0, tables):
        pos = torch.arange(c + n, device="cuda")
        pg = torch.tensor(pages, device="cuda")[pos // page]
        k = kpool[pg, :, pos % page].double().repeat_interleave(rep, 1)
        v = vpool[pg, :, pos % page].double().repeat_interleave(rep, 1)
        s = torch.einsum("thd,nhd->htn", q[at:at + n].double(), k) * scale
        s = cap * torch.tanh(s / cap) if cap else s
        s = s.masked_fill(pos[None, None, :] > (c + torch.arange(n, device="cuda"))[None, :, None], float("-inf"))
        e = (s - s.amax(-1, keepdim=True)).exp()
        p = (e.to(torch.bfloat16).double() if one_term else e) / e.sum(-1, keepdim=True)
        out.append(torch.stack([torch.einsum("htn,nhv->thv", p, v), torch.einsum("htn,nhv->thv", p, v.abs())]))
        at += n
    return torch.cat(out, 1).unbind(0)


# (heads, kv heads, dk, dv, page): every instantiation, groups of 1 to 8, pages that hold less than a tile
@pytest.mark.parametrize("H,Hk,dk,dv,page", [(32, 8, 128, 128, 64), (8, 1, 128, 128, 16), (4, 4, 128, 128, 24), (16, 8, 256, 256, 64), (2, 2, 192, 128, 64),
                                             (8, 2, 64, 64, 8)])
@pytest.mark.parametrize("ctx", [[0, 14, 15, 16, 62, 63, 64, 65], [4095], [1, 3000, 255, 256, 17], [0, 15], [767, 3], [768],
                                 [i * 7 % 256 for i in range(512)], [6000, 4097, 2]])
def test_paged_decode(B, H, Hk, dk, dv, page, ctx):
    """One query per sequence; lengths around a warp's 16 keys and a CTA's 64, one split and many, a warp per CTA and four."""
    meta, tables, kpool, vpool, rnd = paged([1] * len(ctx), ctx, Hk, dk, dv, page)
    q = rnd(len(ctx), H, dk) * 2
    got = B.paged_attention(q, kpool, vpool, meta, dk ** -0.5).double()
    ref, _ = exact(q, kpool, vpool, tables, [1] * len(ctx), ctx, dk ** -0.5)
    # fp32 sums and probabilities (2^-16) of bf16 inputs, one rounding of the result to bf16 (2^-8)
    assert ((got - ref).abs() <= ref.abs() * 2 ** -8 + 2e-4).all(), float((got - ref).abs().max())
    again = B.paged_attention(q, kpool, vpool, meta, dk ** -0.5).double()         # the merge left its tickets as it found them
    assert ((again - ref).abs() <= ref.abs() * 2 ** -8 + 2e-4).all()


def test_paged_decode_capped(B):
    """Capped scores: the hardware's tanh is good to 2^-11 of its result, times the cap 50 in the exponent."""
    ctx = [200, 15, 900]
    meta, tables, kpool, vpool, rnd = paged([1] * 3, ctx, 8, 256, 256, 64)
    q = rnd(3, 16, 256) * 2
    got = B.paged_attention(q, kpool, vpool, meta, 256 ** -0.5, 50.0).double()
    ref, _ = exact(q, kpool, vpool, tables, [1] * 3, ctx, 256 ** -0.5, 50.0)
    assert ((got - ref).norm() / ref.norm()) < 2e-2


RAGGED = [([1, 127, 128, 129, 64, 65], [0] * 6), ([255, 257, 3], [0, 1, 700]), ([300, 1, 40, 1], [63, 2000, 64, 5]), ([700], [1000])]


# every instantiation; heads in pairs (even groups) and rows in pairs (odd groups); pages of a part of a tile, of a tile and of several
@pytest.mark.parametrize("H,Hk,dk,dv,page,cap", [(8, 2, 128, 128, 64, 0.0), (4, 4, 128, 128, 128, 0.0), (6, 2, 128, 128, 16, 0.0), (4, 2, 64, 64, 32, 0.0),
                                                 (3, 3, 192, 128, 64, 0.0), (4, 2, 256, 256, 64, 0.0), (4, 2, 256, 256, 64, 50.0),
                                                 (4, 2, 128, 128, 64, 30.0), (2, 2, 192, 128, 64, 30.0), (2, 1, 64, 64, 16, 30.0)])
@pytest.mark.parametrize("q_lens,ctx0", RAGGED)
def test_flash_prefill(B, H, Hk, dk, dv, page, cap, q_lens, ctx0):
    meta, tables, kpool, vpool, rnd = paged(q_lens, ctx0, Hk, dk, dv, page)
    used = torch.zeros(kpool.shape[0], page, dtype=torch.bool, device="cuda")       # what lies behind a sequence's end may be anything
    for n, c, pages in zip(q_lens, ctx0, tables):
        pos = torch.arange(n + c, device="cuda")
        used[torch.tensor(pages, device="cuda")[pos // page], pos % page] = True
    kpool.masked_fill_(~used[:, None, :, None], float("nan"))
    vpool.masked_fill_(~used[:, None, :, None], float("inf"))
    q = torch.cat([rnd(meta.num_tokens, H, dk) * 3, rnd(meta.num_tokens, H, 8)], -1)[..., :dk]      # strided rows
    assert B.C().flash_prefill_takes(q, kpool, vpool, cap, meta.num_seqs, meta.max_ctx_len)
    got = B.paged_attention(q, kpool, vpool, meta, dk ** -0.5, cap).double()
    ref, mag = exact(q, kpool.nan_to_num(0.0), vpool.nan_to_num(0.0, 0.0, 0.0), tables, q_lens, ctx0, dk ** -0.5, cap)
    # result in bf16 (unit roundoff 2^-8); probabilities in bf16 (2^-8), or as two terms where the scores are capped or heads are 256 wide; the
    # hardware's tanh is good to 2^-11 of its result, so a capped score s moves by |s| 2^-11 (|s| < 30 here) and its probability by as much
    p_err = 30 * 2 ** -11 if cap else (2 ** -16 if dk == 256 else 2 ** -8)
    assert ((got - ref).abs() <= ref.abs() * 1.01 * 2 ** -8 + mag * p_err + 2e-4).all(), float(((got - ref).abs() - mag * p_err).max())


@pytest.mark.parametrize("q_lens,ctx0", RAGGED)
def test_flash_mla(B, q_lens, ctx0):
    """Keys and values read in place of the kv_b product, rotary keys from the latent pool; the step's own rows (nothing cached) and gathered ones."""
    heads, nope, rd, vd, page = 5, 128, 64, 128, 64
    meta, tables, lat, _, rnd = paged(q_lens, ctx0, 1, 576, 64, page)
    fresh = max(ctx0) == 0
    mb = meta.block_tables.shape[1]
    per = -1 if fresh else mb * page
    kv = rnd(meta.num_tokens if fresh else len(q_lens) * mb * page, heads * (nope + vd))
    kpool, vpool = rnd(lat.shape[0], heads, page, nope + rd), rnd(lat.shape[0], heads, page, vd)
    at = 0
    for b, (n, c, pages) in enumerate(zip(q_lens, ctx0, tables)):
        pos = torch.arange(n + c, device="cuda")
        pg = torch.tensor(pages, device="cuda")[pos // page]
        rows = kv[at + pos] if fresh else kv[b * per + pos]
        rows = rows.view(-1, heads, nope + vd)
        kpool[pg, :, pos % page] = torch.cat([rows[..., :nope], lat[pg, 0, pos % page, 512:].unsqueeze(1).expand(-1, heads, rd)], -1)
        vpool[pg, :, pos % page] = rows[..., nope:]
        at += n
    # what lies behind a sequence's end may be anything: rows of the product (the step's own rows: behind the last sequence), slots of the latent pool
    last = torch.ones(lat.shape[0], page, dtype=torch.bool, device="cuda")
    behind = torch.ones(kv.shape[0] + 64, dtype=torch.bool, device="cuda")
    for b, (n, c, pages) in enumerate(zip(q_lens, ctx0, tables)):
        pos = torch.arange(n + c, device="cuda")
        last[torch.tensor(pages, device="cuda")[pos // page], pos % page] = False
        if not fresh:
            behind[b * per + pos] = False
    if fresh:
        behind[:meta.num_tokens] = False
    lat[:, 0][last] = float("nan")
    kv = torch.cat([kv, rnd(64, kv.shape[1])]).view(-1, heads, nope + vd)
    kv[..., :nope].masked_fill_(behind[:, None, None], float("nan"))
    kv[..., nope:].masked_fill_(behind[:, None, None], float("inf"))
    kv = kv.view(-1, heads * (nope + vd))
    q = rnd(meta.num_tokens, heads, nope + rd) * 2
    got = B.mla_prefill_attention(q, kv, lat, meta, 192 ** -0.5, per).double().view(-1, heads, vd)
    ref, mag = exact(q, kpool, vpool, tables, q_lens, ctx0, 192 ** -0.5)
    assert ((got - ref).abs() <= ref.abs() * 2 ** -8 + mag * 2 ** -8 + 2e-4).all()


def test_mla_prefill_prologue(B):
    """Against the single ops: latent norm, both ropes and the cache append."""
    from mlx_sharding_b200.ops import RopeSpec
    meta, _, pool, _, rnd = paged([37, 5], [0, 0], 1, 576, 64, 64)
    T = meta.num_tokens
    big = rnd(T, 16 * 192 + 576)
    q, ckv, kpe = big[:, :3072].unflatten(1, (16, 192)), big[:, 3072:3584], big[:, 3584:]
    w = rnd(512)
    spec = RopeSpec((10000.0 ** (-torch.arange(0, 64, 2, dtype=torch.float32) / 64)).cuda(), 64, True, 1.1)
    q2, kpe2, pool2 = q.clone(), kpe.clone().view(T, 1, 64), pool.clone()
    lat = B.mla_prefill_prologue(q, ckv, kpe, w, 1e-6, pool, meta, spec)
    B.rope_(q2, meta.positions, spec, 128)
    B.rope_(kpe2, meta.positions, spec, 0)
    lat2 = B.rmsnorm(ckv, w, 1e-6)
    pool2.view(-1, 576)[meta.slot_mapping.long()] = torch.cat([lat2, kpe2.view(T, 64)], 1)
    assert torch.equal(q, q2)
    assert torch.allclose(lat.float(), lat2.float(), rtol=2 ** -7, atol=0)                # (one rounding; sums in another order)
    assert torch.allclose(pool.float(), pool2.float(), rtol=2 ** -7, atol=0) and torch.equal(pool.view(-1, 576)[meta.slot_mapping.long(), :512], lat)


@pytest.mark.parametrize("H,Hk,D,dv,page,T", [(32, 8, 128, 128, 64, 1), (32, 8, 128, 128, 64, 300), (4, 2, 256, 256, 64, 7), (3, 1, 48, 24, 16, 5), (2, 2, 64, 64, 64, 1000)])
def test_rope_kv_append(B, H, Hk, D, dv, page, T):
    """Bit for bit the single ops, from strided rows."""
    from mlx_sharding_b200.ops import RopeSpec
    meta, _, kpool, vpool, rnd = paged([T], [70], Hk, D, dv, page)
    spec = RopeSpec((500000.0 ** (-torch.arange(0, D, 2, dtype=torch.float32) / D)).cuda(), D)
    rows = rnd(T, (H + Hk) * D + Hk * dv + 8)
    cut = lambda r: (r[:, :H * D].unflatten(1, (H, D)), r[:, H * D:(H + Hk) * D].unflatten(1, (Hk, D)), r[:, (H + Hk) * D:(H + Hk) * D + Hk * dv].unflatten(1, (Hk, dv)))
    (q, k, v), k2, v2 = cut(rows.clone()), kpool.clone(), vpool.clone()
    assert B.C().rope_append(q, k, v, k2, v2, meta.slot_mapping, meta.positions, spec.inv_freq, 1.0)
    q1, k1, v1 = cut(rows)
    B.rope_(q1, meta.positions, spec)
    B.rope_(k1, meta.positions, spec)
    B.kv_write(k1, v1, kpool, vpool, meta.slot_mapping)
    assert torch.equal(q, q1) and torch.equal(k2, kpool) and torch.equal(v2, vpool)


# many items per CTA: every barrier and ring goes around several times; heads in pairs, rows in pairs and single streams
@pytest.mark.parametrize("H,Hk,dk,dv,cap", [(32, 8, 128, 128, 0.0), (5, 5, 192, 128, 0.0), (16, 8, 256, 256, 50.0), (64, 16, 64, 64, 0.0)])
def test_flash_prefill_many_items(B, H, Hk, dk, dv, cap):
    r = random.Random(3)
    q_lens = [r.choice((1, 5, 64, 100, 128, 129, 200, 257, 300)) for _ in range(60)] + [1500]
    ctx0 = [r.choice((0, 0, 3, 64, 130)) for _ in range(60)] + [200]
    meta, tables, kpool, vpool, rnd = paged(q_lens, ctx0, Hk, dk, dv, 64)
    q = rnd(meta.num_tokens, H, dk) * 3
    got = B.paged_attention(q, kpool, vpool, meta, dk ** -0.5, cap).double()
    ref, mag = exact(q, kpool, vpool, tables, q_lens, ctx0, dk ** -0.5, cap)
    p_err = 30 * 2 ** -11 if cap else 2 ** -8
    assert ((got - ref).abs() <= ref.abs() * 1.01 * 2 ** -8 + mag * p_err + 2e-4).all()


# the rules that keep a few short prompts off the tcgen05 kernel, on both sides of each line; heads of 256: decode kernel with one tile per warp and with a ring
@pytest.mark.parametrize("H,Hk,dk,dv,cap", [(32, 8, 128, 128, 0.0), (16, 16, 192, 128, 0.0), (16, 8, 256, 256, 50.0), (8, 2, 64, 64, 0.0)])
@pytest.mark.parametrize("q_lens", [[1, 16], [16] * 16, [32] * 4, [31, 33], [127], [128], [127] * 40, [129, 3], [65], [60] * 5, [500], [513], [32] * 17])
def test_short_prompts(B, H, Hk, dk, dv, cap, q_lens):
    ctx0 = [0] * len(q_lens)
    meta, tables, kpool, vpool, rnd = paged(q_lens, ctx0, Hk, dk, dv, 64)
    q = rnd(meta.num_tokens, H, dk)
    got = B.paged_attention(q, kpool, vpool, meta, dk ** -0.5, cap).double()
    ref, mag = exact(q, kpool, vpool, tables, q_lens, ctx0, dk ** -0.5, cap)
    p_err = 30 * 2 ** -11 if cap else 2 ** -8
    assert ((got - ref).abs() <= ref.abs() * 1.01 * 2 ** -8 + mag * p_err + 2e-4).all()


@pytest.mark.parametrize("H,Hk,d,page", [(8, 2, 128, 64), (3, 1, 128, 32), (4, 4, 64, 128), (4, 2, 64, 16)])
@pytest.mark.parametrize("block,window,keep,gate,sink", [(0, 100, 5, "head", True), (0, 300, 130, "elem", False), (200, 0, 0, None, True), (0, 0, 0, None, False),
                                                        (96, 64, 70, "head", True)])
@pytest.mark.parametrize("max_ctx", [0, 448, 449])                     # (a bound of 448 keys sends few rows to the mma.sync form; either is right for any context)
def test_sink_flash(B, H, Hk, d, page, block, window, keep, gate, sink, max_ctx):
    """Windows, blocks, kept first tokens, sinks and gates on the tensor cores against fp64; any sign of the score factor."""
    q_lens, ctx0 = [300, 40, 129, 513], [0, 1000, 63, 300]
    meta, tables, kpool, vpool, rnd = paged(q_lens, ctx0, Hk, d, d, page)
    unused = torch.ones(kpool.shape[0], page, dtype=torch.bool, device="cuda")      # what lies behind a sequence's end may be anything
    for n, c, pages in zip(q_lens, ctx0, tables):
        pos = torch.arange(n + c, device="cuda")
        unused[torch.tensor(pages, device="cuda")[pos // page], pos % page] = False
    kpool.masked_fill_(unused[:, None, :, None], float("nan"))
    vpool.masked_fill_(unused[:, None, :, None], float("inf"))
    T, scale = meta.num_tokens, -2.0 * d ** -0.5
    q = rnd(T, H, d).float() * 1.001 + 1e-3                                # not representable in bf16
    sk = torch.linspace(-1, 3, H, device="cuda") if sink else None
    gt = None if gate is None else rnd(T, H if gate == "head" else H * d)
    out = torch.zeros(T, H * d + 16, dtype=torch.bfloat16, device="cuda")
    B.C().hy_sink_flash(q, kpool, vpool, sk, meta.block_tables, meta.context_lens, meta.cu_seqlens, scale, block, window, 0.5, out, 8, keep, gt, None, None, max_ctx)
    at = 0
    for n, c, pages in zip(q_lens, ctx0, tables):
        pos = torch.arange(c + n, device="cuda")
        pg = torch.tensor(pages, device="cuda")[pos // page]
        k = kpool[pg, :, pos % page].double().repeat_interleave(H // Hk, 1)
        v = vpool[pg, :, pos % page].double().repeat_interleave(H // Hk, 1)
        s = torch.einsum("thd,nhd->htn", q[at:at + n].double(), k) * scale
        me, it = (c + torch.arange(n, device="cuda"))[:, None], pos[None, :]
        hide = torch.zeros(n, c + n, dtype=torch.bool, device="cuda")
        if block:
            hide |= it // block != me // block
        if window:
            hide |= it <= me - window
        s = s.masked_fill(((it > me) | (hide & (it >= keep)))[None], float("-inf"))
        e = (s - s.amax(-1, keepdim=True)).exp()
        den = e.sum(-1, keepdim=True) + (0 if sk is None else (sk.double()[:, None, None] - s.amax(-1, keepdim=True)).exp())
        p = e / den
        ref, mag = torch.einsum("htn,nhv->thv", p, v) * 0.5, torch.einsum("htn,nhv->thv", p, v.abs()) * 0.5
        if gate is not None:
            g = torch.sigmoid(gt[at:at + n].double()).view(n, H, -1)
            ref, mag = ref * g, mag * g
        got = out[at:at + n, 8:8 + H * d].double().view(n, H, d)
        assert ((got - ref).abs() <= ref.abs() * 1.01 * 2 ** -8 + mag * 2 ** -8 + 2e-4).all(), float((got - ref).abs().max())
        at += n
    assert (out[:, :8] == 0).all() and (out[:, 8 + H * d:] == 0).all()


@pytest.mark.parametrize("q_lens,ctx0", [([1, 1, 1], [3, 900, 64]), ([40, 129], [0, 70])])
@pytest.mark.parametrize("H,Hk,dk,dv,cap", [(8, 2, 128, 128, 0.0), (4, 2, 256, 256, 50.0), (2, 2, 192, 128, 0.0)])
def test_pools_at_odd_offsets(B, H, Hk, dk, dv, cap, q_lens, ctx0):
    """Pools that are views four bytes into a buffer: the kernels copy 16 bytes at a time."""
    meta, tables, kpool, vpool, rnd = paged(q_lens, ctx0, Hk, dk, dv, 64)
    at_odd = lambda p: torch.empty(p.numel() + 2, dtype=p.dtype, device="cuda")[2:].view(p.shape).copy_(p)
    q = rnd(meta.num_tokens, H, dk)
    got = B.paged_attention(q, at_odd(kpool), at_odd(vpool), meta, dk ** -0.5, cap).double()
    ref, mag = exact(q, kpool, vpool, tables, q_lens, ctx0, dk ** -0.5, cap)
    assert ((got - ref).abs() <= ref.abs() * 1.01 * 2 ** -8 + mag * (30 * 2 ** -11 if cap else 2 ** -8) + 2e-4).all()
    with pytest.raises(RuntimeError, match="16 bytes"):
        B.kv_write(q[:, :Hk, :dk].contiguous(), torch.zeros(meta.num_tokens, Hk, dv, dtype=torch.bfloat16, device="cuda"), at_odd(kpool), vpool,
                   meta.slot_mapping)


@pytest.mark.parametrize("H,Hk,dk,dv", [(4, 2, 256, 256), (8, 2, 128, 128)])
@pytest.mark.parametrize("factor,cap", [(-1.0, 0.0), (0.0, 0.0), (-1.0, 30.0), (1.0, -1.0)])
def test_prompts_with_any_score_factor(B, H, Hk, dk, dv, factor, cap):
    """A factor that is not positive turns the order of the scores around; a negative cap is none."""
    q_lens, ctx0 = [150, 40], [0, 70]
    meta, tables, kpool, vpool, rnd = paged(q_lens, ctx0, Hk, dk, dv, 64)
    q, scale = rnd(meta.num_tokens, H, dk) * 2, factor * dk ** -0.5
    got = B.paged_attention(q, kpool, vpool, meta, scale, cap).double()
    ref, mag = exact(q, kpool, vpool, tables, q_lens, ctx0, scale, max(cap, 0.0))
    assert ((got - ref).abs() <= ref.abs() * 1.01 * 2 ** -8 + mag * (30 * 2 ** -11 if cap > 0 else 2 ** -16) + 2e-4).all()


@pytest.mark.parametrize("H,Hk,dk,dv,cap", [(8, 2, 128, 128, 0.0), (4, 4, 192, 128, 0.0), (4, 2, 64, 64, 0.0), (4, 2, 256, 256, 0.0), (4, 2, 128, 128, 1e4)])
@pytest.mark.parametrize("gain", [0.5, 2.0, 6.0])
def test_precision_of_prompt_probabilities(B, H, Hk, dk, dv, cap, gain):
    """Flat to peaked softmaxes, maxima that grow slowly.  Heads of 256 and capped scores: beside the rounding of the result there is the 2^-17 of a probability in
    two terms (a cap far above the scores changes them by less than 2^-11).  The others: the error of probabilities that are rounded to bf16 relative to the exact
    maximum, whose own is 1; relative to a maximum that lags, it is an eighth more at a gain of 2."""
    q_lens, ctx0 = [400, 129], [0, 900]
    meta, tables, kpool, vpool, rnd = paged(q_lens, ctx0, Hk, dk, dv, 64)
    q = rnd(meta.num_tokens, H, dk) * gain
    got = B.paged_attention(q, kpool, vpool, meta, dk ** -0.5, cap).double()
    ref, mag = exact(q, kpool, vpool, tables, q_lens, ctx0, dk ** -0.5, cap)
    if cap or dk == 256:
        rounding = (ref.to(torch.bfloat16).double() - ref).norm()
        assert (got - ref).norm() <= 1.02 * rounding + mag.norm() * (4 * gain * 2 ** -11 if cap else 2 ** -16)
    else:
        one_term, _ = exact(q, kpool, vpool, tables, q_lens, ctx0, dk ** -0.5, one_term=True)
        assert (got - ref).norm() <= 1.03 * (one_term.to(torch.bfloat16).double() - ref).norm()


# one or two query heads per kv head over a few keys: both sides of the lines between the vector and the matrix form, in keys and in rows
@pytest.mark.parametrize("H,Hk,dk,dv,cap", [(16, 16, 192, 128, 0.0), (32, 32, 128, 128, 0.0), (4, 4, 256, 256, 0.0), (16, 8, 256, 256, 50.0)])
@pytest.mark.parametrize("n,keys", [(1, 1), (3, 8), (3, 9), (2, 16), (9, 16), (600, 16), (2, 17), (300, 24), (5, 25), (70, 8), (65, 7)])
def test_paged_decode_few_keys(B, H, Hk, dk, dv, cap, n, keys):
    ctx = [keys - 1] + [i * 5 % keys for i in range(n - 1)]
    meta, tables, kpool, vpool, rnd = paged([1] * n, ctx, Hk, dk, dv, 16)
    q = rnd(n, H, dk) * 2
    got = B.paged_attention(q, kpool, vpool, meta, dk ** -0.5, cap).double()
    ref, mag = exact(q, kpool, vpool, tables, [1] * n, ctx, dk ** -0.5, cap)
    assert ((got - ref).abs() <= ref.abs() * 2 ** -8 + mag * (30 * 2 ** -11 if cap else 0.0) + 2e-4).all(), float((got - ref).abs().max())
