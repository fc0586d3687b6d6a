"""Bounded waits inside kernels: a kernel whose waits run out gives its memory back and returns, the host gets an error, and the next launch is right."""
import pytest
import torch

from mlx_sharding_b200.ops import get_backend
from mlx_sharding_b200.ops.meta import BatchMeta

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def C():
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    return get_backend("b200").C()


# one stream of rows whose halves meet at barriers, two query heads, two row tiles; many items per CTA
@pytest.mark.parametrize("H,Hk,dk,dv", [(8, 4, 256, 256), (8, 2, 128, 128), (3, 3, 192, 128)])
def test_prompt_attention_returns(C, H, Hk, dk, dv):
    q_lens, ctx0 = [700, 1500, 40, 129] * 4, [0, 300, 64, 1000] * 4
    need = [(a + b + 63) // 64 for a, b in zip(q_lens, ctx0)]
    tables, at = [], 1
    for n in need:
        tables.append(list(range(at, at + n)))
        at += n
    meta = BatchMeta.build(q_lens, ctx0, tables, 64, device="cuda")
    g = torch.Generator(device="cuda").manual_seed(0)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda").to(torch.bfloat16)
    q, k, v = rnd(meta.num_tokens, H, dk), rnd(at, Hk, 64, dk), rnd(at, Hk, 64, dv)
    call = lambda **kw: C.flash_prefill(q, k, v, meta.block_tables, meta.cu_seqlens, meta.context_lens, dk ** -0.5, meta.num_tokens, 0.0, meta.max_ctx_len, **kw)
    want = call()
    torch.cuda.synchronize()
    for spins in (0, 3, 20):                                     # a wait gives up at its first failed looks: in every phase of the kernel
        call(wait_spins=spins)
        torch.cuda.synchronize()
        if spins == 0:                                           # (a few looks may be enough)
            with pytest.raises(RuntimeError, match="prompt attention"):
                C.check_waits()
        else:
            try:
                C.check_waits()
            except RuntimeError:
                pass
    assert torch.equal(call(), want)
    torch.cuda.synchronize()
    C.check_waits()


# one accumulator set and two, fp32 results; several tiles per pair
@pytest.mark.parametrize("dual,fp32", [(False, False), (True, False), (False, True)])
def test_many_row_gemm_returns(C, dual, fp32):
    g = torch.Generator(device="cuda").manual_seed(0)
    rnd = lambda *s: (torch.randn(*s, generator=g, device="cuda") * 0.05).to(torch.bfloat16)
    x, w, w2 = rnd(5000, 1024), rnd(4096, 1024), rnd(4096, 1024) if dual else None
    call = lambda **kw: C.linear(x, w, w2, act=1 if dual else 0, out_fp32=fp32, pair=1, **kw)
    want = call()
    torch.cuda.synchronize()
    for spins in (0, 3, 20):
        call(wait_spins=spins)
        torch.cuda.synchronize()
        if spins == 0:
            with pytest.raises(RuntimeError, match="GEMM"):
                call()                                           # a later launch says so, and is not made
        else:
            try:
                C.check_waits()
            except RuntimeError:
                pass
    assert torch.equal(call(), want)
    torch.cuda.synchronize()
    C.check_waits()
