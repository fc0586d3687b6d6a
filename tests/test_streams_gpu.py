"""Ops whose CTAs meet through scratch memory, on several streams at once."""
import pytest
import torch

from mlx_sharding_b200.ops import LinearWeight, get_backend
from mlx_sharding_b200.ops.meta import BatchMeta

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def B():
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    return get_backend("b200")


def test_decode_attention_on_two_streams(B):
    """Launches of different split counts that overlap: neither takes the other's tickets or partial sums, then or later."""
    g = torch.Generator(device="cuda").manual_seed(0)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda").to(torch.bfloat16)
    jobs = []
    for n, ctx in ((1, 7000), (3, 2500), (2, 900)):
        per = (ctx + 64) // 64
        tables = [list(range(1 + i * per, 1 + (i + 1) * per)) for i in range(n)]
        meta = BatchMeta.build([1] * n, [ctx] * n, tables, 64, device="cuda")
        q, k, v = rnd(n, 32, 128), rnd(1 + n * per, 8, 64, 128), rnd(1 + n * per, 8, 64, 128)
        w = LinearWeight(weight=rnd(512, 4096) * 0.02)
        jobs.append(lambda q=q, k=k, v=v, meta=meta, w=w: (lambda a: (a, B.linear(a.flatten(1), w)))(B.paged_attention(q, k, v, meta, 128 ** -0.5)))
    want = [j() for j in jobs]
    streams = [torch.cuda.Stream() for _ in jobs]
    torch.cuda.synchronize()
    for s, j in zip(streams, jobs):                              # (workspaces of the streams exist)
        with torch.cuda.stream(s):
            j()
    torch.cuda.synchronize()
    got = [[] for _ in jobs]
    for _ in range(200):
        for s, j, o in zip(streams, jobs, got):
            with torch.cuda.stream(s):
                o.append(j())
    torch.cuda.synchronize()
    for w, outs in zip(want, got):
        assert all(torch.equal(a, w[0]) and torch.equal(y, w[1]) for a, y in outs)
    for w, j in zip(want, jobs):
        assert torch.equal(j()[0], w[0])
