"""Matrix products of many rows (tiles on pairs of SMs) against fp64 products of the same bf16 operands: edges of tiles in rows, features and K,
every epilogue, ragged and empty experts."""
import pytest
import torch

from mlx_sharding_b200.ops import get_backend

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def C():
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    return get_backend("b200").C()


def rnd(*s, seed=0, scale=1.0):
    return (torch.randn(*s, generator=torch.Generator(device="cuda").manual_seed(seed), device="cuda") * scale).to(torch.bfloat16)


def close(got, ref, mag, terms):
    """fp32 sums of ``terms`` exact products (2^-24 of the sum of magnitudes each, in any order), one rounding of the result to bf16 (2^-8)."""
    bound = ref.abs() * 2 ** -8 + mag * terms ** 0.5 * 2 ** -22 + 1e-5
    assert ((got.double() - ref).abs() <= bound).all(), float(((got.double() - ref).abs() - bound).max())


@pytest.mark.parametrize("T", [257, 288, 300, 511, 512, 2200])
@pytest.mark.parametrize("N,K", [(136, 64), (256, 72), (392, 1000), (1408, 2048)])
@pytest.mark.parametrize("kind", ["plain", "fp32", "residual_bias", "relu2", "gate_up"])
def test_dense(C, T, N, K, kind):
    x = rnd(T, K + 8, seed=1)[:, :K]                                      # strided rows
    w, w2 = rnd(N, K, seed=2, scale=K ** -0.5), rnd(N, K, seed=3, scale=K ** -0.5)
    y, mag = x.double() @ w.double().t(), x.double().abs() @ w.double().abs().t()
    if kind == "plain":
        close(C.linear(x, w, None, None, None, 0, 0.0, False, None, 0, 0, 0, pair=1), y, mag, K)
    elif kind == "fp32":
        got = C.linear(x, w, None, None, None, 0, 0.0, True, None, 0, 0, 0, pair=1)
        assert got.dtype == torch.float32 and ((got.double() - y).abs() <= mag * K ** 0.5 * 2 ** -22 + 1e-6).all()
    elif kind == "residual_bias":
        r, b = rnd(T, N + 2, seed=4)[:, :N], rnd(N, seed=5)
        out = torch.zeros(T + 1, N + 6, dtype=torch.bfloat16, device="cuda")[:, 2:N + 2]
        C.linear(x, w, None, r, b, 0, 0.0, False, out, 0, 0, 0, pair=1)
        close(out[:T], y + r.double() + b.double(), mag, K)
        assert (out[T] == 0).all()
    elif kind == "relu2":
        ref = y.clamp(min=0).square()
        got = C.linear(x, w, None, None, None, 4, 0.0, False, None, 0, 0, 0, pair=1).double()
        assert ((got - ref).abs() <= ref * 2 ** -8 + 2 * y.abs() * mag * K ** 0.5 * 2 ** -22 + 1e-5).all()
    else:
        u, mu = x.double() @ w2.double().t(), x.double().abs() @ w2.double().abs().t()
        ref = y * torch.sigmoid(y) * u
        got = C.linear(x, w, w2, None, None, 1, 0.0, False, None, 0, 0, 0, pair=1).double()
        # the products' errors enter through both factors (|d silu| <= 1.1); the hardware's exp and division are good to 2^-20
        assert ((got - ref).abs() <= ref.abs() * (2 ** -8 + 2 ** -18) + (1.1 * u.abs() * mag + y.abs() * mu) * K ** 0.5 * 2 ** -22 + 1e-5).all()


@pytest.mark.parametrize("rows", [[300, 0, 1, 255, 256, 257, 0, 513], [0, 0, 40, 2000], [129] * 9 + [0] * 30])
@pytest.mark.parametrize("N,K", [(128, 192), (384, 256)])
def test_grouped(C, rows, N, K):
    E, T = len(rows), max(rows)
    offs = torch.tensor([0] + rows).cumsum(0).to(torch.int32).cuda()
    x, w, w2 = rnd(sum(rows), K, seed=1), rnd(E, N, K, seed=2, scale=K ** -0.5), rnd(E, N, K, seed=3, scale=K ** -0.5)
    y = C.grouped_linear(x, w, None, offs, T, 0, True, pair=1).double()
    h = C.grouped_linear(x, w, w2, offs, T, 1, False, pair=1).double()
    at = 0
    for e, n in enumerate(rows):
        xs = x[at:at + n].double()
        g, u = xs @ w[e].double().t(), xs @ w2[e].double().t()
        mag, mu = xs.abs() @ w[e].double().abs().t(), xs.abs() @ w2[e].double().abs().t()
        assert ((y[at:at + n] - g).abs() <= mag * K ** 0.5 * 2 ** -22 + 1e-6).all()
        ref = g * torch.sigmoid(g) * u
        assert ((h[at:at + n] - ref).abs() <= ref.abs() * (2 ** -8 + 2 ** -18) + (1.1 * u.abs() * mag + g.abs() * mu) * K ** 0.5 * 2 ** -22 + 1e-5).all()
        at += n


# both sides of the rule's lines: rows in one and two tiles, one round and several, short and long K
@pytest.mark.parametrize("T,N,K,dual", [(257, 256, 128, False), (320, 10944, 512, False), (640, 10944, 512, False), (1500, 3648, 2048, False), (300, 4096, 14336, False),
                                        (513, 14336, 3584, True), (512, 14336, 3584, True), (600, 1408, 2048, True)])
def test_rule(C, T, N, K, dual):
    """Pairs of SMs, single SMs, and whichever the rule takes."""
    x, w, w2 = rnd(T, K, seed=1), rnd(N, K, seed=2, scale=K ** -0.5), rnd(N, K, seed=3, scale=K ** -0.5) if dual else None
    one, two, auto = (C.linear(x, w, w2, act=1 if dual else 0, pair=p) for p in (0, 1, -1))
    assert torch.equal(auto, one) or torch.equal(auto, two)
    y, mag = x.double() @ w.double().t(), x.double().abs() @ w.double().abs().t()
    if dual:
        u, mu = x.double() @ w2.double().t(), x.double().abs() @ w2.double().abs().t()
        y, mag = y * torch.sigmoid(y) * u, 1.1 * u.abs() * mag + y.abs() * mu
    for got in (one, two):
        assert ((got.double() - y).abs() <= y.abs() * (2 ** -8 + 2 ** -18) + mag * K ** 0.5 * 2 ** -22 + 1e-5).all()
