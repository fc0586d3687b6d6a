"""Split-K GEMM of a cluster: the reduction's batches of tokens (remainders, the last rank's share), residual, two weights, fp32 results."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T", [1, 3, 16, 31, 33, 64, 65, 100, 128])
@pytest.mark.parametrize("splits", [0, 2, 4])
@pytest.mark.parametrize("N,K", [(256, 2048), (5000, 1032)])
def test_split_reduction(T, splits, N, K):
    from mlx_sharding_b200.ops import get_backend
    C = get_backend("b200").C()
    gen = torch.Generator("cuda").manual_seed(T + N)
    r = lambda *s: torch.randn(*s, device="cuda", generator=gen).bfloat16()
    x, w, w2, res = r(T, K), r(N, K), r(N, K), r(T, N)
    y = x.double() @ w.double().T
    # fp32 sums of K exact products: K * 2^-24 * |x|.|w| at most; bf16 results: two roundings of 2^-8 with a residual between
    mag = (x.double().abs() @ w.double().abs().T) * K * 2 ** -24
    got = C.linear(x, w, out_fp32=True, splits=splits).double()
    assert ((got - y).abs() <= mag + y.abs() * 2 ** -23).all()
    got = C.linear(x, w, residual=res, splits=splits).double()
    want = y + res.double()
    assert ((got - want).abs() <= mag + y.abs() * 2 ** -8 + want.abs() * 1.01 * 2 ** -8).all()
    if T <= 64:
        u = x.double() @ w2.double().T
        got = C.linear(x, w * 0.02, w2, act=1, splits=splits).double()
        g = x.double() @ (w * 0.02).double().T
        want = torch.nn.functional.silu(g) * u
        # the gate's sum and the fast exponential: 2^-8 relative covers both beside the rounding of the result
        assert ((got - want).abs() <= want.abs() * 2 ** -6 + mag * 2 + 1e-3).all()


@pytest.mark.parametrize("T", [1, 8, 64, 100])
@pytest.mark.parametrize("splits", [0, 1, 2, 4])
def test_squared_relu_of_split_sums(T, splits):
    """The activation of a single-weight product applies to the whole sum, whoever adds it up."""
    from mlx_sharding_b200.ops import get_backend
    C = get_backend("b200").C()
    gen = torch.Generator("cuda").manual_seed(T)
    r = lambda *s: torch.randn(*s, device="cuda", generator=gen).bfloat16()
    x, w, b = r(T, 2048), (r(256, 2048) * 0.03).bfloat16(), r(256)
    y = x.double() @ w.double().T + b.double()
    want = y.clamp(min=0).square()
    mag = x.double().abs() @ w.double().abs().T * 2048 * 2 ** -24
    got = C.linear(x, w, bias=b, act=4, splits=splits).double()
    assert ((got - want).abs() <= want * 2 ** -8 + 2 * y.abs() * mag + mag.square() + 1e-6).all()
