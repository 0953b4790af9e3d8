"""Row kernels on rows that 16-byte vectors cannot address (odd lengths, odd offsets) and around the
lengths where the LayerNorm dispatch changes kernel, against float64.

Bounds.  fp32: sums of `cols` (or `rows`) terms in fp32, worst case n 2^-24 of the sum of their
sizes; LayerNorm output is O(1) after division by the deviation, so 1e-5 + cols 2^-24 covers mean,
variance and the last three operations; GELU's tanh adds a few ulps.  bf16 results are
rounded once more: 2^-8 of themselves."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _rows(g, rows, cols, dtype, offset):
    t = torch.randn(rows * cols + offset, generator=g, device="cuda").to(dtype)
    return t[offset:].view(rows, cols)


@pytest.mark.parametrize("cols", [1, 31, 33, 255, 257, 511, 513, 1023, 1025, 2049, 4095, 4096, 4097, 8191, 8193])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("offset", [0, 1])
def test_layernorm_gelu_colsum_any_row(cols, dtype, offset):
    from luatorch_b200 import _backend as B
    g = torch.Generator(device="cuda").manual_seed(cols)
    rows = 19 if cols > 1 else 300
    x = _rows(g, rows, cols, dtype, offset)
    gamma, beta, bias = (_rows(g, 1, cols, dtype, offset)[0] for _ in range(3))
    xd = x.double()
    lost = 2.0 ** -8 if dtype == torch.bfloat16 else 0.0

    y, mean, rstd = B.layernorm(x, gamma, beta)
    mu = xd.mean(1, keepdim=True)
    rs = (xd.var(1, unbiased=False, keepdim=True) + 1e-5).rsqrt()
    want = (xd - mu) * rs * gamma.double() + beta.double()
    # a row of one value: its deviation is 0 and eps alone divides what rounding leaves of it
    tol = (1e-5 + cols * 2.0 ** -24) * (1 + gamma.double().abs() * (1 + (xd - mu).abs() * rs)) + lost * want.abs()
    assert bool(((y.double() - want).abs() <= tol).all())
    torch.testing.assert_close(mean.double(), mu[:, 0], atol=1e-6 + cols * 2.0 ** -24, rtol=0)
    torch.testing.assert_close(rstd.double(), rs[:, 0], atol=0, rtol=1e-5 + cols * 2.0 ** -24)

    z = xd + bias.double()
    act = 0.5 * z * (1 + torch.tanh(math.sqrt(2 / math.pi) * (z + 0.044715 * z ** 3)))
    got = B.gelu_bias(x, bias)
    assert bool(((got.double() - act).abs() <= 2e-6 * (1 + z.abs()) + lost * act.abs()).all())

    s = B.column_sum(x)
    bound = rows * 2.0 ** -24 * xd.abs().sum(0) + lost * xd.sum(0).abs()
    assert bool(((s.double() - xd.sum(0)).abs() <= bound + 1e-30).all())


@pytest.mark.parametrize("cols", [1, 31, 64, 255, 256, 257, 512, 513, 1000, 1023, 1024, 1025, 2048])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("offset", [0, 1])
def test_softmax_any_row(cols, dtype, offset):
    """exp2 and the scaled argument are good to a few 2^-23 of arguments up to 2^6, the sum to
    cols 2^-24: 2e-5 of each value covers them; infinities and NaN as torch has them."""
    from luatorch_b200 import _backend as B
    g = torch.Generator(device="cuda").manual_seed(cols)
    x = _rows(g, 21, cols, dtype, offset).mul_(5)
    x[1, 0] = -math.inf
    x[2] = -math.inf
    x[3, cols // 2] = math.inf
    x[4, cols - 1] = math.nan
    want = torch.softmax(x.double(), 1)
    got = B.softmax(x)
    assert torch.equal(got.isnan(), want.isnan())
    tol = (2e-5 + cols * 2.0 ** -24 + (2.0 ** -8 if dtype == torch.bfloat16 else 0.0)) * want + 1e-37
    assert bool(((got.double() - want).abs() <= tol)[~want.isnan()].all())


@pytest.mark.parametrize("rows", [127, 128, 129, 2049, 4111])
@pytest.mark.parametrize("cols", [1, 33])
def test_column_sum_slabs(rows, cols):
    """Slabs of 128 rows, sixteen partial sums at a time."""
    from luatorch_b200 import _backend as B
    g = torch.Generator(device="cuda").manual_seed(rows)
    x = torch.randn(rows, cols, generator=g, device="cuda")
    xd = x.double()
    out = torch.ones(cols, device="cuda")
    B.column_sum(x, out, True)
    bound = (rows + 1) * 2.0 ** -24 * (xd.abs().sum(0) + 1)
    assert bool(((out.double() - 1 - xd.sum(0)).abs() <= bound).all())


@pytest.mark.parametrize("cols", [1, 31, 64, 257, 1000, 1024])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
def test_softmax_of_extreme_rows(cols, dtype):
    """Rows of the type's lowest value (a mask that leaves nothing) are uniform, as in torch; large
    values keep the bound, because the difference to the maximum is taken before anything is scaled:
    arguments down to -87 count, each to 87 2^-23 of its exponential, and the sum to cols 2^-24."""
    from luatorch_b200 import _backend as B
    g = torch.Generator(device="cuda").manual_seed(cols)
    low = torch.finfo(dtype).min
    x = torch.randn(8, cols, generator=g, device="cuda").to(dtype)
    x[0] = low
    x[1, ::2] = low
    x[2, 1:] = low
    x[3:6] *= 1000
    x[6] = torch.finfo(dtype).max
    y = B.softmax(x).double()
    ref = torch.softmax(x.double(), 1)
    lost = {torch.float32: 0.0, torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11}[dtype]
    tiny = 2.0 ** -24 if dtype == torch.float16 else 1e-37      # subnormal results
    assert bool(((y - ref).abs() <= (2e-5 + cols * 2.0 ** -24 + lost) * ref + tiny).all()), float((y - ref).abs().max())
