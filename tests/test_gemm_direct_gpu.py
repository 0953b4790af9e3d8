"""Products whose operands TMA cannot address (fp32, odd row lengths, narrow outputs): the direct
kernel, the packed route and the SIMT kernel against a float64 reference.

Bounds.  fp32: each operand loses at most 2^-18 of itself beyond its bf16 hi + lo parts and the
lo * lo product (2^-18) is left out, so an element is off by at most 2^-16 sum|a||b|, plus fp32
accumulation of 3 K terms, 3 K 2^-24 sum|a||b| worst case.  bf16 operands are exact: the rounding
of the result (2^-8 of it) and the accumulation (K 2^-23 sum|a||b|) remain."""
import pytest
import torch

pytestmark = pytest.mark.gpu

SIZES = [(1, 1, 1), (5, 3, 7), (16, 16, 512), (128, 64, 64), (129, 65, 65), (127, 63, 63), (256, 10, 784),
         (61, 300, 2001), (257, 129, 1000), (1021, 1333, 777), (1, 1000, 300), (2049, 2047, 515)]


def _check(out, a, b, dtype, extra=None):
    ad, bd = a.double(), b.double()
    ref = ad @ bd
    mag = ad.abs() @ bd.abs()
    K = a.shape[1]
    if extra is not None:
        ref, mag = ref + extra, mag + extra.abs()
    bound = mag * (2.0 ** -16 + 3 * K * 2.0 ** -24) if dtype == torch.float32 else ref.abs() * 2.0 ** -8 + mag * K * 2.0 ** -23
    assert bool(((out.double() - ref).abs() <= bound + 1e-30).all()), float(((out.double() - ref).abs() / (bound + 1e-30)).max())


@pytest.mark.parametrize("M,N,K", SIZES)
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("a_t,b_t", [(False, False), (False, True), (True, False), (True, True)])
def test_any_operands(M, N, K, dtype, a_t, b_t):
    from luatorch_b200 import _C, _backend as B
    g = torch.Generator(device="cuda").manual_seed(M * 31 + N * 7 + K)
    # odd offsets and row lengths: views into a larger buffer
    def mat(rows, cols):
        t = torch.randn(rows * (cols + 1) + 1, generator=g, device="cuda").to(dtype)
        return t[1:].view(rows, cols + 1)[:, :cols]
    a = mat(K, M) if a_t else mat(M, K)
    b = mat(N, K) if b_t else mat(K, N)
    out = B.gemm(a, b, a_t=a_t, b_t=b_t, out_dtype=dtype)
    _check(out, a.t() if a_t else a, b.t() if b_t else b, dtype)
    assert _C.gemm_device_error() == 0


@pytest.mark.parametrize("M,N,K", [(33, 10, 300), (1021, 1333, 777)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_epilogue_and_repeatability(M, N, K, dtype):
    """Bias, scale and accumulation, and the same bits twice."""
    from luatorch_b200 import _backend as B
    g = torch.Generator(device="cuda").manual_seed(5)
    a, b = (torch.randn(s, generator=g, device="cuda").to(dtype) for s in ((M, K), (K, N)))
    bias = torch.randn(N, generator=g, device="cuda")
    outs = []
    for _ in range(2):
        out = torch.ones(M, N, device="cuda")
        B.gemm(a, b, out=out, alpha=0.5, bias=bias, accumulate=True)
        outs.append(out)
    _check(outs[0], 0.5 * a, b, torch.float32, extra=(bias + 1.0).double().expand(M, N))
    assert torch.equal(*outs)


def test_batched_fp32():
    from luatorch_b200 import _backend as B
    g = torch.Generator(device="cuda").manual_seed(6)
    a, b = torch.randn(5, 37, 70, generator=g, device="cuda"), torch.randn(5, 70, 131, generator=g, device="cuda")
    out = B.bmm(a, b)
    for i in range(5):
        _check(out[i], a[i], b[i], torch.float32)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("M,N,K", [(3, 5, 4), (1, 2, 200), (64, 33, 64)])
def test_more_matrices_than_a_grid_dimension_holds(M, N, K, dtype):
    from luatorch_b200 import _C, _backend as B
    g = torch.Generator(device="cuda").manual_seed(7)
    n = 65600
    a, b = torch.randn(n, M, K, generator=g, device="cuda").to(dtype), torch.randn(n, K, N, generator=g, device="cuda").to(dtype)
    out = B.bmm(a, b)
    for i in (0, 1, 32767, 65535, 65536, n - 1):
        _check(out[i], a[i], b[i], dtype)
    assert _C.gemm_device_error() == 0


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("a_t,b_t", [(False, False), (False, True), (True, False), (True, True)])
@pytest.mark.parametrize("M,N,K,packed", [(1030, 777, 1001, True), (2047, 1029, 150, True), (64, 24, 700, False)])
def test_batches_in_two_levels(M, N, K, packed, a_t, b_t, dtype):
    """Four matrices as 2 x 2 with gaps between them, on the packed and the direct route."""
    import luatorch_b200 as lf
    from luatorch_b200 import _C
    g = torch.Generator(device="cuda").manual_seed(M + K)

    def mats(rows, cols):       # odd rows, a gap behind each matrix and another behind each pair
        ld, inner = cols + 1, rows * (cols + 1) + 3
        outer = 2 * inner + 5
        return torch.randn(2 * outer, generator=g, device="cuda").to(dtype), ld, inner, outer

    def matrix(t, i, o, rows, cols, ld, inner, outer):
        return t[o * outer + i * inner:][:rows * ld].view(rows, ld)[:, :cols]

    sa, sb = ((K, M) if a_t else (M, K)), ((N, K) if b_t else (K, N))
    a, b = mats(*sa), mats(*sb)
    out = torch.zeros(2, 2, M, N, device="cuda", dtype=dtype)
    before = sum(lf.launch_counts())
    _C.gemm(a[0], b[0], out, M, N, K, a[1], b[1], N, a_t, not b_t, 2, 2, a[2], a[3], b[2], b[3], M * N, 2 * M * N,
            1.0, False, None, 0, None, 0, None, None, 0, 0)
    assert sum(lf.launch_counts()) - before == (2 if packed else 1)
    for o in range(2):
        for i in range(2):
            x, y = matrix(a[0], i, o, *sa, *a[1:]), matrix(b[0], i, o, *sb, *b[1:])
            _check(out[o, i], x.t() if a_t else x, y.t() if b_t else y, dtype)
    assert _C.gemm_device_error() == 0


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("batch,M,N,K,simt", [
    (1, 1000, 1000, 32, True), (1, 1000, 1025, 32, False),          # 1024 tile steps and one column more
    (1, 256, 1024, 128, True), (1, 256, 1024, 129, False),          # four steps of k and one value more
    (64, 32, 127, 128, True), (65, 32, 127, 128, False),
])
def test_border_of_the_simt_kernel(batch, M, N, K, simt, dtype):
    """One launch of fp32 FMAs up to the border: no part of an fp32 operand is lost there."""
    from luatorch_b200 import _backend as B
    g = torch.Generator(device="cuda").manual_seed(N)
    a, b = torch.randn(batch, M, K, generator=g, device="cuda").to(dtype), torch.randn(batch, K, N + 1, generator=g, device="cuda").to(dtype)
    b = b[:, :, :N].contiguous()
    out = B.bmm(a, b)
    for i in {0, batch - 1}:
        _check(out[i], a[i], b[i], dtype)
        if simt and dtype == torch.float32:
            ad, bd = a[i].double(), b[i].double()
            assert bool(((out[i].double() - ad @ bd).abs() <= K * 2.0 ** -24 * (ad.abs() @ bd.abs())).all())


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("M,N,K", [(40, 33, 50), (61, 24, 700), (1030, 777, 1001)])     # SIMT, direct, packed
@pytest.mark.parametrize("what", ["gelu", "dgelu", "relu", "drelu", "residual"])
def test_fused_epilogues_on_every_route(M, N, K, what, dtype):
    """bf16 results.  Beside the product's bound: one rounding of the result (2^-8 of it) and of the
    intermediate written to aux_out, and tanh.approx (2^-11) through gelu (|z| / 2 of it) and gelu'."""
    from luatorch_b200 import _backend as B
    g = torch.Generator(device="cuda").manual_seed(K)
    a, b = (torch.randn(r, c + 1, generator=g, device="cuda").to(dtype)[:, :c] for r, c in ((M, K), (K, N)))
    a = a * (K ** -0.5)
    x = torch.randn(M, N, generator=g, device="cuda").bfloat16()
    bias = torch.randn(N, generator=g, device="cuda")
    kw = {"gelu": dict(act=1, bias=bias), "dgelu": dict(act=2, aux_in=x), "relu": dict(act=3, bias=bias),
          "drelu": dict(act=4, aux_in=x), "residual": dict(residual=x, bias=bias)}[what]
    pre = torch.empty(M, N, device="cuda", dtype=torch.bfloat16) if what in ("gelu", "relu") else None
    out = B.gemm(a, b, out_dtype=torch.bfloat16, aux_out=pre, **kw).double()
    z, mag = a.double() @ b.double(), a.double().abs() @ b.double().abs()
    if what in ("gelu", "relu", "residual"):
        z = z + bias.double()
        mag = mag + bias.double().abs()
    err = mag * (2.0 ** -16 + 3 * K * 2.0 ** -24)
    xd, c0, c1 = x.double(), 0.7978845608, 0.044715
    if what == "gelu":
        ref = torch.nn.functional.gelu(z, approximate="tanh")
        err = 1.2 * err + 0.5 * z.abs() * 2.0 ** -11
    elif what == "dgelu":
        t = torch.tanh(c0 * (xd + c1 * xd ** 3))
        ref = z * (0.5 * (1 + t) + 0.5 * xd * (1 - t * t) * c0 * (1 + 3 * c1 * xd * xd))
        err = 1.2 * err + z.abs() * 2.0 ** -11 * (0.5 + xd.abs() * c0 * (1 + 3 * c1 * xd * xd))
    elif what == "residual":
        ref = z + xd
    else:
        ref = z.clamp(min=0) if what == "relu" else torch.where(xd > 0, z, torch.zeros_like(z))
    assert bool(((out - ref).abs() <= err + 2.0 ** -8 * ref.abs() + 1e-6).all()), float((out - ref).abs().max())
    if pre is not None:
        assert bool(((pre.double() - z).abs() <= mag * (2.0 ** -16 + 3 * K * 2.0 ** -24) + 2.0 ** -8 * z.abs() + 1e-6).all())


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_no_matrices(dtype):
    """A batch of none has nothing to read."""
    from luatorch_b200 import _backend as B
    out = B.bmm(torch.empty(0, 20, 30, device="cuda", dtype=dtype), torch.empty(0, 30, 40, device="cuda", dtype=dtype))
    assert out.shape == (0, 20, 40) and out.dtype == dtype
    torch.cuda.synchronize()
