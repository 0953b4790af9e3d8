"""The convolution's data movement and long reductions at the edges of their dispatch: im2col, the
halving col2im, column sums of narrow rows, split-K reductions shared by several warps."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("B,C,H,W,k,stride,pad,ld", [
    (1, 1, 1, 1, 1, 1, 0, 8),           # one value
    (5, 3, 7, 13, 3, 1, 1, 32),         # rows that vectors cannot address
    (2, 4, 9, 10, 3, 2, 1, 40),         # halving, odd height
    (3, 2, 8, 9, 3, 2, 1, 24),          # halving, odd width: the general col2im
    (2, 8, 12, 16, 5, 2, 2, 200),
    (2, 32, 32, 32, 3, 2, 1, 288),
    (1, 512, 16, 16, 3, 2, 1, 4608),    # too large to stage in shared memory
    (2, 2, 20, 24, 11, 3, 9, 248),
])
def test_im2col_col2im(dtype, B, C, H, W, k, stride, pad, ld):
    from luatorch_b200 import _C
    g = torch.Generator(device="cuda").manual_seed(H * W + k)
    x = torch.randn(B, C, H, W, generator=g, device="cuda").to(dtype)
    patch = C * k * k
    cols = _C.im2col(x.reshape(-1), B, C, H, W, k, stride, pad, ld)
    ref = torch.nn.functional.unfold(x.float(), k, padding=pad, stride=stride).transpose(1, 2).reshape(-1, patch)
    assert torch.equal(cols[:, :patch].float(), ref) and not cols[:, patch:].any()
    gr = torch.randn(cols.shape, generator=g, device="cuda").to(dtype)
    din = _C.col2im(gr[:, :patch], B, C, H, W, k, stride, pad).view(B, C, H, W).double()
    taps = gr[:, :patch].double().view(B, -1, patch).transpose(1, 2)
    fold = lambda t: torch.nn.functional.fold(t, (H, W), k, padding=pad, stride=stride)
    # at most k k terms summed in fp32, the result rounded to the type
    lost = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -24
    assert bool(((din - fold(taps)).abs() <= k * k * 2.0 ** -24 * fold(taps.abs()) + lost * fold(taps).abs()).all())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("rows", [1, 7, 8, 255, 2049, 70001])
@pytest.mark.parametrize("cols", [8, 32, 64, 128])
def test_column_sum_of_narrow_rows(dtype, rows, cols):
    from luatorch_b200 import _backend as B
    g = torch.Generator(device="cuda").manual_seed(rows + cols)
    x = torch.randn(rows, cols, generator=g, device="cuda").to(dtype)
    out = torch.full((cols,), 0.5, device="cuda")
    B.column_sum(x, out, True)
    xd = x.double()
    assert bool(((out.double() - 0.5 - xd.sum(0)).abs() <= (rows + 1) * 2.0 ** -24 * (xd.abs().sum(0) + 1)).all())
    again = torch.full((cols,), 0.5, device="cuda")
    B.column_sum(x, again, True)
    assert torch.equal(out, again)


@pytest.mark.parametrize("M,N,K", [(32, 27, 131072), (64, 288, 32768), (128, 576, 8192), (72, 5, 65536), (256, 256, 16384)])
def test_split_k_reduction(M, N, K):
    """Long products with few outputs (weight gradients)."""
    from luatorch_b200 import _backend as B
    g = torch.Generator(device="cuda").manual_seed(N)
    ld = (N + 7) // 8 * 8
    a = torch.randn(K, M, generator=g, device="cuda").bfloat16()
    b = torch.randn(K, ld, generator=g, device="cuda").bfloat16()
    out = torch.ones(M, N, device="cuda")
    B.gemm(a, b, a_t=True, out=out, accumulate=True, n_valid=N)
    ad, bd = a.double().t(), b.double()[:, :N]
    assert bool(((out.double() - 1 - ad @ bd).abs() <= K * 2.0 ** -24 * (ad.abs() @ bd.abs() + 1)).all())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("rows", [1, 9, 130, 4095, 131072])
@pytest.mark.parametrize("cols", [4, 8, 16, 32, 64, 128])
def test_column_sum_does_not_depend_on_the_row_stride(dtype, rows, cols):
    """Rows that lie back to back and the same rows further apart: the same order of sums."""
    from luatorch_b200 import _backend as B
    g = torch.Generator(device="cuda").manual_seed(rows + cols)
    x = torch.randn(rows, cols, generator=g, device="cuda").to(dtype)
    wide = torch.zeros(rows, cols + 8, device="cuda", dtype=dtype)
    wide[:, :cols] = x
    for acc in (False, True):
        a, b = torch.full((cols,), 0.5, device="cuda"), torch.full((cols,), 0.5, device="cuda")
        B.column_sum(x, a, acc)
        B.column_sum(wide[:, :cols], b, acc)
        assert torch.equal(a, b)


@pytest.mark.parametrize("M,N,K", [(32, 27, 131072), (16, 8, 65536), (64, 288, 32768)])
def test_split_k_slices_are_added_in_index_order(M, N, K):
    """One product that is not zero per 2048 values of K (so that a slice has at most one), of very
    different sizes: the result is their fp32 sum from the first to the last."""
    import numpy as np
    from luatorch_b200 import _backend as B
    g = torch.Generator().manual_seed(K)
    n = K // 2048
    a, b = torch.zeros(K, M), torch.zeros(K, (N + 7) // 8 * 8)
    v = (torch.randn(n, M, generator=g) * torch.exp(3 * torch.randn(n, M, generator=g))).bfloat16().float()
    a[::2048] = v
    b[::2048] = 1.0
    out = torch.zeros(M, N, device="cuda")
    B.gemm(a.cuda().bfloat16(), b.cuda().bfloat16(), a_t=True, out=out, n_valid=N)
    ref = np.zeros(M, dtype=np.float32)
    for row in v.numpy():
        ref = ref + row
    assert torch.equal(out.cpu(), torch.from_numpy(ref)[:, None].expand(M, N))
