"""The tensor-core product at up to 128 rows where the columns leave SMs idle: K is cut over the CTAs of a cluster, and the finish of a
tile reads the partial sums of all of them."""
import pytest
import torch

from quamba_b200 import ops

pytestmark = pytest.mark.gpu


def _operands(m, k, n, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed + m * 7 + n)
    a = torch.randint(-127, 128, (m, k), device="cuda", generator=g).to(torch.int8)
    w = torch.randint(-127, 128, (n, k), device="cuda", generator=g).to(torch.int8)
    return a, w, (a.double() @ w.double().t()).float(), g       # |sum| < 2^53, and int32 -> fp32 rounds once on both sides


def _convert(r, dtype):
    return torch.clamp(torch.round(r), -128, 127).to(torch.int8) if dtype == torch.int8 else r.to(dtype)


@pytest.mark.parametrize("dtype", [torch.int8, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("m", [9, 16, 64, 128])
def test_scalar_by_value_with_k_split(m, dtype):
    """cutlass_scaled_mv_dq passes its scalar by value and no scale pointers, for any number of rows: alpha * sum, one fp32
    product of the same operands on both sides."""
    k, n, alpha = 1536, 768, 2.5e-4
    a, w, acc, _ = _operands(m, k, n)
    c = torch.empty((m, n), dtype=dtype, device="cuda")
    ops.quant_linear_cuda.cutlass_scaled_mv_dq(c, w, a, alpha, 0.0)
    assert torch.equal(c, _convert(torch.tensor(alpha, device="cuda") * acc, dtype))


def _tile(m, n, k):
    import ctypes
    from quamba_b200 import _lib
    out = [ctypes.c_int32() for _ in range(3)]
    _lib.check(_lib.lib().qb_gemm_tile(m, n, k, *map(ctypes.byref, out)))
    return tuple(v.value for v in out)                            # rows, columns, splits


def test_tile_columns_are_mma_shapes():
    """The int8 MMA of a CTA pair takes multiples of 32 columns, that of one CTA multiples of 16; both up to 256."""
    for m in (9, 16, 65, 128, 129, 300, 512, 777, 1024, 2048, 3000, 4096, 8192, 16384):
        for n in (16, 64, 192, 320, 768, 1536, 2560, 3024, 4096, 5120, 8192, 8512, 10240, 10576, 18560, 50288):
            rows, cols, splits = _tile(m, n, 2560)
            assert 64 <= cols <= 256 and cols % (16 if rows == 128 else 32) == 0, (m, n, rows, cols)
            assert rows == (128 if m <= 128 else 256) and splits in ((1, 2, 4, 8) if m <= 128 else (1,)), (m, n, rows, splits)


@pytest.mark.parametrize("m,n,k,splits", [
    (16, 4096, 1536, 2), (128, 4736, 1536, 2),                                            # tiles of 64 columns
    (9, 2560, 1040, 4), (65, 3000, 1536, 4), (128, 4096, 2048, 4), (16, 4736, 4096, 4),   # 80, 96, 128 and 144; N off the tile, K with a tail
    (9, 192, 5136, 8), (65, 1536, 5136, 8), (33, 2000, 5136, 8), (128, 2304, 5136, 8),    # 64, 112, 144 and 160
    (33, 768, 528, 1)])                                                                   # too short to cut
def test_k_split_equals_the_exact_product(m, n, k, splits):
    """Integer sums are exact in any order, so the only roundings are int32 -> fp32, the two scale products and the conversion, the
    same on both sides.  Rows of A and C with a pitch of their own, and rows of C whose tail vector stores cannot take."""
    assert _tile(m, n, k)[2] == splits
    a, w, acc, g = _operands(m, k, n)
    apitch = torch.empty((m, k + 32), dtype=torch.int8, device="cuda")[:, :k]
    apitch.copy_(a)
    for rows in (1, m):
        sa = torch.rand((rows, 1), device="cuda", generator=g) * 4e-3 + 1e-3
        sb = torch.rand((1, n), device="cuda", generator=g) * 4e-3 + 1e-3
        want = sa * (sb * acc)
        for dtype in (torch.int8, torch.float16, torch.bfloat16):
            c = torch.zeros((m, -(-n // 16) * 16 + 16), dtype=dtype, device="cuda")
            ops.quant_linear_cuda.cutlass_scaled_mm_dq(c[:, :n], apitch, w.t(), sa, sb)
            assert torch.equal(c[:, :n], _convert(want, dtype)) and not c[:, n:].any(), (rows, dtype)


@pytest.mark.parametrize("m", [65, 129, 300, 515])
@pytest.mark.parametrize("per_channel", [True, False])
def test_row_and_column_tails_of_every_output(m, per_channel):
    """Pair tiles (and one-CTA tiles at 65 rows) with rows and columns left over: bf16 outputs and the transposed form, neither of
    which leaves by TMA, next to the row-major ones that do."""
    from quamba_b200.modules import W4A8B16O16Linear
    k, n = 640, 832
    a, w, acc, g = _operands(m, k, n)
    sa, sb = torch.rand((m, 1), device="cuda", generator=g) * 4e-3 + 1e-3, torch.rand((1, n), device="cuda", generator=g) * 4e-3 + 1e-3
    for dtype in (torch.int8, torch.float16, torch.bfloat16):
        c = torch.empty((m, n), dtype=dtype, device="cuda")
        ops.quant_linear_cuda.cutlass_scaled_mm_dq(c, a, w.t(), sa, sb)
        assert torch.equal(c, _convert(sa * (sb * acc), dtype))
    lin = W4A8B16O16Linear(k, n, device="cuda")
    lin.weight.random_(-2 ** 31, 2 ** 31 - 1, generator=g)
    lin.s_channel.uniform_(1e-3, 2e-3, generator=g)
    if per_channel:
        lin.s_group = torch.empty(0, dtype=torch.float16, device="cuda")
    else:
        lin.s_group.uniform_(8.0, 15.5, generator=g)
    prep = lin.prepared()
    acc = (a.double() @ prep.need_w8().double().t()).float()
    want = (acc * prep.sc) * sa
    for transpose in (False, True):
        for out_int8, dtype in ((True, torch.int8), (False, torch.float16)):
            got = ops.w4a8_linear(a, prep, sa.reshape(-1), transpose, out_int8)
            assert torch.equal(got.t() if transpose else got, _convert(want, dtype)), (transpose, dtype)
    ops._lib.read_device_status(torch.cuda.current_stream().cuda_stream)


@pytest.mark.parametrize("m,n,k", [(300, 512, 256), (65, 9600, 256), (16, 768, 1536), (5, 256, 256)])   # pair, one CTA, K split, dp4a
def test_scales_that_are_not_finite(m, n, k):
    """A product that is not a number becomes the int8 0 and an infinite one the end of the range, whichever form the size selects."""
    a, w, acc, g = _operands(m, k, n)
    sa, sb = torch.rand((m, 1), device="cuda", generator=g) * 4e-3 + 1e-3, torch.rand((1, n), device="cuda", generator=g) * 4e-3 + 1e-3
    inf, nan = float("inf"), float("nan")
    for i, v in enumerate((nan, inf, -inf, 1e38, -3e38)):
        sb[0, 3 + 17 * i] = v
        sa[min(i, m - 2), 0] = (nan, inf, -inf, 0.0, 1e38)[i]
    r = sa * (sb * acc)
    assert r.isnan().any() and r.isinf().any()
    want = torch.clamp(torch.round(r), -128, 127).nan_to_num(nan=0.0).to(torch.int8)
    c = torch.empty((m, n), dtype=torch.int8, device="cuda")
    ops.quant_linear_cuda.cutlass_scaled_mm_dq(c, a, w.t(), sa, sb)
    assert torch.equal(c, want)
    c16 = torch.empty((m, n), dtype=torch.float16, device="cuda")
    ops.quant_linear_cuda.cutlass_scaled_mm_dq(c16, a, w.t(), sa, sb)
    assert torch.equal(c16.isnan(), r.isnan()) and torch.equal(c16.nan_to_num(), r.half().nan_to_num())
