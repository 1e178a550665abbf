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
