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
