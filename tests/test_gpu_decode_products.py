"""The decode-sized W4A8 product at the edge of its shared-memory request: with five columns a warp in one pass, four rows of 2048 and
their staged weights are exactly the 48 KB a kernel gets without asking for more, and its static shared memory comes on top."""
import pytest
import torch

from quamba_b200 import ops
from quamba_b200.modules import W4A8B16O16Linear

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [2, 3, 4])
@pytest.mark.parametrize("k", [1920, 2048, 2176])
def test_decode_product_at_48_kb_of_shared_memory(k, rows):
    g = torch.Generator(device="cuda").manual_seed(k + rows)
    lin = W4A8B16O16Linear(k, 9472, device="cuda")
    lin.weight.random_(-2 ** 31, 2 ** 31 - 1, generator=g)
    lin.s_group = torch.empty(0, dtype=torch.float16, device="cuda")
    lin.input_scale.fill_(0.03)
    lin.s_channel.uniform_(1e-3, 2e-3, generator=g)
    a = torch.randint(-127, 128, (rows, k), device="cuda", generator=g).to(torch.int8)
    prep = lin.prepared()
    assert prep.per_channel
    assert torch.equal(ops.decode_linear(a, prep, lin.input_scale), ops.w4a8_linear(a, prep, lin.input_scale, out_int8=False))
