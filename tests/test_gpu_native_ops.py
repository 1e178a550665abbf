"""Argument forms of the operators at their native entry (csrc/binding.cpp)."""
import pytest
import torch

from quamba_b200 import ops

pytestmark = pytest.mark.gpu


def test_partial_slots_of_one_row():
    """One row has no row pitch: a view whose row stride says otherwise is still contiguous."""
    g = torch.Generator(device="cuda").manual_seed(2)
    buf = torch.randn(3, 4, 256, device="cuda", generator=g).half()
    slots = torch.as_strided(buf, (3, 1, 256), (1024, 512, 1))
    assert slots[0].is_contiguous() and slots.stride(1) != 256
    w = torch.ones(256, device="cuda", dtype=torch.float16)
    call = lambda s: ops._qlayer_norm_fwd(s[0], w, None, 1e-5, static_out_scale=0.05, is_rms_norm=True, partials=(s, -1, None))[0]
    assert torch.equal(call(slots), call(slots.contiguous()))
