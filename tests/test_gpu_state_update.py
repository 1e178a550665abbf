"""The decode-step state update at the batch sizes of serving, where every warp walks its own tiles of state rows: against the oracle
and against the CTA-tile kernel, with what a head shares and what a row has of its own, at ragged head counts."""
import pytest
import torch

from helpers import launched
from oracle import update as oupd
from quamba_b200 import _lib, ops

pytestmark = pytest.mark.gpu


def _case(B, H, P, G, grouped, seed=0, z=False, D="head", dt="head", bias="head", i8_bias=False, A="head"):
    """Inputs on the CPU; dt, D, bias and A_log one per head (expanded, as the module passes them) or one per row."""
    g = torch.Generator().manual_seed(seed + B * 131 + H * 7 + P)
    N = 128
    ri8 = lambda *s: torch.randint(-127, 128, s, generator=g, dtype=torch.int32).to(torch.int8)
    per = lambda kind, t_head, t_row: t_head().unsqueeze(-1) if kind == "head" else t_row()
    c = dict(state=ri8(B, H, P, N), x=ri8(B, H, P), Bm=ri8(B, G, N), Cm=ri8(B, G, N), grouped=grouped,
             dt=per(dt, lambda: ri8(B, H), lambda: ri8(B, H, P)), A=per(A, lambda: ri8(H), lambda: ri8(H, P)),
             D=None if D is None else per(D, lambda: ri8(H), lambda: ri8(H, P)), z=ri8(B, H, P) if z else None,
             sdt=torch.tensor(0.02), sA=torch.tensor(0.015), sD=torch.tensor(0.01), sz=torch.tensor(0.03), sb=None)
    if i8_bias:
        c["bias"], c["sb"] = per(bias, lambda: ri8(H), lambda: ri8(H, P)), torch.tensor(0.02)
    else:
        c["bias"] = per(bias, lambda: (torch.rand(H, generator=g) * 2 - 4).half(), lambda: (torch.rand(H, P, generator=g) * 2 - 4).half())
    if grouped:
        hpg, HG, DG = H // G, 2, 4
        c["hgr"] = torch.tensor([[max(1, hpg // 3), hpg]] * G, dtype=torch.int32)
        cut = [[P // 4 + 1, P // 2 - 1, P - 3, P], [2, 3, P // 2 + 5, P]]            # boundaries on no multiple of four
        c["dgr"] = torch.tensor([cut] * G, dtype=torch.int32)
        c["xs"] = torch.rand(G, HG, DG, generator=g) * 0.02 + 0.01
        c["ss"] = torch.rand(G, HG, DG, N, generator=g) * 0.01 + 0.005
        c["sB"], c["sC"] = torch.rand(G, generator=g) * 0.02 + 0.01, torch.rand(G, generator=g) * 0.02 + 0.01
    else:
        c["hgr"] = c["dgr"] = None
        c["xs"], c["ss"], c["sB"], c["sC"] = torch.tensor([0.02]), torch.tensor([0.01]), torch.tensor([0.015]), torch.tensor([0.017])
    return c


def _args(c, move):
    B, H, P, N = c["state"].shape
    d = {k: move(v) if torch.is_tensor(v) else v for k, v in c.items()}
    wide = lambda t, *s: None if t is None else t.expand(*s)
    lead = [d["x"], d["xs"]] + ([d["hgr"], d["dgr"]] if c["grouped"] else [])
    tail = [d["bias"].expand(H, P)] + ([] if c["grouped"] else [d["sb"]]) + [True]
    return d["state"].clone(), lead + [wide(d["dt"], B, H, P), d["sdt"], d["A"].unsqueeze(-1).expand(H, P, N), d["sA"], d["ss"], d["Bm"], d["sB"], d["Cm"],
                                       d["sC"], wide(d["D"], H, P), d["sD"] if d["D"] is not None else None, d["z"], d["sz"] if d["z"] is not None else None] + tail


def _device(c):
    st, args = _args(c, lambda t: t.cuda())
    y = (ops.quamba2_sscan_update_triton if c["grouped"] else ops.quant_sscan_update_triton)(st, *args)
    return y, st


def _check(c, kernel):
    assert launched(lambda: _device(c), kernel), "another kernel took the call"
    st, args = _args(c, lambda t: t)
    y_ref, _ = (oupd.quamba2_sscan_update if c["grouped"] else oupd.quant_sscan_update)(st, *args)
    y, got = _device(c)
    with _lib.path_override(_lib.PATH_UPDATE_CTA_TILES):
        y_t, got_t = _device(c)
    _lib.read_device_status(torch.cuda.current_stream().cuda_stream)
    scale = y_ref.float().abs().max().item()
    for out, state in ((y, got), (y_t, got_t)):
        assert torch.allclose(out.cpu().float(), y_ref.float(), rtol=2e-3, atol=1e-3 * scale)    # one fp16 rounding each, sums of 128 in fp32
        d = (state.cpu().int() - st.int()).abs()
        assert d.max() <= 1 and (d != 0).float().mean() <= 1e-3                                  # a tie may round either way


@pytest.mark.parametrize("B,H,P,G,z,D", [
    (8, 80, 64, 1, False, "head"), (13, 48, 64, 2, True, "head"), (5, 131, 32, 1, False, None), (9, 72, 96, 8, True, "head")])
@pytest.mark.parametrize("grouped", [False, True])
def test_scalars_of_a_head(B, H, P, G, z, D, grouped):
    if grouped and B * H * P < 512 * 32:
        B *= 2
    _check(_case(B, H, P, G, grouped, z=z, D=D), "sscan_update_warp_kernel")


@pytest.mark.parametrize("B,H,P,G,z,dt,bias,i8_bias,A,D", [
    (8, 80, 64, 1, False, "head", "head", False, "head", "row"),          # D per channel, the rest per head
    (8, 80, 64, 2, True, "row", "head", True, "head", "head"), (7, 45, 96, 1, False, "head", "row", True, "head", "row"),
    (6, 51, 32, 1, False, "head", "head", False, "row", None), (9, 24, 64, 8, True, "row", "row", False, "row", "row"),
    (7, 43, 48, 1, False, "head", "head", False, "head", "head"), (5, 30, 16, 2, True, "row", "row", True, "row", "row"),    # 16-row tiles
    (1, 1, 48, 1, False, "row", "row", False, "row", "row")])
def test_scalars_of_a_row(B, H, P, G, z, dt, bias, i8_bias, A, D):
    _check(_case(B, H, P, G, False, seed=1, z=z, D=D, dt=dt, bias=bias, i8_bias=i8_bias, A=A), "sscan_update_warp_kernel")


def test_channel_D_with_grouped_scales():
    _check(_case(8, 80, 64, 1, True, seed=2, D="row"), "sscan_update_warp_kernel")


@pytest.mark.parametrize("grouped", [False, True])
def test_scales_written_by_the_launch_before(grouped):
    """The update is launched as a programmatic dependent; scales that the kernel before it on the stream writes last are its scales."""
    c = _case(16, 80, 64, 1, grouped, seed=3)
    want_y, want_st = _device(c)
    st, args = _args(c, lambda t: t.cuda())
    names = [i for i, a in enumerate(args) if torch.is_tensor(a) and a.dtype == torch.float32]
    padded = lambda t: torch.nn.functional.pad(t.reshape(-1), (0, -t.numel() % 4))              # 16-byte aligned, as a tensor is
    fresh = torch.cat([torch.zeros(1 << 24, device="cuda")] + [padded(args[i]) for i in names])
    fn = ops.quamba2_sscan_update_triton if grouped else ops.quant_sscan_update_triton
    for _ in range(5):
        buf, state, at = torch.full_like(fresh, float("nan")), st.clone(), 1 << 24
        torch.cuda.synchronize()
        for i in names:                                      # each scale a view of the end of the buffer
            n, shape = args[i].numel(), args[i].shape
            args[i], at = buf[at:at + n].view(shape), at + -(-n // 4) * 4
        buf.copy_(fresh)
        y = fn(state, *args)
        assert torch.equal(y, want_y) and torch.equal(state, want_st)
