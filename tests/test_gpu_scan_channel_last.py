"""The channel-last Mamba1 scan (csrc/sscan_cl.cu) in each of its forms against the sequence-last kernel on the same inputs: enough
rows for two channels a lane, with ranges cut in the middle of a sequence and states handed from one CTA to the next, then one,
two and four lanes a channel, then segments.

Both kernels accumulate in fp32 and round once to fp16, so an output differs by one fp16 step (2^-10 of it) where the sums fall on
either side of a tie, and next to zero by the fp32 error of sums whose terms cancel; an int8 state differs by one at a tie."""
import pytest
import torch

from helpers import launched
from quamba_b200 import _lib, ops

pytestmark = pytest.mark.gpu
N = 16


def _inputs(B, d, L, seed=0, z=True, D=True, bias=True):
    g = torch.Generator(device="cuda").manual_seed(seed + B + d + L)
    code = lambda *s: torch.empty(s, device="cuda").normal_(0.0, 36.0, generator=g).round_().clamp_(-127, 127).to(torch.int8)
    one = lambda v: torch.tensor([v], device="cuda")
    # rows of B and C stand side by side, as x_proj writes them, and z beside the conv's input
    xd, zx = code(B, L, 3 * N), code(B, L, 2 * d) if z else None
    return dict(u=code(B, L, d), dt=code(B, L, d), z=zx[..., d:] if z else None, Bm=xd[..., N:2 * N], Cm=xd[..., 2 * N:], A=code(d, N).abs(),
                D=code(d) if D else None, bias=code(d) // 2 - 70 if bias else None, su=one(0.025), sdt=one(0.03), sz=one(0.03), sB=one(0.03), sC=one(0.031),
                sA=one(0.02), sD=one(0.008), sb=one(0.05), sst=one(0.004))


def _sequence_last(c):
    t = lambda v: None if v is None else v.transpose(1, 2).contiguous()
    return ops.quant_sscan_cuda.fwd(t(c["u"]), c["su"], t(c["dt"]), c["sdt"], c["A"], c["sA"], t(c["Bm"]), c["sB"], t(c["Cm"]), c["sC"], c["sst"], c["D"],
                                    c["sD"], t(c["z"]), c["sz"], c["bias"], c["sb"], True)


def _channel_last(c, workspace=True):
    B, L, d = c["u"].shape
    out = torch.full((B, L, d), float("nan"), dtype=torch.float16, device="cuda")
    xs = torch.full((B, d, -(-L // 2048), N), -128, dtype=torch.int8, device="cuda")
    fin = torch.full((B, d, N), -128, dtype=torch.int8, device="cuda")
    n = _lib.lib().qb_sscan_fwd_workspace_bytes(B, d) if workspace else 0
    ws = torch.full((max(n, 1),), 0xA5, dtype=torch.uint8, device="cuda")
    p = lambda t: None if t is None else t.data_ptr()
    st = lambda name, t: {} if t is None else {f"{name}_sb": t.stride(0), f"{name}_sl": t.stride(1)}
    args = _lib.make("qb_sscan_fwd_args", u=p(c["u"]), delta=p(c["dt"]), z=p(c["z"]), Bm=p(c["Bm"]), Cm=p(c["Cm"]), A_log=p(c["A"]), D=p(c["D"]),
                     delta_bias=p(c["bias"]), u_scale=p(c["su"]), delta_scale=p(c["sdt"]), z_scale=p(c["sz"]), B_scale=p(c["sB"]), C_scale=p(c["sC"]),
                     A_scale=p(c["sA"]), D_scale=p(c["sD"]), delta_bias_scale=p(c["sb"]), ssm_state_scale=p(c["sst"]), out=p(out), x_states=p(xs), batch=B,
                     dim=d, seqlen=L, dstate=N, n_groups=1, delta_softplus=1, channel_last=1, final_state=p(fin), workspace=p(ws) if n else None,
                     workspace_bytes=n, **st("u", c["u"]), **st("delta", c["dt"]), **st("z", c["z"]), **st("B", c["Bm"]), **st("C", c["Cm"]))
    ops._run("qb_sscan_fwd", args, c["u"])
    return out, xs, fin


def _close(got, want):
    y, xs, fin = got
    wy, wxs = want
    assert torch.equal(fin, xs[:, :, -1])
    assert torch.allclose(y.float(), wy.float(), rtol=2 ** -10 * 1.1, atol=1e-4 * wy.float().abs().max().item())
    diff = (xs.int() - wxs.int()).abs()
    assert diff.max() <= 1 and (diff != 0).float().mean() <= 1e-3
    _lib.read_device_status(torch.cuda.current_stream().cuda_stream)


@pytest.mark.parametrize("B,d,L,kernel", [
    (119, 512, 5, "wide"), (150, 512, 37, "wide"), (150, 512, 2055, "wide"),     # 952 rows of 64 channels: one each; 1200 on 1184 warps: cut
    (16, 5120, 130, "wide"), (1200, 36, 29, "wide"), (601, 66, 2049, "wide"),    # channels left over in the last group
    (593, 200, 33, "wide"), (2400, 64, 41, "wide"),                              # two rows a warp
    (80, 511, 40, "<1, false>"), (40, 1024, 37, "<1, false>"), (3, 512, 31, "<1, false>"), (20, 1024, 2053, "<2, false>"), (7, 3001, 33, "<2, false>"),
    (10, 1024, 2050, "<4, false>"), (1, 12288, 39, "<4, false>"), (1, 1536, 4100, "<4, true>"), (2, 100, 32, "<4, true>"), (3, 1000, 515, "<4, true>")])
def test_each_form_against_the_sequence_last_kernel(B, d, L, kernel):
    c = _inputs(B, d, L)
    assert launched(lambda: _channel_last(c), "sscan_cl_wide_kernel" if kernel == "wide" else "sscan_cl_kernel" + kernel)
    _close(_channel_last(c), _sequence_last(c))


@pytest.mark.parametrize("B,d,L", [(160, 512, 45), (40, 1024, 45), (2, 512, 45)])
@pytest.mark.parametrize("z,D,bias", [(False, True, True), (True, False, True), (True, True, False), (False, False, False)])
def test_without_gate_skip_or_bias(B, d, L, z, D, bias):
    c = _inputs(B, d, L, 1, z, D, bias)
    _close(_channel_last(c), _sequence_last(c))


def test_without_workspace_the_rows_run_in_waves():
    c = _inputs(160, 512, 45, 2)
    assert launched(lambda: _channel_last(c, False), "sscan_cl_kernel<1, false>")
    _close(_channel_last(c, False), _sequence_last(c))


def test_hand_over_on_two_streams():
    """Two calls that hand states over, at the same time and again on the same buffers' successors: each equals itself alone."""
    cs = [_inputs(170, 512, 200, s) for s in (3, 4)]
    want = [_channel_last(c) for c in cs]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    for _ in range(20):
        got = []
        for c, s in zip(cs, streams):
            with torch.cuda.stream(s):
                got.append(_channel_last(c))
        torch.cuda.synchronize()
        for a, b in zip(got, want):
            assert all(torch.equal(x, y) for x, y in zip(a, b))
    _lib.read_device_status(torch.cuda.current_stream().cuda_stream)
