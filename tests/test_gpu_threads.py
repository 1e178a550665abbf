"""Several host threads, each on a stream of its own, in a process whose first calls of the library they make at the same time: every
call equals the same call made alone afterwards."""
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

SCRIPT = """
import sys, threading
import torch
from quamba_b200 import ops
from test_gpu_native_layer import _layer, _mamba1_layer
sys.setswitchinterval(1e-5)
g = torch.Generator(device="cuda").manual_seed(1)
ri = lambda *s: torch.randint(-127, 128, s, device="cuda", generator=g).to(torch.int8)
one = lambda v: torch.tensor([[v]], device="cuda")
sa, sb, flat = one(0.01), one(0.01), torch.tensor([0.01], device="cuda")
big, few, w, wk = ri(300, 512), ri(16, 4096), ri(512, 512), ri(768, 4096)
row, st, x = torch.randn(64, 5120, device="cuda", generator=g).half(), ri(64, 16, 64, 128), ri(64, 16, 64)
dt, A, bc = ri(64, 16)[:, :, None].expand(64, 16, 64), ri(16).abs()[:, None, None].expand(16, 64, 128), ri(64, 1, 128)

def mm(a, b):
    c = torch.empty(a.shape[0], b.shape[0], dtype=torch.int8, device="cuda")
    ops.quant_linear_cuda.cutlass_scaled_mm_dq(c, a, b.t(), sa, sb)
    return c

def update():
    s = st.clone()
    return torch.cat([ops.quant_sscan_update_triton(s, x, flat, dt, flat, A, flat, flat, bc, flat, bc, flat).flatten().float(), s.flatten().float()])

def scan(batch):
    d, L = 512, 40
    u = ri(batch, d, L)
    args = (u, flat, u, flat, A1, flat, bc1[:batch], flat, bc1[:batch], flat, flat, None, None, u, flat, None, None, True)
    return lambda: ops.quant_sscan_cuda.fwd(*args)[0]

A1, bc1 = ri(512, 16).abs(), ri(64, 16, 40)
layers = [] if len(sys.argv) < 2 else [_layer("w4", False), _mamba1_layer("w8")]
for m in [m for l in layers for m in l.modules() if hasattr(m, "prepared")]:      # a weight's copies are built on the stream of their first use
    m.prepared().need_w8()
h = torch.randn(2, 70, 256, device="cuda", generator=g).half()
calls = [lambda: mm(big, w), lambda: mm(few, wk), lambda: ops.quant_hadamard.fast_hadamard_transform_40N(row, 0.1), update, scan(3)]
calls += [lambda l=l: l(h, None)[0] for l in layers]
torch.cuda.synchronize()
got, errors, gate = {}, [], threading.Barrier(2 * len(calls))

def work(i):
    try:
        with torch.cuda.stream(torch.cuda.Stream()):
            gate.wait()
            got[i] = [calls[i % len(calls)]() for _ in range(20)]
            torch.cuda.current_stream().synchronize()
    except Exception as e:
        errors.append(repr(e))

threads = [threading.Thread(target=work, args=(i,)) for i in range(2 * len(calls))]
[t.start() for t in threads]
[t.join() for t in threads]
assert not errors, errors
for i, outs in got.items():
    want = calls[i % len(calls)]()
    assert all(torch.equal(o, want) for o in outs), i
ops._lib.read_device_status(torch.cuda.current_stream().cuda_stream)
print("same")
"""


@pytest.mark.parametrize("with_layers", [False, True])
def test_first_calls_from_many_threads(with_layers):
    tests = Path(__file__).resolve().parent
    path = f"import sys; sys.path[:0] = [{str(tests.parent)!r}, {str(tests)!r}]\n"
    r = subprocess.run([sys.executable, "-c", path + SCRIPT] + ["layers"] * with_layers, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "same" in r.stdout, r.stderr[-2000:]
