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


@pytest.mark.parametrize("level", ["operator", "layer"])
def test_other_python_threads_run_while_a_launch_waits(level):
    """Behind a kernel of about half a second the launch queue fills up and a launch waits for room; another thread of the process,
    which only looks at the clock, goes on meanwhile."""
    import threading
    import time
    if level == "operator":
        x = torch.zeros(1, 256, device="cuda", dtype=torch.int8)
        st, w = torch.zeros(1, 256, 4, device="cuda", dtype=torch.int8), torch.zeros(256, 4, device="cuda", dtype=torch.int8)
        call = lambda: ops.quant_causal_conv1d_cuda.update(x, st, 0.1, w, 0.1, 0.1, 0.1, None, True)
        calls = 4000
    else:
        from quamba_b200 import InferenceParams
        from test_gpu_native_layer import _layer
        m = _layer("w4", False).mixer
        u, params = torch.zeros(1, 1, 256, device="cuda", dtype=torch.int8), InferenceParams(max_seqlen=8, max_batch_size=1, seqlen_offset=1)
        call = lambda: m.native_layer(None, u, None, False, params)
        calls = 1000
    call()
    torch.cuda.synchronize()
    gap, stop = [0.0], threading.Event()

    def watch():
        last = time.perf_counter()
        while not stop.is_set():
            now = time.perf_counter()
            gap[0], last = max(gap[0], now - last), now
            time.sleep(0.001)

    t = threading.Thread(target=watch)
    t.start()
    t0 = time.perf_counter()
    torch.cuda._sleep(1_000_000_000)
    for _ in range(calls):
        call()
    torch.cuda.synchronize()
    took = time.perf_counter() - t0
    stop.set()
    t.join()
    assert took > 0.4 and gap[0] < 0.15, (took, gap[0])


def test_errors_keep_their_python_types():
    """An output that does not fit raises torch's out-of-memory error, which callers catch to retry with less."""
    x = torch.zeros(1, 256, device="cuda", dtype=torch.float16).expand(1 << 36, 256)     # 16 TB of int8 asked for
    with pytest.raises(torch.OutOfMemoryError):
        ops.quant_hadamard.fast_hadamard_transform(x, 1.0)
    y = torch.zeros(2, 256, device="cuda", dtype=torch.float16)
    assert ops.quant_hadamard.fast_hadamard_transform(y, 1.0).shape == y.shape
