"""The one-call form of a layer (csrc/binding_layers.cpp) against the same layer walked module by module, which a hook on a
sub-module selects: the same launches on the same data, so outputs and both caches are equal bit for bit."""
import pytest
import torch

from quamba_b200 import InferenceParams

pytestmark = pytest.mark.gpu


def _layer(weights, grouped):
    from quamba_b200 import calibrate as cal
    fm = cal.Mamba2LMFloat(d_model=256, n_layer=1, vocab_size=320, seed=5, w4_group_size={"w4": -1, "w4g128": 128, "w8": None}[weights])
    ids = torch.randint(0, 320, (2, 64), generator=torch.Generator().manual_seed(5))
    scales = cal.calibrate(fm, [ids])
    q = cal.quantize_model(fm, scales, w_bits=8 if weights == "w8" else 4).to("cuda")
    layer = q.backbone.layers[0]
    if grouped:
        m, heads = layer.mixer, layer.mixer.nheads
        hr = torch.tensor([[heads // 2, heads]], dtype=torch.int32, device="cuda")
        dr = torch.tensor([[[16, 64], [32, 64]]], dtype=torch.int32, device="cuda")
        xs = m.conv1d.x_out_scales.reshape(1, 1, 1) * torch.tensor([[[0.8, 1.0], [1.1, 1.2]]], device="cuda")
        for mod in (m.conv1d, m.qchunk_scan):
            mod.x_head_group_range, mod.x_dim_group_range = hr, dr
        m.conv1d.x_out_scales, m.qchunk_scan.x_scales = xs, xs
        m.qchunk_scan.ssm_state_scale = m.qchunk_scan.ssm_state_scale.reshape(1, 1, 1, 1).expand(1, 2, 2, 128).contiguous()
    return layer


def _run(layer, batch, length, decode, with_residual, native):
    g = torch.Generator(device="cuda").manual_seed(batch * 1000 + length)
    h = torch.randn(batch, length, 256, device="cuda", generator=g).half()
    r = torch.randn(batch, length, 256, device="cuda", generator=g) if with_residual else None
    conv, ssm = layer.allocate_inference_cache(batch, 8)
    conv.copy_(torch.randint(-100, 100, conv.shape, device="cuda", generator=g))
    ssm.copy_(torch.randint(-100, 100, ssm.shape, device="cuda", generator=g))
    params = InferenceParams(max_seqlen=8, max_batch_size=batch, seqlen_offset=int(decode), key_value_memory_dict={0: (conv, ssm)})
    hook = None if native else layer.mixer.conv1d.register_forward_hook(lambda *a: None)
    try:
        if native:
            taken = layer.mixer.native_layer(layer.norm, h, r, True, InferenceParams(max_seqlen=8, max_batch_size=batch))
            assert taken is not None, "the layer was not taken by the one-call form"
        out, res = layer(h, r, inference_params=params)
    finally:
        if hook is not None:
            hook.remove()
    return out, res, conv, ssm


@pytest.mark.parametrize("weights,grouped", [("w4", False), ("w4g128", True), ("w8", False), ("w8", True)])
@pytest.mark.parametrize("batch,length,decode,with_residual", [(1, 2, False, True), (2, 3, False, False), (1, 4, False, True), (2, 133, False, True),
                                                               (1, 1, True, True), (3, 1, True, True), (9, 1, True, False)])
def test_one_call_layer_equals_the_module_walk(weights, grouped, batch, length, decode, with_residual):
    layer = _layer(weights, grouped)
    for got, want in zip(_run(layer, batch, length, decode, with_residual, True), _run(layer, batch, length, decode, with_residual, False)):
        assert got.dtype == want.dtype and torch.equal(got, want)


@pytest.mark.parametrize("weights", ["w8", "w4"])
@pytest.mark.parametrize("batch,length", [(1, 1), (2, 3), (1, 31), (1, 33), (2, 70), (1, 515), (1, 2048), (3, 2055), (40, 40)])
def test_mamba1_channel_last_layer_against_the_module_walk(weights, batch, length):
    """The channel-last scan (whole sequences, segments, a chunk boundary, ragged ends) against the sequence-last kernel the
    walk runs.  Both accumulate in fp32; the scan outputs differ by fp16 roundings, so an int8 activation behind the rotation
    flips in at most a few per thousand places: y within 2 % of its norm, states within one step."""
    from quamba_b200 import calibrate as cal
    fm = cal.Mamba1LMFloat(d_model=256, n_layer=1, vocab_size=320, seed=6, w4_group_size=None if weights == "w8" else 128)
    ids = torch.randint(0, 320, (1, 48), generator=torch.Generator().manual_seed(6))
    layer = cal.quantize_mamba1_model(fm, [ids], w_bits=int(weights[1])).to("cuda").backbone.layers[0]
    outs = []
    for native in (True, False):
        hook = None if native else layer.mixer.conv1d.register_forward_hook(lambda *a: None)
        g = torch.Generator(device="cuda").manual_seed(length)
        h = torch.randn(batch, length, 256, device="cuda", generator=g).half()
        params = InferenceParams(max_seqlen=8, max_batch_size=batch)
        out, res = layer(h, None, inference_params=params)
        outs.append((out.float(), res, *params.key_value_memory_dict[0]))
        if hook is not None:
            hook.remove()
    (ya, ra, ca, sa), (yb, rb, cb, sb) = outs
    assert torch.equal(ra, rb) and torch.equal(ca, cb)
    assert (ya - yb).norm() <= 0.02 * yb.norm()
    diff = (sa.int() - sb.int()).abs()
    assert diff.max() <= 1 and (diff != 0).float().mean() <= 2e-3


def _mamba1_layer(weights):
    from quamba_b200 import calibrate as cal
    fm = cal.Mamba1LMFloat(d_model=256, n_layer=1, vocab_size=320, seed=6, w4_group_size=None if weights == "w8" else 128)
    ids = torch.randint(0, 320, (1, 48), generator=torch.Generator().manual_seed(6))
    return cal.quantize_mamba1_model(fm, [ids], w_bits=int(weights[1])).to("cuda").backbone.layers[0]


def _any_layer(family, weights):
    return _layer(weights, False) if family == "mamba2" else _mamba1_layer(weights)


def _call(layer, batch, length, decode, caches=None):
    g = torch.Generator(device="cuda").manual_seed(length)
    params = InferenceParams(max_seqlen=8, max_batch_size=batch, seqlen_offset=int(decode))
    params.key_value_memory_dict[0] = caches if caches is not None else layer.allocate_inference_cache(batch, 8)
    out, res = layer(torch.randn(batch, length, 256, device="cuda", generator=g).half(), None, inference_params=params)
    return (out, res, *params.key_value_memory_dict[0])


FOUR = [(f, w) for f in ("mamba2", "mamba1") for w in ("w4", "w8")]


@pytest.mark.parametrize("decode", [False, True])
@pytest.mark.parametrize("family,weights", FOUR)
def test_scales_in_half_precision_are_refused(family, weights, decode):
    layer = _any_layer(family, weights).half()
    with pytest.raises(RuntimeError, match="float32"):
        _call(layer, 2, 1 if decode else 5, decode)


@pytest.mark.parametrize("decode", [False, True])
@pytest.mark.parametrize("part", ["in_proj", "conv1d", "scan", "out_proj", "norm"])
@pytest.mark.parametrize("family,weights", FOUR)
def test_a_part_left_on_the_cpu_is_refused(family, weights, part, decode):
    layer = _any_layer(family, weights)
    m = layer.mixer
    scan = m.qchunk_scan if family == "mamba2" else m.selective_scan
    {"scan": scan, "norm": layer.norm}.get(part, None if part in ("scan", "norm") else getattr(m, part, None)).cpu()
    with pytest.raises(RuntimeError, match="CUDA"):
        _call(layer, 2, 1 if decode else 5, decode)


@pytest.mark.parametrize("family,weights", FOUR)
def test_caches_elsewhere_than_the_input_are_filled_by_the_walk(family, weights):
    layer = _any_layer(family, weights)
    want = _call(layer, 2, 7, False)
    conv, ssm = layer.allocate_inference_cache(2, 8)
    got = _call(layer, 2, 7, False, (conv, ssm.cpu()))
    tol = 0 if family == "mamba2" else 1                    # (the Mamba1 walk runs the sequence-last scan)
    assert torch.equal(got[2], want[2]) and (got[3].int() - want[3].cpu().int()).abs().max() <= tol


@pytest.mark.parametrize("weights", ["w8", "w4"])
def test_mamba1_prefill_refuses_a_projection_without_the_sequence_last_form(weights):
    """The parallel classes scale every column by itself and have no to_seqlen_last; a decode step takes them."""
    from quamba_b200 import W4A8B8O8LinearParallel, W8A8B8O8LinearParallel
    layer = _mamba1_layer(weights)
    old = layer.mixer.in_proj
    new = (W8A8B8O8LinearParallel if weights == "w8" else W4A8B8O8LinearParallel)(256, old.out_features, device="cuda")
    new.weight = old.weight
    if weights == "w8":
        new.a, new.b = old.a, old.b * torch.linspace(0.5, 1.5, new.b.numel(), device="cuda")[None]
    else:
        new.s_channel, new.s_group, new.input_scale = old.s_channel, old.s_group, old.input_scale
    layer.mixer.in_proj = new
    with pytest.raises(TypeError if weights == "w4" else AttributeError):
        _call(layer, 2, 5, False)
    got = _call(layer, 3, 1, True)
    hook = layer.mixer.conv1d.register_forward_hook(lambda *a: None)
    want = _call(layer, 3, 1, True)
    hook.remove()
    for a, b in zip(got, want):
        assert torch.equal(a, b)


@pytest.mark.parametrize("decode", [False, True])
@pytest.mark.parametrize("family,weights", FOUR)
def test_caches_at_an_odd_address(family, weights, decode):
    """Views of a caller's buffer that start on any byte, the conv cache with its channels innermost."""
    layer = _any_layer(family, weights)
    conv, ssm = layer.allocate_inference_cache(2, 8)
    dim = conv.shape[1]
    g = torch.Generator(device="cuda").manual_seed(1)
    odd = lambda n: torch.randint(-90, 90, (n + 1,), device="cuda", generator=g).to(torch.int8)[1:]
    c1, s1 = odd(2 * 4 * dim).view(2, 4, dim).transpose(1, 2), odd(ssm.numel()).view(ssm.shape)
    c2, s2 = conv.copy_(c1), ssm.copy_(s1)
    got, want = _call(layer, 2, 1 if decode else 6, decode, (c1, s1)), _call(layer, 2, 1 if decode else 6, decode, (c2, s2))
    assert torch.equal(c1, c2) and (s1.int() - s2.int()).abs().max() <= 1          # (an unaligned state takes the plain update kernel)
    assert (got[0].float() - want[0].float()).norm() <= 0.02 * want[0].float().norm()


def test_mamba1_sizes_beyond_the_channel_last_scan():
    """It counts the elements of a sequence in 31 bits and the sequences in 16; the sequence-last kernel has no such limits."""
    layer = _mamba1_layer("w8")
    for shape in ((1, 1 << 21, 256), (65536, 1, 256)):
        u = torch.empty(shape, dtype=torch.int8, device="cuda")
        assert layer.mixer.native_layer(None, u, None, False, None) is None, shape
    g = torch.Generator(device="cuda").manual_seed(4)
    h = torch.randn(65537, 1, 256, device="cuda", generator=g).half()
    for part in (slice(0, 64), slice(65500, 65537)):
        want = layer(h[part], None)[0].float()
        got = layer(h, None)[0][part].float()
        assert (got - want).norm() <= 0.02 * want.norm()


@pytest.mark.parametrize("through_block", [True, False])
@pytest.mark.parametrize("family,weights", FOUR)
def test_methods_of_a_subclass_or_an_instance_are_called(family, weights, through_block):
    """What a user overrides, in a subclass of the mixer or on one module, runs in prefill and in decode."""
    layer = _any_layer(family, weights)
    m = layer.mixer
    scan = m.qchunk_scan if family == "mamba2" else m.selective_scan
    calls = []

    def call(decode):
        if through_block:
            return _call(layer, 2, 1 if decode else 5, decode)
        params = InferenceParams(max_seqlen=8, max_batch_size=2, seqlen_offset=int(decode))
        return m(torch.ones(2, 1 if decode else 5, 256, dtype=torch.int8, device="cuda"), inference_params=params)

    def watched(obj, name):
        old = getattr(obj, name)
        setattr(obj, name, lambda *a, **k: (calls.append(name), old(*a, **k))[1])

    cases = [(m, "step", True), (m.conv1d, "update", True), (scan, "update", True)]
    if family == "mamba1":
        cases += [(m.in_proj, "to_seqlen_last", False), (m.dt_proj, "to_seqlen_last", False)]
    for obj, name, decode in cases:
        watched(obj, name)
        call(decode)
        assert calls == [name], (type(obj).__name__, name)
        delattr(obj, name)
        calls.clear()

    class Mine(type(m)):
        def step(self, *a):
            calls.append("mine")
            return super().step(*a)

    m.__class__ = Mine
    call(True)
    assert calls == ["mine"]


@pytest.mark.parametrize("weights", ["w8", "w4"])
@pytest.mark.parametrize("batch", [1, 2, 9, 16, 40])
def test_mamba1_decode_against_the_module_walk(weights, batch):
    """The same operators on strided views instead of copies: the integer products are equal, the state update may take another
    kernel for the alignment of B and C."""
    layer = _mamba1_layer(weights)
    g = torch.Generator(device="cuda").manual_seed(batch)
    outs = []
    for native in (True, False):
        hook = None if native else layer.mixer.conv1d.register_forward_hook(lambda *a: None)
        conv, ssm = layer.allocate_inference_cache(batch, 8)
        g.manual_seed(batch)
        conv.copy_(torch.randint(-100, 100, conv.shape, device="cuda", generator=g))
        ssm.copy_(torch.randint(-100, 100, ssm.shape, device="cuda", generator=g))
        outs.append(_call(layer, batch, 1, True, (conv, ssm)))
        if hook is not None:
            hook.remove()
    (ya, ra, ca, sa), (yb, rb, cb, sb) = outs
    assert torch.equal(ra, rb) and torch.equal(ca, cb)
    diff = (sa.int() - sb.int()).abs()
    assert diff.max() <= 1 and (diff != 0).float().mean() <= 2e-3
    assert (ya.float() - yb.float()).norm() <= 0.02 * yb.float().norm()


@pytest.mark.parametrize("decode", [False, True])
@pytest.mark.parametrize("family,buffers", [
    ("mamba2", ("conv1d.bias", "conv1d.x_head_group_range", "conv1d.x_out_scales", "qchunk_scan.D", "qchunk_scan.dt_bias", "qchunk_scan.x_dim_group_range",
                "qchunk_scan.ssm_state_scale")),
    ("mamba1", ("conv1d.bias", "selective_scan.D", "selective_scan.dt_bias", "selective_scan.D_scale"))])
def test_a_buffer_left_on_the_cpu_is_refused(family, buffers, decode):
    layer = _layer("w4", True) if family == "mamba2" else _mamba1_layer("w4")
    for path in buffers:
        part, name = path.split(".")
        mod = getattr(layer.mixer, part)
        old = getattr(mod, name)
        setattr(mod, name, old.cpu())
        with pytest.raises(RuntimeError, match="CUDA"):
            _call(layer, 2, 1 if decode else 5, decode)
        setattr(mod, name, old)
    h = torch.zeros(2, 1 if decode else 5, 256, device="cuda", dtype=torch.float16)
    with pytest.raises(RuntimeError, match="CUDA"):
        layer(h, torch.zeros(h.shape))
