"""What the framework's speed is measured on: calls that a user of the quantized Mamba models makes, over the range of sizes,
weight formats and options they are made with.

Three entry levels, all public:
  "lm"     the language model, replayed from the CUDA graphs that ``capture_prefill`` / ``capture_decode`` return
  "block"  one layer (block norm + mixer) of a model, called eagerly as ``model(ids)`` calls it, or replayed from a graph the
           user captured around it: the unit every prompt length and every batch size goes through
  "core"   the conv1d and chunk-scan modules of a Mamba2 mixer on in_proj's int8 output, for users who drop these into their
           own mixer
Models are built the way a checkpoint is loaded (constructed, then every buffer filled); the weights are random codes, the
scales are chosen so that each int8 activation fills its range without clipping.  Prefill cases are one layer deep: int8
activations that differ in a last bit grow from layer to layer, so only a single layer's outputs can be held against those of
another correct implementation.
"""
import math

import torch

from quamba_b200 import InferenceParams, QuambaConfig, QuambaLMHeadModel, QuambaMixerModel, Quamb2Conv1D, Quamba2ChunkScan

# widths of the checkpoints these layers exist for: d_inner = 2 * width is one of the supported Hadamard orders
WIDTHS = (768, 1024, 2048, 2560, 4096)
VOCAB = 50288
ACT = 4.0 / 127.0           # int8 scale of an N(0, 1) activation
OUT = 0.025                 # int8 scale of what leaves the conv
PEAK_TOKENS = 16384         # tokens of the largest prefill call (4 sequences of 4096)


def _case(name, level, family, weights, width, batch, seqlen, **more):
    c = dict(name=name, level=level, family=family, weights=weights, width=width, batch=batch, seqlen=seqlen, phase="prefill",
             layers=1, groups=1, grouped_scales=False, graph=False)
    c.update(more)
    return c


def listed():
    return [
        # greedy decoding of one sequence with the 64-layer 2.7B model, weights int4 per output channel: the interactive case
        _case("token-2.7b", "lm", "mamba2", "w4", 2560, 1, 1, phase="decode", layers=64, graph=True),
        # a few sequences at once on a checkpoint in the default weight format (int4, groups of 128)
        _case("token-2.7b-g128-x3", "lm", "mamba2", "w4g128", 2560, 3, 1, phase="decode", layers=16, graph=True),
        # batched serving: one layer's decode step for 64 sequences, captured
        _case("step-x64", "block", "mamba2", "w4", 2560, 64, 1, phase="decode", graph=True),
        # batched serving of the Mamba1 2.8B model
        _case("step-mamba1-x16", "block", "mamba1", "w8", 2560, 16, 1, phase="decode", graph=True),
        # the smallest call: an eager decode step of a small int8 model with per-head-group scales (two beams)
        _case("step-small-eager", "block", "mamba2", "w8", 768, 2, 1, phase="decode", grouped_scales=True),
        # the captured prefill of a 2048-token prompt, embedding and head included
        _case("prefill-2048", "lm", "mamba2", "w4", 2560, 1, 2048, graph=True),
        # a prompt as long as it happens to be
        _case("prefill-777-g128", "block", "mamba2", "w4g128", 2560, 1, 777),
        # a batch of prompts through an int8 model with per-head-group scales, the default of the layer class
        _case("prefill-4x2048-w8", "block", "mamba2", "w8", 2560, 4, 2048, grouped_scales=True),
        # the largest: one chunk of sequences of the 8B model's prefill (8 SSD groups)
        _case("prefill-8b-4x4096", "block", "mamba2", "w4", 4096, 4, 4096, groups=8),
        # Mamba1 2.8B, batch 16 of 1024 tokens
        _case("prefill-mamba1-16x1024", "block", "mamba1", "w8", 2560, 16, 1024),
        # a single short prompt through a small Mamba1 layer (d_inner 1536)
        _case("prefill-mamba1-512", "block", "mamba1", "w4g128", 768, 1, 512),
        # conv1d and chunk scan on their own
        _case("core-4x2048", "core", "mamba2", "w4", 2560, 4, 2048),
    ]


def _log_int(rng, lo, hi):
    return min(hi, int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))


def draw(rng):
    kind = rng.choice(("token", "step", "step", "prefill", "prefill", "prefill", "prefill-lm", "core"))
    width = rng.choice(WIDTHS)
    if kind == "token":
        c = _case("", "lm", "mamba2", rng.choice(("w4", "w4g128")), rng.choice((1024, 2048, 2560)), rng.randint(1, 4), 1,
                  phase="decode", layers=_log_int(rng, 2, 32), graph=True)
    elif kind == "step":
        family = rng.choice(("mamba2", "mamba2", "mamba1"))
        c = _case("", "block", family, rng.choice(("w4", "w4g128", "w8")), width, _log_int(rng, 1, 96), 1, phase="decode",
                  graph=rng.random() < 0.7)
    elif kind == "prefill":
        family = rng.choice(("mamba2", "mamba2", "mamba1"))
        batch = _log_int(rng, 1, 16)
        top = PEAK_TOKENS // batch // (2 if family == "mamba1" or width == 4096 else 1)
        c = _case("", "block", family, rng.choice(("w4", "w4g128", "w8")), width, batch, _log_int(rng, 5, min(4096, top)))
    elif kind == "prefill-lm":
        c = _case("", "lm", "mamba2", rng.choice(("w4", "w4g128")), rng.choice((1024, 2048, 2560)), rng.randint(1, 3),
                  _log_int(rng, 24, 3000), graph=True)
    else:
        batch = _log_int(rng, 1, 8)
        c = _case("", "core", "mamba2", "w4", width, batch, _log_int(rng, 40, min(4096, PEAK_TOKENS // batch)))
    if c["family"] == "mamba2" and c["level"] != "lm":
        c["grouped_scales"] = rng.random() < 0.35
        if width == 4096:
            c["groups"] = 8
    del c["name"]
    return c


# ---- building a model as a checkpoint would fill it -----------------------------------------------------------------------
def _codes(shape, gen, std=40.0):
    x = torch.empty(shape, dtype=torch.float16, device="cuda").normal_(0.0, std, generator=gen)
    return x.round_().clamp_(-127, 127).to(torch.int8)


def _fill_linear(lin, weights, gen, in_scale, out_std):
    """Random codes; the channel scales bring the outputs to a standard deviation of ``out_std`` (int8 steps or fp16)."""
    k, dev = lin.in_features, "cuda"
    act = 1.0 / ACT                                     # standard deviation of the int8 input
    if hasattr(lin, "s_channel"):                       # int4
        lin.weight.random_(-2 ** 31, 2 ** 31 - 1, generator=gen)
        if weights == "w4":
            lin.s_group = torch.empty(0, dtype=torch.float16, device=dev)
            w_std = 16 * 4.61
        else:
            lin.s_group.uniform_(8.0, 15.5, generator=gen)
            w_std = 4.61 * 11.9
        lin.input_scale.fill_(in_scale)
        lin.s_channel.uniform_(0.8, 1.2, generator=gen)
        lin.s_channel.mul_(out_std / (math.sqrt(k) * act * w_std * in_scale))
    else:
        lin.weight.copy_(_codes((lin.weight.shape[1], k), gen).t())
        s = out_std / (math.sqrt(k) * act * 40.0)
        lin.a.fill_(in_scale)
        lin.b.fill_(s / in_scale)
        if hasattr(lin, "alpha"):
            lin.alpha = s


def _fill_groups(conv, scan, gen):
    """Cumulative head and channel ranges with one scale per (SSD group, head group, channel group)."""
    heads = conv.x_dim // conv.x_headdim // conv.n_groups
    nh, nd = conv.x_nhead_group, conv.x_ndim_group
    hr = torch.tensor([(i + 1) * heads // nh for i in range(nh)], dtype=torch.int32, device="cuda")
    dr = torch.tensor([(i + 1) * conv.x_headdim // nd for i in range(nd)], dtype=torch.int32, device="cuda")
    for m in (conv, scan):
        m.x_head_group_range.copy_(hr.expand_as(m.x_head_group_range))
        m.x_dim_group_range.copy_(dr.expand_as(m.x_dim_group_range))
    conv.x_out_scales.uniform_(0.02, 0.03, generator=gen)
    scan.x_scales.copy_(conv.x_out_scales)
    scan.ssm_state_scale.uniform_(0.0007, 0.0014, generator=gen)


def _fill_conv_and_scan(conv, scan, gen):
    conv.x_scale = conv.B_scale = conv.C_scale = ACT
    conv.wx_scale = conv.wB_scale = conv.wC_scale = 0.4 / 40.0
    conv.bx_scale = conv.bB_scale = conv.bC_scale = 0.02 / 40.0
    conv.weight.copy_(_codes(conv.weight.shape, gen))
    conv.bias.copy_(_codes(conv.bias.shape, gen))
    if conv.x_head_group_range is not None:
        _fill_groups(conv, scan, gen)
    else:
        conv.x_out_scales.fill_(OUT)
        scan.x_scales.fill_(OUT)
        scan.ssm_state_scale.fill_(0.001)
    for name in ("B", "C"):                # one scale per SSD group, or one for all where the scales are per tensor
        s = getattr(scan, name + "_scale").fill_(OUT)
        setattr(conv, name + "_out_scales", s.clone())
    dt0 = torch.rand(scan.dt_bias.shape, device="cuda", generator=gen) * 0.099 + 0.001
    scan.dt_bias.copy_(dt0 + torch.log(-torch.expm1(-dt0)))
    scan.dt_scale.fill_(ACT)
    scan.A_log.random_(0, 128, generator=gen)
    scan.A_log_scale.fill_(math.log(16.0) / 127.0)
    scan.D.fill_(120)
    scan.D_scale.fill_(1.0 / 120.0)


def _fill_block(block, case, gen):
    m, w = block.mixer, case["weights"]
    block.norm.weight.fill_(1.0)
    block.norm.output_scale = ACT
    if case["family"] == "mamba2":
        _fill_linear(m.in_proj, w, gen, ACT, 1.0 / ACT)
        _fill_conv_and_scan(m.conv1d, m.qchunk_scan, gen)
        m.norm.weight.fill_(1.0)
        m.norm.z_scale = ACT
    else:
        _fill_linear(m.in_proj, w, gen, ACT, 1.0 / ACT)
        c, s = m.conv1d, m.selective_scan
        c.weight.copy_(_codes(c.weight.shape, gen))
        c.bias.copy_(_codes(c.bias.shape, gen))
        c.input_scale, c.weight_scale, c.bias_scale, c.output_scale = ACT, 0.4 / 40.0, 0.02 / 40.0, OUT
        _fill_linear(m.x_proj, w, gen, OUT, 1.0 / ACT)
        _fill_linear(m.dt_proj, w, gen, ACT, 1.0 / ACT)
        s.dt_bias.copy_(_codes(s.dt_bias.shape, gen, 20.0) - 70)
        s.A_log.copy_(torch.log(torch.arange(1.0, m.d_state + 1, device="cuda")).mul(127.0 / math.log(m.d_state)).round())
        s.D.fill_(127)
        for name, v in (("dt_bias_scale", 0.05), ("A_scale", math.log(m.d_state) / 127.0), ("D_scale", 1.0 / 127.0), ("u_scale", OUT),
                        ("dt_scale", ACT), ("B_scale", ACT), ("C_scale", ACT), ("z_scale", ACT), ("ssm_state_scale", 0.002)):
            getattr(s, name).fill_(v)
    m.had.x_H_scale = ACT
    _fill_linear(m.out_proj, w, gen, ACT, 1.0)


def _ssm_cfg(case):
    w4 = case["weights"] != "w8"
    if case["family"] == "mamba1":
        return dict(layer="W4A8QMamba" if w4 else "W8A8QMamba", d_state=16, d_conv=4, expand=2)
    n = 4 if case["grouped_scales"] else 0
    return dict(layer="W4A8QMamba2" if w4 else "W8A8QMamba2", d_state=128, d_conv=4, expand=2, headdim=64, ngroups=case["groups"],
                chunk_size=256, x_nhead_group=n, x_ndim_group=n)


def _caches(model, case, gen):
    """One tensor for all conv states and one for all SSM states, handed to the layers as views."""
    conv, ssm = model.layers[0].allocate_inference_cache(case["batch"], 1)
    if conv.is_contiguous():
        conv = torch.stack([conv] * case["layers"])
    else:                                  # Mamba2 keeps the channels innermost
        conv = torch.stack([conv.transpose(1, 2)] * case["layers"]).transpose(2, 3)
    ssm = torch.stack([ssm] * case["layers"])
    if case["phase"] == "decode":
        conv.copy_(_codes(conv.shape, gen))
        ssm.copy_(_codes(ssm.shape, gen))
    params = InferenceParams(max_seqlen=4096, max_batch_size=case["batch"], seqlen_offset=int(case["phase"] == "decode"),
                             key_value_memory_dict={i: (conv[i], ssm[i]) for i in range(case["layers"])})
    return params, conv, ssm


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    return {"lm": _prepare_lm, "block": _prepare_block, "core": _prepare_core}[case["level"]](case, gen)


def _prepare_lm(case, gen):
    cfg = QuambaConfig(d_model=case["width"], n_layer=case["layers"], vocab_size=VOCAB, ssm_cfg=_ssm_cfg(case),
                       embedding_cfg={"layer": "W4O16Embedding"}, lm_head_cfg={"layer": "W4A8B16O16Linear"})
    model = QuambaLMHeadModel(cfg, device="cuda")
    bb = model.backbone
    bb.embedding.weight.random_(-2 ** 31, 2 ** 31 - 1, generator=gen)
    bb.embedding.scales.uniform_(0.15, 0.25, generator=gen)
    for block in bb.layers:
        _fill_block(block, case, gen)
    bb.norm_f.weight.fill_(1.0)
    bb.norm_f.output_scale = ACT
    _fill_linear(model.lm_head, case["weights"], gen, ACT, 2.0)
    ids = torch.randint(0, VOCAB, (case["batch"], case["seqlen"]), device="cuda", generator=gen)
    if case["phase"] == "decode":
        params, conv, ssm = _caches(bb, case, gen)
        runner = model.capture_decode(case["batch"], 4096, inference_params=params)
        runner.input_ids.copy_(ids)
        return dict(level="lm", runner=runner, ids=None, caches=[conv, ssm])
    runner = model.capture_prefill(case["batch"], case["seqlen"])
    caches = [t for layer in runner.inference_params.key_value_memory_dict.values() for t in layer]
    return dict(level="lm", runner=runner, ids=ids, caches=caches)


def _prepare_block(case, gen):
    bb = QuambaMixerModel(case["width"], 1, 8, ssm_cfg=_ssm_cfg(case), device="cuda")
    block = bb.layers[0]
    _fill_block(block, case, gen)
    params, conv, ssm = _caches(bb, case, gen)
    shape = (case["batch"], case["seqlen"], case["width"])
    hidden = torch.randn(shape, device="cuda", generator=gen).half()
    residual = torch.randn(shape, device="cuda", generator=gen)
    state = dict(level="block", block=block, hidden=hidden, residual=residual, params=params, caches=[conv, ssm], graph=None)
    if case["graph"]:
        stream = torch.cuda.Stream()
        stream.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(stream):
            block(hidden, residual, inference_params=params)
            stream.synchronize()
            state["graph"] = torch.cuda.CUDAGraph()
            with torch.cuda.graph(state["graph"], stream=stream):
                state["out"] = block(hidden, residual, inference_params=params)
        torch.cuda.current_stream().wait_stream(stream)
    return state


def _prepare_core(case, gen):
    width, groups = 2 * case["width"], case["groups"]
    n, gn, heads = (4 if case["grouped_scales"] else 0), 128 * groups, width // 64
    conv_dim = width + 2 * gn
    conv = Quamb2Conv1D(width, 64, 128, groups, n, n, conv_dim, conv_dim, 4, groups=conv_dim, padding=3, device="cuda")
    scan = Quamba2ChunkScan(width, 64, 128, groups, False, 256, n, n, device="cuda")
    _fill_conv_and_scan(conv, scan, gen)
    row = width + conv_dim + heads                       # z | x B C | dt of one token, as in_proj writes them
    rows = _codes((case["batch"], case["seqlen"], row), gen, 1.0 / ACT)
    return dict(level="core", conv=conv, scan=scan, rows=rows, split=[width, conv_dim, heads], heads=heads, groups=groups)


def run(state):
    if state["level"] == "lm":
        runner = state["runner"]
        if state["ids"] is not None:
            runner.input_ids.copy_(state["ids"])
            return [runner.replay()] + state["caches"]
        return [runner.replay(), runner.input_ids] + state["caches"]
    if state["level"] == "block":
        if state["graph"] is not None:
            state["graph"].replay()
            out = state["out"]
        else:
            out = state["block"](state["hidden"], state["residual"], inference_params=state["params"])
        return list(out) + state["caches"]
    _, xbc, dt = torch.split(state["rows"], state["split"], dim=-1)
    x, B, C = (t.transpose(1, 2) for t in state["conv"](xbc.transpose(1, 2)))
    y, last = state["scan"](x.unflatten(-1, (state["heads"], 64)), dt, B.unflatten(-1, (state["groups"], 128)),
                            C.unflatten(-1, (state["groups"], 128)), return_final_states=True)
    return [y, last]


# ---- what a pass cannot do without ----------------------------------------------------------------------------------------
def _linear(k, n, rows, weights, out_bytes):
    """Bytes and operations of a product; the int8 rows in between need not leave the chip."""
    w = k * n if weights == "w8" else k * n // 2 + (k // 128 * n * 2 if weights == "w4g128" else 0)
    return w + 4 * n + rows * n * out_bytes, 2 * rows * k * n


def work(case):
    d, b, length, g = case["width"], case["batch"], case["seqlen"], case["groups"]
    tokens, inner = b * length, 2 * d
    by = fl = 0
    decode = case["phase"] == "decode"
    if case["family"] == "mamba2":
        heads, conv_dim = inner // 64, inner + 256 * g
        state = heads * 64 * 128
        # per 128-token block and head: C.B^T, the masked product, the carried-in part, the state
        fl += tokens * heads * (2 * 128 * (128 + 64 + 64 + 64) if not decode else 6 * 64 * 128)
        if case["level"] == "core":
            by += tokens * (conv_dim + heads + 2 * inner) + 5 * conv_dim + b * state
            return {"bytes": by, "flops": fl}
        lins = [(d, inner + conv_dim + heads), (inner, d)]
    else:
        conv_dim, state = inner, inner * 16
        fl += tokens * inner * 16 * 8
        rank = math.ceil(d / 16)
        lins = [(d, 2 * inner), (inner, rank + 32), (rank, inner), (inner, d)]
    for k, n in lins:
        x, y = _linear(k, n, tokens, case["weights"], 0)
        by, fl = by + x, fl + y
    by += 5 * conv_dim + b * (state + 4 * conv_dim) * (2 if decode else 1)
    by, fl = by * case["layers"], fl * case["layers"]
    if case["level"] == "lm":
        x, y = _linear(d, VOCAB, b, case["weights"], 2)
        return {"bytes": by + x + tokens * (8 + d // 2), "flops": fl + y}
    return {"bytes": by + tokens * d * (2 + 4 + 4 + 2), "flops": fl}


def tolerance(case):
    # fp16 outputs behind int8 activations whose last bit may fall either way where the value before rounding differs by an
    # fp16 rounding; the integer products are exact
    return {"rel": 1e-2, "differ": 1e-2}
