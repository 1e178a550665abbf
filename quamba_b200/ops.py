"""Extension-level API of the reference, served by the B200 library.

Each namespace below has the name and the call signatures of one compiled extension
(or Triton entry point) of the reference, so the quantized modules and the parity tests
read the same way; underneath, every call marshals raw device pointers into the C ABI of
``libquamba_b200.so`` on torch's current stream (csrc/binding.cpp for the operators of every
layer; ctypes here for what runs once per model or inside captured decode steps).  Outputs
come from torch's caching allocator exactly as in the reference's bindings.  There is no
fallback path: a missing library or a rejected argument raises ``RuntimeError``.

Reference interfaces mirrored (paths inside the reference project):
  quant_sscan_cuda.fwd                      csrc/selective_scan/quant_sscan.cpp:122-270
  quant_causal_conv1d_cuda.fwd / .update    csrc/causal_conv1d/quant_causal_conv1d.cpp:77-231
  quamba2_conv1d_cuda.fwd / .update         csrc/causal_conv1d/quamba2_conv1d.cpp:122-385
  quant_hadamard.fast_hadamard_transform*   csrc/hadamard/quant_hadamard.cpp:72-294
  quant_linear_cuda.*                       csrc/linear/quant_linear.cpp:62-75
  _quant_/_quamba2_mamba_chunk_scan_combined_fwd   quamba/triton/quant_ssd_combined.py:11-166
  quant_/quamba2_sscan_update_triton        quamba/triton/selective_state_update.py:129-478
  _qlayer_norm_fwd / _qlayer_normgated_fwd  quamba/triton/quant_norm.py:134-206, quant_normgated.py:85-132
  quant_embedding_cuda.*                    csrc/embedding/quant_embedding_kernel.cuh:87-139, :207-260
"""
import ctypes
import weakref

import torch

from . import _lib

__all__ = ["quant_sscan_cuda", "quant_causal_conv1d_cuda", "quamba2_conv1d_cuda", "quant_hadamard",
           "quant_linear_cuda", "_quant_mamba_chunk_scan_combined_fwd", "_quamba2_mamba_chunk_scan_combined_fwd",
           "quant_sscan_update_triton", "quamba2_sscan_update_triton", "prepare_w4a8_weight", "_qlayer_norm_fwd",
           "_qlayer_normgated_fwd", "quant_embedding_cuda"]


def _p(t):
    return None if t is None else t.data_ptr()


def _stream(t):
    return torch.cuda.current_stream(t.device).cuda_stream


def _req(cond, msg):
    if not cond:
        raise RuntimeError(msg)


def _no_states(seq_idx, initial_states, final_states_out):
    for name, v in (("seq_idx", seq_idx), ("initial_states", initial_states), ("final_states_out", final_states_out)):
        if v is not None:
            raise RuntimeError(f"No implementation for {name}")


_n = _lib.native          # the native host path: argument checks, output allocation and the C-ABI call of each operator


def _run(fn, args, ref_tensor):
    with torch.cuda.device(ref_tensor.device):
        _lib.call(fn, args, _stream(ref_tensor))


# ------------------------------------------------------------------------------------------------
class quant_causal_conv1d_cuda:
    @staticmethod
    def fwd(x, scale_x, weight, scale_w, scale_out, scale_b, bias=None, seq_idx=None, initial_states=None,
            final_states_out=None, silu_activation=True):
        _no_states(seq_idx, initial_states, final_states_out)
        return _n().conv1_fwd(x, scale_x, weight, scale_w, scale_out, scale_b, bias, silu_activation)

    @staticmethod
    def update(x, conv_state, scale_x, weight, scale_w, scale_out, scale_b, bias=None, silu_activation=True):
        return _n().conv1_update(x, conv_state, scale_x, weight, scale_w, scale_out, scale_b, bias, silu_activation)


class quamba2_conv1d_cuda:
    @staticmethod
    def fwd(xBC, scale_x, scale_B, scale_C, x_dim, x_headdim, d_state, n_groups, x_head_group_range,
            x_dim_group_range, x_scales, B_scales, C_scales, weight, scale_wx, scale_wB, scale_wC, bias,
            scale_bx, scale_bB, scale_bC, seq_idx=None, initial_states=None, final_states_out=None,
            silu_activation=True):
        _no_states(seq_idx, initial_states, final_states_out)
        return _n().conv2_fwd(xBC, scale_x, scale_B, scale_C, x_dim, x_headdim, d_state, n_groups, x_head_group_range,
                              x_dim_group_range, x_scales, B_scales, C_scales, weight, scale_wx, scale_wB, scale_wC, bias,
                              scale_bx, scale_bB, scale_bC, silu_activation)

    @staticmethod
    def update(xBC, conv_state, scale_x, scale_B, scale_C, x_dim, x_headdim, d_state, n_groups, x_head_group_range,
               x_dim_group_range, x_scales, B_scales, C_scales, weight, scale_wx, scale_wB, scale_wC, bias,
               scale_bx, scale_bB, scale_bC, seq_idx=None, initial_states=None, final_states_out=None,
               silu_activation=True):
        return _n().conv2_update(xBC, conv_state, scale_x, scale_B, scale_C, x_dim, x_headdim, d_state, n_groups,
                                 x_head_group_range, x_dim_group_range, x_scales, B_scales, C_scales, weight, scale_wx,
                                 scale_wB, scale_wC, bias, scale_bx, scale_bB, scale_bC, silu_activation)


# ------------------------------------------------------------------------------------------------
def _hadamard(x, scale, special):
    return _n().hadamard(x, scale, special)


class quant_hadamard:
    fast_hadamard_transform = staticmethod(lambda x, scale: _hadamard(x, scale, 1))
    fast_hadamard_transform_12N = staticmethod(lambda x, scale: _hadamard(x, scale, 12))
    fast_hadamard_transform_20N = staticmethod(lambda x, scale: _hadamard(x, scale, 20))
    fast_hadamard_transform_28N = staticmethod(lambda x, scale: _hadamard(x, scale, 28))
    fast_hadamard_transform_40N = staticmethod(lambda x, scale: _hadamard(x, scale, 40))


# ------------------------------------------------------------------------------------------------
class quant_sscan_cuda:
    @staticmethod
    def fwd(u, scale_u, delta, scale_delta, A, scale_A, B, scale_B, C, scale_C, scale_ssm_state, D=None,
            scale_D=None, z=None, scale_z=None, delta_bias=None, scale_delta_bias=None, delta_softplus=False):
        return _n().sscan_fwd(u, scale_u, delta, scale_delta, A, scale_A, B, scale_B, C, scale_C, scale_ssm_state, D, scale_D,
                              z, scale_z, delta_bias, scale_delta_bias, delta_softplus)


# ------------------------------------------------------------------------------------------------
# Programmatic early launch between the kernels of a fused decode step: the kernels named in the header's early_launch note
# read their producer's output past L1, so each may let its successor start while it runs.  The switch is on only inside
# QuambaMixerModel.decode_step_fused, whose launch sequence consists of exactly those kernels.
_EARLY = False


class early_dependents:
    def __enter__(self):
        global _EARLY
        self.prev, _EARLY = _EARLY, True

    def __exit__(self, *exc):
        global _EARLY
        _EARLY = self.prev


def quant_sscan_update_triton(state, q_x, x_scale, q_dt, dt_scale, q_A_log, A_log_scale, ssm_state_scale, q_B, B_scale,
                              q_C, C_scale, q_D=None, D_scale=None, q_z=None, z_scale=None, dt_bias=None,
                              dt_bias_scale=None, dt_softplus=False):
    """state int8 (batch, dim, dstate) or (batch, nheads, dim, dstate), updated in place; returns out fp16."""
    return _n().sscan_update(state, q_x, x_scale, None, None, q_dt, dt_scale, q_A_log, A_log_scale, ssm_state_scale, q_B,
                             B_scale, q_C, C_scale, q_D, D_scale, q_z, z_scale, dt_bias, dt_bias_scale, dt_softplus, _EARLY)


def quamba2_sscan_update_triton(state, q_x, x_scales, x_head_group_range, x_dim_group_range, q_dt, dt_scale, q_A_log,
                                A_log_scale, ssm_state_scale, q_B, B_scale, q_C, C_scale, q_D=None, D_scale=None,
                                q_z=None, z_scale=None, dt_bias=None, dt_softplus=False):
    """Grouped-scale variant: x_scales [G,HG,DG], ssm_state_scale [G,HG,DG,N], B/C scales [G]."""
    _req(x_head_group_range.dtype == torch.int32 and x_dim_group_range.dtype == torch.int32, "group ranges must be int32")
    return _n().sscan_update(state, q_x, x_scales, x_head_group_range, x_dim_group_range, q_dt, dt_scale, q_A_log, A_log_scale,
                             ssm_state_scale, q_B, B_scale, q_C, C_scale, q_D, D_scale, q_z, z_scale, dt_bias, None, dt_softplus,
                             _EARLY)


# ------------------------------------------------------------------------------------------------
def _ssd(q_x, x_scales, hgr, dgr, q_dt, dt_scale, q_A_log, A_log_scale, q_B, B_scale, q_C, C_scale, ssm_state_scale,
         chunk_size, q_D, D_scale, q_z, z_scale, dt_bias, initial_states, seq_idx, cu_seqlens, dt_softplus, dt_limit):
    if initial_states is not None:
        raise NotImplementedError("Only supports initial_states=None")
    if seq_idx is not None:
        raise NotImplementedError("Only supports seq_idx=None")
    if cu_seqlens is not None:
        raise NotImplementedError("Only supports `cu_seqlens=None`")
    return _n().ssd(q_x, x_scales, hgr, dgr, q_dt, dt_scale, q_A_log, A_log_scale, q_B, B_scale, q_C, C_scale, ssm_state_scale,
                    chunk_size, q_D, D_scale, q_z, z_scale, dt_bias, dt_softplus, dt_limit[0], dt_limit[1])


def _quant_mamba_chunk_scan_combined_fwd(q_x, x_scale, q_dt, dt_scale, q_A_log, A_log_scale, q_B, B_scale, q_C, C_scale,
                                         ssm_state_scale, chunk_size, q_D=None, D_scale=None, q_z=None, z_scale=None,
                                         dt_bias=None, initial_states=None, seq_idx=None, cu_seqlens=None,
                                         dt_softplus=False, dt_limit=(0.0, float("inf")), mm_dtype=torch.float16):
    return _ssd(q_x, x_scale, None, None, q_dt, dt_scale, q_A_log, A_log_scale, q_B, B_scale, q_C, C_scale,
                ssm_state_scale, chunk_size, q_D, D_scale, q_z, z_scale, dt_bias, initial_states, seq_idx, cu_seqlens,
                dt_softplus, dt_limit)


def _quamba2_mamba_chunk_scan_combined_fwd(q_x, x_scales, x_head_group_range, x_dim_group_range, q_dt, dt_scale,
                                           q_A_log, A_log_scale, q_B, B_scale, q_C, C_scale, ssm_state_scale,
                                           chunk_size, q_D=None, D_scale=None, q_z=None, z_scale=None, dt_bias=None,
                                           initial_states=None, seq_idx=None, cu_seqlens=None, dt_softplus=False,
                                           dt_limit=(0.0, float("inf")), mm_dtype=torch.float16):
    _req(x_head_group_range.dim() == 2, "x_head_group_range must have shape [n_ssd_group, x_nhead_group]")
    _req(x_dim_group_range.dim() == 3, "x_dim_group_range must have shape [n_ssd_group, x_nhead_group, n_dim_group]")
    _req(x_head_group_range.dtype == torch.int32 and x_dim_group_range.dtype == torch.int32, "group ranges must be int32")
    return _ssd(q_x, x_scales, x_head_group_range, x_dim_group_range, q_dt, dt_scale, q_A_log, A_log_scale, q_B, B_scale, q_C,
                C_scale, ssm_state_scale, chunk_size, q_D, D_scale, q_z, z_scale, dt_bias, initial_states, seq_idx, cu_seqlens,
                dt_softplus, dt_limit)


# ------------------------------------------------------------------------------------------------
class W4A8Prepared:
    """The streaming copies of one Marlin-QQQ packed weight, owned by whoever prepared it (a linear module keeps
    one; nothing global holds it).  ``sc`` fp32 (N) channel scales in natural order; ``w8`` int8 (N, K) the values
    the reference kernel multiplies with; ``w4`` uint8 (N, K / 2) nibble copy of a per-channel weight for
    decode-sized calls.  ``w8`` and ``w4`` are built on first use and can be dropped with :meth:`release`."""

    def __init__(self, b_q_weight, s_ch, s_group, size_n, size_k):
        _req(b_q_weight.is_cuda and b_q_weight.dtype == torch.int32, "b_q_weight must be an int32 CUDA tensor")
        _req(size_k % 16 == 0, f"size_k = {size_k} is not divisible by tile_size = 16")
        _req(b_q_weight.shape[0] == size_k // 16, "Shape mismatch: b_q_weight.size(0) != size_k / tile_size")
        _req(b_q_weight.shape[1] == size_n * 2, "Shape mismatch: b_q_weight.size(1) != size_n * tile_size / pack_factor")
        _req(s_ch.numel() == size_n, f"Shape mismatch: s_ch.numel() = {s_ch.numel()}, size_n = {size_n}")
        self.per_channel = s_group.numel() == 0
        self.group = -1 if self.per_channel else size_k // s_group.shape[0]
        _req(self.group in (-1, 128), f"Unexpected groupsize = {self.group}")
        if not self.per_channel:
            _req(s_group.dtype == torch.float16 and s_group.shape[1] == size_n, "s_group must be fp16 (K/128, N)")
        # weak references: the prepared copies must not keep a deleted layer's buffers alive
        self._src = tuple(weakref.ref(t) for t in (b_q_weight, s_ch, s_group))
        self.size_n, self.size_k = size_n, size_k
        self.versions = (b_q_weight._version, s_ch._version, s_group._version)
        self.w8 = self.w4 = self.sc = self.w4g = self.sg_nat = None

    def stale(self, b_q_weight, s_ch, s_group):
        live = tuple(r() for r in self._src)
        return (live[0] is not b_q_weight or live[1] is not s_ch or live[2] is not s_group
                or self.versions != (b_q_weight._version, s_ch._version, s_group._version))

    def _unpack(self):
        packed, s_ch, s_group = (r() for r in self._src)
        _req(packed is not None and s_ch is not None and s_group is not None, "the packed weight was freed")
        dev = packed.device
        w8 = torch.empty((self.size_n, self.size_k), dtype=torch.int8, device=dev)
        sc = torch.empty((self.size_n,), dtype=torch.float32, device=dev)
        args = _lib.make("qb_w4a8_unpack_args", packed=_p(packed.contiguous()),
                         s_group=None if self.per_channel else _p(s_group.contiguous()),
                         s_channel=_p(s_ch.contiguous().float()), w8=_p(w8), s_channel_nat=_p(sc),
                         size_k=self.size_k, size_n=self.size_n, group_size=self.group if self.group > 0 else self.size_k)
        _run("qb_w4a8_unpack", args, packed)
        return w8, sc

    def need_w8(self):
        if self.w8 is None:
            self.w8, self.sc = self._unpack()
        return self.w8

    def need_w4(self):
        """Nibble copy (per-channel weights only); the int8 expansion it is built from is not kept unless it
        already exists."""
        if self.w4 is None:
            w8 = self.w8
            if w8 is None:
                w8, self.sc = self._unpack()
            w4 = torch.empty((self.size_n, self.size_k // 2), dtype=torch.uint8, device=w8.device)
            with torch.cuda.device(w8.device):
                f = _lib.lib().qb_w4a8_pack_nibbles
                f.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int32, ctypes.c_int32, ctypes.c_void_p]
                _lib.check(f(w8.data_ptr(), w4.data_ptr(), self.size_n, self.size_k, ctypes.c_void_p(_stream(w8))))
            self.w4 = w4
        return self.w4

    def need_w4g(self):
        """Group-128 weights as the decode kernels stream them: (codes, scales) with ``codes`` uint8 (N, K / 2), the raw
        4-bit codes in the nibble layout of :meth:`need_w4` (byte b of 32-bit word i of a row: k = 8 i + b low, k = 8 i + 4 + b
        high), and ``scales`` fp16 (N, K / 128), the group scales in natural order.  Built once, from the packed buffer."""
        if self.w4g is None:
            from . import packing
            packed, s_ch, s_group = (r() for r in self._src)
            _req(packed is not None and s_ch is not None and s_group is not None, "the packed weight was freed")
            _req(not self.per_channel, "need_w4g is for group-quantised weights")
            q = packing.unpack_int4(packed, self.size_k, self.size_n, False)                 # (K, N) codes 0..15
            sg, sc = packing.unpermute_scales(s_group, s_ch, self.size_n, False)             # (K / 128, N), (1, N)
            qt = q.t().contiguous().to(torch.uint8).view(self.size_n, self.size_k // 8, 2, 4)
            self.w4g = (qt[:, :, 0, :] | (qt[:, :, 1, :] << 4)).reshape(self.size_n, self.size_k // 2).contiguous()
            self.sg_nat = sg.t().contiguous().to(torch.float16)
            if self.sc is None:
                self.sc = sc.reshape(-1).float().contiguous()
        return self.w4g, self.sg_nat

    def release(self, w8=True, w4=True):
        if w8:
            self.w8 = None
        if w4:
            self.w4 = self.w4g = self.sg_nat = None

    def nbytes(self):
        return sum(t.numel() * t.element_size() for t in (self.w8, self.w4, self.sc, self.w4g, self.sg_nat) if t is not None)


def prepare_w4a8_weight(b_q_weight, s_ch, s_group, size_n, size_k):
    """Wrap a Marlin-QQQ packed weight for the B200 kernels.  The caller owns the result (and with it the
    streaming copies); nothing is cached globally."""
    return W4A8Prepared(b_q_weight, s_ch, s_group, size_n, size_k)


# Extension-level calls receive raw tensors on every call.  Their prepared copies are remembered per weight
# OBJECT (id of the packed tensor, checked against a weak reference, dropped by a finalizer when the tensor
# dies), so an address re-used by the allocator can never hit another weight's entry.
_W4A8_BY_ID = {}


def _prepared_for(b_q_weight, s_ch, s_group, size_n, size_k):
    key = id(b_q_weight)
    hit = _W4A8_BY_ID.get(key)
    if hit is not None and not hit.stale(b_q_weight, s_ch, s_group) and (hit.size_n, hit.size_k) == (size_n, size_k):
        return hit
    prep = W4A8Prepared(b_q_weight, s_ch, s_group, size_n, size_k)
    _W4A8_BY_ID[key] = prep
    weakref.finalize(b_q_weight, _W4A8_BY_ID.pop, key, None)
    return prep


def w4a8_linear(a, prep, s_tok, output_transpose=False, out_int8=False):
    """The W4A8 product on a weight prepared once with :func:`prepare_w4a8_weight` (what the linear modules call)."""
    return _n().w4a8(a, prep, s_tok, a.shape[0], output_transpose, out_int8)


class quant_linear_cuda:
    @staticmethod
    def w4a8o16_gemm(a, b_q_weight, s_tok, s_ch, s_group, workspace, size_m, size_n, size_k, output_transpose=False):
        prep = _prepared_for(b_q_weight, s_ch, s_group, size_n, size_k)
        return _n().w4a8(a, prep, s_tok, size_m, output_transpose, False)

    @staticmethod
    def w4a8o8_gemm(a, b_q_weight, s_tok, s_ch, s_group, workspace, size_m, size_n, size_k, output_transpose=False):
        prep = _prepared_for(b_q_weight, s_ch, s_group, size_n, size_k)
        return _n().w4a8(a, prep, s_tok, size_m, output_transpose, True)

    @staticmethod
    def cutlass_scaled_mm_dq(c, a, b, a_scales, b_scales):
        """c (M,N) = cvt(a_scales * (b_scales * (a (M,K) @ b (K,N)))), a row-major, b column-major."""
        _n().w8a8_mm(c, a, b, a_scales, b_scales)

    @staticmethod
    def cutlass_scaled_mv_dq(c, a, b, alpha, beta):
        """c (1,N) = cvt(alpha * (a (N,K) @ b (1,K)^T)); beta must be 0 (the reference never passes another value)."""
        _req(float(beta) == 0.0, "beta != 0 is not supported")
        _n().w8a8_mv(c, a, b, alpha, None, None)

    @staticmethod
    def w8a8o8_gemv(c, a, b, scale_a, scale_b):
        """c (1,N) int8 = clamp(roundf(scale_a[n] * scale_b * (a (N,K) @ b (1,K)^T)))."""
        _n().w8a8_mv(c, a, b, None, scale_a, scale_b)
        return c


# ------------------------------------------------------------------------------------------------
def _qlayer_norm_fwd(x, weight, bias, eps, residual=None, static_out_scale=None, residual_dtype=None, is_rms_norm=False,
                     partials=None, out=None):
    """quamba/triton/quant_norm.py:134-206: returns (y int8, residual_out, per_token_scale or None).  ``partials`` (not in
    the reference): (slots, own_index, own) with slots fp16 (n, M, N) -- the input is then the fp16-rounded fp32 sum of
    the n slots, slot ``own_index`` read from the (M, N) tensor ``own`` when that is given; ``x`` must be ``slots[0]``."""
    slots, own_i, own = partials if partials is not None else (None, -1, None)
    code = 0
    if residual_dtype is not None and residual is None:
        _req(residual_dtype in (torch.float16, torch.float32), "residual_dtype must be float16 or float32")
        code = 2 if residual_dtype == torch.float32 else 1
    return _n().norm_fwd(x, weight, bias, eps, residual, static_out_scale, code, is_rms_norm, slots, own_i, own, out)


def _qlayer_normgated_fwd(x, weight, bias, eps, q_z=None, z_scale=None, static_out_scale=None, use_float16_output=False,
                          group_size=None, norm_before_gate=True, is_rms_norm=False):
    """quamba/triton/quant_normgated.py:85-132: returns (out fp16 or int8, per_token_scale (ngroups * M))."""
    return _n().normgated_fwd(x, weight, bias, eps, q_z, z_scale, static_out_scale, use_float16_output, group_size,
                              norm_before_gate, is_rms_norm)


class quant_embedding_cuda:
    """csrc/embedding/quant_embedding.cpp: w4a16_embedding_lookup / w8a16_embedding_lookup (+ the fp16 table)."""

    @staticmethod
    def _lookup(input, weight, scale, kind, dim):
        _req(weight.dim() == 2 and weight.is_cuda, "weight must be a 2-D CUDA tensor")
        _req(input.dim() in (1, 2), "input must be a 1D or 2D tensor")
        _req(input.is_cuda and input.dtype == torch.int64, "input must be an int64 CUDA tensor")
        vocab = weight.shape[0]
        if kind:
            _req(scale.dim() == 1 and scale.is_cuda and scale.dtype == torch.float16 and scale.numel() == vocab,
                 "scale must be a float16 CUDA tensor with one entry per row")
        tokens = input.contiguous()
        out = torch.empty((*tokens.shape, dim), dtype=torch.float16, device=input.device)
        args = _lib.make("qb_embedding_args", table=_p(weight.contiguous()), scales=_p(scale) if kind else None,
                         tokens=_p(tokens), out=_p(out), n_tokens=tokens.numel(), dim=dim, vocab=vocab, kind=kind)
        _run("qb_embedding_lookup", args, input)
        return out

    @staticmethod
    def w4a16_embedding_lookup(input, weight, scale):
        _req(weight.dtype == torch.int32, "weight's dtype must be int32")
        return quant_embedding_cuda._lookup(input, weight, scale, 2, weight.shape[1] * 8)

    @staticmethod
    def w8a16_embedding_lookup(input, weight, scale):
        _req(weight.dtype == torch.int8, "weight's dtype must be int8")
        return quant_embedding_cuda._lookup(input, weight, scale, 1, weight.shape[1])

    @staticmethod
    def f16_embedding_lookup(input, weight):
        _req(weight.dtype == torch.float16, "weight's dtype must be float16")
        return quant_embedding_cuda._lookup(input, weight, None, 0, weight.shape[1])


def greedy_next_token(logits, out=None):
    """Row-wise argmax of fp16 logits (rows, vocab) -> int64 (rows); ``out`` lets a captured step write in place."""
    _req(logits.is_cuda and logits.dtype == torch.float16 and logits.dim() == 2 and logits.stride(1) == 1,
         "logits must be a 2-D float16 CUDA tensor, contiguous in its last dim")
    rows, n = logits.shape
    if out is None:
        out = torch.empty((rows,), dtype=torch.int64, device=logits.device)
    _req(out.dtype == torch.int64 and out.numel() == rows and out.is_contiguous(), "out must be int64 (rows,)")
    f = _lib.lib().qb_argmax_rows
    f.argtypes = [ctypes.c_void_p, ctypes.c_int64, ctypes.c_int32, ctypes.c_int32, ctypes.c_void_p, ctypes.c_void_p]
    with torch.cuda.device(logits.device):
        _lib.check(f(logits.data_ptr(), logits.stride(0), rows, n, out.data_ptr(), ctypes.c_void_p(_stream(logits))))
    return out


# ------------------------------------------------------------------------------------------------
# Fused decode-step launches (1 to 4 rows).  ``prep`` is a W4A8Prepared; per-channel weights stream their nibble copy.
def _decode_weight(prep):
    """(weight copy, w_is_s4, group scales or None) for the decode kernels: nibbles for both weight formats."""
    if prep.per_channel and prep.size_k % 32 == 0:
        return prep.need_w4(), 1, None
    if not prep.per_channel and prep.size_k % 128 == 0 and GROUP_NIBBLES:
        w, sg = prep.need_w4g()
        return w, 1, sg
    return prep.need_w8(), 0, None


# Group-128 weights at decode: True streams the 4-bit codes + group scales and rebuilds the int8 weights in registers
# (half the bytes, bit-identical results, no int8 copy needed by a decode-only deployment); False streams the int8
# expansion.  Measured on the 2.7B model (batch 1): 1.86 ms per token from the codes against 1.53 ms from the expansion
# -- the decode step is bound by latency, not by bytes, and the ~2.4 instructions per weight of the fp16 rebuild sit on the
# critical path -- so the expansion is the default.
GROUP_NIBBLES = False


def decode_norm_linear(x, residual, norm_weight, eps, norm_out_scale, prep, s_tok, out_int8, residual_in_fp32=True, conv=None):
    """residual add + RMSNorm + quantise + W4A8 product for (rows, k) fp16 ``x``.  Returns (out (rows, n) int8 or fp16,
    residual_out).  ``conv``: dict(state, weight, bias, col0, x_dim, gn, scale_in, scale_bias, out_scales) runs the conv1d
    decode step on columns [col0, col0 + x_dim + 2 gn) in the epilogue and adds ``x``, ``B``, ``C`` int8 outputs to it."""
    rows, k = x.shape
    w, s4, sg = _decode_weight(prep)
    dt = torch.int8 if out_int8 else torch.float16
    out = torch.empty((rows, prep.size_n), dtype=dt, device=x.device)
    res_dtype = residual.dtype if residual is not None else (torch.float32 if residual_in_fp32 else torch.float16)
    residual_out = torch.empty((rows, k), dtype=res_dtype, device=x.device)
    kw = {}
    if conv is not None:
        st = conv["state"]
        conv["x"] = torch.empty((rows, conv["x_dim"]), dtype=torch.int8, device=x.device)
        conv["B"] = torch.empty((rows, conv["gn"]), dtype=torch.int8, device=x.device)
        conv["C"] = torch.empty((rows, conv["gn"]), dtype=torch.int8, device=x.device)
        so = conv["out_scales"]
        kw = dict(conv_state=_p(st), conv_weight=_p(conv["weight"]), conv_bias=_p(conv["bias"]), conv_x=_p(conv["x"]),
                  conv_B=_p(conv["B"]), conv_C=_p(conv["C"]), x_out_scale=_p(so[0]), B_out_scale=_p(so[1]), C_out_scale=_p(so[2]),
                  conv_state_sb=st.stride(0), conv_state_sd=st.stride(1), conv_state_sw=st.stride(2), conv_col0=conv["col0"],
                  conv_dim=conv["x_dim"] + 2 * conv["gn"], conv_x_dim=conv["x_dim"], conv_gn=conv["gn"],
                  conv_scale_in_x=conv["scale_in"][0], conv_scale_in_B=conv["scale_in"][1], conv_scale_in_C=conv["scale_in"][2],
                  conv_scale_bias_x=conv["scale_bias"][0], conv_scale_bias_B=conv["scale_bias"][1],
                  conv_scale_bias_C=conv["scale_bias"][2])
    args = _lib.make("qb_decode_norm_linear_args", x=_p(x), residual=_p(residual), residual_out=_p(residual_out),
                     norm_weight=_p(norm_weight), w=_p(w), s_channel_nat=_p(prep.sc), s_group_nat=_p(sg), s_tok=_p(s_tok), out=_p(out),
                     x_row_stride=x.stride(0), residual_row_stride=residual.stride(0) if residual is not None else 0,
                     residual_out_row_stride=residual_out.stride(0), out_row_stride=out.stride(0), rows=rows, n=prep.size_n,
                     k=k, w_is_s4=s4, out_int8=int(out_int8), residual_is_f32=int(residual is not None and residual.dtype == torch.float32),
                     residual_out_is_f32=int(res_dtype == torch.float32), eps=float(eps), norm_out_scale=float(norm_out_scale),
                     early_launch=int(_EARLY), **kw)
    _run("qb_decode_norm_linear", args, x)
    return out, residual_out


def decode_linear(a, prep, s_tok, out_int8=False):
    """Decode-sized W4A8 product of int8 rows ``a`` (1 to 4 rows) on the low-latency kernel: (rows, n) fp16 or int8."""
    rows, k = a.shape
    w, s4, sg = _decode_weight(prep)
    out = torch.empty((rows, prep.size_n), dtype=torch.int8 if out_int8 else torch.float16, device=a.device)
    args = _lib.make("qb_decode_norm_linear_args", a_int8=_p(a), w=_p(w), s_channel_nat=_p(prep.sc), s_group_nat=_p(sg), s_tok=_p(s_tok), out=_p(out),
                     x_row_stride=a.stride(0), out_row_stride=out.stride(0), rows=rows, n=prep.size_n, k=k, w_is_s4=s4,
                     out_int8=int(out_int8), early_launch=int(_EARLY))
    _run("qb_decode_norm_linear", args, a)
    return out


def decode_gate_had_quant(y, z, z_scale, norm_weight, eps, group_size, had_scale):
    """y (rows, d) fp16, z (rows, d) int8 (a strided view is fine) -> gate, grouped RMSNorm, Hadamard rotation, int8:
    QRMSNormGated (fp16 output) followed by QHadamard in one launch.  Returns (rows, d) int8."""
    rows, d = y.shape
    out = torch.empty((rows, d), dtype=torch.int8, device=y.device)
    args = _lib.make("qb_decode_gate_had_quant_args", y=_p(y), z=_p(z), norm_weight=_p(norm_weight), out=_p(out),
                     y_row_stride=y.stride(0), z_row_stride=z.stride(0), out_row_stride=out.stride(0), rows=rows, d=d,
                     group_size=group_size, z_scale=float(z_scale), eps=float(eps), had_scale=float(had_scale),
                     early_launch=int(_EARLY))
    _run("qb_decode_gate_had_quant", args, y)
    return out
