// The host path of the package as one CPython extension (quamba_b200/_native.so) on top of the C ABI.
//
// An eager call of this library is a few microseconds of GPU work, so what the host does around a launch decides how long
// such a call takes: filling an argument struct field by field through ctypes, torch.empty, a device context and the module
// machinery came to about 40 us per launch, against 3 to 15 us for most kernels.  Here a call unpacks its tensors with the
// C API, allocates outputs straight from the caching allocator and enters the C ABI: 3 us including the launch.  Two levels:
//   * one function per extension entry point of the reference (the Python functions in ops.py keep names and arguments);
//   * mamba2_layer / mamba1_layer: the launch sequence of a whole layer in one call.  They read the sub-modules' buffers and
//     scales from the module dictionaries on every call, so nothing can go stale, and return None when a module carries
//     hooks, is of a subclass, or a tensor has a layout they do not take: the caller then walks the modules one by one.
// Nothing here synchronises; all work goes to torch's current stream of the inputs' device.
#include "binding.h"

namespace qbn {

PyObject* g_trace = nullptr;   // callable(entry point, 0 | 1, stream) around every launch, or null

namespace {
void call_trace(PyObject* trace, const char* name, int phase, cudaStream_t st) {
  PyObject* r = PyObject_CallFunction(trace, "siK", name, phase, (unsigned long long)(uintptr_t)st);
  if (r == nullptr) throw PyErr{};
  Py_DECREF(r);
}
}  // namespace

void run_call(const char* name, int (*f)(const void*, void*), const void* args, cudaStream_t st) {
  const Ref trace = Ref::share(g_trace);
  if (trace != nullptr) call_trace(trace, name, 0, st);
  int rc;
  {
    const NoGil released;
    rc = f(args, st);
  }
  if (rc != QB_OK) throw std::runtime_error("quamba_b200 error " + std::to_string(rc) + ": " + qb_last_error());
  if (trace != nullptr) call_trace(trace, name, 1, st);
}

namespace {

PyObject* set_trace(PyObject*, PyObject* f) {
  PyObject* old = g_trace;
  g_trace = f == Py_None ? nullptr : Py_NewRef(f);
  Py_XDECREF(old);
  Py_RETURN_NONE;
}

// ---- conv1d ---------------------------------------------------------------------------------------------------------------
// (x, scale_x, weight, scale_w, scale_out, scale_b, bias, silu)
PyObject* conv1_fwd(const Args& a) {
  const Tensor x = a.tensor(0), w = contiguous(a.tensor(2)), bias = a.opt_tensor(6);
  cuda_i8(x, "x"); cuda_i8(w, "weight");
  need(x.dim() == 3, "x must be (batch, dim, seqlen)");
  const int64_t batch = x.size(0), dim = x.size(1), len = x.size(2), width = w.size(-1);
  need(w.dim() == 2 && w.size(0) == dim, "weight must have shape (dim, width)");
  need(x.stride(2) == 1 || x.stride(1) == 1, "x must be contiguous in seqlen or in channels");
  if (bias.defined()) { cuda_i8(bias, "bias"); need(bias.dim() == 1 && bias.size(0) == dim && bias.stride(0) == 1, "bias must have shape (dim,)"); }
  Device dev(x);
  // a dense input keeps its layout; a view of a wider tensor (one half of in_proj's columns) gets a dense output of its own
  const bool seq_last = x.stride(2) == 1;
  Tensor out = x.is_non_overlapping_and_dense() ? dev.empty_strided(x.sizes(), x.strides(), at::kChar)
                                                : dev.empty_strided(x.sizes(), seq_last ? strides3(dim * len, len, 1) : strides3(dim * len, 1, dim), at::kChar);
  qb_conv1d_fwd_args s{};
  s.x = i8(x); s.out = i8(out); s.weight = i8(w); s.bias = i8(bias);
  s.x_sb = x.stride(0); s.x_sd = x.stride(1); s.x_sl = x.stride(2);
  s.out_sb = out.stride(0); s.out_sd = out.stride(1); s.out_sl = out.stride(2);
  s.batch = batch; s.dim = dim; s.seqlen = len; s.width = width;
  s.scale_x = a.num(1); s.scale_w = a.num(3); s.scale_out = a.num(4); s.scale_b = a.num(5); s.silu = a.flag(7);
  QBN_CALL(qb_causal_conv1d_fwd, s, dev.stream);
  return wrap(out);
}

// (x, conv_state, scale_x, weight, scale_w, scale_out, scale_b, bias, silu)
PyObject* conv1_update(const Args& a) {
  const Tensor x = a.tensor(0), st = a.tensor(1), w = contiguous(a.tensor(3)), bias = a.opt_tensor(7);
  cuda_i8(x, "x"); cuda_i8(st, "conv_state"); cuda_i8(w, "weight");
  need(x.dim() == 2, "x must be (batch, dim)");
  const int64_t batch = x.size(0), dim = x.size(1), width = w.size(-1);
  need(st.dim() == 3 && st.size(0) == batch && st.size(1) == dim && st.size(2) == width, "conv_state must have shape (batch, dim, width)");
  need(w.dim() == 2 && w.size(0) == dim, "weight must have shape (dim, width)");
  on_gpu(bias, "bias");
  Device dev(x);
  Tensor out = dev.empty({batch, dim}, at::kChar);
  qb_conv1d_update_args s{};
  s.x = i8(x); s.conv_state = i8(st); s.out = i8(out); s.weight = i8(w); s.bias = i8(bias);
  s.x_sb = x.stride(0); s.x_sd = x.stride(1); s.state_sb = st.stride(0); s.state_sd = st.stride(1); s.state_sw = st.stride(2);
  s.out_sb = dim; s.out_sd = 1; s.batch = batch; s.dim = dim; s.width = width;
  s.scale_x = a.num(2); s.scale_w = a.num(4); s.scale_out = a.num(5); s.scale_b = a.num(6); s.silu = a.flag(8);
  QBN_CALL(qb_causal_conv1d_update, s, dev.stream);
  return wrap(out);
}

// scales and ranges of a Quamba2 conv from positional arguments `k` on:
// (scale_x, scale_B, scale_C, x_dim, x_headdim, d_state, n_groups, head_range, dim_range, x_scales, B_scales, C_scales,
//  weight, scale_wx, scale_wB, scale_wC, bias, scale_bx, scale_bB, scale_bC, silu)
Conv2 conv2_from(const Args& a, int k) {
  Conv2 c;
  for (int i = 0; i < 3; ++i) {
    c.in[i] = a.num(k + i);
    c.w_scale[i] = a.num(k + 13 + i);
    c.b_scale[i] = a.num_or(k + 17 + i, 0.0);
  }
  c.x_dim = a.integer(k + 3); c.headdim = a.integer(k + 4); c.d_state = a.integer(k + 5); c.groups = a.integer(k + 6);
  c.hgr = a.opt_tensor(k + 7); c.dgr = a.opt_tensor(k + 8);
  c.out_scale[0] = a.tensor(k + 9); c.out_scale[1] = a.tensor(k + 10); c.out_scale[2] = a.tensor(k + 11);
  c.weight = contiguous(a.tensor(k + 12)); c.bias = a.opt_tensor(k + 16);
  c.silu = a.flag(k + 20);
  return c;
}

PyObject* conv2_fwd(const Args& a) {
  const Tensor x = a.tensor(0);
  Conv2 c = conv2_from(a, 1);
  cuda_i8(x, "xBC"); cuda_i8(c.weight, "weight");
  need(x.dim() == 3, "xBC must be (batch, dim, seqlen)");
  const int64_t batch = x.size(0), dim = x.size(1), len = x.size(2);
  need(c.weight.dim() == 2 && c.weight.size(0) == dim, "weight must have shape (dim, width)");
  need(x.stride(1) == 1 && x.stride(2) > 1, "only support channel_last");
  if (c.bias.defined()) { cuda_i8(c.bias, "bias"); need(c.bias.dim() == 1 && c.bias.size(0) == dim, "bias must have shape (dim,)"); }
  c.check();
  Device dev(x);
  const int64_t gn = c.d_state * c.groups;
  Tensor ox = dev.empty({batch, len, c.x_dim}, at::kChar), oB = dev.empty({batch, len, gn}, at::kChar), oC = dev.empty({batch, len, gn}, at::kChar);
  qb_quamba2_conv1d_fwd_args s = c.fwd_args(dim);
  s.xBC = i8(x); s.xBC_sb = x.stride(0); s.xBC_sl = x.stride(2);
  s.x = i8(ox); s.Bm = i8(oB); s.Cm = i8(oC);
  s.batch = batch; s.seqlen = len;
  QBN_CALL(qb_quamba2_conv1d_fwd, s, dev.stream);
  return wrap_list({ox.transpose(1, 2), oB.transpose(1, 2), oC.transpose(1, 2)});
}

PyObject* conv2_update(const Args& a) {
  const Tensor x = a.tensor(0), st = a.tensor(1);
  Conv2 c = conv2_from(a, 2);
  cuda_i8(x, "xBC"); cuda_i8(st, "conv_state"); cuda_i8(c.weight, "weight");
  need(x.dim() == 2, "xBC must be (batch, dim)");
  const int64_t batch = x.size(0), dim = x.size(1);
  need(st.dim() == 3 && st.size(0) == batch && st.size(1) == dim && st.size(2) == c.weight.size(-1), "conv_state must have shape (batch, dim, width)");
  need(c.weight.dim() == 2 && c.weight.size(0) == dim, "weight must have shape (dim, width)");
  need(x.stride(1) == 1, "xBC must be contiguous in channels");
  c.check();
  Device dev(x);
  const int64_t gn = c.d_state * c.groups;
  Tensor ox = dev.empty({batch, c.x_dim}, at::kChar), oB = dev.empty({batch, gn}, at::kChar), oC = dev.empty({batch, gn}, at::kChar);
  qb_quamba2_conv1d_update_args s = c.update_args(dim);
  s.xBC = i8(x); s.xBC_sb = x.stride(0); s.conv_state = i8(st);
  s.state_sb = st.stride(0); s.state_sd = st.stride(1); s.state_sw = st.stride(2);
  s.x = i8(ox); s.Bm = i8(oB); s.Cm = i8(oC); s.batch = batch;
  QBN_CALL(qb_quamba2_conv1d_update, s, dev.stream);
  return wrap_list({ox, oB, oC});
}

// ---- Hadamard: (x, scale, special) ----------------------------------------------------------------------------------------
PyObject* hadamard(const Args& a) {
  Tensor x = a.tensor(0);
  need(x.is_cuda(), "x must be a CUDA tensor");
  const auto t = x.scalar_type();
  need(t == at::kHalf || t == at::kBFloat16 || t == at::kFloat, "x must be fp16, bf16 or fp32");
  const int64_t dim = x.size(-1);
  Device dev(x);
  Tensor out = dev.empty(x.sizes(), at::kChar);
  Tensor x2 = x.dim() == 2 ? x : x.reshape({-1, dim});
  if (x2.stride(-1) != 1) x2 = x2.contiguous();
  qb_hadamard_quant_args s{};
  s.x = x2.data_ptr(); s.out = i8(out); s.x_row_stride = x2.stride(0); s.out_row_stride = dim;
  s.rows = x2.size(0); s.dim = dim; s.special = a.integer(2);
  s.in_dtype = t == at::kHalf ? 0 : (t == at::kBFloat16 ? 1 : 2); s.scale = a.num(1);
  QBN_CALL(qb_hadamard_quant, s, dev.stream);
  return wrap(out);
}

// ---- Mamba1 scan ----------------------------------------------------------------------------------------------------------
// (u, scale_u, delta, scale_delta, A, scale_A, B, scale_B, C, scale_C, scale_ssm_state, D, scale_D, z, scale_z, delta_bias,
//  scale_delta_bias, delta_softplus)
PyObject* sscan_fwd(const Args& a) {
  const Tensor u = a.tensor(0), delta = a.tensor(2), A = contiguous(a.tensor(4)), D = a.opt_tensor(11), z = a.opt_tensor(13), bias = a.opt_tensor(15);
  Tensor B = a.tensor(6), C = a.tensor(8);
  cuda_i8(u, "u"); cuda_i8(delta, "delta"); cuda_i8(A, "A"); cuda_i8(B, "B"); cuda_i8(C, "C");
  need(u.dim() == 3, "u must be (batch, dim, seqlen)");
  const int64_t batch = u.size(0), dim = u.size(1), len = u.size(2), n = A.size(1);
  need(B.dim() >= 3 && C.dim() >= 3, "Must be input-dependent B and C");
  if (B.dim() == 3) B = B.unsqueeze(1);
  if (C.dim() == 3) C = C.unsqueeze(1);
  const int64_t groups = B.size(1);
  need(n <= 256, "quant_sscan only supports state dimension <= 256");
  need(delta.sizes() == u.sizes(), "delta must have the shape of u");
  need(A.size(0) == dim, "A must be (dim, dstate)");
  const int64_t want[4] = {batch, groups, n, len};
  need(B.sizes() == at::IntArrayRef(want, 4), "B must be (batch, n_groups, dstate, seqlen)");
  need(C.sizes() == at::IntArrayRef(want, 4), "C must be (batch, n_groups, dstate, seqlen)");
  const Tensor* chk[4] = {&u, &delta, &B, &C};
  const char* nm[4] = {"u", "delta", "B", "C"};
  for (int i = 0; i < 4; ++i)
    need(chk[i]->stride(-1) == 1 || chk[i]->size(-1) == 1, std::string(nm[i]) + " must be contiguous in seqlen");
  const int sc[6] = {1, 3, 5, 7, 9, 10};
  const char* sn[6] = {"scale_u", "scale_delta", "scale_A", "scale_B", "scale_C", "scale_ssm_state"};
  const float* sp[6];
  for (int i = 0; i < 6; ++i) {
    const Tensor t = a.opt_tensor(sc[i]);
    need(t.defined(), std::string(sn[i]) + " is required");
    need(t.is_cuda() && t.scalar_type() == at::kFloat, std::string(sn[i]) + " must be a float32 CUDA tensor");
    need(t.numel() == 1, std::string(sn[i]) + " must have 1 element");
    sp[i] = f32(t);
  }
  const Tensor zs = a.opt_tensor(14), Ds = a.opt_tensor(12), bs = a.opt_tensor(16);
  on_gpu(D, "D"); on_gpu(bias, "delta_bias");
  if (Ds.defined()) cuda_f32(Ds, "scale_D");
  if (bs.defined()) cuda_f32(bs, "scale_delta_bias");
  if (z.defined()) {
    cuda_i8(z, "z");
    need(z.sizes() == u.sizes() && (z.stride(-1) == 1 || z.size(-1) == 1), "z must match u");
    need(zs.defined(), "scale_z is required");
    need(zs.is_cuda() && zs.scalar_type() == at::kFloat, "scale_z must be a float32 CUDA tensor");
  }
  Device dev(u);
  const int64_t chunks = (len + 2047) / 2048;
  Tensor out = dev.empty({batch, len, dim}, at::kHalf), x = dev.empty({batch, dim, chunks, n}, at::kChar);
  qb_sscan_fwd_args s{};
  s.u = i8(u); s.delta = i8(delta); s.z = i8(z); s.Bm = i8(B); s.Cm = i8(C); s.A_log = i8(A); s.D = i8(D); s.delta_bias = i8(bias);
  s.u_scale = sp[0]; s.delta_scale = sp[1]; s.A_scale = sp[2]; s.B_scale = sp[3]; s.C_scale = sp[4]; s.ssm_state_scale = sp[5];
  s.z_scale = z.defined() ? f32(zs) : nullptr; s.D_scale = D.defined() ? f32(Ds) : nullptr; s.delta_bias_scale = bias.defined() ? f32(bs) : nullptr;
  s.out = out.data_ptr(); s.x_states = i8(x);
  s.u_sb = u.stride(0); s.u_sd = u.stride(1); s.delta_sb = delta.stride(0); s.delta_sd = delta.stride(1);
  if (z.defined()) { s.z_sb = z.stride(0); s.z_sd = z.stride(1); }
  s.B_sb = B.stride(0); s.B_sg = B.stride(1); s.B_sn = B.stride(2); s.C_sb = C.stride(0); s.C_sg = C.stride(1); s.C_sn = C.stride(2);
  s.batch = batch; s.dim = dim; s.seqlen = len; s.dstate = n; s.n_groups = groups; s.delta_softplus = a.flag(17);
  QBN_CALL(qb_sscan_fwd, s, dev.stream);
  return wrap_list({out, x});
}

// ---- single-step state update ---------------------------------------------------------------------------------------------
// (state, x, x_scales, head_range, dim_range, dt, dt_scale, A_log, A_scale, state_scale, B, B_scale, C, C_scale, D, D_scale, z,
//  z_scale, dt_bias, dt_bias_scale, dt_softplus, early)
PyObject* sscan_update(const Args& a) {
  Tensor st = a.tensor(0), x = a.tensor(1), dt = a.tensor(5), A = a.tensor(7), B = a.tensor(10), C = a.tensor(12);
  Tensor D = a.opt_tensor(14), z = a.opt_tensor(16), bias = a.opt_tensor(18);
  Tensor xs = a.tensor(2), hgr = a.opt_tensor(3), dgr = a.opt_tensor(4), ss = a.tensor(9);
  const bool grouped = hgr.defined();
  const bool heads = st.dim() > 3;
  if (st.dim() == 3) st = st.unsqueeze(1);
  if (x.dim() == 2) x = x.unsqueeze(1);
  if (dt.dim() == 2) dt = dt.unsqueeze(1);
  if (A.dim() == 2) A = A.unsqueeze(0);
  if (B.dim() == 2) B = B.unsqueeze(1);
  if (C.dim() == 2) C = C.unsqueeze(1);
  if (D.defined() && D.dim() == 1) D = D.unsqueeze(0);
  if (z.defined() && z.dim() == 2) z = z.unsqueeze(1);
  if (bias.defined() && bias.dim() == 1) bias = bias.unsqueeze(0);
  need(st.dim() == 4 && x.dim() == 3 && B.dim() == 3, "state must be (batch, [nheads,] dim, dstate)");
  const int64_t groups = B.size(1), batch = st.size(0), nh = st.size(1), dim = st.size(2), n = st.size(3);
  auto is = [](const Tensor& t, std::initializer_list<int64_t> v) { return t.sizes() == at::IntArrayRef(v.begin(), v.size()); };
  cuda_i8(st, "state"); cuda_i8(x, "q_x");
  on_gpu(dt, "q_dt"); on_gpu(A, "q_A_log"); on_gpu(B, "q_B"); on_gpu(C, "q_C"); on_gpu(D, "q_D"); on_gpu(z, "q_z"); on_gpu(bias, "dt_bias");
  on_gpu(hgr, "x_head_group_range"); on_gpu(dgr, "x_dim_group_range");
  cuda_f32(xs, "x_scales"); cuda_f32(ss, "ssm_state_scale"); cuda_f32(a.tensor(6), "dt_scale"); cuda_f32(a.tensor(8), "A_log_scale");
  cuda_f32(a.tensor(11), "B_scale"); cuda_f32(a.tensor(13), "C_scale");
  need(is(x, {batch, nh, dim}), "q_x must have shape (batch, nheads, dim)");
  need(dt.sizes() == x.sizes(), "q_dt must have the shape of q_x");
  need(is(A, {nh, dim, n}), "q_A_log must have shape (nheads, dim, dstate)");
  need(nh % groups == 0, "nheads must be divisible by ngroups");
  need(is(B, {batch, groups, n}) && C.sizes() == B.sizes(), "q_B / q_C must be (batch, ngroups, dstate)");
  need(st.stride(-1) == 1 && x.stride(-1) == 1 && B.stride(-1) == 1 && C.stride(-1) == 1, "state, x, B, C must be contiguous in their last dim");
  const Tensor Bs = a.tensor(11), Cs = a.tensor(13);
  if (grouped) {
    hgr = contiguous(hgr); dgr = contiguous(dgr); ss = contiguous(ss);
    need(xs.numel() == groups * hgr.size(1) * dgr.size(2), "x_scales must be [G, HG, DG]");
    need(Bs.numel() == groups && Cs.numel() == groups, "B / C scales must be [G]");
  } else {
    need(Bs.numel() == 1 && Cs.numel() == 1, "B / C scales must have 1 element");
  }
  if (D.defined()) need(is(D, {nh, dim}), "q_D must have shape (nheads, dim)");
  if (z.defined()) need(z.sizes() == x.sizes() && z.stride(-1) == 1, "q_z must have the shape of q_x");
  const Tensor bias_s = a.opt_tensor(19);
  bool half = false;
  if (bias.defined()) {
    need(is(bias, {nh, dim}), "dt_bias must have shape (nheads, dim)");
    if (bias.scalar_type() == at::kChar) {
      need(bias_s.defined(), "int8 dt_bias needs dt_bias_scale");
    } else {
      need(bias.scalar_type() == at::kHalf, "dt_bias must be int8 (with a scale) or float16");
      half = true;
    }
  }
  Device dev(x);
  Tensor out = heads ? dev.empty({batch, nh, dim}, at::kHalf) : dev.empty({batch, dim}, at::kHalf);
  qb_sscan_update_args s{};
  s.state = i8(st); s.x = i8(x); s.dt = i8(dt); s.A_log = i8(A); s.Bm = i8(B); s.Cm = i8(C); s.D = i8(D); s.z = i8(z);
  s.dt_bias = bias.defined() ? bias.data_ptr() : nullptr;
  s.x_scales = f32(xs); s.dt_scale = f32(a.tensor(6)); s.A_scale = f32(a.tensor(8)); s.state_scale = f32(ss); s.B_scale = f32(Bs); s.C_scale = f32(Cs);
  s.D_scale = D.defined() ? scale_of(a.tensor(15), "D_scale") : nullptr; s.z_scale = z.defined() ? scale_of(a.tensor(17), "z_scale") : nullptr;
  s.dt_bias_scale = bias.defined() && !half ? scale_of(bias_s, "dt_bias_scale") : nullptr;
  s.head_group_range = i32(hgr); s.dim_group_range = i32(dgr); s.out = out.data_ptr();
  s.state_sb = st.stride(0); s.state_sh = st.stride(1); s.state_sp = st.stride(2);
  s.x_sb = x.stride(0); s.x_sh = x.stride(1); s.dt_sb = dt.stride(0); s.dt_sh = dt.stride(1); s.dt_sp = dt.stride(2);
  s.A_sh = A.stride(0); s.A_sp = A.stride(1); s.A_sn = A.stride(2);
  s.B_sb = B.stride(0); s.B_sg = B.stride(1); s.C_sb = C.stride(0); s.C_sg = C.stride(1);
  if (D.defined()) { s.D_sh = D.stride(0); s.D_sp = D.stride(1); }
  if (z.defined()) { s.z_sb = z.stride(0); s.z_sh = z.stride(1); }
  if (bias.defined()) { s.bias_sh = bias.stride(0); s.bias_sp = bias.stride(1); }
  s.out_sb = nh * dim; s.out_sh = dim; s.batch = batch; s.nheads = nh; s.headdim = dim; s.dstate = n; s.ngroups = groups;
  s.grouped = grouped; s.nhead_groups = grouped ? hgr.size(1) : 0; s.ndim_groups = grouped ? dgr.size(2) : 0;
  s.dt_bias_is_half = half; s.dt_softplus = a.flag(20); s.early_launch = a.flag(21);
  QBN_CALL(qb_sscan_update, s, dev.stream);
  return wrap(out);
}

// ---- SSD chunk scan -------------------------------------------------------------------------------------------------------
// (x, x_scales, head_range, dim_range, dt, dt_scale, A_log, A_scale, B, B_scale, C, C_scale, state_scale, chunk, D, D_scale, z,
//  z_scale, dt_bias, dt_softplus, dt_min, dt_max)
PyObject* ssd(const Args& a) {
  Tensor x = a.tensor(0), dt = a.tensor(4), A = a.tensor(6), B = a.tensor(8), C = a.tensor(10);
  Tensor D = a.opt_tensor(14), z = a.opt_tensor(16), bias = a.opt_tensor(18);
  Tensor hgr = a.opt_tensor(2), dgr = a.opt_tensor(3), xs = a.tensor(1), ss = a.tensor(12);
  const Tensor Bs = a.tensor(9), Cs = a.tensor(11);
  const bool grouped = hgr.defined();
  need(x.dim() == 4 && B.dim() == 4, "q_x must be (batch, seqlen, nheads, headdim), q_B (batch, seqlen, ngroups, dstate)");
  const int64_t batch = x.size(0), len = x.size(1), nh = x.size(2), hd = x.size(3), groups = B.size(2), n = B.size(3);
  need(groups > 0 && nh % groups == 0, "nheads must be divisible by ngroups");
  cuda_i8(x, "q_x"); cuda_i8(B, "q_B"); cuda_i8(dt, "q_dt"); cuda_i8(A, "q_A_log"); cuda_i8(C, "q_C");
  on_gpu(D, "q_D"); on_gpu(z, "q_z"); on_gpu(bias, "dt_bias"); on_gpu(hgr, "x_head_group_range"); on_gpu(dgr, "x_dim_group_range");
  cuda_f32(xs, "x_scales"); cuda_f32(ss, "ssm_state_scale"); cuda_f32(a.tensor(5), "dt_scale"); cuda_f32(a.tensor(7), "A_log_scale");
  cuda_f32(Bs, "B_scale"); cuda_f32(Cs, "C_scale");
  auto is = [](const Tensor& t, std::initializer_list<int64_t> v) { return t.sizes() == at::IntArrayRef(v.begin(), v.size()); };
  need(is(B, {batch, len, groups, n}) && C.sizes() == B.sizes(), "q_B / q_C shape mismatch");
  need(is(dt, {batch, len, nh}), "q_dt must be (batch, seqlen, nheads)");
  need(is(A, {nh}), "q_A_log must be (nheads,)");
  for (Tensor* t : {&B, &C, &x, &dt})
    if (t->stride(-1) != 1) *t = t->contiguous();
  if (z.defined()) {
    need(z.sizes() == x.sizes(), "q_z must have the shape of q_x");
    if (z.stride(-1) != 1) z = z.contiguous();
  }
  if (D.defined()) {
    need(is(D, {nh, hd}) || is(D, {nh}), "q_D must be (nheads, headdim) or (nheads,)");
    D = contiguous(D);
  }
  if (bias.defined()) {
    need(is(bias, {nh}), "dt_bias must be (nheads,)");
    if (bias.scalar_type() != at::kHalf) bias = bias.to(at::kHalf);
    bias = contiguous(bias);
  }
  if (grouped) {
    hgr = contiguous(hgr); dgr = contiguous(dgr); ss = contiguous(ss);
    need(xs.numel() == groups * hgr.size(1) * dgr.size(2), "x_scales must be [G, HG, DG]");
    need(Bs.numel() == groups && Cs.numel() == groups, "B / C scales must be [G]");
    need(is(ss, {groups, hgr.size(1), dgr.size(2), n}), "ssm_state_scale must be [G, HG, DG, N]");
  } else {
    need(xs.numel() == 1 && Bs.numel() == 1 && Cs.numel() == 1, "scales must have 1 element");
  }
  Device dev(x);
  const int64_t chunk = a.integer(13);
  Tensor out = dev.empty({batch, len, nh, hd}, at::kHalf), fin = dev.empty({batch, nh, hd, n}, at::kChar);
  const int64_t wsb = qb_ssd_workspace_bytes(batch, len, nh, hd, groups, n, chunk);
  need(wsb > 0, "invalid SSD shape");
  Tensor ws = dev.empty({wsb}, at::kByte);
  qb_ssd_args s{};
  s.x = i8(x); s.dt = i8(dt); s.Bm = i8(B); s.Cm = i8(C); s.A_log = i8(A); s.D = i8(D); s.z = i8(z); s.dt_bias = bias.defined() ? bias.data_ptr() : nullptr;
  s.x_scales = f32(xs); s.dt_scale = f32(a.tensor(5)); s.A_scale = f32(a.tensor(7)); s.B_scale = f32(Bs); s.C_scale = f32(Cs);
  s.D_scale = D.defined() ? scale_of(a.tensor(15), "D_scale") : nullptr; s.z_scale = z.defined() ? scale_of(a.tensor(17), "z_scale") : nullptr; s.ssm_state_scale = f32(ss);
  s.head_group_range = i32(hgr); s.dim_group_range = i32(dgr); s.out = out.data_ptr(); s.final_states = i8(fin); s.workspace = ws.data_ptr(); s.workspace_bytes = wsb;
  s.x_sb = x.stride(0); s.x_sl = x.stride(1); s.x_sh = x.stride(2); s.dt_sb = dt.stride(0); s.dt_sl = dt.stride(1);
  s.B_sb = B.stride(0); s.B_sl = B.stride(1); s.B_sg = B.stride(2); s.C_sb = C.stride(0); s.C_sl = C.stride(1); s.C_sg = C.stride(2);
  if (z.defined()) { s.z_sb = z.stride(0); s.z_sl = z.stride(1); s.z_sh = z.stride(2); }
  s.batch = batch; s.seqlen = len; s.nheads = nh; s.headdim = hd; s.ngroups = groups; s.dstate = n; s.chunk_size = chunk;
  s.grouped = grouped; s.nhead_groups = grouped ? hgr.size(1) : 0; s.ndim_groups = grouped ? dgr.size(2) : 0;
  s.D_has_hdim = D.defined() && D.dim() == 2; s.dt_softplus = a.flag(19); s.dt_min = a.num(20); s.dt_max = std::min(a.num(21), 3.0e38);
  QBN_CALL(qb_ssd_chunk_scan_fwd, s, dev.stream);
  return wrap_tuple({out, fin});
}

// ---- linears --------------------------------------------------------------------------------------------------------------
void check_w4a8(const Tensor& x, const Tensor& s_tok, int64_t m, int64_t k) {
  cuda_i8(x, "a");
  need(x.dim() == 2 && x.stride(1) == 1, "a must be a row-major (m, k) matrix");
  need(m == x.size(0), "Shape mismatch: a.size(0) = " + std::to_string(x.size(0)) + ", size_m = " + std::to_string(m));
  need(k == x.size(1), "Shape mismatch: a.size(1) = " + std::to_string(x.size(1)) + ", size_k = " + std::to_string(k));
  need(s_tok.numel() == 1 || s_tok.numel() == m, "s_tok.numel() = " + std::to_string(s_tok.numel()) + " is not 1 or equal to size_m = " + std::to_string(m));
  need(s_tok.is_cuda() && s_tok.scalar_type() == at::kFloat, "s_tok must be a float32 CUDA tensor");
}

// (a, prepared weight, s_tok, m, output_transpose, out_int8)
PyObject* w4a8(const Args& a) {
  const Tensor x = a.tensor(0), s_tok = a.tensor(2);
  PyObject* prep = a.object(1);
  const W4Dims w = w4_dims(prep);
  const int64_t m = a.integer(3);
  const bool tr = a.flag(4), int8 = a.flag(5);
  check_w4a8(x, s_tok, m, w.k);
  Device dev(x);
  Tensor out = tr ? dev.empty({w.n, m}, int8 ? at::kChar : at::kHalf) : dev.empty({m, w.n}, int8 ? at::kChar : at::kHalf);
  if (m > 0) w4a8_run(prep, w, i8(x), x.stride(0), m, f32(s_tok), s_tok.numel() != 1, out.data_ptr(), out.stride(0), int8, tr, dev.stream);
  return wrap(out);
}

int out_code(const Tensor& c) {
  const auto t = c.scalar_type();
  need(t == at::kChar || t == at::kHalf || t == at::kBFloat16, "unsupported output type");
  return t == at::kChar ? 0 : (t == at::kHalf ? 1 : 2);
}

// (c, a, b, a_scales, b_scales)
PyObject* w8a8_mm(const Args& a) {
  const Tensor c = a.tensor(0), x = a.tensor(1), b = a.tensor(2), sa = a.opt_tensor(3), sb = a.opt_tensor(4);
  cuda_i8(x, "a"); cuda_i8(b, "b");
  need(x.dim() == 2 && b.dim() == 2 && c.dim() == 2, "a, b, c must be matrices");
  need(c.size(0) == x.size(0) && x.size(1) == b.size(0) && b.size(1) == c.size(1), "shape mismatch");
  need(sa.defined() && sb.defined() && (sa.numel() == 1 || sa.numel() == x.size(0)) && (sb.numel() == 1 || sb.numel() == b.size(1)), "scale shape mismatch");
  need(x.stride(1) == 1 && c.stride(1) == 1, "a and c must be row-major");
  need(b.stride(0) == 1, "b must be column-major");
  need(c.stride(0) % 16 == 0 && b.stride(1) % 16 == 0, "16 byte alignment of c rows and b columns");
  need(sa.is_cuda() && sa.scalar_type() == at::kFloat, "a_scales must be a float32 CUDA tensor");
  need(sb.is_cuda() && sb.scalar_type() == at::kFloat, "b_scales must be a float32 CUDA tensor");
  need(sa.is_contiguous() && sb.is_contiguous(), "scales must be contiguous");
  qb_w8a8_gemm_args s{};
  s.out_dtype = out_code(c);
  Device dev(x);
  s.a = i8(x); s.b = i8(b); s.a_scale = f32(sa); s.b_scale = f32(sb); s.out = c.data_ptr();
  s.a_row_stride = x.stride(0); s.b_col_stride = b.stride(1); s.out_row_stride = c.stride(0);
  s.m = x.size(0); s.n = b.size(1); s.k = x.size(1); s.a_scale_per_row = sa.numel() != 1; s.b_scale_per_col = sb.numel() != 1;
  QBN_CALL(qb_w8a8_gemm, s, dev.stream);
  Py_RETURN_NONE;
}

// (c, a (N, K), b (1, K), alpha | None, scale_a | None, scale_b | None): the single-row forms, the scalar by value or by
// device pointers with round-half-away (w8a8o8_gemv)
PyObject* w8a8_mv(const Args& a) {
  const Tensor c = a.tensor(0), w = a.tensor(1), x = a.tensor(2), sa = a.opt_tensor(4), sb = a.opt_tensor(5);
  cuda_i8(w, "a"); cuda_i8(x, "b");
  need(w.dim() == 2 && x.dim() == 2 && c.dim() == 2, "a, b, c must be matrices");
  if (sa.defined()) {
    cuda_i8(c, "c");
    need(sa.numel() == w.size(0), "Shape mismatch: scale_a.numel() = " + std::to_string(sa.numel()) + ", size_n = " + std::to_string(w.size(0)));
    need(sb.numel() == 1, "Shape mismatch: scale_b.numel() = " + std::to_string(sb.numel()));
  }
  need(c.size(0) == x.size(0) && w.size(1) == x.size(1) && w.size(0) == c.size(1), "shape mismatch");
  need(w.stride(1) == 1 && x.stride(1) == 1 && c.stride(1) == 1, "a, b, c must be row-major");
  qb_w8a8_gemm_args s{};
  s.out_dtype = out_code(c);
  const Tensor sac = sa.defined() ? contiguous(sa) : sa;
  if (sa.defined()) {
    s.a_scale = f32(sb); s.b_scale = f32(sac); s.b_scale_per_col = 1; s.round_half_away = 1;
  } else {
    s.use_alpha = 1; s.alpha = a.num(3);
  }
  Device dev(w);
  s.a = i8(x); s.b = i8(w); s.out = c.data_ptr(); s.a_row_stride = x.stride(0); s.b_col_stride = w.stride(0); s.out_row_stride = c.stride(0);
  s.m = x.size(0); s.n = w.size(0); s.k = w.size(1);
  QBN_CALL(qb_w8a8_gemm, s, dev.stream);
  Py_RETURN_NONE;
}

// ---- norms ----------------------------------------------------------------------------------------------------------------
void check_norm(const Tensor& x, const Tensor& w, const Tensor& bias) {
  need(x.is_cuda() && x.scalar_type() == at::kHalf && x.dim() == 2, "x must be a 2-D float16 CUDA tensor");
  need(x.stride(-1) == 1, "x must be contiguous in its last dim");
  const int64_t n = x.size(1);
  on_gpu(w, "weight"); on_gpu(bias, "bias");
  need(w.dim() == 1 && w.size(0) == n && w.stride(0) == 1 && w.scalar_type() == at::kHalf, "weight must be fp16 (N,)");
  if (bias.defined()) need(bias.dim() == 1 && bias.size(0) == n && bias.stride(0) == 1 && bias.scalar_type() == at::kHalf, "bias must be fp16 (N,)");
}

// (x, weight, bias, eps, residual, static_scale | None, residual_code, is_rms, slots | None, own_index, own | None, out | None)
// residual_code: what residual_out is stored as when there is no residual: 0 nothing, 1 fp16, 2 fp32
PyObject* norm_fwd(const Args& a) {
  const Tensor x = a.tensor(0), w = a.tensor(1), bias = a.opt_tensor(2), res = a.opt_tensor(4), slots = a.opt_tensor(8), own = a.opt_tensor(10);
  Tensor y = a.opt_tensor(11);
  if (slots.defined()) {
    need(slots.dim() == 3 && slots.scalar_type() == at::kHalf && slots.select(0, 0).is_contiguous() && x.data_ptr() == slots.data_ptr(),
         "partials: fp16 (n, M, N) slots with contiguous rows, x = slots[0]");
    need(!own.defined() || (own.sizes() == x.sizes() && own.scalar_type() == at::kHalf && own.strides() == x.strides()),
         "partials: own piece must have the shape and strides of a slot");
  }
  check_norm(x, w, bias);
  const int64_t m = x.size(0), n = x.size(1);
  int code = a.integer(6);
  on_gpu(res, "residual");
  if (res.defined()) {
    need(res.sizes() == x.sizes() && res.stride(-1) == 1, "residual must have the shape of x");
    need(res.scalar_type() == at::kHalf || res.scalar_type() == at::kFloat, "residual must be float16 or float32");
    code = res.scalar_type() == at::kFloat ? 2 : 1;
  } else if (code == 1) {
    code = 0;                     // x itself is the fp16 residual
  }
  need(n * 2 < 65536, "This layer norm doesn't support feature dim >= 64KB.");
  Device dev(x);
  if (y.defined())
    need(y.scalar_type() == at::kChar && y.dim() == 2 && y.size(0) == m && y.size(1) == n && y.stride(1) == 1 && y.device() == x.device(),
         "out must be an int8 (M, N) tensor on x's device, contiguous in its last dim");
  else
    y = dev.empty({m, n}, at::kChar);
  Tensor ro;
  if (code != 0) ro = dev.empty({m, n}, code == 2 ? at::kFloat : at::kHalf);
  const double scale = a.num_or(5, 0.0);
  const bool fixed = scale != 0.0;   // the reference tests truthiness: None and 0.0 both mean per-token scales
  Tensor dyn;
  if (!fixed) dyn = dev.empty({m}, at::kFloat);
  if (m > 0) {
    qb_rmsnorm_args s{};
    s.x = x.data_ptr(); s.weight = w.data_ptr(); s.bias = ptr(bias); s.residual = ptr(res); s.residual_out = ptr(ro); s.out = y.data_ptr();
    s.dyn_scale = fixed ? nullptr : f32(dyn);
    s.x_row_stride = x.stride(0); s.out_row_stride = y.stride(0);
    if (res.defined()) { s.residual_row_stride = res.stride(0); s.residual_is_f32 = res.scalar_type() == at::kFloat; }
    if (ro.defined()) { s.residual_out_row_stride = n; s.residual_out_is_f32 = code == 2; }
    s.rows = m; s.group_size = n; s.ngroups = 1; s.out_kind = fixed ? 0 : 1; s.norm_before_gate = 1; s.is_rms_norm = a.flag(7);
    s.eps = a.num(3); s.out_scale = scale;
    if (slots.defined()) {
      s.n_partials = slots.size(0); s.partial_stride = slots.stride(0); s.own_index = own.defined() ? a.integer(9) : -1; s.own_partial = ptr(own);
    }
    QBN_CALL(qb_rmsnorm_quant, s, dev.stream);
  }
  return wrap_tuple({y, ro.defined() ? ro : x, dyn});
}

// (x, weight, bias, eps, z, z_scale, static_scale | None, fp16_out, group_size, norm_before_gate, is_rms)
PyObject* normgated_fwd(const Args& a) {
  const Tensor x = a.tensor(0), w = a.tensor(1), bias = a.opt_tensor(2), z = a.opt_tensor(4);
  need(x.is_cuda() && x.scalar_type() == at::kHalf && x.dim() == 2, "x must be a 2-D float16 CUDA tensor");
  const int64_t m = x.size(0), n = x.size(1), gs = a.is_none(8) ? n : a.integer(8);
  need(gs > 0 && n % gs == 0, "the feature dim must be divisible by group_size");
  if (z.defined()) {
    cuda_i8(z, "q_z");
    need(z.sizes() == x.sizes() && z.stride(-1) == 1, "q_z must have the shape of x");
    need(!a.is_none(5), "q_z needs z_scale");
  }
  check_norm(x, w, bias);
  need(gs * 2 < 65536, "This layer norm doesn't support feature dim >= 64KB.");
  const bool half = a.flag(7);
  Device dev(x);
  Tensor out = dev.empty({m, n}, half ? at::kHalf : at::kChar), dyn = dev.empty({n / gs * m}, at::kFloat);
  if (m > 0) {
    qb_rmsnorm_args s{};
    s.x = x.data_ptr(); s.weight = w.data_ptr(); s.bias = ptr(bias); s.z = i8(z); s.out = out.data_ptr(); s.dyn_scale = f32(dyn);
    s.x_row_stride = x.stride(0); s.out_row_stride = n; s.z_row_stride = z.defined() ? z.stride(0) : 0;
    s.rows = m; s.group_size = gs; s.ngroups = n / gs; s.out_kind = half ? 2 : (a.is_none(6) ? 1 : 0);
    s.norm_before_gate = a.flag(9); s.is_rms_norm = a.flag(10); s.eps = a.num(3);
    s.out_scale = s.out_kind == 0 ? a.num(6) : 0.0; s.z_scale = a.num_or(5, 0.0);
    QBN_CALL(qb_rmsnorm_gated, s, dev.stream);
  }
  return wrap_tuple({out, dyn});
}

PyMethodDef kMethods[] = {
    {"set_trace", set_trace, METH_O, nullptr},
    {"set_types", set_types, METH_O, nullptr},
    QBN_METHOD(conv1_fwd), QBN_METHOD(conv1_update), QBN_METHOD(conv2_fwd), QBN_METHOD(conv2_update), QBN_METHOD(hadamard),
    QBN_METHOD(sscan_fwd), QBN_METHOD(sscan_update), QBN_METHOD(ssd), QBN_METHOD(w4a8), QBN_METHOD(w8a8_mm), QBN_METHOD(w8a8_mv),
    QBN_METHOD(norm_fwd), QBN_METHOD(normgated_fwd), QBN_METHOD(mamba2_layer), QBN_METHOD(mamba1_layer),
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_native", "Host path of quamba_b200 (see csrc/binding.cpp).", -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace
}  // namespace qbn

PyMODINIT_FUNC PyInit__native() {
  PyObject* m = PyModule_Create(&qbn::kModule);
  if (m != nullptr && PyModule_AddStringConstant(m, "torch_version", QBN_TORCH_VERSION) < 0) {
    Py_DECREF(m);
    return nullptr;
  }
  return m;
}
