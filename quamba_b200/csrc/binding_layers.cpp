// Whole layers in one host call (see binding.cpp): the launch sequence of the Python modules' forward / step, issued from
// their buffers and scales with intermediates taken straight from the caching allocator.
#include "binding.h"

namespace qbn {

Types g_types{};

namespace {
PyObject *g_hooks = nullptr, *g_pre_hooks = nullptr;         // torch's hooks on every module
PyTypeObject *g_w4_mamba2 = nullptr, *g_w8_mamba2 = nullptr, *g_w4_mamba1 = nullptr, *g_w8_mamba1 = nullptr;
}  // namespace

PyObject* set_types(PyObject*, PyObject* dict) {
  auto type = [&](const char* name) -> PyTypeObject* {
    PyObject* o = PyDict_GetItemString(dict, name);
    if (o == nullptr || !PyType_Check(o)) return nullptr;
    return reinterpret_cast<PyTypeObject*>(Py_NewRef(o));
  };
  Types& t = g_types;
  t.QRMSNorm = type("QRMSNorm"); t.QRMSNormGated = type("QRMSNormGated"); t.Quamb2Conv1D = type("Quamb2Conv1D");
  t.Quamba2ChunkScan = type("Quamba2ChunkScan"); t.QHadamard = type("QHadamard"); t.QCausalConv1D = type("QCausalConv1D");
  t.QSScan = type("QSScan"); t.W4A8B16O16Linear = type("W4A8B16O16Linear"); t.W4A8B8O8Linear = type("W4A8B8O8Linear");
  t.W4A8B8O8LinearParallel = type("W4A8B8O8LinearParallel"); t.W8A8B8O8Linear = type("W8A8B8O8Linear");
  t.W8A8B8O8LinearParallel = type("W8A8B8O8LinearParallel"); t.W8A8B16O16Linear = type("W8A8B16O16Linear");
  g_w4_mamba2 = type("W4A8QMamba2"); g_w8_mamba2 = type("W8A8QMamba2");
  g_w4_mamba1 = type("W4A8QMamba"); g_w8_mamba1 = type("W8A8QMamba");
  g_hooks = PyDict_GetItemString(dict, "forward_hooks");
  g_pre_hooks = PyDict_GetItemString(dict, "forward_pre_hooks");
  Py_XINCREF(g_hooks);
  Py_XINCREF(g_pre_hooks);
  Py_RETURN_NONE;
}

Mod::Mod(PyObject* o) : self(Ref::share(o)), attrs(Ref::own(PyObject_GenericGetDict(o, nullptr))) {
  if (attrs == nullptr) throw PyErr{};
  buffers = Ref::share(PyDict_GetItem(attrs, QBN_NAME(_buffers)));
  if (buffers == nullptr) throw NotPlain{};
}

void Mod::require_plain(PyTypeObject* type) const {
  auto empty = [&](PyObject* name) {
    PyObject* d = PyDict_GetItem(attrs, name);
    return d == nullptr || (PyDict_Check(d) && PyDict_GET_SIZE(d) == 0);
  };
  if ((type != nullptr && Py_TYPE(self) != type) || !empty(QBN_NAME(_forward_hooks)) || !empty(QBN_NAME(_forward_pre_hooks)) ||
      PyDict_GetItem(attrs, QBN_NAME(forward)) != nullptr)
    throw NotPlain{};
}

void Mod::require_own(PyObject* method) const {
  if (PyDict_GetItem(attrs, method) != nullptr) throw NotPlain{};
}

Mod Mod::child(PyObject* name, PyTypeObject* type) const {
  PyObject* mods = PyDict_GetItem(attrs, QBN_NAME(_modules));
  PyObject* c = mods != nullptr ? PyDict_GetItem(mods, name) : nullptr;
  if (c == nullptr || c == Py_None) throw NotPlain{};
  Mod m(c);
  m.require_plain(type);
  return m;
}

void Conv2::check() {
  on_gpu(bias, "bias"); on_gpu(hgr, "x_head_group_range"); on_gpu(dgr, "x_dim_group_range");
  cuda_f32(out_scale[0], "x_scales"); cuda_f32(out_scale[1], "B_scales"); cuda_f32(out_scale[2], "C_scales");
  if (hgr.defined() && dgr.defined()) {
    need(hgr.scalar_type() == at::kInt && dgr.scalar_type() == at::kInt, "group ranges must be int32");
    need(hgr.size(0) == groups && dgr.size(0) == groups, "x_head_group_range.shape[0] / x_dim_group_range.shape[0] must equal the number of groups");
    const int64_t nh = hgr.size(1), nd = dgr.size(2);
    need(dgr.size(1) == nh, "x_dim_group_range.shape[1] must equal the number of head groups");
    need(out_scale[0].numel() == groups * nh * nd, "number of x scales must equal the number of groups");
    need(out_scale[1].numel() == groups && out_scale[2].numel() == groups, "number of B / C scales must equal the number of SSD groups");
    hgr = contiguous(hgr);
    dgr = contiguous(dgr);
  } else {
    need(!hgr.defined() && !dgr.defined(), "x_head_group_range and x_dim_group_range must be both None or both set");
    need(out_scale[0].numel() == 1 && out_scale[1].numel() == 1 && out_scale[2].numel() == 1, "number of x / B / C scales must be equal to 1");
  }
}

// ---- linears --------------------------------------------------------------------------------------------------------------
namespace {
PyObject* attrs_of(PyObject* o) {
  PyObject* d = PyObject_GenericGetDict(o, nullptr);
  if (d == nullptr) throw PyErr{};
  Py_DECREF(d);
  return d;
}
PyObject* item(PyObject* d, PyObject* name) {
  PyObject* r = PyDict_GetItem(d, name);
  if (r == nullptr) throw std::runtime_error("prepared weight without " + std::string(PyUnicode_AsUTF8(name)));
  return r;
}
// a streaming copy of the prepared weight: the attribute, or what the method that builds it returns
Tensor copy_of(PyObject* prep, PyObject* d, PyObject* attr, PyObject* method) {
  PyObject* t = item(d, attr);
  if (t != Py_None) return as_tensor(t);
  PyObject* made = PyObject_CallMethodNoArgs(prep, method);
  if (made == nullptr) throw PyErr{};
  Tensor r = as_tensor(made);
  Py_DECREF(made);
  return r;
}
}  // namespace

W4Dims w4_dims(PyObject* prep) {
  PyObject* d = attrs_of(prep);
  return {as_long(item(d, QBN_NAME(size_n))), as_long(item(d, QBN_NAME(size_k))), PyObject_IsTrue(item(d, QBN_NAME(per_channel))) == 1};
}

void w4a8_run(PyObject* prep, const W4Dims& w, const int8_t* a, int64_t lda, int64_t m, const float* s_tok, bool per_row, void* out,
              int64_t ldo, bool int8, bool transpose, cudaStream_t st) {
  PyObject* d = attrs_of(prep);
  auto common = [&](auto& s) {
    s.a = a; s.s_tok = s_tok; s.out = out; s.a_row_stride = lda; s.out_row_stride = ldo; s.m = m; s.n = w.n; s.k = w.k;
    s.s_tok_per_row = per_row; s.out_int8 = int8; s.output_transpose = transpose;
  };
  if (m <= 8 && w.per_channel && w.k % 32 == 0 && lda % 16 == 0 && reinterpret_cast<uintptr_t>(a) % 16 == 0) {
    // a few rows on per-channel weights: stream the nibble copy (half the bytes, identical results); from nine rows on the
    // tensor-core kernel on the int8 copy is faster than re-streaming the weights for every eight rows
    const Tensor w4 = copy_of(prep, d, QBN_NAME(w4), QBN_NAME(need_w4)), sc = as_tensor(item(d, QBN_NAME(sc)));
    qb_w4a8_gemv_s4_args s{};
    common(s);
    s.w4 = static_cast<const uint8_t*>(w4.data_ptr()); s.s_channel_nat = f32(sc);
    QBN_CALL(qb_w4a8_gemv_s4, s, st);
    return;
  }
  const Tensor w8 = copy_of(prep, d, QBN_NAME(w8), QBN_NAME(need_w8)), sc = as_tensor(item(d, QBN_NAME(sc)));
  qb_w4a8_gemm_args s{};
  common(s);
  s.w8 = i8(w8); s.s_channel_nat = f32(sc);
  QBN_CALL(qb_w4a8_gemm, s, st);
}

namespace {

// One linear module of a layer: n output columns (padded), of which `features` are the caller's.
struct Lin {
  Mod m;
  int64_t k, n, features;
  bool w4, int8;
  Tensor w, sa, sb;                                          // W8A8: weight and scales; W4A8: the input scale in sa
  Ref alpha;                                                 // W8A8 with one scale per side: what a single row is scaled by
  Lin(const Mod& parent, PyObject* name, c10::Device dev) : m(open(parent, name)) {
    const Types& t = g_types;
    PyTypeObject* ty = Py_TYPE(m.self);
    w4 = ty == t.W4A8B16O16Linear || ty == t.W4A8B8O8Linear || ty == t.W4A8B8O8LinearParallel;
    if (!w4 && ty != t.W8A8B8O8Linear && ty != t.W8A8B8O8LinearParallel && ty != t.W8A8B16O16Linear) throw NotPlain{};
    int8 = ty != t.W4A8B16O16Linear && ty != t.W8A8B16O16Linear;
    features = m.integer(QBN_NAME(out_features));
    k = m.integer(QBN_NAME(in_features));
    n = features + m.integer(QBN_NAME(pad_out));
    if (w4) {
      if (m.integer(QBN_NAME(size_n)) != n || m.integer(QBN_NAME(size_k)) != k) throw NotPlain{};
      m.tensor_on(QBN_NAME(weight), at::kInt, dev);
      sa = m.tensor_on(QBN_NAME(input_scale), at::kFloat, dev);
    } else {
      w = m.tensor_on(QBN_NAME(weight), at::kChar, dev); sa = m.tensor_on(QBN_NAME(a), at::kFloat, dev); sb = m.tensor_on(QBN_NAME(b), at::kFloat, dev);
      if (ty != t.W8A8B8O8LinearParallel) alpha = Ref::share(m.get(QBN_NAME(alpha)));
      if (w.dim() != 2 || w.size(0) != k || w.size(1) != n || w.stride(0) != 1 || w.stride(1) % 16 != 0 || !sa.is_contiguous() || !sb.is_contiguous() ||
          sa.numel() != 1 || (sb.numel() != 1 && sb.numel() != n))
        throw NotPlain{};
    }
  }
  // has to_seqlen_last, the form a Mamba1 prefill multiplies with: one scale per side, whose places it swaps
  bool seqlen_last() const {
    const PyTypeObject* ty = Py_TYPE(m.self);
    return ty == g_types.W4A8B8O8Linear || (ty == g_types.W8A8B8O8Linear && sb.numel() == 1);
  }
  static Mod open(const Mod& parent, PyObject* name) { return parent.child(name, nullptr); }

  // the module's prepared weight, built or rebuilt by prepared() when a buffer was replaced or written in place
  Ref prepared() const {
    const Ref p = Ref::share(PyDict_GetItem(m.attrs, QBN_NAME(_prep)));
    if (p != nullptr && p != Py_None) {
      PyObject* d = attrs_of(p);
      PyObject* src = item(d, QBN_NAME(_src));
      PyObject* ver = item(d, QBN_NAME(versions));
      PyObject* names[3] = {QBN_NAME(weight), QBN_NAME(s_channel), QBN_NAME(s_group)};
      bool fresh = true;
      for (int i = 0; i < 3 && fresh; ++i) {
        PyObject* b = m.get(names[i]);
        fresh = PyWeakref_GetObject(PyTuple_GET_ITEM(src, i)) == b && as_long(PyTuple_GET_ITEM(ver, i)) == (long)as_tensor(b)._version();
      }
      if (fresh) return p;
    }
    const Ref q = Ref::own(PyObject_CallMethodNoArgs(m.self, QBN_NAME(prepared)));
    if (q == nullptr) throw PyErr{};
    return q;
  }

  // as_matrix: the matrix form even for one row, with the two scales applied in the order of to_seqlen_last
  void run(const int8_t* a, int64_t lda, int64_t rows, void* out, int64_t ldo, cudaStream_t st, bool as_matrix = false) const {
    if (w4) {
      const Ref p = prepared();
      const W4Dims d = w4_dims(p);
      need(d.n == n && d.k == k, "the weight was replaced by one of another shape during the call");
      w4a8_run(p, d, a, lda, rows, f32(sa), false, out, ldo, int8, false, st);
      return;
    }
    qb_w8a8_gemm_args s{};
    s.a = a; s.b = i8(w); s.out = out; s.a_row_stride = lda; s.b_col_stride = w.stride(1); s.out_row_stride = ldo;
    s.m = rows; s.n = n; s.k = k; s.out_dtype = int8 ? 0 : 1;
    if (as_matrix) {
      s.a_scale = f32(sb); s.b_scale = f32(sa);
    } else if (rows == 1 && alpha != nullptr) {
      s.use_alpha = 1;
      s.alpha = as_double(alpha);
    } else {
      s.a_scale = f32(sa); s.b_scale = f32(sb); s.b_scale_per_col = sb.numel() != 1;
      s.round_half_away = rows == 1;
    }
    QBN_CALL(qb_w8a8_gemm, s, st);
  }
};

// The block norm in front of a layer: hidden (+ residual) -> int8 rows and the new residual.
struct BlockNorm {
  Tensor rows, residual;
  BlockNorm(PyObject* norm, const Tensor& x, PyObject* res_obj, bool fp32, int64_t m, int64_t n, const Device& dev) {
    Mod nm(norm);
    nm.require_plain(g_types.QRMSNorm);
    const Tensor w = nm.tensor_on(QBN_NAME(weight), at::kHalf, dev.dev), bias = nm.opt_tensor(QBN_NAME(bias));
    const double scale = nm.num_or(QBN_NAME(output_scale), 0.0);
    if (scale == 0.0 || bias.defined() || w.numel() != n || !w.is_contiguous() || x.scalar_type() != at::kHalf || n * 2 >= 65536)
      throw NotPlain{};
    qb_rmsnorm_args s{};
    bool f32_out = fp32;
    if (res_obj != Py_None) {
      const Tensor r = as_tensor(res_obj);
      if (r.sizes() != x.sizes() || r.device() != x.device() || !r.is_contiguous() || (r.scalar_type() != at::kHalf && r.scalar_type() != at::kFloat)) throw NotPlain{};
      f32_out = r.scalar_type() == at::kFloat;
      s.residual = r.data_ptr(); s.residual_row_stride = n; s.residual_is_f32 = f32_out;
    }
    rows = dev.empty({m, n}, at::kChar);
    if (res_obj != Py_None || f32_out) {
      residual = dev.empty(x.sizes(), f32_out ? at::kFloat : at::kHalf);
      s.residual_out = residual.data_ptr(); s.residual_out_row_stride = n; s.residual_out_is_f32 = f32_out;
    } else {
      residual = x;
    }
    s.x = x.data_ptr(); s.weight = w.data_ptr(); s.out = rows.data_ptr(); s.x_row_stride = n; s.out_row_stride = n;
    s.rows = m; s.group_size = n; s.ngroups = 1; s.norm_before_gate = 1; s.is_rms_norm = 1;
    s.eps = nm.num(QBN_NAME(eps)); s.out_scale = scale;
    QBN_CALL(qb_rmsnorm_quant, s, dev.stream);
  }
};

struct Rotation {
  int64_t blocks, special;
  double scale;
  explicit Rotation(const Mod& had) : blocks(had.integer(QBN_NAME(blocks))), special(had.integer(QBN_NAME(N))) {
    if (special == 2) special = 1;
    scale = had.num(QBN_NAME(had_scale)) / had.num(QBN_NAME(x_H_scale));
  }
  void run(const Tensor& y, const Tensor& out, int64_t rows, int64_t width, cudaStream_t st) const {
    qb_hadamard_quant_args s{};
    s.x = y.data_ptr(); s.out = i8(out); s.dim = width / blocks; s.x_row_stride = s.out_row_stride = s.dim; s.rows = rows * blocks;
    s.special = special; s.scale = scale;
    QBN_CALL(qb_hadamard_quant, s, st);
  }
};

// (rows, n) fp16 -> (batch, len, features)
Tensor layer_output(const Tensor& out, int64_t batch, int64_t len, const Lin& lin) {
  if (lin.features == lin.n) return out;
  return out.narrow(-1, 0, lin.features).reshape({batch, len, lin.features});
}

}  // namespace

// (norm | None, mixer, hidden, residual | None, residual_in_fp32, conv_state | None, ssm_state | None, decode)
// -> (output, residual), or the output alone without a norm; None when the layer has to be walked module by module.
// hidden (batch, len, d_model): fp16 with a norm, the norm's int8 rows without.
PyObject* mamba2_layer(const Args& a) {
  const Mod mx(a.object(1));
  const bool has_norm = !a.is_none(0), decode = a.flag(7);
  if (Py_TYPE(mx.self) != g_w4_mamba2 && Py_TYPE(mx.self) != g_w8_mamba2) throw NotPlain{};   // a subclass may have a forward or step of its own
  if (has_norm) mx.require_plain(nullptr);
  if (decode) mx.require_own(QBN_NAME(step));
  if ((g_hooks != nullptr && PyDict_GET_SIZE(g_hooks) != 0) || (g_pre_hooks != nullptr && PyDict_GET_SIZE(g_pre_hooks) != 0)) throw NotPlain{};
  const Tensor x = a.tensor(2);
  if (!x.is_cuda() || x.dim() != 3 || !x.is_contiguous() || x.numel() == 0) throw NotPlain{};
  const int64_t batch = x.size(0), len = x.size(1), dm = x.size(2), rows = batch * len;
  if (decode && len != 1) throw NotPlain{};
  const c10::Device on = x.device();
  const Lin in(mx, QBN_NAME(in_proj), on), outp(mx, QBN_NAME(out_proj), on);
  const Mod conv = mx.child(QBN_NAME(conv1d), g_types.Quamb2Conv1D), scan = mx.child(QBN_NAME(qchunk_scan), g_types.Quamba2ChunkScan),
            gn_m = mx.child(QBN_NAME(norm), g_types.QRMSNormGated), had_m = mx.child(QBN_NAME(had), g_types.QHadamard);
  if (decode) { conv.require_own(QBN_NAME(update)); scan.require_own(QBN_NAME(update)); }
  const int64_t d = mx.integer(QBN_NAME(d_ssm)), groups = mx.integer(QBN_NAME(ngroups)), ds = mx.integer(QBN_NAME(d_state)),
                nh = mx.integer(QBN_NAME(nheads)), hd = mx.integer(QBN_NAME(headdim)), gn = groups * ds, dim = d + 2 * gn;
  if (in.k != dm || !in.int8 || outp.int8 || outp.k != d || in.features != d + dim + nh || nh * hd != d) throw NotPlain{};
  const Tensor conv_st = a.opt_tensor(5), ssm_st = a.opt_tensor(6);
  auto is = [](const Tensor& t, std::initializer_list<int64_t> v) { return t.sizes() == at::IntArrayRef(v.begin(), v.size()); };
  if (decode && !conv_st.defined()) throw NotPlain{};
  if (conv_st.defined() && (conv_st.scalar_type() != at::kChar || !is(conv_st, {batch, dim, 4}) || ssm_st.scalar_type() != at::kChar ||
                            !is(ssm_st, {batch, nh, hd, ds}) || !ssm_st.is_contiguous() || conv_st.device() != on || ssm_st.device() != on ||
                            (conv_st.stride(1) == 1 && (conv_st.stride(0) % 4 != 0 || conv_st.stride(2) % 4 != 0 || reinterpret_cast<uintptr_t>(conv_st.data_ptr()) % 4 != 0))))
    throw NotPlain{};

  Conv2 c;
  c.weight = conv.tensor_on(QBN_NAME(weight), at::kChar, on); c.bias = conv.opt_tensor_on(QBN_NAME(bias), at::kChar, on);
  c.hgr = conv.opt_tensor_on(QBN_NAME(x_head_group_range), at::kInt, on); c.dgr = conv.opt_tensor_on(QBN_NAME(x_dim_group_range), at::kInt, on);
  PyObject* so[3] = {QBN_NAME(x_out_scales), QBN_NAME(B_out_scales), QBN_NAME(C_out_scales)};
  PyObject* si[3] = {QBN_NAME(x_scale), QBN_NAME(B_scale), QBN_NAME(C_scale)};
  PyObject* sw[3] = {QBN_NAME(wx_scale), QBN_NAME(wB_scale), QBN_NAME(wC_scale)};
  PyObject* sb[3] = {QBN_NAME(bx_scale), QBN_NAME(bB_scale), QBN_NAME(bC_scale)};
  for (int i = 0; i < 3; ++i) {
    c.out_scale[i] = conv.tensor_on(so[i], at::kFloat, on);
    c.in[i] = conv.num(si[i]); c.w_scale[i] = conv.num(sw[i]); c.b_scale[i] = conv.num_or(sb[i], 0.0);
  }
  c.x_dim = conv.integer(QBN_NAME(x_dim)); c.headdim = conv.integer(QBN_NAME(x_headdim)); c.d_state = conv.integer(QBN_NAME(d_state));
  c.groups = conv.integer(QBN_NAME(n_groups));
  if (c.x_dim != d || c.d_state * c.groups != gn || !is(c.weight, {dim, 4}) || !c.weight.is_contiguous() || (c.bias.defined() && !c.bias.is_contiguous()))
    throw NotPlain{};
  c.check();

  auto scale = [&](PyObject* name) { return scan.tensor_on(name, at::kFloat, on); };
  const Tensor A = scan.tensor_on(QBN_NAME(A_log), at::kChar, on), D = scan.opt_tensor_on(QBN_NAME(D), at::kChar, on),
               bias = scan.opt_tensor_on(QBN_NAME(dt_bias), at::kHalf, on), ss = scale(QBN_NAME(ssm_state_scale)), xs = scale(QBN_NAME(x_scales)),
               Bs = scale(QBN_NAME(B_scale)), Cs = scale(QBN_NAME(C_scale)), dts = scale(QBN_NAME(dt_scale)), As = scale(QBN_NAME(A_log_scale)),
               hgr = scan.opt_tensor_on(QBN_NAME(x_head_group_range), at::kInt, on), dgr = scan.opt_tensor_on(QBN_NAME(x_dim_group_range), at::kInt, on);
  const Tensor Ds = D.defined() ? scale(QBN_NAME(D_scale)) : Tensor();
  const bool hdim = scan.flag(QBN_NAME(D_has_hdim)), grouped = hgr.defined();
  if (A.numel() != nh || !A.is_contiguous() || (D.defined() && (D.numel() != (hdim ? d : nh) || !D.is_contiguous())) ||
      (bias.defined() && (bias.numel() != nh || !bias.is_contiguous())) || grouped != dgr.defined() ||
      (grouped && (!hgr.is_contiguous() || !dgr.is_contiguous() || hgr.dim() != 2 || dgr.dim() != 3 || !is(ss, {groups, hgr.size(1), dgr.size(2), ds}) || !ss.is_contiguous() ||
                   xs.numel() != groups * hgr.size(1) * dgr.size(2) || Bs.numel() != groups || Cs.numel() != groups)) ||
      (!grouped && (xs.numel() != 1 || Bs.numel() != 1 || Cs.numel() != 1 || ss.numel() != 1)))
    throw NotPlain{};
  const Tensor gw = gn_m.tensor_on(QBN_NAME(weight), at::kHalf, on);
  const int64_t gsize = gn_m.get(QBN_NAME(group_size)) == Py_None ? d : gn_m.integer(QBN_NAME(group_size));
  if (!gn_m.flag(QBN_NAME(use_float16_output)) || gn_m.get(QBN_NAME(bias)) != Py_None || gw.numel() != d || !gw.is_contiguous() ||
      gsize <= 0 || d % gsize != 0)
    throw NotPlain{};
  PyObject* lim = scan.get(QBN_NAME(dt_limit));
  if (!PyTuple_Check(lim) || PyTuple_GET_SIZE(lim) != 2) throw NotPlain{};
  const double dt_min = as_double(PyTuple_GET_ITEM(lim, 0)), dt_max = std::min(as_double(PyTuple_GET_ITEM(lim, 1)), 3.0e38);
  const bool softplus = scan.flag(QBN_NAME(delta_softplus)), before_gate = gn_m.flag(QBN_NAME(norm_before_gate));
  const int64_t chunk = scan.integer(QBN_NAME(chunk_size));
  const double g_eps = gn_m.num(QBN_NAME(eps)), g_z = gn_m.num(QBN_NAME(z_scale));
  const Rotation had(had_m);
  if (had.blocks <= 0 || d % had.blocks != 0) throw NotPlain{};

  const Device dev(x);
  const cudaStream_t st = dev.stream;
  Tensor u = x, residual;
  if (has_norm) {
    BlockNorm n(a.object(0), x, a.object(3), a.flag(4), rows, dm, dev);
    u = n.rows;
    residual = n.residual;
  } else if (x.scalar_type() != at::kChar) {
    throw NotPlain{};
  }
  // in_proj: one int8 row [z | x B C | dt] per token, read below through strided views
  const Tensor zx = dev.empty({rows, in.n}, at::kChar);
  in.run(i8(u), dm, rows, zx.data_ptr(), in.n, st);
  int8_t* z = i8(zx);
  int8_t *xbc = z + d, *dt = z + d + dim;
  const Tensor cx = dev.empty({rows, d}, at::kChar), cB = dev.empty({rows, gn}, at::kChar), cC = dev.empty({rows, gn}, at::kChar);
  Tensor y = dev.empty({rows, d}, at::kHalf);
  auto scan_common = [&](auto& s) {
    s.x = i8(cx); s.dt = dt; s.Bm = i8(cB); s.Cm = i8(cC); s.A_log = i8(A); s.D = i8(D); s.dt_bias = ptr(bias);
    s.x_scales = f32(xs); s.dt_scale = f32(dts); s.A_scale = f32(As); s.B_scale = f32(Bs); s.C_scale = f32(Cs); s.D_scale = f32(Ds);
    s.head_group_range = i32(hgr); s.dim_group_range = i32(dgr); s.out = y.data_ptr();
    s.batch = batch; s.nheads = nh; s.headdim = hd; s.ngroups = groups; s.dstate = ds; s.grouped = grouped;
    s.nhead_groups = grouped ? hgr.size(1) : 0; s.ndim_groups = grouped ? dgr.size(2) : 0; s.dt_softplus = softplus;
  };
  if (decode) {
    qb_quamba2_conv1d_update_args s = c.update_args(dim);
    s.xBC = xbc; s.xBC_sb = in.n; s.conv_state = i8(conv_st); s.state_sb = conv_st.stride(0); s.state_sd = conv_st.stride(1); s.state_sw = conv_st.stride(2);
    s.x = i8(cx); s.Bm = i8(cB); s.Cm = i8(cC); s.batch = batch;
    QBN_CALL(qb_quamba2_conv1d_update, s, st);
    qb_sscan_update_args t{};
    scan_common(t);
    t.state = i8(ssm_st); t.state_scale = f32(ss); t.state_sb = d * ds; t.state_sh = hd * ds; t.state_sp = ds;
    t.x_sb = d; t.x_sh = hd; t.dt_sb = in.n; t.dt_sh = 1; t.A_sh = 1; t.B_sb = t.C_sb = gn; t.B_sg = t.C_sg = ds;
    t.D_sh = D.defined() ? (hdim ? hd : 1) : 0; t.D_sp = D.defined() && hdim ? 1 : 0; t.bias_sh = bias.defined() ? 1 : 0;
    t.out_sb = d; t.out_sh = hd; t.dt_bias_is_half = bias.defined();
    QBN_CALL(qb_sscan_update, t, st);
  } else {
    qb_quamba2_conv1d_fwd_args s = c.fwd_args(dim);
    s.xBC = xbc; s.xBC_sb = len * in.n; s.xBC_sl = in.n; s.x = i8(cx); s.Bm = i8(cB); s.Cm = i8(cC); s.batch = batch; s.seqlen = len;
    if (conv_st.defined()) {       // the last four inputs of every channel go to the decode cache
      s.conv_state = i8(conv_st); s.state_sb = conv_st.stride(0); s.state_sd = conv_st.stride(1); s.state_sw = conv_st.stride(2);
    }
    QBN_CALL(qb_quamba2_conv1d_fwd, s, st);
    qb_ssd_args t{};
    scan_common(t);
    const int64_t wsb = qb_ssd_workspace_bytes(batch, len, nh, hd, groups, ds, chunk);
    need(wsb > 0, "invalid SSD shape");
    const Tensor ws = dev.empty({wsb}, at::kByte);
    const Tensor fin = ssm_st.defined() ? ssm_st : dev.empty({batch, nh, hd, ds}, at::kChar);
    t.ssm_state_scale = f32(ss); t.final_states = i8(fin); t.workspace = ws.data_ptr(); t.workspace_bytes = wsb;
    t.x_sb = len * d; t.x_sl = d; t.x_sh = hd; t.dt_sb = len * in.n; t.dt_sl = in.n; t.B_sb = t.C_sb = len * gn; t.B_sl = t.C_sl = gn; t.B_sg = t.C_sg = ds;
    t.seqlen = len; t.chunk_size = chunk; t.D_has_hdim = D.defined() && hdim;
    t.dt_min = dt_min; t.dt_max = dt_max;
    QBN_CALL(qb_ssd_chunk_scan_fwd, t, st);
  }
  const Tensor g = dev.empty({rows, d}, at::kHalf);
  qb_rmsnorm_args s{};
  s.x = y.data_ptr(); s.weight = gw.data_ptr(); s.z = z; s.out = g.data_ptr(); s.x_row_stride = s.out_row_stride = d; s.z_row_stride = in.n;
  s.rows = rows; s.group_size = gsize; s.ngroups = d / gsize; s.out_kind = 2; s.norm_before_gate = before_gate; s.is_rms_norm = 1;
  s.eps = g_eps; s.z_scale = g_z;
  QBN_CALL(qb_rmsnorm_gated, s, st);
  const Tensor q = dev.empty({rows, d}, at::kChar);
  had.run(g, q, rows, d, st);
  Tensor out = dev.empty({batch, len, outp.n}, at::kHalf);
  outp.run(i8(q), d, rows, out.data_ptr(), outp.n, st);
  out = layer_output(out, batch, len, outp);
  return has_norm ? wrap_tuple({out, residual}) : wrap(out);
}

// The Mamba1 counterpart: (norm | None, mixer, hidden, residual | None, residual_in_fp32, conv_state | None, ssm_state | None,
// decode).  Prefill runs channel-last from in_proj to the scan, so none of the module walk's transposes exist here.
PyObject* mamba1_layer(const Args& a) {
  const Mod mx(a.object(1));
  const bool has_norm = !a.is_none(0), decode = a.flag(7);
  if (Py_TYPE(mx.self) != g_w4_mamba1 && Py_TYPE(mx.self) != g_w8_mamba1) throw NotPlain{};   // a subclass may have a forward or step of its own
  if (has_norm) mx.require_plain(nullptr);
  if (decode) mx.require_own(QBN_NAME(step));
  if ((g_hooks != nullptr && PyDict_GET_SIZE(g_hooks) != 0) || (g_pre_hooks != nullptr && PyDict_GET_SIZE(g_pre_hooks) != 0)) throw NotPlain{};
  const Tensor x = a.tensor(2);
  if (!x.is_cuda() || x.dim() != 3 || !x.is_contiguous() || x.numel() == 0) throw NotPlain{};
  const int64_t batch = x.size(0), len = x.size(1), dm = x.size(2), rows = batch * len;
  if (decode && len != 1) throw NotPlain{};
  const c10::Device on = x.device();
  const Lin in(mx, QBN_NAME(in_proj), on), xp(mx, QBN_NAME(x_proj), on), dtp(mx, QBN_NAME(dt_proj), on), outp(mx, QBN_NAME(out_proj), on);
  const Mod conv = mx.child(QBN_NAME(conv1d), g_types.QCausalConv1D), scan = mx.child(QBN_NAME(selective_scan), g_types.QSScan),
            had_m = mx.child(QBN_NAME(had), g_types.QHadamard);
  if (decode) { conv.require_own(QBN_NAME(update)); scan.require_own(QBN_NAME(update)); }
  else { in.m.require_own(QBN_NAME(to_seqlen_last)); dtp.m.require_own(QBN_NAME(to_seqlen_last)); }
  const int64_t d = mx.integer(QBN_NAME(d_inner)), ds = mx.integer(QBN_NAME(d_state)), rank = mx.integer(QBN_NAME(dt_rank));
  if (in.k != dm || in.features != 2 * d || xp.k != d || xp.features != rank + 2 * ds || dtp.k != rank || dtp.features != d || dtp.n != d || outp.k != d ||
      !in.int8 || !xp.int8 || !dtp.int8 || outp.int8 || (!decode && (!in.seqlen_last() || !dtp.seqlen_last())) || ds != 16 || d % 16 != 0 || rank % 4 != 0)
    throw NotPlain{};
  // the channel-last scan counts a sequence's elements in 31 bits and the sequences in 16
  if (!decode && (std::max({in.n, xp.n, d}) * len >= (int64_t(1) << 31) || batch >= 65536)) throw NotPlain{};
  const Tensor conv_st = a.opt_tensor(5), ssm_st = a.opt_tensor(6);
  auto is = [](const Tensor& t, std::initializer_list<int64_t> v) { return t.sizes() == at::IntArrayRef(v.begin(), v.size()); };
  const Tensor cw = conv.tensor_on(QBN_NAME(weight), at::kChar, on), cb = conv.opt_tensor_on(QBN_NAME(bias), at::kChar, on);
  if (decode && !conv_st.defined()) throw NotPlain{};
  if (cw.dim() != 2 || cw.size(0) != d || cw.size(1) != 4 || !cw.is_contiguous() || (cb.defined() && !cb.is_contiguous()) ||
      (conv_st.defined() && (conv_st.scalar_type() != at::kChar || !is(conv_st, {batch, d, 4}) || ssm_st.scalar_type() != at::kChar ||
                             !is(ssm_st, {batch, d, ds}) || !ssm_st.is_contiguous() || conv_st.device() != on || ssm_st.device() != on ||
                             (conv_st.stride(1) == 1 && (conv_st.stride(0) % 4 != 0 || conv_st.stride(2) % 4 != 0 || reinterpret_cast<uintptr_t>(conv_st.data_ptr()) % 4 != 0)))))
    throw NotPlain{};
  const Tensor A = scan.tensor_on(QBN_NAME(A_log), at::kChar, on), D = scan.opt_tensor_on(QBN_NAME(D), at::kChar, on),
               bias = scan.opt_tensor_on(QBN_NAME(dt_bias), at::kChar, on);
  auto scale = [&](PyObject* name) {
    const Tensor t = scan.tensor_on(name, at::kFloat, on);
    if (t.numel() != 1) throw NotPlain{};
    return t;
  };
  const Tensor As = scale(QBN_NAME(A_scale)), us = scale(QBN_NAME(u_scale)), dts = scale(QBN_NAME(dt_scale)), Bs = scale(QBN_NAME(B_scale)),
               Cs = scale(QBN_NAME(C_scale)), zs = scale(QBN_NAME(z_scale)), ss = scale(QBN_NAME(ssm_state_scale)), Ds = scale(QBN_NAME(D_scale)),
               bs = scale(QBN_NAME(dt_bias_scale));
  if (!is(A, {d, ds}) || !A.is_contiguous() || (D.defined() && (D.numel() != d || !D.is_contiguous())) ||
      (bias.defined() && (bias.numel() != d || !bias.is_contiguous())))
    throw NotPlain{};
  const double c_in = conv.num(QBN_NAME(input_scale)), c_w = conv.num(QBN_NAME(weight_scale)), c_out = conv.num(QBN_NAME(output_scale)),
               c_b = conv.num(QBN_NAME(bias_scale));
  const bool softplus = scan.flag(QBN_NAME(delta_softplus));
  const Rotation had(had_m);
  if (had.blocks <= 0 || d % had.blocks != 0) throw NotPlain{};

  const Device dev(x);
  const cudaStream_t st = dev.stream;
  Tensor u = x, residual;
  if (has_norm) {
    BlockNorm n(a.object(0), x, a.object(3), a.flag(4), rows, dm, dev);
    u = n.rows;
    residual = n.residual;
  } else if (x.scalar_type() != at::kChar) {
    throw NotPlain{};
  }
  const Tensor xz = dev.empty({rows, in.n}, at::kChar), cx = dev.empty({rows, d}, at::kChar), xd = dev.empty({rows, xp.n}, at::kChar),
               dt = dev.empty({rows, d}, at::kChar), y = dev.empty({rows, d}, at::kHalf), q = dev.empty({rows, d}, at::kChar);
  in.run(i8(u), dm, rows, xz.data_ptr(), in.n, st, !decode);
  int8_t* z = i8(xz) + d;
  auto conv_common = [&](auto& s) {
    s.x = i8(xz); s.out = i8(cx); s.weight = i8(cw); s.bias = i8(cb); s.batch = batch; s.dim = d; s.width = 4; s.x_sd = 1; s.out_sd = 1; s.silu = 1;
    s.scale_x = c_in; s.scale_w = c_w; s.scale_out = c_out; s.scale_b = c_b;
    if (conv_st.defined()) { s.conv_state = i8(conv_st); s.state_sb = conv_st.stride(0); s.state_sd = conv_st.stride(1); s.state_sw = conv_st.stride(2); }
  };
  if (decode) {
    qb_conv1d_update_args s{};
    conv_common(s);
    s.x_sb = in.n; s.out_sb = d;
    QBN_CALL(qb_causal_conv1d_update, s, st);
  } else {
    qb_conv1d_fwd_args s{};
    conv_common(s);
    s.seqlen = len; s.x_sb = len * in.n; s.x_sl = in.n; s.out_sb = len * d; s.out_sl = d;
    QBN_CALL(qb_causal_conv1d_fwd, s, st);
  }
  xp.run(i8(cx), d, rows, xd.data_ptr(), xp.n, st);
  dtp.run(i8(xd), xp.n, rows, dt.data_ptr(), d, st, !decode);
  int8_t *B = i8(xd) + rank, *C = B + ds;
  if (decode) {
    qb_sscan_update_args t{};
    t.state = i8(ssm_st); t.x = i8(cx); t.dt = i8(dt); t.A_log = i8(A); t.Bm = B; t.Cm = C; t.D = i8(D); t.z = z; t.dt_bias = ptr(bias);
    t.x_scales = f32(us); t.dt_scale = f32(dts); t.A_scale = f32(As); t.state_scale = f32(ss); t.B_scale = f32(Bs); t.C_scale = f32(Cs); t.D_scale = f32(Ds);
    t.z_scale = f32(zs); t.dt_bias_scale = f32(bs); t.out = y.data_ptr();
    t.state_sb = d * ds; t.state_sh = d * ds; t.state_sp = ds; t.x_sb = t.x_sh = d; t.dt_sb = t.dt_sh = d; t.dt_sp = 1; t.A_sh = d * ds; t.A_sp = ds; t.A_sn = 1;
    t.B_sb = t.B_sg = t.C_sb = t.C_sg = xp.n; t.D_sh = d; t.D_sp = 1; t.z_sb = t.z_sh = in.n; t.bias_sh = d; t.bias_sp = 1; t.out_sb = t.out_sh = d;
    t.batch = batch; t.nheads = 1; t.headdim = d; t.dstate = ds; t.ngroups = 1; t.dt_softplus = softplus;
    QBN_CALL(qb_sscan_update, t, st);
  } else {
    qb_sscan_fwd_args t{};
    t.u = i8(cx); t.delta = i8(dt); t.z = z; t.Bm = B; t.Cm = C; t.A_log = i8(A); t.D = i8(D); t.delta_bias = i8(bias);
    t.u_scale = f32(us); t.delta_scale = f32(dts); t.z_scale = f32(zs); t.B_scale = f32(Bs); t.C_scale = f32(Cs); t.A_scale = f32(As); t.D_scale = f32(Ds);
    t.delta_bias_scale = f32(bs); t.ssm_state_scale = f32(ss); t.out = y.data_ptr();
    t.u_sb = t.delta_sb = len * d; t.u_sl = t.delta_sl = d; t.u_sd = t.delta_sd = t.z_sd = 1; t.z_sb = len * in.n; t.z_sl = in.n;
    t.B_sb = t.C_sb = len * xp.n; t.B_sl = t.C_sl = xp.n; t.B_sn = t.C_sn = 1;
    t.batch = batch; t.dim = d; t.seqlen = len; t.dstate = ds; t.n_groups = 1; t.delta_softplus = softplus;
    t.channel_last = 1;
    t.final_state = ssm_st.defined() ? i8(ssm_st) : nullptr;
    t.workspace_bytes = qb_sscan_fwd_workspace_bytes(batch, d);
    const Tensor ws = t.workspace_bytes > 0 ? dev.empty({t.workspace_bytes}, at::kByte) : Tensor();
    t.workspace = ptr(ws);
    QBN_CALL(qb_sscan_fwd, t, st);
  }
  had.run(y, q, rows, d, st);
  Tensor out = dev.empty({batch, len, outp.n}, at::kHalf);
  outp.run(i8(q), d, rows, out.data_ptr(), outp.n, st);
  out = layer_output(out, batch, len, outp);
  return has_norm ? wrap_tuple({out, residual}) : wrap(out);
}

}  // namespace qbn
