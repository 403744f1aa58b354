// Generation step of plain transformer blocks: the checks of their modules, weights and caches, and the call that issues the kernels.
//
// A block on one new token runs five kernels of 4 to 7 us (a 125M model), yet Python needs about 130 attribute and tensor calls
// to see that the block is a plain one: 17 us of checks and 4 us to hand the addresses over, per block, against 12 us to launch.  Here the same checks
// take 2 us.  Whatever is not plainly covered is answered with None and left to the Python path (ops/fused_infer.py), which
// holds the rules; nothing is remembered between calls.
//
// One token through a model of 12 blocks of 768 columns: 482 -> 275 us (now what the device takes); six sequences, whose attention of
// heads of 64 is the library's and comes back from Python for every block, 1321 -> 911; one block of 2048 columns 54 -> 45 us.
//
// A CPython module because the checks read Python objects; tensors are read through PyTorch's own C++ interface.
#include <Python.h>

#include <ATen/ATen.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <algorithm>
#include <cmath>
#include <vector>

namespace {

using BlocksDecode = int (*)(const long long*, const double*, int, void*);

// Classes and the native entry, set once by configure().
struct Config {
  PyObject *attention = nullptr, *mlp = nullptr, *norm = nullptr, *cache = nullptr, *parameter = nullptr;
  BlocksDecode decode = nullptr;
  long max_rows = 0, norm_rows = 0;
} g;

PyObject* name(const char* s) { return PyUnicode_InternFromString(s); }
struct Names {
  PyObject *modules = name("_modules"), *parameters = name("_parameters"), *buffers = name("_buffers"),
           *fwd_hooks = name("_forward_hooks"), *pre_hooks = name("_forward_pre_hooks"), *forward = name("forward"),
           *attention = name("attention"), *mlp = name("mlp"), *attention_norm = name("attention_norm"), *mlp_norm = name("mlp_norm"),
           *tp = name("tp"), *q_norm = name("q_norm"), *k_norm = name("k_norm"), *capture = name("capture_attention_weights"),
           *fp8 = name("fp8"), *fp8_block = name("_kf_fp8_block"), *fp8_weight = name("_kf_fp8"), *flat = name("_kf_flat"),
           *head_dim = name("head_dim"), *q_proj = name("q_proj"), *k_proj = name("k_proj"), *v_proj = name("v_proj"),
           *o_proj = name("o_proj"), *gate_proj = name("gate_proj"), *up_proj = name("up_proj"), *down_proj = name("down_proj"),
           *weight = name("weight"), *eps = name("eps"), *k = name("k"), *v = name("v"), *seq_len = name("seq_len");
};
Names& n() {
  static Names names;
  return names;
}

// The attribute dictionary of an object, held for as long as the caller looks into it.
class Attributes {
 public:
  explicit Attributes(PyObject* o) : dict_(o ? PyObject_GenericGetDict(o, nullptr) : nullptr) {
    if (!dict_) PyErr_Clear();
  }
  ~Attributes() { Py_XDECREF(dict_); }
  Attributes(const Attributes&) = delete;
  Attributes& operator=(const Attributes&) = delete;
  PyObject* get(PyObject* key) const {  // borrowed, null when absent
    return dict_ && PyDict_Check(dict_) ? PyDict_GetItemWithError(dict_, key) : nullptr;
  }
  PyObject* table(PyObject* key, PyObject* item) const {  // self.<key>[item]
    PyObject* t = get(key);
    return t && PyDict_Check(t) ? PyDict_GetItemWithError(t, item) : nullptr;
  }

 private:
  PyObject* dict_;
};

bool empty_dict(PyObject* d) { return d && PyDict_Check(d) && PyDict_GET_SIZE(d) == 0; }

// No hooks and no replaced forward.
bool plain(const Attributes& m) { return empty_dict(m.get(n().fwd_hooks)) && empty_dict(m.get(n().pre_hooks)) && !m.get(n().forward); }

// Whether an optional flag of a module is certainly off: absent everywhere, or present in its dictionary and false.
bool flag_off(PyObject* o, const Attributes& m, PyObject* key) {
  if (PyObject* v = m.get(key)) return v == Py_False || v == Py_None;
  return !_PyType_Lookup(Py_TYPE(o), key) && !m.table(n().parameters, key) && !m.table(n().buffers, key) && !m.table(n().modules, key);
}

// A tensor that is no subclass but nn.Parameter and has memory of its own (no wrapper of a transform or of a dispatch mode).
const at::Tensor* tensor(PyObject* o) {
  if (!o || !(Py_TYPE(o) == reinterpret_cast<PyTypeObject*>(THPVariableClass) || reinterpret_cast<PyObject*>(Py_TYPE(o)) == g.parameter))
    return nullptr;
  const at::Tensor& t = THPVariable_Unpack(o);
  return t.defined() && t.has_storage() && !t.unsafeGetTensorImpl()->is_python_dispatch() && !t.is_sparse() ? &t : nullptr;
}

long long aligned(const void* p) { return reinterpret_cast<uintptr_t>(p) & 15 ? 0 : reinterpret_cast<long long>(p); }
long long address(const at::Tensor& t) { return aligned(t.const_data_ptr()); }
// Of what the kernels write: memory that a lazy clone shares with its original is its own after this.
long long target(const at::Tensor& t) { return aligned(t.mutable_data_ptr()); }

// Address of the dense bf16 (rows, cols) weight of self.<sub>, 0 for anything else; rows < 0: any number, reported in *rows_out.
long long matrix(const Attributes& m, PyObject* sub, long long rows, long long cols, long long* rows_out = nullptr) {
  const Attributes linear(m.table(n().modules, sub));
  PyObject* w = linear.table(n().parameters, n().weight);
  const at::Tensor* t = tensor(w);
  if (!t || t->scalar_type() != at::kBFloat16 || !t->is_cuda() || t->dim() != 2 || t->size(1) != cols || !t->is_contiguous()) return 0;
  if (rows < 0) *rows_out = t->size(0);
  else if (t->size(0) != rows) return 0;
  const Attributes own(w);
  if (own.get(n().fp8_weight) || _PyType_Lookup(Py_TYPE(w), n().fp8_weight) || own.get(n().flat)) {
    if (own.get(n().fp8_weight) || _PyType_Lookup(Py_TYPE(w), n().fp8_weight)) return 0;
    PyObject* unit = own.get(n().flat);  // a flat unit: fine unless it is sharded
    PyObject* s = PyObject_GetAttrString(unit, "sharded");
    if (!s) PyErr_Clear();
    const bool off = !s || s == Py_False;
    Py_XDECREF(s);
    if (!off) return 0;
  }
  return address(*t);
}

// Address of a plain RMSNorm's bf16 gain of width d and its epsilon, 0 for any other norm.
long long gain(PyObject* norm, long long d, double* eps) {
  if (!norm || reinterpret_cast<PyObject*>(Py_TYPE(norm)) != g.norm) return 0;
  const Attributes m(norm);
  PyObject* e = m.get(n().eps);
  const at::Tensor* t = tensor(m.table(n().parameters, n().weight));
  if (!plain(m) || !e || !PyFloat_Check(e) || !t || t->scalar_type() != at::kBFloat16 || !t->is_cuda() || t->dim() != 1 || t->size(0) != d ||
      !t->is_contiguous())
    return 0;
  *eps = PyFloat_AS_DOUBLE(e);
  return address(*t);
}

constexpr int INTS = 31, REALS = 3;  // per block, see kf_blocks_decode_bf16

struct Plan {
  long long weights[9], kc, vc, h, hkv, hd, f, past, step;  // gain, q, k, v, o, gain, gate, up, down
  double eps1, eps2;
};

// foreign: attention of heads of 64 for several sequences (the library's) can be called between two parts of the block.
bool plan(PyObject* block, PyObject* cache, long long b, long long d, const at::Tensor& cos, bool as_layer, bool foreign, Plan& p) {
  const Attributes m(block);
  if (as_layer && !plain(m)) return false;
  PyObject *att = m.table(n().modules, n().attention), *mlp = m.table(n().modules, n().mlp);
  if (!att || !mlp || reinterpret_cast<PyObject*>(Py_TYPE(att)) != g.attention || reinterpret_cast<PyObject*>(Py_TYPE(mlp)) != g.mlp ||
      reinterpret_cast<PyObject*>(Py_TYPE(cache)) != g.cache || !flag_off(block, m, n().fp8) || !flag_off(block, m, n().fp8_block))
    return false;
  const Attributes a(att), f(mlp), c(cache);
  if (!plain(a) || !plain(f) || a.get(n().tp) != Py_None || f.get(n().tp) != Py_None || a.get(n().q_norm) != Py_None ||
      a.get(n().k_norm) != Py_None || a.table(n().modules, n().q_norm) || a.table(n().modules, n().k_norm) || a.get(n().capture) != Py_False)
    return false;
  PyObject* hd = a.get(n().head_dim);
  if (!hd || !PyLong_CheckExact(hd)) return false;
  p.hd = PyLong_AsLongLong(hd);
  if ((p.hd != 64 && p.hd != 128) || cos.size(1) != p.hd / 2 || (p.hd == 64 && b > 1 && !foreign)) return false;
  long long qc = 0, kvc = 0;
  p.weights[0] = gain(m.table(n().modules, n().attention_norm), d, &p.eps1);
  p.weights[1] = matrix(a, n().q_proj, -1, d, &qc);
  p.weights[2] = matrix(a, n().k_proj, -1, d, &kvc);
  if (qc <= 0 || kvc <= 0 || qc % p.hd || kvc % p.hd || qc % kvc) return false;
  p.weights[3] = matrix(a, n().v_proj, kvc, d);
  p.weights[4] = matrix(a, n().o_proj, d, qc);
  p.weights[5] = gain(m.table(n().modules, n().mlp_norm), d, &p.eps2);
  p.weights[6] = matrix(f, n().gate_proj, -1, d, &p.f);
  if (p.f <= 0 || p.f % 8) return false;
  p.weights[7] = matrix(f, n().up_proj, p.f, d);
  p.weights[8] = matrix(f, n().down_proj, d, p.f);
  for (int i = 0; i < 9; ++i)
    if (!p.weights[i]) return false;
  p.h = qc / p.hd;
  p.hkv = kvc / p.hd;
  PyObject* past = c.get(n().seq_len);
  const at::Tensor *k = tensor(c.get(n().k)), *v = tensor(c.get(n().v));
  if (!past || !PyLong_CheckExact(past) || !k || !v || k->scalar_type() != at::kBFloat16 || v->scalar_type() != at::kBFloat16 ||
      k->dim() != 4 || k->sizes() != v->sizes() || k->size(0) != b || k->size(2) != p.hkv || k->size(3) != p.hd || !k->is_contiguous() ||
      !v->is_contiguous() || !k->is_cuda() || !v->is_cuda())
    return false;
  p.past = PyLong_AsLongLong(past);
  if (p.past < 0 || p.past + 1 > k->size(1)) return false;
  p.kc = target(*k);
  p.vc = target(*v);
  p.step = k->stride(0);
  return p.kc && p.vc;
}

// decode(blocks, caches, x, cos, sin, foreign, stream, sms): blocks and caches are lists.  (y, launches), or None when some block is not
// covered (nothing has been done then); an error code of the native call as an integer.  foreign: None when the
// blocks are called by the model in their stead (their own hooks count then); for the single block of a call, foreign(q (B, H hd), H, hd,
// position) -> (B, H hd) is the attention of heads of 64 for several sequences.
PyObject* decode(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  if (nargs != 8 || !PyList_Check(args[0]) || !PyList_Check(args[1]) || !g.decode) {
    PyErr_SetString(PyExc_TypeError, "decode(blocks, caches, x, cos, sin, foreign, stream, sms) after configure()");
    return nullptr;
  }
  const Py_ssize_t count = PyList_GET_SIZE(args[0]);
  PyObject* foreign = args[5];
  const bool as_layers = foreign == Py_None;
  const long long stream = PyLong_AsLongLong(args[6]), sms = PyLong_AsLongLong(args[7]);
  if (PyErr_Occurred()) return nullptr;
  const at::Tensor *x = tensor(args[2]), *cos = tensor(args[3]), *sin = tensor(args[4]);
  if (count < 1 || PyList_GET_SIZE(args[1]) < count || !x || !cos || !sin || x->dim() != 3 || x->size(1) != 1 ||
      x->scalar_type() != at::kBFloat16 || !x->is_cuda() || !x->is_contiguous() || x->numel() == 0 || x->is_conj() || x->is_neg() ||
      cos->scalar_type() != at::kFloat || sin->scalar_type() != at::kFloat || cos->dim() != 2 || cos->sizes() != sin->sizes() ||
      cos->size(0) < 1 || !cos->is_cuda() || !cos->is_contiguous() || !sin->is_contiguous())
    Py_RETURN_NONE;
  const long long b = x->size(0), d = x->size(2), xp = address(*x), cosp = address(*cos), sinp = address(*sin);
  if (b > g.max_rows || d % 8 || !xp || !cosp || !sinp) Py_RETURN_NONE;
  std::vector<Plan> plans(static_cast<size_t>(count));
  long long cols = 0, heads = 0;
  for (Py_ssize_t i = 0; i < count; ++i) {
    Plan& p = plans[static_cast<size_t>(i)];
    PyObject* cache = PyList_GET_ITEM(args[1], i);
    for (Py_ssize_t j = 0; j < i; ++j)
      if (PyList_GET_ITEM(args[1], j) == cache) Py_RETURN_NONE;
    if (!plan(PyList_GET_ITEM(args[0], i), cache, b, d, *cos, as_layers, !as_layers && count == 1, p)) {
      if (PyErr_Occurred()) return nullptr;
      Py_RETURN_NONE;
    }
    cols = std::max(cols, 2 * d + 2 * p.h * p.hd + p.f);
    heads = std::max(heads, p.h);
  }
  HANDLE_TH_ERRORS
  {
    // The blocks share one buffer of intermediates and hand x on through two more: each kernel of the chain writes only after all
    // before it are complete.  n (D) | q (H hd) | hidden (F) | h1 (D) | attention (H hd) | outputs of even and odd blocks | rstd, lse
    const at::Tensor scratch = at::empty({b * cols + 2 * b + 2 * heads + 2 * b * d}, x->options());
    at::Tensor y = at::empty_like(*x);
    const auto base = reinterpret_cast<long long>(scratch.mutable_data_ptr());
    const long long hand[2] = {base + 2 * b * cols, base + 2 * b * (cols + d)}, rstd = base + 2 * b * (cols + 2 * d);
    std::vector<long long> ints(static_cast<size_t>(count) * INTS);
    std::vector<double> reals(static_cast<size_t>(count) * REALS);
    long long src = xp;
    for (Py_ssize_t i = 0; i < count; ++i) {
      const Plan& p = plans[static_cast<size_t>(i)];
      const long long h1 = base + 2 * b * (d + p.h * p.hd + p.f);
      const long long dst = i == count - 1 ? reinterpret_cast<long long>(y.mutable_data_ptr()) : hand[i & 1];
      const long long row[INTS] = {src, p.weights[0], p.weights[1], p.weights[2], p.weights[3], p.weights[4], p.weights[5], p.weights[6],
                                   p.weights[7], p.weights[8], p.kc, p.vc, base, rstd, h1, dst, cosp, sinp, b, d, p.h, p.hkv, p.hd, p.f,
                                   p.past, p.step, sms, 7, p.hd == 64, h1 + 2 * b * d, rstd + 4 * b};
      std::copy(row, row + INTS, ints.begin() + i * INTS);
      reals[static_cast<size_t>(i) * REALS] = p.eps1;
      reals[static_cast<size_t>(i) * REALS + 1] = p.eps2;
      reals[static_cast<size_t>(i) * REALS + 2] = 1.0 / std::sqrt(static_cast<double>(p.hd));
      src = dst;
    }
    auto issue = [&] {
      int rc = 0;
      Py_BEGIN_ALLOW_THREADS
      rc = g.decode(ints.data(), reals.data(), static_cast<int>(count), reinterpret_cast<void*>(stream));
      Py_END_ALLOW_THREADS
      return rc;
    };
    const bool split = plans[0].hd == 64 && b > 1;
    if (split) ints[27] = 1;
    int rc = issue();
    if (rc) return PyLong_FromLong(rc);
    at::Tensor attended;  // lives until its reader has been issued
    if (split) {
      const Plan& p = plans[0];
      PyObject* q = THPVariable_Wrap(scratch.narrow(0, b * d, b * p.h * p.hd).view({b, p.h * p.hd}));
      PyObject* out = q ? PyObject_CallFunction(foreign, "OLLL", q, p.h, p.hd, p.past) : nullptr;
      Py_XDECREF(q);
      if (!out) return nullptr;
      const at::Tensor* t = tensor(out);
      const bool fits = t && t->scalar_type() == at::kBFloat16 && t->is_cuda() && t->dim() == 2 && t->size(0) == b &&
                        t->size(1) == p.h * p.hd && t->is_contiguous() && address(*t);
      if (fits) attended = *t;
      Py_DECREF(out);
      if (!fits) {
        PyErr_SetString(PyExc_RuntimeError, "the attention between two parts of a block has to return dense bf16 rows");
        return nullptr;
      }
      ints[27] = 4;
      ints[29] = address(attended);
      rc = issue();
      if (rc) return PyLong_FromLong(rc);
    }
    for (Py_ssize_t i = 0; i < count; ++i) {
      PyObject* end = PyLong_FromLongLong(plans[static_cast<size_t>(i)].past + 1);
      const bool ok = end && PyObject_SetAttr(PyList_GET_ITEM(args[1], i), n().seq_len, end) == 0;
      Py_XDECREF(end);
      if (!ok) return nullptr;
    }
    PyObject* out = THPVariable_Wrap(std::move(y));
    return out ? Py_BuildValue("(Nn)", out, count * ((split ? 4 : 5) + (b <= g.norm_rows ? 0 : 2))) : nullptr;
  }
  END_HANDLE_TH_ERRORS
}

// configure(Attention, SwiGLUMLP, RMSNorm, KVCache, Parameter, address of kf_blocks_decode_bf16, largest batch, batch up to which the
// projections take their norms along)
PyObject* configure(PyObject*, PyObject* args) {
  Config c;
  unsigned long long fn = 0;
  if (!PyArg_ParseTuple(args, "OOOOOKll", &c.attention, &c.mlp, &c.norm, &c.cache, &c.parameter, &fn, &c.max_rows, &c.norm_rows)) return nullptr;
  for (PyObject* o : {c.attention, c.mlp, c.norm, c.cache, c.parameter}) Py_INCREF(o);
  c.decode = reinterpret_cast<BlocksDecode>(fn);
  g = c;
  Py_RETURN_NONE;
}

PyMethodDef methods[] = {
    {"decode", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(decode)), METH_FASTCALL, "one new token per sequence through blocks"},
    {"configure", configure, METH_VARARGS, "classes and the native entry"},
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "kf_steps", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit_kf_steps() { return PyModule_Create(&module); }
