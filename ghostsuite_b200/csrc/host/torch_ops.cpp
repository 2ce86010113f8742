// Host side of the operations on torch tensors: operand preparation, workspaces, output allocation and
// the calls into libghost_b200, in one native call per operation.  A hooked layer's work is a few
// launches of a few microseconds; the same steps in Python and ctypes (a stream lookup, an output
// allocation, an argument conversion each) took 20 to 60 us per operation and bound every step that
// does not fill the GPU.  Entry points take positional arguments only (METH_FASTCALL); ghostsuite_b200/
// ops.py holds the documented signatures.
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/function_hook.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/autograd/variable.h>

#include <algorithm>
#include <map>
#include <mutex>
#include <stdexcept>
#include <string>
#include <unordered_map>
#include <unordered_set>
#include <utility>
#include <vector>

#include "../../../include/ghost_b200.h"
#include "../launch_rules.h"

namespace {

using at::Tensor;

// ---- errors ------------------------------------------------------------------------------------
struct GhostError : std::runtime_error {
  int code;
  GhostError(int c, const std::string& m) : std::runtime_error(m), code(c) {}
};
[[noreturn]] void invalid(const std::string& m) { throw GhostError(GHOST_ERR_INVALID, m); }
void check(int status) {
  if (status != GHOST_OK) throw GhostError(status, ghost_last_error());
}
PyObject* g_kernel_error = nullptr;     // ghostsuite_b200._lib.GhostKernelError

template <typename F> PyObject* guarded(F&& f) {
  try {
    return f();
  } catch (const GhostError& e) {
    PyObject* type = e.code == GHOST_ERR_INVALID ? PyExc_ValueError
                   : e.code == GHOST_ERR_INDEX ? PyExc_IndexError
                   : e.code == GHOST_ERR_DEVICE || e.code > 0 || g_kernel_error == nullptr ? PyExc_RuntimeError
                                                                                           : g_kernel_error;
    const std::string text = e.code == GHOST_ERR_DEVICE ? std::string("ghostsuite_b200 needs a B200 (sm_100) GPU: ") + e.what()
                                                        : std::string(e.what());
    PyErr_SetString(type, text.c_str());
  } catch (const c10::OutOfMemoryError& e) {
    // torch.cuda.OutOfMemoryError where torch exposes it, as from torch.empty
    PyObject* mod = PyImport_ImportModule("torch");
    PyObject* type = mod ? PyObject_GetAttrString(mod, "OutOfMemoryError") : nullptr;
    PyErr_Clear();
    PyErr_SetString(type ? type : PyExc_RuntimeError, e.what_without_backtrace());
    Py_XDECREF(type);
    Py_XDECREF(mod);
  } catch (python_error& e) {
    if (!PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, e.what());
  } catch (const std::exception& e) {
    PyErr_SetString(PyExc_RuntimeError, e.what());
  }
  return nullptr;
}

// ---- arguments -----------------------------------------------------------------------------------
constexpr int kNotCuda = 1;             // positive codes: plain RuntimeError
bool present(PyObject* o) { return o != nullptr && o != Py_None; }
const Tensor& tensor(PyObject* o) {
  if (!THPVariable_Check(o)) invalid("expected a tensor");
  return THPVariable_Unpack(o);
}
const Tensor& cuda_tensor(PyObject* o) {
  const Tensor& t = tensor(o);
  if (!t.is_cuda()) throw GhostError(kNotCuda, "ghostsuite_b200 kernels need CUDA tensors (no CPU fallback exists)");
  return t;
}
long long integer(PyObject* o) {
  const long long v = PyLong_AsLongLong(o);
  if (v == -1 && PyErr_Occurred()) { PyErr_Clear(); invalid("expected an integer"); }
  return v;
}
float real(PyObject* o) {
  const double v = PyFloat_AsDouble(o);
  if (v == -1.0 && PyErr_Occurred()) { PyErr_Clear(); invalid("expected a number"); }
  return static_cast<float>(v);
}
void need(Py_ssize_t have, Py_ssize_t want, const char* who) {
  if (have != want) invalid(std::string(who) + ": wrong number of arguments");
}
PyObject* wrap(Tensor t) { return THPVariable_Wrap(std::move(t)); }
PyObject* wrap_or_none(const Tensor& t) {
  if (t.defined()) return THPVariable_Wrap(t);
  Py_RETURN_NONE;
}

int is_f32(const Tensor& t) {
  if (t.scalar_type() == at::kFloat) return 1;
  if (t.scalar_type() == at::kBFloat16) return 0;
  invalid(std::string("unsupported dtype ") + c10::toString(t.scalar_type()) + ": the kernels take float32 and bfloat16");
}
// [N, d] -> [N, 1, d]; [N, ..., d] -> [N, T, d], contiguous; float16 / float64 become float32
Tensor as3d(const Tensor& x0) {
  Tensor x = x0;
  if (x.scalar_type() == at::kHalf || x.scalar_type() == at::kDouble) x = x.to(at::kFloat);
  if (x.dim() == 3) return x.is_contiguous() ? x : x.contiguous();
  if (x.dim() <= 2) x = x.unsqueeze(1);
  else x = x.reshape({x.size(0), -1, x.size(-1)});
  return x.contiguous();
}
Tensor ids2d(const Tensor& x0) {
  Tensor x = x0.dim() == 2 ? x0 : x0.reshape({x0.size(0), -1});
  if (x.scalar_type() != at::kLong) x = x.to(at::kLong);
  return x.contiguous();
}
bool tma_ready(const Tensor& x) {
  return x.scalar_type() == at::kBFloat16 && x.size(-1) % 8 == 0 && (reinterpret_cast<uintptr_t>(x.data_ptr()) & 15u) == 0;
}
// A caller's result buffer, which the kernels write as rows x cols elements from its start.
void check_result(const Tensor& out, long long rows, long long cols, const Tensor& like, const char* who) {
  if (out.numel() != rows * cols || !out.is_contiguous() || out.get_device() != like.get_device())
    invalid(std::string(who) + ": the output must be a contiguous " + std::to_string(rows) + " x " + std::to_string(cols) +
            " tensor on the operands' device");
}
long long pad8(long long n) { return (n + 7) / 8 * 8; }
Tensor empty(at::IntArrayRef size, const Tensor& like, at::ScalarType dt) { return at::empty(size, like.options().dtype(dt)); }

// Device and stream of one operation.
struct Launch {
  c10::cuda::CUDAGuard guard;
  c10::cuda::CUDAStream stream;
  explicit Launch(const Tensor& t) : guard(t.device()), stream(c10::cuda::getCurrentCUDAStream(t.get_device())) {}
  void* st() const { return static_cast<void*>(stream.stream()); }
};

// ---- workspace -------------------------------------------------------------------------------------
// One growing buffer per (device, stream).  A buffer that is replaced goes back to torch's caching
// allocator, which hands it out again in stream order, so kernels queued on it are safe; callers hold
// the GIL for a whole operation, so two threads on one stream cannot mix their parts.
std::mutex g_arena_mu;
std::map<std::pair<int, void*>, Tensor> g_arenas;

class Workspace {
 public:
  long long plan(long long nbytes) {
    const long long at = total_;
    total_ += (nbytes + 255) / 256 * 256;
    return at;
  }
  char* commit(const Launch& L, const Tensor& like) {
    const long long want = total_ + 256;
    std::lock_guard<std::mutex> lock(g_arena_mu);
    Tensor& buf = g_arenas[{like.get_device(), L.st()}];
    if (!buf.defined() || buf.numel() < want) {
      buf = Tensor();
      buf = at::empty({want > (1 << 20) ? want : (1 << 20)}, like.options().dtype(at::kByte));
    }
    const uintptr_t base = reinterpret_cast<uintptr_t>(buf.data_ptr());
    return reinterpret_cast<char*>((base + 255) / 256 * 256);
  }

 private:
  long long total_ = 0;
};

PyObject* py_arena_clear(PyObject*, PyObject* const*, Py_ssize_t) {
  std::lock_guard<std::mutex> lock(g_arena_mu);
  g_arenas.clear();
  Py_RETURN_NONE;
}

// hi/lo layouts of an fp32 operand pair so that sum_k L[k] R[k] = hi*hi + lo*hi + hi*lo
constexpr int kSplitLeft[3] = {0, 1, 0};
enum { kSideBySide = 0 };      // where the parts of a copy lie

// An operand [N, T, cols] of the layer math: a tensor with exactly these dimensions, or a convolution
// operand [N, C, H, W] whose tokens are the output positions.
struct Conv { int C, H, W, kh, kw, sy, sx, py, px, dy, dx; };
struct Operand {
  const Tensor& t;
  long long N, T, cols;
  const Conv* conv;
  explicit Operand(const Tensor& x) : t(x), N(x.size(0)), T(x.size(1)), cols(x.size(2)), conv(nullptr) {}
  Operand(const Tensor& x, const Conv& c, long long tokens)
      : t(x), N(x.size(0)), T(tokens), cols(static_cast<long long>(c.C) * c.kh * c.kw), conv(&c) {}
  int f32() const { return is_f32(t); }
  // readable as it is by the tensor-core entry points
  bool ready() const { return conv == nullptr && tma_ready(t); }
  // bf16 copy of samples [first, first + samples) of a tensor
  void cast(long long first, long long samples, void* dst, long long ld_dst, long long cpad, int parts, const int (&kinds)[3],
            int stack, void* st) const {
    const char* p = static_cast<const char*>(t.data_ptr()) + first * T * cols * t.element_size();
    check(ghost_cast_split_bf16(p, f32(), samples, T, static_cast<int>(cols), cols, dst, ld_dst, static_cast<int>(cpad), parts, kinds[0],
                                kinds[1], kinds[2], stack, st));
  }
};

void check_split(long long n_train, long long n_val, const char* who) {
  if (n_train <= 0) invalid("No training samples to compute dot product, check batch sizes.");
  if (n_val <= 0) invalid(std::string(who) + " needs at least one validation sample");
}

// ---- operands of the tensor-core paths -----------------------------------------------------------------
// Two operands of the entry points that take one or two bf16 parts.  A float32 operand makes both two parts; otherwise
// what is not readable as it is is copied with its rows padded.  `merged`: one sample holding all rows.
struct XtyOperands {
  const Operand* x[2];
  long long count, T, ld[2], off[2] = {0, 0};      // samples that are read and their tokens
  bool merged, copy[2], split;
  XtyOperands(Workspace& ws, const Operand& X, const Operand& Y, long long count_, bool merged_)
      : count(count_), T(X.T), merged(merged_) {
    x[0] = &X;
    x[1] = &Y;
    split = X.f32() || Y.f32();
    for (int i = 0; i < 2; ++i) {
      copy[i] = split || !x[i]->ready();
      ld[i] = copy[i] ? (x[i]->cols + 63) / 64 * 64 : x[i]->cols;
      if (copy[i]) off[i] = ws.plan(count * parts() * T * ld[i] * 2);
    }
  }
  int parts() const { return split ? 2 : 1; }
  const void* where(int i, char* base) const { return copy[i] ? static_cast<const void*>(base + off[i]) : x[i]->t.data_ptr(); }
  // Lays out what has to be copied, with the column sums of operand sums_of (1 or 2, both operands copied) on the way
  void prepare(char* base, void* st, int sums_of = 0, float* sums = nullptr) const {
    if (x[0]->conv) {                    // the out-grad, then the input under its window
      const Conv &b = *x[0]->conv, &a = *x[1]->conv;
      check(ghost_conv_operands(x[1]->t.data_ptr(), x[1]->f32(), x[0]->t.data_ptr(), x[0]->f32(), count, a.C, a.H, a.W, a.kh, a.kw,
                                a.sy, a.sx, a.py, a.px, a.dy, a.dx, b.C, b.H, b.W, parts(), merged ? 1 : 0, base + off[1],
                                base + off[0], sums_of == 1 ? sums : nullptr, st));
    } else if (copy[0] || copy[1]) {
      auto src = [&](int i) { return copy[i] ? x[i]->t.data_ptr() : nullptr; };
      auto dst = [&](int i) { return copy[i] ? base + off[i] : nullptr; };
      check(ghost_split_operands(src(0), x[0]->f32(), static_cast<int>(x[0]->cols), src(1), x[1]->f32(), static_cast<int>(x[1]->cols),
                                 parts(), count, T, merged ? 1 : 0, dst(0), dst(1), sums_of == 1 ? sums : nullptr,
                                 sums_of == 2 ? sums : nullptr, st));
    }
  }
};

// ---- Gram path -----------------------------------------------------------------------------------------
void launch_gram(const Launch& L, const XtyOperands& ops, int a, char* base, long long n_val, int round_mode, float scale, Tensor& M) {
  const int g = 1 - a;
  check(ghost_gram_dot_parts(ops.where(a, base), ops.where(g, base), ops.parts(), static_cast<int>(ops.count - n_val),
                             static_cast<int>(n_val), ops.T, static_cast<int>(ops.x[a]->cols), static_cast<int>(ops.x[g]->cols),
                             ops.ld[a], ops.ld[g], round_mode, scale, M.data_ptr<float>(), L.st()));
}

Tensor gram_dot(const Launch& L, const Operand& A, const Operand& G, long long n_val, int round_mode, float scale) {
  check_split(A.N - n_val, n_val, "gram_dot");
  if (G.N != A.N || G.T != A.T) invalid("gram_dot: activation and out-grad disagree on [batch, tokens]");
  Tensor M = empty({n_val, A.N - n_val}, A.t, at::kFloat);
  Workspace ws;
  XtyOperands ops(ws, A, G, A.N, true);
  char* base = ws.commit(L, A.t);
  ops.prepare(base, L.st());
  launch_gram(L, ops, 0, base, n_val, round_mode, scale, M);
  return M;
}

PyObject* py_gram_dot(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    need(n, 5, "gram_dot");
    const Tensor &A0 = cuda_tensor(a[0]), &G0 = cuda_tensor(a[1]);
    Launch L(A0);
    const Tensor A = as3d(A0), G = as3d(G0);
    return wrap(gram_dot(L, Operand(A), Operand(G), integer(a[2]), static_cast<int>(integer(a[3])), real(a[4])));
  });
}

// ---- token-contracted GEMMs --------------------------------------------------------------------------
// scale * sum over the first `samples` samples of X^T Y, into out
void wgrad(const Launch& L, const Operand& X, const Operand& Y, long long samples, float scale, Tensor& out, bool accumulate) {
  const int m = static_cast<int>(X.cols), n = static_cast<int>(Y.cols);
  Workspace ws;
  const long long ws_bytes = ghost_wgrad_workspace_bytes(m, n);
  const long long off_ws = ws.plan(ws_bytes);
  XtyOperands ops(ws, X, Y, samples, true);
  char* base = ws.commit(L, X.t);
  ops.prepare(base, L.st());
  check(ghost_wgrad_parts(ops.where(0, base), ops.where(1, base), ops.parts(), samples * ops.T, samples * ops.T, m, n, ops.ld[0], ops.ld[1], scale, accumulate ? 1 : 0,
                          out.data_ptr(), is_f32(out), base + off_ws, ws_bytes, L.st()));
}

// (X, Y, scale, f32_out, out or None, accumulate)
PyObject* py_wgrad(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    need(n, 6, "wgrad");
    const Tensor &X0 = cuda_tensor(a[0]), &Y0 = cuda_tensor(a[1]);
    Launch L(X0);
    const Tensor X = as3d(X0), Y = as3d(Y0);
    if (Y.size(0) != X.size(0) || Y.size(1) != X.size(1)) invalid("wgrad operands disagree on the token layout");
    const bool have = present(a[4]);
    Tensor out = have ? cuda_tensor(a[4]) : empty({X.size(2), Y.size(2)}, X, integer(a[3]) ? at::kFloat : at::kBFloat16);
    if (have) check_result(out, X.size(2), Y.size(2), X, "wgrad");
    wgrad(L, Operand(X), Operand(Y), X.size(0), real(a[2]), out, have && integer(a[5]));
    return wrap(out);
  });
}

// ---- per-sample path -----------------------------------------------------------------------------------
struct PerSample { Tensor M, grad, colsums; };

PerSample persample_dot(const Launch& L, const Operand& X, const Operand& Y, long long n_val, float dot_scale, bool want_grad,
                        float grad_scale, at::ScalarType grad_dt, int colsum_of, int split_sums_of) {
  const long long N = X.N, T = X.T, n_train = N - n_val;
  const int m = static_cast<int>(X.cols), n = static_cast<int>(Y.cols);
  check_split(n_train, n_val, "persample_dot");
  if (Y.N != N || Y.T != T) invalid("persample_dot operands disagree on the token layout");
  PerSample r;
  r.M = empty({n_val, n_train}, X.t, at::kFloat);
  if (want_grad) r.grad = empty({m, n}, X.t, grad_dt);
  Workspace ws;
  XtyOperands ops(ws, X, Y, N, false);
  const int f32 = ops.split ? 1 : 0;
  const long long ws_bytes = ghost_persample_workspace_bytes(static_cast<int>(n_train), static_cast<int>(n_val), m, n, f32);
  const long long off_ws = ws.plan(ws_bytes);
  char* base = ws.commit(L, X.t);
  // Column sums: of bf16 operands the GEMM pass takes them along (colsum_of), of float32 ones their conversion does
  // (split_sums_of) unless a sample has too few rows for a block of it; of a convolution's, the copy does.
  const int sums_of = X.conv ? split_sums_of : !ops.split ? colsum_of : T >= 16 ? split_sums_of : 0;
  if (sums_of) r.colsums = empty({N, ops.x[sums_of - 1]->cols}, X.t, at::kFloat);
  float* sums = sums_of ? r.colsums.data_ptr<float>() : nullptr;
  if (ops.split || X.conv) ops.prepare(base, L.st(), sums_of, sums);
  else ops.prepare(base, L.st());
  check(ghost_persample_dot_parts(ops.where(0, base), ops.where(1, base), ops.parts(), static_cast<int>(n_train),
                                  static_cast<int>(n_val), T, m, n, ops.ld[0], ops.ld[1], dot_scale, r.M.data_ptr<float>(),
                                  want_grad ? r.grad.data_ptr() : nullptr, want_grad ? is_f32(r.grad) : 0, grad_scale, 0,
                                  ops.split || X.conv ? 0 : sums_of, ops.split || X.conv ? nullptr : sums, base + off_ws, ws_bytes, L.st()));
  return r;
}

// (X, Y, n_val, dot_scale, want_grad, grad_scale, grad_is_f32, colsum_of: 0 / 1 = X / 2 = Y)
PyObject* py_persample_dot(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    need(n, 8, "persample_dot");
    const Tensor &X0 = cuda_tensor(a[0]), &Y0 = cuda_tensor(a[1]);
    Launch L(X0);
    const Tensor X = as3d(X0), Y = as3d(Y0);
    PerSample r = persample_dot(L, Operand(X), Operand(Y), integer(a[2]), real(a[3]), integer(a[4]) != 0, real(a[5]),
                                integer(a[6]) ? at::kFloat : at::kBFloat16, static_cast<int>(integer(a[7])), 0);
    return Py_BuildValue("(NNN)", wrap(r.M), wrap_or_none(r.grad), wrap_or_none(r.colsums));
  });
}

// ---- column sums, norms --------------------------------------------------------------------------------
Tensor colsum(const Launch& L, const Tensor& G) {
  const long long N = G.size(0), T = G.size(1), p = G.size(2);
  Tensor out = empty({N, p}, G, at::kFloat);
  check(ghost_colsum(G.data_ptr(), is_f32(G), static_cast<int>(N), T, static_cast<int>(p), p, out.data_ptr<float>(), L.st()));
  return out;
}

PyObject* py_colsum(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    need(n, 1, "colsum");
    const Tensor& G0 = cuda_tensor(a[0]);
    Launch L(G0);
    return wrap(colsum(L, as3d(G0)));
  });
}

struct Norm { Tensor gw, gb; };

Norm norm_persample(const Launch& L, Tensor A, Tensor G, float eps, bool rms) {
  if (A.scalar_type() != G.scalar_type()) {
    const at::ScalarType common = c10::promoteTypes(A.scalar_type(), G.scalar_type());
    A = A.to(common);
    G = G.to(common);
  }
  A = as3d(A);
  G = as3d(G);
  const long long N = A.size(0), T = A.size(1), F = A.size(2);
  if (G.sizes() != A.sizes()) invalid("LayerNorm input and out-grad shapes differ");
  Tensor both = empty({2, N, F}, A, at::kFloat);
  Norm r{both.select(0, 0), both.select(0, 1)};
  Workspace ws;
  const long long ws_bytes = ghost_layernorm_workspace_bytes(static_cast<int>(N), T, static_cast<int>(F));
  const long long off = ws.plan(ws_bytes);
  char* base = ws.commit(L, A);
  auto fn = rms ? ghost_rmsnorm_persample : ghost_layernorm_persample;
  check(fn(A.data_ptr(), G.data_ptr(), is_f32(A), static_cast<int>(N), T, static_cast<int>(F), eps, r.gw.data_ptr<float>(),
           r.gb.data_ptr<float>(), base + off, ws_bytes, L.st()));
  return r;
}

// (A, G, eps, rms) -> (gw, gb)
PyObject* py_norm_persample(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    need(n, 4, "norm_persample");
    const Tensor &A = cuda_tensor(a[0]), &G = cuda_tensor(a[1]);
    Launch L(A);
    Norm r = norm_persample(L, A, G, real(a[2]), integer(a[3]) != 0);
    return Py_BuildValue("(NN)", wrap(r.gw), wrap(r.gb));
  });
}

// ---- whole hooks ----------------------------------------------------------------------------------------
// dtype argument of an optional output: -1 = not wanted, 0 = bfloat16, 1 = float32
Tensor optional_empty(at::IntArrayRef size, const Tensor& like, long long dt) {
  return dt < 0 ? Tensor() : empty(size, like, dt ? at::kFloat : at::kBFloat16);
}

// One of the two tensor-core paths, with the train gradient (dtype code gdt) and, where it costs nothing
// extra, the column sums of B for a layer with a bias (`fuse`: also those that a GEMM pass takes along).
void dense_paths(const Launch& L, const Operand& A, const Operand& B, long long n_val, bool in_by_out, bool gram, long long gdt,
                 float scale, bool bias, bool fuse, Tensor& M, Tensor& grad, Tensor& sums) {
  const Operand &X = in_by_out ? A : B, &Y = in_by_out ? B : A;
  if (gram) {
    // one copy of what has to be copied serves the Grams and the gradient, and gives the bias its sums
    const long long N = A.N;
    const int m = static_cast<int>(X.cols), n = static_cast<int>(Y.cols), b = in_by_out ? 1 : 0;
    check_split(N - n_val, n_val, "gram_dot");
    M = empty({n_val, N - n_val}, A.t, at::kFloat);
    grad = optional_empty({X.cols, Y.cols}, X.t, gdt);
    Workspace ws;
    const long long ws_bytes = grad.defined() ? ghost_wgrad_workspace_bytes(m, n) : 0, off_ws = ws.plan(ws_bytes);
    XtyOperands ops(ws, X, Y, N, true);
    char* base = ws.commit(L, A.t);
    const bool take = bias && (A.conv || (ops.split && A.T >= 16));
    if (take) sums = empty({N, B.cols}, A.t, at::kFloat);
    ops.prepare(base, L.st(), take ? b + 1 : 0, take ? sums.data_ptr<float>() : nullptr);
    const int a = 1 - b;
    check(ghost_gram_pass(ops.where(a, base), ops.where(b, base), ops.parts(), static_cast<int>(N - n_val), static_cast<int>(n_val), A.T,
                          static_cast<int>(A.cols), static_cast<int>(B.cols), ops.ld[a], ops.ld[b], in_by_out ? 1 : 0, M.data_ptr<float>(), scale,
                          grad.defined() ? grad.data_ptr() : nullptr, grad.defined() ? is_f32(grad) : 0, base + off_ws, ws_bytes, L.st()));
  } else {
    PerSample r = persample_dot(L, X, Y, n_val, 1.f, gdt >= 0, scale, gdt == 0 ? at::kBFloat16 : at::kFloat,
                                !fuse ? 0 : in_by_out ? 2 : 1, !bias ? 0 : in_by_out ? 2 : 1);
    M = r.M;
    grad = r.grad;
    sums = r.colsums;
  }
}

// Everything the backward hook of a Linear / Conv1D layer computes or allocates:
// (A, B, n_val, weight_is_in_by_out, use_gram, weight grad dtype, grad scale, has_bias, bias grad dtype, any_path,
// fuse_colsums)
// -> (M, weight grad, column sums of B, unfilled bias matrix, unfilled bias grad), None where not wanted.
PyObject* py_dense_hook(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    need(n, 11, "dense_hook");
    const Tensor &A0 = cuda_tensor(a[0]), &B0 = cuda_tensor(a[1]);
    Launch L(A0);
    const Tensor A = as3d(A0), B = as3d(B0);
    const long long n_val = integer(a[2]), N = A.size(0), n_train = N - n_val, p = B.size(2);
    const bool in_by_out = integer(a[3]) != 0, gram = integer(a[4]) != 0, bias = integer(a[7]) != 0;
    const long long gdt = integer(a[5]), bdt = integer(a[8]);
    const bool fuse = bias && integer(a[10]) != 0;
    const float scale = real(a[6]);
    const Tensor &X = in_by_out ? A : B, &Y = in_by_out ? B : A;
    Tensor M, grad, sums;
    const int dI = static_cast<int>(A.size(2)), pI = static_cast<int>(p);
    check_split(n_train, n_val, "dense_hook");
    if (B.size(0) != N || B.size(1) != A.size(1)) invalid("activation and out-grad disagree on [batch, tokens]");
    if (integer(a[9]) && A.scalar_type() == B.scalar_type() &&
        ghost_dense_small_fits(is_f32(A), static_cast<int>(n_train), static_cast<int>(n_val), A.size(1), dI, pI)) {
      M = empty({n_val, n_train}, A, at::kFloat);
      grad = optional_empty({X.size(2), Y.size(2)}, X, gdt);
      // written out even for one float32 token, whose row is the sum: they are read when the pass ends
      if (fuse) sums = empty({N, p}, A, at::kFloat);
      check(ghost_dense_small(A.data_ptr(), B.data_ptr(), is_f32(A), static_cast<int>(n_train), static_cast<int>(n_val),
                              A.size(1), dI, pI, in_by_out ? 1 : 0, M.data_ptr<float>(), grad.defined() ? grad.data_ptr() : nullptr,
                              grad.defined() ? is_f32(grad) : 0, scale, fuse ? sums.data_ptr<float>() : nullptr, L.st()));
    } else {
      dense_paths(L, Operand(A), Operand(B), n_val, in_by_out, gram, gdt, scale, bias, fuse, M, grad, sums);
    }
    if (bias && !sums.defined()) sums = colsum(L, B);
    Tensor Mb = bias ? empty({n_val, n_train}, A, at::kFloat) : Tensor();
    Tensor sb = optional_empty({p}, A, bias ? bdt : -1);
    return Py_BuildValue("(NNNNN)", wrap(M), wrap_or_none(grad), wrap_or_none(sums), wrap_or_none(Mb), wrap_or_none(sb));
  });
}

// The same for a Conv2d layer with groups == 1: (A [N, C, H, W], B [N, p, Ho, Wo], n_val, (kh, kw, sy, sx, py, px, dy,
// dx), use_gram, weight grad dtype, grad scale, has_bias, bias grad dtype); the weight gradient is [p, C * kh * kw]
PyObject* py_conv_hook(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    need(n, 9, "conv_hook");
    const Tensor &A0 = cuda_tensor(a[0]), &B0 = cuda_tensor(a[1]);
    Launch L(A0);
    const Tensor A = A0.contiguous(), B = B0.contiguous();
    if (A.dim() != 4 || B.dim() != 4 || A.size(0) != B.size(0)) invalid("conv_hook takes [N, C, H, W] and [N, p, Ho, Wo]");
    if (!PyTuple_Check(a[3]) || PyTuple_GET_SIZE(a[3]) != 8) invalid("conv_hook: bad window");
    int w[8];
    for (int i = 0; i < 8; ++i) w[i] = static_cast<int>(integer(PyTuple_GET_ITEM(a[3], i)));
    const Conv ca = {static_cast<int>(A.size(1)), static_cast<int>(A.size(2)), static_cast<int>(A.size(3)), w[0], w[1], w[2],
                     w[3], w[4], w[5], w[6], w[7]};
    const Conv cb = {static_cast<int>(B.size(1)), static_cast<int>(B.size(2)), static_cast<int>(B.size(3)), 1, 1, 1, 1, 0, 0, 1, 1};
    if (w[2] <= 0 || w[3] <= 0 || (ca.H + 2 * w[4] - w[6] * (w[0] - 1) - 1) / w[2] + 1 != B.size(2) ||
        (ca.W + 2 * w[5] - w[7] * (w[1] - 1) - 1) / w[3] + 1 != B.size(3))
      invalid("conv_hook: the out-grad is not this convolution's output size");
    const long long T = B.size(2) * B.size(3), N = A.size(0), p = B.size(1), n_val = integer(a[2]), n_train = N - n_val;
    check_split(n_train, n_val, "conv_hook");
    const bool bias = integer(a[7]) != 0;
    Tensor M, grad, sums;
    dense_paths(L, Operand(A, ca, T), Operand(B, cb, T), n_val, false, integer(a[4]) != 0, integer(a[5]), real(a[6]), bias, false, M,
                grad, sums);
    Tensor Mb = bias ? empty({n_val, n_train}, A, at::kFloat) : Tensor();
    Tensor sb = optional_empty({p}, A, bias ? integer(a[8]) : -1);
    return Py_BuildValue("(NNNNN)", wrap(M), wrap_or_none(grad), wrap_or_none(sums), wrap_or_none(Mb), wrap_or_none(sb));
  });
}

// The same for a LayerNorm / RMS norm layer: (A, G, eps, rms, n_val, weight grad dtype, bias grad dtype) ->
// (gw, gb, unfilled weight matrix, bias matrix, weight grad, bias grad); no bias: dtype -1, two Nones
PyObject* py_norm_hook(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    need(n, 7, "norm_hook");
    const Tensor &A = cuda_tensor(a[0]), &G = cuda_tensor(a[1]);
    Launch L(A);
    Norm r = norm_persample(L, A, G, real(a[2]), integer(a[3]) != 0);
    const long long n_val = integer(a[4]), n_train = r.gw.size(0) - n_val, F = r.gw.size(1), bdt = integer(a[6]);
    check_split(n_train, n_val, "norm_hook");
    Tensor M = empty({bdt >= 0 ? 2 : 1, n_val, n_train}, A, at::kFloat);
    return Py_BuildValue("(NNNNNN)", wrap(r.gw), wrap(r.gb), wrap(M.select(0, 0)), wrap_or_none(bdt >= 0 ? M.select(0, 1) : Tensor()),
                         wrap_or_none(optional_empty({F}, A, integer(a[5]))), wrap_or_none(optional_empty({F}, A, bdt)));
  });
}

// ---- embedding ------------------------------------------------------------------------------------------
// (ids, G, n_val, vocab, scale)
PyObject* py_embedding_dot(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    need(n, 5, "embedding_dot");
    const Tensor &ids0 = cuda_tensor(a[0]), &G0 = cuda_tensor(a[1]);
    Launch L(G0);
    const Tensor ids = ids2d(ids0), G = as3d(G0);
    const long long N = G.size(0), T = G.size(1), d = G.size(2), n_val = integer(a[2]), vocab = integer(a[3]);
    if (ids.size(0) != N || ids.size(1) != T) invalid("embedding ids and out-grad disagree on [batch, tokens]");
    const long long n_train = N - n_val;
    if (n_train <= 0) invalid("No training samples to compute dot product, check batch sizes.");
    Tensor M = empty({n_val, n_train}, G, at::kFloat);
    Workspace ws;
    const long long ws_bytes = ghost_embedding_pass_workspace_bytes(static_cast<int>(n_train), static_cast<int>(n_val), T,
                                                                    static_cast<int>(vocab), static_cast<int>(d));
    const long long off = ws.plan(ws_bytes);
    char* base = ws.commit(L, G);
    check(ghost_embedding_dot(reinterpret_cast<const long long*>(ids.data_ptr()), G.data_ptr(), is_f32(G),
                              static_cast<int>(n_train), static_cast<int>(n_val), T, static_cast<int>(d),
                              static_cast<int>(vocab), real(a[4]), M.data_ptr<float>(), base + off, ws_bytes, L.st()));
    return wrap(M);
  });
}

// dot products and train gradient in one pass: (ids, G, n_val, vocab, pre_scale) -> (M, grad in the dtype of G)
PyObject* py_embedding_hook(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    need(n, 5, "embedding_hook");
    const Tensor &ids0 = cuda_tensor(a[0]), &G0 = cuda_tensor(a[1]);
    Launch L(G0);
    const Tensor ids = ids2d(ids0), G = as3d(G0);
    const long long N = G.size(0), T = G.size(1), d = G.size(2), n_val = integer(a[2]), vocab = integer(a[3]), n_train = N - n_val;
    if (ids.size(0) != N || ids.size(1) != T) invalid("embedding ids and out-grad disagree on [batch, tokens]");
    check_split(n_train, n_val, "embedding_hook");
    Tensor M = empty({n_val, n_train}, G, at::kFloat), grad = empty({vocab, d}, G, G.scalar_type());
    Workspace ws;
    const long long ws_bytes = ghost_embedding_pass_workspace_bytes(static_cast<int>(n_train), static_cast<int>(n_val), T,
                                                                    static_cast<int>(vocab), static_cast<int>(d));
    const long long off = ws.plan(ws_bytes);
    char* base = ws.commit(L, G);
    check(ghost_embedding_pass(reinterpret_cast<const long long*>(ids.data_ptr()), G.data_ptr(), is_f32(G),
                               static_cast<int>(n_train), static_cast<int>(n_val), T, static_cast<int>(d),
                               static_cast<int>(vocab), 1.f, M.data_ptr<float>(), real(a[4]), static_cast<float>(n_train), 0,
                               grad.data_ptr(), base + off, ws_bytes, L.st()));
    return Py_BuildValue("(NN)", wrap(M), wrap(grad));
  });
}

// (ids, G, n_train, vocab, pre_scale, divisor, out or None, accumulate)
PyObject* py_embedding_wgrad(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    need(n, 8, "embedding_wgrad");
    const Tensor &ids0 = cuda_tensor(a[0]), &G0 = cuda_tensor(a[1]);
    Launch L(G0);
    const Tensor ids = ids2d(ids0), G = as3d(G0);
    const long long T = G.size(1), d = G.size(2), n_train = integer(a[2]), vocab = integer(a[3]);
    const bool have = present(a[6]);
    Tensor out = have ? cuda_tensor(a[6]) : empty({vocab, d}, G, G.scalar_type());
    if (out.scalar_type() != G.scalar_type()) invalid("embedding_wgrad output must have the dtype of the out-grad");
    if (have) check_result(out, vocab, d, G, "embedding_wgrad");
    if (n_train > G.size(0) || ids.size(0) < n_train || ids.size(1) != T)
      invalid("embedding ids and out-grad do not hold the train samples");
    Workspace ws;
    const long long ws_bytes = ghost_embedding_wgrad_workspace_bytes(static_cast<int>(n_train), T, static_cast<int>(vocab));
    const long long off = ws.plan(ws_bytes);
    char* base = ws.commit(L, G);
    check(ghost_embedding_wgrad(reinterpret_cast<const long long*>(ids.data_ptr()), G.data_ptr(), is_f32(G),
                                static_cast<int>(n_train), T, static_cast<int>(d), static_cast<int>(vocab), real(a[4]),
                                real(a[5]), have && integer(a[7]) ? 1 : 0, out.data_ptr(), base + off, ws_bytes, L.st()));
    return wrap(out);
  });
}

// ---- GradProj ---------------------------------------------------------------------------------------------
void check_projection_out(const Tensor& out, long long B, long long k, const char* who) {
  if (out.scalar_type() != at::kFloat || out.dim() != 2 || out.size(0) != B || out.stride(1) != 1 || out.size(1) < k)
    invalid(std::string(who) + " output must be a float32 [B, >= k_r*k_c] row-major view");
}

// (G, A, P_r, P_c, k_r, k_c, scale, out or None: a new [B, k_r, k_c])
PyObject* py_gradproj_dense(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    need(n, 8, "gradproj_dense");
    const Tensor &G0 = cuda_tensor(a[0]), &A0 = cuda_tensor(a[1]), &P_r = cuda_tensor(a[2]), &P_c = cuda_tensor(a[3]);
    Launch L(G0);
    const Tensor G = as3d(G0), A = as3d(A0);
    const long long B = G.size(0), T = G.size(1), k_r = integer(a[4]), k_c = integer(a[5]);
    if (A.size(0) != B || A.size(1) != T)
      throw GhostError(kNotCuda, "Batch size mismatch between activations and output gradients");
    const bool have = present(a[7]);
    const Tensor out = have ? cuda_tensor(a[7]) : empty({B, k_r, k_c}, G, at::kFloat);
    if (have) check_projection_out(out, B, k_r * k_c, "gradproj");
    const bool split = is_f32(G) || is_f32(A);
    const long long n_r = G.size(2), n_c = A.size(2), cp_r = pad8(n_r), cp_c = pad8(n_c);
    if (P_r.size(1) != (split ? 3 : 1) * cp_r || P_c.size(1) != (split ? 3 : 1) * cp_c)
      invalid("projection matrices were prepared for a different dtype/feature size");
    const bool copies = !split && gb::gradproj_copies(B, T, n_r, n_c, tma_ready(G), tma_ready(A), ghost_sm_count());
    if (k_r <= 64 && k_c <= 64 && !copies) {
      // the prepared split lays a float32 matrix out as (hi, hi, lo): the residual part starts at 2 * cp
      const int f32 = !split ? 0 : !is_f32(A) ? 2 : !is_f32(G) ? 3 : 1;
      check(ghost_gradproj_dense(G.data_ptr(), A.data_ptr(), f32, static_cast<int>(B), T, static_cast<int>(n_r),
                                 static_cast<int>(n_c), n_r, n_c, P_r.data_ptr(), P_c.data_ptr(), static_cast<int>(k_r),
                                 static_cast<int>(k_c), P_r.size(1), P_c.size(1), split ? static_cast<int>(2 * cp_r) : 0,
                                 split ? static_cast<int>(2 * cp_c) : 0, real(a[6]), out.data_ptr<float>(), out.stride(0), L.st()));
    } else {
      Workspace ws;
      const Tensor* x[2] = {&G, &A};
      const long long cp[2] = {cp_r, cp_c};
      long long off[2] = {0, 0}, len[2];
      const void* at[2];
      for (int i = 0; i < 2; ++i) {
        len[i] = (split ? 3 : 1) * cp[i];
        if (split || !tma_ready(*x[i])) off[i] = ws.plan(B * T * len[i] * 2);
      }
      char* base = ws.commit(L, G);
      for (int i = 0; i < 2; ++i) {
        const bool copy = split || !tma_ready(*x[i]);
        at[i] = copy ? base + off[i] : x[i]->data_ptr();
        if (copy) Operand(*x[i]).cast(0, B, base + off[i], len[i], cp[i], split ? 3 : 1, kSplitLeft, kSideBySide, L.st());
      }
      check(ghost_gradproj_dense_bf16(at[0], at[1], static_cast<int>(B), T, static_cast<int>(len[0]), static_cast<int>(len[1]), len[0],
                                      len[1], P_r.data_ptr(), P_c.data_ptr(), static_cast<int>(k_r), static_cast<int>(k_c),
                                      P_r.size(1), P_c.size(1), real(a[6]), out.data_ptr<float>(), out.stride(0), L.st()));
    }
    if (!have) return wrap(out);
    Py_INCREF(a[7]);
    return a[7];
  });
}

// (ids, G, P_o, P_i_t, k_o, k_i, scale, out or None)
PyObject* py_gradproj_embedding(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    need(n, 8, "gradproj_embedding");
    const Tensor &ids0 = cuda_tensor(a[0]), &G0 = cuda_tensor(a[1]), &P_o = cuda_tensor(a[2]), &P_i_t = cuda_tensor(a[3]);
    Launch L(G0);
    const Tensor ids = ids2d(ids0), G = as3d(G0);
    const long long B = G.size(0), T = G.size(1), d = G.size(2), k_o = integer(a[4]), k_i = integer(a[5]);
    if (ids.size(0) != B || ids.size(1) != T)
      throw GhostError(kNotCuda, "Batch size mismatch between token ids and output gradients");
    const bool split = is_f32(G) != 0;
    const long long cp = pad8(d);
    if (P_o.scalar_type() != at::kBFloat16 || P_o.dim() != 2 || P_o.size(0) != k_o || P_o.size(1) != (split ? 3 : 1) * cp)
      invalid("P_o was prepared for a different dtype/feature size");
    if (P_i_t.scalar_type() != at::kFloat || P_i_t.dim() != 2 || P_i_t.size(1) != k_i || !P_i_t.is_contiguous())
      invalid("P_i must be passed as the contiguous float32 [vocab, k_i] transpose");
    Tensor out = present(a[7]) ? cuda_tensor(a[7]) : empty({B, k_o * k_i}, G, at::kFloat);
    check_projection_out(out, B, k_o * k_i, "embedding projection");
    // The prepared split lays a float32 matrix out as (hi, hi, lo): the residual part starts at 2 * cp.
    // The kernel covers up to 64 x 64 of a sample's block per launch; larger projections go block by
    // block into the zeroed output.
    const bool chunked = k_o > 64 || k_i > 64;
    if (chunked) out.narrow(1, 0, k_o * k_i).zero_();
    const long long ld_po = P_o.size(1);
    for (long long o0 = 0; o0 < k_o; o0 += 64)
      for (long long i0 = 0; i0 < k_i; i0 += 64)
        check(ghost_gradproj_embedding(reinterpret_cast<const long long*>(ids.data_ptr()), G.data_ptr(), is_f32(G),
                                       static_cast<int>(B), T, static_cast<int>(d), d,
                                       static_cast<const char*>(P_o.data_ptr()) + o0 * ld_po * 2, ld_po, static_cast<int>(cp),
                                       split ? static_cast<int>(2 * cp) : 0, P_i_t.data_ptr<float>() + i0, k_i,
                                       static_cast<int>(P_i_t.size(0)), static_cast<int>(std::min(64ll, k_o - o0)),
                                       static_cast<int>(std::min(64ll, k_i - i0)), real(a[6]), chunked ? 1 : 0,
                                       out.data_ptr<float>() + o0 * k_i + i0, out.stride(0), static_cast<int>(k_i), L.st()));
    return wrap(out);
  });
}

// (P1, P2, scale)
PyObject* py_projection_similarity(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    need(n, 3, "projection_similarity");
    Tensor P1 = cuda_tensor(a[0]), P2 = cuda_tensor(a[1]);
    Launch L(P1);
    if (P1.dim() != 2 || P2.dim() != 2 || P1.size(1) != P2.size(1)) invalid("projection sets have different dimensions");
    if (P1.scalar_type() != P2.scalar_type()) {
      const at::ScalarType common = c10::promoteTypes(P1.scalar_type(), P2.scalar_type());
      P1 = P1.to(common);
      P2 = P2.to(common);
    }
    if (P1.scalar_type() != at::kFloat && P1.scalar_type() != at::kBFloat16) {
      P1 = P1.to(at::kFloat);
      P2 = P2.to(at::kFloat);
    }
    if (P1.stride(1) != 1) P1 = P1.contiguous();
    if (P2.stride(1) != 1) P2 = P2.contiguous();
    Tensor S = empty({P1.size(0), P2.size(0)}, P1, at::kFloat);
    check(ghost_projection_similarity(P1.data_ptr(), P2.data_ptr(), is_f32(P1), static_cast<int>(P1.size(0)),
                                      static_cast<int>(P2.size(0)), P1.size(1), P1.stride(0), P2.stride(0), real(a[2]),
                                      S.data_ptr<float>(), S.stride(0), L.st()));
    return wrap(S);
  });
}

// ---- end of a backward pass ---------------------------------------------------------------------------------
PyObject *k_X, *k_M, *k_sum_out, *k_n_train, *k_n_val, *k_dot_scale, *k_sum_scale, *k_Xv;
PyObject *k_param, *k_matrix, *k_vector, *k_train_grad, *k_add, *k_parameters, *k_modules, *k_named_modules;

PyObject* item(PyObject* dict, PyObject* key) { return PyDict_GetItemWithError(dict, key); }   // borrowed

ghost_pass_job read_job(PyObject* d, int* device) {
  if (!PyDict_Check(d)) invalid("small_reduce_batch takes a list of dicts");
  ghost_pass_job j = {};
  PyObject *x = item(d, k_X), *m = item(d, k_M), *s = item(d, k_sum_out);
  if (!present(x)) invalid("small_reduce_batch: a job has no input");
  const Tensor& X = cuda_tensor(x);
  if (X.scalar_type() != at::kFloat || X.dim() != 2 || !X.is_contiguous())
    invalid("small_reduce_batch takes contiguous float32 [N, F] tensors");
  PyObject *nt = item(d, k_n_train), *nv = item(d, k_n_val);
  if (!present(nt) || !present(nv)) invalid("small_reduce_batch: a job has no n_train / n_val");
  *device = X.get_device();
  j.X = X.data_ptr<float>();
  j.F = static_cast<int>(X.size(1));
  j.n_train = static_cast<int>(integer(nt));
  j.n_val = static_cast<int>(integer(nv));
  j.dot_scale = present(item(d, k_dot_scale)) ? real(item(d, k_dot_scale)) : 1.f;
  j.sum_scale = present(item(d, k_sum_scale)) ? real(item(d, k_sum_scale)) : 1.f;
  j.sum_is_f32 = 1;
  if (present(m)) {
    const Tensor& M = cuda_tensor(m);
    if (M.scalar_type() != at::kFloat || !M.is_contiguous() || M.numel() != static_cast<long long>(j.n_val) * j.n_train)
      invalid("small_reduce_batch: M must be a contiguous float32 [n_val, n_train] tensor");
    j.M = M.data_ptr<float>();
  }
  if (present(s)) {
    const Tensor& out = cuda_tensor(s);
    if (!out.is_contiguous() || out.numel() != X.size(1)) invalid("small_reduce_batch: sum_out must be a contiguous [F] tensor");
    j.sum_out = out.data_ptr();
    j.sum_is_f32 = is_f32(out);
  }
  PyObject* xv = item(d, k_Xv);
  if (present(xv)) {
    if (!PyTuple_Check(xv) || PyTuple_GET_SIZE(xv) != 3) invalid("small_reduce_batch: bad layout of the separate validation rows");
    const Tensor& g = cuda_tensor(PyTuple_GET_ITEM(xv, 0));
    const long long offset = integer(PyTuple_GET_ITEM(xv, 1)), per_rank = integer(PyTuple_GET_ITEM(xv, 2));
    if (g.scalar_type() != at::kFloat || g.dim() != 2 || !g.is_contiguous() || offset + per_rank * X.size(1) > g.size(1) ||
        g.size(0) * per_rank != j.n_val || X.size(0) < j.n_train)
      invalid("small_reduce_batch: bad layout of the separate validation rows");
    j.Xv = g.data_ptr<float>() + offset;
    j.v_rank_pitch = g.size(1);
    j.v_per_rank = static_cast<int>(per_rank);
  }
  return j;
}

// The jobs' reductions and every matrix's sum over the validation samples, one launch per device; the sums, one vector per
// matrix.  A matrix that a job fills gets its sum from that job.
std::vector<Tensor> reduce_pass(PyObject* jobs, const std::vector<PyObject*>& mats) {
  struct OnDevice { int device; Tensor any; std::vector<ghost_pass_job> jobs; };      // a tensor of it, for its stream
  std::vector<OnDevice> devices;
  auto on = [&](int device, const Tensor& t) -> size_t {
    for (size_t i = 0; i < devices.size(); ++i)
      if (devices[i].device == device) return i;
    devices.push_back({device, t, {}});
    devices.back().jobs.reserve(mats.size() + static_cast<size_t>(PyList_GET_SIZE(jobs)));
    return devices.size() - 1;
  };
  struct Filled { size_t device, job; const Tensor* vec; };
  std::unordered_map<const float*, Filled> filled;
  for (Py_ssize_t i = 0; i < PyList_GET_SIZE(jobs); ++i) {
    PyObject* d = PyList_GET_ITEM(jobs, i);
    int dev = 0;
    ghost_pass_job j = read_job(d, &dev);
    if (j.M == nullptr && j.sum_out == nullptr) invalid("small_reduce_batch: a job has no output");
    const size_t at = on(dev, cuda_tensor(item(d, k_X)));
    if (j.M) filled[j.M] = {at, devices[at].jobs.size(), nullptr};
    devices[at].jobs.push_back(j);
  }
  std::vector<Tensor> out(mats.size());
  // one buffer per run of equal column counts keeps the vectors' allocations to one or two
  for (size_t i = 0; i < mats.size();) {
    const Tensor first = cuda_tensor(mats[i]);
    size_t e = i;
    while (e < mats.size()) {
      const Tensor& t = cuda_tensor(mats[e]);
      if (t.scalar_type() != at::kFloat || t.dim() != 2 || !t.is_contiguous())
        invalid("pass_reduce: matrices are contiguous float32 [n_val, n_train]");
      if (t.size(1) != first.size(1) || t.get_device() != first.get_device()) break;
      ++e;
    }
    Tensor vecs = empty({static_cast<long long>(e - i), first.size(1)}, first, at::kFloat);
    for (size_t k = i; k < e; ++k) {
      const Tensor& t = cuda_tensor(mats[k]);
      auto it = filled.find(t.data_ptr<float>());
      if (it != filled.end() && it->second.vec != nullptr) {
        out[k] = *it->second.vec;           // listed again: a job of its own would read the matrix while the first one writes it
        continue;
      }
      out[k] = vecs.select(0, static_cast<long long>(k - i));
      float* vp = out[k].data_ptr<float>();
      if (it != filled.end()) {
        devices[it->second.device].jobs[it->second.job].vec = vp;
        it->second.vec = &out[k];
      } else {
        ghost_pass_job j = {};
        j.M = t.data_ptr<float>();
        j.vec = vp;
        j.n_val = static_cast<int>(t.size(0));
        j.n_train = static_cast<int>(t.size(1));
        devices[on(t.get_device(), t)].jobs.push_back(j);
      }
    }
    i = e;
  }
  for (OnDevice& d : devices) {
    Launch L(d.any);
    check(ghost_pass_reduce(d.jobs.data(), static_cast<int>(d.jobs.size()), L.st()));
  }
  return out;
}

// (jobs: list of dicts, matrices: list of [n_val, n_train] tensors) -> list of [n_train] tensors, one per matrix
PyObject* py_pass_reduce(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    need(n, 2, "pass_reduce");
    if (!PyList_Check(a[0]) || !PyList_Check(a[1])) invalid("pass_reduce takes two lists");
    std::vector<PyObject*> mats(static_cast<size_t>(PyList_GET_SIZE(a[1])));
    for (size_t i = 0; i < mats.size(); ++i) mats[i] = PyList_GET_ITEM(a[1], static_cast<Py_ssize_t>(i));
    const std::vector<Tensor> vecs = reduce_pass(a[0], mats);
    PyObject* out = PyList_New(static_cast<Py_ssize_t>(vecs.size()));
    if (!out) throw std::bad_alloc();
    for (size_t i = 0; i < vecs.size(); ++i) PyList_SET_ITEM(out, static_cast<Py_ssize_t>(i), wrap(vecs[i]));
    return out;
  });
}

// A new reference that is given up at the end of the scope; null: a Python error is set.
struct Owned {
  PyObject* o;
  explicit Owned(PyObject* p) : o(p) {
    if (!o) throw python_error();
  }
  Owned(const Owned&) = delete;
  Owned& operator=(const Owned&) = delete;
  ~Owned() { Py_DECREF(o); }
};
// The instance dictionary of a parameter (a tensor of any class)
PyObject* instance_dict(PyObject* o) { return PyObject_GenericGetDict(o, nullptr); }
void set_item(PyObject* dict, PyObject* key, PyObject* value) {
  if (PyDict_SetItem(dict, key, value) != 0) throw python_error();
}

// (jobs: list of dicts, dots: list of (parameter, matrix), observer or None) -> whether it was done: all matrices are on GPUs.
// The hooks' lists at the end of a backward pass: pass_reduce, the vectors as <parameter>.grad_dot_prod, and the jobs'
// train gradients as <parameter>.train_grad or added to it.  A parameter that is listed again keeps its last matrix, as it does
// when every hook overwrites the attribute.
PyObject* py_finish_pass(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    need(n, 3, "finish_pass");
    if (!PyList_Check(a[0]) || !PyList_Check(a[1])) invalid("finish_pass takes two lists");
    std::vector<PyObject*> params, mats;
    std::unordered_map<PyObject*, size_t> where;
    for (Py_ssize_t i = 0; i < PyList_GET_SIZE(a[1]); ++i) {
      PyObject* e = PyList_GET_ITEM(a[1], i);
      if (!PyTuple_Check(e) || PyTuple_GET_SIZE(e) != 2) invalid("finish_pass: pairs of a parameter and its matrix");
      PyObject *param = PyTuple_GET_ITEM(e, 0), *m = PyTuple_GET_ITEM(e, 1);
      if (!tensor(m).is_cuda()) Py_RETURN_FALSE;
      const auto [it, is_new] = where.emplace(param, params.size());
      if (is_new) {
        params.push_back(param);
        mats.push_back(m);
      } else {
        mats[it->second] = m;
      }
    }
    const std::vector<Tensor> vecs = reduce_pass(a[0], mats);
    for (size_t i = 0; i < vecs.size(); ++i) {
      Owned own(instance_dict(params[i]));
      if (item(own.o, k_matrix) != mats[i]) continue;
      Owned v(wrap(vecs[i]));
      set_item(own.o, k_vector, v.o);
    }
    for (Py_ssize_t i = 0; i < PyList_GET_SIZE(a[0]); ++i) {
      PyObject *job = PyList_GET_ITEM(a[0], i), *param = item(job, k_param), *grad = item(job, k_sum_out);
      if (!present(param) || !present(grad)) continue;
      const Tensor &g = tensor(grad), &p = tensor(param);
      Owned mine(g.sizes() == p.sizes() ? Py_NewRef(grad) : wrap(g.view(p.sizes())));
      Owned own(instance_dict(param));
      PyObject* sum = item(own.o, k_train_grad);
      if (sum == nullptr) {
        set_item(own.o, k_train_grad, mine.o);
      } else {
        const Owned added(PyObject_CallMethodOneArg(sum, k_add, mine.o));
      }
      if (present(a[2])) {
        const Owned told(PyObject_CallOneArg(a[2], param));
      }
    }
    Py_RETURN_TRUE;
  });
}

// (matrices: list of equal [n_val, n_train]) -> float32 buffer of n_val * n_train + n_train + 1 elements: the
// summed matrix, its column sums, and the device error word (bits of an int32)
PyObject* py_matrix_sum(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    need(n, 1, "matrix_sum");
    if (!PyList_Check(a[0]) || PyList_GET_SIZE(a[0]) == 0) invalid("matrix_sum takes a list of matrices");
    const Tensor& first = cuda_tensor(PyList_GET_ITEM(a[0], 0));
    if (first.dim() != 2) invalid("matrix_sum: matrices are [n_val, n_train]");
    Launch L(first);
    const long long nv = first.size(0), nt = first.size(1);
    std::vector<const float*> p;
    for (Py_ssize_t i = 0; i < PyList_GET_SIZE(a[0]); ++i) {
      const Tensor& t = cuda_tensor(PyList_GET_ITEM(a[0], i));
      if (t.scalar_type() != at::kFloat || !t.is_contiguous() || t.sizes() != first.sizes() || t.get_device() != first.get_device())
        invalid("matrix_sum: matrices must be contiguous float32 of one shape on one device");
      p.push_back(t.data_ptr<float>());
    }
    Tensor out = empty({nv * nt + nt + 1}, first, at::kFloat);
    float* o = out.data_ptr<float>();
    check(ghost_matrix_sum(p.data(), static_cast<int>(p.size()), static_cast<int>(nv), static_cast<int>(nt), o, o + nv * nt,
                           reinterpret_cast<int*>(o + nv * nt + nt), L.st()));
    return wrap(out);
  });
}

// (module, torch.nn.Module.named_modules) -> [(qualified name, parameter)] as module.named_parameters() gives
// them: every parameter once, modules in depth-first order.  The engines walk the model three times a
// step.  False: a module keeps its tables elsewhere than in its dictionary (scripted modules) or lists its
// modules in a way of its own, and the caller asks torch.
struct Walk {
  PyObject* named_modules;
  std::unordered_set<PyObject*> seen;                // modules and parameters
  std::unordered_set<PyTypeObject*> plain;           // module types with torch's own listing
};
bool walk_parameters(PyObject* module, const std::string& prefix, Walk& walk, PyObject* out) {
  if (!walk.seen.insert(module).second) return true;
  if (walk.plain.find(Py_TYPE(module)) == walk.plain.end()) {
    PyObject* listing = PyObject_GetAttr(reinterpret_cast<PyObject*>(Py_TYPE(module)), k_named_modules);
    if (!listing) PyErr_Clear();
    const bool own = listing != walk.named_modules;
    Py_XDECREF(listing);
    if (own) return false;
    walk.plain.insert(Py_TYPE(module));
  }
  PyObject* dict = PyObject_GenericGetDict(module, nullptr);
  if (!dict) { PyErr_Clear(); return false; }
  Owned hold(dict);
  PyObject *key, *value;
  Py_ssize_t pos = 0;
  PyObject *params = item(dict, k_parameters), *modules = item(dict, k_modules);
  if (!params || !PyDict_Check(params) || !modules || !PyDict_Check(modules) || item(dict, k_named_modules)) return false;
  while (PyDict_Next(params, &pos, &key, &value)) {
    if (value == Py_None || !walk.seen.insert(value).second) continue;
    Py_ssize_t size = 0;
    const char* name = PyUnicode_AsUTF8AndSize(key, &size);
    if (!name) throw python_error();
    const std::string full = prefix + std::string(name, static_cast<size_t>(size));
    Owned text(PyUnicode_FromStringAndSize(full.data(), static_cast<Py_ssize_t>(full.size())));
    Owned entry(PyTuple_Pack(2, text.o, value));
    if (PyList_Append(out, entry.o) != 0) throw python_error();
  }
  pos = 0;
  while (PyDict_Next(modules, &pos, &key, &value)) {
    if (value == Py_None) continue;
    Py_ssize_t size = 0;
    const char* name = PyUnicode_AsUTF8AndSize(key, &size);
    if (!name) throw python_error();
    if (!walk_parameters(value, prefix + std::string(name, static_cast<size_t>(size)) + ".", walk, out)) return false;
  }
  return true;
}

PyObject* py_named_parameters(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    need(n, 2, "named_parameters");
    PyObject* out = PyList_New(0);
    if (!out) throw std::bad_alloc();
    Walk walk{a[1], {}, {}};
    try {
      if (!walk_parameters(a[0], "", walk, out)) {
        Py_DECREF(out);
        Py_RETURN_NONE;
      }
    } catch (...) {
      Py_DECREF(out);
      throw;
    }
    return out;
  });
}

// ---- the gradient of a layer's output -----------------------------------------------------------------------
// Calls fn(gradient in the output's shape, or None) before the node runs.
class OutputHook : public torch::autograd::FunctionPreHook {
 public:
  OutputHook(PyObject* fn, size_t index, at::IntArrayRef shape) : fn_(fn), index_(index), shape_(shape.vec()) { Py_INCREF(fn_); }
  ~OutputHook() override {
    if (!Py_IsInitialized()) return;
    const PyGILState_STATE gil = PyGILState_Ensure();
    Py_DECREF(fn_);
    PyGILState_Release(gil);
  }
  torch::autograd::variable_list operator()(const torch::autograd::variable_list& grads) override {
    const PyGILState_STATE gil = PyGILState_Ensure();
    try {
      call(grads[index_]);
    } catch (...) {
      PyGILState_Release(gil);
      throw;
    }
    PyGILState_Release(gil);
    return grads;
  }

 private:
  void call(const Tensor& grad) const {
    PyObject* arg = !grad.defined() ? Py_NewRef(Py_None) : wrap(grad.sizes() == shape_ ? grad : grad.reshape(shape_));
    PyObject* result = arg ? PyObject_CallOneArg(fn_, arg) : nullptr;
    Py_XDECREF(arg);
    if (!result) {
      python_error error;
      error.persist();
      throw std::move(error);
    }
    Py_DECREF(result);
  }
  PyObject* fn_;
  size_t index_;
  std::vector<int64_t> shape_;
};

// (output, fn): hook the node that hands the output's gradient on.  Linear layers return a reshaped view of
// their product; an in-place operation on a view gives it a new node and drops the old one with its hooks, so
// there the base's node is taken.  False: no node has produced it.
PyObject* py_hook_output(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    need(n, 2, "hook_output");
    const Tensor& out = tensor(a[0]);
    torch::autograd::Edge edge = torch::autograd::impl::gradient_edge(out);
    if (out.is_view()) {
      const Tensor base(out._base());
      if (base.requires_grad() && base.grad_fn() && base.numel() == out.numel() && base.is_contiguous() && out.is_contiguous())
        edge = torch::autograd::impl::gradient_edge(base);
    }
    if (!out.grad_fn()) Py_RETURN_FALSE;
    edge.function->add_pre_hook(std::make_unique<OutputHook>(a[1], edge.input_nr, out.sizes()));
    Py_RETURN_TRUE;
  });
}

PyObject* py_set_kernel_error(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n == 1) {
    Py_XDECREF(g_kernel_error);
    Py_INCREF(a[0]);
    g_kernel_error = a[0];
  }
  Py_RETURN_NONE;
}

#define GB_METHOD(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(py_##name)), METH_FASTCALL, nullptr}
PyMethodDef kMethods[] = {
    GB_METHOD(gram_dot),          GB_METHOD(wgrad),
    GB_METHOD(persample_dot),     GB_METHOD(colsum),
    GB_METHOD(norm_persample),    GB_METHOD(embedding_dot),
    GB_METHOD(embedding_wgrad),   GB_METHOD(gradproj_dense),
    GB_METHOD(gradproj_embedding), GB_METHOD(projection_similarity),
    GB_METHOD(pass_reduce),       GB_METHOD(finish_pass),
    GB_METHOD(matrix_sum),
    GB_METHOD(dense_hook),        GB_METHOD(conv_hook),
    GB_METHOD(norm_hook),
    GB_METHOD(embedding_hook),    GB_METHOD(named_parameters),
    GB_METHOD(hook_output),
    GB_METHOD(arena_clear),       GB_METHOD(set_kernel_error),
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_ghost_torch", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

// The torch release whose headers this was compiled against; looked for in the file before it is loaded.
extern "C" __attribute__((visibility("default"), used)) const char ghost_torch_built_for[] =
    "ghost_torch built for torch " GHOST_TORCH_VERSION "\n";

PyMODINIT_FUNC PyInit__ghost_torch() {
  struct { PyObject** at; const char* name; } keys[] = {{&k_X, "X"}, {&k_M, "M"}, {&k_sum_out, "sum_out"}, {&k_n_train, "n_train"},
                                                        {&k_n_val, "n_val"}, {&k_dot_scale, "dot_scale"},
                                                        {&k_sum_scale, "sum_scale"}, {&k_Xv, "Xv"}, {&k_param, "param"},
                                                        {&k_matrix, "grad_dot_prod_matrix"}, {&k_vector, "grad_dot_prod"},
                                                        {&k_train_grad, "train_grad"}, {&k_add, "add_"},
                                                        {&k_parameters, "_parameters"}, {&k_modules, "_modules"},
                                                        {&k_named_modules, "named_modules"}};
  for (auto& k : keys) *k.at = PyUnicode_InternFromString(k.name);
  return PyModule_Create(&kModule);
}
