// Native host path of the package: argument checks, output and scratch allocation, stream lookup and
// the autograd rules of every op, between Python and the C ABI (include/s2cnn_b200.h).
//
// The layers of this library are short kernels (a small network's forward pass is five launches of
// 3 - 30 us), so the host work per op decides the latency of small calls and of training steps: with
// the checks, allocations and ctypes calls in Python an op cost 20 - 30 us and its Python autograd
// rule as much again.  Here an op costs a few microseconds, and its backward runs in the autograd
// engine's thread without the interpreter lock.
//
// One `Ops` object wraps one build of the library, found by path: the CUDA build in the product, the
// host-emulation build in the CPU tests - the same code drives both.
#include <dlfcn.h>

#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/extension.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/jit/frontend/tracer.h>

#include <atomic>
#include <cmath>
#include <optional>
#include <string>
#include <tuple>
#include <vector>

#include <nvtx3/nvToolsExt.h>

#include "../../include/s2cnn_b200.h"

namespace {

using at::Tensor;
using OptTensor = std::optional<Tensor>;
using torch::autograd::AutogradContext;
using torch::autograd::tensor_list;
using torch::autograd::Variable;

// ---- errors ---------------------------------------------------------------------------------------
// Set as Python exceptions and carried as python_error, so that the type survives the autograd
// engine (which rethrows the exception of a backward pass in the thread that called it).
PyObject* g_s2c_error = nullptr;   // s2cnn_b200._lib.S2cError
PyObject* g_traced = nullptr;      // s2cnn_b200.ops._traced
// Whether torch.jit.trace is recording this thread's calls, other than within an op that it records as one node.
thread_local int g_inside_traced_op = 0;
bool tracing() { return torch::jit::tracer::isTracing() && g_inside_traced_op == 0; }
struct InsideTracedOp {   // a Python context manager
  void enter() { ++g_inside_traced_op; }
  void exit(pybind11::args) { --g_inside_traced_op; }
};

[[noreturn]] void raise(PyObject* type, const std::string& msg) {
  pybind11::gil_scoped_acquire gil;
  PyErr_SetString(type, msg.c_str());
  python_error e;
  e.persist();
  throw e;
}
[[noreturn]] void raise_s2c(const std::string& msg) { raise(g_s2c_error, msg); }
inline void check(bool ok, const char* what) {
  if (!ok) raise(PyExc_AssertionError, what);
}

long so3_nspec(long b) { return b * (4 * b * b - 1) / 3; }
long so3_bandwidth(long nspec) {   // as s2cnn/soft/so3_fft.py:121-122
  const long b = std::lround(std::cbrt(0.75 * (double)nspec));
  if (so3_nspec(b) != nspec)
    raise(PyExc_AssertionError, "not an SO(3) spectrum length: " + std::to_string(nspec));
  return b;
}
long s2_bandwidth(long nspec) {
  const long b = std::lround(std::sqrt((double)nspec));
  if (b * b != nspec) raise(PyExc_AssertionError, "not an S2 spectrum length: " + std::to_string(nspec));
  return b;
}

// ---- one build of the library ---------------------------------------------------------------------
#define S2C_API(X)                                                                                 \
  X(last_error) X(is_cuda_build) X(tables_computed) X(so3_analysis_workspace) X(so3_synthesis_workspace) X(so3_rfft)               \
  X(so3_rfft_relu) X(so3_rfft_sums_ws) X(so3_relay_workspace) X(s2_conv_relu_so3_rfft_workspace) X(s2_conv_relu_so3_rfft_ws) X(so3_rifft_relu_rfft_ws) X(so3_rifft_relu_grad_ws) X(so3_fft) X(so3_rifft)                 \
  X(so3_rifft_relu_integrate)                      \
  X(s2_conv_synthesis_workspace) X(s2_conv_synthesis) X(s2_conv_real_synthesis_workspace) X(s2_conv_real_synthesis) X(s2_conv_real_relu_so3_rfft) X(so3_ifft) X(s2_fft_workspace) X(s2_fft)    \
  X(s2_ifft) X(so3_mm) X(so3_mm_gradx_ws) X(so3_mm_gradx_workspace) X(so3_mm_grady_ws) X(so3_mm_grady_workspace) X(so3_mm_real) X(so3_mm_real_workspace) X(so3_mm_tc_status) X(s2_mm) X(s2_mm_gradx) \
  X(s2_mm_grady) X(s2_mm_real_gradx) X(s2_mm_real_grady) X(rft_forward) X(rft_forward_t) X(rft_forward_scaled) X(rft_backward_scaled) X(rft_backward_workspace) X(so3_integrate)                  \
  X(so3_integrate_backward) X(so3_rotate_spectrum) X(project_on_sphere)

struct Ops {
#define X(name) decltype(&::s2c_##name) name##_ = nullptr;
  S2C_API(X)
#undef X
  bool is_cuda = false, nvtx = false, check_tc = false;
  std::atomic<long> tables_seen{0};
  PyObject* on_new_tables = nullptr;   // called with (what) when a call has built tables

  Ops(const std::string& path, pybind11::object on_tables, bool use_nvtx, bool check_tensor_cores) {
    void* h = dlopen(path.c_str(), RTLD_NOW | RTLD_LOCAL);
    if (!h) raise_s2c(std::string("cannot load ") + path + ": " + dlerror());
#define X(name)                                                                       \
  name##_ = reinterpret_cast<decltype(name##_)>(dlsym(h, "s2c_" #name));              \
  if (!name##_) raise_s2c(std::string("symbol s2c_" #name " missing in ") + path);
    S2C_API(X)
#undef X
    is_cuda = is_cuda_build_() != 0;
    nvtx = use_nvtx && is_cuda;
    check_tc = check_tensor_cores && is_cuda;
    on_new_tables = on_tables.release().ptr();
  }

  // -- helpers --------------------------------------------------------------------------------------
  // These ops write through raw pointers, which neither a tracer (it would record the allocation of the
  // result and nothing that fills it) nor forward-mode differentiation sees: refused here.  The
  // differentiable ops are recorded by a tracer as one node each, see S2C_TRACED.
  void prep(const Tensor& t) const {
    if (tracing())
      raise(PyExc_RuntimeError, "s2cnn_b200: torch.jit.trace cannot record this op (the differentiable layers and transforms can be traced)");
    if (t._fw_grad(0).defined())
      raise(PyExc_NotImplementedError, "s2cnn_b200 ops do not implement forward-mode automatic differentiation (no jvp)");
    if (t.scalar_type() != at::kFloat)
      raise(PyExc_TypeError, std::string("s2cnn_b200 kernels are float32 only, got ") + c10::toString(t.scalar_type()));
    if (t.is_cuda() != is_cuda)
      raise_s2c("s2cnn_b200: tensor on " + t.device().str() + " but the loaded library is the " +
                (is_cuda ? "CUDA" : "emulation") + " build - the product path runs on CUDA only");
  }
  void prep(const OptTensor& t) const {
    if (t) prep(*t);
  }

  // Device and stream of a call: the tensor's device is made current, its current stream is used.
  struct Ctx {
    std::optional<c10::cuda::CUDAGuard> guard;
    void* stream = nullptr;
    Ctx(const Ops& o, const Tensor& t) {
      if (o.is_cuda) {
        guard.emplace(t.device());
        stream = c10::cuda::getCurrentCUDAStream(t.device().index()).stream();
      }
    }
  };

  template <class F, class... A>
  int call_rc(const char* name, F fn, A... args) const {
    if (nvtx) nvtxRangePushA(name);
    const int rc = fn(args...);
    if (nvtx) nvtxRangePop();
    return rc;
  }
  template <class F, class... A>
  void call(const char* name, F fn, A... args) const {
    const int rc = call_rc(name, fn, args...);
    if (rc != 0)
      raise_s2c(std::string(name) + " failed (status " + std::to_string(rc) + "): " + last_error_());
  }
#define S2C_CALL(name, ...) call("s2c_" #name, name##_, __VA_ARGS__)

  // The reference logs "Compute Wigner ..." on the "trainer" logger whenever a table is built
  // (s2cnn/soft/so3_fft.py:223, s2_fft.py:127); same here, from the library's counter.
  void log_new_tables(const char* what, long b_in, long b_out) {
    const long n = tables_computed_();
    if (n == tables_seen.load(std::memory_order_relaxed)) return;
    tables_seen = n;
    pybind11::gil_scoped_acquire gil;
    const pybind11::handle callback(on_new_tables);
    callback(std::string(what) + " b " + std::to_string(b_in) + " -> " + std::to_string(b_out), n);
  }

  static long lead_numel(at::IntArrayRef s) {
    long n = 1;
    for (auto v : s) n *= v;
    return n;
  }
  static std::vector<int64_t> spectrum_shape(long nspec, at::IntArrayRef lead) {
    std::vector<int64_t> s;
    s.reserve(lead.size() + 2);
    s.push_back(nspec);
    s.insert(s.end(), lead.begin(), lead.end());
    s.push_back(2);
    return s;
  }
  static std::vector<int64_t> signal_shape(at::IntArrayRef lead, long n, int axes, bool complex) {
    std::vector<int64_t> s(lead.begin(), lead.end());
    for (int i = 0; i < axes; ++i) s.push_back(n);
    if (complex) s.push_back(2);
    return s;
  }
  static Tensor empty_like_shape(const Tensor& like, at::IntArrayRef shape) { return at::empty(shape, like.options()); }
  // scratch space of one call; none where the kernels it will take need none
  struct Scratch {
    Tensor keep;
    void* p = nullptr;
    size_t n = 0;
    Scratch(size_t bytes, const Tensor& like) : n(bytes) {
      if (!bytes) return;
      keep = at::empty({(int64_t)bytes}, like.options().dtype(at::kByte));
      p = keep.mutable_data_ptr();
    }
  };
  // bias -> (contiguous flat tensor kept alive, pointer, count); the feature axis is the last of `lead`
  static const float* bias_ptr(const OptTensor& bias, Tensor& keep, int& nfeat) {
    nfeat = 0;
    if (!bias) return nullptr;
    keep = bias->contiguous();
    nfeat = (int)keep.numel();
    return keep.const_data_ptr<float>();
  }
  static long b_or(const std::optional<int64_t>& b, long otherwise) { return b ? (long)*b : otherwise; }
  static const float* cptr(const Tensor& t) { return t.const_data_ptr<float>(); }
  static float* ptr(const Tensor& t) { return t.mutable_data_ptr<float>(); }

  // -- SO(3) transforms -----------------------------------------------------------------------------
  static long so3_side(const Tensor& x, int first_trailing) {
    const long d = x.dim();
    check(d >= first_trailing, "SO(3) signal: too few axes");
    const long n = x.size(d - first_trailing);
    check(n % 2 == 0 && n > 0 && x.size(d - first_trailing + 1) == n && x.size(d - first_trailing + 2) == n,
          "SO(3) signal: the last three axes must be 2b x 2b x 2b");
    return n / 2;
  }

  Tensor so3_rfft(const Tensor& x_, bool for_grad, std::optional<int64_t> b_out_, bool relu) {
    prep(x_);
    const long b_in = so3_side(x_, 3), b_out = b_or(b_out_, b_in);
    const Tensor x = x_.contiguous();
    const auto lead = x.sizes().slice(0, x.dim() - 3);
    const long nb = lead_numel(lead);
    Tensor out = empty_like_shape(x, spectrum_shape(so3_nspec(b_out), lead));
    Ctx c(*this, x);
    const Scratch ws(so3_analysis_workspace_(nb, b_in, b_out), x);
    if (relu) {
      check(!for_grad, "so3_rfft: relu goes with the forward weighting");
      S2C_CALL(so3_rfft_relu, cptr(x), ptr(out), nb, (int)b_in, (int)b_out, ws.p, ws.n, c.stream);
    } else {
      S2C_CALL(so3_rfft, cptr(x), ptr(out), nb, (int)b_in, (int)b_out, (int)for_grad, ws.p, ws.n, c.stream);
    }
    log_new_tables("so3_rfft", b_in, b_out);
    return out;
  }

  std::tuple<Tensor, Tensor> so3_rfft_with_sums(const Tensor& x_, bool for_grad, std::optional<int64_t> b_out_) {
    prep(x_);
    const long b_in = so3_side(x_, 3), b_out = b_or(b_out_, b_in);
    const Tensor x = x_.contiguous();
    const auto lead = x.sizes().slice(0, x.dim() - 3);
    const long nb = lead_numel(lead);
    if (2 * b_in < 64) {
      Tensor out = empty_like_shape(x, spectrum_shape(so3_nspec(b_out), lead));
      Tensor sums = empty_like_shape(x, lead);
      Ctx c(*this, x);
      const Scratch ws(so3_analysis_workspace_(nb, b_in, b_out), x);
      const int rc = call_rc("s2c_so3_rfft_sums_ws", so3_rfft_sums_ws_, cptr(x), ptr(out), ptr(sums), nb, (int)b_in,
                             (int)b_out, (int)for_grad, ws.p, ws.n, c.stream);
      if (rc == 0) {
        log_new_tables("so3_rfft", b_in, b_out);
        return {out, sums};
      }
      if (rc != 4)   // 4: no such kernel for this size, nothing written
        raise_s2c("s2c_so3_rfft_sums_ws failed (status " + std::to_string(rc) + "): " + last_error_());
    }
    return {so3_rfft(x, for_grad, b_out, false), x.sum({-3, -2, -1})};
  }

  Tensor so3_fft(const Tensor& x_, bool for_grad, std::optional<int64_t> b_out_) {
    prep(x_);
    check(x_.dim() >= 4 && x_.size(-1) == 2, "so3_fft: the last axis holds (re, im)");
    const long b_in = so3_side(x_, 4), b_out = b_or(b_out_, b_in);
    const Tensor x = x_.contiguous();
    const auto lead = x.sizes().slice(0, x.dim() - 4);
    const long nb = lead_numel(lead);
    Tensor out = empty_like_shape(x, spectrum_shape(so3_nspec(b_out), lead));
    Ctx c(*this, x);
    const Scratch ws(so3_analysis_workspace_(nb, b_in, b_out), x);
    S2C_CALL(so3_fft, cptr(x), ptr(out), nb, (int)b_in, (int)b_out, (int)for_grad, ws.p, ws.n, c.stream);
    return out;
  }

  Tensor so3_rifft(const Tensor& x_, bool for_grad, std::optional<int64_t> b_out_, const OptTensor& bias) {
    prep(x_);
    prep(bias);
    check(x_.dim() >= 2 && x_.size(-1) == 2, "so3_rifft: the last axis holds (re, im)");
    const long b_in = so3_bandwidth(x_.size(0)), b_out = b_or(b_out_, b_in);
    const Tensor x = x_.contiguous();
    const auto lead = x.sizes().slice(1, x.dim() - 2);
    const long nb = lead_numel(lead);
    Tensor out = empty_like_shape(x, signal_shape(lead, 2 * b_out, 3, false)), keep;
    int nfeat;
    const float* bp = bias_ptr(bias, keep, nfeat);
    check(!bp || (!lead.empty() && lead.back() == nfeat), "so3_rifft: one bias per feature (last leading axis)");
    Ctx c(*this, x);
    const Scratch ws(so3_synthesis_workspace_(nb, b_in, b_out), x);
    S2C_CALL(so3_rifft, cptr(x), ptr(out), nb, (int)b_in, (int)b_out, (int)for_grad, bp, nfeat, ws.p, ws.n, c.stream);
    log_new_tables("so3_rifft", b_in, b_out);
    return out;
  }

  Tensor so3_rifft_relu_grad(const Tensor& x_, const Tensor& act_) {
    prep(x_);
    prep(act_);
    const long b_in = so3_bandwidth(x_.size(0)), b_out = so3_side(act_, 3);
    const Tensor x = x_.contiguous(), act = act_.contiguous();
    const auto lead = act.sizes().slice(0, act.dim() - 3);
    check(x.size(-1) == 2 && x.sizes().slice(1, x.dim() - 2) == lead, "so3_rifft_relu_grad: shapes differ");
    Tensor out = at::empty_like(act);
    Ctx c(*this, x);
    const long nb = lead_numel(lead);
    const Scratch ws(so3_synthesis_workspace_(nb, b_in, b_out), x);
    S2C_CALL(so3_rifft_relu_grad_ws, cptr(x), cptr(act), ptr(out), nb, (int)b_in, (int)b_out, ws.p, ws.n, c.stream);
    return out;
  }

  Tensor so3_rifft_relu_integrate(const Tensor& x_, const OptTensor& bias, std::optional<int64_t> b_out_) {
    prep(x_);
    prep(bias);
    check(x_.dim() >= 2 && x_.size(-1) == 2, "so3_rifft_relu_integrate: the last axis holds (re, im)");
    const long b_in = so3_bandwidth(x_.size(0)), b_out = b_or(b_out_, b_in);
    const Tensor x = x_.contiguous();
    const auto lead = x.sizes().slice(1, x.dim() - 2);
    Tensor out = empty_like_shape(x, lead), keep;
    int nfeat;
    const float* bp = bias_ptr(bias, keep, nfeat);
    check(!bp || (!lead.empty() && lead.back() == nfeat), "so3_rifft_relu_integrate: one bias per feature");
    Ctx c(*this, x);
    S2C_CALL(so3_rifft_relu_integrate, cptr(x), ptr(out), lead_numel(lead), (int)b_in, (int)b_out, bp, nfeat, c.stream);
    return out;
  }

  struct S2Product { long nspec, nb, fi, fo, b; };
  static S2Product s2_product_dims(const Tensor& xs, const Tensor& ys) {
    check(xs.dim() == 4 && ys.dim() == 4 && xs.size(3) == 2 && ys.size(3) == 2, "s2 product: [l * m, ., ., complex] operands");
    S2Product d{xs.size(0), xs.size(1), xs.size(2), ys.size(2), 0};
    check(ys.size(0) == d.nspec && ys.size(1) == d.fi, "s2 product: operands do not match");
    d.b = s2_bandwidth(d.nspec);
    return d;
  }

  // `real`: the factors are spectra of real signals
  Tensor s2_conv_relu_so3_rfft(const Tensor& xs_, const Tensor& ys_, const OptTensor& bias, int64_t b_next, bool real) {
    prep(xs_); prep(ys_); prep(bias);
    const S2Product d = s2_product_dims(xs_, ys_);
    const Tensor xs = xs_.contiguous(), ys = ys_.contiguous();
    Tensor keep;
    int nfeat;
    const float* bp = bias_ptr(bias, keep, nfeat);
    check(!bp || nfeat == d.fo, "s2_conv_relu_so3_rfft: one bias per output feature");
    Tensor out = empty_like_shape(xs, {so3_nspec(b_next), d.nb, d.fo, 2});
    Ctx c(*this, xs);
    const Scratch ws(s2_conv_relu_so3_rfft_workspace_((int)d.nb, (int)d.fo, (int)d.b, (int)b_next), xs);
    if (real)
      S2C_CALL(s2_conv_real_relu_so3_rfft, cptr(xs), cptr(ys), ptr(out), (int)d.nb, (int)d.fi, (int)d.fo, (int)d.b, (int)b_next, bp, ws.p, ws.n, c.stream);
    else
      S2C_CALL(s2_conv_relu_so3_rfft_ws, cptr(xs), cptr(ys), ptr(out), (int)d.nb, (int)d.fi, (int)d.fo, (int)d.b, (int)b_next, bp, ws.p, ws.n, c.stream);
    return out;
  }

  Tensor so3_rifft_relu_rfft(const Tensor& x_, const OptTensor& bias, int64_t b_mid, int64_t b_next) {
    prep(x_);
    prep(bias);
    check(x_.dim() >= 2 && x_.size(-1) == 2, "so3_rifft_relu_rfft: the last axis holds (re, im)");
    const long b_in = so3_bandwidth(x_.size(0));
    const Tensor x = x_.contiguous();
    const auto lead = x.sizes().slice(1, x.dim() - 2);
    Tensor keep;
    int nfeat;
    const float* bp = bias_ptr(bias, keep, nfeat);
    check(!bp || (!lead.empty() && lead.back() == nfeat), "so3_rifft_relu_rfft: one bias per feature");
    Tensor out = empty_like_shape(x, spectrum_shape(so3_nspec(b_next), lead));
    Ctx c(*this, x);
    const long nb = lead_numel(lead);
    const Scratch ws(so3_relay_workspace_(nb, (int)b_in, (int)b_mid, (int)b_next), x);
    S2C_CALL(so3_rifft_relu_rfft_ws, cptr(x), ptr(out), nb, (int)b_in, (int)b_mid, (int)b_next, bp, nfeat, ws.p, ws.n, c.stream);
    return out;
  }

  Tensor s2_conv_synthesis(const Tensor& xs_, const Tensor& ys_, const OptTensor& bias, bool real) {
    prep(xs_); prep(ys_); prep(bias);
    const S2Product d = s2_product_dims(xs_, ys_);
    const Tensor xs = xs_.contiguous(), ys = ys_.contiguous();
    Tensor keep;
    int nfeat;
    const float* bp = bias_ptr(bias, keep, nfeat);
    check(!bp || nfeat == d.fo, "s2_conv_synthesis: one bias per output feature");
    const long n = 2 * d.b;
    Tensor out = empty_like_shape(xs, {d.nb, d.fo, n, n, n});
    Ctx c(*this, xs);
    const Scratch ws((real ? s2_conv_real_synthesis_workspace_ : s2_conv_synthesis_workspace_)((int)d.nb, (int)d.fo, (int)d.b), xs);
    if (real)
      S2C_CALL(s2_conv_real_synthesis, cptr(xs), cptr(ys), ptr(out), (int)d.nb, (int)d.fi, (int)d.fo, (int)d.b, bp, ws.p, ws.n, c.stream);
    else
      S2C_CALL(s2_conv_synthesis, cptr(xs), cptr(ys), ptr(out), (int)d.nb, (int)d.fi, (int)d.fo, (int)d.b, bp, ws.p, ws.n, c.stream);
    return out;
  }

  Tensor so3_ifft(const Tensor& x_, bool for_grad, std::optional<int64_t> b_out_) {
    prep(x_);
    check(x_.dim() >= 2 && x_.size(-1) == 2, "so3_ifft: the last axis holds (re, im)");
    const long b_in = so3_bandwidth(x_.size(0)), b_out = b_or(b_out_, b_in);
    const Tensor x = x_.contiguous();
    const auto lead = x.sizes().slice(1, x.dim() - 2);
    const long nb = lead_numel(lead);
    Tensor out = empty_like_shape(x, signal_shape(lead, 2 * b_out, 3, true));
    Ctx c(*this, x);
    const Scratch ws(so3_synthesis_workspace_(nb, b_in, b_out), x);
    S2C_CALL(so3_ifft, cptr(x), ptr(out), nb, (int)b_in, (int)b_out, (int)for_grad, ws.p, ws.n, c.stream);
    return out;
  }

  // -- S2 transforms --------------------------------------------------------------------------------
  Tensor s2_fft(const Tensor& x_, bool for_grad, std::optional<int64_t> b_out_, bool x_is_real) {
    prep(x_);
    const long d = x_.dim(), t = x_is_real ? 2 : 3;
    check(d >= t && (x_is_real || x_.size(-1) == 2), "s2_fft: signal axes");
    const long n = x_.size(d - t);
    check(n % 2 == 0 && n > 0 && x_.size(d - t + 1) == n, "S2 signal: 2b x 2b samples");
    const long b_in = n / 2, b_out = b_or(b_out_, b_in);
    check(b_out <= b_in, "s2_fft: b_out <= b_in");   // s2cnn/soft/s2_fft.py:24
    const Tensor x = x_.contiguous();
    const auto lead = x.sizes().slice(0, d - t);
    const long nb = lead_numel(lead);
    Tensor out = empty_like_shape(x, spectrum_shape(b_out * b_out, lead));
    Ctx c(*this, x);
    const Scratch ws(s2_fft_workspace_(nb, b_in, b_out), x);
    S2C_CALL(s2_fft, cptr(x), (int)x_is_real, ptr(out), nb, (int)b_in, (int)b_out, (int)for_grad, ws.p, ws.n, c.stream);
    return out;
  }

  Tensor s2_ifft(const Tensor& x_, bool for_grad, std::optional<int64_t> b_out_, bool out_is_real) {
    prep(x_);
    check(x_.dim() >= 2 && x_.size(-1) == 2, "s2_ifft: the last axis holds (re, im)");
    const long b_in = s2_bandwidth(x_.size(0)), b_out = b_or(b_out_, b_in);
    check(b_out >= b_in, "s2_ifft: b_out >= b_in");   // s2cnn/soft/s2_fft.py:71
    const Tensor x = x_.contiguous();
    const auto lead = x.sizes().slice(1, x.dim() - 2);
    const long nb = lead_numel(lead);
    Tensor out = empty_like_shape(x, signal_shape(lead, 2 * b_out, 2, !out_is_real));
    Ctx c(*this, x);
    const Scratch ws(s2_fft_workspace_(nb, b_in, b_out), x);
    S2C_CALL(s2_ifft, cptr(x), ptr(out), (int)out_is_real, nb, (int)b_in, (int)b_out, (int)for_grad, ws.p, ws.n, c.stream);
    return out;
  }

  // -- spectral products ----------------------------------------------------------------------------
  template <class F>
  Tensor mm(const char* name, F fn, const Tensor& a_, const Tensor& b_, at::IntArrayRef shape, long nl, long nb, long fi, long fo) {
    prep(a_);
    prep(b_);
    const Tensor a = a_.contiguous(), b = b_.contiguous();
    Tensor out = empty_like_shape(a, shape);
    Ctx c(*this, a);
    call(name, fn, cptr(a), cptr(b), ptr(out), (int)nl, (int)nb, (int)fi, (int)fo, c.stream);
    if (check_tc) check_tensor_core_status();
    return out;
  }
  // a gradient product: the parts of tiles shared by several thread blocks lie in a workspace
  template <class F, class W>
  Tensor mm_grad(const char* name, F fn, W workspace_bytes, const Tensor& a_, const Tensor& b_, at::IntArrayRef shape, long nl, long nb, long fi, long fo) {
    prep(a_);
    prep(b_);
    const Tensor a = a_.contiguous(), b = b_.contiguous();
    Tensor out = empty_like_shape(a, shape);
    Ctx c(*this, a);
    const Scratch ws(workspace_bytes((int)nl, (int)nb, (int)fi, (int)fo), a);
    call(name, fn, cptr(a), cptr(b), ptr(out), (int)nl, (int)nb, (int)fi, (int)fo, ws.p, ws.n, c.stream);
    if (check_tc) check_tensor_core_status();
    return out;
  }
  // Waits for the device and raises if a tensor-core product has given up on one of its bounded
  // barrier waits since the library was loaded (its output is then undefined).
  void check_tensor_core_status() const {
    const int rc = so3_mm_tc_status_();
    if (rc != 0)
      raise_s2c("s2cnn_b200: a tensor-core spectral product reported a barrier time-out (status " +
                std::to_string(rc) + "); its results are invalid");
  }
  Tensor so3_mm(const Tensor& x, const Tensor& y) {
    check(x.dim() == 4 && y.dim() == 4 && x.size(3) == 2 && y.size(3) == 2 && y.size(1) == x.size(2) && y.size(0) == x.size(0),
          "so3_mm: x [l * m * n, batch, f_in, 2] and y [l * m * n, f_in, f_out, 2]");
    const long nl = so3_bandwidth(x.size(0)), nb = x.size(1), fi = x.size(2), fo = y.size(2);
    return mm("s2c_so3_mm", so3_mm_, x, y, {so3_nspec(nl), nb, fo, 2}, nl, nb, fi, fo);
  }
  Tensor so3_mm_gradx(const Tensor& gz, const Tensor& y, int64_t nb, int64_t fi) {
    const long nl = so3_bandwidth(y.size(0)), fo = y.size(2);
    return mm_grad("s2c_so3_mm_gradx", so3_mm_gradx_ws_, so3_mm_gradx_workspace_, gz, y, {so3_nspec(nl), nb, fi, 2}, nl, nb, fi, fo);
  }
  Tensor so3_mm_grady(const Tensor& gz, const Tensor& x, int64_t fo) {
    const long nl = so3_bandwidth(x.size(0)), nb = x.size(1), fi = x.size(2);
    return mm_grad("s2c_so3_mm_grady", so3_mm_grady_ws_, so3_mm_grady_workspace_, gz, x, {so3_nspec(nl), fi, fo, 2}, nl, nb, fi, fo);
  }
  // products of spectra of real signals; op as in s2c_so3_mm_real
  Tensor mm_real(int op, const Tensor& u_, const Tensor& v_, at::IntArrayRef shape, long nl, long nb, long fi, long fo) {
    prep(u_);
    prep(v_);
    const Tensor u = u_.contiguous(), v = v_.contiguous();
    Tensor out = empty_like_shape(u, shape);
    Ctx c(*this, u);
    const Scratch ws(so3_mm_real_workspace_(op, (int)nl, (int)nb, (int)fi, (int)fo), u);
    S2C_CALL(so3_mm_real, op, cptr(u), cptr(v), ptr(out), (int)nl, (int)nb, (int)fi, (int)fo, ws.p, ws.n, c.stream);
    if (check_tc) check_tensor_core_status();
    return out;
  }
  Tensor so3_mm_real(const Tensor& x, const Tensor& y) {
    check(x.dim() == 4 && y.dim() == 4 && x.size(3) == 2 && y.size(3) == 2 && y.size(1) == x.size(2) && y.size(0) == x.size(0),
          "so3_mm: x [l * m * n, batch, f_in, 2] and y [l * m * n, f_in, f_out, 2]");
    const long nl = so3_bandwidth(x.size(0)), nb = x.size(1), fi = x.size(2), fo = y.size(2);
    return mm_real(0, x, y, {so3_nspec(nl), nb, fo, 2}, nl, nb, fi, fo);
  }
  Tensor so3_mm_real_gradx(const Tensor& gz, const Tensor& y, int64_t nb, int64_t fi) {
    const long nl = so3_bandwidth(y.size(0)), fo = y.size(2);
    return mm_real(1, gz, y, {so3_nspec(nl), nb, fi, 2}, nl, nb, fi, fo);
  }
  Tensor so3_mm_real_grady(const Tensor& gz, const Tensor& x, int64_t fo) {
    const long nl = so3_bandwidth(x.size(0)), nb = x.size(1), fi = x.size(2);
    return mm_real(2, gz, x, {so3_nspec(nl), fi, fo, 2}, nl, nb, fi, fo);
  }
  Tensor s2_mm(const Tensor& x, const Tensor& y) {
    const S2Product d = s2_product_dims(x, y);
    return mm("s2c_s2_mm", s2_mm_, x, y, {so3_nspec(d.b), d.nb, d.fo, 2}, d.b, d.nb, d.fi, d.fo);
  }
  Tensor s2_mm_gradx(const Tensor& gz, const Tensor& y, int64_t nb, int64_t fi, bool real) {
    const long nl = s2_bandwidth(y.size(0)), fo = y.size(2);
    return mm("s2c_s2_mm_gradx", real ? s2_mm_real_gradx_ : s2_mm_gradx_, gz, y, {nl * nl, nb, fi, 2}, nl, nb, fi, fo);
  }
  Tensor s2_mm_grady(const Tensor& gz, const Tensor& x, int64_t fo, bool real) {
    const long nl = s2_bandwidth(x.size(0)), nb = x.size(1), fi = x.size(2);
    return mm("s2c_s2_mm_grady", real ? s2_mm_real_grady_ : s2_mm_grady_, gz, x, {nl * nl, fi, fo, 2}, nl, nb, fi, fo);
  }

  // -- kernel-grid -> spectrum ----------------------------------------------------------------------
  // x [..., n_grid], F [n_grid, nspec, 2] -> [nspec, ..., 2]
  Tensor rft_forward(const Tensor& x_, const Tensor& F_) {
    prep(x_);
    prep(F_);
    const long ng = x_.size(-1), ns = F_.size(1);
    check(F_.size(0) == ng && F_.size(2) == 2, "rft_forward: F [n_grid, nspec, 2]");
    const Tensor x = x_.contiguous(), F = F_.contiguous();
    const auto lead = x.sizes().slice(0, x.dim() - 1);
    Tensor out = empty_like_shape(x, spectrum_shape(ns, lead));
    Ctx c(*this, x);
    S2C_CALL(rft_forward, cptr(x), cptr(F), ptr(out), (int)lead_numel(lead), (int)ng, (int)ns, c.stream);
    return out;
  }
  // the same product on the tensor cores: Ft [nspec, 2, n_grid]; CUDA build, even n_grid
  Tensor rft_forward_t(const Tensor& x_, const Tensor& Ft_) {
    prep(x_);
    prep(Ft_);
    const long ng = x_.size(-1), ns = Ft_.size(0);
    check(Ft_.size(2) == ng && Ft_.size(1) == 2, "rft_forward_t: Ft [nspec, 2, n_grid]");
    const Tensor x = x_.contiguous(), Ft = Ft_.contiguous();
    const auto lead = x.sizes().slice(0, x.dim() - 1);
    Tensor out = empty_like_shape(x, spectrum_shape(ns, lead));
    Ctx c(*this, x);
    S2C_CALL(rft_forward_t, cptr(x), cptr(Ft), ptr(out), (int)lead_numel(lead), (int)ng, (int)ns, c.stream);
    return out;
  }
  // rft of scale * x; Ft optional (the tensor cores want it)
  Tensor rft_forward_scaled(const Tensor& x_, const Tensor& F_, const OptTensor& Ft, double scale) {
    prep(x_);
    prep(F_);
    prep(Ft);
    const long ng = x_.size(-1), ns = F_.size(1);
    check(F_.size(0) == ng && F_.size(2) == 2 && F_.is_contiguous(), "rft_forward_scaled: F [n_grid, nspec, 2]");
    check(!Ft || (Ft->size(0) == ns && Ft->size(1) == 2 && Ft->size(2) == ng && Ft->is_contiguous()), "rft_forward_scaled: Ft [nspec, 2, n_grid]");
    const Tensor x = x_.contiguous();
    const auto lead = x.sizes().slice(0, x.dim() - 1);
    Tensor out = empty_like_shape(x, spectrum_shape(ns, lead));
    Ctx c(*this, x);
    S2C_CALL(rft_forward_scaled, cptr(x), cptr(F_), Ft ? cptr(*Ft) : nullptr, ptr(out), (int)lead_numel(lead), (int)ng, (int)ns, (float)scale, c.stream);
    return out;
  }
  // scale * F^T g: g [nspec, nf, 2], F [n_grid, nspec, 2] -> [nf, n_grid]
  Tensor rft_backward(const Tensor& g_, const Tensor& F_, double scale) {
    prep(g_);
    prep(F_);
    const long ns = g_.size(0), nf = g_.size(1), ng = F_.size(0);
    check(F_.size(1) == ns, "rft_backward: F [n_grid, nspec, 2]");
    const Tensor g = g_.contiguous(), F = F_.contiguous();
    Tensor out = empty_like_shape(g, {nf, ng});
    Ctx c(*this, g);
    const Scratch ws(rft_backward_workspace_((int)nf, (int)ng, (int)ns), g);
    S2C_CALL(rft_backward_scaled, cptr(g), cptr(F), ptr(out), (int)nf, (int)ng, (int)ns, (float)scale, ws.p, ws.n, c.stream);
    return out;
  }

  // -- integration ----------------------------------------------------------------------------------
  Tensor so3_integrate(const Tensor& x_, bool relu) {
    prep(x_);
    const long b = so3_side(x_, 3);
    const Tensor x = x_.contiguous();
    const auto lead = x.sizes().slice(0, x.dim() - 3);
    Tensor out = empty_like_shape(x, lead);
    Ctx c(*this, x);
    S2C_CALL(so3_integrate, cptr(x), ptr(out), lead_numel(lead), (int)b, (int)relu, c.stream);
    return out;
  }
  Tensor so3_integrate_backward(const Tensor& g_, int64_t b, const OptTensor& x_, bool relu) {
    prep(g_);
    prep(x_);
    const Tensor g = g_.contiguous();
    Tensor x;
    if (x_) x = x_->contiguous();
    Tensor out = empty_like_shape(g, signal_shape(g.sizes(), 2 * b, 3, false));
    Ctx c(*this, g);
    S2C_CALL(so3_integrate_backward, cptr(g), x.defined() ? cptr(x) : nullptr, ptr(out), (long)g.numel(), (int)b, (int)relu, c.stream);
    return out;
  }

  // -- rotation, projection -------------------------------------------------------------------------
  Tensor so3_rotate_spectrum(const Tensor& U, const Tensor& x_, int64_t b, bool adjoint) {
    prep(U);
    prep(x_);
    if (x_.dim() < 2 || x_.size(0) != so3_nspec(b) || x_.size(-1) != 2 || U.dim() != 2 || U.size(0) != so3_nspec(b) || U.size(1) != 2)
      raise(PyExc_ValueError, "so3_rotate_spectrum: bad shapes");
    const Tensor x = x_.contiguous();
    Tensor out = at::empty_like(x);
    Ctx c(*this, x);
    S2C_CALL(so3_rotate_spectrum, cptr(U), cptr(x), ptr(out), (int)b, lead_numel(x.sizes().slice(1, x.dim() - 2)), (int)adjoint, c.stream);
    return out;
  }

  // verts [nv, 3] float32, faces [nf, 3] int32, grid [nr, 3] float32 -> [3, nr] float32
  // (distance to the first hit, normal . ray, |normal x ray|; see include/s2cnn_b200.h)
  Tensor project_on_sphere(const Tensor& verts_, const Tensor& faces_, const Tensor& grid_) {
    prep(verts_);
    prep(grid_);
    if (faces_.scalar_type() != at::kInt || faces_.is_cuda() != is_cuda)
      raise(PyExc_TypeError, "faces must be an int32 tensor on the library's device");
    check(verts_.dim() == 2 && verts_.size(1) == 3 && faces_.dim() == 2 && faces_.size(1) == 3, "project_on_sphere: [n, 3] meshes");
    check(grid_.dim() == 2 && grid_.size(1) == 3, "project_on_sphere: grid [n, 3]");
    check(faces_.min().item<int>() >= 0 && faces_.max().item<int>() < verts_.size(0), "face index out of range");
    const Tensor verts = verts_.contiguous(), faces = faces_.contiguous(), grid = grid_.contiguous();
    Tensor out = empty_like_shape(verts, {3, grid.size(0)});
    Ctx c(*this, verts);
    S2C_CALL(project_on_sphere, cptr(verts), (int)verts.size(0), faces.const_data_ptr<int>(), (int)faces.size(0), cptr(grid), (int)grid.size(0), ptr(out), c.stream);
    return out;
  }
};

// ---- autograd rules -------------------------------------------------------------------------------
// The rules are the reference's: the transpose of a transform is the opposite transform with the other
// table weighting.  Where nothing asks for a gradient the op runs without a graph node.
template <class... T>
bool wants_grad(const T&... t) {
  return at::GradMode::is_enabled() && (t.requires_grad() || ...);
}
Ops* ops_of(AutogradContext* ctx) { return reinterpret_cast<Ops*>(ctx->saved_data["ops"].toInt()); }
void keep_ops(AutogradContext* ctx, int64_t ops) { ctx->saved_data["ops"] = ops; }
std::optional<int64_t> opt_b(int64_t b) { return b > 0 ? std::optional<int64_t>(b) : std::nullopt; }

// s2cnn/soft/s2_fft.py:226-236
struct S2FftReal : torch::autograd::Function<S2FftReal> {
  static Tensor forward(AutogradContext* ctx, int64_t ops, const Tensor& x, int64_t b_out) {
    keep_ops(ctx, ops);
    ctx->saved_data["b_in"] = x.size(-1) / 2;
    return reinterpret_cast<Ops*>(ops)->s2_fft(x, false, opt_b(b_out), true);
  }
  static tensor_list backward(AutogradContext* ctx, tensor_list g) {
    return {Variable(), ops_of(ctx)->s2_ifft(g[0], true, ctx->saved_data["b_in"].toInt(), true), Variable()};
  }
};
// s2cnn/soft/s2_fft.py:239-250
struct S2IfftReal : torch::autograd::Function<S2IfftReal> {
  static Tensor forward(AutogradContext* ctx, int64_t ops, const Tensor& x, int64_t b_out) {
    keep_ops(ctx, ops);
    ctx->saved_data["b_in"] = (int64_t)s2_bandwidth(x.size(0));
    return reinterpret_cast<Ops*>(ops)->s2_ifft(x, false, opt_b(b_out), true);
  }
  static tensor_list backward(AutogradContext* ctx, tensor_list g) {
    return {Variable(), ops_of(ctx)->s2_fft(g[0], true, ctx->saved_data["b_in"].toInt(), true), Variable()};
  }
};
// s2cnn/soft/so3_fft.py:446-456; with `relu` the transform of max(x, 0), the mask of its gradient
// applied inside the synthesis kernel
struct So3FftReal : torch::autograd::Function<So3FftReal> {
  static Tensor forward(AutogradContext* ctx, int64_t ops, const Tensor& x, int64_t b_out, bool relu) {
    keep_ops(ctx, ops);
    ctx->saved_data["b_in"] = x.size(-1) / 2;
    if (relu) ctx->save_for_backward({x});
    return reinterpret_cast<Ops*>(ops)->so3_rfft(x, false, opt_b(b_out), relu);
  }
  static tensor_list backward(AutogradContext* ctx, tensor_list g) {
    const auto saved = ctx->get_saved_variables();
    Tensor gx = saved.empty() ? ops_of(ctx)->so3_rifft(g[0], true, ctx->saved_data["b_in"].toInt(), std::nullopt)
                              : ops_of(ctx)->so3_rifft_relu_grad(g[0], saved[0]);
    return {Variable(), gx, Variable(), Variable()};
  }
};
// s2cnn/soft/so3_fft.py:459-469
struct So3IfftReal : torch::autograd::Function<So3IfftReal> {
  static Tensor forward(AutogradContext* ctx, int64_t ops, const Tensor& x, int64_t b_out) {
    keep_ops(ctx, ops);
    ctx->saved_data["b_in"] = (int64_t)so3_bandwidth(x.size(0));
    return reinterpret_cast<Ops*>(ops)->so3_rifft(x, false, opt_b(b_out), std::nullopt);
  }
  static tensor_list backward(AutogradContext* ctx, tensor_list g) {
    return {Variable(), ops_of(ctx)->so3_rfft(g[0], true, ctx->saved_data["b_in"].toInt(), false), Variable()};
  }
};

// Gradient of the bias that was added to every sample of a [batch, feature, ...] signal, and of the
// spectrum below it: for small bandwidths the sums are a by-product of the analysis kernel.
std::tuple<Tensor, Tensor> spectrum_and_bias_grad(Ops* o, const Tensor& g, bool want_spec, bool want_bias,
                                                  int64_t b, at::IntArrayRef bias_shape) {
  Tensor gs, gb;
  if (want_spec && want_bias && g.dim() == 5) {
    Tensor sums;
    std::tie(gs, sums) = o->so3_rfft_with_sums(g, true, b);
    gb = sums.sum(0).reshape(bias_shape);
  } else {
    if (want_spec) gs = o->so3_rfft(g, true, b, false);
    if (want_bias) gb = g.sum({0, 2, 3, 4}).reshape(bias_shape);
  }
  return {gs, gb};
}

// SO3_ifft_real followed by "+ bias" ([1, f_out, 1, 1, 1]), s2cnn/soft/so3_conv.py:55-56
struct So3IfftRealBias : torch::autograd::Function<So3IfftRealBias> {
  static Tensor forward(AutogradContext* ctx, int64_t ops, const Tensor& x, const Tensor& bias) {
    keep_ops(ctx, ops);
    ctx->saved_data["b_in"] = (int64_t)so3_bandwidth(x.size(0));
    ctx->saved_data["bias_shape"] = bias.sizes().vec();
    return reinterpret_cast<Ops*>(ops)->so3_rifft(x, false, std::nullopt, bias);
  }
  static tensor_list backward(AutogradContext* ctx, tensor_list g) {
    Tensor gx, gb;
    std::tie(gx, gb) = spectrum_and_bias_grad(ops_of(ctx), g[0].contiguous(), ctx->needs_input_grad(0), ctx->needs_input_grad(1),
                                              ctx->saved_data["b_in"].toInt(), ctx->saved_data["bias_shape"].toIntVector());
    return {Variable(), gx, gb};
  }
};
// s2_mm -> SO3_ifft_real -> + bias (s2cnn/soft/s2_conv.py:42-45) as one op; backward is the reference's
// chain: so3_rfft(for_grad) of the output gradient, then the grad-x / grad-y products
struct S2ProductSynthesis : torch::autograd::Function<S2ProductSynthesis> {
  static Tensor forward(AutogradContext* ctx, int64_t ops, const Tensor& x, const Tensor& y, const Tensor& bias) {
    keep_ops(ctx, ops);
    ctx->save_for_backward({x, y});
    ctx->saved_data["bias_shape"] = bias.sizes().vec();
    // (the full product, as in SpectralMm: a kernel spectrum is a mirror of itself but for single last bits)
    return reinterpret_cast<Ops*>(ops)->s2_conv_synthesis(x, y, bias, false);
  }
  static tensor_list backward(AutogradContext* ctx, tensor_list g) {
    const auto saved = ctx->get_saved_variables();
    const Tensor &x = saved[0], &y = saved[1];
    Ops* o = ops_of(ctx);
    Tensor gz, gx, gy, gb;
    const bool wx = ctx->needs_input_grad(0), wy = ctx->needs_input_grad(1);
    std::tie(gz, gb) = spectrum_and_bias_grad(o, g[0].contiguous(), wx || wy, ctx->needs_input_grad(2),
                                              s2_bandwidth(x.size(0)), ctx->saved_data["bias_shape"].toIntVector());
    if (wx) gx = o->s2_mm_gradx(gz, y, x.size(1), x.size(2), true);
    if (wy) gy = o->s2_mm_grady(gz, x, y.size(2), true);
    return {Variable(), gx, gy, gb};
  }
};
// s2cnn/so3_mm.py:95-122 and s2cnn/s2_mm.py:67-101
enum MmKind { kSo3Mm, kSo3MmReal, kS2Mm };
template <MmKind KIND>
struct SpectralMm : torch::autograd::Function<SpectralMm<KIND>> {
  static Tensor forward(AutogradContext* ctx, int64_t ops, const Tensor& x, const Tensor& y) {
    keep_ops(ctx, ops);
    ctx->save_for_backward({x, y});
    Ops* o = reinterpret_cast<Ops*>(ops);
    // The forward product of a recorded pass stays the full one: the half product rounds differently, and through the
    // ReLUs that follow a changed last bit of an activation moves a deep network's gradients by 1e-4 and more.
    return KIND == kS2Mm ? o->s2_mm(x, y) : o->so3_mm(x, y);
  }
  static tensor_list backward(AutogradContext* ctx, tensor_list g) {
    const auto saved = ctx->get_saved_variables();
    const Tensor &x = saved[0], &y = saved[1];
    Ops* o = ops_of(ctx);
    Tensor gx, gy;
    const Tensor gz = g[0].contiguous();
    const long nb = x.size(1), fi = x.size(2), fo = y.size(2);
    if (ctx->needs_input_grad(0))
      gx = KIND == kSo3Mm ? o->so3_mm_gradx(gz, y, nb, fi) : KIND == kSo3MmReal ? o->so3_mm_real_gradx(gz, y, nb, fi) : o->s2_mm_gradx(gz, y, nb, fi, false);
    if (ctx->needs_input_grad(1))
      gy = KIND == kSo3Mm ? o->so3_mm_grady(gz, x, fo) : KIND == kSo3MmReal ? o->so3_mm_real_grady(gz, x, fo) : o->s2_mm_grady(gz, x, fo, false);
    return {Variable(), gx, gy};
  }
};
// scale * kernel [..., n_grid] -> [nspec, ..., 2]: the einsum of s2cnn/s2_ft.py:22 and s2cnn/so3_ft.py:22,
// with the layers' constant scaling of the kernel
struct Rft : torch::autograd::Function<Rft> {
  static Tensor forward(AutogradContext* ctx, int64_t ops, const Tensor& x, const Tensor& F, const OptTensor& Ft, double scale) {
    keep_ops(ctx, ops);
    ctx->save_for_backward({F});
    ctx->saved_data["shape"] = x.sizes().vec();
    ctx->saved_data["scale"] = scale;
    return reinterpret_cast<Ops*>(ops)->rft_forward_scaled(x, F, Ft, scale);
  }
  static tensor_list backward(AutogradContext* ctx, tensor_list g) {
    const auto saved = ctx->get_saved_variables();
    const Tensor& F = saved[0];
    const Tensor gx = ops_of(ctx)->rft_backward(g[0].contiguous().view({F.size(1), -1, 2}), F, ctx->saved_data["scale"].toDouble());
    return {Variable(), gx.view(ctx->saved_data["shape"].toIntVector()), Variable(), Variable(), Variable()};
  }
};
// s2cnn/soft/so3_integrate.py:7-29, optionally of max(x, 0)
struct So3Integrate : torch::autograd::Function<So3Integrate> {
  static Tensor forward(AutogradContext* ctx, int64_t ops, const Tensor& x, bool relu) {
    keep_ops(ctx, ops);
    ctx->saved_data["b"] = x.size(-1) / 2;
    if (relu) ctx->save_for_backward({x});
    return reinterpret_cast<Ops*>(ops)->so3_integrate(x, relu);
  }
  static tensor_list backward(AutogradContext* ctx, tensor_list g) {
    const auto saved = ctx->get_saved_variables();
    const bool relu = !saved.empty();
    OptTensor x;
    if (relu) x = saved[0];
    return {Variable(), ops_of(ctx)->so3_integrate_backward(g[0], ctx->saved_data["b"].toInt(), x, relu), Variable()};
  }
};
// s2cnn/soft/so3_rotation.py:22-41: backward is the transposed product
struct RotateSpectrum : torch::autograd::Function<RotateSpectrum> {
  static Tensor forward(AutogradContext* ctx, int64_t ops, const Tensor& x, const Tensor& U, int64_t b) {
    keep_ops(ctx, ops);
    ctx->save_for_backward({U});
    ctx->saved_data["b"] = b;
    return reinterpret_cast<Ops*>(ops)->so3_rotate_spectrum(U, x, b, false);
  }
  static tensor_list backward(AutogradContext* ctx, tensor_list g) {
    const auto saved = ctx->get_saved_variables();
    return {Variable(), ops_of(ctx)->so3_rotate_spectrum(saved[0], g[0], ctx->saved_data["b"].toInt(), true), Variable(), Variable()};
  }
};

// Under torch.jit.trace an op runs as a Python autograd function (ops._traced), which the tracer records as one
// node that calls the op again.
template <class... A>
Tensor traced(Ops& o, const char* name, const A&... args) {
  pybind11::gil_scoped_acquire gil;
  const pybind11::handle fn(g_traced);
  return fn(pybind11::cast(&o, pybind11::return_value_policy::reference), name, args...).template cast<Tensor>();
}
#define S2C_TRACED(name, ...) \
  if (tracing()) return traced(o, name, __VA_ARGS__)

int64_t id(Ops& o) { return reinterpret_cast<int64_t>(&o); }
int64_t b_arg(const std::optional<int64_t>& b) { return b ? *b : 0; }

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  namespace py = pybind11;
  py::register_exception_translator([](std::exception_ptr p) {
    try {
      if (p) std::rethrow_exception(p);
    } catch (python_error& e) {
      e.restore();
    }
  });
  pybind11::class_<InsideTracedOp>(m, "InsideTracedOp")
      .def(pybind11::init<>())
      .def("__enter__", &InsideTracedOp::enter)
      .def("__exit__", &InsideTracedOp::exit);
  m.def("set_traced", [](py::object f) { g_traced = f.release().ptr(); });
  m.def("set_error_type", [](py::object t) { g_s2c_error = t.release().ptr(); });
  using namespace py::literals;
  const auto nogil = py::call_guard<py::gil_scoped_release>();
  const auto none = py::none();
  py::class_<Ops, std::unique_ptr<Ops, py::nodelete>>(m, "Ops")   // outlives every graph node that points to it
      .def(py::init<const std::string&, py::object, bool, bool>())
      .def("so3_rfft", &Ops::so3_rfft, "x"_a, "for_grad"_a = false, "b_out"_a = none, "relu"_a = false, nogil)
      .def("so3_rfft_with_sums", &Ops::so3_rfft_with_sums, "x"_a, "for_grad"_a = false, "b_out"_a = none, nogil)
      .def("so3_fft", &Ops::so3_fft, "x"_a, "for_grad"_a = false, "b_out"_a = none, nogil)
      .def("so3_rifft", &Ops::so3_rifft, "x"_a, "for_grad"_a = false, "b_out"_a = none, "bias"_a = none, nogil)
      .def("so3_rifft_relu_grad", &Ops::so3_rifft_relu_grad, "x"_a, "act"_a, nogil)
      .def("so3_rifft_relu_integrate", &Ops::so3_rifft_relu_integrate, "x"_a, "bias"_a = none, "b_out"_a = none, nogil)
      .def("s2_conv_relu_so3_rfft", &Ops::s2_conv_relu_so3_rfft, "xs"_a, "ys"_a, "bias"_a, "b_next"_a, "real"_a = false, nogil)
      .def("so3_rifft_relu_rfft", &Ops::so3_rifft_relu_rfft, "x"_a, "bias"_a, "b_mid"_a, "b_next"_a, nogil)
      .def("s2_conv_synthesis", &Ops::s2_conv_synthesis, "xs"_a, "ys"_a, "bias"_a = none, "real"_a = false, nogil)
      .def("so3_ifft", &Ops::so3_ifft, "x"_a, "for_grad"_a = false, "b_out"_a = none, nogil)
      .def("s2_fft", &Ops::s2_fft, "x"_a, "for_grad"_a = false, "b_out"_a = none, "x_is_real"_a = false, nogil)
      .def("s2_ifft", &Ops::s2_ifft, "x"_a, "for_grad"_a = false, "b_out"_a = none, "out_is_real"_a = false, nogil)
      .def("check_tensor_core_status", &Ops::check_tensor_core_status, nogil)
      .def("so3_mm", &Ops::so3_mm, "x"_a, "y"_a, nogil)
      .def("so3_mm_gradx", &Ops::so3_mm_gradx, "gz"_a, "y"_a, "nb"_a, "fi"_a, nogil)
      .def("so3_mm_grady", &Ops::so3_mm_grady, "gz"_a, "x"_a, "fo"_a, nogil)
      .def("so3_mm_real", &Ops::so3_mm_real, "x"_a, "y"_a, nogil)
      .def("so3_mm_real_gradx", &Ops::so3_mm_real_gradx, "gz"_a, "y"_a, "nb"_a, "fi"_a, nogil)
      .def("so3_mm_real_grady", &Ops::so3_mm_real_grady, "gz"_a, "x"_a, "fo"_a, nogil)
      .def("s2_mm", &Ops::s2_mm, "x"_a, "y"_a, nogil)
      .def("s2_mm_gradx", &Ops::s2_mm_gradx, "gz"_a, "y"_a, "nb"_a, "fi"_a, "real"_a = false, nogil)
      .def("s2_mm_grady", &Ops::s2_mm_grady, "gz"_a, "x"_a, "fo"_a, "real"_a = false, nogil)
      .def("rft_forward", &Ops::rft_forward, "x"_a, "F"_a, nogil)
      .def("rft_forward_t", &Ops::rft_forward_t, "x"_a, "Ft"_a, nogil)
      .def("rft_backward", &Ops::rft_backward, "g"_a, "F"_a, "scale"_a = 1.0, nogil)
      .def("so3_integrate", &Ops::so3_integrate, "x"_a, "relu"_a = false, nogil)
      .def("so3_integrate_backward", &Ops::so3_integrate_backward, "g"_a, "b"_a, "x"_a = none, "relu"_a = false, nogil)
      .def("so3_rotate_spectrum", &Ops::so3_rotate_spectrum, "U"_a, "x"_a, "b"_a, "adjoint"_a = false, nogil)
      .def("project_on_sphere", &Ops::project_on_sphere, "verts"_a, "faces"_a, "grid"_a, nogil)
      // -- the same ops with their autograd rules
      .def("ag_s2_fft_real", [](Ops& o, const Tensor& x, std::optional<int64_t> b) {
            S2C_TRACED("ag_s2_fft_real", x, b);
            return wants_grad(x) ? S2FftReal::apply(id(o), x, b_arg(b)) : o.s2_fft(x, false, b, true);
          }, "x"_a, "b_out"_a = none, nogil)
      .def("ag_s2_ifft_real", [](Ops& o, const Tensor& x, std::optional<int64_t> b) {
            S2C_TRACED("ag_s2_ifft_real", x, b);
            return wants_grad(x) ? S2IfftReal::apply(id(o), x, b_arg(b)) : o.s2_ifft(x, false, b, true);
          }, "x"_a, "b_out"_a = none, nogil)
      .def("ag_so3_fft_real", [](Ops& o, const Tensor& x, std::optional<int64_t> b, bool relu) {
            S2C_TRACED("ag_so3_fft_real", x, b, relu);
            return wants_grad(x) ? So3FftReal::apply(id(o), x, b_arg(b), relu) : o.so3_rfft(x, false, b, relu);
          }, "x"_a, "b_out"_a = none, "relu"_a = false, nogil)
      .def("ag_so3_ifft_real", [](Ops& o, const Tensor& x, std::optional<int64_t> b) {
            S2C_TRACED("ag_so3_ifft_real", x, b);
            return wants_grad(x) ? So3IfftReal::apply(id(o), x, b_arg(b)) : o.so3_rifft(x, false, b, std::nullopt);
          }, "x"_a, "b_out"_a = none, nogil)
      .def("ag_so3_ifft_real_bias", [](Ops& o, const Tensor& x, const Tensor& bias) {
            S2C_TRACED("ag_so3_ifft_real_bias", x, bias);
            return wants_grad(x, bias) ? So3IfftRealBias::apply(id(o), x, bias) : o.so3_rifft(x, false, std::nullopt, bias);
          }, "x"_a, "bias"_a, nogil)
      .def("ag_s2_product_synthesis", [](Ops& o, const Tensor& x, const Tensor& y, const Tensor& bias) {
            S2C_TRACED("ag_s2_product_synthesis", x, y, bias);
            return wants_grad(x, y, bias) ? S2ProductSynthesis::apply(id(o), x, y, bias) : o.s2_conv_synthesis(x, y, bias, true);
          }, "x"_a, "y"_a, "bias"_a, nogil)
      .def("ag_so3_mm", [](Ops& o, const Tensor& x, const Tensor& y) {
            S2C_TRACED("ag_so3_mm", x, y);
            return wants_grad(x, y) ? SpectralMm<kSo3Mm>::apply(id(o), x, y) : o.so3_mm(x, y);
          }, "x"_a, "y"_a, nogil)
      .def("ag_so3_mm_real", [](Ops& o, const Tensor& x, const Tensor& y) {
            S2C_TRACED("ag_so3_mm_real", x, y);
            return wants_grad(x, y) ? SpectralMm<kSo3MmReal>::apply(id(o), x, y) : o.so3_mm_real(x, y);
          }, "x"_a, "y"_a, nogil)
      .def("ag_s2_mm", [](Ops& o, const Tensor& x, const Tensor& y) {
            S2C_TRACED("ag_s2_mm", x, y);
            return wants_grad(x, y) ? SpectralMm<kS2Mm>::apply(id(o), x, y) : o.s2_mm(x, y);
          }, "x"_a, "y"_a, nogil)
      .def("ag_rft", [](Ops& o, const Tensor& x, const Tensor& F, const OptTensor& Ft, double scale) {
            S2C_TRACED("ag_rft", x, F, Ft, scale);
            return wants_grad(x) ? Rft::apply(id(o), x, F, Ft, scale) : o.rft_forward_scaled(x, F, Ft, scale);
          }, "x"_a, "F"_a, "Ft"_a = none, "scale"_a = 1.0, nogil)
      .def("ag_so3_integrate", [](Ops& o, const Tensor& x, bool relu) {
            S2C_TRACED("ag_so3_integrate", x, relu);
            return wants_grad(x) ? So3Integrate::apply(id(o), x, relu) : o.so3_integrate(x, relu);
          }, "x"_a, "relu"_a = false, nogil)
      .def("ag_rotate_spectrum", [](Ops& o, const Tensor& x, const Tensor& U, int64_t b) {
            S2C_TRACED("ag_rotate_spectrum", x, U, b);
            return wants_grad(x) ? RotateSpectrum::apply(id(o), x, U, b) : o.so3_rotate_spectrum(U, x, b, false);
          }, "x"_a, "U"_a, "b"_a, nogil);
}
