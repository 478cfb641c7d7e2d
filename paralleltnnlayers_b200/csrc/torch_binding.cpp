// CPython / torch binding of the hot operators: argument checks, output and workspace allocation, the C-ABI call and
// the autograd nodes of the layers, in one native call per operator.
//
// What bounds the small operators is the host: the same calls through ctypes took 22-26 us for a forward convolution
// (6 descriptors, tensor checks, torch.cuda.device and current_stream round trips, torch.empty), 80-98 us for the
// training step and 215-280 us for a layer's forward and backward under a Python autograd.Function, against 5-60 us on
// the GPU.  Only the operators a training or serving loop calls are here; the rest of ops.py stays on ctypes.
// The library itself (libb200cp.so) keeps no dependency on torch.
#include <Python.h>

#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/utils/pybind.h>

#include <array>
#include <string>
#include <vector>

#include "b200cp.h"

namespace {

using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::Variable;
using torch::autograd::variable_list;

PyObject* g_error_class = nullptr;  // paralleltnnlayers_b200._lib.B200CPError

// A failed status becomes the Python exception whichever thread it is raised on (backward runs on the engine's own).
[[noreturn]] void raise_status(int status) {
  std::string msg = b200cp_last_error_string();
  if (msg.empty()) msg = b200cp_status_string(status);
  pybind11::gil_scoped_acquire gil;
  PyObject* args = Py_BuildValue("(is)", status, msg.c_str());
  PyErr_SetObject(g_error_class ? g_error_class : PyExc_RuntimeError, args);
  Py_XDECREF(args);
  python_error e;
  e.persist();
  throw e;
}
inline void ok(int status) {
  if (C10_UNLIKELY(status != B200CP_OK)) raise_status(status);
}

// float32, CUDA, contiguous: the tensor itself where it already is
Tensor dev(const Tensor& t, const char* name) {
  TORCH_CHECK_TYPE(t.defined() && t.is_cuda() && t.scalar_type() == at::kFloat, name, " must be a float32 CUDA tensor");
  return t.is_contiguous() ? t : t.contiguous();
}
// The same, on the device of the call: the kernels read every operand by address.
Tensor dev(const Tensor& t, const char* name, const Tensor& input) {
  Tensor c = dev(t, name);
  TORCH_CHECK_VALUE(c.device() == input.device(), name, " is on ", c.device(), ", the input on ", input.device());
  return c;
}
// A tensor the kernels index by another operand's sizes
void check_size(const Tensor& t, const char* name, at::IntArrayRef size) {
  TORCH_CHECK_VALUE(t.numel() == c10::multiply_integers(size), name, " has ", t.numel(), " values where the shapes of the call give ",
                    size);
}
inline const float* cp(const Tensor& t) { return static_cast<const float*>(t.const_data_ptr()); }
inline float* mp(const Tensor& t) { return static_cast<float*>(t.mutable_data_ptr()); }
inline Tensor empty(at::IntArrayRef size, const Tensor& like) {
  return at::detail::empty_cuda(size, at::kFloat, like.device(), std::nullopt);
}
inline void* stream(const Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.device().index()).stream(); }
inline Tensor workspace(size_t bytes, const Tensor& like) {
  return empty({(int64_t)(std::max<size_t>(bytes, 4) / 4)}, like);
}
inline size_t ws_bytes(const Tensor& ws) { return (size_t)ws.numel() * 4; }
struct Scratch {   // a workspace that may be of no bytes (then nothing is allocated)
  Tensor t;
  void* ptr = nullptr;
  size_t bytes;
  Scratch(size_t n, const Tensor& like) : bytes(n) {
    if (n == 0) return;
    t = workspace(n, like);
    ptr = t.mutable_data_ptr();
  }
};

// ---- CP4 / three-factor CP ------------------------------------------------------------------------------------------
struct Conv {  // operands of a CP4 convolution, checked and contiguous
  Tensor in, FT, FC, FY, FX;
  b200cp_tensor_shape s;
  Conv(const Tensor& in_, const char* in_name, const Tensor& ft, const Tensor& fc, const Tensor& fy, const Tensor& fx,
       int64_t pad, bool in_is_upstream)
      : in(dev(in_, in_name)), FT(dev(ft, "FT", in)), FC(dev(fc, "FC", in)), FY(dev(fy, "FY", in)), FX(dev(fx, "FX", in)) {
    TORCH_CHECK_VALUE(in.dim() == 4, "input must be a rank-4 NCHW tensor");
    const Tensor* f[4] = {&FT, &FC, &FY, &FX};
    const char* nm[4] = {"FT", "FC", "FY", "FX"};
    for (int i = 0; i < 4; ++i)
      TORCH_CHECK_VALUE(f[i]->dim() == 2 && FT.dim() == 2 && f[i]->size(1) == FT.size(1), nm[i],
                        " must be [dim, rank] with the same rank as FT");
    const int64_t ch = in_is_upstream ? FT.size(0) : FC.size(0);
    TORCH_CHECK_VALUE(in.size(1) == ch, "input has ", in.size(1), " channels, the factor has ", ch);
    s = {(unsigned)in.size(0), (unsigned)in.size(2), (unsigned)in.size(3), (unsigned)pad, (unsigned)FT.size(0),
         (unsigned)FC.size(0), (unsigned)FY.size(0), (unsigned)FX.size(0), (unsigned)FT.size(1)};
  }
  Tensor out_like(unsigned channels) const { return empty({s.N, channels, s.H, s.W}, in); }
  // the rank planes, the upstream gradient and the input of a convolution of this shape
  void check_plane(const Tensor& P, const char* name) const { check_size(P, name, {s.N, s.Rank, s.H, s.W}); }
  void check_out(const Tensor& dU, const char* name) const { check_size(dU, name, {s.N, s.T, s.H, s.W}); }
  void check_in(const Tensor& X, const char* name) const { check_size(X, name, {s.N, s.C, s.H, s.W}); }
  void check_upstream(const Tensor& dU, const char* what) const {
    TORCH_CHECK_VALUE(dU.dim() == 4 && dU.size(0) == s.N && dU.size(1) == s.T && dU.size(2) == s.H && dU.size(3) == s.W,
                      what);
  }
};

using Grads4 = std::array<Tensor, 4>;
Grads4 split4(const Tensor& dK, const b200cp_tensor_shape& s) {
  const int64_t R = s.Rank, d[4] = {s.T, s.C, s.Y, s.X};
  Grads4 g;
  int64_t o = dK.storage_offset();
  for (int i = 0; i < 4; ++i) {
    g[i] = dK.as_strided({d[i], R}, {R, 1}, o);   // (one operator where narrow and view are three)
    o += d[i] * R;
  }
  return g;
}

Tensor cp4_forward(const Tensor& X, const Tensor& FT, const Tensor& FC, const Tensor& FY, const Tensor& FX, int64_t pad,
                   int flags, Tensor* plane = nullptr) {
  const Conv c(X, "Input", FT, FC, FY, FX, pad, false);
  const c10::cuda::OptionalCUDAGuard guard(c.in.device());
  Tensor U = c.out_like(c.s.T);
  if (plane) *plane = c.out_like(c.s.Rank);
  const Scratch ws(b200cp_cp4_fwd_workspace_bytes(&c.s, plane != nullptr, flags), c.in);
  ok(b200cp_cp4_fwd_ws(&c.s, cp(c.in), cp(c.FT), cp(c.FC), cp(c.FY), cp(c.FX), mp(U), plane ? mp(*plane) : nullptr, ws.ptr,
                       ws.bytes, stream(c.in), flags));
  return U;
}

Tensor cp4_backward_data(const Tensor& dU, const Tensor& FT, const Tensor& FC, const Tensor& FY, const Tensor& FX,
                         int64_t pad, int flags, Tensor* plane = nullptr) {
  const Conv c(dU, "Upstream", FT, FC, FY, FX, pad, true);
  const c10::cuda::OptionalCUDAGuard guard(c.in.device());
  Tensor dX = c.out_like(c.s.C);
  if (plane) *plane = c.out_like(c.s.Rank);
  const Scratch ws(b200cp_cp4_bwd_data_workspace_bytes(&c.s, plane != nullptr, flags), c.in);
  ok(b200cp_cp4_bwd_data_ws(&c.s, cp(c.in), cp(c.FT), cp(c.FC), cp(c.FY), cp(c.FX), mp(dX), plane ? mp(*plane) : nullptr,
                            ws.ptr, ws.bytes, stream(c.in), flags));
  return dX;
}

// dX and the packed factor gradients from the forward's rank plane
Tensor cp4_backward_saved(const Tensor& dU, const Tensor& In, const Tensor& P_, const Tensor& FT, const Tensor& FC,
                          const Tensor& FY, const Tensor& FX, int64_t pad, int flags, Tensor* dK, b200cp_tensor_shape* shape) {
  const Conv c(dU, "Upstream", FT, FC, FY, FX, pad, true);
  const Tensor P = dev(P_, "P", c.in), X = dev(In, "In", c.in);
  c.check_plane(P, "P");
  c.check_in(X, "In");
  const c10::cuda::OptionalCUDAGuard guard(c.in.device());
  const b200cp_tensor_shape& s = c.s;
  Tensor dX = c.out_like(s.C);
  *dK = empty({(int64_t)(s.T + s.C + s.Y + s.X) * s.Rank}, c.in);
  const Scratch ws(b200cp_cp4_bwd_saved_workspace_bytes(&s, flags), c.in);
  ok(b200cp_cp4_bwd_saved(&s, cp(X), cp(c.in), cp(P), cp(c.FT), cp(c.FC), cp(c.FY), cp(c.FX), mp(dX), mp(*dK), ws.ptr, ws.bytes,
                          stream(c.in), flags));
  *shape = s;
  return dX;
}

// the packed gradient buffer [dFT|dFC|dFY|dFX]
Tensor cp4_backward_filter(const Tensor& dU_, const Tensor& In, const Tensor& FT, const Tensor& FC, const Tensor& FY,
                           const Tensor& FX, int64_t pad, int flags, b200cp_tensor_shape* shape) {
  const Conv c(In, "In", FT, FC, FY, FX, pad, false);
  const Tensor dU = dev(dU_, "dLdO", c.in);
  c.check_upstream(dU, "dLdO must be [N,T,H,W]");
  const c10::cuda::OptionalCUDAGuard guard(c.in.device());
  const b200cp_tensor_shape& s = c.s;
  Tensor dK = empty({(int64_t)(s.T + s.C + s.Y + s.X) * s.Rank}, c.in);
  Tensor ws = workspace(b200cp_cp4_bwd_filter_workspace_bytes(&s, flags), c.in);
  ok(b200cp_cp4_bwd_filter(&s, cp(c.in), cp(dU), cp(c.FT), cp(c.FC), cp(c.FY), cp(c.FX), mp(dK), mp(ws), ws_bytes(ws),
                           stream(c.in), flags));
  *shape = s;
  return dK;
}

Tensor cp4_backward_filter_saved(const Tensor& dU_, const Tensor& In, const Tensor& P_, const Tensor& Q_, const Tensor& FT,
                                 const Tensor& FC, const Tensor& FY, const Tensor& FX, int64_t pad, int flags,
                                 b200cp_tensor_shape* shape) {
  const Conv c(In, "In", FT, FC, FY, FX, pad, false);
  const Tensor dU = dev(dU_, "dLdO", c.in), P = dev(P_, "P", c.in), Q = dev(Q_, "Q", c.in);
  c.check_out(dU, "dLdO");
  c.check_plane(P, "P");
  c.check_plane(Q, "Q");
  const c10::cuda::OptionalCUDAGuard guard(c.in.device());
  const b200cp_tensor_shape& s = c.s;
  Tensor dK = empty({(int64_t)(s.T + s.C + s.Y + s.X) * s.Rank}, c.in);
  Tensor ws = workspace(b200cp_cp4_bwd_filter_saved_workspace_bytes(&s, flags), c.in);
  ok(b200cp_cp4_bwd_filter_saved(&s, cp(c.in), cp(dU), cp(P), cp(Q), cp(c.FY), cp(c.FX), mp(dK), mp(ws), ws_bytes(ws),
                                 stream(c.in), flags));
  *shape = s;
  return dK;
}

struct Conv3 {
  Tensor in, KT, KC_in, KC;
  b200cp_tensor_shape s;
  Conv3(const Tensor& in_, const char* in_name, const Tensor& kt, const Tensor& kcin, const Tensor& kc, int64_t pad,
        bool in_is_upstream)
      : in(dev(in_, in_name)), KT(dev(kt, "KT", in)), KC_in(dev(kcin, "KCin", in)), KC(dev(kc, "KC", in)) {
    TORCH_CHECK_VALUE(in.dim() == 4 && KT.dim() == 2 && KC_in.dim() == 2 && KC.dim() == 3,
                      "expected input [N,ch,H,W], KT [T,R], KCin [C,R], KC [Y,X,R]");
    const int64_t R = KT.size(1);
    TORCH_CHECK_VALUE(KC_in.size(1) == R && KC.size(2) == R, "all factors must have the same rank");
    TORCH_CHECK_VALUE(in.size(1) == (in_is_upstream ? KT.size(0) : KC_in.size(0)),
                      "channel count of the input does not match the factor");
    s = {(unsigned)in.size(0), (unsigned)in.size(2), (unsigned)in.size(3), (unsigned)pad, (unsigned)KT.size(0),
         (unsigned)KC_in.size(0), (unsigned)KC.size(0), (unsigned)KC.size(1), (unsigned)R};
  }
};

Tensor cp3_forward(const Tensor& X, const Tensor& KT, const Tensor& KCin, const Tensor& KC, int64_t pad, int flags,
                   Tensor* plane = nullptr) {
  const Conv3 c(X, "Input", KT, KCin, KC, pad, false);
  const c10::cuda::OptionalCUDAGuard guard(c.in.device());
  Tensor U = empty({c.s.N, c.s.T, c.s.H, c.s.W}, c.in);
  if (plane) *plane = empty({c.s.N, c.s.Rank, c.s.H, c.s.W}, c.in);
  const Scratch ws(b200cp_cp3_fwd_workspace_bytes(&c.s, plane != nullptr, flags), c.in);
  ok(b200cp_cp3_fwd_ws(&c.s, cp(c.in), cp(c.KT), cp(c.KC_in), cp(c.KC), mp(U), plane ? mp(*plane) : nullptr, ws.ptr, ws.bytes,
                       stream(c.in), flags));
  return U;
}

Tensor cp3_backward_data(const Tensor& dU, const Tensor& KT, const Tensor& KCin, const Tensor& KC, int64_t pad, int flags) {
  const Conv3 c(dU, "Upstream", KT, KCin, KC, pad, true);
  const c10::cuda::OptionalCUDAGuard guard(c.in.device());
  Tensor dX = empty({c.s.N, c.s.C, c.s.H, c.s.W}, c.in);
  const Scratch ws(b200cp_cp3_bwd_data_workspace_bytes(&c.s, flags), c.in);
  ok(b200cp_cp3_bwd_data_ws(&c.s, cp(c.in), cp(c.KT), cp(c.KC_in), cp(c.KC), mp(dX), ws.ptr, ws.bytes, stream(c.in), flags));
  return dX;
}

std::array<Tensor, 3> split3(const Tensor& dK, const b200cp_tensor_shape& s) {
  const int64_t R = s.Rank, nT = s.T * R, nC = s.C * R, o = dK.storage_offset();
  return {dK.as_strided({s.T, R}, {R, 1}, o), dK.as_strided({s.C, R}, {R, 1}, o + nT),
          dK.as_strided({s.Y, s.X, R}, {s.X * R, R, 1}, o + nT + nC)};
}

// dX (where it is wanted) and the factor gradients from the forward's rank plane
Tensor cp3_backward_saved(const Tensor& dU, const Tensor& In, const Tensor& P_, const Tensor& KT, const Tensor& KCin,
                          const Tensor& KC, int64_t pad, int flags, bool need_dx, std::array<Tensor, 3>* grads) {
  const Conv3 c(dU, "Upstream", KT, KCin, KC, pad, true);
  const b200cp_tensor_shape& s = c.s;
  const Tensor P = dev(P_, "P", c.in), X = dev(In, "In", c.in);
  check_size(P, "P", {s.N, s.Rank, s.H, s.W});
  check_size(X, "In", {s.N, s.C, s.H, s.W});
  const c10::cuda::OptionalCUDAGuard guard(c.in.device());
  Tensor dX = need_dx ? empty({s.N, s.C, s.H, s.W}, c.in) : Tensor();
  Tensor dK = empty({(int64_t)(s.T + s.C + s.Y * s.X) * s.Rank}, c.in);
  const Scratch ws(b200cp_cp3_bwd_saved_workspace_bytes(&s, flags), c.in);
  ok(b200cp_cp3_bwd_saved(&s, cp(X), cp(c.in), cp(P), cp(c.KT), cp(c.KC_in), cp(c.KC), need_dx ? mp(dX) : nullptr, mp(dK), ws.ptr, ws.bytes,
                          stream(c.in), flags));
  *grads = split3(dK, s);
  return dX;
}

std::array<Tensor, 3> cp3_backward_filter(const Tensor& dU_, const Tensor& In, const Tensor& KT, const Tensor& KCin,
                                          const Tensor& KC, int64_t pad, int flags) {
  const Conv3 c(In, "In", KT, KCin, KC, pad, false);
  const b200cp_tensor_shape& s = c.s;
  const Tensor dU = dev(dU_, "dLdO", c.in);
  check_size(dU, "dLdO", {s.N, s.T, s.H, s.W});
  const c10::cuda::OptionalCUDAGuard guard(c.in.device());
  Tensor dK = empty({(int64_t)(s.T + s.C + s.Y * s.X) * s.Rank}, c.in);
  Tensor ws = workspace(b200cp_cp3_bwd_filter_workspace_bytes(&s, flags), c.in);
  ok(b200cp_cp3_bwd_filter(&s, cp(c.in), cp(dU), cp(c.KT), cp(c.KC_in), cp(c.KC), mp(dK), mp(ws), ws_bytes(ws),
                           stream(c.in), flags));
  return split3(dK, s);
}

// The default path of these layers takes the fastest product; a caller who names a path keeps to FFMA.
int product_flags(int flags) { return (flags & B200CP_PATH_MASK) == B200CP_PATH_AUTO ? flags | B200CP_TENSOR_PRODUCTS : flags; }

// ---- reshaped-CP conv and CP dense ------------------------------------------------------------------------------------
struct Modes {
  std::vector<Tensor> F;
  int order = 0, R = 0;
  std::vector<int> a, b;
  std::vector<const float*> ptr;
  int64_t na = 1, nb = 1;
  Modes(at::TensorList f, const char* what, const Tensor& input) {
    order = (int)f.size();
    TORCH_CHECK_VALUE(order >= 1, what, ": no kernels given");
    for (int k = 0; k < order; ++k) {
      F.push_back(dev(f[k], ("kernel" + std::to_string(k)).c_str(), input));
      const Tensor& t = F.back();
      TORCH_CHECK_VALUE(t.dim() == 3 && t.size(2) == F[0].size(2), what, ": kernel ", k,
                        " must be [in, out, rank] with a common rank");
      a.push_back((int)t.size(0));
      b.push_back((int)t.size(1));
      na *= t.size(0);
      nb *= t.size(1);
      ptr.push_back(cp(t));
    }
    R = (int)F[0].size(2);
  }
  Tensor core(const Tensor& KC_, const Tensor& input) const {   // the spatial core of a convolution with these modes
    const Tensor KC = dev(KC_, "kernelc", input);
    TORCH_CHECK_VALUE(KC.dim() == 3 && KC.size(2) == R, "kernelc must be [FH, FW, rank]");
    return KC;
  }
};

Tensor rcp_forward(const Tensor& U_, at::TensorList A, const Tensor& KC_, int flags) {
  flags = product_flags(flags);
  const Tensor U = dev(U_, "input");
  const Modes m(A, "conv2d_rcp_fused_nchw", U);
  const Tensor KC = m.core(KC_, U);
  const int64_t nd = U.dim();
  const bool folded = nd == 4;
  if (!folded) {
    bool match = nd == m.order + 3;
    for (int k = 0; match && k < m.order; ++k) match = U.size(1 + k) == m.a[k];
    TORCH_CHECK_VALUE(match, "input modes do not match the kernels");
  }
  const int64_t N = U.size(0), H = U.size(nd - 2), W = U.size(nd - 1);
  TORCH_CHECK_VALUE(U.numel() == N * m.na * H * W, "input channel count does not match the kernels");
  const c10::cuda::OptionalCUDAGuard guard(U.device());
  Tensor V = empty({N, m.nb, H, W}, U);
  const int FH = (int)KC.size(0), FW = (int)KC.size(1);
  Tensor ws = workspace(b200cp_rcp_fwd_workspace_bytes((int)N, (int)H, (int)W, m.order, m.a.data(), m.b.data(), m.R, FH, FW,
                                                       flags), U);
  ok(b200cp_rcp_fwd_ws((int)N, (int)H, (int)W, m.order, m.a.data(), m.b.data(), m.R, FH, FW, cp(U), m.ptr.data(), cp(KC),
                       mp(V), mp(ws), ws_bytes(ws), stream(U), flags));
  if (folded) return V;
  std::vector<int64_t> shape{N};
  for (int t : m.b) shape.push_back(t);
  shape.push_back(H);
  shape.push_back(W);
  return V.view(shape);
}

struct FactorGrads {
  Tensor dx, ds;
  std::vector<Tensor> df;
};

FactorGrads rcp_backward(const Tensor& U_, const Tensor& dV_, at::TensorList A, const Tensor& KC_, int flags, bool need_dx,
                         bool need_dw) {
  flags = product_flags(flags);
  const Tensor U = dev(U_, "input"), dV = dev(dV_, "dV", U);
  const Modes m(A, "rcp_conv2d_backward", U);
  const Tensor KC = m.core(KC_, U);
  const int64_t nd = U.dim();
  TORCH_CHECK_VALUE(nd >= 2, "input must be [N, S0, .., H, W]");
  const int64_t N = U.size(0), H = U.size(nd - 2), W = U.size(nd - 1);
  check_size(U, "input", {N, m.na, H, W});
  check_size(dV, "dV", {N, m.nb, H, W});
  const c10::cuda::OptionalCUDAGuard guard(U.device());
  FactorGrads g;
  std::vector<float*> dp;
  if (need_dx) g.dx = empty(U.sizes(), U);
  if (need_dw) {
    for (const Tensor& f : m.F) {
      g.df.push_back(empty(f.sizes(), U));
      dp.push_back(mp(g.df.back()));
    }
    g.ds = empty(KC.sizes(), U);
  }
  const int FH = (int)KC.size(0), FW = (int)KC.size(1);
  Tensor ws = workspace(b200cp_rcp_bwd_workspace_bytes((int)N, (int)H, (int)W, m.order, m.a.data(), m.b.data(), m.R, FH, FW,
                                                       flags), U);
  ok(b200cp_rcp_bwd((int)N, (int)H, (int)W, m.order, m.a.data(), m.b.data(), m.R, FH, FW, cp(U), cp(dV), m.ptr.data(),
                    cp(KC), need_dx ? mp(g.dx) : nullptr, need_dw ? dp.data() : nullptr, need_dw ? mp(g.ds) : nullptr,
                    mp(ws), ws_bytes(ws), stream(U), flags));
  return g;
}

Tensor dense_forward(const Tensor& U_, at::TensorList F, int flags) {
  flags = product_flags(flags);
  const Tensor U = dev(U_, "input");
  const Modes m(F, "dense_cp", U);
  const int64_t B = U.size(0);
  TORCH_CHECK_VALUE(U.numel() == B * m.na, "input size does not match the kernels");
  const c10::cuda::OptionalCUDAGuard guard(U.device());
  Tensor Y = empty({B, m.nb}, U);
  Tensor ws = workspace(b200cp_dense_fwd_workspace_bytes((int)B, m.order, m.a.data(), m.b.data(), m.R, flags), U);
  ok(b200cp_dense_fwd_ws((int)B, m.order, m.a.data(), m.b.data(), m.R, cp(U), m.ptr.data(), mp(Y), mp(ws), ws_bytes(ws),
                         stream(U), flags));
  if (U.dim() == 2) return Y;
  std::vector<int64_t> shape{B};
  for (int o : m.b) shape.push_back(o);
  return Y.view(shape);
}

FactorGrads dense_backward(const Tensor& U_, const Tensor& dV_, at::TensorList F, int flags, bool need_dx, bool need_dw) {
  flags = product_flags(flags);
  const Tensor U = dev(U_, "input"), dV = dev(dV_, "dV", U);
  const Modes m(F, "dense_cp_backward", U);
  const int B = (int)U.size(0);
  check_size(U, "input", {B, m.na});
  check_size(dV, "dV", {B, m.nb});
  const c10::cuda::OptionalCUDAGuard guard(U.device());
  FactorGrads g;
  std::vector<float*> dp;
  if (need_dx) g.dx = empty(U.sizes(), U);
  if (need_dw)
    for (const Tensor& f : m.F) {
      g.df.push_back(empty(f.sizes(), U));
      dp.push_back(mp(g.df.back()));
    }
  Tensor ws = workspace(b200cp_dense_bwd_workspace_bytes(B, m.order, m.a.data(), m.b.data(), m.R, flags), U);
  ok(b200cp_dense_bwd(B, m.order, m.a.data(), m.b.data(), m.R, cp(U), cp(dV), m.ptr.data(), need_dx ? mp(g.dx) : nullptr,
                      need_dw ? dp.data() : nullptr, mp(ws), ws_bytes(ws), stream(U), flags));
  return g;
}

// ---- autograd nodes -------------------------------------------------------------------------------------------------------
// `grad`: gradients are recorded where the node is applied (inside a forward the mode is always off; the factors of a
// module require a gradient under no_grad too, where a rank plane would be written and dropped)
struct CP4Node : torch::autograd::Function<CP4Node> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& FT, const Tensor& FC, const Tensor& FY,
                        const Tensor& FX, int64_t pad, int64_t flags, bool grad) {
    ctx->saved_data["pad"] = pad;
    ctx->saved_data["flags"] = flags;
    // with 3x3 filters the forward keeps its rank plane for the factor gradients (a quarter of x at C = 4R)
    bool shared = false;
    if (grad && (FT.requires_grad() || FC.requires_grad() || FY.requires_grad() || FX.requires_grad()) && x.dim() == 4) {
      const Conv c(x, "Input", FT, FC, FY, FX, pad, false);
      shared = b200cp_cp4_shares_planes(&c.s, (int)flags) != 0;
    }
    if (shared) {
      Tensor P;
      Tensor y = cp4_forward(x, FT, FC, FY, FX, pad, (int)flags, &P);
      ctx->save_for_backward({x, FT, FC, FY, FX, P});
      return y;
    }
    ctx->save_for_backward({x, FT, FC, FY, FX});
    return cp4_forward(x, FT, FC, FY, FX, pad, (int)flags);
  }
  static variable_list backward(AutogradContext* ctx, const variable_list& grads) {
    const variable_list v = ctx->get_saved_variables();
    const int64_t pad = ctx->saved_data["pad"].toInt();
    const int flags = (int)ctx->saved_data["flags"].toInt();
    const Tensor dy = grads[0].contiguous();
    const Tensor &x = v[0], &FT = v[1], &FC = v[2], &FY = v[3], &FX = v[4];
    b200cp_tensor_shape s;
    variable_list out(8);
    if (v.size() == 6) {
      Tensor dK;
      Tensor dx = cp4_backward_saved(dy, x, v[5], FT, FC, FY, FX, pad, flags, &dK, &s);
      const Grads4 g = split4(dK, s);
      if (ctx->needs_input_grad(0)) out[0] = dx;
      for (int i = 0; i < 4; ++i) out[1 + i] = g[i];
      return out;
    }
    if (ctx->needs_input_grad(0)) out[0] = cp4_backward_data(dy, FT, FC, FY, FX, pad, flags);
    if (ctx->needs_input_grad(1) || ctx->needs_input_grad(2) || ctx->needs_input_grad(3) || ctx->needs_input_grad(4)) {
      const Grads4 g = split4(cp4_backward_filter(dy, x, FT, FC, FY, FX, pad, flags, &s), s);
      for (int i = 0; i < 4; ++i) out[1 + i] = g[i];
    }
    return out;
  }
};

struct CP3Node : torch::autograd::Function<CP3Node> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& KT, const Tensor& KCin, const Tensor& KC,
                        int64_t pad, bool grad) {
    ctx->saved_data["pad"] = pad;
    // where the gradients are formed from whole rank planes the forward keeps its own
    bool shared = false;
    if (grad && (KT.requires_grad() || KCin.requires_grad() || KC.requires_grad()) && x.dim() == 4) {
      const Conv3 c(x, "Input", KT, KCin, KC, pad, false);
      shared = b200cp_cp3_shares_planes(&c.s, 0) != 0;
    }
    if (shared) {
      Tensor P;
      Tensor y = cp3_forward(x, KT, KCin, KC, pad, 0, &P);
      ctx->save_for_backward({x, KT, KCin, KC, P});
      return y;
    }
    ctx->save_for_backward({x, KT, KCin, KC});
    return cp3_forward(x, KT, KCin, KC, pad, 0);
  }
  static variable_list backward(AutogradContext* ctx, const variable_list& grads) {
    const variable_list v = ctx->get_saved_variables();
    const int64_t pad = ctx->saved_data["pad"].toInt();
    const Tensor dy = grads[0].contiguous();
    variable_list out(6);
    const bool need_dw = ctx->needs_input_grad(1) || ctx->needs_input_grad(2) || ctx->needs_input_grad(3);
    if (v.size() == 5 && need_dw) {
      std::array<Tensor, 3> g;
      out[0] = cp3_backward_saved(dy, v[0], v[4], v[1], v[2], v[3], pad, 0, ctx->needs_input_grad(0), &g);
      for (int i = 0; i < 3; ++i) out[1 + i] = g[i];
      return out;
    }
    if (ctx->needs_input_grad(0)) out[0] = cp3_backward_data(dy, v[1], v[2], v[3], pad, 0);
    if (need_dw) {
      const std::array<Tensor, 3> g = cp3_backward_filter(dy, v[0], v[1], v[2], v[3], pad, 0);
      for (int i = 0; i < 3; ++i) out[1 + i] = g[i];
    }
    return out;
  }
};

struct RCPNode : torch::autograd::Function<RCPNode> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& KC, at::TensorList A) {
    variable_list save{x, KC};
    save.insert(save.end(), A.begin(), A.end());
    ctx->save_for_backward(std::move(save));
    return rcp_forward(x, A, KC, 0);
  }
  static variable_list backward(AutogradContext* ctx, const variable_list& grads) {
    const variable_list v = ctx->get_saved_variables();
    const Tensor& x = v[0];
    const int64_t nd = x.dim();
    const Tensor dy = grads[0].contiguous().view({x.size(0), -1, x.size(nd - 2), x.size(nd - 1)});
    FactorGrads g = rcp_backward(x, dy, at::TensorList(v).slice(2), v[1], 0, true, true);
    variable_list out{g.dx, g.ds};
    out.insert(out.end(), g.df.begin(), g.df.end());
    return out;
  }
};

struct DenseNode : torch::autograd::Function<DenseNode> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, at::TensorList F) {
    variable_list save{x};
    save.insert(save.end(), F.begin(), F.end());
    ctx->save_for_backward(std::move(save));
    return dense_forward(x, F, 0);
  }
  static variable_list backward(AutogradContext* ctx, const variable_list& grads) {
    const variable_list v = ctx->get_saved_variables();
    const Tensor& x = v[0];
    const Tensor dy = grads[0].contiguous().reshape({x.size(0), -1});
    FactorGrads g = dense_backward(x.dim() == 2 ? x : x.reshape({x.size(0), -1}), dy, at::TensorList(v).slice(1), 0, true, true);
    variable_list out{x.dim() == 2 ? g.dx : g.dx.view(x.sizes())};
    out.insert(out.end(), g.df.begin(), g.df.end());
    return out;
  }
};

// ---- Python surface: positional arguments only (ops.py keeps the names and defaults) -----------------------------------
const Tensor& tensor_arg(PyObject* o, const char* name) {
  TORCH_CHECK_TYPE(THPVariable_Check(o), name, " must be a float32 CUDA tensor");
  return THPVariable_Unpack(o);
}
int64_t int_arg(PyObject* o) {
  const long long v = PyLong_AsLongLong(o);
  if (v == -1 && PyErr_Occurred()) throw python_error();
  return v;
}
std::vector<Tensor> tensor_args(PyObject* const* a, Py_ssize_t n) {
  std::vector<Tensor> v;
  v.reserve(n);
  for (Py_ssize_t i = 0; i < n; ++i) v.push_back(tensor_arg(a[i], ("kernel" + std::to_string(i)).c_str()));
  return v;
}
void count_args(Py_ssize_t n, Py_ssize_t want) { TORCH_CHECK_TYPE(n == want, "expected ", want, " arguments, got ", n); }
PyObject* wrap(const Tensor& t) {
  if (!t.defined()) Py_RETURN_NONE;
  return THPVariable_Wrap(t);
}
template <size_t K>
PyObject* wrap_tuple(const std::array<Tensor, K>& ts) {
  PyObject* r = PyTuple_New(K);
  if (!r) throw python_error();
  for (size_t i = 0; i < K; ++i) PyTuple_SET_ITEM(r, i, wrap(ts[i]));
  return r;
}
PyObject* wrap_list(const std::vector<Tensor>& ts) {
  PyObject* r = PyList_New((Py_ssize_t)ts.size());
  if (!r) throw python_error();
  for (size_t i = 0; i < ts.size(); ++i) PyList_SET_ITEM(r, (Py_ssize_t)i, wrap(ts[i]));
  return r;
}
// the GIL is given up while the operator runs: a launch may block on a full queue
template <typename Fn>
auto unlocked(Fn&& fn) {
  pybind11::gil_scoped_release nogil;
  return fn();
}

#define PYFN(name) PyObject* name(PyObject*, PyObject* const* a, Py_ssize_t n)

PYFN(py_cp4_forward) {
  HANDLE_TH_ERRORS
  count_args(n, 7);
  const Tensor &x = tensor_arg(a[0], "Input"), &ft = tensor_arg(a[1], "FT"), &fc = tensor_arg(a[2], "FC"),
               &fy = tensor_arg(a[3], "FY"), &fx = tensor_arg(a[4], "FX");
  const int64_t pad = int_arg(a[5]), flags = int_arg(a[6]);
  return wrap(unlocked([&] { return cp4_forward(x, ft, fc, fy, fx, pad, (int)flags); }));
  END_HANDLE_TH_ERRORS
}
PYFN(py_cp4_forward_save) {
  HANDLE_TH_ERRORS
  count_args(n, 7);
  const Tensor &x = tensor_arg(a[0], "Input"), &ft = tensor_arg(a[1], "FT"), &fc = tensor_arg(a[2], "FC"),
               &fy = tensor_arg(a[3], "FY"), &fx = tensor_arg(a[4], "FX");
  const int64_t pad = int_arg(a[5]), flags = int_arg(a[6]);
  std::array<Tensor, 2> r;
  unlocked([&] { r[0] = cp4_forward(x, ft, fc, fy, fx, pad, (int)flags, &r[1]); });
  return wrap_tuple(r);
  END_HANDLE_TH_ERRORS
}
PYFN(py_cp4_backward_data) {
  HANDLE_TH_ERRORS
  count_args(n, 7);
  const Tensor &x = tensor_arg(a[0], "Upstream"), &ft = tensor_arg(a[1], "FT"), &fc = tensor_arg(a[2], "FC"),
               &fy = tensor_arg(a[3], "FY"), &fx = tensor_arg(a[4], "FX");
  const int64_t pad = int_arg(a[5]), flags = int_arg(a[6]);
  return wrap(unlocked([&] { return cp4_backward_data(x, ft, fc, fy, fx, pad, (int)flags); }));
  END_HANDLE_TH_ERRORS
}
PYFN(py_cp4_backward_data_save) {
  HANDLE_TH_ERRORS
  count_args(n, 7);
  const Tensor &x = tensor_arg(a[0], "Upstream"), &ft = tensor_arg(a[1], "FT"), &fc = tensor_arg(a[2], "FC"),
               &fy = tensor_arg(a[3], "FY"), &fx = tensor_arg(a[4], "FX");
  const int64_t pad = int_arg(a[5]), flags = int_arg(a[6]);
  std::array<Tensor, 2> r;
  unlocked([&] { r[0] = cp4_backward_data(x, ft, fc, fy, fx, pad, (int)flags, &r[1]); });
  return wrap_tuple(r);
  END_HANDLE_TH_ERRORS
}
PYFN(py_cp4_forward_backward_data) {
  HANDLE_TH_ERRORS
  count_args(n, 9);
  const Tensor &x = tensor_arg(a[0], "Input"), &du = tensor_arg(a[1], "Upstream"), &ft = tensor_arg(a[2], "FT"),
               &fc = tensor_arg(a[3], "FC"), &fy = tensor_arg(a[4], "FY"), &fx = tensor_arg(a[5], "FX");
  const int64_t pad = int_arg(a[6]), flags = int_arg(a[7]);
  const int save = PyObject_IsTrue(a[8]);
  if (save < 0) throw python_error();
  std::array<Tensor, 4> r;
  unlocked([&] {
    const Conv c(x, "Input", ft, fc, fy, fx, pad, false);
    const Tensor dU = dev(du, "Upstream", c.in);
    c.check_upstream(dU, "Upstream must be [N, T, H, W]");
    const c10::cuda::OptionalCUDAGuard guard(c.in.device());
    r[0] = c.out_like(c.s.T);
    r[1] = c.out_like(c.s.C);
    if (save) {
      r[2] = c.out_like(c.s.Rank);
      r[3] = c.out_like(c.s.Rank);
    }
    ok(b200cp_cp4_fwd_bwd_data(&c.s, cp(c.in), cp(dU), cp(c.FT), cp(c.FC), cp(c.FY), cp(c.FX), mp(r[0]), mp(r[1]),
                               save ? mp(r[2]) : nullptr, save ? mp(r[3]) : nullptr, stream(c.in), (int)flags));
  });
  return save ? wrap_tuple(r) : wrap_tuple(std::array<Tensor, 2>{r[0], r[1]});
  END_HANDLE_TH_ERRORS
}
PYFN(py_cp4_backward_filter) {
  HANDLE_TH_ERRORS
  count_args(n, 9);
  const Tensor &du = tensor_arg(a[0], "dLdO"), &x = tensor_arg(a[1], "In"), &ft = tensor_arg(a[2], "FT"),
               &fc = tensor_arg(a[3], "FC"), &fy = tensor_arg(a[4], "FY"), &fx = tensor_arg(a[5], "FX");
  const int64_t pad = int_arg(a[6]), flags = int_arg(a[7]);
  const int packed = PyObject_IsTrue(a[8]);
  if (packed < 0) throw python_error();
  b200cp_tensor_shape s;
  Tensor dK = unlocked([&] { return cp4_backward_filter(du, x, ft, fc, fy, fx, pad, (int)flags, &s); });
  return packed ? wrap(dK) : wrap_tuple(split4(dK, s));
  END_HANDLE_TH_ERRORS
}
PYFN(py_cp4_backward_filter_saved) {
  HANDLE_TH_ERRORS
  count_args(n, 10);
  const Tensor &du = tensor_arg(a[0], "dLdO"), &x = tensor_arg(a[1], "In"), &p = tensor_arg(a[2], "P"),
               &q = tensor_arg(a[3], "Q"), &ft = tensor_arg(a[4], "FT"), &fc = tensor_arg(a[5], "FC"),
               &fy = tensor_arg(a[6], "FY"), &fx = tensor_arg(a[7], "FX");
  const int64_t pad = int_arg(a[8]), flags = int_arg(a[9]);
  b200cp_tensor_shape s;
  Tensor dK = unlocked([&] { return cp4_backward_filter_saved(du, x, p, q, ft, fc, fy, fx, pad, (int)flags, &s); });
  return wrap_tuple(split4(dK, s));
  END_HANDLE_TH_ERRORS
}
PYFN(py_cp4_step) {
  HANDLE_TH_ERRORS
  count_args(n, 8);
  const Tensor &x = tensor_arg(a[0], "X"), &du = tensor_arg(a[1], "dU"), &ft = tensor_arg(a[2], "FT"),
               &fc = tensor_arg(a[3], "FC"), &fy = tensor_arg(a[4], "FY"), &fx = tensor_arg(a[5], "FX");
  const int64_t pad = int_arg(a[6]), flags = int_arg(a[7]);
  std::array<Tensor, 3> r;
  unlocked([&] {
    const Conv c(x, "X", ft, fc, fy, fx, pad, false);
    const Tensor dU = dev(du, "dU", c.in);
    c.check_upstream(dU, "dU must be [N,T,H,W]");
    const c10::cuda::OptionalCUDAGuard guard(c.in.device());
    const b200cp_tensor_shape& s = c.s;
    r[0] = c.out_like(s.T);
    r[1] = c.out_like(s.C);
    r[2] = empty({(int64_t)(s.T + s.C + s.Y + s.X) * s.Rank}, c.in);
    Tensor ws = workspace(b200cp_cp4_step_workspace_bytes(&s, (int)flags), c.in);
    ok(b200cp_cp4_step(&s, cp(c.in), cp(dU), cp(c.FT), cp(c.FC), cp(c.FY), cp(c.FX), mp(r[0]), mp(r[1]), mp(r[2]), mp(ws),
                       ws_bytes(ws), stream(c.in), (int)flags));
  });
  return wrap_tuple(r);
  END_HANDLE_TH_ERRORS
}
PYFN(py_cp3_forward) {
  HANDLE_TH_ERRORS
  count_args(n, 6);
  const Tensor &x = tensor_arg(a[0], "Input"), &kt = tensor_arg(a[1], "KT"), &kcin = tensor_arg(a[2], "KCin"),
               &kc = tensor_arg(a[3], "KC");
  const int64_t pad = int_arg(a[4]), flags = int_arg(a[5]);
  return wrap(unlocked([&] { return cp3_forward(x, kt, kcin, kc, pad, (int)flags); }));
  END_HANDLE_TH_ERRORS
}
PYFN(py_cp3_backward_data) {
  HANDLE_TH_ERRORS
  count_args(n, 6);
  const Tensor &x = tensor_arg(a[0], "Upstream"), &kt = tensor_arg(a[1], "KT"), &kcin = tensor_arg(a[2], "KCin"),
               &kc = tensor_arg(a[3], "KC");
  const int64_t pad = int_arg(a[4]), flags = int_arg(a[5]);
  return wrap(unlocked([&] { return cp3_backward_data(x, kt, kcin, kc, pad, (int)flags); }));
  END_HANDLE_TH_ERRORS
}
PYFN(py_cp3_backward_filter) {
  HANDLE_TH_ERRORS
  count_args(n, 7);
  const Tensor &du = tensor_arg(a[0], "dLdO"), &x = tensor_arg(a[1], "In"), &kt = tensor_arg(a[2], "KT"),
               &kcin = tensor_arg(a[3], "KCin"), &kc = tensor_arg(a[4], "KC");
  const int64_t pad = int_arg(a[5]), flags = int_arg(a[6]);
  return wrap_tuple(unlocked([&] { return cp3_backward_filter(du, x, kt, kcin, kc, pad, (int)flags); }));
  END_HANDLE_TH_ERRORS
}
// (flags, input, kernelc, kernel0, kernel1, ...)
PYFN(py_rcp_forward) {
  HANDLE_TH_ERRORS
  TORCH_CHECK_TYPE(n >= 4, "conv2d_rcp_fused_nchw needs an input, at least one kernel and kernelc");
  const int64_t flags = int_arg(a[0]);
  const Tensor &u = tensor_arg(a[1], "input"), &kc = tensor_arg(a[2], "kernelc");
  const std::vector<Tensor> A = tensor_args(a + 3, n - 3);
  return wrap(unlocked([&] { return rcp_forward(u, A, kc, (int)flags); }));
  END_HANDLE_TH_ERRORS
}
// (flags, need_dx, need_dw, input, dV, kernelc, kernel0, ...)
PYFN(py_rcp_backward) {
  HANDLE_TH_ERRORS
  TORCH_CHECK_TYPE(n >= 7, "rcp_conv2d_backward needs an input, dV, at least one kernel and kernelc");
  const int64_t flags = int_arg(a[0]);
  const int need_dx = PyObject_IsTrue(a[1]), need_dw = PyObject_IsTrue(a[2]);
  if (need_dx < 0 || need_dw < 0) throw python_error();
  const Tensor &u = tensor_arg(a[3], "input"), &dv = tensor_arg(a[4], "dV"), &kc = tensor_arg(a[5], "kernelc");
  const std::vector<Tensor> A = tensor_args(a + 6, n - 6);
  const FactorGrads g = unlocked([&] { return rcp_backward(u, dv, A, kc, (int)flags, need_dx, need_dw); });
  PyObject* r = PyTuple_New(3);
  if (!r) throw python_error();
  PyTuple_SET_ITEM(r, 0, wrap(g.dx));
  if (need_dw) {
    PyTuple_SET_ITEM(r, 1, wrap_list(g.df));
  } else {
    Py_INCREF(Py_None);
    PyTuple_SET_ITEM(r, 1, Py_None);
  }
  PyTuple_SET_ITEM(r, 2, wrap(g.ds));
  return r;
  END_HANDLE_TH_ERRORS
}
// (flags, input, kernel0, ...)
PYFN(py_dense_forward) {
  HANDLE_TH_ERRORS
  TORCH_CHECK_TYPE(n >= 3, "dense_cp needs an input and at least one kernel");
  const int64_t flags = int_arg(a[0]);
  const Tensor& u = tensor_arg(a[1], "input");
  const std::vector<Tensor> F = tensor_args(a + 2, n - 2);
  return wrap(unlocked([&] { return dense_forward(u, F, (int)flags); }));
  END_HANDLE_TH_ERRORS
}
// (flags, need_dx, need_dw, input, dV, kernel0, ...)
PYFN(py_dense_backward) {
  HANDLE_TH_ERRORS
  TORCH_CHECK_TYPE(n >= 6, "dense_cp_backward needs an input, dV and at least one kernel");
  const int64_t flags = int_arg(a[0]);
  const int need_dx = PyObject_IsTrue(a[1]), need_dw = PyObject_IsTrue(a[2]);
  if (need_dx < 0 || need_dw < 0) throw python_error();
  const Tensor &u = tensor_arg(a[3], "input"), &dv = tensor_arg(a[4], "dV");
  const std::vector<Tensor> F = tensor_args(a + 5, n - 5);
  const FactorGrads g = unlocked([&] { return dense_backward(u, dv, F, (int)flags, need_dx, need_dw); });
  PyObject* r = PyTuple_New(2);
  if (!r) throw python_error();
  PyTuple_SET_ITEM(r, 0, wrap(g.dx));
  if (need_dw) {
    PyTuple_SET_ITEM(r, 1, wrap_list(g.df));
  } else {
    Py_INCREF(Py_None);
    PyTuple_SET_ITEM(r, 1, Py_None);
  }
  return r;
  END_HANDLE_TH_ERRORS
}

PYFN(py_cp4_apply) {
  HANDLE_TH_ERRORS
  TORCH_CHECK_TYPE(n >= 5 && n <= 7, "CP4Conv2dFunction.apply(x, FT, FC, FY, FX, pad=1, flags=0)");
  const Tensor &x = tensor_arg(a[0], "Input"), &ft = tensor_arg(a[1], "FT"), &fc = tensor_arg(a[2], "FC"),
               &fy = tensor_arg(a[3], "FY"), &fx = tensor_arg(a[4], "FX");
  const int64_t pad = n > 5 ? int_arg(a[5]) : 1, flags = n > 6 ? int_arg(a[6]) : 0;
  return wrap(unlocked([&] { return CP4Node::apply(x, ft, fc, fy, fx, pad, flags, at::GradMode::is_enabled()); }));
  END_HANDLE_TH_ERRORS
}
PYFN(py_cp3_apply) {
  HANDLE_TH_ERRORS
  TORCH_CHECK_TYPE(n >= 4 && n <= 5, "CP3Conv2dFunction.apply(x, KT, KCin, KC, pad=1)");
  const Tensor &x = tensor_arg(a[0], "Input"), &kt = tensor_arg(a[1], "KT"), &kcin = tensor_arg(a[2], "KCin"),
               &kc = tensor_arg(a[3], "KC");
  const int64_t pad = n > 4 ? int_arg(a[4]) : 1;
  return wrap(unlocked([&] { return CP3Node::apply(x, kt, kcin, kc, pad, at::GradMode::is_enabled()); }));
  END_HANDLE_TH_ERRORS
}
PYFN(py_rcp_apply) {
  HANDLE_TH_ERRORS
  TORCH_CHECK_TYPE(n >= 3, "RCPConv2dFunction.apply(x, KC, K0, K1, ...)");
  const Tensor &x = tensor_arg(a[0], "input"), &kc = tensor_arg(a[1], "kernelc");
  const std::vector<Tensor> A = tensor_args(a + 2, n - 2);
  return wrap(unlocked([&] { return RCPNode::apply(x, kc, at::TensorList(A)); }));
  END_HANDLE_TH_ERRORS
}
PYFN(py_dense_apply) {
  HANDLE_TH_ERRORS
  TORCH_CHECK_TYPE(n >= 2, "CPDenseFunction.apply(x, K0, K1, ...)");
  const Tensor& x = tensor_arg(a[0], "input");
  const std::vector<Tensor> F = tensor_args(a + 1, n - 1);
  return wrap(unlocked([&] { return DenseNode::apply(x, at::TensorList(F)); }));
  END_HANDLE_TH_ERRORS
}
PyObject* py_set_error_class(PyObject*, PyObject* cls) {
  Py_XINCREF(cls);
  Py_XDECREF(g_error_class);
  g_error_class = cls;
  Py_RETURN_NONE;
}

#define FAST(name) {#name, (PyCFunction)(void (*)(void))py_##name, METH_FASTCALL, nullptr}
PyMethodDef g_methods[] = {FAST(cp4_forward), FAST(cp4_forward_save), FAST(cp4_backward_data), FAST(cp4_backward_data_save),
                           FAST(cp4_forward_backward_data), FAST(cp4_backward_filter), FAST(cp4_backward_filter_saved),
                           FAST(cp4_step), FAST(cp3_forward), FAST(cp3_backward_data), FAST(cp3_backward_filter),
                           FAST(rcp_forward), FAST(rcp_backward), FAST(dense_forward), FAST(dense_backward),
                           FAST(cp4_apply), FAST(cp3_apply), FAST(rcp_apply), FAST(dense_apply),
                           {"set_error_class", py_set_error_class, METH_O, nullptr},
                           {nullptr, nullptr, 0, nullptr}};
PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "_C", "native operator bindings", -1, g_methods, nullptr, nullptr, nullptr,
                        nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__C(void) { return PyModule_Create(&g_module); }
