// Which form of the reshaped-CP conv and the CP dense layer runs: the factored register-tiled kernels, or the weight
// multiplied out and one product with it.
#include <algorithm>
#include <climits>

#include "b200cp_test.h"
#include "common.cuh"

namespace b200cp {
namespace {

long prod(const int* d, int n) {
  long p = 1;
  for (int k = 0; k < n; ++k) p *= d[k];
  return p;
}

// the weight as kron_weight_launch writes it
size_t weight_floats(int order, const int* idims, const int* odims, int taps, bool transposed) {
  const long slow = prod(transposed ? odims : idims, order), fast = prod(transposed ? idims : odims, order);
  return (size_t)slow * taps * kron_weight_ld((int)fast);
}

// The form with the smaller estimated time runs (what the estimates are made of, and how good they are, stands beside
// them: chain_kernel, the register-tiled kernels, kron_small.cu).  Either side of the line, us, factored / multiplied out:
//   4096 samples of 16x16x16 -> 16x16x16   R = 4 386 / 3823    R = 16 1102 / 3830    R = 64 4006 / 3880    R = 256 15551 / 4095
//   64 samples of the same                 R = 4 49 / 125      R = 16 152 / 134
//   4096 samples of 10x10x10 -> 10x10x10   R = 4 127 / 257     R = 16 401 / 259
//   one sample of 8x8x8x8 -> 8x8x8x4       R = 4 39 / 40       R = 16 131 / 45
//   32 images of 28x28, 16x16 -> 16x16     R = 4 616 / 968     R = 8 1130 / 968;   4x8x8 -> 4x8x8 R = 64 894 / 973
//   8 images of 32x32, 6x6x6 -> 6x6x6      R = 4 161 / 275     R = 8 300 / 275
// A weight of more than kMostWeight bytes of scratch is multiplied out only for what the factored form does not take (it does
// not fit on chip), up to kMostEntries.
constexpr size_t kMostWeight = size_t{256} << 20;
constexpr double kMostEntries = 1e9;

// With fewer ranks the factored kernels' sums are short enough to round less than the tensor product does (R = 4, 4096 samples of
// 10x10x10 -> 10x10x10: 1.4e-7 of the result against 1.55e-7), and they are not far behind or ahead.
constexpr int kLeastRanks = 8;
// Below this many multiply-adds the FFMA product takes less than the tensor one's fixed 20 us (512 x 512 -> 512: 19 us), and the
// search for its tiles is not worth the host's time.
constexpr double kLeastMacs = 1e8;
// The tensor product holds hi / lo planes of the weight and of the activations: as much again as the layer's input.
constexpr size_t kMostPlanes = size_t{1} << 30;
bool tensor_may(int flags, int R, double macs) {
  if (!(flags & B200CP_TENSOR_PRODUCTS)) return false;
  return gemm_tc_mode() == 2 || (R >= kLeastRanks && macs >= kLeastMacs);
}

enum class Form { factored, ffma, tensor, inside };   // inside: ffma, the weight formed by the product's CTAs

// `floats`: of the weight; a form's time is negative where it does not take the sizes
Form pick(size_t floats, double entries, double ffma_us, double tensor_us, double factored_us) {
  if (tensor_us >= 0 && gemm_tc_mode() == 2) return Form::tensor;
  const bool tensor = tensor_us >= 0 && tensor_us < ffma_us && floats * sizeof(float) <= kMostWeight;
  const Form out = tensor ? Form::tensor : Form::ffma;
  if (factored_us < 0) return entries <= kMostEntries ? out : Form::factored;
  return factored_us > (tensor ? tensor_us : ffma_us) && floats * sizeof(float) <= kMostWeight ? out : Form::factored;
}

struct DensePlan {
  Form form;
  int K, N;               // inputs and outputs of the product
  size_t weight, bytes;   // floats of the weight, bytes of the workspace
};
// the tensor form reads the weight with the other side contiguous
DensePlan dense_plan(int B, int order, const int* idims, const int* odims, int R, bool transposed, int flags) {
  DensePlan p{};
  p.K = (int)prod(transposed ? odims : idims, order);
  p.N = (int)prod(transposed ? idims : odims, order);
  const double ffma = dense_kron_us(B, order, idims, odims, R, transposed);
  const bool may = tensor_may(flags, R, (double)B * p.K * p.N) && dense_tc_takes();
  const KronWeight w{order, idims, odims, R, nullptr, nullptr, !transposed, false};
  const size_t planes = may ? align_up(dense_tc_scratch_floats(B, p.K, p.N, w) * sizeof(float), 256) : 0;
  const double tensor = may && planes <= kMostPlanes ? dense_tc_us(B, p.K, p.N, w) : -1;
  const double least = tensor >= 0 ? std::min(ffma, tensor) : ffma;
  p.weight = weight_floats(order, idims, odims, 1, transposed);
  p.form = pick(p.weight, (double)p.K * p.N, ffma, tensor, dense_factored_us(B, order, idims, odims, R, transposed, least));
  if (p.form == Form::tensor) {
    p.bytes = planes;
  } else if (p.form == Form::ffma) {
    p.bytes = align_up(p.weight * sizeof(float), 256);
  }
  return p;
}

DensePlan rcp_plan(int N, int H, int W, int order, const int* cdims, const int* tdims, int R, int FH, int FW, bool transposed,
                   int flags) {
  DensePlan p{};
  if (FH != 3 || FW != 3) return p;
  p.K = (int)prod(transposed ? tdims : cdims, order);
  p.N = (int)prod(transposed ? cdims : tdims, order);
  bool inside = false;
  const double ffma = rcp_kron_us(N, H, W, order, cdims, tdims, R, transposed, &inside);
  const bool may = tensor_may(flags, R, 9.0 * N * H * W * p.K * p.N) && conv_tc_takes(N, p.K, p.N, H, W);
  const size_t planes = may ? align_up(conv_tc_scratch_floats(N, p.K, p.N, H, W) * sizeof(float), 256) : 0;
  const double tensor = may && planes <= kMostPlanes
                            ? kron_weight_us(order, cdims, tdims, R, 9, !transposed) + conv_tc_us(N, p.K, p.N, H, W) : -1;
  const double least = tensor >= 0 ? std::min(ffma, tensor) : ffma;
  p.weight = weight_floats(order, cdims, tdims, 9, transposed);
  p.form = pick(p.weight, 9.0 * p.K * p.N, ffma, tensor,
                rcp_factored_us(N, H, W, order, cdims, tdims, R, FH, FW, transposed, least));
  if (p.form == Form::tensor) {
    p.bytes = planes;
  } else if (p.form == Form::ffma) {
    // (formed inside nothing is stored; but a call without a workspace runs the factored kernels, so this one asks for some)
    p.bytes = inside ? 256 : align_up(p.weight * sizeof(float), 256);
    if (inside) p.form = Form::inside;
  }
  return p;
}

bool fits(const DensePlan& p, const void* ws, size_t ws_bytes) {
  return p.bytes && ws && ws_bytes >= p.bytes && !(reinterpret_cast<uintptr_t>(ws) & 15);
}
}  // namespace

size_t dense_product_workspace(int B, int order, const int* idims, const int* odims, int R, bool transposed, int flags) {
  if (check_kron_modes(order, idims, odims, R, "dense_cp") || B < 1) return 0;
  if (B > 0x7fffffff - 64) return 0;
  return dense_plan(B, order, idims, odims, R, transposed, flags).bytes;
}

int dense_product_launch(int B, int order, const int* idims, const int* odims, int R, const float* X,
                         const float* const* F, float* Y, bool transposed, void* ws, size_t ws_bytes, cudaStream_t st,
                         int flags) {
  if (int rc = check_kron_modes(order, idims, odims, R, "dense_cp")) return rc;
  if (B < 1) return fail(B200CP_ERR_INVALID_ARG, "dense_cp: batch must be positive");
  const DensePlan p = B > 0x7fffffff - 64 ? DensePlan{} : dense_plan(B, order, idims, odims, R, transposed, flags);
  if (!fits(p, ws, ws_bytes)) return dense_chain_launch(B, order, idims, odims, R, X, F, Y, transposed, st);
  float* Wt = static_cast<float*>(ws);
  if (p.form == Form::tensor)
    return dense_tc_launch(B, p.K, p.N, X, KronWeight{order, idims, odims, R, F, nullptr, !transposed, false}, Y, Wt, st);
  if (int rc = kron_weight_launch(order, idims, odims, R, F, nullptr, 1, transposed, false, Wt, st)) return rc;
  return small_gemm_launch(B, p.N, p.K, X, Wt, Y, st);
}

size_t rcp_product_workspace(int N, int H, int W, int order, const int* cdims, const int* tdims, int R, int FH, int FW,
                             bool transposed, int flags) {
  if (check_kron_modes(order, cdims, tdims, R, "rcp") || N < 1 || H < 1 || W < 1) return 0;
  return rcp_plan(N, H, W, order, cdims, tdims, R, FH, FW, transposed, flags).bytes;
}

int rcp_product_launch(int N, int H, int W, int order, const int* cdims, const int* tdims, int R, int FH, int FW,
                       const float* X, const float* const* A, const float* S, float* V, bool transposed, void* ws,
                       size_t ws_bytes, cudaStream_t st, int flags) {
  if (int rc = check_kron_modes(order, cdims, tdims, R, "rcp")) return rc;
  const bool sizes = N >= 1 && H >= 1 && W >= 1;
  const DensePlan p = sizes ? rcp_plan(N, H, W, order, cdims, tdims, R, FH, FW, transposed, flags) : DensePlan{};
  if (!fits(p, ws, ws_bytes))
    return rcp_chain_launch(N, H, W, order, cdims, tdims, R, FH, FW, X, A, S, V, transposed, st);
  if (p.form == Form::inside) return small_conv_launch(N, H, W, order, cdims, tdims, R, A, S, transposed, X, nullptr, V, st);
  float* Wt = static_cast<float*>(ws);
  if (p.form == Form::tensor)
    return conv_tc_launch(N, p.K, p.N, H, W, X, KronWeight{order, cdims, tdims, R, A, S, !transposed, transposed}, V, Wt, st);
  return small_conv_launch(N, H, W, order, cdims, tdims, R, A, S, transposed, X, Wt, V, st);
}

}  // namespace b200cp

extern "C" int b200cp_test_rcp_product(int N, int H, int W, int order, const int* cdims, const int* tdims, int R, int transposed, int flags,
                                       int* out) {
  using namespace b200cp;
  if (int rc = check_kron_modes(order, cdims, tdims, R, "rcp")) return rc;
  const DensePlan p = rcp_plan(N, H, W, order, cdims, tdims, R, 3, 3, transposed != 0, flags);
  out[0] = (int)p.form;
  return conv_shares(N, p.K, p.N, H, W, p.form == Form::inside ? R : INT_MAX, out + 1);
}
