// Which form of the reshaped-CP conv and the CP dense layer runs: the factored register-tiled kernels, or the weight
// multiplied out and one product with it.
#include <algorithm>

#include "common.cuh"

namespace b200cp {
namespace {

long prod(const int* d, int n) {
  long p = 1;
  for (int k = 0; k < n; ++k) p *= d[k];
  return p;
}

// Estimated times in seconds.  Rates are what the kernels measured on a B200: multiply-adds per second of the small FFMA
// products and of the register-tiled factored kernels at their own shapes; the multiplied-out form has one launch more.
constexpr double kSmallGemmRate = 15e12, kSmallConvRate = 14e12, kDenseFastRate = 21e12, kRcpFastRate = 11e12;
constexpr double kLaunch = 3e-6;

bool is_fast_dense(int order, const int* a, const int* b) {
  if (order != 4) return false;
  for (int k = 0; k < 4; ++k)
    if (a[k] != 8 || b[k] != 8) return false;
  return true;
}
bool is_fast_rcp(int order, const int* a, const int* b, int FH, int FW) {
  return order == 3 && FH == 3 && FW == 3 && a[0] == 4 && b[0] == 4 && a[1] == 8 && b[1] == 8 && a[2] == 8 && b[2] == 8;
}

// the weight as kron_weight_launch writes it
size_t weight_floats(int order, const int* idims, const int* odims, int taps, bool transposed) {
  const long slow = prod(transposed ? odims : idims, order), fast = prod(transposed ? idims : odims, order);
  return (size_t)slow * taps * kron_weight_ld((int)fast);
}

enum class Form { kFactored, kSmall };

Form dense_form(int B, int order, const int* idims, const int* odims, int R) {
  const double I = (double)prod(idims, order), O = (double)prod(odims, order);
  if (I * O > 1e9) return Form::kFactored;
  if (is_fast_dense(order, idims, odims)) {
    const double fact = (double)B * R * 4 * 4096 * 8;
    if (fact / kDenseFastRate < (double)B * I * O / kSmallGemmRate + kLaunch) return Form::kFactored;
  }
  return Form::kSmall;
}

Form rcp_form(int N, int H, int W, int order, const int* cdims, const int* tdims, int R, int FH, int FW) {
  if (FH != 3 || FW != 3) return Form::kFactored;
  const double C = (double)prod(cdims, order), T = (double)prod(tdims, order), px = (double)N * H * W;
  if (C * T * 9 > 1e9) return Form::kFactored;
  if (is_fast_rcp(order, cdims, tdims, FH, FW)) {
    const double fact = px * R * (256.0 * 9 + 256.0 * 20);
    if (fact / kRcpFastRate < px * C * T * 9 / kSmallConvRate + kLaunch) return Form::kFactored;
  }
  return Form::kSmall;
}

}  // namespace

size_t dense_product_workspace(int B, int order, const int* idims, const int* odims, int R, bool transposed) {
  if (check_kron_modes(order, idims, odims, R, "dense_cp") || B < 1) return 0;
  if (dense_form(B, order, idims, odims, R) == Form::kFactored) return 0;
  return align_up(weight_floats(order, idims, odims, 1, transposed) * sizeof(float), 256);
}

int dense_product_launch(int B, int order, const int* idims, const int* odims, int R, const float* X,
                         const float* const* F, float* Y, bool transposed, void* ws, size_t ws_bytes, cudaStream_t st) {
  if (int rc = check_kron_modes(order, idims, odims, R, "dense_cp")) return rc;
  if (B < 1) return fail(B200CP_ERR_INVALID_ARG, "dense_cp: batch must be positive");
  const size_t need = dense_product_workspace(B, order, idims, odims, R, transposed);
  if (!need || !ws || ws_bytes < need || (reinterpret_cast<uintptr_t>(ws) & 15))
    return dense_chain_launch(B, order, idims, odims, R, X, F, Y, transposed, st);
  float* Wt = static_cast<float*>(ws);
  if (int rc = kron_weight_launch(order, idims, odims, R, F, nullptr, 1, transposed, Wt, st)) return rc;
  const int I = (int)prod(idims, order), O = (int)prod(odims, order);
  return small_gemm_launch(B, transposed ? I : O, transposed ? O : I, X, Wt, Y, st);
}

size_t rcp_product_workspace(int N, int H, int W, int order, const int* cdims, const int* tdims, int R, int FH, int FW,
                             bool transposed) {
  if (check_kron_modes(order, cdims, tdims, R, "rcp") || N < 1 || H < 1 || W < 1) return 0;
  if (rcp_form(N, H, W, order, cdims, tdims, R, FH, FW) == Form::kFactored) return 0;
  return align_up(weight_floats(order, cdims, tdims, FH * FW, transposed) * sizeof(float), 256);
}

int rcp_product_launch(int N, int H, int W, int order, const int* cdims, const int* tdims, int R, int FH, int FW,
                       const float* X, const float* const* A, const float* S, float* V, bool transposed, void* ws,
                       size_t ws_bytes, cudaStream_t st) {
  if (int rc = check_kron_modes(order, cdims, tdims, R, "rcp")) return rc;
  const size_t need = rcp_product_workspace(N, H, W, order, cdims, tdims, R, FH, FW, transposed);
  if (!need || !ws || ws_bytes < need || (reinterpret_cast<uintptr_t>(ws) & 15))
    return rcp_chain_launch(N, H, W, order, cdims, tdims, R, FH, FW, X, A, S, V, transposed, st);
  float* Wt = static_cast<float*>(ws);
  if (int rc = kron_weight_launch(order, cdims, tdims, R, A, S, FH * FW, transposed, Wt, st)) return rc;
  const int C = (int)prod(cdims, order), T = (int)prod(tdims, order);
  return small_conv_launch(N, transposed ? T : C, transposed ? C : T, H, W, X, Wt, V, st);
}

}  // namespace b200cp
