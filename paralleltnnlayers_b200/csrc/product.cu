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

bool multiplies_out(size_t floats, double entries, double kron_us, double factored_us) {
  if (factored_us < 0) return entries <= kMostEntries;
  return factored_us > kron_us && floats * sizeof(float) <= kMostWeight;
}

}  // namespace

size_t dense_product_workspace(int B, int order, const int* idims, const int* odims, int R, bool transposed) {
  if (check_kron_modes(order, idims, odims, R, "dense_cp") || B < 1) return 0;
  if (B > 0x7fffffff - 64) return 0;
  const size_t floats = weight_floats(order, idims, odims, 1, transposed);
  const double kron = dense_kron_us(B, order, idims, odims, R, transposed);
  const double entries = (double)prod(idims, order) * prod(odims, order);
  if (!multiplies_out(floats, entries, kron, dense_factored_us(B, order, idims, odims, R, transposed, kron))) return 0;
  return align_up(floats * sizeof(float), 256);
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
  if (FH != 3 || FW != 3) return 0;
  const size_t floats = weight_floats(order, cdims, tdims, 9, transposed);
  const double kron = rcp_kron_us(N, H, W, order, cdims, tdims, R, transposed);
  const double entries = 9.0 * prod(cdims, order) * prod(tdims, order);
  if (!multiplies_out(floats, entries, kron, rcp_factored_us(N, H, W, order, cdims, tdims, R, FH, FW, transposed, kron))) return 0;
  return align_up(floats * sizeof(float), 256);
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
