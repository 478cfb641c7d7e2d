// Convolutions and factor gradients as products over whole rank planes (cp_planes.cu).
#pragma once

#include "common.cuh"

namespace b200cp {

// What to compute is what has an output pointer: U, dX, the packed factor gradients dK.  The rank planes
// P = K1^T X and Q = K0^T dU ([N][R][H][W]) are read where they are given (P, Q), else computed -- into Psave / Qsave
// where the caller wants them, else into the workspace.
struct PlanesJob {
  const b200cp_tensor_shape* s = nullptr;
  const float *X = nullptr, *dU = nullptr, *K0 = nullptr, *K1 = nullptr;
  const float *KH = nullptr, *KW = nullptr, *KC = nullptr;   // KH and KW, or the free [3][3][R] core
  const float *P = nullptr, *Q = nullptr;
  float *Psave = nullptr, *Qsave = nullptr;
  float *U = nullptr, *dX = nullptr, *dK = nullptr;
};
enum { kPlanesFwd = 1, kPlanesBwd = 2, kPlanesGrads = 4, kPlanesNoP = 8, kPlanesNoQ = 16 };   // NoP / NoQ: given or saved
extern std::atomic<int> g_planes_test;   // b200cp_test_set_planes: which calls take them (abi.cu)
bool planes_supported(const b200cp_tensor_shape& s);
size_t planes_workspace(const b200cp_tensor_shape& s, int parts);
int planes_launch(const PlanesJob& j, void* ws, size_t ws_bytes, cudaStream_t st);
int planes_device_status(int* out);
int planes_forms(const b200cp_tensor_shape& s);   // on the tensor cores: bit 0 one product, 1 two in a launch, 2 the factor gradients

}  // namespace b200cp
