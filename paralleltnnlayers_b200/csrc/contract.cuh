// Contraction of a dense gradient with the factors: shared by contract_peel.cu (mode by mode) and contract_halves.cu.
#pragma once

#include "common.cuh"

namespace b200cp {

struct PeelMode {
  int nc, nt;      // p = c * nt + t
  long gc, gt;     // offset in G per c and per t
  const float* vec;  // [nc * nt][R]
};

bool halves_take(int L, const int* sizes, int R, bool has_s);
size_t halves_scratch_floats(int L, const int* sizes, int R);
int halves_launch(int L, const PeelMode* modes, int R, const float* G, float* const* grads, float* scratch, cudaStream_t st);
int halves_device_status(int* out);

}  // namespace b200cp
