// CP dense layer of order 4: register-tiled kernel on CUDA cores (exact fp32).
//
//   Y[n,(o1,o2,o3,o4)] = sum_r sum_{i1..i4} X[n,(i1,i2,i3,i4)] F1[i1,o1,r] F2[i2,o2,r] F3[i3,o3,r] F4[i4,o4,r]
// (test/layers.py:445-465; the reference's fused kernel, Kernels/dense_cp.cu:4-46, is this sum for one fixed
// order-3 shape).  A CTA owns kS samples; their inputs stay in shared memory for the whole rank loop.  Per rank:
//   phase A  a thread owns one sample, one (i1,i2) pair and half of o4: it contracts i4 -> o4 and i3 -> o3 in
//            registers and writes T[(i1,i2)][(o3,o4)] to shared memory;
//   phase B  a thread owns one sample, one (o3,o4) pair and half of o2: it reads the column T[:, (o3,o4)],
//            contracts i2 -> o2 and i1 -> o1 and adds into its [o1][o2/2] accumulators, which stay in
//            registers across all ranks.
// The data gradient is the same kernel with the factors read transposed.
#include <algorithm>
#include <cstdlib>

#include "common.cuh"

namespace b200cp {

namespace {

struct DenseFastArgs {
  const float* X;
  const float* F[4];
  float* Y;
  int B, R;
  int fsi[4], fso[4];  // element (contracted i, produced o) of factor k at F[k][(i*fsi + o*fso)*R + r]
};

template <int I1, int O1, int I2, int O2, int I3, int O3, int I4, int O4>
struct DenseFastCfg {
  static constexpr int kS = 2, NT = 256;
  static constexpr int QI = I1 * I2, PI = I3 * I4;   // input viewed as [QI][PI]
  static constexpr int QO = O1 * O2, PO = O3 * O4;   // output viewed as [QO][PO]
  static constexpr int XP = PI + 4, TP = PO + 4;     // row pitches: 16-byte rows, conflict-free float4 access
  static constexpr int OFF2 = I1 * O1, OFF3 = OFF2 + I2 * O2, OFF4 = OFF3 + I3 * O3, FPR = OFF4 + I4 * O4;
  static constexpr int H4 = O4 / 2, H2 = O2 / 2;
  static_assert(QI * 2 * kS == NT && PO * 2 * kS == NT, "one thread per (sample, pair, half)");
  static_assert(PI % 4 == 0 && PO % 4 == 0 && O1 % 4 == 0 && O3 % 4 == 0 && H4 == 4 && H2 == 4 && I4 % 4 == 0 && FPR % 4 == 0,
                "vector accesses");
  static size_t smem_bytes(int R) { return sizeof(float) * ((size_t)R * FPR + kS * QI * XP + kS * QI * TP); }
};

template <int I1, int O1, int I2, int O2, int I3, int O3, int I4, int O4>
__global__ void __launch_bounds__(256, 2) dense4_fast_kernel(const DenseFastArgs a) {
  using K = DenseFastCfg<I1, O1, I2, O2, I3, O3, I4, O4>;
  extern __shared__ __align__(16) float sm[];
  float* Fs = sm;                                  // [R][F1 | F2 | F3 | F4], each [i][o]
  float* Xs = Fs + (size_t)a.R * K::FPR;           // [kS][QI][XP]
  float* Ts = Xs + K::kS * K::QI * K::XP;          // [kS][QI][TP]
  const int tid = threadIdx.x;
  const int n0 = blockIdx.x * K::kS;

  for (int i = tid; i < a.R * K::FPR; i += K::NT) {
    const int r = i / K::FPR, e = i - r * K::FPR;
    int k, q, od;
    if (e < K::OFF2) { k = 0; q = e; od = O1; }
    else if (e < K::OFF3) { k = 1; q = e - K::OFF2; od = O2; }
    else if (e < K::OFF4) { k = 2; q = e - K::OFF3; od = O3; }
    else { k = 3; q = e - K::OFF4; od = O4; }
    const int ii = q / od, oo = q - ii * od;
    Fs[i] = __ldg(a.F[k] + (size_t)(ii * a.fsi[k] + oo * a.fso[k]) * a.R + r);
  }
  {
    constexpr int IN = K::QI * K::PI;
    for (int i = tid; i < K::kS * IN / 4; i += K::NT) {
      const int s = i / (IN / 4), e = (i - s * (IN / 4)) * 4;
      const int q = e / K::PI, k = e - q * K::PI;
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      if (n0 + s < a.B) v = __ldg(reinterpret_cast<const float4*>(a.X + (size_t)(n0 + s) * IN + e));
      *reinterpret_cast<float4*>(Xs + (size_t)(s * K::QI + q) * K::XP + k) = v;
    }
  }
  const int half = tid / (K::NT / 2);          // warp-uniform
  const int s = (tid / K::QI) % K::kS;
  const int qa = tid % K::QI;                  // phase A: (i1,i2) pair;  phase B: (o3,o4) pair (QI == PO threads)
  float acc[O1][K::H2];
#pragma unroll
  for (int i = 0; i < O1; ++i)
#pragma unroll
    for (int j = 0; j < K::H2; ++j) acc[i][j] = 0.f;
  __syncthreads();

  const float* xrow = Xs + (size_t)(s * K::QI + qa) * K::XP;
  float* trow = Ts + (size_t)(s * K::QI + qa) * K::TP;
  const float* tcol = Ts + (size_t)s * K::QI * K::TP + qa;

  for (int r = 0; r < a.R; ++r) {
    const float* F = Fs + (size_t)r * K::FPR;
    // ---- phase A: modes 4 and 3 ----
    {
      float a4[I4][K::H4];
#pragma unroll
      for (int i4 = 0; i4 < I4; ++i4) {
        const float4 v = *reinterpret_cast<const float4*>(F + K::OFF4 + i4 * O4 + half * K::H4);
        a4[i4][0] = v.x; a4[i4][1] = v.y; a4[i4][2] = v.z; a4[i4][3] = v.w;
      }
      float t[O3][K::H4];
#pragma unroll
      for (int o = 0; o < O3; ++o)
#pragma unroll
        for (int j = 0; j < K::H4; ++j) t[o][j] = 0.f;
#pragma unroll
      for (int i3 = 0; i3 < I3; ++i3) {
        float x[I4];
#pragma unroll
        for (int v4 = 0; v4 < I4 / 4; ++v4) {
          const float4 v = *reinterpret_cast<const float4*>(xrow + i3 * I4 + v4 * 4);
          x[v4 * 4] = v.x; x[v4 * 4 + 1] = v.y; x[v4 * 4 + 2] = v.z; x[v4 * 4 + 3] = v.w;
        }
        float tmp[K::H4];
#pragma unroll
        for (int j = 0; j < K::H4; ++j) tmp[j] = 0.f;
#pragma unroll
        for (int i4 = 0; i4 < I4; ++i4)
#pragma unroll
          for (int j = 0; j < K::H4; ++j) tmp[j] = fmaf(x[i4], a4[i4][j], tmp[j]);
#pragma unroll
        for (int v4 = 0; v4 < O3 / 4; ++v4) {
          const float4 w = *reinterpret_cast<const float4*>(F + K::OFF3 + i3 * O3 + v4 * 4);
          const float w3[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
          for (int u = 0; u < 4; ++u)
#pragma unroll
            for (int j = 0; j < K::H4; ++j) t[v4 * 4 + u][j] = fmaf(w3[u], tmp[j], t[v4 * 4 + u][j]);
        }
      }
#pragma unroll
      for (int o = 0; o < O3; ++o)
        *reinterpret_cast<float4*>(trow + o * O4 + half * K::H4) = make_float4(t[o][0], t[o][1], t[o][2], t[o][3]);
    }
    __syncthreads();
    // ---- phase B: modes 2 and 1 ----
    {
      float a2[I2][K::H2];
#pragma unroll
      for (int i2 = 0; i2 < I2; ++i2) {
        const float4 v = *reinterpret_cast<const float4*>(F + K::OFF2 + i2 * O2 + half * K::H2);
        a2[i2][0] = v.x; a2[i2][1] = v.y; a2[i2][2] = v.z; a2[i2][3] = v.w;
      }
#pragma unroll 2
      for (int i1 = 0; i1 < I1; ++i1) {
        float t[I2];
#pragma unroll
        for (int i2 = 0; i2 < I2; ++i2) t[i2] = tcol[(size_t)(i1 * I2 + i2) * K::TP];
        float tmp[K::H2];
#pragma unroll
        for (int j = 0; j < K::H2; ++j) tmp[j] = 0.f;
#pragma unroll
        for (int i2 = 0; i2 < I2; ++i2)
#pragma unroll
          for (int j = 0; j < K::H2; ++j) tmp[j] = fmaf(t[i2], a2[i2][j], tmp[j]);
#pragma unroll
        for (int v4 = 0; v4 < O1 / 4; ++v4) {
          const float4 w = *reinterpret_cast<const float4*>(F + i1 * O1 + v4 * 4);
          const float w1[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
          for (int u = 0; u < 4; ++u)
#pragma unroll
            for (int j = 0; j < K::H2; ++j) acc[v4 * 4 + u][j] = fmaf(w1[u], tmp[j], acc[v4 * 4 + u][j]);
        }
      }
    }
    __syncthreads();
  }

  if (n0 + s < a.B) {
    float* y = a.Y + (size_t)(n0 + s) * K::QO * K::PO + qa;
#pragma unroll
    for (int o1 = 0; o1 < O1; ++o1)
#pragma unroll
      for (int j = 0; j < K::H2; ++j) y[(size_t)(o1 * O2 + half * K::H2 + j) * K::PO] = acc[o1][j];
  }
}

}  // namespace

using DenseFast = DenseFastCfg<8, 8, 8, 8, 8, 8, 8, 8>;

// The shape the register-tiled kernel is compiled for (order 4, every mode 8 -> 8), at a rank whose factors fit beside
// the samples in shared memory.
bool dense_fast_takes(int order, const int* din, const int* dout, int R, const DeviceInfo& di) {
  if (order != 4) return false;
  for (int k = 0; k < 4; ++k)
    if (din[k] != 8 || dout[k] != 8) return false;
  return DenseFast::smem_bytes(R) <= (size_t)di.smem_optin && !getenv("B200CP_NO_FAST");
}

// Estimated microseconds: waves of CTAs, per rank 1.98 us alone on an SM and 3.5 us where two share one (up to about 47 ranks).
// Measured: 1024 samples R = 16 117, R = 64 516; 4096 samples R = 16 402, R = 32 803, R = 64 1831; one sample R = 64 129.
double dense_fast_us(int B, int R, const DeviceInfo& di) {
  const int ctas = ceil_div(B, DenseFast::kS);
  const bool two = ctas > di.sm_count && 2 * (DenseFast::smem_bytes(R) + 1024) <= 228 * 1024;
  return 3.0 + (double)R * (two ? 3.5 * ceil_div(ctas, 2 * di.sm_count) : 1.98 * ceil_div(ctas, di.sm_count));
}

// for layers dense_fast_takes
int dense_fast_launch(int B, const int* fsi, const int* fso, int R, const float* X, const float* const* F, float* Y,
                      cudaStream_t st) {
  DenseFastArgs a{};
  a.X = X; a.Y = Y; a.B = B; a.R = R;
  for (int k = 0; k < 4; ++k) { a.F[k] = F[k]; a.fsi[k] = fsi[k]; a.fso[k] = fso[k]; }
  const size_t smem = DenseFast::smem_bytes(R);
  auto kern = dense4_fast_kernel<8, 8, 8, 8, 8, 8, 8, 8>;
  B200CP_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  kern<<<(unsigned)ceil_div(B, DenseFast::kS), DenseFast::NT, smem, st>>>(a);
  B200CP_LAUNCH_OK("dense4_fast_kernel");
  return B200CP_OK;
}

}  // namespace b200cp
